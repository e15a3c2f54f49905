// Dense blocks of K for the hierarchical approximation (hmatrix.cu): the
// per-source records of one patch family on the device and the block
// assembly entry point (assemble.cu).
#pragma once
#include <vector>
#include "ucg_internal.cuh"
#include "okada92.cuh"
#include "nikkhoo15.cuh"

namespace ucg {

// device tables of the triangular sources (in the context's workspaces)
struct TriTables {
    const double *rec = nullptr;   // NW_SIZE records, field-major
    const int *edge = nullptr;     // 3 x ns, side-major: 2 edge + (1 where the side runs against the edge)
    const double *ed = nullptr;    // NE_SIZE records of the mesh's unique edges, field-major
    int ns = 0, ne = 0;
};

struct BlockSources {
    int family = 0;          // 0 rectangles, 1 triangles
    int okada_mode = UCG_OKADA_FP64;
    const double *src = nullptr;   // rectangles: SoA source records on the device
    TriTables tri;           // triangles
    int ns = 0;
    OkMed med{};
    NwConst cst{};
};

// records of the context's single patch family and the receiver table (c->rcv);
// UCG_E_UNSUPPORTED for volumes or mixed rectangles and triangles
int block_sources_build(ucg_ctx *c, int okada_mode, BlockSources *bs);
// K rows of receivers ridx[0..nrb) by columns of sources sidx[0..nsb) (device
// element-id arrays) into out, row-major (3 nrb) x (2 nsb); enqueued on c->stream
void assemble_block(ucg_ctx *c, const BlockSources &bs, const int *ridx, int nrb, const int *sidx, int nsb,
                    double *out);
// bounding box (lo, hi) and centre of every patch, in K's element order
void element_boxes(const ucg_ctx *c, std::vector<double> &box, std::vector<double> &ctr);

}  // namespace ucg
