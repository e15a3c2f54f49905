// Dense blocks of K for the hierarchical approximation (hmatrix.cu): the
// per-source records of one patch family on the device and the block
// assembly entry point (assemble.cu).
#pragma once
#include <vector>
#include "ucg_internal.cuh"
#include "okada92.cuh"
#include "nikkhoo15.cuh"

namespace ucg {

// a context workspace of at least `bytes` (its earlier contents are lost)
template <class T>
inline int workspace(ucg_ctx *c, int which, size_t bytes, T **out)
{
    if (c->ws_bytes[which] < bytes) {
        UCG_CUDA(cudaStreamSynchronize(c->stream));
        if (c->ws[which]) cudaFree(c->ws[which]);
        c->ws[which] = nullptr;
        c->ws_bytes[which] = 0;
        const cudaError_t e = cudaMalloc(&c->ws[which], bytes);
        if (e != cudaSuccess) {
            c->ws[which] = nullptr;
            return cuda_fail(c, e, "cudaMalloc(assembly workspace)");
        }
        c->ws_bytes[which] = bytes;
    }
    *out = static_cast<T *>(c->ws[which]);
    return UCG_OK;
}

// a host table into a workspace
template <class T, class H>
inline int workspace_upload(ucg_ctx *c, int which, const std::vector<H> &h, T **out)
{
    const int rc = workspace(c, which, sizeof(H) * h.size(), out);
    if (rc) return rc;
    UCG_CUDA(cudaMemcpyAsync(*out, h.data(), sizeof(H) * h.size(), cudaMemcpyHostToDevice, c->stream));
    return UCG_OK;
}

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

// a dense block: receivers [r0, r0 + nr) by sources [s0, s0 + ns), positions in
// the permuted order; out is row-major (3 nr) x (2 ns), on the device
struct BlockJob {
    double *out;
    int r0, nr, s0, ns;
};

// UCG_E_UNSUPPORTED for volumes or mixed rectangles and triangles
int block_family(const ucg_ctx *c);
// source records of the context's single patch family in the order perm, and
// the receiver table (c->rcv, K's order)
int block_sources_build(ucg_ctx *c, int okada_mode, const std::vector<int> &perm, BlockSources *bs);
// all the blocks in one launch, enqueued on c->stream; perm_d: the device copy of
// perm.  The job list is copied before the call returns.
int assemble_blocks(ucg_ctx *c, const BlockSources &bs, const int *perm_d, const std::vector<BlockJob> &jobs);
// bounding box (lo, hi) and centre of every patch, in K's element order
void element_boxes(const ucg_ctx *c, std::vector<double> &box, std::vector<double> &ctr);

}  // namespace ucg
