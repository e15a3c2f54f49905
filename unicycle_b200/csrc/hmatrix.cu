// Hierarchical (H-matrix) approximation of K for fault models, built and
// applied on the device.
//
// The reference's MATLAB toolbox runs large models through a hierarchical
// matrix (matlab/+unicycle/+ode/+hmmvp/rateandstate.m:71-143, the hmmvp
// library); the Fortran drivers hold K dense.  Here:
//
//   ordering   patches are permuted by a cluster tree: recursive bisection of
//              their centres along the longest extent of the cluster, down to
//              `leaf` patches; every cluster is a contiguous range of the
//              permutation.
//   blocks     a pair of clusters (tau, sigma) is admissible when
//              max(diam tau, diam sigma) <= eta dist(tau, sigma) (bounding boxes
//              of the patches' vertices) and the block fits the build scratch;
//              admissible pairs become low-rank blocks, pairs of leaves that are
//              not admissible dense blocks, other pairs are split (the non-leaf
//              side, or both).
//   build      each block is assembled densely on the device into scratch by the
//              same pair kernels as K (assemble_blocks), so K itself is never
//              held: N beyond what a dense K fits in HBM works.  A low-rank
//              block is compressed by adaptive cross approximation with partial
//              pivoting (one CTA per block) to relative accuracy eps, then
//              checked against the dense block on a pseudo-random probe
//              vector; a block that fails the check, or whose factors would not
//              be smaller, is kept dense.
//   storage    FP64.  V is stored rank-major (k x n); the rows of U and of the
//              dense blocks are repacked into panels, one per row leaf (of at most 42
//              patches: a tree leaf or a part of one) and chunk of at most 24 KB,
//              each a column-major (rows x columns) slab of one kind, dense or U.
//   product    t = H v on v in the permuted order (every block's columns are a
//              contiguous slice), two launches of k_hm_rows: the first forms
//              z_b = V_b^T v_sigma of the low-rank blocks (one warp per two rank
//              vectors) and, in CTAs between them, the dense chunks; the second
//              the chunks of U.  A CTA copies its chunk's panel into shared memory
//              with one bulk copy (two in the split form) and one thread per row
//              multiplies it by the matching entries of v or z.  Inside an attempt
//              the stage kernel (rk.cu) adds a leaf's chunks in order and writes the
//              next v permuted; by itself, k_hm_gather permutes v before and
//              k_hm_reduce adds up and writes K's row order after.  Every stored
//              byte is read once per product and the summation order is fixed
//              (deterministic).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_bf16.h>
#include <cstring>
#include <numeric>
#include <utility>
#include <vector>
#include "ucg_internal.cuh"
#include "blocks.cuh"

namespace ucg {

struct HBlock {              // a block in the permuted element order
    int r0, r1, s0, s1;      // receiver and source element ranges
    int lowrank;             // 1: low-rank candidate (admissible)
};

struct HLowRank {            // device descriptor of a stored low-rank block
    const double *U, *V;     // k x m and k x n, rank-major
    int k, m, n, s0;         // rank, rows, columns, first source element (permuted)
    int r0;                  // first receiver element (permuted)
    int zoff;                // offset of its z in the product's workspace
    long vsoff;              // offset of its V in the split (bf16 hi / lo) copy
};

struct HLeafTerm {           // the rows of one row leaf in one block (or a range of its columns)
    const double *A;         // while building: the block's column-major rows at the leaf (stride lda)
    int lda;                 // while building: the block's m
    int cols;                // columns of this piece
    int xsel;                // 0: dense columns times xp; 1: U columns times z
    long xoff;               // first entry of xp (dense) or z (low-rank) multiplying the piece
};

struct HChunk {              // consecutive terms [q0, q1) of one row leaf, packed contiguously
    int rows, cols;          // rows of the leaf; columns over the terms
    int q0, q1;
    int bytes;               // of its panel (a multiple of 16)
    int id;                  // its place in the leaf's order: slot of its partial sums
    long off;                // panel offset (doubles)
};

struct HMat {
    int np = 0, leaf = 0;
    double eta = 0, eps = 0;
    std::vector<int> perm;               // permuted position -> element
    int *perm_d = nullptr;
    // storage
    std::vector<void *> allocs;
    size_t bytes = 0;                    // stored factors and dense blocks
    long n_dense = 0, n_lowrank = 0, n_fallback = 0;
    int max_rank = 0;
    double build_ms = 0;
    // product
    HLowRank *lr_d = nullptr;            // low-rank descriptors
    int2 *items_d = nullptr;             // (block, first rank index) work items of the first kernel
    long n_items = 0;
    HLeafTerm *terms_d = nullptr;        // per row leaf, its terms (consecutive)
    HChunk *chunks_d = nullptr;          // work of the row kernel
    int *leaf_chunk_d = nullptr;         // per row leaf, its chunks (CSR)
    int n_chunks = 0, n_dense_chunks = 0;
    int *leaf_e0_d = nullptr;            // row leaves: element ranges (permuted)
    int n_leaves = 0, max_leaf = 0;
    int tree_leaf = 0;                   // patches of the cluster tree's largest leaf
    int max_cols = 0;                    // columns of the widest chunk
    double *z_d = nullptr;               // low-rank workspace
    long nz = 0;
    double *part_d = nullptr;            // partial row sums (chunk, row)
    double *xp_d = nullptr;              // the product's input in the permuted order
    double *panel = nullptr;             // the row data of every chunk, chunk after chunk
    long panel_len = 0;                  // doubles
    std::vector<HLowRank> lr_h;          // host copy of the low-rank descriptors
    std::vector<int> leaf_e0_h, leaf_term0_h;   // host copies of the leaves and their term ranges
    std::vector<HLeafTerm> terms_h;
    std::vector<long> term_poff_h;       // panel offset (doubles) of every term
    // split copies (hi and lo bf16 of every value) for UCG_PREC_HMATRIX_SPLIT
    __nv_bfloat16 *ph = nullptr, *pl = nullptr, *vh = nullptr, *vl = nullptr;
    int *status_d = nullptr;             // nonzero: a bulk copy of the row kernel timed out
    double *t_d = nullptr;               // product output (K's row order)
};

namespace {

// ---- cluster tree and block tree (host) -------------------------------------------

struct Node {
    int e0, e1;
    double lo[3], hi[3];
    int c[2];
};

struct TreeBuilder {
    const std::vector<double> &box, &ctr;
    std::vector<int> &perm;
    std::vector<Node> nodes;
    int leaf;

    int build(int e0, int e1)
    {
        Node nd;
        nd.e0 = e0;
        nd.e1 = e1;
        nd.c[0] = nd.c[1] = -1;
        for (int k = 0; k < 3; k++) {
            nd.lo[k] = INFINITY;
            nd.hi[k] = -INFINITY;
        }
        double clo[3] = {INFINITY, INFINITY, INFINITY}, chi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int i = e0; i < e1; i++) {
            const int e = perm[i];
            for (int k = 0; k < 3; k++) {
                nd.lo[k] = std::min(nd.lo[k], box[6L * e + k]);
                nd.hi[k] = std::max(nd.hi[k], box[6L * e + 3 + k]);
                clo[k] = std::min(clo[k], ctr[3L * e + k]);
                chi[k] = std::max(chi[k], ctr[3L * e + k]);
            }
        }
        const int id = (int)nodes.size();
        nodes.push_back(nd);
        if (e1 - e0 > leaf) {
            int ax = 0;
            for (int k = 1; k < 3; k++)
                if (chi[k] - clo[k] > chi[ax] - clo[ax]) ax = k;
            const int mid = e0 + (e1 - e0) / 2;
            std::nth_element(perm.begin() + e0, perm.begin() + mid, perm.begin() + e1,
                             [&](int a, int b) { return ctr[3L * a + ax] < ctr[3L * b + ax]; });
            const int a = build(e0, mid);
            const int b = build(mid, e1);
            nodes[id].c[0] = a;
            nodes[id].c[1] = b;
        }
        return id;
    }
};

double diam(const Node &a)
{
    double s = 0;
    for (int k = 0; k < 3; k++) s += (a.hi[k] - a.lo[k]) * (a.hi[k] - a.lo[k]);
    return std::sqrt(s);
}

double dist(const Node &a, const Node &b)
{
    double s = 0;
    for (int k = 0; k < 3; k++) {
        const double d = std::max(0.0, std::max(a.lo[k] - b.hi[k], b.lo[k] - a.hi[k]));
        s += d * d;
    }
    return std::sqrt(s);
}

void block_tree(const std::vector<Node> &nd, int t, int s, double eta, double max_entries, std::vector<HBlock> &out)
{
    const Node &a = nd[t], &b = nd[s];
    const bool la = a.c[0] < 0, lb = b.c[0] < 0;
    const double entries = 6.0 * (a.e1 - a.e0) * (double)(b.e1 - b.e0);
    const bool fits = entries <= max_entries || (la && lb);
    if (fits && std::max(diam(a), diam(b)) <= eta * dist(a, b)) {
        out.push_back({a.e0, a.e1, b.e0, b.e1, 1});
        return;
    }
    if (la && lb) {
        out.push_back({a.e0, a.e1, b.e0, b.e1, 0});
    } else if (la) {
        block_tree(nd, t, b.c[0], eta, max_entries, out);
        block_tree(nd, t, b.c[1], eta, max_entries, out);
    } else if (lb) {
        block_tree(nd, a.c[0], s, eta, max_entries, out);
        block_tree(nd, a.c[1], s, eta, max_entries, out);
    } else {
        for (int i = 0; i < 2; i++)
            for (int j = 0; j < 2; j++) block_tree(nd, a.c[i], b.c[j], eta, max_entries, out);
    }
}

// ---- adaptive cross approximation (device) --------------------------------------------

struct AcaJob {
    const double *B;         // dense block, row-major m x n
    int m, n, kmax;
    double *U, *V;           // kmax x m, kmax x n
    unsigned char *used;     // m row flags
};

constexpr int ACA_THREADS = 512;
constexpr int ACA_KMAX = 256;

__device__ double aca_probe(long j)
{
    // deterministic pseudo-random value in [-1, 1] (splitmix64 of j)
    unsigned long long x = (unsigned long long)j * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
    x ^= x >> 31;
    x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 27;
    return (double)(x >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// block-wide sum (every thread gets the result)
__device__ double block_sum(double v, double *sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double s = 0.0;
    for (int i = 0; i < ACA_THREADS / 32; i++) s += sh[i];
    return s;
}

// block-wide argmax of v >= 0 (ties: lowest index); bi < 0 where no thread had a candidate
__device__ void block_argmax(double v, int idx, double *shv, int *shi, double &bv, int &bi)
{
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (oi >= 0 && (idx < 0 || ov > v || (ov == v && oi < idx))) {
            v = ov;
            idx = oi;
        }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) {
        shv[w] = v;
        shi[w] = idx;
    }
    __syncthreads();
    bv = -1.0;
    bi = -1;
    for (int i = 0; i < ACA_THREADS / 32; i++)
        if (shi[i] >= 0 && (bi < 0 || shv[i] > bv || (shv[i] == bv && shi[i] < bi))) {
            bv = shv[i];
            bi = shi[i];
        }
}

// b[j] - sum_l cs[l] F[l, j] for j < len, handed to put(j, r): a row (or column) of
// a block less the crosses so far.  Four entries a thread at a time, eight crosses
// deep: the loads, not the arithmetic, take the time.
template <class Put>
__device__ __forceinline__ void aca_residual(const double *b, long stride, const double *F, int len, int k,
                                             const double *cs, int tid, Put put)
{
    for (int j0 = tid; j0 < len; j0 += 4 * ACA_THREADS) {
        int j[4];
        double r[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            j[q] = min(j0 + q * ACA_THREADS, len - 1);
            r[q] = b[j[q] * stride];
        }
#pragma unroll 8
        for (int l = 0; l < k; l++)
#pragma unroll
            for (int q = 0; q < 4; q++) r[q] -= cs[l] * F[(long)l * len + j[q]];
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (j0 + q * ACA_THREADS < len) put(j[q], r[q]);
    }
}

// the probe vector, shared by all blocks
__global__ void k_probe(double *__restrict__ w, int n)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) w[j] = aca_probe(j);
}

// Adaptive cross approximation with partial pivoting, one CTA per block.  rank and
// z (ACA_KMAX a block) receive the number of crosses and V^T w.  The largest blocks
// come first and set the kernel's time, a rank at a time: the products of a new
// cross with the earlier ones (for the norm) go one warp each, not one after the
// other through the whole CTA with eight barriers each, and the check against the
// dense block is a kernel of its own over all SMs (N = 7,200: 25 -> 7.9 ms).
__global__ void __launch_bounds__(ACA_THREADS) k_aca(const AcaJob *__restrict__ jobs, double eps,
                                                     const double *__restrict__ probe, int *__restrict__ rank,
                                                     double *__restrict__ z)
{
    const AcaJob J = jobs[blockIdx.x];
    __shared__ double shv[ACA_THREADS / 32];
    __shared__ int shi[ACA_THREADS / 32];
    __shared__ double cs[ACA_KMAX];
    const int m = J.m, n = J.n, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const double *B = J.B;
    for (int i = tid; i < m; i += ACA_THREADS) J.used[i] = 0;
    __syncthreads();
    int k = 0, row = m / 2, misses = 0;
    double frob2 = 0.0;
    while (k < J.kmax) {
        double *v = J.V + (long)k * n;
        double *u = J.U + (long)k * m;
        // residual of the row; its largest entry picks the pivot column
        double best = -1.0;
        int bj = -1;
        for (int l = tid; l < k; l += ACA_THREADS) cs[l] = J.U[(long)l * m + row];
        __syncthreads();
        aca_residual(B + (long)row * n, 1, J.V, n, k, cs, tid, [&](int j, double r) {
            v[j] = r;
            if (fabs(r) > best) { best = fabs(r); bj = j; }
        });
        if (tid == 0) J.used[row] = 1;
        double pv;
        int pj;
        block_argmax(best, bj, shv, shi, pv, pj);
        if (!(pv > 0.0)) {
            // a zero residual row: try the next unused one
            if (++misses > 16) break;
            int nr = -1;
            for (int i = 0; i < m; i++) {
                const int cand = (row + 1 + i) % m;
                if (!J.used[cand]) { nr = cand; break; }
            }
            __syncthreads();
            if (nr < 0) break;
            row = nr;
            continue;
        }
        const double p = v[pj];
        __syncthreads();
        for (int j = tid; j < n; j += ACA_THREADS) v[j] = v[j] / p;
        // residual of the pivot column
        for (int l = tid; l < k; l += ACA_THREADS) cs[l] = J.V[(long)l * n + pj];
        __syncthreads();
        aca_residual(B + pj, n, J.U, m, k, cs, tid, [&](int i, double r) { u[i] = r; });
        __syncthreads();
        // ||S_k||_F^2 update: |u|^2 |v|^2 + 2 sum_l (u_l . u)(v_l . v)
        double a = 0.0, b = 0.0;
        for (int i = tid; i < m; i += ACA_THREADS) a += u[i] * u[i];
        for (int j = tid; j < n; j += ACA_THREADS) b += v[j] * v[j];
        const double nu2 = block_sum(a, shv), nv2 = block_sum(b, shv);
        double cross = 0.0;
        for (int l = w; l < k; l += ACA_THREADS / 32) {
            double cu = 0.0, cv = 0.0;
#pragma unroll 8
            for (int i = lane; i < m; i += 32) cu += J.U[(long)l * m + i] * u[i];
#pragma unroll 8
            for (int j = lane; j < n; j += 32) cv += J.V[(long)l * n + j] * v[j];
            for (int o = 16; o > 0; o >>= 1) {
                cu += __shfl_xor_sync(0xffffffffu, cu, o);
                cv += __shfl_xor_sync(0xffffffffu, cv, o);
            }
            if (lane == 0) cross += cu * cv;
        }
        cross = block_sum(cross, shv);
        frob2 += nu2 * nv2 + 2.0 * cross;
        k++;
        if (sqrt(nu2 * nv2) <= eps * sqrt(fabs(frob2))) break;
        // next row: the largest entry of the new column among the unused rows
        best = -1.0;
        int bi = -1;
        for (int i = tid; i < m; i += ACA_THREADS)
            if (!J.used[i] && fabs(u[i]) > best) { best = fabs(u[i]); bi = i; }
        int ni;
        block_argmax(best, bi, shv, shi, pv, ni);
        if (ni < 0) break;
        row = ni;
    }
    if (tid == 0) rank[blockIdx.x] = k;
    __syncthreads();
    for (int l = w; l < k; l += ACA_THREADS / 32) {
        double s = 0.0;
#pragma unroll 4
        for (int j = lane; j < n; j += 32) s += J.V[(long)l * n + j] * probe[j];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) z[(long)blockIdx.x * ACA_KMAX + l] = s;
    }
}

// The check of every block against its dense form for the probe vector w: sums of
// |B w - U z|^2 and |B w|^2 over one tile of rows
constexpr int CHECK_ROWS = 32;

__global__ void __launch_bounds__(256) k_aca_check(const AcaJob *__restrict__ jobs, const int2 *__restrict__ tiles,
                                                   const double *__restrict__ probe, const int *__restrict__ rank,
                                                   const double *__restrict__ z, double2 *__restrict__ sums)
{
    __shared__ double2 sh[8];
    const int2 tile = tiles[blockIdx.x];
    const AcaJob J = jobs[tile.x];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, k = rank[tile.x];
    const double *zj = z + (long)tile.x * ACA_KMAX;
    double e2 = 0.0, y2 = 0.0;
    for (int i = tile.y + w; i < min(J.m, tile.y + CHECK_ROWS); i += 8) {
        double s = 0.0, a = 0.0;
#pragma unroll 4
        for (int j = lane; j < J.n; j += 32) s += J.B[(long)i * J.n + j] * probe[j];
        for (int l = lane; l < k; l += 32) a += J.U[(long)l * J.m + i] * zj[l];
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            a += __shfl_xor_sync(0xffffffffu, a, o);
        }
        e2 += (s - a) * (s - a);
        y2 += s * s;
    }
    if (lane == 0) sh[w] = make_double2(e2, y2);
    __syncthreads();
    if (threadIdx.x == 0) {
        double2 t = sh[0];
        for (int i = 1; i < 8; i++) {
            t.x += sh[i].x;
            t.y += sh[i].y;
        }
        sums[blockIdx.x] = t;
    }
}

// rank of every block, or -1 where it stays dense: the probe error above `check`,
// or factors of more than half its size.  first: first tile of every block.
__global__ void k_aca_accept(const AcaJob *__restrict__ jobs, int n_jobs, const int *__restrict__ first,
                             const double2 *__restrict__ sums, double check, int *__restrict__ rank)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_jobs) return;
    double e2 = 0.0, y2 = 0.0;
    for (int t = first[q]; t < first[q + 1]; t++) {
        e2 += sums[t].x;
        y2 += sums[t].y;
    }
    const double err = y2 > 0.0 ? sqrt(e2 / y2) : (e2 > 0.0 ? INFINITY : 0.0);
    const int k = rank[q], m = jobs[q].m, n = jobs[q].n;
    const bool smaller = (double)k * (m + n) < 0.5 * (double)m * n;
    if (!(err <= check && smaller)) rank[q] = -1;
}

// What a batch keeps, in one launch: copies of the factors and column-major
// copies of the dense blocks.  A CTA takes KEEP_TILE values of one job.
struct KeepJob {
    const double *src;   // row-major m x n
    double *dst;
    int m, n;
    int transpose;
};

constexpr int KEEP_TILE = 4096;

__global__ void __launch_bounds__(256) k_keep(const KeepJob *__restrict__ jobs, const int2 *__restrict__ tiles)
{
    const int2 tile = tiles[blockIdx.x];
    const KeepJob J = jobs[tile.x];
    const long tot = (long)J.m * J.n, t0 = (long)tile.y * KEEP_TILE, t1 = min(tot, t0 + KEEP_TILE);
    for (long t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
        if (J.transpose) {
            const long j = t / J.m, i = t - j * J.m;
            J.dst[t] = J.src[i * J.n + j];
        } else {
            J.dst[t] = J.src[t];
        }
    }
}

int keep_blocks(ucg_ctx *c, const std::vector<KeepJob> &jobs)
{
    if (jobs.empty()) return UCG_OK;
    std::vector<int2> tiles;
    for (size_t q = 0; q < jobs.size(); q++) {
        const long n = ((long)jobs[q].m * jobs[q].n + KEEP_TILE - 1) / KEEP_TILE;
        for (long t = 0; t < n; t++) tiles.push_back(make_int2((int)q, (int)t));
    }
    KeepJob *jd;
    int2 *td;
    int rc;
    if ((rc = workspace_upload(c, WS_JOBS, jobs, &jd)) || (rc = workspace_upload(c, WS_TILES, tiles, &td))) return rc;
    k_keep<<<(int)tiles.size(), 256, 0, c->stream>>>(jd, td);
    c->launches.count++;
    UCG_CUDA(cudaGetLastError());
    return UCG_OK;
}

// ---- the product --------------------------------------------------------------------
//
// The kernels are launched with programmatic dependent launch: each lets the next
// be scheduled and waits for the ones before it itself, the row kernel only after
// it has asked for its panel, which does not depend on them.

// v in the permuted element order (so that every block's columns are a
// contiguous range of xp)
__global__ void k_hm_gather(const int *__restrict__ perm, int np, const double *__restrict__ v,
                            double *__restrict__ xp)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    reinterpret_cast<double2 *>(xp)[i] = reinterpret_cast<const double2 *>(v)[perm[i]];
}

// Two kernels form the partial sums, bound by HBM.  The first works on z and, in
// every other CTA, on the chunks of dense blocks, which do not need it; the second
// on the chunks of low-rank factors, which do.  (z by itself took 29 us of a product
// at N = 7,200 for 17 us worth of its 110 MB, the few longest blocks being the tail.)
//
// z_b[l] = V_b[l, :] . xp(sigma_b): one warp per (block, HM_ZR rank indices), which
// share the loads of xp, with HM_ZU loads of each in flight, the longest blocks
// first.  Stage of an attempt at N = 7,200, FP64 / split / N = 1,800: HM_ZR, HM_ZU =
// 2, 2 135 / 92 / 26.5 us; 1, 4 148 / 91 / 27; 2, 4 139 / 91 / 27; 4, 2 132 / 97 / 30.
//
// Partial row sums over one chunk of a row leaf's terms: the chunk's panel
// (at most HM_CHUNK_BYTES, contiguous) arrives in shared memory by one bulk
// copy, asked for first of all; meanwhile the entries of xp (dense) or z
// (low-rank) that multiply its columns are gathered beside it; then one thread per
// row multiplies.  k_hm_reduce (in an attempt k_hm_stage, rk.cu) adds a leaf's
// chunks in order.  Many small CTAs per SM keep many copies in flight.  The wait
// for the copy is bounded (about 4 s); when it runs out the chunk writes NaN, which
// the integrator reports as a non-finite rate, and the kernel flags status.  24 KB
// chunks: 16 KB 4 % slower for the split form, whose chunks are half as large, 32 KB
// 5 % for FP64 (fewer CTAs an SM).  Before these kernels a stage took 150 / 120 / 46.
constexpr long HM_CHUNK_BYTES = 24 * 1024;
constexpr int HM_THREADS = 128;   // at most; the launch takes a leaf's rows rounded up to warps
constexpr int HM_LEAF = HM_THREADS / 3;   // patches of a row leaf: a thread a row
constexpr int HM_ZR = 2, HM_ZU = 2;
constexpr unsigned long long HM_TIMEOUT_NS = 4000000000ull;

__device__ __forceinline__ uint32_t hm_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool hm_try(uint64_t *bar)
{
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
                 " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(hm_smem(bar)) : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool hm_wait(uint64_t *bar)
{
    if (hm_try(bar)) return true;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (unsigned it = 1;; it++) {
        if (hm_try(bar)) return true;
        if ((it & 255u) == 0u) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t - t0 > HM_TIMEOUT_NS) return false;
        }
    }
}

// ---- split (hi + lo) form ---------------------------------------------------------------
//
// Every stored value x is kept as its FP32 rounding split into two 16-bit
// planes: hi, the upper half (a bf16 number: sign, exponent, 7 significand
// bits) and lo, the lower 16 significand bits.  hi and lo together give the
// FP32 value exactly (relative error <= 2^-24); the anchored Runge-Kutta
// stages read both for every stage (4 bytes per value, half the FP64 stream)
// and sum in FP64.

__device__ __forceinline__ void split32(double v, __nv_bfloat16 &hi, __nv_bfloat16 &lo)
{
    const uint32_t b = __float_as_uint(__double2float_rn(v));
    hi = __ushort_as_bfloat16((unsigned short)(b >> 16));
    lo = __ushort_as_bfloat16((unsigned short)(b & 0xffffu));
}
__device__ __forceinline__ float join32(__nv_bfloat16 hi, __nv_bfloat16 lo)
{
    return __uint_as_float(((uint32_t)__bfloat16_as_ushort(hi) << 16) | (uint32_t)__bfloat16_as_ushort(lo));
}

__global__ void k_split_flat(const double *__restrict__ x, long n, __nv_bfloat16 *__restrict__ hi,
                             __nv_bfloat16 *__restrict__ lo)
{
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
        split32(x[t], hi[t], lo[t]);
}

struct SplitJob {
    const double *src;
    long n, dst;
};

__global__ void k_split_jobs(const SplitJob *__restrict__ jobs, __nv_bfloat16 *__restrict__ hi,
                             __nv_bfloat16 *__restrict__ lo)
{
    const SplitJob J = jobs[blockIdx.x];
    for (long t = threadIdx.x; t < J.n; t += blockDim.x) split32(J.src[t], hi[J.dst + t], lo[J.dst + t]);
}

// ---- product kernels ----------------------------------------------------------------

struct HmProduct {
    const HLowRank *lr;
    const int2 *items;        // (block, first rank index) of the z warps
    long n_items;
    const HLeafTerm *terms;
    const HChunk *chunks;     // of dense blocks, then of low-rank factors
    int n_dense;
    const double *panel;                      // FP64 form
    const __nv_bfloat16 *ph, *pl, *vh, *vl;   // split form
    const double *xp;
    double *z, *part;
    int rows_max;
    int *status;
};

// two columns of V of one rank index, FP64 or split
template <bool SPLIT> struct ZPair;
template <> struct ZPair<false> {
    const double2 *v;
    double2 x;
    __device__ __forceinline__ void at(const HmProduct &P, const HLowRank &b, int l)
    {
        (void)P;
        v = reinterpret_cast<const double2 *>(b.V + (long)l * b.n);
    }
    __device__ __forceinline__ void load(int j) { x = v[j]; }
    __device__ __forceinline__ double2 get() const { return x; }
};
template <> struct ZPair<true> {
    const __nv_bfloat162 *h, *l;
    __nv_bfloat162 xh, xl;
    __device__ __forceinline__ void at(const HmProduct &P, const HLowRank &b, int r)
    {
        const long o = b.vsoff + (long)r * b.n;
        h = reinterpret_cast<const __nv_bfloat162 *>(P.vh + o);
        l = reinterpret_cast<const __nv_bfloat162 *>(P.vl + o);
    }
    __device__ __forceinline__ void load(int j) { xh = h[j]; xl = l[j]; }
    __device__ __forceinline__ double2 get() const
    {
        return make_double2((double)join32(xh.x, xl.x), (double)join32(xh.y, xl.y));
    }
};

template <bool SPLIT>
__device__ __forceinline__ void hm_z(const HmProduct &P, long w)
{
    if (w >= P.n_items) return;
    const int lane = threadIdx.x & 31;
    const int2 it = P.items[w];
    const HLowRank b = P.lr[it.x];
    const int n2 = b.n >> 1;
    const double2 *x = reinterpret_cast<const double2 *>(P.xp + 2L * b.s0);
    ZPair<SPLIT> v[HM_ZR][HM_ZU];
#pragma unroll
    for (int r = 0; r < HM_ZR; r++)
#pragma unroll
        for (int u = 0; u < HM_ZU; u++)   // past the last rank: the last one again, not stored
            v[r][u].at(P, b, min(it.y + r, b.k - 1));
    double s[HM_ZR][2] = {};
    auto add = [&](int r, double2 a, double2 xx) {
        s[r][0] = fma(a.x, xx.x, s[r][0]);
        s[r][1] = fma(a.y, xx.y, s[r][1]);
    };
    int j = lane;
    for (; j + 32 * (HM_ZU - 1) < n2; j += 32 * HM_ZU) {
        double2 xx[HM_ZU];
#pragma unroll
        for (int u = 0; u < HM_ZU; u++) {
            xx[u] = x[j + 32 * u];
#pragma unroll
            for (int r = 0; r < HM_ZR; r++) v[r][u].load(j + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < HM_ZU; u++)
#pragma unroll
            for (int r = 0; r < HM_ZR; r++) add(r, v[r][u].get(), xx[u]);
    }
    for (; j < n2; j += 32) {
        const double2 xx = x[j];
#pragma unroll
        for (int r = 0; r < HM_ZR; r++) {
            v[r][0].load(j);
            add(r, v[r][0].get(), xx);
        }
    }
#pragma unroll
    for (int r = 0; r < HM_ZR; r++) {
        double t = s[r][0] + s[r][1];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0 && it.y + r < b.k) P.z[b.zoff + it.y + r] = t;
    }
}

// FIRST: z and the chunks of dense blocks; otherwise the chunks of low-rank factors
template <bool SPLIT, bool FIRST>
__global__ void __launch_bounds__(HM_THREADS) k_hm_rows(HmProduct P, int zblocks)
{
    extern __shared__ __align__(128) double sm[];
    __shared__ __align__(8) uint64_t bar;
    int slot = blockIdx.x;
    if (FIRST) {
        // z and dense CTAs in turn until one kind runs out: z alone keeps too little in flight
        const int both = 2 * min(zblocks, P.n_dense);
        const bool z = slot < both ? !(slot & 1) : zblocks > P.n_dense;
        slot = slot < both ? slot >> 1 : slot - (both >> 1);
        if (z) {
            pdl_wait();
            pdl_launch();
            hm_z<SPLIT>(P, ((long)slot * blockDim.x + threadIdx.x) >> 5);
            return;
        }
    }
    const HChunk ch = P.chunks[FIRST ? slot : P.n_dense + slot];
    const int i = threadIdx.x, rows = ch.rows;
    const long nel = ch.bytes / 8;                      // values in the chunk
    const __nv_bfloat16 *sb = reinterpret_cast<const __nv_bfloat16 *>(sm);   // split: hi, then lo
    double *xs = sm + (SPLIT ? HM_CHUNK_BYTES / 16 : HM_CHUNK_BYTES / 8);
    if (i == 0 && nel) {
        const uint32_t bytes = SPLIT ? ch.bytes / 2 : ch.bytes, half = ch.bytes / 4;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(hm_smem(&bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(hm_smem(&bar)), "r"(bytes)
                     : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(hm_smem(sm)), "l"(SPLIT ? (const void *)(P.ph + ch.off) : (const void *)(P.panel + ch.off)),
                     "r"(SPLIT ? half : bytes), "r"(hm_smem(&bar)) : "memory");
        if (SPLIT)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(hm_smem(sb + nel)), "l"(P.pl + ch.off), "r"(half), "r"(hm_smem(&bar)) : "memory");
    }
    pdl_wait();
    pdl_launch();
    double *part = P.part + (long)ch.id * P.rows_max + i;
    if (nel == 0) {
        if (i < rows) *part = 0.0;
        return;
    }
    // the entries of xp or z, column after column of the chunk's terms
    for (int q = ch.q0, base = 0; q < ch.q1; q++) {
        const HLeafTerm T = P.terms[q];
        const double *x = (FIRST ? P.xp : P.z) + T.xoff;
        for (int j = i; j < T.cols; j += blockDim.x) xs[base + j] = x[j];
        base += T.cols;
    }
    __syncthreads();
    if (!hm_wait(&bar)) {
        if (i == 0) atomicExch(P.status, 1);
        if (i < rows) *part = nan("");
        hm_wait(&bar);   // the copy may still land in this CTA's shared memory: wait once more (bounded)
        return;
    }
    if (i >= rows) return;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    long off = 0;
    const double *x = xs;
    for (int q = ch.q0; q < ch.q1; q++) {
        const int cols = P.terms[q].cols;
        auto val = [&](int j) -> double {
            const long o = off + i + (long)j * rows;
            return SPLIT ? (double)join32(sb[o], sb[nel + o]) : sm[o];
        };
        int j = 0;
        for (; j + 3 < cols; j += 4) {
            a0 = fma(val(j), x[j], a0);
            a1 = fma(val(j + 1), x[j + 1], a1);
            a2 = fma(val(j + 2), x[j + 2], a2);
            a3 = fma(val(j + 3), x[j + 3], a3);
        }
        for (; j < cols; j++) a0 = fma(val(j), x[j], a0);
        off += ((long)rows * cols + 7) & ~7L;
        x += cols;
    }
    *part = (a0 + a1) + (a2 + a3);
}

struct PackJob {
    const double *src;       // column-major, leading dimension lda
    int lda, rows, cols;
    long dst;                // offset of the rows x cols panel
};

__global__ void k_pack(const PackJob *__restrict__ jobs, double *__restrict__ panel)
{
    const PackJob J = jobs[blockIdx.x];
    const long tot = (long)J.rows * J.cols;
    for (long t = threadIdx.x; t < tot; t += blockDim.x) {
        const long j = t / J.rows, i = t % J.rows;
        panel[J.dst + t] = J.src[j * J.lda + i];
    }
}

// t for one row leaf: blockDim / gs groups of gs threads (gs >= rows) each add
// every ng-th chunk of the leaf, then group 0 adds the groups' sums in order.
__global__ void k_hm_reduce(const int *__restrict__ leaf_e0, const int *__restrict__ leaf_chunk,
                            const int *__restrict__ perm, const double *__restrict__ part, int rows_max,
                            double *__restrict__ t, int gs)
{
    extern __shared__ double sh[];
    const int L = blockIdx.x;
    const int e0 = leaf_e0[L], rows = 3 * (leaf_e0[L + 1] - e0);
    const int c0 = leaf_chunk[L], c1 = leaf_chunk[L + 1];
    const int ng = blockDim.x / gs, g = threadIdx.x / gs, i = threadIdx.x % gs;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    if (i < rows) {
        int c = c0 + g;
        for (; c + 3 * ng < c1; c += 4 * ng) {
            s0 += part[(long)c * rows_max + i];
            s1 += part[(long)(c + ng) * rows_max + i];
            s2 += part[(long)(c + 2 * ng) * rows_max + i];
            s3 += part[(long)(c + 3 * ng) * rows_max + i];
        }
        for (; c < c1; c += ng) s0 += part[(long)c * rows_max + i];
    }
    sh[threadIdx.x] = (s0 + s1) + (s2 + s3);
    __syncthreads();
    if (g == 0 && i < rows) {
        double s = 0.0;
        for (int k = 0; k < ng; k++) s += sh[k * gs + i];
        t[3L * perm[e0 + i / 3] + i % 3] = s;
    }
}

}  // namespace

// ---- host entry points ---------------------------------------------------------------

void hmatrix_free(ucg_ctx *c)
{
    HMat *h = c->hm;
    if (!h) return;
    rk_drop_graph(c);
    cudaStreamSynchronize(c->stream);
    for (void *p : h->allocs) cudaFree(p);
    void *ps[] = {h->perm_d, h->lr_d, h->items_d, h->terms_d, h->chunks_d, h->leaf_chunk_d, h->leaf_e0_d, h->z_d,
                  h->t_d, h->part_d, h->xp_d, h->status_d, h->ph, h->pl, h->vh, h->vl};
    for (void *p : ps)
        if (p) cudaFree(p);
    delete h;
    c->hm = nullptr;
}

// temp_allocs: storage of the build alone, the caller's to free when it fails
static int build_matrix(ucg_ctx *c, int okada_mode, double eta, double eps, int leaf, std::vector<void *> &temp_allocs)
{
    hmatrix_free(c);
    const int np = c->nr + c->nt;
    BlockSources bs;
    int rc = block_family(c);
    if (rc) {
        c->err = "hierarchical matrix: one patch family (rectangles or triangles) and no volumes";
        return rc;
    }
    HMat *h = new HMat();
    c->hm = h;
    h->np = np;
    h->leaf = leaf;
    h->eta = eta;
    h->eps = eps;
    cudaEvent_t ev0, ev1;
    UCG_CUDA(cudaEventCreate(&ev0));
    UCG_CUDA(cudaEventCreate(&ev1));
    UCG_CUDA(cudaEventRecord(ev0, c->stream));

    // cluster tree and blocks; the build scratch bounds the size of a block
    std::vector<double> box, ctr;
    element_boxes(c, box, ctr);
    h->perm.resize(np);
    std::iota(h->perm.begin(), h->perm.end(), 0);
    TreeBuilder tb{box, ctr, h->perm, {}, leaf};
    tb.build(0, np);
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const size_t bound = std::min<size_t>((size_t)8 << 30, free_b / 4);   // of the build scratch
    std::vector<HBlock> blocks;
    block_tree(tb.nodes, 0, 0, eta, 0.4 * (double)bound / sizeof(double), blocks);
    // row leaves of the product: the tree's, those of more patches than a CTA of the
    // row kernel has threads for cut into equal parts
    std::vector<int> leaf_e0;
    for (const Node &nd : tb.nodes) {
        if (nd.c[0] >= 0) continue;
        const int sz = nd.e1 - nd.e0, parts = (sz + HM_LEAF - 1) / HM_LEAF;
        for (int k = 0; k < parts; k++) leaf_e0.push_back(nd.e0 + (int)((long)sz * k / parts));
        h->tree_leaf = std::max(h->tree_leaf, sz);
    }
    std::sort(leaf_e0.begin(), leaf_e0.end());
    h->n_leaves = (int)leaf_e0.size();
    leaf_e0.push_back(np);
    for (int L = 0; L < h->n_leaves; L++) h->max_leaf = std::max(h->max_leaf, leaf_e0[L + 1] - leaf_e0[L]);
    UCG_CUDA(cudaMalloc(&h->perm_d, sizeof(int) * np));
    UCG_CUDA(cudaMemcpyAsync(h->perm_d, h->perm.data(), sizeof(int) * np, cudaMemcpyHostToDevice, c->stream));

    if ((rc = block_sources_build(c, okada_mode, h->perm, &bs))) return rc;

    // scratch of a batch: what all blocks need, within the bound (few large batches:
    // each waits for its largest block)
    auto block_need = [&](const HBlock &B) -> size_t {   // doubles
        const long m = 3L * (B.r1 - B.r0), n = 2L * (B.s1 - B.s0);
        const long kmax = std::min<long>(ACA_KMAX, std::min(m, n));
        const size_t need = (size_t)m * n + (B.lowrank ? (size_t)kmax * (m + n) + (m + 7) / 8 + 2 : 0);
        return (need + 31) & ~(size_t)31;
    };
    size_t total_need = 0, largest = 0;
    for (const HBlock &B : blocks) {
        total_need += block_need(B);
        largest = std::max(largest, block_need(B));
    }
    const size_t scratch =
        std::min(bound, std::max(sizeof(double) * largest, sizeof(double) * total_need));
    double *sc = nullptr;
    UCG_CUDA(cudaMalloc(&sc, scratch));
    struct Done {
        int b;            // block index
        int rank;         // -1: dense
        const double *A;  // dense (column-major) or U
        const double *V;
    };
    std::vector<Done> done;
    // storage: bump allocation over large device chunks; pool 0 keeps V, pool 1
    // holds U and the dense blocks until they are repacked into row panels
    const size_t CHUNK = (size_t)256 << 20;
    size_t chunk_left[2] = {0, 0};
    char *chunk_ptr[2] = {nullptr, nullptr};
    auto store = [&](int pool, size_t bytes, double **out) -> int {
        bytes = (bytes + 255) & ~(size_t)255;
        if (bytes > chunk_left[pool]) {
            const size_t sz = std::max(bytes, CHUNK);
            void *p = nullptr;
            cudaError_t e = cudaMalloc(&p, sz);
            if (e != cudaSuccess) return cuda_fail(c, e, "cudaMalloc(hierarchical matrix storage)");
            (pool == 0 ? h->allocs : temp_allocs).push_back(p);
            chunk_ptr[pool] = (char *)p;
            chunk_left[pool] = sz;
        }
        *out = (double *)chunk_ptr[pool];
        chunk_ptr[pool] += bytes;
        chunk_left[pool] -= bytes;
        return UCG_OK;
    };
    const int MAXJOBS = 4096;
    AcaJob *jobs_d = nullptr;
    int *ranks_d = nullptr;
    double *aca_z = nullptr, *probe_d = nullptr;
    UCG_CUDA(cudaMalloc(&jobs_d, sizeof(AcaJob) * MAXJOBS));
    UCG_CUDA(cudaMalloc(&ranks_d, sizeof(int) * MAXJOBS));
    UCG_CUDA(cudaMalloc(&aca_z, sizeof(double) * (size_t)MAXJOBS * ACA_KMAX));
    UCG_CUDA(cudaMalloc(&probe_d, sizeof(double) * 2 * np));
    k_probe<<<(2 * np + 255) / 256, 256, 0, c->stream>>>(probe_d, 2 * np);
    c->launches.count++;
    auto cleanup = [&]() {
        cudaStreamSynchronize(c->stream);
        cudaFree(sc);
        cudaFree(jobs_d);
        cudaFree(ranks_d);
        cudaFree(aca_z);
        cudaFree(probe_d);
    };

    // the blocks in batches that fit the scratch
    size_t bi = 0;
    std::vector<AcaJob> jobs;
    std::vector<int> job_block;
    std::vector<BlockJob> build;
    std::vector<KeepJob> keep;
    while (bi < blocks.size()) {
        size_t off = 0;   // in doubles
        jobs.clear();
        job_block.clear();
        build.clear();
        keep.clear();
        std::vector<std::pair<int, size_t>> dense_in_batch;
        while (bi < blocks.size() && (int)jobs.size() < MAXJOBS) {
            const HBlock &B = blocks[bi];
            const long m = 3L * (B.r1 - B.r0), n = 2L * (B.s1 - B.s0);
            const int kmax = (int)std::min<long>(ACA_KMAX, std::min(m, n));
            const size_t need = block_need(B);
            if ((off + need) * sizeof(double) > scratch) {
                if (off == 0) {
                    cleanup();
                    c->err = "hierarchical matrix: a dense leaf block exceeds the build scratch (use a smaller leaf)";
                    return UCG_E_OOM;
                }
                break;
            }
            double *Bd = sc + off;
            build.push_back({Bd, B.r0, B.r1 - B.r0, B.s0, B.s1 - B.s0});
            if (B.lowrank) {
                AcaJob J;
                J.B = Bd;
                J.m = (int)m;
                J.n = (int)n;
                J.kmax = kmax;
                J.U = Bd + (size_t)m * n;
                J.V = J.U + (size_t)kmax * m;
                J.used = (unsigned char *)(J.V + (size_t)kmax * n);
                jobs.push_back(J);
                job_block.push_back((int)bi);
            } else {
                dense_in_batch.push_back({(int)bi, off});
            }
            off += need;
            bi++;
        }
        if ((rc = assemble_blocks(c, bs, h->perm_d, build))) {
            cleanup();
            return rc;
        }
        std::vector<int> ranks(jobs.size());
        if (!jobs.empty()) {
            // the largest first
            std::vector<int> order(jobs.size());
            std::iota(order.begin(), order.end(), 0);
            std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
                return (long)jobs[x].m + jobs[x].n > (long)jobs[y].m + jobs[y].n;
            });
            std::vector<AcaJob> sorted;
            std::vector<int> sorted_block, first(1, 0);
            std::vector<int2> tiles;
            for (int q : order) {
                for (int i = 0; i < jobs[q].m; i += CHECK_ROWS) tiles.push_back(make_int2((int)sorted.size(), i));
                first.push_back((int)tiles.size());
                sorted.push_back(jobs[q]);
                sorted_block.push_back(job_block[q]);
            }
            jobs.swap(sorted);
            job_block.swap(sorted_block);
            int2 *td;
            int *fd;
            double2 *sums;
            if ((rc = workspace_upload(c, WS_TILES, tiles, &td)) || (rc = workspace_upload(c, WS_JOBS, first, &fd)) ||
                (rc = workspace(c, WS_SCRATCH, sizeof(double2) * tiles.size(), &sums))) {
                cleanup();
                return rc;
            }
            const int nj = (int)jobs.size();
            cudaMemcpyAsync(jobs_d, jobs.data(), sizeof(AcaJob) * jobs.size(), cudaMemcpyHostToDevice, c->stream);
            k_aca<<<nj, ACA_THREADS, 0, c->stream>>>(jobs_d, eps, probe_d, ranks_d, aca_z);
            k_aca_check<<<(int)tiles.size(), 256, 0, c->stream>>>(jobs_d, td, probe_d, ranks_d, aca_z, sums);
            k_aca_accept<<<(nj + 127) / 128, 128, 0, c->stream>>>(jobs_d, nj, fd, sums, 10.0 * eps, ranks_d);
            c->launches.count += 3;
            cudaMemcpyAsync(ranks.data(), ranks_d, sizeof(int) * jobs.size(), cudaMemcpyDeviceToHost, c->stream);
        }
        cudaError_t e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) {
            cleanup();
            return cuda_fail(c, e, "hierarchical matrix compression");
        }
        // keep the factors of the compressed blocks and column-major copies of the dense ones
        auto keep_dense = [&](int b, const double *src) -> int {
            const HBlock &B = blocks[b];
            const int m = 3 * (B.r1 - B.r0), n = 2 * (B.s1 - B.s0);
            double *d = nullptr;
            int r = store(1, sizeof(double) * (size_t)m * n, &d);
            if (r) return r;
            keep.push_back({src, d, m, n, 1});
            h->bytes += sizeof(double) * (size_t)m * n;
            done.push_back({b, -1, d, nullptr});
            return UCG_OK;
        };
        for (auto &d : dense_in_batch) {
            if ((rc = keep_dense(d.first, sc + d.second))) {
                cleanup();
                return rc;
            }
            h->n_dense++;
        }
        for (size_t q = 0; q < jobs.size(); q++) {
            const int b = job_block[q], k = ranks[q];
            if (k < 0) {
                if ((rc = keep_dense(b, jobs[q].B))) {
                    cleanup();
                    return rc;
                }
                h->n_fallback++;
                continue;
            }
            const AcaJob &J = jobs[q];
            double *U = nullptr, *V = nullptr;
            if ((rc = store(1, sizeof(double) * (size_t)k * J.m, &U)) || (rc = store(0, sizeof(double) * (size_t)k * J.n, &V))) {
                cleanup();
                return rc;
            }
            if (k > 0) {
                keep.push_back({J.U, U, k, J.m, 0});
                keep.push_back({J.V, V, k, J.n, 0});
            }
            h->bytes += sizeof(double) * (size_t)k * (J.m + J.n);
            h->n_lowrank++;
            h->max_rank = std::max(h->max_rank, k);
            done.push_back({b, k, U, V});
        }
        if ((rc = keep_blocks(c, keep))) {
            cleanup();
            return rc;
        }
        e = cudaStreamSynchronize(c->stream);   // the scratch is reused by the next batch
        if (e != cudaSuccess) {
            cleanup();
            return cuda_fail(c, e, "hierarchical matrix storage");
        }
    }
    cleanup();

    // product structures, in block-tree order (fixed summation order)
    std::vector<HLowRank> lr;
    std::vector<int2> items;
    std::vector<std::vector<HLeafTerm>> per_leaf(h->n_leaves);
    long zoff = 0;
    auto leaf_of = [&](int e) {
        return (int)(std::upper_bound(leaf_e0.begin(), leaf_e0.end() - 1, e) - leaf_e0.begin()) - 1;
    };
    std::sort(done.begin(), done.end(), [](const Done &a, const Done &b) { return a.b < b.b; });
    for (const Done &d : done) {
        const HBlock &B = blocks[d.b];
        const int m = 3 * (B.r1 - B.r0), n = 2 * (B.s1 - B.s0);
        if (d.rank < 0) {
            for (int L = leaf_of(B.r0); L < h->n_leaves && leaf_e0[L] < B.r1; L++)
                per_leaf[L].push_back({d.A + 3L * (leaf_e0[L] - B.r0), m, n, 0, 2L * B.s0});
        } else if (d.rank > 0) {
            const int id = (int)lr.size();
            lr.push_back({d.A, d.V, d.rank, m, n, B.s0, B.r0, (int)zoff});
            for (int l = 0; l < d.rank; l += HM_ZR) items.push_back(make_int2(id, l));
            for (int L = leaf_of(B.r0); L < h->n_leaves && leaf_e0[L] < B.r1; L++)
                per_leaf[L].push_back({d.A + 3L * (leaf_e0[L] - B.r0), m, d.rank, 1, zoff});
            zoff += d.rank;
        }
    }
    // terms cut into column pieces and grouped into chunks of at most
    // HM_CHUNK_BYTES; every piece's rows are packed into one panel, chunk after
    // chunk, each piece padded to 16 bytes
    std::vector<HLeafTerm> terms;
    std::vector<HChunk> chunks;
    std::vector<int> leaf_chunk(1, 0);
    std::vector<HChunk> by_kind[2];   // chunks of dense and of low-rank pieces
    std::vector<PackJob> pk;
    long poff = 0;
    for (int L = 0; L < h->n_leaves; L++) {
        const int rows = 3 * (leaf_e0[L + 1] - leaf_e0[L]);
        const int maxc = (int)std::max<long>(1, HM_CHUNK_BYTES / (8L * rows + 16));
        // dense pieces first: a chunk is of one kind
        for (int kind = 0; kind < 2; kind++) {
            HChunk ch{rows, 0, (int)terms.size(), (int)terms.size(), 0, 0, poff};
            auto close = [&]() {
                ch.id = (int)chunks.size();
                chunks.push_back(ch);
                by_kind[kind].push_back(ch);
                ch = HChunk{rows, 0, (int)terms.size(), (int)terms.size(), 0, 0, poff};
            };
            for (const HLeafTerm &T : per_leaf[L]) {
                if (T.xsel != kind) continue;
                for (int c0 = 0; c0 < T.cols; c0 += maxc) {
                    const int nc = std::min(maxc, T.cols - c0);
                    const long sz = ((long)rows * nc + 7) & ~7L;   // padded to 8 elements (64 / 16 bytes)
                    if (ch.bytes + 8L * sz > HM_CHUNK_BYTES) close();
                    HLeafTerm P = T;
                    P.cols = nc;
                    P.xoff = T.xoff + c0;
                    pk.push_back({T.A + (long)c0 * T.lda, T.lda, rows, nc, poff});
                    terms.push_back(P);
                    poff += sz;
                    ch.q1 = (int)terms.size();
                    ch.bytes += (int)(8L * sz);
                    ch.cols += nc;
                    h->max_cols = std::max(h->max_cols, ch.cols);
                }
            }
            if (ch.bytes || kind == 0) close();   // possibly empty: the leaf's dense rows are then zero
        }
        leaf_chunk.push_back((int)chunks.size());
    }
    h->n_chunks = (int)chunks.size();
    h->leaf_e0_h = leaf_e0;
    h->leaf_term0_h.assign(1, 0);
    for (int L = 0; L < h->n_leaves; L++) h->leaf_term0_h.push_back(chunks[leaf_chunk[L + 1] - 1].q1);
    h->term_poff_h.resize(pk.size());
    for (size_t q = 0; q < pk.size(); q++) h->term_poff_h[q] = pk[q].dst;
    {
        double *panel = nullptr;
        UCG_CUDA(cudaMalloc(&panel, sizeof(double) * std::max<long>(poff, 2)));
        h->allocs.push_back(panel);
        h->panel = panel;
        h->panel_len = poff;
        if (!pk.empty()) {
            PackJob *pk_d = nullptr;
            UCG_CUDA(cudaMalloc(&pk_d, sizeof(PackJob) * pk.size()));
            UCG_CUDA(cudaMemcpyAsync(pk_d, pk.data(), sizeof(PackJob) * pk.size(), cudaMemcpyHostToDevice, c->stream));
            k_pack<<<(int)pk.size(), 256, 0, c->stream>>>(pk_d, panel);
            c->launches.count++;
            UCG_CUDA(cudaStreamSynchronize(c->stream));
            cudaFree(pk_d);
        }
        for (void *p : temp_allocs) cudaFree(p);
        temp_allocs.clear();
        for (HLowRank &b : lr) b.U = nullptr;   // the product reads U from the panels
        for (HLeafTerm &T : terms) T.A = nullptr;
        h->terms_h = terms;
    }
    // the longest blocks' warps first
    std::stable_sort(items.begin(), items.end(), [&](const int2 &x, const int2 &y) { return lr[x.x].n > lr[y.x].n; });
    h->n_items = (long)items.size();
    h->n_dense_chunks = (int)by_kind[0].size();
    h->nz = std::max<long>(zoff, 1);
    UCG_CUDA(cudaMalloc(&h->lr_d, sizeof(HLowRank) * std::max<size_t>(lr.size(), 1)));
    UCG_CUDA(cudaMalloc(&h->items_d, sizeof(int2) * std::max<size_t>(items.size(), 1)));
    UCG_CUDA(cudaMalloc(&h->terms_d, sizeof(HLeafTerm) * std::max<size_t>(terms.size(), 1)));
    UCG_CUDA(cudaMalloc(&h->chunks_d, sizeof(HChunk) * chunks.size()));
    UCG_CUDA(cudaMalloc(&h->leaf_chunk_d, sizeof(int) * leaf_chunk.size()));
    UCG_CUDA(cudaMalloc(&h->leaf_e0_d, sizeof(int) * leaf_e0.size()));
    UCG_CUDA(cudaMalloc(&h->z_d, sizeof(double) * h->nz));
    UCG_CUDA(cudaMalloc(&h->t_d, sizeof(double) * (3L * np + 2)));
    UCG_CUDA(cudaMalloc(&h->xp_d, sizeof(double) * (2L * np + 2)));
    UCG_CUDA(cudaMalloc(&h->status_d, sizeof(int)));
    UCG_CUDA(cudaMemset(h->status_d, 0, sizeof(int)));
    UCG_CUDA(cudaMalloc(&h->part_d, sizeof(double) * (size_t)h->n_chunks * 3 * h->max_leaf));
    {
        long vs = 0;
        for (HLowRank &b : lr) {
            b.vsoff = vs;
            vs += (long)b.k * b.n;
        }
    }
    h->lr_h = lr;
    if (!lr.empty()) UCG_CUDA(cudaMemcpyAsync(h->lr_d, lr.data(), sizeof(HLowRank) * lr.size(), cudaMemcpyHostToDevice, c->stream));
    if (!items.empty())
        UCG_CUDA(cudaMemcpyAsync(h->items_d, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, c->stream));
    if (!terms.empty())
        UCG_CUDA(cudaMemcpyAsync(h->terms_d, terms.data(), sizeof(HLeafTerm) * terms.size(), cudaMemcpyHostToDevice, c->stream));
    // on the device the dense chunks come first: the two product kernels take one kind each
    by_kind[0].insert(by_kind[0].end(), by_kind[1].begin(), by_kind[1].end());
    UCG_CUDA(cudaMemcpyAsync(h->chunks_d, by_kind[0].data(), sizeof(HChunk) * chunks.size(), cudaMemcpyHostToDevice, c->stream));
    UCG_CUDA(cudaMemcpyAsync(h->leaf_chunk_d, leaf_chunk.data(), sizeof(int) * leaf_chunk.size(), cudaMemcpyHostToDevice, c->stream));
    UCG_CUDA(cudaMemcpyAsync(h->leaf_e0_d, leaf_e0.data(), sizeof(int) * leaf_e0.size(), cudaMemcpyHostToDevice, c->stream));
    UCG_CUDA(cudaEventRecord(ev1, c->stream));
    UCG_CUDA(cudaEventSynchronize(ev1));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    h->build_ms = ms;
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    return UCG_OK;
}

// A build that fails leaves no matrix: its parts would be taken for one.
int hmatrix_build(ucg_ctx *c, int okada_mode, double eta, double eps, int leaf)
{
    std::vector<void *> temp_allocs;
    int rc = build_matrix(c, okada_mode, eta, eps, leaf, temp_allocs);
    // the split planes belong to the matrix that a run in the split form reads
    if (!rc && c->precision == UCG_PREC_HMATRIX_SPLIT) rc = hmatrix_split_build(c);
    if (!rc) return UCG_OK;
    cudaStreamSynchronize(c->stream);
    for (void *p : temp_allocs) cudaFree(p);
    hmatrix_free(c);
    return rc;
}

// the chunks' partial row sums of H xp (split: of its FP32 planes), enqueued on
// the context stream
template <bool SPLIT>
static cudaError_t launch_products(ucg_ctx *c)
{
    HMat *h = c->hm;
    const HmProduct P{h->lr_d, h->items_d, h->n_items, h->terms_d, h->chunks_d, h->n_dense_chunks, h->panel,
                      h->ph, h->pl, h->vh, h->vl, h->xp_d, h->z_d, h->part_d, 3 * h->max_leaf, h->status_d};
    const size_t smem = (SPLIT ? HM_CHUNK_BYTES / 2 : HM_CHUNK_BYTES) + sizeof(double) * h->max_cols;
    const int thr = (3 * h->max_leaf + 31) & ~31;
    const int zb = (int)((h->n_items * 32 + thr - 1) / thr), lowrank = h->n_chunks - h->n_dense_chunks;
    cudaError_t e = launch_pdl(k_hm_rows<SPLIT, true>, dim3(zb + h->n_dense_chunks), dim3(thr), smem, c->stream, P, zb);
    c->launches.count++;
    if (e == cudaSuccess && lowrank > 0) {
        e = launch_pdl(k_hm_rows<SPLIT, false>, dim3(lowrank), dim3(thr), smem, c->stream, P, 0);
        c->launches.count++;
    }
    return e;
}

cudaError_t hmatrix_products(ucg_ctx *c, bool split)
{
    return split ? launch_products<true>(c) : launch_products<false>(c);
}

HmParts hmatrix_parts(const ucg_ctx *c)
{
    const HMat *h = c->hm;
    return HmParts{h->leaf_e0_d, h->leaf_chunk_d, h->perm_d, h->part_d, h->xp_d, 3 * h->max_leaf, h->n_leaves};
}

// t = H v (K's row order), enqueued on the context stream
cudaError_t hmatrix_apply(ucg_ctx *c, const double *v, double *t)
{
    HMat *h = c->hm;
    k_hm_gather<<<(h->np + 255) / 256, 256, 0, c->stream>>>(h->perm_d, h->np, v, h->xp_d);
    const cudaError_t e = hmatrix_products(c, false);
    if (e != cudaSuccess) return e;
    const int rows = 3 * h->max_leaf, gs = ((rows + 31) / 32) * 32, nthr = std::max(gs, (1024 / gs) * gs);
    k_hm_reduce<<<h->n_leaves, nthr, sizeof(double) * nthr, c->stream>>>(h->leaf_e0_d, h->leaf_chunk_d, h->perm_d,
                                                                         h->part_d, rows, t, gs);
    c->launches.count += 2;
    return cudaGetLastError();
}

// hi / lo planes of the FP32 copies of the panels and of V (once; kept with the matrix)
int hmatrix_split_build(ucg_ctx *c)
{
    HMat *h = c->hm;
    if (!h) return UCG_E_STATE;
    if (h->ph) return UCG_OK;
    long vn = 0;
    for (const HLowRank &b : h->lr_h) vn += (long)b.k * b.n;
    const long pn = std::max<long>(h->panel_len, 8);
    UCG_CUDA(cudaMalloc(&h->ph, sizeof(__nv_bfloat16) * pn));
    UCG_CUDA(cudaMalloc(&h->pl, sizeof(__nv_bfloat16) * pn));
    UCG_CUDA(cudaMalloc(&h->vh, sizeof(__nv_bfloat16) * std::max<long>(vn, 8)));
    UCG_CUDA(cudaMalloc(&h->vl, sizeof(__nv_bfloat16) * std::max<long>(vn, 8)));
    if (h->panel_len > 0) {
        k_split_flat<<<8 * c->sms, 256, 0, c->stream>>>(h->panel, h->panel_len, h->ph, h->pl);
        c->launches.count++;
    }
    std::vector<SplitJob> jobs;
    for (const HLowRank &b : h->lr_h)
        if (b.k > 0) jobs.push_back({b.V, (long)b.k * b.n, b.vsoff});
    if (!jobs.empty()) {
        SplitJob *jd = nullptr;
        UCG_CUDA(cudaMalloc(&jd, sizeof(SplitJob) * jobs.size()));
        UCG_CUDA(cudaMemcpyAsync(jd, jobs.data(), sizeof(SplitJob) * jobs.size(), cudaMemcpyHostToDevice, c->stream));
        k_split_jobs<<<(int)jobs.size(), 256, 0, c->stream>>>(jd, h->vh, h->vl);
        c->launches.count++;
        UCG_CUDA(cudaStreamSynchronize(c->stream));
        cudaFree(jd);
    }
    UCG_CUDA(cudaStreamSynchronize(c->stream));
    return UCG_OK;
}

double *hmatrix_t(ucg_ctx *c) { return c->hm ? c->hm->t_d : nullptr; }

bool hmatrix_layout(const ucg_ctx *c, HLayout *out)
{
    const HMat *h = c->hm;
    if (!h) return false;
    out->np = h->np;
    out->n_leaves = h->n_leaves;
    out->tree_leaf = h->tree_leaf;
    out->perm = h->perm;
    out->leaf_e0 = h->leaf_e0_h;
    out->leaf_term0 = h->leaf_term0_h;
    out->terms.clear();
    for (size_t q = 0; q < h->terms_h.size(); q++) {
        const HLeafTerm &T = h->terms_h[q];
        out->terms.push_back({h->term_poff_h[q], T.cols, T.xsel, T.xoff});
    }
    out->lr.clear();
    for (const HLowRank &b : h->lr_h) out->lr.push_back({b.V, b.k, b.n, b.s0, b.zoff, b.r0, b.m});
    out->panel = h->panel;
    return true;
}

void hmatrix_info(const ucg_ctx *c, long *n_dense, long *n_lowrank, long *n_fallback, size_t *bytes, int *max_rank,
                  double *build_ms)
{
    const HMat *h = c->hm;
    if (n_dense) *n_dense = h ? h->n_dense + h->n_fallback : 0;
    if (n_lowrank) *n_lowrank = h ? h->n_lowrank : 0;
    if (n_fallback) *n_fallback = h ? h->n_fallback : 0;
    if (bytes) *bytes = h ? h->bytes : 0;
    if (max_rank) *max_rank = h ? h->max_rank : 0;
    if (build_ms) *build_ms = h ? h->build_ms : 0.0;
}

}  // namespace ucg
