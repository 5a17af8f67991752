// Gauss-Seidel row updates shared by the stationary multigrid (dv_gmg.cu) and
// the V-cycle of the multigrid-preconditioned CG (dv_mgpcg.cuh).
//
// Row update x_i = (b_i - sum_{j != i} a_ij x_j) / a_ii in column order, each
// product and difference rounded separately (GaussSeidelIterationCsrDuVi.cs:22-50).
// A launch updates the rows of one independent group: one dependency level of
// the forward sweep (the reference's own order) or the node blocks of one color.
#pragma once

#include "dv_kernels.cuh"

namespace dvk {

template <class T> __device__ __forceinline__ T rn_mul(T a, T b);
template <> __device__ __forceinline__ double rn_mul<double>(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ float rn_mul<float>(float a, float b) { return __fmul_rn(a, b); }
template <class T> __device__ __forceinline__ T rn_sub(T a, T b);
template <> __device__ __forceinline__ double rn_sub<double>(double a, double b) { return __dsub_rn(a, b); }
template <> __device__ __forceinline__ float rn_sub<float>(float a, float b) { return __fsub_rn(a, b); }
template <class T> __device__ __forceinline__ T rn_div(T a, T b);
template <> __device__ __forceinline__ double rn_div<double>(double a, double b) { return __ddiv_rn(a, b); }
template <> __device__ __forceinline__ float rn_div<float>(float a, float b) { return __fdiv_rn(a, b); }

template <class T>
__device__ __forceinline__ void gs_row_csr(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                           const T *__restrict__ va, const T *__restrict__ b, T *x, int32_t i) {
    T s = b[i], d = T(0);
    for (int32_t k = rp[i]; k < rp[i + 1]; ++k) {
        const int32_t c = ci[k];
        const T a = va[k];
        if (c != i) s = rn_sub<T>(s, rn_mul<T>(a, ((volatile T *)x)[c]));
        else d = a;
    }
    x[i] = rn_div<T>(s, d);
}

template <class VI, class T>
__device__ __forceinline__ void gs_row_duvi(const DuviArgs &A, const T *__restrict__ b, T *x, int32_t i) {
    const T *tab = static_cast<const T *>(A.values);
    const VI *vi = static_cast<const VI *>(A.vidx);
    T s = b[i], d = T(0);
    uint32_t di = A.row_to_dist[i];
    for (uint32_t bl = A.row_to_col[i]; bl < A.row_to_col[i + 1]; ++bl) {
        uint32_t c = A.col_idx[bl];
        const int cnt = A.dist[di];
        for (int k = 0;; ++k) {
            const T a = tab[vi[di]];
            if ((int32_t)c != i) s = rn_sub<T>(s, rn_mul<T>(a, ((volatile T *)x)[c]));
            else d = a;
            ++di;
            if (k == cnt) break;
            c += A.dist[di] + 1u;
        }
    }
    x[i] = rn_div<T>(s, d);
}

// rows[0..count): first rows of the group's blocks of bs consecutive rows
template <class T>
__global__ void k_gs_csr(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci, const T *__restrict__ va,
                         const T *__restrict__ b, T *x, const int32_t *__restrict__ rows, int32_t count, int bs,
                         const int *__restrict__ done) {
    if (chain_done(done)) return;
    for (int32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const int32_t r0 = rows[t];
        for (int q = 0; q < bs; ++q) gs_row_csr<T>(rp, ci, va, b, x, r0 + q);
    }
}
template <class VI, class T>
__global__ void k_gs_duvi(DuviArgs A, const T *__restrict__ b, T *x, const int32_t *__restrict__ rows, int32_t count,
                          int bs, const int *__restrict__ done) {
    if (chain_done(done)) return;
    for (int32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const int32_t r0 = rows[t];
        for (int q = 0; q < bs; ++q) gs_row_duvi<VI, T>(A, b, x, r0 + q);
    }
}

// Multicolor node-block update on the node-pattern layout: one thread per node of the color,
// its pattern's records from shared memory.  One pass over the records gathers every column
// of another node once and subtracts it from all three rows (fused multiply-adds); the node's
// own 3 x 3 block is then solved row by row in order, each row using the rows of the node
// already updated in this sweep and the old values of the later ones (the block Gauss-Seidel
// step of the raw kernels above, with the neighbour sum taken first).
template <class T>
__global__ void __launch_bounds__(256) k_gs_pattern(const uint16_t *__restrict__ pid, const uint32_t *__restrict__ pstart,
                                                    const PatRec<T> *__restrict__ grec, int32_t npat, int32_t nrec,
                                                    const T *__restrict__ b, T *x, const int32_t *__restrict__ rows,
                                                    int32_t count, const int *__restrict__ done) {
    if (chain_done(done)) return;
    extern __shared__ uint4 gs_smem[];
    const PatRec<T> *rec = reinterpret_cast<const PatRec<T> *>(gs_smem);
    const uint32_t *st = reinterpret_cast<const uint32_t *>(rec + nrec);
    stage_patterns<T>(gs_smem, grec, pstart, npat, nrec);
    __syncthreads();
    for (int32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const int32_t r0 = rows[t];
        const uint32_t p = __ldg(pid + r0 / 3);
        const uint32_t kb = st[p], ke = st[p + 1];
        T s0 = b[r0], s1 = b[r0 + 1], s2 = b[r0 + 2];
        T a[3][3] = {{T(0), T(0), T(0)}, {T(0), T(0), T(0)}, {T(0), T(0), T(0)}};
#pragma unroll 4
        for (uint32_t k = kb; k < ke; ++k) {
            const PatRec<T> q = rec[k];
            if (q.off >= 0 && q.off < 3) {   // the node's own block, column q.off
                if (q.off == 0) { a[0][0] = q.v[0]; a[1][0] = q.v[1]; a[2][0] = q.v[2]; }
                else if (q.off == 1) { a[0][1] = q.v[0]; a[1][1] = q.v[1]; a[2][1] = q.v[2]; }
                else { a[0][2] = q.v[0]; a[1][2] = q.v[1]; a[2][2] = q.v[2]; }
                continue;
            }
            const T xv = __ldg(x + (r0 + q.off));
            s0 = fma(-q.v[0], xv, s0);
            s1 = fma(-q.v[1], xv, s1);
            s2 = fma(-q.v[2], xv, s2);
        }
        const T x1o = x[r0 + 1], x2o = x[r0 + 2];
        const T x0 = (s0 - a[0][1] * x1o - a[0][2] * x2o) / a[0][0];
        const T x1 = (s1 - a[1][0] * x0 - a[1][2] * x2o) / a[1][1];
        const T x2 = (s2 - a[2][0] * x0 - a[2][1] * x1) / a[2][2];
        x[r0] = x0;
        x[r0 + 1] = x1;
        x[r0 + 2] = x2;
    }
}

// ---------------------------------------------------------------------------
// Forward sweeps in the reference's row order by one block, for systems whose x fits its shared
// memory
//
// A dependency level of a small system holds a few dozen rows, and a launch per level waits for the
// launch before and then walks each row's entries one after another in one thread.  Here one block
// runs all levels of all sweeps with x in shared memory and a barrier between levels.  A warp takes
// a row: the lanes load its entries (those of the warp's next row are in flight across the
// barrier), form the products a_ij x_j side by side and leave them in shared memory, from where
// they are subtracted one after another in column order: products and differences are rounded
// one by one as in gs_row_csr, so the result is the same bit for bit (the diagonal and the padding
// subtract +0, which changes nothing).  Bound by that chain of dependent subtractions.
// 12 x 4 x 4 elements, two levels, to 1e-3: 950 -> 109 ms (about 12 -> 1.3 us a dependency level).
// ---------------------------------------------------------------------------
constexpr int kGsWarps = 32;
constexpr int kGsLane = 3;   // entries of a row a lane holds at a time (96 a warp)

template <class T>
__global__ void __launch_bounds__(kGsWarps * 32) k_gs_block(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                            const T *__restrict__ va, const T *__restrict__ b, T *x,
                                                            const int32_t *__restrict__ rows,
                                                            const int32_t *__restrict__ off, int32_t nlevels, int32_t n,
                                                            int sweeps, const int *__restrict__ done) {
    if (chain_done(done)) return;
    extern __shared__ uint4 gsb_smem[];
    constexpr int W = 32 * kGsLane;
    T *prod = reinterpret_cast<T *>(gsb_smem) + (threadIdx.x >> 5) * W;   // this warp's products
    T *xs = reinterpret_cast<T *>(gsb_smem) + kGsWarps * W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int32_t i = threadIdx.x; i < n; i += kGsWarps * 32) xs[i] = x[i];
    // a row and the first W of its entries, held by the warp
    struct Row {
        int32_t i, s, len, c[kGsLane];
        T v[kGsLane], b;
    } q;
    auto load = [&](int32_t t) {
        q.i = __ldg(rows + t);
        q.s = __ldg(rp + q.i);
        q.len = __ldg(rp + q.i + 1) - q.s;
        q.b = b[q.i];
#pragma unroll
        for (int u = 0; u < kGsLane; ++u) {
            const int32_t k = lane + 32 * u;
            q.c[u] = k < q.len ? __ldg(ci + q.s + k) : q.i;   // padding: as the diagonal, but without a value
            q.v[u] = k < q.len ? __ldg(va + q.s + k) : T(0);
        }
    };
    const int32_t last = sweeps * nlevels;
    int32_t t0 = __ldg(off), t1 = __ldg(off + 1);
    if (t0 + warp < t1) load(t0 + warp);
    for (int32_t l = 0; l < last; ++l) {
        __syncthreads();   // the rows of the level before are in xs
        int32_t n0 = 0, n1 = 0;   // the next level's rows
        if (l + 1 < last) {
            const int32_t m = (l + 1) % nlevels;
            n0 = __ldg(off + m);
            n1 = __ldg(off + m + 1);
        }
        for (int32_t t = t0 + warp; t < t1; t += kGsWarps) {
            T s = q.b, d = T(0);
            const int32_t i = q.i;
            for (int32_t k0 = 0;; k0 += W) {
                const int32_t cnt = min(W, q.len - k0);
#pragma unroll
                for (int u = 0; u < kGsLane; ++u) {
                    const bool diag = q.c[u] == i;
                    if (diag && k0 + lane + 32 * u < q.len) d = q.v[u];
                    prod[lane + 32 * u] = diag ? T(0) : rn_mul<T>(q.v[u], xs[q.c[u]]);
                }
                __syncwarp();
#pragma unroll 4
                for (int32_t k = 0; k < cnt; k += 4) {   // W is a multiple of 4: the padding subtracts +0
                    T p[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[u] = prod[k + u];
#pragma unroll
                    for (int u = 0; u < 4; ++u) s = rn_sub<T>(s, p[u]);
                }
                __syncwarp();
                if (k0 + W >= q.len) break;
#pragma unroll
                for (int u = 0; u < kGsLane; ++u) {   // the next W entries of a longer row
                    const int32_t k = k0 + W + lane + 32 * u;
                    q.c[u] = k < q.len ? __ldg(ci + q.s + k) : i;
                    q.v[u] = k < q.len ? __ldg(va + q.s + k) : T(0);
                }
            }
            // the next row of this warp, in this level or the next one
            const bool more = t + kGsWarps < t1;
            const unsigned has = __ballot_sync(0xffffffffu, d != T(0));
            d = __shfl_sync(0xffffffffu, d, has ? __ffs(has) - 1 : 0);
            if (more) load(t + kGsWarps);
            else if (n0 + warp < n1) load(n0 + warp);
            if (lane == 0) xs[i] = rn_div<T>(s, d);
        }
        if (t0 + warp >= t1 && n0 + warp < n1) load(n0 + warp);   // no row in this level
        t0 = n0;
        t1 = n1;
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += kGsWarps * 32) x[i] = xs[i];
}

// ---------------------------------------------------------------------------
// The same by node groups: 3 consecutive rows with one column list of at most 96 columns.  A warp takes
// a node, with a barrier per level of nodes (a third of the rows' levels).  Every product with another
// node's value is formed at once; lanes 0 .. 2 subtract the three rows' products up to the node's own
// columns side by side, then row by row the node's own terms (new values of the rows before, old ones
// of the rows after), the rest of the row and the division: 39 + 3 x 41 subtractions after one
// another for a hex node instead of 3 x 81, in each row's own order.  The next node's entries are
// loaded while they run.  12 x 4 x 4 elements, two levels, to 1e-3: 91.9 -> 82.0 ms (3.1 us a level of nodes).
// ---------------------------------------------------------------------------
constexpr int kGsCols = 96;          // columns of a node, 3 a lane
constexpr int kGsStride = kGsCols + 2;   // a row's products in shared memory: the three lanes' loads in different banks

template <class T>
__global__ void __launch_bounds__(kGsWarps * 32) k_gs_block_nodes(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                                  const T *__restrict__ va, const T *__restrict__ b, T *x,
                                                                  const int32_t *__restrict__ nodes,
                                                                  const int32_t *__restrict__ off, int32_t nlevels,
                                                                  int32_t n, int sweeps, const int *__restrict__ done) {
    if (chain_done(done)) return;
    extern __shared__ uint4 gsb_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T *prod = reinterpret_cast<T *>(gsb_smem) + warp * (3 * kGsStride + 9);   // this warp's products, own 3 x 3 block
    T *block = prod + 3 * kGsStride;
    T *xs = reinterpret_cast<T *>(gsb_smem) + kGsWarps * (3 * kGsStride + 9);
    for (int32_t i = threadIdx.x; i < n; i += kGsWarps * 32) xs[i] = x[i];
    const int row = min(lane, 2);
    struct Node {
        int32_t node, len, c[3];
        T v[3][3], b;
    } q;
    auto load = [&](int32_t t) {
        q.node = __ldg(nodes + t);
        const int32_t s = __ldg(rp + 3 * q.node);
        q.len = __ldg(rp + 3 * q.node + 1) - s;
        q.b = b[3 * q.node + row];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const int32_t k = lane + 32 * u;
            q.c[u] = k < q.len ? __ldg(ci + s + k) : 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) q.v[u][d] = k < q.len ? __ldg(va + s + d * q.len + k) : T(0);
        }
    };
    const int32_t last = sweeps * nlevels;
    int32_t t0 = __ldg(off), t1 = __ldg(off + 1);
    if (t0 + warp < t1) load(t0 + warp);
    for (int32_t l = 0; l < last; ++l) {
        __syncthreads();   // the nodes of the level before are in xs
        int32_t n0 = 0, n1 = 0;   // the next level's nodes
        if (l + 1 < last) {
            const int32_t m = (l + 1) % nlevels;
            n0 = __ldg(off + m);
            n1 = __ldg(off + m + 1);
        }
        for (int32_t t = t0 + warp; t < t1; t += kGsWarps) {
            const int32_t r0 = 3 * q.node, len = q.len;
            int first = len, own = 0;   // the node's own columns: position of the first, and which of the three are there
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const int32_t k = lane + 32 * u, o = q.c[u] - r0;
                const bool mine = k < len && o >= 0 && o < 3;
                const unsigned m = __ballot_sync(0xffffffffu, mine);
                if (m && first == len) first = 32 * u + __ffs(m) - 1;
#pragma unroll
                for (int e = 0; e < 3; ++e)
                    if (__ballot_sync(0xffffffffu, mine && o == e)) own |= 1 << e;
                const T xv = xs[q.c[u]];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    if (mine) block[3 * d + o] = q.v[u][d];
                    prod[d * kGsStride + k] = mine || k >= len ? T(0) : rn_mul<T>(q.v[u][d], xv);
                }
            }
            T s = q.b;
            __syncwarp();
            const bool more = t + kGsWarps < t1;
            if (more) load(t + kGsWarps);
            else if (n0 + warp < n1) load(n0 + warp);
            const T *pr = prod + row * kGsStride;
            const T *ar = block + 3 * row;
#pragma unroll 8
            for (int k = 0; k < first; ++k) s = rn_sub<T>(s, pr[k]);
            T xn[3] = {xs[r0], xs[r0 + 1], xs[r0 + 2]};   // old values, replaced row by row
            const int rest = first + __popc(own);
#pragma unroll
            for (int d = 0; d < 3; ++d) {   // row d: lane d's result counts
                T w = s;
#pragma unroll
                for (int o = 0; o < 3; ++o)
                    if (o != d && ((own >> o) & 1)) w = rn_sub<T>(w, rn_mul<T>(ar[o], xn[o]));
#pragma unroll 8
                for (int k = rest; k < len; ++k) w = rn_sub<T>(w, pr[k]);
                w = rn_div<T>(w, (own >> d) & 1 ? block[4 * d] : T(0));
                xn[d] = __shfl_sync(0xffffffffu, w, d);
            }
            if (lane < 3) xs[r0 + lane] = lane == 0 ? xn[0] : lane == 1 ? xn[1] : xn[2];
            __syncwarp();
        }
        if (t0 + warp >= t1 && n0 + warp < n1) load(n0 + warp);   // no node in this level
        t0 = n0;
        t1 = n1;
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += kGsWarps * 32) x[i] = xs[i];
}

// Row groups of one Gauss-Seidel ordering (device rows + host group offsets).
struct GsOrder {
    DevMem rows;
    std::vector<int32_t> off;
    int bs = 1;
    bool lex = false;
    bool block = false;          // swept by one block (k_gs_block): level offsets and, for DuVi, the entries
    bool nodes = false;          // ... by node groups (k_gs_block_nodes): d_nodes in levels d_off
    int32_t nlevels = 0;
    DevMem d_off, d_nodes, col, val;
};

// Builds the ordering: lex = dependency levels of the forward sweep (rows);
// otherwise a greedy coloring of node blocks (3 or 2 consecutive rows when the size allows).
inline void gs_build_order(const dv_csr_host &a, bool lex, cudaStream_t s, GsOrder &o) {
    std::vector<int32_t> rows;
    o.lex = lex;
    if (lex) {
        dv_gs_level_sets(a, rows, o.off);
        o.bs = 1;
    } else {
        o.bs = (a.n_rows % 3 == 0) ? 3 : (a.n_rows % 2 == 0 ? 2 : 1);
        std::vector<int32_t> color;
        const int nc = dv_block_coloring(a, o.bs, color);
        o.off.assign(nc + 1, 0);
        rows.resize(color.size());
        for (int32_t c : color) o.off[c + 1]++;
        for (int c = 0; c < nc; ++c) o.off[c + 1] += o.off[c];
        std::vector<int32_t> fill(o.off.begin(), o.off.end() - 1);
        for (size_t b = 0; b < color.size(); ++b) rows[fill[color[b]]++] = (int32_t)b * o.bs;
    }
    o.rows.alloc(4 * rows.size());
    DV_CUDA(cudaMemcpyAsync(o.rows.p, rows.data(), 4 * rows.size(), cudaMemcpyHostToDevice, s));
    DV_CUDA(cudaStreamSynchronize(s));
}

template <class T>
constexpr size_t gs_block_smem(int32_t n, bool nodes) {
    return sizeof(T) * ((size_t)n + kGsWarps * (nodes ? 3 * kGsStride + 9 : 32 * kGsLane));
}

// Whether one block sweeps these levels faster than a launch a level does: its warps take 32 rows or nodes at a
// time, at most `passes` times a level on average.  Measured at 19,200 rows, a level by the block against a launch
// (FP64, 5 / 27 / 81 entries a row): 96 rows 3.4 / 4.2 / 5.7 against 8.4 / 12 / 18 us, 192 rows 6.4 / 7.8 / 12
// against 7.0 / 11 / 19, 384 rows 12 / 15 / 25 against 7.1 / 11 / 20: six passes of rows.  By node groups (9 / 81
// entries a row, a level of nodes against three of rows): 256 nodes 20 / 36 against 26 / 68 us, 512 nodes
// 36 / 68 against 27 / 67: ten passes of nodes.
inline bool gs_levels_narrow(const std::vector<int32_t> &off, int passes) {
    int64_t need = 0;
    for (size_t l = 0; l + 1 < off.size(); ++l) need += (off[l + 1] - off[l] + kGsWarps - 1) / kGsWarps;
    return need <= passes * (int64_t)(off.size() - 1);
}

// Prepares the one-block sweep of A's row-order levels (a: its host copy) where x fits a block's shared
// memory (FP64 up to 25,856 rows, by node groups up to 19,232) and the levels are narrow; wide levels (a
// red-black or a nearly diagonal matrix, as against a hex grid's few dozen rows) stay a launch each over all SMs.
template <class T>
void gs_prepare_block(const dv_matrix *A, const dv_csr_host &a, GsOrder &o) {
    dv_context *ctx = A->ctx;
    const size_t room = (size_t)ctx->max_smem_optin - 1024;
    if (!o.lex || A->n_rows == 0 || gs_block_smem<T>(A->n_rows, false) > room) return;
    cudaStream_t s = ctx->stream;
    std::vector<int32_t> perm, off;
    bool nodes = gs_block_smem<T>(A->n_rows, true) <= room && dv_csr_row_group(a) == 3;
    for (int32_t i = 0; i < a.n_rows && nodes; i += 3) nodes = a.rowptr[i + 1] - a.rowptr[i] <= kGsCols;
    if (nodes) dv_gs_node_level_sets(a, perm, off);
    if (nodes ? !gs_levels_narrow(off, 10) : !gs_levels_narrow(o.off, 6)) return;
    o.nodes = nodes;
    if (o.nodes) {
        o.d_nodes.alloc(4 * perm.size());
        DV_CUDA(cudaMemcpyAsync(o.d_nodes.p, perm.data(), 4 * perm.size(), cudaMemcpyHostToDevice, s));
    } else {
        off = o.off;
    }
    o.nlevels = (int32_t)off.size() - 1;
    o.d_off.alloc(4 * off.size());
    DV_CUDA(cudaMemcpyAsync(o.d_off.p, off.data(), 4 * off.size(), cudaMemcpyHostToDevice, s));
    if (A->format == DV_FORMAT_DUVI) {
        o.col.alloc(4 * (size_t)A->nnz);
        o.val.alloc(sizeof(T) * (size_t)A->nnz);
        duvi_decode<T>(A, o.col.as<int32_t>(), o.val.as<T>());
    }
    DV_CUDA(cudaStreamSynchronize(s));
    o.block = true;
}

// One forward sweep over all groups of the ordering (x updated in place).
template <class T>
void gs_sweep(const LaunchEnv &e, const dv_matrix *A, const GsOrder &o, const T *b, T *x) {
    dv_context *ctx = e.ctx;
    const int32_t ngroups = (int32_t)o.off.size() - 1;
    for (int32_t q = 0; q < ngroups; ++q) {
        const int32_t cnt = o.off[q + 1] - o.off[q];
        const int32_t *rows = o.rows.as<int32_t>() + o.off[q];
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((cnt + kThreads - 1) / kThreads, ctx->num_sms * 8));
        if (o.bs == 3 && A->format == DV_FORMAT_DUVI && A->pat_ok && A->lanes_group == 3 && !A->pat_based &&
            sizeof(T) == (A->precision == DV_F64 ? 8 : 4)) {
            // node blocks of one color on the pattern layout
            const size_t smem = sizeof(PatRec<T>) * (size_t)A->pat_entries + 4 * ((size_t)A->pat_count + 1);
            static SmemLimit limit;   // per instantiation and device
            limit.raise(k_gs_pattern<T>, smem, ctx->device);
            launch_chain(k_gs_pattern<T>, grid, kThreads, smem, e.stream, A->pat_id.as<uint16_t>(), A->pat_start.as<uint32_t>(),
                                                               static_cast<const PatRec<T> *>(A->pat_rec.p),
                                                               A->pat_count, A->pat_entries, b, x, rows, cnt, e.done);
        } else if (A->format == DV_FORMAT_CSR) {
            launch_chain(k_gs_csr<T>, grid, kThreads, 0, e.stream, A->rowptr.as<int32_t>(), A->col.as<int32_t>(),
                                                         static_cast<const T *>(A->val.p), b, x, rows, cnt, o.bs, e.done);
        } else if (A->vi_bits == 8) {
            launch_chain(k_gs_duvi<uint8_t, T>, grid, kThreads, 0, e.stream, duvi_args(A), b, x, rows, cnt, o.bs, e.done);
        } else if (A->vi_bits == 16) {
            launch_chain(k_gs_duvi<uint16_t, T>, grid, kThreads, 0, e.stream, duvi_args(A), b, x, rows, cnt, o.bs, e.done);
        } else {
            launch_chain(k_gs_duvi<uint32_t, T>, grid, kThreads, 0, e.stream, duvi_args(A), b, x, rows, cnt, o.bs, e.done);
        }
        DV_CUDA(cudaGetLastError());
        ctx->count();
    }
}

// `sweeps` forward sweeps.
template <class T>
void gs_sweeps(const LaunchEnv &e, const dv_matrix *A, const GsOrder &o, const T *b, T *x, int sweeps) {
    if (!o.block) {
        for (int k = 0; k < sweeps; ++k) gs_sweep<T>(e, A, o, b, x);
        return;
    }
    if (sweeps < 1) return;
    const bool csr = A->format == DV_FORMAT_CSR;
    const int32_t *rp = csr ? A->rowptr.as<int32_t>() : A->row_to_dist.as<int32_t>();
    const int32_t *col = csr ? A->col.as<int32_t>() : o.col.as<int32_t>();
    const T *val = csr ? static_cast<const T *>(A->val.p) : o.val.as<T>();
    const size_t smem = gs_block_smem<T>(A->n_rows, o.nodes);
    auto kern = o.nodes ? k_gs_block_nodes<T> : k_gs_block<T>;
    static SmemLimit limit[2];   // per kernel, instantiation and device
    limit[o.nodes].raise(kern, smem, e.ctx->device);
    launch_chain(kern, 1, kGsWarps * 32, smem, e.stream, rp, col, val, b, x, (o.nodes ? o.d_nodes : o.rows).template as<int32_t>(),
                 o.d_off.as<int32_t>(), o.nlevels, A->n_rows, sweeps, e.done);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

}  // namespace dvk
