// Device kernels of libduvigpu.so for sm_100a.
//
// The sparse path is HBM-bound integer/byte decode plus FMAs (about 0.1 flop
// per byte), so there are no tensor-core tiles here: the kernels are built
// around coalesced 16-byte staging of the index/byte streams into shared
// memory, L2-resident gathers of the vector, warp-shuffle reductions and
// epilogues that fuse the vector updates of each algorithm step into the
// pass over the matrix.
#pragma once

#include <cstddef>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <utility>

#include "dv_internal.cuh"

#include <cuda_runtime.h>

namespace dvk {

constexpr int kThreads = 256;            // CSR and vector kernels
constexpr int kDuviWarps = 8;            // warps per block, staged DuVi kernel (8/16-bit indices)
constexpr int kDuviWarps32 = 4;          // 32-bit value indices (larger stage)
constexpr int kStageD = 3072;            // per-warp stage of entry bytes (>= kBundleBytes + 32)
constexpr int kStageC = 512;             // per-warp stage of block column starts (>= kBundleBlocks + 8)
constexpr int kMaxRed = 4;               // doubles per block in a grid reduction

static_assert(kStageD >= kBundleBytes + 32, "stage too small");
static_assert(kStageC >= kBundleBlocks + 8, "column stage too small");

// The dynamic shared memory a kernel may use is an attribute of each device: a
// launcher raises it to every new largest size on each device it launches on.
// Host threads may launch on several contexts at once: the caches of launch settings
// below are updated under one lock, so a raise never lowers a limit another thread set.
inline std::mutex &launch_cache_mutex() {
    static std::mutex m;
    return m;
}

constexpr int kMaxDevices = 64;
struct SmemLimit {
    size_t set[kMaxDevices] = {};
    template <class K>
    void raise(K kern, size_t smem, int device) {
        DV_REQUIRE(device >= 0 && device < kMaxDevices, DV_ERR_ARG, "device ordinal out of range");
        std::lock_guard<std::mutex> lock(launch_cache_mutex());
        if (smem > set[device]) {
            DV_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            set[device] = smem;
        }
    }
};

// Resident blocks per SM of a kernel at a dynamic shared-memory size on a device (occupancy
// query, remembered for the last few (device, size) pairs; the current device is `device`).
struct OccupancyCache {
    size_t smem[8] = {};
    int dev[8] = {};
    int blocks[8] = {};
    int next = 0;
    template <class K>
    int get(K kern, int threads, size_t smem_bytes, int device) {
        std::lock_guard<std::mutex> lock(launch_cache_mutex());
        for (int i = 0; i < 8; ++i)
            if (blocks[i] > 0 && smem[i] == smem_bytes && dev[i] == device) return blocks[i];
        int occ = 0;
        DV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem_bytes));
        occ = std::max(occ, 1);
        smem[next] = smem_bytes;
        dev[next] = device;
        blocks[next] = occ;
        next = (next + 1) % 8;
        return occ;
    }
};

// ---------------------------------------------------------------------------
// chains of dependent kernels
//
// The kernels of an iteration depend on one another and are short on all but the finest levels, so the
// time from the last block of one to the first of the next counts.  They are launched with
// programmatic stream serialisation: a kernel's blocks may be set up when the blocks of the one before
// have left, and wait (griddepcontrol.wait) for that kernel's writes to be visible before they touch
// anything but constant tables.  Every kernel launched by launch_chain calls chain_done first (a kernel
// that did not wait could complete before the one it depends on, and release the next), and what it
// reads comes after the branch on its result.  With against without: mixed solve 16^3 963 -> 845 us,
// 12 uneven meshes 2.34 -> 2.13 ms, adjoint pair 48x24x24 8.10 -> 7.50 ms, mixed solve 128^3 7.49 -> 7.27
// ms, a product of 1,200 rows called over and over 4.0 -> 3.5 us.  Letting the next kernel's blocks in
// as soon as all of this one's have started (griddepcontrol.launch_dependents) was slower for all but
// the smallest: they settle on the SMs that happen to have room and stay there (adjoint pair 9.3 ms).
// DV_CHAIN=0 launches plainly (A/B comparisons).
// ---------------------------------------------------------------------------
// waits for the kernel before; then whether the solve has stopped
__device__ __forceinline__ bool chain_done(const int *done) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return done && *(volatile const int *)done;
}
template <class... P, class... A>
void launch_chain(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
    static const bool on = [] {
        const char *v = getenv("DV_CHAIN");
        return !(v && v[0] == '0');
    }();
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute serial = {};
    serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    serial.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &serial;
    c.numAttrs = on ? 1 : 0;
    DV_CUDA(cudaLaunchKernelEx(&c, kern, static_cast<P>(args)...));
}

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// Sum over aligned groups of W lanes (all lanes of a group must be converged).
template <int W, class T>
__device__ __forceinline__ T group_sum(T v) {
    if constexpr (W == 1) {
        return v;
    } else {
        const unsigned lane = threadIdx.x & 31u;
        const unsigned mask = (W == 32) ? 0xffffffffu : (((1u << W) - 1u) << (lane & ~(unsigned)(W - 1)));
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
        return v;
    }
}

// Block reduction of N doubles: bit i of MAXMASK selects max instead of sum.
// Result valid in thread 0.  All threads of the block must call it.
template <int N, unsigned MAXMASK>
__device__ void block_reduce(double (&v)[N]) {
    __shared__ double sh[kMaxRed][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        double t = ((MAXMASK >> i) & 1u) ? warp_max(v[i]) : warp_sum(v[i]);
        if (lane == 0) sh[i][warp] = t;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            double t = lane < nw ? sh[i][lane] : 0.0;
            v[i] = ((MAXMASK >> i) & 1u) ? warp_max(t) : warp_sum(t);
        }
    }
    __syncthreads();
}

// Deterministic grid reduction: per-block partials, then the last block to
// arrive sums them in block order.  Returns true in thread 0 of the last block,
// with the totals in out.  Resets the ticket for the next launch.
template <int N, unsigned MAXMASK>
__device__ bool grid_reduce(double (&v)[N], double *partials, unsigned *ticket, double (&out)[N]) {
    block_reduce<N, MAXMASK>(v);
    __shared__ int is_last;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) partials[(size_t)blockIdx.x * N + i] = v[i];
        __threadfence();
        unsigned t = atomicAdd(ticket, 1u);
        is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    double acc[N];
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int i = 0; i < N; ++i) {
            double p = __ldcg(partials + (size_t)b * N + i);
            acc[i] = ((MAXMASK >> i) & 1u) ? fmax(acc[i], p) : acc[i] + p;
        }
    block_reduce<N, MAXMASK>(acc);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) out[i] = acc[i];
        *ticket = 0;
        return true;
    }
    return false;
}

// ---------------------------------------------------------------------------
// gathers: value of the vector at a column (the x of y = A x)
// ---------------------------------------------------------------------------
template <class XT, class AT>
struct GatherVec {
    const XT *__restrict__ x;
    __device__ __forceinline__ AT operator()(uint32_t c) const { return (AT)__ldg(x + c); }
};
// x = w .* b on the fly: the first Jacobi sweep from a zero guess fused into the second.
template <class T>
struct GatherWB {
    const T *__restrict__ w;
    const T *__restrict__ b;
    __device__ __forceinline__ T operator()(uint32_t c) const { return __ldg(w + c) * __ldg(b + c); }
};

// Multiply-add policy: FP64 paths round the product and the sum separately
// (bit-identical to the reference's sequential kernels and to the .NET CPU
// code); FP32 V-cycle paths contract to FMA.
template <class AT>
__device__ __forceinline__ AT madd(AT acc, AT a, AT b);
template <>
__device__ __forceinline__ double madd<double>(double acc, double a, double b) { return __dadd_rn(acc, __dmul_rn(a, b)); }
template <>
__device__ __forceinline__ float madd<float>(float acc, float a, float b) { return fmaf(a, b, acc); }

// Epilogues that set FUSED = true accept one fused multiply-add per term in FP64
// (more accurate, half the FP64 operations); all others keep the reference's order
// of a rounded product followed by a rounded add.
template <class Op, class = void>
struct op_fused : std::false_type {};
template <class Op>
struct op_fused<Op, std::void_t<decltype(Op::FUSED)>> : std::integral_constant<bool, Op::FUSED> {};
template <class AT, bool FUSED>
__device__ __forceinline__ AT madd_op(AT acc, AT a, AT b) {
    if constexpr (FUSED) return fma(a, b, acc);
    else return madd<AT>(acc, a, b);
}

// ---------------------------------------------------------------------------
// epilogues (row operators).  Each has NRED reduction slots and MAXMASK.  load(r) reads what row r
// needs and store(r, sum, loaded, slots) finishes it: a thread that finishes several rows loads for all of
// them before it stores the first (finish_rows), because no load may pass a store to an array it
// might alias, and a load, a store, a load, a store .. is a chain of full memory latencies (mixed solve
// 128^3 7.24 -> 6.82 ms, its FP32 residual 38.1 -> 36.2 us, 64 load cases on 48^3 35.0 -> 33.7 ms).
// An epilogue may define touch(r): a prefetch of what load() will read at rows r .. r+2, issued by the
// streaming kernels one step before they finish those rows.
// ---------------------------------------------------------------------------
struct NoIn {};
template <class Op, class AT, int N>
__device__ __forceinline__ void finish_rows(const Op &op, int32_t r, const AT (&s)[N], double *red) {
    decltype(op.load(r)) in[N];
#pragma unroll
    for (int d = 0; d < N; ++d) in[d] = op.load(r + d);
#pragma unroll
    for (int d = 0; d < N; ++d) op.store(r + d, s[d], in[d], red);
}
template <class Op, class AT>
__device__ __forceinline__ void finish_row(const Op &op, int32_t r, AT s, double *red) {
    op.store(r, s, op.load(r), red);
}
struct NoRed {
    static constexpr int NRED = 0;
    static constexpr unsigned MAXMASK = 0;
    __device__ void finish(const double *) const {}
};

template <class T>
__device__ __forceinline__ void prefetch_l1(const T *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
template <class Op, class = void>
struct op_touch : std::false_type {};
template <class Op>
struct op_touch<Op, std::void_t<decltype(std::declval<const Op &>().touch(0))>> : std::true_type {};
template <class Op>
__device__ __forceinline__ void touch_rows(const Op &op, int32_t r) {
    if constexpr (op_touch<Op>::value) op.touch(r);
}

// y = A x (clear) or y += A x, accumulating onto the old y in entry order.
template <class YT, class AT>
struct OpSpmv : NoRed {
    YT *__restrict__ y;
    int clear;
    __device__ __forceinline__ AT init(int32_t r) const { return clear ? AT(0) : (AT)y[r]; }
    __device__ __forceinline__ NoIn load(int32_t) const { return {}; }
    __device__ __forceinline__ void store(int32_t r, AT s, NoIn, double *) const { y[r] = (YT)s; }
    __device__ __forceinline__ void touch(int32_t) const {}
};

// y = A x (restriction into the next level's right-hand side) and wb = w .* y, the product the
// next level's first Jacobi sweep gathers
template <class T>
struct OpRestrictWB : NoRed {
    T *__restrict__ y;
    T *__restrict__ wb;
    const T *__restrict__ w;
    __device__ __forceinline__ T init(int32_t) const { return T(0); }
    __device__ __forceinline__ T load(int32_t r) const { return w[r]; }
    __device__ __forceinline__ void store(int32_t r, T s, T wr, double *) const {
        y[r] = s;
        wb[r] = wr * s;
    }
    __device__ __forceinline__ void touch(int32_t) const {}
};

// r = b - A x
template <class T>
struct OpResid : NoRed {
    const T *__restrict__ b;
    T *__restrict__ r;
    __device__ __forceinline__ T init(int32_t) const { return T(0); }
    __device__ __forceinline__ T load(int32_t i) const { return b[i]; }
    __device__ __forceinline__ void store(int32_t i, T s, T bi, double *) const { r[i] = bi - s; }
    __device__ __forceinline__ void touch(int32_t i) const { prefetch_l1(b + i); }
};

// y = x + w .* (b - A x)  (jacobi_iteration, CsrGeometricMultigrid.cl:176-194)
template <class T>
struct OpJacobi : NoRed {
    const T *__restrict__ x;
    const T *__restrict__ w;
    const T *__restrict__ b;
    T *__restrict__ y;
    __device__ __forceinline__ T init(int32_t) const { return T(0); }
    struct In {
        T x, w, b;
    };
    __device__ __forceinline__ In load(int32_t i) const { return {x[i], w[i], b[i]}; }
    __device__ __forceinline__ void store(int32_t i, T s, const In &a, double *) const { y[i] = a.x + a.w * (a.b - s); }
    __device__ __forceinline__ void touch(int32_t i) const {
        prefetch_l1(x + i);
        prefetch_l1(w + i);
        prefetch_l1(b + i);
    }
};
// Second sweep from a zero guess: x1 = w .* b, y = x1 + w .* (b - A x1).
template <class T>
struct OpJacobiFromZero : NoRed {
    const T *__restrict__ w;
    const T *__restrict__ b;
    T *__restrict__ y;
    __device__ __forceinline__ T init(int32_t) const { return T(0); }
    struct In {
        T w, b;
    };
    __device__ __forceinline__ In load(int32_t i) const { return {w[i], b[i]}; }
    __device__ __forceinline__ void store(int32_t i, T s, const In &a, double *) const {
        y[i] = a.w * a.b + a.w * (a.b - s);
    }
    __device__ __forceinline__ void touch(int32_t i) const {
        prefetch_l1(w + i);
        prefetch_l1(b + i);
    }
};

// Device scalars shared by the solver kernels of one solve.
struct SolverScalars {
    double rz, rz_new, pap, alpha, beta;   // Jacobi PCG
    double zr, zq, pq;                     // flexible CG
    double rr, bb, tol2, res_max, res_norm2;
    int it, max_it, done, converged, failed, restart, cycle, pad;
};

// Last Jacobi sweep of the finest level with the flexible-CG dot products of its
// result z fused in: z.q, z.r and beta = -(z.q)/(p.q) (0 on a restart), as k_fcg_red.
template <class T>
struct OpJacobiFcgRed {
    static constexpr int NRED = 2;
    static constexpr unsigned MAXMASK = 0;
    const T *__restrict__ x;
    const T *__restrict__ w;
    const T *__restrict__ b;
    T *__restrict__ y;
    const double *__restrict__ q;
    const double *__restrict__ r;
    SolverScalars *sc;
    __device__ __forceinline__ T init(int32_t) const { return T(0); }
    struct In {
        T x, w, b;
        double q, r;
    };
    __device__ __forceinline__ In load(int32_t i) const { return {x[i], w[i], b[i], q[i], r[i]}; }
    __device__ __forceinline__ void store(int32_t i, T s, const In &a, double *red) const {
        const T z = a.x + a.w * (a.b - s);
        y[i] = z;
        red[0] += (double)z * a.q;
        red[1] += (double)z * a.r;
    }
    __device__ __forceinline__ void touch(int32_t i) const {
        prefetch_l1(x + i);
        prefetch_l1(w + i);
        prefetch_l1(b + i);
        prefetch_l1(q + i);
        prefetch_l1(r + i);
    }
    __device__ void finish(const double *t) const {
        sc->zq = t[0];
        sc->zr = t[1];
        sc->beta = sc->restart ? 0.0 : -t[0] / sc->pq;
        sc->restart = 0;
    }
};

// PCG: Ap = A p and p.Ap; alpha = rz / pAp (dot_finalize_and_calc_a, CsrCG.cl:223-241).
struct OpPcgAp {
    static constexpr int NRED = 1;
    static constexpr unsigned MAXMASK = 0;
    const double *__restrict__ p;
    double *__restrict__ ap;
    SolverScalars *sc;
    __device__ __forceinline__ double init(int32_t) const { return 0.0; }
    __device__ __forceinline__ double load(int32_t i) const { return p[i]; }
    __device__ __forceinline__ void store(int32_t i, double s, double pi, double *red) const {
        ap[i] = s;
        red[0] = __dadd_rn(red[0], __dmul_rn(pi, s));
    }
    __device__ void finish(const double *t) const {
        sc->pap = t[0];
        sc->alpha = sc->rz / t[0];
    }
};

// Flexible CG outer product: s = (A z)_i, q = s + beta q, p = z + beta p, p.q.
template <class ZT>
struct OpFcg {
    static constexpr int NRED = 1;
    static constexpr unsigned MAXMASK = 0;
    static constexpr bool FUSED = true;   // products may use fused multiply-adds (not a parity path)
    const ZT *__restrict__ z;
    double *__restrict__ p;
    double *__restrict__ q;
    SolverScalars *sc;
    double beta;   // unused placeholder: beta is read from sc in load()
    __device__ __forceinline__ double init(int32_t) const { return 0.0; }
    struct In {
        double bt, q, p;
        ZT z;
    };
    __device__ __forceinline__ In load(int32_t i) const { return {sc->beta, q[i], p[i], z[i]}; }
    __device__ __forceinline__ void store(int32_t i, double s, const In &a, double *red) const {
        double qi = s + a.bt * a.q;
        double pi = (double)a.z + a.bt * a.p;
        q[i] = qi;
        p[i] = pi;
        red[0] += pi * qi;
    }
    __device__ __forceinline__ void touch(int32_t i) const {
        prefetch_l1(z + i);
        prefetch_l1(p + i);
        prefetch_l1(q + i);
    }
    __device__ void finish(const double *t) const {
        sc->pq = t[0];
        sc->alpha = sc->zr / t[0];
    }
};

// r = b - A x with the max-norm / NaN check of residual_with_check
// (CsrGeometricMultigrid.cl:121-141): converged when all |r_i| <= tol, failed
// on NaN or |r_i| > 1e50.  Also ||r||^2.  The last block updates the cycle
// counter and the stop decision of the V-cycle driver.
struct OpResidCheck {
    static constexpr int NRED = 3;
    static constexpr unsigned MAXMASK = 0b011;
    const double *__restrict__ b;
    double *__restrict__ r;
    SolverScalars *sc;
    double tol;
    __device__ __forceinline__ double init(int32_t) const { return 0.0; }
    __device__ __forceinline__ double load(int32_t i) const { return b[i]; }
    __device__ __forceinline__ void store(int32_t i, double s, double bi, double *red) const {
        double ri = __dsub_rn(bi, s);
        r[i] = ri;
        double c = fabs(ri);
        if (isnan(ri) || c > 1e50) red[1] = 1.0;
        else red[0] = fmax(red[0], c);
        red[2] += ri * ri;
    }
    __device__ void finish(const double *t) const {
        bool failed = t[1] != 0.0;
        bool converged = !failed && t[0] <= tol;
        sc->res_max = t[0];
        sc->res_norm2 = sqrt(t[2]);
        sc->converged = converged;
        sc->failed = failed;
        if (converged || failed || sc->cycle > sc->max_it) sc->done = 1;
        else sc->cycle += 1;
    }
};

// ---------------------------------------------------------------------------
// CSR row kernel: TPR threads per row, grid-stride over rows
// ---------------------------------------------------------------------------
template <int TPR, class MT, class AT, class Gather, class Op>
__global__ void __launch_bounds__(kThreads) k_csr(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                  const MT *__restrict__ va, int32_t n, Gather g, Op op,
                                                  const int *__restrict__ done, double *partials, unsigned *ticket) {
    if (chain_done(done)) return;
    // entries per lane per step: all index/value loads, then all gathers, then the FMAs (one lane a row: the
    // 27 entries of a restriction row in three steps, summed in order)
    constexpr int U = TPR == 1 ? 9 : 4;
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    const int sub = threadIdx.x % TPR;
    const int gpb = kThreads / TPR;
    for (int32_t row = blockIdx.x * gpb + threadIdx.x / TPR; row < n; row += gridDim.x * gpb) {
        const int32_t s0 = __ldg(rp + row), s1 = __ldg(rp + row + 1);
        AT s = (TPR == 1) ? op.init(row) : AT(0);
        for (int32_t base = s0 + sub; base < s1; base += TPR * U) {
            int32_t c[U];
            AT v[U], xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int32_t k = base + u * TPR;
                c[u] = k < s1 ? __ldcs(ci + k) : 0;
                v[u] = k < s1 ? (AT)__ldcs(va + k) : AT(0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = (base + u * TPR < s1) ? g((uint32_t)c[u]) : AT(0);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (base + u * TPR < s1) s = madd<AT>(s, v[u], xv[u]);
        }
        s = group_sum<TPR>(s);
        if (TPR > 1) s = op.init(row) + s;
        if (sub == 0) finish_row(op, row, s, red);
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

// ---------------------------------------------------------------------------
// CSR node kernel: W threads per node group of 3 consecutive rows that share one column list
// (dv_matrix::row_group == 3, checked over the whole matrix at upload)
//
// HBM-bound.  Read row by row a product moves (4 + s_v) bytes an entry; here the columns and the
// gathered x are read once for the three rows, 4/3 + s_v bytes an entry (FP64 9.33 instead of 12,
// FP32 5.33 instead of 8), from the caller's CSR arrays as they are (the list of the group's first
// row).  Each lane loads U columns and 3 U values, then gathers, then multiplies; the three row
// sums are reduced over the W lanes and lanes 0 .. 2 finish one row each.  64 x 48 x 48 elements
// (36 M entries), FP64: 84.3 -> 69.4 us (365 MB of DRAM traffic, 5.3 TB/s; the gathers and the
// unaligned value runs make 660 MB between L2 and the SMs); 37 x 29 x 23, FP32, in cache:
// 16.2 -> 11.2 us.  A register double buffer (the next group's loads ahead of the multiplies) left
// both unchanged.
// ---------------------------------------------------------------------------
template <int W, class AT, class Gather, class Op>
__global__ void __launch_bounds__(kThreads) k_csr_nodes(const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                        const AT *__restrict__ va, int32_t ngroups, Gather g, Op op,
                                                        const int *__restrict__ done, double *partials,
                                                        unsigned *ticket) {
    if (chain_done(done)) return;
    constexpr int U = 3;
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    const int sub = threadIdx.x % W;
    constexpr int gpb = kThreads / W;
    for (int32_t grp = blockIdx.x * gpb + threadIdx.x / W; grp < ngroups; grp += gridDim.x * gpb) {
        const int32_t r0 = 3 * grp;
        const int32_t s0 = __ldg(rp + r0), len = __ldg(rp + r0 + 1) - s0;
        const int32_t *cp = ci + s0;
        const AT *vp = va + s0;   // the rows' values follow each other: row d starts at d * len
        AT s[3] = {AT(0), AT(0), AT(0)};
        for (int32_t base = sub; base < len; base += W * U) {
            int32_t c[U];
            AT v[U][3], xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int32_t k = base + u * W;
                c[u] = k < len ? __ldcs(cp + k) : 0;
#pragma unroll
                for (int d = 0; d < 3; ++d) v[u][d] = k < len ? __ldcs(vp + (size_t)d * len + k) : AT(0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = (base + u * W < len) ? g((uint32_t)c[u]) : AT(0);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (base + u * W < len)
#pragma unroll
                    for (int d = 0; d < 3; ++d) s[d] = fma(v[u][d], xv[u], s[d]);   // one rounding a term
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) s[d] = group_sum<W>(s[d]);
        if (sub < 3) {
            const AT t = sub == 0 ? s[0] : sub == 1 ? s[1] : s[2];
            finish_row(op, r0 + sub, op.init(r0 + sub) + t, red);
        }
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

// ---------------------------------------------------------------------------
// DuVi row-bundle kernel
//
// One warp per bundle of <= 32 consecutive rows.  The warp copies the
// bundle's entry bytes (Distances), value indices and block column starts into
// its shared-memory stage with 16-byte loads (ranges widened to 16-byte
// boundaries; device arrays carry tail padding), then each lane walks one row
// of the stage in the order of DuViGeometricMultigrid.cl:84-98.  Tables of at
// most 256 distinct values are staged per block.
// ---------------------------------------------------------------------------
struct DuviArgs {
    const uint32_t *__restrict__ row_to_col;
    const uint32_t *__restrict__ row_to_dist;
    const uint32_t *__restrict__ col_idx;
    const uint8_t *__restrict__ dist;
    const void *__restrict__ vidx;
    const void *__restrict__ values;
    const int32_t *__restrict__ bundles;
    int32_t nbundles;
    int32_t nuniq;
};

template <class VI>
__device__ __forceinline__ void copy16(void *dst, const void *src, int nbytes16, int lane) {
    const uint4 *s = static_cast<const uint4 *>(src);
    uint4 *d = static_cast<uint4 *>(dst);
    for (int i = lane; i < nbytes16; i += 32) d[i] = __ldg(s + i);
}

template <class VI, class AT, class Gather, class Op, int WARPS, int BATCH>
__global__ void __launch_bounds__(WARPS * 32, 2) k_duvi(DuviArgs A, Gather g, Op op, const int *__restrict__ done,
                                                     double *partials, unsigned *ticket) {
    if (chain_done(done)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool kSmemTable = sizeof(VI) == 1;
    AT *tab = reinterpret_cast<AT *>(smem);
    unsigned char *wbase = smem + (kSmemTable ? 256 * sizeof(AT) : 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *sdist = wbase + (size_t)warp * (kStageD + kStageD * sizeof(VI) + kStageC * 4);
    VI *svi = reinterpret_cast<VI *>(sdist + kStageD);
    uint32_t *scol = reinterpret_cast<uint32_t *>(sdist + kStageD + kStageD * sizeof(VI));
    const AT *gtab = static_cast<const AT *>(A.values);
    const VI *gvi = static_cast<const VI *>(A.vidx);
    if (kSmemTable) {
        for (int i = threadIdx.x; i < A.nuniq; i += blockDim.x) tab[i] = gtab[i];
        __syncthreads();
    }
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;

    for (int32_t bi = blockIdx.x * WARPS + warp; bi < A.nbundles; bi += gridDim.x * WARPS) {
        const int32_t r0 = __ldg(A.bundles + bi), r1 = __ldg(A.bundles + bi + 1);
        const int32_t rl = min(r0 + lane, r1);
        const uint32_t rd_l = __ldg(A.row_to_dist + rl), rc_l = __ldg(A.row_to_col + rl);
        const uint32_t d0 = __shfl_sync(0xffffffffu, rd_l, 0), c0 = __shfl_sync(0xffffffffu, rc_l, 0);
        const uint32_t d1 = __ldg(A.row_to_dist + r1), c1 = __ldg(A.row_to_col + r1);
        const int32_t row = r0 + lane;
        if (d1 - d0 <= (uint32_t)kBundleBytes && c1 - c0 <= (uint32_t)kBundleBlocks) {
            // stage
            const uint32_t a0 = d0 & ~15u;
            const int nd16 = (int)((d1 - a0 + 15u) >> 4);
            copy16<VI>(sdist, A.dist + a0, nd16, lane);
            const uint64_t vb0 = ((uint64_t)d0 * sizeof(VI)) & ~(uint64_t)15;
            const int nv16 = (int)(((uint64_t)d1 * sizeof(VI) - vb0 + 15u) >> 4);
            copy16<VI>(svi, reinterpret_cast<const unsigned char *>(gvi) + vb0, nv16, lane);
            const uint32_t ca0 = c0 & ~3u;
            const int nc16 = (int)((c1 - ca0 + 3u) >> 2);
            copy16<VI>(scol, A.col_idx + ca0, nc16, lane);
            __syncwarp();
            if (row < r1) {
                uint32_t di = rd_l - a0;
                uint32_t dv = rd_l - (uint32_t)(vb0 / sizeof(VI));
                const uint32_t b_end = __ldg(A.row_to_col + row + 1) - ca0;
                AT s = op.init(row);
                for (uint32_t b = rc_l - ca0; b < b_end; ++b) {
                    const uint32_t n = sdist[di] + 1u;   // entries of the block
                    uint32_t cc = scol[b];
                    uint32_t k = 0;
                    // batches of BATCH entries: column prefix from the gap bytes, then
                    // BATCH independent gathers, then the FMAs in entry order
                    for (; k + BATCH <= n; k += BATCH) {
                        uint32_t cols[BATCH];
                        AT vals[BATCH], xs[BATCH];
#pragma unroll
                        for (int u = 0; u < BATCH; ++u) {
                            cols[u] = cc;
                            cc += sdist[di + k + u + 1] + 1u;   // gap to the next entry (the last read is unused)
                            vals[u] = kSmemTable ? tab[svi[dv + k + u]] : __ldg(gtab + svi[dv + k + u]);
                        }
#pragma unroll
                        for (int u = 0; u < BATCH; ++u) xs[u] = g(cols[u]);
#pragma unroll
                        for (int u = 0; u < BATCH; ++u) s = madd<AT>(s, vals[u], xs[u]);
                    }
                    for (; k < n; ++k) {
                        const AT v = kSmemTable ? tab[svi[dv + k]] : __ldg(gtab + svi[dv + k]);
                        const AT xv = g(cc);
                        cc += sdist[di + k + 1] + 1u;
                        s = madd<AT>(s, v, xv);
                    }
                    di += n;
                    dv += n;
                }
                finish_row(op, row, s, red);
            }
            __syncwarp();
        } else if (lane == 0) {
            // a row longer than the stage: walk it from global memory
            for (int32_t rr = r0; rr < r1; ++rr) {
                uint32_t di = __ldg(A.row_to_dist + rr);
                const uint32_t be = __ldg(A.row_to_col + rr + 1);
                AT s = op.init(rr);
                for (uint32_t b = __ldg(A.row_to_col + rr); b < be; ++b) {
                    uint32_t c = __ldg(A.col_idx + b);
                    int cnt = __ldg(A.dist + di);
                    s = madd<AT>(s, kSmemTable ? tab[__ldg(gvi + di)] : __ldg(gtab + __ldg(gvi + di)), g(c));
                    for (int k = 0; k < cnt; ++k) {
                        ++di;
                        c += __ldg(A.dist + di) + 1u;
                        s = madd<AT>(s, kSmemTable ? tab[__ldg(gvi + di)] : __ldg(gtab + __ldg(gvi + di)), g(c));
                    }
                    ++di;
                }
                finish_row(op, rr, s, red);
            }
        }
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

template <class VI, class AT>
constexpr size_t duvi_smem_bytes(int warps) {
    return (sizeof(VI) == 1 ? 256 * sizeof(AT) : 0) + (size_t)warps * (kStageD + kStageD * sizeof(VI) + kStageC * 4);
}

// ---------------------------------------------------------------------------
// launch dispatch
// ---------------------------------------------------------------------------
struct LaunchEnv {
    dv_context *ctx;
    cudaStream_t stream;
    const int *done;
    double *partials;
    unsigned *ticket;
    int max_blocks;
};

// ---------------------------------------------------------------------------
// DuVi lane kernel (lane-interleaved derived layout, see DuviLanesHost)
//
// One warp per bundle of 32 row groups, one lane per group.  The loop over the
// bundle's 4-entry words is warp-uniform; each lane decodes its leader row's
// columns once (entry byte 255: next block column; otherwise column += byte + 1)
// and applies every gathered x value to the G rows of its group, which share
// the column structure.  Words whose 4 entries all belong to the lane take a
// path without per-entry predicates; only a lane's last word is predicated.
// With SCALED, 8-bit value indices are byte offsets into the shared-memory
// table (one byte extract and one shared load per value).  No staging: every
// stream load is a coalesced 128-byte warp transaction, issued one word ahead
// (register double buffer, streaming loads).  Each row still sums its entries
// in order, so FP64 results equal the reference walk bit for bit.
// ---------------------------------------------------------------------------
template <class VI> struct ViChunk;
template <> struct ViChunk<uint8_t> { using T = uint32_t; };
template <> struct ViChunk<uint16_t> { using T = uint2; };
template <> struct ViChunk<uint32_t> { using T = uint4; };

__device__ __forceinline__ uint32_t vi_get(uint32_t c, int k) { return __byte_perm(c, 0u, 0x4440u + (unsigned)k); }
__device__ __forceinline__ uint32_t vi_get(uint2 c, int k) { return ((k < 2 ? c.x : c.y) >> (16 * (k & 1))) & 0xFFFFu; }
__device__ __forceinline__ uint32_t vi_get(uint4 c, int k) { return k == 0 ? c.x : k == 1 ? c.y : k == 2 ? c.z : c.w; }

struct DuviLanesArgs {
    const uint32_t *__restrict__ meta;
    const uint32_t *__restrict__ dist;
    const void *__restrict__ vi;
    const uint32_t *__restrict__ cols;
    const uint32_t *__restrict__ nent;
    const void *__restrict__ values;
    const void *__restrict__ tuples;   // node-tuple mode: 4 values per tuple
    const int32_t *__restrict__ offsets;   // stencil mode: column - first row of the group
    int64_t ngroups;
    int32_t nbundles;
    int32_t nuniq;
    int32_t ntup;
    int32_t noff;
};

// the (up to) 3 row values of a node tuple: one 16-byte shared load (FP32) or two (FP64)
__device__ __forceinline__ void tup_get(const float *t, uint32_t idx, float (&v)[4]) {
    const float4 q = reinterpret_cast<const float4 *>(t)[idx];
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void tup_get(const double *t, uint32_t idx, double (&v)[4]) {
    const double2 *p = reinterpret_cast<const double2 *>(t) + 2 * idx;
    const double2 a = p[0], b = p[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

template <class AT, bool SCALED, bool SMEM, class Chunk>
__device__ __forceinline__ AT lane_value(const AT *tab, const AT *gtab, const Chunk &c, int k) {
    const uint32_t idx = vi_get(c, k);
    if constexpr (SCALED) return *reinterpret_cast<const AT *>(reinterpret_cast<const char *>(tab) + idx);
    else if constexpr (SMEM) return tab[idx];
    else return __ldg(gtab + idx);
}

template <class VI, class AT, class Gather, class Op, int G, bool SCALED, bool SHIFT, bool TUP, bool STEN>
__global__ void __launch_bounds__(256) k_duvi_lanes(DuviLanesArgs A, Gather g, Op op, const int *__restrict__ done,
                                                    double *partials, unsigned *ticket) {
    if (chain_done(done)) return;
    using Chunk = typename ViChunk<VI>::T;
    constexpr bool kSmemTable = sizeof(VI) == 1;
    constexpr int NV = TUP ? 1 : G;   // index chunks per word
    __shared__ __align__(16) AT tab[TUP ? 1024 : (kSmemTable ? 256 : 1)];
    const AT *gtab = static_cast<const AT *>(A.values);
    __shared__ int32_t soff[STEN ? 256 : 1];
    if constexpr (STEN)
        for (int i = threadIdx.x; i < A.noff; i += blockDim.x) soff[i] = A.offsets[i];
    if constexpr (TUP) {
        const AT *tg = static_cast<const AT *>(A.tuples);
        for (int i = threadIdx.x; i < 4 * A.ntup; i += blockDim.x) tab[i] = tg[i];
        __syncthreads();
    } else if (kSmemTable) {
        for (int i = threadIdx.x; i < A.nuniq; i += blockDim.x) tab[i] = gtab[i];
        __syncthreads();
    }
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const Chunk *vbase = static_cast<const Chunk *>(A.vi);
    for (int32_t bi = blockIdx.x * wpb + (threadIdx.x >> 5); bi < A.nbundles; bi += gridDim.x * wpb) {
        const uint32_t d_base = __ldg(A.meta + 5 * bi), v_base = __ldg(A.meta + 5 * bi + 1);
        const uint32_t c_base = __ldg(A.meta + 5 * bi + 2), words = __ldg(A.meta + 5 * bi + 3);
        const int64_t grp = (int64_t)bi * 32 + lane;
        const bool valid = grp < A.ngroups;
        const uint32_t ne = valid ? __ldg(A.nent + grp) : 0u;
        const uint32_t full = ne >> 2;   // words whose 4 entries are all this lane's
        const int32_t r0 = (int32_t)(grp * G);
        AT s[G];
#pragma unroll
        for (int d = 0; d < G; ++d) s[d] = valid ? op.init(r0 + d) : AT(0);
        const uint32_t *dp = A.dist + d_base + lane;
        const Chunk *vp = vbase + v_base + lane;
        const uint32_t *cp = A.cols + c_base + lane;
        uint32_t c = 0;
        // register double buffer: the streams of word w+1 are in flight while word w is decoded
        uint32_t dw_next = 0;
        Chunk vw_next[NV];
        if (words > 0) {
            dw_next = __ldcs(dp);
#pragma unroll
            for (int d = 0; d < NV; ++d) vw_next[d] = __ldcs(vp + (size_t)d * 32);
        }
        for (uint32_t w = 0; w < words; ++w) {
            const uint32_t dw = dw_next;
            Chunk vw[NV];
#pragma unroll
            for (int d = 0; d < NV; ++d) vw[d] = vw_next[d];
            if (w + 1 < words) {
                dw_next = __ldcs(dp + (size_t)(w + 1) * 32);
#pragma unroll
                for (int d = 0; d < NV; ++d) vw_next[d] = __ldcs(vp + ((size_t)(w + 1) * NV + d) * 32);
            }
            if (w < full) {
                uint32_t cols[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t byte = __byte_perm(dw, 0u, 0x4440u + (unsigned)k);
                    if constexpr (STEN) {
                        c = (uint32_t)(r0 + soff[byte]);
                    } else if (byte == 255u) {
                        c = __ldcs(cp);
                        cp += 32;
                    } else {
                        c += byte + 1u;
                    }
                    cols[k] = c;
                }
                if constexpr (SHIFT) {   // row d reads column + d
                    AT xs[4][G];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int d = 0; d < G; ++d) xs[k][d] = g(cols[k] + (uint32_t)d);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        AT tv[4];
                        if constexpr (TUP) tup_get(tab, vi_get(vw[0], k), tv);
#pragma unroll
                        for (int d = 0; d < G; ++d)
                            s[d] = madd<AT>(s[d], TUP ? tv[d] : lane_value<AT, SCALED, kSmemTable>(tab, gtab, vw[TUP ? 0 : d], k),
                                            xs[k][d]);
                    }
                } else {
                    AT xv[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) xv[k] = g(cols[k]);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        AT tv[4];
                        if constexpr (TUP) tup_get(tab, vi_get(vw[0], k), tv);
#pragma unroll
                        for (int d = 0; d < G; ++d)
                            s[d] = madd<AT>(s[d], TUP ? tv[d] : lane_value<AT, SCALED, kSmemTable>(tab, gtab, vw[TUP ? 0 : d], k),
                                            xv[k]);
                    }
                }
            } else if (w * 4 < ne) {   // the lane's last, partial word
                uint32_t cols[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t byte = __byte_perm(dw, 0u, 0x4440u + (unsigned)k);
                    if (w * 4 + k < ne) {
                        if constexpr (STEN) {
                            c = (uint32_t)(r0 + soff[byte]);
                        } else if (byte == 255u) {
                            c = __ldcs(cp);
                            cp += 32;
                        } else {
                            c += byte + 1u;
                        }
                    }
                    cols[k] = c;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (w * 4 + k < ne) {
                        const AT x0 = SHIFT ? AT(0) : g(cols[k]);
                        AT tv[4];
                        if constexpr (TUP) tup_get(tab, vi_get(vw[0], k), tv);
#pragma unroll
                        for (int d = 0; d < G; ++d)
                            s[d] = madd<AT>(s[d], TUP ? tv[d] : lane_value<AT, SCALED, kSmemTable>(tab, gtab, vw[TUP ? 0 : d], k),
                                            SHIFT ? g(cols[k] + (uint32_t)d) : x0);
                    }
                }
            }
        }
        if (valid) finish_rows(op, r0, s, red);
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

template <class VI, class AT, class Gather, class Op, int G>
void launch_duvi_lanes_g(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    DuviLanesArgs a;
    a.meta = m->lanes_meta.as<uint32_t>();
    a.dist = m->lanes_dist.as<uint32_t>();
    a.vi = m->lanes_vi.p;
    a.cols = m->lanes_cols.as<uint32_t>();
    a.nent = m->lanes_nent.as<uint32_t>();
    a.values = m->values.p;
    a.tuples = m->lanes_tup.p;
    a.offsets = m->lanes_off.as<int32_t>();
    a.noff = m->lanes_noff;
    a.ngroups = m->lanes_groups;
    a.nbundles = (int32_t)m->lanes_bundles;
    a.nuniq = (int32_t)m->nuniq;
    a.ntup = m->lanes_ntup;
    int blocks = (int)((m->lanes_bundles + 7) / 8);
    if (blocks > e.max_blocks) blocks = e.max_blocks;
    if (blocks < 1) blocks = 1;
    const bool sh = G > 1 && m->lanes_shift;
    bool done_launch = false;
    if constexpr (sizeof(VI) == 1) {
        if constexpr (G > 1) {
            if (m->lanes_stencil) {
                launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, false, false, true, true>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
                done_launch = true;
            } else if (m->lanes_tuples) {
                if (sh) launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, false, true, true, false>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
                else launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, false, false, true, false>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
                done_launch = true;
            }
        }
        if (!done_launch && m->lanes_scaled) {
            if (sh) launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, true, G != 1, false, false>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
            else launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, true, false, false, false>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
            done_launch = true;
        }
    }
    if (!done_launch) {
        if (sh) launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, false, G != 1, false, false>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
        else launch_chain(k_duvi_lanes<VI, AT, Gather, Op, G, false, false, false, false>, blocks, 256, 0, e.stream, a, g, op, e.done, e.partials, e.ticket);
    }
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

template <class VI, class AT, class Gather, class Op>
void launch_duvi_lanes(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    if (m->lanes_group == 3) launch_duvi_lanes_g<VI, AT, Gather, Op, 3>(e, m, g, op);
    else if (m->lanes_group == 2) launch_duvi_lanes_g<VI, AT, Gather, Op, 2>(e, m, g, op);
    else launch_duvi_lanes_g<VI, AT, Gather, Op, 1>(e, m, g, op);
}


// ---------------------------------------------------------------------------
// DuVi node-pattern kernel (derived layout, see DuviPatternHost)
//
// One thread per node group.  The group's pattern id selects a run of records
// {column offset from the group's first row, the G row values} staged in shared
// memory; the thread gathers x at each offset and applies it to its G rows,
// summing every row in its entry order (FP64 results equal the reference walk
// bit for bit).  The matrix costs 2 bytes per group in DRAM; the product is
// bound by the x gathers.
// ---------------------------------------------------------------------------
template <class AT>
struct alignas(16) PatRec {
    int32_t off;
    AT v[3];
};
static_assert(sizeof(PatRec<float>) == 16 && offsetof(PatRec<float>, v) == 4, "FP32 pattern record layout");
static_assert(sizeof(PatRec<double>) == 32 && offsetof(PatRec<double>, v) == 8, "FP64 pattern record layout");

// Stages a pattern table (records and pattern starts) in shared memory.
template <class AT>
__device__ __forceinline__ void stage_patterns(uint4 *smem, const PatRec<AT> *__restrict__ grec,
                                               const uint32_t *__restrict__ pstart, int32_t npat, int32_t nrec) {
    uint32_t *st = reinterpret_cast<uint32_t *>(reinterpret_cast<PatRec<AT> *>(smem) + nrec);
    const uint4 *src = reinterpret_cast<const uint4 *>(grec);
    const int n16 = nrec * (int)(sizeof(PatRec<AT>) / 16);
    for (int i = threadIdx.x; i < n16; i += blockDim.x) smem[i] = __ldg(src + i);
    for (int i = threadIdx.x; i <= npat; i += blockDim.x) st[i] = __ldg(pstart + i);
}

// One node group from its pattern records (shared memory): every row summed in entry order.
// BASED: offsets from the group's first column (base[]), else from its first row;
// SHIFT: row d of the group reads column + d.
template <class AT, class Gather, class Op, int G, bool BASED, bool SHIFT>
__device__ __forceinline__ void pattern_group(int64_t gi, const PatRec<AT> *rec, const uint32_t *st,
                                              const uint16_t *__restrict__ pid, const uint32_t *__restrict__ base,
                                              const Gather &g, const Op &op, double *red) {
    const uint32_t p = __ldg(pid + gi);
    const uint32_t b = st[p], e = st[p + 1];
    const int32_t r0 = (int32_t)(gi * G);
    const int32_t c0 = BASED ? (int32_t)__ldg(base + gi) : r0;
    AT s[G];
#pragma unroll
    for (int d = 0; d < G; ++d) s[d] = op.init(r0 + d);
    uint32_t k = b;
    // B records at a time: their columns, then all gathers, then the multiply-adds.  A group's walk is a chain of
    // B-wide steps, each as long as a gather from L2; hex patterns have 81, 54, 36 or 24 records.
    constexpr int B = SHIFT ? 4 : 9;
    for (; k + B <= e; k += B) {
        if constexpr (SHIFT) {
            PatRec<AT> q[B];
#pragma unroll
            for (int u = 0; u < B; ++u) q[u] = rec[k + u];
            AT x[B][G];
#pragma unroll
            for (int u = 0; u < B; ++u)
#pragma unroll
                for (int d = 0; d < G; ++d) x[u][d] = g((uint32_t)(c0 + q[u].off + d));
#pragma unroll
            for (int u = 0; u < B; ++u)
#pragma unroll
                for (int d = 0; d < G; ++d) s[d] = madd_op<AT, op_fused<Op>::value>(s[d], q[u].v[d], x[u][d]);
        } else {
            AT x[B];
#pragma unroll
            for (int u = 0; u < B; ++u) x[u] = g((uint32_t)(c0 + rec[k + u].off));
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const PatRec<AT> q = rec[k + u];
#pragma unroll
                for (int d = 0; d < G; ++d) s[d] = madd_op<AT, op_fused<Op>::value>(s[d], q.v[d], x[u]);
            }
        }
    }
    for (; k < e; ++k) {
        const PatRec<AT> q = rec[k];
#pragma unroll
        for (int d = 0; d < G; ++d) s[d] = madd_op<AT, op_fused<Op>::value>(s[d], q.v[d], g((uint32_t)(c0 + q.off + (SHIFT ? d : 0))));
    }
    finish_rows(op, r0, s, red);
}

template <class AT, class Gather, class Op, int G, bool BASED, bool SHIFT>
__global__ void __launch_bounds__(256) k_duvi_pattern(const uint16_t *__restrict__ pid, const uint32_t *__restrict__ pstart,
                                                      const PatRec<AT> *__restrict__ grec, const uint32_t *__restrict__ base,
                                                      int32_t npat, int32_t nrec, int64_t ngroups, Gather g, Op op,
                                                      const int *__restrict__ done, double *partials, unsigned *ticket) {
    extern __shared__ uint4 pat_smem[];
    const PatRec<AT> *rec = reinterpret_cast<const PatRec<AT> *>(pat_smem);
    const uint32_t *st = reinterpret_cast<const uint32_t *>(rec + nrec);
    stage_patterns<AT>(pat_smem, grec, pstart, npat, nrec);
    if (chain_done(done)) return;
    __syncthreads();
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    for (int64_t gi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; gi < ngroups; gi += (int64_t)gridDim.x * blockDim.x)
        pattern_group<AT, Gather, Op, G, BASED, SHIFT>(gi, rec, st, pid, base, g, op, red);
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

// ---------------------------------------------------------------------------
// DuVi grid-stencil kernel (derived layout, see DuviGridHost)
//
// Operators whose node groups sit on an lx x ly x lz box (x fastest, 3 rows per group) and
// whose interior groups share one pattern coupling the 27 box neighbours.  A block owns a
// tile of 32 x 8 groups of the xy plane and a run of zc planes; it streams the planes z0-1 ..
// z1 through shared memory (the tile plus a one-group halo, 3 values per group, double
// buffered, the next plane's loads in flight during the current plane's arithmetic).  Each
// staged value is read once per thread and applied to the three groups it couples to in z
// (the plane below, at and above it), so a group's three rows collect the 81 columns in
// column order: plane z-1, then z, then z+1, each plane by y, x and dof.  With the same
// multiply-add rounding this is the node-pattern kernel's sum bit for bit.  The interior
// pattern's values are kernel parameters (constant-bank operands of the FMAs): no record
// loads, one shared-memory load per staged value.  Groups on the box faces, and interior
// groups of other patterns, are listed and run through their pattern records by the first
// blocks of the same launch.
// ---------------------------------------------------------------------------

// Structure of the interior row block of an isotropic trilinear hexahedron operator on a uniform
// grid (3 rows of a node against its 27 neighbours x 3 dofs, entry k and row d at 3 k + d): the
// entries of one class are equal and class -1 entries are zero, for every modulus and Poisson
// ratio.  The equalities come from the element's reflection and rotation symmetries, the zeros
// from the cancellation of the 8 elements that share the node (90 of the 243 entries).  Ten
// values then describe the whole stencil.  A matrix is checked against this table when its
// grid layout is built and uses it only if every equality and zero holds exactly.
constexpr int kHexClasses = 10;
#define DV_HEX_CLASS_TABLE \
    0,  1,  1,  1,  0,  1,  1,  1,  0,  2, -1, -1, -1,  3,  4, -1,  4,  3,  0,  5,  5,  5,  0,  1,  5,  1,  0, \
    3, -1,  4, -1,  2, -1,  4, -1,  3,  6, -1, -1, -1,  6, -1, -1, -1,  7,  3, -1,  8, -1,  2, -1,  8, -1,  3, \
    0,  5,  1,  5,  0,  5,  1,  5,  0,  2, -1, -1, -1,  3,  8, -1,  8,  3,  0,  1,  5,  1,  0,  5,  5,  5,  0, \
    3,  4, -1,  4,  3, -1, -1, -1,  2,  6, -1, -1, -1,  7, -1, -1, -1,  6,  3,  8, -1,  8,  3, -1, -1, -1,  2, \
    7, -1, -1, -1,  6, -1, -1, -1,  6,  9, -1, -1, -1,  9, -1, -1, -1,  9,  7, -1, -1, -1,  6, -1, -1, -1,  6, \
    3,  8, -1,  8,  3, -1, -1, -1,  2,  6, -1, -1, -1,  7, -1, -1, -1,  6,  3,  4, -1,  4,  3, -1, -1, -1,  2, \
    0,  1,  5,  1,  0,  5,  5,  5,  0,  2, -1, -1, -1,  3,  8, -1,  8,  3,  0,  5,  1,  5,  0,  5,  1,  5,  0, \
    3, -1,  8, -1,  2, -1,  8, -1,  3,  6, -1, -1, -1,  6, -1, -1, -1,  7,  3, -1,  4, -1,  2, -1,  4, -1,  3, \
    0,  5,  5,  5,  0,  1,  5,  1,  0,  2, -1, -1, -1,  3,  4, -1,  4,  3,  0,  1,  1,  1,  0,  1,  1,  1,  0
// The same table in device and host memory: device code indexes the __device__ copy, which
// the compiler folds to constants after unrolling (a table local to a constexpr function
// would be rebuilt at every inlined call).
__device__ constexpr signed char kHexClassDev[243] = {DV_HEX_CLASS_TABLE};
constexpr signed char kHexClassHost[243] = {DV_HEX_CLASS_TABLE};
__host__ __device__ __forceinline__ constexpr int hex_class(int i) {
#ifdef __CUDA_ARCH__
    return kHexClassDev[i];
#else
    return kHexClassHost[i];
#endif
}

constexpr int kGridTX = 32, kGridTY = 8;   // tile of groups per block: one warp per row (of NY rows each)
constexpr int kGridPX = kGridTX + 2;       // with halo
constexpr int kGridPitch = 104;            // staged values of a tile row: 3 x 34, padded to whole 16-byte copies
template <int NY>
struct PlaneDims {
    static constexpr int TY = kGridTY * NY;             // tile rows
    static constexpr int PY = TY + 2;                   // with halo
    static constexpr int PLANE = kGridPitch * PY;       // staged values per plane
    static constexpr int LOADS = (PLANE + 255) / 256;   // staging slots per thread
};
constexpr int kGridPlane = PlaneDims<1>::PLANE;   // 1040

template <class AT>
struct GridCoef {
    AT v[81][3];           // interior pattern: entry k = 27 dz' + 9 dy' + 3 dx' + c (primes: offset + 1), row d
    AT cls[kHexClasses];   // its class values when it has the hex structure (hex_class)
};

struct GridGeom {
    int32_t lx, ly, lz;        // group box
    int32_t ntx, nty, zc;      // tiles per plane in x and y, planes per z run
    int32_t ntile;             // ntx * nty * ceil((lz - 2) / zc): tiles over the interior nodes
    int32_t tile_blocks;       // blocks [0, tile_blocks) run the tiles, the rest the boundary list
    int32_t hot, all_hot;      // interior pattern id; 1 when no interior group has another pattern
    int64_t nbound;
};

// One term of a stencil row: the coefficient of entry k, row d.  HEX takes it from the ten class
// values (zero entries skipped where SKIP0, i.e. wherever the result need not equal the sequential
// sum over every stored entry bit for bit: NaN or infinite x and the sign of a zero sum are the
// only differences), otherwise from the full table.
template <class AT, bool FUSED, bool HEX, bool SKIP0>
__device__ __forceinline__ AT grid_term(AT acc, const GridCoef<AT> &cf, int k, int d, AT v) {
    if constexpr (HEX) {
        const int c = hex_class(3 * k + d);
        if (c >= 0) return madd_op<AT, FUSED>(acc, cf.cls[c], v);
        if constexpr (SKIP0) return acc;
        else return madd_op<AT, FUSED>(acc, AT(0), v);
    } else {
        return madd_op<AT, FUSED>(acc, cf.v[k][d], v);
    }
}

// Asynchronous global -> shared copies (cp.async, zero fill when `valid` is false: no global read).
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(void *dst, const void *src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(BYTES), "r"(valid ? BYTES : 0)
                 : "memory");
}
// 16 bytes, of which the first `bytes` are read and the rest zero; through the L1 cache (.ca), where an epilogue
// that reads x at its own rows finds it again
__device__ __forceinline__ void cp_async_part16(void *dst, const void *src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// How a gather is staged through shared memory: its source arrays (x; or w and b when the
// gathered value is w .* b) are copied plane by plane, and a staged value is formed from them
// (the same arithmetic as the gather, so results do not depend on the path).
template <class G>
struct StageSrc;
template <class XT, class AT>
struct StageSrc<GatherVec<XT, AT>> {
    using ST = XT;
    static constexpr int N = 1;
    __device__ static const XT *src(const GatherVec<XT, AT> &g, int) { return g.x; }
    template <int PLANE = kGridPlane>
    __device__ static AT value(const XT *pl, int i) { return (AT)pl[i]; }
};
template <class T>
struct StageSrc<GatherWB<T>> {
    using ST = T;
    static constexpr int N = 2;
    __device__ static const T *src(const GatherWB<T> &g, int k) { return k == 0 ? g.w : g.b; }
    template <int PLANE = kGridPlane>
    __device__ static T value(const T *pl, int i) { return pl[i] * pl[i + PLANE]; }
};
constexpr int kGridStages = 4;   // staged planes in flight per block (a plane is consumed 3 steps after its copy)

// Staging of a thread: values k = threadIdx.x + 256 j of the plane (row k / kGridPitch, x-dof k % kGridPitch) ...
template <int NY, class ST, bool VEC>
struct StageSlots {
    static constexpr int PLANE = PlaneDims<NY>::PLANE;
    static constexpr int LOADS = PlaneDims<NY>::LOADS;
    int32_t poff[LOADS];   // offset in a plane of the lx x ly node box (-1: outside the box, -2: past the plane)
    __device__ void plane_offsets(int x0, int y0, int lx, int ly) {
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int k = threadIdx.x + 256 * j, row = k / kGridPitch, col = 3 * (x0 - 1) + k - kGridPitch * row;
            const int yn = y0 - 1 + row;
            poff[j] = k >= PLANE ? -2 : yn >= 0 && yn < ly && col >= 0 && col < 3 * lx ? 3 * lx * yn + col : -1;
        }
    }
    // copies plane z (zero outside 0 <= z < lz) of every source of the gather into one ring slot
    template <class SS, class Gather>
    __device__ void issue(const Gather &g, ST *slot, int z, int lz, int32_t plane_len) const {
        const bool zin = z >= 0 && z < lz;
        const int64_t base = zin ? (int64_t)z * plane_len : 0;
#pragma unroll
        for (int k = 0; k < SS::N; ++k) {
            const ST *src = SS::src(g, k);
#pragma unroll
            for (int j = 0; j < LOADS; ++j)
                if (poff[j] > -2) {
                    const bool v = zin && poff[j] >= 0;
                    cp_async_zfill<sizeof(ST)>(slot + k * PLANE + threadIdx.x + 256 * j, v ? src + base + poff[j] : src, v);
                }
        }
        cp_async_commit();
    }
};
// ... or, where every row of an FP32 vector starts on a 16-byte boundary (an lx that is a multiple of 4), the
// 16-byte pieces k = threadIdx.x + 256 j: two copies a thread and plane instead of eight
// (FP32 residual 128^3 36.2 -> 33.6 us, mixed solve 6.78 -> 6.58 ms).
template <int NY, class ST>
struct StageSlots<NY, ST, true> {
    static constexpr int PLANE = PlaneDims<NY>::PLANE;
    static constexpr int E = 16 / (int)sizeof(ST);
    static constexpr int LOADS = (PLANE / E + 255) / 256;
    int32_t poff[LOADS], bytes[LOADS];   // bytes: of the piece, inside the box's row
    __device__ void plane_offsets(int x0, int y0, int lx, int ly) {
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int k = E * (threadIdx.x + 256 * j), row = k / kGridPitch, col = 3 * (x0 - 1) + k - kGridPitch * row;
            const int yn = y0 - 1 + row, have = max(0, min(E, 3 * lx - col));
            poff[j] = k >= PLANE ? -2 : yn >= 0 && yn < ly && have > 0 ? 3 * lx * yn + col : -1;
            bytes[j] = have * (int)sizeof(ST);
        }
    }
    template <class SS, class Gather>
    __device__ void issue(const Gather &g, ST *slot, int z, int lz, int32_t plane_len) const {
        const bool zin = z >= 0 && z < lz;
        const int64_t base = zin ? (int64_t)z * plane_len : 0;
#pragma unroll
        for (int k = 0; k < SS::N; ++k) {
            const ST *src = SS::src(g, k);
#pragma unroll
            for (int j = 0; j < LOADS; ++j)
                if (poff[j] > -2) {
                    const bool v = zin && poff[j] >= 0;
                    cp_async_part16(slot + k * PLANE + E * (threadIdx.x + 256 * j), v ? src + base + poff[j] : src,
                                    v ? bytes[j] : 0);
                }
        }
        cp_async_commit();
    }
};
// Whether every row of a gather's sources starts on a 16-byte boundary (host).
template <class ST>
inline bool rows_aligned16(const ST *p, int32_t lx) {
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (3 * (int64_t)lx * (int64_t)sizeof(ST)) % 16 == 0;
}
template <class XT, class AT>
inline bool stage_aligned16(const GatherVec<XT, AT> &g, int32_t lx) { return rows_aligned16(g.x, lx); }
template <class T>
inline bool stage_aligned16(const GatherWB<T> &g, int32_t lx) { return rows_aligned16(g.w, lx) && rows_aligned16(g.b, lx); }

// One staged plane applied to the three accumulated groups of each of the thread's NY nodes
// (rows q = 0 .. NY-1 of its column of the tile): below (DI: group p+1 takes the plane as its
// dz = -1 neighbours), at (DM: group p, dz = 0) and above (DF: group p-1, dz = +1).  A staged
// value of plane row r is loaded once and serves every node q with r - q in 0 .. 2.
template <class AT, class SS, int NY, bool FUSED, bool HEX, bool SKIP0, bool DI, bool DM, bool DF>
__device__ __forceinline__ void grid_plane_step(const typename SS::ST *__restrict__ pl, int tx, int ty,
                                                const GridCoef<AT> &cf, AT (&a0)[NY][3], AT (&a1)[NY][3],
                                                AT (&a2)[NY][3]) {
    constexpr int PLANE = PlaneDims<NY>::PLANE;
#pragma unroll
    for (int r = 0; r < NY + 2; ++r)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const AT v = SS::template value<PLANE>(pl, (NY * ty + r) * kGridPitch + (tx + dx) * 3 + c);
#pragma unroll
                for (int q = 0; q < NY; ++q) {
                    const int dy = r - q;
                    if (dy < 0 || dy > 2) continue;
                    const int k = 9 * dy + 3 * dx + c;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if (DI) a2[q][d] = grid_term<AT, FUSED, HEX, SKIP0>(a2[q][d], cf, k, d, v);
                        if (DM) a1[q][d] = grid_term<AT, FUSED, HEX, SKIP0>(a1[q][d], cf, 27 + k, d, v);
                        if (DF) a0[q][d] = grid_term<AT, FUSED, HEX, SKIP0>(a0[q][d], cf, 54 + k, d, v);
                    }
                }
            }
}

template <class AT, class Gather, class Op, bool HEX, int NY, bool VEC>
__global__ void __launch_bounds__(256, 3)   // 3 blocks an SM: FP64 fits 80 registers without spills
    k_duvi_grid(GridGeom G, GridCoef<AT> cf, const uint16_t *__restrict__ pid, const uint32_t *__restrict__ pstart,
                const PatRec<AT> *__restrict__ grec, const uint32_t *__restrict__ bnode, int32_t npat, int32_t nrec,
                Gather g, Op op, const int *__restrict__ done, double *partials, unsigned *ticket) {
    extern __shared__ uint4 grid_smem[];
    constexpr bool FU = op_fused<Op>::value;
    constexpr bool S0 = FU || sizeof(AT) == 4;   // FP64 parity epilogues multiply the zeros too
    // What the epilogue reads is loaded before the step's multiplies where the staged vector is FP32 (mixed solve
    // 128^3 6.58 -> 6.49 ms); elsewhere it is prefetched a step ahead and loaded after them: with FP64 staging the
    // early loads' registers cost more than they hide (FP64 solve 96 x 48 x 48 2.73 -> 2.79 ms), and the full
    // coefficient table leaves none.
    constexpr bool EARLY = HEX && sizeof(typename StageSrc<Gather>::ST) == 4;
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    if ((int32_t)blockIdx.x >= G.tile_blocks) {
        // boundary groups from their pattern records: short blocks, last, so that they fill the SMs that
        // finish their tiles first
        const PatRec<AT> *rec = reinterpret_cast<const PatRec<AT> *>(grid_smem);
        const uint32_t *st = reinterpret_cast<const uint32_t *>(rec + nrec);
        stage_patterns<AT>(grid_smem, grec, pstart, npat, nrec);
        if (chain_done(done)) return;
        __syncthreads();
        const int64_t bblk = (int64_t)blockIdx.x - G.tile_blocks, nbblk = (int64_t)gridDim.x - G.tile_blocks;
        for (int64_t i = bblk * blockDim.x + threadIdx.x; i < G.nbound; i += nbblk * blockDim.x)
            pattern_group<AT, Gather, Op, 3, false, false>((int64_t)__ldg(bnode + i), rec, st, pid, nullptr, g, op, red);
    } else {
        if (chain_done(done)) return;
        using SS = StageSrc<Gather>;
        using ST = typename SS::ST;
        using SL = StageSlots<NY, ST, VEC>;
        constexpr int SLOT = SS::N * SL::PLANE;
        ST *ring = reinterpret_cast<ST *>(grid_smem);   // kGridStages slots of SS::N staged planes
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
        SL slots;
        const int64_t lxy = (int64_t)G.lx * G.ly;
        const int32_t plane_len = (int32_t)(3 * lxy);
        for (int t = (int)blockIdx.x; t < G.ntile; t += G.tile_blocks) {
            const int txi = t % G.ntx, tyi = (t / G.ntx) % G.nty, tzi = t / (G.ntx * G.nty);
            // tiles cover the interior nodes 1 .. l-2 of each axis (the faces are boundary groups)
            const int x0 = 1 + txi * kGridTX, y0 = 1 + tyi * PlaneDims<NY>::TY, z0 = 1 + tzi * G.zc,
                      z1 = min(G.lz - 1, z0 + G.zc);
            const int ix = x0 + tx;
            int32_t col_xy[NY];   // group index in its plane of the thread's nodes
            bool inxy[NY];
#pragma unroll
            for (int q = 0; q < NY; ++q) {
                const int iy = y0 + NY * ty + q;
                col_xy[q] = ix + G.lx * iy;
                inxy[q] = ix >= 1 && ix <= G.lx - 2 && iy >= 1 && iy <= G.ly - 2;
            }
            slots.plane_offsets(x0, y0, G.lx, G.ly);
            // a stencil group (off the faces, interior pattern) that this thread finishes
            auto active = [&](int q, int z) {
                if (!inxy[q] || z < 1 || z > G.lz - 2) return false;
                return G.all_hot || (int)__ldg(pid + col_xy[q] + lxy * z) == G.hot;
            };
#pragma unroll
            for (int s2 = 0; s2 < kGridStages - 1; ++s2) {
                if (z0 - 1 + s2 <= z1) slots.template issue<SS>(g, ring + s2 * SLOT, z0 - 1 + s2, G.lz, plane_len);
                else cp_async_commit();
            }
            AT a0[NY][3], a1[NY][3], a2[NY][3];
            bool act0[NY], act1[NY];
#pragma unroll
            for (int q = 0; q < NY; ++q) {
                act0[q] = act1[q] = false;
#pragma unroll
                for (int d = 0; d < 3; ++d) a0[q][d] = a1[q][d] = a2[q][d] = AT(0);
            }
            for (int p = z0 - 1, k = 0; p <= z1; ++p, ++k) {
                cp_async_wait<kGridStages - 2>();   // plane p has landed (this thread's copies)
                __syncthreads();                     // ... and everyone's; the slot of plane p-1 is free
                if (p + kGridStages - 1 <= z1)
                    slots.template issue<SS>(g, ring + ((k + kGridStages - 1) % kGridStages) * SLOT, p + kGridStages - 1,
                                             G.lz, plane_len);
                else
                    cp_async_commit();
                const ST *pl = ring + (k % kGridStages) * SLOT;
                const bool di = p + 1 >= z0 && p + 1 < z1, dm = p >= z0 && p < z1, df = p - 1 >= z0 && p - 1 < z1;
                bool act2[NY];
#pragma unroll
                for (int q = 0; q < NY; ++q) {
                    act2[q] = di && active(q, p + 1);
                    if (di) {
                        const int32_t r = (int32_t)(3 * (col_xy[q] + lxy * (p + 1)));
#pragma unroll
                        for (int d = 0; d < 3; ++d) a2[q][d] = act2[q] ? op.init(r + d) : AT(0);
                    }
                    if (!EARLY && dm && act1[q])
                        touch_rows(op, (int32_t)(3 * (col_xy[q] + lxy * p)));   // finished next step
                }
                const int64_t below = lxy * (p - 1);
                decltype(op.load(0)) in[NY][3];
                auto load_below = [&] {
#pragma unroll
                    for (int q = 0; q < NY; ++q)
                        if (act0[q])
#pragma unroll
                            for (int d = 0; d < 3; ++d) in[q][d] = op.load((int32_t)(3 * (col_xy[q] + below)) + d);
                };
                if (EARLY && df) load_below();
                if (di && dm && df) grid_plane_step<AT, SS, NY, FU, HEX, S0, true, true, true>(pl, tx, ty, cf, a0, a1, a2);
                else if (di && dm) grid_plane_step<AT, SS, NY, FU, HEX, S0, true, true, false>(pl, tx, ty, cf, a0, a1, a2);
                else if (dm && df) grid_plane_step<AT, SS, NY, FU, HEX, S0, false, true, true>(pl, tx, ty, cf, a0, a1, a2);
                else if (di) grid_plane_step<AT, SS, NY, FU, HEX, S0, true, false, false>(pl, tx, ty, cf, a0, a1, a2);
                else if (dm) grid_plane_step<AT, SS, NY, FU, HEX, S0, false, true, false>(pl, tx, ty, cf, a0, a1, a2);
                else if (df) grid_plane_step<AT, SS, NY, FU, HEX, S0, false, false, true>(pl, tx, ty, cf, a0, a1, a2);
                if (df) {
                    if (!EARLY) load_below();
#pragma unroll
                    for (int q = 0; q < NY; ++q)
                        if (act0[q])
#pragma unroll
                            for (int d = 0; d < 3; ++d) op.store((int32_t)(3 * (col_xy[q] + below)) + d, a0[q][d], in[q][d], red);
                }
#pragma unroll
                for (int q = 0; q < NY; ++q) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        a0[q][d] = a1[q][d];
                        a1[q][d] = a2[q][d];
                    }
                    act0[q] = act1[q];
                    act1[q] = act2[q];
                }
            }
            cp_async_wait<0>();
            __syncthreads();   // the next tile refills the ring
        }
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

// Planes per z run of the grid stencil's tiles.  A tile of zc planes takes zc + 2 steps, a boundary block
// about kBoundSteps; tiles start first, boundary blocks fill in.  The time is at least the tiles' waves and at
// least all work spread over the wave; the run with the smallest bound, the longer one at a tie (fewer
// planes staged twice).  128^3 FP32 residual 45.1 -> 38.7 us, mixed solve 8.09 -> 7.55 ms: with the boundary
// blocks first and runs of a power of two, 68 of 512 tiles were left to a second wave.
constexpr int kBoundSteps = 3;
inline int grid_run_length(int64_t plane_tiles, int lz, int64_t wave, int64_t bound_blocks) {
    int best = 1;
    double best_cost = 1e300;
    for (int zc = 1; zc <= std::min(lz, 64); ++zc) {
        const int64_t tiles = plane_tiles * ((lz + zc - 1) / zc);
        const double waves = (double)((tiles + wave - 1) / wave) * (zc + 2);
        const double spread = ((double)tiles * (zc + 2) + (double)bound_blocks * kBoundSteps) / (double)wave;
        const double cost = std::max(waves, spread);
        if (cost <= best_cost) {
            best_cost = cost;
            best = zc;
        }
    }
    return best;
}

// Grid-stencil launch: tile blocks over runs of zc planes, then the boundary blocks.
template <class AT, class Gather, class Op, bool HEX, bool VEC>
void launch_duvi_grid_h(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    // FP32: two nodes per thread in y (staged rows shared, per-step work amortised); FP64: one
    // (registers)
    constexpr int NY = sizeof(AT) == 4 ? 2 : 1;
    auto kern = k_duvi_grid<AT, Gather, Op, HEX, NY, VEC>;
    using SS = StageSrc<Gather>;
    const size_t smem = std::max(sizeof(typename SS::ST) * SS::N * kGridStages * (size_t)PlaneDims<NY>::PLANE,
                                 sizeof(PatRec<AT>) * (size_t)m->pat_entries + 4 * ((size_t)m->pat_count + 1));
    static SmemLimit limit;   // per instantiation and device
    limit.raise(kern, smem, e.ctx->device);
    static OccupancyCache occupancy;   // per instantiation
    const int occ = occupancy.get(kern, 256, smem, e.ctx->device);
    GridCoef<AT> cf;
    for (int k = 0; k < 81; ++k)
        for (int d = 0; d < 3; ++d) cf.v[k][d] = (AT)m->grid_coef[3 * k + d];
    for (int c = 0; c < kHexClasses; ++c) cf.cls[c] = HEX ? (AT)m->grid_cls[c] : AT(0);
    GridGeom G;
    G.lx = m->grid_lx;
    G.ly = m->grid_ly;
    G.lz = m->grid_lz;
    G.ntx = std::max(0, (G.lx - 2 + kGridTX - 1) / kGridTX);   // tiles over the interior nodes 1 .. l-2
    G.nty = std::max(0, (G.ly - 2 + PlaneDims<NY>::TY - 1) / PlaneDims<NY>::TY);
    G.hot = m->grid_hot;
    G.all_hot = m->grid_all_hot;
    G.nbound = m->grid_nb;
    const int64_t wave = (int64_t)e.ctx->num_sms * occ;
    // one boundary group a thread (measured: two or four a thread slowed the solve by 6 and 14 %)
    const int64_t bound_blocks = G.nbound == 0 ? 0
                                 : std::min<int64_t>((G.nbound + 255) / 256, std::max<int64_t>(1, e.max_blocks / 4));
    const int64_t plane_tiles = (int64_t)G.ntx * G.nty;
    const int lzi = std::max(1, G.lz - 2);
    G.zc = grid_run_length(plane_tiles, lzi, wave, bound_blocks);
    G.ntile = G.lz > 2 ? (int32_t)(plane_tiles * ((lzi + G.zc - 1) / G.zc)) : 0;
    G.tile_blocks = (int32_t)std::min<int64_t>(G.ntile, std::max<int64_t>(1, e.max_blocks - bound_blocks));
    const int blocks = (int)std::max<int64_t>(1, G.tile_blocks + bound_blocks);
    launch_chain(kern, blocks, 256, smem, e.stream, G, cf, m->pat_id.as<uint16_t>(), m->pat_start.as<uint32_t>(),
                                          static_cast<const PatRec<AT> *>(m->pat_rec.p), m->grid_bnode.as<uint32_t>(),
                                          m->pat_count, m->pat_entries, g, op, e.done, e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

template <class AT, class Gather, class Op, int G, bool BASED, bool SHIFT>
void launch_duvi_pattern_gbs(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    auto kern = k_duvi_pattern<AT, Gather, Op, G, BASED, SHIFT>;
    const size_t smem = sizeof(PatRec<AT>) * (size_t)m->pat_entries + 4 * ((size_t)m->pat_count + 1);
    // Raise the kernel's dynamic shared-memory limit to every new largest size: epilogues
    // that reduce add static shared memory, so even tables under 48 KB can need it.
    static SmemLimit limit;   // per instantiation and device
    limit.raise(kern, smem, e.ctx->device);
    // Whole waves: past one wave of resident blocks (SMs x blocks per SM at this table size
    // and register count), a multiple of it, so that the last wave is not a partial one.
    static OccupancyCache occupancy;   // per instantiation
    const int occ = occupancy.get(kern, 256, smem, e.ctx->device);
    const int64_t ng = m->n_rows / G;
    const int64_t need = std::max<int64_t>(1, (ng + 255) / 256), wave = (int64_t)e.ctx->num_sms * occ;
    const int64_t cap = std::min<int64_t>(need, e.max_blocks);
    const int blocks = (int)(cap <= wave ? cap : cap / wave * wave);
    launch_chain(kern, blocks, 256, smem, e.stream, m->pat_id.as<uint16_t>(), m->pat_start.as<uint32_t>(),
                                          static_cast<const PatRec<AT> *>(m->pat_rec.p), m->pat_base.as<uint32_t>(),
                                          m->pat_count, m->pat_entries, ng, g, op, e.done, e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}


template <class AT, class Gather, class Op, int G>
void launch_duvi_pattern_g(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op);

// The hex-structured stencil when the matrix has it; the general stencil (243 coefficients) in
// FP32 otherwise.  FP64 matrices without the hex structure keep the node patterns (grid_ok is
// not set for them); the fallback below only guards against a stale variant.
template <class AT, class Gather, class Op>
void launch_duvi_grid(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    if (m->grid_hex) {
        if constexpr (sizeof(typename StageSrc<Gather>::ST) == 4) {
            if (stage_aligned16(g, m->grid_lx)) {
                launch_duvi_grid_h<AT, Gather, Op, true, true>(e, m, g, op);
                return;
            }
        }
        launch_duvi_grid_h<AT, Gather, Op, true, false>(e, m, g, op);
    } else if constexpr (sizeof(AT) == 4) launch_duvi_grid_h<AT, Gather, Op, false, false>(e, m, g, op);
    else launch_duvi_pattern_g<AT, Gather, Op, 3>(e, m, g, op);
}

template <class AT, class Gather, class Op, int G>
void launch_duvi_pattern_g(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    if (!m->pat_based) launch_duvi_pattern_gbs<AT, Gather, Op, G, false, false>(e, m, g, op);
    else if (G > 1 && m->pat_shift) launch_duvi_pattern_gbs<AT, Gather, Op, G, true, (G > 1)>(e, m, g, op);
    else launch_duvi_pattern_gbs<AT, Gather, Op, G, true, false>(e, m, g, op);
}

template <class AT, class Gather, class Op>
void launch_duvi_pattern(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    if (m->lanes_group == 3) launch_duvi_pattern_g<AT, Gather, Op, 3>(e, m, g, op);
    else if (m->lanes_group == 2) launch_duvi_pattern_g<AT, Gather, Op, 2>(e, m, g, op);
    else launch_duvi_pattern_g<AT, Gather, Op, 1>(e, m, g, op);
}

template <class VI, class AT, class Gather, class Op, int BATCH>
void launch_duvi_vi(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    constexpr int W = sizeof(VI) == 4 ? kDuviWarps32 : kDuviWarps;
    const size_t smem = duvi_smem_bytes<VI, AT>(W);
    auto kern = k_duvi<VI, AT, Gather, Op, W, BATCH>;
    static SmemLimit limit;   // per instantiation and device
    limit.raise(kern, smem, e.ctx->device);
    DuviArgs a;
    a.row_to_col = m->row_to_col.as<uint32_t>();
    a.row_to_dist = m->row_to_dist.as<uint32_t>();
    a.col_idx = m->col_idx.as<uint32_t>();
    a.dist = m->dist.as<uint8_t>();
    a.vidx = m->vidx.p;
    a.values = m->values.p;
    a.bundles = m->bundles.as<int32_t>();
    a.nbundles = m->nbundles;
    a.nuniq = (int32_t)m->nuniq;
    int blocks = (m->nbundles + W - 1) / W;
    if (blocks > e.max_blocks) blocks = e.max_blocks;
    if (blocks < 1) blocks = 1;
    launch_chain(kern, blocks, W * 32, smem, e.stream, a, g, op, e.done, e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

// Columns and values of a DuVi matrix, entry by entry, for kernels that walk a row's entries side by
// side (row offsets: row_to_dist).
template <class VI, class T>
__global__ void k_duvi_decode(DuviArgs A, int32_t n, int32_t *__restrict__ col, T *__restrict__ val) {
    const T *tab = static_cast<const T *>(A.values);
    const VI *vi = static_cast<const VI *>(A.vidx);
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t di = A.row_to_dist[i];
        for (uint32_t bl = A.row_to_col[i]; bl < A.row_to_col[i + 1]; ++bl) {
            uint32_t c = A.col_idx[bl];
            const int cnt = A.dist[di];
            for (int k = 0;; ++k) {
                col[di] = (int32_t)c;
                val[di] = tab[vi[di]];
                ++di;
                if (k == cnt) break;
                c += A.dist[di] + 1u;
            }
        }
    }
}

inline DuviArgs duvi_args(const dv_matrix *m) {
    DuviArgs a;
    a.row_to_col = m->row_to_col.as<uint32_t>();
    a.row_to_dist = m->row_to_dist.as<uint32_t>();
    a.col_idx = m->col_idx.as<uint32_t>();
    a.dist = m->dist.as<uint8_t>();
    a.vidx = m->vidx.p;
    a.values = m->values.p;
    a.bundles = m->bundles.as<int32_t>();
    a.nbundles = m->nbundles;
    a.nuniq = (int32_t)m->nuniq;
    return a;
}

template <class T>
void duvi_decode(const dv_matrix *m, int32_t *col, T *val) {
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)m->n_rows + 255) / 256, m->ctx->num_sms * 16));
    cudaStream_t s = m->ctx->stream;
    if (m->vi_bits == 8) k_duvi_decode<uint8_t, T><<<grid, 256, 0, s>>>(duvi_args(m), m->n_rows, col, val);
    else if (m->vi_bits == 16) k_duvi_decode<uint16_t, T><<<grid, 256, 0, s>>>(duvi_args(m), m->n_rows, col, val);
    else k_duvi_decode<uint32_t, T><<<grid, 256, 0, s>>>(duvi_args(m), m->n_rows, col, val);
    DV_CUDA(cudaGetLastError());
    m->ctx->count();
}

// Row offsets of a CSR matrix, or of a DuVi matrix's decoded entries.
inline const int32_t *row_offsets(const dv_matrix *m) {
    return (m->format == DV_FORMAT_CSR ? m->rowptr : m->row_to_dist).as<int32_t>();
}

template <int TPR, class AT, class Gather, class Op>
void launch_csr_tpr(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    const int gpb = kThreads / TPR;
    int blocks = (m->n_rows + gpb - 1) / gpb;
    if (blocks > e.max_blocks) blocks = e.max_blocks;
    if (blocks < 1) blocks = 1;
    launch_chain(k_csr<TPR, AT, AT, Gather, Op>, blocks, kThreads, 0, e.stream, 
        row_offsets(m), m->col.as<int32_t>(), static_cast<const AT *>(m->val.p), m->n_rows, g, op, e.done,
        e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

template <int W, class AT, class Gather, class Op>
void launch_csr_nodes(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    auto kern = k_csr_nodes<W, AT, Gather, Op>;
    const int32_t ngroups = m->n_rows / 3;
    const int64_t need = std::max<int64_t>(1, ((int64_t)ngroups * W + kThreads - 1) / kThreads);
    int64_t blocks = need;
    if (Op::NRED > 0) {   // one wave of resident blocks, so that few partial sums are left to add
        static OccupancyCache occupancy;   // per instantiation
        const int64_t wave = (int64_t)e.ctx->num_sms * occupancy.get(kern, kThreads, 0, e.ctx->device);
        blocks = std::min<int64_t>(need, std::min<int64_t>(wave, e.max_blocks));
    }
    launch_chain(kern, (unsigned)blocks, kThreads, 0, e.stream, row_offsets(m), m->col.as<int32_t>(),
                                                      static_cast<const AT *>(m->val.p), ngroups, g, op, e.done,
                                                      e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

// ---------------------------------------------------------------------------
// Matrix-free hexahedral operator (DV_FORMAT_HEX): y = K(E) x with K = sum_e f_e Ke on a
// structured grid of unit-cube trilinear hexahedra, f_e = scale * E_e per element, the
// nodes of the x = 0 face clamped (FemCantileverBase.cs:87-158, FemCantilever3D.cs:27-132).
//
// Nothing of the matrix is stored: a product reads the element factors (one value per
// element), x and writes y.  Bound by arithmetic: 24 x 24 multiply-adds an element if Ke is
// applied as it stands (and by corner, 48 scalings of x more).  Ke commutes with the element's
// three mirror images, so in sums and differences over opposite corners (a Walsh-Hadamard
// transform of the 8 corner values of each component, signs (-1)^(s.b) for corner b and
// character s) it falls apart into eight 3 x 3 blocks, one per parity t: component c of block t is
// character s = t xor e_c.  For the isotropic cube these blocks hold 8 different numbers in all
// (HexModes); rigid motions are exact zeros.  One element then takes 33 operations and 18
// scalings, and the transforms 24 + 24 additions in xy (once per node plane and element
// column) and 24 + 24 in z: about 170 operations an element instead of 670.
//
// A thread owns one element column of a tile of W x R columns and streams node planes: the
// plane's four corner values (staged in shared memory, kGridStages planes in flight) are
// transformed in xy, combined with the plane below in z, multiplied, and the two faces' parts
// added while still transformed; the inverse in xy gives the column's share of its 4 nodes of the
// plane.  Shares of other threads' nodes are exchanged through shared memory across the next
// step's barrier (so a step has one), and every thread finishes the node at its column's upper
// right corner: (W - 1) x (R - 1) nodes a tile.  W and R are chosen per mesh for the fewest tiles
// (hex_tile).  Elements outside the mesh have factor 0 and clamped or outside nodes have x = 0,
// so face and edge nodes need no special case.  The sum order differs from the assembled
// operator's, so FP64 products agree with the assembled matrix to rounding (not bit for bit).
// 128^3, log-uniform moduli, FP64 product: 212.9 -> 68 us (119 MB of vectors and factors: 18 us;
// 170 FP64 operations a node: 19 us), relative error against 64 bits 4.7e-16 -> 2.1e-16.
// Sums and differences over corners turn an infinite x into Inf - Inf, and overflow for a finite x near
// the type's limit: a node whose sums are not finite is formed again from the entries of Ke
// (hex_node_direct), so it has the signed infinity, the NaN or the finite value of Ke times x.
// ---------------------------------------------------------------------------
template <class AT>
struct HexModes {
    AT a0, b0;   // t = 0 (the three normal strains): diagonal minus off-diagonal, off-diagonal
    AT p, q;     // t = one axis: the two components that are not translations
    AT r, w;     // t = two axes: shear (all four entries equal), the third component alone
    AT g0, h0;   // t = three axes: as t = 0
};

// One mesh of a (possibly batched) matrix-free operator: its element counts, the tiles it is
// streamed in, its first tile in the launch, and where its rows and element factors start.
struct HexMesh {
    int32_t ne0, ne1, ne2;     // elements per axis (free-node box: ne0 x (ne1 + 1) x (ne2 + 1))
    int32_t ntx, nty, zc;      // tiles per plane in x and y, planes per z run
    int32_t wn, rn;            // nodes of a tile in x and y (one element column more in each)
    int32_t tile0, pad;        // first tile of this mesh
    int64_t row0, fac0;        // first row, first element factor
};

constexpr int kHexThreads = 256;
constexpr int kHexLoads = 4;                               // staging slots per thread
constexpr int kHexPlane = kHexLoads * kHexThreads;         // staged values of a plane, at most

// Tile of a mesh plane of lx x ly free nodes: (wn + 1) x (rn + 1) element columns, one a thread,
// whose (wn + 2) x (rn + 2) nodes fit the staging slots; the fewest tiles, the widest at a tie.
inline void hex_tile(int32_t lx, int32_t ly, int32_t &wn, int32_t &rn) {
    int64_t best = INT64_MAX;
    wn = rn = 1;
    for (int32_t nt = 1; nt <= lx; ++nt) {
        const int32_t w = (lx + nt - 1) / nt;
        int32_t r = std::min<int32_t>(kHexThreads / (w + 1) - 1, ly);
        while (r >= 1 && 3 * (w + 2) * (r + 2) > kHexPlane) --r;
        if (r < 1) continue;
        const int32_t my = (ly + r - 1) / r;
        const int64_t tiles = (int64_t)((lx + w - 1) / w) * my;
        if (tiles < best) {
            best = tiles;
            wn = w;
            rn = (ly + my - 1) / my;
        }
        if (w <= 8) break;
    }
}

// Corner values v[by][bx] of one component in a plane -> characters s = sx + 2 sy.
template <class AT>
__device__ __forceinline__ void hex_xy(AT v00, AT v10, AT v01, AT v11, AT (&s)[4]) {
    const AT a = v00 + v10, b = v00 - v10, c = v01 + v11, d = v01 - v11;
    s[0] = a + c;
    s[1] = b + d;
    s[2] = a - c;
    s[3] = b - d;
}

// The mesh of tile t: the last with tile0 <= t.
__device__ __forceinline__ int hex_mesh_of(const HexMesh *__restrict__ meshes, int32_t nmesh, int t) {
    int lo = 0, hi = nmesh - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (meshes[mid].tile0 <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The three rows from r of tile t's mesh, added to s entry by entry: the element layer below the node
// and the one above, each by its lower and its upper corners (plane z - 1; z, above and below; z + 1).  As
// everywhere, an element outside the mesh has factor 0 and a node outside it x = 0.  Out of line: it
// takes no registers from the kernel's step.
template <class AT>
struct HexRows {
    AT v[3];
};
template <class AT, bool FUSED, class Gather>
__device__ __noinline__ HexRows<AT> hex_node_direct(const HexMesh *__restrict__ meshes, int32_t nmesh, int t,
                                                    const AT *__restrict__ ef_all, const AT *__restrict__ ke, Gather g,
                                                    int32_t r, HexRows<AT> s) {
    constexpr int vtk[8] = {0, 1, 3, 2, 4, 5, 7, 6};
    const HexMesh G = meshes[hex_mesh_of(meshes, nmesh, t)];
    const int32_t lx = G.ne0, ly = G.ne1 + 1, q = (int32_t)(r - G.row0) / 3;
    const int iz = q / (lx * ly), iy = q / lx - ly * iz, ix = q % lx;
#pragma unroll 1
    for (int part = 0; part < 4; ++part) {
        const int above = part & 1, bz = part >> 1, layer = iz - 1 + above, z = layer + bz;
#pragma unroll 1
        for (int el = 0; el < 4; ++el) {
            const int ex = ix + (el & 1), ey = iy - 1 + (el >> 1);
            const bool inside = ex < G.ne0 && ey >= 0 && ey < G.ne1 && layer >= 0 && layer < G.ne2;
            const AT f = inside ? ef_all[G.fac0 + ex + (int64_t)G.ne0 * (ey + (int64_t)G.ne1 * layer)] : AT(0);
            const int a = vtk[3 - el + (above ? 0 : 4)];   // the node among the element's corners
#pragma unroll 1
            for (int c = 0; c < 12; ++c) {   // corner c / 3 of the plane, dof c % 3
                const int corner = c / 3, d = c - 3 * corner;
                const int x = ex - 1 + (corner & 1), y = ey + (corner >> 1);
                const bool node = x >= 0 && x < lx && y >= 0 && y < ly && z >= 0 && z <= G.ne2;
                const AT w = f * (node ? g((uint32_t)(G.row0 + 3 * (x + (int64_t)lx * (y + (int64_t)ly * z)) + d)) : AT(0));
                const AT *col = ke + 72 * a + 3 * vtk[corner + 4 * bz] + d;
#pragma unroll
                for (int i = 0; i < 3; ++i) s.v[i] = madd_op<AT, FUSED>(s.v[i], col[24 * i], w);
            }
        }
    }
    return s;
}
// Whether any of the sums is an infinity or a NaN.
__device__ __forceinline__ bool any_nonfinite(const double (&s)[3]) {
    const int a = __double2hiint(s[0]) & 0x7fffffff, b = __double2hiint(s[1]) & 0x7fffffff, c = __double2hiint(s[2]) & 0x7fffffff;
    return max(a, max(b, c)) >= 0x7ff00000;
}
__device__ __forceinline__ bool any_nonfinite(const float (&s)[3]) {
    const int a = __float_as_int(s[0]) & 0x7fffffff, b = __float_as_int(s[1]) & 0x7fffffff, c = __float_as_int(s[2]) & 0x7fffffff;
    return max(a, max(b, c)) >= 0x7f800000;
}

template <class AT, class Gather, class Op>
__global__ void __launch_bounds__(kHexThreads, sizeof(AT) == 8 ? 2 : 3)
    k_hex_elem(const HexMesh *__restrict__ meshes, int32_t nmesh, int32_t ntile, HexModes<AT> kc,
               const AT *__restrict__ ke, const AT *__restrict__ ef_all, Gather g, Op op, const int *__restrict__ done,
               double *partials, unsigned *ticket) {
    if (chain_done(done)) return;
    extern __shared__ uint4 hex_smem[];
    using SS = StageSrc<Gather>;
    using ST = typename SS::ST;
    constexpr int SLOT = SS::N * kHexPlane;
    ST *ring = reinterpret_cast<ST *>(hex_smem);                      // kGridStages slots of node planes
    AT *share = reinterpret_cast<AT *>(ring + kGridStages * SLOT);    // 2 x 9 shares a thread
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        const HexMesh G = meshes[hex_mesh_of(meshes, nmesh, t)];
        const int32_t lx = G.ne0, ly = G.ne1 + 1, lz = G.ne2 + 1;
        const int32_t plane_len = 3 * lx * ly, layer_len = G.ne0 * G.ne1;
        const int W = G.wn + 1, R = G.rn + 1;   // element columns
        const int tl = t - G.tile0;
        const int txi = tl % G.ntx, tyi = (tl / G.ntx) % G.nty, tzi = tl / (G.ntx * G.nty);
        const int x0 = txi * G.wn, y0 = tyi * G.rn, z0 = tzi * G.zc, z1 = min(lz, z0 + G.zc);
        const int ty = (int)threadIdx.x / W, tx = (int)threadIdx.x - W * ty;
        const bool column = ty < R;
        const int ix = x0 + tx, iy = y0 + ty;   // the node this thread finishes; its element is (ix, iy - 1)
        const bool node = column && tx < W - 1 && ty < R - 1 && ix < lx && iy < ly;
        const bool inside = column && ix < G.ne0 && iy >= 1 && iy <= G.ne1;
        const AT *ef = ef_all + G.fac0 + (inside ? ix + (int64_t)G.ne0 * (iy - 1) : 0);
        auto factor = [&](int l) { return inside && l >= 0 && l < G.ne2 ? __ldg(ef + (int64_t)l * layer_len) : AT(0); };
        const int32_t r_xy = (int32_t)G.row0 + 3 * (ix + lx * iy);
        // staged plane: node (x0 - 1 + j, y0 - 1 + i), dof c at 3 ((W + 1) i + j) + c; offsets in the plane, -1
        // outside the mesh, -2 past the tile
        int32_t poff[kHexLoads];
        const int staged = 3 * (W + 1) * (R + 1);
#pragma unroll
        for (int j = 0; j < kHexLoads; ++j) {
            const int k = threadIdx.x + kHexThreads * j, nd = k / 3, i = nd / (W + 1);
            const int xn = x0 - 1 + nd - (W + 1) * i, yn = y0 - 1 + i;
            poff[j] = k >= staged ? -2 : xn >= 0 && xn < lx && yn >= 0 && yn < ly ? 3 * (xn + lx * yn) + (k - 3 * nd) : -1;
        }
        auto issue = [&](int z, int k) {
            const bool zin = z >= 0 && z < lz;
            const int64_t base = zin ? G.row0 + (int64_t)z * plane_len : 0;
            ST *slot = ring + (k % kGridStages) * SLOT;
#pragma unroll
            for (int q = 0; q < SS::N; ++q) {
                const ST *src = SS::src(g, q);
#pragma unroll
                for (int j = 0; j < kHexLoads; ++j)
                    if (poff[j] > -2) {
                        const bool v = zin && poff[j] >= 0;
                        cp_async_zfill<sizeof(ST)>(slot + q * kHexPlane + threadIdx.x + kHexThreads * j,
                                                   v ? src + base + poff[j] : src, v);
                    }
            }
            cp_async_commit();
        };
#pragma unroll
        for (int q = 0; q < kGridStages - 1; ++q) {
            if (z0 - 1 + q <= z1) issue(z0 - 1 + q, q);
            else cp_async_commit();
        }
        AT sp[3][4], up[3][4];   // the plane below, transformed; its part from the layer under it
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int s = 0; s < 4; ++s) sp[c][s] = up[c][s] = AT(0);
        AT own[3] = {AT(0), AT(0), AT(0)};
        AT fa = factor(z0 - 1), fb = factor(z0);
        const int corner = column ? 3 * ((W + 1) * ty + tx) : 0;
        for (int p = z0 - 1, k = 0; p <= z1 + 1; ++p, ++k) {
            cp_async_wait<kGridStages - 2>();   // plane p has landed (this thread's copies)
            __syncthreads();                     // ... and everyone's, and the shares of plane p - 2
            if (p - 2 >= z0 && node) {   // finish node plane p - 2
                const AT *sh = share + ((k + 1) & 1) * 9 * kHexThreads + threadIdx.x;
                const int32_t r = r_xy + (p - 2) * plane_len;
                // one value a row is loaded before the branch, which no load is moved across (residuals 96^3, loaded after
                // it and before it: FP64 27.4 -> 26.1 us, FP32 21.3 -> 20.9; 25.8 and 20.3 without the check); more would spill
                constexpr bool EARLY = sizeof(op.load(r)) <= sizeof(AT);
                decltype(op.load(r)) in[3];
                if constexpr (EARLY)
#pragma unroll
                    for (int c = 0; c < 3; ++c) in[c] = op.load(r + c);
                AT s[3];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    s[c] = op.init(r + c) + ((own[c] + sh[c * kHexThreads + 1]) +
                                             (sh[(3 + c) * kHexThreads + W] + sh[(6 + c) * kHexThreads + W + 1]));
                if (any_nonfinite(s)) {
                    const HexRows<AT> v = hex_node_direct<AT, op_fused<Op>::value>(
                        meshes, nmesh, t, ef_all, ke, g, r, HexRows<AT>{{op.init(r), op.init(r + 1), op.init(r + 2)}});
#pragma unroll
                    for (int c = 0; c < 3; ++c) s[c] = v.v[c];
                }
                if constexpr (!EARLY)
#pragma unroll
                    for (int c = 0; c < 3; ++c) in[c] = op.load(r + c);
#pragma unroll
                for (int c = 0; c < 3; ++c) op.store(r + c, s[c], in[c], red);
            }
            if (p > z1) break;
            if (p + kGridStages - 1 <= z1) issue(p + kGridStages - 1, k + kGridStages - 1);
            else cp_async_commit();
            const ST *pl = ring + (k % kGridStages) * SLOT + corner;
            AT sc[3][4];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                hex_xy<AT>(SS::template value<kHexPlane>(pl, c), SS::template value<kHexPlane>(pl, 3 + c),
                           SS::template value<kHexPlane>(pl, 3 * (W + 1) + c),
                           SS::template value<kHexPlane>(pl, 3 * (W + 1) + 3 + c), sc[c]);
            if (p >= z0) {
                // element layer p - 1 .. p: X+ = lower + upper (sz = 0), X- = lower - upper (sz = 1)
                const AT f = fa;
                fa = fb;
                fb = factor(p + 1);
                if (p - 1 >= z0 && node) touch_rows(op, r_xy + (p - 1) * plane_len);   // finished next step
                AT xp[3][4], xm[3][4];
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        xp[c][s] = sp[c][s] + sc[c][s];
                        xm[c][s] = sp[c][s] - sc[c][s];
                    }
                AT yp[3][4], ym[3][4];
                auto three = [&](AT u, AT v, AT w, AT d, AT o, AT &yu, AT &yv, AT &yw) {
                    const AT m = o * (u + v + w);
                    yu = f * fma(d, u, m);
                    yv = f * fma(d, v, m);
                    yw = f * fma(d, w, m);
                };
                auto two = [&](AT u, AT v, AT &yu, AT &yv) {
                    yu = f * fma(kc.p, u, kc.q * v);
                    yv = f * fma(kc.p, v, kc.q * u);
                };
                const AT fr = f * kc.r, fw = f * kc.w;
                yp[0][0] = yp[1][0] = yp[2][0] = AT(0);                                                   // translations
                three(xp[0][1], xp[1][2], xm[2][0], kc.a0, kc.b0, yp[0][1], yp[1][2], ym[2][0]);         // t = 000
                two(xp[1][3], xm[2][1], yp[1][3], ym[2][1]);                                              // x
                two(xp[0][3], xm[2][2], yp[0][3], ym[2][2]);                                              // y
                two(xm[0][1], xm[1][2], ym[0][1], ym[1][2]);                                              // z
                yp[0][2] = yp[1][1] = fr * (xp[0][2] + xp[1][1]);                                         // xy
                ym[2][3] = fw * xm[2][3];
                ym[0][0] = yp[2][1] = fr * (xm[0][0] + xp[2][1]);                                         // xz
                ym[1][3] = fw * xm[1][3];
                ym[1][0] = yp[2][2] = fr * (xm[1][0] + xp[2][2]);                                         // yz
                ym[0][3] = fw * xm[0][3];
                three(xm[0][2], xm[1][1], xp[2][3], kc.g0, kc.h0, ym[0][2], ym[1][1], yp[2][3]);         // xyz
                // plane p - 1: the part from below and this layer's lower face, back to corners
                if (p - 1 >= z0) {
                    AT *sh = share + (k & 1) * 9 * kHexThreads + threadIdx.x;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        AT n[4], T[4];
#pragma unroll
                        for (int s = 0; s < 4; ++s) T[s] = up[c][s] + (yp[c][s] + ym[c][s]);
                        hex_xy<AT>(T[0], T[1], T[2], T[3], n);   // its own inverse but for the factor: n[bx + 2 by]
                        own[c] = n[3];
                        sh[c * kHexThreads] = n[2];         // (bx, by) = (0, 1): the node to the left
                        sh[(3 + c) * kHexThreads] = n[1];   // (1, 0): the node below
                        sh[(6 + c) * kHexThreads] = n[0];
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int s = 0; s < 4; ++s) up[c][s] = yp[c][s] - ym[c][s];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int s = 0; s < 4; ++s) sp[c][s] = sc[c][s];
        }
        cp_async_wait<0>();
        __syncthreads();   // the next tile refills the rings
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

template <class AT, class Gather, class Op>
void launch_hex_elem(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    auto kern = k_hex_elem<AT, Gather, Op>;
    using SS = StageSrc<Gather>;
    const size_t smem = sizeof(typename SS::ST) * SS::N * kGridStages * (size_t)kHexPlane +
                        sizeof(AT) * 18 * (size_t)kHexThreads;
    static SmemLimit limit;   // per instantiation and device
    limit.raise(kern, smem, e.ctx->device);
    const double *c = m->hex_modes;
    const HexModes<AT> kc{(AT)c[0], (AT)c[1], (AT)c[2], (AT)c[3], (AT)c[4], (AT)c[5], (AT)c[6], (AT)c[7]};
    const int blocks = (int)std::min<int64_t>(m->hex_ntile, e.max_blocks);
    launch_chain(kern, blocks, kHexThreads, smem, e.stream, m->hex_meshes.as<HexMesh>(), m->hex_nmesh, m->hex_ntile, kc,
                                                  m->hex_factor.as<AT>(), m->hex_factor.as<AT>() + 576, g, op, e.done,
                                                  e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

// ---------------------------------------------------------------------------
// Trilinear transfers without a matrix (DV_FORMAT_TRILINEAR): the factor-2 coarsening of an even
// structured grid (coarse nodes at the even fine nodes, x = 0 clamped), prolongation y_f = P x_c
// (a fine node takes 1 or 2 coarse nodes per axis, weights 1 or 1/2) and restriction y_c = P^T x_f
// (a coarse node takes the fine nodes at -1, 0, +1 per axis, weights 1/2, 1, 1/2).  Each row sums
// its columns in increasing order with the same multiply-add rounding as a stored matrix, so the
// products equal those of the assembled P and P^T (dv_hex_trilinear) bit for bit.
// ---------------------------------------------------------------------------
struct TriGeom {
    int32_t f0, f1, f2;   // fine element counts (even)
    __host__ __device__ int64_t nodes(bool restrict_) const {   // rows / 3
        return restrict_ ? (int64_t)(f0 / 2) * (f1 / 2 + 1) * (f2 / 2 + 1) : (int64_t)f0 * (f1 + 1) * (f2 + 1);
    }
    __host__ __device__ int64_t items(bool restrict_) const { return restrict_ ? nodes(true) : nodes(false) / 2; }
};

// Adds to s the rows of the fine nodes 2 q and 2 q + 1 (prolongation; fine element counts are even, so X = 2 m + 1
// and 2 m + 2 lie in one row and share the coarse nodes m and m + 1 of up to four coarse rows), or of coarse
// node q (restriction), in increasing column order.  g(column) gathers; dof d takes column d of each node.  All of a
// pair's values (restriction: a fine plane's) are loaded before the first is added: added one after another
// as they come, a row waits for up to 8 (27) loads in turn.  Mixed solve 128^3 6.50 -> 6.27 ms, 16^3 0.86 -> 0.82 ms,
// FP64 solve 96 x 48 x 48 2.80 -> 2.67 ms; 64 load cases on 48^3
// (k_bprod_tri) 26.3 -> 25.2 ms.
template <class AT, bool FU, class F>
__device__ __forceinline__ void tri_prolong(const TriGeom &G, uint32_t q, F &&g, AT (&s)[6]) {
    // 32-bit index arithmetic throughout: rows and columns are below 2^31
    const uint32_t ny = G.f1 + 1, cx = G.f0 / 2, cy = G.f1 / 2 + 1;
    const uint32_t t = q / cx, m = q - t * cx, Z = t / ny, Y = t - Z * ny;
    const bool oy = Y & 1, oz = Z & 1;   // between two coarse nodes: weights 1/2
    AT v[4][2][3];
#pragma unroll
    for (int i = 0; i < 4; ++i)   // coarse rows, y fastest
        if ((!(i & 1) || oy) && (!(i & 2) || oz)) {
            const uint32_t col = 3u * (m + cx * (Y / 2 + (i & 1) + cy * (Z / 2 + (i >> 1))));
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                v[i][0][d] = m > 0 ? g(col - 3 + d) : AT(0);   // coarse node 0 is clamped
                v[i][1][d] = g(col + d);
            }
        }
    const AT w = (oy ? AT(0.5) : AT(1)) * (oz ? AT(0.5) : AT(1)), wh = AT(0.5) * w;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if ((!(i & 1) || oy) && (!(i & 2) || oz))
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (m > 0) s[d] = madd_op<AT, FU>(s[d], wh, v[i][0][d]);
                s[d] = madd_op<AT, FU>(s[d], wh, v[i][1][d]);
                s[3 + d] = madd_op<AT, FU>(s[3 + d], w, v[i][1][d]);
            }
}
template <class AT, bool FU, class F>
__device__ __forceinline__ void tri_restrict(const TriGeom &G, uint32_t q, F &&g, AT (&s)[3]) {
    const uint32_t ny = G.f1 + 1, cx = G.f0 / 2, cy = G.f1 / 2 + 1;
    const uint32_t t = q / cx, m = q - t * cx;
    const int32_t Zc = (int32_t)(t / cy), Yc = (int32_t)(t - (uint32_t)Zc * cy), X0 = 2 * (int32_t)m + 1;
#pragma unroll
    for (int c = -1; c <= 1; ++c) {
        const int32_t Z = 2 * Zc + c;
        if (Z < 0 || Z > G.f2) continue;
        AT v[3][9];   // the fine nodes X0 .. X0 + 2 of three rows
#pragma unroll
        for (int b = -1; b <= 1; ++b) {
            const int32_t Y = 2 * Yc + b;
            if (Y < 0 || Y > G.f1) continue;
            const uint32_t col = 3u * ((uint32_t)(X0 - 1) + (uint32_t)G.f0 * ((uint32_t)Y + ny * (uint32_t)Z));
#pragma unroll
            for (int k = 0; k < 9; ++k) v[b + 1][k] = X0 + k / 3 <= G.f0 ? g(col + k) : AT(0);
        }
#pragma unroll
        for (int b = -1; b <= 1; ++b) {
            const int32_t Y = 2 * Yc + b;
            if (Y < 0 || Y > G.f1) continue;
#pragma unroll
            for (int k = 0; k < 9; ++k)
                if (X0 + k / 3 <= G.f0) {
                    const AT w = (k / 3 != 1 ? AT(0.5) : AT(1)) * (b ? AT(0.5) : AT(1)) * (c ? AT(0.5) : AT(1));
                    s[k % 3] = madd_op<AT, FU>(s[k % 3], w, v[b + 1][k]);
                }
        }
    }
}
template <bool RESTRICT, class AT, bool FU, class F, int R>
__device__ __forceinline__ void tri_rows(const TriGeom &G, uint32_t q, F &&g, AT (&s)[R]) {
    static_assert(R == (RESTRICT ? 3 : 6), "rows of an item");
    if constexpr (RESTRICT) tri_restrict<AT, FU>(G, q, g, s);
    else tri_prolong<AT, FU>(G, q, g, s);
}

// One thread per pair of fine nodes (prolongation) or coarse node (restriction).
template <bool RESTRICT, class AT, class Gather, class Op>
__global__ void __launch_bounds__(256) k_tri(TriGeom G, Gather g, Op op, const int *__restrict__ done,
                                             double *partials, unsigned *ticket) {
    if (chain_done(done)) return;
    constexpr bool FU = op_fused<Op>::value;
    constexpr int R = RESTRICT ? 3 : 6;
    double red[Op::NRED > 0 ? Op::NRED : 1];
#pragma unroll
    for (int i = 0; i < (Op::NRED > 0 ? Op::NRED : 1); ++i) red[i] = 0.0;
    const uint32_t items = (uint32_t)G.items(RESTRICT);
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < items; q += gridDim.x * blockDim.x) {
        AT s[R];
#pragma unroll
        for (int d = 0; d < R; ++d) s[d] = op.init((int32_t)(R * q) + d);
        tri_rows<RESTRICT, AT, FU>(G, q, g, s);
        finish_rows(op, (int32_t)(R * q), s, red);
    }
    if constexpr (Op::NRED > 0) {
        double tot[Op::NRED];
        if (grid_reduce<Op::NRED, Op::MAXMASK>(red, partials, ticket, tot)) op.finish(tot);
    }
}

template <class AT, class Gather, class Op>
void launch_trilinear(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    const TriGeom G{m->tri_ne[0], m->tri_ne[1], m->tri_ne[2]};
    const int64_t items = G.items(m->tri_restrict);
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, e.max_blocks));
    if (m->tri_restrict) launch_chain(k_tri<true, AT, Gather, Op>, blocks, 256, 0, e.stream, G, g, op, e.done, e.partials, e.ticket);
    else launch_chain(k_tri<false, AT, Gather, Op>, blocks, 256, 0, e.stream, G, g, op, e.done, e.partials, e.ticket);
    DV_CUDA(cudaGetLastError());
    e.ctx->count();
}

// CSR rows, or the decoded entries of a DuVi matrix.
template <class AT, class Gather, class Op>
void launch_csr(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    switch (m->csr_tpr) {
        case 1: launch_csr_tpr<1, AT>(e, m, g, op); break;
        case 4: launch_csr_tpr<4, AT>(e, m, g, op); break;
        case 8: launch_csr_tpr<8, AT>(e, m, g, op); break;
        case 16: launch_csr_tpr<16, AT>(e, m, g, op); break;
        case 3 * 16: launch_csr_nodes<16, AT>(e, m, g, op); break;
        case 3 * 32: launch_csr_nodes<32, AT>(e, m, g, op); break;
        default: launch_csr_tpr<32, AT>(e, m, g, op); break;
    }
}

// Runs op over every row of m with the accumulator type AT (= value precision).
template <class AT, class Gather, class Op>
void launch_rows(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    if (m->format == DV_FORMAT_HEX) {
        launch_hex_elem<AT>(e, m, g, op);
        return;
    }
    if (m->format == DV_FORMAT_TRILINEAR) {
        launch_trilinear<AT>(e, m, g, op);
        return;
    }
    if (m->entries_ok) {
        launch_csr<AT>(e, m, g, op);
        return;
    }
    if (m->format == DV_FORMAT_DUVI && m->duvi_variant == 3) {
        launch_duvi_grid<AT>(e, m, g, op);
        return;
    }
    if (m->format == DV_FORMAT_DUVI && m->duvi_variant == 2) {
        launch_duvi_pattern<AT>(e, m, g, op);
        return;
    }
    if (m->format == DV_FORMAT_DUVI && m->duvi_variant == 1) {
        if (m->vi_bits == 8) launch_duvi_lanes<uint8_t, AT>(e, m, g, op);
        else if (m->vi_bits == 16) launch_duvi_lanes<uint16_t, AT>(e, m, g, op);
        else launch_duvi_lanes<uint32_t, AT>(e, m, g, op);
        return;
    }
    if (m->format == DV_FORMAT_DUVI) {
        // batch width matched to the dominant block length (chosen at upload)
        if (m->duvi_batch == 9) {
            if (m->vi_bits == 8) launch_duvi_vi<uint8_t, AT, Gather, Op, 9>(e, m, g, op);
            else if (m->vi_bits == 16) launch_duvi_vi<uint16_t, AT, Gather, Op, 9>(e, m, g, op);
            else launch_duvi_vi<uint32_t, AT, Gather, Op, 9>(e, m, g, op);
        } else {
            if (m->vi_bits == 8) launch_duvi_vi<uint8_t, AT, Gather, Op, 4>(e, m, g, op);
            else if (m->vi_bits == 16) launch_duvi_vi<uint16_t, AT, Gather, Op, 4>(e, m, g, op);
            else launch_duvi_vi<uint32_t, AT, Gather, Op, 4>(e, m, g, op);
        }
        return;
    }
    launch_csr<AT>(e, m, g, op);
}

// r = b - A x for the residual that a PCG solve reports.  Close to the limit of FP64 its last digits depend on the order
// of the row sums, so it does not follow the kernel that is fastest for the iterations: CSR rows are summed one
// thread a row in the stored order, as DuVi rows are and as a host would.  Long rows, on the average, are split as
// the products split them: one after another, 1,200 and 3,000 entries a row took 0.28 and 0.6 ms of a solve of
// 22 iterations (0.8 and 1.5 ms); 81 entries a row take 0.03 ms of 1.5 (13,872 rows) and 0.14 of 8.9 (117,612).
constexpr int64_t kStoredOrderEntries = 96;   // a row
template <class Gather, class Op>
void launch_reported_residual(const LaunchEnv &e, const dv_matrix *m, Gather g, Op op) {
    if (m->format == DV_FORMAT_CSR && m->nnz <= kStoredOrderEntries * m->n_rows) launch_csr_tpr<1, double>(e, m, g, op);
    else launch_rows<double>(e, m, g, op);
}

// ---------------------------------------------------------------------------
// vector kernels
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_scale(const T *__restrict__ w, const T *__restrict__ b, T *__restrict__ x, int32_t n,
                        const int *__restrict__ done) {
    if (chain_done(done)) return;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] = w[i] * b[i];
}
template <class T>
__global__ void k_copy(const T *__restrict__ a, T *__restrict__ b, int32_t n, const int *__restrict__ done) {
    if (chain_done(done)) return;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = a[i];
}
template <class T>
__global__ void k_fill(T *__restrict__ a, T v, int32_t n, const int *__restrict__ done) {
    if (chain_done(done)) return;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = v;
}
template <class A, class B>
__global__ void k_convert(const A *__restrict__ a, B *__restrict__ b, int32_t n) {
    chain_done(nullptr);   // launched in a chain, whatever comes before it
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = (B)a[i];
}
// x += y
template <class T>
__global__ void k_axpy1(const T *__restrict__ y, T *__restrict__ x, int32_t n, const int *__restrict__ done) {
    if (chain_done(done)) return;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] = x[i] + y[i];
}

// Dense y = Ainv b (coarse solve), one warp per row.
template <class T>
__global__ void k_dense_gemv(const T *__restrict__ a, const T *__restrict__ b, T *__restrict__ y, int32_t n,
                             const int *__restrict__ done) {
    if (chain_done(done)) return;
    const int lane = threadIdx.x & 31;
    const int32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (int32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
        const T *ar = a + (size_t)r * n;
        T s = 0;
        for (int32_t k = lane; k < n; k += 32) s += ar[k] * __ldg(b + k);
        s = warp_sum(s);
        if (lane == 0) y[r] = s;
    }
}

// Dense y = Ainv b with one block of 128 threads per row (the coarse solve of the MG-PCG V-cycle):
// every row's products split over 4 warps, two partial sums per thread, a shared-memory sum.
template <class T>
__global__ void __launch_bounds__(128) k_dense_gemv_rows(const T *__restrict__ a, const T *__restrict__ b,
                                                         T *__restrict__ y, int32_t n, const int *__restrict__ done) {
    if (chain_done(done)) return;
    __shared__ T part[4];
    for (int32_t r = blockIdx.x; r < n; r += gridDim.x) {
        const T *ar = a + (size_t)r * n;
        T s0 = 0, s1 = 0;
        int32_t k = threadIdx.x;
        for (; k + 128 < n; k += 256) {
            s0 += ar[k] * __ldg(b + k);
            s1 += ar[k + 128] * __ldg(b + k + 128);
        }
        if (k < n) s0 += ar[k] * __ldg(b + k);
        T v = warp_sum(s0 + s1);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) y[r] = (part[0] + part[1]) + (part[2] + part[3]);
        __syncthreads();
    }
}

}  // namespace dvk
