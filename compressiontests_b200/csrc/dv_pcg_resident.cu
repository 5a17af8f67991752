// Jacobi PCG as one kernel for systems that are bound by launches, not by memory.
//
// Three launches an iteration (product with p.Ap, update with the stop test, new direction) cost
// about 7 us each on a system of a few thousand rows, where the work itself takes about one: every
// launch waits for the last block of the one before, reads the stop flag, and its last block adds
// the partial sums alone.  Here one cooperative launch runs every iteration.  Block b owns a
// contiguous run of node groups; two exchanges an iteration carry the sums (p.Ap; the residual's),
// and every block adds all blocks' partial sums itself, in block order, so that all take the same
// alpha, beta and stop decision without a third exchange.  The new direction
// p = z + beta p is formed where the product gathers it (its own rows are also stored, into the
// other of two buffers), which saves the third barrier.
// 16^3 cantilever (13,872 rows), 143 iterations through the host interface: 3.31 -> 1.88 ms in CSR (2.74
// with k_csr_nodes alone), most of the 10 us an iteration being the two exchanges.
#include "dv_pcg_resident.cuh"

#include <algorithm>

using namespace dvk;

namespace {

constexpr int kThreadsR = 1024;      // one block an SM: 32 warps, one node group each
constexpr unsigned kSpinLimit = 1u << 22;   // loads of the counter: seconds

struct ResidentArgs {
    const double *M;                 // the inverse diagonal, or the diagonal (invert)
    int invert;
    double *x, *r, *z, *p0, *p1, *ap;
    double *partials;                // p.Ap, then the residual's four sums, of every block
    unsigned *arrived;               // arrivals so far (starts at 0)
    SolverScalars *sc;
    double tol;
    int32_t ngroups;
    int rel_l2;
};

// Sums (bit i of MAXMASK: the maximum) over all blocks, and the barrier between them: this block's go
// out, it arrives at a counter, and when all have arrived it adds all blocks' sums in block order.
// What any block wrote before is visible to all after it.  False when the others did not come within
// the limit; all blocks then leave.  (Without the counter, every block polling every other block's sum,
// an iteration took 4 us more.)
template <int N, unsigned MAXMASK>
__device__ bool grid_total(double (&v)[N], double *partials, unsigned *arrived, unsigned target) {
    __shared__ double tot[N];
    __shared__ int ok;
    block_reduce<N, MAXMASK>(v);   // ends with a barrier: every thread's writes are before the release
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) __stcg(partials + (size_t)i * gridDim.x + blockIdx.x, v[i]);
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
        unsigned spins = 0, seen;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
        } while ((int)(seen - target) < 0 && ++spins < kSpinLimit);
        ok = (int)(seen - target) >= 0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < N) {
        const bool mx = (MAXMASK >> warp) & 1u;
        double a = 0.0;
        for (unsigned b = lane; b < gridDim.x; b += 32) {
            const double q = __ldcg(partials + (size_t)warp * gridDim.x + b);
            a = mx ? fmax(a, q) : a + q;
        }
        a = mx ? warp_max(a) : warp_sum(a);
        if (lane == 0) tot[warp] = a;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = tot[i];
    return ok != 0;
}

// Entries of a node group's three rows: CSR (one column list for the three, see k_csr_nodes) ...
struct CsrGroups {
    const int32_t *rp, *ci;
    const double *va;
    struct Group {
        const int32_t *c;
        const double *v;
        int32_t len;
    };
    __device__ void stage() const {}
    __device__ Group group(int32_t g) const {
        const int32_t s = __ldg(rp + 3 * g), len = __ldg(rp + 3 * g + 1) - s;
        return {ci + s, va + s, len};
    }
    __device__ static uint32_t col(const Group &q, int32_t k) { return (uint32_t)__ldg(q.c + k); }
    __device__ static void values(const Group &q, int32_t k, double (&v)[3]) {
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = __ldg(q.v + (size_t)d * q.len + k);
    }
};
// ... and node patterns (records staged in shared memory, offsets from the group's first row)
struct PatternGroups {
    const uint16_t *pid;
    const uint32_t *start;
    const PatRec<double> *rec;
    int32_t npat, nrec;
    struct Group {
        const PatRec<double> *q;
        int32_t len, r0;
    };
    __device__ static uint4 *smem() {
        extern __shared__ uint4 pcg_smem[];
        return pcg_smem;
    }
    __device__ void stage() const {
        stage_patterns<double>(smem(), rec, start, npat, nrec);
        __syncthreads();
    }
    __device__ Group group(int32_t g) const {
        const PatRec<double> *s = reinterpret_cast<const PatRec<double> *>(smem());
        const uint32_t *st = reinterpret_cast<const uint32_t *>(s + nrec);
        const uint32_t p = __ldg(pid + g);
        return {s + st[p], (int32_t)(st[p + 1] - st[p]), 3 * g};
    }
    __device__ static uint32_t col(const Group &q, int32_t k) { return (uint32_t)(q.r0 + q.q[k].off); }
    __device__ static void values(const Group &q, int32_t k, double (&v)[3]) {
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = q.q[k].v[d];
    }
};

template <class Groups>
__global__ void __launch_bounds__(kThreadsR) k_pcg_resident(Groups G, ResidentArgs a) {
    G.stage();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t per = (a.ngroups + (int32_t)gridDim.x - 1) / (int32_t)gridDim.x;
    const int32_t g0 = min(a.ngroups, (int32_t)blockIdx.x * per), g1 = min(a.ngroups, g0 + per);
    const int32_t i0 = 3 * g0, i1 = 3 * g1;
    double *part_pap = a.partials, *part_res = a.partials + gridDim.x;
    double rz = a.sc->rz, beta = 0.0;
    const double bb = a.sc->bb;
    const int max_it = a.sc->max_it;
    int it = a.sc->it;
    double *pold = a.p0, *pnew = a.p1;
    for (unsigned target = gridDim.x;; target += 2 * gridDim.x) {
        // p = z + beta p, Ap and p.Ap (OpPcgAp, k_pcg_p)
        double pap[1] = {0.0};
        for (int32_t g = g0 + warp; g < g1; g += kThreadsR / 32) {
            const typename Groups::Group q = G.group(g);
            double s[3] = {0.0, 0.0, 0.0};
            for (int32_t base = lane; base < q.len; base += 96) {
                uint32_t c[3];
                double pz[3], pp[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) c[u] = base + 32 * u < q.len ? G.col(q, base + 32 * u) : 0u;
#pragma unroll
                for (int u = 0; u < 3; ++u) {   // other blocks' rows: not through the L1 cache
                    pz[u] = __ldcg(a.z + c[u]);
                    pp[u] = __ldcg(pold + c[u]);
                }
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (base + 32 * u < q.len) {
                        double v[3];
                        G.values(q, base + 32 * u, v);
                        const double xv = pz[u] + beta * pp[u];
#pragma unroll
                        for (int d = 0; d < 3; ++d) s[d] = fma(v[d], xv, s[d]);
                    }
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) s[d] = warp_sum(s[d]);
            if (lane < 3) {
                const int32_t i = 3 * g + lane;
                const double t = lane == 0 ? s[0] : lane == 1 ? s[1] : s[2];
                const double pi = __ldcg(a.z + i) + beta * __ldcg(pold + i);
                __stcg(pnew + i, pi);
                a.ap[i] = t;
                pap[0] = __dadd_rn(pap[0], __dmul_rn(pi, t));
            }
        }
        if (!grid_total<1, 0>(pap, part_pap, a.arrived, target)) return;
        const double alpha = rz / pap[0];
        // x += alpha p, r -= alpha Ap, z = M r and the stop test (k_pcg_update)
        double red[4] = {0.0, 0.0, 0.0, 0.0};
        for (int32_t i = i0 + (int32_t)threadIdx.x; i < i1; i += kThreadsR) {
            a.x[i] = a.x[i] + alpha * __ldcg(pnew + i);
            const double ri = a.r[i] - alpha * a.ap[i];
            a.r[i] = ri;
            const double m = a.M[i];
            const double zi = (a.invert ? 1 / m : m) * ri;
            __stcg(a.z + i, zi);
            const double c = fabs(ri);
            if (isnan(ri) || c > 1e50) red[1] = 1.0;
            else red[0] = fmax(red[0], c);
            red[2] += ri * zi;
            red[3] += ri * ri;
        }
        if (!grid_total<4, 0b0011>(red, part_res, a.arrived, target + gridDim.x)) return;
        const bool failed = red[1] != 0.0;
        const bool converged = !failed && (a.rel_l2 ? red[3] <= a.tol * a.tol * bb : red[0] <= a.tol);
        const bool stop = converged || failed || it > max_it;
        if (stop) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                a.sc->it = it;
                a.sc->res_max = red[0];
                a.sc->res_norm2 = sqrt(red[3]);
                a.sc->converged = converged;
                a.sc->failed = failed;
                a.sc->done = 1;
            }
            return;
        }
        beta = red[2] / rz;
        rz = red[2];
        it += 1;
        double *t = pold;
        pold = pnew;
        pnew = t;
    }
}

template <class Groups>
bool launch_resident(dv_context *ctx, const Groups &G, ResidentArgs a, size_t smem) {
    auto kern = k_pcg_resident<Groups>;
    static SmemLimit limit;   // per instantiation and device
    limit.raise(kern, smem, ctx->device);
    void *args[] = {const_cast<Groups *>(&G), &a};
    const cudaError_t err = cudaLaunchCooperativeKernel(reinterpret_cast<void *>(kern), dim3(ctx->num_sms), dim3(kThreadsR),
                                                        args, smem, ctx->stream);   // one block an SM
    if (err == cudaErrorCooperativeLaunchTooLarge || err == cudaErrorNotSupported) {
        cudaGetLastError();
        return false;
    }
    DV_CUDA(err);
    ctx->count();
    return true;
}

}  // namespace

size_t dv_pcg_resident_bytes(dv_context *ctx) { return 64 + 5 * sizeof(double) * (size_t)ctx->num_sms; }

bool dv_pcg_resident_ok(const dv_matrix *A) {
    if (A->precision != DV_F64 || A->n_rows > kPcgResidentRows || A->n_rows % 3 != 0 || A->n_rows == 0) return false;
    if (A->format == DV_FORMAT_CSR) return A->row_group == 3;
    return A->n_rows <= kPcgResidentPatternRows && A->format == DV_FORMAT_DUVI && A->pat_ok && A->lanes_group == 3 && !A->pat_based && !A->pat_shift &&
           sizeof(PatRec<double>) * (size_t)A->pat_entries + 4 * ((size_t)A->pat_count + 1) <=
               (size_t)std::min(160 * 1024, A->ctx->max_smem_optin - 2048);   // less the sums' own shared memory
}

bool dv_pcg_resident(dv_matrix *A, const double *M, int invert, double *x, double *r, double *z, double *p0, double *p1, double *ap,
                     void *work, SolverScalars *sc, double tol, int rel_l2) {
    dv_context *ctx = A->ctx;
    ResidentArgs a;
    a.M = M;
    a.invert = invert;
    a.x = x;
    a.r = r;
    a.z = z;
    a.p0 = p0;
    a.p1 = p1;
    a.ap = ap;
    a.arrived = static_cast<unsigned *>(work);
    a.partials = reinterpret_cast<double *>(static_cast<char *>(work) + 64);
    a.sc = sc;
    a.tol = tol;
    a.ngroups = A->n_rows / 3;
    a.rel_l2 = rel_l2;
    DV_CUDA(cudaMemsetAsync(work, 0, 64, ctx->stream));
    DV_CUDA(cudaMemsetAsync(p0, 0, sizeof(double) * (size_t)A->n_rows, ctx->stream));   // read with beta = 0 first
    if (A->format == DV_FORMAT_CSR)
        return launch_resident(ctx, CsrGroups{A->rowptr.as<int32_t>(), A->col.as<int32_t>(), A->val.as<double>()}, a, 0);
    return launch_resident(ctx, PatternGroups{A->pat_id.as<uint16_t>(), A->pat_start.as<uint32_t>(),
                                              static_cast<const PatRec<double> *>(A->pat_rec.p), A->pat_count,
                                              A->pat_entries}, a,
                           sizeof(PatRec<double>) * (size_t)A->pat_entries + 4 * ((size_t)A->pat_count + 1));
}
