// Jacobi PCG in one cooperative kernel, for systems small enough to be bound by launches.
#pragma once

#include "dv_kernels.cuh"

// Largest system that takes it.  An iteration costs 10 us plus its work at the pace of one block an SM;
// the launches cost about 18 us plus the work at full pace.  Measured an iteration, launches -> one
// kernel: CSR 13,872 rows 19.5 -> 10.6 us, 45,000 rows 26.5 -> 16.5 (crossing near 120,000; five vectors
// of 104,000 rows fit the fixed array of dv_pcg_solve_noalloc); node patterns 19.5 -> 10.8, 19.5 -> 16.0
// (crossing near 70,000, their product reads less).
constexpr int32_t kPcgResidentRows = 104000, kPcgResidentPatternRows = 65536;

// Whether the kernel has a product for this matrix (FP64, node groups of 3 rows: CSR with one column
// list a group, or the node-pattern layout) and the system is small enough.
bool dv_pcg_resident_ok(const dv_matrix *A);
// Bytes of `work` below (barrier and partial sums).
size_t dv_pcg_resident_bytes(dv_context *ctx);
// Iterates from r, z = M r and sc (rz, bb, it, max_it) until sc->done, the same steps and stop test as
// dv_pcg_solve's chunks; M is the inverse diagonal, or with invert the diagonal; p0, p1, ap are work
// vectors.  Context stream, asynchronous.  sc->done stays
// 0 if the blocks lost one another (a bounded wait ran out).  False where the driver does not take the
// cooperative launch (fewer SMs for this process than the device has): p1, r, z and sc are then as they came, and the
// caller iterates in chunks.
bool dv_pcg_resident(dv_matrix *A, const double *M, int invert, double *x, double *r, double *z, double *p0, double *p1, double *ap,
                     void *work, dvk::SolverScalars *sc, double tol, int rel_l2);
