"""The allocation-free Jacobi PCG entry point (dv_pcg_solve_noalloc).

For callers that cannot allocate device memory while they solve (a host that
reserved all device memory up front, or a time-critical loop that cannot afford
cudaFree's device-wide synchronisation).  Called through the C ABI, its result must match the allocating entry
point (dv_pcg_solve) on the same matrix and right-hand side, within the
tolerance of the other PCG tests, on two calls in a row: the second call finds
the previous call's data in the shared device array and must not depend on it.
This file is collected last on purpose.
"""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

REL = 1e-7   # tolerance of test_pcg_matches_oracle


@pytest.mark.parametrize("fmt", ["csr", "duvi"])
def test_noalloc_pcg_matches_allocating_pcg(ctx, native, oracle, fmt):
    import torch
    N = native._native
    m = oracle.Model((16, 4, 4), (20, 1, 1))
    A, b = m.kff.to_scipy(), m.rhs()
    ref = native.CudaCsrPcgSolver(ctx, 2000, 1e-8, fmt=fmt).Initialize(A=A, b=b)
    x_ref, st_ref = ref.Solve()
    assert st_ref.HasConverged
    M = native.SparseMatrix(ctx, A, fmt, "f64")
    db = torch.from_numpy(b).cuda()
    dx = torch.full_like(db, float("nan"))
    torch.cuda.synchronize()
    for call in range(2):
        st = N.Stats()
        # free device memory around the call: the warm (second) call must not allocate
        free_before = torch.cuda.mem_get_info()[0]
        N.check(N.lib().dv_pcg_solve_noalloc(M.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()), 0, 2000,
                                             1e-8, C.byref(st)))
        free_after = torch.cuda.mem_get_info()[0]
        if call == 1:
            assert free_after == free_before, (free_before, free_after)
        x = dx.cpu().numpy()
        assert st.converged and not st.failed, call
        assert st.iterations == st_ref.NumIterationsRequired, call
        assert np.max(np.abs(x - x_ref)) <= REL * np.max(np.abs(x_ref)), call
        # the relative residual is recomputed in FP64 at exit, as for the allocating solver
        true_rel = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        assert abs(st.relative_residual - true_rel) <= 1e-3 * true_rel, call
        assert abs(st.relative_residual - st_ref.RelativeResidual) <= 1e-3 * st_ref.RelativeResidual, call
        dx.fill_(float("nan"))   # the next call must not read the old solution
        torch.cuda.synchronize()
    # warm start from the solution: converged at once
    dx.copy_(torch.from_numpy(x_ref))
    torch.cuda.synchronize()
    st = N.Stats()
    N.check(N.lib().dv_pcg_solve_noalloc(M.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()), 1, 2000, 1e-8,
                                         C.byref(st)))
    assert st.converged and st.iterations <= 1
    ref.ReleaseCudaResources()
    M.release()


def test_noalloc_rejects_systems_above_the_limit(ctx, native):
    import torch
    N = native._native
    n = 131073
    A = sp.identity(n, format="csr") * 2.0
    M = native.SparseMatrix(ctx, A, "csr", "f64")
    db = torch.ones(n, dtype=torch.float64, device="cuda")
    dx = torch.zeros_like(db)
    torch.cuda.synchronize()
    st = N.Stats()
    status = N.lib().dv_pcg_solve_noalloc(M.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()), 0, 10, 1e-8,
                                          C.byref(st))
    assert status == N.DV_ERR_ARG
    assert b"131072" in N.lib().dv_last_error()
    M.release()


@pytest.mark.parametrize("fmt,ne", [("csr", (33, 32, 31)), ("csr", (42, 31, 31)), ("duvi", (30, 28, 28)), ("duvi", (42, 31, 31)),
                                    ("csr", (35, 29, 32)), ("duvi", (27, 27, 27))])
def test_noalloc_pcg_sizes(ctx, native, fmt, ne):
    # Systems that iterate by launches (CSR from 104,001 rows, node patterns from 65,537, up to the array's 131,072), and those
    # just below, whose five vectors of n rows share the array (103,950 rows in CSR; 63,504 on patterns).
    import torch
    N = native._native
    A, b = native.hex_stiffness(ne), native.traction_rhs(ne)
    ref = native.CudaCsrPcgSolver(ctx, 2000, 1e-8, fmt=fmt).Initialize(A=A, b=b)
    x_ref, st_ref = ref.Solve()
    assert st_ref.HasConverged
    M = native.SparseMatrix(ctx, A, fmt, "f64")
    db = torch.from_numpy(b).cuda()
    for guess in (0, 1):
        dx = torch.from_numpy(0.5 * x_ref).cuda() if guess else torch.full_like(db, float("nan"))
        torch.cuda.synchronize()
        st = N.Stats()
        N.check(N.lib().dv_pcg_solve_noalloc(M.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()), guess, 2000, 1e-8,
                                             C.byref(st)))
        assert st.converged and not st.failed
        assert guess or abs(st.iterations - st_ref.NumIterationsRequired) <= 1
        x = dx.cpu().numpy()
        assert np.max(np.abs(x - x_ref)) <= REL * np.max(np.abs(x_ref))
    ref.ReleaseCudaResources()
    M.release()


@pytest.mark.parametrize("fmt", ["csr", "duvi"])
@pytest.mark.parametrize("first", [0, 1])
def test_noalloc_after_one_call_with_the_format(fmt, first):
    # After one call with the format, in a fresh process, another call takes no device memory: a small system solved in one kernel
    # and then a large one by launches from a start vector, or the other way round.
    import json
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", f"""
import ctypes as C, json
import numpy as np, torch
import compressiontests_b200 as cb
N, ctx = cb._native, cb.CudaContext(0)
calls = []
for ne in ((16, 4, 4), (36, 32, 32)):
    A, b = cb.hex_stiffness(ne), cb.traction_rhs(ne)
    M = cb.SparseMatrix(ctx, A, "{fmt}", "f64")
    db = torch.from_numpy(b).cuda()
    calls.append((M, db, torch.zeros_like(db)))
if {first}: calls.reverse()
torch.cuda.synchronize()
free, ok = [], []
for k, (M, db, dx) in enumerate(calls):
    st = N.Stats()
    free.append(torch.cuda.mem_get_info()[0])
    N.check(N.lib().dv_pcg_solve_noalloc(M.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()), k, 2000, 1e-6, C.byref(st)))
    ok.append(bool(st.converged))
free.append(torch.cuda.mem_get_info()[0])
print(json.dumps([ok, free]))
"""], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    ok, free = json.loads(r.stdout.strip().splitlines()[-1])
    assert all(ok) and free[1] == free[2], (ok, free)
