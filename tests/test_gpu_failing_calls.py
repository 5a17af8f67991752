"""CUDA calls that fail: what the library does when an allocation has no room or a launch is refused.

The failure comes from a stand-in for the runtime's entry point, preloaded into a child process: it asks for more memory
than there is, or returns the launch's error code and calls nothing, so nothing runs on the GPU.
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STAND_IN = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static size_t lo = 1, hi = 0;   /* allocations of lo .. hi bytes fail */
static int fail_cooperative, failed;
void fail_allocations(size_t from, size_t to) { lo = from; hi = to; }
void fail_cooperative_launches(int on) { fail_cooperative = on; }
int failed_calls(void) { return failed; }
static void *real(const char *name) {
    void *lib = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
    return dlsym(lib, name);
}
int cudaMalloc(void **p, size_t bytes) {
    if (bytes >= lo && bytes <= hi) { failed++; bytes = (size_t)1 << 50; }   /* more than any device has: out of memory */
    return ((int (*)(void **, size_t))real("cudaMalloc"))(p, bytes);
}
typedef struct { unsigned x, y, z; } Dim;
int cudaLaunchCooperativeKernel(const void *f, Dim grid, Dim block, void **args, size_t smem, void *stream) {
    if (fail_cooperative) { failed++; return 720; }   /* cudaErrorCooperativeLaunchTooLarge */
    return ((int (*)(const void *, Dim, Dim, void **, size_t, void *))real("cudaLaunchCooperativeKernel"))(f, grid, block, args,
                                                                                                           smem, stream);
}
"""
PRELUDE = """
import ctypes, json, sys
import numpy as np
import compressiontests_b200 as cb
fake = ctypes.CDLL(None)
fake.fail_allocations.argtypes = [ctypes.c_size_t, ctypes.c_size_t]
ctx = cb.CudaContext(0)
"""


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    """Runs a script in a process with the stand-in loaded first; the script prints one JSON line."""
    d = tmp_path_factory.mktemp("stand_in")
    (d / "f.c").write_text(STAND_IN)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(d / "f.so"), str(d / "f.c"), "-ldl"], check=True)

    def run(script):
        env = dict(os.environ, LD_PRELOAD=str(d / "f.so"), PYTHONPATH=ROOT)
        r = subprocess.run([sys.executable, "-c", PRELUDE + script], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return json.loads(r.stdout.strip().splitlines()[-1])

    return run


def test_solver_without_room_for_decoded_entries(child):
    # The decoded copy of the outer operator has no room: the solver keeps that operator on its layout and solves as with the copy.
    r = child("""
ne = (12, 8, 8)
A, P = cb.hex_hierarchy(ne, coarse_ne=4)
b = cb.traction_rhs(ne)
out = []
for fail in (False, True):
    n = 8 * A[0].nnz + 64
    if fail: fake.fail_allocations(n, n)
    s = cb.MultigridPcgSolver(ctx, A, P, precision="mixed", fmt="duvi")
    fake.fail_allocations(1, 0)
    x, st = s.Solve(b)
    out.append((x, st.HasConverged, st.NumIterationsRequired))
print(json.dumps(dict(failed=fake.failed_calls(), ok=[o[1] for o in out], its=[o[2] for o in out],
                      diff=float(np.max(np.abs(out[0][0] - out[1][0])) / np.max(np.abs(out[0][0]))))))
""")
    # two solves to a relative residual of 1e-8, each within 1e-6 of the solution
    assert r["failed"] == 1 and r["ok"] == [True, True] and r["its"][0] == r["its"][1] and r["diff"] < 2e-6, r


@pytest.mark.parametrize("fmt", ["csr", "duvi"])
def test_pcg_where_the_cooperative_launch_is_refused(child, fmt):
    # A process that has fewer SMs than the device reports: the driver refuses the one-kernel solve and the solvers
    # iterate in chunks, with and without a start vector.
    r = child(f"""
import torch
N = cb._native
ne = (16, 6, 5)
A, b = cb.hex_stiffness(ne), cb.traction_rhs(ne)
out = []
for fail in (0, 1):
    fake.fail_cooperative_launches(fail)
    s = cb.CudaCsrPcgSolver(ctx, 2000, 1e-9, fmt="{fmt}").Initialize(A=A, b=b)
    x, st = s.Solve()
    x2, st2 = s.Solve(xInitialGuess=0.5 * x)
    M = cb.SparseMatrix(ctx, A, "{fmt}", "f64")
    db = torch.from_numpy(b).cuda()
    dx = torch.zeros_like(db)
    torch.cuda.synchronize()
    sn = N.Stats()
    N.check(N.lib().dv_pcg_solve_noalloc(M.h, ctypes.c_void_p(db.data_ptr()), ctypes.c_void_p(dx.data_ptr()), 0, 2000, 1e-9,
                                         ctypes.byref(sn)))
    out.append(([x, x2, dx.cpu().numpy()], [st.HasConverged, st2.HasConverged, bool(sn.converged)],
                [st.NumIterationsRequired, st2.NumIterationsRequired, sn.iterations]))
print(json.dumps(dict(failed=fake.failed_calls(), ok=[o[1] for o in out], its=[o[2] for o in out],
                      diff=[float(np.max(np.abs(p - q)) / np.max(np.abs(p))) for p, q in zip(out[0][0], out[1][0])])))
""")
    assert r["failed"] == 3 and all(r["ok"][0]) and all(r["ok"][1]), r
    assert all(abs(p - q) <= 1 for p, q in zip(*r["its"])) and max(r["diff"]) < 1e-7, r


@pytest.mark.parametrize("which", ["V-cycle block", "outer block", "scalars"])
def test_load_cases_after_an_allocation_failed(child, which):
    # Resizing the block buffers for another number of load cases has no room once: that call raises, the next one with the
    # same number allocates them anew and solves (8 columns in FP32 and FP64 blocks, 8 columns' scalars).
    r = child(f"""
ne, k = (12, 8, 8), 8
B = cb.random_face_loads(ne, k, seed=2)
s = cb.MultigridPcgSolver.from_hex(ctx, ne, coarse_ne=4, precision="mixed", tol=1e-9)
ref = s.solve_many(B)[0]
s.solve_many(B[:, :3])
n = {{"V-cycle block": 4 * k * B.shape[0] + 64, "outer block": 8 * k * B.shape[0] + 64}}.get("{which}")
if n is None: fake.fail_allocations(64 + 8 * k, 1024)
else: fake.fail_allocations(n, n)
raised = ""
try:
    s.solve_many(B)
except cb.DuviError as e:
    raised = str(e)
fake.fail_allocations(1, 0)
X, st, conv = s.solve_many(B)
print(json.dumps(dict(raised=raised, ok=bool(conv.all()), same=bool(np.array_equal(X, ref)))))
""")
    assert "memory" in r["raised"] and r["ok"] and r["same"], r
