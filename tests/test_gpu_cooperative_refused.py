"""Cooperative launches that the device refuses: the solves, the adjoint and the polish go on with
ordinary launches.  The refusal is made on the host: the library's objects are linked once more with
cudaLaunchCooperativeKernel replaced by a function that answers an error code (nothing is launched
then), and a child process runs on that library.

The same library with a cooperative launch one block short: the block before the missing one waits for
edges that nobody writes.  The wait is bounded (a few seconds), the call reports it, and the handle solves
again afterwards.  (Every index stays within the buffers, which hold the words of a block per SM.)

Results against the same calls with the launches accepted: FP64 bit for bit (the paths keep one order of
sums), mixed solves within the bounds of test_gpu_resident, gradients within those of test_gpu_cg."""
import glob
import os
import subprocess
import sys

import pytest

from pasc_inference_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <cuda_runtime.h>
extern "C" {
int coop_answer = 0;   // 0: the real launch; > 0: the error it answers; -1: a block short
int coop_calls = 0;
cudaError_t __real_cudaLaunchCooperativeKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t);
cudaError_t __wrap_cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s)
{
    coop_calls++;
    if (coop_answer < 0) g.x -= 1;
    return coop_answer > 0 ? (cudaError_t)coop_answer : __real_cudaLaunchCooperativeKernel(f, g, b, a, m, s);
}
}
"""

CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from pasc_inference_gb300 import capi
capi.LIB_PATH = sys.argv[2]
from pasc_inference_gb300 import PASC_PREC_FP64, PASC_PREC_MIXED, Problem
lib = capi.load()
answer, calls = (C.c_int.in_dll(lib, n) for n in ("coop_answer", "coop_calls"))
T, K = 30_000, 3
rng = np.random.default_rng(1)
data = rng.integers(0, K, T) + 0.5 * rng.standard_normal(T)
x0 = rng.random(T * K)
dg = rng.standard_normal(T * K) / T
theta = np.arange(K) + 0.1

def solve(prec, cut):
    with Problem(T, K, 10.0, prec) as p:
        p.set_data(data); p.set_gamma(x0); p.set_theta(theta); p.update_b()
        o = capi.spgqp_opts(maxit=3, m=10, eps=0.0)
        if cut:
            p.spgqp_start(o); p.spgqp_iterate(1); st = p.spgqp_iterate(2)
        else:
            st = p.spgqp_solve(o)
        assert (st.it, st.hessmult, st.status) == (3, 4, capi.PASC_SPG_MAXIT)
        return st.fx, p.get_gamma(), st.kernel_launches

def adjoint():
    with Problem(T, K, 200.0, PASC_PREC_MIXED) as p:
        g = np.zeros((T, K)); t = np.arange(T); on = (t % 80) < 40; on[-1] = False
        g[t, (t // 80) % K] = 1.0
        mix = np.random.default_rng(2).random((T, K)) + 0.5
        g[on] = mix[on] / mix[on].sum(1, keepdims=True)
        p.set_data(data); p.set_theta(theta); p.set_gamma(g.astype(np.float32).astype(float).ravel())
        deps, dX, dth, st = p.adjoint(dg, opts=capi.adjoint_opts(cg_tol=1e-11))
        assert st.status == 1
        pst = p.polish()
        return deps, dX, dth, pst.fx

def run(code):
    answer.value, calls.value = code, 0
    return [solve(p, cut) for p in (PASC_PREC_FP64, PASC_PREC_MIXED) for cut in (False, True)] + [adjoint()], calls.value

want, n = run(0)
assert n >= 8, n
for code in (int(v) for v in sys.argv[3:]):
    got, n = run(code)
    assert n == 5, n  # every handle asks once and remembers
    for i in (0, 1):
        assert got[i][0] == want[i][0] and np.array_equal(got[i][1], want[i][1])
    for i in (2, 3):
        assert abs(got[i][0] - want[i][0]) <= 2e-6 * abs(want[i][0])
        assert np.linalg.norm(got[i][1] - want[i][1]) <= 1e-5 * np.linalg.norm(want[i][1])
        assert got[i][2] > want[i][2]
    for a, b in zip(got[4], want[4]):
        a, b = np.atleast_1d(a), np.atleast_1d(b)
        assert np.max(np.abs(a - b)) <= 1e-5 * max(np.max(np.abs(b)), 1e-300)
print("ok")
"""


@pytest.fixture(scope="module")
def refusing_library(gpulib, tmp_path_factory):
    d = tmp_path_factory.mktemp("coop")
    src, obj, lib = d / "shim.cu", d / "shim.o", d / "libpasc_refusing.so"
    src.write_text(SHIM)
    B.build()  # (the objects: nothing to do where the library was built here)
    objs = sorted(glob.glob(os.path.join(B.BUILD_DIR, "*.o")))
    subprocess.check_call([B.nvcc(), *B.ARCH_FLAGS, "-Xcompiler", "-fPIC", "-c", str(src), "-o", str(obj)])
    subprocess.check_call([B.nvcc(), *B.ARCH_FLAGS, "-shared", "-o", str(lib), *objs, str(obj), "-Xlinker",
                           "--wrap=cudaLaunchCooperativeKernel"])
    return str(lib)


def test_refused_launches_fall_back(refusing_library):
    # cudaErrorCooperativeLaunchTooLarge, cudaErrorNotSupported, cudaErrorNotPermitted
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, refusing_library, "720", "801", "800"], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


TIMEOUT_CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from pasc_inference_gb300 import capi
capi.LIB_PATH = sys.argv[2]
from pasc_inference_gb300 import PASC_PREC_MIXED, PascError, Problem
answer = C.c_int.in_dll(capi.load(), "coop_answer")
T, K = 20_000, 3
rng = np.random.default_rng(1)
x0 = rng.random(T * K)
o = capi.spgqp_opts(maxit=3, m=10, eps=0.0)
with Problem(T, K, 10.0, PASC_PREC_MIXED) as p:
    p.set_data(rng.integers(0, K, T) + 0.5 * rng.standard_normal(T)); p.set_gamma(x0); p.set_theta(np.arange(K) + 0.1)
    want = p.spgqp_solve(o).fx, p.get_gamma()
    p.set_gamma(x0)
    answer.value = -1
    try:
        p.spgqp_solve(o)
    except PascError as e:
        assert e.code == capi.PASC_ERR_TIMEOUT and "another block" in str(e), e
    else:
        raise AssertionError("no error")
    answer.value = 0
    p.set_gamma(x0)
    assert p.spgqp_solve(o).fx == want[0]
    assert np.array_equal(p.get_gamma(), want[1])
print("ok")
"""


def test_wait_for_a_missing_block_is_reported(refusing_library):
    r = subprocess.run([sys.executable, "-c", TIMEOUT_CHILD, ROOT, refusing_library], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
