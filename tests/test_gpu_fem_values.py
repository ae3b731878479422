"""The mixed path's FEM-SUM kernels on values at the ends of their range, called by themselves (their
sums are not readable through the ABI): infinities stay infinities, and sums that leave the FP32 range
before they are scaled back into it are kept; a block whose first value lies far from all others keeps
its digits.

A sum is stored in FP32: 2^-24 relative to the exact one; 2^-23 leaves room for the FP64 rounding in front
of it."""
import ctypes as C
import math
import re
import subprocess

import numpy as np
import pytest

from pasc_inference_gb300 import capi

pytestmark = pytest.mark.gpu


def _launcher(lib, name, *argtypes):
    """A launcher of the library's internal interface (a C++ symbol)."""
    names = subprocess.run(["nm", "-D", "--defined-only", capi.LIB_PATH], capture_output=True, text=True, check=True).stdout
    sym = re.findall(rf"\b(_ZN4pasc{len(name)}{name}E\w+)", names)
    assert len(sym) == 1, sym
    f = getattr(lib, sym[0])
    f.restype, f.argtypes = C.c_int, list(argtypes)
    return f


def _check(got, want):
    ok = np.isfinite(want)
    np.testing.assert_array_equal(got[~ok], want[~ok])
    np.testing.assert_allclose(got[ok], want[ok], rtol=2.0**-23, atol=0.0)


def test_fem_sum_field_range(gpulib):
    torch = pytest.importorskip("torch")
    launch = _launcher(gpulib, "launch_fem_sum_field", C.c_void_p, C.c_void_p, C.c_void_p, C.c_long, C.c_int, C.c_double,
                       C.c_void_p)
    K, lo = 3, np.array([0, 5, 9, 9, 30, 31, 1031], dtype=np.int32)
    T1, T2 = int(lo[-1]), len(lo) - 1
    rng = np.random.default_rng(3)
    g = rng.standard_normal((T1, K)).astype(np.float32)
    g[5:9, 0] = 3e38             # four of them: beyond FP32, in FP64 not
    g[6, 1] = np.inf
    g[7, 2] = np.nan
    g[12, 0], g[20, 1] = -np.inf, 3e38
    for scale in (1.0, 2.0**-10, -0.1):
        gd, ld = torch.tensor(g, device="cuda"), torch.tensor(lo, device="cuda")
        out = torch.full((T2, K), 7.0, device="cuda")
        assert launch(gd.data_ptr(), out.data_ptr(), ld.data_ptr(), T2, K, scale, None) == 0
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            want = np.array([[np.float32(scale * float(np.sum(g[a:b, k].astype(np.float64))))
                              for k in range(K)] for a, b in zip(lo[:-1], lo[1:])])
        _check(out.cpu().numpy(), want)


def test_fem_sum_residual_cancellation_and_range(gpulib):
    torch = pytest.importorskip("torch")
    launch = _launcher(gpulib, "launch_fem_sum_residual", C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_long, C.c_int,
                       C.c_double, C.c_void_p)
    n = 400_000
    lo = np.array([0, n, n + 10, n + 10, n + 20, n + 30, n + 40, n + 41, 2 * n], dtype=np.int32)
    T1, T2, K = int(lo[-1]), len(lo) - 1, 3
    theta = np.array([0.3, 0.3000001, 2.0])
    rng = np.random.default_rng(4)
    x = theta[0] + 1e-3 * rng.standard_normal(T1)
    x[:n] = 0.3000001
    x[0] = 1e4                    # far from all others: sum (x - x[0])^2 is n times the result
    x[n + 10], x[n + 25], x[n + 33] = np.inf, -np.inf, np.nan
    x[n + 40] = theta[0]          # a block of one timestep, on a theta: exactly 0
    for scale in (1.0, -1.0 / T2):
        xd, td, ld = (torch.tensor(v, device="cuda") for v in (x, theta, lo))
        out = torch.full((T2, K), 7.0, dtype=torch.float32, device="cuda")
        assert launch(xd.data_ptr(), td.data_ptr(), out.data_ptr(), ld.data_ptr(), T2, K, scale, None) == 0
        torch.cuda.synchronize()
        want = np.array([[np.float32(scale * (math.fsum((x[a:b] - theta[k]) ** 2) if np.all(np.isfinite(x[a:b]))
                                              else np.sum((x[a:b] - theta[k]) ** 2)))
                          for k in range(K)] for a, b in zip(lo[:-1], lo[1:])])
        _check(out.cpu().numpy(), want)
