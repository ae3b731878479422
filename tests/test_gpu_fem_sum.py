"""The mixed path's FEM-SUM kernels (bounds made once, float-float field sums, shifted residual sums,
copy back) against the FP64 path, at block counts around the kernels' blocks of 256, coarse steps of
one to all timesteps, and data far from zero.

One outer iteration with no SPG iteration: theta, the reduced b and gamma, the projected start point,
its objective and the prolongated gamma.  The reduced gamma, sums of up to n = 1/reduce + 1 values
below 1, is stored in FP32 before it is projected: half an ulp of a sum (n 6e-8) on the value and on the
threshold, 2.4e-7 n with the projection's own rounding; f moves by as much times its slope, a few
units per timestep: 1e-6 n."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_FP64, PASC_PREC_MIXED, Problem, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,reduce", [(5, 0.2), (256, 0.5), (257, 0.999), (2560, 0.1), (2561, 0.1), (5119, 0.05), (30_000, 0.0001),
                                      (77_777, 0.37)])
@pytest.mark.parametrize("K,offset", [(1, 0.0), (2, 0.0), (3, 1000.0), (5, -20.0), (8, 0.0)])
def test_fem_sum_mixed_vs_fp64(gpulib, T, reduce, K, offset):
    rng = np.random.default_rng(T + K)
    data = (offset + rng.integers(0, K, T) + 0.5 * rng.standard_normal(T)).astype(np.float32).astype(np.float64)
    g0 = rng.random(T * K).astype(np.float32).astype(np.float64)
    theta = offset + np.arange(K) + 0.25
    res = []
    for prec in (PASC_PREC_FP64, PASC_PREC_MIXED):
        with Problem(T, K, 1.0, prec) as p:
            p.set_fem(reduce, 0)
            p.set_data(data)
            p.set_gamma(g0)
            p.set_theta(theta)
            st = p.ts_solve(capi.ts_opts(maxit=1, thetasolved=1), capi.spgqp_opts(maxit=0))
            res.append((st.L, p.get_gamma()))
    (L64, g64), (L32, g32) = res
    n = min(T, 1.0 / reduce + 1.0)
    assert np.max(np.abs(g64 - g32)) <= 2.4e-7 * n
    assert abs(L64 - L32) <= 1e-6 * n * max(abs(L64), 1.0)
