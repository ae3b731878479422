"""FP64 solves in one cooperative launch (K <= 8, 1-D) against the oracle, at the edges of the plan:
tiles of 64, 128 and 256 timesteps, short last blocks, the two forms on both sides of 256 * 4 * SMs
entries, and K = 9, which keeps one kernel per operation.

Per entry the arithmetic is the oracle's; the sums differ by their order (about 1e-16 relative each).  Ten iterations of the oracle move by
1e-13 relative in f under a 1-ulp change of a step length: f is held to 1e-12 relative, gamma to
1e-10 (the bound of the FP64 trajectories of the other tests is 1e-12 after three iterations).  A solve
cut into start and iterate calls keeps g, d and Ad: equal bit for bit."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_FP64, Problem, capi

pytestmark = pytest.mark.gpu

CASES = [(1, 300), (2, 5), (2, 128), (2, 129), (2, 9728), (2, 77_824), (2, 77_825), (3, 255), (3, 256), (3, 257),
         (3, 51_882), (3, 51_883), (4, 64), (4, 9800), (5, 30_720), (6, 513), (7, 1000), (8, 65), (8, 19_456),
         (8, 19_457), (3, 154_500), (9, 300)]


@pytest.mark.parametrize("K,T", CASES)
@pytest.mark.parametrize("tp", [False, True])
def test_fp64_fused_edges(gpulib, oracle, K, T, tp):
    rng = np.random.default_rng(1000 * K + T)
    data = rng.integers(0, K, T) + 0.5 * rng.standard_normal(T)
    theta = np.arange(K) + 0.5
    x0 = rng.random(T * K)
    b = oracle.residual_b(data, theta, T, K)
    coeff = oracle.A_coeff(10.0, T)
    oo = oracle.spg_opts(maxit=10, m=10, eps=0.0)
    xo, ro = (oracle.spgqp_solve_kc(b, x0, T, K, coeff * theta * theta, oo) if tp
              else oracle.spgqp_solve(b, x0, T, K, coeff, oo))[:2]
    opts = capi.spgqp_opts(maxit=10, m=10, eps=0.0)
    with Problem(T, K, 10.0, PASC_PREC_FP64) as p:
        p.set_data(data)
        p.set_gamma(x0)
        if tp:
            p.set_usethetainpenalty(True)
        p.set_theta(theta)
        p.update_b()
        st = p.spgqp_solve(opts)
        g = p.get_gamma()
        p.set_gamma(x0)
        p.spgqp_start(opts)
        p.spgqp_iterate(4)
        st2 = p.spgqp_iterate(6)
        np.testing.assert_array_equal(p.get_gamma(), g)
    assert st.it == st2.it and st.fx == st2.fx and st.gP == st2.gP and st.status == st2.status
    if K == 1:  # gamma is 1 everywhere: the solve ends at once
        assert st.it == 0 and np.all(g == 1.0)
        return
    assert st.it == ro.it == 10
    assert abs(st.fx - ro.fx) <= 1e-12 * abs(ro.fx), (st.fx, ro.fx)
    assert np.max(np.abs(g - xo)) <= 1e-10
