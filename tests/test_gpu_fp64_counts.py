"""FP64 solves cut into spgqp_start and spgqp_iterate calls: iterations, Hessian products and status
after every call are those of the iterations asked for, though the cooperative launch (K <= 8) has
formed the direction after them already.  A running solve has made 1 + it products; one that ends because
the next direction vanished (DAD_ZERO) has formed that direction too and says so in the call that asks
for it."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_FP64, PascError, Problem, capi

pytestmark = pytest.mark.gpu


def _problem(T, K, seed=5):
    rng = np.random.default_rng(seed)
    p = Problem(T, K, 10.0, PASC_PREC_FP64)
    p.set_data(rng.integers(0, K, T) + 0.5 * rng.standard_normal(T))
    x0 = rng.random(T * K)
    p.set_gamma(x0)
    p.set_theta(np.arange(K) + 0.5)
    p.update_b()
    return p, x0


@pytest.mark.parametrize("K,T", [(2, 300), (3, 60_000), (8, 700), (9, 300)])
def test_counts_after_every_call(gpulib, K, T):
    p, _ = _problem(T, K)
    with p:
        p.spgqp_start(capi.spgqp_opts(maxit=10, m=10, eps=0.0))
        for n, it in ((0, 0), (1, 1), (0, 1), (4, 5), (100, 10), (3, 10)):
            st = p.spgqp_iterate(n)
            status = capi.PASC_SPG_MAXIT if it == 10 else capi.PASC_SPG_RUNNING
            assert (st.it, st.hessmult, st.status) == (it, it + 1, status), n


@pytest.mark.parametrize("K,T", [(1, 50), (9, 1), (2, 1)])
def test_a_vanished_direction_is_reported_by_the_call_that_asks_for_it(gpulib, K, T):
    """K = 1, or one timestep: no iteration moves gamma for long."""
    p, x0 = _problem(T, K)
    with p:
        opts = capi.spgqp_opts(maxit=200, m=10, eps=0.0, stop_difff=0)
        whole = p.spgqp_solve(opts)
        assert whole.status == capi.PASC_SPG_DAD_ZERO and whole.hessmult == whole.it + 2
        g = p.get_gamma()
        p.set_gamma(x0)
        p.spgqp_start(opts)
        for it in range(whole.it + 1):  # running up to the last iteration
            st = p.spgqp_iterate(0 if it == 0 else 1)
            assert (st.it, st.hessmult, st.status) == (it, it + 1, capi.PASC_SPG_RUNNING)
        for _ in range(2):
            st = p.spgqp_iterate(5)
            assert (st.it, st.hessmult, st.status) == (whole.it, whole.it + 2, capi.PASC_SPG_DAD_ZERO)
        assert st.fx == whole.fx and st.gP == whole.gP
        np.testing.assert_array_equal(p.get_gamma(), g)


@pytest.mark.parametrize("K", [3, 9])
def test_get_fx_belongs_to_iterate(gpulib, K):
    """The objective is handed out after an iterate call, not after a start alone."""
    p, x0 = _problem(300, K)
    with p:
        p.spgqp_start(capi.spgqp_opts(maxit=10, m=10, eps=0.0))
        with pytest.raises(PascError) as e:
            p.get_fx()
        assert e.value.code == capi.PASC_ERR_STATE
        st = p.spgqp_iterate(0)
        assert p.get_fx() == st.fx
        st = p.spgqp_iterate(3)
        assert p.get_fx() == st.fx
        p.set_gamma(x0)
        st = p.spgqp_solve(capi.spgqp_opts(maxit=5, m=10, eps=0.0))
        assert p.get_fx() == st.fx
