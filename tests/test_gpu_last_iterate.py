"""spgqp_last_iterate: device time and launches of the iterations of the last spgqp_iterate or
spgqp_solve.  The start (a sweep of its own on the sweep kernels) is part of the solve's time and not
of the iterations'."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, Problem, capi

pytestmark = pytest.mark.gpu


def _problem(T, K, variant):
    rng = np.random.default_rng(T)
    p = Problem(T, K, 10.0, PASC_PREC_MIXED)
    p.set_data(rng.integers(0, K, T) + 0.5 * rng.standard_normal(T))
    p.set_gamma(rng.random(T * K))
    p.set_theta(np.arange(K) + 0.5)
    p.set_sweep_variant(variant)
    return p


@pytest.mark.parametrize("variant", [0, 1])
def test_solve_on_the_sweep_kernels(gpulib, variant):
    with _problem(300_000, 3, variant) as p:
        st = p.spgqp_solve(capi.spgqp_opts(maxit=5, eps=0.0))
        ms, n = p.spgqp_last_iterate()
        assert st.it == 5 and n == 5 and st.kernel_launches == 6
        assert 0.0 < ms * 1e-3 < st.time_s


def test_solve_in_one_launch(gpulib):
    with _problem(20_000, 3, -1) as p:
        opts = capi.spgqp_opts(maxit=5, eps=0.0)
        st = p.spgqp_solve(opts)
        ms, n = p.spgqp_last_iterate()
        assert st.it == 5 and n == 1 and 0.0 < ms * 1e-3 <= st.time_s
        p.spgqp_start(opts)
        assert p.spgqp_last_iterate() == (0.0, 0)  # a start alone iterates nothing
        st = p.spgqp_iterate(2)
        ms, n = p.spgqp_last_iterate()
        assert st.it == 2 and n == 1 and 0.0 < ms * 1e-3 < st.time_s
        p.spgqp_iterate(0)  # nothing of the call before is left over
        assert p.spgqp_last_iterate() == (0.0, 0)
