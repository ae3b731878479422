"""The adjoint's FP32 conjugate gradients over the list of active timesteps (one cooperative launch)
at the edges of its plan: one block, short last blocks, one entry per thread and several, and a
problem whose active timesteps do not fit in shared memory (all timesteps, one kernel per half
iteration).  Active timesteps come in runs of given length, so neighbours of the list are
neighbours in time inside a run only.

Against the FP64 oracle on the same gamma, both solves to a relative residual of 1e-12 (1e-10 for
the large one, whose refinement ends above 1e-12 with all timesteps as well): gradients within 1e-5
(the FP32 steps run inside FP64 refinement; the bound of the other mixed adjoint tests)."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, Problem, capi

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = np.atleast_1d(a), np.atleast_1d(b)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


# T, K, length of the runs, timesteps between their starts (the free sets grow by a timestep or
# two on each side: gaps stay wide enough to pin every run), tolerance
CASES = [(40, 2, 1, 7, 1e-12), (2049, 3, 40, 80, 1e-12), (5000, 3, 400, 500, 1e-12), (60_000, 3, 30, 47, 1e-12),
         (90_000, 8, 20, 50, 1e-12), (300_000, 8, 45, 50, 1e-10)]


@pytest.mark.parametrize("T,K,run,step,tol", CASES)
def test_cg_over_active_timesteps(gpulib, oracle, T, K, run, step, tol):
    rng = np.random.default_rng(T + K)
    eps2 = 200.0
    t = np.arange(T)
    on = (t % step) < run
    on[-1] = False  # no cluster is free at every timestep
    g = np.zeros((T, K))
    g[t, (t // step) % K] = 1.0
    mix = rng.random((T, K)) + 0.5
    g[on] = mix[on] / mix[on].sum(1, keepdims=True)
    x = g.astype(np.float32).astype(np.float64).ravel()
    theta = np.linspace(0.0, 1.0, K)
    data = theta[(t // step) % K] + 0.1 * rng.standard_normal(T)
    dg = rng.standard_normal(T * K) / T
    deps_o, dX_o, dth_o, _, r = oracle.adjoint(x, data, theta, dg, T, K, eps2, cg_tol=tol)
    assert r.status == 1 and r.free_dims > 0
    with Problem(T, K, eps2, PASC_PREC_MIXED) as p:
        p.set_data(data)
        p.set_theta(theta)
        p.set_gamma(x)
        deps, dX, dth, st = p.adjoint(dg, opts=capi.adjoint_opts(cg_tol=tol))
        assert st.status == 1 and st.free_dims == r.free_dims
        assert _rel(deps, deps_o) <= 1e-5 and _rel(dX, dX_o) <= 1e-5 and _rel(dth, dth_o) <= 1e-5
        # the same handle with another epssqr: nothing of the first solve's operator is kept
        p.set_epssqr(2.0 * eps2)
        deps2, dX2, _, st2 = p.adjoint(dg, opts=capi.adjoint_opts(cg_tol=tol))
    d2, x2, _, _, r2 = oracle.adjoint(x, data, theta, dg, T, K, 2.0 * eps2, cg_tol=tol)
    assert st2.status == 1 and r2.status == 1
    assert _rel(deps2, d2) <= 1e-5 and _rel(dX2, x2) <= 1e-5
