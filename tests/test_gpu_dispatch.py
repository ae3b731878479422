"""Which path a solve took, by its kernel launches: the cooperative launches where their plans apply,
and the ordinary kernels where they do not.  (Both give the same results, so no other test tells a plan
that stopped applying.)"""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_FP64, PASC_PREC_MIXED, Problem, capi

pytestmark = pytest.mark.gpu


def _problem(T, K, prec, xdim=1):
    rng = np.random.default_rng(T + K)
    p = Problem(T, K, 10.0, prec, xdim=xdim)
    p.set_data((rng.integers(0, K, T)[:, None] + 0.5 * rng.standard_normal((T, xdim))).ravel())
    p.set_gamma(rng.random(T * K))
    p.set_theta(np.repeat(np.arange(K) + 0.5, xdim))
    p.update_b()
    return p


@pytest.mark.parametrize("T,K,fits", [(5, 2, True), (4097, 2, True), (77_825, 3, True), (1_150_000, 3, True),
                                      (1_300_000, 3, False), (58_369, 8, True), (470_000, 8, True), (600_000, 8, False)])
@pytest.mark.parametrize("form", ["data", "b", "penalty"])
def test_mixed_solve(gpulib, T, K, fits, form):
    if form == "b" and T > 100_000 and fits:
        T = T * 2 // 3  # (b takes K values per timestep of the shared memory, the data one)
    opts = capi.spgqp_opts(maxit=20, m=10, eps=0.0)
    with _problem(T, K, PASC_PREC_MIXED, 2 if form == "b" else 1) as p:
        if form == "penalty":
            p.set_usethetainpenalty(True)
        st = p.spgqp_solve(opts)
        assert st.it == 20
        assert (st.kernel_launches == 1) == fits, st.kernel_launches
        assert fits or st.kernel_launches >= 21
        for variant in (0, 1):  # a pinned kernel is taken as it is
            p.set_sweep_variant(variant)
            assert p.spgqp_solve(opts).kernel_launches >= 21


@pytest.mark.parametrize("T,K,fused", [(5, 2, True), (300, 8, True), (60_000, 3, True), (300_000, 5, True), (300, 9, False)])
def test_fp64_solve(gpulib, T, K, fused):
    with _problem(T, K, PASC_PREC_FP64) as p:
        st = p.spgqp_solve(capi.spgqp_opts(maxit=10, m=10, eps=0.0))
        assert st.it == 10
        assert st.kernel_launches <= 4 if fused else st.kernel_launches >= 80


@pytest.mark.parametrize("T,K,run,step,tol,fits", [(2049, 3, 40, 80, 1e-12, True), (90_000, 8, 20, 50, 1e-12, True),
                                                   (300_000, 8, 45, 50, 1e-10, False)])
def test_adjoint(gpulib, T, K, run, step, tol, fits):
    rng = np.random.default_rng(T + K)
    t = np.arange(T)
    on = (t % step) < run
    on[-1] = False
    g = np.zeros((T, K))
    g[t, (t // step) % K] = 1.0
    mix = rng.random((T, K)) + 0.5
    g[on] = mix[on] / mix[on].sum(1, keepdims=True)
    theta = np.linspace(0.0, 1.0, K)
    with Problem(T, K, 200.0, PASC_PREC_MIXED) as p:
        p.set_data(theta[(t // step) % K] + 0.1 * rng.standard_normal(T))
        p.set_theta(theta)
        p.set_gamma(g.astype(np.float32).astype(np.float64).ravel())
        st = p.adjoint(rng.standard_normal(T * K) / T, opts=capi.adjoint_opts(cg_tol=tol))[3]
    assert st.status == 1 and st.cg_it > 40
    assert (st.kernel_launches < st.cg_it) if fits else (st.kernel_launches >= 2 * st.cg_it)
