"""Cooperative launches from several handles and in several launches: FP64 solves and adjoints driven
from two threads at once give what they give alone, bit for bit, and a mixed solve of more iterations
than one launch makes goes on in the next one as if nothing had happened."""
import threading

import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_FP64, PASC_PREC_MIXED, Problem, capi

pytestmark = pytest.mark.gpu


def _both(work):
    """work(n) for n = 0, 1, alone and then at the same time from two threads."""
    want = [work(n) for n in (0, 1)]
    got, errors = [None, None], []

    def run(n):
        try:
            for _ in range(8):
                got[n] = work(n)
        except Exception as e:  # reported by the test's thread
            errors.append(e)

    th = [threading.Thread(target=run, args=(n,)) for n in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    for n in (0, 1):
        for a, b in zip(got[n], want[n]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("T,K", [(9000, 2), (250_000, 3)])
def test_fp64_solves_on_two_handles_at_once(gpulib, T, K):
    ps, x0 = [], []
    for n in (0, 1):
        rng = np.random.default_rng(n)
        p = Problem(T, K, 10.0, PASC_PREC_FP64)
        p.set_data(rng.integers(0, K, T) + 0.5 * rng.standard_normal(T))
        p.set_theta(np.arange(K) + 0.5)
        x0.append(rng.random(T * K))
        p.set_gamma(x0[n])
        p.update_b()
        ps.append(p)

    def work(n):
        ps[n].set_gamma(x0[n])
        st = ps[n].spgqp_solve(capi.spgqp_opts(maxit=15, m=10, eps=0.0))
        return st.fx, ps[n].get_gamma()

    _both(work)
    for p in ps:
        p.close()


def test_adjoints_on_two_handles_at_once(gpulib):
    T, K = 40_000, 3
    t = np.arange(T)
    ps, dg = [], []
    for n in (0, 1):
        rng = np.random.default_rng(n)
        on = (t % 80) < 30 + 20 * n
        on[-1] = False
        g = np.zeros((T, K))
        g[t, (t // 80) % K] = 1.0
        mix = rng.random((T, K)) + 0.5
        g[on] = mix[on] / mix[on].sum(1, keepdims=True)
        theta = np.linspace(0.0, 1.0, K)
        p = Problem(T, K, 200.0, PASC_PREC_MIXED)
        p.set_data(theta[(t // 80) % K] + 0.1 * rng.standard_normal(T))
        p.set_theta(theta)
        p.set_gamma(g.astype(np.float32).astype(np.float64).ravel())
        dg.append(rng.standard_normal(T * K) / T)
        ps.append(p)
    _both(lambda n: ps[n].adjoint(dg[n], opts=capi.adjoint_opts(cg_tol=1e-10))[:3])
    for p in ps:
        p.close()


def test_solve_of_more_iterations_than_a_launch_makes(gpulib):
    T, K, n = 3000, 3, 6000  # 4096 sweeps a launch
    rng = np.random.default_rng(3)
    x0 = rng.random(T * K)
    opts = capi.spgqp_opts(maxit=n, m=10, eps=0.0, stop_difff=0)
    with Problem(T, K, 2000.0, PASC_PREC_MIXED) as p:
        p.set_data(np.repeat(rng.integers(0, K, T // 100), 100) + 0.5 * rng.standard_normal(T))
        p.set_theta(np.arange(K) + 0.1)
        p.set_gamma(x0)
        st = p.spgqp_solve(opts)
        g = p.get_gamma()
        assert st.it > 4096 and st.kernel_launches == 2
        p.set_gamma(x0)
        p.spgqp_start(opts)
        p.spgqp_iterate(1000)
        st2 = p.spgqp_iterate(n)
        assert (st2.it, st2.fx, st2.status) == (st.it, st.fx, st.status)
        np.testing.assert_array_equal(p.get_gamma(), g)
