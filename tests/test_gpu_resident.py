"""The resident solve (one cooperative launch, state in shared memory; taken when the kernel is
left to the library and the state fits) at the edges of its plan: one block and several, short
last blocks, rows of one to many timesteps per thread, the largest signal that fits.

Against the FP64 oracle the objective after 0 and 3 iterations is held to 2e-6 relative, the bound
of the other sweeps' trajectories (FP32 state).  Against the pinned bulk-copy sweep, which does the
same FP32 arithmetic per entry and differs only in the grouping of the sums: a sum differs by at
most a few FP32 ulps of its terms (1e-6 relative), which moves the step lengths by as much; after
three steps gamma is held to 1e-5 (2-norm).  A solve cut into start and iterate calls recomputes its
direction from the stored gamma with the same arithmetic: equal bit for bit."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, Problem, capi

pytestmark = pytest.mark.gpu


def _inputs(T, K, xdim, seed):
    rng = np.random.default_rng(seed)
    data = rng.integers(0, K, T).astype(float)[:, None] + 0.5 * rng.standard_normal((T, xdim))
    return data.ravel(), np.repeat(np.arange(K) + 0.5, xdim), rng.random(T * K)


def _problem(T, K, mode, data, theta, x0, variant):
    p = Problem(T, K, 10.0, PASC_PREC_MIXED, xdim=2 if mode == 1 else 1)
    p.set_data(data)
    p.set_gamma(x0)
    if mode == 2:
        p.set_usethetainpenalty(True)
    p.set_theta(theta)
    p.set_sweep_variant(variant)
    return p


SIZES = {1: [5, 4096, 4097], 2: [7, 2049, 4097, 77823], 3: [1024, 2047, 2048, 2049, 77825], 4: [2561],
         5: [2048, 3000, 123457], 6: [1023, 1025], 7: [1024, 1537], 8: [6, 1024, 1025, 58369]}


@pytest.mark.parametrize("K", sorted(SIZES))
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_resident_edges(gpulib, oracle, K, mode):
    for T in SIZES[K]:
        data, theta, x0 = _inputs(T, K, 2 if mode == 1 else 1, 100 * K + T)
        opts = capi.spgqp_opts(maxit=3, m=10, eps=0.0)
        with _problem(T, K, mode, data, theta, x0, -1) as p:
            st = p.spgqp_solve(opts)
            g = p.get_gamma()
            p.set_gamma(x0)
            p.spgqp_start(opts)
            p.spgqp_iterate(1)
            st2 = p.spgqp_iterate(2)
            assert st.it == st2.it and st.fx == st2.fx
            np.testing.assert_array_equal(p.get_gamma(), g)
        with _problem(T, K, mode, data, theta, x0, 1) as p:
            st1 = p.spgqp_solve(opts)
            g1 = p.get_gamma()
        # (one cluster: gamma is 1 everywhere and the solve ends at once)
        assert st.it == st1.it == (3 if K > 1 else 0) and abs(st.fx - st1.fx) <= 2e-6 * abs(st1.fx), (T, st.fx, st1.fx)
        assert np.linalg.norm(g - g1) <= 1e-5 * np.linalg.norm(g1), T
        if mode == 0:
            x0r = x0.astype(np.float32).astype(np.float64)
            _, ro, _ = oracle.spgqp_solve(oracle.residual_b(data, theta, T, K), x0r, T, K, oracle.A_coeff(10.0, T),
                                          oracle.spg_opts(maxit=3, m=10))
            assert abs(st.fx - ro.fx) <= 2e-6 * abs(ro.fx), (T, st.fx, ro.fx)


@pytest.mark.parametrize("T,K", [(1_150_000, 3), (1_160_001, 3), (1_300_000, 3), (470_000, 8)])
def test_resident_at_the_limit_of_shared_memory(gpulib, T, K):
    data, theta, x0 = _inputs(T, K, 1, T)
    opts = capi.spgqp_opts(maxit=3, m=10, eps=0.0)
    res = []
    for variant in (-1, 1):
        with _problem(T, K, 0, data, theta, x0, variant) as p:
            st = p.spgqp_solve(opts)
            res.append((st.it, st.fx, p.get_gamma()))
    assert res[0][0] == res[1][0] == 3
    assert abs(res[0][1] - res[1][1]) <= 2e-6 * abs(res[1][1])
    assert np.linalg.norm(res[0][2] - res[1][2]) <= 1e-5 * np.linalg.norm(res[1][2])


def test_resident_solves_on_two_handles_at_once(gpulib):
    """Two handles driven from two threads: each solve gives what it gives alone."""
    import threading
    T, K = 200_001, 3
    opts = capi.spgqp_opts(maxit=30, m=10, eps=0.0)
    ins = [_inputs(T, K, 1, s) for s in (1, 2)]
    ps = [_problem(T, K, 0, *i, -1) for i in ins]
    want = []
    for p in ps:
        p.spgqp_solve(opts)
        want.append(p.get_gamma())
    got = [None, None]

    def work(n):
        for _ in range(10):
            ps[n].set_gamma(ins[n][2])
            ps[n].spgqp_solve(opts)
        got[n] = ps[n].get_gamma()
    th = [threading.Thread(target=work, args=(n,)) for n in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for n in (0, 1):
        np.testing.assert_array_equal(got[n], want[n])
        ps[n].close()
