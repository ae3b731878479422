"""The sums of the mixed path's theta step (FP32 per thread, three FP32 terms per warp, FP64 beyond) at
the edges of its warps, blocks and grid, and at data whose sums leave the FP32 range while theta does
not.

Against 64-bit sums of the same FP32 values.  theta_k = sum gamma x / sum gamma: every product is
rounded once, 2^-24 of itself, which moves theta by at most 2^-24 max|x|; the sums' own errors are
far below.  Bound: 2^-23 max|x|.  With theta in the penalty the denominator has squares of FP32
differences as well, 2^-22 relative, and |theta| <= max|x|: 2^-21 max|x|."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, Problem

pytestmark = pytest.mark.gpu


def _theta(T, K, data, gamma, tp, epssqr=3.0):
    with Problem(T, K, epssqr, PASC_PREC_MIXED) as p:
        p.set_data(data)
        p.set_gamma(gamma)
        if tp:
            p.set_usethetainpenalty(True)
        p.update_theta()
        first = p.get_theta()
        p.update_theta()  # nothing of the first call is left over
        np.testing.assert_array_equal(p.get_theta(), first)
        return first


def _exact(T, K, data, gamma, tp, epssqr=3.0):
    g = gamma.reshape(T, K)
    num, den = g.T @ data, g.sum(0)
    if tp:
        den = den + epssqr / T * (np.diff(g, axis=0) ** 2).sum(0)
    return num / den


@pytest.mark.parametrize("tp", [False, True])
@pytest.mark.parametrize("K", range(1, 9))
def test_theta_sums(gpulib, K, tp):
    for T in (1, 31, 33, 255, 257, 1025, 4097, 155_649, 1_000_003):
        rng = np.random.default_rng(100 * K + T)
        gamma = (rng.random((T, K)) + 0.01).astype(np.float32)
        gamma = (gamma / gamma.sum(1, keepdims=True)).astype(np.float32).astype(np.float64).ravel()
        base = rng.integers(0, K, T) + 0.5 * rng.standard_normal(T)
        # data of order 1; one far from it in a warp of others; and 2^125: 32 of them leave the FP32 range
        spike = base.copy()
        spike[T // 2] = 1e30
        for data in (base, spike, (base / np.abs(base).max()) * 2.0**125):
            data = data.astype(np.float32).astype(np.float64)
            got, want = _theta(T, K, data, gamma, tp), _exact(T, K, data, gamma, tp)
            bound = (2.0**-21 if tp else 2.0**-23) * np.abs(data).max()
            assert np.max(np.abs(got - want)) <= bound, (T, got, want)


def test_theta_of_an_infinite_value_is_not_finite(gpulib):
    T, K = 5000, 2
    data = np.zeros(T)
    data[1234] = np.inf
    got = _theta(T, K, data, np.full(T * K, 0.5), False)
    assert not np.any(np.isfinite(got))
