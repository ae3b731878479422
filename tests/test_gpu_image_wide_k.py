"""The image sweep with five to eight clusters, whose pixels are moved 8 or 16 bytes at a time (even
K) or written through shared memory (odd K): widths around the 29 owned columns of a strip and its
32 lanes, heights around its rows, border strips and inner ones, against the general graph sweep.

The bounds of test_gpu_image_tiles: after five iterations the objectives agree within 2e-6 (FP32 state)
and gamma within 1e-5 (2-norm).  Nothing outside the image's own pixels is written: a second problem's
gamma, allocated beside the first one's buffers, stays bit for bit what it was."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, BGMGraphGrid2D, Problem, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2, 3), (27, 4), (29, 9), (30, 2), (31, 5), (32, 33), (33, 3), (57, 8), (60, 31), (89, 64), (640, 211)])
@pytest.mark.parametrize("K", [5, 6, 7, 8])
def test_image_wide_pixels(gpulib, W, H, K):
    rng = np.random.default_rng(W * 1000 + H * 10 + K)
    img = rng.integers(0, K, W * H) + 0.4 * rng.standard_normal(W * H)
    x0 = rng.random(W * H * K)
    grid = BGMGraphGrid2D(W, H)
    grid.process_grid()
    res = []
    with Problem(1, K, 2.0, PASC_PREC_MIXED, graph=grid) as beside:
        beside.set_gamma(x0)
        kept = beside.get_gamma()
        for variant in (1, 0):
            with Problem(1, K, 2.0, PASC_PREC_MIXED, graph=grid) as p:
                p.set_sweep_variant(variant)
                p.set_data(img)
                p.set_gamma(x0)
                p.set_theta(np.arange(K) + 0.0)
                st = p.spgqp_solve(capi.spgqp_opts(maxit=5, m=10, eps=0.0))
                res.append((st.it, st.fx, p.get_gamma()))
        np.testing.assert_array_equal(beside.get_gamma(), kept)
    (it1, f1, g1), (it0, f0, g0) = res
    assert it1 == it0 == 5
    assert abs(f1 - f0) <= 2e-6 * max(abs(f0), 1e-9)
    assert np.linalg.norm(g1 - g0) <= 1e-5 * np.linalg.norm(g0)
