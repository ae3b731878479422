"""The fused image sweep at the edges of its strip tiles (29 owned columns, th owned rows chosen from
the size), one warp wide and many, against the general graph sweep on the same image: the same FP32
arithmetic per pixel up to the order of four neighbour differences, sums in another grouping.  After
five iterations the objectives agree within 2e-6 (FP32 state) and gamma within 1e-5 (2-norm)."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, BGMGraphGrid2D, Problem, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2, 2), (3, 70), (28, 5), (29, 6), (30, 7), (31, 64), (58, 63), (59, 66), (87, 3), (300, 201),
                                 (1100, 401)])
@pytest.mark.parametrize("K", [1, 2, 3, 5, 8])
def test_image_strip_edges(gpulib, W, H, K):
    rng = np.random.default_rng(W * 1000 + H * 10 + K)
    img = rng.integers(0, K, W * H) + 0.4 * rng.standard_normal(W * H)
    x0 = rng.random(W * H * K)
    grid = BGMGraphGrid2D(W, H)
    grid.process_grid()
    res = []
    for variant in (1, 0):
        with Problem(1, K, 2.0, PASC_PREC_MIXED, graph=grid) as p:
            p.set_sweep_variant(variant)
            p.set_data(img)
            p.set_gamma(x0)
            p.set_theta(np.arange(K) + 0.0)
            st = p.spgqp_solve(capi.spgqp_opts(maxit=5, m=10, eps=0.0))
            res.append((st.it, st.fx, p.get_gamma()))
    (it1, f1, g1), (it0, f0, g0) = res
    assert it1 == it0
    assert abs(f1 - f0) <= 2e-6 * max(abs(f0), 1e-9)
    assert np.linalg.norm(g1 - g0) <= 1e-5 * np.linalg.norm(g0)
