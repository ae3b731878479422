"""Device memory of a mixed problem's adjoint: the vectors of the path it takes and no others.

Per entry (T K of them) gamma, dl/dgamma, lambda and the residual in FP64 and three FP32 vectors, 44
bytes; per timestep mask, list, clean signal and dl/dx, 24.  Where the active timesteps do not fit the
cooperative solve two FP32 vectors more, 8 bytes per entry.  Other allocations (partial sums, words,
tables) and the allocator's granularity of 2 MB for each of about a dozen: below 32 MB."""
import numpy as np
import pytest

from pasc_inference_gb300 import PASC_PREC_MIXED, Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run,extra", [(2, 0), (45, 8)])
def test_adjoint_memory(gpulib, run, extra):
    torch = pytest.importorskip("torch")
    T, K = 2_000_000, 4
    rng = np.random.default_rng(1)
    t = np.arange(T)
    on = (t % 50) < run
    on[-1] = False
    g = np.zeros((T, K))
    g[t, (t // 50) % K] = 1.0
    g[on] = 1.0 / K
    theta = np.linspace(0.0, 1.0, K)
    with Problem(T, K, 200.0, PASC_PREC_MIXED) as p:
        p.set_data(theta[(t // 50) % K] + 0.1 * rng.standard_normal(T))
        p.set_theta(theta)
        p.set_gamma(g.ravel())
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        p.adjoint(rng.standard_normal(T * K) / T)
        used = before - torch.cuda.mem_get_info()[0]
        lower, slack = (44 + extra) * T * K + 24 * T, 32 << 20
        assert lower <= used <= lower + slack, (used, lower)
