"""Lead decimation at the sizes where its LU panels change width: last panels of up to 8 columns, of up to half
the panel and wider, for 32-wide (n <= 256) and 16-wide panels."""
import numpy as np
import pytest
import torch

from oracle import lead_oracle

pytestmark = pytest.mark.gpu
RTOL = 1e-9  # as for the other decimation tests; the leads below converge in about ten well-conditioned steps


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 40, 41, 48, 49, 57, 264, 265, 273])
def test_decimation_matches_oracle(n):
    from dpnegf_b200.surface_green import LeadArena, LeadBlocks, self_energies
    rng = np.random.default_rng(n)
    c = lambda s: (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) * s / np.sqrt(n)
    herm = lambda x: (x + x.conj().T) / 2
    h, h01 = herm(c(0.5)) + np.diag(rng.uniform(-2, 2, n)), c(0.4)
    s, s01 = np.eye(n) + herm(c(0.02)), c(0.01)
    hdl, sdl = c(0.4), c(0.01)
    t = lambda x: torch.as_tensor(x, dtype=torch.complex128, device="cuda")
    arena = LeadArena([LeadBlocks(*map(t, (h, h01, s, s01, hdl, sdl)))])
    E, eta = np.array([-0.6, 0.1, 0.8]), 0.05
    res = self_energies(arena, [0] * 3, E, eta, want_gs=True)
    for k, e in enumerate(E):
        sig, gs, st, it = lead_oracle.self_energy(h, h01, s, s01, e, hdl, sdl, etaLead=eta)
        assert st == lead_oracle.LS_OK and res.status[k] == 0 and abs(int(res.iters[k]) - it) <= 1
        for got, want in ((res.gs[k], gs), (res.sigma[k], sig)):
            assert np.abs(got.cpu().numpy() - want).max() <= RTOL * np.abs(want).max(), (n, e)
