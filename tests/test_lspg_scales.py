"""The normal equations' solve inside the fused Gauss-Newton iteration over the
scale of the trial space: a basis times 2^e and latent coordinates times 2^-e are
the same states, and the decoder, the residual and its Jacobian are exact in that
factor.  JR^T JR is 2^2e times its usual size; e = +-100 stay within the solve's
usual path, which is exact in the factor too, e = +-300 take the one for extreme
pivots, which rounds differently: k^2 products with a relative error of 1.1e-16
times the condition of JR^T JR, below 1e4 for random directions over 270 sample
dofs, leave 32^2 * 1.1e-16 * 1e4 = 1.1e-9 of the correction at most.  Where the
products of the elimination leave their range instead, the step loses its
digits: 9e-4 of the correction."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("k", [6, 32])
def test_scaled_basis_gives_the_same_states(pda, k):
    import torch
    n = 20
    full = pda.create_full_mesh((n, n), (-5, 5, -5, 5), 7)
    rng = np.random.default_rng(200 + k)
    gids = np.sort(rng.choice(n * n, 90, replace=False))
    sm, st = pda.create_sample_mesh(full, gids)
    weno5 = pda.InviscidFluxReconstruction.Weno5
    ps, pf = (pda.create_problem(m, pda.Swe2d(0), weno5, 1) for m in (sm, full))
    u0 = pf.initialCondition().cpu().numpy().reshape(-1, 3)[st].reshape(-1)
    phi, _ = np.linalg.qr(rng.normal(0, 1, (u0.size, k)))
    x0 = rng.normal(0, 0.05, k)
    states = []
    for e in (0, -100, -300, 100, 300):
        rom = pda.LspgRom.affine(ps, np.searchsorted(st, gids), torch.from_numpy(u0).cuda(),
                                 torch.from_numpy(phi * 2.0 ** e).cuda())
        x = torch.from_numpy(x0 * 2.0 ** -e).cuda()
        rom.advance_bdf1(x, 0.002, 3, gn_iters=2, tol=0.0)
        states.append(rom.decode(x))
        assert torch.isfinite(states[-1]).all()
        moved = torch.linalg.norm(states[0] - torch.from_numpy(u0).cuda())
        off = torch.linalg.norm(states[-1] - states[0])
        assert moved > 0 and off <= (0 if abs(e) <= 100 else 1.1e-9 * moved), (e, off / moved)
