"""The normal equations' solve inside the fused Gauss-Newton iteration, over the
latent sizes where its split over the block changes: fewer pairs of the augmented
triangle than a warp, fewer than the block has threads, and more (24 and 32
columns).  The assembled path solves them by its own
kernel, so the two latent trajectories agree to rounding: the JR^T JR of random
directions over 270 sample dofs has a condition below 1e4, so sums of 270 terms
leave 270 * 1.1e-16 * 1e4 = 3e-10 relative at most; a lost or doubled pair
changes the step by far more."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("k", [2, 6, 12, 20, 24, 32])
def test_fused_iteration_over_latent_sizes(pda, k):
    import torch
    n = 20
    full = pda.create_full_mesh((n, n), (-5, 5, -5, 5), 7)
    rng = np.random.default_rng(100 + k)
    gids = np.sort(rng.choice(n * n, 90, replace=False))
    sm, st = pda.create_sample_mesh(full, gids)
    params = {"gravity": 7.0, "coriolis": -2.0, "pulseMagnitude": 0.15}
    weno5 = pda.InviscidFluxReconstruction.Weno5
    ps = pda.create_problem(sm, pda.Swe2d(0), weno5, 1, params)
    pf = pda.create_problem(full, pda.Swe2d(0), weno5, 1, params)
    u0 = pf.initialCondition().cpu().numpy().reshape(-1, 3)[st].reshape(-1)
    phi, _ = np.linalg.qr(rng.normal(0, 1, (u0.size, k)))
    x0 = rng.normal(0, 0.05, k)
    out = []
    for fused in (True, False):
        rom = pda.LspgRom.affine(ps, np.searchsorted(st, gids), torch.from_numpy(u0).cuda(),
                                 torch.from_numpy(phi).cuda())
        rom.set_fused(fused)
        x = torch.from_numpy(x0.copy()).cuda()
        rom.advance_bdf1(x, 0.002, 3, gn_iters=3, tol=0.0, use_graph=fused)
        out.append(x.cpu().numpy())
    assert np.all(np.isfinite(out[0]))
    assert np.linalg.norm(out[0] - out[1]) <= 3e-10 * np.linalg.norm(out[1]), out
