"""The fused Gauss-Newton iteration with single-precision Jacobian terms over
latent sizes, against the assembled path in double: one iteration of one step.
The terms carry about 40 operations of 6e-8 each, 2.4e-6 of JR, and a least
squares step is off by at most twice the condition of JR (below 100: random
directions over 270 sample dofs) times that, 5e-4 of the correction; a lost or
doubled pair of the solve changes it by more than 1e-2."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("k", [2, 12, 24, 32])
def test_single_precision_terms_over_latent_sizes(pda, k):
    import torch
    n = 20
    full = pda.create_full_mesh((n, n), (-5, 5, -5, 5), 7)
    rng = np.random.default_rng(300 + k)
    gids = np.sort(rng.choice(n * n, 90, replace=False))
    sm, st = pda.create_sample_mesh(full, gids)
    weno5 = pda.InviscidFluxReconstruction.Weno5
    ps, pf = (pda.create_problem(m, pda.Swe2d(0), weno5, 1) for m in (sm, full))
    u0 = pf.initialCondition().cpu().numpy().reshape(-1, 3)[st].reshape(-1)
    phi, _ = np.linalg.qr(rng.normal(0, 1, (u0.size, k)))
    x0 = rng.normal(0, 0.05, k)
    out = []
    for fused in (True, False):
        rom = pda.LspgRom.affine(ps, np.searchsorted(st, gids), torch.from_numpy(u0).cuda(),
                                 torch.from_numpy(phi).cuda())
        rom.set_fused(fused)
        if fused:
            rom.set_jacobian_precision(32)
        x = torch.from_numpy(x0.copy()).cuda()
        rom.advance_bdf1(x, 0.05, 1, gn_iters=1, tol=0.0, use_graph=fused)
        out.append(x.cpu().numpy())
    moved = np.linalg.norm(out[1] - x0)
    assert moved > 0 and 0 < np.linalg.norm(out[0] - out[1]) <= 5e-4 * moved, out
