"""The fused Gauss-Newton iteration on more rows than two blocks per SM hold, where
single-precision terms with few columns take the form with the fluxes on the face
values' own warps (and 12 columns do not): one iteration of one step against the
assembled path in double, 5e-4 of the correction as on small samples (40
operations of 6e-8, twice the condition of JR, below 100)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("family,scheme,k", [("swe2d", 2, 2), ("swe2d", 1, 10), ("swe2d", 2, 12), ("euler2d", 2, 8),
                                             ("euler2d", 0, 4), ("euler1d", 2, 6), ("euler3d", 1, 4)])
def test_many_rows_match_the_assembled_path(pda, family, scheme, k):
    import torch
    shape, bounds, enum, ic = {"swe2d": ((64, 60), (-5.0, 5.0), pda.Swe2d.SlipWall, 1),
                               "euler2d": ((64, 60), (0.0, 1.0), pda.Euler2d.Riemann, 2),
                               "euler1d": ((3500,), (-0.5, 0.5), pda.Euler1d.Sod, 1),
                               "euler3d": ((13, 12, 14), (-1.0, 1.0), pda.Euler3d.PeriodicSmooth, 1)}[family]
    full = pda.create_full_mesh(shape, list(bounds) * len(shape), 2 * scheme + 3, (family == "euler3d",) * 3)
    n = int(np.prod(shape))
    rng = np.random.default_rng(400 + k)
    gids = np.sort(rng.choice(n, n * 9 // 10, replace=False))
    sm, st = pda.create_sample_mesh(full, gids)
    ps, pf = pda.create_problem(sm, enum, scheme, ic), pda.create_problem(full, enum, scheme, ic)
    u0 = pf.initialCondition().cpu().numpy().reshape(-1, pf.numDofPerCell())[st].reshape(-1)
    phi, _ = np.linalg.qr(rng.normal(0, 1, (u0.size, k)))
    x0 = rng.normal(0, 0.02, k)
    out = []
    for fused in (True, False):
        rom = pda.LspgRom.affine(ps, np.searchsorted(st, gids), torch.from_numpy(u0).cuda(),
                                 torch.from_numpy(phi).cuda())
        rom.set_fused(fused)
        if fused:
            rom.set_jacobian_precision(32)
        x = torch.from_numpy(x0.copy()).cuda()
        rom.advance_bdf1(x, 0.05 * (bounds[1] - bounds[0]) / max(shape), 1, gn_iters=1, tol=0.0, use_graph=fused)
        out.append(x.cpu().numpy())
    moved = np.linalg.norm(out[1] - x0)
    assert moved > 0 and 0 < np.linalg.norm(out[0] - out[1]) <= 5e-4 * moved, out
