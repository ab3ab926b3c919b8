"""Velocity of 1D rows that follow one another, whose blocks form each face
between their rows once: meshes where the last block holds one row, is one row
short, or where the block grows to two warps a side, with and without boundary
rows beside them, and sample meshes with gaps, whose rows keep their own faces.
Equal to the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("n,rows", [(7, None), (15, None), (16, None), (24, None), (25, None), (1520, None),
                                    (1700, None), (3046, None), (3065, None), (60, (20, 30)), (60, (3, 9, 11, 40))])
def test_chained_rows(pda, oracle, tmp_path, n, rows, scheme, periodic):
    import torch
    mesh = pda.create_full_mesh((n,), (0.0, 1.0), 2 * scheme + 3, (periodic,) * 3)
    if rows is not None:
        gids = np.arange(*rows) if len(rows) == 2 else np.array(rows)
        mesh, _ = pda.create_sample_mesh(mesh, gids)
    mesh.write(str(tmp_path / "m"))
    om = oracle.mesh_load(str(tmp_path / "m"))
    if periodic:
        p, o = pda.create_problem(mesh, pda.Euler1d.PeriodicSmooth, scheme), oracle.problem(om, 0, 0, scheme, 1)
    else:
        p, o = pda.create_problem(mesh, pda.Euler1d.Sod, scheme), oracle.problem(om, 0, 1, scheme, 1)
    rng = np.random.default_rng(n)
    cells = p.totalDofStencilMesh() // 3
    u = 0.3 * rng.standard_normal((cells, 3))
    u[:, 0] = 1.0 + 0.1 * rng.random(cells)
    u[:, 2] = 5.0 + rng.random(cells)
    u[::7, 1] = 0.0
    V = p.createVelocity()
    p.velocity(torch.from_numpy(u.reshape(-1)).cuda(), 0.0, V)
    assert np.array_equal(V.cpu().numpy(), o.velocity(u.reshape(-1)))
