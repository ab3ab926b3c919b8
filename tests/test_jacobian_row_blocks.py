"""V and J of row sets (sample meshes) where the row kernel's split changes: the
last block's rows (one row, one below and above the rows of a block) and rows
whose neighbours repeat on periodic meshes shorter than the stencil, which take
the ordered sums instead of a thread per entry.  V, the CSR pattern and the
values equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("euler1d", 2, (40,), k) for k in (1, 9, 10, 11)] + [("euler1d", 2, (n,), n) for n in (4, 5, 6, 7)] + \
        [("euler1d", 1, (3,), 3)] + \
        [("euler2d", 2, (12, 9), k) for k in (1, 3, 4, 5)] + [("euler2d", 2, s, s[0] * s[1]) for s in ((5, 9), (9, 6), (4, 4))] + \
        [("euler2d", 1, (4, 7), 28), ("euler3d", 1, (4, 5, 6), 50), ("euler3d", 2, (7, 8, 6), 9)]


@pytest.mark.parametrize("family,scheme,shape,rows", CASES)
def test_row_blocks(pda, oracle, tmp_path, family, scheme, shape, rows):
    import torch
    full = pda.create_full_mesh(shape, [0.0, 1.0] * len(shape), 2 * scheme + 3, (True,) * 3)
    n = int(np.prod(shape))
    rng = np.random.default_rng(rows)
    mesh, _ = pda.create_sample_mesh(full, np.sort(rng.choice(n, rows, replace=False)))
    mesh.write(str(tmp_path / "m"))
    om = oracle.mesh_load(str(tmp_path / "m"))
    enum = {"euler1d": pda.Euler1d.PeriodicSmooth, "euler2d": pda.Euler2d.PeriodicSmooth,
            "euler3d": pda.Euler3d.PeriodicSmooth}[family]
    nd = len(shape) + 2
    p, o = pda.create_problem(mesh, enum, scheme), oracle.problem(om, len(shape) - 1, 0, scheme, 1)
    cells = p.totalDofStencilMesh() // nd
    u = 0.3 * rng.standard_normal((cells, nd))
    u[:, 0] = 1.0 + 0.1 * rng.random(cells)
    u[:, -1] = 5.0 + rng.random(cells)
    V, J = p.createVelocity(), p.createJacobian()
    p.rightHandSideAndJacobian(torch.from_numpy(u.reshape(-1)).cuda(), 0.0, V, J)
    oracle.set_cube_mode(1)
    try:
        vo, rp, ci, jo = o.velocity_and_jacobian(u.reshape(-1))
    finally:
        oracle.set_cube_mode(0)
    assert np.array_equal(J.rowptr.cpu().numpy(), rp) and np.array_equal(J.colidx.cpu().numpy(), ci)
    assert np.array_equal(V.cpu().numpy(), vo)
    assert np.array_equal(J.values.cpu().numpy(), jo)
