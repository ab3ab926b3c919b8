"""The forms of the face tile kernels at the sizes where they end: a warp per dof
(small meshes) with one face more or less than its tiles hold, and the narrow
and wide tiles of larger meshes, on ordinary states and on states whose products
leave the integer pipe's operand window.  The velocity equals the oracle's bit
for bit (the shallow-water flux to 1e-13, as elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("euler2d", 2, (n, 9)) for n in (7, 27, 28, 29, 57)] + [("euler2d", 1, (9, n)) for n in (28, 29, 30, 60)] + \
        [("swe2d", 2, (28, 57)), ("swe2d", 1, (59, 30))] + \
        [("euler3d", 2, (28, 7, 8)), ("euler3d", 1, (7, 30, 6)), ("euler3d", 2, (8, 7, 29))] + \
        [("euler2d", 2, (256, 250)), ("euler2d", 1, (301, 256)), ("swe2d", 2, (300, 256))]


@pytest.mark.parametrize("kind", ["ordinary", "mixed"])
@pytest.mark.parametrize("family,scheme,shape", CASES)
def test_face_tile_forms(pda, oracle, tmp_path, family, scheme, shape, kind):
    import torch
    euler, three = family != "swe2d", family == "euler3d"
    mesh = pda.create_full_mesh(shape, [0.0, 1.0] * len(shape), 2 * scheme + 3, (three,) * 3)
    mesh.write(str(tmp_path / "m"))
    om = oracle.mesh_load(str(tmp_path / "m"))
    if three:
        p, o = pda.create_problem(mesh, pda.Euler3d.PeriodicSmooth, scheme), oracle.problem(om, 2, 0, scheme, 1)
    elif euler:
        p, o = pda.create_problem(mesh, pda.Euler2d.Riemann, scheme, 2), oracle.problem(om, 1, 4, scheme, 2)
    else:
        p, o = pda.create_problem(mesh, pda.Swe2d.SlipWall, scheme, 1), oracle.problem(om, 3, 0, scheme, 1)
    rng = np.random.default_rng(21)
    n, nd = int(np.prod(shape)), {"euler2d": 4, "euler3d": 5, "swe2d": 3}[family]
    u = 0.3 * rng.standard_normal((n, nd))
    u[:, 0] = 1.0 + 0.1 * rng.random(n)
    if euler:
        u[:, -1] = 5.0 + rng.random(n)
    if kind == "mixed":  # at rest, uniform, and scaled far up and down in bands of cells
        band = (np.arange(n) // 5) % 8
        u[band == 1, 1:-1 if euler else nd] = 0.0
        u[band == 3] = u[0]
        u[band == 5] *= 1e-85
        u[band == 7] *= 1e85
    V = p.createVelocity()
    p.velocity(torch.from_numpy(u.reshape(-1)).cuda(), 0.0, V)
    got, want = V.cpu().numpy(), o.velocity(u.reshape(-1))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fine = np.isfinite(want)
    assert np.array_equal(got[~fine & ~np.isnan(want)], want[~fine & ~np.isnan(want)])
    if euler:
        assert np.array_equal(got[fine], want[fine])
    else:
        scale = np.maximum(np.abs(want[fine]), 1e-3 * np.abs(want[fine]).max())
        assert np.all(np.abs(got[fine] - want[fine]) <= 1e-13 * scale)
