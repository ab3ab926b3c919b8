"""Face tile kernels on states whose products leave the integer pipe's operand
window (zeros, uniform flow, very small and very large values, and mixtures of
these with ordinary cells): the velocity equals the oracle's bit for bit (the
shallow-water flux to 1e-13, as elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (70, 9)  # more than one tile along x, fewer cells than a tile along y


def _state(kind, nd, euler, rng):
    n = SHAPE[0] * SHAPE[1]
    u = np.empty((n, nd))
    u[:, 0] = 1.0 + 0.1 * rng.random(n)
    u[:, 1:] = 0.3 * rng.standard_normal((n, nd - 1))
    if euler:
        u[:, -1] = 5.0 + rng.random(n)
    pick = rng.random(n) < 0.5
    if kind == "zeros":  # one momentum zero everywhere, the other in half of the cells
        u[:, 1] = 0.0
        u[pick, 2] = 0.0
    elif kind == "uniform":
        u[:] = u[0]
        u[:, 1] = 0.0
    elif kind == "small":
        u[pick] *= 1e-85
    elif kind == "large":
        u[pick] *= 1e85
    return u.reshape(-1)


@pytest.mark.parametrize("kind", ["zeros", "uniform", "small", "large"])
@pytest.mark.parametrize("scheme", [1, 2])
@pytest.mark.parametrize("family", ["euler2d", "swe2d"])
def test_velocity_outside_the_operand_window(pda, oracle, tmp_path, family, scheme, kind):
    import torch
    euler = family == "euler2d"
    mesh = pda.create_full_mesh(SHAPE, (0.0, 1.0, 0.0, 1.0), 7)
    mesh.write(str(tmp_path / "m"))
    om = oracle.mesh_load(str(tmp_path / "m"))
    if euler:
        p = pda.create_problem(mesh, pda.Euler2d.Riemann, scheme, 2)
        o = oracle.problem(om, 1, 4, scheme, 2)
    else:
        p = pda.create_problem(mesh, pda.Swe2d.SlipWall, scheme, 1)
        o = oracle.problem(om, 3, 0, scheme, 1)
    u = _state(kind, 4 if euler else 3, euler, np.random.default_rng(11))
    V = p.createVelocity()
    p.velocity(torch.from_numpy(u).cuda(), 0.0, V)
    got, want = V.cpu().numpy(), o.velocity(u)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fine = np.isfinite(want)
    assert np.array_equal(got[~fine & ~np.isnan(want)], want[~fine & ~np.isnan(want)])
    if euler:
        assert np.array_equal(got[fine], want[fine])
    else:
        # a cell's terms cancel: relative to the largest flux difference of the cell's neighbourhood
        scale = np.maximum(np.abs(want[fine]), 1e-3 * np.abs(want[fine]).max())
        assert np.all(np.abs(got[fine] - want[fine]) <= 1e-13 * scale)
