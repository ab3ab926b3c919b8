"""The Jacobian tile kernel where its tiles of 31 cells end, and on states
whose flux Jacobians are not finite (the kernel leaves out products with known
zeros): V, the CSR pattern and the values equal the oracle's bit for bit
(shallow water to the bars of the other tests), NaN for NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("euler2d", 2, (n, 9)) for n in (37, 38, 36, 7, 68)] + [("euler2d", 1, (9, 35)), ("euler2d", 1, (36, 9))] + \
        [("swe2d", 2, (38, 11)), ("swe2d", 1, (11, 35)), ("euler3d", 2, (32, 7, 8)), ("euler3d", 1, (7, 31, 6))]


def _problems(pda, oracle, tmp_path, family, scheme, shape):
    periodic = family == "euler3d"
    mesh = pda.create_full_mesh(shape, [0.0, 1.0] * len(shape), 2 * scheme + 3, (periodic,) * 3)
    mesh.write(str(tmp_path / "m"))
    om = oracle.mesh_load(str(tmp_path / "m"))
    if family == "euler2d":
        return pda.create_problem(mesh, pda.Euler2d.Riemann, scheme, 2), oracle.problem(om, 1, 4, scheme, 2)
    if family == "euler3d":
        return pda.create_problem(mesh, pda.Euler3d.PeriodicSmooth, scheme), oracle.problem(om, 2, 0, scheme, 1)
    return pda.create_problem(mesh, pda.Swe2d.SlipWall, scheme, 1), oracle.problem(om, 3, 0, scheme, 1)


def _state(family, shape, rng):
    n = int(np.prod(shape))
    nd = {"euler2d": 4, "euler3d": 5, "swe2d": 3}[family]
    u = np.empty((n, nd))
    u[:, 0] = 1.0 + 0.1 * rng.random(n)
    u[:, 1:] = 0.3 * rng.standard_normal((n, nd - 1))
    if family != "swe2d":
        u[:, -1] = 5.0 + rng.random(n)
    return u


def _compare(pda, oracle, p, o, u, exact):
    import torch
    V, J = p.createVelocity(), p.createJacobian()
    p.rightHandSideAndJacobian(torch.from_numpy(u.reshape(-1).copy()).cuda(), 0.0, V, J)
    oracle.set_cube_mode(1)
    try:
        vo, rp, ci, jo = o.velocity_and_jacobian(u.reshape(-1))
    finally:
        oracle.set_cube_mode(0)
    assert np.array_equal(J.rowptr.cpu().numpy(), rp) and np.array_equal(J.colidx.cpu().numpy(), ci)
    v, j = V.cpu().numpy(), J.values.cpu().numpy()
    if exact:
        assert np.array_equal(v, vo, equal_nan=True)
        assert np.array_equal(j, jo, equal_nan=True)
        return jo
    scale = np.maximum.reduceat(np.abs(jo), rp[:-1])
    assert np.all(np.abs(j - jo) <= 1e-12 * np.repeat(scale, np.diff(rp)))
    return jo


@pytest.mark.parametrize("family,scheme,shape", CASES)
def test_tile_edges(pda, oracle, tmp_path, family, scheme, shape):
    p, o = _problems(pda, oracle, tmp_path, family, scheme, shape)
    _compare(pda, oracle, p, o, _state(family, shape, np.random.default_rng(3)), family != "swe2d")


@pytest.mark.parametrize("kind", ["pressure", "density", "infinite", "nan", "at_rest"])
@pytest.mark.parametrize("scheme", [1, 2])
def test_states_without_finite_jacobians(pda, oracle, tmp_path, scheme, kind):
    shape = (40, 17)
    p, o = _problems(pda, oracle, tmp_path, "euler2d", scheme, shape)
    u = _state("euler2d", shape, np.random.default_rng(4))
    cells = [8 * 40 + 20, 9 * 40 + 33]
    if kind == "pressure":
        u[cells, 3] = -2.0
    elif kind == "density":
        u[cells, 0] = -1.0
    elif kind == "infinite":
        u[cells, 2] = np.inf
    elif kind == "nan":
        u[cells, 1] = np.nan
    else:
        u[:] = u[0]
        u[:, 1:3] = 0.0
        u[cells, 0] += 0.01
    jo = _compare(pda, oracle, p, o, u, True)
    assert kind == "at_rest" or np.isnan(jo).any()
