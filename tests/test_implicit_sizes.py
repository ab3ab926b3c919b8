"""The linear solver's one-launch form over its ranges: one block with fewer
rows than lanes, odd row counts, one block per SM, and several rounds of rows
per block.  Tight tolerances, so that the state is the discrete solution,
which a host Newton with direct solves on the oracle's V and J also reaches
(1e-9, as in the other implicit test)."""
import numpy as np
import pytest

from test_implicit import _host_newton

pytestmark = pytest.mark.gpu

CASES = [("euler1d", 0, (5,)), ("euler1d", 1, (23,)), ("euler2d", 1, (9, 7)), ("swe2d", 2, (41, 33)),
         ("euler2d", 0, (150, 140))]


@pytest.mark.parametrize("family,scheme,shape", CASES)
def test_row_counts(pda, oracle, tmp_path, family, scheme, shape):
    import torch
    mesh = pda.create_full_mesh(shape, [0.0, 1.0] * len(shape), 2 * scheme + 3)
    mesh.write(str(tmp_path / "m"))
    om = oracle.mesh_load(str(tmp_path / "m"))
    enum, fam, prob, ic = {"euler1d": (pda.Euler1d.Sod, 0, 1, 1), "euler2d": (pda.Euler2d.Riemann, 1, 4, 2),
                           "swe2d": (pda.Swe2d.SlipWall, 3, 0, 1)}[family]
    p, o = pda.create_problem(mesh, enum, scheme, ic), oracle.problem(om, fam, prob, scheme, ic)
    n = int(np.prod(shape))
    u = o.initial_condition() * (1 + 0.01 * np.random.default_rng(5).random(n * p.numDofPerCell()))
    dt = 0.2 / max(shape)
    want = _host_newton(o, u, dt, 1, "cn", tol=1e-12)
    U = torch.from_numpy(u.copy()).cuda()
    for _ in range(2):  # a second call on the kept buffers
        U.copy_(torch.from_numpy(u))
        info = p.advance_implicit(U, 0.0, dt, 1, scheme="cn", newton_tol=1e-11, linear_tol=1e-13,
                                  linear_max_iters=5000)
        assert np.allclose(U.cpu().numpy(), want, rtol=1e-9, atol=1e-11)
        assert info["linear_iters"] > 0
