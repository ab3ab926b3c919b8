"""Explicit steps by graphs of one and of several steps, and by launches: the
same states bit for bit, for step counts around the lengths where the graphs
change, a first call and a repeated one, and a changed step size."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ssprk3", "rk4"])
@pytest.mark.parametrize("problem", ["sod1d", "smooth1d", "swe2d", "sedov2d"])
def test_graphs_equal_launches(pda, problem, kind):
    import torch
    s = torch.cuda.Stream()
    if problem == "sod1d":
        mesh = pda.create_full_mesh((60,), (-0.5, 0.5), 7)
        p = pda.create_problem(mesh, pda.Euler1d.Sod, 2, stream=s)
    elif problem == "smooth1d":  # periodic: structured faces in one dimension
        mesh = pda.create_full_mesh((300,), (-1.0, 1.0), 7, (True,))
        p = pda.create_problem(mesh, pda.Euler1d.PeriodicSmooth, 2, stream=s)
    elif problem == "swe2d":
        mesh = pda.create_full_mesh((20, 17), (-5.0, 5.0, -5.0, 5.0), 7)
        p = pda.create_problem(mesh, pda.Swe2d.SlipWall, 2, stream=s)
    else:  # structured inner box and near-boundary rows
        mesh = pda.create_full_mesh((24, 21), (0.0, 1.2, 0.0, 1.2), 5)
        p = pda.create_problem(mesh, pda.Euler2d.SedovSymmetry, 1, stream=s)
    advance = getattr(p, "advance_" + kind)
    with torch.cuda.stream(s):
        a, b = p.initialCondition(), p.initialCondition()
    for steps, dt in ((1, 1e-4), (31, 1e-4), (32, 1e-4), (50, 1e-4), (50, 2e-4), (33, 2e-4)):
        advance(a, 0.0, dt, steps)
        advance(b, 0.0, dt, steps, use_graph=False)
        s.synchronize()
        assert torch.equal(a, b), (steps, dt)
    assert not torch.isnan(a).any()
