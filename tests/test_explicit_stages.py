"""SSP-RK3 stages inside the evaluations' kernels against stages composed from
velocity calls, bit for bit: structured faces in 1D (8192 cells and more), alone
and with near-boundary rows in the same stage, and the stage of the batched
balance, on ordinary states and on states whose products leave the integer
pipe's operand window."""
import pytest

pytestmark = pytest.mark.gpu


def _state(torch, problem, kind):
    u = problem.initialCondition()
    nd = problem.numDofPerCell()
    g = torch.Generator(device="cuda").manual_seed(17)
    w = (u * (1 + 1e-2 * torch.rand(u.shape, generator=g, device="cuda", dtype=torch.float64))).view(-1, nd)
    if kind == "mixed":  # at rest, uniform, and scaled far up and down in bands of cells
        band = (torch.arange(len(w), device="cuda") // 40) % 8
        w[band == 1, 1] = 0.0
        w[band == 3] = w[0].clone()
        w[band == 5] *= 1e-85
        w[band == 7] *= 1e85
    return w.reshape(-1).contiguous()


def _composed(problem, u, dt, steps):
    """As the stages associate: each product rounded, sums from left to right."""
    v = problem.createVelocity()

    def f(x, t):
        problem.velocity(x, t, v)
        return v

    t = 0.0
    for _ in range(steps):
        a = u + f(u, t) * dt
        b = (a * (1.0 / 4.0) + u * (3.0 / 4.0)) + f(a, t + dt) * (1.0 / 4.0 * dt)
        u = (u * (1.0 / 3.0) + b * (2.0 / 3.0)) + f(b, t + dt / 2.0) * (2.0 / 3.0 * dt)
        t += dt
    return u


def _equal(torch, got, want):
    return torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(0.0), want.nan_to_num(0.0))


@pytest.mark.parametrize("kind", ["ordinary", "mixed"])
@pytest.mark.parametrize("problem,scheme", [("PeriodicSmooth", 0), ("PeriodicSmooth", 1), ("PeriodicSmooth", 2),
                                            ("Sod", 1), ("Sod", 2)])
def test_structured_1d(pda, problem, scheme, kind):
    import torch
    s = torch.cuda.Stream()
    mesh = pda.create_full_mesh((8200,), (-1.0, 1.0), 2 * scheme + 3, (problem != "Sod",))
    p = pda.create_problem(mesh, getattr(pda.Euler1d, problem), scheme, stream=s)
    with torch.cuda.stream(s):
        start = _state(torch, p, kind)
        for steps, dt in ((1, 1e-5), (3, 1e-5), (35, 1e-6)):
            want = _composed(p, start, dt, steps)
            for use_graph in (True, False):
                u = start.clone()
                p.advance_ssprk3(u, 0.0, dt, steps, use_graph=use_graph)
                assert _equal(torch, u, want), (steps, use_graph)
        s.synchronize()
    assert want.isfinite().all() or kind == "mixed"


@pytest.mark.parametrize("dt", [1e-3, 1e-90])
@pytest.mark.parametrize("kind", ["ordinary", "mixed"])
def test_batched_stage(pda, kind, dt):
    import torch
    s = torch.cuda.Stream()
    probs = [pda.create_problem(pda.create_full_mesh(shape, (-5, 5, -5, 5), 7), pda.Swe2d.SlipWall, 2, 1,
                                {"gravity": g, "coriolis": -2.0, "pulseMagnitude": 0.1}, stream=s)
             for shape, g in (((33, 20), 7.0), ((64, 41), 9.0))]
    batch = pda.create_batch(probs, stream=s)
    with torch.cuda.stream(s):
        states = [_state(torch, p, kind) for p in probs]
        u = batch.createState()
        for i, x in enumerate(states):
            batch.instance(u, i).copy_(x)
        batch.advance_ssprk3(u, 0.0, dt, 2)
        for i, (p, x) in enumerate(zip(probs, states)):
            assert _equal(torch, batch.instance(u, i), _composed(p, x, dt, 2)), i
        s.synchronize()
