"""V and J of a mesh with more tiles of faces along a line than one grid
dimension holds (65,535 of 31 faces).  The state repeats, so each period's rows
are those of a short mesh with the same cell width, bit for bit; the rows at the
short mesh's ends, whose columns wrap around, are compared on a state that is
shifted by half a period."""
import pytest

pytestmark = pytest.mark.gpu

CELLS, PERIOD = 2 ** 21, 4096


@pytest.mark.parametrize("scheme", [1, 2])
def test_long_line_repeats_a_short_one(pda, scheme):
    import torch
    width = 2.0 ** -20

    def evaluate(cells, u):
        mesh = pda.create_full_mesh((cells,), (0.0, cells * width), 2 * scheme + 3, (True,))
        p = pda.create_problem(mesh, pda.Euler1d.PeriodicSmooth, scheme)
        v, j = p.createVelocity(), p.createJacobian()
        p.rightHandSideAndJacobian(u, 0.0, v, j)
        torch.cuda.synchronize()
        assert j.values.numel() == cells * 9 * (2 * scheme + 3)  # every row has its full stencil
        return v.view(cells, 3), j.values.view(cells, -1)

    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.arange(PERIOD, device="cuda", dtype=torch.float64) * (2 * torch.pi / PERIOD)
    rho = 1 + 0.2 * torch.sin(x) + 1e-3 * torch.rand(PERIOD, generator=g, device="cuda", dtype=torch.float64)
    u = torch.stack([rho, 0.7 * rho, 2.5 + 0.5 * 0.7 ** 2 * rho], 1)
    v, j = evaluate(CELLS, u.repeat(CELLS // PERIOD, 1).reshape(-1))
    half = PERIOD // 2
    for shift in (0, half):
        vs, js = evaluate(PERIOD, u.roll(-shift, 0).reshape(-1).contiguous())
        inner = slice(half // 2, PERIOD - half // 2)
        vl = v.roll(-shift, 0).view(-1, PERIOD, 3)[1:-1]
        jl = j.view(-1, PERIOD, j.shape[1])
        jl = jl[1:-1] if shift == 0 else torch.cat([jl[:-1, half:], jl[1:, :half]], 1)
        assert torch.equal(vl, vs.expand_as(vl))
        assert torch.equal(jl[:, inner], js[inner].expand_as(jl[:, inner]))
