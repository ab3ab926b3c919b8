"""The implicit stepper's device buffers: a problem keeps small ones between
calls and gives large ones (here 317 MiB: 400^2 cells with four rows of 52
entries) back at the end of a call."""
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@pytest.mark.parametrize("n", [32, 400])
def test_large_buffers_are_given_back(pda, n):
    import torch

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    mesh = pda.create_full_mesh((n, n), (0.0, 1.0, 0.0, 1.0), 7)
    p = pda.create_problem(mesh, pda.Euler2d.Riemann, 2, 2)
    u, v, j = p.initialCondition(), p.createVelocity(), p.createJacobian()
    p.velocity(u, 0.0, v)
    p.rightHandSideAndJacobian(u, 0.0, v, j)  # the problem's own tables
    before = used()
    for _ in range(2):
        p.advance_implicit(u, 0.0, 1e-4, 1, newton_max_iters=1, linear_max_iters=3)
        assert used() - before <= 256 * MIB
    assert torch.isfinite(u).all()
