"""The backward pass of fused training runs on two streams, side by side with the
output layer's update.  With a wide output layer that update takes long enough to
overlap every launch of the other stream; weights, biases and losses equal those
of the separate optimizer pass, which stays on one stream, bit for bit."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_wide_output_layer_equals_one_stream(pda):
    import torch
    n = 49152
    g = torch.Generator(device="cuda").manual_seed(5)
    waves = torch.sin(torch.arange(1, 9, device="cuda")[:, None] * torch.linspace(0, 6.0, n, device="cuda"))
    x = torch.tanh(torch.randn(512, 8, generator=g, device="cuda") @ waves / 3).to(torch.bfloat16).contiguous()
    out = []
    for fused in (True, False):
        ae = pda.AutoEncoder(n, 12, 1024, 256, seed=4)
        ae.set_fused(fused)
        losses = ae.train(x, batch=128, epochs=2, lr=1e-3, seed=9)
        out.append((losses, [ae.layer(l) for l in range(6)]))
    (la, wa), (lb, wb) = out
    assert np.array_equal(la, lb) and np.isfinite(la).all()
    for l in range(6):
        assert torch.equal(wa[l][0], wb[l][0]) and torch.equal(wa[l][1], wb[l][1]), l
