"""The backward pass over batch sizes: error gradients, transposes and bias sums
go through the rows 128 at a time, so batches of half a group, of one and a half
groups and of many, against the oracle's replay of the same bf16 roundings (3e-2
of each layer's gradient, one bf16 unit in the last place of an operand, as in
the other gradient test)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [64, 192, 256, 1088])
def test_gradients_match_oracle(pda, batch):
    import torch
    import mlp_oracle
    n, k, ha, hb = 192, 4, 128, 64
    ae = pda.AutoEncoder(n, k, ha, hb, seed=3)
    x = torch.from_numpy(np.random.default_rng(6).normal(0, 0.5, (batch, n))).cuda().to(torch.bfloat16)
    loss, g = ae.gradients(x)
    layers = [tuple(t.double().cpu().numpy() for t in ae.layer(l)) for l in range(6)]
    want, gw, gb = mlp_oracle.loss_and_gradients([w for w, _ in layers], [b for _, b in layers],
                                                 x.float().cpu().numpy(), bf16=True)
    assert abs(loss - want) <= 1e-3 * want
    g, off = g.double().cpu().numpy(), 0
    for l in range(6):
        for ref in (gw[l], gb[l]):
            got = g[off: off + ref.size].reshape(ref.shape)
            off += ref.size
            assert np.linalg.norm(got - ref) <= 3e-2 * np.linalg.norm(ref), l
