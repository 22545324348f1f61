"""The proposal network's kernels at the edges of their tiles (128 candidates, the grids
of one and of two tiles per CTA), forward and gradients, against the CPU restatement.
Tolerances: the restatement's sums are in float64, the kernels' in fp32: 64 + 16 terms
of order one forward, `n` terms of order 1/n in a gradient."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 128, 129, 255, 257, 38912, 38913, 97281, 200000])
def test_forward_and_gradients(n):
    import torch
    from minimumcyclebasis_gb300.learned import ProposalNet, init_params
    rng = np.random.default_rng(n)
    p = init_params(3)
    p[1024:1088] -= 0.05  # some units off for most candidates
    net = ProposalNet(p)
    x = omlp.bf16_round(rng.normal(size=(n, 16)).astype(np.float32))
    y = (rng.random(n) < 0.3).astype(np.uint8)
    xd, yd = torch.from_numpy(x).to(torch.bfloat16).cuda(), torch.from_numpy(y).cuda()
    want, _ = omlp.forward(p, x)
    for _ in range(2):
        assert np.allclose(net.forward(xd).cpu().numpy(), want, atol=1e-5, rtol=1e-5)
    wl, wg = omlp.loss_and_grads(p, x, y, 2.0)
    for _ in range(2):  # recomputed, not accumulated
        loss, g = net.gradients(xd, yd, pos_weight=2.0)
        assert abs(loss - wl) < 1e-5 * max(1.0, abs(wl))
        assert np.allclose(g, wg, atol=1e-5, rtol=1e-4), np.abs(g - wg).max()
    net.close()
