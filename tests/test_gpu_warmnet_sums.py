"""The network's weight gradients over many bricks a block.  Every brick is the
same and every value is exact in BF16, so a gradient is the brick's FP64
gradient times the bricks, and what remains is the rounding of the sums: a
brick's up to 32 accumulating steps (truncated, at most two units of 2^-23 of
the running sum each: 4e-6 of the brick's sum), up to 108 bricks in a block's
register (2^-24 each: 3.2e-6) and 27 additions of the blocks' parts (1.6e-6)."""
import numpy as np
import pytest

from oracle import warmnet as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 16384])
def test_gradient_sums(native_lib, nb):
    from mrfmap_gb300 import warmstart as W
    x = 150 / 128  # eight mantissa bits
    P = {name: np.zeros(shp) for name, shp in R.SHAPES}
    P["b1"][:] = x
    P["W2"][13] = np.eye(16)  # both activations are x everywhere
    P["W3"][13] = 0.75
    p = R.pack(P)
    feat = np.tile(np.array([150, 171, 225, 251]) / 128, (1, 512, 1))
    target = np.full((1, 512), 16 * 0.75 * x - x)  # the output's gradient is x
    w = np.ones((1, 512))
    _, g = R.gradients(p, feat, target, w, 2.0, bf16=True)
    net = W.WarmNet(seed=0)
    net.params.copy_(torch.from_numpy(p.astype(np.float32)))
    many = [torch.from_numpy(a.astype(np.float32)).cuda().repeat(nb, *[1] * (a.ndim - 1)) for a in (feat, target, w)]
    net.gradients(*many, 2.0)
    out = net.grads.cpu().numpy().astype(np.float64)
    np.testing.assert_allclose(out, nb * g, rtol=1e-5, atol=0)
