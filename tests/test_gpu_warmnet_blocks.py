"""The network's kernels at brick counts around a block's share: one brick, an
odd few, one more than the SMs (a block with two bricks), one more than two
blocks per SM; ramps that make every tap, channel and brick face matter.
Against the CPU reference with the kernels' BF16 rounding, at the tolerances
of the network's other tests."""
import numpy as np
import pytest

from oracle import warmnet as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 3, 153, 305])
def test_forward_and_gradients(native_lib, nb):
    from mrfmap_gb300 import warmstart as W
    rng = np.random.default_rng(nb)
    feat = rng.normal(0, 1, (nb, 512, 4)).astype(np.float32)
    feat += np.linspace(0, 1, 512, dtype=np.float32)[None, :, None] * np.arange(4, dtype=np.float32)
    target = rng.normal(0, 2, (nb, 512)).astype(np.float32)
    w = (rng.random((nb, 512)) < 0.6).astype(np.float32)
    net = W.WarmNet(seed=nb)
    net.params += torch.from_numpy(rng.normal(0, 0.02, net.params.numel()).astype(np.float32)).cuda()
    p = net.params.cpu().numpy().astype(np.float64)
    ft, tt, wt = (torch.from_numpy(a).cuda() for a in (feat, target, w))
    y = net.predict(ft).cpu().numpy()
    yr, _ = R.forward(p, feat.astype(np.float64), bf16=True)
    assert np.abs(y - np.asarray(yr).reshape(y.shape)).max() <= 1e-2 * np.abs(yr).max()
    norm = float(w.sum())
    runs = []
    for _ in range(2):
        loss = net.gradients(ft, tt, wt, norm)
        runs.append(net.grads.cpu().numpy().copy())
    np.testing.assert_array_equal(runs[0], runs[1])
    lr, gr = R.gradients(p, feat.astype(np.float64), target.astype(np.float64), w.astype(np.float64), norm, bf16=True)
    assert float(loss.item()) == pytest.approx(lr, rel=1e-3)
    o = 0
    for name, shp in R.SHAPES:
        n = int(np.prod(shp))
        a, b = runs[0][o:o + n], gr[o:o + n]
        assert np.abs(a - b).max() <= 2e-2 * np.abs(b).max() + 1e-7, (name, np.abs(a - b).max(), np.abs(b).max())
        o += n
