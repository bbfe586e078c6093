"""Features and workspace that start at any float, as a view into a larger
tensor does: the same bits as from arrays on 16 bytes, and nothing written
behind the workspace."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _at(a, words):
    """a's values at `words` floats behind an aligned start."""
    buf = torch.zeros(a.numel() + words, device="cuda")
    v = buf[words:].view(a.shape)
    v.copy_(a)
    assert v.data_ptr() % 16 == 4 * (words % 4)
    return v


@pytest.mark.parametrize("words", [1, 2, 3])
@pytest.mark.parametrize("nb", [1, 64, 305])
def test_offset_arrays(native_lib, nb, words):
    from mrfmap_gb300 import warmstart as W
    g = torch.Generator(device="cuda")
    g.manual_seed(nb)
    feat, target, weight = (torch.randn(nb, 512, *k, generator=g, device="cuda") for k in ((4,), (), ()))
    weight = weight.abs()
    net = W.WarmNet(seed=2)
    ref = net.predict(feat)
    loss = net.gradients(feat, target, weight, 100.0)
    want = (ref, loss, net.grads.clone())
    n = native_lib.mrf_net_workspace_bytes(nb)
    ws = torch.full((n + 4 * words + 256,), 0x5A, dtype=torch.uint8, device="cuda")
    p = lambda t, o=0: C.c_void_p(t.data_ptr() + o)  # noqa: E731
    f, t, w, out, grads, params = (_at(a, words) for a in (feat, target, weight, ref, net.grads, net.params))
    out.zero_()
    grads.zero_()
    l2 = torch.zeros(1, device="cuda")
    assert native_lib.mrf_net_forward(p(params), p(f), nb, p(out), p(ws, 4 * words), None) == 0
    assert native_lib.mrf_net_gradients(p(params), p(f), p(t), p(w), nb, 100.0, p(grads), p(l2), p(ws, 4 * words),
                                        None) == 0
    for a, b in zip((out, l2, grads), want):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    assert (ws[n + 4 * words:] == 0x5A).all() and (ws[:4 * words] == 0x5A).all()
