"""Calls that need every view's structures (Jacobi iterations, their tuners, the
warm start, its features) right after views were added to a built full-ray map:
the build that these calls make is a full one, not an append.  Against a map
whose views were all there before its first build, bit for bit."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _jacobi(m):
    m.infer(iters=3, flags=L.JACOBI)
    return m.logodds()


def _warm_start(m):
    m.warm_start(np.linspace(-3, 2, m.num_bricks * 512, dtype=np.float32), sweeps=2)
    return m.logodds()


def _features(m):
    f = torch.zeros(m.num_bricks, 512, 4, device="cuda")
    torch.cuda.synchronize()
    m.warm_features(f.data_ptr())
    m.synchronize()
    return f.cpu().numpy()


def _autotune(m):
    m.autotune(reps=1, flags=L.JACOBI)
    return _jacobi(m)


def _home_share(m):
    m.autotune_home_share((50, 90), reps=1, flags=L.JACOBI)
    return _jacobi(m)


@pytest.mark.parametrize("built", ["gauss-seidel", "jacobi"])
@pytest.mark.parametrize("call", [_jacobi, _warm_start, _features, _autotune, _home_share])
def test_after_adding_views(native_lib, call, built):
    w = synthetic.small_room(0)
    out = []
    for first in (2, len(w.poses)):
        m = L.MRFMap(w.params, activation=L.ACT_FULL_RAY)
        for k, (P, D) in enumerate(zip(w.poses, w.depths)):
            m.add_view(P, D)
            if k + 1 == first:
                m.infer(iters=1, flags=L.JACOBI if built == "jacobi" else 0)
                m.reset_state()
        builds = m.stats()["builds_full"] if first == len(w.poses) else None
        out.append(call(m))
        s = m.stats()
        assert s["builds_appended"] == 0
        if builds is not None:
            assert s["builds_full"] == builds
        m.close()
    np.testing.assert_array_equal(out[0], out[1])
