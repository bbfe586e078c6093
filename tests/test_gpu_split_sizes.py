"""Image sizes on both sides of the rules that change a kernel's split of the
work: likelihood and expected depth with several lanes a ray up to ten 8 x 4
tiles per SM and one lane a ray beyond; runs of dynamic incidences longer than
the pair update's tile and what it gathers ahead; Jacobi iterations past the
second, which visit loud pairs and voxels only.  Against the FP64 oracle at the
project's tolerances."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


ROOM = synthetic.Scene(room=np.array([-1.96, -1.96, 0.04, 1.96, 1.96, 2.96]),
                       boxes=np.array([[0.2, 0.3, 0.04, 0.9, 0.8, 1.1], [-0.6, -1.2, 0.04, -0.2, -0.4, 1.6]]))


def _params(rows, cols, res, f=0.8):
    return synthetic.sensor_params(MapParams(res=res, dims=(4.0, 4.0, 3.0), rows=rows, cols=cols, fx=f * cols,
                                             fy=f * cols, cx=cols / 2, cy=rows / 2, prior=0.1, max_iters=4))


def _views(p, n):
    eyes = [[-1.2, 0.2, 1.4], [1.1, -0.4, 1.5], [0.1, 1.2, 1.3]][:n]
    poses = [synthetic.look_at(e, [-0.8 * e[0], -0.8 * e[1], 1.2]) for e in eyes]
    return [(P, synthetic.render_depth(ROOM, p, P).astype(np.float32)) for P in poses]


def _pair(p, views):
    m, om = L.MRFMap(p, activation=L.ACT_FULL_RAY), O.OracleMap(p, threads=8)
    for P, D in views:
        m.add_view(P, D)
        om.add_view(P, D, O.ACT_FULL_RAY)
    return m, om


@pytest.mark.parametrize("over", [0, 1], ids=["at the rule", "beyond"])
def test_score_and_depth_on_both_sides_of_the_split(native_lib, oracle_lib, over):
    import torch
    tiles = 10 * torch.cuda.get_device_properties(0).multi_processor_count
    cols = 8 * 19  # ragged: the last tile column and row are partly filled
    rows = 4 * (tiles // 19 + over) - 1
    p = _params(rows, cols - 3, 0.08)
    m, om = _pair(p, _views(p, 2))
    m.infer(iters=2)
    om.set_beliefs(m.beliefs().astype(np.float64))
    Q = synthetic.look_at([-1.15, 0.25, 1.45], [1.0, -0.2, 1.2])
    D = synthetic.render_depth(ROOM, p, Q).astype(np.float32)
    ref = om.likelihood(Q, D)
    np.testing.assert_allclose(m.likelihood(Q, D)[1], ref[1] if isinstance(ref, tuple) else ref, rtol=0, atol=1e-3)
    depth, want = m.render(L.RENDER_EXPECTED_DEPTH, Q, D)[0], om.render(L.RENDER_EXPECTED_DEPTH, Q, D, 0.0)
    want = want[0] if isinstance(want, tuple) else want
    np.testing.assert_allclose(depth, want, rtol=0, atol=2e-3)
    m.close()
    om.close()


@pytest.mark.parametrize("rows,cols", [(24, 43), (33, 32), (60, 64)])
def test_runs_longer_than_a_tile(native_lib, oracle_lib, rows, cols):
    """1 m voxels: a wall's returns, up to 3840 rays, fall into a few voxels --
    runs just short of, just past and several times the pair update's tile."""
    p = _params(rows, cols, 1.0, 6.0)
    rng = np.random.default_rng(rows)
    P = synthetic.look_at([-1.5, 0.45, 1.45], [1.5, 0.45, 1.45])
    views = [(P, rng.uniform(2.1, 2.4, (rows, cols)).astype(np.float32))]
    for flags in (0, L.JACOBI):
        m, om = _pair(p, views)
        if rows == 60:
            t = om.view_trace(0)
            assert np.bincount(t["vox"][t["mu"] > 0].astype(np.int64)).max() > 1024 + 32
        m.infer(iters=4, flags=flags)
        om.infer(iters=4, flags=O.JACOBI if flags else 0)
        assert np.abs(m.beliefs() - om.beliefs()).max() <= 1e-3
        # FP32 sums of up to 3840 terms: 2e-4 of the sum at worst
        np.testing.assert_allclose(m.logodds(), om.logodds(), rtol=1e-3, atol=1e-3)
        m.close()
        om.close()


@pytest.mark.parametrize("views", [1, 3])
@pytest.mark.parametrize("path", [0, L.QUIET_PREFIX], ids=["auto", "quiet"])
def test_later_jacobi_iterations(native_lib, oracle_lib, views, path):
    p = _params(36, 44, 0.08)
    m, om = _pair(p, _views(p, views))
    m.infer(iters=6, flags=L.JACOBI | path)
    om.infer(iters=6, flags=O.JACOBI)
    b, ob = m.beliefs(), om.beliefs()
    s = m.stats()
    assert s["n_pairs_dyn"] < s["n_pairs"]
    assert np.abs(b - ob).max() <= 1e-3
    m.close()
    om.close()
