"""Brick-wise steps of the traversal (dda_cross) against voxel-wise ones: the
count pass leaves bricks in one go and the emit pass steps their voxels, the
incidence lists are compared with the oracle's bit for bit, over poses whose
rays run along an axis, along diagonals (ties), through brick corners and
edges, from outside the volume, and from inside an inactive brick; scene boxes
included.  The likelihood and the expected depth cross inactive bricks the same
way."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EYES = {
    "axis_x": ([-0.9, 0.0, 0.5], [0.9, 0.0, 0.5]),          # a boundary of voxels and bricks
    "axis_y_off": ([0.013, -0.91, 0.507], [0.013, 0.9, 0.507]),
    "diagonal": ([-0.8, -0.8, 0.2], [0.8, 0.8, 0.2]),        # ties of x and y in every voxel
    "corner": ([-0.96, -0.96, 0.0], [0.96, 0.96, 0.96]),     # ties of all three, brick corners
    "outside": ([-1.7, 0.3, 0.4], [0.5, -0.2, 0.6]),
    "down": ([0.111, -0.05, 0.93], [0.1101, 0.0499, 0.02]),
}


def _params(rows, cols, res):
    return synthetic.sensor_params(MapParams(res=res, dims=(1.92, 1.92, 1.0), rows=rows, cols=cols, fx=0.9 * cols,
                                             fy=0.9 * cols, cx=cols / 2, cy=rows / 2, prior=0.1, max_iters=2))


@pytest.mark.parametrize("policy", [L.ACT_ENDPOINT, L.ACT_FULL_RAY], ids=["endpoint", "fullray"])
@pytest.mark.parametrize("eye", EYES)
@pytest.mark.parametrize("rows,cols,res", [(3, 3, 0.04), (17, 23, 0.02), (12, 31, 0.013)])
def test_lists_bit_exact(native_lib, oracle_lib, rows, cols, res, eye, policy):
    p = _params(rows, cols, res)
    rng = np.random.default_rng(5)
    P = synthetic.look_at(*EYES[eye])
    D = rng.uniform(0.2, 2.5, (rows, cols)).astype(np.float32)
    m = L.MRFMap(p, activation=policy)
    om = O.OracleMap(p, threads=4)
    m.add_view(P, D)
    om.add_view(P, D, policy)
    assert m.num_bricks == om.num_bricks
    meta, vox, ln, mu = m.view_incidences(0)
    t = om.view_trace(0)
    ometa = np.zeros((rows * cols, 5), np.int32)
    ometa[t["pix"]] = t["meta"]
    np.testing.assert_array_equal(meta, ometa)
    np.testing.assert_array_equal(vox.astype(np.int64), t["vox"].astype(np.int64))
    np.testing.assert_array_equal(ln.view(np.uint32), t["len"].view(np.uint32))
    np.testing.assert_array_equal(mu == 0, t["mu"] == 0)
    # the same field on both sides: likelihood within the project's 1e-3, the
    # expected depth within 2e-3
    if m.num_bricks:
        m.infer(iters=2)
        b = m.beliefs().astype(np.float64)
        om.set_beliefs(b)
        Q = synthetic.look_at(np.add(EYES[eye][0], [0.01, 0.02, 0.015]), EYES[eye][1])
        img, ref = m.likelihood(Q, D)[1], om.likelihood(Q, D)
        ref = ref[1] if isinstance(ref, tuple) else ref
        np.testing.assert_allclose(img, ref, rtol=0, atol=1e-3)
    m.close()
    om.close()


def test_pose_without_a_direction(native_lib):
    """NaN poses give no voxels and end."""
    p = _params(6, 8, 0.04)
    m = L.MRFMap(p, activation=L.ACT_FULL_RAY)
    for k in (0, 3):
        P = synthetic.look_at(*EYES["outside"]).copy()
        P[0, k] = np.nan
        m.add_view(P, np.full((6, 8), 1.0, np.float32))
    m.infer(iters=1)
    assert m.stats()["n_inc_pre"] == 0
    m.close()
