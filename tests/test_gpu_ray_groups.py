"""The ray kernel's lane groups at the sizes where they can go wrong: rays of
every length from a few incidences to more than 512 (one chunk, several, the
FP64 sums), mixed in one warp, dynamic windows that start at any offset in a
vector, counts that do not fill a warp's groups, rays that leave the volume
(the infinity term) and invalid pixels -- against the FP64 oracle at the
project's belief tolerance, with the static prefixes in full and from their
quiet sums."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _ramp(rows, cols, res, seed):
    """Two views facing each other, the depths of each a shuffled ramp."""
    rng = np.random.default_rng(seed)
    p = synthetic.sensor_params(MapParams(res=res, dims=(6.0, 6.0, 3.0), rows=rows, cols=cols, fx=1.5 * cols,
                                          fy=1.5 * cols, cx=cols / 2, cy=rows / 2, prior=0.1, max_iters=4))
    views = []
    for x in (-2.8, 2.8):
        d = rng.permutation(np.linspace(0.12, 5.9, rows * cols)).astype(np.float32)
        d[rng.random(d.size) < 0.02] = 0.0
        d[0] = np.nan
        views.append((synthetic.look_at([x, 0.1 * x, 1.4], [-x, 0.0, 1.5]), d.reshape(rows, cols)))
    return p, views


@pytest.mark.parametrize("rows,cols,res", [(1, 1, 0.05), (1, 5, 0.02), (7, 9, 0.04), (23, 29, 0.01)])
@pytest.mark.parametrize("flags", [0, L.JACOBI, L.FIX_PRE_RESET], ids=["gauss-seidel", "jacobi", "fix-reset"])
def test_ray_groups_against_oracle(native_lib, oracle_lib, rows, cols, res, flags):
    p, views = _ramp(rows, cols, res, 11)
    om = O.OracleMap(p, threads=8)
    for P, D in views:
        om.add_view(P, D, O.ACT_FULL_RAY)
    om.infer(iters=4, flags=(O.JACOBI if flags & L.JACOBI else 0) | (O.FIX_PRE_RESET if flags & L.FIX_PRE_RESET else 0))
    ob = om.beliefs()
    om.close()
    for path in (L.FULL_RAYS, L.QUIET_PREFIX):
        m = L.MRFMap(p, activation=L.ACT_FULL_RAY)
        for P, D in views:
            m.add_view(P, D)
        m.infer(iters=4, flags=flags | path)
        b = m.beliefs()
        if rows > 20:
            n_pre = np.concatenate([m.view_incidences(v)[0][:, 0] for v in (0, 1)])
            assert n_pre.max() > 512 and 0 < n_pre[n_pre > 0].min() < 33
        m.close()
        assert b.shape == ob.shape
        if not b.size:
            continue
        assert np.abs(b - ob).max() <= 1e-3
        touched = (b > 0) | (ob > 0)
        assert not touched.any() or ((b > 0.5) == (ob > 0.5))[touched].mean() >= 0.999
