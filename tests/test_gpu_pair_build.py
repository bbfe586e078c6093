"""The pair build at the sizes where it can go wrong: images whose pixel count
does not fill a block's rays, rays shorter and longer than the 64 incidences
collected in shared memory, more near voxels in one block than its table holds
(a wide camera), bricks with one voxel touched and with all 512, pairs with
and without dynamic incidences.

Every incidence's voxel, and the pairs' cumulative lengths through the
messages they gate, come back as the FP64 oracle has them: the incidence lists
bit for bit, the pair and dynamic counts exactly, beliefs at the project's
tolerance."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _view(rows, cols, f, res, seed):
    rng = np.random.default_rng(seed)
    p = synthetic.sensor_params(MapParams(res=res, dims=(4.0, 4.0, 3.0), rows=rows, cols=cols, fx=f * cols,
                                          fy=f * cols, cx=cols / 2, cy=rows / 2, prior=0.1, max_iters=3))
    d = (1.2 + 0.5 * rng.random((rows, cols))).astype(np.float32)
    d[rng.random((rows, cols)) < 0.05] = 0.0
    return p, synthetic.look_at([0.3, -1.7, 1.4], [0.1, 1.5, 1.5]), d


@pytest.mark.parametrize("policy", [L.ACT_ENDPOINT, L.ACT_FULL_RAY], ids=["endpoint", "fullray"])
@pytest.mark.parametrize("rows,cols,f,res", [(1, 1, 1.0, 0.04), (3, 21, 1.0, 0.05), (5, 13, 4.0, 0.005),
                                             (24, 32, 0.25, 0.01)])
def test_pairs_against_oracle(native_lib, oracle_lib, rows, cols, f, res, policy):
    p, P, D = _view(rows, cols, f, res, 3)
    m = L.MRFMap(p, activation=policy)
    om = O.OracleMap(p, threads=8)
    m.add_view(P, D)
    om.add_view(P, D, policy)
    meta, vox, ln, mu = m.view_incidences(0)
    t = om.view_trace(0)
    np.testing.assert_array_equal(vox.astype(np.int64), t["vox"].astype(np.int64))
    np.testing.assert_array_equal(ln.view(np.uint32), t["len"].view(np.uint32))
    # the pairs past the length gate, from the traced lengths in 64 bits
    post = np.concatenate([np.arange(a) < b for a, b in meta[:, :2]]) if len(vox) else np.zeros(0, bool)
    cum = np.bincount(vox[post], weights=ln[post].astype(np.float64)) if post.any() else np.zeros(1)
    st = m.stats()
    assert st["n_pairs"] == len(np.unique(vox))
    assert abs(st["n_pairs_active"] - (cum > 0.1).sum()) <= ((cum > 0.1 - 1e-6) & (cum < 0.1 + 1e-6)).sum()
    m.infer(iters=3)
    om.infer(iters=3)
    b, ob = m.beliefs(), om.beliefs()
    m.close()
    om.close()
    assert b.shape == ob.shape
    if b.size:
        assert np.abs(b - ob).max() <= 1e-3
