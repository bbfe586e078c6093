"""Expected depth and likelihood from poses whose rays run along an axis, along
diagonals (ties), through brick corners and from outside the volume, with
several lanes a ray (small images) and with one (the large one), against the
FP64 oracle on the same beliefs at the project's tolerances."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EYES = {
    "axis_x": ([-0.9, 0.0, 0.5], [0.9, 0.0, 0.5]),
    "axis_y_off": ([0.013, -0.91, 0.507], [0.013, 0.9, 0.507]),
    "diagonal": ([-0.8, -0.8, 0.2], [0.8, 0.8, 0.2]),
    "corner": ([-0.96, -0.96, 0.0], [0.96, 0.96, 0.96]),
    "outside": ([-1.7, 0.3, 0.4], [0.5, -0.2, 0.6]),
    "down": ([0.111, -0.05, 0.93], [0.1101, 0.0499, 0.02]),
}


@pytest.mark.parametrize("policy", [L.ACT_ENDPOINT, L.ACT_FULL_RAY], ids=["endpoint", "fullray"])
@pytest.mark.parametrize("eye", EYES)
@pytest.mark.parametrize("rows,cols", [(3, 3), (17, 23), (201, 263)])
def test_views(native_lib, oracle_lib, rows, cols, eye, policy):
    import torch
    tiles = ((rows + 3) // 4) * ((cols + 7) // 8)
    assert (tiles > 10 * torch.cuda.get_device_properties(0).multi_processor_count) == (rows > 200)
    p = synthetic.sensor_params(MapParams(res=0.04, dims=(1.92, 1.92, 1.0), rows=rows, cols=cols, fx=0.9 * cols,
                                          fy=0.9 * cols, cx=cols / 2, cy=rows / 2, prior=0.1, max_iters=2))
    D = np.random.default_rng(5).uniform(0.2, 2.5, (rows, cols)).astype(np.float32)
    P = synthetic.look_at(*EYES[eye])
    m, om = L.MRFMap(p, activation=policy), O.OracleMap(p, threads=8)
    m.add_view(P, D)
    om.add_view(P, D, policy)
    if m.num_bricks:
        m.infer(iters=2)
        om.set_beliefs(m.beliefs().astype(np.float64))
        img, ref = m.likelihood(P, D)[1], om.likelihood(P, D)[1]
        np.testing.assert_allclose(img, ref, rtol=0, atol=1e-3)
        depth, want = m.render(L.RENDER_EXPECTED_DEPTH, P, D)[0], om.render(L.RENDER_EXPECTED_DEPTH, P, D, 0.0)[0]
        np.testing.assert_allclose(depth, want, rtol=0, atol=2e-3)
    m.close()
    om.close()
