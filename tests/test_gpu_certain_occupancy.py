"""Loaded occupancies of exactly 0 and exactly 1: behind a voxel of occupancy 1
the visibility is 0, on either side of the rule that splits a ray over several
lanes.  An image of a third of the rows and columns, with a third of the focal
lengths and centre, has the middle pixels' rays of the large one bit for bit:
the small one takes the split path, the large one and the allocation-free entry
point take one lane a ray."""
import ctypes as C

import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams

pytestmark = pytest.mark.gpu

ROWS, COLS, RES = 75, 80, 0.05
EYE = np.array([-0.813, 0.117, 0.731])


def _map(scale, points, occ):
    k = float(scale)
    p = synthetic.sensor_params(MapParams(res=RES, dims=(2.0, 2.0, 1.5), rows=ROWS * scale, cols=COLS * scale,
                                          fx=70 * k, fy=70 * k, cx=40 * k, cy=37.5 * k, prior=0.1, max_iters=2))
    m = L.MRFMap(p)
    m.load_map(points, occ)
    return m


def _noalloc(m, pose, depth):
    import torch
    d = torch.from_numpy(depth).cuda()
    img, s = torch.zeros_like(d), torch.zeros(1, device="cuda")
    fp = np.ascontiguousarray(pose, np.float32).ctypes.data_as(C.POINTER(C.c_float))
    assert L.load().mrf_likelihood_device_noalloc(m.handle, fp, C.c_void_p(d.data_ptr()), C.c_void_p(img.data_ptr()),
                                                  C.c_void_p(s.data_ptr())) == 0
    m.synchronize()
    return s.item(), img.cpu().numpy()


@pytest.mark.parametrize("share", [0.01, 0.2], ids=["sparse", "dense"])
def test_occupancy_one(native_lib, share):
    import torch
    tiles = 10 * torch.cuda.get_device_properties(0).multi_processor_count
    assert 10 * 19 <= tiles < 30 * 57  # 8 x 4 pixels each: small image at most, large one more
    rng = np.random.default_rng(3)
    pts = np.stack(np.meshgrid(*[np.arange(k) + 0.5 for k in (40, 40, 30)], indexing="ij"), -1).reshape(-1, 3)
    occ = (rng.random(len(pts)) < share).astype(np.float32)
    at = pts * RES - [1.0, 1.0, 0.0]
    occ[np.linalg.norm(at - EYE, axis=1) < 0.35] = 0.0  # nothing within the near limit
    small, large = _map(1, pts, occ), _map(3, pts, occ)
    P = synthetic.look_at(EYE, [0.79, 0.013, 0.677])
    D = rng.uniform(0.3, 1.6, (ROWS, COLS)).astype(np.float32)
    big = np.repeat(np.repeat(D, 3, 0), 3, 1)
    (s, img), one = small.likelihood(P, D), _noalloc(small, P, D)
    ref = large.likelihood(P, big)[1][1::3, 1::3]
    assert np.isfinite(ref).all() and np.isfinite(img).all()
    np.testing.assert_allclose(img, ref, rtol=0, atol=1e-3)
    np.testing.assert_allclose(img, one[1], rtol=0, atol=1e-3)
    assert s == pytest.approx(one[0], rel=1e-5)
    depth = small.render(L.RENDER_EXPECTED_DEPTH, P, D)[0]
    ref = large.render(L.RENDER_EXPECTED_DEPTH, P, big)[0][1::3, 1::3]
    assert np.isfinite(ref).all() and ref.max() > 0
    np.testing.assert_allclose(depth, ref, rtol=0, atol=2e-3)
    small.close()
    large.close()
