"""Builds whose views do not fit one launch: more views than a trace launch
takes, queues cut by their number of views and by their pixels, and region
lists made again around a retired view.  A ray that a cut lost or doubled
changes a message, so variants that read different queues, builds that cut
differently and the FP64 oracle must agree."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic
from mrfmap_gb300.params import MapParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ROOM = synthetic.Scene(room=np.array([-1.96, -1.96, 0.04, 1.96, 1.96, 2.96]),
                       boxes=np.array([[0.2, 0.3, 0.04, 0.9, 0.8, 1.1], [-0.6, -1.2, 0.04, -0.2, -0.4, 1.6]]))


def _params(rows, cols, res):
    return synthetic.sensor_params(MapParams(res=res, dims=(4.0, 4.0, 3.0), rows=rows, cols=cols, fx=0.8 * cols,
                                             fy=0.8 * cols, cx=cols / 2, cy=rows / 2, prior=0.1, max_iters=4))


def _views(p, n):
    rng = np.random.default_rng(n)
    out = []
    for _ in range(n):
        eye = rng.uniform([-1.4, -1.4, 0.9], [1.4, 1.4, 1.8])
        P = synthetic.look_at(eye, [-0.7 * eye[0], -0.7 * eye[1], 1.2])
        out.append((P, synthetic.render_depth(ROOM, p, P).astype(np.float32)))
    return out


def _map(p, views):
    m = L.MRFMap(p, activation=L.ACT_FULL_RAY)
    for P, D in views:
        m.add_view(P, D)
    return m


@pytest.mark.parametrize("n", [16, 17, 65], ids=["one trace launch", "two", "two queue batches"])
def test_many_views(native_lib, oracle_lib, n):
    """Every view's lists are the oracle's bit for bit, and the iterations give
    the bits of a map whose views were built one by one."""
    p = _params(12, 16, 0.1)
    views = _views(p, n)
    m, om, one = _map(p, views), O.OracleMap(p, threads=8), L.MRFMap(p, activation=L.ACT_FULL_RAY)
    for P, D in views:
        om.add_view(P, D, O.ACT_FULL_RAY)
        one.add_view(P, D)
        one.infer(iters=1)
    for k in range(n):
        meta, vox, ln, mu = m.view_incidences(k)
        t = om.view_trace(k)
        want = np.zeros((12 * 16, 5), np.int32)
        want[t["pix"]] = t["meta"]
        np.testing.assert_array_equal(meta, want)
        np.testing.assert_array_equal(vox.astype(np.int64), t["vox"].astype(np.int64))
        np.testing.assert_array_equal(ln.view(np.uint32), t["len"].view(np.uint32))
        np.testing.assert_array_equal(mu == 0, t["mu"] == 0)
    for variant in (0, 4):
        m.set_ray_variant(variant)
        for flags in (0, L.JACOBI):
            out = []
            for x in (m, one):
                x.reset_state()
                x.infer(iters=3, flags=flags)
                out.append(x.logodds())
            np.testing.assert_array_equal(out[0], out[1])
    m.close()
    om.close()
    one.close()


def test_queues_cut_by_pixels(native_lib):
    """Four views of 640x480 pass the million pixels of a batch: built at once
    and one by one, by the queue of all rays and by the regions."""
    p = _params(480, 640, 0.1)
    views = _views(p, 4)
    out = []
    for appended in (False, True):
        for variant in (0, 4):
            m = L.MRFMap(p, activation=L.ACT_FULL_RAY)
            for P, D in views:
                m.add_view(P, D)
                if appended:
                    m.infer(iters=1)
            m.set_ray_variant(variant)
            for flags in (0, L.JACOBI):
                m.reset_state()
                m.infer(iters=3, flags=flags)
                out.append((flags, m.logodds()))
            m.close()
    for flags in (0, L.JACOBI):
        same = [lo for f, lo in out if f == flags]
        for lo in same[1:]:
            np.testing.assert_array_equal(lo, same[0])


@pytest.mark.parametrize("appended", [False, True], ids=["one build", "appended"])
def test_region_lists_again_around_a_retired_view(native_lib, appended):
    p = _params(48, 64, 0.08)
    views = _views(p, 5)
    out = []
    for share in (None, 30, 95):
        m = L.MRFMap(p, activation=L.ACT_FULL_RAY)
        for P, D in views:
            m.add_view(P, D)
            if appended:
                m.infer(iters=1, flags=L.INCREMENTAL)
        m.set_ray_variant(4)
        m.infer(iters=2, flags=L.INCREMENTAL)
        m.retire_view(2)
        m.infer(iters=1, flags=L.INCREMENTAL)
        if share:
            m.set_home_share(share)
        m.infer(iters=2, flags=L.INCREMENTAL)
        m.infer(iters=2, flags=L.INCREMENTAL | L.JACOBI)
        out.append(m.logodds())
        m.close()
    for lo in out[1:]:
        np.testing.assert_array_equal(lo, out[0])
