"""Tuning of maps whose Jacobi launches cover several views: they run the
longest-first variant unless told otherwise, which reads no regions, so the
home share is tuned on the launches that it governs; and both schedules'
variants can be read and put back."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic

pytestmark = pytest.mark.gpu


def _map(views):
    w = synthetic.full_room(1, n_frames=views, rows=24, cols=32, res=0.1)
    m = L.MRFMap(w.params, activation=L.ACT_FULL_RAY)
    for P, D in zip(w.poses, w.depths):
        m.add_view(P, D)
    m.infer(iters=1, flags=L.JACOBI)
    return m


def test_home_share_is_tuned_where_it_counts(native_lib):
    """A Jacobi iteration is a handful of launches, a Gauss-Seidel one as many
    per view: over 16 tiny views their times tell which was timed."""
    m = _map(16)
    best, share_ms = m.autotune_home_share((50, 90), reps=10, flags=L.JACOBI)
    assert best in (50, 90) and m.tuning()[1] == best
    _, jacobi_ms = m.autotune(reps=10, flags=L.JACOBI)
    _, gs_ms = m.autotune(reps=10)
    assert np.median(gs_ms) > 3 * np.median(jacobi_ms)  # what the test rests on
    assert share_ms.min() > 2 * np.median(jacobi_ms)
    # a chosen variant with regions: the Jacobi iterations themselves
    m.set_ray_variant(3)
    _, share_ms = m.autotune_home_share((50, 90), reps=10, flags=L.JACOBI)
    assert share_ms.max() < 0.5 * np.median(gs_ms)
    m.close()


def test_variants_of_both_schedules_can_be_put_back(native_lib):
    m = _map(3)
    assert (m.tuning()[0], m.ray_variant(), m.ray_variant(L.JACOBI)) == (4, 4, 1)
    keep = m.ray_variant(), m.ray_variant(L.JACOBI)
    m.reset_state()
    m.infer(iters=3, flags=L.JACOBI)
    b = m.beliefs()
    m.set_ray_variant(6)
    assert (m.ray_variant(), m.ray_variant(L.JACOBI)) == (6, 6)
    best, _ = m.autotune(reps=1, flags=L.JACOBI)
    assert (m.ray_variant(), m.ray_variant(L.JACOBI)) == (best, best)
    m.set_ray_variant(keep[0], flags=0)
    m.set_ray_variant(keep[1], flags=L.JACOBI)
    assert (m.tuning()[0], m.ray_variant(), m.ray_variant(L.JACOBI)) == (4, 4, 1)
    m.reset_state()
    m.infer(iters=3, flags=L.JACOBI)
    np.testing.assert_array_equal(m.beliefs(), b)
    for bad in (-1, 99):
        with pytest.raises(L.MrfError):
            m.set_ray_variant(bad, flags=L.JACOBI)
    assert (m.ray_variant(), m.ray_variant(L.JACOBI)) == (4, 1)
    m.close()
