"""A call's result does not depend on the calls before it: from the same reset
state, the same number of iterations gives the same bits before and after calls
that make the lists of the quiet-prefix path (long calls, the autotuners)."""
import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300 import synthetic

pytestmark = pytest.mark.gpu

BEFORE = {
    "long call": lambda m, f: m.infer(iters=12, flags=f),
    "autotune": lambda m, f: (m.autotune(reps=1, flags=f), m.set_ray_variant(4)),
    "home share": lambda m, f: m.autotune_home_share((60, 90), reps=1, flags=f),
    "forced": lambda m, f: m.infer(iters=3, flags=f | L.QUIET_PREFIX),
}


@pytest.mark.parametrize("flags", [0, L.JACOBI], ids=["gauss-seidel", "jacobi"])
@pytest.mark.parametrize("call", BEFORE)
def test_same_bits(native_lib, call, flags):
    w = synthetic.small_room(0)
    m = L.MRFMap(w.params, activation=L.ACT_FULL_RAY)
    for P, D in zip(w.poses, w.depths):
        m.add_view(P, D)
    seen = {}
    for after in (False, True):
        for n in (3, 4, 5, 7):
            m.reset_state()
            m.infer(iters=n, flags=flags)
            seen[after, n] = (m.logodds(), m.stats()["quiet_prefix_used"])
        if not after:
            BEFORE[call](m, flags)
    for n in (3, 4, 5, 7):
        np.testing.assert_array_equal(seen[True, n][0], seen[False, n][0])
        assert seen[True, n][1] == seen[False, n][1]
    # both paths are in reach of this map
    m.reset_state()
    m.infer(iters=12, flags=flags)
    assert m.stats()["quiet_prefix_used"] == 1 and seen[False, 3][1] == 0
    m.close()
