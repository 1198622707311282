"""An FP64 window of a batch gives the same bits whichever windows are beside it
(below 1,024 poses in all, from which on b_s is summed by whole poses)."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


def _first(wins):
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_batch(wins)
        _, reps, _ = h.solve_batch(3)
        return (*h.get_window_state(0), reps[0].chi2_final)


@pytest.mark.parametrize("K,L", [(6, 90), (20, 1500)])
def test_neighbours(zs_lib, K, L):
    w = [scenes.arc_scene(K, L, seed=s) for s in range(4)]
    alone = _first(w[:1])
    for beside in (w[:2], w, [w[0], scenes.arc_scene(5, 40, seed=9)]):
        got = _first(beside)
        assert np.array_equal(got[0], alone[0]) and np.array_equal(got[1], alone[1])
        assert got[2] == alone[2]
