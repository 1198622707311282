"""The FP64 windows' factors (one launch over all windows) at the edges of
their 32-wide tiles, beside a window whose system is not finite, and when a
dependency never comes."""

import os
import subprocess
import sys

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# n = 6 K: within one tile, just past one, two and four, three tiles exactly, the most
KS = (1, 2, 5, 6, 10, 11, 16, 21, 22, 27, 32)


def _windows():
    return [scenes.arc_scene(K, 60 + 7 * K, seed=K) for K in KS]


def _batch(wins, iterations):
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_batch(wins)
        _, reps, _ = h.solve_batch(iterations)
        return reps, [h.get_window_state(w) for w in range(len(wins))]


def test_windows_match_single_solves(zs_lib):
    wins = _windows()
    reps, states = _batch(wins, 4)
    for w, sc in enumerate(wins):
        with ba.BundleAdjuster(precision=ba.FP64) as h:
            h.set_problem(sc)
            r = h.solve(4)
            p, x = h.get_state()
        assert (reps[w].accepted, reps[w].attempts) == (r.accepted, r.attempts), w
        assert abs(reps[w].chi2_final - r.chi2_final) <= 1e-9 * r.chi2_final + 1e-300, w
        assert np.abs(states[w][0] - p).max() <= 1e-7 * np.abs(p).max(), w
        assert np.abs(states[w][1] - x).max() <= 1e-7 * np.abs(x).max(), w


def test_failed_window_leaves_the_others(zs_lib):
    wins = _windows()
    wins.insert(5, scenes.arc_scene(20, 200, seed=99))
    reps, states = _batch(wins, 4)
    wins[5].landmarks[3] = np.nan
    reps2, states2 = _batch(wins, 4)
    assert reps2[5].accepted == 0 and reps2[5].cholesky_failures == reps2[5].attempts >= 1
    for w in range(len(wins)):
        if w == 5:
            continue
        assert reps2[w].chi2_final == reps[w].chi2_final, w
        assert np.array_equal(states2[w][0], states[w][0]) and np.array_equal(states2[w][1], states[w][1]), w


CHILD = r"""
import numpy as np
from zeroslam_gb300 import ba, scenes
wins = [scenes.arc_scene(K, 200, seed=K) for K in (8, 20, 12)]
for graph in (1, 0):
    with ba.BundleAdjuster(precision=ba.FP64, batch_graph=graph) as h:
        h.set_batch(wins)
        try:
            h.solve_batch(3)
            raise SystemExit("no timeout")
        except ba.ZsError as e:
            assert e.status == ba.ZS_ERR_TIMEOUT, e
        assert np.array_equal(h.get_window_state(1)[0], wins[1].poses)  # where it was
        assert not np.array_equal(h.get_window_state(0)[0], wins[0].poses)
    with ba.BundleAdjuster(precision=ba.MIXED) as h:
        h.set_batch(wins)
        assert h.solve_batch(3)[0] >= 3
print("timeout reported, context usable")
"""


def test_stalled_window_times_out(zs_lib):
    env = dict(os.environ, ZS_TEST_STALL_FX_TASK="0")  # the first tile of the largest window
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "timeout reported" in r.stdout
