"""The plain linearisation (no loss, no information matrices) against the
general one, which identity information matrices take, at the edges of its
blocks of 256 observations, with fixed poses and landmarks and points behind
their camera."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


def _cut(sc, M):
    for name in ("obs_pose", "obs_landmark", "obs_uv"):
        setattr(sc, name, getattr(sc, name)[:M].copy())
    return sc


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("M", [64, 255, 256, 257, 1000])
def test_plain_linearisation(zs_lib, M, fixed):
    sc = _cut(scenes.arc_scene(6, 200, seed=9), M)
    if fixed:
        sc.pose_fixed[3] = 1
        sc.landmark_fixed[::3] = 1
    for at, shift in ((5, 12.0), (17, 40.0)):
        sc.landmarks[at, 2] -= shift
    out = []
    for info in (None, np.tile(np.array([1.0, 0.0, 0.0, 1.0]), (sc.M, 1))):
        sc.obs_info = info
        with ba.BundleAdjuster(precision=ba.FP64) as h:
            h.set_problem(sc)
            out.append(h.linear_step(1e3))
    p, g = out
    # every entry sums at most M products of two terms, each rounded at 2^-53
    # of H_pp (its largest entry bounds S's: S + E V^-1 E^T = H_pp + lambda I)
    tol = 4 * (sc.M + 2) * 2.0**-53
    assert p["ok"] and g["ok"]
    assert np.abs(p["S"] - g["S"]).max() <= tol * np.abs(g["S"]).max()
    assert np.abs(p["bs"] - g["bs"]).max() <= tol * max(np.abs(g["bs"]).max(), np.abs(g["b"]).max())
    assert np.abs(p["b"] - g["b"]).max() <= tol * np.abs(g["b"]).max()
