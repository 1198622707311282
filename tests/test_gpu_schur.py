"""The FP64 Schur products at the sizes where their split can go wrong:
pairs of poses that share a few landmarks (below, at and above the eight that
a warp takes at a time), segments at their shortest and longest, and more
than one segment a pair. S and b_s against the oracle."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,L", [(2, 1), (3, 7), (3, 8), (4, 9), (5, 31), (3, 33), (2, 513), (6, 520), (30, 1100)])
def test_schur_products(zs_lib, oracle, K, L):
    sc = scenes.arc_scene(K, L, seed=K + L)
    o = oracle.linear_step(sc, 30.0)
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_problem(sc)
        d = h.linear_step(30.0)
    # at most 1100 products a pair, each sum rounded at 2^-53 of H_pp: 1.2e-13 of it
    scale = np.abs(o["hpp"]).max()
    assert np.abs(d["S"] - o["S"]).max() <= 1e-12 * scale
    assert np.abs(d["bs"] - o["bs"]).max() <= 1e-12 * max(np.abs(o["bs"]).max(), np.abs(o["b"]).max())


@pytest.mark.parametrize("f", [1e-90, 1e-9, 1e12, 1e90])
def test_schur_scales(zs_lib, oracle, f):
    sc = scenes.arc_scene(7, 61, seed=3)
    rng = np.random.default_rng(1)
    w = f * 10.0 ** rng.uniform(-3, 3, sc.M)  # an information a million times another's
    sc.obs_info = np.stack([w, 0 * w, 0 * w, w], 1)
    o = oracle.linear_step(sc, 30.0 * f)
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_problem(sc)
        d = h.linear_step(30.0 * f)
    # as above, and each 3 x 3 inverse, formed by both with their own rounding,
    # is only good to its condition number
    tol = 1e-12 + 4 * np.linalg.cond(o["hll"] + 30.0 * f * np.eye(3)).max() * 2.0**-53
    assert np.abs(d["S"] - o["S"]).max() <= tol * np.abs(o["hpp"]).max()
    assert np.abs(d["bs"] - o["bs"]).max() <= tol * max(np.abs(o["bs"]).max(), np.abs(o["b"]).max())


def test_schur_overflow(zs_lib, oracle):
    sc = scenes.arc_scene(5, 40, seed=4)
    sc.obs_info = np.tile(np.array([1e306, 0, 0, 1e306]), (sc.M, 1))
    assert not oracle.linear_step(sc, 1.0)["ok"]
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_problem(sc)
        assert not h.linear_step(1.0)["ok"]
