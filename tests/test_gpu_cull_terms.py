"""The cull's error terms at distances from far below a pixel to beyond the
range that the integer square root takes, and where they are not finite:
means and decisions equal the oracle's bit for bit."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.0, 1e-3, 1.0, 1e4, 1e15, 1e32, "special"])
def test_terms(zs_lib, oracle, scale):
    cm = scenes.cull_map(scenes.arc_scene(9, 700, seed=31), seed=31, truth=True)
    rng = np.random.default_rng(32)
    kp = cm.obs_keypoint
    if scale == "special":
        kp[rng.integers(0, kp.shape[0], 40), rng.integers(0, 2, 40)] = np.float32(np.inf)
        kp[rng.integers(0, kp.shape[0], 40), rng.integers(0, 2, 40)] = np.float32(1e-40)
        kp[rng.integers(0, kp.shape[0], 10), 0] = np.float32(np.nan)
    else:
        kp += (scale * rng.normal(size=kp.shape)).astype(np.float32)
    e_o, m_o, n_o = oracle.map_cull(cm)
    with ba.BundleAdjuster() as h:
        e, m, rep = h.map_cull(cm)
    assert np.array_equal(e, e_o) and rep.erased == n_o
    assert np.array_equal(m, m_o, equal_nan=True)
