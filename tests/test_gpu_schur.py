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
