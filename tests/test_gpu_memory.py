"""Device memory of an FP64 problem: the records of the linearisation and those
of the Schur products are never needed together and share their memory."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


def test_bytes_per_observation(zs_lib):
    torch = pytest.importorskip("torch")
    K, L = 8, 60000
    sc = scenes.arc_scene(K, 100, seed=1)
    X = np.tile(sc.landmarks, (L // 100, 1))
    pose, lm = np.meshgrid(np.arange(K, dtype=np.int32), np.arange(L, dtype=np.int32))
    sc.landmarks, sc.landmark_fixed = X, np.zeros(L, np.uint8)
    sc.obs_pose, sc.obs_landmark = pose.ravel().copy(), lm.ravel().copy()
    sc.obs_uv = np.full((K * L, 2), 250.0)
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_problem(scenes.arc_scene(K, 100, seed=1))
        h.linear_step(1.0)  # (the context and the kernels are loaded)
        before = torch.cuda.mem_get_info()[0]
        h.set_problem(sc)
        used = before - torch.cuda.mem_get_info()[0]
    # H_pl and W 144 bytes each, the shared records 320, the index arrays and
    # pixels 41, the triples (K + 1) / 2 x 8 = 36 an observation and the landmarks'
    # arrays about 300 / K = 38; a tenth for the allocator
    assert used <= 1.1 * (144 + 144 + 320 + 41 + 36 + 38) * sc.M
