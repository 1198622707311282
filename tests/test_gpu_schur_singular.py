"""A landmark whose damped block counts as singular (it then has no inverse and
adds nothing to the reduced system) takes no bits from the Schur products of
the landmarks beside it, however large its own H_pl: one seen once, close to
a camera, added to a scene."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


def _with_near(sc, pose, depth):
    """sc and a landmark at `depth` of camera `pose`, which alone sees it."""
    q, t = scenes.unpack_poses(sc.poses[pose:pose + 1])
    X = scenes.quat_to_matrix(q)[0].T @ (depth * np.array([0.2, 0.1, 1.0]) - t[0])
    out = sc.copy()
    out.landmarks = np.vstack([sc.landmarks, X])
    out.landmark_fixed = np.append(sc.landmark_fixed, np.uint8(0))
    out.obs_pose = np.append(sc.obs_pose, np.int32(pose))
    out.obs_landmark = np.append(sc.obs_landmark, np.int32(sc.L))
    out.obs_uv = np.vstack([sc.obs_uv, [[400.0, 300.0]]])
    return out


def _step(sc, lam):
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        h.set_problem(sc)
        return h.linear_step(lam)


@pytest.mark.parametrize("depth", [0.3, 1e-2, 1e-5])
def test_neighbours_keep_their_bits(zs_lib, depth):
    sc = scenes.arc_scene(6, 90, seed=61)
    lam, pose = 1e-9, 2
    a, b = _step(sc, lam), _step(_with_near(sc, pose, depth), lam)
    K = sc.K
    SA, SB = a["S"].reshape(K, 6, K, 6), b["S"].reshape(K, 6, K, 6)
    for i in range(K):
        for j in range(i + 1):
            if (i, j) != (pose, pose):
                assert np.array_equal(SA[i, :, j], SB[i, :, j]), (i, j)



@pytest.mark.parametrize("depth,lam", [(3.0, 1e-6), (3.0, 1e-2), (0.3, 1e-4), (0.3, 1.0), (1e-2, 1e-2), (1e-2, 100.0)])
def test_damping_alone_holds_it(zs_lib, oracle, depth, lam):
    """The same landmark where the damping makes its block regular: the inverse
    is up to 10^12 times larger along the ray, along which H_pl has no part."""
    sc = scenes.arc_scene(6, 90, seed=61)
    pose, K = 2, sc.K
    two = _with_near(sc, pose, depth)
    a, b = _step(sc, lam), _step(two, lam)
    d = np.sqrt(lam + np.concatenate([np.diag(h) for h in oracle.linear_step(two, lam)["hpp"].reshape(K, 6, 6)]))
    err = np.tril(np.abs(a["S"] - b["S"])) / (d[:, None] * d[None, :])
    err[6 * pose:6 * pose + 6, 6 * pose:6 * pose + 6] = 0.0
    # a pair's sum of at most L products, each rounded at 2^-53 of the two rows' own scale
    assert err.max() <= two.L * 2.0**-53
