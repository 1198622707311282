"""The one-launch tracking solve at the edges of its sums: a warp's 32
observations, the four warps of a task, the 256 of a chunk, and the chunk
counts (8, 16, more) at which the sums over chunks change their split; one to
four free poses. Against the general path."""

import numpy as np
import pytest

from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu


def _tracking(M, free, huber):
    """At most M observations of each free pose, and the fixed poses' own."""
    sc = scenes.arc_scene(free + 3, 6000 if M > 300 else 400, seed=M + free, huber=huber)
    sc.landmark_fixed[:] = 1
    sc.pose_fixed[:] = 1
    sc.pose_fixed[1:1 + free] = 0
    keep = np.ones(sc.M, bool)
    for k in range(1, 1 + free):
        keep[np.flatnonzero(sc.obs_pose == k)[M:]] = False
    for name in ("obs_pose", "obs_landmark", "obs_uv"):
        setattr(sc, name, getattr(sc, name)[keep].copy())
    return sc


def _solve(sc, path, iterations):
    with ba.BundleAdjuster(precision=ba.FP64, pose_only_path=path) as h:
        h.set_problem(sc)
        r = h.solve(iterations)
        return r, h.get_state()[0]


@pytest.mark.parametrize("huber", [False, True])
@pytest.mark.parametrize("M,free", [(6, 1), (31, 1), (32, 2), (33, 4), (127, 1), (129, 3), (255, 1), (257, 2), (2047, 1),
                                    (2049, 2), (4097, 1), (5001, 4)])
def test_sums(zs_lib, M, free, huber):
    sc = _tracking(M, free, huber)
    # under Huber the last bit of a pose decides an outlier's second-order
    # weight in the next linearisation, so there the first step is compared
    n = 1 if huber else 3
    r, p = _solve(sc, 1, n)
    r0, p0 = _solve(sc, 0, n)
    assert r.kernel_launches == 1 and r0.kernel_launches > 1
    assert (r.accepted, r.attempts) == (r0.accepted, r0.attempts)
    # sums of up to 40,000 terms in another order: 40,000 2^-53 = 4.4e-12 of
    # the cost (each term is at least zero); the poses that follow keep nine digits
    assert abs(r.chi2_final - r0.chi2_final) <= 5e-12 * r0.chi2_final
    assert np.abs(p - p0).max() <= 1e-9 * np.abs(p0).max()
