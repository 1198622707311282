"""The adjoint's two preconditioners (the exact Hessian's factorisation, and
the Gauss-Newton matrix's where a landmark's block is singular) on the inputs
that its blocks handle in code of their own, against the FP64 reference."""

import numpy as np
import pytest

from conftest import rel_err
from gradcheck import harness as H
from zeroslam_gb300 import ba, scenes

pytestmark = pytest.mark.gpu

ADJ_TOL = 1e-5  # of the reference's central differences
# With the exact factorisation what is left to the iterations is its rounding
# and a damping of 1e-13; with the Gauss-Newton matrix it is the curvature of
# residuals of a pixel.
EXACT_ITERATIONS = 4


def _append(sc, pose, landmark, uv):
    sc.obs_pose = np.append(sc.obs_pose, np.int32(pose))
    sc.obs_landmark = np.append(sc.obs_landmark, np.int32(landmark))
    sc.obs_uv = np.vstack([sc.obs_uv, uv])


def _scene(kind):
    sc = scenes.arc_scene(5, 40, seed=51, min_obs=2, **scenes.ADJOINT_INIT_NOISE)
    sc.pose_fixed[1] = 1
    rng = np.random.default_rng(52)
    if kind == "info":
        A = rng.normal(size=(sc.M, 2, 2)) / 3 + np.eye(2)
        sc.obs_info = np.ascontiguousarray((A @ A.transpose(0, 2, 1)).reshape(sc.M, 4))
        sc.obs_info[:, 2] = sc.obs_info[:, 1]
    elif kind == "duplicates":
        for o in (0, 7, 7, 31):
            _append(sc, sc.obs_pose[o], sc.obs_landmark[o], sc.obs_uv[o] + 0.3 * rng.normal(size=2))
    elif kind == "fixed":
        sc.landmark_fixed[::3] = 1
    return sc


def _camera(pose):
    q, t = scenes.unpack_poses(pose[None])
    return scenes.quat_to_matrix(q)[0], t[0]


@pytest.mark.parametrize("kind", ["plain", "info", "duplicates", "fixed", "behind"])
def test_exact_preconditioner(zs_lib, oracle, kind):
    sc = _scene(kind)
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        x = H.converge(h, sc)
        if kind == "behind":  # a landmark to the side: before three cameras, at the back of the last
            X = np.array([20.0, 0.5, 2.0])
            Xc = [_camera(p)[0] @ X + _camera(p)[1] for p in x[0]]
            assert min(c[2] for c in Xc[:3]) > 1 and Xc[4][2] < -1
            f = sc.intrinsics
            for k in (0, 1, 2):
                _append(sc, k, sc.L, [f[0] * Xc[k][0] / Xc[k][2] + f[2], f[1] * Xc[k][1] / Xc[k][2] + f[3]])
            _append(sc, 4, sc.L, [300.0, 200.0])
            sc.landmark_fixed = np.append(sc.landmark_fixed, np.uint8(0))
            sc.landmarks = np.vstack([sc.landmarks, X])
            x = (x[0], np.vstack([x[1], X]))
            h.set_problem(sc)
            h.set_state(*x)
        rng = np.random.default_rng(53)
        a_p = rng.normal(size=(sc.K, 6)) * (sc.pose_fixed == 0)[:, None]
        a_l = rng.normal(size=(sc.L, 3)) * (sc.landmark_fixed == 0)[:, None]
        duv, dint, rep = h.adjoint(a_p, a_l)
    ref_uv, ref_int = H.reference_gradient(oracle, sc, x, a_p, a_l)
    if kind == "info":  # d(-gradient)/d(pixel) carries the information matrix
        ref_uv = np.einsum("mij,mj->mi", sc.obs_info.reshape(-1, 2, 2), ref_uv)
    if kind == "behind":  # its penalty does not depend on the pixel; its rows, 40 times
        ref_uv[-1] = 0.0  # the others', leave a residual of 1600 times theirs
    assert rep.rel_residual < (1e-8 if kind == "behind" else 1e-10)
    assert rep.iterations <= EXACT_ITERATIONS
    assert rel_err(dint, ref_int) < ADJ_TOL
    assert rel_err(duv, ref_uv) < ADJ_TOL


@pytest.mark.parametrize("kind", ["unseen", "once"])
def test_singular_landmark_takes_gauss_newton(zs_lib, oracle, kind):
    sc = _scene("plain")
    a_l = np.zeros((sc.L, 3))
    a_p = np.random.default_rng(54).normal(size=(sc.K, 6)) * (sc.pose_fixed == 0)[:, None]
    with ba.BundleAdjuster(precision=ba.FP64) as h:
        x = H.converge(h, sc)
        ref_uv, ref_int = H.reference_gradient(oracle, sc, x, a_p, a_l)
        # A landmark that nothing, or one pixel that it meets, holds: it takes up
        # the pixel's residual whatever the pose does, and no other value changes.
        R, t = _camera(x[0][3])
        X = R.T @ (np.array([0.3, -0.2, 4.0]) - t)
        two = sc.copy()
        two.landmarks = np.vstack([sc.landmarks, X])
        two.landmark_fixed = np.append(sc.landmark_fixed, np.uint8(0))
        if kind == "once":
            f = two.intrinsics
            _append(two, 3, sc.L, np.array([f[0] * 0.3 / 4.0 + f[2], f[1] * -0.2 / 4.0 + f[3]]))
            ref_uv = np.vstack([ref_uv, np.zeros(2)])
        h.set_problem(two)
        h.set_state(x[0], np.vstack([x[1], X]))
        duv, dint, rep, v = h.adjoint(a_p, np.zeros((two.L, 3)), want_state=True)
    assert rep.iterations > EXACT_ITERATIONS, "the exact Hessian's factorisation took a singular block"
    assert rep.rel_residual < 1e-10
    if kind == "unseen":
        assert np.all(v[-3:] == 0.0)
    assert rel_err(dint, ref_int) < ADJ_TOL
    assert rel_err(duv, ref_uv) < ADJ_TOL
