"""A wait of the triangular solve that runs out inside the adjoint's
preconditioner is reported, not taken for a gradient."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import numpy as np
from zeroslam_gb300 import ba, scenes
sc = scenes.arc_scene(14, 300, seed=41, min_obs=2, sigma_px=0.0)
sc.pose_fixed[:2] = 1
sc.poses, sc.landmarks = sc.gt_poses, sc.gt_landmarks  # no residual: the Hessian is positive definite
with ba.BundleAdjuster(precision=ba.FP64) as h:
    h.set_problem(sc)
    try:
        _, _, rep = h.adjoint(np.ones((sc.K, 6)), None)
        raise SystemExit("no timeout: rel_residual %g after %d iterations" % (rep.rel_residual, rep.iterations))
    except ba.ZsError as e:
        assert e.status == ba.ZS_ERR_TIMEOUT, e
    assert h.chi2() < 1e-9
print("timeout reported, context usable")
"""


def test_stalled_solve_times_out(zs_lib):
    env = dict(os.environ, ZS_TEST_STALL_TRISOLVE="0")  # the first of three blocks
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "timeout reported" in r.stdout
