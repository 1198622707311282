"""The FP64 triangular solves (blocks of 32 rows, an owner CTA each) at ragged
last blocks, one block, and more blocks than SMs; a factor that fails the
reference's solve test (source/matrix_decomposition_cholesky.hpp:74,80); a
block that never comes."""

import os
import subprocess
import sys

import numpy as np
import pytest

from zeroslam_gb300 import ba

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 95, 161, 1200, 4865, 5001])
def test_solution(zs_lib, n):
    rng = np.random.default_rng(n)
    U = rng.normal(size=(n, 8))
    A = U @ U.T + np.diag(rng.uniform(1.0, 100.0, n))
    b = rng.normal(size=n)
    ok, L, x = ba.dense_cholesky_solve(A, b)
    assert ok
    # two substitutions of n terms, each sum rounded at 2^-53 of |L| |y|
    y = np.abs(L.T @ x)
    r = np.abs(L @ (L.T @ x) - b)
    assert np.all(r <= 8 * (n + 32) * 2.0**-53 * (np.abs(L) @ (np.abs(L).T @ np.abs(x) + y)))


@pytest.mark.parametrize("n", [40, 300])
def test_solve_test(zs_lib, n):
    A = np.eye(n)
    A[n - 2, n - 2] = 1e-14 * 0.9  # L_ii = 0.95e-7 max |L_ii|; the pivot test rejects it too
    assert not ba.dense_cholesky_solve(A, np.ones(n))[0]
    A[n - 2, n - 2] = 1.2e-14
    ok, L, x = ba.dense_cholesky_solve(A, np.ones(n))
    assert ok and abs(x[n - 2] * 1.2e-14 - 1) < 1e-12


CHILD = r"""
import numpy as np
from zeroslam_gb300 import ba
n = 200
A = np.eye(n) * 2; b = np.ones(n)
st = ba.dense_cholesky_status(A, b, precision=ba.FP64)
assert st == ba.ZS_ERR_TIMEOUT, st
ok, _, x = ba.dense_cholesky_solve(A, b, precision=ba.MIXED)
assert ok and np.max(np.abs(x - 0.5)) < 1e-12
print("timeout reported, context usable")
"""


def test_stalled_block_times_out(zs_lib):
    env = dict(os.environ, ZS_TEST_STALL_TRISOLVE="2")
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "timeout reported" in r.stdout
