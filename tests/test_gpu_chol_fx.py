"""The FP64 factor (fixed-point products, FP64 diagonal blocks) at the edges
of its tiles and of the two tile sizes, on rows of very different scale and
on ill-conditioned matrices; matrices that are not positive definite fail as
matrix::decompose_cholesky does (source/matrix_decomposition_cholesky.hpp:40,53);
a dependency that never comes is reported, not waited for."""

import os
import subprocess
import sys

import numpy as np
import pytest

from zeroslam_gb300 import ba

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _spd(n, seed, kind):
    rng = np.random.default_rng(seed)
    if kind == "ill":  # condition 1e10
        Q, _ = np.linalg.qr(rng.normal(size=(n, n)))
        A = (Q * np.logspace(0, -10, n)) @ Q.T
        return 0.5 * (A + A.T)
    A = rng.normal(size=(n, n))
    A = A @ A.T / n + np.eye(n)
    if kind == "scaled":
        d = 10.0 ** rng.uniform(-3, 0, n)
        A = A * d[:, None] * d[None, :]
    return A


@pytest.mark.parametrize("kind", ["plain", "scaled", "ill"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 97, 200, 385, 1535, 1536, 1537, 1600, 1665])
def test_factor(zs_lib, n, kind):
    A = _spd(n, n, kind)
    b = np.random.default_rng(n + 1).normal(size=n)
    ok, L, x = ba.dense_cholesky_solve(A, b)
    assert ok
    # Backward error of an entry in FP64: at most (n + 1) 2^-53 of its row and
    # column scales; the factor's last rounding and this product's own add as much.
    s = np.sqrt(np.diag(A))
    err = np.abs(np.tril(L @ L.T - A)) / (s[:, None] * s[None, :])
    assert err.max() <= 3 * (n + 2) * 2.0**-53
    r = np.linalg.norm(A @ x - b)
    assert r <= 40 * (n + 2) * 2.0**-53 * np.linalg.norm(A, 2) * np.linalg.norm(x)


@pytest.mark.parametrize("n", [1, 2, 33, 70, 4640])
def test_pivots_of_powers_of_four(zs_lib, n):
    """Pivots that are powers of four, the lowest of their scaled range, and
    factors that FP64 holds: L's diagonal is the positive root."""
    rng = np.random.default_rng(n)
    L = np.eye(n) + np.diag(rng.choice([-0.25, 0.0, 0.25], n - 1), -1)
    L = 2.0 ** rng.integers(-3, 4, n)[:, None] * L
    ok, F, _ = ba.dense_cholesky_solve(L @ L.T, np.ones(n))
    assert ok
    # A pivot's error is a few 2^-60 of its scale and what it passes on shrinks
    # sixteenfold from row to row: the last conversion's 2^-53 and as much again.
    assert (np.abs(F - L) <= 2.0**-52 * np.sqrt(np.diag(L @ L.T))[:, None]).all()


@pytest.mark.parametrize("n", [4608, 4609, 4641, 4705])
def test_factor_large(zs_lib, n):
    """Either side of the change of tiles (n = 4608), and the 64-wide tiles' ragged ends."""
    test_factor(zs_lib, n, "plain")


@pytest.mark.parametrize("kind", ["late", "nan"])
def test_not_positive_definite_large(zs_lib, kind):
    test_not_positive_definite(zs_lib, kind, 4700)


@pytest.mark.parametrize("n", [2, 40, 130, 1600])
@pytest.mark.parametrize("kind", ["negative", "zero", "large", "correlated", "late", "nan", "inf"])
def test_not_positive_definite(zs_lib, kind, n):
    A = _spd(n, n + 7, "scaled")
    if kind == "negative":
        A[n - 1, n - 1] *= -1
    elif kind == "zero":
        A[n // 2, n // 2] = 0.0
    elif kind == "large":  # an entry above its row and column scales
        A[n - 1, 0] = A[0, n - 1] = 1.2 * np.sqrt(A[0, 0] * A[n - 1, n - 1]) if n == 2 else 1e6
    elif kind == "correlated":  # every 2 x 2 minor positive, the matrix indefinite (n > 2)
        A = np.full((n, n), -0.99)
        np.fill_diagonal(A, 0.98 if n == 2 else 1.0)
    elif kind == "late":  # the last pivot alone is negative, by 1e-6 of its diagonal
        L = np.linalg.cholesky(A)
        L[n - 1, n - 1] = 0.0
        A = L @ L.T
        A[n - 1, n - 1] *= 1.0 - 1e-6
    elif kind == "nan":
        A[n - 1, 0] = np.nan
    else:
        A[n - 1, 0] = np.inf
    ok, _, _ = ba.dense_cholesky_solve(A, np.ones(n))
    assert not ok
    A = _spd(n, n + 8, "plain")  # and the next call is not affected
    ok, _, x = ba.dense_cholesky_solve(A, A @ np.ones(n))
    assert ok and np.abs(x - 1).max() < 1e-10


CHILD = r"""
import numpy as np
from zeroslam_gb300 import ba
rng = np.random.default_rng(0)
for n in (200, 4700):
    G = rng.normal(size=(n, n)); A = G @ G.T / n + np.eye(n); b = rng.normal(size=n)
    st = ba.dense_cholesky_status(A, b, precision=ba.FP64)
    assert st == ba.ZS_ERR_TIMEOUT, st
    ok, _, x = ba.dense_cholesky_solve(A, b, precision=ba.MIXED)
    assert ok and np.max(np.abs(x - np.linalg.solve(A, b))) < 1e-9 * np.max(np.abs(x))
print("timeout reported, context usable")
"""


@pytest.mark.parametrize("task", [0, 2])
def test_stalled_dependency_times_out(zs_lib, task):
    env = dict(os.environ, ZS_TEST_STALL_FX_TASK=str(task))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert "timeout reported" in r.stdout
