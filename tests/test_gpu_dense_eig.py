"""The dense Hermitian eigensolver at the edges of its tiles (64) and panels (32), on matrices that reach its special
cases: reducible ones, zero columns (reflectors that do nothing), low rank, entries of very different sizes.  Against
LAPACK; the bound is the backward error of a stable reduction, n eps ||A|| for the eigenvalues and 8 sqrt(n) eps ||A||_F
for the residuals."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from wtb_gb300 import api  # noqa: E402

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def matrix(n, kind):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    A = (X + X.conj().T) / 2
    if kind == "dominant":
        return 1e-3 * A + np.diag(rng.uniform(1.5, 8.0, n))
    if kind == "graded":
        s = 10.0 ** rng.uniform(-8.0, 0.0, n)
        return A * s[:, None] * s[None]
    if kind == "low rank":
        return X[:, :3] @ X[:, :3].conj().T
    if kind == "reducible":
        A[: n // 2, n // 2:] = 0.0
        A[n // 2:, : n // 2] = 0.0
    if kind == "diagonal":
        return np.diag(rng.normal(size=n)).astype(complex)
    return np.zeros_like(A) if kind == "zero" else A


@pytest.mark.parametrize("kind", ["random", "dominant", "graded", "low rank", "reducible", "diagonal", "zero"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 34, 64, 65, 66, 97, 129, 200])
def test_eigenvalues(ctx, n, kind):
    A = matrix(n, kind)
    W, ref = ctx.zheev(A), np.linalg.eigvalsh(A)
    assert np.abs(W - ref).max() <= max(n, 4) * EPS * np.abs(ref).max() + 1e-300


@pytest.mark.parametrize("kind", ["random", "dominant", "reducible"])
@pytest.mark.parametrize("n", [2, 33, 65, 200, 333])
def test_eigenpairs(ctx, n, kind):
    A = matrix(n, kind)
    W, Z = ctx.zheev_vectors(A)
    nrm = np.linalg.norm(A)
    assert np.linalg.norm(A @ Z - Z * W) <= 8.0 * np.sqrt(n) * EPS * nrm
    # eigenvectors of values closer than 1e-7 ||A|| are orthogonalised, the others by their gaps (eps / 1e-7)
    assert np.abs(Z.conj().T @ Z - np.eye(n)).max() <= 1e-8


@pytest.mark.parametrize("scale", [1e-154, 1e-150, 1e-100, 1e150])
@pytest.mark.parametrize("n", [33, 130])
def test_scaled_eigenvalues(ctx, n, scale):
    A = matrix(n, "random") * scale
    W, ref = ctx.zheev(A), np.linalg.eigvalsh(A)
    assert np.abs(W - ref).max() <= n * EPS * np.abs(ref).max()


# columns a CTA of the back-transformation and slices of a column: 1 and 256, 2 and 128, 3 and 85 (no multiple of the eight
# lanes that add them up)
@pytest.mark.parametrize("n", [608, 609, 1216, 1217, 1300, 1368])
def test_eigenpairs_by_columns_a_block(ctx, n):
    test_eigenpairs(ctx, n, "random")


# A row c without couplings and rows [[c, b], [b, a]], c one of the points at which the bisection for the pair's upper
# eigenvalue counts: both pivots there are zero exactly.  (c, b, a), beside rows 1 and -1.
@pytest.mark.parametrize("c,b,a", [("0x1.187f742108421p-3", "0x1p-10", "-0x1.23c53b869337cp-4"),
                                   ("0x1.83600b18c6319p-7", "0x1p-11", "-0x1.bc6fe52111fc6p-3"),
                                   ("0x1.c5b08aa5294a5p-2", "0x1p-11", "0x1.87a34f57a09a0p-5"),
                                   ("0x1.38a4315ad6b5bp-5", "0x1p-10", "-0x1.e29bfe55f4160p-3")])
def test_counts_at_two_zero_pivots(ctx, c, b, a):
    c, b, a = (float.fromhex(x) for x in (c, b, a))
    A = np.diag([1.0, -1.0, c, c, a]).astype(complex)
    A[3, 4] = A[4, 3] = b
    W, ref = ctx.zheev(A), np.linalg.eigvalsh(A)
    assert np.abs(W - ref).max() <= 5 * EPS * np.abs(ref).max()


# Eigenvalues +-g/2 of rows [[0, g/2], [g/2, 0]] beside an uncoupled row 1.  The reduction changes nothing, and the rounding of
# the elimination is an ulp of g, so each vector is that of the matrix with its last diagonal entry off by at most the
# smallest pivot, 2^-56 of the norm, which turns it by half of that over g; 64 ulp for the normalisation and the rest.
@pytest.mark.parametrize("g", [3e-7, 5e-7, 1e-6, 2e-6, 3e-6, 5e-6, 7e-6, 1e-5, 2e-5, 4e-5])
def test_vectors_of_close_eigenvalues(ctx, g):
    A = np.diag([1.0, 0.0, 0.0]).astype(complex)
    A[1, 2] = A[2, 1] = g / 2
    Z = np.asarray(ctx.zheev_vectors(A)[1])
    assert np.abs(Z.conj().T @ Z - np.eye(3)).max() <= 2.0 ** -56 * (1 + 1e-12) / g + 64 * EPS
