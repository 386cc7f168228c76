"""The FP64 FFT contraction (k_fft64.cu) against the oracle's factored operator, over the transform lengths and mesh
shapes where its passes differ: one factor, two factors, unit dimensions, one to three dimensions, ragged batches of
planes, and the first mesh that does not fit (the product by the table)."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from oracle import wtb_oracle as O  # noqa: E402
from wtb_gb300 import api  # noqa: E402
from wtb_gb300.synthetic import BSEParams, make_system  # noqa: E402

pytestmark = pytest.mark.gpu

# (mesh, FFT form expected)
MESHES = [((1, 1, 1), True), ((2, 1, 1), True), ((1, 3, 1), True), ((3, 2, 1), True), ((8, 8, 1), True),
          ((9, 5, 1), True), ((1, 17, 13), True), ((24, 23, 1), True), ((45, 7, 1), True), ((31, 36, 1), True),
          ((120, 1, 1), True), ((121, 1, 1), False), ((2, 3, 4), True), ((5, 4, 6), True), ((9, 8, 7), True),
          ((3, 2, 30), True), ((13, 2, 10), True)]


@pytest.mark.parametrize("ngrid,fft", MESHES)
def test_operator_matches_the_oracle(built, ngrid, fft):
    three = ngrid[2] > 1
    s = make_system(5, 4, "cubic" if three else "hex", 2 if three else 3, 1.5, tuple(min(n, 6) for n in ngrid))
    p = BSEParams(ngrid=ngrid, nc=2, nv=1, coultype="V3DL" if three else "V2DRK", ediel=(1.0, 4.0, 1.0), r0=40.0, nev=1)
    ctx = api.Context(0)
    ctx.set_hr(s)
    ctx.bsesolver(p, precision="fp64", op="matfree")
    assert ctx.operator_form() == ("FP64 FFT convolution" if fft else "FP64 CUDA-core product")
    rng = np.random.default_rng(1)
    ncol = 3
    X = rng.normal(size=(p.dim, ncol)) + 1j * rng.normal(size=(p.dim, ncol))
    Y = ctx.bse_matvec(p, X, precision="fp64", op="matfree")
    kpt = O.monhkhorst_pack(*ngrid, p.mshift, s.rlat)
    eigv, vec, _ = O.bands(s, p, kpt)
    ref = O.bse_matvec_factored(X, eigv, O.gauge_fix(vec), kpt, p, s.rlat)
    # the transforms' rounding is a few log2(P) ulp of the column's norm, the bands 1e-13 relative
    assert np.linalg.norm(Y - ref) <= 1e-12 * np.linalg.norm(ref)
    ctx.close()


# every pruned first factor (2, 4, 8, 10, 16), with coprime second factors and with twiddles, on meshes of half the length
# and shorter, and twiddles without pruning
@pytest.mark.parametrize("ngrid", [(5, 1, 1), (18, 3, 1), (15, 4, 1), (20, 6, 1), (5, 5, 5), (4, 4, 10), (3, 50, 1),
                                   (3, 49, 1), (100, 2, 1), (64, 5, 1), (13, 4, 3)])
def test_pruned_and_twiddled_factors(built, ngrid):
    test_operator_matches_the_oracle(built, ngrid, True)


# one application and the adjoint's linear solves do not depend on the number of excitons, nor does the form they take
@pytest.mark.parametrize("nev", [6, 7, 12])
def test_applications_whatever_the_excitons(built, nev):
    s = make_system(5, 4, "hex", 3, 1.5, (6, 6, 1))
    p = BSEParams(ngrid=(9, 8, 1), nc=2, nv=1, coultype="V2DRK", ediel=(1.0, 4.0, 1.0), r0=40.0, nev=nev)
    ctx = api.Context(0)
    ctx.set_hr(s)
    ctx.bsesolver(p, precision="fp64", op="matfree")
    rng = np.random.default_rng(1)
    X = rng.normal(size=(p.dim, 3)) + 1j * rng.normal(size=(p.dim, 3))
    Y = ctx.bse_matvec(p, X, precision="fp64", op="matfree")
    assert ctx.operator_form() == "FP64 FFT convolution"
    p.nev = 1
    assert np.array_equal(Y, ctx.bse_matvec(p, X, precision="fp64", op="matfree"))
    p.nev = nev
    ctx.bsesolver(p, precision="fp64", op="matfree")
    ctx.bse_backward(p, np.ones(nev), np.ones(nev), precision="fp64")
    assert ctx.operator_form() == "FP64 FFT convolution"
    ctx.close()
