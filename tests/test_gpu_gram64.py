"""FP64 solves at the sizes where the FP64 Gram kernels change their work per thread (few, some and many reduction parts)
and where the block fills its largest basis, against the oracle's dense eigenvalues."""
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


# (mesh, nev, block): dims 128 (1 part), 392 (3 parts, 33 and 78 basis columns), 2,178 (12 parts)
@pytest.mark.parametrize("n,nev,block", [(8, 3, 0), (14, 5, 11), (14, 20, 26), (33, 4, 0)])
def test_lowest_energies(built, n, nev, block):
    s = make_system(7, 4, "hex", 3, 1.5, (6, 6, 1))
    p = BSEParams(ngrid=(n, n, 1), nc=2, nv=1, coultype="V2DRK", r0=40.0, nev=nev)
    ctx = api.Context(0)
    ctx.set_hr(s)
    E = ctx.bsesolver(p, precision="fp64", op="dense", block=block)["E"]
    kpt = O.monhkhorst_pack(n, n, 1, p.mshift, s.rlat)
    eigv, vec, _ = O.bands(s, p, kpt)
    ref = np.linalg.eigvalsh(O.bse_build(eigv, O.gauge_fix(vec), kpt, p, s.rlat))[:nev]
    # residuals of 1e-8 relative leave the eigenvalues within their squares; 1e-9 eV is the repository's bound
    assert np.abs(E - ref).max() <= 1e-9
    ctx.close()


# the upper triangles alone (FFT form of the contraction): 3 b columns with b = 1, 7, 16, 26, few and many reduction
# parts, two and three dimensions
@pytest.mark.parametrize("ngrid,nev,block", [((8, 8, 1), 1, 1), ((14, 14, 1), 3, 7), ((14, 14, 1), 6, 16),
                                             ((33, 30, 1), 4, 26), ((6, 5, 4), 9, 0)])
def test_upper_triangles(built, ngrid, nev, block):
    three = ngrid[2] > 1
    s = make_system(7, 4, "cubic" if three else "hex", 2 if three else 3, 1.5, tuple(min(n, 6) for n in ngrid))
    p = BSEParams(ngrid=ngrid, nc=2, nv=1, coultype="V3DL" if three else "V2DRK", ediel=(1.0, 4.0, 1.0), r0=40.0, nev=nev)
    ctx = api.Context(0)
    ctx.set_hr(s)
    E = ctx.bsesolver(p, precision="fp64", op="matfree", block=block)["E"]
    assert ctx.operator_form() == "FP64 FFT convolution"
    ctx.close()
    kpt = O.monhkhorst_pack(*ngrid, p.mshift, s.rlat)
    eigv, vec, _ = O.bands(s, p, kpt)
    ref = np.linalg.eigvalsh(O.bse_build(eigv, O.gauge_fix(vec), kpt, p, s.rlat))[:nev]
    # as above
    assert np.abs(E - ref).max() <= 1e-9
