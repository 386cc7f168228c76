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
