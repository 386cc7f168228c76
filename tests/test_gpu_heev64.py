"""FP64 projected eigenproblems where their kernel changes: the smallest, columns that do not fill the cluster's CTAs or
warps, the largest block, and the most systems of which each gets a cluster and one more."""
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


def _system(n, nev):
    s = make_system(7, 4, "hex", 3, 1.5, (6, 6, 1))
    return s, BSEParams(ngrid=(n, n, 1), nc=2, nv=1, coultype="V2DRK", r0=40.0, nev=nev)


def _dense(s, p):
    n = p.ngrid[0]
    kpt = O.monhkhorst_pack(n, n, 1, p.mshift, s.rlat)
    eigv, vec, _ = O.bands(s, p, kpt)
    return np.linalg.eigvalsh(O.bse_build(eigv, O.gauge_fix(vec), kpt, p, s.rlat))


# block b: up to 3 b columns
@pytest.mark.parametrize("nev,block", [(1, 1), (1, 3), (2, 7), (3, 11), (8, 16), (20, 25), (20, 26)])
def test_lowest_energies(built, nev, block):
    s, p = _system(14, nev)
    ctx = api.Context(0)
    ctx.set_hr(s)
    E = ctx.bsesolver(p, precision="fp64", op="dense", block=block)["E"]
    ctx.close()
    # residuals of 1e-8 relative leave the eigenvalues within their squares; 1e-9 eV is the repository's bound
    assert np.abs(E - _dense(s, p)[:nev]).max() <= 1e-9


@pytest.mark.parametrize("nsys", [19, 20])
def test_joint_batch(built, nsys):
    s, p = _system(8, 3)
    b = api.Batch(0, nworkers=1)
    try:
        out, _ = b.bsesolver([(s, p)] * nsys, precision="fp64", op="matfree")
    finally:
        b.close()
    ref = _dense(s, p)[:3]
    for o in out:
        assert o["status"] == 0
        assert np.abs(o["E"] - ref).max() <= 1e-9
