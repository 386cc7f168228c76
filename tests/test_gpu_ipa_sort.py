"""The IPA records' stable sort around the rows of a CTA (512) and the keys of a tile (2,048), with ties (k and -k), and the
broadened sums around the rows of a statistics block (2,048) and of a staged tile, with energies on a photon energy."""
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
SYS = make_system(7, 4, "hex", 3, 1.5, (6, 6, 1))


@pytest.mark.parametrize("nk,nc,nv", [(1, 1, 1), (7, 2, 1), (511, 1, 1), (512, 1, 1), (513, 1, 1), (512, 2, 1),
                                      (1025, 1, 1), (2049, 1, 1), (1500, 2, 2)])
def test_stable_sort(built, nk, nc, nv):
    p = BSEParams(ngrid=(nk, 1, 1), nc=nc, nv=nv, coultype="V2DRK", r0=40.0, nev=1)
    ctx = api.Context(0)
    ctx.set_hr(SYS)
    rec = ctx.spoptics(p)
    ctx.close()
    kpt = O.monhkhorst_pack(nk, 1, 1, p.mshift, SYS.rlat).astype(np.float32)
    where = {tuple(k): i for i, k in enumerate(kpt)}
    no = rec[:, 3].astype(int)
    c, v = rec[:, 4].astype(int) - no - 1, rec[:, 5].astype(int) - no + nv - 1
    index = (np.array([where[tuple(r[:3])] for r in rec]) * nc + c) * nv + v
    assert np.array_equal(np.sort(index), np.arange(p.dim))
    step, key = np.diff(index), np.diff(rec[:, 6])
    assert np.all((key > 0) | ((key == 0) & (step > 0)))


@pytest.mark.parametrize("n", [1, 2, 255, 257, 2047, 2048, 2049, 6001])
def test_broadened_sums(built, n):
    rng = np.random.default_rng(n)
    p = BSEParams(ngrid=(8, 8, 1), nc=2, nv=1, coultype="V2DRK", r0=40.0, nev=1)
    p.numbse, p.ebse0, p.ebsef, p.renorm = 129, 0.0, 8.0, False
    esp = np.sort(rng.uniform(1.0, 9.0, n))
    esp[n // 2] = 4.0  # on a photon energy
    esp = np.sort(esp)
    acts = {c: rng.uniform(0.0, 1.0, n) for c in O.COMPONENTS}
    ctx = api.Context(0)
    ctx.set_hr(SYS)
    d = ctx.spdielraw(p, esp, acts)
    ctx.close()
    ref = O.spdielraw(esp, acts, p.ngrid, SYS.rlat, p)
    for c in O.COMPONENTS:
        # the bound of the repository's other comparison of these sums
        np.testing.assert_allclose(d[c], ref[c], rtol=1e-10, atol=1e-12 * max(1.0, np.abs(ref[c]).max()))
