"""The FP64 contraction's form on both sides of each bound of its rule, and what the FFT gives for many excitons against the
product: a 2D mesh just above 1,800 points, a thin 3D slab, a 3D mesh.

The bounds: both forms' energies are within the squares of their residuals (1e-8 relative) of the operator's, 1e-9 eV; a
residual of 1e-8 of the energy turns a vector by that over its gap, so activities of separate excitons agree to
2 * 1e-8 E / gap, here with gaps of 1e-3 eV and E of a few eV, 1e-4 of the largest."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from wtb_gb300 import api  # noqa: E402
from wtb_gb300.synthetic import BSEParams, make_system  # noqa: E402

pytestmark = pytest.mark.gpu
FFT, PRODUCT = "FP64 FFT convolution", "FP64 CUDA-core product"


def _case(ngrid, nev):
    three = ngrid[2] > 1
    s = make_system(5, 4, "cubic" if three else "hex", 2 if three else 3, 1.5, tuple(min(n, 6) for n in ngrid))
    p = BSEParams(ngrid=ngrid, nc=1, nv=1, coultype="V3DL" if three else "V2DRK", ediel=(1.0, 4.0, 1.0), r0=40.0, nev=nev)
    return s, p


def _solve(ngrid, nev):
    s, p = _case(ngrid, nev)
    ctx = api.Context(0)
    ctx.set_hr(s)
    r = ctx.bsesolver(p, precision="fp64", op="matfree")
    form = ctx.operator_form()
    ctx.close()
    return r, form


@pytest.mark.parametrize("ngrid,nev,form", [
    ((9, 8, 1), 6, FFT), ((9, 8, 1), 7, PRODUCT),            # excitons
    ((45, 40, 1), 7, FFT), ((46, 39, 1), 7, PRODUCT),        # 1,800 points and 1,794
    ((9, 8, 2), 7, FFT), ((9, 8, 1), 12, PRODUCT),           # three dimensions
    ((80, 80, 1), 1, FFT), ((81, 81, 1), 1, PRODUCT),        # the largest square mesh that fits one CTA
    ((18, 18, 18), 1, FFT), ((19, 19, 19), 1, PRODUCT),      # the largest cube
])
def test_form(built, ngrid, nev, form):
    assert _solve(ngrid, nev)[1] == form


@pytest.mark.parametrize("ngrid,nev", [((43, 42, 1), 12), ((24, 24, 2), 14), ((11, 10, 9), 12)])
def test_many_excitons(built, ngrid, nev, tmp_path):
    r, form = _solve(ngrid, nev)
    assert form == FFT
    out = str(tmp_path / "product.npz")
    code = ("import sys; sys.path.insert(0, %r); import numpy as np; from tests.test_gpu_forms64 import _solve, PRODUCT\n"
            "r, form = _solve(%r, %d); assert form == PRODUCT\n"
            "np.savez(%r, E=r['E'], **r['acts'])" % (ROOT, ngrid, nev, out))
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, WTB_FFT="0"))
    ref = np.load(out)
    assert np.abs(r["E"] - ref["E"]).max() <= 1e-9
    gap = np.diff(ref["E"])
    apart = np.flatnonzero(np.minimum(np.append(np.inf, gap[:-1]), gap) >= 1e-3)  # of the excitons but the last
    assert len(apart)
    for c in api.COMPONENTS:
        assert np.abs(r["acts"][c] - ref[c])[apart].max() <= 1e-4 * max(np.abs(ref[c]).max(), 1e-300), c
