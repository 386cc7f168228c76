"""The broadened sums' reciprocal: within an ulp of the division inside its range, the division itself outside."""
import ctypes
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu
LOW, HIGH = 2.0 ** -1007, 2.0 ** 993  # the range of the Newton step


@pytest.fixture(scope="module")
def lib(built, tmp_path_factory):
    import __graft_entry__ as g

    out = str(tmp_path_factory.mktemp("kernels") / "spectrum_kernels.so")
    g._run([g._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
            "-I", g.CSRC, "-o", out, os.path.join(ROOT, "tests", "spectrum_kernels.cu"), g.LIB,
            "-Xlinker", "-rpath=" + os.path.dirname(g.LIB), "-lcudart"])
    return ctypes.CDLL(out)


def _both(lib, x):
    import torch

    x = torch.tensor(x, dtype=torch.float64, device="cuda")
    r, q = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    assert lib.reciprocals(*(ctypes.c_void_p(t.data_ptr()) if k != 1 else t for k, t in enumerate((x, len(x), r, q)))) == 0
    return r.cpu().numpy(), q.cpu().numpy()


@pytest.mark.parametrize("exponents", [(-1007, 992), (-20, 20), (0, 0)])
def test_within_an_ulp(lib, exponents):
    rng = np.random.default_rng(exponents[0] + 5000)
    n = 1 << 20
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(exponents[0], exponents[1] + 1, n))
    x[:4] = np.ldexp([1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5], exponents[0])
    r, q = _both(lib, x)
    assert np.array_equal(q, 1.0 / x)
    assert np.all(np.abs(r - q) <= np.spacing(q))


def test_outside_the_range(lib):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, np.nextafter(LOW, 0.0), HIGH, 1e308, -1.0, -3.0, -1e-320])
    r, q = _both(lib, x)
    assert np.array_equal(r, q, equal_nan=True)
    r, q = _both(lib, [LOW, np.nextafter(HIGH, 0.0)])
    assert np.all(np.abs(r - q) <= np.spacing(q))
