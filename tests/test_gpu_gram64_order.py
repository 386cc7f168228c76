"""The FP64 Grams' order of operations: whatever the work per thread (two entries, one, a component, single warps), a part's
sums are the same chain of fused multiply-adds over its rows, and the parts are added in the same order, so the bits do
not depend on it.  The chain is restated with exact rational products, rounded once per step."""
import ctypes
import os
import sys
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(built, tmp_path_factory):
    import __graft_entry__ as g

    out = str(tmp_path_factory.mktemp("kernels") / "gram_kernels.so")
    g._run([g._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
            "-I", g.CSRC, "-o", out, os.path.join(ROOT, "tests", "gram_kernels.cu"), g.LIB,
            "-Xlinker", "-rpath=" + os.path.dirname(g.LIB), "-lcudart"])
    return ctypes.CDLL(out)


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def chain(A, B):
    """A^H B of one part's rows"""
    out = np.zeros((A.shape[1], B.shape[1]), dtype=complex)
    for i in range(A.shape[1]):
        for j in range(B.shape[1]):
            re = im = 0.0
            for a, b in zip(A[:, i], B[:, j]):
                re = fma(a.imag, b.imag, fma(a.real, b.real, re))
                im = fma(-a.imag, b.real, fma(a.real, b.imag, im))
            out[i, j] = complex(re, im)
    return out


def added(parts):
    """the parts' sums: every eighth part in order, then the eight in order"""
    total = np.zeros(parts.shape[1:], dtype=complex)
    for w in range(8):
        s = np.zeros(parts.shape[1:], dtype=complex)
        for b in range(w, len(parts), 8):
            s = s + parts[b]
        total = total + s
    return total


def _data(nrow, p, q):
    rng = np.random.default_rng(nrow + p)
    f = lambda k: rng.normal(size=(nrow, k)) + 1j * rng.normal(size=(nrow, k))  # noqa: E731
    return f(p), f(q)


def _dev(*arrays):
    import torch

    t = [torch.tensor(a, device="cuda") for a in arrays]
    torch.cuda.synchronize()
    return t


def _check(parts, A, B, npart, upper=False):
    per = -(-len(A) // npart)
    for b in sorted({0, 1, npart // 2, npart - 1}):
        ref = chain(A[b * per:(b + 1) * per], B[b * per:(b + 1) * per])
        got = np.triu(parts[b]) if upper else parts[b]
        assert np.array_equal(got, np.triu(ref) if upper else ref), b


# parts: two entries a thread from 1,216 on, one from 912, components from 9,728 entries in all, else single warps
@pytest.mark.parametrize("npart,nrow", [(1216, 2432), (1000, 2999), (700, 2100), (3, 97)])
def test_gram(lib, npart, nrow):
    p, q = 4, 5
    A, B = _data(nrow, p, q)
    a, b, out, partial = _dev(A, B, np.zeros((p, q), dtype=complex), np.zeros((npart, p, q), dtype=complex))
    assert lib.gram64(*(ctypes.c_void_p(x.data_ptr()) if hasattr(x, "data_ptr") else x
                        for x in (a, p, b, q, nrow, npart, out, partial))) == 0
    parts = partial.cpu().numpy()
    _check(parts, A, B, npart)
    assert np.array_equal(out.cpu().numpy(), added(parts))


@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("npart,nrow", [(1216, 2432), (1000, 2999), (700, 2100), (3, 97)])
def test_pair(lib, npart, nrow, upper):
    p = 4
    A, B = _data(nrow, p, p)
    z = np.zeros((p, p), dtype=complex)
    a, b, M, G, partial = _dev(A, B, z, z, np.zeros((2, npart, p, p), dtype=complex))
    assert lib.gram_pair64(*(ctypes.c_void_p(x.data_ptr()) if hasattr(x, "data_ptr") else x
                             for x in (a, b, p, nrow, npart, int(upper), M, G, partial))) == 0
    for X, C, parts in ((A, M, partial[0].cpu().numpy()), (B, G, partial[1].cpu().numpy())):
        _check(parts, A, X, npart, upper)
        ref, got = added(parts), C.cpu().numpy()
        if upper:
            assert np.array_equal(np.triu(got), np.triu(ref))
            assert np.array_equal(np.tril(got, -1), np.triu(ref, 1).conj().T)
        else:
            assert np.array_equal(got, ref)
