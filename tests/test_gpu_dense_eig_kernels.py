"""The fixed-point back-transformation by itself: columns in shared memory and in global memory (matrices of more than 12,800
rows), and the longest sums a thread forms there, with every product at its largest."""
import ctypes
import math
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(built, tmp_path_factory):
    import __graft_entry__ as g

    out = str(tmp_path_factory.mktemp("kernels") / "dense_eig_kernels.so")
    g._run([g._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
            "-I", g.CSRC, "-o", out, os.path.join(ROOT, "tests", "dense_eig_kernels.cu"), g.LIB,
            "-Xlinker", "-rpath=" + os.path.dirname(g.LIB), "-lcudart"])
    return ctypes.CDLL(out)


def _run(lib, v, n, ncol, tau, Zt, kc, in_smem, blocks):
    import torch

    torch.cuda.synchronize()
    exv = torch.zeros(n, dtype=torch.int32, device="cuda")
    Z = torch.empty((n, n), dtype=torch.complex128, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (v, tau, exv, Zt, Z)]
    assert lib.back_transform(p[0], n, ncol, p[1], p[2], p[3], p[4], kc, in_smem, blocks) == 0
    return Z


@pytest.mark.parametrize("n,kc", [(40, 1), (40, 8), (257, 3), (300, 5), (300, 16)])
def test_columns_in_global_memory(lib, n, kc):
    import torch

    rng = np.random.default_rng(n + kc)
    V = np.zeros((n - 1, n), dtype=complex)
    tau = np.zeros(n - 1, dtype=complex)
    for j in range(n - 1):
        V[j, j + 1] = 1.0
        V[j, j + 2:] = rng.uniform(-1, 1, n - j - 2) + 1j * rng.uniform(-1, 1, n - j - 2)
        tau[j] = 2.0 / np.vdot(V[j], V[j]).real
    Zt = np.linalg.qr(rng.normal(size=(n, n)))[0]
    ref = Zt.astype(complex)
    for j in range(n - 2, -1, -1):
        ref -= tau[j] * np.outer(V[j], V[j].conj() @ ref)
    t = [torch.tensor(x, device="cuda") for x in (tau, Zt)]
    blocks = (n + kc - 1) // kc
    Z = [_run(lib, torch.tensor(V, device="cuda"), n, n - 1, *t, kc, s, blocks).cpu().numpy() for s in (0, 1)]
    assert np.array_equal(Z[0], Z[1])
    # n reflectors, each within 2^-52 of the entry's and the product's exact value in units of a column's length
    assert np.abs(Z[0] - ref).max() <= 4 * n * 2.0 ** -52


def test_longest_sums(lib):
    import torch

    n, kc = 20000, 8  # 625 rows a thread
    c = (1 - 2.0 ** -30) * 2.0 ** -8  # v's high limb at its largest
    z = (2.0 ** 53 / 141 // 2 ** 32 * 2 ** 32 + 0x7fffff00) * 2.0 ** -60  # z's low limb at its largest
    tau = 2.0 / (1 + (n - 2) * c * c)
    V = torch.full((n,), c, dtype=torch.complex128, device="cuda")
    T = torch.zeros(n - 1, dtype=torch.complex128, device="cuda")
    T[0] = tau
    Zt = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    Zt[:, :kc] = z
    Z = _run(lib, V, n, 1, T, Zt, kc, 0, 1)[:, :kc].cpu().numpy()
    f = tau * math.fsum([z] + [c * z] * (n - 2))
    ref = np.full(n, z - c * f)
    ref[0], ref[1] = z, z - f
    # the sum to 2^-53, f to 2^-53 of itself twice, the update to 2^-61
    assert np.abs(Z - ref[:, None]).max() <= 4 * 2.0 ** -53 * max(abs(f), 1.0)
