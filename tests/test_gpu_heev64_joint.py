"""The FP64 projected eigenproblem of many systems in one launch, more than there are clusters of SMs, against each system
by itself (the same bits) and against LAPACK."""
import ctypes
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(built, tmp_path_factory):
    import __graft_entry__ as g

    out = str(tmp_path_factory.mktemp("kernels") / "heev_kernels.so")
    g._run([g._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
            "-I", g.CSRC, "-o", out, os.path.join(ROOT, "tests", "heev_kernels.cu"), g.LIB,
            "-Xlinker", "-rpath=" + os.path.dirname(g.LIB), "-lcudart"])
    return ctypes.CDLL(out)


def _run(lib, A, nwant):
    import torch

    nsys, n = A.shape[:2]
    a = torch.tensor(A, device="cuda")
    E = torch.empty((nsys, nwant), dtype=torch.float64, device="cuda")
    V = torch.empty((nsys, n, nwant), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (a, E, V)]
    assert lib.heev64(p[0], n, nwant, nsys, p[1], p[2]) == 0
    return E.cpu().numpy(), V.cpu().numpy()


@pytest.mark.parametrize("n,nwant", [(1, 1), (3, 3), (33, 11), (48, 16), (78, 26)])
@pytest.mark.parametrize("nsys", [19, 20, 64])
def test_joint_and_single(lib, n, nwant, nsys):
    rng = np.random.default_rng(n + nsys)
    X = rng.normal(size=(nsys, n, n)) + 1j * rng.normal(size=(nsys, n, n))
    A = X + X.conj().transpose(0, 2, 1)
    E, V = _run(lib, A, nwant)
    for q in range(nsys):
        e, v = _run(lib, A[q:q + 1], nwant)
        assert np.array_equal(e[0], E[q]) and np.array_equal(v[0], V[q])
    ref = np.linalg.eigvalsh(A)[:, :nwant]
    nrm = np.linalg.norm(A, axis=(1, 2))
    eps = np.finfo(float).eps
    # a stable reduction: n eps ||A|| for the eigenvalues, 8 sqrt(n) eps ||A||_F for the residuals
    assert np.all(np.abs(E - ref).max(1) <= max(n, 4) * eps * nrm)
    res = np.linalg.norm(A @ V - V * E[:, None], axis=(1, 2))
    assert np.all(res <= 8 * np.sqrt(n) * np.sqrt(nwant) * eps * nrm)
