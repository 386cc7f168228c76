"""The back-transformation's columns a block are a rule on the size: few bounds, not a choice that flips from size to size."""
import ctypes
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_columns_a_block(built, tmp_path):
    import __graft_entry__ as g

    out = str(tmp_path / "dense_eig_kernels.so")
    g._run([g._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
            "-I", g.CSRC, "-o", out, os.path.join(ROOT, "tests", "dense_eig_kernels.cu"), g.LIB,
            "-Xlinker", "-rpath=" + os.path.dirname(g.LIB), "-lcudart"])
    lib = ctypes.CDLL(out)
    kc = [lib.block_columns(n) for n in range(1, 12802)]
    assert kc[-1] == 0 and min(kc[:-1]) >= 1  # 200 KB hold a column of 12,800 rows
    assert sum(a != b for a, b in zip(kc, kc[1:])) <= 8
