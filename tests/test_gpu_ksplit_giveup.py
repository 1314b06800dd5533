"""A K-split GEMM whose bounded wait runs out leaves C alone.

The kernel is built once more with a wait limit of 2 ms (ksplit_giveup.cu) and
run on one tile of two CTAs: with whole loads it adds the product, with loads
that bring fewer bytes than a stage's barrier expects the wait expires, the
status word says so, and no share that was never put is added into C.
"""
import ctypes as ct
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
ERR_TIMEOUT = 4  # PHPC_ERR_TIMEOUT


@pytest.fixture(scope="module")
def ksplit_tile(built, tmp_path_factory):
    import build

    so = tmp_path_factory.mktemp("ksplit") / "ksplit_giveup.so"
    subprocess.run([build.NVCC, *build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-DPHPC_WAIT_LIMIT_NS=2000000ull", f"-I{build.INC}", f"-I{build.CSRC}",
                    str(HERE / "ksplit_giveup.cu"), str(build.CSRC / "runtime.cu"), "-o", str(so)], check=True)
    f = ct.CDLL(str(so)).ksplit_tile
    f.argtypes = [ct.c_int, ct.c_void_p, ct.POINTER(ct.c_int)]
    f.restype = ct.c_int
    return f


@pytest.mark.parametrize("short_rows", [0, 8])
def test_a_missing_share_is_not_added(ksplit_tile, torch_cuda, short_rows):
    c0 = np.arange(128 * 128, dtype=np.float32).reshape(128, 128)
    c, status = c0.copy(), ct.c_int(-1)
    assert ksplit_tile(short_rows, c.ctypes.data, ct.byref(status)) == 0
    if short_rows:
        assert status.value & 0xFF == ERR_TIMEOUT
        np.testing.assert_array_equal(c, c0)
    else:
        assert status.value == 0
        np.testing.assert_array_equal(c, c0 + 6 * 512)
