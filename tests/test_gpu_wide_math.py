"""The wide rows' arithmetic (sampler_wide_math.cuh) on the device, bit for bit against what the multi-pass path
computes: a row's probabilities must not depend on the path it took, and a draw shows a last bit only where it lands on one."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("wide_math") / "wide_math.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared",
                    "-o", str(so), str(HERE / "wide_math.cu")], check=True)
    return C.CDLL(str(so))


def test_every_exponential(lib):
    """All floats from -0 to -130, denormal arguments and results and what the clamp at -120 takes among them; and -inf."""
    for first, last in ((np.float32(0.0), np.float32(130.0)), (np.float32(np.inf), np.float32(np.inf))):
        a, b = (int(v.view(np.uint32)) for v in (first, last))
        differ, which = C.c_ulonglong(), C.c_uint()
        assert lib.exp_differs(C.c_uint(a), C.c_uint(b - a + 1), C.byref(differ), C.byref(which)) == 0
        assert differ.value == 0, (differ.value, -np.uint32(which.value).view(np.float32))


def test_every_mass(lib):
    """All floats from 0 to 1 as 64-bit masses in units of 2^-62."""
    differ = C.c_ulonglong()
    assert lib.mass_differs(C.c_uint(int(np.float32(1.0).view(np.uint32))), C.byref(differ)) == 0
    assert differ.value == 0
