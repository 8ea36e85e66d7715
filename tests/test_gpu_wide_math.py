"""The wide rows' arithmetic (sampler_wide_math.cuh) on the device, bit for bit against what the multi-pass path
computes: a row's probabilities must not depend on the path it took, and a draw shows a last bit only where it lands on one."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import to_dev

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


@pytest.mark.parametrize("near", [False, True])
def test_quotients(lib, near):
    """(float) ((double) e / S) with e in (1e-14, 1] and S in [1, 2^21], what a row of up to 2^21 columns can have; and where
    the quotient lies within 2^-53 of itself of the midpoint of two floats, powers of two among those."""
    import torch
    rng = np.random.default_rng(31)
    n = 1 << 22
    e = np.exp(-rng.uniform(0.0, 32.0, n)).astype(np.float32)
    e[:1000] = 1.0
    S = np.exp2(rng.uniform(0.0, 21.0, n))
    if near:
        p = (e / S).astype(np.float32)
        p[::7] = np.exp2(np.floor(np.log2(p[::7])))
        side = np.where(rng.random(n) < 0.5, np.float32(0.0), np.float32(np.inf))
        mid = (p.astype(np.float64) + np.nextafter(p, side).astype(np.float64)) * 0.5
        S = e.astype(np.float64) / mid
        S = np.where(rng.random(n) < 0.5, S, np.nextafter(S, np.where(rng.random(n) < 0.5, 0.0, np.inf)))
    got, unsure = torch.empty(n, dtype=torch.float32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    de, dS = to_dev(e), to_dev(S)
    torch.cuda.synchronize()
    assert lib.quotients(*(C.c_void_p(t.data_ptr()) for t in (de, dS, got, unsure)), n) == 0
    want = (e.astype(np.float64) / S).astype(np.float32)
    differ = np.nonzero(got.cpu().numpy().view(np.uint32) != want.view(np.uint32))[0]
    assert differ.size == 0, (differ.size, e[differ[:4]], S[differ[:4]])
    # 2^-43 of the quotients' range, of 2^-23 between two floats, wants the division
    assert int(unsure) == n if near else int(unsure) < 64
