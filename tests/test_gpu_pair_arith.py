"""The packed arithmetic (csrc/rsf_pair.cuh) against the correctly rounded intrinsics and the scalar
arithmetic: reciprocal, square root, delta and H over every bit pattern of their ranges, quotient and
normals over random arguments with the ends of every guard among them.  The kernels' bit-exactness rests
on these, and on the device's approximations that they correct."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RCP, SQRT, DIRAC, HEAVISIDE, DIV, NORMALS = range(6)


def _bits(v):
    return int(np.float32(v).view(np.uint32))


@pytest.fixture(scope="module")
def sweep(cuda, rsflib, tmp_path_factory):
    from rsf_gb300 import build

    so = tmp_path_factory.mktemp("pair") / "pair_arith.so"
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", str(Path(__file__).with_name("pair_arith.cu")), "-o", str(so),
                    "-lcudart"], check=True, capture_output=True)
    fn = ctypes.CDLL(str(so)).pair_sweep
    fn.restype = ctypes.c_longlong
    fn.argtypes = [ctypes.c_int, ctypes.c_uint, ctypes.c_uint, ctypes.c_ulonglong, ctypes.c_float,
                   ctypes.POINTER(ctypes.c_float)]

    def run(what, lo, hi, n, eps=1.0):
        arg = (ctypes.c_float * 3)()
        bad = fn(what, lo, hi, n, eps, arg)
        assert bad == 0, (bad, [float(v).hex() for v in arg])

    return run


def test_reciprocal(sweep):
    lo, hi = _bits(2.0 ** -126), _bits(2.0 ** 126)
    sweep(RCP, lo, 0, hi - lo + 1)
    sweep(RCP, lo | 0x80000000, 0, hi - lo + 1)


def test_square_root(sweep):
    lo = _bits(2.0 ** -102)
    sweep(SQRT, lo, 0, 0x7f800000 - lo)
    sweep(SQRT, 0, 0, 1)


EPS = [1.0, 0.2, 0.1, 1e-3, 7.3, 2.0 ** -20, 2.0 ** 20, 1.9999999, 3e-8, 1e-12, 5e6]


@pytest.mark.parametrize("eps", EPS)
def test_delta_and_heaviside(eps, sweep):
    for sign in (0, 0x80000000):
        sweep(DIRAC, sign, 0, _bits(2.0 ** 59) + 1, eps)  # beyond, delta's denominator is held (see dirac2)
        sweep(HEAVISIDE, sign, 0, 0x80000000, eps)  # infinities and NaNs too


# exponent fields: everything, the ordinary range, and both sides of the guards at 2^-100 and 2^120
RANGES = [(0, 255), (100, 140), (20, 34), (1, 60), (240, 255), (118, 136)]


@pytest.mark.parametrize("lo,hi", RANGES)
def test_quotient(lo, hi, sweep):
    sweep(DIV, lo, hi, 1 << 30)


@pytest.mark.parametrize("lo,hi", RANGES + [(74, 80), (60, 90)])
def test_normals(lo, hi, sweep):
    sweep(NORMALS, lo, hi, 1 << 29)
