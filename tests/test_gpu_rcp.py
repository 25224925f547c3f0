"""The FP64 reciprocal of the evaluation and the 2x2 solves (nurbs_math.cuh: fast::rcp)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

_dp = np.ctypeslib.ndpointer(dtype=np.float64, flags="C_CONTIGUOUS")


@pytest.fixture(scope="module")
def rcp(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("rcp") / "librcp.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "gpu-nurbs_gb300", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "rcp_check.cu")], check=True, capture_output=True)
    f = C.CDLL(out).rcp_check
    f.argtypes = [_dp, _dp, C.c_longlong]

    def call(x):
        x = np.ascontiguousarray(x, np.float64)
        y = np.empty_like(x)
        assert f(x, y, len(x)) == 0
        return y

    return call


def mantissas():
    m = np.random.default_rng(1).integers(0, 1 << 52, 1 << 18, dtype=np.uint64)
    m[: 1 << 16] |= np.uint64(0xffffffff)            # the approximation ignores the low word
    m[1 << 16: 1 << 17] &= ~np.uint64(0xffffffff)
    m[-4:] = [0, 1, (1 << 52) - 1, (1 << 52) - 2]
    return m


@pytest.mark.parametrize("exponent", [8, 9, 400, 1022, 1023, 1024, 1700, 2036, 2037])
def test_error(rcp, exponent):
    """An approximation to 2^-20 and a third-order step: 2^-60, 2^-7 ulp, before the last rounding."""
    x = (mantissas() | np.uint64(exponent << 52)).view(np.float64)
    y = rcp(x)
    scaled = np.ldexp(x, 1023 - exponent), np.ldexp(y, exponent - 1023)
    e = np.abs(scaled[0].astype(np.longdouble) * scaled[1].astype(np.longdouble) - 1)
    assert float((e / scaled[0] / np.spacing(scaled[1])).max()) <= 0.5 + 2.0 ** -7
    assert np.array_equal(rcp(-x), -y)


@pytest.mark.parametrize("exponent", [0, 1, 6, 7, 2038, 2039, 2046])
def test_ends_of_the_exponent_range(rcp, exponent):
    x = (mantissas() | np.uint64(exponent << 52)).view(np.float64)
    with np.errstate(all="ignore"):
        for s in (x, -x):
            assert np.array_equal(rcp(s), 1.0 / s)


def test_special_values(rcp):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324])
    with np.errstate(all="ignore"):
        want = 1.0 / x
    got = rcp(x)
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.signbit(got[:4]), np.signbit(want[:4]))
