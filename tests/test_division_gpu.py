"""The quantisers' quotients (quantize_common.cuh) against __fdiv_rn on the device, over all 2^23
significands: amax / 6 and sf / gs bit for bit, on both sides of every limit where they fall back to a
division, and the e2m1 values of x / step around every rounding boundary."""

import ctypes
import pathlib
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from mosaicist_b200 import build

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not pathlib.Path(nvcc).exists():
        pytest.skip("nvcc is needed to build the check")
    so = tmp_path_factory.mktemp("division") / "division_check.so"
    subprocess.run([nvcc, *build.ARCH, *build.COMMON, "-shared", "-Xcompiler", "-fPIC", "-cudart", "static", "-o", str(so),
                    str(HERE / "division_check.cu")], check=True, capture_output=True)
    lib = ctypes.CDLL(str(so))

    def run(which, exponent):
        bad, seen = ctypes.c_ulonglong(), ctypes.c_ulonglong()
        assert lib.division_check(which, exponent, ctypes.byref(bad), ctypes.byref(seen)) == 0
        return bad.value, seen.value

    return run


# biased exponents: 0 subnormals, 27 / 28 around 1e-30, 226 / 227 around 1e30, 254 the largest
@pytest.mark.parametrize("exponent", [0, 1, 2, 24, 26, 27, 28, 60, 126, 127, 128, 200, 225, 226, 227, 253, 254])
def test_amax_over_6(check, exponent):
    assert check(0, exponent) == (0, 1 << 23)


# 43 / 44 around 1e-25, 210 / 211 around 1e25
@pytest.mark.parametrize("exponent", [1, 20, 43, 44, 45, 100, 127, 128, 154, 209, 210, 211, 230, 254])
def test_scale_step(check, exponent):
    assert check(1, exponent) == (0, 127 << 23)


# steps down to 2^-100: below that the remainder is no longer exact in fp32
@pytest.mark.parametrize("exponent", [27, 60, 100, 117, 127, 137, 200, 240])
def test_packed_values(check, exponent):
    assert check(2, exponent) == (0, 128 << 23)
