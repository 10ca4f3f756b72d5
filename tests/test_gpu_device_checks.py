"""What the kernels' comments claim of their arithmetic, on the GPU: the FP32 roundings
without range tests against CUDA's correctly rounded operations (every FP32 argument, every
quotient near the middle of two numbers), the FP64 operations of the integer pipe against
the FP64 pipe, and the FP64 draws that decide in FP32 against the FP64 methods, from the
same stream, bit for bit.
"""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


class Result(ctypes.Structure):
    _fields_ = [("n", ctypes.c_ulonglong), ("bad", ctypes.c_ulonglong), ("aux", ctypes.c_ulonglong),
                ("worst", ctypes.c_float), ("where", ctypes.c_uint)]


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    from trophic_maelstorm_gb300 import build
    so = str(tmp_path_factory.mktemp("checks") / "checks.so")
    cmd = [build.nvcc()] + build.ARCH + build.NVFLAGS + ["-I", build.CSRC, "-shared", "-o", so,
                                                         os.path.join(HERE, "device_checks.cu"), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)

    def run(name, a=0, b=0):
        out = Result()
        rc = getattr(lib, "chk_" + name)(ctypes.byref(out), ctypes.c_ulonglong(a), ctypes.c_ulonglong(b))
        assert rc == 0, (name, rc)
        assert out.bad == 0, (name, out.bad, out.n, hex(out.where))
        return out
    return run


def test_reciprocal_of_every_float(checks):
    r = checks("reciprocals")
    assert r.aux == 0                                  # none between 2^-100 and 2^100 is handed on
    assert r.n > 2 * 200 * 2 ** 23


def test_inverse_square_root_of_every_float_from_1(checks):
    assert checks("inv_sqrt").n == 128 * 2 ** 23


def test_quotients(checks):
    assert checks("log_quotient").n == 0x3fb504f4 - 0x3f3504f3 + 1
    assert checks("quotient_middles").n > 150_000_000
    assert checks("boost_quotient", 64, 1).n > 2 ** 29


@pytest.mark.parametrize("spread", [0, 1, 3, 60, 520])
def test_fp64_operations(checks, spread):
    assert checks("f64", 1 << 26, spread).n == 1 << 26


def test_fp64_estimates(checks):
    assert checks("recip31").n == 1 << 32
    assert checks("f64_sqrt").n == 1 << 28
    assert checks("open_unit").n == 1 << 26


def test_poisson_search(checks):
    # undecided searches are drawn in FP64: few on the stream's own words
    r = checks("search", 1 << 26, 0)
    assert r.n == 1 << 26 and r.aux < 0.003 * r.n
    r = checks("search", 1 << 26, 1)
    assert r.n == 1 << 26 and 0.3 < r.aux / r.n < 0.9  # around a tail about half
    # the derivation leaves the tails within (m + 2) / (m + 4) of the bound
    assert checks("search_tails", 1 << 22).worst < 17 / 18


@pytest.mark.parametrize("name", ["ptrs", "ptrs_cap", "normal", "normal_cap", "gamma", "gamma_cap"])
def test_draws_match_the_fp64_methods(checks, name):
    assert checks(name, 1 << 26).n == 1 << 26


def test_fp32_uniform(checks):
    assert checks("unit", 1 << 26).worst > 0
