"""jf_sqrt_mid, jf_inv_sqrt_mid and jf_div_mid (jellyfih_b200/csrc/jf_device.cuh)
give the bits of the general square root, reciprocal of the root and quotient:
every operand of 2^-60 .. 2^60 for the roots; for the quotient every mantissa of
the divisor, with numerators at and about the powers of two (where a reciprocal
that is not correctly rounded shows), at and about the divisor's own mantissa
and its complement, and random ones."""
import ctypes
import os
import subprocess

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


class Found(ctypes.Structure):
    _fields_ = [("n", ctypes.c_uint64), ("a", ctypes.c_float), ("b", ctypes.c_float)]


def test_roots_and_quotient_have_the_general_bits(tmp_path):
    from jellyfih_b200 import build
    lib = str(tmp_path / "mid_range.so")
    # the flags of the library's own build
    subprocess.run([build.nvcc_path(), *build.ARCH, "-O3", "-std=c++17", "--shared", "-Xcompiler", "-fPIC", "-I",
                    build.CSRC, "-I", os.path.join(build.REPO, "include"), "-o", lib,
                    os.path.join(HERE, "mid_range.cu")], check=True, timeout=300)
    out = (Found * 3)()
    assert ctypes.CDLL(lib).mid_range(out, 256) == 0
    for what, f in zip(("square root", "reciprocal of the root", "quotient"), out):
        assert f.n == 0, f"{what}: {f.n} operands differ, one of them {float(f.a).hex()}, {float(f.b).hex()}"
