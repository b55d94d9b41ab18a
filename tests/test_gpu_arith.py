"""The arithmetic of csrc/arith.cuh against the device's correctly rounded
operations: no result differs in a bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from aquagpusph_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("arith") / "arith_check.so")
    subprocess.run([build.nvcc()] + build._flags("gnn_tc.cu") +
                   ["-shared", os.path.join(HERE, "arith_check.cu"), "-o", out], check=True)
    so = ctypes.CDLL(out)
    for name in ("check_silu_grad", "check_sqrt", "check_div", "check_div_product",
                 "check_div_small"):
        getattr(so, name).restype = ctypes.c_longlong
    return so


def bits(x):
    return int(np.float32(x).view(np.uint32))


def test_silu_gradient(lib):
    """Every float up to 128, both signs; infinity and NaN."""
    assert lib.check_silu_grad(0, bits(128.0)) == 0
    assert lib.check_silu_grad(bits(np.inf), bits(np.nan)) == 0


def test_quad_sqrt(lib):
    """Every mantissa of two binades, zero, and every float at the ends of the range."""
    assert lib.check_sqrt(bits(1.0), bits(4.0)) == 0
    assert lib.check_sqrt(bits(2.0 ** -100), bits(2.0 ** -99)) == 0
    assert lib.check_sqrt(bits(2.0 ** 99), bits(2.0 ** 100)) == 0
    assert lib.check_sqrt(0, 0) == 0


def test_quad_div(lib):
    """Every mantissa of the divisor, with the numerators whose quotients lie
    nearest to the middle between two floats."""
    assert lib.check_div(64) == 0


def test_quad_div_by_a_product_of_densities(lib):
    assert lib.check_div_product(64) == 0


def test_quad_div_of_the_smallest_numerators(lib):
    assert lib.check_div_small() == 0
