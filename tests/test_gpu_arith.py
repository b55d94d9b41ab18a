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
    for name in ("check_silu_grad",):
        getattr(so, name).restype = ctypes.c_longlong
    return so


def bits(x):
    return int(np.float32(x).view(np.uint32))


def test_silu_gradient(lib):
    """Every float up to 128, both signs; infinity and NaN."""
    assert lib.check_silu_grad(0, bits(128.0)) == 0
    assert lib.check_silu_grad(bits(np.inf), bits(np.nan)) == 0
