"""The packed roots and quotients of the force and adjoint passes are the correctly
rounded ones: every float of their range, and every numerator that could round
wrong, against CUDA's own."""
import ctypes
import os
import subprocess

import pytest

from simplefluid_gb300 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_packed_root_and_quotients_round_as_ieee(tmp_path):
    so = str(tmp_path / "librounding_check.so")
    out = subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-fmad=false", "-I", build.CSRC, "-shared", "-o", so,
                          os.path.join(HERE, "cpp", "rounding_check.cu")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    fn = ctypes.CDLL(so).check_rounding
    fn.argtypes = [ctypes.c_float, ctypes.c_float, ctypes.c_int, ctypes.POINTER(ctypes.c_ulonglong)]
    counts = (ctypes.c_ulonglong * 7)()
    # 2^-90 (kFastR2Min) to 2^80 (kFastHMax squared)
    assert fn(2.0 ** -90, 2.0 ** 80, 64, counts) == 0
    roots, recips, recips_of_squares, bad_r, tried_r, bad_r2, tried_r2 = counts
    assert (roots, recips, recips_of_squares) == (0, 0, 0)
    assert bad_r == 0 and bad_r2 == 0
    assert tried_r > 64 * 2 ** 23 + 10 ** 7 and tried_r2 > 2 * (64 * 2 ** 23 + 10 ** 7)
