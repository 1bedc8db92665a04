"""The branch-free quotients, the FP64 reciprocal and the rotation solve of the
kernels against CUDA's own divisions, bit for bit: random operands over the
ranges that each states (score scales d0^2 in [2^-3, 2^13), squared distances up
to the end of the FP32 range, infinite and NaN), a quarter of them with mantissas
beside all zeros and all ones, and every mantissa of a denominator."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

CHECKS = {"tmterm": (0, 1 << 30), "tmterm_ends": (1, 1 << 22), "div_ord": (2, 1 << 30),
          "div2_neg": (3, 1 << 30), "recip64": (4, 1 << 29), "div64": (5, 1 << 29), "solve": (6, 1 << 25),
          "mantissas": (7, 1 << 27)}


@pytest.mark.parametrize("name", list(CHECKS))
def test_equals_the_ieee_division(name):
    from gtalign_alpha_b200 import build
    L = ctypes.CDLL(build.build_arith_check())
    L.arith_check.argtypes = [ctypes.c_int, ctypes.c_ulonglong, ctypes.c_longlong,
                              ctypes.POINTER(ctypes.c_ulonglong), ctypes.POINTER(ctypes.c_double)]
    what, n = CHECKS[name]
    bad, first = ctypes.c_ulonglong(1), (ctypes.c_double * 3)()
    assert L.arith_check(what, 17, n, ctypes.byref(bad), first) == 0
    assert bad.value == 0, (bad.value, [float.hex(x) for x in first])
