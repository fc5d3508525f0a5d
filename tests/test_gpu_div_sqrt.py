"""The exact mode's quotient and square root (integer long division and digit recurrence,
csrc/lg_x64.cuh) against IEEE-754 double: equal bits, for random significands and exponents
and where a digit, the correction or the rounding can go wrong."""
import ctypes as C

import numpy as np
import pytest

from light_garden_gb300 import abi

pytestmark = pytest.mark.gpu


def _run(a, b):
    lib = C.CDLL(str(abi.LIB_PATH.parent / "liblg_peaks.so"))
    f = lib.lgp_div_sqrt
    f.argtypes = [C.c_int] + [C.POINTER(C.c_double)] * 4 + [C.c_uint64]
    q, s = np.empty_like(a), np.empty_like(a)
    ptr = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in (a, b, q, s)]
    assert f(0, *ptr, len(a)) == 0
    return q, s


def _same(got, want):
    return (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))


@pytest.mark.parametrize("kind", ["random", "near", "few_bits", "many_ones", "squares", "tiny_huge", "special"])
def test_div_sqrt_round_like_ieee(gpu, kind):
    rng = np.random.default_rng(3)
    n = 1 << 21
    bits = rng.integers(0, 1 << 64, (2, n), dtype=np.uint64)
    mant = np.uint64((1 << 52) - 1)
    expo = rng.integers(1000, 1047, (2, n)).astype(np.uint64) << np.uint64(52)  # 2^-23 .. 2^23
    x = (bits & (mant | np.uint64(1 << 63))) | expo
    if kind == "near":          # quotients around 1
        x[1] = x[0] + rng.integers(0, 9, n).astype(np.uint64) - np.uint64(4)
    elif kind == "few_bits":    # exact quotients, remainders of zero
        x &= ~np.uint64((1 << 30) - 1)
    elif kind == "many_ones":
        x |= np.uint64(((1 << 52) - 1) ^ 0xFF)
    elif kind == "tiny_huge":   # results outside the normal range, denormals
        x = bits
    a, b = x[0].view(np.float64).copy(), x[1].view(np.float64).copy()
    if kind == "squares":       # exact roots and their neighbours
        r = ((x[0] & ~np.uint64((1 << 27) - 1)).view(np.float64)) ** 2
        a = (r.view(np.uint64) + rng.integers(0, 3, n).astype(np.uint64) - np.uint64(1)).view(np.float64).copy()
    elif kind == "special":
        v = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 1.7976931348623157e308, 4.0, 2.0])
        a, b = (g.ravel().copy() for g in np.meshgrid(v, v))
    q, s = _run(a, b)
    with np.errstate(all="ignore"):
        assert _same(q, a / b).all()
        assert _same(s, np.sqrt(a)).all()
