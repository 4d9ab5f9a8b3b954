"""The tables of the field solve's FFTs against exp(-2 pi i k / N) in 50 digits:
every entry within 0.51 units in the last place (correctly rounded but for
near ties), and the multiples of a quarter turn exact; in FP32 the second terms
bring an entry to 2^-47 (half a unit in the last place of a term of 2^-24).  No
GPU needed."""
import ctypes
import math
from decimal import Decimal, getcontext

import numpy as np
import pytest

from conftest import load_impz

impz = load_impz()


def roots(logn):
    """exp(-2 pi i k / 2^logn) as pairs of Decimals: half angles, then products."""
    getcontext().prec = 50
    c, s = Decimal(-1), Decimal(0)  # half a turn
    for _ in range(logn - 1):
        c, s = ((1 + c) / 2).sqrt(), ((1 - c) / 2).sqrt()
    out = [(Decimal(1), Decimal(0))]
    for _ in range(2 ** (logn - 2)):  # a quarter turn; the rest by symmetry
        x, y = out[-1]
        out.append((x * c - y * s, y * c + x * s))
    q = out[:-1]
    return ([(x, -y) for x, y in q] + [(-y, -x) for x, y in q] + [(-x, y) for x, y in q] +
            [(y, x) for x, y in q])


@pytest.mark.parametrize("name,dtype,log2e", [("IdE", np.float64, 3), ("IfE", np.float32, 4)])
@pytest.mark.parametrize("logn", [3, 4, 5, 8, 9, 13])
def test_twiddles_are_rounded_once(name, dtype, log2e, logn):
    f = getattr(impz.lib(), "_ZN4impz12fft_twiddles%sEiiPv" % name)
    f.restype = ctypes.c_int
    t = np.zeros((2 ** (logn + (dtype is np.float32)), 2), dtype=dtype)
    count = f(logn, t.ctypes.data_as(ctypes.c_void_p))
    want = []
    if logn > log2e:
        w = roots(logn)
        lns = log2e
        while lns < logn:  # stage by stage, exp(-2 pi i e m / (ns r))
            lr = min(log2e, logn - lns)
            ns, r = 2 ** lns, 2 ** lr
            want += [w[(e * m << (logn - lns - lr)) % 2 ** logn] for e in range(1, r)
                     for m in range(ns)]
            lns += lr
    assert count == len(want)
    worst = 0.0
    for got, exact in zip(t[:count].ravel(), [v for pair in want for v in pair]):
        if abs(exact) < Decimal("1e-40"):
            assert got == 0.0
            continue
        unit = math.ulp(float(exact)) if dtype is np.float64 else float(np.spacing(dtype(abs(float(exact)))))
        worst = max(worst, float(abs(Decimal(float(got)) - exact)) / unit)
    assert worst <= 0.51, worst
    if dtype is np.float32:
        both = t[:count].astype(np.float64) + t[2 ** logn:2 ** logn + count]
        exact = np.array([[float(v) for v in pair] for pair in want]).reshape(count, 2)
        assert count == 0 or np.max(np.abs(both - exact)) <= 2.0 ** -47
