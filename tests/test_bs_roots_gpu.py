"""1/sqrt and 1/x of the FP64 sums (bs_device.cuh) against 80-bit values and against CUDA's functions.

Bound: 2^-52 relative, which holds the derived 1.5 roundings of the root and one of the reciprocal. CUDA's
1/x is correctly rounded and its rsqrt within one place of the last digit, a relative 2^-52, so the two sides
are at most 2^-52 + 2^-53 and 2^-52 + 2^-52 apart."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _roots(wb, x):
    y = np.zeros((4, len(x)))
    call = wb.lib().winds_bs_selftest_roots
    call.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p]
    wb.bs._check(call(np.ascontiguousarray(x).ctypes.data, len(x), y.ctypes.data))
    return y


def test_roots_over_their_range(wb):
    rng = np.random.default_rng(0)
    m = 1.0 + np.arange(4096) / 4096.0
    edge = np.concatenate([[1.0, np.nextafter(2.0, 1.0), np.nextafter(4.0, 1.0)], m])
    x = np.concatenate([2.0 ** rng.uniform(-960.0, 960.0, 400000), rng.uniform(0.25, 4.0, 400000), edge,
                        edge * 2.0 ** -960, edge * 2.0 ** 958, 2.0 ** np.arange(-960.0, 961.0)])
    y = _roots(wb, x)
    assert np.finfo(np.longdouble).nmant >= 63
    xl = x.astype(np.longdouble)
    for got, cuda, ref, apart in ((y[0], y[2], 1 / np.sqrt(xl), 2.0 ** -51), (y[1], y[3], 1 / xl, 1.5 * 2.0 ** -52)):
        assert float(np.max(np.abs(got / ref - 1))) <= 2.0 ** -52
        assert float(np.max(np.abs(got / cuda - 1))) <= apart


def test_roots_outside(wb):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, -1.0, -1e-310])
    y = _roots(wb, x)
    assert not np.isfinite(y[0]).any()
    assert not np.isfinite(y[1][x != -1.0]).any()
    assert y[1][7] == -1.0
