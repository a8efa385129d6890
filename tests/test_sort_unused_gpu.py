"""Targets ordered by counting where some are unused, as in the group of a growing wake: the order has to be
a permutation with every live target before every unused one, at the sizes where the kernel takes one, two
and four targets a lane and at the largest group that is counted."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 4736, 4737, 9472, 9473, 18973])
@pytest.mark.parametrize("live", [0.0, 0.1, 0.7, 1.0])
def test_order_is_a_permutation(wb, n, live):
    rng = np.random.default_rng(n)
    P = np.asfortranarray(rng.uniform(-1.0, 1.0, (n, 3)))
    P[-1] = P.max(0)  # a corner of the box: the last cells of the curve
    unused = np.ascontiguousarray(rng.random(n) >= live, dtype=np.int32)
    perm = np.full(n, -1, dtype=np.int32)
    call = wb.lib().winds_bs_selftest_order
    call.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong, C.c_void_p]
    wb.bs._check(call(P.ctypes.data, unused.ctypes.data, n, perm.ctypes.data))
    assert np.array_equal(np.sort(perm), np.arange(n))
    assert np.array_equal(unused[perm], np.sort(unused))
    tail = perm[n - unused.sum():]
    assert np.array_equal(tail, np.sort(tail))  # equal keys keep their order


def test_order_refuses_larger_groups(wb):
    call = wb.lib().winds_bs_selftest_order
    call.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong, C.c_void_p]
    P, u, perm = np.zeros((18974, 3), order="F"), np.zeros(18974, np.int32), np.zeros(18974, np.int32)
    assert call(P.ctypes.data, u.ctypes.data, 18974, perm.ctypes.data) == 1  # WINDS_BS_ERR_ARG
