"""Evaluations of different sizes from two host threads at once, each on its own stream and scratch (the
library's context, and the no-allocation call): both order their targets by counting with the same kernel,
whose shared memory grows with their number."""
from __future__ import annotations

import ctypes as C
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_counting_sizes_from_two_threads(wb):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).ravel(order="F").copy()).cuda()  # noqa: E731
    fam = (dev([0.0, 0.0, 0.0]), dev([0.0, 0.0, 1.0]), dev([1.0]), dev([0.01]), (1, 3, 1, 1))
    sizes = (18900, 9600)  # four targets a lane in both; 76 and 38 KB of keys
    P = [dev(rng.uniform(1.0, 3.0, (n, 3))) for n in sizes]
    out = [torch.zeros(3 * n, dtype=torch.float64, device="cuda") for n in sizes]
    L = wb.lib()
    call = L.winds_bs_eval_device_noalloc
    call.argtypes = [C.c_void_p, C.c_int] + [C.c_void_p] * 5
    f = wb.bs.Family(*[x.data_ptr() for x in fam[:4]], (C.c_longlong * 4)(*fam[4]))
    prm = wb.bs.Params(wb.bs.CORE_VATISTAS, 2.0, 1e9, wb.bs.PREC_F64, 0)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    errors, end = [], time.time() + 4.0

    def library():
        try:
            while time.time() < end and not errors:
                wb.eval_device([fam], (P[0], (sizes[0], 3, 1, 1)), wb.bs.CORE_VATISTAS, 2.0, 1e9, out[0], "f64")
                wb.sync()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    def noalloc():
        dims = (C.c_longlong * 4)(sizes[1], 3, 1, 1)
        while time.time() < end and not errors:
            if call(C.byref(f), 1, P[1].data_ptr(), dims, C.byref(prm), out[1].data_ptr(), stream.cuda_stream):
                errors.append(RuntimeError(L.winds_bs_last_error().decode()))

    ts = [threading.Thread(target=t) for t in (library, noalloc)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors
