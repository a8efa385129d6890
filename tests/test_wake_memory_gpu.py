"""A closed batch gives its device memory back: the per-step series of long runs above all (16 bytes a step
and case), and the small tables, over many batches."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_closed_batches_leave_no_memory(wb, synth):
    torch = pytest.importorskip("torch")
    wake = importlib.import_module("winds-master_b200.wake")
    rc = synth.RotorCase(nst=3, nb=1, nsteps=4, dpsi_deg=10.0, seed=1, jitter=0.0)
    c = synth.make_wake_case(rc, nsteps=4, pitch_deg=3.0)
    n = 400000  # 6.4 MB of series
    at = np.arange(n) % 4
    c.update(nsteps=n, quarter=c["quarter"][:, :, at], trailing=c["trailing"][:, :, at], wind=c["wind"][:, at])

    def batch():
        b = wake.WakeBatch([c], integrator="fe", precision="f64")
        b.step(1)
        b.close()

    batch()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(10):
        batch()
    assert free - torch.cuda.mem_get_info()[0] <= 16 << 20  # 64 MB of series were allocated
