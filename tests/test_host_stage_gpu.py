"""Host arrays through the staging memory: around one chunk (1 MB), the points where more threads
copy, and more than the memory holds (32 MB), against the same evaluation on device arrays; pinned
arrays, which go directly; several threads at once. Copies: every value has to be equal."""
from __future__ import annotations

import importlib
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [1, 43690, 43691, 87400, 1398200])
@pytest.mark.parametrize("pinned", [False, True])
def test_eval_host_equals_eval_device(wb, nt, pinned):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(nt)
    F1 = np.asfortranarray(rng.uniform(-1.0, 1.0, (5, 3, 1, 1)))
    F2 = np.asfortranarray(F1 + 0.3)
    g, rc = np.ones((5, 1, 1, 1)), np.full((5, 1, 1, 1), 0.01)
    P = np.asfortranarray(rng.uniform(2.0, 9.0, (nt, 3, 1, 1)))
    dev = lambda a: torch.from_numpy(a.ravel(order="F").copy()).cuda()  # noqa: E731
    out = torch.zeros(3 * nt, dtype=torch.float64, device="cuda")
    fams = [(dev(F1), dev(F2), dev(g), dev(rc), F1.shape)]
    wb.set_autotune(False)
    try:
        wb.eval_device(fams, (dev(P), P.shape), wb.bs.CORE_VATISTAS, 2.0, 1e9, out, "f64")
        wb.sync()
        u = np.full((nt, 3, 1, 1), 7.0, order="F")
        if pinned:
            u = torch.empty(3 * nt, dtype=torch.float64, pin_memory=True).numpy().reshape(nt, 3, 1, 1, order="F")
        wb.eval_host([(F1, F2, g, rc)], P, wb.bs.CORE_VATISTAS, 2.0, 1e9, "f64", out=u)
    finally:
        wb.set_autotune(True)
    np.testing.assert_array_equal(u.ravel(order="F"), out.cpu().numpy())


def test_kinematics_from_several_threads(wb):
    kin = importlib.import_module("winds-master_b200.kin")

    def series(k):
        nt, nb, nst, ns = 400 + 37 * k, 3, 17, 16
        t = 0.05 * np.arange(nt)
        return dict(time=t, azimuth=72.0 * t + k, pitch=np.full((nt, nb), 2.0), nac_yaw=np.zeros(nt),
                    ptfm=np.zeros((nt, 6)), wind=np.tile([10.0, 0.0, 0.0], (nt, 1)),
                    r_trail=np.linspace(2.0, 63.0, nst), chord_trail=np.full(nst, 3.0),
                    twist_trail=np.linspace(13.0, 0.0, nst), r_nodes=np.linspace(3.0, 62.0, ns),
                    chord=np.full(ns, 3.0), twist=np.linspace(13.0, 0.0, ns), precone=np.zeros(nb),
                    overhang=-5.0, shaft_tilt=-5.0, tower_ht=87.6, twr2shft=1.96, ptfm_ref=0.0)

    want = [kin.kinematics(series(k)) for k in range(6)]
    got = [None] * 6

    def work(k):
        for _ in range(4):
            got[k] = kin.kinematics(series(k))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for a, b in zip(want, got):
        for key in a:
            np.testing.assert_array_equal(a[key], b[key])
