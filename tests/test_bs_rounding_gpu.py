"""Rounding of the FP32c sums over a wake, against the FP64 sum on the same inputs, in the 2-norm over all
targets. A wake's filaments in chained order put the terms that matter to a target next to one another, so
the error depends on how few of them an uncompensated sum spans. Bound: two thirds of FP32's unit roundoff
(2^-24 = 6.0e-8), which the sum in input order, without chains and 64 filaments at a time, keeps as well."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 2.0 / 3.0 * 2.0 ** -24


def _rel(u, ref):
    return np.linalg.norm(u - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("core,d", [("visc", 2.0), ("cut", 1e-4)])
def test_evaluation(wb, synth, core, d):
    w = synth.make_wake(synth.RotorCase(nst=29, nsteps=347, dpsi_deg=720.0 / 347, seed=3))
    fams = [synth.shed_filaments(w["dom"]) + (w["gamma_shed"], w["rc_shed"]),
            synth.trail_filaments(w["dom"]) + (w["gamma_trail"], w["rc_trail"])]
    code = wb.bs.CORE_CUTOFF if core == "cut" else wb.bs.CORE_VATISTAS
    nt, nf = w["dom"].size // 3, sum(f[2].size for f in fams)
    ref = wb.eval_host(fams, w["dom"], code, d, 1000.0, "f64")
    for T, KF in ((2, 32), (2, 64), (4, 32), (4, 64), (3, 32), (3, 64)):
        for chained in (True, False):
            wb.set_tuning(code, nt, nf, T, KF, 16.0)
            wb.set_layout(code, nt, nf, chained)
            err = _rel(wb.eval_host(fams, w["dom"], code, d, 1000.0, "f32c"), ref)
            assert err <= BOUND, (T, KF, chained, err)


@pytest.mark.parametrize("d", ["visc2", 1e-4])
def test_step(synth, wb, d):
    wake = importlib.import_module("winds-master_b200.wake")
    cases = [synth.make_wake_case(synth.RotorCase(nst=nst, nsteps=n, dpsi_deg=720.0 / n, seed=n, jitter=0.0),
                                  nsteps=4, pitch_deg=4.0) for nst, n in ((29, 348), (41, 200))]
    got = {}
    for prec in ("f64", "f32c"):
        b = wake.WakeBatch(cases, integrator="pcc", d=d, co=1000.0, precision=prec)
        b.step(1, graph=True)
        got[prec] = [b.state(k)["uind"] for k in range(len(cases))]
        b.close()
    for a, c in zip(got["f32c"], got["f64"]):
        assert _rel(a, c) <= BOUND, _rel(a, c)
