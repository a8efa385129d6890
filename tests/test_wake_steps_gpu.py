"""Several steps asked for in one call against the same steps asked for one by one, from the reference's
start-up (no lifting-line iteration at its first step) and from a full wake, eager and replayed."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("startup,na_start", [("reference", 2), ("full", 0)])
@pytest.mark.parametrize("graph", [False, True])
def test_steps_in_one_call(wb, synth, startup, na_start, graph):
    wake = importlib.import_module("winds-master_b200.wake")
    rc = synth.RotorCase(nst=9, nb=3, nsteps=8, dpsi_deg=10.0, seed=1, jitter=0.0)
    c = synth.make_wake_case(rc, nsteps=8, pitch_deg=3.0)
    c["na_start"] = na_start
    kj = synth.make_kj_case(rc, nsteps=8, pitch_deg=3.0, root_cut=0.2)
    got = []
    for calls in ([4], [1, 1, 1, 1], [2, 2], [1, 3]):
        b = wake.WakeBatch([c], integrator="pcc", precision="f64", startup=startup)
        b.set_kj([kj], relax=0.25, tol=1e-8, maxiter=30)
        for n in calls:
            b.step(n, graph=graph)
        live, steps = b.live(0)
        assert steps == 4
        its, res, evals = b.kj_stats()
        # of the wake's columns now, and of the last step's (one fewer while it grows); the
        # other columns of the capacity hold nothing
        st, m = b.state(0), live if na_start == 0 else live - 1
        st = dict(dom=st["dom"][:, :, :live], bound=st["bound"], shed=st["shed"][:, :m],
                  trail=st["trail"][:, :m - 1], rc_shed=st["rc_shed"][:, :m],
                  rc_trail=st["rc_trail"][:, :m - 1], uind=st["uind"][:, :, :m])
        got.append((st, b.loads(), its.tolist(), evals))
        b.close()
    assert got[0][2][0] > 0
    for state, loads, its, evals in got[1:]:
        assert (its, evals) == (got[0][2], got[0][3])
        for k, v in state.items():
            np.testing.assert_array_equal(v, got[0][0][k], err_msg=k)
        for a, b in zip(loads, got[0][1]):
            np.testing.assert_array_equal(a, b)
