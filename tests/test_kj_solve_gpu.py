"""The lifting-line iteration in one launch (kj_solve) at the sizes where it changes form: fewer
points than CTAs of a cluster, matrix rows in shared memory, in the scratch and formed term by term,
working vectors in the scratch; against the FP64 step oracle."""
from __future__ import annotations

import numpy as np
import pytest

import kj_ref
import wake_ref

pytestmark = pytest.mark.gpu

BOUND_TOL = 1e-9  # as the FP64 lifting-line tests


def _case(synth, nst, nb, na, seed):
    rc = synth.RotorCase(nst=nst, nb=nb, nsteps=na - 1, dpsi_deg=10.0, seed=seed, jitter=0.0)
    return (synth.make_wake_case(rc, nsteps=4, pitch_deg=3.0),
            synth.make_kj_case(rc, nsteps=4, pitch_deg=3.0, root_cut=0.2))


def _compare(wb, synth, sizes, maxiter, tol=1e-8, graph=True, steps=2, check=None):
    import importlib
    wake = importlib.import_module("winds-master_b200.wake")
    pairs = [_case(synth, *s, seed=k) for k, s in enumerate(sizes)]
    b = wake.WakeBatch([c for c, _ in pairs], integrator="pcc", precision="f64")
    b.set_kj([k for _, k in pairs], relax=0.25, tol=tol, maxiter=maxiter)
    refs = {i: kj_ref.KJWakeRef(wake_ref.WakeCaseRef(**{k: pairs[i][0][k] for k in wake_ref.WakeCaseRef.__dataclass_fields__}),
                                pairs[i][1], integrator="pcc", relax=0.25, tol=tol, maxiter=maxiter)
            for i in (range(len(pairs)) if check is None else check)}
    for _ in range(steps):
        b.step(1, graph=graph)
        its, res, ev = b.kj_stats()
        assert ev == its.max()
        for i, r in refs.items():
            r.step()
            assert its[i] == r.kj_iters
            assert abs(res[i] - r.kj_res) <= BOUND_TOL
            assert np.abs(b.bound(i) - r.bound).max() <= BOUND_TOL * (np.abs(r.bound).max() + 1.0)
            assert np.abs(b.perf(i)[2] - r.aoa).max() <= 1e-7
    b.close()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("sizes", [[(2, 1, 3)], [(3, 2, 4)], [(9, 3, 12), (4, 1, 5)], [(41, 3, 6)]])
def test_kj_solve_small(wb, synth, sizes, graph):
    _compare(wb, synth, sizes, maxiter=25, graph=graph)


def test_kj_solve_tolerances_end_cases_apart(wb, synth):
    """Cases that converge at different iterations, the batch's count that of the last."""
    _compare(wb, synth, [(9, 3, 12), (17, 3, 5), (5, 2, 7)], maxiter=200, tol=1e-5)


def test_kj_solve_matrix_in_scratch(wb, synth):
    _compare(wb, synth, [(90, 3, 4), (7, 3, 4)], maxiter=6)


def test_kj_solve_vectors_in_scratch(wb, synth):
    _compare(wb, synth, [(1800, 3, 3)], maxiter=2, steps=1)


def test_kj_solve_without_matrix(wb, synth):
    """More cases than the matrix scratch holds: every term formed in every iteration."""
    sizes = [(120, 3, 3)] * 240
    _compare(wb, synth, sizes, maxiter=2, steps=1, check=[0, 239])
