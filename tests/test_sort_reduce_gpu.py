"""The evaluation's target sort (by counting up to 3.6e8 comparisons, 18973 targets of one group, the
device-wide sort above) and the reduction by eight warps, at the sizes where they change.

Filaments and targets are apart, so that a term's rounding is a few 1e-16 and a sum of 200 of them
stays below 1e-13 of the sum of magnitudes: FP64 has to be within 1e-12 of the largest velocity of
the term-by-term oracle, FP32c within 1e-5, the bound of the direct sum's other tests."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _family(rng, dims):
    F1 = np.asfortranarray(rng.uniform(-1.0, 1.0, dims))
    F2 = np.asfortranarray(F1 + rng.normal(0.0, 0.2, dims))
    g = (dims[0], 1) + tuple(dims[2:])
    return (F1, F2, np.asfortranarray(rng.uniform(5.0, 15.0, g)),
            np.asfortranarray(rng.uniform(0.01, 0.02, g)))


@pytest.mark.parametrize("nt", [1, 33, 2048, 2049, 4097, 8192, 8193, 16384, 16385, 20001, 127, 128, 129, 18973,
                                18974])
def test_sorted_evaluation(wb, oracle, nt):
    """Seven families (two packing launches; one is empty), a ragged target count."""
    rng = np.random.default_rng(nt)
    fams = [_family(rng, d) for d in ((7, 3, 3, 1), (1, 3, 1, 1), (4, 3, 2, 2), (0, 3, 1, 1), (33, 3, 1, 1),
                                      (2, 3, 9, 3), (31, 3, 1, 1))]
    P = rng.uniform(-4.0, 4.0, (nt, 3, 1, 1))
    P[:, 0] += 7.0
    P[: nt // 4] = P[0]  # equal places, equal keys
    P = np.asfortranarray(P)
    uo = sum(oracle.c_eval(a, b, P, g, r, "visc2", 1e9) for a, b, g, r in fams if a.size)
    for prec, tol in (("f64", 1e-12), ("f32c", 1e-5)):
        u = wb.eval_host(fams, P, wb.bs.CORE_VATISTAS, 2.0, 1e9, prec)
        assert np.abs(u - uo).max() <= tol * np.abs(uo).max(), prec


@pytest.mark.parametrize("nst,steps", [(9, 20), (17, 60), (33, 80), (41, 120)])
def test_one_cta_and_device_wide_sort_agree(wb, synth, nst, steps):
    """A case alone (its nodes sorted by counting) and beside one of 17k nodes (all sorted together)."""
    import importlib
    wake = importlib.import_module("winds-master_b200.wake")
    case = lambda n, s: synth.make_wake_case(synth.RotorCase(nst=n, nsteps=s), nsteps=3)  # noqa: E731
    small, large = case(nst, steps), case(41, 140)
    alone = wake.WakeBatch([small], integrator="fe", precision="f64")
    both = wake.WakeBatch([large, small], integrator="fe", precision="f64")
    one = wake.WakeBatch([large], integrator="fe", precision="f64")
    for b in (alone, both, one):
        b.step(1)
    for a, b in ((alone.state(0), both.state(1)), (one.state(0), both.state(0))):
        assert np.abs(a["uind"]).max() > 0.1
        assert np.abs(a["uind"] - b["uind"]).max() <= 1e-12 * np.abs(a["uind"]).max()
