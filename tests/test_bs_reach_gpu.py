"""Reaches that are not a number, of either sign (MATLAB's has the sign bit set), or infinite: no pair is
beyond them, as a comparison with NaN is false (BiotSavart.m:111). The same bits as with a reach that holds
the whole set; and a reach of zero, which drops every pair."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REACHES = {"nan": np.array([0x7FF8000000000000], np.uint64).view(np.float64)[0],
           "-nan": np.array([0xFFF8000000000000], np.uint64).view(np.float64)[0],
           "inf": np.inf}


@pytest.mark.parametrize("core,d", [("visc", 2.0), ("visc", 3.0), ("cut", 0.3), ("cut", 0.0)])
@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_reach_without_end(wb, core, d, prec):
    rng = np.random.default_rng(4)
    col = lambda a: np.asfortranarray(a.reshape(len(a), -1, 1, 1))  # noqa: E731
    F1 = rng.uniform(-1.0, 1.0, (37, 3))
    fam = [(col(F1), col(F1 + rng.normal(0.0, 0.4, F1.shape)), col(rng.uniform(1.0, 9.0, (37, 1))),
            col(rng.uniform(1e-6, 0.05, (37, 1))))]
    P = col(rng.uniform(-3.0, 3.0, (150, 3)))
    code = wb.bs.CORE_CUTOFF if core == "cut" else wb.bs.CORE_VATISTAS
    for flags in (0, wb.bs.FLAG_SEQUENTIAL):
        want = wb.eval_host(fam, P, code, d, 1e9, prec, flags=flags)
        assert np.abs(want).max() > 0.1
        for name, co in REACHES.items():
            np.testing.assert_array_equal(wb.eval_host(fam, P, code, d, co, prec, flags=flags), want, err_msg=name)
        assert not wb.eval_host(fam, P, code, d, 0.0, prec, flags=flags).any()
