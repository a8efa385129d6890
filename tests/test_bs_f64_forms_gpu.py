"""The FP64 sum's short forms against the same sum in sequential mode, which has the full term for
every pair: random points, points on a filament's line, next to the segment and on its ends, reaches
that cut through the set, zero-length filaments, circulations and scales outside the forms' range.

Bound: the forms are used where 1 + cos >= 2^-8 and the squared sine to the line >= 2^-9, where both
ways to form a term are within 4 roundings times 512 (2.3e-13) of it; 1e-12 of the sum of the terms'
sizes holds the two and the summation."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _col(a):
    return np.asfortranarray(a.reshape(a.shape[0], -1, 1, 1))


@pytest.mark.parametrize("scale", [1e-120, 1e-70, 1e-3, 1.0, 1e4, 1e70, 1e120])
@pytest.mark.parametrize("core,d", [("visc", 2.0), ("cut", 0.3)])
@pytest.mark.parametrize("reach", [2.5, 1e3, 0.0, -1.0])
def test_short_forms(wb, scale, core, d, reach):
    rng = np.random.default_rng(7)
    nf = 37
    F1 = rng.uniform(-1.0, 1.0, (nf, 3))
    F2 = F1 + rng.normal(0.0, 0.4, (nf, 3))
    F2[5] = F1[5]
    g = rng.uniform(1.0, 9.0, (nf, 1))
    g[3], g[4], g[6], g[8] = np.nan, np.inf, 0.0, -2.0
    rc = rng.uniform(1e-6, 0.05, (nf, 1))
    rc[9] = 0.0
    L, n = F2[0] - F1[0], np.cross(F2[0] - F1[0], [0.3, -0.2, 0.9])
    line = [F1[0] + s * L + o * n for s in (-2.0, -0.1, 0.0, 0.3, 1.0, 1.2, 5.0)
            for o in (0.0, 1e-9, 1e-6, 1e-3, 0.02, 0.06, 0.1)]
    P = np.concatenate([rng.uniform(-3.0, 3.0, (150, 3)), np.array(line), F1[7:9], [[0.0, 1e9, 0.0]]])
    code = wb.bs.CORE_CUTOFF if core == "cut" else wb.bs.CORE_VATISTAS
    with np.errstate(over="ignore", under="ignore"):
        args = (_col(P * scale), code, d * scale ** 2 if core == "cut" else d, reach * scale)
        fam = [tuple(_col(a) for a in (F1 * scale, F2 * scale, g, rc * scale ** 2))]
    u = wb.eval_host(fam, *args, "f64")
    ref = wb.eval_host(fam, *args, "f64", flags=wb.bs.FLAG_SEQUENTIAL)
    size = sum(np.abs(wb.eval_host([tuple(np.asfortranarray(a[k:k + 1]) for a in fam[0])], *args, "f64",
                                   flags=wb.bs.FLAG_SEQUENTIAL)) for k in range(nf))
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(u))
    assert np.all(np.abs(u - ref)[fin] <= 1e-12 * size.max(axis=1, keepdims=True).repeat(3, 1)[fin])
