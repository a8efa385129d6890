"""FP64 sums with a negative squared cut-off, for which only FP64 is offered: the denominator of a pair can
nearly vanish, and what is left of it is the reference's rounding. The short form has to leave such pairs to
the full term, as it is in sequential mode.

Bound: as tests/test_bs_f64_forms_gpu.py, where the short form is used both ways of forming a term are within
4 roundings times 512 of it; 1e-12 of the sum of the terms' sizes holds the two and the summation."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [0.0, 1e-15, 1e-13, 1e-10, 1e-6, 1e-3, 0.1])
@pytest.mark.parametrize("k", [0, 5, 30])
def test_vanishing_denominators(wb, left, k):
    rng = np.random.default_rng(k)
    nf, nt = 37, 300
    F1 = rng.uniform(-1.0, 1.0, (nf, 3))
    F2 = F1 + rng.normal(0.0, 0.4, (nf, 3))
    P = rng.uniform(-3.0, 3.0, (nt, 3))
    a, b = P[k] - F1[k], P[k] - F2[k]
    rr = np.linalg.norm(a) * np.linalg.norm(b)
    d = -(1.0 - left) * rr * (rr + a @ b) / ((F2 - F1)[k] @ (F2 - F1)[k])
    col = lambda x: np.asfortranarray(x.reshape(len(x), -1, 1, 1))  # noqa: E731
    fam = tuple(col(x) for x in (F1, F2, rng.uniform(1.0, 9.0, (nf, 1)), np.full((nf, 1), 0.01)))
    seq = dict(flags=wb.bs.FLAG_SEQUENTIAL)
    args = (col(P), wb.bs.CORE_CUTOFF, d, 1e9, "f64")
    u, ref = wb.eval_host([fam], *args), wb.eval_host([fam], *args, **seq)
    size = sum(np.abs(wb.eval_host([tuple(np.asfortranarray(x[j:j + 1]) for x in fam)], *args, **seq)) for j in range(nf))
    assert np.all(np.abs(u - ref) <= 1e-12 * size.max(axis=1, keepdims=True))
