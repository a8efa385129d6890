"""FP32c sums over sets without connected filaments, whose tiles of 32 have a loop of their own for the
core-free distant groups: whole and ragged tiles, tiles with one link, all groups core-free, some or none.

Bound on each target: a distant term is within some 25 roundings of 2^-24 (|x1 - P|^2 formed from terms up to
(1 + 2/3)^2 of (1 - 2/3)^2), the core left out and the sum of eight by eight within as many again: 64 times
2^-24 of the sum of the terms' sizes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core,d,rc", [("visc", 2.0, 0.02), ("visc", 2.0, 3.0), ("cut", 1e-6, 0.1), ("cut", 40.0, 0.1)])
@pytest.mark.parametrize("nf", [1, 31, 32, 33, 64, 96, 97])
@pytest.mark.parametrize("link", [False, True])
def test_unlinked(wb, oracle, core, d, rc, nf, link):
    rng = np.random.default_rng(nf)
    col = lambda a: np.asfortranarray(a.reshape(len(a), -1, 1, 1))  # noqa: E731
    F1 = rng.uniform(-4.0, 4.0, (nf, 3))
    F2 = F1 + rng.normal(0.0, 0.5, (nf, 3))
    if link and nf > 1:
        F1[nf // 2] = F2[nf // 2 - 1]
    fam = (col(F1), col(F2), col(rng.uniform(5.0, 15.0, (nf, 1))), np.full((nf, 1, 1, 1), rc ** 2, order="F"))
    P = col(np.concatenate([rng.normal(0.0, 1.0, (70, 3)) + [off, 1.0, 0.0] for off in (3.0, 9.0, 14.0, 60.0)]))
    model = d if core == "cut" else "visc2"
    code = wb.bs.CORE_CUTOFF if core == "cut" else wb.bs.CORE_VATISTAS
    terms = [oracle.c_eval(*[np.asfortranarray(a[k:k + 1]) for a in fam[:2]], P,
                           *[np.asfortranarray(a[k:k + 1]) for a in fam[2:]], model, 1e9) for k in range(nf)]
    uo = oracle.c_eval(fam[0], fam[1], P, fam[2], fam[3], model, 1e9)
    size = sum(np.sqrt((t * t).sum(1, keepdims=True)) for t in terms)
    for T in (2, 4, 3, 8):
        for KF in (32, 64):
            wb.set_tuning(code, len(P), nf, T, KF, 16.0)
            for chained in (False, True):
                wb.set_layout(code, len(P), nf, chained)
                u = wb.eval_host([fam], P, code, d, 1e9, "f32c")
                err = np.abs(u - uo) / size
                assert err.max() <= 64 * 2.0 ** -24, (T, KF, chained, err.max())
