"""FP32c sums of more items than workers, each of one or two tiles of filaments, with near-singular pairs
and distant filaments in the same tiles: every worker writes to its stages (prepared records, lists of
near-singular pairs) until the end of an item and fills them again at the start of its next. A write that
came after the copy would change a sum: the same bits in every run, whichever worker takes which item."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core", ["visc", "cut"])
@pytest.mark.parametrize("T,KF,tiles", [(2, 64, 1), (2, 32, 1), (4, 64, 1), (4, 32, 2), (3, 64, 2)])
def test_short_items(wb, core, T, KF, tiles):
    rng = np.random.default_rng(5)
    nf, nt = 640, 60000
    p = np.cumsum(rng.normal(0.0, 0.25, (nf + 1, 3)), axis=0)
    col = lambda a: np.asfortranarray(a.reshape(len(a), -1, 1, 1))  # noqa: E731
    F1, F2 = col(p[:-1]), col(p[1:])
    g, rc = col(rng.uniform(5.0, 15.0, (nf, 1))), np.full((nf, 1, 1, 1), 1e-3, order="F")
    near = p[rng.integers(0, nf, nt // 2)] + rng.normal(0.0, 0.2, (nt // 2, 3))
    P = col(np.concatenate([near, rng.uniform(-30.0, 30.0, (nt - nt // 2, 3))]))
    code = wb.bs.CORE_CUTOFF if core == "cut" else wb.bs.CORE_VATISTAS
    d = 1e-3 if core == "cut" else 2.0
    tiles_of_targets = -(-nt // (32 * {2: 2, 3: 6, 4: 4}[T]))
    wb.set_tuning(code, nt, nf, T, KF, tiles_of_targets * nf / (KF * tiles) / (148 * 8))
    wb.set_layout(code, nt, nf, True)
    try:
        u = [wb.eval_host([(F1, F2, g, rc)], P, code, d, 1e9, "f32c") for _ in range(8)]
    finally:
        wb.set_tuning(code, nt, nf, 4, 64, 16.0)
    for v in u[1:]:
        np.testing.assert_array_equal(v, u[0])
