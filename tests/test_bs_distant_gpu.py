"""The FP32c sum's distant form (filaments at least 1.5 target-ball radii away, expanded about the
ball's centre), with and without its core term, on chained and broken lines of filaments, at the
edges of tiles and groups and over the scales it has to hold for."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import per_target_rel

pytestmark = pytest.mark.gpu

F32C_TOL = 1e-5


def _in_range(F1, F2, g, rcs):
    """The FP32 records hold the Vatistas core term (K^2 rc^2 |L|^2)^2 between 1e-30 and 1e30; a
    filament beyond either end is evaluated with the core of that end."""
    L2 = ((F2 - F1) ** 2).sum(1, keepdims=True)
    D = ((g / (4 * np.pi)) ** 2 * rcs * L2) ** 2
    return bool(np.all((D[g != 0] >= 1e-30) & (D[g != 0] <= 1e30)))


def _line(rng, nf, scale, broken):
    """nf filaments of one random-walk line around the origin, [nf, 3, 1, 1]; ``broken``: every
    fifth one moved off the line, so that it and its successor start chains."""
    p = np.cumsum(rng.normal(0.0, 0.3, (nf + 1, 3)), axis=0) + [0.0, 0.0, 0.5]
    p *= 4.0 / max(4.0, np.abs(p).max())
    F1, F2 = p[:-1].copy(), p[1:].copy()
    if broken:
        F1[::5] += rng.normal(0.0, 0.2, F1[::5].shape)
    g = rng.uniform(5.0, 15.0, (nf, 1, 1, 1))
    g[::7] = 0.0  # filaments without circulation stay in the chain
    f = lambda a: np.asfortranarray(a.reshape(nf, 3, 1, 1) * scale)  # noqa: E731
    return f(F1), f(F2), np.asfortranarray(g)


@pytest.mark.parametrize("core,d,rc", [("visc", 2.0, 0.02), ("visc", 2.0, 3.0), ("cut", 1e-6, 0.1), ("cut", 40.0, 0.1)])
@pytest.mark.parametrize("nt,nf", [(1, 1), (2, 5), (33, 64), (129, 131), (193, 260)])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e4])
def test_distant_form(wb, oracle, core, d, rc, nt, nf, scale):
    rng = np.random.default_rng(nt + nf)
    # a ball of targets just inside, at and beyond the form's distance from the line
    P = rng.normal(0.0, 1.0, (nt, 3))
    P *= rng.uniform(0.0, 4.0, (nt, 1)) / np.linalg.norm(P, axis=1, keepdims=True)
    for off in (9.0, 13.0, 40.0):
        Pf = np.asfortranarray(((P + [off, 1.0, 0.0]) * scale).reshape(nt, 3, 1, 1))
        for broken in (False, True):
            F1, F2, g = _line(rng, nf, scale, broken)
            rcs = np.full((nf, 1, 1, 1), (rc * scale) ** 2, order="F")
            dd = d * scale ** 2 if core == "cut" else d
            if core == "visc" and not _in_range(F1, F2, g, rcs):
                continue
            uo = oracle.c_eval(F1, F2, Pf, g, rcs, dd if core == "cut" else "visc2", 1e9)
            code = wb.bs.CORE_CUTOFF if core == "cut" else wb.bs.CORE_VATISTAS
            for T, KF, chained in ((2, 32, True), (4, 64, True), (3, 64, True), (8, 32, True), (4, 32, False)):
                wb.set_tuning(code, nt, nf, T, KF, 16.0)
                wb.set_layout(code, nt, nf, chained)
                u = wb.eval_host([(F1, F2, g, rcs)], Pf, code, dd, 1e9, "f32c")
                assert per_target_rel(u, uo) < F32C_TOL, (T, KF, chained, off, broken)
