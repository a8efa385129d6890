"""The lifting-line iteration where some CTAs of a case's cluster own no points: fewer points than CTAs
(nb (nst - 1) < 8), and counts that shares of an eighth, rounded up, cover before the last CTA (nst 10, 12
and 15 with three blades: 27, 33 and 42 points); against the FP64 step oracle."""
from __future__ import annotations

import pytest

from test_kj_solve_gpu import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("size", [(2, 1, 3), (4, 1, 5), (3, 3, 4), (10, 3, 6), (12, 3, 5), (15, 3, 4), (18, 1, 4),
                                  (10, 2, 5)])
def test_idle_ctas_against_the_oracle(wb, synth, size, graph):
    _compare(wb, synth, [size], maxiter=25, graph=graph)


@pytest.mark.parametrize("nst", [10, 12, 15])
def test_idle_ctas_beside_other_cases(wb, synth, nst):
    _compare(wb, synth, [(nst, 3, 4), (17, 3, 9), (2, 1, 3), (nst, 1, 5)], maxiter=60)
