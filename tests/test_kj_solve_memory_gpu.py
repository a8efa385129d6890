"""Lifting lines whose influence matrix would take more device memory than is free: formed term by term, with
the oracle's iterations and circulation as everywhere (tests/test_kj_solve_gpu.py)."""
from __future__ import annotations

import pytest

from test_kj_solve_gpu import _compare

pytestmark = pytest.mark.gpu


def test_matrix_beyond_free_memory(wb, synth):
    """100 cases of 357 points and 1074 own filaments: 1.2 GB of matrix, with some 0.7 GB free."""
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - (700 << 20), dtype=torch.uint8, device="cuda")
    try:
        _compare(wb, synth, [(120, 3, 3)] * 100, maxiter=2, steps=1, check=[0, 99])
    finally:
        del held
        torch.cuda.empty_cache()
