"""Parameters set from the host are the ones the next call computes with: the same vector set twice
in a row (the second time long after the first upload) gives the same bits."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_forward_uses_the_parameters_just_set(wb):
    mlp = importlib.import_module("winds-master_b200.mlp")
    m = mlp.Mlp(9, seed=1)
    rng = np.random.default_rng(2)
    x = rng.normal(0.0, 1.0, (256, 9)).astype(np.float32)
    p0 = m.params
    for k in range(20):
        p = (p0 * rng.uniform(0.5, 1.5, p0.shape)).astype(np.float32)
        m.params = p
        y = m.forward(x)
        m.params = p
        np.testing.assert_array_equal(m.forward(x), y)
        m.params = p0
    m.close()
