"""The one-kernel network at the edges of its tiles (128 rows) and of a full device of them (one per
SM, then a second one for some), for the fewest and the most inputs.

Against the oracle with the same BF16 rounding points: the bounds of the other tests of these
kernels, what a different summation order moves across rounding boundaries in a few hundred rows.
For many rows a row's output does not depend on the rows around it: bit for bit that of a short call."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n, n_in):
    mlp = importlib.import_module("winds-master_b200.mlp")
    rng = np.random.default_rng(n + n_in)
    x = rng.normal(0.5, 2.0, (n, n_in)).astype(np.float32)
    t = np.sin(x[:, 0]).astype(np.float32)
    m = mlp.Mlp(n_in, seed=n)
    th = m.params
    th[-1] = 0.1
    m.params = th
    sh, sc = np.full(n_in, 0.5, np.float32), np.full(n_in, 0.5, np.float32)
    m.set_scaling(sh, sc, 1.0)
    return m, x, t, sh, sc


@pytest.mark.parametrize("n_in", [1, 16])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 257])
def test_forward(wb, n, n_in):
    import mlp_ref
    m, x, _, sh, sc = _case(n, n_in)
    y16, _ = mlp_ref.forward(m.params, x, sh, sc, bf16_round=True)
    assert np.abs(m.forward(x) - y16).max() <= 2e-3 * (np.abs(y16).max() + 1e-3)
    m.close()


@pytest.mark.parametrize("n_in", [1, 16])
@pytest.mark.parametrize("n", [18944, 18945, 38017, 65537])
def test_rows_are_independent(wb, n, n_in):
    m, x, _, _, _ = _case(n, n_in)
    y = m.forward(x)
    for a, b in ((0, 200), (n // 2 - 77, n // 2 + 77), (n - 131, n)):
        np.testing.assert_array_equal(m.forward(x[a:b]), y[a:b])
    m.close()


@pytest.mark.parametrize("n_in", [1, 16])
@pytest.mark.parametrize("n", [1, 128, 129, 18944, 19100])
def test_gradient(wb, n, n_in):
    import mlp_ref
    m, x, t, sh, sc = _case(n, n_in)
    loss, g = m.loss_grad(x, t)
    l16, g16 = mlp_ref.loss_grad(m.params, x, t, sh, sc, bf16_round=True)
    assert abs(loss - l16) <= 1e-4 * l16 + 1e-7
    cuts = sorted([mlp_ref.OFF_W[L] for L in range(4)] + [mlp_ref.OFF_B[L] for L in range(4)] +
                  [mlp_ref.OFF_W5, mlp_ref.OFF_B5, mlp_ref.N_PARAM])
    for a, b in zip(cuts[:-1], cuts[1:]):
        assert np.linalg.norm(g[a:b] - g16[a:b]) <= 5e-3 * np.linalg.norm(g16[a:b]) + 1e-7, (a, b)
    m.close()
