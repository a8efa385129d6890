"""The arrays that ``kinematics`` returns are the caller's, each by itself: one that is kept does not keep the
others' memory, and each can be resized, as arrays made one by one."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_arrays_are_their_own(wb, synth):
    kin = importlib.import_module("winds-master_b200.kin")
    out = kin.kinematics(synth.rotor_series(synth.RotorCase(nst=9, nsteps=40), 40))
    assert len(out) == 15
    for name, a in out.items():
        assert a.flags.owndata and a.flags.f_contiguous and a.base is None, name
        assert np.isfinite(a).all(), name
