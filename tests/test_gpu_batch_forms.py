"""The forms a batch's launches take: which knobs choose them, and that they
change no bit of the members' results."""
import numpy as np
import pytest

import fdtd_b200 as F
from cases import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knob,value", [("FDTD_TMA", "0"), ("FDTD_TMA", "1"), ("FDTD_PDL", "0"), ("FDTD_PDL", "1")])
def test_staged_knobs_leave_the_batch_its_launches(knob, value, monkeypatch):
    """FDTD_TMA and FDTD_PDL arrange the staged launches of a simulation of its
    own.  The batch keeps its launches over all members and its graph."""
    params = [make(F, n, precision=F.FDTD_FP32) for n in ("sphere_au", "sphere_big", "slab")]
    out = []
    for env in (False, True):
        if env:
            monkeypatch.setenv(knob, value)
        b = F.Batch(params)
        b.step(140)
        out.append((b.stats(), [b.sim(i).field(c) for i in range(3) for c in range(6)]))
        b.close()
    assert out[0][0] == out[1][0] and out[1][0][1] == 1
    for x, y in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(x, y)
