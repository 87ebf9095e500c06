"""TFSF boxes at the edge of what the setup accepts: two to four cells wide,
so that both faces of an axis fall into one vector of the direct passes, and
with faces on the grid's walls, whose E and H cells the passes do not store.
The wave's polarisation has an x and a y component, so that every face takes
corrections.

Every form of the step gives the same bits: the corrections as the default
has them, asked into the passes (FDTD_TFSF=1) and in a launch of their own
(0), the split entry points and a batch; in FP64 the oracle's fields.
"""
import numpy as np
import pytest

import fdtd_b200 as F
import oracle as O
from cases import make

pytestmark = pytest.mark.gpu

STEPS = 150


def narrow(axis, width, inset):
    """A box of `width` cells along `axis`, its lower face inset + 6 cells in."""
    return dict(tfsf_inset=inset, box_offset=0, **{"NCELL" + "XY"[axis]: 2 * inset - 1 + width})


def wall(axis):
    """Faces one cell inside both walls of `axis`."""
    return dict(tfsf_inset=1, box_offset=0, **{"Ncpml" + "XYZ"[axis]: 0})


# insets 2 to 5: lower faces 8 to 11 cells in, every place in a 4-cell vector
BOXES = ([narrow(0, w, i) for w in (2, 3, 4) for i in (2, 3, 4, 5)] + [narrow(1, 2, 2), narrow(1, 3, 3)]
         + [wall(0), wall(1), wall(2)]
         + [dict(wall(1), NcpmlX=0, NCELLX=3), dict(wall(1), NcpmlX=0, NcpmlZ=0)])


def fields(p):
    s = F.Sim(p)
    s.step(STEPS)
    s.check()
    out = [s.field(c) for c in range(6)]
    s.close()
    return out


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("name", ["vacuum", "slab"])
@pytest.mark.parametrize("box", range(len(BOXES)))
def test_narrow_boxes_and_faces_on_walls(box, name, prec, monkeypatch):
    over = dict(BOXES[box], Tend=STEPS, inc_phi_deg=30.0)
    p = make(F, name, precision=prec, **over)
    monkeypatch.setenv("FDTD_TFSF", "0")
    ref = fields(p)
    assert max(np.abs(f).max() for f in ref) > 0
    if prec == F.FDTD_FP64:
        o = O.OracleSim(make(O, name, **over))
        o.step(STEPS)
        for c in (range(3), range(3, 6)):
            scale = max(np.abs(o.field(q)).max() for q in c)
            assert max(np.abs(ref[q] - o.field(q)).max() for q in c) <= 1e-11 * scale
    for tfsf in (None, "1"):
        if tfsf is None:
            monkeypatch.delenv("FDTD_TFSF")
        else:
            monkeypatch.setenv("FDTD_TFSF", tfsf)
        for got in (fields(p), split_fields(p), batch_fields(p)):
            for c in range(6):
                np.testing.assert_array_equal(got[c], ref[c], err_msg=f"component {c}, FDTD_TFSF={tfsf}")


def split_fields(p):
    s = F.Sim(p)
    for _ in range(STEPS):
        s.update_h()
        s.update_line()
        s.update_e()
    out = [s.field(c) for c in range(6)]
    s.close()
    return out


def batch_fields(p):
    b = F.Batch([p, make(F, "sphere_au", precision=p.precision, Tend=STEPS)])
    b.step(STEPS)
    out = [b.sim(0).field(c) for c in range(6)]
    b.close()
    return out


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
def test_statistics_tell_which_form_runs(prec, monkeypatch):
    """The TFSF launch's entries, none where the passes apply the corrections."""
    def entries(**over):
        s = F.Sim(make(F, "vacuum", precision=prec, **over))
        st = s.stats()
        s.close()
        return st.tfsf_entries_h, st.tfsf_entries_e

    assert entries() == (0, 0)
    for over in (dict(inc_theta_deg=20.0), BOXES[0], BOXES[6], BOXES[14], BOXES[16]):
        assert min(entries(**over)) > 0
    monkeypatch.setenv("FDTD_TFSF", "0")
    assert min(entries()) > 0
