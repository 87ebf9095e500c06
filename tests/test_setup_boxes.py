"""TFSF and flux boxes that reach outside the grid are refused at setup."""
import pytest

import fdtd_b200 as F
from cases import make


@pytest.mark.parametrize("axis", range(3))
@pytest.mark.parametrize("static", [0, 1])
def test_boxes_outside_the_grid_are_refused(axis, static):
    n = "Ncpml" + "XYZ"[axis]
    # faces at index 0: their H cells would be at -1
    for inset, offset in ((0, -1), (-1, -3)):
        with pytest.raises(F.FdtdError) as e:
            F.plan(make(F, "vacuum", tfsf_inset=inset, box_offset=offset, StaticField=static, **{n: 0}))
        assert "do not fit" in str(e.value)
    # faces inside, the absorption box from index -1 on: refused where it is sampled
    p = make(F, "vacuum", tfsf_inset=2, box_offset=-3, StaticField=static, **{n: 0})
    if static:
        assert F.plan(p).abs_start[axis] == -1
    else:
        with pytest.raises(F.FdtdError) as e:
            F.plan(p)
        assert "do not fit" in str(e.value)
    # the outermost box that fits
    d = F.plan(make(F, "vacuum", tfsf_inset=2, box_offset=-2, StaticField=static, **{n: 0}))
    assert d.abs_start[axis] == 0 and d.abs_end[axis] == (d.nx, d.ny, d.nz)[axis]
