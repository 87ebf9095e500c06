"""The oracle's CPML where the x slab is wider than the y slab.  Ey's near-x
slab takes the y axis's ce table (main.cu:2891), which ends before the slab
does; the coefficients beyond it are zero, as the product's tables have them,
and not what lies behind the table in memory."""
import numpy as np
import pytest

import oracle as O
from cases import make


@pytest.mark.parametrize("ny", [0, 2])
def test_x_slab_wider_than_y_slab(ny):
    """Three runs, with other values left in the freed blocks of the tables'
    sizes before each."""
    out = []
    for fill in (0.0, 1e30, -3.0):
        blocks = [np.full(n, fill) for n in range(1, 17) for _ in range(200)]
        del blocks
        s = O.OracleSim(make(O, "vacuum", NcpmlY=ny, tfsf_inset=4, box_offset=0, Tend=150))
        s.step(150)
        out.append([s.field(c) for c in range(6)])
    assert max(np.abs(f).max() for f in out[0][:3]) < 1.0  # the pulse's amplitude
    for other in out[1:]:
        for c in range(6):
            np.testing.assert_array_equal(other[c], out[0][c])
