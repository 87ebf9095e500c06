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


# members whose planes are no multiple of a block's, one at oblique incidence,
# and hydrodynamic ones
SETS = {"local": [("sphere_au", {}), ("sphere_big", dict(NCELLZ=78)), ("slab", dict(NCELLZ=26, inc_theta_deg=20.0))],
        "hydro": [("hydro", {}), ("hydro", dict(NCELLX=25, NCELLZ=36, nano_sphere_radius=8e-9))]}
_ALONE = {}


def members(name, prec):
    return [make(F, n, precision=prec, **over) for n, over in SETS[name]]


def alone(name, prec):
    if (name, prec) not in _ALONE:
        out = []
        for p in members(name, prec):
            s = F.Sim(p)
            s.step(133)
            out.append(([s.field(c) for c in range(6)], s.spectra()))
            s.close()
        _ALONE[name, prec] = out
    return _ALONE[name, prec]


@pytest.mark.parametrize("kz,ring", [(1, 0), (2, 1), (3, 0), (3, 1), (5, 1), (8, 0), (8, 1), (12, 1), (16, 0), (16, 1),
                                     (32, 1), (200, 0)])
@pytest.mark.parametrize("tail", ["0", "1"])
@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("name", sorted(SETS))
def test_every_form_agrees_with_single_runs(name, prec, tail, kz, ring, monkeypatch):
    """Planes per thread, copied ahead or not, and the last blocks split or not:
    what the tuner chooses between, each fixed by its knob."""
    ref = alone(name, prec)
    monkeypatch.setenv("FDTD_PASS", f"flat:{kz}:{ring}")
    monkeypatch.setenv("FDTD_BATCH_TAIL", tail)
    b = F.Batch(members(name, prec))
    tu = b.tuning()
    assert not tu["tuned"] and tu["stages"]["h"] == tu["stages"]["e"] == [4 if ring else 1] * 2
    planes = kz * (8 if kz == 1 else 4 if kz == 2 else 2 if kz <= 4 else 1)
    assert all(q["kchunk"] == planes for q in tu["buckets"])
    b.step(133)
    for i, (f, t) in enumerate(ref):
        for c in range(6):
            np.testing.assert_array_equal(b.sim(i).field(c), f[c], err_msg=f"member {i} component {c}")
        np.testing.assert_array_equal(b.spectra(i), t)
    b.close()


def test_split_last_blocks_of_a_tuned_batch(monkeypatch):
    """The knob holds where the tuner runs too."""
    sizes = ((84, 76, 80), (60, 60, 60))
    params = [make(F, "sphere_big", precision=F.FDTD_FP32, NCELLX=x, NCELLY=y, NCELLZ=z) for x, y, z in sizes]
    out = []
    for tail in ("0", "1"):
        monkeypatch.setenv("FDTD_BATCH_TAIL", tail)
        b = F.Batch(params)
        assert b.tuning()["tuned"]
        b.step(60)
        out.append([b.sim(i).field(c) for i in range(2) for c in range(6)])
        b.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
