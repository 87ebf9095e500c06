"""The direct E and H passes (flat.cuh) against the staged ones.

Both forms do the same operations in the same order per cell, so fields are
bit-identical: over row lengths of every remainder of the 16-byte vector and
of the padded pitch, grids of fewer planes than a thread takes, dispersive
cells inside the CPML, dielectric classes and periodic x and y, with the TFSF
corrections in the passes or in a launch of their own, in the fused step and
through the split entry points.
"""
import numpy as np
import pytest

import fdtd_b200 as F
from cases import make

pytestmark = pytest.mark.gpu

SPECS = ("flat:1", "flat:5", "flat:3:0:128", "flat:2:1", "flat:8:1", "flat:64:1", "flat:200")


def fields(name, prec, spec, monkeypatch, steps, **over):
    monkeypatch.setenv("FDTD_PASS", spec)
    s = F.Sim(make(F, name, precision=prec, **over))
    assert s.stats().h_staged == s.stats().e_staged == int(spec.startswith("staged"))
    s.step(steps)
    s.check()
    out = [s.field(c) for c in range(6)]
    spectra = s.reflectance() if s.params.periodic_xy else s.spectra()
    s.close()
    return out, spectra


def agree(name, prec, specs, monkeypatch, steps=150, **over):
    ref, tab = fields(name, prec, "staged:4:1:16:4", monkeypatch, steps, **over)
    assert max(np.abs(f).max() for f in ref) > 0
    for spec in specs:
        got, t = fields(name, prec, spec, monkeypatch, steps, **over)
        for c in range(6):
            np.testing.assert_array_equal(got[c], ref[c], err_msg=f"{name} {spec} component {c}")
        np.testing.assert_array_equal(t, tab)


@pytest.mark.parametrize("tfsf", ["0", "1"])
@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("name", ["sphere_big", "slab", "disks_slab", "hydro", "fixes", "periodic_spheres"])
def test_direct_passes_agree_with_the_staged_ones(name, prec, tfsf, monkeypatch):
    monkeypatch.setenv("FDTD_TFSF", tfsf)
    agree(name, prec, SPECS, monkeypatch)


@pytest.mark.parametrize("angles", [dict(inc_phi_deg=30.0), dict(inc_phi_deg=90.0, polar_psi_deg=20.0),
                                    dict(inc_theta_deg=25.0, inc_phi_deg=40.0, polar_psi_deg=10.0)])
@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
def test_every_polarisation_and_oblique_incidence(angles, prec, monkeypatch):
    """Oblique incidence keeps the TFSF launch whatever is asked for."""
    monkeypatch.setenv("FDTD_TFSF", "1")
    agree("slab", prec, ("flat:1", "flat:4:1"), monkeypatch, **angles)


@pytest.mark.parametrize("tfsf", ["0", "1"])
@pytest.mark.parametrize("name", ["sphere_big", "slab", "hydro"])
def test_split_entry_points_agree_with_the_fused_step(name, tfsf, monkeypatch):
    """Both in one run too: the clocks of the two forms stay together."""
    monkeypatch.setenv("FDTD_TFSF", tfsf)
    a, b = (F.Sim(make(F, name, precision=F.FDTD_FP32)) for _ in range(2))
    a.step(140)
    b.step(33)
    for _ in range(70):
        b.update_h()
        b.update_line()
        b.update_e()
        b.spectral_accumulate()
    b.step(37)
    for c in range(6):
        np.testing.assert_array_equal(a.field(c), b.field(c))
    np.testing.assert_array_equal(a.probe(), b.probe())
    np.testing.assert_array_equal(a.spectra(), b.spectra())
    a.close()
    b.close()


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("dx", range(8))
def test_every_row_remainder(dx, prec, monkeypatch):
    agree("sphere_au", prec, ("flat:1", "flat:7:1", "flat:2:0:128"), monkeypatch, steps=90, NCELLX=21 + dx, NCELLY=22 - dx % 3)


def test_tuned_and_untuned_direct_passes_agree(monkeypatch):
    """The shape the tuner keeps and the untimed rule's."""
    out = []
    for tune in ("1", "0"):
        monkeypatch.setenv("FDTD_TUNE", tune)
        s = F.Sim(make(F, "sphere_big", precision=F.FDTD_FP32))
        st = s.stats()
        assert st.h_staged == 0 and st.h_kchunk >= 1 and (st.h_ms > 0) == (tune == "1")
        s.step(140)
        out.append([s.field(c) for c in range(6)])
        s.close()
    for c in range(6):
        np.testing.assert_array_equal(out[0][c], out[1][c])


def test_unbuilt_direct_variant_is_rejected(monkeypatch):
    for spec in ("flat:0", "flat:4:2", "flat:4:0:96"):
        monkeypatch.setenv("FDTD_PASS", spec)
        with pytest.raises(F.FdtdError) as e:
            F.Sim(make(F, "vacuum", precision=F.FDTD_FP32))
        assert e.value.status == 1 and "not built" in str(e.value)


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("name,count", [("sphere_au", 1), ("sphere_big", 3), ("hydro", 2), ("slab", 5), ("sphere_big", 9)])
def test_batch_blocks_agree_with_single_runs(name, count, prec):
    """Batches under and over the tuner's size, members whose planes do not
    fill a block's groups, one member at oblique incidence (its TFSF launch
    runs beside the others' passes) and, after the batch, a member stepped by
    itself."""
    params = [make(F, name, precision=prec, NCELLZ=make(F, name).NCELLZ + i) for i in range(count)]
    if count > 2:
        params[1].update(inc_theta_deg=20.0, inc_phi_deg=15.0)
    b = F.Batch(params)
    b.step(133)
    for i, p in enumerate(params):
        alone = F.Sim(p)
        alone.step(140)
        b.sim(i).step(7)
        for c in range(6):
            np.testing.assert_array_equal(b.sim(i).field(c), alone.field(c), err_msg=f"member {i} component {c}")
        np.testing.assert_array_equal(b.sim(i).spectra(), alone.spectra())
        alone.close()
    b.close()


def test_batch_with_the_staged_passes(monkeypatch):
    """A batch whose members the direct passes do not take."""
    monkeypatch.setenv("FDTD_PASS", "staged:4:1:16:4")
    params = [make(F, n, precision=F.FDTD_FP32) for n in ("sphere_au", "sphere_big")]
    b = F.Batch(params)
    b.step(140)
    monkeypatch.delenv("FDTD_PASS")
    for i, p in enumerate(params):
        alone = F.Sim(p)
        alone.step(140)
        for c in range(6):
            np.testing.assert_array_equal(b.sim(i).field(c), alone.field(c), err_msg=f"member {i} component {c}")
        np.testing.assert_array_equal(b.spectra(i), alone.spectra())
        alone.close()
    b.close()


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("nx,ny,nonlocal_", [(0, 0, 0), (1, 3, 0), (2, 1, 3), (3, 2, 0), (5, 0, 3)])
def test_direct_adjoint_agrees_with_coefficient_arrays(nx, ny, nonlocal_, prec, monkeypatch):
    """Row lengths of every remainder and rows that end inside a warp, both
    dispersive models, a dielectric slab under the design box's metal: the
    same sums in the same order; the source's atomics at the corners shared
    by two flux faces leave rounding."""
    gold = dict(metal_custom=1, eps_inf=1.1431, omega_D=1.3202e16, gamma_D=1.0805e14, cp_A=(0.26698, 3.0834),
                cp_phi=(-1.2371, -1.0968), cp_Omega=(3.8711e15, 4.1684e15), cp_Gamma=(4.4642e14, 2.3555e15))
    out = []
    for mode in ("1", "0"):
        monkeypatch.setenv("FDTD_ADJ_FUSED", mode)
        s = F.Sim(make(F, "disks_slab", precision=prec, NCELLX=27 + nx, NCELLY=25 + ny, Tend=260, NONLOCAL=nonlocal_,
                       disk_diameter=4e-9, disk_nx=1, disk_ny=1, slab_thickness=4e-9,
                       design_box=[18, 22, 17, 20, 16, 19], **gold))
        s.set_design(np.random.default_rng(4).uniform(0, 1, (3, 3, 4)).astype(np.float32))
        value = s.forward([2, 5], 60)
        out.append((value, *s.backward()))
        s.close()
    assert out[0][0] == out[1][0]
    tol = 1e-11 if prec == F.FDTD_FP64 else 1e-5
    assert np.abs(out[1][1]).max() > 0
    assert np.abs(out[0][1] - out[1][1]).max() <= tol * np.abs(out[1][1]).max()
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=tol)
