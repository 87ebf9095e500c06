"""The dispersive cells in blocks of the pass launches and in launches of their
own beside the E pass (FDTD_CELLS; by default by their number): the same
bits."""
import numpy as np
import pytest

import fdtd_b200 as F
from cases import make

pytestmark = pytest.mark.gpu

GOLD = dict(metal_custom=1, eps_inf=1.1431, omega_D=1.3202e16, gamma_D=1.0805e14, cp_A=(0.26698, 3.0834),
            cp_phi=(-1.2371, -1.0968), cp_Omega=(3.8711e15, 4.1684e15), cp_Gamma=(4.4642e14, 2.3555e15))


def state(s):
    out = [s.field(c) for c in range(6)]
    out.append(s.reflectance() if s.params.periodic_xy else s.spectra())
    s.close()
    return out


def same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("passes", ["flat:4:0", "flat:2:1", "staged:4:1:16:4"])
@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("name", ["sphere_au", "slab", "hydro", "disks_slab", "periodic_spheres", "oblique"])
def test_blocks_and_launches_agree(name, prec, passes, monkeypatch):
    monkeypatch.setenv("FDTD_PASS", passes)
    over = dict(inc_theta_deg=20.0, inc_phi_deg=30.0) if name == "oblique" else {}
    p = make(F, "slab" if name == "oblique" else name, precision=prec, **over)
    out = []
    for cells in ("0", "1"):
        monkeypatch.setenv("FDTD_CELLS", cells)
        s = F.Sim(p)
        s.step(150)
        s.check()
        out.append(state(s))
        s = F.Sim(p)  # eager and graph steps, split calls
        s.step(20)
        for _ in range(40):
            s.update_h()
            s.update_line()
            s.update_e()
            s.spectral_accumulate()
        s.step(90)
        out.append(state(s))
    for other in out[1:]:
        same(out[0], other)


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("name", ["slab", "hydro"])
def test_batch_blocks_and_launches_agree(name, prec, monkeypatch):
    params = [make(F, name, precision=prec, NCELLX=21 + 3 * i) for i in range(3)]
    out = []
    for cells in ("0", "1"):
        monkeypatch.setenv("FDTD_CELLS", cells)
        b = F.Batch(params)
        b.step(140)  # one graph period and eager steps
        out.append([b.sim(i).field(c) for i in range(3) for c in range(6)] + [b.spectra(i) for i in range(3)])
        b.close()
    same(*out)


@pytest.mark.parametrize("model", [0, 3])
def test_recorded_trajectories_agree(model, monkeypatch):
    """The forward's record and the recomputed segments, FP64."""
    out = []
    for cells in ("0", "1"):
        monkeypatch.setenv("FDTD_CELLS", cells)
        for gb in ("1", "0"):
            monkeypatch.setenv("FDTD_ADJ_RECORD_GB", gb)
            s = F.Sim(make(F, "sphere_big", precision=F.FDTD_FP64, nano_sphere=0, Tend=300, NONLOCAL=model,
                           design_box=[40, 48, 40, 46, 44, 48], **GOLD))
            s.set_design(np.random.default_rng(3).uniform(0, 1, (4, 6, 8)).astype(np.float32))
            out.append((s.forward([2, 5], 40), *s.backward()))
            s.close()
    for o in out[1:]:
        assert o[0] == out[0][0]
        assert np.abs(o[1] - out[0][1]).max() <= 1e-11 * np.abs(out[0][1]).max() and np.abs(o[1]).max() > 0
        np.testing.assert_allclose(o[2], out[0][2], rtol=1e-11)


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("model", [0, 3])
def test_count_chooses(model, prec, monkeypatch):
    """Just under and over one wave of blocks on 148 multiprocessors (75,776
    cells): the launches of one step tell which form runs."""
    import torch
    wave = 2 * 256 * torch.cuda.get_device_properties(0).multi_processor_count

    def sim(r):
        return F.Sim(make(F, "hydro" if model else "sphere_au", precision=prec, NCELLX=47, NCELLY=47, NCELLZ=47,
                          nano_sphere_radius=r * 2e-9 + 1e-10))

    for r in (16, 18, 19):  # 51,240, 73,092 and 86,034 cells
        monkeypatch.delenv("FDTD_CELLS", raising=False)
        s = sim(r)
        n = sum(s.dims.n_metal_cells)
        s.step(2)  # (the first step has the DFT's launches too)
        before = s.stats().kernels
        s.step(1)
        assert s.stats().kernels - before == 2 + (n > wave) * (3 if model else 1), (r, n)
        s.step(120)
        auto = state(s)
        monkeypatch.setenv("FDTD_CELLS", "0" if n > wave else "1")
        s = sim(r)
        s.step(123)
        same(auto, state(s))
