"""The two forms of the adjoint's transposed sub-steps: the direct passes (the
default) and the coefficient arrays (FDTD_ADJ_FUSED=0)."""
import numpy as np
import pytest

import fdtd_b200 as F
from cases import make

pytestmark = pytest.mark.gpu

GOLD = dict(metal_custom=1, eps_inf=1.1431, omega_D=1.3202e16, gamma_D=1.0805e14, cp_A=(0.26698, 3.0834),
            cp_phi=(-1.2371, -1.0968), cp_Omega=(3.8711e15, 4.1684e15), cp_Gamma=(4.4642e14, 2.3555e15))


def design_sim(prec, name="sphere_big", box=(40, 48, 40, 48, 44, 48), **over):
    s = F.Sim(make(F, name, precision=prec, nano_sphere=0, design_box=list(box), **GOLD, **over))
    b = s.params.design_box
    rng = np.random.default_rng(3)
    s.set_design(rng.uniform(0, 1, (b[5] - b[4], b[3] - b[2], b[1] - b[0])).astype(np.float32))
    return s


def test_one_form_is_held(monkeypatch):
    """The adjoint's device memory: the adjoint fields and coefficient arrays,
    and the psi adjoints of the form that runs, once for the coefficient
    arrays and twice for the direct passes (psi: the psi slabs' bytes)."""
    import torch
    n, nc, es = 200, 20, 8
    psi = 12 * (2 * nc + 1) * n * n * es
    used = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("FDTD_ADJ_FUSED", mode)
        s = design_sim(F.FDTD_FP64, box=(98, 102, 98, 102, 98, 102), Tend=59,
                       **{k + a: v for a in "XYZ" for k, v in (("NCELL", n - 2 * nc - 1), ("Ncpml", nc))})
        assert (s.dims.nx, s.dims.ny, s.dims.nz) == (n, n, n)
        s.step(10)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s.forward([2], 30)
        s.backward()
        st = s.stats()
        used[mode] = before - torch.cuda.mem_get_info()[0] - 12 * n ** 3 * es - st.adj_record_bytes - st.dft_rows * 16
        s.close()
    slack = 48 << 20  # allocation granularity, graphs
    assert used["0"] <= 1.1 * psi + slack
    assert used["1"] <= 2.2 * psi + slack


@pytest.mark.parametrize("first", ["1", "0"])
def test_form_may_change_between_sweeps(first, monkeypatch):
    """The knob is read at each backward, whatever the forward found."""
    monkeypatch.setenv("FDTD_ADJ_FUSED", first)
    s = design_sim(F.FDTD_FP64, Tend=210)
    s.forward([2, 5], 40)
    out = []
    for mode in (first, "0" if first == "1" else "1", first):
        monkeypatch.setenv("FDTD_ADJ_FUSED", mode)
        out.append(s.backward())
    s.close()
    assert np.abs(out[0][0]).max() > 0
    for g, gp in out[1:]:
        assert np.abs(g - out[0][0]).max() <= 1e-11 * np.abs(out[0][0]).max()
        np.testing.assert_allclose(gp, out[0][1], rtol=1e-11)


# planes per thread 2, 3, 8 (the adjoint takes 2 to 8), blocks of 128 and 256
# threads; the last two ask the forward for the copied-ahead form and for more
# planes than the adjoint takes
SHAPES = ("flat:1", "flat:2", "flat:3:0:128", "flat:8:0:128", "flat:8:1", "flat:64")
_ARRAYS = {}


@pytest.mark.parametrize("prec", [F.FDTD_FP32, F.FDTD_FP64])
@pytest.mark.parametrize("model", [0, 3])
@pytest.mark.parametrize("shape", SHAPES)
def test_every_shape_agrees_with_the_coefficient_arrays(shape, model, prec, monkeypatch):
    """97 x 89 x 93 cells: the same sums in the same order; the source's atomics
    at the corners shared by two flux faces leave rounding."""
    def gradient(mode):
        monkeypatch.setenv("FDTD_ADJ_FUSED", mode)
        s = design_sim(prec, Tend=300, NONLOCAL=model)
        value = s.forward([2, 5], 40)
        out = (value, *s.backward())
        s.close()
        return out

    if (model, prec) not in _ARRAYS:
        _ARRAYS[model, prec] = gradient("0")
    value, g, gp = _ARRAYS[model, prec]
    monkeypatch.setenv("FDTD_PASS", shape)
    v1, g1, gp1 = gradient("1")
    tol = 1e-11 if prec == F.FDTD_FP64 else 1e-5
    assert v1 == value and np.abs(g).max() > 0
    assert np.abs(g1 - g).max() <= tol * np.abs(g).max()
    np.testing.assert_allclose(gp1, gp, rtol=tol)
