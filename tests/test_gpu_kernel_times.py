"""a3g_kernel_times counts the launches that happened: explicit diffusion with
its horizontal sweeps in one launch and in two, forward and transposed, and
the Crank-Nicolson tables only when they are rebuilt."""
import numpy as np
import pytest

from gpu_common import random_state, random_winds
from volcano_ash3d_b200 import synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu


def _model(uneven=False, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=20, jvent=10, fall_mps=(0.1, 0.8), bin_mass=(0.5, 0.5), plume_km=1.0,
              volume_km3=1.0e-3, duration_h=1.0, use_cn=False, sim_hours=1.0, winds="random", seed=91)
    kw.update(over)
    cfg = syn.Config("times", 40, 21, 11, 2, **kw)
    geo = syn.geometry(cfg)
    if uneven:  # cells whose size varies along i: the horizontal sweeps one by one
        geo["kappa"] = np.asfortranarray(geo["kappa"] * (1.0 + 0.01 * np.arange(cfg.nx + 4))[:, None, None])
    m = Ash3dGPU(cfg, geo=geo)
    m.set_interior(random_state(cfg, 3))
    m.set_winds(*random_winds(cfg, 4))
    m.set_dt(0.005)
    return m


def _counts(m, *calls):
    for c in calls:
        c()
    m.kernel_timing(True)
    for c in calls:
        c()
    t = m.kernel_times()
    m.kernel_timing(False)
    assert all((ms > 0.0) == (n > 0) for ms, n in t.values())
    return {k: n for k, (_, n) in t.items() if n}


@pytest.mark.parametrize("uneven", [False, True])
def test_explicit_diffusion(uneven):
    m = _model(uneven)
    got = _counts(m, lambda: m.DiffuseHorz(1), lambda: m.DiffuseHorz(2), m.DiffuseVert)
    assert got == (dict(diff_x=2, diff_y=2, diff_z=1) if uneven else dict(diff_x=2, diff_z=1))
    lam = np.ones((40, 21, 11, 2), order="F")
    got = _counts(m, lambda: m.adj_diffuse_horz(lam, 1))
    assert got["adjoint"] == (2 if uneven else 1)
    m.close()


def test_factor_tables():
    m = _model(use_cn=True)
    assert "cn_table" not in _counts(m, lambda: m.DiffuseHorz(1), m.DiffuseVert)
    got = _counts(m, lambda: m.set_dt(0.006), lambda: m.DiffuseHorz(1), m.DiffuseVert)
    assert got["cn_table"] == 1 and got["cn_solve_x"] == got["cn_solve_y"] == got["cn_solve_z"] == 1
    m.close()
