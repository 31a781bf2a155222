"""The marched sweeps over terrain, where the geometry varies along i: lines of
a few cells and of several chunks and segments of either length, one grain and
many, both terrain scalings, bit for bit against the oracle; and cells whose
size varies along i without terrain, which take the same z and y marches."""
import numpy as np
import pytest

import ash3d_oracle as orc
from gpu_common import random_state, random_winds
from topo_common import level_winds
from volcano_ash3d_b200 import synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3, 1), (33, 9, 10, 2), (50, 97, 11, 1), (99, 49, 18, 3), (200, 100, 33, 1), (193, 66, 40, 9)]


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, use_cn=True,
              fall_mps=tuple(0.1 * (g + 1) for g in range(ns)), bin_mass=(1.0 / ns,) * ns, plume_km=1.0,
              volume_km3=1.0e-3, duration_h=1.0, winds="random", seed=81)
    kw.update(over)
    return syn.Config("terrain", nx, ny, nz, ns, **kw)


def _compare(cfg, geo, winds, box=None):
    gpu, ref = Ash3dGPU(cfg, geo=geo), orc.OracleModel(cfg, geo=geo)
    q = random_state(cfg, 5)
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.005)
        if box:
            m.set_subgrid(box)
        for op in ("advect_x", "AdvectVert", "advect_y", "AdvectVert"):
            m.Set_BC(1)
            getattr(m, op)()
    bad = np.argwhere(gpu.interior() != ref.interior())
    assert bad.size == 0, f"{len(bad)} cells differ, first {bad[:3].tolist()}"
    a, b = gpu.outflows(), ref.outflows()
    for name in a:
        assert np.array_equal(a[name], b[name]), name
    gpu.close()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("scaling", [1, 2])
@pytest.mark.parametrize("boxed", [False, True])
def test_terrain_sweeps_bitwise(size, scaling, boxed):
    cfg = _cfg(*size, zscaling_id=scaling, topo_km=0.4, topo_width_km=20.0, fast_subgrid=boxed)
    nx, ny, nz, _ = size
    box = (min(2, nx - 1), nx, 1, max(2, ny - 3), 1, max(2, nz - 2)) if boxed else None
    _compare(cfg, syn.geometry(cfg), level_winds(cfg, 6), box)


def test_two_grains_a_thread_bitwise():
    """Enough rows for the x sweep that takes two grains of a row together."""
    cfg = _cfg(193, 129, 40, 17, zscaling_id=2, topo_km=0.4, topo_width_km=20.0)
    _compare(cfg, syn.geometry(cfg), level_winds(cfg, 6))


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("limiter", ["superbee", "none", "mc"])
def test_uneven_cells_bitwise(size, limiter):
    cfg = _cfg(*size, limiter=limiter)
    geo = syn.geometry(cfg)
    geo["kappa"] = np.asfortranarray(geo["kappa"] * (1.0 + 0.01 * np.arange(cfg.nx + 4))[:, None, None])
    geo["sig_nz"] = np.asfortranarray(geo["sig_nz"] * (1.0 + 0.003 * np.arange(cfg.nx + 4))[:, None, None])
    _compare(cfg, geo, random_winds(cfg, 6))
