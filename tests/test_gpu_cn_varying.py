"""Crank-Nicolson lines taken a batch of rows at a time: the y and z solves
where the coefficients vary along i (terrain), bit for bit, and the transposed
solves, to the 1e-12 of the largest value that the adjoint's differing order
of sums allows.  Lines of two rows, a batch more or less, chunks of 32 and one
cell beside them, and more grains than a block holds."""
import numpy as np
import pytest

import ash3d_oracle as orc
from gpu_common import pair, random_state, random_winds
from topo_common import level_winds
from volcano_ash3d_b200 import synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3, 1), (31, 9, 10, 2), (32, 8, 8, 9), (33, 17, 11, 3), (65, 41, 18, 1), (97, 10, 25, 10)]


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, use_cn=True,
              fall_mps=tuple(0.1 * (g + 1) for g in range(ns)), bin_mass=(1.0 / ns,) * ns, plume_km=1.0,
              volume_km3=1.0e-3, duration_h=1.0, winds="random", seed=71)
    kw.update(over)
    return syn.Config("varying", nx, ny, nz, ns, **kw)


TERRAIN = dict(zscaling_id=2, topo_km=0.4, topo_width_km=20.0)


def _state(m, cfg, winds, dt):
    m.set_interior(random_state(cfg, 5))
    m.set_winds(*winds)
    m.set_dt(dt)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("boxed", [False, True])
def test_terrain_solves_bitwise(size, boxed):
    cfg, gpu, ref = pair(_cfg(*size, fast_subgrid=boxed, **TERRAIN))
    nx, ny, nz, ns = size
    aloft = np.ones(ns, dtype=np.int32)
    if ns > 1:
        aloft[1] = 0
    for m in (gpu, ref):
        _state(m, cfg, level_winds(cfg, 6), 0.02)
        m.set_aloft(aloft)
        if boxed:
            m.set_subgrid((1, max(2, nx - 1), 2, ny, 1, max(2, nz - 1)))
        for n in (1, 2):
            m.Set_BC(2)
            m.DiffuseHorz(n)
            m.DiffuseVert()
    bad = np.argwhere(gpu.interior() != ref.interior())
    assert bad.size == 0, f"{len(bad)} cells differ, first {bad[:3].tolist()}"
    gpu.close()


# the adjoint refuses terrain, not cells whose size varies along i
GRIDS = {"projected": {}, "lonlat": dict(latlon=True, de=0.5, dn=0.5, latLL=20.0), "uneven": {}}


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("grid", GRIDS)
def test_transposed_solves(size, grid):
    cfg = _cfg(*size, **GRIDS[grid])
    geo = syn.geometry(cfg)
    if grid == "uneven":
        geo["kappa"] = np.asfortranarray(geo["kappa"] * (1.0 + 0.01 * np.arange(cfg.nx + 4))[:, None, None])
    gpu, ref = Ash3dGPU(cfg, geo=geo), orc.OracleModel(cfg, geo=geo)
    for m in (gpu, ref):
        _state(m, cfg, random_winds(cfg, 6), 0.02)
    rng = np.random.default_rng(8)
    lam = np.asfortranarray(rng.standard_normal(size))
    for op, args in (("adj_diffuse_horz", (1,)), ("adj_diffuse_horz", (2,)), ("adj_diffuse_vert", ())):
        a, b = getattr(gpu, op)(lam, *args), getattr(ref, op)(lam, *args)
        assert np.abs(a - b).max() <= 1.0e-12 * np.abs(b).max(), (op, args)
    gpu.close()
