"""Explicit diffusion: the fused horizontal sweeps and the marched vertical one
against the oracle (forward, bit for bit) and against the transpose applied
sweep by sweep (adjoint), on rows around the 30 columns of a warp, lines of one
segment and several, periodic rows, sub-boxes of either parity and stretched
levels."""
import numpy as np
import pytest

from gpu_common import pair, random_winds
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2,
              fall_mps=(0.3,) * ns, bin_mass=(1.0 / ns,) * ns, plume_km=0.4, volume_km3=1.0e-3,
              duration_h=1.0, use_cn=False, sim_hours=1.0, winds="random", seed=71)
    kw.update(over)
    return syn.Config("explicit", nx, ny, nz, ns, **kw)


def _state(cfg, seed):
    rng = np.random.default_rng(seed)
    q = rng.uniform(0.0, 1.0e3, (cfg.nx, cfg.ny, cfg.nz, cfg.ns))
    q[rng.uniform(size=q.shape) < 0.3] = 0.0
    q[rng.uniform(size=q.shape) < 0.05] = 3.0e-310
    return np.asfortranarray(q)


KINDS = dict(projected={}, lonlat=dict(latlon=True, de=0.5, dn=0.5, latLL=25.0),
             periodic=dict(latlon=True, periodic=True, dn=0.5, latLL=25.0))
SIZES = [(2, 3, 3, 1), (3, 8, 9, 2), (29, 17, 3, 1), (30, 16, 8, 2), (31, 33, 17, 1), (62, 70, 40, 2)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("kind", list(KINDS))
def test_sweeps_bitwise(size, kind):
    over = dict(KINDS[kind])
    if kind == "periodic":
        over["de"] = 360.0 / size[0]
    if kind == "projected":
        over["dz_profile"] = tuple(0.4 + 0.1 * (k % 3) for k in range(size[2]))
    cfg, gpu, ref = pair(_cfg(*size, **over))
    q = _state(cfg, 1)
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_dt(0.01)
        for itime in (1, 2):
            m.Set_BC(2)
            m.DiffuseHorz(itime)
            m.DiffuseVert()
    assert np.array_equal(gpu.interior(), ref.interior())
    gpu.close()


@pytest.mark.parametrize("box", [(2, 59, 3, 68, 2, 39), (31, 60, 9, 24, 5, 6), (1, 30, 1, 70, 1, 40)])
@pytest.mark.parametrize("itime", [1, 2])
def test_boxes_bitwise(box, itime):
    cfg, gpu, ref = pair(_cfg(62, 70, 40, 2, fast_subgrid=True))
    q = _state(cfg, 2)
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_subgrid(box)
        m.set_dt(0.02)
        m.Set_BC(2)
        m.DiffuseHorz(itime)
        m.DiffuseVert()
    assert np.array_equal(gpu.interior(), ref.interior())
    gpu.close()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("kind", list(KINDS))
def test_transpose(size, kind):
    """<D q, lam> = <q, D^T lam>: each side sums n products of terms below 1e3, exact to n roundings."""
    over = dict(KINDS[kind])
    if kind == "periodic":
        over["de"] = 360.0 / size[0]
    cfg, gpu, _ = pair(_cfg(*size, **over))
    rng = np.random.default_rng(3)
    q, lam = (rng.standard_normal((cfg.nx, cfg.ny, cfg.nz, cfg.ns)) for _ in range(2))
    gpu.set_winds(*random_winds(cfg, 4))  # the adjoint asks for winds, although these sweeps use none
    gpu.set_dt(0.01)
    for itime in (1, 2):
        gpu.set_interior(np.asfortranarray(q))
        gpu.DiffuseHorz(itime)
        gpu.DiffuseVert()
        fwd = float(np.sum(gpu.interior() * lam))
        back = gpu.adj_diffuse_horz(gpu.adj_diffuse_vert(lam), itime)
        scale = float(np.sum(np.abs(q) * np.abs(back)) + np.sum(np.abs(lam) * np.abs(gpu.interior())))
        assert abs(fwd - float(np.sum(q * back))) <= 2.0**-53 * q.size * scale
    gpu.close()
