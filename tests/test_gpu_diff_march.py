"""The marched explicit vertical diffusion (grids of 250,000 cells and more):
columns of a few levels to several segments, rows that end inside a warp,
sub-boxes, stretched levels; forward bit for bit against the oracle, the
transpose by <D q, lam> = <q, D^T lam>."""
import numpy as np
import pytest

from gpu_common import pair, random_winds
from volcano_ash3d_b200 import synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu

SIZES = [(63, 70, 57, 1), (300, 281, 3, 2), (29, 33, 263, 1)]


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, fall_mps=(0.3,) * ns,
              bin_mass=(1.0 / ns,) * ns, plume_km=0.4, volume_km3=1.0e-3, duration_h=1.0, use_cn=False, sim_hours=1.0,
              winds="random", seed=71, dz_profile=tuple(0.4 + 0.1 * (k % 3) for k in range(nz)))
    kw.update(over)
    return syn.Config("diffmarch", nx, ny, nz, ns, **kw)


def _state(cfg, seed):
    rng = np.random.default_rng(seed)
    q = rng.uniform(0.0, 1.0e3, (cfg.nx, cfg.ny, cfg.nz, cfg.ns))
    q[rng.uniform(size=q.shape) < 0.3] = 0.0
    return np.asfortranarray(q)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("boxed", [False, True])
def test_sweep_bitwise(size, boxed):
    cfg, gpu, ref = pair(_cfg(*size, fast_subgrid=boxed))
    q = _state(cfg, 1)
    for m in (gpu, ref):
        m.set_interior(q)
        if boxed:
            m.set_subgrid((3, cfg.nx - 1, 2, cfg.ny, 1, max(2, cfg.nz - 2)))
        m.set_dt(0.01)
        for _ in range(2):
            m.Set_BC(2)
            m.DiffuseVert()
    assert np.array_equal(gpu.interior(), ref.interior())
    gpu.close()


@pytest.mark.parametrize("size", SIZES)
def test_transpose(size):
    """Each side sums n products of terms below 1e3: exact to n roundings."""
    cfg = _cfg(*size)
    gpu = Ash3dGPU(cfg)
    rng = np.random.default_rng(3)
    q, lam = (rng.standard_normal((cfg.nx, cfg.ny, cfg.nz, cfg.ns)) for _ in range(2))
    gpu.set_winds(*random_winds(cfg, 4))
    gpu.set_dt(0.01)
    gpu.set_interior(np.asfortranarray(q))
    gpu.DiffuseVert()
    out = gpu.interior()
    back = gpu.adj_diffuse_vert(lam)
    scale = float(np.sum(np.abs(q) * np.abs(back)) + np.sum(np.abs(lam) * np.abs(out)))
    assert abs(float(np.sum(out * lam)) - float(np.sum(q * back))) <= 2.0**-53 * q.size * scale
    gpu.close()
