"""The marched adjoint sweeps against the one-cell-per-thread gather (the same
expressions, so the same bits), on lines of one chunk and less, of several
chunks and segments, rows that end inside a tile, every limiter, and limiter
ratios on the class bounds."""
import numpy as np
import pytest

from gpu_common import random_winds
from volcano_ash3d_b200 import _lib, synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2,
              fall_mps=tuple(0.2 * (g + 1) for g in range(ns)), bin_mass=(1.0 / ns,) * ns, plume_km=1.0,
              volume_km3=1.0e-3, duration_h=1.0, use_cn=True, sim_hours=1.0, winds="random", seed=61)
    kw.update(over)
    return syn.Config("adjoint", nx, ny, nz, ns, **kw)


def _sweeps(m, cfg, seed):
    rng = np.random.default_rng(seed)
    shape = (cfg.nx, cfg.ny, cfg.nz, cfg.ns)
    q = rng.integers(0, 7, shape) * 0.5 * (rng.uniform(size=shape) < 0.7)
    some = rng.uniform(size=shape) < 0.3
    q[some] = rng.uniform(0.0, 50.0, some.sum())
    tiny = rng.uniform(size=shape) < 0.1
    q[tiny] = 10.0 ** rng.uniform(-323.0, -8.0, tiny.sum())
    lam = rng.standard_normal(shape)
    m.set_interior(np.asfortranarray(q))
    m.set_winds(*random_winds(cfg, seed + 1))
    m.set_dt(0.01)
    dep = np.asfortranarray(rng.standard_normal((cfg.nx, cfg.ny, cfg.ns)))
    return [m.adj_advect_x(lam), m.adj_advect_y(lam), m.adj_advect_z(lam, dep)]


def _compare(cfg, seed=3):
    a, b = Ash3dGPU(cfg), Ash3dGPU(cfg)
    b.set_variant(5, 1)
    for name, x, y in zip("xyz", _sweeps(a, cfg, seed), _sweeps(b, cfg, seed)):
        bad = np.argwhere(x != y)
        assert bad.size == 0, f"{name}: {len(bad)} cells differ, first {bad[:3].tolist()}"
    for m in (a, b):
        m.close()


@pytest.mark.parametrize("size", [(3, 3, 3, 1), (33, 9, 10, 2), (17, 21, 11, 1), (40, 57, 19, 3), (65, 130, 61, 1)])
@pytest.mark.parametrize("latlon", [False, True])
def test_sizes(size, latlon):
    _compare(_cfg(*size, latlon=latlon, de=0.5, dn=0.5, latLL=20.0))


@pytest.mark.parametrize("limiter", ["none", "minmod", "superbee", "mc", "laxwen", "bw", "fromm"])
@pytest.mark.parametrize("nocycle", [0, 1])
def test_limiters(limiter, nocycle, monkeypatch):
    lib = _lib.load()
    plain = lib.a3g_default_params

    def params(p):
        plain(p)
        p._obj.nocycle = nocycle

    monkeypatch.setattr(lib, "a3g_default_params", params)
    _compare(_cfg(40, 31, 19, 2, limiter=limiter), seed=5)
