"""The marched advection sweeps at the sizes where a march can go wrong: lines
of one cell to several chunks and segments, rows that end inside a tile, sub-boxes
of either parity, clouds with still air around them, and limiter ratios on
the class bounds 0, 1/2, 1 and 2.  Bit for bit against the oracle; NOCYCLE
against the block kernels."""
import numpy as np
import pytest

from gpu_common import pair, random_winds
from volcano_ash3d_b200 import _lib, synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu


def _cfg(nx, ny, nz, ns, **over):
    ns_f = tuple(float(v) for v in np.linspace(0.05, 1.5, ns))
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, fall_mps=ns_f,
              bin_mass=(1.0 / ns,) * ns, plume_km=1.0, volume_km3=1.0e-3, duration_h=1.0, use_cn=True,
              sim_hours=1.0, winds="random", seed=31)
    kw.update(over)
    return syn.Config("march", nx, ny, nz, ns, **kw)


def _cloud(cfg, seed):
    """A blob of a few cells' width in exact zeros, small dyadic values (equal and doubled differences), a band
    of values whose differences straddle EPS_THRESH, and a tail down to the subnormals."""
    rng = np.random.default_rng(seed)
    shape = (cfg.nx, cfg.ny, cfg.nz, cfg.ns)
    i, j, k, g = np.meshgrid(*(np.arange(n) for n in shape), indexing="ij")
    r = np.abs(i - cfg.nx // 3) / 4.0 + np.abs(j - cfg.ny // 2) / 5.0 + np.abs(k - cfg.nz // 2) / 3.0
    q = np.where(r < 3.0, rng.uniform(0.0, 1.0e4, shape), 0.0)
    dy = (r >= 2.0) & (r < 4.0)
    q[dy] = rng.integers(0, 9, dy.sum()) * 0.25
    thin = (r >= 4.0) & (r < 5.0)
    q[thin] = rng.uniform(0.0, 4.0e-10, thin.sum())
    tail = (r >= 5.0) & (r < 6.0)
    q[tail] = 10.0 ** rng.uniform(-323.0, -100.0, tail.sum())
    return np.asfortranarray(q)


def _run(cfg, models, seed, box, ops):
    q, winds = _cloud(cfg, seed), random_winds(cfg, seed + 1)
    for m in models:
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.01)
        m.set_subgrid(box)
        for _ in range(2):
            for op in ops:
                getattr(m, op)()
    return [m.interior() for m in models], [m.outflows() for m in models]


def _same(states, flows):
    bad = np.argwhere(states[0] != states[1])
    assert bad.size == 0, f"{len(bad)} cells differ, first {bad[:3].tolist()}"
    for name in flows[0]:
        assert np.array_equal(flows[0][name], flows[1][name]), name


# (nx, ny, nz, ns): single cells, one cell beside a chunk of 8 or a segment of 10, odd rows, rows past a 32-lane tile
SIZES = [(3, 3, 3, 1), (33, 9, 10, 2), (17, 21, 11, 1), (40, 57, 19, 3), (65, 130, 61, 1)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("op", ["advect_x", "advect_y", "AdvectVert"])
@pytest.mark.parametrize("latlon", [False, True])
def test_marched_sweep_bitwise(size, op, latlon):
    cfg = _cfg(*size, latlon=latlon, de=0.5, dn=0.5, latLL=20.0)
    cfg, gpu, ref = pair(cfg)
    nx, ny, nz, _ = size
    _same(*_run(cfg, (gpu, ref), 7, (1, nx, 1, ny, 1, nz), [op]))
    gpu.close()


@pytest.mark.parametrize("box", [(1, 40, 1, 57, 1, 19), (4, 31, 9, 33, 2, 9), (3, 36, 8, 57, 3, 18), (9, 9, 20, 20, 5, 6)])
@pytest.mark.parametrize("op", ["advect_x", "advect_y", "AdvectVert"])
def test_marched_sweep_in_a_box_bitwise(box, op):
    cfg = _cfg(40, 57, 19, 2, fast_subgrid=True)
    cfg, gpu, ref = pair(cfg)
    _same(*_run(cfg, (gpu, ref), 8, box, [op]))
    gpu.close()


@pytest.mark.parametrize("limiter", ["none", "minmod", "superbee", "mc", "laxwen", "bw", "fromm"])
def test_limiters_bitwise(limiter):
    cfg = _cfg(40, 57, 19, 2, limiter=limiter)
    cfg, gpu, ref = pair(cfg)
    _same(*_run(cfg, (gpu, ref), 9, (1, 40, 1, 57, 1, 19), ["advect_x", "advect_y", "AdvectVert"]))
    gpu.close()


@pytest.mark.parametrize("limiter", ["superbee", "mc"])
def test_nocycle_matches_the_block_kernels(limiter, monkeypatch):
    lib = _lib.load()
    plain = lib.a3g_default_params

    def no_cycle(p):
        plain(p)
        p._obj.nocycle = 1

    monkeypatch.setattr(lib, "a3g_default_params", no_cycle)
    cfg = _cfg(40, 57, 19, 2, limiter=limiter)
    models = Ash3dGPU(cfg), Ash3dGPU(cfg)
    for d in range(3):
        models[1].set_variant(d, 1)
    _same(*_run(cfg, models, 10, (1, 40, 1, 57, 1, 19), ["advect_x", "advect_y", "AdvectVert"]))
    for m in models:
        m.close()
