"""NaN and infinite concentrations and missing (NaN) winds in the marched
sweeps: the block kernels, which form every interface by itself, give the same
cells the same values, so that what a broken cell reaches does not depend on the
kernel that swept it.  The sign of a zero aside, bit for bit."""
import numpy as np
import pytest

from gpu_common import pair, random_state, random_winds
from topo_common import level_winds
from volcano_ash3d_b200 import _lib, synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu

SIZE = (43, 57, 21, 2)
KINDS = {"projected": {}, "lonlat": dict(latlon=True, de=0.5, dn=0.5, latLL=20.0),
         "periodic": dict(latlon=True, periodic=True, de=360.0 / SIZE[0], dn=0.5, latLL=20.0),
         "terrain": dict(zscaling_id=1, topo_km=0.4, topo_width_km=20.0)}


def _cfg(**over):
    nx, ny, nz, ns = SIZE
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=20, jvent=30, fall_mps=(0.1, 0.8), bin_mass=(0.5, 0.5), plume_km=1.0,
              volume_km3=1.0e-3, duration_h=1.0, use_cn=True, sim_hours=1.0, winds="random", seed=91)
    kw.update(over)
    return syn.Config("nonfinite", nx, ny, nz, ns, **kw)


def _cells(rng, shape, n):
    return tuple(rng.integers(0, m, n) for m in shape)


def _state(cfg, seed, broken):
    """A cloud in the middle of still air, with single broken cells in both."""
    rng = np.random.default_rng(seed)
    q = random_state(cfg, seed)
    q[:, :, : cfg.nz // 3] = 0.0
    q[: cfg.nx // 4] = 0.0
    if broken == "nan":
        q[_cells(rng, q.shape, 40)] = np.nan
        q[_cells(rng, q.shape, 40)] = -np.nan
    elif broken == "inf":
        q[_cells(rng, q.shape, 40)] = np.inf
    elif broken == "huge":
        q[_cells(rng, q.shape, 40)] = 1.0e300
    return np.asfortranarray(q)


def _winds(cfg, seed, missing):
    rng = np.random.default_rng(seed + 50)
    w = level_winds(cfg, seed) if cfg.zscaling_id else random_winds(cfg, seed)
    if missing:
        for v in w:
            v[_cells(rng, v.shape, 60)] = np.nan
            v[_cells(rng, v.shape, 60)] = -np.nan
    return w


def _compare(cfg, q, winds, ops, general, box=None):
    out = []
    geo = syn.geometry(cfg)
    for variants in ({}, general):
        m = Ash3dGPU(cfg, geo=geo)
        for d, v in variants.items():
            m.set_variant(d, v)
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.005)
        if box:
            m.set_subgrid(box)
        for op in ops:
            m.Set_BC(1)
            getattr(m, op[0])(*op[1:]) if isinstance(op, tuple) else getattr(m, op)()
        out.append((m.interior(), m.outflows()))
        m.close()
    (a, fa), (b, fb) = out
    assert np.isnan(b).any() or not np.isnan(q).any()
    bad = np.argwhere(~((a == b) | (np.isnan(a) & np.isnan(b))))
    assert bad.size == 0, f"{len(bad)} cells differ, first {[(t.tolist(), a[tuple(t)], b[tuple(t)]) for t in bad[:3]]}"
    for name in fa:
        assert np.array_equal(fa[name], fb[name], equal_nan=True), name


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("op", ["advect_x", "advect_y", "AdvectVert"])
@pytest.mark.parametrize("broken", ["nan", "inf", "huge"])
def test_broken_cells(kind, op, broken):
    cfg = _cfg(**KINDS[kind])
    _compare(cfg, _state(cfg, 3, broken), _winds(cfg, 4, False), [op], {0: 1, 1: 1, 2: 1})


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("op", ["advect_x", "advect_y", "AdvectVert"])
def test_missing_winds(kind, op):
    cfg = _cfg(**KINDS[kind])
    _compare(cfg, _state(cfg, 5, ""), _winds(cfg, 6, True), [op], {0: 1, 1: 1, 2: 1})


@pytest.mark.parametrize("broken", ["nan", "inf"])
def test_broken_cells_in_a_box(broken):
    cfg = _cfg(fast_subgrid=True)
    for op in ("advect_x", "advect_y", "AdvectVert"):
        _compare(cfg, _state(cfg, 7, broken), _winds(cfg, 8, True), [op], {0: 1, 1: 1, 2: 1}, (4, 38, 3, 55, 2, 18))


@pytest.mark.parametrize("limiter", ["none", "minmod", "mc", "laxwen", "bw", "fromm"])
def test_other_limiters(limiter):
    cfg = _cfg(limiter=limiter)
    for op in ("advect_x", "advect_y", "AdvectVert"):
        _compare(cfg, _state(cfg, 9, "nan"), _winds(cfg, 10, True), [op], {0: 1, 1: 1, 2: 1})


@pytest.mark.parametrize("kind", ["projected", "lonlat", "terrain"])
@pytest.mark.parametrize("op", [("DiffuseHorz", 1), ("DiffuseHorz", 2), ("DiffuseVert",)])
@pytest.mark.parametrize("broken", ["nan", "inf", "huge"])
def test_broken_cells_in_the_solves(kind, op, broken):
    cfg = _cfg(**KINDS[kind])
    _compare(cfg, _state(cfg, 11, broken), _winds(cfg, 12, False), [op], {3: 1, 4: 0})


@pytest.mark.parametrize("kind", ["projected", "lonlat"])
@pytest.mark.parametrize("broken", ["nan", "inf", "huge", ""])
def test_adjoint_sweeps(kind, broken):
    """The marched transposed sweeps against the one-cell-per-thread gather, over broken states (or missing winds)."""
    cfg = _cfg(**KINDS[kind])
    q, winds = _state(cfg, 13, broken), _winds(cfg, 14, not broken)
    lam = np.asfortranarray(np.random.default_rng(15).standard_normal(q.shape))
    geo = syn.geometry(cfg)
    out = []
    for variant in (0, 1):
        m = Ash3dGPU(cfg, geo=geo)
        m.set_variant(5, variant)
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.005)
        out.append([m.adj_advect_x(lam), m.adj_advect_y(lam), m.adj_advect_z(lam, None)])
        m.close()
    for name, a, b in zip("xyz", *out):
        assert np.isnan(b).any() == (broken != "huge"), name
        assert np.array_equal(a, b, equal_nan=True), name


@pytest.mark.parametrize("latlon", [False, True])
def test_a_missing_level_sets_no_time_step(latlon):
    """Adjust_DT passes over cells whose wind is missing: a thin level without any wind does not bring the settling
    speed's limit in."""
    dz = tuple(0.02 if k == 5 else 0.5 for k in range(SIZE[2]))
    cfg, gpu, ref = pair(_cfg(dz_profile=dz, latlon=latlon, de=0.5, dn=0.5, latLL=20.0))
    winds = [0.01 * v for v in random_winds(cfg, 16)]
    winds[2][:, :, 2 + 5] = np.nan
    winds[2][7, 9, 2 + 8] = np.nan
    for m in (gpu, ref):
        m.set_winds(*winds)
    dt = ref.Adjust_DT(0.0, 1.0e9, 1.0e9)
    assert gpu.Adjust_DT(0.0, 1.0e9, 1.0e9) == dt
    gpu.close()
