"""FAST_SUBGRID with boxes that move, shrink, grow and jump: cells that an earlier
box left behind come back as zeros, whichever writer set them (an uploaded
level, a restart file, a snapshot, a source column beside the box, the
sweeps).  Bit for bit against the oracle, cell by cell over the whole grid."""
import numpy as np
import pytest

from gpu_common import pair, random_state, random_winds
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

N = (70, 41, 23)
# moved without overlap, nested, odd and even first cells, one plane, the whole grid
BOXES = [(3, 20, 2, 9, 2, 8), (40, 66, 20, 40, 10, 22), (45, 60, 25, 30, 12, 15), (30, 30, 20, 35, 1, 23),
         (1, 70, 1, 41, 1, 23), (18, 33, 5, 36, 4, 11), (64, 70, 41, 41, 23, 23), (2, 69, 1, 41, 3, 20)]


def _cfg(**over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=35, jvent=20, fall_mps=(0.2, 0.9, 1.5), bin_mass=(0.4, 0.3, 0.3),
              plume_km=8.0, volume_km3=1.0e-3, duration_h=1.0, sim_hours=1.0, winds="random", seed=5,
              fast_subgrid=True)
    kw.update(over)
    return syn.Config("cover", *N, 3, **kw)


def _same(gpu, ref, where):
    bad = np.argwhere(gpu.interior() != ref.interior())
    assert bad.size == 0, (where, f"{len(bad)} cells differ, first {bad[:3].tolist()}")
    vg, mg = gpu.TimeStepTotals()
    vr, mr = ref.TimeStepTotals()
    np.testing.assert_allclose(vg, vr, rtol=1e-12, atol=1e-300)
    np.testing.assert_allclose(mg, mr, rtol=1e-12, atol=1e-300)


KINDS = {"explicit": dict(use_cn=False), "cn": dict(use_cn=True),
         "lonlat": dict(use_cn=True, latlon=True, de=0.5, dn=0.5, latLL=20.0),
         "south": dict(use_cn=False, latlon=True, de=0.5, dn=0.5, latLL=-30.0)}


@pytest.mark.parametrize("kind", KINDS)
def test_boxes_that_move(kind):
    cfg, gpu, ref = pair(_cfg(**KINDS[kind]))
    winds = random_winds(cfg, 3)
    q = random_state(cfg, 4)
    flux = np.full((cfg.nz + 1, cfg.ns), 3.0e4, order="F")
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.005)
    gpu.snapshot_alloc(1)
    gpu.snapshot_save(0)
    for n, box in enumerate(BOXES):
        for m in (gpu, ref):
            m.set_subgrid(box)
            if n % 2:
                m.add_source(flux, 0.1)
            m.Set_BC(1)
            m.AdvectHorz(n)
            m.AdvectVert()
            m.Set_BC(2)
            m.DiffuseHorz(n)
            m.DiffuseVert()
        _same(gpu, ref, (n, box))
        if n == 2:  # a whole level again
            gpu.snapshot_load(0)
            ref.set_interior(q)
        if n == 4:
            for m in (gpu, ref):
                m.set_interior(q[::-1, ::-1])
    gpu.close()


@pytest.mark.parametrize("op", ["advect_x", "advect_y", "AdvectVert", "DiffuseVert"])
def test_one_sweep_after_the_box_jumps(op):
    """Every kernel by itself over a target that the box before filled."""
    for cn in (False, True):
        cfg, gpu, ref = pair(_cfg(use_cn=cn))
        winds, q = random_winds(cfg, 3), random_state(cfg, 4)
        for m in (gpu, ref):
            m.set_interior(q)
            m.set_winds(*winds)
            m.set_dt(0.005)
        for n, box in enumerate([BOXES[4], BOXES[1], BOXES[5], BOXES[4], BOXES[0], BOXES[2]]):
            for m in (gpu, ref):
                m.set_subgrid(box)
                m.add_source(np.full((cfg.nz + 1, cfg.ns), 2.0e4, order="F"), 0.1)
                getattr(m, op)()
            _same(gpu, ref, (op, cn, n, box))
        gpu.close()


def test_the_box_follows_the_cloud():
    """The occupied planes, and with them the next box, from a state inside one box."""
    cfg, gpu, ref = pair(_cfg(use_cn=True))
    q = np.zeros((cfg.nx, cfg.ny, cfg.nz, cfg.ns), order="F")
    q[30:40, 18:22, 3:9] = 1.0e5
    winds = random_winds(cfg, 3)
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.005)
    for n in range(4):
        assert tuple(gpu.get_minmax_index()) == tuple(ref.get_minmax_index())
        for m in (gpu, ref):
            m.Set_BC(1)
            m.AdvectHorz(n)
            m.AdvectVert()
            m.Set_BC(2)
            m.DiffuseHorz(n)
            m.DiffuseVert()
        _same(gpu, ref, n)
    gpu.close()
