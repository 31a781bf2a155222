"""The x march (a row per lane) on grids with rows enough for it, over row
lengths whose last chunk, ghost cells and segments fall every way, wrapped
rows among them: the wrapped ghosts of a row of 8m+1 cells lie in two chunks.
Whole grids and boxes, with a grain that is not aloft, bit for bit against the
oracle; and the same rows where they are too few, which take a warp each."""
import numpy as np
import pytest

from gpu_common import pair, random_state, random_winds
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

MANY, FEW = (53, 51, 2), (9, 11, 2)  # ny, nz, ns: 5406 rows, 198 rows; 53*51 is no multiple of 32


def _cfg(nx, rows, **over):
    ny, nz, ns = rows
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, fall_mps=(0.1, 0.8),
              bin_mass=(0.5, 0.5), plume_km=1.0, volume_km3=1.0e-3, duration_h=1.0, use_cn=True, sim_hours=1.0,
              winds="random", seed=31)
    kw.update(over)
    return syn.Config("rowmarch", nx, ny, nz, ns, **kw)


def _sweeps(cfg, box=None, aloft=(1, 1)):
    cfg, gpu, ref = pair(cfg)
    q, winds = random_state(cfg, 3), random_winds(cfg, 4)
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_winds(*winds)
        m.set_dt(0.01)
        m.set_aloft(aloft)
        if box:
            m.set_subgrid(box)
        for _ in range(2):
            m.advect_x()
    bad = np.argwhere(gpu.interior() != ref.interior())
    assert bad.size == 0, f"{len(bad)} cells differ, first {bad[:3].tolist()}"
    a, b = gpu.outflows(), ref.outflows()
    for name in a:
        assert np.array_equal(a[name], b[name]), name
    gpu.close()


@pytest.mark.parametrize("nx", [3, 9, 17, 32, 33, 39, 65, 361])
@pytest.mark.parametrize("rows", [MANY, FEW])
@pytest.mark.parametrize("periodic", [False, True])
def test_rows(nx, rows, periodic):
    over = dict(latlon=True, periodic=True, de=360.0 / nx, dn=0.5, latLL=20.0) if periodic else {}
    _sweeps(_cfg(nx, rows, **over), aloft=(1, 0) if nx == 33 else (1, 1))


@pytest.mark.parametrize("nx", [33, 65])
def test_a_box_over_wrapped_rows(nx):
    cfg = _cfg(nx, MANY, latlon=True, periodic=True, de=360.0 / nx, dn=0.5, latLL=20.0, fast_subgrid=True)
    _sweeps(cfg, box=(1, nx, 4, 47, 3, 50))


@pytest.mark.parametrize("box", [(4, 31, 9, 33, 2, 9), (3, 36, 8, 53, 3, 18), (9, 9, 20, 20, 5, 6), (1, 40, 1, 53, 1, 51)])
def test_boxes(box):
    _sweeps(_cfg(40, MANY, fast_subgrid=True), box=box, aloft=(0, 1))
