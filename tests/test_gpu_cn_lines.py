"""The tiled Crank-Nicolson solves and the factor tables at the line lengths
where a chunk of 16 cells can go wrong (2 cells, a chunk and its neighbours,
two and three chunks), in boxes of either parity, on clouds whose diffused
tails reach the subnormals, with geometry that is constant along the line or
not; bit for bit against the oracle, over two values of dt."""
import numpy as np
import pytest

from gpu_common import pair
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, fall_mps=(0.5,) * ns,
              bin_mass=(1.0 / ns,) * ns, plume_km=0.4, volume_km3=1.0e-3, duration_h=1.0, use_cn=True,
              sim_hours=1.0, winds="random", seed=41)
    kw.update(over)
    return syn.Config("lines", nx, ny, nz, ns, **kw)


def _state(cfg, seed):
    """Two point sources in exact zeros, a dense corner, and a tail through the subnormals."""
    rng = np.random.default_rng(seed)
    q = np.zeros((cfg.nx, cfg.ny, cfg.nz, cfg.ns), order="F")
    q[cfg.nx // 2, cfg.ny // 2, cfg.nz // 2, :] = 1.0e5
    q[-1, -1, -1, :] = 3.0
    a, b, c = (max(1, n // 3) for n in q.shape[:3])
    q[:a, :b, :c, :] = rng.uniform(0.0, 1.0e3, (a, b, c, cfg.ns))
    q[-a:, :b, -c:, :] = 10.0 ** rng.uniform(-323.0, -250.0, (a, b, c, cfg.ns))
    return q


def _compare(cfg, ops, box):
    cfg, gpu, ref = pair(cfg)
    q = _state(cfg, 5)
    for m in (gpu, ref):
        m.set_interior(q)
        m.set_subgrid(box)
    for dt in (0.02, 0.02, 0.31):
        for op in ops:
            for m in (gpu, ref):
                m.set_dt(dt)
                op(m)
        a, b = gpu.interior(), ref.interior()
        bad = np.argwhere(a != b)
        assert bad.size == 0, f"dt {dt}: {len(bad)} cells differ, first {bad[:3].tolist()}"
    gpu.close()


HORZ = [lambda m: m.DiffuseHorz(1), lambda m: m.DiffuseHorz(2)]
VERT = [lambda m: m.DiffuseVert()]


@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 18, 32, 33, 49])
@pytest.mark.parametrize("kind", ["projected", "lonlat", "stretched"])
def test_lines_bitwise(n, kind):
    over = dict(latlon=True, de=0.5, dn=0.5, latLL=30.0) if kind == "lonlat" else {}
    if kind == "stretched":
        over["dz_profile"] = tuple(0.3 + 0.1 * (k % 3) for k in range(n))
    m = max(3, n)
    box = (1, m, 1, m, 1, n)
    _compare(_cfg(m, m, n, 2, **over), HORZ + VERT, box)


@pytest.mark.parametrize("box", [(2, 34, 3, 36, 2, 20), (5, 35, 4, 19, 1, 23), (8, 9, 20, 21, 7, 8), (3, 18, 17, 33, 5, 24)])
def test_boxes_bitwise(box):
    # DiffuseHorz widens the box by a cell where FAST_SUBGRID is on: give the solves this one
    cfg = _cfg(37, 38, 24, 2)
    cfg, gpu, ref = pair(cfg)
    gpu.close()
    _compare(_cfg(37, 38, 24, 2), VERT, box)
    wide = _cfg(37, 38, 24, 2, fast_subgrid=True)
    inner = (box[0] + 1, max(box[0] + 1, box[1] - 1), box[2] + 1, max(box[2] + 1, box[3] - 1), box[4], box[5])
    _compare(wide, HORZ[:1], inner)


def test_many_distinct_lines_bitwise():
    # over 1024 distinct lines: the tables' 32-lines-a-block form (x of a lon/lat grid; y and z over terrain)
    _compare(_cfg(40, 70, 16, 1, latlon=True, de=0.5, dn=0.5, latLL=10.0), HORZ + VERT, (1, 40, 1, 70, 1, 16))
    _compare(_cfg(41, 39, 33, 2, zscaling_id=2, topo_km=1.5, topo_width_km=30.0), HORZ + VERT, (1, 41, 1, 39, 1, 33))
