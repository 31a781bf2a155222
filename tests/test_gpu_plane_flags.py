"""The occupied planes that FAST_SUBGRID's box comes from, against numpy: rows
from one column to several turns of a warp, one grain to more than a block's
share, ash in every cell, in single cells (the last grain's, the last
column's), above, at and just below the threshold, NaN cells, and nothing."""
import numpy as np
import pytest

from gpu_common import pair, random_state
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

SIZES = [(3, 40, 9, 2), (4, 7, 30, 1), (5, 5, 5, 60), (33, 9, 8, 3), (64, 31, 5, 9), (129, 12, 7, 4), (300, 17, 9, 5)]


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2, fall_mps=(0.3,) * ns,
              bin_mass=(1.0 / ns,) * ns, plume_km=1.0, volume_km3=1.0e-3, duration_h=1.0, use_cn=True, sim_hours=1.0,
              winds="random", seed=5, fast_subgrid=True)
    kw.update(over)
    return syn.Config("planes", nx, ny, nz, ns, **kw)


@pytest.mark.parametrize("size", SIZES)
def test_boxes(size):
    cfg, gpu, ref = pair(_cfg(*size))
    nx, ny, nz, ns = size
    rng = np.random.default_rng(8)
    dense = random_state(cfg, 4) + 1.0
    empty = np.zeros_like(dense)
    states = [dense, empty, np.full_like(dense, np.nan)]
    for n in range(12):
        q = empty.copy()
        at = tuple(rng.integers(0, m) for m in size)
        value = [1.0e-7, np.nextafter(1.0e-7, 0.0), 5.0][n % 3]
        q[at] = value
        q[nx - 1, at[1], at[2], ns - 1] = value
        q[0, 0, nz - 1, 0] = np.nan
        states.append(q)
    for q in states:
        for m in (gpu, ref):
            m.set_interior(np.asfortranarray(q))
        assert tuple(gpu.get_minmax_index()) == tuple(ref.get_minmax_index())
    gpu.close()
