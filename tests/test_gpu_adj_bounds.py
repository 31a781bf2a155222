"""The marched transposed advection sweeps against the oracle's, on states whose
limiter ratios lie on the class bounds (0, 1/2, 1, 2), tails down to the
subnormals and tiny differences, with a grain that is not aloft.  The two take
the same branches and sum their terms in different orders: 1e-12 of the field's
largest value, as the adjoint sweeps are compared elsewhere."""
import numpy as np
import pytest

from gpu_common import pair, random_winds
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(33, 9, 10, 2), (40, 57, 19, 3)])
@pytest.mark.parametrize("aloft", [None, 0, 1])
@pytest.mark.parametrize("latlon", [False, True])
def test_class_bounds(size, aloft, latlon):
    nx, ny, nz, ns = size
    cfg = syn.Config("bounds", nx, ny, nz, ns, dx=4.0, dy=5.0, dz=0.5, ivent=(nx + 1) // 2, jvent=(ny + 1) // 2,
                     fall_mps=tuple(0.2 * (g + 1) for g in range(ns)), bin_mass=(1.0 / ns,) * ns, plume_km=1.0,
                     volume_km3=1.0e-3, duration_h=1.0, use_cn=True, sim_hours=1.0, winds="random", seed=61,
                     latlon=latlon, de=0.5, dn=0.5, latLL=20.0)
    cfg, gpu, ref = pair(cfg)
    rng = np.random.default_rng(7)
    shape = (nx, ny, nz, ns)
    q = rng.integers(0, 7, shape) * 0.5 * (rng.uniform(size=shape) < 0.7)
    tiny = rng.uniform(size=shape) < 0.1
    q[tiny] = 10.0 ** rng.uniform(-323.0, -8.0, tiny.sum())
    lam = np.asfortranarray(rng.standard_normal(shape))
    dep = np.asfortranarray(rng.standard_normal((nx, ny, ns)))
    flags = np.ones(ns, dtype=np.int32)
    if aloft is not None:
        flags[aloft] = 0
    for m in (gpu, ref):
        m.set_interior(np.asfortranarray(q))
        m.set_winds(*random_winds(cfg, 8))
        m.set_dt(0.01)
        m.set_aloft(flags)
    for op, args in (("adj_advect_x", ()), ("adj_advect_y", ()), ("adj_advect_z", (dep,))):
        a, b = getattr(gpu, op)(lam, *args), getattr(ref, op)(lam, *args)
        assert np.abs(a - b).max() <= 1.0e-12 * np.abs(b).max(), op
        if aloft is not None:
            assert not a[..., aloft].any(), op
    gpu.close()
