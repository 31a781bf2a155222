"""The kernels that give a warp a row (CFL maxima and dt, wind interpolation,
mass totals, NetCDF arrays and restart) at row lengths around a warp's 32
lanes, a lane's eight cells and a pass of 256, and on grids of a single block
or many."""
import math

import numpy as np
import pytest

from gpu_common import pair, random_winds
from topo_common import level_winds
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3, 1), (31, 4, 5, 2), (33, 9, 7, 3), (65, 40, 37, 1), (255, 3, 4, 2), (257, 5, 3, 2), (520, 6, 4, 1)]


def _cfg(nx, ny, nz, ns, **over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=2, jvent=2, fall_mps=tuple(0.1 * (g + 1) for g in range(ns)),
              bin_mass=(1.0 / ns,) * ns, plume_km=1.0, volume_km3=1.0e-3, duration_h=1.0, winds="random", seed=51)
    kw.update(over)
    return syn.Config("rows", nx, ny, nz, ns, **kw)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("kind", ["projected", "lonlat", "terrain"])
def test_rows(size, kind):
    over = dict(lonlat=dict(latlon=True, de=0.5, dn=0.5, latLL=20.0),
                terrain=dict(zscaling_id=2, topo_km=0.4, topo_width_km=20.0)).get(kind, {})
    cfg, gpu, ref = pair(_cfg(*size, **over))
    rng = np.random.default_rng(3)
    # dt from ghosted winds, bit for bit, twice (the block counters are back at zero)
    for seed in (4, 5):
        w = (level_winds if kind == "terrain" else random_winds)(cfg, seed)
        for m in (gpu, ref):
            m.set_winds(*w)
        assert np.array_equal(gpu.cfl_maxima(), ref.cfl_maxima())
        assert gpu.Adjust_DT(0.0, 1.0e9, 1.0e9) == ref.Adjust_DT(0.0, 1.0e9, 1.0e9)
    # interpolated winds, seen through dt and one sweep
    met = syn.MetSource(cfg)
    q = rng.uniform(0.0, 1.0e3, (cfg.nx, cfg.ny, cfg.nz, cfg.ns))
    for m in (gpu, ref):
        m.set_met_steps(met.step(0), met.step(1))
        m.interp_winds(0.37)
        m.set_interior(np.asfortranarray(q))
    assert gpu.Adjust_DT(0.0, 1.0e9, 1.0e9) == ref.Adjust_DT(0.0, 1.0e9, 1.0e9)
    for m in (gpu, ref):
        m.Set_BC(1)
        m.AdvectHorz(1)
        m.AdvectVert()
    c = gpu.interior()
    assert np.array_equal(c, ref.interior())
    # totals against exact sums of the same state and outflows
    kap = gpu.geo["kappa"]
    vols, mass = gpu.TimeStepTotals()
    inner = kap[2:-2, 2:-2, 2:-2]
    want = [math.fsum((c[..., g] * inner).ravel()) for g in range(cfg.ns)]
    assert np.allclose(mass, want, rtol=1.0e-15 * 8, atol=0.0)
    again, _ = ref.TimeStepTotals()
    assert np.allclose(vols, again, rtol=1.0e-13, atol=0.0)
    ticket = gpu.totals_async()
    assert np.array_equal(gpu.totals_get(ticket)[0], vols)
    # the arrays of the writer, and back
    ash, dep = gpu.output_ashcon()
    assert np.array_equal(ash, c.astype(np.float32))
    gpu.restart_load(ash, dep)
    assert np.array_equal(gpu.interior(), ash.astype(np.float64))
    gpu.close()
