"""The vertical Crank-Nicolson solve of columns too tall for a tile (more than
256 levels): whole columns and boxes, one grain and several, tables that the
whole grid or a row shares; bit for bit against the oracle, over two values of
dt."""
import numpy as np
import pytest

from gpu_common import pair
from volcano_ash3d_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [256, 257, 300])
@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("kind", ["projected", "lonlat", "boxed"])
def test_tall_columns_bitwise(nz, ns, kind):
    over = dict(latlon=True, de=0.5, dn=0.5, latLL=30.0) if kind == "lonlat" else {}
    cfg = syn.Config("tall", 37, 5, nz, ns, dx=4.0, dy=5.0, dz=0.5, ivent=18, jvent=3, fall_mps=(0.5,) * ns,
                     bin_mass=(1.0 / ns,) * ns, plume_km=25.0, volume_km3=1.0e-3, duration_h=1.0, use_cn=True,
                     sim_hours=1.0, winds="random", seed=43, fast_subgrid=kind == "boxed",
                     dz_profile=tuple(0.5 + 0.05 * (k % 4) for k in range(nz)), **over)
    cfg, gpu, ref = pair(cfg)
    rng = np.random.default_rng(5)
    q = rng.uniform(0.0, 1.0e3, (cfg.nx, cfg.ny, nz, ns))
    q[:, :, nz // 3: nz // 2] = 0.0
    q[:, :, nz // 2: nz // 2 + 9] = 1.0e-300
    for m in (gpu, ref):
        m.set_interior(np.asfortranarray(q))
        if kind == "boxed":
            m.set_subgrid((2, 35, 1, 4, 3, nz - 4))
    for dt in (0.02, 0.02, 0.31):
        for m in (gpu, ref):
            m.set_dt(dt)
            m.DiffuseVert()
        assert np.array_equal(gpu.interior(), ref.interior())
    gpu.close()
