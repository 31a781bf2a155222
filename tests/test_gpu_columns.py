"""The column sums (cloud load and the output products) for grain counts and
levels that are no multiples of what a thread takes at a time, against sums in
the same order (grains in order within a level, levels upwards), bit for bit."""
import numpy as np
import pytest

from gpu_common import random_state
from volcano_ash3d_b200 import synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 2, 3, 4, 5, 7, 8, 9, 12, 60])
@pytest.mark.parametrize("nz", [3, 4, 5, 8, 11])
def test_column_sums(nz, ns):
    cfg = syn.Config("columns", 33, 7, nz, ns, dx=4.0, dy=5.0, dz=0.5, ivent=16, jvent=4, fall_mps=(0.5,) * ns,
                     bin_mass=(1.0 / ns,) * ns, plume_km=1.0, volume_km3=1.0e-3, duration_h=1.0, use_cn=True,
                     sim_hours=1.0, winds="random", seed=43, dz_profile=tuple(0.4 + 0.1 * (k % 3) for k in range(nz)))
    m = Ash3dGPU(cfg)
    q = random_state(cfg, 3)
    q[:8] = 0.0
    m.set_interior(q)
    m.set_output_params()
    dz = np.asarray(m.geo["dz_vec"])[2:]
    load, top = np.zeros((33, 7)), np.zeros((33, 7))
    for k in range(nz):
        t = np.zeros((33, 7))
        for g in range(ns):
            t = t + q[:, :, k, g]
        load = load + t * dz[k] / 1.0e3
        top = np.maximum(top, t)
    assert np.array_equal(m.cloud_load(), load)
    out = m.output_vars(1.0)
    seen = load >= 0.2  # CLOUDLOAD_THRESH
    assert np.array_equal(out["cloud_load"], np.where(seen, load, 0.0))
    assert np.array_equal(out["max_conc"], np.where(seen, top * 1.0e6 / 1.0e9, 0.0))
    m.close()
