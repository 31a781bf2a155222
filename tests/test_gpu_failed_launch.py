"""A launch that fails leaves no state that says it ran.  The failure is an
error code on the host: the context's stream is put into capture, the capture
is invalidated by a synchronisation, and every launch into it is then refused
until the capture is ended; nothing reaches the GPU."""
import ctypes as C

import numpy as np
import pytest

from gpu_common import random_state, random_winds
from volcano_ash3d_b200 import _lib, synthetic as syn
from volcano_ash3d_b200.model import Ash3dGPU

pytestmark = pytest.mark.gpu

RELAXED = 2


class Refusing:
    """Launches into the model's stream are refused inside the block."""

    def __init__(self, model):
        self.model, self.stream = model, C.c_void_p(model.stream_handle())
        self.cuda = C.CDLL("libcuda.so.1")

    def __enter__(self):
        self.model.sync()
        assert self.cuda.cuStreamBeginCapture_v2(self.stream, C.c_int(RELAXED)) == 0
        assert self.cuda.cuStreamSynchronize(self.stream) != 0

    def __exit__(self, *exc):
        graph = C.c_void_p()
        assert self.cuda.cuStreamEndCapture(self.stream, C.byref(graph)) != 0  # no graph comes of it
        assert not graph.value
        assert self.cuda.cuStreamSynchronize(self.stream) == 0


def _model(**over):
    kw = dict(dx=4.0, dy=5.0, dz=0.5, ivent=20, jvent=10, fall_mps=(0.1, 0.8), bin_mass=(0.5, 0.5), plume_km=1.0,
              volume_km3=1.0e-3, duration_h=1.0, use_cn=False, sim_hours=1.0, winds="random", seed=91)
    kw.update(over)
    cfg = syn.Config("refused", 40, 21, 11, 2, **kw)
    m = Ash3dGPU(cfg)
    m.set_interior(random_state(cfg, 3))
    m.set_winds(*random_winds(cfg, 4))
    return m


def _async_dt(m):
    return m.lib.a3g_adjust_dt_async(m.ctx, C.c_double(0.0), C.c_double(1.0e9), C.c_double(1.0e9))


def _swept(m, dt):
    m.set_dt(dt)
    m.advect_x()
    m.AdvectVert()
    return m.interior()


def _fast_dt(m):
    return m.lib.a3g_fast_dt_async(m.ctx, C.c_double(0.5), C.c_double(0.0), C.c_double(1.0e9), C.c_double(1.0e9))


@pytest.mark.parametrize("form_dt", [_async_dt, _fast_dt])
def test_dt_over_kappa(form_dt):
    """A refused dt kernel has not formed dt/kappa: the next dt's sweeps form it."""
    want = _swept(_model(), 0.013)
    m = _model()
    m.Adjust_DT(0.0, 1.0e9, 1.0e9)
    with Refusing(m):
        assert form_dt(m) != 0
    assert np.array_equal(_swept(m, 0.013), want)
    m.close()


def test_explicit_diffusion_factors():
    """A refused table launch has not filled the explicit sweeps' table."""
    def diffused(m):
        m.set_dt(0.013)
        m.DiffuseHorz(1)
        return m.interior()

    want = diffused(_model())
    m = _model()
    m.set_dt(0.013)
    with Refusing(m):
        assert m.lib.a3g_diffuse_horz(m.ctx, 1) != 0
    assert np.array_equal(diffused(m), want)
    m.close()
