"""Kernel profile: what a step launches is what it reports.  A world sorted in
one launch has no scatter and no gather; one particle more has all four."""
import ctypes

import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,launches", [(10_000, (3, 0, 0, 3)), (24_576, (3, 0, 0, 3)), (24_577, (3, 3, 3, 3))])
def test_launches_per_kernel(gpu, n, launches):
    from plgpu.physics import GpuWorld

    spec = uniform_world(n, 4, 0.02, seed=5, vel_scale=0.01)
    w = GpuWorld(2, n)
    try:
        w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, beta=spec.beta, wrap=spec.wrap)
        w.set_matrix(spec.matrix)
        w.upload(spec.pos, spec.vel, spec.types)
        assert w.lib.plg_profile_enable(w.ctx, 1) == 0
        w.step(3)
        for k, want in enumerate(launches):
            ms, count = ctypes.c_double(-1), ctypes.c_int64(-1)
            assert w.lib.plg_profile_read(w.ctx, k, ctypes.byref(ms), ctypes.byref(count)) == 0
            assert count.value == want
            assert (ms.value > 0) == (want > 0)
    finally:
        w.close()
