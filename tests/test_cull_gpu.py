"""The 3D force kernel's two walks over a window (distance test, then the
kept terms) at the sizes where its words and passes end: a world of 3 cells
per axis, whose every window holds every particle.  Against the FP64 oracle
(pair sets exact, accelerations and states within the parity tolerances of
test_parity_gpu.py), and every tile variant's plain step against the
instrumented one, bit for bit."""
import numpy as np
import pytest

from worlds import compare_with_oracle, run_gpu_debug, uniform_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [True, False])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 64, 65, 255, 256, 257, 288, 289, 513, 1729, 2177])
def test_window_sizes(gpu, n, wrap):
    from plgpu.physics import GpuWorld

    spec = uniform_world(n, 5, 0.33, seed=400 + n, dim=3, vel_scale=0.01, wrap=wrap)
    g, state = run_gpu_debug(spec)
    compare_with_oracle(spec, g, state)
    for variant in range(3):
        w = GpuWorld(3, n)
        try:
            w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, beta=spec.beta, wrap=spec.wrap)
            w.set_matrix(spec.matrix)
            w.set_tile(variant)
            w.upload(spec.pos, spec.vel, spec.types)
            w.step(1)
            for a, b in zip(w.download(), state):
                assert np.array_equal(a, b)
        finally:
            w.close()
