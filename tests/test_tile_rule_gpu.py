"""The default tiles of crowded 2D worlds (alone and in a batch) and of large
3D worlds: on both sides of each line, with the same bits as the other tiles."""
import numpy as np
import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,crowded", [(4799, False), (4800, True)])  # 10 x 10 cells: 48 per cell
def test_crowded_worlds(gpu, n, crowded):
    from plgpu.batch import GpuBatch, WorldDesc
    from plgpu.physics import GpuWorld

    spec = uniform_world(n, 4, 0.0999, seed=55, vel_scale=0.01)
    states = []
    for variant in (None, 0, 2):
        w = GpuWorld(2, n)
        try:
            w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, beta=spec.beta, wrap=spec.wrap)
            w.set_matrix(spec.matrix)
            if variant is not None:
                w.set_tile(variant)
            w.upload(spec.pos, spec.vel, spec.types)
            assert w.tile() == ((1 if crowded else 2) if variant is None else variant)
            w.step(3)
            states.append(w.download())
        finally:
            w.close()
    d = WorldDesc(pos=spec.pos, types=spec.types, matrix=spec.matrix, rmax=spec.rmax, friction=spec.friction,
                  force=spec.force, dt=spec.dt, beta=spec.beta, wrap=spec.wrap, vel=spec.vel)
    b = GpuBatch(2, 2 * n, 2, 400)
    try:
        (a,) = b.update(add=[d])
        assert b.world_tile(a) == (1 if crowded else 0)
        b.step(3)
        states.append(b.download(a))
        b.set_tile(0)
        (c,) = b.update(add=[d])  # a variant set by hand stays for new worlds
        assert b.world_tile(c) == 0
    finally:
        b.close()
    for s in states[1:]:
        for x, y in zip(s, states[0]):
            assert np.array_equal(x, y)


# 27^3 cells: 10.2 per cell at 200,000 particles; 26^3: 11.4, past the line.
@pytest.mark.parametrize("n,nx,tile", [(199_999, 27, 0), (200_000, 27, 2), (200_000, 26, 0)])
def test_large_3d_worlds(gpu, n, nx, tile):
    from plgpu.physics import GpuWorld

    spec = uniform_world(n, 4, 0.999 / nx, seed=56, dim=3, vel_scale=0.01)
    states = []
    for variant in (None, 0, 1, 2):
        w = GpuWorld(3, n)
        try:
            w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, beta=spec.beta, wrap=spec.wrap)
            w.set_matrix(spec.matrix)
            if variant is not None:
                w.set_tile(variant)
            w.upload(spec.pos, spec.vel, spec.types)
            assert w.tile() == (tile if variant is None else variant)
            w.step(2)
            states.append(w.download())
        finally:
            w.close()
    for s in states[1:]:
        for x, y in zip(s, states[0]):
            assert np.array_equal(x, y)
