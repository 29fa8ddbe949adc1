"""The splat where whole pixels and crossed ones meet: disks smaller than a
pixel, of a few pixels and larger than the image, whose squares end on and
between sample positions, against the numpy restatement bit for bit, and
pictures of changing size from one context (its buffers are kept and grow)."""
import numpy as np
import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("size", [0.001, 0.0625 / 4, 0.0625, 0.07, 0.3, 2.5])
def test_disk_sizes(gpu, size, wrap):
    import splat_ref
    from plgpu.physics import GpuWorld

    spec = uniform_world(700, 5, 0.05, seed=81)
    spec.pos[:64, 0] = np.arange(64) / 64.0  # centres on and beside sample positions
    spec.pos[:64, 1] = (np.arange(64) % 16 + 0.125) / 16.0
    pal = np.random.default_rng(5).random((5, 4)).astype(np.float32)
    w = GpuWorld(2, spec.n)
    try:
        w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, wrap=True)
        w.set_matrix(spec.matrix)
        w.upload(spec.pos, spec.vel, spec.types)
        pos, _, types, _ = w.download()
        for width, height in ((16, 16), (33, 20), (8, 40), (16, 16)):
            got = w.render(width, height, pal, size=size, wrap=wrap)
            ref = splat_ref.splat(pos.astype(np.float32), types, pal, width, height, size=size, wrap=wrap)
            assert np.array_equal(got, ref)
    finally:
        w.close()
