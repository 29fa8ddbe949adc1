"""Windows too full for one tile variant's staging and not for another's: one
cluster around a corner of the box (its four or eight cells are images of each
other's neighbours), of sizes around each staging's capacity.  All variants
give the same bits, and the default one agrees with the oracle."""
import numpy as np
import pytest

from worlds import WorldSpec, compare_with_oracle, f32, rng_of, run_gpu_debug

pytestmark = pytest.mark.gpu


def _corner(dim, n, wrap):
    rng = rng_of(1000 * dim + n)
    rmax = 0.05
    pos = np.zeros((n, 3))
    p = f32(rng.uniform(-0.9 * rmax, 0.9 * rmax, (n, dim)))
    p = p - np.floor(p) if wrap else 0.5 + p  # without wrapping: the same cluster in the middle
    p = np.asarray(p, np.float32)
    p[p >= 1.0] = 0.0
    pos[:, :dim] = p
    vel = np.zeros((n, 3))
    vel[:, :dim] = f32(0.01 * rng.standard_normal((n, dim)))
    types = rng.integers(0, 5, n).astype(np.int32)
    return WorldSpec(dim, pos, vel, types, f32(rng.uniform(-1, 1, (5, 5))), rmax, dt=0.001, wrap=wrap)


@pytest.mark.parametrize("wrap", [True, False])
@pytest.mark.parametrize("dim,n", [(2, 1160), (2, 1281), (2, 2047), (2, 2300), (3, 840), (3, 1779), (3, 2177), (3, 2500)])
def test_variants_agree(gpu, dim, n, wrap):
    from plgpu.physics import GpuWorld

    spec = _corner(dim, n, wrap)
    states = []
    for variant in (0, 1, 2):
        w = GpuWorld(dim, n)
        try:
            w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, beta=spec.beta, wrap=spec.wrap)
            w.set_matrix(spec.matrix)
            w.set_tile(variant)
            w.upload(spec.pos, spec.vel, spec.types)
            w.step(2)
            states.append(w.download())
        finally:
            w.close()
    for s in states[1:]:
        for x, y in zip(s, states[0]):
            assert np.array_equal(x, y)
    compare_with_oracle(spec, *run_gpu_debug(spec))
