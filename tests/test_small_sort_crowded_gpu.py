"""Crowded cells in the one-launch sort of small worlds: the order is the
oracle's for cells on both sides of the crowding line and across the blocks'
shares of the slots, and the sort of a world crowded into one or a few cells
takes no longer than the three launches take for one particle more."""
import ctypes

import numpy as np
import pytest

from worlds import f32, rng_of, run_gpu_debug, run_oracle_debug, uniform_world

pytestmark = pytest.mark.gpu


def _packed(sizes, dim, nx, seed):
    """sizes[k] particles in the k-th cell (rows of nx cells), in mixed order."""
    n = sum(sizes)
    spec = uniform_world(n, 3, 0.999 / nx, seed=seed, dim=dim)
    rng = rng_of(seed + 1)
    cell = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    at = np.stack([cell // nx**k % nx for k in range(dim)], axis=1)
    spec.pos[:, :dim] = f32((at + 0.1 + 0.8 * rng.random((n, dim))) * spec.rmax)
    return spec


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize(
    "sizes",
    [
        (255, 256, 257, 258, 255),
        (0, 257, 1, 257, 257, 257, 0, 3),
        (511, 1, 512, 1, 513, 0, 1025),
        (512, 513, 511, 513, 514),
        (0, 513, 1, 513, 513, 0, 3, 509),
        (300, 212, 256, 256, 257, 255, 600, 1, 1),
        (2, 4095, 1, 4097, 256, 3),
        (257,),
        (256,),
        (1, 24575),
        (12288, 12288),
    ],
)
def test_order_of_crowded_cells(gpu, dim, sizes):
    spec = _packed(sizes, dim, 4, 300 + len(sizes))
    g, state = run_gpu_debug(spec)
    d, o = run_oracle_debug(spec)
    assert np.array_equal(state[3], o.ids) and np.array_equal(state[2], o.types)
    assert np.array_equal(g["cell"], d["cell"])


def _sort_us(n, nx, box):
    """Mean time of the step's launches before the force kernel."""
    from plgpu.physics import GpuWorld

    spec = uniform_world(n, 4, 0.999 / nx, seed=17)
    if box < 1:
        spec.pos[:, :2] = f32(0.501 + box * spec.pos[:, :2])
    w = GpuWorld(2, n)
    try:
        w.set_settings(spec.rmax, spec.friction, spec.force, 1e-6, beta=spec.beta, wrap=spec.wrap)
        w.set_matrix(spec.matrix)
        w.upload(spec.pos, spec.vel, spec.types)
        w.step(2)
        assert w.lib.plg_profile_enable(w.ctx, 1) == 0
        w.step(4)
        total = 0.0
        for k in range(3):
            ms, launches = ctypes.c_double(), ctypes.c_int64()
            assert w.lib.plg_profile_read(w.ctx, k, ctypes.byref(ms), ctypes.byref(launches)) == 0
            total += 1e3 * ms.value / 4
        return total
    finally:
        w.close()


@pytest.mark.parametrize("nx,box", [(50, 0.015), (3, 1.0), (5, 1.0)])
def test_crowded_cells_take_no_longer_than_three_launches(gpu, nx, box):
    """24,576 particles are the most the one launch takes; 24,577 go to the three.  The margin is for noise."""
    assert _sort_us(24_576, nx, box) <= 1.2 * _sort_us(24_577, nx, box)
