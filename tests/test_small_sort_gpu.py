"""The one-launch sort of small worlds against the oracle (stable order, cell
of every particle, pair sets) at the ends of its range: one particle, whole
and partial groups of four, a block's share of the slots, all particles in one
cell (beyond a block's shared list), the largest world it takes and the first
it leaves to the three launches."""
import numpy as np
import pytest

from worlds import compare_with_oracle, f32, rng_of, run_gpu_debug, run_oracle_debug, uniform_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 511, 512, 513, 1025, 4095, 24575, 24576, 24577])
def test_sizes(gpu, dim, n):
    rmax = max(0.02, (10 / n) ** (1 / dim) / 2) if dim == 2 else max(0.05, (10 / n) ** (1 / dim) / 2)
    spec = uniform_world(n, 4, min(rmax, 0.3), seed=700 + n, dim=dim, vel_scale=0.01)
    compare_with_oracle(spec, *run_gpu_debug(spec))


@pytest.mark.parametrize("n,spread", [(5000, 0.0), (6000, 1e-3), (24576, 0.3)])
def test_crowded_cells(gpu, n, spread):
    """One cell with every member but a few (positions and pair sets only:
    the force of thousands of near neighbours is not the point)."""
    spec = uniform_world(n, 3, 0.25, seed=9)
    rng = rng_of(10)
    spec.pos[:-5, :2] = f32(0.3 + spread * (rng.random((n - 5, 2)) - 0.5))
    g, state = run_gpu_debug(spec)
    d, o = run_oracle_debug(spec)
    assert np.array_equal(state[3], o.ids) and np.array_equal(state[2], o.types)
    assert np.array_equal(g["cell"], d["cell"])


def test_cell_limit(gpu):
    """128 x 128 cells are the most it takes; 129 x 129 go the other way."""
    for nx in (128, 129):
        spec = uniform_world(6000, 4, 1.0 / nx * (1 - 1e-6), seed=31, vel_scale=0.01)
        assert int(1 / spec.rmax) == nx
        compare_with_oracle(spec, *run_gpu_debug(spec))


def test_many_steps(gpu):
    """Counts and offsets stay right from step to step, graph and plain launches alike."""
    from plgpu.physics import GpuWorld

    spec = uniform_world(9001, 5, 0.02, seed=33, vel_scale=0.05)
    out = []
    for graph in (1, 0):
        w = GpuWorld(2, spec.n)
        try:
            w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, wrap=True)
            w.set_matrix(spec.matrix)
            w.lib.plg_set_use_graph(w.ctx, graph)
            w.upload(spec.pos, spec.vel, spec.types)
            w.step(40)
            out.append(w.download())
        finally:
            w.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.array_equal(np.sort(out[0][3]), np.arange(spec.n))
