"""Batched step graphs of one and of several steps: any count of steps, step
budgets that run out inside a graph, one force launch a step and several, and
changes between calls give the bits of plain launches."""
import numpy as np
import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


def _descs(dim, sizes):
    from plgpu.batch import WorldDesc

    out = []
    for k, n in enumerate(sizes):
        s = uniform_world(n, 3 + k, (0.03 if dim == 2 else 0.08) + 0.01 * k, seed=95 + k, dim=dim, vel_scale=0.02)
        out.append(WorldDesc(pos=s.pos, types=s.types, matrix=s.matrix, rmax=s.rmax, friction=s.friction, force=s.force,
                             dt=s.dt, beta=s.beta, wrap=s.wrap, vel=s.vel))
    return out


@pytest.mark.parametrize("dim,mixed", [(2, False), (2, True), (3, False), (3, True)])
def test_counts_budgets_and_changes(gpu, dim, mixed):
    from plgpu.batch import GpuBatch

    worlds = _descs(dim, (1, 700, 5_001, 20_000))
    batches = []
    try:
        for graph in (1, 0):
            b = GpuBatch(dim, 60_000, 8, 60_000)
            batches.append(b)
            assert b.lib.plg_batch_set_use_graph(b.b, graph) == 0
            ids = b.update(add=worlds)
            if mixed:
                for k, i in enumerate(ids):
                    b.set_world_tile(i, k % 3)
            states = []
            for k, steps in enumerate((1, 33, 32, 3, 38)):
                if k == 1:
                    b.set_steps(ids[1], 18)  # runs out inside a graph of several steps
                    b.set_steps(ids[2], 0)
                if k == 3:
                    b.set_steps(ids[1], 2)
                    b.set_steps(ids[2], -1)
                if k == 4:
                    (new,) = b.update(remove=[ids[3]], add=[worlds[3]])
                    ids = ids[:3] + [new]
                b.step(steps)
                assert b.steps_left(ids[1]) == (-1 if k == 0 else 0)
                assert b.steps_left(ids[2]) == (0 if k in (1, 2) else -1)
                states.append([b.download(i) for i in ids])
            batches[-1] = (b, states)
        for x, y in zip(batches[0][1], batches[1][1]):
            for p, q in zip(x, y):
                for u, v in zip(p, q):
                    assert np.array_equal(u, v)
        frozen, running = batches[0][1][2], batches[0][1][1]
        for u, v in zip(frozen[1], running[1]):  # its budget had run out: not moved
            assert np.array_equal(u, v)
        assert not np.array_equal(frozen[3][0], running[3][0])
    finally:
        for b in batches:
            (b[0] if isinstance(b, tuple) else b).close()
