"""Tile variants that a batch gives its worlds: crowded 2D worlds open no force
launch of their own unless they are large and dense, whatever joins or leaves,
and a variant set for a world stays."""
import numpy as np
import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


def _desc(n, nx, seed):
    from plgpu.batch import WorldDesc

    s = uniform_world(n, 4, 0.9999 / nx, seed=seed, vel_scale=0.01)
    return WorldDesc(pos=s.pos, types=s.types, matrix=s.matrix, rmax=s.rmax, friction=s.friction, force=s.force, dt=s.dt,
                     beta=s.beta, wrap=s.wrap, vel=s.vel)


def test_one_launch_whatever_joins(gpu):
    from plgpu.batch import GpuBatch

    ordinary, tiny, dense = _desc(3000, 50, 1), _desc(432, 3, 2), _desc(4000, 6, 3)
    b = GpuBatch(2, 20_000, 8, 10_000)
    try:
        tiles = lambda: [b.world_tile(i) for i in b.world_ids()]  # noqa: E731
        b.update(add=[ordinary, tiny])
        assert tiles() == [0, 0]
        b.update(remove=b.world_ids(), add=[tiny, dense])  # crowded throughout
        assert tiles() == [1, 1]
        (c,) = b.update(add=[ordinary])
        assert tiles() == [0, 0, 0]
        b.update(remove=[c])
        assert tiles() == [1, 1]
        a = b.world_ids()[0]
        b.set_world_tile(a, 2)
        b.step(2)
        assert tiles() == [2, 1]
        b.update(add=[dense])  # the set variant stays, and the batch is not on the dense tile throughout
        assert tiles() == [2, 0, 0]
    finally:
        b.close()


@pytest.mark.parametrize("n,nx,tile", [(100_000, 31, 1), (99_999, 31, 0), (102_400, 32, 1), (102_399, 32, 0)])
def test_large_dense_worlds_have_their_launch(gpu, n, nx, tile):
    from plgpu.batch import GpuBatch

    b = GpuBatch(2, 110_000, 4, 10_000)
    try:
        b.update(add=[_desc(3000, 50, 1), _desc(n, nx, 6)])
        assert [b.world_tile(i) for i in b.world_ids()] == [0, tile]
        b.step(2)
    finally:
        b.close()


def test_tuned_variants_stay(gpu):
    from plgpu.batch import GpuBatch

    b = GpuBatch(2, 20_000, 8, 10_000)
    try:
        b.update(add=[_desc(432, 3, 2), _desc(3000, 50, 1)])
        choice, _ = b.autotune_worlds(2)
        (c,) = b.update(add=[_desc(2000, 40, 4)])
        assert {i: b.world_tile(i) for i in choice} == choice
        v, _ = b.autotune(2)
        assert [b.world_tile(i) for i in b.world_ids()] == [v] * 3
        (d,) = b.update(add=[_desc(4000, 6, 3)])  # one variant for the batch: new worlds take it
        assert b.world_tile(d) == v
    finally:
        b.close()


def test_variants_given_do_not_change_bits(gpu):
    from plgpu.batch import GpuBatch

    worlds = [_desc(4000, 6, 3), _desc(432, 3, 2), _desc(3000, 50, 1)]
    states = []
    for apart in (False, True):
        b = GpuBatch(2, 20_000, 8, 10_000)
        try:
            if apart:  # the crowded worlds alone first, on the dense tile
                ids = b.update(add=worlds[:2])
                b.step(3)
                ids += b.update(add=worlds[2:])
                b.step(3)
            else:
                ids = b.update(add=worlds)
                b.step(3)
                third = b.download(ids[2])
                b.step(3)
            states.append([b.download(i) for i in ids[:2]] + [third if not apart else None, b.download(ids[2])])
        finally:
            b.close()
    for x, y in zip(states[0][:2], states[1][:2]):
        for u, v in zip(x, y):
            assert np.array_equal(u, v)
    for u, v in zip(states[0][2], states[1][3]):  # three steps of the world that joined later
        assert np.array_equal(u, v)
