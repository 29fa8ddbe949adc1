"""Step graphs of one and of several steps: any count of steps, in one call or
several, and changes between calls (settings, matrix, particle count, tile)
give the bits of plain launches; a stop request ends a long call."""
import threading
import time

import numpy as np
import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


def _world(spec, graph, capacity=None):
    from plgpu.physics import GpuWorld

    w = GpuWorld(spec.dim, capacity or spec.n)
    w.set_settings(spec.rmax, spec.friction, spec.force, spec.dt, beta=spec.beta, wrap=spec.wrap)
    w.set_matrix(spec.matrix)
    assert w.lib.plg_set_use_graph(w.ctx, graph) == 0
    w.upload(spec.pos, spec.vel, spec.types)
    return w


@pytest.mark.parametrize("dim,n,rmax", [(2, 5_001, 0.03), (2, 60_000, 0.008), (3, 30_001, 0.06)])
def test_counts_and_changes(gpu, dim, n, rmax):
    spec = uniform_world(n, 5, rmax, seed=91, dim=dim, vel_scale=0.02)
    extra = uniform_world(700, 5, rmax, seed=92, dim=dim, vel_scale=0.02)
    a, b = _world(spec, 1, n + 700), _world(spec, 0, n + 700)
    try:
        for k, steps in enumerate((1, 31, 32, 33, 3, 70, 35, 4, 66)):
            for w in (a, b):
                if k == 4:
                    w.set_settings(spec.rmax, spec.friction, 0.7, 0.5 * spec.dt, beta=spec.beta, wrap=spec.wrap)
                if k == 5:
                    w.set_matrix(-spec.matrix)
                if k == 6:
                    w.append(extra.pos, extra.vel, extra.types)
                if k == 7:
                    w.set_tile(1)
                if k == 8:
                    w.set_settings(0.9 * spec.rmax, spec.friction, 0.7, 0.5 * spec.dt, beta=spec.beta, wrap=False)
                w.step(steps)
            for x, y in zip(a.download(), b.download()):
                assert np.array_equal(x, y)
    finally:
        a.close()
        b.close()


def test_a_stop_request_ends_a_long_call(gpu):
    from plgpu import _lib

    spec = uniform_world(20_000, 5, 0.01, seed=93, vel_scale=0.01)
    w = _world(spec, 1)
    status = []
    try:
        t = threading.Thread(target=lambda: status.append(w.lib.plg_step(w.ctx, 2_000_000)))
        t.start()
        time.sleep(0.2)
        assert w.lib.plg_request_stop(w.ctx) == 0
        t.join(20)
        assert not t.is_alive() and status == [_lib.PLG_E_STOPPED]
        w.step(1)
        assert np.array_equal(np.sort(w.download()[3]), np.arange(spec.n))
    finally:
        w.close()
