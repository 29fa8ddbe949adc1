"""A stop request in a long call: no more than the eight steps in flight are
still done (timed on a world of slow steps), the state is that of a whole
number of steps, and the next call runs."""
import threading
import time

import numpy as np
import pytest

from worlds import uniform_world

pytestmark = pytest.mark.gpu


def test_steps_done_after_a_stop_request(gpu):
    from plgpu import _lib
    from plgpu.physics import GpuWorld

    spec = uniform_world(60_000, 4, 0.33, seed=31)  # 9 cells: milliseconds a step
    w = GpuWorld(2, spec.n)
    status = []
    try:
        w.set_settings(spec.rmax, spec.friction, spec.force, 1e-6, beta=spec.beta, wrap=spec.wrap)
        w.set_matrix(spec.matrix)
        w.upload(spec.pos, spec.vel, spec.types)
        w.step(32)  # builds the graphs
        t0 = time.perf_counter()
        w.step(16)
        step = (time.perf_counter() - t0) / 16
        t = threading.Thread(target=lambda: status.append(w.lib.plg_step(w.ctx, 100_000)))
        t.start()
        time.sleep(40 * step)
        t0 = time.perf_counter()
        assert w.lib.plg_request_stop(w.ctx) == 0
        t.join(30)
        took = time.perf_counter() - t0
        assert not t.is_alive() and status == [_lib.PLG_E_STOPPED]
        assert took <= 11 * step, (took / step, step)  # eight, and time for the host
        w.step(1)
        assert np.array_equal(np.sort(w.download()[3]), np.arange(spec.n))
    finally:
        w.close()
