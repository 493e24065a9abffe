"""The synchronous solver calls draw their scratch from a pool that keeps its memory between calls:
calls from several threads on their own streams give the bits of the same calls made one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(12, 14, 16), (9, 11, 13)])
def test_concurrent_calls_share_the_scratch_pool(gpu, shape):
    import torch
    rng = np.random.default_rng(sum(shape))
    T0, Q = rng.uniform(20, 120, shape), rng.uniform(0, 900, shape)
    k, rho = rng.uniform(2e-4, 6e-4, shape), rng.uniform(1.5e-3, 4e-3, shape)
    void = rng.uniform(size=shape) < 0.7
    C0 = rng.uniform(0, 1, shape) * void
    z = np.zeros(shape)

    def one():
        ctx = gpu.MetalAblationContext(*shape, 0.03, 0.025, 0.02, 1e-5, 10e-6, 20.0, 100.0, 300.0,
                                       plume_params={'D_xy': 1.5, 'D_z': 2.5, 'vz': 4.0, 'tau_linger': 0.02})
        ctx.set_state(T0, z, z, z, z.astype(np.uint8), z.astype(np.uint8), Q, k, rho, plume=C0, plume_void=void)
        for _ in range(5):
            ctx.advance_substeps(3)
        return ctx.get_state()[0], ctx.get_plume()

    want = one()
    got = [None] * 4

    def worker(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = one()

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in got:
        assert np.array_equal(g[0], want[0]) and np.array_equal(g[1], want[1])
