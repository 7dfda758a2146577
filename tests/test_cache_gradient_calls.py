"""Gradient calls of the cache in a row: each returns its own samples' loss and
gradient, with a loss pointer or without, training steps between."""
import numpy as np
import pytest

import mlp_oracle as mo
from test_cache import BOX, INV, LO, _samples


@pytest.mark.gpu
def test_each_call_returns_its_own_loss_and_gradient():
    import torch
    import photonmap
    ctx = photonmap.Context(0)
    params = mo.init_params(21)
    ctx.cache_init(seed=1, out_scale=2.0, aabb=BOX)
    for seed, n in ((1, 5000), (2, 129), (3, 1), (4, 5000)):
        pos, nrm, tgt = _samples(n, seed)
        tgt *= seed                                             # losses far apart
        ctx.cache_set_params(params)
        g, loss = ctx.cache_gradient(pos, nrm, tgt)
        _, loss_cpu, g_cpu = mo.forward_backward(params, pos, nrm, tgt, None, LO, INV, 2.0, 2.0 / (3 * n))
        # the oracle test's bounds
        assert abs(loss - loss_cpu / (3 * n)) <= 1e-2 * (loss_cpu / (3 * n))
        for a, b in zip(g.reshape(5, 64, 64), g_cpu.reshape(5, 64, 64)):
            assert np.linalg.norm(a - b) < 2e-2 * np.linalg.norm(b)
        dev = [torch.from_numpy(x).cuda() for x in (pos, nrm, tgt)]
        torch.cuda.synchronize()
        h = np.zeros_like(g)
        ctx._check(ctx.L.pm_cache_gradient(ctx.h, *(x.data_ptr() for x in dev), None, n, h.ctypes.data, None), "gradient")
        # the same sums in another order of float32 additions
        assert np.linalg.norm(h - g) <= 1e-5 * np.linalg.norm(g)
        step = ctx.cache_train_step(pos, nrm, tgt)
        assert abs(step - loss) <= 1e-5 * loss
    ctx.close()
