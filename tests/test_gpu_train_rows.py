"""Training over device rows at any float's address, and over batches from one
CTA's rows to more CTAs than parameters divide evenly among: the rows' 16-byte
loads and the single ones, and the optimiser fused (its partials staged) or as a
second launch, give the same bits."""
import ctypes

import numpy as np
import pytest

from cloudgb import _lib, surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("batch", [128, 384, 9600, 19456])
def test_rows_and_shares(ctx, layers, batch):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(batch)
    n, steps = 20011, 6
    x = rng.uniform(0.0, 3.0, (n, surrogate.N_FEATURES)).astype(np.float32)
    tau = rng.uniform(0.0, 2.0, n).astype(np.float32)
    flat = torch.zeros(x.size + 4, dtype=torch.float32, device="cuda")
    target = torch.from_numpy(tau).cuda()
    results = []
    for shift, separate in [(0, 0), (1, 0), (2, 0), (0, 1), (3, 1)]:
        flat[shift:shift + x.size] = torch.from_numpy(x.reshape(-1)).cuda()
        torch.cuda.synchronize()
        net = surrogate.SunMLP(ctx, seed=3, hidden_layers=layers)
        tp = _lib.cg_train_params()
        _lib.load().cg_train_params_default(ctypes.byref(tp))
        tp.steps, tp.batch, tp.sigma, tp.seed, tp.separate_adam = steps, batch, 2.0, 1, separate
        losses = np.empty(steps, np.float32)
        _lib.check(_lib.load().cg_mlp_train(
            net.handle, ctypes.c_void_p(flat.data_ptr() + 4 * shift),
            ctypes.c_void_p(target.data_ptr()), n, ctypes.byref(tp),
            losses.ctypes.data_as(_lib.FP)), "cg_mlp_train")
        params, m, v, step = net.get_params()
        assert np.isfinite(losses).all() and step == steps
        results.append((losses, params, m, v))
    for r in results[1:]:
        for a, b in zip(r, results[0]):
            assert np.array_equal(a, b)
