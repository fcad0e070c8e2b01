"""Inference over caller's rows on the device at any float's address: the rows'
16-byte loads and the single ones give the same bits, whatever the number of rows
left for the last tile."""
import ctypes

import numpy as np
import pytest

from cloudgb import _lib, surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 5000, 200001])
def test_rows_at_any_address(ctx, n, layers):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    lib = _lib.load()
    x = rng.uniform(-3.0, 3.0, (n, surrogate.N_FEATURES)).astype(np.float32)
    net = surrogate.SunMLP(ctx, hidden_layers=layers)
    flat = torch.zeros(n * surrogate.N_FEATURES + 4, dtype=torch.float32, device="cuda")
    outs = []
    for shift in range(4):
        flat[shift:shift + x.size] = torch.from_numpy(x.reshape(-1)).cuda()
        out = torch.full((n + 1,), -7.0, device="cuda")
        torch.cuda.synchronize()
        _lib.check(lib.cg_mlp_infer(net.handle, ctypes.c_void_p(flat.data_ptr() + 4 * shift), n,
                                    ctypes.c_void_p(out.data_ptr()), 1, None), "cg_mlp_infer")
        ctx.synchronize()
        outs.append(out.cpu().numpy())
        assert outs[-1][n] == -7.0
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
    assert np.array_equal(outs[0][:n], net.infer(x))
