"""GPU tests of the one-call training of a layer (qgru_train_forward / qgru_train_backward) against the dense
per-direction entry points, which the other tests compare with the oracle: outputs bit for bit, gradients as
fp32 sums in another order."""
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named, gen_x

QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
pytestmark = pytest.mark.gpu


def _pass(m, fn, x, hx, g_out, g_hn):
    import torch
    leaves = [t.clone().requires_grad_() for t in ((x,) if hx is None else (x, hx))]
    out, hn = fn(leaves[0], leaves[1] if hx is not None else None)
    wrt = leaves + list(m.parameters())
    return out.detach(), hn.detach(), torch.autograd.grad((out, hn), wrt, (g_out, g_hn))


# (T, B, I, H): one unit, K of the recurrence over one warp (ragged, full tiles) and over two in clusters of 2, 3, 4
@pytest.mark.parametrize("T,B,I,H", [(1, 1, 3, 1), (5, 3, 40, 64), (4, 150, 33, 131), (6, 9, 20, 256), (3, 70, 65, 321), (4, 37, 12, 512)])
@pytest.mark.parametrize("storage,cfg", [("float", None), ("float32", "cfg2"), ("float32", "unsigned_x"), ("float32", "gate_in16"),
                                         ("int32", "default"), ("int32", "ih16"), ("int32", "gate_in16"), ("int32", "wide16")])
@pytest.mark.parametrize("bidir,batch_first,bias", [(False, False, True), (True, True, False)])
def test_train_layer_equals_dense_calls(cuda_device, storage, cfg, T, B, I, H, bidir, batch_first, bias):
    import torch
    torch.manual_seed(T * H)
    rng = np.random.default_rng(T + 7 * H)
    D = 2 if bidir else 1
    x = torch.from_numpy(np.ascontiguousarray(gen_x(rng, B, T, I))).to(cuda_device)            # [B, T, I]
    if not batch_first:
        x = x.transpose(0, 1).contiguous()
    hx = torch.randn(D, B, H, device=cuda_device) * 0.3 if H != 256 else None
    m = QuantGRU(I, H, bias=bias, bidirectional=bidir, batch_first=batch_first,
                 quant_storage_dtype="float32" if storage == "float" else storage).to(cuda_device)
    m.use_quantization = storage != "float"
    if m.use_quantization:
        m.load_bitwidth_config(config_named(cfg).to_json_dict())
        m.use_quantization = True
        m.calibrating = True
        m(x * 0.6)                          # (a part of what follows is clamped)
        m.calibrating = False
        m.finalize_calibration()
    m.train()
    g_out = torch.randn(*x.shape[:2], D * H, device=cuda_device)
    g_hn = torch.randn(D, B, H, device=cuda_device)
    out, hn, grads = _pass(m, m, x, hx, g_out, g_hn)
    want_out, want_hn, want = _pass(m, m._forward_train_stepwise, x, hx, g_out, g_hn)
    if storage == "float":
        assert torch.allclose(out, want_out, rtol=0, atol=1e-6) and torch.allclose(hn, want_hn, rtol=0, atol=1e-6)
    else:
        assert torch.equal(out, want_out) and torch.equal(hn, want_hn)
    for a, b in zip(grads, want):
        assert a.shape == b.shape and (a - b).abs().max() <= 2e-5 * max(float(b.abs().max()), 1e-30)
