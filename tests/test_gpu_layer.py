"""GPU tests of the one-call layer forward (qgru_layer_forward*): strided inputs and outputs, both
directions and the last states against the dense per-direction entry points, for every form of the
recurrence it can meet."""
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named, gen_x

gru_ops = importlib.import_module(PKG_NAME + ".gru_ops")
params_mod = importlib.import_module(PKG_NAME + ".params")
QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
pytestmark = pytest.mark.gpu


def _module(cfg, I, H, bidir, batch_first, storage, x, dev):
    import torch
    torch.manual_seed(I * H)
    m = QuantGRU(I, H, bidirectional=bidir, batch_first=batch_first, quant_storage_dtype=storage).to(dev).eval()
    m.load_bitwidth_config(config_named(cfg).to_json_dict())
    m.calibrating = True
    m(x.transpose(0, 1)[:8, :6] if not batch_first else x[:6, :8])
    m.calibrating = False
    m.finalize_calibration()
    return m


# (T, B, I, H): one CTA per row, clusters of 1 and 4, timestep chunks, a layer without a cluster form
@pytest.mark.parametrize("cfg,storage", [("default", "int32"), ("cfg2", "float32"), ("wide16", "int32"), ("unsigned_x", "int32")])
@pytest.mark.parametrize("T,B,I,H", [(1, 1, 3, 5), (5, 3, 40, 64), (7, 150, 33, 130), (270, 18, 20, 300), (2, 5, 12, 1100)])
def test_layer_forward_equals_dense_forwards(cuda_device, cfg, storage, T, B, I, H):
    import torch
    rng = np.random.default_rng(T + 7 * H)
    x = torch.from_numpy(np.ascontiguousarray(gen_x(rng, B, T, I))).to(cuda_device)            # [B, T, I]
    h0 = torch.from_numpy((rng.standard_normal((2, B, H)) * 0.3).astype(np.float32)).to(cuda_device)
    m = _module(cfg, I, H, True, True, storage, x, cuda_device)
    xt = x.transpose(0, 1).contiguous()
    with torch.no_grad():
        out, hn = m(x, h0)
        out0, hn0 = m(x)
        strided, _ = m(torch.cat([x, x], dim=2)[:, :, I:], h0)        # rows that are not dense
        m.batch_first = False
        out_t, hn_t = m(xt, h0)
        m.batch_first = True
    assert out.is_contiguous() and torch.equal(out, out_t.transpose(0, 1)) and torch.equal(hn, hn_t)
    assert torch.equal(out, strided)
    for d in range(2):
        hd = m._dirs[d].handle
        fwd = hd.forward_f32 if storage == "int32" else hd.forward_fstorage
        for got, got_n, init in ((out, hn, h0[d]), (out0, hn0, None)):
            h = fwd(xt, init, reverse=d == 1)
            want = (h[1:] if d == 0 else h[:T]).transpose(0, 1)
            assert torch.equal(got[:, :, d * H:(d + 1) * H], want)
            assert torch.equal(got_n[d], h[T] if d == 0 else h[0])
    if storage == "int32":
        o = m.quant_params.c.op[0]
        lo = 0 if o.is_unsigned else -(1 << (o.bits - 1))
        x_q = torch.from_numpy(rng.integers(lo, lo + (1 << o.bits), (B, T, I)).astype(np.int32)).to(cuda_device)
        out_q, hn_q = m.forward_quantized(x_q)
        for d in range(2):
            h = m._dirs[d].handle.forward_i32(x_q.transpose(0, 1).contiguous(), reverse=d == 1)
            assert torch.equal(out_q[:, :, d * H:(d + 1) * H], (h[1:] if d == 0 else h[:T]).transpose(0, 1))
            assert torch.equal(hn_q[d], h[T] if d == 0 else h[0])


@pytest.mark.parametrize("storage,H", [("int32", 64), ("float32", 300), ("float", 200)])
def test_batch_sizes_that_alternate(cuda_device, storage, H):
    """One module, batches of changing size (a last short one among them): plans, workspace and tensor maps follow."""
    import torch
    I, T = 20, 6
    rng = np.random.default_rng(H)
    xs = [torch.from_numpy(np.ascontiguousarray(gen_x(rng, b, T, I))).to(cuda_device) for b in (32, 7, 300, 31)]

    def module():
        m = _module("default", I, H, True, True, "float32" if storage == "float" else storage, xs[0], cuda_device)
        m.use_quantization = storage != "float"
        return m

    def step(m, x):
        out, hn = m.train()(x)
        grads = torch.autograd.grad(out.sum() + hn.sum(), list(m.parameters()))
        with torch.no_grad():
            return [out.detach(), hn.detach(), *grads, *m.eval()(x)]
    want = [step(module(), x) for x in xs]
    m = module()
    for i in (0, 1, 0, 2, 3, 2, 1, 0):
        assert all(torch.equal(a, b) for a, b in zip(step(m, xs[i]), want[i])), i
