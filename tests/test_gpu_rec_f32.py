"""GPU tests of the fp32 recurrences and of the fp32 matrix product behind them, at the sizes where their
plans change: one CTA per row group, clusters of 2 to 16, layers wider than the registers of a
cluster hold, ragged rows and units, split and unsplit K."""
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME
from oracle.backward_np import gru_backward
from tests.cases import gen_weights, gen_x

gru_ops = importlib.import_module(PKG_NAME + ".gru_ops")
pytestmark = pytest.mark.gpu


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


@pytest.mark.parametrize("T,B,I,H", [(3, 1, 1, 1), (5, 3, 7, 31), (4, 2, 64, 32), (7, 40, 5, 33), (6, 9, 129, 128), (3, 17, 3, 129),
                                     (40, 65, 12, 160), (3, 5, 20, 200), (3, 150, 66, 262), (2, 33, 16, 385), (3, 70, 8, 512),
                                     (2, 3, 8, 513)])
def test_float_forward_and_backward(oracle, cuda_device, T, B, I, H):
    rng = np.random.default_rng(100 * H + B)
    W, R, bw, br = gen_weights(rng, I, H)
    x = gen_x(rng, T, B, I)
    h0 = (rng.standard_normal((B, H)) * 0.3).astype(np.float32)
    want_h, want_v = oracle.forward_float(T, B, I, H, W, R, bw, br, x, h0, want_v=True)
    dh_new = rng.standard_normal((T + 1, B, H)).astype(np.float32)
    with gru_ops.Handle(I, H, device=0) as hd:
        d = [_t(a, cuda_device) for a in (W, R, bw, br, x)]
        h, v = hd.forward_float(*d, h0=_t(h0, cuda_device), want_v=True)
        assert np.abs(h.cpu().numpy() - want_h).max() <= 1e-5
        assert np.abs(v.cpu().numpy() - want_v).max() <= 1e-5 * max(1.0, np.abs(want_v).max())
        got = hd.backward(d[0], d[1], d[4], _t(dh_new, cuda_device), _t(want_h, cuda_device), _t(want_v, cuda_device))
    want = gru_backward(W, R, x, dh_new, want_h, want_v)
    for g, w in zip(got, want):
        g = g.cpu().numpy().reshape(w.shape)
        assert np.abs(g - w).max() <= 2e-5 * max(np.abs(w).max(), 1e-30)


# a cell a thread with 9, 11 and 16 rows a cluster, the next number of rows, CTAs of 32 and 64 units on either side of their line
@pytest.mark.parametrize("T,B,I,H", [(3, 130, 5, 262), (3, 75, 8, 512), (2, 112, 8, 500), (2, 119, 8, 512), (3, 96, 9, 256), (3, 128, 9, 256),
                                     (3, 140, 6, 160), (4, 300, 5, 100), (5, 33, 4, 128)])
def test_float_recurrences_between_their_forms(oracle, cuda_device, T, B, I, H):
    test_float_forward_and_backward(oracle, cuda_device, T, B, I, H)


def test_two_directions_share_an_odd_number_of_clusters(cuda_device):
    """65 rows of 262 units in both directions: the last clusters have two rows; the same as torch.nn.GRU."""
    import torch
    torch.manual_seed(4)
    QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
    T, B, I, H = 5, 65, 12, 262
    m = QuantGRU(I, H, bidirectional=True).to(cuda_device).train()
    m.use_quantization = False
    ref = torch.nn.GRU(I, H, bidirectional=True).double()
    with torch.no_grad():
        for name, p in ref.named_parameters():
            p.copy_(getattr(m, name).double().cpu())
    x = torch.randn(T, B, I)
    g = torch.randn(T, B, 2 * H)
    xs = [x.to(cuda_device).requires_grad_(), x.double().requires_grad_()]
    out = m(xs[0])[0]
    want = ref(xs[1])[0]
    assert (out.detach().cpu() - want.detach()).abs().max() <= 2e-6
    wrt = [[xs[0]] + [getattr(m, n) for n, _ in ref.named_parameters()], [xs[1]] + [p for _, p in ref.named_parameters()]]
    got = torch.autograd.grad(out, wrt[0], g.to(cuda_device))
    for a, b in zip(got, torch.autograd.grad(want, wrt[1], g.double())):
        assert (a.cpu() - b).abs().max() <= 1e-5 * b.abs().max()


def _grid_of(call, name):
    """CTAs of the launches of a kernel during the call, as the profiler saw them."""
    import json
    import os
    import tempfile
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        p.export_chrome_trace(os.path.join(d, "t.json"))
        with open(os.path.join(d, "t.json")) as f:
            events = json.load(f)["traceEvents"]
    return [e["args"]["grid"][0] for e in events if name in e.get("name", "") and "grid" in e.get("args", {})]


@pytest.mark.parametrize("H", [256, 512])
def test_recurrences_are_planned_within_the_sm_limit(cuda_device, H):
    """One direction with sm_limit 20 is cut into clusters for 20 SMs (two waves of them at the most here), also where two
    such directions would fit the chip."""
    import torch
    torch.manual_seed(H)
    QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
    T, B, I = 4, 30, 16
    x = torch.randn(T, B, I, device=cuda_device)

    def step(m):
        out = m(x)[0]
        return out, torch.autograd.grad(out, list(m.parameters()), torch.ones_like(out))
    m = QuantGRU(I, H).to(cuda_device).train()
    m.use_quantization = False
    free = step(m)
    assert max(_grid_of(lambda: step(m), "k_float_chain")) > 2 * 20
    m.set_option("sm_limit", 20)
    kept = step(m)
    for name in ("k_float_chain", "k_bwd_chain"):
        grids = _grid_of(lambda: step(m), name)
        assert len(grids) == 1 and grids[0] <= 2 * 20, (name, grids)
    # other clusters, the same sums in another order
    for a, b in zip((kept[0], *kept[1]), (free[0], *free[1])):
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()


@pytest.mark.parametrize("H,few,many", [(200, 300, 3000), (320, 300, 2500), (512, 100, 1100)])
def test_float_forward_of_very_many_rows(cuda_device, H, few, many):
    """Beyond some number of rows the forward goes step by step: the same states as the rows give in smaller batches."""
    import torch
    T, I = 3, 20
    rng = np.random.default_rng(H)
    w = [_t(a, cuda_device) for a in gen_weights(rng, I, H)]
    x = _t(gen_x(rng, T, many, I), cuda_device)
    h0 = _t((rng.standard_normal((many, H)) * 0.3).astype(np.float32), cuda_device)
    with gru_ops.Handle(I, H, device=0) as hd:
        launches = hd.launch_count()
        want, want_v = hd.forward_float(*w, x[:, :few].contiguous(), h0=h0[:few], want_v=True)
        in_one = hd.launch_count() - launches
        got, got_v = hd.forward_float(*w, x, h0=h0, want_v=True)
        assert hd.launch_count() - launches - in_one >= 2 * T > in_one      # step by step, and in one launch
    # sums of H products in another order, |r|, |h| <= 1: a few ulp of values of order one
    assert (got[:, :few] - want).abs().max() <= 2e-6 and (got_v[:, :few] - want_v).abs().max() <= 2e-5
