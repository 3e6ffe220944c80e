"""GPU tests of the chain of state gradients of a quantized layer on the tensor cores, at the edges of its plans."""
import importlib

import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named

QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
pytestmark = pytest.mark.gpu


# (B, H, bidirectional): one row, ragged groups of four rows, one and several tiles of units, units that are no multiple of four, 64 units
# a CTA, several waves of clusters
@pytest.mark.parametrize("B,H,bidir", [(1, 97, False), (5, 128, True), (9, 129, False), (2, 190, False), (70, 257, True), (259, 300, False),
                                       (41, 383, False), (230, 512, False), (600, 512, False), (300, 500, True)])
@pytest.mark.parametrize("storage,cfg", [("float32", "cfg2"), ("int32", "default")])
def test_chain_of_state_gradients(cuda_device, storage, cfg, B, H, bidir):
    import torch
    torch.manual_seed(B + H)
    T, I, D = 4, 24, 2 if bidir else 1
    m = QuantGRU(I, H, bidirectional=bidir, quant_storage_dtype=storage).to(cuda_device)
    x = torch.randn(T, B, I, device=cuda_device)
    m.load_bitwidth_config(config_named(cfg).to_json_dict())
    m.use_quantization = True
    m.calibrating = True
    m(x * 0.6)                              # (a part of what follows is clamped)
    m.calibrating = False
    m.finalize_calibration()
    m.train()
    hx = (torch.randn(D, B, H, device=cuda_device) * 0.3).requires_grad_()
    x.requires_grad_()
    g_out, g_hn = torch.randn(T, B, D * H, device=cuda_device), torch.randn(D, B, H, device=cuda_device)
    wrt = [x, hx] + list(m.parameters())
    got = torch.autograd.grad(m(x, hx), wrt, (g_out, g_hn))
    want = torch.autograd.grad(m._forward_train_stepwise(x, hx), wrt, (g_out, g_hn))
    for a, b in zip(got, want):
        # the same fp32 gradients with R * dq summed in another order over 3H products, through T steps
        assert (a - b).norm() <= 2e-6 * b.norm() and (a - b).abs().max() <= 2e-5 * b.abs().max()


# 4, 16 and 28 rows a cluster; two, three and four tiles; warps that only read accumulators, and none
@pytest.mark.parametrize("H,B,sms", [(190, 4, 8), (190, 56, 8), (257, 16, 12), (300, 56, 12), (512, 4, 24), (512, 16, 24), (512, 56, 24),
                                     (512, 300, 0)])
def test_long_chain_repeats_its_bits(cuda_device, H, B, sms):
    """Operand, accumulators and partial sums are written again in each of 250 steps; sums have a fixed order, so every pass gives the
    same bits, and the gradients of the stepwise path."""
    import torch
    torch.manual_seed(H + B)
    T, I = 250, 16
    m = QuantGRU(I, H, quant_storage_dtype="int32").to(cuda_device)
    x = torch.randn(T, B, I, device=cuda_device)
    m.calibrating = True
    m(x)
    m.calibrating = False
    m.finalize_calibration()
    m.use_quantization = True
    m.train()
    if sms:
        m.set_option("sm_limit", sms)       # one or two clusters
    hx = (torch.randn(1, B, H, device=cuda_device) * 0.3).requires_grad_()
    x.requires_grad_()
    g_out = torch.randn(T, B, H, device=cuda_device)
    wrt = [x, hx] + list(m.parameters())
    got = [torch.autograd.grad(m(x, hx)[0], wrt, g_out) for _ in range(4)]
    assert m._dirs[0].handle.train_saved_bytes(2, T, B)     # (it was the one-call form)
    for again in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], again))
    want = torch.autograd.grad(m._forward_train_stepwise(x, hx)[0], wrt, g_out)
    for a, b in zip(got[0], want):
        # as above; a step's error of 2e-7 fades with the gate (z about 1/2, so two steps' worth), in sums over 250 steps of mixed sign
        assert (a - b).norm() <= 2e-6 * b.norm() and (a - b).abs().max() <= 2e-5 * b.abs().max()


@pytest.mark.parametrize("scale", [2.0 ** -112, 2.0 ** -118, 2.0 ** 60, 2.0 ** 100])
def test_chain_of_very_small_and_large_gradients(cuda_device, scale):
    """Near the ends of fp32 (2^-126, 2^128) the chain is as exact as in the middle: gradients that were scaled by a power of two
    come back scaled, save for what rounds below 2^-126."""
    import torch
    torch.manual_seed(11)
    T, B, I, H = 4, 24, 24, 200
    m = QuantGRU(I, H, quant_storage_dtype="float32").to(cuda_device)
    x = torch.randn(T, B, I, device=cuda_device)
    m.calibrating = True
    m(x)
    m.calibrating = False
    m.finalize_calibration()
    m.use_quantization = True
    m.train()
    hx = (torch.randn(1, B, H, device=cuda_device) * 0.3).requires_grad_()
    g_out = torch.randn(T, B, H, device=cuda_device)
    got = torch.autograd.grad(m(x, hx)[0], [hx, m.weight_hh_l0], g_out * scale)
    want = torch.autograd.grad(m(x, hx)[0], [hx, m.weight_hh_l0], g_out)
    for a, b in zip(got, want):
        a = a.double() / scale
        # sums of some 3H products, in four steps, of 2^-149 / 2 each at the most where a product rounds below 2^-126
        assert (a - b).norm() <= 1e-7 * b.norm() + 2.0 ** -149 / scale * (4 * 3 * H * b.numel()) ** 0.5


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_chain_keeps_what_is_not_finite(cuda_device, value):
    """An infinite or undefined gradient of one row reaches what it reached in fp32, and no other row."""
    import torch
    torch.manual_seed(5)
    T, B, I, H = 3, 6, 24, 130
    m = QuantGRU(I, H, quant_storage_dtype="float32").to(cuda_device)
    x = torch.randn(T, B, I, device=cuda_device)
    m.calibrating = True
    m(x)
    m.calibrating = False
    m.finalize_calibration()
    m.use_quantization = True
    m.train()
    hx = torch.zeros(1, B, H, device=cuda_device, requires_grad=True)
    x.requires_grad_()
    g_out = torch.randn(T, B, H, device=cuda_device)
    g_out[T - 1, 2, 17] = value
    got = torch.autograd.grad(m(x, hx)[0], [x, hx], g_out)
    want = torch.autograd.grad(m._forward_train_stepwise(x, hx)[0], [x, hx], g_out)
    for a, b, at in zip(got, want, (1, 1)):
        rows = [k for k in range(B) if k != 2]
        a, b = a.transpose(0, at), b.transpose(0, at)
        assert (a[rows] - b[rows]).abs().max() <= 2e-5 * b[rows].abs().max()
        assert torch.equal(torch.isfinite(a[2]), torch.isfinite(b[2]))
