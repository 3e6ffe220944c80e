"""GPU tests of the fp32 product on the tensor cores (three bf16 parts per operand), at the edges of its tiles and for values
that have no such parts."""
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import gen_weights

gru_ops = importlib.import_module(PKG_NAME + ".gru_ops")
pytestmark = pytest.mark.gpu


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _backward_without_r(dev, T, B, I, H, x_scale=1.0, dh_scale=1.0):
    """dx, dW, dR of the library (R = 0: dp and dq of a step depend on its own gradient and what comes through the update gate)
    and the same in float64."""
    import torch
    rng = np.random.default_rng(I * H)
    W, R, _, _ = gen_weights(rng, I, H)
    v = torch.rand(T, B, 4 * H, device=dev)
    h = torch.randn(T + 1, B, H, device=dev) * 0.3
    x = torch.randn(T, B, I, device=dev) * x_scale
    dh = torch.randn(T + 1, B, H, device=dev) * dh_scale
    with gru_ops.Handle(I, H, device=0) as hd:
        dx, dW, dR, dbw, dbr, _ = hd.backward(_t(W, dev), _t(R * 0, dev), x, dh, h, v)
    z, r, g, q = (v[..., k * H:(k + 1) * H].double() for k in range(4))
    carry = torch.zeros(B, H, dtype=torch.float64, device=dev)
    dp = torch.empty(T, B, 3 * H, dtype=torch.float64, device=dev)
    dq = torch.empty_like(dp)
    for t in range(T - 1, -1, -1):
        d = dh[t + 1].double() + carry
        dg = (1 - g[t] ** 2) * (1 - z[t]) * d
        dz = z[t] * (1 - z[t]) * (h[t].double() - g[t]) * d
        dr = r[t] * (1 - r[t]) * dg * q[t]
        dp[t], dq[t] = torch.cat([dz, dr, dg], 1), torch.cat([dz, dr, dg * r[t]], 1)
        carry = z[t] * d
    P, Q = dp.reshape(T * B, -1), dq.reshape(T * B, -1)
    want = [P @ _t(W, dev).double().t(), x.reshape(-1, I).double().t() @ P, h[:T].reshape(-1, H).double().t() @ Q]
    return [a.double().reshape(b.shape) for a, b in zip((dx, dW, dR), want)], want


# (T * B, I, H): I and 3H at and beside tiles of 128 and 256, rows in groups of four, two and one, K with and without a rest
@pytest.mark.parametrize("T,B,I,H", [(16, 256, 128, 128), (31, 131, 130, 86), (50, 81, 257, 43), (33, 128, 16, 171), (67, 96, 64, 256)])
def test_products_of_the_backward(cuda_device, T, B, I, H):
    for a, b in zip(*_backward_without_r(cuda_device, T, B, I, H)):
        # dp and dq carry a few fp32 roundings each (2^-24 of values with a spread of order one); sums over K of them less
        assert (a - b).norm() <= 5e-7 * b.norm()
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()


@pytest.mark.parametrize("x_scale,dh_scale", [(2.0 ** -118, 1.0), (1.0, 2.0 ** -118), (2.0 ** 50, 2.0 ** 40), (2.0 ** 105, 2.0 ** -30)])
def test_products_of_very_small_and_large_values(cuda_device, x_scale, dh_scale):
    """Near the ends of fp32 (2^-126, 2^128) the products are as exact as in the middle; every result here is a normal number."""
    for a, b in zip(*_backward_without_r(cuda_device, 16, 256, 128, 128, x_scale, dh_scale)):
        # as above, and what is below 2^-126 rounds to 2^-149: of sums near 2^-120 over 384 terms and more, 2^-150 each, less than 1e-7
        assert (a - b).norm() <= 6e-7 * b.norm()
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()


@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan"), 3.4e38])
def test_input_projection_of_values_without_bf16_parts(cuda_device, value):
    """A row with such a value takes the fp32 multiply-adds of its tile; the other rows are as before."""
    import torch
    T, B, I, H = 2, 700, 128, 300
    rng = np.random.default_rng(3)
    W, R, bw, br = (_t(a, cuda_device) for a in gen_weights(rng, I, H))
    x = torch.randn(T, B, I, device=cuda_device)
    bad = x.clone()
    bad[0, 130, 7] = value
    with gru_ops.Handle(I, H, device=0) as hd:
        clean = hd.forward_float(W, R, bw, br, x)
        got = hd.forward_float(W, R, bw, br, bad)
    # the step in float64 for the one row (a finite product that overflows in fp32 is an infinity here too: |w| >= 2^-10)
    pre = torch.where(W[7].abs() * abs(value) > 3.4028235e38, torch.sign(W[7]) * torch.sign(torch.tensor(value)).item() * float("inf"),
                      (bad[0, 130].double() @ W.double())) if np.isinf(value) else bad[0, 130].double() @ W.double()
    pre = pre + bw.double()
    z, r = torch.sigmoid(pre[:H] + br[:H].double()), torch.sigmoid(pre[H:2 * H] + br[H:2 * H].double())
    want = (1 - z) * torch.tanh(pre[2 * H:] + r * br[2 * H:].double())
    row = got[1, 130].double()
    assert torch.equal(torch.isnan(row), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert (row - want)[ok].abs().max() <= 2e-6 if ok.any() else True
    others = [b for b in range(B) if b != 130]
    # (sums in another order where the tile was multiplied again)
    assert (got[:, others] - clean[:, others]).abs().max() <= 2e-6


@pytest.mark.parametrize("T,B,I,H", [(16, 256, 128, 128), (31, 131, 130, 86), (40, 100, 260, 44)])
def test_masked_products_of_the_backward(cuda_device, T, B, I, H):
    """The clamp masks of x, W and R zero their gradients' elements and change no other (rows in groups of four and single)."""
    import torch
    rng = np.random.default_rng(I * H)
    W, R, _, _ = (_t(a, cuda_device) for a in gen_weights(rng, I, H))
    rand = lambda *s: torch.randn(*s, device=cuda_device)
    v, h, x, dh = torch.rand(T, B, 4 * H, device=cuda_device), rand(T + 1, B, H) * 0.3, rand(T, B, I), rand(T + 1, B, H)
    shapes = {"x": (T * B, I), "h0": (B, H), "W": (I, 3 * H), "R": (H, 3 * H), "bw": (3 * H,), "br": (3 * H,),
              "ih_linear": (T * B, 3 * H), "hh_linear": (T * B, 3 * H), "gate_input": (T * B, 3 * H),
              "gate_output": (T * B, 3 * H), "h": (T * B, H)}
    ones = {n: torch.ones(s, dtype=torch.uint8, device=cuda_device) for n, s in shapes.items()}
    some = {n: (torch.rand(shapes[n], device=cuda_device) < 0.7).to(torch.uint8) for n in ("x", "W", "R")}
    with gru_ops.Handle(I, H, device=0) as hd:
        all_ = hd.backward(W, R, x, dh, h, v, masks=ones)
        part = hd.backward(W, R, x, dh, h, v, masks={**ones, **some})
    for a, b, n in zip(all_[:3], part[:3], ("x", "W", "R")):
        assert torch.equal(a.reshape(b.shape) * some[n].reshape(b.shape), b), n
