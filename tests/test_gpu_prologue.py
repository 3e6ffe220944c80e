"""GPU tests of the activations' quantization (k_prologue): 128-bit rows quantized by the reciprocal, with the division where a half
may lie between the two, against numpy's fp32 division and against the scalar path, at values around every half."""
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import OP, config_named, make_case

gru_ops = importlib.import_module(PKG_NAME + ".gru_ops")
pytestmark = pytest.mark.gpu


def around_halves(scale, zp, lo, hi):
    """fp32 values whose quotient by scale is a half, some ulps to either side of it, or an integer; and what no rule may assume."""
    q = np.arange(lo - 3, hi + 4, dtype=np.float64)[:, None] - zp + np.array([0.0, 0.5])
    x = (q * np.float64(scale)).astype(np.float32).ravel()
    ulp = np.spacing(np.abs(x) + np.float32(1e-30)).astype(np.float32)
    x = np.concatenate([x + np.float32(k) * ulp for k in (-9, -3, -2, -1, 0, 1, 2, 3, 9)])
    odd = np.array([0.0, -0.0, 1e-45, -1e-45, 1e-38, 3.4e38, -3.4e38, 2.0 ** 19 * scale, 2.0 ** 22 * scale, -2.0 ** 23 * scale])
    return np.concatenate([x, odd.astype(np.float32)])


@pytest.mark.parametrize("I", [4, 128, 132, 384])
@pytest.mark.parametrize("scale,zp", [(0.0625, 0), (1 / 3, -7), (0.013, 101), (0.9999999, -128), (1.7e-4, 0)])
def test_rows_of_four_equal_division(oracle, cuda_device, I, scale, zp):
    import torch
    B, H = 3, 8
    case = make_case(I, 2, B, I, H, oracle, config_named("default"))
    op = case.params.c.op[OP["x"]]
    op.scale, op.zero_point = scale, zp
    s, lo, hi = oracle.dequantize(np.array([zp + 1]), case.params.c, OP["x"])[0], -128, 127     # (as its M and shift have it)
    values = around_halves(s, zp, lo, hi)
    T = max(3, -(-len(values) // (B * I)))
    x = np.random.default_rng(I).permutation(np.resize(values, T * B * I)).reshape(T, B, I)
    flat = torch.zeros(x.size + 4, device=cuda_device)
    aligned, shifted = flat[:x.size].view(T, B, I), flat[1:x.size + 1].view(T, B, I)
    w = [torch.from_numpy(a).to(cuda_device) for a in (case.W, case.R, case.bw, case.br)]
    with gru_ops.Handle(I, H, device=cuda_device.index or 0) as hd:
        hd.set_params(case.params)
        hd.set_weights_f32(*w)
        for int_storage in (False, True):
            runs = []
            for view in (aligned, shifted):              # (a base that is no multiple of 16 bytes: the scalar path)
                view.copy_(torch.from_numpy(x).to(cuda_device))
                h, v, x_q, masks = hd.forward_fstorage_train(*w, view, int_storage=int_storage)
                runs.append([x_q, masks["x"], h, v])
            for a, b in zip(*runs):
                assert torch.equal(a, b)
            with np.errstate(over="ignore"):
                t = x / s
                raw = np.rint(t) + np.float32(zp) if int_storage else np.rint(t + np.float32(zp))
            assert np.array_equal(runs[0][0].cpu().numpy(), np.clip(raw, lo, hi))
            assert np.array_equal(runs[0][1].cpu().numpy().reshape(T, B, I) != 0, (raw >= lo) & (raw <= hi))


def test_not_a_number_and_infinity_as_the_scalar_path_has_them(oracle, cuda_device):
    import torch
    T, B, I, H = 2, 3, 8, 8
    case = make_case(5, T, B, I, H, oracle, config_named("default"))
    x = torch.from_numpy(case.x).to(cuda_device)
    x.view(-1)[::5] = torch.tensor([float("nan"), float("inf"), float("-inf")], device=cuda_device).repeat(4)[:len(x.view(-1)[::5])]
    shifted = torch.empty(x.numel() + 4, device=cuda_device)[1:x.numel() + 1].view(T, B, I)
    shifted.copy_(x)
    w = [torch.from_numpy(a).to(cuda_device) for a in (case.W, case.R, case.bw, case.br)]
    with gru_ops.Handle(I, H, device=cuda_device.index or 0) as hd:
        hd.set_params(case.params)
        hd.set_weights_f32(*w)
        for int_storage in (False, True):
            a, b = [hd.forward_fstorage_train(*w, view, int_storage=int_storage) for view in (x, shifted)]
            assert torch.equal(a[2], b[2]) and torch.equal(a[3]["x"], b[3]["x"]) and torch.equal(a[0], b[0])
