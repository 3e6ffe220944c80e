"""Timed cases of the quantized GRU: what a program built on ``QuantGRU`` spends its time in.

Four things are done with the module, and every case is one of them, called the way a program
calls it:

``infer``      ``module(x, hx)`` in eval mode with quantization on (float in, float out), through the
               integer path (``quant_storage_dtype="int32"``) or the float-storage path ("float32")
``int_io``     ``module.forward_quantized(x_q, h_q)``: integers in, integers out
``train``      one forward in train mode and the gradients of its outputs with respect to every parameter,
               the input and the initial state: quantization-aware (either storage) or float
``calibrate``  ``calibrating = True``, a few batches, ``finalize_calibration()`` by one of the three methods

A case is a dict: ``do`` (above), ``I``, ``H``, ``B``, ``T`` (input size, hidden size, batch, timesteps),
``bidir``, ``batch_first``, ``h0`` (an initial state is passed), ``bits`` (a bit-width configuration of
``workloads.config_named``), ``storage`` ("int32", "float32", or "float" for an unquantized module), ``x`` (the
input's distribution) and, for ``calibrate``, ``method`` and ``batches``.

Quantization parameters come from ranges that a float64 GRU written here in plain torch takes over the
first rows and steps of the input, so that they depend on the seed alone and not on the library's own
calibration pass, whose fp32 rounding may change.
"""
import importlib
import math

import numpy as np
import torch

from __graft_entry__ import PKG_NAME, load_package

load_package()
_params = importlib.import_module(PKG_NAME + ".params")
_workloads = importlib.import_module(PKG_NAME + ".workloads")
QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
_OP = importlib.import_module(PKG_NAME + "._cabi").OP_INDEX

_DEFAULTS = {"do": "infer", "bidir": False, "batch_first": False, "h0": False, "bits": "default", "storage": "int32",
             "x": "normal", "method": "", "batches": 0}


def _case(**kw):
    return {**_DEFAULTS, **kw}


def listed():
    return [
        # one frame of a streaming recogniser, state carried by the caller: nothing but call latency
        _case(name="stream_frame", I=80, H=256, B=1, T=1, h0=True, bits="cfg5", x="ar1"),
        # a small model's batch (keyword spotting size): few microseconds per kernel
        _case(name="small_batch", I=64, H=128, B=32, T=50, batch_first=True, bits="sym8_tensor"),
        # the bidirectional encoder layer that the benchmark reports
        _case(name="bidir_encoder", I=256, H=512, B=256, T=200, bidir=True, bits="cfg2"),
        # offline throughput: very many short sequences
        _case(name="throughput", I=128, H=256, B=4096, T=100, bits="cfg3", x="outliers"),
        # wide layer, long sequences: bound by the recurrence
        _case(name="wide_long", I=1024, H=1024, B=64, T=1000, bits="sym8_tensor", x="normal05"),
        # one very long sequence (a recording), batch 1
        _case(name="long_stream", I=80, H=256, B=1, T=16000, bits="cfg5", x="ar1"),
        # the module's default storage and bit widths, sizes that are no multiple of anything
        _case(name="float_storage_odd", I=161, H=321, B=37, T=127, bidir=True, h0=True, batch_first=True, storage="float32"),
        # integers in and out with 16-bit activations
        _case(name="int_io_16bit_odd", do="int_io", I=45, H=100, B=21, T=61, h0=True, bits="wide16"),
        # quantization-aware fine-tuning of the encoder layer, module defaults (float32 storage)
        _case(name="qat_encoder", do="train", I=256, H=512, B=256, T=200, bits="cfg2", storage="float32"),
        # quantization-aware training of the small model on the integer path
        _case(name="qat_small_int", do="train", I=64, H=128, B=32, T=50, h0=True, batch_first=True, bits="sym8_tensor"),
        # float pre-training, odd sizes
        _case(name="float_train_odd", do="train", I=130, H=262, B=65, T=91, bidir=True, storage="float"),
        # post-training calibration by the SQNR search, per-channel weights
        _case(name="calibrate_sqnr", do="calibrate", I=128, H=256, B=64, T=200, method="sqnr", batches=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choices(["infer", "int_io", "train", "calibrate"], [5, 1, 3, 1.5])[0]
    bits8 = ["default", "sym8_tensor", "cfg2", "cfg3", "cfg5", "pot2", "pot2_asym", "ih16", "gate_in16", "unsigned_x"]
    c = _case(do=do, bidir=rng.random() < 0.35, batch_first=rng.random() < 0.5, h0=rng.random() < 0.5,
              bits=rng.choice(bits8), storage=rng.choice(["int32", "int32", "float32"]),
              x=rng.choice(["normal", "normal05", "outliers", "ar1"]))
    if do == "infer":
        top = {"I": (8, 1024), "H": (16, 1024), "B": (1, 4096), "T": (1, 2000)}
        most = 1.0e11                     # multiply-adds of a pass
        if rng.random() < 0.2:            # a stream: batch 1, many or very few steps
            top.update(B=(1, 1), H=(16, 512), T=(1, 16000))
    elif do == "int_io":
        c["bits"], c["storage"] = rng.choice(["wide16"] + bits8), "int32"
        top = {"I": (8, 256), "H": (16, 256), "B": (1, 64), "T": (1, 200)}
        most = 2.0e9
    elif do == "train":
        c["storage"] = rng.choice(["float", "float32", "float32", "int32"])
        top = {"I": (8, 512), "H": (16, 512), "B": (1, 256), "T": (4, 200)}
        most = 2.0e10
    else:
        c.update(storage="int32", h0=False, bidir=False)
        c["method"], c["batches"] = rng.choice(["minmax", "sqnr", "percentile"]), rng.choice([1, 2])
        top = {"I": (8, 256), "H": (16, 256), "B": (1, 128), "T": (4, 200)}
        most = 5.0e9
    while True:
        for k, (lo, hi) in top.items():
            c[k] = _log(rng, lo, hi)
        if _macs(c) <= most and c["T"] * c["B"] * c["H"] <= 5.0e7:
            return c


# ------------------------------------------------------------------------------------- inputs
def _dirs(c):
    return 2 if c["bidir"] else 1


def _macs(c):
    n = c["T"] * c["B"] * 3 * c["H"] * (c["I"] + c["H"]) * _dirs(c)
    return n * max(1, c["batches"])


def _make_x(c, g, dev):
    """[T, B, I] fp32 of the case's distribution, generated on the device."""
    shape = (c["T"], c["B"], c["I"])
    x = torch.randn(shape, generator=g, device=dev)
    if c["x"] == "normal05":
        x *= 0.5
    elif c["x"] == "outliers":            # 1 % of the entries scaled by 8
        x = torch.where(torch.rand(shape, generator=g, device=dev) < 0.01, 8.0 * x, x)
    elif c["x"] == "ar1":                 # per-channel AR(1), coefficient 0.9, unit variance: a doubling scan over time
        x[1:] *= math.sqrt(1 - 0.81)
        for k in (1, 2, 4, 8, 16, 32, 64, 128):
            if k < c["T"]:
                x = torch.cat([x[:k], x[k:] + 0.9 ** k * x[:-k]])
    return x


def _ranges(c, weights, x, reverse):
    """Operator ranges of the float GRU over the first rows and steps of x (float64, plain torch)."""
    W, R, bw, br = (w.double() for w in weights)   # [3H, I], [3H, H], [3H], [3H]; gate order r, z, n
    H = c["H"]
    x = x[:24, :16].double()
    if reverse:
        x = x.flip(0)
    bound = x.abs().flatten()
    if c["x"] == "outliers":               # as percentile calibration would: the outliers clip
        bound = bound.sort().values[: max(1, int(0.999 * bound.numel()))]
    bound = bound.max()
    h = torch.zeros(x.shape[1], H, dtype=torch.float64, device=x.device)
    seen = {"x": [x.clamp(-bound, bound)]}
    for t in range(x.shape[0]):
        ih, hh = x[t] @ W.t() + bw, h @ R.t() + br
        r_in, z_in = ih[:, :H] + hh[:, :H], ih[:, H:2 * H] + hh[:, H:2 * H]
        r, z = torch.sigmoid(r_in), torch.sigmoid(z_in)
        n_in = ih[:, 2 * H:] + r * hh[:, 2 * H:]
        n = torch.tanh(n_in)
        old, new = z * h, (1 - z) * n
        h = old + new
        for name, v in (("h", h), ("weight_ih_linear", ih), ("weight_hh_linear", hh), ("update_gate_input", z_in),
                        ("reset_gate_input", r_in), ("new_gate_input", n_in), ("update_gate_output", z),
                        ("reset_gate_output", r), ("new_gate_output", n), ("mul_reset_hidden", r * hh[:, 2 * H:]),
                        ("mul_old_contribution", old), ("mul_new_contribution", new)):
            seen.setdefault(name, []).append(v)
    out = _params.Ranges(H)
    for name, vs in seen.items():
        v = torch.cat([a.flatten() for a in vs])
        out.min_v[_OP[name]], out.max_v[_OP[name]] = (float(e) for e in torch.aminmax(v))
    for name, w in zip(("W", "R", "bw", "br"), weights):
        w = torch.cat([w[H:2 * H], w[:H], w[2 * H:]])   # channel order of the library: z, r, n
        lo, hi = torch.aminmax(w.reshape(3 * H, -1), dim=1)
        out.ch_min[name], out.ch_max[name] = lo.cpu().numpy().copy(), hi.cpu().numpy().copy()
        out.min_v[_OP[name]], out.max_v[_OP[name]] = float(lo.min()), float(hi.max())
    return out


class _State:
    pass


def prepare(case, seed):
    c = {**_DEFAULTS, **case}
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(int(seed) % (1 << 60))
    D, T, B, H = _dirs(c), c["T"], c["B"], c["H"]
    s = _State()
    s.case = c
    s.module = m = QuantGRU(c["I"], H, batch_first=c["batch_first"], bidirectional=c["bidir"],
                            quant_storage_dtype="float32" if c["storage"] == "float" else c["storage"]).to(dev)
    with torch.no_grad():
        for p in m.parameters():
            p.uniform_(-1 / math.sqrt(H), 1 / math.sqrt(H), generator=g)
    m.train(c["do"] == "train")
    m.load_bitwidth_config(_workloads.config_named(c["bits"]).to_json_dict())
    m.use_quantization = c["storage"] != "float"
    x = _make_x(c, g, dev)
    s.hx = torch.rand((D, B, H), generator=g, device=dev) - 0.5 if c["h0"] else None
    if c["do"] == "calibrate":
        m.calibration_method, m.percentile_value = c["method"], 99.9
        s.batches = [x] + [_make_x(c, g, dev) for _ in range(c["batches"] - 1)]
        if c["batch_first"]:
            s.batches = [b.transpose(0, 1).contiguous() for b in s.batches]
        return s
    if c["storage"] != "float":
        for d, suffix in enumerate(["", "_reverse"][:D]):
            ws = [getattr(m, n + suffix).detach() for n in ("weight_ih_l0", "weight_hh_l0", "bias_ih_l0", "bias_hh_l0")]
            setattr(m, "quant_ranges" + suffix, _ranges(c, ws, x, d == 1))
        m.finalize_calibration()
    if c["do"] == "int_io":
        p = m.quant_params.c
        q = []
        for v, name in ((x, "x"), (s.hx, "h")):
            o = p.op[_OP[name]]
            lo = 0 if o.is_unsigned else -(1 << (o.bits - 1))
            q.append(None if v is None else (torch.round(v / o.scale) + o.zero_point).clamp(lo, lo + (1 << o.bits) - 1).to(torch.int32))
        x, s.hx = q
    if c["batch_first"]:
        x = x.transpose(0, 1).contiguous()
    if c["do"] == "train":
        shape = (B, T, D * H) if c["batch_first"] else (T, B, D * H)
        s.g_out = torch.randn(shape, generator=g, device=dev)
        s.g_hn = torch.randn((D, B, H), generator=g, device=dev)
        x.requires_grad_()
        if s.hx is not None:
            s.hx.requires_grad_()
    s.x = x
    return s


def run(state):
    s, do = state, state.case["do"]
    m = s.module
    if do == "infer":
        with torch.no_grad():
            return m(s.x, s.hx)
    if do == "int_io":
        return m.forward_quantized(s.x, s.hx)
    if do == "train":
        out, hn = m(s.x, s.hx)
        wrt = [s.x] + ([s.hx] if s.hx is not None else []) + list(m.parameters())
        return [out.detach(), hn.detach()] + list(torch.autograd.grad((out, hn), wrt, (s.g_out, s.g_hn)))
    m.reset_calibration()
    m.calibrating = True
    outs = [m(b) for b in s.batches]
    m.calibrating = False
    m.finalize_calibration()
    # the parameters that a quant-param file would hold: the real interval of every operator
    spans = []
    for p in [m.quant_params] + ([m.quant_params_reverse] if m.bidirectional else []):
        ops = [e for e in p.to_export_dict().values()]
        spans.append(np.concatenate([np.atleast_1d(np.asarray(e[k], np.float64)) for e in ops for k in ("real_min", "real_max")]))
    return outs, spans


def work(case):
    """Operands and results at the types the entry point takes and gives; weights as the inference paths
    hold them (one byte each, quantized once) or, where a pass starts from the float parameters, as fp32."""
    c = {**_DEFAULTS, **case}
    D, T, B, I, H = _dirs(c), c["T"], c["B"], c["I"], c["H"]
    w = D * (3 * H * (I + H) + 6 * H)
    x, out, state = T * B * I, T * B * D * H, D * B * H
    macs = T * B * 3 * H * (I + H) * D
    if c["do"] == "train":     # x, weights, gradients of both outputs in; outputs and a gradient for each input out
        return {"bytes": 4 * (2 * x + 2 * w + 2 * out + 4 * state), "flops": 2 * 3 * macs}
    if c["do"] == "calibrate":
        n = c["batches"]
        return {"bytes": 4 * (n * (x + out + state) + w), "flops": 2 * n * macs}
    return {"bytes": 4 * (x + out + 2 * state) + w, "flops": 2 * macs}


def tolerance(case):
    c = {**_DEFAULTS, **case}
    if c["do"] in ("infer", "int_io"):
        return "exact"         # integers, and their products with one scale
    if c["do"] == "train":
        # fp32 sums over T * B products, carried back through T steps
        return {"rel": 2e-5, "max": 1e-3}
    if c["method"] == "minmax":
        return {"rel": 1e-5, "max": 1e-3}
    # ranges come from 2048-bin histograms: a value that rounds into the next bin moves one by a bin or a
    # step of the search
    return {"rel": 5e-3, "max": 5e-2}
