"""``QuantGRU``: the nn.GRU-compatible module of the reference (pytorch/quant_gru.py:1060-2400),
restricted to the inference hot path and running on libqgru_b200.so.

What is kept, with the reference's names and meaning: the constructor signature and parameter
names (``weight_ih_l0`` ... in PyTorch's (r, z, n) gate order), ``batch_first``,
``bidirectional``, ``use_quantization``, ``calibrating`` + ``finalize_calibration`` (MinMax),
``load_bitwidth_config`` / ``set_all_bitwidth``, ``forward`` (float mode, calibration mode,
quantized mode with ``quant_storage_dtype="int32"``: the integer path, or ``"float32"``: the
float-storage path with real sigmoid / tanh, both in eval mode), ``forward_quantized`` (int32 in / out),
``export_quant_params`` / ``load_quant_params``.

What differs by design: each direction owns a ``gru_ops.Handle`` whose packed weights are
re-quantized only when a parameter tensor or the quant params change (the reference
re-quantizes weights and regenerates LUTs on every call); the reverse direction runs on the
same input with reversed time indexing instead of two ``flip`` copies; a quantized forward is one library
call for both directions (they run beside each other on two CUDA streams) that reads and writes
the module's own tensors, batch-first ones too, and does not wait for the GPU: like any torch
operation its results are ordered on the current stream.  A layer has one workspace: calls on different streams run
one after the other on the GPU (a call captured into a graph excepted: whoever launches the graph orders it).  A wait inside
a kernel that runs out is raised by the first call of the module (backward included) that begins after the GPU got
there, or by ``synchronize()``, which waits for the module's work (as ``forward_quantized`` does, which checks its
input's range).  Training: in train() mode with gradients enabled, forward
runs through an autograd function whose backward is qgru_backward - the fp32 GRU in float mode,
and with use_quantization the quantized forward in training mode (float-storage path, or the
integer path with quant_storage_dtype="int32") with its clamp masks as straight-through
estimators (QAT).  ONNX and AIMET hooks are not
built.
"""
import json
import math

import torch
from torch import nn

from . import _cabi, gru_ops
from .params import GRUQuantParams, Histograms, OperatorQuantConfig, Ranges


def reorder_weights_pytorch_to_haste(w):
    """(r, z, n) -> (z, r, n) along dim 0 (pytorch/quant_gru.py:617-639); self-inverse."""
    h3 = w.shape[0] // 3
    return torch.cat([w[h3:2 * h3], w[:h3], w[2 * h3:]], 0).contiguous()


def convert_weights_to_haste_format(weight_ih, weight_hh, bias_ih, bias_hh, hidden_size, device):
    """[3H, I] / [3H, H] PyTorch weights -> W [I, 3H], R [H, 3H], bw, br [3H] in (z, r, n) order
    (pytorch/quant_gru.py:661-712); missing biases become zeros."""
    W = reorder_weights_pytorch_to_haste(weight_ih.detach().to(device, torch.float32)).t().contiguous()
    R = reorder_weights_pytorch_to_haste(weight_hh.detach().to(device, torch.float32)).t().contiguous()
    if bias_ih is not None and bias_hh is not None:
        bw = reorder_weights_pytorch_to_haste(bias_ih.detach().to(device, torch.float32))
        br = reorder_weights_pytorch_to_haste(bias_hh.detach().to(device, torch.float32))
    else:
        bw = torch.zeros(3 * hidden_size, device=device, dtype=torch.float32)
        br = torch.zeros(3 * hidden_size, device=device, dtype=torch.float32)
    return W, R, bw, br


class _FloatGRUFunction(torch.autograd.Function):
    """One direction of the fp32 GRU with its backward pass (the reference's GRUFunction,
    pytorch/quant_gru.py:760-1058, float mode): forward keeps h and the gate buffer v, backward
    is qgru_backward.  Inputs in haste layout: x [T,B,I], W [I,3H], R [H,3H], bw, br [3H],
    h0 [B,H]; returns h [(T+1),B,H] (slot 0 = h0)."""

    @staticmethod
    def forward(ctx, handle, x, W, R, bw, br, h0):
        h, v = handle.forward_float(W, R, bw, br, x, h0, want_v=True)
        ctx.handle = handle
        ctx.save_for_backward(x, W, R, h, v)
        return h

    @staticmethod
    def backward(ctx, dh_all):
        x, W, R, h, v = ctx.saved_tensors
        dh_all = dh_all.contiguous()
        # the gradient of slot 0 (h0 passed through as an output) is added to what flows back to h0
        dx, dW, dR, dbw, dbr, dh0 = ctx.handle.backward(W, R, x, dh_all, h, v)
        return None, dx, dW, dR, dbw, dbr, dh0 + dh_all[0]


class _QuantGRUFunction(torch.autograd.Function):
    """One direction of quantization-aware training (the reference's GRUFunction with
    use_quantization and float32 storage, pytorch/quant_gru.py:826-1050): forward is the
    float-storage quantized forward in training mode (gate buffer and clamp masks kept),
    backward differentiates through the dequantized quantized tensors with the masks as
    straight-through estimators (qgru_backward)."""

    @staticmethod
    def forward(ctx, handle, qp, int_storage, x, W, R, bw, br, h0):
        handle.set_params(qp)
        handle.set_weights_f32(W, R, bw, br)
        # float32 storage: float requantization, real sigmoid / tanh; int32 storage: the integer
        # path (piecewise-linear gates) in training mode
        h, v, x_q, masks = handle.forward_fstorage_train(W, R, bw, br, x, h0, int_storage=int_storage)
        Wd, Rd, _, _ = handle.get_weights_dequantized()
        xd = handle.dequantize_f32(x_q.to(torch.float32), "x")
        ctx.handle, ctx.masks = handle, masks
        ctx.save_for_backward(xd, Wd, Rd, h, v)
        return h

    @staticmethod
    def backward(ctx, dh_all):
        xd, Wd, Rd, h, v = ctx.saved_tensors
        dh_all = dh_all.contiguous()
        dx, dW, dR, dbw, dbr, dh0 = ctx.handle.backward(Wd, Rd, xd, dh_all, h, v, masks=ctx.masks)
        return None, None, None, dx, dW, dR, dbw, dbr, dh0 + dh_all[0]


class _LayerFunction(torch.autograd.Function):
    """Training of the whole layer, both directions, weights in the module's layout: one library call forward,
    one backward (qgru_train_forward / qgru_train_backward; modes as there).  Inputs: x and hx as the
    module takes them (fp32), then w_ih, w_hh, b_ih, b_hh per direction (biases may be None).  What the backward needs
    is in saved tensors (freed after it, hooks apply): the library's block of every direction and, in float mode, x."""

    @staticmethod
    def forward(ctx, module, mode, saved_bytes, x, hx, *params):
        H, D = module.hidden_size, module.num_directions
        t_dim, b_dim = (1, 0) if module.batch_first else (0, 1)
        T, B = x.shape[t_dim], x.shape[b_dim]
        handles = [module._dirs[d].handle for d in range(D)]
        if mode == 0:
            x = x.transpose(0, 1).contiguous() if module.batch_first else x.contiguous()
            x_ts, x_bs = B * x.shape[2], x.shape[2]
        else:
            if x.stride(-1) != 1:
                x = x.contiguous()
            x_ts, x_bs = x.stride(t_dim), x.stride(b_dim)
        saved = torch.empty((D, (saved_bytes + 255) // 256 * 256), dtype=torch.uint8, device=x.device)
        dirs = (_cabi.TrainDir * D)()
        params = [p if p is None else p.contiguous() for p in params]
        for d in range(D):
            for name, p in zip(("W", "R", "bw", "br"), params[4 * d:4 * d + 4]):
                setattr(dirs[d], name, p.data_ptr() if p is not None else None)
            dirs[d].saved = saved[d].data_ptr()
        out = torch.empty((B, T, D * H) if module.batch_first else (T, B, D * H), device=x.device)
        h_n = torch.empty((D, B, H), device=x.device)
        h = handles[0]
        h._ck(h._lib.qgru_train_forward(h._h, handles[1]._h if D == 2 else None, mode, T, B, x.data_ptr(), x_ts, x_bs,
                                        hx.data_ptr() if hx is not None else None, dirs, out.data_ptr(), out.stride(t_dim),
                                        out.stride(b_dim), h_n.data_ptr(), gru_ops._stream(x.device)), "qgru_train_forward")
        ctx.handles, ctx.mode, ctx.batch_first, ctx.shares_x = handles, mode, module.batch_first, [d.shares_x for d in dirs]
        ctx.shape, ctx.param_shapes = (T, B, x.shape[2], H), [None if p is None else p.shape for p in params]
        ctx.set_materialize_grads(False)
        keep = [saved, x] if mode == 0 else [saved]
        ctx.kept_as = [(t.dtype, t.shape, t.device) for t in keep]
        ctx.save_for_backward(*keep)
        return out, h_n

    @staticmethod
    def backward(ctx, dout, dh_n):
        keep = ctx.saved_tensors
        if any((t.dtype, t.shape, t.device) != as_ for t, as_ in zip(keep, ctx.kept_as)):
            raise RuntimeError("a saved-tensor hook has returned another type, shape or device than it was given")
        saved, *x = [t.contiguous() for t in keep]
        if saved.data_ptr() % 256:      # (a hook's view: the library reads the block's parts as words and vectors)
            saved = saved.clone()
        T, B, I, H = ctx.shape
        D, dev = len(ctx.handles), saved.device
        t_dim, b_dim = (1, 0) if ctx.batch_first else (0, 1)
        if dout is None:
            dout = torch.zeros((B, T, D * H) if ctx.batch_first else (T, B, D * H), device=dev)
        elif dout.stride(-1) != 1:
            dout = dout.contiguous()
        if dh_n is not None:
            dh_n = dh_n.contiguous()
        need = ctx.needs_input_grad
        dx = torch.empty((T, B, I), device=dev) if need[3] else None
        dh0 = torch.empty((D, B, H), device=dev) if need[4] else None
        grads = [torch.empty(s, device=dev) if s is not None and n else None for s, n in zip(ctx.param_shapes, need[5:])]
        dirs = (_cabi.TrainDir * D)()
        for d in range(D):
            dirs[d].saved, dirs[d].shares_x = saved[d].data_ptr(), ctx.shares_x[d]
            for name, g in zip(("dW", "dR", "dbw", "dbr"), grads[4 * d:4 * d + 4]):
                setattr(dirs[d], name, g.data_ptr() if g is not None else None)
        h = ctx.handles[0]
        h._ck(h._lib.qgru_train_backward(h._h, ctx.handles[1]._h if D == 2 else None, ctx.mode, T, B,
                                         x[0].data_ptr() if x else None, dout.data_ptr(), dout.stride(t_dim),
                                         dout.stride(b_dim), dh_n.data_ptr() if dh_n is not None else None,
                                         dx.data_ptr() if dx is not None else None, dh0.data_ptr() if dh0 is not None else None,
                                         dirs, gru_ops._stream(dev)), "qgru_train_backward")
        if dx is not None and ctx.batch_first:
            dx = dx.transpose(0, 1)
        return (None, None, None, dx, dh0, *grads)


class _Direction:
    """Per-direction run-time state: handle, haste-layout weights, what the handle holds."""

    def __init__(self):
        self.handle = None
        self.weights = None
        self.weights_key = None
        self.params_key = None
        self.loaded_key = None


class QuantGRU(nn.Module):
    def __init__(self, input_size, hidden_size, num_layers=1, bias=True, batch_first=False,
                 dropout=0.0, bidirectional=False, use_quantization=False, use_pot2_scale=False,
                 quant_storage_dtype="float32"):
        super().__init__()
        if num_layers != 1:
            raise NotImplementedError("only num_layers=1 is supported")
        if dropout > 0:
            raise NotImplementedError("dropout is not supported")
        if quant_storage_dtype not in ("float32", "int32"):
            raise ValueError(f"quant_storage_dtype must be 'float32' or 'int32', got {quant_storage_dtype}")
        self.input_size, self.hidden_size, self.num_layers = input_size, hidden_size, num_layers
        self.bias, self.batch_first, self.dropout = bias, batch_first, dropout
        self.bidirectional = bidirectional
        self.num_directions = 2 if bidirectional else 1
        self.use_quantization = use_quantization
        self.quant_storage_dtype = quant_storage_dtype
        suffixes = [""] + (["_reverse"] if bidirectional else [])
        for s in suffixes:
            setattr(self, "weight_ih_l0" + s, nn.Parameter(torch.empty(3 * hidden_size, input_size)))
            setattr(self, "weight_hh_l0" + s, nn.Parameter(torch.empty(3 * hidden_size, hidden_size)))
            if bias:
                setattr(self, "bias_ih_l0" + s, nn.Parameter(torch.empty(3 * hidden_size)))
                setattr(self, "bias_hh_l0" + s, nn.Parameter(torch.empty(3 * hidden_size)))
            else:
                self.register_parameter("bias_ih_l0" + s, None)
                self.register_parameter("bias_hh_l0" + s, None)
        self.reset_parameters()
        self._bitwidth_config = OperatorQuantConfig()
        self._bitwidth_config.use_pot2 = bool(use_pot2_scale)
        self.calibration_method = "minmax"
        self.percentile_value = 100.0
        self.calibrating = False
        self.quant_ranges = self.quant_params = None
        self.quant_ranges_reverse = self.quant_params_reverse = None
        self.hist_collectors = self.hist_collectors_reverse = None
        self._quant_params_dirty = False
        self._dirs = [_Direction() for _ in suffixes]

    # ------------------------------------------------------------------ configuration
    @property
    def use_pot2_scale(self):
        return self._bitwidth_config.use_pot2

    @use_pot2_scale.setter
    def use_pot2_scale(self, v):
        self._bitwidth_config.use_pot2 = bool(v)
        self._quant_params_dirty = True

    def reset_parameters(self):
        stdv = 1.0 / math.sqrt(self.hidden_size)
        for p in self.parameters():
            nn.init.uniform_(p, -stdv, stdv)

    def load_bitwidth_config(self, config_file, verbose=False):
        if self.is_calibrated():
            return  # as the reference: ignored once params exist (pytorch/quant_gru.py:1389-1397)
        cfg = OperatorQuantConfig.from_json(config_file)
        self.use_quantization = not cfg.disable_quantization
        self._bitwidth_config = cfg
        self._quant_params_dirty = True

    def set_all_bitwidth(self, bitwidth=8, is_symmetric=True, verbose=False):
        self._bitwidth_config.set_all_bitwidth(bitwidth, is_symmetric)
        self._quant_params_dirty = True

    def is_calibrated(self):
        if self.bidirectional:
            return self.quant_params is not None and self.quant_params_reverse is not None
        return self.quant_params is not None

    def reset_calibration(self):
        self.quant_ranges = self.quant_params = None
        self.quant_ranges_reverse = self.quant_params_reverse = None
        self.hist_collectors = self.hist_collectors_reverse = None
        self._quant_params_dirty = False

    def _check_method(self):
        if self.calibration_method not in ("minmax", "sqnr", "percentile"):
            raise ValueError(f"calibration_method must be 'minmax', 'sqnr' or 'percentile', "
                             f"got {self.calibration_method!r}")

    def finalize_calibration(self, verbose=False):
        """Ranges (minmax) or histograms (sqnr / percentile) -> quant params and LUTs
        (pytorch/quant_gru.py finalize_calibration)."""
        self._check_method()
        if self.calibration_method == "minmax":
            if self.quant_ranges is None or (self.bidirectional and self.quant_ranges_reverse is None):
                raise RuntimeError("no calibration data: set calibrating=True and call forward() first")
            self.quant_params = gru_ops.calculate_gru_quantitative_parameters(self.quant_ranges, self._bitwidth_config)
            if self.bidirectional:
                self.quant_params_reverse = gru_ops.calculate_gru_quantitative_parameters(
                    self.quant_ranges_reverse, self._bitwidth_config)
        else:
            if self.hist_collectors is None or (self.bidirectional and self.hist_collectors_reverse is None):
                raise RuntimeError("no calibration data: set calibrating=True and call forward() first")
            pct = self.calibration_method == "percentile"
            self.quant_params = gru_ops.calculate_gru_quantitative_parameters_from_histograms(
                self.hist_collectors, self._bitwidth_config, pct, self.percentile_value)
            if self.bidirectional:
                self.quant_params_reverse = gru_ops.calculate_gru_quantitative_parameters_from_histograms(
                    self.hist_collectors_reverse, self._bitwidth_config, pct, self.percentile_value)
        self._quant_params_dirty = False

    # ---------------------------------------------------------- quant-param JSON files
    def export_quant_params(self, path):
        """Write the reference's quant-param JSON layout (pytorch/quant_gru.py:4252-4330)."""
        if not self.is_calibrated():
            raise RuntimeError("QuantGRU not calibrated")
        doc = {"model_info": {"input_size": self.input_size, "hidden_size": self.hidden_size,
                              "bias": self.bias, "batch_first": self.batch_first,
                              "bidirectional": self.bidirectional,
                              "use_pot2_scale": bool(self._bitwidth_config.use_pot2)},
               "operators": self.quant_params.to_export_dict()}
        if self.bidirectional:
            doc["operators_reverse"] = self.quant_params_reverse.to_export_dict()
        with open(path, "w", encoding="utf-8") as f:
            json.dump(doc, f, indent=2)

    def load_quant_params(self, path):
        with open(path, "r", encoding="utf-8") as f:
            doc = json.load(f)
        info = doc.get("model_info", {})
        if info.get("hidden_size", self.hidden_size) != self.hidden_size or \
                info.get("input_size", self.input_size) != self.input_size:
            raise ValueError("quant-param file was exported for a different input/hidden size")
        if bool(info.get("bidirectional", False)) != self.bidirectional:   # pytorch/quant_gru.py:4379-4383
            raise ValueError(f"bidirectional mismatch: file {info.get('bidirectional')}, module {self.bidirectional}")
        if "operators" not in doc:
            raise ValueError(f"unsupported quant-param file: no 'operators' (has {list(doc)})")
        pot2 = bool(info.get("use_pot2_scale", False))
        self.quant_params = GRUQuantParams.from_export_dict(doc["operators"], self.hidden_size, pot2)
        if self.bidirectional:
            if "operators_reverse" not in doc:
                raise ValueError("bidirectional module needs 'operators_reverse' in the file")
            self.quant_params_reverse = GRUQuantParams.from_export_dict(doc["operators_reverse"],
                                                                        self.hidden_size, pot2)
            # both directions quantize the same input (pytorch/quant_gru.py:4428-4433)
            fi, ri = doc["operators"].get("input", {}), doc["operators_reverse"].get("input", {})
            for field in ("multiplier", "shift", "zero_point"):
                if (field in fi or field in ri) and fi.get(field) != ri.get(field):
                    raise ValueError(f"operators.input and operators_reverse.input differ in {field}")
        self._bitwidth_config = self.quant_params.config()
        self.use_quantization = True
        self._quant_params_dirty = False

    # ----------------------------------------------------------------- run-time plumbing
    def _params_of(self, d):
        if d == 1:
            return [self.weight_ih_l0_reverse, self.weight_hh_l0_reverse, self.bias_ih_l0_reverse, self.bias_hh_l0_reverse]
        return [self.weight_ih_l0, self.weight_hh_l0, self.bias_ih_l0, self.bias_hh_l0]

    def _handle(self, d, device):
        st = self._dirs[d]
        if st.handle is None or st.handle.device != (device.index or 0):
            st.handle = gru_ops.Handle(self.input_size, self.hidden_size, device=device.index or 0)
            st.handle.set_option("rec", "fast")
            if self.bidirectional:
                # the two directions run side by side: each persistent kernel takes half the SMs
                sms = torch.cuda.get_device_properties(device).multi_processor_count
                st.handle.set_option("sm_limit", max(1, sms // 2))
            st.weights_key = st.params_key = st.loaded_key = None
        return st

    def _direction(self, d, device):
        st = self._dirs[d]
        if st.handle is None or st.handle.device != (device.index or 0):
            st = self._handle(d, device)
        ps = self._params_of(d)
        key = tuple((p.data_ptr(), p._version) if p is not None else None for p in ps)
        if key != st.weights_key:
            st.weights = convert_weights_to_haste_format(*ps, self.hidden_size, device)
            st.weights_key = key
            st.loaded_key = None
        return st

    def _load_params(self, st, d):
        """The direction's quant params on its handle; returns what identifies them."""
        qp = self.quant_params_reverse if d == 1 else self.quant_params
        key = (id(qp), qp.to_bytes())
        if key != st.params_key:
            st.params_key = st.loaded_key = None
            st.handle.set_params(qp)
            st.params_key = key
        return key

    def _ready_quant(self, d, device):
        st = self._direction(d, device)
        key = (st.weights_key, self._load_params(st, d))
        if key != st.loaded_key:
            st.handle.set_weights_f32(*st.weights)
            st.loaded_key = key
        return st

    def _split_h0(self, hx, batch, device, dtype):
        if hx is None:
            return [None] * self.num_directions
        want = (self.num_directions, batch, self.hidden_size)
        if tuple(hx.shape) != want:
            raise ValueError(f"hx must have shape {list(want)}, got {list(hx.shape)}")
        hx = hx.to(device=device, dtype=dtype)
        return [hx[d].contiguous() for d in range(self.num_directions)]

    def _has_calibration_data(self):
        have = self.quant_ranges if self.calibration_method == "minmax" else self.hist_collectors
        have_r = self.quant_ranges_reverse if self.calibration_method == "minmax" else self.hist_collectors_reverse
        return have is not None and (not self.bidirectional or have_r is not None)

    def _ensure_quant_ready(self):
        """Quant params are (re)derived whenever calibration data or the bit-width configuration
        changed since they were last computed, as the reference's forward does
        (pytorch/quant_gru.py:2106-2125): the documented flow `calibrating=True; forward();
        calibrating=False; forward()` needs no explicit finalize_calibration() for any method."""
        if self._quant_params_dirty and self._has_calibration_data():
            self.finalize_calibration()
        elif not self.is_calibrated():
            if self.quant_ranges is not None or self.hist_collectors is not None:
                self.finalize_calibration()   # raises if the data of the chosen method is missing
            else:
                raise RuntimeError("quantization is enabled but the module is not calibrated: set "
                                   "calibrating=True, run forward() on calibration data, then "
                                   "calibrating=False")

    def _combine(self, outs, T):
        """outs[d] = h [(T+1),B,H]; forward slots 1..T are the outputs, reverse slots 0..T-1."""
        of = outs[0][1:]
        hn = outs[0][T:T + 1]
        if not self.bidirectional:
            return of.contiguous(), hn.contiguous()
        orv = outs[1][:T]
        return torch.cat([of, orv], dim=-1), torch.cat([hn, outs[1][0:1]], dim=0)

    def _layer_forward(self, input, hx, device, dtype):
        """One quantized forward of every direction in one library call: (output, h_n)."""
        # (one frame of a stream is host time from end to end: no conversion, attribute or temporary that is not needed)
        x = input
        if x.dtype is not dtype or x.device != device or x.stride(-1) != 1:
            x = x.to(device=device, dtype=dtype).contiguous()
        shape = x.shape
        if len(shape) != 3 or shape[2] != self.input_size:
            raise ValueError(f"input must have {self.input_size} features in three dimensions, got {list(shape)}")
        H, D, batch_first = self.hidden_size, self.num_directions, self.batch_first
        if batch_first:
            B, T, _ = shape
            x_bs, x_ts, _ = x.stride()
        else:
            T, B, _ = shape
            x_ts, x_bs, _ = x.stride()
        h0 = None
        if hx is not None:
            if tuple(hx.shape) != (D, B, H):
                raise ValueError(f"hx must have shape {[D, B, H]}, got {list(hx.shape)}")
            if hx.dtype is not dtype or hx.device != device or not hx.is_contiguous():
                hx = hx.to(device=device, dtype=dtype).contiguous()
            h0 = hx.data_ptr()
        h = self._ready_quant(0, device).handle
        rev = self._ready_quant(1, device).handle._h if D == 2 else None
        # (the library keeps offsets inside a timestep in 32 bits: very long batch-first outputs are transposed)
        direct = not batch_first or T * D * H <= 1 << 25
        if batch_first and direct:
            out = x.new_empty((B, T, D * H))
            o_ts, o_bs = D * H, T * D * H
        else:
            out = x.new_empty((T, B, D * H))
            o_ts, o_bs = B * D * H, D * H
        h_n = x.new_empty((D, B, H))
        stream = torch._C._cuda_getCurrentRawStream(device.index or 0)
        if dtype is torch.int32:
            rc = h._lib.qgru_layer_forward_i32(h._h, rev, T, B, x.data_ptr(), x_ts, x_bs, h0, out.data_ptr(), o_ts, o_bs, h_n.data_ptr(), stream)
        else:
            rc = h._lib.qgru_layer_forward(h._h, rev, self.quant_storage_dtype != "int32", T, B, x.data_ptr(), x_ts, x_bs, h0, out.data_ptr(),
                                           o_ts, o_bs, h_n.data_ptr(), stream)
        if rc:
            h._ck(rc, "qgru_layer_forward")
        return out if direct else out.transpose(0, 1).contiguous(), h_n

    def _forward_train(self, input, hx):
        """Float mode and QAT with autograd."""
        device = input.device
        if input.dim() != 3 or input.shape[2] != self.input_size:
            raise ValueError(f"input must have {self.input_size} features in three dimensions, got {list(input.shape)}")
        params = [p for d in range(self.num_directions) for p in self._params_of(d)]
        for p in params:
            if p is not None and p.device != device:
                raise ValueError(f"input is on {device}, the parameters on {p.device}")
        states = [self._handle(d, device) for d in range(self.num_directions)]
        mode = 0 if not self.use_quantization else 2 if self.quant_storage_dtype == "int32" else 1
        if mode:
            for d, st in enumerate(states):
                self._load_params(st, d)
        B, T = input.shape[:2] if self.batch_first else (input.shape[1], input.shape[0])
        sizes = [st.handle.train_saved_bytes(mode, T, B) for st in states]
        if not all(sizes):
            return self._forward_train_stepwise(input, hx)
        for st in states:
            st.loaded_key = None        # the quantized weights of this step replace the loaded ones
        # (conversions outside the autograd function: torch carries the gradients back through them)
        params = [p if p is None or p.dtype == torch.float32 else p.to(torch.float32) for p in params]
        if hx is not None:
            hx = hx.to(device=device, dtype=torch.float32).contiguous()
        return _LayerFunction.apply(self, mode, max(sizes), input.to(torch.float32), hx, *params)

    def _forward_train_stepwise(self, input, hx):
        """Layers without the one-call form (H > 512, operands wider than 8 bit).
        Every tensor operation outside the two library calls is a
        torch operation, so gradients reach the module's parameters in their PyTorch layout."""
        x = input.transpose(0, 1) if self.batch_first else input
        device = x.device
        x = x.to(torch.float32).contiguous()
        T, B, _ = x.shape
        H = self.hidden_size
        outs, hns = [], []
        for d in range(self.num_directions):
            st = self._direction(d, device)
            w_ih, w_hh, b_ih, b_hh = self._params_of(d)
            W = reorder_weights_pytorch_to_haste(w_ih.to(torch.float32)).t().contiguous()
            R = reorder_weights_pytorch_to_haste(w_hh.to(torch.float32)).t().contiguous()
            if b_ih is not None and b_hh is not None:
                bw = reorder_weights_pytorch_to_haste(b_ih.to(torch.float32))
                br = reorder_weights_pytorch_to_haste(b_hh.to(torch.float32))
            else:
                bw = torch.zeros(3 * H, device=device)
                br = torch.zeros(3 * H, device=device)
            h0 = hx[d].to(torch.float32).contiguous() if hx is not None else torch.zeros(B, H, device=device)
            xd = x.flip(0).contiguous() if d == 1 else x
            if self.use_quantization:
                qp = self.quant_params_reverse if d == 1 else self.quant_params
                h = _QuantGRUFunction.apply(st.handle, qp, self.quant_storage_dtype == "int32", xd, W, R, bw, br, h0)
                st.params_key = st.loaded_key = None   # the handle was reloaded outside the module's cache
            else:
                h = _FloatGRUFunction.apply(st.handle, xd, W, R, bw, br, h0)
            outs.append(h[1:].flip(0) if d == 1 else h[1:])
            hns.append(h[T:T + 1])
        output = torch.cat(outs, dim=-1) if self.bidirectional else outs[0]
        h_n = torch.cat(hns, dim=0)
        if self.batch_first:
            output = output.transpose(0, 1).contiguous()
        return output, h_n

    # --------------------------------------------------------------------------- forward
    def forward(self, input, hx=None):
        if not torch.is_grad_enabled():
            return self._forward_impl(input, hx)
        needs_grad = (input.requires_grad or (hx is not None and hx.requires_grad) or
                      any(p.requires_grad for p in self.parameters()))
        if needs_grad and self.training and not self.calibrating:
            if self.use_quantization:
                self._ensure_quant_ready()
            if not input.is_cuda:
                raise ValueError("input must be a CUDA tensor")
            want = (self.num_directions, input.shape[0 if self.batch_first else 1], self.hidden_size)
            if hx is not None and tuple(hx.shape) != want:
                raise ValueError(f"hx must have shape {list(want)}, got {list(hx.shape)}")
            return self._forward_train(input, hx)
        with torch.no_grad():
            return self._forward_impl(input, hx)

    def _forward_impl(self, input, hx=None):
        device = input.device if input.is_cuda else torch.device("cuda", torch.cuda.current_device())
        if self.use_quantization and not self.calibrating:
            self._ensure_quant_ready()
            return self._layer_forward(input, hx, device, torch.float32)
        if self.batch_first:
            input = input.transpose(0, 1)
        x = input.to(device=device, dtype=torch.float32).contiguous()
        T, B, _ = x.shape
        h0 = self._split_h0(hx, B, device, torch.float32)

        if self.calibrating:
            self._check_method()
            outs = []
            for d in range(self.num_directions):
                st = self._direction(d, device)
                xd = x.flip(0).contiguous() if d == 1 else x
                if self.calibration_method == "minmax":
                    rng_name = "quant_ranges_reverse" if d == 1 else "quant_ranges"
                    if getattr(self, rng_name) is None:
                        setattr(self, rng_name, Ranges(self.hidden_size))
                    h = st.handle.calibrate_minmax(*st.weights, xd, getattr(self, rng_name), h0[d], want_h=True)
                else:
                    name = "hist_collectors_reverse" if d == 1 else "hist_collectors"
                    if getattr(self, name) is None:
                        setattr(self, name, Histograms(self.hidden_size, device.index or 0))
                    h = st.handle.calibrate_hist(*st.weights, xd, getattr(self, name),
                                                 self._bitwidth_config.granularity_list(), h0[d], want_h=True)
                    for w in st.weights:    # still being counted when the call returns, maybe not on the stream they were made on
                        w.record_stream(torch.cuda.current_stream(device))
                outs.append(torch.cat([h[1:].flip(0), h[0:1]], 0) if d == 1 else h)
            self._quant_params_dirty = True
        else:
            outs = []
            for d in range(self.num_directions):
                st = self._direction(d, device)
                xd = x.flip(0).contiguous() if d == 1 else x
                h = st.handle.forward_float(*st.weights, xd, h0[d])
                outs.append(torch.cat([h[1:].flip(0), h[0:1]], 0) if d == 1 else h)
        output, h_n = self._combine(outs, T)
        if self.batch_first:
            output = output.transpose(0, 1).contiguous()
        return output, h_n

    @torch.no_grad()
    def forward_quantized(self, input, hx=None):
        """int32 in / int32 out inference (pytorch/quant_gru.py:2318-2380)."""
        if not self.is_calibrated() or self.quant_params is None:
            raise RuntimeError("QuantGRU not calibrated")
        if input.is_floating_point():
            raise TypeError("forward_quantized only accepts already quantized integer input "
                            f"(int in / int out); got dtype={input.dtype}")
        device = input.device if input.is_cuda else torch.device("cuda", torch.cuda.current_device())
        out = self._layer_forward(input, hx, device, torch.int32)
        for st in self._dirs:
            st.handle.synchronize()     # values outside the operators' ranges are an error of this call
        return out

    def synchronize(self):
        """Waits for the module's work on the current stream and raises what went wrong in it on the GPU."""
        for st in self._dirs:
            if st.handle:
                st.handle.synchronize()

    def last_plans(self):
        return [st.handle.describe_plan() if st.handle else "" for st in self._dirs]

    def last_timings(self):
        return [st.handle.last_timing() for st in self._dirs if st.handle]

    def launch_count(self):
        return sum(st.handle.launch_count() for st in self._dirs if st.handle)

    def set_option(self, name, value):
        """Forward a kernel-selection option to every direction's handle (after first use)."""
        for st in self._dirs:
            if st.handle:
                st.handle.set_option(name, value)
