"""GPU tests of calls on streams of the caller's own: torch's streams do not wait for the default stream, so whatever a
call needs has to be queued on the stream it comes on or be ordered with it."""
import importlib

import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named

QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
pytestmark = pytest.mark.gpu


def _module(I, H, storage, cfg="cfg2", bidir=True, train=True, seed=0):
    import torch
    torch.manual_seed(seed)
    m = QuantGRU(I, H, bidirectional=bidir, quant_storage_dtype="float32" if storage == "float" else storage).to("cuda:0")
    m.use_quantization = storage != "float"
    if m.use_quantization:
        m.load_bitwidth_config(config_named(cfg).to_json_dict())
        m.use_quantization = True
        m.calibrating = True
        m(torch.randn(12, 8, I, device="cuda:0") * 0.7)
        m.calibrating = False
        m.finalize_calibration()
    return m.train(train)


def _step(m, x):
    import torch
    out, hn = m(x)
    return [out.detach(), hn.detach()] + list(torch.autograd.grad(out.sum() + hn.sum(), list(m.parameters())))


def test_size_query_queues_nothing(cuda_device):
    """qgru_train_saved_bytes has no stream: what it queued would not be ordered with the forward."""
    m = _module(12, 64, "float32")
    m._load_params(m._handle(0, cuda_device), 0)
    hd = m._dirs[0].handle
    before = hd.launch_count()
    assert hd.train_saved_bytes(1, 5, 3) > 0
    assert hd.launch_count() == before


@pytest.mark.parametrize("storage", ["float32", "int32", "float"])
def test_first_training_step_on_a_side_stream(cuda_device, storage):
    """New parameters, then the first step on a stream of the caller's while the default stream is busy."""
    import torch
    m = _module(40, 96, storage)
    x = torch.randn(20, 33, 40, device=cuda_device)
    want = _step(m, x)
    busy = torch.randn(4096, 4096, device=cuda_device)
    for _ in range(5):
        if m.use_quantization:
            m.finalize_calibration()
        torch.cuda.synchronize()
        for _ in range(8):
            busy = torch.tanh(busy @ busy)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            got = _step(m, x)
        side.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
        torch.cuda.synchronize()


def _on(stream, fn):
    import torch
    with torch.cuda.stream(stream):
        return fn()


def _infer(m, x, h0=None):
    import torch
    with torch.no_grad():
        return list(m(x, h0))


# the register-resident forms, clusters on tcgen05 with timestep chunks, 16-bit states (one launch; step by step)
@pytest.mark.parametrize("storage,cfg,T,H,bidir", [("int32", "cfg2", 60, 256, True), ("int32", "sym8_tensor", 300, 384, False),
                                                   ("float32", "default", 60, 320, True), ("int32", "wide16", 40, 100, True),
                                                   ("int32", "wide16", 20, 300, False), ("float", "", 60, 128, False)])
def test_inference_on_two_streams(cuda_device, storage, cfg, T, H, bidir):
    """Two inputs of different sizes, each on a stream of its own, without waiting in between: one workspace."""
    import torch
    m = _module(48, H, storage, cfg, bidir, train=False)
    D = 2 if bidir else 1
    xs = [torch.randn(T, 150, 48, device=cuda_device), torch.randn(T // 2 + 1, 70, 48, device=cuda_device)]
    hs = [None, torch.rand(D, 70, H, device=cuda_device) - 0.5]
    want = [_infer(m, x, h) for x, h in zip(xs, hs)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    got = [_on(streams[i & 1], lambda: _infer(m, xs[i & 1], hs[i & 1])) for i in range(12)]
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, want[i & 1])), i


@pytest.mark.parametrize("storage,H,bidir", [("float32", 128, True), ("int32", 256, False), ("float", 262, True), ("float32", 520, False)])
def test_training_on_two_streams(cuda_device, storage, H, bidir):
    """A step on one stream, a step of another size on the other, and inference with reloaded weights between them."""
    import torch
    m = _module(40, H, storage, "default", bidir)
    xs = [torch.randn(30, 65, 40, device=cuda_device), torch.randn(17, 20, 40, device=cuda_device)]
    want = [_step(m, x) for x in xs]
    want_i = _infer(m.eval(), xs[1])
    m.train()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    got = []
    for i in range(8):
        got.append((want[i & 1], _on(streams[i & 1], lambda: _step(m, xs[i & 1]))))
        if i == 3:
            got.append((want_i, _on(streams[0], lambda: _infer(m.eval(), xs[1]))))
            m.train()
    torch.cuda.synchronize()
    for k, (w, g) in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, w)), k


@pytest.mark.parametrize("method", ["sqnr", "percentile", "minmax"])
def test_calibration_on_two_streams(cuda_device, method):
    import torch
    torch.manual_seed(3)
    m = QuantGRU(64, 128, quant_storage_dtype="int32").to(cuda_device)
    m.load_bitwidth_config(config_named("default").to_json_dict())
    m.calibration_method, m.percentile_value = method, 99.9
    xs = [torch.randn(40 - 7 * i, 50, 64, device=cuda_device) * (1 + i) for i in range(4)]

    def run(streams):
        m.reset_calibration()
        m.calibrating = True
        torch.cuda.synchronize()
        outs = [_on(streams[i % len(streams)], lambda: m(xs[i])[0]) for i in range(4)]
        m.calibrating = False
        m.finalize_calibration()
        torch.cuda.synchronize()
        return outs, m.quant_params.to_bytes()
    want, want_p = run([torch.cuda.current_stream()])
    got, got_p = run([torch.cuda.Stream(), torch.cuda.Stream()])
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and got_p == want_p


def test_imported_counts_wait_for_what_had_the_memory_before(cuda_device):
    """A collector's counts live in torch's cached memory: on a side stream its last owner's kernels may still be writing it."""
    import numpy as np
    import torch
    Histograms = importlib.import_module(PKG_NAME + ".params").Histograms
    H, side = 64, torch.cuda.Stream()
    counts = np.arange(2048, dtype=np.float32)
    busy = torch.randn(4096, 4096, device=cuda_device)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        n = Histograms(H)._storage.numel()
        for _ in range(3):
            for _ in range(8):
                busy = torch.tanh(busy @ busy)
            junk = torch.empty(n, dtype=torch.uint8, device=cuda_device)
            at = junk.data_ptr()
            junk.fill_(7)
            del junk
            hs = Histograms(H)
            assert hs._storage.data_ptr() == at      # the very memory that the fill has not reached yet
            hs.put(5, counts, -1.0, 2.0, float(counts.sum(dtype=np.float64)))
            side.synchronize()
            assert np.array_equal(np.asarray(hs.get(5)[0]), counts)


def test_new_parameters_wait_for_what_is_in_flight(cuda_device):
    """Parameters and weights are replaced by host copies and by calls on another stream."""
    import torch
    m = _module(48, 256, "int32", "cfg2", True, train=False)
    ranges = m.quant_ranges
    x = torch.randn(120, 150, 48, device=cuda_device)
    want = _infer(m, x)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        torch.cuda.synchronize()
        got = _on(a, lambda: _infer(m, x))
        with torch.no_grad(), torch.cuda.stream(b):
            m.set_all_bitwidth(7)
            m.finalize_calibration()
            m(x[:3].contiguous())
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(got, want))
        m.load_state_dict(m.state_dict())
        m._bitwidth_config = type(m._bitwidth_config).from_json(config_named("cfg2").to_json_dict())
        m.quant_ranges = ranges
        m.finalize_calibration()


def test_captured_forward(cuda_device):
    """A forward captured into a graph after eager calls on other streams, replayed between more of them."""
    import torch
    m = _module(48, 256, "int32", "cfg2", True, train=False)
    x = torch.randn(20, 30, 48, device=cuda_device)
    x2 = torch.randn(20, 30, 48, device=cuda_device)
    want, want2 = _infer(m, x), _infer(m, x2)
    side = torch.cuda.Stream()
    _on(side, lambda: _infer(m, x2))
    torch.cuda.synchronize()
    graph, static = torch.cuda.CUDAGraph(), x.clone()
    with torch.cuda.graph(graph):
        out = _infer(m, static)
    for _ in range(2):
        assert all(torch.equal(p, q) for p, q in zip(_on(side, lambda: _infer(m, x2)), want2))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(out, want))
    assert m.last_timings()[0]["total_ms"] > 0
