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
