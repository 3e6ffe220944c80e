"""GPU tests of what a training step keeps between forward and backward: it belongs to autograd, like the saved tensors of
any function - freed by the backward, kept on request, seen by hooks, one block per forward."""
import importlib

import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named

QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
pytestmark = pytest.mark.gpu
STORAGE = pytest.mark.parametrize("storage", ["float", "float32", "int32"])


def _module(storage, dev, I=40, H=96, batch_first=False):
    import torch
    torch.manual_seed(11)
    m = QuantGRU(I, H, bidirectional=True, batch_first=batch_first, quant_storage_dtype="float32" if storage == "float" else storage).to(dev)
    if storage != "float":
        m.load_bitwidth_config(config_named("cfg2").to_json_dict())
        m.use_quantization = True
        m.calibrating = True
        m(torch.randn(12, 8, I, device=dev) * 0.7)
        m.calibrating = False
        m.finalize_calibration()
    return m.train()


def _grads(m, out, hn, **kw):
    import torch
    return torch.autograd.grad(out.square().sum() + hn.sum(), list(m.parameters()), **kw)


@STORAGE
def test_the_backward_frees_what_was_kept(cuda_device, storage):
    import torch
    m = _module(storage, cuda_device)
    x = torch.randn(50, 64, 40, device=cuda_device)
    _grads(m, *m(x))
    torch.cuda.synchronize()
    kept = 2 * m._dirs[0].handle.train_saved_bytes(0 if storage == "float" else 1 if storage == "float32" else 2, 50, 64)
    before = torch.cuda.memory_allocated()
    out, hn = m(x)
    assert torch.cuda.memory_allocated() - before > kept
    _grads(m, out, hn)
    results = 4 * (out.numel() + hn.numel())
    assert torch.cuda.memory_allocated() - before < results + kept // 10          # out is still alive
    with pytest.raises(RuntimeError, match="second time"):
        _grads(m, out, hn)


@STORAGE
@pytest.mark.parametrize("batch_first", [False, True])
def test_kept_graphs_hooks_and_checkpoints_give_the_same(cuda_device, storage, batch_first):
    import torch
    from torch.utils.checkpoint import checkpoint
    m = _module(storage, cuda_device, batch_first=batch_first)
    x = torch.randn(21, 33, 40, device=cuda_device)
    want = _grads(m, *m(x))
    out, hn = m(x)
    first, second = _grads(m, out, hn, retain_graph=True), _grads(m, out, hn)
    with torch.autograd.graph.save_on_cpu(pin_memory=True):
        out, hn = m(x)
    hooked = _grads(m, out, hn)
    out, hn = checkpoint(m, x, use_reentrant=False)
    again = _grads(m, out, hn)
    for g in (first, second, hooked, again):
        assert all(torch.equal(a, b) for a, b in zip(g, want))


def test_a_hook_that_returns_something_else_is_an_error(cuda_device):
    import torch
    m = _module("float32", cuda_device)
    x = torch.randn(5, 3, 40, device=cuda_device)
    for unpack in (lambda t: t.cpu(), lambda t: t[:1], lambda t: t.float()):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            out, hn = m(x)
            loss = out.sum()
        with pytest.raises(RuntimeError, match="hook"):
            loss.backward()


@STORAGE
def test_a_hook_may_return_a_view_at_any_byte(cuda_device, storage):
    """Hooks that keep every tensor as bytes of one buffer: the block comes back off its alignment."""
    import torch
    m = _module(storage, cuda_device, H=132)
    x = torch.randn(9, 7, 40, device=cuda_device)
    want = _grads(m, *m(x))

    def pack(t):
        if t.dtype != torch.uint8:
            return t
        flat = torch.empty(t.numel() + 3, dtype=t.dtype, device=t.device)
        flat[3:].copy_(t.reshape(-1))
        return flat[3:].view(t.shape)
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        out, hn = m(x)
    assert all(torch.equal(a, b) for a, b in zip(_grads(m, out, hn), want))


@STORAGE
def test_two_live_forwards_and_parameters_changed_before_the_backward(cuda_device, storage):
    """Forwards of different sizes alive at once, backwards in either order, parameters stepped in place in between."""
    import torch
    m = _module(storage, cuda_device)
    xs = [torch.randn(30, 65, 40, device=cuda_device), torch.randn(17, 20, 40, device=cuda_device)]
    want = [_grads(m, *m(x)) for x in xs]
    state = {k: v.clone() for k, v in m.state_dict().items()}
    for order in ((0, 1), (1, 0)):
        m.load_state_dict(state)
        outs = [m(x) for x in xs]
        with torch.no_grad():
            for p in m.parameters():
                p.add_(0.25 * torch.randn_like(p))
        for i in order:
            assert all(torch.equal(a, b) for a, b in zip(_grads(m, *outs[i]), want[i]))
