"""GPU tests of how a module reports a wait inside a kernel that ran out.  The failure is made as in test_gpu_forward.py: the
dp4a recurrence's group barrier with a limit of 2000 polls and one CTA that leaves out an arrival (host-set
options); the kernel returns, nothing faults or waits without a bound."""
import importlib

import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named

_cabi = importlib.import_module(PKG_NAME + "._cabi")
QuantGRU = importlib.import_module(PKG_NAME + ".quant_gru").QuantGRU
pytestmark = pytest.mark.gpu


def _module(dev):
    import torch
    torch.manual_seed(5)
    m = QuantGRU(24, 300, quant_storage_dtype="int32").to(dev).eval()
    m.load_bitwidth_config(config_named("default").to_json_dict())
    x = torch.randn(6, 9, 24, device=dev)
    m.calibrating = True
    m(x)
    m.calibrating = False
    m.finalize_calibration()
    return m, x


def _expire(m, x):
    """One forward whose wait runs out; the module's options are as before afterwards."""
    import torch
    for k, v in (("rec", "dp4a"), ("spin_limit", 2000), ("test_withhold_arrive", 1)):
        m.set_option(k, v)
    with torch.no_grad():
        m(x)
    torch.cuda.synchronize()
    assert "rec=dp4a" in m.last_plans()[0] and "P=3" in m.last_plans()[0]
    for k, v in (("rec", "fast"), ("spin_limit", 1 << 24), ("test_withhold_arrive", 0)):
        m.set_option(k, v)


def _raises():
    return pytest.raises(_cabi.QgruError, match="ran out")


@pytest.mark.parametrize("then", ["forward", "integer_forward", "reloaded_weights", "new_params", "synchronize", "train_forward"])
def test_first_call_after_the_expiry_raises_it_once(cuda_device, then):
    import torch
    m, x = _module(cuda_device)
    x_q = torch.randint(-100, 100, x.shape, device=cuda_device, dtype=torch.int32)
    with torch.no_grad():
        want, want_q = m(x), m.forward_quantized(x_q)
        _expire(m, x)
        if then == "reloaded_weights":
            m.weight_hh_l0.mul_(1.0)
        if then == "new_params":
            m.finalize_calibration()
        with _raises() as err:
            if then == "integer_forward":
                m.forward_quantized(x_q)
            elif then == "synchronize":
                m.synchronize()
            elif then == "train_forward":
                with torch.enable_grad():
                    m.train()(x)
            else:
                m(x)
        assert err.value.status == _cabi.QGRU_ERR_TIMEOUT
        m.eval()
        assert all(torch.equal(a, b) for a, b in zip(m(x), want))
        assert all(torch.equal(a, b) for a, b in zip(m.forward_quantized(x_q), want_q))
        m.synchronize()


def test_backward_raises_the_expiry(cuda_device):
    """An optimizer step must not run on what a forward in between has left: the backward asks too."""
    import torch
    m, x = _module(cuda_device)
    m(x)
    out, _ = m.train()(x)
    m.eval()
    _expire(m, x)
    with _raises():
        out.sum().backward()
    assert m.weight_hh_l0.grad is None
    out, _ = m.train()(x)
    out.sum().backward()
    assert bool(torch.isfinite(m.weight_hh_l0.grad).all())
