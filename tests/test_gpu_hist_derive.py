"""GPU test of the parameter derivation from histograms (qgru_calc_params_from_hist: the SQNR search and the
percentile scan run on the GPU) against the host function of one histogram, for histograms with one,
few and all bins occupied, odd bin counts, and counts above 2^24."""
import ctypes as C
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME

_cabi = importlib.import_module(PKG_NAME + "._cabi")
params_mod = importlib.import_module(PKG_NAME + ".params")
pytestmark = pytest.mark.gpu


def _host(counts, mn, mx, total, op, pot2, pct, percentile):
    out = _cabi.Op()
    C.memmove(C.byref(out), C.byref(op), C.sizeof(op))
    st = _cabi.lib().qgru_calibrate_from_histogram(counts.ctypes.data_as(C.POINTER(C.c_float)), counts.size, mn, mx, int(total),
                                                   int(pot2), int(pct), percentile, C.byref(out))
    assert st == 0
    return out.scale, out.zero_point


@pytest.mark.parametrize("pct", [False, True])
@pytest.mark.parametrize("bins,occupied,gran", [(2048, 1, "PER_CHANNEL"), (2048, 97, "PER_CHANNEL"), (2048, 2048, "PER_GATE"),
                                                (2047, 300, "PER_TENSOR"), (33, 20, "PER_CHANNEL"), (1, 1, "PER_TENSOR")])
def test_derivation_equals_host(cuda_device, bins, occupied, gran, pct):
    H, rng = 5, np.random.default_rng(bins + occupied)
    cfg = params_mod.OperatorQuantConfig()
    cfg.bits["x"], cfg.bits["h"], cfg.unsigned["x"], cfg.symmetric["h"] = 4, 16, True, True
    for n in params_mod.WEIGHT_OPS:
        cfg.granularity[n] = params_mod.GRANULARITY[gran]
    hs = params_mod.Histograms(H, 0, num_bins=bins)
    data = {}
    for idx in range(hs.count()):
        counts = np.zeros(bins, np.float32)
        at = rng.choice(bins, min(occupied, bins), replace=False)
        counts[at] = rng.integers(1, 50, at.size) if idx % 3 else rng.integers(1, 60000, at.size)
        c = float(rng.normal(0, 0.2))
        w = float(abs(rng.normal(0, 1)) + 0.05)
        data[idx] = (counts, c - w, c + w, float(counts.sum(dtype=np.float64)))
        hs.put(idx, *data[idx])
    got = params_mod.GRUQuantParams.from_histograms(hs, cfg, pct, 99.0)
    want = _cabi.Params()
    cfg.fill(want)
    for i, name in enumerate(_cabi.OPS):
        if name not in params_mod.WEIGHT_OPS:
            assert (got.c.op[i].scale, got.c.op[i].zero_point) == _host(*data[i], want.op[i], False, pct, 99.0), name
    for k, name in enumerate(params_mod.WEIGHT_OPS):
        op = want.op[_cabi.OP_INDEX[name]]
        if gran == "PER_TENSOR":
            idx = [_cabi.OP_INDEX[name]] * (3 * H)
        elif gran == "PER_GATE":
            idx = [_cabi.HIST_GATE0 + 3 * k + c // H for c in range(3 * H)]
        else:
            idx = [_cabi.HIST_CHANNEL0 + k * 3 * H + c for c in range(3 * H)]
        for c in range(3 * H):
            assert float(got.scales[name][c]) == _host(*data[idx[c]], op, False, pct, 99.0)[0], (name, c)
