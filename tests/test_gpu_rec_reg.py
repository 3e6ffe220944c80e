"""GPU tests of the recurrence with R in registers (option rec=reg, qgru_rec_reg.cu) against the oracle: every split of
K over warps and of the units over CTAs, ragged rows and units, both directions, all cells."""
import importlib

import numpy as np
import pytest

from __graft_entry__ import PKG_NAME
from tests.cases import config_named, make_case

gru_ops = importlib.import_module(PKG_NAME + ".gru_ops")
pytestmark = pytest.mark.gpu

# (T, B, H): one CTA with 64 .. 256 inputs a warp (one row, full and ragged tiles of eight, several tiles), K over two
# warps in clusters of 3 and 4, over four warps in clusters of 9 and 16
SHAPES = [(1, 1, 1), (4, 3, 64), (5, 300, 60), (3, 1500, 33), (6, 9, 130), (4, 19, 192), (5, 1, 255), (3, 1400, 256),
          (5, 2, 257), (6, 37, 321), (4, 70, 384), (5, 41, 512), (3, 300, 500), (4, 2, 513), (5, 5, 600), (3, 90, 1001), (4, 1, 1024)]


@pytest.mark.parametrize("T,B,H", SHAPES)
@pytest.mark.parametrize("cfg", ["default", "cfg2", "cfg3", "ih16", "unsigned_x"])
def test_reg_recurrence_equals_oracle(oracle, cuda_device, cfg, T, B, H):
    import torch
    I = 7
    case = make_case(T * 131 + H, T, B, I, H, oracle, config_named(cfg))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    want = oracle.forward_i32(T, B, I, H, case.wq, case.x_q, case.h0_q, case.params.c, case.params.scale_list())
    with gru_ops.Handle(I, H, device=cuda_device.index or 0) as hd:
        hd.set_params(case.params)
        hd.set_weights_i32(*[dev(a) for a in case.wq])
        x, xf = dev(case.x_q), dev(case.x)
        h0 = None if case.h0_q is None else dev(case.h0_q)
        f0 = None if case.h0 is None else dev(case.h0)
        base = [hd.forward_f32(xf, f0, reverse=True), hd.forward_fstorage(xf, f0), hd.forward_i32(x, h0, reverse=True)]
        hd.set_option("rec", "reg")
        assert np.array_equal(hd.forward_i32(x, h0).cpu().numpy(), want)
        assert "r_in=registers" in hd.describe_plan()
        for cell in ("auto", "generic"):
            hd.set_option("cell", cell)
            got = [hd.forward_f32(xf, f0, reverse=True), hd.forward_fstorage(xf, f0), hd.forward_i32(x, h0, reverse=True)]
            for a, b in zip(base, got):
                assert torch.equal(a, b), hd.describe_plan()


# one unit, ragged units, one and several 16-byte chunks per thread, every row count a CTA wave can end with
@pytest.mark.parametrize("T,B,H", [(1, 1, 1), (5, 3, 33), (4, 21, 100), (3, 300, 130), (4, 2, 256), (3, 2, 257)])
@pytest.mark.parametrize("cfg", ["wide16", "pot2_wide16", "unsigned_wide16"])
def test_wide_recurrence_equals_oracle(oracle, cuda_device, cfg, T, B, H):
    """States of up to 16 bits in one launch (option rec=fast; H > 256: step by step)."""
    import torch
    I = 9
    c = config_named("wide16")
    if cfg == "pot2_wide16":
        c.use_pot2 = True
    if cfg == "unsigned_wide16":
        c.unsigned["h"] = c.unsigned["x"] = True
        c.bits["h"] = 12
    case = make_case(T * 17 + H, T, B, I, H, oracle, c)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    want = oracle.forward_i32(T, B, I, H, case.wq, case.x_q, case.h0_q, case.params.c, case.params.scale_list())
    with gru_ops.Handle(I, H, device=cuda_device.index or 0) as hd:
        hd.set_params(case.params)
        hd.set_weights_i32(*[dev(a) for a in case.wq])
        x, h0 = dev(case.x_q), None if case.h0_q is None else dev(case.h0_q)
        xf, f0 = dev(case.x), None if case.h0 is None else dev(case.h0)
        base = [hd.forward_i32(x, h0, reverse=True), hd.forward_f32(xf, f0)]
        hd.set_option("rec", "fast")
        assert np.array_equal(hd.forward_i32(x, h0).cpu().numpy(), want)
        assert ("path=wide" in hd.describe_plan()) == (H <= 256)
        assert torch.equal(base[0], hd.forward_i32(x, h0, reverse=True)) and torch.equal(base[1], hd.forward_f32(xf, f0))


@pytest.mark.parametrize("H,P,rows", [(512, 4, 8), (384, 3, 8), (1024, 16, 16), (600, 10, 16)])
def test_fast_on_either_side_of_its_line(oracle, cuda_device, H, P, rows):
    """rec=fast takes clusters with R in registers up to so many rows a cluster (one tile of eight, two above H = 512) and
    tcgen05 beyond; sm_limit keeps the number of clusters, and so the rows, small."""
    import torch
    T, I = 5, 7
    with gru_ops.Handle(I, H, device=cuda_device.index or 0) as hd:
        hd.set_option("rec", "fast")
        hd.set_option("sm_limit", 2 * P)
        seen = set()
        for B in (rows - 1, rows, rows + 1, 2 * rows, 2 * rows + 1):
            case = make_case(B * 31 + H, T, B, I, H, oracle, config_named("cfg2"))
            hd.set_params(case.params)
            hd.set_weights_i32(*[torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device) for a in case.wq])
            want = oracle.forward_i32(T, B, I, H, case.wq, case.x_q, case.h0_q, case.params.c, case.params.scale_list())
            h0 = None if case.h0_q is None else torch.from_numpy(case.h0_q).to(cuda_device)
            got = hd.forward_i32(torch.from_numpy(case.x_q).to(cuda_device), h0)
            assert np.array_equal(got.cpu().numpy(), want), hd.describe_plan()
            plan = dict(w.split("=") for w in hd.describe_plan().split() if "=" in w)
            if plan["r_in"] == "registers":
                assert int(plan["Bt"]) <= rows
            seen.add((plan["r_in"] == "registers", int(plan.get("Bt", 0))))
        assert (True, rows) in seen and any(not reg for reg, _ in seen), seen


@pytest.mark.parametrize("H", [33, 64, 256])
@pytest.mark.parametrize("cfg", ["default", "cfg2", "ih16"])
def test_tiles_of_two_to_four_rows(oracle, cuda_device, cfg, H):
    """One CTA a row range: a tile of two to four rows puts each row in two columns of the product.  sm_limit makes the CTAs'
    rows 1 .. 5 and 12 (a last tile of four), the last CTA's fewer; inference and training cells of both storages."""
    import torch
    T, I = 4, 8
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)
    with gru_ops.Handle(I, H, device=cuda_device.index or 0) as hd:
        hd.set_option("sm_limit", 3)
        for B in (3, 5, 6, 8, 9, 11, 12, 13, 36):
            case = make_case(B * 31 + H, T, B, I, H, oracle, config_named(cfg), with_h0=True)
            hd.set_params(case.params)
            w, x, h0 = [dev(a) for a in (case.W, case.R, case.bw, case.br)], dev(case.x), dev(case.h0)
            hd.set_weights_f32(*w)
            want = oracle.forward_i32(T, B, I, H, case.wq, case.x_q, case.h0_q, case.params.c, case.params.scale_list())

            def run():
                out = [hd.forward_f32(x, h0, reverse=True), hd.forward_fstorage(x, h0)]
                for int_storage in (False, True):
                    h, v, x_q, masks = hd.forward_fstorage_train(*w, x, h0, int_storage=int_storage)
                    out += [h, v, x_q, *masks.values()]
                return out

            hd.set_option("rec", "generic")
            base = run()
            hd.set_option("rec", "reg")
            assert np.array_equal(hd.forward_i32(dev(case.x_q), dev(case.h0_q)).cpu().numpy(), want), B
            assert "r_in=registers" in hd.describe_plan()
            for a, b in zip(base, run()):
                assert torch.equal(a, b), (B, hd.describe_plan())
