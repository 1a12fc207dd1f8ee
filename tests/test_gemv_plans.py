"""The launch planner of the decode product: every plan of the accepted range is one the kernel can run (no GPU needed), and products over shapes whose plans differ most
give the same bits as the exposed chunk sums, row for row whatever the number of rows (GPU)."""
import random

import pytest
import torch

from kyojin_mac_b200 import ops, synth
from kyojin_mac_b200.layout import FMT_ID, TILE_BYTES

KC_MAX, SMEM_MAX, SMS = 8, 226 * 1024, 148
MINS = {"q4_k": 256, "q5_k": 256, "q2_k": 512}          # staged sums per block and column tile


@pytest.mark.parametrize("fmt", sorted(FMT_ID))
def test_plans_are_runnable(fmt):
    rng = random.Random(FMT_ID[fmt])
    for _ in range(300):
        n, nb, m = int(2 ** rng.uniform(0, 17)), int(2 ** rng.uniform(0, 9)), rng.randint(1, 32)
        p = ops.gemv_plan(fmt, n, nb * 256, m)
        where = (fmt, n, nb * 256, m, p)
        assert 4 <= p["warps"] <= 12 and p["warps"] * 32 <= (512 if p["nt"] <= 2 else 384 if p["nt"] == 3 or fmt not in ("q5_k", "q6_k", "q8_0") else 256) and p["smem"] <= SMEM_MAX, where
        assert 8 * p["nt"] >= m and 1 <= p["kc"] <= KC_MAX and p["grid"] <= SMS, where
        assert p["kbp"] * p["ksplit"] >= nb and p["kbp"] * (p["ksplit"] - 1) < nb and p["grid"] % p["ksplit"] == 0, where   # the parts cover k and none is empty
        assert p["kbp"] == nb or p["kbp"] % p["kc"] == 0, where                              # a part is whole chunks
        assert (ops.gemv_workspace_bytes(fmt, n, nb * 256, m) > 0) == (p["aligned"] == 0 or (p["aligned"] == 1 and p["ksplit"] > 1)), where


@pytest.mark.parametrize("fmt", sorted(FMT_ID))
def test_plans_without_a_workspace_are_runnable(fmt):
    """A caller without scratch gets a form without chunk sums in memory that the kernel can run, wherever such a form fits shared memory; nothing fits only where
    the staged activations of all of k do not."""
    rng = random.Random(100 + FMT_ID[fmt])
    served = 0
    for _ in range(300):
        n, nb, m = int(2 ** rng.uniform(0, 17)), int(2 ** rng.uniform(0, 8)), rng.randint(1, 32)
        p = ops.gemv_plan(fmt, n, nb * 256, m, 0)
        where = (fmt, n, nb * 256, m, p)
        two_launches = p["aligned"] == 0 or (p["aligned"] == 1 and p["ksplit"] > 1)
        if two_launches:                                                                     # refused by the product for want of a workspace
            staged = nb * (16 * p["nt"] * min(8, 1 << max(0, (m - 1).bit_length())) * 32 + MINS.get(fmt, 0) * p["nt"])
            assert staged + 4 * (2 * TILE_BYTES[fmt] + 1312) > SMEM_MAX, where               # rings, scale scratch and barriers of four warps
            continue
        served += 1
        assert p["ksplit"] == 1 and p["kbp"] == nb and p["smem"] <= SMEM_MAX and 4 <= p["warps"] <= 12 and p["grid"] <= SMS, where
    assert served >= 100


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,n,k", [("q6_k", 1577, 6912), ("q4_k", 609, 5120), ("q5_k", 4100, 8192), ("q3_k", 865, 5888), ("nvfp4", 2400, 1280), ("q8_0", 33, 13568),
                                     ("iq4_xs", 16, 1792), ("nvfp4", 320, 1792), ("q2_k", 5376, 512), ("q4_k", 38, 256)])
def test_rows_do_not_depend_on_the_plan(fmt, n, k):
    from kyojin_mac_b200 import mma_gemv
    from kyojin_mac_b200.foreign_linear import DevPack
    dev = DevPack.from_t16(fmt, synth.t16_random_device(fmt, n, k, seed=5), n, k)
    g = torch.Generator(device="cuda").manual_seed(6)
    x, x2 = ((torch.randn((32, k), device="cuda", generator=g) * 0.5).to(torch.float16) for _ in range(2))
    want = mma_gemv.finalize_rows(dev, mma_gemv.partial_mma(dev, x, 32), 32)
    gated = ops.gemv(fmt, dev.t16, n, k, ops.silu_mul(x, x2))
    ref = x.double() @ dev.dequant(torch.float32).double().T
    assert ((want.double() - ref).norm() / ref.norm()).item() <= 1e-3
    for m in (1, 2, 4, 7, 8, 9, 16, 17, 24, 25, 32):
        assert torch.equal(ops.gemv(fmt, dev.t16, n, k, x[:m]), want[:m]), (m, ops.gemv_plan(fmt, n, k, m))
        assert torch.equal(ops.gemv(fmt, dev.t16, n, k, x[:m], x2=x2[:m]), gated[:m]), (m, ops.gemv_plan(fmt, n, k, m))
    ops.check_device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,n,k,m", [("q4_k", 9216, 2560, 12), ("q4_k", 9216, 2560, 24)])
def test_products_without_a_workspace(fmt, n, k, m):
    """A shape whose best plan uses a workspace although another form serves it: a caller without one gets that form, the same bits."""
    from kyojin_mac_b200 import _lib
    assert ops.gemv_workspace_bytes(fmt, n, k, m) > 0 and ops.gemv_plan(fmt, n, k, m, 0)["aligned"] == 1
    t16 = synth.t16_random_device(fmt, n, k, seed=7)
    x = torch.randn((m, k), device="cuda").to(torch.float16)
    y = torch.empty((m, n), dtype=torch.float16, device="cuda")
    L = _lib.lib()
    rc = L.kyb_gemv_t16(ops._fmt(fmt), t16.data_ptr(), n, k, x.data_ptr(), m, x.stride(0), 1.0, y.data_ptr(), y.stride(0), None, 0, 0, ops._stream())
    assert rc == 0, L.kyb_last_error()
    assert torch.equal(y, ops.gemv(fmt, t16, n, k, x))
