"""The launch planner of the prefill product (no GPU needed): every row count of the accepted range gets items that the kernel can run and that cover the rows."""
import random

import pytest

from kyojin_mac_b200 import ops
from kyojin_mac_b200.layout import FMT_ID

EDGES = [1, 31, 32, 33, 96, 127, 128, 129, 255, 256, 257, 300, 4001, 393216, 393217, 1048575, 1048576, 1048577, 2000000, 10**8, 2**31 - 1]


def _rows(rng):
    return EDGES + [int(2 ** rng.uniform(0, 31)) for _ in range(40)]


@pytest.mark.parametrize("split", [1, 4])
@pytest.mark.parametrize("fmt", sorted(FMT_ID))
def test_plans_are_runnable(fmt, split):
    rng = random.Random(split)
    for m in _rows(rng):
        for n, k in ((1, 1024), (300, 2048), (16384, 1024), (int(2 ** rng.uniform(0, 17)), 1024 * rng.randint(1, 20))):
            p = ops.gemm_kq_plan(fmt, n, k, m, split)
            where = (fmt, n, k, m, split, p)
            assert p["rows"] % 32 == 0 and 32 <= p["rows"] <= 256, where                     # TMA boxes of up to 256 rows, MMAs of up to 256 columns
            assert p["rows"] - 32 < m, where                                                 # no item wider than the rows need
            tiles = (n + (255 if p["pair"] else 127)) // (256 if p["pair"] else 128)
            assert p["items"] == tiles * ((m + p["rows"] - 1) // p["rows"]) * split, where


@pytest.mark.parametrize("n,k,m", [(8192, 7168, 2048), (2048, 7168, 2048), (1536, 3072, 4096), (7168, 18432, 1024)])
def test_items_of_several_destinations_stay_narrow(n, k, m):
    """Up to 128 rows an item's epilogue (stores to all ranks) runs under the next item's MMAs; wider items would make the MMAs wait for the stores."""
    assert ops.gemm_kq_plan("q4_k", n, k, m)["rows"] > 128
    for destinations in (2, 4, 8):
        assert ops.gemm_kq_plan("q4_k", n, k, m, destinations=destinations)["rows"] <= 128


@pytest.mark.gpu
def test_more_than_a_million_rows():
    """2^20 + 33 rows (4097 items of 256 rows): the result is that of the same rows in a small product, bit for bit."""
    import torch
    from kyojin_mac_b200 import synth
    fmt, n, k, m = "q4_k", 16, 256, (1 << 20) + 33
    t16 = synth.t16_random_device(fmt, n, k, seed=8)
    x = torch.randn((m, k), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9)).to(torch.float16)
    y = ops.gemm_kq(fmt, t16, n, k, x)
    ops.check_device_status()
    for lo in (0, m // 2, m - 300):
        assert torch.equal(y[lo:lo + 300], ops.gemm_kq(fmt, t16, n, k, x[lo:lo + 300]))
