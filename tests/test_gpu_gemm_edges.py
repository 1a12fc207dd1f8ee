"""Edges of the prefill GEMM whose weights are decoded into tensor memory: row counts around the 32-row MMA granularity and the 128- / 256-row accumulators, outputs
around the 128-row decode block and the 16-byte output pieces, one and an odd number of 256-input blocks, more items than CTA pairs, expert segments of every kind.
Oracle: fp64 product of this library's fp32 decode. Bounds: the whole result within 1e-3 (2-norm); every element within 4e-3 |x| |w|: by Cauchy-Schwarz the error is at
most |x| |dw|, a K-quant weight s q - z carries at most three roundings of relative size 2^-11 on parts that together are at most about 2.5 |w| in the 2-norm for
these draws (3 * 2.5 * 2^-11 = 3.7e-3; their signs are random, so what is seen is far smaller), while a wrong element is off by |x| |w| / sqrt(k) > 2e-2 |x| |w|."""
import pytest
import torch

from kyojin_mac_b200 import foreign_kqgmm as KQ, ops, synth
from kyojin_mac_b200.foreign_linear import DevPack

pytestmark = pytest.mark.gpu


def _check(y, x, w):
    """y against x w^T, both operands float64."""
    want = x @ w.T
    d = (y.double() - want).abs()
    assert (d.norm() / want.norm()).item() <= 1e-3
    rel = d / (x.norm(dim=1, keepdim=True) * w.norm(dim=1))
    assert rel.max().item() <= 4e-3, (rel.max().item(), divmod(int(rel.argmax()), w.shape[0]))


@pytest.mark.parametrize("fmt,n,k,m", [("q4_k", 16, 256, 1), ("q4_k", 128, 256, 33), ("q6_k", 144, 768, 64), ("q3_k", 264, 512, 65), ("q5_k", 1040, 1280, 96), ("nvfp4", 384, 256, 127),
                                       ("q8_0", 512, 768, 128), ("q2_k", 272, 512, 129), ("iq4_xs", 256, 1024, 161), ("q4_k", 520, 2048, 257), ("q4_k", 20480, 256, 70),
                                       ("q6_k", 20736, 768, 300), ("q4_k", 33, 512, 100), ("q3_k", 1001, 768, 600)])
def test_rows_and_outputs_at_the_edges(fmt, n, k, m):
    t16 = synth.t16_random_device(fmt, n, k, seed=n + m)
    g = torch.Generator(device="cuda").manual_seed(k + m)
    x = torch.randn((m, k), device="cuda", generator=g).to(torch.float16)
    out = torch.full((m + 2, n + 24), 7.0, dtype=torch.float16, device="cuda")          # nothing outside the result is written
    y = ops.gemm_kq(fmt, t16, n, k, x, split=1)
    ops.gemm_kq(fmt, t16, n, k, x, split=1, out=out[1:m + 1, 8:n + 8])
    ops.check_device_status()
    _check(y, x.double(), ops.dequant(fmt, t16, n, k, torch.float32).double())
    assert torch.equal(out[1:m + 1, 8:n + 8], y)
    out[1:m + 1, 8:n + 8] = 7.0
    assert (out == 7.0).all()
    for msub in (1, 2):                                                                  # the one-CTA form gives the same bits
        assert torch.equal(ops.gemm_kq(fmt, t16, n, k, x, msub=msub), y)


@pytest.mark.parametrize("mt", [128, 256])
@pytest.mark.parametrize("rows", [(1, 0, 31, 33, 128), (129, 255, 256, 257, 0, 64), (300, 1, 512)])
def test_expert_segments(rows, mt):
    """Grouped products over segments of every kind (empty, shorter than an MMA step, one row more than a block, several items) equal the per-expert products."""
    fmt, n, k, E = "q4_k", 256, 768, len(rows)
    dev = DevPack.from_t16(fmt, synth.t16_random_device(fmt, E * n, k, seed=3), n, k, E)
    up = DevPack.from_t16(fmt, synth.t16_random_device(fmt, E * n, k, seed=4), n, k, E)
    ids = torch.cat([torch.full((r,), e, dtype=torch.int32) for e, r in enumerate(rows)]).cuda()
    S = ids.numel()
    g = torch.Generator(device="cuda").manual_seed(S)
    ids = ids[torch.randperm(S, device="cuda", generator=g)]
    x = (torch.randn((S, k), device="cuda", generator=g) * 0.3).to(torch.float16)
    order, tb, off = KQ.csort(ids, E, mt)
    xg = KQ.gather_perm(x, order, 1)
    y = KQ.gmm(dev, xg, tb, off, S, mt, orow=order)
    a, b = KQ.gmm(dev, xg, tb, off, S, mt), KQ.gmm(up, xg, tb, off, S, mt)
    h = ops.gemm_kq_grouped_glu(fmt, dev.t16, up.t16, n, k, E, xg, tb, off, mt=mt)
    ops.check_device_status()
    assert torch.equal(h, ops.silu_mul(a, b))
    for e, r in enumerate(rows):
        if r:
            sel = (ids == e).nonzero().flatten()
            _check(y[sel], x[sel].double(), dev.expert(e).dequant(torch.float32).double())
    assert torch.equal(y[order.long()], a)
