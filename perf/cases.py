"""The work whose speed this framework is judged by: quantized linears, gated MLPs and routed-expert layers over the sizes that decoding, batched decoding,
chunked prefill and prefill give them, each through the public call that a user's program makes.

A case is a dict of plain values; `prepare` builds the inputs and the modules from a seed, `run` is one pass, `exact` the same outputs in 64 bits from the stored GGUF
blocks by plain torch. Sizes are those of the benchmark configurations (hidden 5120 / MLP 27648, hidden 3072 / 12288, hidden 7168 / 18432 / expert width 2048) and
generic ones around them."""
import math

import torch

from kyojin_mac_b200 import foreign_linear as FL
from kyojin_mac_b200 import foreign_moe as FM
from kyojin_mac_b200 import moe_fused as MF
from kyojin_mac_b200 import ops

DEV = "cuda"
# inputs per stored block, bytes per stored block
BLOCK = {"q4_k": (256, 144), "q5_k": (256, 176), "q6_k": (256, 210), "q3_k": (256, 110), "q8_0": (32, 34), "nvfp4": (64, 36)}
FORMATS = ("q4_k", "q4_k", "q6_k", "q3_k", "q5_k", "q8_0", "nvfp4")        # drawn formats (the most used one twice)
GSCALE = 0.05                                                               # per-tensor scale of the NVFP4 matrices


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one attention projection of a small model, one token: latency
        dict(name="decode_proj_m1", kind="linear", fmt="q4_k", n=4096, k=4096, m=1),
        # the gated MLP of a 32B-class layer, one token: weight bandwidth (Q4_K gate | up, Q6_K down)
        dict(name="decode_mlp_m1", kind="mlp", fmt="q4_k", fmt_down="q6_k", h=5120, i=27648, m=1),
        # an output head with an odd vocabulary, a batch of decoding sequences
        dict(name="decode_head_m20", kind="linear", fmt="q6_k", n=32001, k=4096, m=20),
        # one projection for a batch of 96 decoding sequences (or a short prompt)
        dict(name="rows_q4k_m96", kind="linear", fmt="q4_k", n=13824, k=5120, m=96),
        # a chunk of a prompt through the down projection of a large MLP
        dict(name="chunk_q6k_m300", kind="linear", fmt="q6_k", n=5120, k=27648, m=300),
        # prefill of 2048 tokens through both projections of a small MLP
        dict(name="prefill_q3k_up", kind="linear", fmt="q3_k", n=12288, k=3072, m=2048),
        dict(name="prefill_q3k_down", kind="linear", fmt="q3_k", n=3072, k=12288, m=2048),
        # a long ragged prompt through a wide projection
        dict(name="prefill_q4k_ragged", kind="linear", fmt="q4_k", n=16384, k=7168, m=4001),
        # NVFP4 weights with activations quantised on the fly
        dict(name="prefill_nvfp4_a4", kind="a4", n=18432, k=7168, m=4096),
        # a routed-expert block (router, experts, combine) for 64 decoding sequences
        dict(name="moe_block_t64", kind="moe_block", fmt="q4_k", e=256, topk=8, h=7168, i=2048, t=64),
        # the routed experts of a 4096-token prefill, weighted sum included
        dict(name="moe_prefill_t4096", kind="moe", fmt="q4_k", e=256, topk=8, h=7168, i=2048, t=4096),
        # the router of that prefill: logits, shared-expert gate, top-k
        dict(name="router_t4096", kind="router", e=256, topk=8, h=7168, t=4096),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(("decode", "decode", "rows", "prefill", "prefill", "mlp", "a4", "moe_block", "moe", "router"))
    fmt = rng.choice(FORMATS)
    if kind == "decode":                                                     # 1 .. 32 rows, any number of outputs
        n, k = _log(rng, 512, 65536, rng.choice((1, 16, 256))), _log(rng, 1024, 28672, 256)
        return dict(kind="linear", fmt=fmt, n=n, k=k, m=_log(rng, 1, 32))
    if kind == "rows":                                                       # 33 .. 256 rows
        return dict(kind="linear", fmt=fmt, n=_log(rng, 1024, 32768, rng.choice((8, 128))), k=_log(rng, 1024, 28672, 256), m=_log(rng, 33, 256))
    if kind == "prefill":                                                    # longer chunks and whole prompts
        return dict(kind="linear", fmt=fmt, n=_log(rng, 2048, 16384, rng.choice((16, 256))), k=_log(rng, 2048, 14336, 256), m=_log(rng, 257, 4096))
    if kind == "mlp":
        return dict(kind="mlp", fmt=rng.choice(("q4_k", "q5_k", "nvfp4")), fmt_down=rng.choice(("q4_k", "q6_k", "q8_0")), h=_log(rng, 1024, 8192, 256), i=_log(rng, 2048, 28672, 256),
                    m=_log(rng, 1, 32))
    if kind == "a4":
        return dict(kind="a4", n=_log(rng, 2048, 18432, 256), k=_log(rng, 1024, 7168, 256), m=_log(rng, 33, 4096))
    e, h, i = rng.choice((32, 64, 128, 256)), _log(rng, 1024, 7168, 256), _log(rng, 512, 2048, 256)
    if kind == "moe_block":
        return dict(kind="moe_block", fmt=rng.choice(("q4_k", "q6_k", "q3_k")), e=e, topk=rng.choice((2, 4, 8)), h=h, i=i, t=_log(rng, 1, 96))
    if kind == "moe":
        return dict(kind="moe", fmt=rng.choice(("q4_k", "q6_k", "q3_k")), e=e, topk=rng.choice((4, 8)), h=h, i=i, t=_log(rng, 512, 4096))
    return dict(kind="router", e=e, topk=8, h=_log(rng, 1024, 7168, 64), t=_log(rng, 1, 4096))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _raw(fmt, n, k, g):
    """Stored GGUF rows uint8 [n, row_bytes]: random codes and block scales, super-block scales that give weights of about 0.02 with a mean near zero."""
    be, bb = BLOCK[fmt]
    b = torch.randint(0, 256, (n, k // be, bb), dtype=torch.uint8, device=DEV, generator=g)

    def put(off, v):
        b[..., off:off + 2] = v.to(torch.float16).contiguous().view(torch.uint8).reshape(n, k // be, 2)

    u = 0.5 + torch.rand((n, k // be), device=DEV, generator=g)
    if fmt == "q4_k":
        put(0, 1.4e-4 * u), put(2, 1.05e-3 * u)
    elif fmt == "q5_k":
        put(0, 7e-5 * u), put(2, 1.085e-3 * u)
    elif fmt == "q6_k":
        put(208, 6e-5 * u)
        b[..., 192:208] = torch.randint(-32, 32, (n, k // be, 16), dtype=torch.int8, device=DEV, generator=g).view(torch.uint8)
    elif fmt == "q3_k":
        put(108, 5e-4 * u)
    elif fmt == "q8_0":
        put(0, 2.8e-4 * u)
    else:                                                                    # NVFP4: e4m3 scales of 2^U[-8, 0]
        s = torch.exp2(-8.0 * torch.rand((n, k // be, 4), device=DEV, generator=g))
        b[..., 0:4] = s.to(torch.float8_e4m3fn).view(torch.uint8)
    return b.reshape(n, -1)


def _gscale(fmt):
    return GSCALE if fmt == "nvfp4" else 1.0


def _dev(fmt, n, k, g, experts=None):
    rows = n * (experts or 1)
    return FL.DevPack.from_t16(fmt, ops.raw_to_t16(fmt, _raw(fmt, rows, k, g), rows, k), n, k, experts, _gscale(fmt))


def _x(m, k, g, dtype=torch.float16):
    return torch.randn((m, k), device=DEV, generator=g).to(dtype)


class _MLP(torch.nn.Module):
    def __init__(self, gate, up, down):
        super().__init__()
        self.gate_proj, self.up_proj, self.down_proj = FL.ForeignLinear(gate), FL.ForeignLinear(up), FL.ForeignLinear(down)

    def forward(self, x):
        return self.down_proj(torch.nn.functional.silu(self.gate_proj(x)) * self.up_proj(x))


class _Layer(torch.nn.Module):
    """Holds the MLP as a model holds it, so that the installers can replace its parts."""

    def __init__(self, mlp):
        super().__init__()
        self.mlp = mlp

    def forward(self, x):
        return self.mlp(x)


def _ids(t, e, topk, g):
    """Routed experts and weights of t tokens: top-k of N(0, 1) logits, weights normalised to one."""
    p, ids = torch.softmax(torch.randn((t, e), device=DEV, generator=g), -1).topk(topk, -1)
    return ids.to(torch.int32), p / p.sum(-1, keepdim=True)


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "linear":
        lin = FL.ForeignLinear(_dev(case["fmt"], case["n"], case["k"], g))
        return dict(kind=kind, lin=lin, x=_x(case["m"], case["k"], g))
    if kind == "mlp":
        gate, up = _dev(case["fmt"], case["i"], case["h"], g), _dev(case["fmt"], case["i"], case["h"], g)
        layer, x = _Layer(_MLP(gate, up, _dev(case["fmt_down"], case["h"], case["i"], g))), _x(case["m"], case["h"], g)
        FL.group_same_input(layer, (x,), log=lambda s: None)
        FL.install_dense_glu(layer, log=lambda s: None)
        return dict(kind=kind, layer=layer, x=x)
    if kind == "a4":
        dev = _dev("nvfp4", case["n"], case["k"], g)
        x = _x(case["m"], case["k"], g, torch.bfloat16)
        dev.apply_a4(x[:1], torch.bfloat16)                                  # the code / scale arrays of the weights are laid out by the first call
        return dict(kind=kind, dev=dev, x=x)
    if kind == "router":
        gw = 0.02 * torch.randn((case["e"], case["h"]), device=DEV, generator=g)
        sgw = 0.02 * torch.randn((case["h"],), device=DEV, generator=g)
        return dict(kind=kind, gw=gw, sgw=sgw, x=_x(case["t"], case["h"], g), e=case["e"], topk=case["topk"])
    e, h, i = case["e"], case["h"], case["i"]
    glu = FL.ForeignSwitchGLU(_dev(case["fmt"], i, h, g, e), _dev(case["fmt"], i, h, g, e), _dev(case["fmt"], h, i, g, e))
    if kind == "moe_block":
        gw = 0.02 * torch.randn((e, h), device=DEV, generator=g)
        return dict(kind=kind, block=FM.RoutedBlock(gw, glu, case["topk"], True), x=_x(case["t"], h, g))
    x = _x(case["t"], h, g)
    ids, wts = _ids(case["t"], e, case["topk"], g)
    return dict(kind=kind, moe=MF.wrap(glu), x=x, ids=ids, wts=wts)


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"](state["x"])
    if kind == "mlp":
        return state["layer"](state["x"])
    if kind == "a4":
        return state["dev"].apply_a4(state["x"], torch.bfloat16)
    if kind == "router":
        lg = ops.router_logits(state["x"], state["gw"], state["sgw"])
        inds, scs, sgs = ops.moe_select(lg, state["e"], state["topk"], True, has_shared=True)
        return lg, inds, scs, sgs
    if kind == "moe_block":
        return state["block"](state["x"])
    return state["moe"](state["x"], state["ids"], state["wts"])


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _wbytes(fmt, n, k):
    be, bb = BLOCK[fmt]
    return n * (k // be) * bb


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": _wbytes(case["fmt"], n, k) + 2 * m * k + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "mlp":
        m, h, i = case["m"], case["h"], case["i"]
        return {"bytes": 2 * _wbytes(case["fmt"], i, h) + _wbytes(case["fmt_down"], h, i) + 4 * m * h, "flops": 6 * m * h * i}
    if kind == "a4":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": _wbytes("nvfp4", n, k) + 2 * m * k + 2 * m * n, "flops": 2 * m * n * k}
    t, e, h, topk = case["t"], case["e"], case["h"], case["topk"]
    if kind == "router":
        return {"bytes": 4 * (e + 1) * h + 2 * t * h + 4 * t * (e + 1) + 8 * t * topk + 4 * t, "flops": 2 * t * (e + 1) * h}
    i = case["i"]
    touched = e * (1.0 - (1.0 - topk / e) ** t)                              # experts that at least one of the tokens goes to, on average
    byt = int(touched * (2 * _wbytes(case["fmt"], i, h) + _wbytes(case["fmt"], h, i)))
    byt += 2 * t * h + (2 * t * h + 4 * e * h if kind == "moe_block" else 4 * t * h + 8 * t * topk)
    return {"bytes": byt, "flops": 6 * t * topk * h * i + (2 * t * e * h if kind == "moe_block" else 0)}


def tolerance(case):
    """About four times the error against `exact` that was measured for each kind of pass."""
    kind = case["kind"]
    if kind == "linear":                                                     # fp16 result (2e-4); from 64 rows on also fp16 weights (together 3.5e-4)
        return {"rel": 1.5e-3, "max": 1e-2}
    if kind == "mlp":                                                        # gate, up, the gated product and the result in fp16
        return {"rel": 2e-3, "max": 2e-2}
    if kind == "a4":                                                         # bf16 result (1.7e-3); the quantised activations are the same for every implementation
        return {"rel": 7e-3, "max": 3e-2}
    if kind == "router":                                                     # fp32 logits (tensor-core form 8e-6), near ties of the k-th expert
        return {"rel": 4e-5, "max": 1e-3, "differ": 1e-3}
    return {"rel": 3e-3, "max": 3e-2}                                        # four roundings to fp16 on the way through an expert


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _f16(b, off):
    return b[..., off:off + 2].contiguous().view(torch.float16).to(torch.float64)             # [n, nb, 1]


def _q45_scales(s):
    """12 bytes -> eight 6-bit scales and eight 6-bit minimums."""
    lo, mid, hi = s[..., 0:4], s[..., 4:8], s[..., 8:12]
    sc = torch.cat([lo & 63, (hi & 15) | ((lo >> 6) << 4)], -1)
    mn = torch.cat([mid & 63, (hi >> 4) | ((mid >> 6) << 4)], -1)
    return sc.double().unsqueeze(-1), mn.double().unsqueeze(-1)


def _decode(fmt, raw, k):
    """Stored GGUF rows -> float64 [n, k], without the per-tensor scale."""
    be, bb = BLOCK[fmt]
    n = raw.shape[0]
    b = raw.reshape(n, k // be, bb)
    if fmt in ("q4_k", "q5_k"):
        sc, mn = _q45_scales(b[..., 4:16])
        q = b[..., (16 if fmt == "q4_k" else 48):].reshape(n, -1, 4, 1, 32)
        code = torch.cat([q & 15, q >> 4], -2).reshape(n, -1, 8, 32)
        if fmt == "q5_k":
            bit = torch.arange(8, device=b.device, dtype=torch.uint8).reshape(8, 1)
            code = code | (((b[..., 16:48].unsqueeze(-2) >> bit) & 1) << 4)
        w = _f16(b, 0).unsqueeze(-1) * sc * code.double() - _f16(b, 2).unsqueeze(-1) * mn
    elif fmt == "q6_k":
        ql, qh = b[..., 0:128].reshape(n, -1, 2, 2, 32), b[..., 128:192].reshape(n, -1, 2, 1, 32)
        lo = torch.cat([ql & 15, ql >> 4], -2)                                                # [.., half, quarter, 32]
        sh = torch.arange(0, 8, 2, device=b.device, dtype=torch.uint8).reshape(4, 1)
        code = (lo | (((qh >> sh) & 3) << 4)).double() - 32.0
        sc = b[..., 192:208].contiguous().view(torch.int8).double().unsqueeze(-1)
        w = _f16(b, 208).unsqueeze(-1) * sc * code.reshape(n, -1, 16, 16)
    elif fmt == "q3_k":
        sh = torch.arange(0, 8, 2, device=b.device, dtype=torch.uint8).reshape(4, 1)
        lo = (b[..., 32:96].reshape(n, -1, 2, 1, 32) >> sh) & 3
        bit = torch.arange(8, device=b.device, dtype=torch.uint8).reshape(2, 4, 1)
        hb = (b[..., 0:32].reshape(n, -1, 1, 1, 32) >> bit) & 1
        code = (lo | (hb << 2)).double() - 4.0
        s = b[..., 96:108]
        low = torch.cat([s[..., 0:8] & 15, s[..., 0:8] >> 4], -1)
        high = (s[..., 8:12].unsqueeze(-2) >> sh) & 3
        sc = (low | (high.reshape(n, -1, 16) << 4)).double() - 32.0
        w = _f16(b, 108).unsqueeze(-1) * sc.unsqueeze(-1) * code.reshape(n, -1, 16, 16)
    elif fmt == "q8_0":
        w = _f16(b, 0) * b[..., 2:34].contiguous().view(torch.int8).double()
    else:
        grid = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device=b.device)
        grid = torch.cat([grid, -grid])
        q = b[..., 4:36].reshape(n, -1, 4, 8)
        code = torch.cat([q & 15, q >> 4], -1)                                                # byte j of a block of 16: inputs j and j + 8
        w = grid[code.long()] * b[..., 0:4].contiguous().view(torch.float8_e4m3fn).double().unsqueeze(-1)
    return w.reshape(n, k)


def _product(fmt, raw, k, x):
    """x (float64) times the transposed decoded matrix, a slice of rows at a time."""
    step = max(1, (1 << 26) // k)
    return torch.cat([x @ _decode(fmt, raw[i:i + step], k).T for i in range(0, raw.shape[0], step)], -1) * _gscale(fmt)


def _sat(y):
    return y.clamp(-65504.0, 65504.0)


def _silu_mul(a, b):
    return a / (1.0 + torch.exp(-a)) * b


def _quantised(x):
    """The NVFP4 rule for activations: blocks of 16, scale = e4m3 nearest to amax / 6 (at least 2^-9), values to the nearest e2m1 (ties to even)."""
    m, k = x.shape
    v = x.float().reshape(m, k // 16, 16)
    s = (v.abs().amax(-1).clamp_min(6.0 / 512.0) / 6.0).to(torch.float8_e4m3fn).float().unsqueeze(-1)
    q = (v / s).clamp(-6.0, 6.0)
    a = q.abs()
    code = sum((a > t).long() for t in (0.25, 1.25, 2.5, 5.0)) + sum((a >= t).long() for t in (0.75, 1.75, 3.5))
    grid = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device=x.device)
    return (torch.sign(q).double() * grid[code] * s.double()).reshape(m, k)


def _experts(case, raws, x, ids, wts):
    """Weighted sum over the routed experts, [t, h] float64."""
    h, i, fmt = case["h"], case["i"], case["fmt"]
    xd, out = x.double(), torch.zeros((case["t"], h), dtype=torch.float64, device=x.device)
    for e in range(case["e"]):
        tok, slot = (ids == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        wg, wu, wd = raws[0][e * i:(e + 1) * i], raws[1][e * i:(e + 1) * i], raws[2][e * h:(e + 1) * h]
        y = _product(fmt, wd, i, _silu_mul(_product(fmt, wg, h, xd[tok]), _product(fmt, wu, h, xd[tok])))
        out.index_add_(0, tok, _sat(y) * wts[tok, slot].double().unsqueeze(-1))
    return out


def exact(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "linear":
        raw = _raw(case["fmt"], case["n"], case["k"], g)
        return _sat(_product(case["fmt"], raw, case["k"], _x(case["m"], case["k"], g).double()))
    if kind == "mlp":
        h, i = case["h"], case["i"]
        rg, ru, rd = _raw(case["fmt"], i, h, g), _raw(case["fmt"], i, h, g), _raw(case["fmt_down"], h, i, g)
        x = _x(case["m"], h, g).double()
        return _sat(_product(case["fmt_down"], rd, i, _silu_mul(_product(case["fmt"], rg, h, x), _product(case["fmt"], ru, h, x))))
    if kind == "a4":
        raw = _raw("nvfp4", case["n"], case["k"], g)
        return _product("nvfp4", raw, case["k"], _quantised(_x(case["m"], case["k"], g, torch.bfloat16)))
    if kind == "router":
        gw = 0.02 * torch.randn((case["e"], case["h"]), device=DEV, generator=g)
        sgw = 0.02 * torch.randn((case["h"],), device=DEV, generator=g)
        lg = _x(case["t"], case["h"], g).double() @ torch.cat([gw, sgw[None]]).double().T
        top, inds = torch.softmax(lg[:, :case["e"]], -1).topk(case["topk"], -1)
        return lg, inds.to(torch.int32).reshape(-1), (top / top.sum(-1, keepdim=True)).reshape(-1), torch.sigmoid(lg[:, case["e"]])
    e, h, i = case["e"], case["h"], case["i"]
    raws = [_raw(case["fmt"], e * i, h, g), _raw(case["fmt"], e * i, h, g), _raw(case["fmt"], e * h, i, g)]
    if kind == "moe_block":
        gw = 0.02 * torch.randn((e, h), device=DEV, generator=g)
        x = _x(case["t"], h, g)
        top, ids = torch.softmax(x.double() @ gw.double().T, -1).topk(case["topk"], -1)
        return _sat(_experts(case, raws, x, ids, top / top.sum(-1, keepdim=True)))
    x = _x(case["t"], h, g)
    ids, wts = _ids(case["t"], e, case["topk"], g)
    return _experts(case, raws, x, ids, wts)
