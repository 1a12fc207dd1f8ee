// Prefill GEMM with the dequantisation fused into the operand producer: D[m, n] = sat_f16(gscale * sum_k A[m, k] * W[n, k]), W read as T16 tiles
// (every format of the library) and never written to HBM as fp16. Replaces the two-step large-row path of kyojin_mlx/foreign_linear.py:710 / :737
// (`x2 @ self.dequant().T`) and, in grouped form, the sorted grouped product of kyojin_mlx/foreign_kqgmm.py:225-239 (`gmm`).
//
// The weights are the M-side operand and live in tensor memory: the decoders' registers are already the 16 x 256-bit fragments that `tcgen05.st.16x256b` stores (a
// T16 row tile is 16 rows; lane (g, t) holds four consecutive inputs of rows g and g + 8 of every 16-input slice), so one store instruction per 16 rows x 64 inputs
// replaces eight swizzled shared-memory stores and their selects, and neither the decoded weights nor the MMA's reads of them touch shared memory. The activations
// are the N-side operand (TMA, 128-byte swizzle), so an item costs MMA time in proportion to its rows (N = rows rounded up to 16; 32 by pairs) instead of whole
// 128-row blocks, and the accumulator holds D transposed (lanes = outputs, columns = activation rows).
//
// One persistent CTA per SM, 22 warps:
//   warp 0      TMA: activation boxes (64 inputs of all the rows that the CTA needs for an item; grouped form: of 64 rows) into a ring of shared-memory stages
//   warp 1      tcgen05.mma issuer (M = 128 output rows, A from tensor memory, two accumulator slots of 128 columns), tcgen05.commit hands stages back
//   warps 2-5   epilogue: tcgen05.ld 16x256b, output scale, stmatrix.trans turns the fragments around into [activation row][output] staging tiles, which leave as
//               tiled bulk stores (two warps per store of 32 rows x 64 outputs) or as coalesced row pieces
//   warps 6-21  decoders: warp (q = warp % 4, j) owns row tile 2 q + (j & 1) of the CTA's 128 output rows (the tensor-memory lanes a warp may touch are those of its
//               quarter q) and every second T16 tile of it (parity j >> 1). It keeps one T16 tile in registers, each unit refilled from its next tile right after its
//               use (across items too), unpacks a 64-input quarter with LOP3 / PRMT into fp16 pairs, applies the block scales with half2 arithmetic (scale and
//               min rounded to fp16, then one fma per pair: the rounding points of the reference's few-row kernels, kyojin_mlx/foreign_metal.py:1357-1358,
//               :1382-1383) and stores it into half of one of four tensor-memory stages (64 columns each).
// PAIR (tcgen05 cta_group::2): two CTAs of neighbouring SMs compute 256 outputs; each decodes its own 128 rows into its own tensor memory and loads half of the
// activation rows, one MMA of the leader (cluster rank 0) drives both tensor cores. full barriers, acc_empty in the leader; empty and acc_full in each CTA
// (commit to the pair). Remote arrivals use the plain (CTA-scope release) form: what they publish sits in the arriving CTA's own tensor memory.
// Every mbarrier wait is bounded; a wait that gives up sets the device status word and the CTA drains.
//
// What bounds it: wide items (N = 256) the tensor core, their exposed epilogue and, in a long run of them, the power limit; narrow ones the decoders (330 clocks per 64
// inputs of 128 outputs for Q4_K, up to 555 for IQ4_XS, against 256 of MMA at 128 rows); few inputs the epilogue. Measured, the form with the decoded weights in shared
// memory -> now: Q4_K 13824 x 5120, 96 rows 50.6 -> 24.0 us; 8192 x 4096, 128 rows 40.8 -> 17.5; Q6_K 5120 x 27648, 300 rows 146 -> 114.7; Q3_K 12288 x 3072, 2048
// rows 156 -> 140, 3072 x 12288 169 -> 138; 256 experts of 2048 x 7168, 4096 tokens x 8, weighted sum included 5055 -> 3996 us. 8192 outputs of 512 or 1024 inputs and
// 4096 rows are 7 to 14 % slower than in that form. The sums are the same bits: the MMA adds the same products in the same order with its operands exchanged.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "t16_decode.cuh"
#include "tc_common.cuh"

namespace kyb {

constexpr int KQ_BN = 128, KQ_BK = 128, KQ_DW = 16, KQ_THREADS = (6 + KQ_DW) * 32;  // output rows per CTA, inputs per stage
constexpr int KQ_SA = 4;                                // weight stages in tensor memory: two T16 tiles, one per decoder parity
constexpr uint32_t KQ_COL_A = 256;                      // tensor memory: accumulator slots [0, 128) and [128, 256), weight stage s at 256 + 64 s
constexpr int KQ_TORD = 2048;                           // grouped form: tile order table in shared memory (u16 entries)
constexpr uint32_t KQ_SCR = 1280;                       // per decoder warp: block scales of one T16 tile as half2 pairs
constexpr uint32_t KQ_STG = 8192;                       // epilogue staging tile: 32 activation rows x 128 outputs as two 128-byte-swizzled halves; two of them
using KqOutMaps = KybOutMaps;                           // dense form: the [m, col0 + n] fp16 output matrix of every receiving rank

struct KqParams {
    const uint8_t* t16;
    __half* d[8];               // output matrix on every rank that receives the tiles (one entry without sharding), already offset to this rank's first column
    int nout;
    int64_t ldd;
    int m, n, k, nb;            // rows of A, rows of one W matrix, inputs, 256-input blocks
    int rt_total;               // 16-row tiles in the whole T16 buffer (row tiles past it are clamped; their outputs are never stored)
    float gscale;
    unsigned int* status;
    const uint32_t* tb;         // grouped form: first mt-row tile of every expert (E + 1 entries), else null
    const uint32_t* off;        // grouped form: first sorted row of every expert (E + 1 entries)
    const uint32_t* row_map;    // optional: output row of every sorted row
    const float* gs;            // optional: per-expert output scale
    int experts;
    int tiles_m, tiles_n;
    int mt;                     // activation rows per item (multiple of 32, at most 256)
    int bstages;                // shared-memory ring: 4 stages, or 2 of twice the size, of `bstage_bytes` (two halves of 64 inputs)
    uint32_t bstage_bytes;
    uint32_t box_rows;          // activation rows per TMA box (64 inputs wide)
    int tma_out, col0;          // dense form: the epilogue stores through the tensor maps (tiled bulk stores of 32 rows x 64 outputs), at column col0 + n0
    int vec_out;                // row stores: 16-byte pieces are aligned in every destination
    // split-k (dense form, one destination): the k-blocks are cut into ksplit equal ranges, an item is (tile, range) and writes its fp32 accumulator to
    // part [range][m][ldp] instead of d; gemm_kq_reduce_kernel adds the ranges in k order, scales, saturates and stores d
    int ksplit, mpad;           // mpad: rows of a range in part
    float* part;
    int64_t ldp;
    // gated pair (grouped form): an item's 128 weight rows are 64 rows of the gate stack (t16) and the same 64 rows of the up stack (t16b), 16-row tiles alternating,
    // so that one epilogue thread holds both products of an output; it writes fp16(silu(a) * b) of the two fp16-rounded products
    // (kyojin_mlx/foreign_kqgmm.py:293-314 `mlp`: gmm, gmm, silu_perm in one launch)
    const uint8_t* t16b;
    const float* gsb;           // per-expert output scale of the up stack (or null)
    int glu;
    float limit;                // > 0: a = min(a, limit), b = clamp(b, -limit, limit) as the activation kernel does
};

struct KqItem {
    int m0, m_end, n0;          // first activation row, end of the rows that may be stored, first output of this CTA
    int rt0;                    // T16 row tile of output n0
    int nn;                     // MMA width: the item's rows rounded up
    int tb0, ntb, sp;           // first 256-input block, number of blocks and index of the item's k-range (the whole of k without split-k)
    float gscale, gscale_b;
    bool valid;
};

template <bool PAIR>
__device__ __forceinline__ KqItem kq_item(const KqParams& p, int t, uint32_t rank, const uint16_t* tord = nullptr) {
    KqItem it;
    it.valid = true, it.gscale = p.gscale, it.gscale_b = p.gscale;
    it.tb0 = 0, it.ntb = p.nb, it.sp = 0;
    if (!p.tb) {
        if (p.ksplit > 1) {                                                             // tiles fastest, k-ranges slowest
            const int tiles = p.tiles_m * p.tiles_n;
            it.sp = t / tiles, t -= it.sp * tiles;
            it.ntb = p.nb / p.ksplit, it.tb0 = it.sp * it.ntb;
        }
        const int tn = t / p.tiles_m, tm = t - tn * p.tiles_m;                         // m fastest: CTAs running together share the weight rows
        it.n0 = (PAIR ? 2 * tn + (int)rank : tn) * KQ_BN;
        it.m0 = tm * p.mt, it.m_end = min(p.m, it.m0 + p.mt), it.rt0 = it.n0 >> 4;
        it.nn = PAIR ? (it.m_end - it.m0 + 31) & ~31 : (it.m_end - it.m0 + 15) & ~15;
        return it;
    }
    int tm = t / p.tiles_n;
    const int tn = t - tm * p.tiles_n;                                                   // n fastest: CTAs running together share the activation rows
    it.n0 = (PAIR ? 2 * tn + (int)rank : tn) * (p.glu ? KQ_BN / 2 : KQ_BN);
    if ((uint32_t)tm >= p.tb[p.experts]) {
        it.valid = false;
        return it;
    }
    if (tord) tm = (int)tord[tm];                                                        // wide tiles first (see the kernel's prologue)
    int lo = 0, hi = p.experts;                                                          // largest e with tb[e] <= tm (empty experts repeat a value)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (p.tb[mid] <= (uint32_t)tm) lo = mid; else hi = mid;
    }
    it.m0 = (int)(p.off[lo] + ((uint32_t)tm - p.tb[lo]) * (uint32_t)p.mt);
    it.m_end = min((int)p.off[lo + 1], it.m0 + p.mt);
    it.nn = PAIR ? (it.m_end - it.m0 + 31) & ~31 : (it.m_end - it.m0 + 15) & ~15;
    it.rt0 = (lo * p.n + it.n0) >> 4;
    if (p.gs) it.gscale = p.gs[lo];
    if (p.gsb) it.gscale_b = p.gsb[lo];
    return it;
}

// ------------------------------------------------------------------------------------------------ decoder: tile registers, scales, quarters
__device__ __forceinline__ uint4 ldg128s(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ldg64s(const uint8_t* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg32s(const uint8_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg16s(const uint8_t* p) {
    unsigned short v;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) { asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory"); }

__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) {
    __half2 r = __hsub2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    __half2 r = __hfma2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b), *reinterpret_cast<__half2*>(&c));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2_splat(float v) {
    __half2 r = __half2half2(sat_half(v));
    return *reinterpret_cast<uint32_t*>(&r);
}

// What one lane holds of a T16 tile: its 16-byte units of the code planes (the lane's MMA-fragment bytes, see kyojin_mac_b200/layout.py) and the scale bytes
// of row lane / 2 (half lane % 2) for the scale preparation.
template <int FMT>
struct KqTile {
    uint4 q[FMT == KYB_FMT_Q6_K ? 6 : FMT == KYB_FMT_Q3_K ? 3 : FMT == KYB_FMT_Q5_K ? 5 : FMT == KYB_FMT_Q8_0 ? 8 : FMT == KYB_FMT_Q2_K ? 2 : 4];
    uint4 sc;
    uint32_t d16;
};

template <int FMT>
__device__ __forceinline__ void kq_load(const uint8_t* tile, int lane, KqTile<FMT>& tr) {
    const int r = lane >> 1, hf = lane & 1;
    if constexpr (FMT == KYB_FMT_Q4_K) {
#pragma unroll
        for (int G = 0; G < 4; ++G) tr.q[G] = ldg128s(tile + (G * 32 + lane) * 16);
        tr.sc = ldg128s(tile + 2048 + r * 16);
        tr.d16 = 0;
    } else if constexpr (FMT == KYB_FMT_Q5_K) {
#pragma unroll
        for (int P = 0; P < 4; ++P) tr.q[P] = ldg128s(tile + (P * 32 + lane) * 16);
        tr.q[4] = ldg128s(tile + 2048 + lane * 16);                                           // the fifth bits of all four quarters
        tr.sc = ldg128s(tile + 2560 + r * 16);
        tr.d16 = 0;
    } else if constexpr (FMT == KYB_FMT_Q8_0) {
#pragma unroll
        for (int P = 0; P < 8; ++P) tr.q[P] = ldg128s(tile + (P * 32 + lane) * 16);
        tr.sc = ldg128s(tile + 4096 + r * 16);                                                // the row's eight fp16 d
        tr.d16 = 0;
    } else if constexpr (FMT == KYB_FMT_Q2_K) {
        tr.q[0] = ldg128s(tile + lane * 16);
        tr.q[1] = ldg128s(tile + (32 + lane) * 16);
        tr.sc = ldg128s(tile + 1024 + r * 16);                                                // the row's 16 scale | min << 4 bytes
        tr.d16 = ldg32s(tile + 1280 + r * 4);                                                 // d | dmin << 16
    } else if constexpr (FMT == KYB_FMT_IQ4_XS) {
#pragma unroll
        for (int P = 0; P < 4; ++P) tr.q[P] = ldg128s(tile + (P * 32 + lane) * 16);
        const uint2 mw = ldg64s(tile + 2048 + r * 8);                                         // d | scales_h << 16, four scales_l bytes
        tr.sc = make_uint4(mw.x, mw.y, 0, 0);
        tr.d16 = 0;
    } else if constexpr (FMT == KYB_FMT_Q6_K) {
#pragma unroll
        for (int P = 0; P < 4; ++P) tr.q[P] = ldg128s(tile + (P * 32 + lane) * 16);
        tr.q[4] = ldg128s(tile + 2048 + lane * 16);
        tr.q[5] = ldg128s(tile + 2048 + (32 + lane) * 16);
        const uint2 s = ldg64s(tile + 3072 + r * 16 + 8 * hf);
        tr.sc = make_uint4(s.x, s.y, 0, 0);
        tr.d16 = ldg16s(tile + 3328 + r * 2);
    } else if constexpr (FMT == KYB_FMT_Q3_K) {
        tr.q[0] = ldg128s(tile + lane * 16);
        tr.q[1] = ldg128s(tile + (32 + lane) * 16);
        tr.q[2] = ldg128s(tile + 1024 + lane * 16);
        const uint8_t* sp = tile + 1536 + r * 12;
        tr.sc = make_uint4(ldg32s(sp), ldg32s(sp + 4), ldg32s(sp + 8), 0);
        tr.d16 = ldg16s(tile + 1728 + r * 2);
    } else {
#pragma unroll
        for (int P = 0; P < 4; ++P) tr.q[P] = ldg128s(tile + (P * 32 + lane) * 16);
        const uint2 s = ldg64s(tile + 2048 + r * 16 + 8 * hf);
        tr.sc = make_uint4(s.x, s.y, 0, 0);
        tr.d16 = 0;
    }
}

// (lo, hi) fp16 pair -> the two (v, v) pairs, clamped to the finite fp16 range (an overflowing block scale must not turn into inf * 0)
__device__ __forceinline__ uint32_t h2_clamp(uint32_t a) {
    __half2 v = *reinterpret_cast<__half2*>(&a);
    const uint32_t hi_bits = 0x7BFF7BFFu, lo_bits = 0xFBFFFBFFu;
    v = __hmax2(__hmin2(v, *reinterpret_cast<const __half2*>(&hi_bits)), *reinterpret_cast<const __half2*>(&lo_bits));
    return *reinterpret_cast<uint32_t*>(&v);
}
// four byte codes c (unsigned, as (1024 + c) - bias in fp16, exact) times the fp16 pair d2 -> four (v, v) pairs; fp16(d * code) is the single rounding of the
// exact product, the same value as the float32 product rounded to fp16
__device__ __forceinline__ uint4 kq_scale4(uint32_t codes, uint32_t bias2, uint32_t d2) {
    const uint32_t a = h2_clamp(h2_mul(h2_sub(prmt(codes, 0x64646464u, 0x4140u), bias2), d2));
    const uint32_t b = h2_clamp(h2_mul(h2_sub(prmt(codes, 0x64646464u, 0x4342u), bias2), d2));
    return make_uint4(prmt(a, 0u, 0x1010u), prmt(a, 0u, 0x3232u), prmt(b, 0u, 0x1010u), prmt(b, 0u, 0x3232u));
}

// Block scales of the tile as half2 pairs (value, value) in the warp's scratch. Q4_K / Q5_K: (S, Z)[row][8] at row * 80 (scale and minus min of the eight
// 32-input sub-blocks, interleaved: one 16-byte read gives both of the two sub-blocks of a quarter); Q8_0 / IQ4_XS: S[row][8] at row * 48; the others: S[row][16]
// at row * 80 (one scale per 16 inputs). With the 80- and 48-byte pitches the reads of rows g = 0 .. 7 fall on distinct banks: a warp's read costs the minimum
// number of shared-memory wavefronts (a 32-byte pitch puts rows g and g + 4 on the same banks and doubles them).
template <int FMT>
__device__ __forceinline__ void kq_prep_scales(const KqTile<FMT>& tr, uint32_t scr, int lane) {
    const int r = lane >> 1, hf = lane & 1;
    if constexpr (FMT == KYB_FMT_Q2_K) {
        // one scale and one minimum per 16 inputs: word (fp16(d sc), fp16(-dmin mn)) per slice at row * 80 + 4 * slice (lane half hf covers slices 8 hf .. 8 hf + 7)
        const uint32_t d2 = prmt(tr.d16, 0u, 0x1010u), dm2 = prmt(tr.d16, 0u, 0x3232u) ^ 0x80008000u;
        const uint32_t w0 = hf ? tr.sc.z : tr.sc.x, w1 = hf ? tr.sc.w : tr.sc.y;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint32_t w = q ? w1 : w0;
            const uint32_t sl = w & 0x0F0F0F0Fu, ml = (w >> 4) & 0x0F0F0F0Fu;
            const uint32_t sa = h2_clamp(h2_mul(h2_sub(prmt(sl, 0x64646464u, 0x4140u), 0x64006400u), d2)), sb = h2_clamp(h2_mul(h2_sub(prmt(sl, 0x64646464u, 0x4342u), 0x64006400u), d2));
            const uint32_t za = h2_clamp(h2_mul(h2_sub(prmt(ml, 0x64646464u, 0x4140u), 0x64006400u), dm2)), zb = h2_clamp(h2_mul(h2_sub(prmt(ml, 0x64646464u, 0x4342u), 0x64006400u), dm2));
            sts128(scr + r * 80 + 32 * hf + 16 * q, make_uint4(prmt(sa, za, 0x5410u), prmt(sa, za, 0x7632u), prmt(sb, zb, 0x5410u), prmt(sb, zb, 0x7632u)));
        }
    } else if constexpr (FMT == KYB_FMT_IQ4_XS) {
        // 6-bit scales of sub-blocks 4 hf .. 4 hf + 3 (4 low bits from scales_l, 2 high bits from scales_h), minus 32, times d: S[row][8] as (v, v) pairs at row * 48
        const uint32_t sh = tr.sc.x >> (16 + 8 * hf), sl = tr.sc.y >> (16 * hf);
        const uint32_t lsw = ((sl & 15u) | ((sh & 3u) << 4)) | ((((sl >> 4) & 15u) | (((sh >> 2) & 3u) << 4)) << 8) | ((((sl >> 8) & 15u) | (((sh >> 4) & 3u) << 4)) << 16) |
                             ((((sl >> 12) & 15u) | (((sh >> 6) & 3u) << 4)) << 24);
        sts128(scr + r * 48 + 16 * hf, kq_scale4(lsw, 0x64206420u, prmt(tr.sc.x, 0u, 0x1010u)));
    } else if constexpr (FMT == KYB_FMT_Q8_0) {
        // one fp16 d per 32 inputs: S[row][8] as (d, d) pairs at row * 48 (lane half hf covers blocks 4 hf .. 4 hf + 3)
        const uint32_t w0 = hf ? tr.sc.z : tr.sc.x, w1 = hf ? tr.sc.w : tr.sc.y;
        sts128(scr + r * 48 + 16 * hf, make_uint4(h2_clamp(prmt(w0, 0u, 0x1010u)), h2_clamp(prmt(w0, 0u, 0x3232u)), h2_clamp(prmt(w1, 0u, 0x1010u)), h2_clamp(prmt(w1, 0u, 0x3232u))));
    } else if constexpr (FMT == KYB_FMT_Q4_K || FMT == KYB_FMT_Q5_K) {
        const uint4 mt = tr.sc;
        const uint32_t scw = ((hf ? mt.w : mt.y) & (hf ? 0x0f0f0f0fu : 0x3f3f3f3fu)) | ((mt.y >> 2) & (hf ? 0x30303030u : 0u));
        const uint32_t mnw = ((hf ? mt.w >> 4 : mt.z) & (hf ? 0x0f0f0f0fu : 0x3f3f3f3fu)) | ((mt.z >> 2) & (hf ? 0x30303030u : 0u));
        const uint32_t d2 = prmt(mt.x, 0u, 0x1010u), dm2 = prmt(mt.x, 0u, 0x3232u) ^ 0x80008000u;           // (d, d) and (-dmin, -dmin)
        const uint4 sv = kq_scale4(scw, 0x64006400u, d2), zv = kq_scale4(mnw, 0x64006400u, dm2);
        sts128(scr + r * 80 + 32 * hf, make_uint4(sv.x, zv.x, sv.y, zv.y));
        sts128(scr + r * 80 + 32 * hf + 16, make_uint4(sv.z, zv.z, sv.w, zv.w));
    } else if constexpr (FMT == KYB_FMT_Q6_K) {
        const uint32_t d2 = prmt(tr.d16, 0u, 0x1010u);
        // int8 scale + 128 as an unsigned byte, bias 1024 + 128
        sts128(scr + r * 80 + 32 * hf, kq_scale4(tr.sc.x ^ 0x80808080u, 0x64806480u, d2));
        sts128(scr + r * 80 + 32 * hf + 16, kq_scale4(tr.sc.y ^ 0x80808080u, 0x64806480u, d2));
    } else if constexpr (FMT == KYB_FMT_Q3_K) {
        const uint32_t w0 = tr.sc.x, w1 = tr.sc.y, w2 = tr.sc.z;
        const uint32_t ga = hf ? (((w0 >> 4) & 0x0f0f0f0fu) | (w2 & 0x30303030u)) : ((w0 & 0x0f0f0f0fu) | ((w2 << 4) & 0x30303030u));
        const uint32_t gb = hf ? (((w1 >> 4) & 0x0f0f0f0fu) | ((w2 >> 2) & 0x30303030u)) : ((w1 & 0x0f0f0f0fu) | ((w2 << 2) & 0x30303030u));
        const uint32_t d2 = prmt(tr.d16, 0u, 0x1010u);
        sts128(scr + r * 80 + 32 * hf, kq_scale4(ga, 0x64206420u, d2));                                     // 6-bit scale - 32
        sts128(scr + r * 80 + 32 * hf + 16, kq_scale4(gb, 0x64206420u, d2));
    } else {
        // e4m3 magnitude (7 bits) << 7 is the fp16 of value * 2^-8; code 0x7F decodes to 0
        auto four = [](uint32_t w) -> uint4 {
            w &= 0x7f7f7f7fu;
            const uint32_t is7f = ((w + 0x01010101u) & 0x80808080u) >> 7;                                    // 1 in every byte that is 0x7F
            w ^= is7f * 0x7fu;
            const uint32_t a = h2_mul(prmt(w, 0u, 0x4140u) << 7, 0x5C005C00u), b = h2_mul(prmt(w, 0u, 0x4342u) << 7, 0x5C005C00u);   // * 2^8, exact
            return make_uint4(prmt(a, 0u, 0x1010u), prmt(a, 0u, 0x3232u), prmt(b, 0u, 0x1010u), prmt(b, 0u, 0x3232u));
        };
        sts128(scr + r * 80 + 32 * hf, four(tr.sc.x));
        sts128(scr + r * 80 + 32 * hf + 16, four(tr.sc.y));
    }
}

// Quarter P (inputs [64 P, 64 P + 64)) of the tile: this lane's fp16 weights of rows g (h = 0) and g + 8 (h = 1), four consecutive inputs of every 16-input slice i
// as the two registers r[4 i + 2 h], r[4 i + 2 h + 1].
template <int FMT, int P>
__device__ __forceinline__ void kq_compute_quarter(const KqTile<FMT>& tr, uint32_t scr, int lane, uint32_t (&r)[16]) {
    const int g = lane >> 2;
    if constexpr (FMT == KYB_FMT_Q4_K) {
        const uint4 u = tr.q[P];
        const uint4 sg = lds128(scr + g * 80 + 16 * P), sh = lds128(scr + (g + 8) * 80 + 16 * P);   // (scale, minus min) of sub-blocks 2 P and 2 P + 1
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t w = h ? (c ? u.w : u.y) : (c ? u.z : u.x);
                const uint32_t s_lo = h ? sh.x : sg.x, s_hi = h ? sh.z : sg.z, z_lo = h ? sh.y : sg.y, z_hi = h ? sh.w : sg.w;
                const uint32_t p01 = prmt(w, 0u, 0x4140u), p23 = prmt(w, 0u, 0x4342u);       // bytes (b0, 0, b1, 0), (b2, 0, b3, 0)
                // low nibbles: 1024 + q, minus 1024; high nibbles: (1024 + 16 q) / 16 - 64; both exact
                const uint32_t l01 = h2_sub(and_or(p01, 0x000F000Fu, 0x64006400u), 0x64006400u), l23 = h2_sub(and_or(p23, 0x000F000Fu, 0x64006400u), 0x64006400u);
                const uint32_t h01 = h2_fma(and_or(p01, 0x00F000F0u, 0x64006400u), 0x2C002C00u, 0xD400D400u);
                const uint32_t h23 = h2_fma(and_or(p23, 0x00F000F0u, 0x64006400u), 0x2C002C00u, 0xD400D400u);
                r[4 * c + 2 * h] = h2_fma(l01, s_lo, z_lo), r[4 * c + 2 * h + 1] = h2_fma(l23, s_lo, z_lo);
                r[4 * (2 + c) + 2 * h] = h2_fma(h01, s_hi, z_hi), r[4 * (2 + c) + 2 * h + 1] = h2_fma(h23, s_hi, z_hi);
            }
        }
    } else if constexpr (FMT == KYB_FMT_Q5_K) {
        const uint4 u = tr.q[P], hb = tr.q[4];
        const uint4 sg = lds128(scr + g * 80 + 16 * P), sh = lds128(scr + (g + 8) * 80 + 16 * P);   // (scale, minus min) of sub-blocks 2 P and 2 P + 1
#pragma unroll
        for (int i = 0; i < 4; ++i) {                                                    // slice s = 4 P + i, sub-block 2 P + i / 2
            const int p = i >> 1, i8 = 4 * (P & 1) + i;                                      // fifth bit of slice s: bit s & 7 of word s >> 3
            uint32_t wg = p ? u.z : u.x, wh = p ? u.w : u.y;
            if (i & 1) wg >>= 4, wh >>= 4;
            uint32_t bg = (P & 2) ? hb.z : hb.x, bh = (P & 2) ? hb.w : hb.y;
            if (i8 < 4) bg <<= (4 - i8), bh <<= (4 - i8);
            else bg >>= (i8 - 4), bh >>= (i8 - 4);
            const uint32_t vg = and_or(wg, 0x0F0F0F0Fu, bg & 0x10101010u), vh = and_or(wh, 0x0F0F0F0Fu, bh & 0x10101010u);
            // bytes -> fp16 (1024 + v) - 1024 = v, exact; then one fma per pair with the fp16 scale and minus min of the sub-block
            const uint32_t sgi = p ? sg.z : sg.x, zgi = p ? sg.w : sg.y, shi = p ? sh.z : sh.x, zhi = p ? sh.w : sh.y;
            r[4 * i] = h2_fma(h2_sub(prmt(vg, 0x64646464u, 0x4140u), 0x64006400u), sgi, zgi);
            r[4 * i + 1] = h2_fma(h2_sub(prmt(vg, 0x64646464u, 0x4342u), 0x64006400u), sgi, zgi);
            r[4 * i + 2] = h2_fma(h2_sub(prmt(vh, 0x64646464u, 0x4140u), 0x64006400u), shi, zhi);
            r[4 * i + 3] = h2_fma(h2_sub(prmt(vh, 0x64646464u, 0x4342u), 0x64006400u), shi, zhi);
        }
    } else if constexpr (FMT == KYB_FMT_Q2_K) {
        const uint4 u = tr.q[P >> 1];
        const uint4 sg4 = lds128(scr + g * 80 + 16 * P), sh4 = lds128(scr + (g + 8) * 80 + 16 * P);
        const uint32_t sg[4] = {sg4.x, sg4.y, sg4.z, sg4.w}, sh[4] = {sh4.x, sh4.y, sh4.z, sh4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {                                                    // slice 4 P + i: codes at bits 2 i of word (P & 1)
            const uint32_t vg = (((P & 1) ? u.z : u.x) >> (2 * i)) & 0x03030303u, vh = (((P & 1) ? u.w : u.y) >> (2 * i)) & 0x03030303u;
            const uint32_t Sg = prmt(sg[i], 0u, 0x1010u), Zg = prmt(sg[i], 0u, 0x3232u), Sh = prmt(sh[i], 0u, 0x1010u), Zh = prmt(sh[i], 0u, 0x3232u);
            r[4 * i] = h2_fma(h2_sub(prmt(vg, 0x64646464u, 0x4140u), 0x64006400u), Sg, Zg);
            r[4 * i + 1] = h2_fma(h2_sub(prmt(vg, 0x64646464u, 0x4342u), 0x64006400u), Sg, Zg);
            r[4 * i + 2] = h2_fma(h2_sub(prmt(vh, 0x64646464u, 0x4140u), 0x64006400u), Sh, Zh);
            r[4 * i + 3] = h2_fma(h2_sub(prmt(vh, 0x64646464u, 0x4342u), 0x64006400u), Sh, Zh);
        }
    } else if constexpr (FMT == KYB_FMT_IQ4_XS) {
        const uint4 u = tr.q[P];
        const uint2 sg = lds64(scr + g * 48 + 8 * P), sh = lds64(scr + (g + 8) * 48 + 8 * P);
        auto grid4 = [](uint32_t idx) -> uint32_t {                                      // four 4-bit codes (one per byte) -> their grid values + 128
            const uint32_t x = idx & 0x07070707u, y = x | (x >> 4);
            const uint32_t sel = prmt(y, 0u, 0x4420u);
            const uint32_t lo = prmt(0xBFAD9881u, 0xF6EADDCFu, sel), hi = prmt(0x26190D01u, 0x71594535u, sel);
            const uint32_t m = ((idx >> 3) & 0x01010101u) * 0xFFu;
            return ((lo & ~m) | (hi & m)) ^ 0x80808080u;
        };
#pragma unroll
        for (int i = 0; i < 4; ++i) {                                                    // slice 4 P + i, sub-block 2 P + i / 2
            const int p = i >> 1;
            uint32_t wg = p ? u.z : u.x, wh = p ? u.w : u.y;
            if (i & 1) wg >>= 4, wh >>= 4;
            const uint32_t vg = grid4(wg & 0x0F0F0F0Fu), vh = grid4(wh & 0x0F0F0F0Fu);
            const uint32_t sgi = p ? sg.y : sg.x, shi = p ? sh.y : sh.x;
            r[4 * i] = h2_mul(h2_sub(prmt(vg, 0x64646464u, 0x4140u), 0x64806480u), sgi);
            r[4 * i + 1] = h2_mul(h2_sub(prmt(vg, 0x64646464u, 0x4342u), 0x64806480u), sgi);
            r[4 * i + 2] = h2_mul(h2_sub(prmt(vh, 0x64646464u, 0x4140u), 0x64806480u), shi);
            r[4 * i + 3] = h2_mul(h2_sub(prmt(vh, 0x64646464u, 0x4342u), 0x64806480u), shi);
        }
    } else if constexpr (FMT == KYB_FMT_Q8_0) {
        const uint2 sg = lds64(scr + g * 48 + 8 * P), sh = lds64(scr + (g + 8) * 48 + 8 * P);
#pragma unroll
        for (int i = 0; i < 4; ++i) {                                                    // slice 4 P + i = half i & 1 of unit 2 P + i / 2 (one 32-input block)
            const uint4 u = tr.q[2 * P + (i >> 1)];
            const uint32_t vg = ((i & 1) ? u.z : u.x) ^ 0x80808080u, vh = ((i & 1) ? u.w : u.y) ^ 0x80808080u;   // int8 -> value + 128
            const uint32_t sgi = (i >> 1) ? sg.y : sg.x, shi = (i >> 1) ? sh.y : sh.x;
            // bytes -> fp16 (1024 + v + 128) - 1152 = v, exact
            r[4 * i] = h2_mul(h2_sub(prmt(vg, 0x64646464u, 0x4140u), 0x64806480u), sgi);
            r[4 * i + 1] = h2_mul(h2_sub(prmt(vg, 0x64646464u, 0x4342u), 0x64806480u), sgi);
            r[4 * i + 2] = h2_mul(h2_sub(prmt(vh, 0x64646464u, 0x4140u), 0x64806480u), shi);
            r[4 * i + 3] = h2_mul(h2_sub(prmt(vh, 0x64646464u, 0x4342u), 0x64806480u), shi);
        }
    } else {
        const uint4 sg4 = lds128(scr + g * 80 + 16 * P), sh4 = lds128(scr + (g + 8) * 80 + 16 * P);
        const uint32_t sg[4] = {sg4.x, sg4.y, sg4.z, sg4.w}, sh[4] = {sh4.x, sh4.y, sh4.z, sh4.w};
        uint4 u, hi = make_uint4(0, 0, 0, 0), hb = make_uint4(0, 0, 0, 0);
        if constexpr (FMT == KYB_FMT_Q6_K) {
            u = tr.q[P];
            hi = tr.q[4 + (P >> 1)];
        } else if constexpr (FMT == KYB_FMT_Q3_K) {
            u = tr.q[P >> 1];
            hb = tr.q[2];
        } else {
            u = tr.q[P];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int s = 4 * P + i;
            uint32_t g01, g23, h01, h23;                                                     // rows g / g + 8: weights (0, 1) and (2, 3) of the slice
            if constexpr (FMT == KYB_FMT_Q6_K) {
                const int p = i >> 1;
                uint32_t wg = p ? u.z : u.x, wh = p ? u.w : u.y;
                if (i & 1) wg >>= 4, wh >>= 4;
                uint32_t hg = (P & 1) ? hi.z : hi.x, hh = (P & 1) ? hi.w : hi.y;
                if (i == 0) hg <<= 4, hh <<= 4;
                else if (i == 1) hg <<= 2, hh <<= 2;
                else if (i == 3) hg >>= 2, hh >>= 2;
                const uint32_t vg = and_or(wg, 0x0F0F0F0Fu, hg & 0x30303030u), vh = and_or(wh, 0x0F0F0F0Fu, hh & 0x30303030u);
                // bytes -> fp16 (1024 + v) - 1056 = v - 32, exact
                g01 = h2_sub(prmt(vg, 0x64646464u, 0x4140u), 0x64206420u), g23 = h2_sub(prmt(vg, 0x64646464u, 0x4342u), 0x64206420u);
                h01 = h2_sub(prmt(vh, 0x64646464u, 0x4140u), 0x64206420u), h23 = h2_sub(prmt(vh, 0x64646464u, 0x4342u), 0x64206420u);
            } else if constexpr (FMT == KYB_FMT_Q3_K) {
                uint32_t wg = (P & 1) ? u.z : u.x, wh = (P & 1) ? u.w : u.y;
                wg >>= 2 * i, wh >>= 2 * i;
                uint32_t bg = (P & 2) ? hb.z : hb.x, bh = (P & 2) ? hb.w : hb.y;
                const int i8 = s & 7;                                                        // bit i8 -> bit 2
                if (i8 < 2) bg <<= (2 - i8), bh <<= (2 - i8);
                else bg >>= (i8 - 2), bh >>= (i8 - 2);
                const uint32_t vg = and_or(wg, 0x03030303u, bg & 0x04040404u), vh = and_or(wh, 0x03030303u, bh & 0x04040404u);
                // (1024 + v) - 1028 = v - 4
                g01 = h2_sub(prmt(vg, 0x64646464u, 0x4140u), 0x64046404u), g23 = h2_sub(prmt(vg, 0x64646464u, 0x4342u), 0x64046404u);
                h01 = h2_sub(prmt(vh, 0x64646464u, 0x4140u), 0x64046404u), h23 = h2_sub(prmt(vh, 0x64646464u, 0x4342u), 0x64046404u);
            } else {
                const int p = i >> 1;
                const uint32_t wg = p ? u.z : u.x, wh = p ? u.w : u.y;
                uint32_t eg, og, eh, oh;                                                     // (w0, w2) and (w1, w3) as fp16 bits of value * 2^-14
                if ((i & 1) == 0) {
                    eg = wg & 0x8E008E00u, eh = wh & 0x8E008E00u;
                    og = (wg << 3) & 0x8E008E00u, oh = (wh << 3) & 0x8E008E00u;
                } else {
                    eg = and_or(wg << 6, 0x0E000E00u, (wg << 2) & 0x80008000u), eh = and_or(wh << 6, 0x0E000E00u, (wh << 2) & 0x80008000u);
                    og = and_or(wg << 9, 0x0E000E00u, (wg << 1) & 0x80008000u), oh = and_or(wh << 9, 0x0E000E00u, (wh << 1) & 0x80008000u);
                }
                eg = h2_mul(eg, 0x74007400u), og = h2_mul(og, 0x74007400u), eh = h2_mul(eh, 0x74007400u), oh = h2_mul(oh, 0x74007400u);   // * 2^14: the e2m1 value, exact
                g01 = prmt(eg, og, 0x5410u), g23 = prmt(eg, og, 0x7632u);
                h01 = prmt(eh, oh, 0x5410u), h23 = prmt(eh, oh, 0x7632u);
            }
            r[4 * i] = h2_mul(g01, sg[i]), r[4 * i + 1] = h2_mul(g23, sg[i]);
            r[4 * i + 2] = h2_mul(h01, sh[i]), r[4 * i + 3] = h2_mul(h23, sh[i]);
        }
    }
}
// After quarter P of a tile has been computed, the registers it alone used are refilled from the next tile (in place: one register set, every unit is requested a
// whole tile ahead of its next use). Units shared by two quarters are refilled after the second one.
template <int FMT, int P>
__device__ __forceinline__ void kq_refill(const uint8_t* next, int lane, KqTile<FMT>& tr) {
    if constexpr (FMT == KYB_FMT_Q4_K || FMT == KYB_FMT_NVFP4 || FMT == KYB_FMT_IQ4_XS) {
        tr.q[P] = ldg128s(next + (P * 32 + lane) * 16);
    } else if constexpr (FMT == KYB_FMT_Q2_K) {
        if constexpr (P == 1) tr.q[0] = ldg128s(next + lane * 16);                           // 2-bit codes of quarters 0, 1
        if constexpr (P == 3) tr.q[1] = ldg128s(next + (32 + lane) * 16);
    } else if constexpr (FMT == KYB_FMT_Q5_K) {
        tr.q[P] = ldg128s(next + (P * 32 + lane) * 16);
        if constexpr (P == 1) {                                                              // fifth bits of quarters 0, 1
            const uint2 hb = ldg64s(next + 2048 + lane * 16);
            tr.q[4].x = hb.x, tr.q[4].y = hb.y;
        }
        if constexpr (P == 3) {
            const uint2 hb = ldg64s(next + 2048 + lane * 16 + 8);
            tr.q[4].z = hb.x, tr.q[4].w = hb.y;
        }
    } else if constexpr (FMT == KYB_FMT_Q8_0) {
        tr.q[2 * P] = ldg128s(next + (2 * P * 32 + lane) * 16);
        tr.q[2 * P + 1] = ldg128s(next + ((2 * P + 1) * 32 + lane) * 16);
    } else if constexpr (FMT == KYB_FMT_Q6_K) {
        tr.q[P] = ldg128s(next + (P * 32 + lane) * 16);
        if constexpr (P == 1) tr.q[4] = ldg128s(next + 2048 + lane * 16);                    // 2-bit planes of quarters 0, 1
        if constexpr (P == 3) tr.q[5] = ldg128s(next + 2048 + (32 + lane) * 16);             // ... of quarters 2, 3
    } else {
        if constexpr (P == 1) {
            tr.q[0] = ldg128s(next + lane * 16);                                             // 2-bit codes of quarters 0, 1 and their high bits
            const uint2 hb = ldg64s(next + 1024 + lane * 16);
            tr.q[2].x = hb.x, tr.q[2].y = hb.y;
        }
        if constexpr (P == 3) {
            tr.q[1] = ldg128s(next + (32 + lane) * 16);
            const uint2 hb = ldg64s(next + 1024 + lane * 16 + 8);
            tr.q[2].z = hb.x, tr.q[2].w = hb.y;
        }
    }
}

// The scale bytes of the next tile, requested once the scales of the current one have been prepared.
template <int FMT>
__device__ __forceinline__ void kq_refill_scales(const uint8_t* tile, int lane, KqTile<FMT>& tr) {
    const int r = lane >> 1, hf = lane & 1;
    if constexpr (FMT == KYB_FMT_Q4_K) {
        tr.sc = ldg128s(tile + 2048 + r * 16);
    } else if constexpr (FMT == KYB_FMT_Q5_K) {
        tr.sc = ldg128s(tile + 2560 + r * 16);
    } else if constexpr (FMT == KYB_FMT_Q8_0) {
        tr.sc = ldg128s(tile + 4096 + r * 16);
    } else if constexpr (FMT == KYB_FMT_Q2_K) {
        tr.sc = ldg128s(tile + 1024 + r * 16);
        tr.d16 = ldg32s(tile + 1280 + r * 4);
    } else if constexpr (FMT == KYB_FMT_IQ4_XS) {
        const uint2 mw = ldg64s(tile + 2048 + r * 8);
        tr.sc.x = mw.x, tr.sc.y = mw.y;
    } else if constexpr (FMT == KYB_FMT_Q6_K) {
        const uint2 s = ldg64s(tile + 3072 + r * 16 + 8 * hf);
        tr.sc.x = s.x, tr.sc.y = s.y;
        tr.d16 = ldg16s(tile + 3328 + r * 2);
    } else if constexpr (FMT == KYB_FMT_Q3_K) {
        const uint8_t* sp = tile + 1536 + r * 12;
        tr.sc.x = ldg32s(sp), tr.sc.y = ldg32s(sp + 4), tr.sc.z = ldg32s(sp + 8);
        tr.d16 = ldg16s(tile + 1728 + r * 2);
    } else {
        const uint2 s = ldg64s(tile + 2048 + r * 16 + 8 * hf);
        tr.sc.x = s.x, tr.sc.y = s.y;
    }
}

// ------------------------------------------------------------------------------------------------ tensor-memory and matrix-transpose building blocks
// D[tmem] (+)= A[tmem] * B[smem]^T, issued by one thread
template <bool PAIR>
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
// 16 lanes x 32 columns: repeat i covers columns 8 i .. 8 i + 7; lane (g, t): registers 4 i, 4 i + 1 = row g, columns 2 t, 2 t + 1; 4 i + 2, 4 i + 3 = row g + 8
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
                   "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// four 8 x 8 matrices of 16-bit elements, transposed: lane l gives the address of the 16 bytes that receive column l & 7 of matrix l >> 3
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// A bounded wait of the whole warp whose answer is a vote. Every wait of this kernel is one: lanes poll on their own and may give up at different times, and behind
// each wait stand warp-wide instructions (tcgen05.ld / st, __syncwarp) that must not be met by a part of the warp.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_fast(bar, parity)) != 0; }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void half_barrier(int h) { asm volatile("bar.sync %0, 64;" ::"r"(2 + h) : "memory"); }   // the two epilogue warps of 64 outputs
__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }      // the four epilogue warps
__device__ __forceinline__ uint32_t pack_sat(uint32_t a, uint32_t b, float s) {
    __half2 h = sat_half2(__uint_as_float(a) * s, __uint_as_float(b) * s);
    return *reinterpret_cast<uint32_t*>(&h);
}

// The tiles of one decoder warp over all its items: every second T16 tile (parity kp of the CTA's running tile count) of one row tile.
template <int TB, bool PAIR>
struct KqWalk {
    const uint8_t* ptr;         // current tile
    int t, kb, ntb, base;       // item, block inside the item's range, blocks of the range, parity of the tiles before the item
    bool ok;

    __device__ __forceinline__ void enter(const KqParams& p, int num_items, int stride, uint32_t rank, const uint16_t* tord, int kp, int q, int half) {
        ok = false;
        for (; t < num_items; t += stride) {
            const KqItem it = kq_item<PAIR>(p, t, rank, tord);
            if (!it.valid) return;                                                     // grouped form: all items behind it are invalid too
            ntb = it.ntb, kb = kp ^ base;
            if (kb < ntb) {
                const int rt = min(it.rt0 + (p.glu ? q : 2 * q + half), p.rt_total - 1);
                ptr = ((p.glu && half) ? p.t16b : p.t16) + ((size_t)rt * (size_t)p.nb + (size_t)(it.tb0 + kb)) * TB;
                ok = true;
                return;
            }
            base ^= ntb & 1;
        }
    }
    __device__ __forceinline__ void advance(const KqParams& p, int num_items, int stride, uint32_t rank, const uint16_t* tord, int kp, int q, int half) {
        kb += 2;
        if (kb < ntb) {
            ptr += 2 * TB;
            return;
        }
        base ^= ntb & 1, t += stride;
        enter(p, num_items, stride, rank, tord, kp, q, half);
    }
};

template <int FMT, bool PAIR>
__global__ void __launch_bounds__(KQ_THREADS, 1) gemm_kq_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ KqOutMaps outs, const KqParams p,
                                                                 const int num_items) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int TB = kyb_tile_bytes(FMT);
    const uint32_t BS = (uint32_t)p.bstages;                                         // 4 or 2
    const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stg0 = smem0 + (uint32_t)BS * p.bstage_bytes;
    const uint32_t scr0 = stg0 + 2 * KQ_STG;
    const uint32_t bars = scr0 + KQ_DW * KQ_SCR;                                    // full[4], empty[4], acc_full[2], acc_empty[2], tmem slot
    const uint32_t full0 = bars, empty0 = bars + 32, accf0 = bars + 64, acce0 = bars + 80, tmem_slot = bars + 96;
    const uint32_t tord_a = bars + 112;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    const int first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, stride = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    constexpr uint32_t TMEM_COLS = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < KQ_SA; ++s) mbar_init_a(full0 + 8 * s, (PAIR ? 2 : 1) * KQ_DW / 2 + 1), mbar_init_a(empty0 + 8 * s, 1);
        for (int a = 0; a < 2; ++a) mbar_init_a(accf0 + 8 * a, 1), mbar_init_a(acce0 + 8 * a, PAIR ? 8 : 4);
        mbar_fence_init();
        prefetch_tmap(&tma_a);
    }
    if (warp == 1) {
        if constexpr (PAIR) tmem_alloc_pair(tmem_slot, TMEM_COLS);
        else tmem_alloc(tmem_slot, TMEM_COLS);
    }
    // Grouped form with items of up to 256 rows: a tile with more than 128 rows costs more than one with fewer, and items go to the CTAs round-robin, so the tiles
    // are renumbered with the wide ones first: every CTA then gets the same number of them (+-1) instead of a random share. Warp 2 builds the table (wide tiles from
    // the front, the others from the back) from the segment offsets; more tiles than the table holds keep their order.
    const uint16_t* tord = nullptr;
    if (p.tb && p.mt == 256) {
        const uint32_t total = p.tb[p.experts];
        if (total <= (uint32_t)KQ_TORD) {
            uint16_t* tw = reinterpret_cast<uint16_t*>(smem_raw + (tord_a - smem_u32(smem_raw)));
            tord = tw;
            if (warp == 2) {
                uint32_t front = 0, back = total;
                for (int e0 = 0; e0 < p.experts; e0 += 32) {
                    const int e = e0 + lane;
                    uint32_t two = 0, one = 0, first_tile = 0;
                    if (e < p.experts) {
                        const uint32_t rows = p.off[e + 1] - p.off[e], nt = (rows + 255u) >> 8;
                        first_tile = p.tb[e];
                        one = (nt && rows - 256u * (nt - 1u) <= 128u) ? 1u : 0u;
                        two = nt - one;
                    }
                    uint32_t a = two, b = one;                                          // inclusive warp scans
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t ua = __shfl_up_sync(0xffffffffu, a, d), ub = __shfl_up_sync(0xffffffffu, b, d);
                        if (lane >= d) a += ua, b += ub;
                    }
                    for (uint32_t i = 0; i < two; ++i) tw[front + a - two + i] = (uint16_t)(first_tile + i);
                    if (one) tw[back - b] = (uint16_t)(first_tile + two);
                    front += __shfl_sync(0xffffffffu, a, 31), back -= __shfl_sync(0xffffffffu, b, 31);
                }
            }
        }
    }
    tc_fence_before();
    if constexpr (PAIR) cluster_sync_all();                                         // both CTAs' barriers exist before either signals the other
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = lds32(tmem_slot);
    bool failed = false;

    if (warp == 0) {
        // ---- TMA producer: activation boxes. Stage i of the run uses barrier full[i % 4] (with the decoders of that stage) and shared-memory stage i % BS, which is free
        // once the MMAs of stage i - BS are done. By pairs each CTA loads its half of the item's rows and all bytes complete on the leader's barrier.
        // This loop and the MMA issuer's are executed by the whole warp, their conditions are warp votes and one elected lane issues, so that addresses and
        // descriptors stay in uniform registers (inside the elected lane's branch every operand of every MMA went through vector registers: 75 clocks per MMA). A
        // stage is 128 inputs because the instructions around a stage (waits, expect_tx, commit: 200-250 clocks in either warp) are paid per stage.
        const bool lead = elect_one();
        const uint32_t fullr0 = PAIR ? map_to_rank(full0, 0) : full0;
        uint32_t i = 0;
        bool ok = true;
        for (int t = first; t < num_items && ok; t += stride) {
            const KqItem it = kq_item<PAIR>(p, t, rank, tord);
            if (!it.valid) break;
            const uint32_t rows = __reduce_max_sync(0xffffffffu, (uint32_t)it.nn) >> (PAIR ? 1 : 0), boxes = (rows + p.box_rows - 1u) / p.box_rows;
            const uint32_t end = i + 2u * __reduce_max_sync(0xffffffffu, (uint32_t)it.ntb), bytes = (PAIR ? 4u : 2u) * boxes * p.box_rows * 128u;
            const int y0 = __reduce_max_sync(0xffffffffu, it.m0) + (PAIR ? (int)(rank * rows) : 0);
            int x = __reduce_max_sync(0xffffffffu, it.tb0) * 256;
            for (; i < end && ok; ++i, x += KQ_BK) {
                if (i >= BS) ok = mbar_wait_warp(empty0 + 8 * ((i - BS) & 3u), ((i - BS) >> 2) & 1u);
                if (lead) {
                    const uint32_t dst = smem0 + (i & (BS - 1u)) * p.bstage_bytes, bar = fullr0 + 8 * (i & 3u);
                    if (rank == 0) mbar_expect_tx_a(full0 + 8 * (i & 3u), bytes);
                    for (uint32_t b = 0; b < boxes; ++b)
#pragma unroll
                        for (uint32_t h = 0; h < 2; ++h) {
                            const uint32_t d = dst + h * (p.bstage_bytes >> 1) + b * p.box_rows * 128u;
                            if constexpr (PAIR) tma_load_2d_pair(d, &tma_a, x + 64 * (int)h, y0 + (int)(p.box_rows * b), bar);
                            else tma_load_2d(d, &tma_a, x + 64 * (int)h, y0 + (int)(p.box_rows * b), bar);
                        }
                }
                __syncwarp();
            }
        }
        failed = !ok;
    } else if (warp == 1) {
        // ---- MMA issuer (by pairs: the leader's)
        if (rank == 0) {
            const bool lead = elect_one();
            uint32_t i = 0, slot = 0, uses = 0;                                     // bit a of uses = parity of the uses of accumulator slot a
            const uint64_t desc0 = umma_desc_sw128(smem0);
            const uint32_t dstage = p.bstage_bytes >> 4, dhalf = p.bstage_bytes >> 5;
            bool ok = true;
            for (int t = first; t < num_items && ok; t += stride) {
                const KqItem it = kq_item<PAIR>(p, t, rank, tord);
                if (!it.valid) break;
                const uint32_t nn = __reduce_max_sync(0xffffffffu, (uint32_t)it.nn), end = i + 2u * __reduce_max_sync(0xffffffffu, (uint32_t)it.ntb);
                const uint32_t idesc = umma_idesc_f16(PAIR ? 256 : 128, (int)nn);
                if (nn > 128u) slot = 0;                                            // a wide item takes both slots
                const uint32_t tmem_d = tmem_base + slot * 128u, used = nn > 128u ? 3u : 1u << slot;
                // the epilogue must have drained an accumulator before the first MMA into it
                ok = mbar_wait_warp(acce0 + 8 * slot, ((uses >> slot) & 1u) ^ 1u);
                if (nn > 128u && ok) ok = mbar_wait_warp(acce0 + 8, ((uses >> 1) & 1u) ^ 1u);
                for (uint32_t acc = 0; i < end && ok; ++i, acc = 1) {
                    ok = mbar_wait_warp(full0 + 8 * (i & 3u), (i >> 2) & 1u);
                    tc_fence_after();
                    const uint32_t tmem_a = tmem_base + KQ_COL_A + 64u * (i & 3u);
                    const uint64_t bd = desc0 + (i & (BS - 1u)) * dstage;
                    if (lead) {
#pragma unroll
                        for (int kk = 0; kk < KQ_BK / 16; ++kk) umma_f16_ta<PAIR>(tmem_d, tmem_a + 8 * kk, bd + (kk >= 4 ? dhalf : 0u) + 2 * (kk & 3), idesc, kk ? 1u : acc);
                        if constexpr (PAIR) umma_commit_pair(empty0 + 8 * (i & 3u));    // the weight stage and the activation stage are free once these MMAs have read them
                        else umma_commit(empty0 + 8 * (i & 3u));
                    }
                    __syncwarp();
                }
                if (lead) {
                    for (uint32_t a = 0; a < 2; ++a)
                        if (used & (1u << a)) {
                            if constexpr (PAIR) umma_commit_pair(accf0 + 8 * a);
                            else umma_commit(accf0 + 8 * a);
                        }
                }
                __syncwarp();
                uses ^= used, slot ^= nn > 128u ? 0u : 1u;
            }
            failed = !ok;
        }
    } else if (warp < 6) {
        // ---- epilogue: warp w may touch TMEM lanes [32 (w % 4), 32 (w % 4) + 32) = outputs n0 + 32 q ..
        const int q = warp & 3;
        const bool issuer = elect_one() && (q & 1) == 0;                              // of the tiled stores of 64 outputs
        const uint32_t xq = __reduce_max_sync(0xffffffffu, 32u * (uint32_t)(q & 2));  // first of the 64 outputs that this warp's half tile holds
        const uint32_t acce = PAIR ? map_to_rank(acce0, 0) : acce0;
        const uint32_t tq = tmem_base + ((uint32_t)(q * 32) << 16);
        uint32_t next = 0, uses = 0, ch = 0;                                          // accumulator slots as the MMA issuer deals them; staged 32-row chunks so far
        for (int t = first; t < num_items; t += stride) {
            const KqItem it = kq_item<PAIR>(p, t, rank, tord);
            if (!it.valid) break;
            const int nsub = it.nn > 128 ? 2 : 1;
            for (int sub = 0; sub < nsub; ++sub) {
                const uint32_t slot = nsub == 2 ? (uint32_t)sub : next;
                if (!failed && !mbar_wait_warp(accf0 + 8 * slot, (uses >> slot) & 1u)) failed = true;
                uses ^= 1u << slot, next = slot ^ 1u;
                tc_fence_after();
                const int cols = min(it.nn - 128 * sub, 128);
                if (p.tma_out) {
                    // ---- dense form with tiled bulk stores: 32 rows x 64 outputs per store. The two warps of 64 outputs share a half tile and a store, so no warp
                    // waits for all four and two lanes issue the boxes; their operands are in uniform registers, the loop has no other form's branches.
                    int row0 = it.m0 + 128 * sub;
                    uint32_t ta = tq + slot * 128u;
                    const bool mine = !failed && it.n0 + (int)xq < p.n;
                    for (int left = cols; left > 0; left -= 32, ta += 32u, row0 += 32, ++ch) {
                        uint32_t va[16], vb[16];                                        // outputs 32 q + g, + 8 and 32 q + 16 + g, + 8, activation rows 8 i + 2 t, + 1
                        tmem_ld_16x256b_x4(ta, va);
                        tmem_ld_16x256b_x4(ta + (16u << 16), vb);
                        tmem_ld_wait();
                        if (left <= 32) {                                               // this warp has read its quarter of the accumulator
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                if constexpr (PAIR) mbar_arrive_remote(acce + 8 * slot);
                                else mbar_arrive_a(acce + 8 * slot);
                            }
                        }
                        const uint32_t stg = stg0 + (ch & 1u) * KQ_STG + 64u * xq;      // this half: 32 rows of 128 bytes
                        const uint32_t c16 = 4u * (q & 1) + (lane >> 3), dst = stg + ((c16 ^ (lane & 7)) << 4) + (lane & 7) * 128u;
#pragma unroll
                        for (int i = 0; i < 4; ++i)                                    // matrices: outputs 0-7, 8-15, 16-23, 24-31 of the warp, activation rows 8 i .. 8 i + 7
                            stmatrix_x4_trans(dst + 1024u * i, pack_sat(va[4 * i], va[4 * i + 1], it.gscale), pack_sat(va[4 * i + 2], va[4 * i + 3], it.gscale),
                                              pack_sat(vb[4 * i], vb[4 * i + 1], it.gscale), pack_sat(vb[4 * i + 2], vb[4 * i + 3], it.gscale));
                        fence_proxy_async_smem();
                        // the other staging tile is free for the next chunk once the store issued from it has read it: waited for before the barrier
                        if (issuer) tma_store_wait_read();
                        half_barrier(q >> 1);
                        if (issuer) {
                            if (mine && row0 < it.m_end) {
                                tma_store_2d(&outs.m[0], stg, p.col0 + it.n0 + (int)xq, row0);
                                for (int pr = 1; pr < p.nout; ++pr) tma_store_2d(&outs.m[pr], stg, p.col0 + it.n0 + (int)xq, row0);
                            }
                            tma_store_commit();
                        }
                    }
                    continue;
                }
                for (int c = 0; c < cols; c += 32) {
                    const int row0 = it.m0 + 128 * sub + c;
                    const bool last = c + 32 >= cols;
                    if (p.part) {
                        // ---- split-k: this range's accumulator as it is (fp32): every column is one activation row, a warp's 32 outputs are 128 contiguous bytes
                        uint32_t v[32];
                        tmem_ld_32x32(tq + slot * 128u + (uint32_t)c, v);
                        tmem_ld_wait();
                        if (last) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                if constexpr (PAIR) mbar_arrive_remote(acce + 8 * slot);
                                else mbar_arrive_a(acce + 8 * slot);
                            }
                        }
                        float* dst = p.part + ((size_t)it.sp * (size_t)p.mpad + (size_t)row0) * (size_t)p.ldp + it.n0 + 32 * q + lane;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (row0 + j < it.m_end && !failed) dst[(size_t)j * (size_t)p.ldp] = __uint_as_float(v[j]);
                        continue;
                    }
                    // rows of the staged chunk that this warp will store (row stores): 8 rows, 16 (gated pair: 8) lanes of 16 bytes each
                    uint32_t orow[4];
                    const int per = p.glu ? 4 : 2;                                      // rows per store instruction
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = row0 + 8 * q + per * i + (p.glu ? lane >> 3 : lane >> 4);
                        orow[i] = (uint32_t)row;
                        if (p.row_map && i < 8 / per && row < it.m_end) orow[i] = p.row_map[row];
                    }
                    uint32_t va[16], vb[16];                                            // outputs 32 q + g, + 8 and 32 q + 16 + g, + 8, activation rows 8 i + 2 t, + 1
                    tmem_ld_16x256b_x4(tq + slot * 128u + (uint32_t)c, va);
                    tmem_ld_16x256b_x4(tq + (16u << 16) + slot * 128u + (uint32_t)c, vb);
                    tmem_ld_wait();
                    if (last) {                                                         // this warp has read its quarter of the accumulator
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            if constexpr (PAIR) mbar_arrive_remote(acce + 8 * slot);
                            else mbar_arrive_a(acce + 8 * slot);
                        }
                    }
                    const uint32_t stg = stg0 + (ch & 1u) * KQ_STG;
                    if (p.glu) {
                        // va holds the gate products, vb the up products of the same 16 outputs; both are rounded to fp16 (what separate launches would have stored)
                        const float ga = it.gscale, gb = it.gscale_b, lim = p.limit;
                        uint32_t w[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            __half2 a2 = sat_half2(__uint_as_float(va[2 * i]) * ga, __uint_as_float(va[2 * i + 1]) * ga);
                            __half2 b2 = sat_half2(__uint_as_float(vb[2 * i]) * gb, __uint_as_float(vb[2 * i + 1]) * gb);
                            float a0 = __low2float(a2), a1 = __high2float(a2), b0 = __low2float(b2), b1 = __high2float(b2);
                            if (lim > 0.f) a0 = fminf(a0, lim), a1 = fminf(a1, lim), b0 = fminf(fmaxf(b0, -lim), lim), b1 = fminf(fmaxf(b1, -lim), lim);
                            __half2 h = sat_half2(a0 * (1.0f / (1.0f + expf(-a0))) * b0, a1 * (1.0f / (1.0f + expf(-a1))) * b1);
                            w[i] = *reinterpret_cast<uint32_t*>(&h);
                        }
#pragma unroll
                        for (int i = 0; i < 4; i += 2) {                               // matrices (i, outputs 0-7), (i, 8-15), (i + 1, 0-7), (i + 1, 8-15)
                            const uint32_t row = 8u * (i + (lane >> 4)) + (lane & 7), c16 = 2u * q + ((lane >> 3) & 1);
                            stmatrix_x4_trans(stg + row * 128u + ((c16 ^ (row & 7u)) << 4), w[2 * i], w[2 * i + 1], w[2 * i + 2], w[2 * i + 3]);
                        }
                    } else {
                        const float gscale = it.gscale;
                        const uint32_t c16 = 4u * (q & 1) + (lane >> 3), half_tile = stg + (uint32_t)(q >> 1) * 4096u + ((c16 ^ (lane & 7)) << 4) + (lane & 7) * 128u;
#pragma unroll
                        for (int i = 0; i < 4; ++i)                                    // matrices: outputs 0-7, 8-15, 16-23, 24-31 of the warp, activation rows 8 i .. 8 i + 7
                            stmatrix_x4_trans(half_tile + 1024u * i, pack_sat(va[4 * i], va[4 * i + 1], gscale), pack_sat(va[4 * i + 2], va[4 * i + 3], gscale),
                                              pack_sat(vb[4 * i], vb[4 * i + 1], gscale), pack_sat(vb[4 * i + 2], vb[4 * i + 3], gscale));
                    }
                    {
                        epilogue_barrier();
                        if (p.glu) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const uint32_t rr = 8u * q + 4u * i + (lane >> 3), c16 = lane & 7;
                                const uint4 o = lds128(stg + rr * 128u + ((c16 ^ (rr & 7u)) << 4));
                                if (row0 + (int)rr < it.m_end && !failed) *reinterpret_cast<uint4*>(p.d[0] + (size_t)orow[i] * p.ldd + it.n0 + 8 * c16) = o;
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t rr = 8u * q + 2u * i + (lane >> 4), c16 = lane & 15;
                                const uint4 o = lds128(stg + (c16 >> 3) * 4096u + rr * 128u + (((c16 & 7u) ^ (rr & 7u)) << 4));
                                const int col = it.n0 + 8 * (int)c16;
                                if (row0 + (int)rr < it.m_end && !failed) {
                                    if (p.vec_out && col + 8 <= p.n) {
                                        for (int pr = 0; pr < p.nout; ++pr) *reinterpret_cast<uint4*>(p.d[pr] + (size_t)orow[i] * p.ldd + col) = o;
                                    } else {
                                        const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
                                        for (int pr = 0; pr < p.nout; ++pr)
#pragma unroll
                                            for (int j = 0; j < 8; ++j)
                                                if (col + j < p.n) p.d[pr][(size_t)orow[i] * p.ldd + col + j] = __ushort_as_half((unsigned short)(ow[j >> 1] >> (16 * (j & 1))));
                                    }
                                }
                            }
                        }
                    }
                    ++ch;
                }
            }
        }
    } else {
        // ---- decoders
        const int dw = warp - 6, q = warp & 3, half = (dw >> 2) & 1, kp = dw >> 3;
        const uint32_t scr = scr0 + dw * KQ_SCR;
        const uint32_t tw = tmem_base + ((uint32_t)(32 * q + 16 * half) << 16) + KQ_COL_A + 128u * (uint32_t)kp;   // this warp's 16 lanes, stages 2 kp and 2 kp + 1
        const uint32_t full = (PAIR ? map_to_rank(full0, 0) : full0) + 16u * (uint32_t)kp, empty = empty0 + 16u * (uint32_t)kp;
        KqWalk<TB, PAIR> wk;
        wk.t = first, wk.base = 0;
        wk.enter(p, num_items, stride, rank, tord, kp, q, half);
        uint32_t parity = 1;                                                            // a fresh barrier passes a wait on the previous phase
        bool more = wk.ok;
        if (more) {
            // Software pipeline over the 64-input quarters: while the tensor-memory store of quarter P is on its way, the registers of quarter P + 1 are computed; the
            // wait for a free stage, the scale loads and the arithmetic overlap it.
            // The refills are unconditional (behind the last tile they read it once more, and what is computed from it is not stored): fewer branches and copies.
            KqTile<FMT> tr;
            uint32_t r[16];
            kq_load<FMT>(wk.ptr, lane, tr);
            kq_prep_scales<FMT>(tr, scr, lane);
            __syncwarp();
            wk.advance(p, num_items, stride, rank, tord, kp, q, half);
            kq_refill_scales<FMT>(wk.ptr, lane, tr);
            kq_compute_quarter<FMT, 0>(tr, scr, lane, r);
            kq_refill<FMT, 0>(wk.ptr, lane, tr);
#define KYB_KQ_WAIT(H)                                                               \
    {                                                                                \
        if (!mbar_wait_warp(empty + 8 * (H), parity)) failed = true;                 \
        tc_fence_after();                                                            \
    }
#define KYB_KQ_PUBLISH(H)                                                            \
    {                                                                                \
        tmem_st_wait();                                                              \
        tc_fence_before();                                                           \
        __syncwarp();                                                                \
        if (lane == 0) {                                                             \
            if constexpr (PAIR) mbar_arrive_remote(full + 8 * (H));                  \
            else mbar_arrive_a(full + 8 * (H));                                      \
        }                                                                            \
    }
            while (more && !failed) {
                more = wk.ok;                                                           // wk is one tile ahead
                KYB_KQ_WAIT(0)
                tmem_st_16x256b_x4(tw, r);
                kq_compute_quarter<FMT, 1>(tr, scr, lane, r);
                kq_refill<FMT, 1>(wk.ptr, lane, tr);
                tmem_st_16x256b_x4(tw + 32u, r);
                KYB_KQ_PUBLISH(0)
                kq_compute_quarter<FMT, 2>(tr, scr, lane, r);
                kq_refill<FMT, 2>(wk.ptr, lane, tr);
                KYB_KQ_WAIT(1)
                tmem_st_16x256b_x4(tw + 64u, r);
                kq_compute_quarter<FMT, 3>(tr, scr, lane, r);
                kq_refill<FMT, 3>(wk.ptr, lane, tr);
                tmem_st_16x256b_x4(tw + 96u, r);
                KYB_KQ_PUBLISH(1)                                                       // its warp barrier also ends every lane's reads of this tile's scales
                kq_prep_scales<FMT>(tr, scr, lane);                                     // tr.sc holds the next tile's scale bytes
                __syncwarp();
                kq_compute_quarter<FMT, 0>(tr, scr, lane, r);                           // quarter 0 of the next tile
                if (more) wk.advance(p, num_items, stride, rank, tord, kp, q, half);
                kq_refill_scales<FMT>(wk.ptr, lane, tr);
                kq_refill<FMT, 0>(wk.ptr, lane, tr);
                parity ^= 1u;
            }
#undef KYB_KQ_WAIT
#undef KYB_KQ_PUBLISH
        }
    }
    if ((warp == 2 || warp == 4) && p.tma_out) tma_store_wait_all();                      // the staging buffer must outlive its stores
    if (failed) atomicExch(p.status, KYB_DEV_TIMEOUT_GEMM);
    tc_fence_before();
    if constexpr (PAIR) cluster_sync_all();                                            // neither CTA frees tensor memory or leaves while the other may still signal it
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
        else tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// split-k, second step: d [m, n] = sat(gscale * (part[0] + part[1] + ... in k order)), eight columns per thread
__global__ void gemm_kq_reduce_kernel(const float* __restrict__ part, int ksplit, int m, int mpad, int n, int64_t ldp, float gscale, __half* __restrict__ d, int64_t ldd) {
    const int n8 = (n + 7) >> 3;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)m * n8) return;
    const int row = (int)(i / n8), c0 = (int)(i % n8) * 8;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int sp = 0; sp < ksplit; ++sp) {
        const float4* src = reinterpret_cast<const float4*>(part + ((size_t)sp * (size_t)mpad + (size_t)row) * (size_t)ldp + c0);
        const float4 a = src[0], b = src[1];                                            // ldp is a multiple of 256: always inside the row
        acc[0] += a.x, acc[1] += a.y, acc[2] += a.z, acc[3] += a.w, acc[4] += b.x, acc[5] += b.y, acc[6] += b.z, acc[7] += b.w;
    }
    __half* dst = d + (size_t)row * (size_t)ldd + c0;
    if (c0 + 8 <= n && (ldd & 7) == 0 && ((uintptr_t)d & 15) == 0) {
        __half2 h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = sat_half2(acc[2 * j] * gscale, acc[2 * j + 1] * gscale);
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(h);
    } else {
        for (int j = 0; j < 8 && c0 + j < n; ++j) dst[j] = sat_half(acc[j] * gscale);
    }
}

}  // namespace kyb

namespace {

template <bool PAIR>
const void* kq_kernel_ptr(int fmt) {
    switch (fmt) {
        case KYB_FMT_Q4_K: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_Q4_K, PAIR>;
        case KYB_FMT_Q6_K: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_Q6_K, PAIR>;
        case KYB_FMT_Q3_K: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_Q3_K, PAIR>;
        case KYB_FMT_Q5_K: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_Q5_K, PAIR>;
        case KYB_FMT_Q8_0: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_Q8_0, PAIR>;
        case KYB_FMT_Q2_K: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_Q2_K, PAIR>;
        case KYB_FMT_IQ4_XS: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_IQ4_XS, PAIR>;
        default: return (const void*)kyb::gemm_kq_kernel<KYB_FMT_NVFP4, PAIR>;
    }
}

constexpr size_t KQ_SMEM_CAP = 227 * 1024;
constexpr size_t KQ_RING = 128 * 1024;                  // activation ring
constexpr size_t KQ_SMEM_FIXED = 1024 + 2 * kyb::KQ_STG + (size_t)kyb::KQ_DW * kyb::KQ_SCR + 112 + 2 * kyb::KQ_TORD;

int kq_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        (void)cudaGetLastError();
        sms = v;
    }
    return sms;
}

// shared-memory attribute once per device, format and form; by pairs also how many CTA pairs the device holds at once (0: none, take the one-CTA form)
template <bool PAIR>
int kq_configure(int fmt, int* pairs) {
    static std::mutex mu;
    static unsigned done[KYB_FMT_COUNT] = {};
    static int pairs_max[KYB_FMT_COUNT][32] = {};
    int dev = 0;
    KYB_CUDA(cudaGetDevice(&dev));
    const void* kern = kq_kernel_ptr<PAIR>(fmt);
    std::lock_guard<std::mutex> lk(mu);
    if (!(done[fmt] & (1u << (dev & 31)))) {
        KYB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KQ_SMEM_CAP));
        if (PAIR) {
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t qc = {};
            qc.gridDim = dim3(2), qc.blockDim = dim3(kyb::KQ_THREADS), qc.dynamicSmemBytes = KQ_SMEM_FIXED + KQ_RING, qc.attrs = attr, qc.numAttrs = 1;
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, kern, &qc) != cudaSuccess || nc <= 0) {
                (void)cudaGetLastError();
                nc = 0;
            }
            pairs_max[fmt][dev & 31] = nc;
        }
        done[fmt] |= 1u << (dev & 31);
    }
    if (pairs) *pairs = pairs_max[fmt][dev & 31];
    return KYB_OK;
}

// units: CTAs (one-CTA form) or pairs that may run at once
template <bool PAIR>
int kq_launch(int fmt, const CUtensorMap& ta, const KybOutMaps& outs, kyb::KqParams p, int num_items, int units, cudaStream_t st) {
    if (int rc = kq_configure<PAIR>(fmt, nullptr)) return rc;
    // a stage of the activation ring is 128 inputs of up to 128 rows per CTA (the one-CTA form with wider items: 256)
    p.bstages = !PAIR && p.mt > 128 ? 2 : 4;
    p.bstage_bytes = (uint32_t)(KQ_RING / p.bstages);
    const size_t smem = KQ_SMEM_FIXED + KQ_RING;
    const int n = std::min(num_items, units);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(PAIR ? 2 * n : n)), cfg.blockDim = dim3(kyb::KQ_THREADS), cfg.dynamicSmemBytes = smem, cfg.stream = st, cfg.attrs = attr, cfg.numAttrs = PAIR ? 1 : 0;
    void* args[] = {(void*)&ta, (void*)&outs, (void*)&p, (void*)&num_items};
    KYB_CUDA(cudaLaunchKernelExC(&cfg, kq_kernel_ptr<PAIR>(fmt), args));
    return kyb_launch_check("gemm_kq");
}

// The form of a dense launch: CTA pairs or not, and activation rows per item (a multiple of 32, at most 256): what a cost model in clocks finds cheapest. An item is
// `stages` stages of 64 inputs, each as long as its MMAs (2 clocks per activation row by pairs; 2.6, above 128 rows 2.8, in the one-CTA form, which reads all of the
// activations through its own shared memory) but never less than the decode of its weights, and an epilogue of 760 clocks per 32 rows. Items of up to 128 rows
// alternate two accumulators: the epilogue of one runs under the next. Wider ones use both, their epilogue is exposed. Launching pairs costs 2900 clocks more.
// Fitted to 1900 timings (four formats, 2048 to 16384 outputs, 256 to 27648 inputs, 64 to 4001 rows, every form): the form it picks is on average 0.2 %, at most 5 %
// slower than the best one. Q4_K 8192 x 1024, 2048 rows: pairs of 256 rows 37.6 us, one CTA of 128 rows 32.9; 300 rows of 2048 x 512 9.2 / 6.8; 96 rows of
// 13824 x 5120 23.7 / 22.7. Items below 64 rows only where m has no more.
// The candidates are the item sizes, not the numbers of items, so any m has the same few of them.
// clocks that the decoders take for 64 inputs of 128 outputs (one CTA, 128 rows of 8192 x 4096, less the start and the epilogue)
constexpr double KQ_DEC_CLOCKS[KYB_FMT_COUNT] = {330.0, 400.0, 356.0, 381.0, 394.0, 345.0, 418.0, 555.0};
struct KqForm {
    bool pair;
    int mt;
    double clocks;
};
KqForm kq_choose(int fmt, int64_t n, int64_t m, int nb, int ksplit, int sms, int pairs, int widest = 256, double epi32 = 760.0) {
    const double stages = 4.0 * nb / ksplit, dec = KQ_DEC_CLOCKS[fmt];
    KqForm best{false, 0, 0.0};
    for (int pair = pairs > 0 ? 1 : 0; pair >= 0; --pair) {
        const int64_t tiles_n = (pair ? (n + 255) / 256 : (n + 127) / 128) * ksplit, units = pair ? pairs : sms;
        bool any = false;
        for (int mt = widest; mt >= 32; mt -= 32) {
            const int64_t tm = (m + mt - 1) / mt;
            if ((m + tm * 32 - 1) / (tm * 32) * 32 != mt) continue;                    // as many items of fewer rows cover m: that size is the candidate
            if (mt < 64 && any) break;
            any = true;
            const int64_t rounds = (tiles_n * tm + units - 1) / units;
            const double walk = stages * std::max(pair ? 1.02 * dec : dec, (pair ? 2.0 : mt > 128 ? 2.8 : 2.59) * mt), epi = epi32 * (mt / 32);
            const double clocks = (pair ? 10850.0 : 7920.0) + (mt > 128 ? (double)rounds * (walk + epi + 160.0) : (double)rounds * std::max(walk + 1417.0, epi + 144.0) + epi);
            if (!best.mt || clocks < best.clocks) best = {pair != 0, mt, clocks};
        }
    }
    return best;
}

// Several destinations: an item's stores to the other GPUs take longer than its MMAs (256 x 256 outputs to seven peers are 0.9 MB, 88 us of a pair's share of the link
// against 30 us of MMAs at 7168 inputs), so the items stay at 128 rows, whose epilogue runs under the next item's MMAs. Reasoned, not measured on several GPUs; with all
// destinations on one GPU the narrow items cost 0 to 10 %.
int kq_widest(int nout) { return nout > 1 ? 128 : 256; }

// CTA pairs the device holds at once; without a device half of the SMs
int kq_pairs(int fmt) {
    int pairs = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || kq_configure<true>(fmt, &pairs) != KYB_OK) pairs = kq_sms() / 2;
    (void)cudaGetLastError();
    return pairs;
}

}  // namespace

static int kq_dense(int fmt, const void* t16, int64_t n, int64_t k, const void* a, int64_t lda, int64_t m, float gscale, void* const* d, int nout, int64_t ldd,
                    int64_t col0, int msub, void* stream, int ksplit = 1, float* part = nullptr) {
    KYB_REQUIRE(fmt >= 0 && fmt < KYB_FMT_COUNT, "unknown weight format %d", fmt);
    KYB_REQUIRE(t16 && a, "null pointer");
    KYB_REQUIRE(m > 0 && n > 0 && k > 0 && k % 256 == 0, "m=%lld n=%lld k=%lld: k must be a positive multiple of 256", (long long)m, (long long)n, (long long)k);
    KYB_REQUIRE(lda >= k && lda % 8 == 0 && ldd >= n, "leading dimensions: lda >= k and a multiple of 8, ldd >= n");
    KYB_REQUIRE(((uintptr_t)a & 15) == 0 && ((uintptr_t)t16 & 15) == 0, "a and t16 must be 16-byte aligned");
    KYB_REQUIRE(m < (1ll << 31) && n < (1ll << 31) && k < (1ll << 24), "dimension too large");
    KYB_REQUIRE(msub >= 0 && msub <= 2, "msub is 0 (automatic), 1 or 2");
    unsigned int* status = kyb_device_status_word();
    KYB_REQUIRE(status, "could not set up the device status word");
    kyb::KqParams p;
    memset(&p, 0, sizeof(p));
    p.t16 = (const uint8_t*)t16, p.ldd = ldd, p.m = (int)m, p.n = (int)n, p.k = (int)k, p.nb = (int)(k / 256), p.rt_total = (int)((n + 15) / 16);
    p.nout = nout, p.gscale = gscale, p.status = status;
    for (int i = 0; i < nout; ++i) p.d[i] = (__half*)d[i] + col0;
    p.ksplit = ksplit, p.mpad = (int)m, p.part = ksplit > 1 ? part : nullptr, p.ldp = (n + 255) / 256 * 256;
    // a given msub asks for the one-CTA form with that many 128-row blocks per item
    int pairs = 0;
    const int sms = kq_sms();
    if (msub == 0)
        if (int rc = kq_configure<true>(fmt, &pairs)) return rc;
    const KqForm form = msub ? KqForm{false, 128 * msub, 0.0} : kq_choose(fmt, n, m, p.nb, ksplit, sms, pairs, kq_widest(nout));
    const bool pair = form.pair;
    p.mt = form.mt;
    CUtensorMap ta;                                                                 // one box is 64 inputs of all the rows that a CTA loads for an item
    p.box_rows = (uint32_t)(pair ? p.mt / 2 : p.mt);
    if (int rc = kyb_make_tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a, (uint64_t)m, (uint64_t)k, (uint64_t)lda * 2, p.box_rows, 64)) return rc;
    p.tiles_n = (int)(pair ? (n + 255) / 256 : (n + 127) / 128);
    p.tiles_m = (int)((m + p.mt - 1) / p.mt);
    // tiled bulk stores need 16-byte aligned bases and row pitches; otherwise the epilogue stores row pieces
    KybOutMaps outs;
    memset(&outs, 0, sizeof(outs));
    p.col0 = (int)col0;
    p.tma_out = (ldd % 8 == 0 && col0 % 8 == 0 && ksplit == 1) ? 1 : 0;
    for (int i = 0; i < nout && p.tma_out; ++i)
        if ((uintptr_t)d[i] & 15) p.tma_out = 0;
    for (int i = 0; i < nout && p.tma_out; ++i)
        if (int rc = kyb_make_tmap_2d(&outs.m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, d[i], (uint64_t)m, (uint64_t)(col0 + n), (uint64_t)ldd * 2, 32, 64)) return rc;
    KYB_REQUIRE((int64_t)p.tiles_n * p.tiles_m * ksplit < (1ll << 31), "m=%lld n=%lld: too many output tiles", (long long)m, (long long)n);
    const int items = p.tiles_n * p.tiles_m * ksplit;
    if (int rc = pair ? kq_launch<true>(fmt, ta, outs, p, items, pairs, (cudaStream_t)stream) : kq_launch<false>(fmt, ta, outs, p, items, sms, (cudaStream_t)stream)) return rc;
    if (ksplit == 1) return KYB_OK;
    const int64_t threads = m * ((n + 7) / 8);
    kyb::gemm_kq_reduce_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(part, ksplit, (int)m, p.mpad, (int)n, p.ldp, gscale, (__half*)d[0], ldd);
    return kyb_launch_check("gemm_kq_reduce");
}

// D fp16 [m, n] (row stride ldd) = sat(gscale * A fp16 [m, k] (row stride lda) x W^T), W = T16 tiles of an [n, k] matrix of format fmt. msub = 0: the library
// chooses (CTA pairs, or the one-CTA form where that fills the SMs better); 1 or 2: the one-CTA form with up to that many blocks of 128 activation rows per item.
// All forms give the same bits.
extern "C" int kyb_gemm_kq(int fmt, const void* t16, int64_t n, int64_t k, const void* a, int64_t lda, int64_t m, float gscale, void* d, int64_t ldd, int msub,
                           void* stream) {
    KYB_REQUIRE(d && ((uintptr_t)d & 1) == 0, "null or odd output pointer");
    void* outs[1] = {d};
    return kq_dense(fmt, t16, n, k, a, lda, m, gscale, outs, 1, ldd, 0, msub, stream);
}

// Diagnostics: the form that kyb_gemm_kq (split = 1), kyb_gemm_kq_splitk or kyb_gemm_kq_ag (destinations > 1) takes for a shape. out3 = {1 by CTA pairs / 0 one CTA, activation rows per item, items}.
// Without a device: as on 148 SMs.
extern "C" int kyb_gemm_kq_plan(int fmt, int64_t n, int64_t k, int64_t m, int split, int destinations, int64_t* out3) {
    KYB_REQUIRE(fmt >= 0 && fmt < KYB_FMT_COUNT && n > 0 && m > 0 && k > 0 && k % 256 == 0 && split >= 1 && split <= 8 && destinations >= 1 && out3, "bad arguments");
    const KqForm f = kq_choose(fmt, n, m, (int)(k / 256), split, kq_sms(), kq_pairs(fmt), kq_widest(destinations));
    out3[0] = f.pair, out3[1] = f.mt, out3[2] = (f.pair ? (n + 255) / 256 : (n + 127) / 128) * ((m + f.mt - 1) / f.mt) * split;
    return KYB_OK;
}

// Split-k for products that leave most SMs idle (e.g. 300 x 768 outputs from 12288 inputs: 3 items of 256 outputs): the k-blocks are cut into `split` equal ranges,
// (tile, range) items fill the SMs, every item leaves its fp32 accumulator in the workspace and a second kernel adds the ranges in k order (the result is
// deterministic; it differs from the unsplit product by fp32 summation order only). kyb_gemm_kq_split: the factor the library suggests (1: do not split);
// kyb_gemm_kq_split_bytes: bytes of 16-byte aligned workspace the call then needs.
extern "C" int kyb_gemm_kq_split(int fmt, int64_t n, int64_t k, int64_t m) {
    if (fmt < 0 || fmt >= KYB_FMT_COUNT || n <= 0 || k <= 0 || k % 256 || m <= 128) return 1;
    const int nb = (int)(k / 256), pairs = kq_pairs(fmt);
    if ((double)n * (double)m > 32.0 * 1024 * 1024) return 1;                          // hundreds of items: the ranges only add traffic
    // The launcher's own cost model with the split form's epilogue (fp32 stores, 1300 clocks per 32 rows), 3.2 us for the second launch, and the ranges and the output
    // at 1.5 and 3.7 MB per us; a split must be 4 % faster. Fitted to 480 timings of 11 shapes, 64 to 2048 rows, Q4_K and Q6_K: from 129 rows on it is on average 0.3 %
    // slower than the best factor and never slower than no split. Q4_K 768 x 12288, 300 rows 37.9 -> 19.3 us (six ranges), 2048 rows stay at 40.3 (six ranges: 60.9); 2048 x 8192, 512 rows
    // 28.1 (four ranges: 33.5); 3072 x 12288, 300 rows 38.9 -> 31.3 (three; six: 40.6).
    const double whole = kq_choose(fmt, n, m, nb, 1, kq_sms(), pairs).clocks / 1900.0;
    int best = 1;
    double best_us = 0.96 * whole;
    for (int sp = 2; sp <= 8; ++sp) {
        if (nb % sp || nb / sp < 4) continue;                                           // equal ranges of at least 1024 inputs
        const double us = kq_choose(fmt, n, m, nb, sp, kq_sms(), pairs, 256, 1300.0).clocks / 1900.0 + 3.2 + (double)m * (double)n / 1.0e6 * (sp * 4 * 0.654 + 2 * 0.273);
        if (us < best_us) best = sp, best_us = us;
    }
    return best;
}
extern "C" size_t kyb_gemm_kq_split_bytes(int64_t n, int64_t m, int split) {
    if (n <= 0 || m <= 0 || split <= 1) return 0;
    return (size_t)split * (size_t)(((m + 255) / 256) * 256) * (size_t)(((n + 255) / 256) * 256) * sizeof(float);   // rows and columns padded to whole work items
}
extern "C" int kyb_gemm_kq_splitk(int fmt, const void* t16, int64_t n, int64_t k, const void* a, int64_t lda, int64_t m, float gscale, void* d, int64_t ldd, int split,
                                  void* workspace, size_t workspace_bytes, void* stream) {
    KYB_REQUIRE(d && ((uintptr_t)d & 1) == 0, "null or odd output pointer");
    KYB_REQUIRE(split >= 2 && split <= 8 && k > 0 && k % 256 == 0 && (k / 256) % split == 0, "split=%d: 2..8 equal ranges of whole 256-input blocks (k=%lld)", split, (long long)k);
    const size_t need = kyb_gemm_kq_split_bytes(n, m, split);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 15)) {
        kyb_set_error("split-k needs %zu bytes of 16-byte aligned workspace, got %zu", need, workspace ? workspace_bytes : (size_t)0);
        return KYB_EWORKSPACE;
    }
    void* outs[1] = {d};
    return kq_dense(fmt, t16, n, k, a, lda, m, gscale, outs, 1, ldd, 0, 0, stream, split, (float*)workspace);
}

// The same product with the all-gather of an N-sharded linear folded into the epilogue: every tile goes to the output matrix of every rank, at column col0.
extern "C" int kyb_gemm_kq_ag(int fmt, const void* t16, int64_t n, int64_t k, const void* a, int64_t lda, int64_t m, float gscale, const kyb_peer_out* out, int64_t ldd,
                              int64_t col0, int msub, void* stream) {
    KYB_REQUIRE(out && out->count >= 1 && out->count <= 8, "peer outputs: 1..8 ranks");
    KYB_REQUIRE(col0 >= 0 && col0 % 8 == 0 && col0 + n <= ldd && ldd % 8 == 0, "col0=%lld: a multiple of 8 with col0 + n <= ldd, ldd a multiple of 8", (long long)col0);
    void* outs[8];
    for (int i = 0; i < out->count; ++i) {
        KYB_REQUIRE(out->ptr[i] && ((uintptr_t)out->ptr[i] & 15) == 0, "peer output %d is null or not 16-byte aligned", i);
        outs[i] = out->ptr[i];
    }
    return kq_dense(fmt, t16, n, k, a, lda, m, gscale, outs, out->count, ldd, col0, msub, stream);
}

// Grouped form for routed experts: a fp16 [s, k] rows sorted by expert (segment e = rows [off[e], off[e + 1])), T16 of the expert stack (experts * n rows),
// tb / off from kyb_moe_plan with the same mt (128 or 256 rows of one expert per work item: with 256 a decoded weight tile serves up to two 128-row blocks, so an
// expert with 129..256 rows is decoded once, not twice), row_map (optional, u32 [s]) = output row of each sorted row, gs (optional) per-expert output scale.
// d [*, n]. The item list is sized for the worst case (s / mt + experts tiles per 256 output columns); items past tb[experts] are skipped.
// t16b != null: the gated pair. t16 / t16b are the gate and up stacks of one shape, d [s, n] = fp16(silu(a) * b) of their fp16-rounded products.
static int kq_grouped(int fmt, const void* t16, const void* t16b, int64_t n, int64_t k, int experts, const void* a, int64_t lda, int64_t s, const void* tb, const void* off,
                      const void* row_map, const void* gs, const void* gsb, float limit, void* d, int64_t ldd, int mt, void* stream) {
    const bool glu = t16b != nullptr;
    KYB_REQUIRE(mt == 128 || mt == 256, "mt=%d: 128 or 256 rows per work item", mt);
    KYB_REQUIRE(fmt >= 0 && fmt < KYB_FMT_COUNT, "unknown weight format %d", fmt);
    KYB_REQUIRE(t16 && a && d && tb && off, "null pointer");
    KYB_REQUIRE(s > 0 && n > 0 && k > 0 && k % 256 == 0 && experts > 0, "s=%lld n=%lld k=%lld experts=%d: k must be a positive multiple of 256", (long long)s, (long long)n,
                (long long)k, experts);
    if (glu) {
        KYB_REQUIRE(n % 128 == 0, "the gated pair needs n %% 128 == 0, got n=%lld", (long long)n);
        KYB_REQUIRE(ldd % 8 == 0 && ((uintptr_t)d & 15) == 0 && ((uintptr_t)t16b & 15) == 0 && !row_map, "the gated pair stores 16-byte pieces in sorted order: ldd %% 8 == 0, aligned d, no row_map");
    } else {
        KYB_REQUIRE(n % 256 == 0, "the grouped product needs n %% 256 == 0 (an output tile must not straddle two experts), got n=%lld", (long long)n);
    }
    KYB_REQUIRE(lda >= k && lda % 8 == 0 && ldd >= n, "leading dimensions: lda >= k and a multiple of 8, ldd >= n");
    KYB_REQUIRE(((uintptr_t)a & 15) == 0 && ((uintptr_t)t16 & 15) == 0, "a and t16 must be 16-byte aligned");
    KYB_REQUIRE(s < (1ll << 31) && (int64_t)experts * n < (1ll << 31) && k < (1ll << 24), "dimension too large");
    unsigned int* status = kyb_device_status_word();
    KYB_REQUIRE(status, "could not set up the device status word");
    CUtensorMap ta;
    if (int rc = kyb_make_tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a, (uint64_t)s, (uint64_t)k, (uint64_t)lda * 2, 64, 64)) return rc;
    kyb::KqParams p;
    memset(&p, 0, sizeof(p));
    p.t16 = (const uint8_t*)t16, p.ldd = ldd, p.m = (int)s, p.n = (int)n, p.k = (int)k, p.nb = (int)(k / 256);
    p.nout = 1, p.d[0] = (__half*)d;
    p.rt_total = (int)((int64_t)experts * n / 16);
    p.gscale = 1.0f, p.status = status, p.tb = (const uint32_t*)tb, p.off = (const uint32_t*)off, p.row_map = (const uint32_t*)row_map, p.gs = (const float*)gs, p.experts = experts;
    p.mt = mt, p.ksplit = 1;
    p.t16b = (const uint8_t*)t16b, p.gsb = (const float*)gsb, p.glu = glu ? 1 : 0, p.limit = limit;
    int pairs = 0;
    if (int rc = kq_configure<true>(fmt, &pairs)) return rc;
    p.box_rows = 64;                                                               // segments have any number of rows: boxes of 64 as needed
    p.tiles_n = (int)(n / (glu ? kyb::KQ_BN / 2 : kyb::KQ_BN)) / (pairs > 0 ? 2 : 1), p.tiles_m = (int)((s + mt - 1) / mt) + experts;
    p.vec_out = (ldd % 8 == 0 && ((uintptr_t)d & 15) == 0) ? 1 : 0;                // rows are scattered (row_map) or end inside a tile: no tensor map fits
    KybOutMaps outs;
    memset(&outs, 0, sizeof(outs));
    const int items = p.tiles_n * p.tiles_m;
    if (int rc = pairs > 0 ? kq_launch<true>(fmt, ta, outs, p, items, pairs, (cudaStream_t)stream) : kq_launch<false>(fmt, ta, outs, p, items, kq_sms(), (cudaStream_t)stream)) return rc;
    return kyb_zero_tail_rows(d, ldd, n, row_map, (const uint32_t*)off + experts, s, (cudaStream_t)stream);   // slots that belong to no expert: rows of zeros
}

extern "C" int kyb_gemm_kq_grouped(int fmt, const void* t16, int64_t n, int64_t k, int experts, const void* a, int64_t lda, int64_t s, const void* tb, const void* off,
                                   const void* row_map, const void* gs, void* d, int64_t ldd, int mt, void* stream) {
    return kq_grouped(fmt, t16, nullptr, n, k, experts, a, lda, s, tb, off, row_map, gs, nullptr, 0.f, d, ldd, mt, stream);
}

// Gate and up of a routed SwiGLU layer as ONE grouped product with the gated activation in its epilogue: h fp16 [s, n] (sorted order) = silu(a) * b with
// a = fp16(x W_gate^T), b = fp16(x W_up^T) (the values the two-launch form would have written) and the optional clamp of kyb_silu_mul. Replaces two
// kyb_gemm_kq_grouped calls and kyb_silu_mul (kyojin_mlx/foreign_kqgmm.py:293-314 `mlp`: gmm, gmm, silu_perm).
extern "C" int kyb_gemm_kq_grouped_glu(int fmt, const void* t16_gate, const void* t16_up, int64_t n, int64_t k, int experts, const void* a, int64_t lda, int64_t s,
                                       const void* tb, const void* off, const void* gs_gate, const void* gs_up, float limit, void* h, int64_t ldh, int mt, void* stream) {
    KYB_REQUIRE(t16_up, "null pointer");
    return kq_grouped(fmt, t16_gate, t16_up, n, k, experts, a, lda, s, tb, off, nullptr, gs_gate, gs_up, limit, h, ldh, mt, stream);
}
