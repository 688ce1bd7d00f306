// Warp-cooperative fp8 e4m3 quantisation of bf16 rows: shared by the append operator, the indexer-query operator and the
// fused decode-step prologue.
//
// The definition is code = e4m3(x / s) with an IEEE f32 division and s = absmax / 448. A division per value (704 of them per
// token) costs more than everything else together, so the quotient is the product with a two-term reciprocal
// r + rl ~ 1 / s (r = RN(1 / s), rl = RN(RN(1 - r s) r)):  q = RN(x r + RN(x rl)), one multiply and one fused multiply-add.
// For the operands that occur here - x and the absmax behind s are bf16 numbers - this IS the correctly rounded x / s: all
// 128 x 128 pairs of mantissas were compared (exponents only shift the result while nothing under- or overflows, which
// rv_quant_scale's range guarantees for every quotient that gives a normal code). Codes without an exponent (zeros and
// subnormals, where the reference rounds ties away from zero and the converter to even) and scales outside the range take
// the division and the software codec.
#pragma once

#include "codec.cuh"
#include "common.cuh"

struct QuantScale { float s, r, rl; };   // the scale, its reciprocal (r = 0: outside the range of the fast quotient) and the rest
__device__ __forceinline__ QuantScale rv_quant_scale(float amax) {
    QuantScale q;
    q.s = rv_scale_from_amax(amax);
    q.r = (q.s >= 8.077935669463161e-28f && q.s <= 1.2379400392853803e27f) ? __frcp_rn(q.s) : 0.0f;   // 2^-90 .. 2^90
    q.rl = __fmul_rn(fmaf(-q.r, q.s, 1.0f), q.r);
    return q;
}

// Largest |value| of eight packed bf16 values, in both halves of a bf16x2 word (a NaN loses against a number).
__device__ __forceinline__ uint32_t rv_max_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t rv_absmax8(const uint4& p) {
    const uint32_t m = rv_max_bf16x2(rv_max_bf16x2(p.x & 0x7fff7fffu, p.y & 0x7fff7fffu), rv_max_bf16x2(p.z & 0x7fff7fffu, p.w & 0x7fff7fffu));
    return rv_max_bf16x2(m, __byte_perm(m, m, 0x1032));
}

// Eight packed bf16 values -> eight codes by the fast quotient. Bits come up in `redo` if any of them has to be done by
// rv_codes8_exact: a byte whose exponent bits are all zero borrows into its top bit (no byte of the masked word exceeds
// 0x78).
__device__ __forceinline__ uint2 rv_codes8(const uint4& p, const QuantScale& q, uint32_t& redo) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
    uint16_t h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float x0 = __uint_as_float(w[i] << 16), x1 = __uint_as_float(w[i] & 0xffff0000u);
        const float lo = fmaf(x0, q.r, __fmul_rn(x0, q.rl)), hi = fmaf(x1, q.r, __fmul_rn(x1, q.rl));
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(h[i]) : "f"(hi), "f"(lo));
    }
    uint2 o;
    asm("mov.b32 %0, {%1, %2};" : "=r"(o.x) : "h"(h[0]), "h"(h[1]));
    asm("mov.b32 %0, {%1, %2};" : "=r"(o.y) : "h"(h[2]), "h"(h[3]));
    redo |= ((o.x & 0x78787878u) - 0x01010101u) | ((o.y & 0x78787878u) - 0x01010101u);
    return o;
}
constexpr uint32_t RV_REDO = 0x80808080u;
__device__ __forceinline__ uint2 rv_codes8_exact(const uint4& p, float s) {
    uint2 o = make_uint2(0u, 0u);
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const uint32_t v = i == 0 ? p.x : (i == 1 ? p.y : (i == 2 ? p.z : p.w));
        const uint32_t h = rv_f32x2_to_e4m3x2(__fdiv_rn(__uint_as_float(v << 16), s), __fdiv_rn(__uint_as_float(v & 0xffff0000u), s));
        if (i < 2) o.x |= h << (16 * i); else o.y |= h << (16 * (i - 2));
    }
    return o;
}

// Quantise a vector of `n` bf16 values (n % 16 == 0, n <= 512) by one warp: lane l takes the chunks of eight l and l + 32.
// Returns the scale (all lanes).
__device__ __forceinline__ float quant_vec(const uint16_t* __restrict__ src, int n, uint8_t* __restrict__ dst, int lane) {
    uint4 v[2];
    uint32_t m = 0u;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = (lane + 32 * u) * 8;
        v[u] = i < n ? *reinterpret_cast<const uint4*>(src + i) : make_uint4(0u, 0u, 0u, 0u);
        m = rv_max_bf16x2(m, rv_absmax8(v[u]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = rv_max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, o));
    const QuantScale q = rv_quant_scale(__uint_as_float(m << 16));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = (lane + 32 * u) * 8;
        if (i < n) {
            uint32_t redo = q.r == 0.0f ? RV_REDO : 0u;
            uint2 c = rv_codes8(v[u], q, redo);
            if (redo & RV_REDO) c = rv_codes8_exact(v[u], q.s);
            *reinterpret_cast<uint2*>(dst + i) = c;
        }
    }
    return q.s;
}

// ------------------------------------------------------------------------------------------
// One token row into the paged pools, by one warp: the latent row (c_kv | k_rope, one scale) and the indexer key (one scale)
// as ONE run of 8-value chunks, lane l taking the chunks l, l + 32, ...: every load is 512 contiguous bytes of a warp, and
// at the model's 576 + 128 values three passes do it with 92 % of the lanes (16-value chunks, latent and key apart: three
// passes with 46 %). All loads and the page lookup are issued together, so the position -> page -> store chain costs two
// memory round trips. PASSES * 32 chunks cover the geometry (rv_append_chunks).
// 65,537 tokens take 34.3 us (4.1 TB/s read and written; two thirds of the issue slots are in use, 400 instructions a
// token); 109 us with divisions. A persistent grid with the next row requested ahead took 44 us (fewer warps).
// ------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ int rv_append_chunks(const DsaGeom& g) { return (g.kv_lora + g.rope_dim + g.index_dim) / 8; }

template <int PASSES>
struct AppendRow {
    uint4 v[PASSES];
    int page, pos;
};
// Requests a row's values and its page (no use of either).
template <int PASSES>
__device__ __forceinline__ void append_row_load(AppendRow<PASSES>& a, const DsaGeom& g, const uint16_t* __restrict__ latent,
                                                const uint16_t* __restrict__ index_key, int row, int seq, int pos,
                                                const int32_t* __restrict__ block_table, int lane) {
    const int w = g.kv_lora + g.rope_dim, hd = g.index_dim, nl = w / 8, n = nl + hd / 8;
    const int lp = pos >> rv_log2(g.page_tokens);
    a.pos = pos;
    a.page = -1;
    if (pos >= 0 && lp < g.max_pages_per_seq) a.page = block_table[(size_t)seq * g.max_pages_per_seq + lp];
    const uint4* src = reinterpret_cast<const uint4*>(latent + (size_t)row * w);
    const uint4* key = reinterpret_cast<const uint4*>(index_key + (size_t)row * hd) - nl;
#pragma unroll
    for (int u = 0; u < PASSES; ++u) {
        const int i = lane + 32 * u;
        a.v[u] = i < n ? (i < nl ? src : key)[i] : make_uint4(0u, 0u, 0u, 0u);
    }
}
// Quantises and stores a loaded row.
template <int PASSES>
__device__ __forceinline__ void append_row_store(const AppendRow<PASSES>& a, const DsaGeom& g, uint8_t* __restrict__ latent_pool,
                                                 float* __restrict__ latent_scale, uint8_t* __restrict__ index_pool,
                                                 float* __restrict__ index_scale, int32_t* __restrict__ status, int lane) {
    const int w = g.kv_lora + g.rope_dim, hd = g.index_dim, nl = w / 8, n = nl + hd / 8;
    uint32_t m = 0u;                       // running maxima: latent in the low half, key in the high half
#pragma unroll
    for (int u = 0; u < PASSES; ++u) m = rv_max_bf16x2(m, rv_absmax8(a.v[u]) & (lane + 32 * u < nl ? 0x0000ffffu : 0xffff0000u));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = rv_max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, o));
    // the lower half-warp works out the latent row's scale, the upper the key's
    const QuantScale mine = rv_quant_scale(__uint_as_float(lane < 16 ? m << 16 : m & 0xffff0000u));
    QuantScale ql, qk;
    ql.s = __shfl_sync(0xffffffffu, mine.s, 0); ql.r = __shfl_sync(0xffffffffu, mine.r, 0);
    qk.s = __shfl_sync(0xffffffffu, mine.s, 16); qk.r = __shfl_sync(0xffffffffu, mine.r, 16);
    ql.rl = __shfl_sync(0xffffffffu, mine.rl, 0); qk.rl = __shfl_sync(0xffffffffu, mine.rl, 16);
    if (a.page < 0 || a.page >= g.n_pool_pages) {
        if (lane == 0 && status) atomicOr(status, 1);
        return;
    }
    const size_t r = (size_t)a.page * g.page_tokens + (a.pos & (g.page_tokens - 1));
    uint2* dl = reinterpret_cast<uint2*>(latent_pool + r * w);
    uint2* dk = reinterpret_cast<uint2*>(index_pool + r * hd) - nl;
#pragma unroll
    for (int u = 0; u < PASSES; ++u) {
        const int i = lane + 32 * u;
        if (i < n) {
            const bool lat = i < nl;
            QuantScale q;
            q.s = lat ? ql.s : qk.s;
            q.r = lat ? ql.r : qk.r;
            q.rl = lat ? ql.rl : qk.rl;
            uint32_t redo = q.r == 0.0f ? RV_REDO : 0u;
            uint2 c = rv_codes8(a.v[u], q, redo);
            if (redo & RV_REDO) c = rv_codes8_exact(a.v[u], q.s);   // rare: about one lane in fifteen rows of normal data
            (lat ? dl : dk)[i] = c;
        }
    }
    if (lane == 0) {
        latent_scale[r] = ql.s;
        index_scale[r] = qk.s;
    }
}
