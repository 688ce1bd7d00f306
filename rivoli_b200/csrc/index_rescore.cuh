// Exact lightning-indexer score of LISTED tokens, in the fold order of rivoli_index_score_paged (bit-identical to it):
//   cd = left fold over d of qcode[h][d] * kcode[t][d]   (each product of two e4m3 values is exact in f32, so the fused
//        multiply-add IS the reference's acc + q * k: crates/engine/tests/indexer_kernel.rs:237-249)
//   dot = (cd * s_q[h]) * s_k[t];  term_h = (w[h] * wscale) * max(dot * dscale, 0);  score = fold over h ascending.
// A warp takes four consecutive listed tokens per pass (their loads are in flight together and they share the q values), lane =
// head (index_heads <= 32), index_dim = 128 (one 4-code word per lane). Two tokens ride in one packed f32x2 multiply-add, each
// half rounded as the scalar one is; the tokens of a dim lie side by side.
#pragma once

#include "codec.cuh"
#include "common.cuh"

constexpr int RS_HD = 128;

// Word e of the q codes of one sequence, PACKED as they lie in memory (word w of head h = its dims 4w .. 4w+3) and transposed
// to [word][head] (lane = head on both sides: no bank conflicts); RS_QWORDS of them. The fold decodes a word into its four
// values on the fly (exactly): as (q, q) f32 pairs in shared memory they cost eight times its bandwidth, which then bounds the
// fold (99 tokens on an SM: 14,000 cycles, 6,300 so).
constexpr int RS_QWORDS = 32 * (RS_HD / 4);
__device__ __forceinline__ uint32_t rv_rescore_q_word(const uint8_t* __restrict__ qcodes_seq, int nh, int e) {
    const int h = e & 31, d4 = e >> 5;
    return h < nh ? *reinterpret_cast<const uint32_t*>(qcodes_seq + (size_t)h * RS_HD + d4 * 4) : 0u;
}

__device__ __forceinline__ uint64_t rs_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Pool row of token t (rows of unmapped pages stand in as page 0).
__device__ __forceinline__ uint32_t rv_pool_row(const DsaGeom& g, const int32_t* __restrict__ bt, uint32_t t) {
    const int pshift = 31 - __clz(g.page_tokens), pg = bt[t >> pshift];   // page sizes are powers of two
    return ((pg < 0 || pg >= g.n_pool_pages ? 0u : (uint32_t)pg) << pshift) + (t & (uint32_t)(g.page_tokens - 1));
}

// Scores `ln` listed tokens, row_of(position) being a token's pool row: a pass covers WARPS * 4 of them, warp w taking
// positions base + 4 w .. + 3.
// kf = this WARP's staging of four key rows as f32, [dim][token] (RS_HD * 4 floats, 16-byte aligned). my_sq / my_wh = this
// lane's head scale and weight * wscale (0 for lanes >= nh). emit(position, score) is called by one lane per token.
template <int WARPS, class RowOf, class Emit>
__device__ __forceinline__ void rv_rescore_listed(RowOf row_of, uint32_t ln, const uint32_t* qf, float* kf, const DsaGeom& g,
                                                  const uint8_t* __restrict__ index_pool,
                                                  const float* __restrict__ index_scale, float my_sq, float my_wh,
                                                  Emit emit) {
    constexpr int TOK = 4, PAD = 36;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
    for (uint32_t p0 = warp * TOK; p0 < ln; p0 += WARPS * TOK) {
        const int n_here = min(TOK, (int)(ln - p0));
        uint32_t cw[TOK];
        float skv[TOK];
#pragma unroll
        for (int e = 0; e < TOK; ++e) {
            cw[e] = 0u; skv[e] = 0.0f;
            if (e < n_here) {
                const size_t rr = row_of(p0 + e);
                cw[e] = *reinterpret_cast<const uint32_t*>(index_pool + rr * RS_HD + lane * 4);
                skv[e] = index_scale[rr];
            }
        }
        float2 lo[TOK], hi[TOK];
#pragma unroll
        for (int e = 0; e < TOK; ++e) { lo[e] = rv_e4m3x2_to_f32x2((uint16_t)(cw[e] & 0xffff)); hi[e] = rv_e4m3x2_to_f32x2((uint16_t)(cw[e] >> 16)); }
        float4* dst = reinterpret_cast<float4*>(kf) + lane * 4;
        dst[0] = make_float4(lo[0].x, lo[1].x, lo[2].x, lo[3].x);
        dst[1] = make_float4(lo[0].y, lo[1].y, lo[2].y, lo[3].y);
        dst[2] = make_float4(hi[0].x, hi[1].x, hi[2].x, hi[3].x);
        dst[3] = make_float4(hi[0].y, hi[1].y, hi[2].y, hi[3].y);
        __syncwarp();
        uint64_t c01 = 0ull, c23 = 0ull;
#pragma unroll 4
        for (int d = 0; d < RS_HD; d += 4) {
            const uint32_t qc = qf[d * 8 + lane];
            const float2 qa = rv_e4m3x2_to_f32x2((uint16_t)(qc & 0xffff)), qb = rv_e4m3x2_to_f32x2((uint16_t)(qc >> 16));
            const float q4[4] = {qa.x, qa.y, qb.x, qb.y};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ulonglong2 k4 = reinterpret_cast<const ulonglong2*>(kf)[d + i];   // broadcast read
                uint64_t q2;
                asm("mov.b64 %0, {%1, %1};" : "=l"(q2) : "f"(q4[i]));
                c01 = rs_fma2(q2, k4.x, c01);
                c23 = rs_fma2(q2, k4.y, c23);
            }
        }
        const float cd[TOK] = {__uint_as_float((uint32_t)c01), __uint_as_float((uint32_t)(c01 >> 32)),
                               __uint_as_float((uint32_t)c23), __uint_as_float((uint32_t)(c23 >> 32))};
        __syncwarp();
#pragma unroll
        for (int e = 0; e < TOK; ++e) {
            const float dot = __fmul_rn(__fmul_rn(cd[e], my_sq), skv[e]);
            float rr = __fmul_rn(dot, g.index_dscale);
            rr = rr > 0.0f ? rr : 0.0f;
            kf[e * PAD + lane] = __fmul_rn(my_wh, rr);     // (an absent head's term is +0, which changes no sum)
        }
        __syncwarp();
        if (lane < n_here) {
            float acc = 0.0f;
#pragma unroll
            for (int h = 0; h < 32; h += 4) {
                const float4 t4 = *reinterpret_cast<const float4*>(kf + lane * PAD + h);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, t4.x), t4.y), t4.z), t4.w);
            }
            emit(p0 + lane, acc);
        }
        __syncwarp();
    }
}
