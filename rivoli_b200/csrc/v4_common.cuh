// Shared pieces of the V4 cousin path (block indexer, selection, sparse attention, KV compressor).
#pragma once

#include "codec.cuh"
#include "common.cuh"

__device__ __forceinline__ float v4_rbf16(float x) { return rv_bf16_to_f32(rv_f32_to_bf16(x)); }

// One element of an f32 or a bf16 array, widened exactly.
__device__ __forceinline__ float v4_load_f32(const float* p, size_t i) { return p[i]; }
__device__ __forceinline__ float v4_load_f32(const uint16_t* p, size_t i) { return rv_bf16_to_f32(p[i]); }

constexpr int V4_ROT_MAX = 256;
constexpr float V4_FP4_MAX = 6.0f;

// e2m1 round trip of q (already clamped to [-6, 6]): nearest grid point, midpoints to the even code.
__device__ __forceinline__ float v4_e2m1_roundtrip(float q) {
    const float a = fabsf(q);
    int code = 0;
    code += a > 0.25f;
    code += a >= 0.75f;
    code += a > 1.25f;
    code += a >= 1.75f;
    code += a > 2.5f;
    code += a >= 3.5f;
    code += a > 5.0f;
    const float mag = code < 4 ? 0.5f * (float)code : (code == 4 ? 2.0f : (code == 5 ? 3.0f : (code == 6 ? 4.0f : 6.0f)));
    return signbit(q) ? -mag : mag;
}

// Smallest power of two >= amax / 6, from the exponent field of the product.
__device__ __forceinline__ float v4_round_scale(float amax) {
    const uint32_t b = __float_as_uint(__fmul_rn(amax, __fdiv_rn(1.0f, V4_FP4_MAX)));
    const int e = (int)((b >> 23) & 0xffu) - 127 + ((b & 0x7fffffu) ? 1 : 0);
    return __uint_as_float((uint32_t)(e + 127) << 23);
}

// Hadamard + fp4 spread of one row. One WARP per row, the row in registers: lane l holds the E = d / 32 consecutive values from l * E. The butterfly visits
// the operand pairs (j, j + h) stage by stage exactly as the host loop does - in a thread while h < E, between lanes
// (shuffle) beyond - and which thread evaluates a pair does not change the value. A block of 32 is 32 / E lanes. The scale
// is a power of two, so the quotient is the exact product with its reciprocal (a normal number: the scale lies between
// 2^-126 and 2^125; an infinite row has an infinite scale and the reciprocal 0, with which an infinite value gives NaN and a
// finite one 0, both NaN once multiplied by the scale, as with the division). 4,095 rows of 128: 10.3 us with a CTA per row and the row in shared memory, 3.8 us now.
template <int E>
__device__ __forceinline__ void v4_spread_row(float (&v)[E], int lane) {
    constexpr int D = E * 32;
#pragma unroll
    for (int h = 1; h < E; h <<= 1)
#pragma unroll
        for (int j = 0; j < E; ++j)
            if (!(j & h)) {
                const float a = v[j], b = v[j + h];
                v[j] = __fadd_rn(a, b);
                v[j + h] = __fsub_rn(a, b);
            }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const float other = __shfl_xor_sync(0xffffffffu, v[j], o);
            v[j] = (lane & o) ? __fsub_rn(other, v[j]) : __fadd_rn(v[j], other);
        }
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)D));
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < E; ++j) { v[j] = v4_rbf16(__fmul_rn(v[j], scale)); amax = fmaxf(amax, fabsf(v[j])); }
#pragma unroll
    for (int o = 1; o < 32 / E; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));   // exact under any association
    const float s = v4_round_scale(fmaxf(amax, __fmul_rn(V4_FP4_MAX, __uint_as_float(1u << 23))));
    const float inv = isinf(s) ? 0.0f : __uint_as_float((254u << 23) - __float_as_uint(s));
#pragma unroll
    for (int j = 0; j < E; ++j) {
        float q = __fmul_rn(v[j], inv);
        q = q < -V4_FP4_MAX ? -V4_FP4_MAX : (q > V4_FP4_MAX ? V4_FP4_MAX : q);
        v[j] = v4_rbf16(__fmul_rn(v4_e2m1_roundtrip(q), s));
    }
}

static inline int v4_check_geom(const V4Geom* g, int n_seqs) {
    if (!g || n_seqs <= 0) return 1001;
    if (g->n_heads <= 0 || g->head_dim <= 0 || g->window <= 0 || g->index_heads <= 0 || g->index_dim <= 0 ||
        g->index_topk <= 0 || g->ratio <= 1 || g->max_comp <= 0)
        return 1001;
    return 0;
}
