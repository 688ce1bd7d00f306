// V4 cousin of the decode path, part 3: the KV compressor (deposit, pooling, finish) and the fp8 prefix quantiser.
#include "v4_common.cuh"

namespace {

// ---------------------------------------------------------------------------------------------------
// KV compressor, decode arm: deposit one token into the pooling state; when a block closes, pool it
// (softmax over the ENTRY axis per feature), bf16 store, RMSNorm, rotate the last rd dims at the block's
// first position, then the finishing quantisation (spread for the indexer's compressor, fp8 block-64
// on the un-rotated dims for the attention compressor).
// Reference: crates/backend/kernels/kvcompress.hip (deposit / decode / pool_row / finish_row),
// crates/oracles/src/v4oracle/compress.rs:131-200.
// ---------------------------------------------------------------------------------------------------
constexpr int CP_THREADS = 256;
constexpr int CP_ENTS_MAX = 128;
constexpr float CP_FP8_MAX = 448.0f;

__device__ __forceinline__ float cp_block_sum(float v, float* red) {   // red: CP_THREADS / 32 floats
    v = rv_warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < CP_THREADS / 32; ++i) t += red[i];
    __syncthreads();
    return t;
}

// e4m3 round trip with round-to-nearest-even everywhere and saturation at 448: the hardware converter's rule.
__device__ __forceinline__ float cp_e4m3_roundtrip(float q) {
    uint16_t c;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(c) : "f"(q), "f"(0.0f));
    return rv_e4m3x2_to_f32x2(c).x;
}

// fp8 quantise-dequantise of one block of `block` values starting at seg (one warp; power-of-two scale,
// amax floor 1e-4): crates/backend/kernels/mla.hip:319-338. Exact: the maximum is associative, the rest is
// per element.
__device__ __forceinline__ void cp_act_quant_block(const float* seg, float* out, int block) {
    const int lane = threadIdx.x & 31;
    float amax = 1e-4f;
    for (int i = lane; i < block; i += 32) amax = fmaxf(amax, fabsf(seg[i]));
    amax = rv_warp_max(amax);
    const uint32_t bits = __float_as_uint(__fmul_rn(amax, __fdiv_rn(1.0f, CP_FP8_MAX)));
    const int e = (int)((bits >> 23) & 0xffu) - 127 + ((bits & 0x7fffffu) ? 1 : 0);
    const float s = __uint_as_float((uint32_t)(e + 127) << 23);
    for (int i = lane; i < block; i += 32) {
        float q = __fdiv_rn(seg[i], s);
        q = q < -CP_FP8_MAX ? -CP_FP8_MAX : (q > CP_FP8_MAX ? CP_FP8_MAX : q);
        out[i] = __fmul_rn(cp_e4m3_roundtrip(q), s);
    }
}

// The scale of a block (a power of two) and its reciprocal (2^-e is a normal number: e >= -22), by which a quotient is exact.
// An infinite block has an infinite scale (e = 128) and the reciprocal 0, which gives what the division by infinity does: NaN
// for an infinite value, 0 for any other, and NaN for both once multiplied by the scale.
__device__ __forceinline__ float cp_f8_scale(float amax, float& inv) {
    const uint32_t bits = __float_as_uint(__fmul_rn(amax, __fdiv_rn(1.0f, CP_FP8_MAX)));
    const int e = (int)((bits >> 23) & 0xffu) - 127 + ((bits & 0x7fffffu) ? 1 : 0);
    inv = e == 128 ? 0.0f : __uint_as_float((uint32_t)(127 - e) << 23);
    return __uint_as_float((uint32_t)(e + 127) << 23);
}
__device__ __forceinline__ float cp_f8_roundtrip(float x, float s, float inv) {
    float q = __fmul_rn(x, inv);
    q = q < -CP_FP8_MAX ? -CP_FP8_MAX : (q > CP_FP8_MAX ? CP_FP8_MAX : q);
    return __fmul_rn(cp_e4m3_roundtrip(q), s);
}

// The same for blocks of 64 with 16-byte accesses: a thread holds four values, sixteen neighbours a block. Bound by
// memory (read once, written once); 4,095 rows of 448: 10.3 us with one warp per block and two values per lane, 5.2 us now.
__global__ void __launch_bounds__(256)
cp_act_quant_f8_prefix64_kernel(const float* src, float* dst, int rows, int row_stride, int n) {
    const int per_row = n / 4;
    const size_t id = (size_t)blockIdx.x * 256 + threadIdx.x, row = id / per_row;
    const int c = (int)(id - row * per_row) * 4;
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    const bool live = row < (size_t)rows;
    const float4 v = live ? *reinterpret_cast<const float4*>(src + row * row_stride + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    float inv;
    const float s = cp_f8_scale(fmaxf(amax, 1e-4f), inv);
    auto one = [&](float x) { return cp_f8_roundtrip(x, s, inv); };
    if (live) *reinterpret_cast<float4*>(dst + row * row_stride + c) = make_float4(one(v.x), one(v.y), one(v.z), one(v.w));
}

__global__ void cp_act_quant_f8_prefix_kernel(const float* src, float* dst, int rows, int row_stride, int n, int block) {
    const int nb = n / block;
    const size_t id = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);   // one warp per block
    if (id >= (size_t)rows * (size_t)nb) return;
    const size_t off = (size_t)(id / nb) * row_stride + (size_t)(id % nb) * block;
    cp_act_quant_block(src + off, dst + off, block);
}

struct CpState {
    float* kv;      // [ents][cd]
    float* score;   // [ents][cd]
};

// bf16 row -> RMSNorm (bf16 store) -> rotation of the last rd dims at `pos` (bf16 store), in place, by one CTA.
// red: CP_THREADS / 32 floats of shared memory.
__device__ __forceinline__ void cp_finish_row(float* row, const float* __restrict__ norm, const float* __restrict__ freqs,
                                              CompGeom p, int pos, float* red) {
    const int tid = threadIdx.x, d = p.d;
    float part = 0.0f;
    for (int e = tid; e < d; e += CP_THREADS) part += row[e] * row[e];
    const float rs = 1.0f / sqrtf(cp_block_sum(part, red) / (float)d + p.eps);
    for (int e = tid; e < d; e += CP_THREADS) row[e] = v4_rbf16(norm[e] * (row[e] * rs));
    __syncthreads();
    float* seg = row + (d - p.rd);
    for (int i = tid; i < p.rd / 2; i += CP_THREADS) {
        const float c = freqs[(size_t)pos * p.rd + 2 * i], sn = freqs[(size_t)pos * p.rd + 2 * i + 1];
        const float a = seg[2 * i], b = seg[2 * i + 1];
        seg[2 * i] = v4_rbf16(__fsub_rn(__fmul_rn(a, c), __fmul_rn(b, sn)));
        seg[2 * i + 1] = v4_rbf16(__fadd_rn(__fmul_rn(a, sn), __fmul_rn(b, c)));
    }
    __syncthreads();
}

// Pool + bf16 + RMSNorm + rotation of one sequence's state into row[d] (shared or global), by one CTA;
// then the overlap half of the state moves down.
__device__ __forceinline__ void cp_pool_finish(CpState st, const float* __restrict__ norm,
                                               const float* __restrict__ freqs, float* row, CompGeom p,
                                               int start_pos, float* red) {
    const int tid = threadIdx.x, d = p.d, cd = p.cd, overlap = p.coff == 2;
    for (int e = tid; e < d; e += CP_THREADS) {
        float mx = -INFINITY;
        for (int j = 0; j < p.ents; ++j) mx = fmaxf(mx, st.score[(size_t)j * cd + ((overlap && j >= p.ratio) ? d : 0) + e]);
        float o = 0.0f;
        if (isfinite(mx)) {
            float sum = 0.0f;
            for (int j = 0; j < p.ents; ++j)
                sum += expf(st.score[(size_t)j * cd + ((overlap && j >= p.ratio) ? d : 0) + e] - mx);
            for (int j = 0; j < p.ents; ++j) {
                const size_t a = (size_t)j * cd + ((overlap && j >= p.ratio) ? d : 0) + e;
                o += st.kv[a] * (expf(st.score[a] - mx) / sum);
            }
        }
        row[e] = v4_rbf16(o);
    }
    __syncthreads();
    cp_finish_row(row, norm, freqs, p, (start_pos / p.ratio) * p.ratio, red);
    if (overlap) {   // every pooling read is done (barriers above): the overlap half moves down
        const size_t n = (size_t)p.ratio * cd;
        for (size_t i = tid; i < n; i += CP_THREADS) {
            st.kv[i] = st.kv[n + i];
            st.score[i] = st.score[n + i];
        }
    }
    __syncthreads();
}

// Prefill arm: block b of a prompt that starts at position 0. Entry j of its window is row j - ratio of block b
// (second half of the projected row) or, with overlap, row j of block b - 1 (first half; absent for block 0);
// scores get the positional bias of the row's place in ITS block.
__global__ void __launch_bounds__(CP_THREADS) cp_prefill_kernel(const float* __restrict__ kv,
                                                                const float* __restrict__ score,
                                                                const float* __restrict__ ape, CompFinish f, CompGeom p) {
    __shared__ float red[CP_THREADS / 32];
    const int b = blockIdx.x, tid = threadIdx.x, d = p.d, cd = p.cd, overlap = p.coff == 2;
    float* row = f.out + (size_t)b * d;
    for (int e = tid; e < d; e += CP_THREADS) {
        float mx = -INFINITY;
        float sum = 0.0f, o = 0.0f;
        for (int pass = 0; pass < 3; ++pass) {   // 0: maximum, 1: sum of exponentials, 2: weighted values
            for (int j = 0; j < p.ents; ++j) {
                int sblk, src_j, half;
                if (!overlap) { sblk = b; src_j = j; half = 0; }
                else if (j >= p.ratio) { sblk = b; src_j = j - p.ratio; half = d; }
                else if (b > 0) { sblk = b - 1; src_j = j; half = 0; }
                else continue;
                const size_t src = (size_t)(sblk * p.ratio + src_j) * cd + half + e;
                const float sc = score[src] + ape[(size_t)src_j * cd + half + e];
                if (pass == 0) mx = fmaxf(mx, sc);
                else if (pass == 1) sum += expf(sc - mx);
                else o += kv[src] * (expf(sc - mx) / sum);
            }
            if (pass == 0 && !isfinite(mx)) break;
        }
        row[e] = v4_rbf16(isfinite(mx) ? o : 0.0f);
    }
    __syncthreads();
    cp_finish_row(row, f.norm, f.freqs, p, b * p.ratio, red);
}

// The same for the overlapping ratio-4 compressor with d = 128, 256 or 512 (what both compressors of a layer are): eight
// entries per block and feature, every projected value used exactly once (8.8 bytes a value): bound by HBM, 4.6 TB/s at
// d 512, and the issue slots of the exponentials and quotients. A thread owns two features of one block, d / 2 threads a block:
// its 8 scores and 8 values are all requested before the first is used (128 bytes per thread; two features and not four, so that
// several CTAs share an SM: the exponentials of one cover the loads of another); the maximum, the exponentials (one per entry instead of two) and the weighted sum run from
// registers. Values and their order are those of the kernel above and of the decode arms, the quotients and the norm's partial
// sums included (a row meets in shared memory in the order of a 256-thread CTA): a block has the same bits whether it was
// pooled from a prompt or token by token. (The sum divided once and the norm summed as the features lie would take 27.7 us
// instead of 30.9 at 4,095 blocks of d 512, and land on other codes now and then.) The positional bias sits in shared memory for
// the CTA's walk over the grid's blocks. Three passes over global memory took 124 us; four CTAs per SM are 2.4 us faster than
// five, at whose registers the quotients spill, and 11 faster than three.
constexpr int CP4_THREADS = 256, CP4_CTAS = 4;
template <int D>
__global__ void __launch_bounds__(CP4_THREADS, CP4_CTAS) cp_prefill4_kernel(const float* __restrict__ kv,
                                                                            const float* __restrict__ score,
                                                                            const float* __restrict__ ape, CompFinish f,
                                                                            CompGeom p, int nblk) {
    constexpr int WPB = D / 64, GROUPS = CP4_THREADS / 32 / WPB, CD = 2 * D;   // warps per block, blocks per CTA and step
    constexpr int NV = D == 512 ? 1 : 2;                // the norm's partial sums a warp takes
    __shared__ float s_red[8 * GROUPS];
    __shared__ __align__(16) float s_row[GROUPS * D];
    __shared__ __align__(16) float bias[8][D];          // row j: the positional bias entry j adds to its scores
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = warp / WPB;
    const int e = ((warp - group * WPB) * 32 + lane) * 2;
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    for (int i = tid * 4; i < 8 * D; i += CP4_THREADS * 4) {
        const int j = i / D, c = i - j * D;
        *reinterpret_cast<float4*>(&bias[j][c]) = *reinterpret_cast<const float4*>(ape + (size_t)(j & 3) * CD + (j >> 2) * D + c);
    }
    const float2 gain = *reinterpret_cast<const float2*>(f.norm + e);
    __syncthreads();
    float* my = s_row + group * D;
    // whole groups of the CTA step together (the norm's barriers); a group past the end works on the last block and stores nothing
    for (int b0 = blockIdx.x * GROUPS; b0 < nblk; b0 += gridDim.x * GROUPS) {
        const bool live = b0 + group < nblk;
        const int b = live ? b0 + group : nblk - 1;
        float2 sc[8], kx[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {                  // entry j: row j of block b - 1 (first half), row j - 4 of block b (second)
            const int sb = j < 4 ? max(b - 1, 0) : b;  // (block 0 has no predecessor: its first four are not used)
            const size_t src = (size_t)(sb * 4 + (j & 3)) * CD + (j >> 2) * D + e;
            sc[j] = *reinterpret_cast<const float2*>(score + src);
            kx[j] = *reinterpret_cast<const float2*>(kv + src);
        }
        float2 freq = make_float2(0.f, 0.f);
        const int r0 = e - (D - p.rd);                 // place in the rotated tail (rd is even)
        if (r0 >= 0) freq = *reinterpret_cast<const float2*>(f.freqs + (size_t)(b * 4) * p.rd + r0);
        const int j0 = b > 0 ? 0 : 4;
        float row[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float x[8], mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                x[j] = (c ? sc[j].y : sc[j].x) + bias[j][e + c];
                if (j >= j0) mx = fmaxf(mx, x[j]);
            }
            float o = 0.0f;
            if (isfinite(mx)) {
                float sum = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; ++j) if (j >= j0) { x[j] = expf(x[j] - mx); sum += x[j]; }
#pragma unroll
                for (int j = 0; j < 8; ++j) if (j >= j0) o += (c ? kx[j].y : kx[j].x) * (x[j] / sum);
            }
            row[c] = v4_rbf16(o);
        }
        *reinterpret_cast<float2*>(my + e) = make_float2(row[0], row[1]);
        __syncthreads();
        const int w = warp - group * WPB;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int t = (v * WPB + w) * 32 + lane;
            float part = my[t] * my[t];
            if (D == 512) part += my[t + 256] * my[t + 256];
            part = rv_warp_sum(part);
            if (lane == 0) s_red[group * 8 + v * WPB + w] = part;
        }
        __syncthreads();                               // (the row is written again behind this, the sums behind the next)
        float part = 0.0f;
#pragma unroll
        for (int i = 0; i < NV * WPB; ++i) part += s_red[group * 8 + i];
        const float rs = 1.0f / sqrtf(part / (float)D + p.eps);
        row[0] = v4_rbf16(gain.x * (row[0] * rs));
        row[1] = v4_rbf16(gain.y * (row[1] * rs));
        if (r0 >= 0) {
            const float a = row[0], c = row[1];
            row[0] = v4_rbf16(__fsub_rn(__fmul_rn(a, freq.x), __fmul_rn(c, freq.y)));
            row[1] = v4_rbf16(__fadd_rn(__fmul_rn(a, freq.y), __fmul_rn(c, freq.x)));
        }
        if (live) *reinterpret_cast<float2*>(f.out + (size_t)b * D + e) = make_float2(row[0], row[1]);
    }
}

__global__ void __launch_bounds__(CP_THREADS) cp_deposit_kernel(const float* __restrict__ kv,
                                                                const float* __restrict__ score,
                                                                const float* __restrict__ ape, float* kv_state,
                                                                float* score_state, CompGeom p, int s, int slot0) {
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    const int remainder = s % p.ratio, cutoff = s - remainder, overlap = p.coff == 2;
    const int state_off = overlap ? p.ratio : 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x, tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (overlap && cutoff >= p.ratio) {   // the last full block's rows become the overlap half
        const size_t n = (size_t)p.ratio * p.cd;
        for (size_t i = tid; i < n; i += stride) {
            const size_t src = (size_t)(cutoff - p.ratio) * p.cd + i;
            kv_state[i] = kv[src];
            score_state[i] = score[src] + ape[i];
        }
    }
    if (remainder > 0) {                  // the open block's rows, from slot0 on
        const size_t n = (size_t)remainder * p.cd, dst0 = (size_t)(state_off + slot0) * p.cd;
        for (size_t i = tid; i < n; i += stride) {
            const size_t src = (size_t)cutoff * p.cd + i;
            kv_state[dst0 + i] = kv[src];
            score_state[dst0 + i] = score[src] + ape[(size_t)slot0 * p.cd + i];
        }
    }
}

__global__ void __launch_bounds__(CP_THREADS) cp_decode_kernel(float* kv_state, float* score_state, CompFinish f,
                                                               CompGeom p, int start_pos) {
    __shared__ float red[CP_THREADS / 32];
    cp_pool_finish(CpState{kv_state, score_state}, f.norm, f.freqs, f.out, p, start_pos, red);
}

// Batched decode step: one CTA per sequence. cache row = cache + (b * cache_rows + cache_row0 + block) * d (bf16).
__global__ void __launch_bounds__(CP_THREADS) cp_step_kernel(CompGeom p, const int32_t* __restrict__ pos,
                                                             const float* __restrict__ kv_proj,
                                                             const float* __restrict__ score_proj,
                                                             const float* __restrict__ ape, float* kv_state,
                                                             float* score_state, const float* __restrict__ norm,
                                                             const float* __restrict__ freqs, int rotate,
                                                             uint16_t* __restrict__ cache, int cache_rows,
                                                             int cache_row0, float* __restrict__ prequant,
                                                             uint8_t* __restrict__ packed,
                                                             uint32_t* __restrict__ packed_exp) {
    extern __shared__ __align__(16) float cp_row[];   // [d]
    __shared__ float red[CP_THREADS / 32];
    __shared__ uint32_t exp_word;
    __shared__ int row_lo, row_hi;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sp = pos[b], slot = sp % p.ratio, d = p.d;
    const size_t st_n = (size_t)p.ents * p.cd;
    CpState st{kv_state + (size_t)b * st_n, score_state + (size_t)b * st_n};
    const size_t dst = (size_t)((p.coff == 2 ? p.ratio : 0) + slot) * p.cd;
    for (int e = tid; e < p.cd; e += CP_THREADS) {
        st.kv[dst + e] = kv_proj[(size_t)b * p.cd + e];
        st.score[dst + e] = score_proj[(size_t)b * p.cd + e] + ape[(size_t)slot * p.cd + e];
    }
    if ((sp + 1) % p.ratio != 0) return;   // the block is still open
    __syncthreads();
    cp_pool_finish(st, norm, freqs, cp_row, p, sp, red);
    if (prequant) for (int e = tid; e < d; e += CP_THREADS) prequant[(size_t)b * d + e] = cp_row[e];
    if (rotate) {
        // the spread of blockindex.hip:97-138 on the row in shared memory
        for (int h = 1; h < d; h <<= 1) {
            for (int t = tid; t < (d >> 1); t += CP_THREADS) {
                const int j = 2 * t - (t & (h - 1));
                const float a = cp_row[j], c = cp_row[j + h];
                cp_row[j] = __fadd_rn(a, c);
                cp_row[j + h] = __fsub_rn(a, c);
            }
            __syncthreads();
        }
        const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)d));
        for (int i = tid; i < d; i += CP_THREADS) cp_row[i] = v4_rbf16(__fmul_rn(cp_row[i], scale));
        __syncthreads();
        const float floor_ = __fmul_rn(V4_FP4_MAX, __uint_as_float(1u << 23));
        for (int blk = warp; blk < d / 32; blk += CP_THREADS / 32) {
            const float v = cp_row[blk * 32 + lane];
            const float s = v4_round_scale(fmaxf(rv_warp_max(fabsf(v)), floor_));
            float q = __fdiv_rn(v, s);
            q = q < -V4_FP4_MAX ? -V4_FP4_MAX : (q > V4_FP4_MAX ? V4_FP4_MAX : q);
            cp_row[blk * 32 + lane] = __fmul_rn(v4_e2m1_roundtrip(q), s);
        }
    } else {
        // fp8 block-64 on the dims that were not rotated (crates/oracles/src/v4oracle/compress.rs:235-247)
        for (int blk = warp; blk < (d - p.rd) / 64; blk += CP_THREADS / 32) cp_act_quant_block(cp_row + blk * 64, cp_row + blk * 64, 64);
    }
    if (tid == 0) { exp_word = 0u; row_lo = 1000; row_hi = -1000; }
    __syncthreads();
    uint16_t* out = cache + ((size_t)b * cache_rows + cache_row0 + sp / p.ratio) * d;
    for (int e = tid; e < d; e += CP_THREADS) out[e] = rv_f32_to_bf16(cp_row[e]);
    if (packed) {
        // the scorer's second form of the same row (d == 128, cache_rows rows per sequence): int8 multiples of the row's
        // unit 2^(pmin - 130), pmin = the smallest biased exponent any non-empty block's largest magnitude has; the
        // row's word holds pmin, 0 for an all-zero row, 0xff when the row is not of that form (blocks more than 3
        // binades apart, magnitudes outside 2^-40 .. 2^40)
        const size_t prow = (size_t)b * cache_rows + cache_row0 + sp / p.ratio;
        float v = 0.0f;
        if (warp < 4) {
            v = rv_bf16_to_f32(rv_f32_to_bf16(cp_row[warp * 32 + lane]));
            int pb = (int)((__float_as_uint(v) >> 23) & 0xffu);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) pb = max(pb, __shfl_xor_sync(0xffffffffu, pb, o));
            if (lane == 0 && pb > 0) { atomicMin(&row_lo, pb); atomicMax(&row_hi, pb); }
        }
        __syncthreads();
        const int lo = row_lo, hi = row_hi;
        const bool form = hi < lo || (lo >= 87 && hi <= 167 && hi - lo <= 3);
        if (warp < 4) {
            const float x = (form && hi >= lo) ? v * __int_as_float((257 - lo) << 23) : 0.0f;
            const int m = __float2int_rn(x);
            bool ok = form && (float)m == x && (hi >= lo || (__float_as_uint(v) & 0x7fffffffu) == 0);
            ok = __all_sync(0xffffffffu, ok);
            packed[prow * 128 + warp * 32 + lane] = (uint8_t)(m & 0xff);
            if (lane == 0 && !ok) atomicOr(&exp_word, 1u);
        }
        __syncthreads();
        if (tid == 0) packed_exp[prow] = exp_word ? 0xffu : (hi >= lo ? (uint32_t)lo : 0u);
    }
}

// The same for the overlapping ratio-4 compressor with d = 128, 256 or 512 (what both compressors of a layer are), one or two
// compressors and the ring write of a decode token in ONE launch: 512 / d sequences per CTA, a thread owns two features of
// one sequence, so deposit, pooling and the move of the overlap half need no exchange - a closing block's loads (10 rows'
// worth, the token's own row comes from the projections) are all in flight at once. Values and their order are those of the
// kernel above, the norm's partial sums included (they meet in shared memory in the order of a 256-thread CTA). Bound by
// latency: two dependent trips to memory; 128 sequences of d 512 14.4 -> 6.9 us (d 128: 10.3 -> 5.8).
struct CpStepJob {
    const float* kv_proj; const float* score_proj; const float* ape; float* kv_state; float* score_state;
    const float* norm; const float* freqs; uint16_t* cache; float* prequant; uint8_t* packed; uint32_t* packed_exp;
    float eps; int d, rd, rotate, cache_rows, cache_row0;
    int cta_end;              // the job's CTAs end here
};
struct CpStepArgs {
    CpStepJob job[2]; const int32_t* pos; int n_jobs, n_seqs;
    const uint16_t* entry; uint16_t* ring; size_t ring_rows; int window, ring_d;   // ring write: behind the jobs' CTAs
};

template <int D>
__device__ __forceinline__ void cp_step4(const CpStepJob& J, const int32_t* __restrict__ pos, int cta, int n_seqs, float* s_row, float* s_red) {
    constexpr int WPS = D / 64, SEQS = 8 / WPS, CD = 2 * D, NV = D == 512 ? 1 : 2;   // warps per sequence, sequences per CTA
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = warp / WPS, w = warp - grp * WPS;
    const int b = cta * SEQS + grp, e = (w * 32 + lane) * 2;
    const bool mine = b < n_seqs;
    const int sp = mine ? pos[b] : 0, slot = sp & 3;
    const bool closing = mine && slot == 3;
    float* kv = J.kv_state + (size_t)(mine ? b : 0) * 8 * CD;
    float* sc = J.score_state + (size_t)(mine ? b : 0) * 8 * CD;
    auto ld = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
    auto st = [](float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; };
    float2 dk[2], ds[2];      // the token's row, both halves
    float2 x[8], k[8], x0[3], k0[3];
    if (mine) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            dk[h] = ld(J.kv_proj + (size_t)b * CD + h * D + e);
            const float2 s = ld(J.score_proj + (size_t)b * CD + h * D + e), a = ld(J.ape + (size_t)slot * CD + h * D + e);
            ds[h] = make_float2(s.x + a.x, s.y + a.y);
        }
    }
    if (closing) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { x[j] = ld(sc + j * CD + e); k[j] = ld(kv + j * CD + e); }
#pragma unroll
        for (int j = 4; j < 7; ++j) { x[j] = ld(sc + j * CD + D + e); k[j] = ld(kv + j * CD + D + e); x0[j - 4] = ld(sc + j * CD + e); k0[j - 4] = ld(kv + j * CD + e); }
    }
    if (mine) {
#pragma unroll
        for (int h = 0; h < 2; ++h) { st(kv + (4 + slot) * CD + h * D + e, dk[h]); st(sc + (4 + slot) * CD + h * D + e, ds[h]); }
    }
    float row[2] = {0.0f, 0.0f};
    float* my = s_row + grp * D;
    if (closing) {
        x[7] = ds[1]; k[7] = dk[1];
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // the overlap half moves down
            st(sc + j * CD + e, j < 3 ? x0[j] : ds[0]); st(kv + j * CD + e, j < 3 ? k0[j] : dk[0]);
            st(sc + j * CD + D + e, x[4 + j]); st(kv + j * CD + D + e, k[4 + j]);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float v[8], mx = -INFINITY, o = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) { v[j] = c ? x[j].y : x[j].x; mx = fmaxf(mx, v[j]); }
            if (isfinite(mx)) {
                float sum = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; ++j) { v[j] = expf(v[j] - mx); sum += v[j]; }
#pragma unroll
                for (int j = 0; j < 8; ++j) o += (c ? k[j].y : k[j].x) * (v[j] / sum);
            }
            row[c] = v4_rbf16(o);
        }
        st(my + e, make_float2(row[0], row[1]));
    }
    __syncthreads();
    if (closing) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int t = (v * WPS + w) * 32 + lane;
            float part = 0.0f;
            part += my[t] * my[t];
            if (D == 512) part += my[t + 256] * my[t + 256];
            part = rv_warp_sum(part);
            if (lane == 0) s_red[grp * 8 + v * WPS + w] = part;
        }
    }
    __syncthreads();
    if (closing) {
        float t = 0.0f;
#pragma unroll
        for (int i = 0; i < NV * WPS; ++i) t += s_red[grp * 8 + i];
        const float rs = 1.0f / sqrtf(t / (float)D + J.eps);
        const float2 gain = ld(J.norm + e);
        row[0] = v4_rbf16(gain.x * (row[0] * rs));
        row[1] = v4_rbf16(gain.y * (row[1] * rs));
        const int r0 = e - (D - J.rd);
        if (r0 >= 0) {
            const float c = J.freqs[(size_t)(sp - 3) * J.rd + r0], sn = J.freqs[(size_t)(sp - 3) * J.rd + r0 + 1];
            const float a = row[0], z = row[1];
            row[0] = v4_rbf16(__fsub_rn(__fmul_rn(a, c), __fmul_rn(z, sn)));
            row[1] = v4_rbf16(__fadd_rn(__fmul_rn(a, sn), __fmul_rn(z, c)));
        }
        if (J.prequant) st(J.prequant + (size_t)b * D + e, make_float2(row[0], row[1]));
    }
    const size_t orow = (size_t)(mine ? b : 0) * J.cache_rows + J.cache_row0 + (sp >> 2);
    if (!J.rotate) {
        if (closing) {
            if (w * 64 < D - J.rd) {   // fp8 block-64 on the dims that were not rotated: a block is a warp
                const float amax = fmaxf(1e-4f, rv_warp_max(fmaxf(fabsf(row[0]), fabsf(row[1]))));
                float inv;
                const float s = cp_f8_scale(amax, inv);
                row[0] = cp_f8_roundtrip(row[0], s, inv);
                row[1] = cp_f8_roundtrip(row[1], s, inv);
            }
            *reinterpret_cast<uint32_t*>(J.cache + orow * D + e) = (uint32_t)rv_f32_to_bf16(row[0]) | ((uint32_t)rv_f32_to_bf16(row[1]) << 16);
        }
        return;
    }
    if constexpr (D <= V4_ROT_MAX) {
        if (closing) st(my + e, make_float2(row[0], row[1]));
        __syncthreads();
        if (!closing || w != 0) return;
        constexpr int E = D / 32;
        float v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = my[lane * E + j];
        v4_spread_row<E>(v, lane);
        uint32_t o[E / 2];
#pragma unroll
        for (int j = 0; j < E; j += 2) o[j / 2] = (uint32_t)rv_f32_to_bf16(v[j]) | ((uint32_t)rv_f32_to_bf16(v[j + 1]) << 16);
#pragma unroll
        for (int j = 0; j < E / 2; ++j) reinterpret_cast<uint32_t*>(J.cache + orow * D + lane * E)[j] = o[j];
        if constexpr (D == 128) if (J.packed) {
            // the scorer's second form of the same row: int8 multiples of the row's unit 2^(pmin - 130), pmin = the smallest
            // biased exponent any non-empty block's largest magnitude has; the row's word holds pmin, 0 for an all-zero
            // row, 0xff when the row is not of that form (blocks more than 3 binades apart, magnitudes outside 2^-40 .. 2^40)
            int pb = 0;
#pragma unroll
            for (int j = 0; j < E; ++j) { v[j] = rv_bf16_to_f32(rv_f32_to_bf16(v[j])); pb = max(pb, (int)((__float_as_uint(v[j]) >> 23) & 0xffu)); }
#pragma unroll
            for (int q = 1; q < 8; q <<= 1) pb = max(pb, __shfl_xor_sync(0xffffffffu, pb, q));
            int lo = pb > 0 ? pb : 1000, hi = pb > 0 ? pb : -1000;
#pragma unroll
            for (int q = 8; q < 32; q <<= 1) { lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, q)); hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, q)); }
            const bool form = hi < lo || (lo >= 87 && hi <= 167 && hi - lo <= 3);
            bool ok = form;
            uint32_t bytes = 0;
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const float xq = (form && hi >= lo) ? v[j] * __int_as_float((257 - lo) << 23) : 0.0f;
                const int m = __float2int_rn(xq);
                ok = ok && (float)m == xq && (hi >= lo || (__float_as_uint(v[j]) & 0x7fffffffu) == 0);
                bytes |= (uint32_t)(m & 0xff) << (8 * j);
            }
            ok = __all_sync(0xffffffffu, ok);
            reinterpret_cast<uint32_t*>(J.packed + orow * 128)[lane] = bytes;
            if (lane == 0) J.packed_exp[orow] = ok ? (hi >= lo ? (uint32_t)lo : 0u) : 0xffu;
        }
    }
}

__global__ void __launch_bounds__(CP_THREADS) cp_step4_kernel(CpStepArgs A) {
    __shared__ __align__(16) float s_row[512];
    __shared__ float s_red[64];
    // the wait comes first: whatever is launched behind this kernel then starts after everything in front of it is complete
    rv_grid_dep_wait();
    rv_grid_dep_trigger();
    int cta = (int)blockIdx.x, first = 0;
    for (int j = 0; j < A.n_jobs; ++j) {
        const CpStepJob& J = A.job[j];
        if (cta < J.cta_end) {
            if (J.d == 512) cp_step4<512>(J, A.pos, cta - first, A.n_seqs, s_row, s_red);
            else if (J.d == 256) cp_step4<256>(J, A.pos, cta - first, A.n_seqs, s_row, s_red);
            else cp_step4<128>(J, A.pos, cta - first, A.n_seqs, s_row, s_red);
            return;
        }
        first = J.cta_end;
    }
    // the token's window entry into ring slot pos % window: a warp per sequence
    const int b = (cta - first) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= A.n_seqs) return;
    const int r = A.pos[b] % A.window, slot = r < 0 ? r + A.window : r;
    const uint16_t* src = A.entry + (size_t)b * A.ring_d;
    uint16_t* dst = A.ring + ((size_t)b * A.ring_rows + slot) * A.ring_d;
    if (A.ring_d % 8 == 0 && (((uintptr_t)A.entry | (uintptr_t)A.ring) & 15) == 0) {
        for (int i = lane; i < A.ring_d / 8; i += 32) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    } else {
        for (int i = lane; i < A.ring_d; i += 32) dst[i] = src[i];
    }
}

static int cp_guard(const CompGeom& p) {
    if (p.ratio <= 1 || p.d <= 0 || p.rd <= 0 || p.coff < 1 || p.coff > 2) return 1001;
    if (p.rd > p.d || (p.rd & 1)) return 1002;
    if (p.cd != p.coff * p.d || p.ents != p.coff * p.ratio) return 1003;
    if (p.ents > CP_ENTS_MAX) return 1004;
    if ((p.coff == 2) != (p.ratio == 4)) return 1010;
    return 0;
}
}  // namespace

RIVOLI_API int rivoli_act_quant_f8_prefix(const float* src, float* dst, int rows, int row_stride, int n, int block,
                                          void* stream) {
    if (rows <= 0 || n <= 0 || block <= 0 || row_stride < n) return 1001;
    if (src != dst && n != row_stride) return 1002;   // the untouched tail of a row only survives in place
    if (n % block) return 1004;
    const size_t total = (size_t)rows * (size_t)(n / block);
    rv_drain_error();
    if (block == 64 && row_stride % 4 == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0) {
        const size_t threads = (size_t)rows * (size_t)(n / 4);
        rv_launch_dependent(cp_act_quant_f8_prefix64_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, (cudaStream_t)stream,
                            src, dst, rows, row_stride, n);
        return rv_launch_status();
    }
    cp_act_quant_f8_prefix_kernel<<<(unsigned)((total + 7) / 8), 256, 0, (cudaStream_t)stream>>>(src, dst, rows, row_stride,
                                                                                                n, block);
    return rv_launch_status();
}

RIVOLI_API int rivoli_kv_compress_deposit(const float* kv, const float* score, const float* ape, float* kv_state,
                                          float* score_state, const CompGeom* pp, int s, int slot0, void* stream) {
    if (!pp) return 1000;
    const CompGeom p = *pp;
    if (int g = cp_guard(p)) return g;
    if (s <= 0) return 1005;
    if (slot0 < 0 || slot0 + s % p.ratio > p.ratio) return 1008;
    const int rem = s % p.ratio;
    const size_t n = (size_t)(p.ratio > rem ? p.ratio : rem) * p.cd;
    rv_drain_error();
    rv_launch_dependent(cp_deposit_kernel, dim3((unsigned)((n + CP_THREADS - 1) / CP_THREADS)), dim3(CP_THREADS), 0, (cudaStream_t)stream,
                        kv, score, ape, kv_state, score_state, p, s, slot0);
    return rv_launch_status();
}

RIVOLI_API int rivoli_kv_compress_prefill(const float* kv, const float* score, const float* ape, const CompFinish* ff,
                                          const CompGeom* pp, int nblk, void* stream) {
    if (!pp || !ff) return 1000;
    const CompGeom p = *pp;
    if (int g = cp_guard(p)) return g;
    if (nblk <= 0) return 1006;
    cudaStream_t st = (cudaStream_t)stream;
    rv_drain_error();
    const bool wide = (((uintptr_t)kv | (uintptr_t)score | (uintptr_t)ape | (uintptr_t)ff->norm | (uintptr_t)ff->freqs | (uintptr_t)ff->out) & 15) == 0;
    if (p.ratio == 4 && wide && (p.d == 128 || p.d == 256 || p.d == 512)) {
        const int groups = CP4_THREADS / (p.d / 2), most = CP4_CTAS * rv_sm_count();
        const int ctas = (nblk + groups - 1) / groups;
        const dim3 grid((unsigned)(ctas < most ? ctas : most));
        if (p.d == 512) rv_launch_dependent(cp_prefill4_kernel<512>, grid, dim3(CP4_THREADS), 0, st, kv, score, ape, *ff, p, nblk);
        else if (p.d == 256) rv_launch_dependent(cp_prefill4_kernel<256>, grid, dim3(CP4_THREADS), 0, st, kv, score, ape, *ff, p, nblk);
        else rv_launch_dependent(cp_prefill4_kernel<128>, grid, dim3(CP4_THREADS), 0, st, kv, score, ape, *ff, p, nblk);
        return rv_launch_status();
    }
    cp_prefill_kernel<<<(unsigned)nblk, CP_THREADS, 0, st>>>(kv, score, ape, *ff, p);
    return rv_launch_status();
}

RIVOLI_API int rivoli_kv_compress_decode(float* kv_state, float* score_state, const CompFinish* ff, const CompGeom* pp,
                                         int start_pos, void* stream) {
    if (!pp || !ff) return 1000;
    const CompGeom p = *pp;
    if (int g = cp_guard(p)) return g;
    if (start_pos <= 0) return 1007;                 // position 0 belongs to the prefill arm
    if ((start_pos + 1) % p.ratio != 0) return 1009; // the block has not closed
    rv_drain_error();
    cp_decode_kernel<<<1, CP_THREADS, 0, (cudaStream_t)stream>>>(kv_state, score_state, *ff, p, start_pos);
    return rv_launch_status();
}

static int cp_step_guard(const CompGeom& p, int rotate, int cache_rows, int cache_row0, const void* packed, const void* packed_exp) {
    if (int g = cp_guard(p)) return g;
    if (cache_rows <= 0 || cache_row0 < 0) return 1001;
    if (rotate && (p.d > V4_ROT_MAX || (p.d & (p.d - 1)) || p.d % 32)) return 1002;
    if (!rotate && (p.d - p.rd) % 64) return 1004;
    if ((packed != nullptr) != (packed_exp != nullptr)) return 1001;
    if (packed && (!rotate || p.d != 128)) return 1002;   // the packed form is the indexer's: spread rows of width 128
    if ((size_t)p.d * 4 > 48 * 1024) return 1002;
    return 0;
}

// The step takes the two-features-per-thread kernel (else: one CTA per sequence, any geometry).
static bool cp_step4_ok(const CompGeom& p, const CompStep& c, int rotate) {
    return p.ratio == 4 && (p.d == 128 || p.d == 256 || (p.d == 512 && !rotate)) &&
           (((uintptr_t)c.kv_proj | (uintptr_t)c.score_proj | (uintptr_t)c.ape | (uintptr_t)c.kv_state | (uintptr_t)c.score_state |
             (uintptr_t)c.norm | (uintptr_t)c.prequant) & 7) == 0 && (((uintptr_t)c.cache | (uintptr_t)c.packed) & 3) == 0;
}

static CpStepJob cp_step4_job(const CompGeom& p, const CompStep& c, int n_seqs, int first_cta) {
    const int seqs = 512 / p.d;
    return CpStepJob{c.kv_proj, c.score_proj, c.ape, c.kv_state, c.score_state, c.norm, c.freqs, c.cache, c.prequant, c.packed,
                     c.packed_exp, p.eps, p.d, p.rd, c.rotate, c.cache_rows, c.cache_row0, first_cta + (n_seqs + seqs - 1) / seqs};
}

static int cp_step_launch(const CompGeom& p, int n_seqs, const int32_t* pos, const CompStep& c, cudaStream_t st) {
    if (cp_step4_ok(p, c, c.rotate)) {
        CpStepArgs a{};
        a.job[0] = cp_step4_job(p, c, n_seqs, 0);
        a.pos = pos; a.n_jobs = 1; a.n_seqs = n_seqs;
        rv_launch_dependent(cp_step4_kernel, dim3((unsigned)a.job[0].cta_end), dim3(CP_THREADS), 0, st, a);
    } else {
        cp_step_kernel<<<(unsigned)n_seqs, CP_THREADS, (size_t)p.d * 4, st>>>(
            p, pos, c.kv_proj, c.score_proj, c.ape, c.kv_state, c.score_state, c.norm, c.freqs, c.rotate, c.cache, c.cache_rows,
            c.cache_row0, c.prequant, c.packed, c.packed_exp);
    }
    return rv_launch_status();
}

RIVOLI_API int rivoli_v4_compress_step_bf16(const CompGeom* pp, int n_seqs, const int32_t* pos, const float* kv_proj,
                                            const float* score_proj, const float* ape, float* kv_state,
                                            float* score_state, const float* norm, const float* freqs, int rotate,
                                            uint16_t* cache, int cache_rows, int cache_row0, float* prequant,
                                            unsigned char* packed, uint32_t* packed_exp, void* stream) {
    if (!pp) return 1000;
    const CompGeom p = *pp;
    if (int g = cp_guard(p)) return g;
    if (n_seqs <= 0) return 1001;
    if (int g = cp_step_guard(p, rotate, cache_rows, cache_row0, packed, packed_exp)) return g;
    rv_drain_error();
    return cp_step_launch(p, n_seqs, pos, CompStep{kv_proj, score_proj, ape, kv_state, score_state, norm, freqs, cache, prequant,
                                                   packed, packed_exp, rotate, cache_rows, cache_row0}, (cudaStream_t)stream);
}

int rivoli_v4_sparse_attend_launch(const V4Geom* g, int n_seqs, const uint16_t* q, const uint16_t* kv_cache, const float* sink,
                                   const int32_t* sel, int cols, uint16_t* out, int force_simt, int q_early, cudaStream_t st);

RIVOLI_API int rivoli_v4_token_step_bf16(const V4Geom* g, int n_seqs, const int32_t* pos, const uint16_t* kv_entry,
                                         const CompGeom* attn, const CompStep* attn_step, const CompGeom* index,
                                         const CompStep* index_step, const uint16_t* q, const uint16_t* index_q,
                                         const float* index_w, const float* sink, int32_t* sel, void* scratch, uint16_t* out,
                                         void* stream) {
    if (!attn || !index || !attn_step || !index_step) return 1000;
    if (int rc = v4_check_geom(g, n_seqs)) return rc;
    if (!pos || !kv_entry) return 1001;
    for (int j = 0; j < 2; ++j) {
        const CompStep& c = j ? *attn_step : *index_step;
        if (int e = cp_step_guard(j ? *attn : *index, c.rotate, c.cache_rows, c.cache_row0, c.packed, c.packed_exp)) return e;
    }
    if (index->d != g->index_dim || index_step->cache_rows != g->max_comp || index_step->cache_row0 != 0) return 1003;
    if (attn->d != g->head_dim || attn_step->cache_rows != g->window + g->max_comp || attn_step->cache_row0 < g->window) return 1003;
    cudaStream_t st = (cudaStream_t)stream;
    rv_drain_error();
    CpStepArgs a{};
    a.pos = pos; a.n_seqs = n_seqs;
    a.entry = kv_entry; a.ring = attn_step->cache; a.ring_rows = (size_t)attn_step->cache_rows; a.window = g->window; a.ring_d = g->head_dim;
    int ctas = 0;
    for (int j = 0; j < 2; ++j) {   // what the joint launch does not take goes in front of it, on its own
        const CompGeom& p = j ? *attn : *index;
        const CompStep& c = j ? *attn_step : *index_step;
        if (!cp_step4_ok(p, c, c.rotate)) {
            if (int e = cp_step_launch(p, n_seqs, pos, c, st)) return e;
        } else {
            a.job[a.n_jobs] = cp_step4_job(p, c, n_seqs, ctas);
            ctas = a.job[a.n_jobs++].cta_end;
        }
    }
    rv_launch_dependent(cp_step4_kernel, dim3((unsigned)(ctas + (n_seqs + 7) / 8)), dim3(CP_THREADS), 0, st, a);
    if (int e = rv_launch_status()) return e;
    if (int e = rivoli_v4_select_blocks_bf16(g, n_seqs, pos, index_q, index_w, index_step->cache, index_step->packed,
                                             index_step->packed_exp, sel, scratch, 0, stream))
        return e;
    return rivoli_v4_sparse_attend_launch(g, n_seqs, q, attn_step->cache, sink, sel, g->window + g->index_topk, out, 0, 1, st);
}
