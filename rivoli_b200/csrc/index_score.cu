// Lightning-indexer scores on CUDA cores, in the reference's exact arithmetic order.
//
//   rivoli_index_score        : the reference operator (f32 q, bf16 key slab, one sequence;
//                               crates/backend/kernels/indexer.hip:60-93).
//   rivoli_index_score_paged  : batched, paged, fp8 keys and fp8 q. Bit-reproducible:
//                               the code dot is a left fold over d (each product of two e4m3
//                               values is exact in f32, so fma(q,k,acc) IS round(acc + q*k)),
//                               scales are applied to the finished dot, heads fold ascending.
//
// The paged kernel is a register-tiled f32 "GEMM" (tokens x heads x dims) whose k-loop is
// sequential per output, which is what keeps the fold order fixed. It is the definitional
// path: ~62 FLOP per key byte means CUDA cores cannot keep up with HBM here; the
// tensor-core scorer uses this kernel's arithmetic only for the tokens near the top-k cut.
#include "codec.cuh"
#include "common.cuh"

// ------------------------------------------------------------------------------------------
// Reference layout. One warp per cached token; lanes split hd; heads fold in list order on
// lane 0 so the per-token sum has the reference's head order. The per-head dot is a
// shuffle-tree sum (the reference's own kernel also differs from its host fold here, and
// holds the comparison to 1e-5 relative: crates/engine/tests/indexer_kernel.rs:340-356).
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
index_score_slab_kernel(const float* __restrict__ q, const float* __restrict__ w,
                        const unsigned short* __restrict__ kcache, const unsigned int* __restrict__ heads,
                        int nt, int nact, int hd, float wscale, float dscale, float* __restrict__ scores) {
    extern __shared__ float kf[];  // [8 warps][hd]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * 8 + warp;
    if (t >= nt) return;
    float* krow = kf + (size_t)warp * hd;
    for (int i = lane; i < hd; i += 32) krow[i] = rv_bf16_to_f32(kcache[(size_t)t * hd + i]);
    __syncwarp();
    float acc = 0.0f;
    for (int a = 0; a < nact; ++a) {
        const int h = heads ? (int)heads[a] : a;
        const float* qh = q + (size_t)h * hd;
        float part = 0.0f;
        for (int i = lane; i < hd; i += 32) part = fmaf(qh[i], krow[i], part);
        part = rv_warp_sum(part);
        const float r = fmaxf(__fmul_rn(part, dscale), 0.0f);
        acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(w[h], wscale), r));
    }
    if (lane == 0) scores[t] = acc;
}

// ------------------------------------------------------------------------------------------
// The same scores, bit for bit, for key rows of 128 values and up to 64 heads: a register tile of 2 tokens x 4 heads per
// thread. The kernel above spends 5 shuffles and as many additions per (token, head) in every lane on the reduction of
// 4 products a lane. Here one thread evaluates the whole reduction tree of a (token, head) itself - "lane" l's partial is
// the fold over the dims l, l + 32, l + 64, l + 96, and partials meet in the butterfly's order (16, 8, 4, 2, 1), walked
// depth first with one running sum per level - so an operand read from shared memory serves 2 or 4 products.
// CTA = 64 tokens, 8 warps of 4 heads each (a second pass for more than 32 heads); bound by the multiply-adds and the
// shared-memory reads that feed them. 8,193 tokens x 32 heads: 26.7 -> 12.0 us.
// ------------------------------------------------------------------------------------------
constexpr int SL_TOK = 64, SL_HD = 128, SL_HP = 32, SL_THREADS = 256, SL_HW = SL_HP / (SL_THREADS / 32);   // heads per warp
constexpr int SL_QP = (SL_HP + 1) * 4;   // pitch of a partial's heads (padded: the staging stores spread over the banks)
constexpr int SL_SMEM = (SL_HD * SL_TOK + 32 * SL_QP + SL_HP * SL_TOK) * (int)sizeof(float);

__global__ void __launch_bounds__(SL_THREADS)
index_score_slab128_kernel(const float* __restrict__ q, const float* __restrict__ w,
                           const unsigned short* __restrict__ kcache, const unsigned int* __restrict__ heads,
                           int nt, int nact, float wscale, float dscale, float* __restrict__ scores) {
    extern __shared__ __align__(16) float sl_smem[];
    float2* kT = reinterpret_cast<float2*>(sl_smem);                                   // [dim][lane]: tokens lane and lane + 32
    float4* qs = reinterpret_cast<float4*>(sl_smem + SL_HD * SL_TOK);                  // [partial l][head]: dims l + 32 k
    float* cs = sl_smem + SL_HD * SL_TOK + 32 * SL_QP;                                  // [head][token] contributions
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t0 = blockIdx.x * SL_TOK;
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    {   // keys: a thread takes a quarter of one token's row, all loads in flight, and spreads it over the dims
        constexpr int PART = SL_HD / (SL_THREADS / SL_TOK);
        const int tl = tid & 63, part = tid >> 6, t = t0 + tl;
        uint4 v[PART / 8];
#pragma unroll
        for (int c = 0; c < PART / 8; ++c)
            v[c] = t < nt ? *reinterpret_cast<const uint4*>(kcache + (size_t)t * SL_HD + part * PART + c * 8) : make_uint4(0, 0, 0, 0);
        float* dst = reinterpret_cast<float*>(kT) + (tl & 31) * 2 + (tl >> 5);
#pragma unroll
        for (int c = 0; c < PART / 8; ++c) {
            const uint32_t ww[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                dst[(part * PART + c * 8 + 2 * e) * SL_TOK] = __uint_as_float(ww[e] << 16);
                dst[(part * PART + c * 8 + 2 * e + 1) * SL_TOK] = __uint_as_float(ww[e] & 0xffff0000u);
            }
        }
    }
    float total = 0.0f;                                                                  // of token t0 + tid, heads in order
    for (int h0 = 0; h0 < nact; h0 += SL_HP) {
        __syncthreads();
        for (int e = tid; e < SL_HP * SL_HD; e += SL_THREADS) {
            const int a = e >> 7, d = e & 127;                                           // lanes along a head's row
            const int h = h0 + a < nact ? (heads ? (int)heads[h0 + a] : h0 + a) : -1;
            reinterpret_cast<float*>(qs)[(d & 31) * SL_QP + a * 4 + (d >> 5)] = h >= 0 ? q[(size_t)h * SL_HD + d] : 0.0f;
        }
        __syncthreads();
        float sum[SL_HW][2];
        const float4* qw = qs + warp * SL_HW;
        auto leaf = [&](int l, float (&p)[SL_HW][2]) {                                        // the partials of "lane" l
            float2 k[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) k[e] = kT[(l + 32 * e) * 32 + lane];
#pragma unroll
            for (int h = 0; h < SL_HW; ++h) {
                const float4 qv = qw[l * (SL_QP / 4) + h];
                p[h][0] = fmaf(qv.w, k[3].x, fmaf(qv.z, k[2].x, fmaf(qv.y, k[1].x, fmaf(qv.x, k[0].x, 0.0f))));
                p[h][1] = fmaf(qv.w, k[3].y, fmaf(qv.z, k[2].y, fmaf(qv.y, k[1].y, fmaf(qv.x, k[0].y, 0.0f))));
            }
        };
        float sd[SL_HW][2];
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {                                                    // subtrees l = 0, 2 | 1, 3 of the last two levels
            const int base = (u >> 1) + 2 * (u & 1);
            float sb[SL_HW][2], sc[SL_HW][2];
#pragma unroll
            for (int b4 = 0; b4 < 2; ++b4) {                                             // base, base + 4
#pragma unroll
                for (int a8 = 0; a8 < 2; ++a8) {                                         // + 0, + 8
                    const int l = base + 4 * b4 + 8 * a8;
                    float p0[SL_HW][2], p1[SL_HW][2];
                    leaf(l, p0);
                    leaf(l + 16, p1);
#pragma unroll
                    for (int h = 0; h < SL_HW; ++h)
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            const float a = __fadd_rn(p0[h][t], p1[h][t]);
                            sb[h][t] = a8 == 0 ? a : __fadd_rn(sb[h][t], a);
                        }
                }
#pragma unroll
                for (int h = 0; h < SL_HW; ++h)
#pragma unroll
                    for (int t = 0; t < 2; ++t) sc[h][t] = b4 == 0 ? sb[h][t] : __fadd_rn(sc[h][t], sb[h][t]);
            }
#pragma unroll
            for (int h = 0; h < SL_HW; ++h)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (u & 1) {
                        const float d = __fadd_rn(sd[h][t], sc[h][t]);
                        sum[h][t] = u == 1 ? d : __fadd_rn(sum[h][t], d);
                    } else {
                        sd[h][t] = sc[h][t];
                    }
                }
        }
#pragma unroll
        for (int h = 0; h < SL_HW; ++h) {
            const int a = h0 + warp * SL_HW + h;
            const float wh = a < nact ? __fmul_rn(w[heads ? heads[a] : (unsigned)a], wscale) : 0.0f;
#pragma unroll
            for (int t = 0; t < 2; ++t) cs[(warp * SL_HW + h) * SL_TOK + lane + 32 * t] = __fmul_rn(wh, fmaxf(__fmul_rn(sum[h][t], dscale), 0.0f));
        }
        __syncthreads();
        if (tid < SL_TOK)
            for (int h = 0; h < min(SL_HP, nact - h0); ++h) total = __fadd_rn(total, cs[h * SL_TOK + tid]);
    }
    if (tid < SL_TOK && t0 + tid < nt) scores[t0 + tid] = total;
}

RIVOLI_API int rivoli_index_score(const float* q, const float* w, const unsigned short* kcache,
                                  const unsigned int* heads, int nt, int nh, int nact, int hd,
                                  float wscale, float dscale, float* scores) {
    if (nt <= 0 || nh <= 0 || nact <= 0 || nact > nh || hd <= 0) return 1001;
    // Same bounds the reference's launcher states (block = next pow2 >= nact, <= 1024;
    // staging (hd + block) floats <= 64 KiB), so the same shapes are accepted and rejected.
    int bd = 1;
    while (bd < nact) bd <<= 1;
    if (bd < 32) bd = 32;
    if (bd > 1024) return 1002;
    if (((size_t)hd + bd) * sizeof(float) > 65536) return 1002;
    const size_t smem = (size_t)8 * hd * sizeof(float);
    rv_drain_error();
    if (hd == SL_HD && nact <= 2 * SL_HP && ((uintptr_t)kcache & 15) == 0) {
        rv_allow_smem<index_score_slab128_kernel>(SL_SMEM);
        rv_launch_dependent(index_score_slab128_kernel, dim3((unsigned)((nt + SL_TOK - 1) / SL_TOK)), dim3(SL_THREADS), (size_t)SL_SMEM,
                            (cudaStream_t)0, q, w, kcache, heads, nt, nact, wscale, dscale, scores);
        return rv_launch_status();
    }
    if (smem > 48 * 1024)
        rv_allow_smem<index_score_slab_kernel>(227 * 1024);
    index_score_slab_kernel<<<(nt + 7) / 8, 256, smem>>>(q, w, kcache, heads, nt, nact, hd, wscale, dscale, scores);
    return rv_launch_status();
}

// ------------------------------------------------------------------------------------------
// Paged exact scorer. CTA = 128 threads = 128 tokens of one sequence.
//   thread (tx = tid % 32, ty = tid / 32) owns tokens 4*tx..4*tx+3 and heads ty*HPW..+HPW-1
//   dims are staged 64 at a time: kf[64][128] (token minor) and qf[64][4*HPW] (head minor)
// ------------------------------------------------------------------------------------------
constexpr int IS_TOK = 128;   // tokens per CTA
constexpr int IS_DCH = 64;    // dims per staged chunk

template <int HPW>
__global__ void __launch_bounds__(128)
index_score_paged_kernel(DsaGeom g, const uint8_t* __restrict__ qcodes, const float* __restrict__ qscales,
                         const float* __restrict__ w, const uint8_t* __restrict__ index_pool,
                         const float* __restrict__ index_scale, const int32_t* __restrict__ block_table,
                         const int32_t* __restrict__ seq_len, float* __restrict__ scores, int score_stride) {
    constexpr int NHP = 4 * HPW;  // padded head count
    constexpr int CST = NHP + 1;  // odd pitch of the per-(token, head) contribution tile
    __shared__ __align__(16) float smem[IS_DCH * IS_TOK + IS_DCH * NHP];
    float (*kf)[IS_TOK] = reinterpret_cast<float (*)[IS_TOK]>(smem);
    float (*qf)[NHP] = reinterpret_cast<float (*)[NHP]>(smem + IS_DCH * IS_TOK);
    // After the k-loop both tiles are dead: cs overlays the front, sks sits at the very end.
    float* cs = smem;
    float* sks = smem + IS_DCH * IS_TOK + IS_DCH * NHP - IS_TOK;
    static_assert(IS_TOK * CST <= IS_DCH * IS_TOK + IS_DCH * NHP - IS_TOK, "epilogue tiles overlap");
    const int b = blockIdx.y, t0 = blockIdx.x * IS_TOK, tid = threadIdx.x;
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    const int nt = seq_len[b];
    if (t0 >= nt) return;
    const int nh = g.index_heads, hd = g.index_dim;
    const int tx = tid & 31, ty = tid >> 5;

    // This thread stages token t0 + tid.
    const int t = t0 + tid;
    const uint8_t* krow = nullptr;
    float sk = 0.0f;
    if (t < nt) {
        const int page = block_table[(size_t)b * g.max_pages_per_seq + t / g.page_tokens];
        const size_t r = (size_t)page * g.page_tokens + (t & (g.page_tokens - 1));
        krow = index_pool + r * hd;
        sk = index_scale[r];
    }

    float acc[4][HPW];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < HPW; ++j) acc[i][j] = 0.0f;

    for (int d0 = 0; d0 < hd; d0 += IS_DCH) {
        const int dn = min(IS_DCH, hd - d0);
        __syncthreads();
        // keys: 16 codes at a time from this thread's row
        for (int c = 0; c < dn; c += 16) {
            uint4 p = make_uint4(0, 0, 0, 0);
            if (krow) p = *reinterpret_cast<const uint4*>(krow + d0 + c);
            const uint32_t wv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float2 a = rv_e4m3x2_to_f32x2((uint16_t)(wv[k] & 0xffff));
                float2 bq = rv_e4m3x2_to_f32x2((uint16_t)(wv[k] >> 16));
                kf[c + 4 * k + 0][tid] = a.x; kf[c + 4 * k + 1][tid] = a.y;
                kf[c + 4 * k + 2][tid] = bq.x; kf[c + 4 * k + 3][tid] = bq.y;
            }
        }
        // q: [dn][NHP], zero for padded heads
        for (int e = tid; e < dn * NHP; e += 128) {
            const int d = e / NHP, h = e % NHP;
            float v = 0.0f;
            if (h < nh) v = rv_e4m3_to_f32(qcodes[((size_t)b * nh + h) * hd + d0 + d]);
            qf[d][h] = v;
        }
        __syncthreads();
        for (int d = 0; d < dn; ++d) {
            const float4 kv = *reinterpret_cast<const float4*>(&kf[d][tx * 4]);
            float qv[HPW];
#pragma unroll
            for (int j = 0; j < HPW; j += 2) {
                const float2 q2 = *reinterpret_cast<const float2*>(&qf[d][ty * HPW + j]);
                qv[j] = q2.x; qv[j + 1] = q2.y;
            }
#pragma unroll
            for (int j = 0; j < HPW; ++j) {
                acc[0][j] = fmaf(qv[j], kv.x, acc[0][j]);
                acc[1][j] = fmaf(qv[j], kv.y, acc[1][j]);
                acc[2][j] = fmaf(qv[j], kv.z, acc[2][j]);
                acc[3][j] = fmaf(qv[j], kv.w, acc[3][j]);
            }
        }
    }
    __syncthreads();
    // Per-(token, head) contribution into smem, then a sequential fold over heads.
    sks[tid] = sk;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < HPW; ++j) {
        const int h = ty * HPW + j;
        if (h < nh) {
            const float sq = qscales[(size_t)b * nh + h];
            const float wh = __fmul_rn(w[(size_t)b * nh + h], g.index_wscale);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int tl = tx * 4 + i;
                const float dot = __fmul_rn(__fmul_rn(acc[i][j], sq), sks[tl]);
                float r = __fmul_rn(dot, g.index_dscale);
                r = r > 0.0f ? r : 0.0f;
                cs[tl * CST + h] = __fmul_rn(wh, r);
            }
        }
    }
    __syncthreads();
    if (t < nt) {
        float s = 0.0f;
        for (int h = 0; h < nh; ++h) s = __fadd_rn(s, cs[tid * CST + h]);
        scores[(size_t)b * score_stride + t] = s;
    }
}

RIVOLI_API int rivoli_index_score_paged(const DsaGeom* g, const uint8_t* qcodes, const float* qscales,
                                        const float* w, const uint8_t* index_pool,
                                        const float* index_scale, const int32_t* block_table,
                                        const int32_t* seq_len, int B, float* scores, int score_stride,
                                        void* stream) {
    if (int e = rv_check_geom(g)) return e;
    if (B <= 0 || score_stride <= 0 || !qcodes || !qscales || !w || !index_pool || !index_scale ||
        !block_table || !seq_len || !scores)
        return 1001;
    if ((uintptr_t)index_pool & 15) return 1005;
    if ((long long)score_stride > (long long)g->max_pages_per_seq * g->page_tokens) return 1002;
    dim3 grid((score_stride + IS_TOK - 1) / IS_TOK, B);
    cudaStream_t st = (cudaStream_t)stream;
    rv_drain_error();
#define RV_LAUNCH_IS(HPW)                                                                         \
    rv_launch_dependent(index_score_paged_kernel<HPW>, grid, dim3(128), 0, st, *g, qcodes, qscales, w, \
                        index_pool, index_scale, block_table, seq_len, scores, score_stride)
    if (g->index_heads <= 8) RV_LAUNCH_IS(2);
    else if (g->index_heads <= 16) RV_LAUNCH_IS(4);
    else if (g->index_heads <= 32) RV_LAUNCH_IS(8);
    else RV_LAUNCH_IS(16);
#undef RV_LAUNCH_IS
    return rv_launch_status();
}
