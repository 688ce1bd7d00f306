// MLA decode attention in latent space on CUDA cores (f32 accumulate):
//     out_h = sum_t softmax_t((q_h . [L_t | R_t]) * scale) * L_t
//
//   rivoli_mla_attend             : the reference operator (f32 q, fp8 latent slab with
//                                   per-128 block scales, bf16 roped keys, one sequence;
//                                   crates/backend/kernels/attn.hip:119-308).
//   rivoli_attend_simt_paged_bf16 : the same arithmetic on the paged fp8 pool (bf16 q,
//                                   one scale per token, fp8 roped keys), batched. This is the
//                                   f32 cross-check of the tensor-core kernel and the path
//                                   used for geometries that kernel does not cover.
//
// What bounds it: instruction issue. There are 2 * H * rows * (2 kvl + rope) f32 operations and only a megabyte or two
// of rows, so the work is spread over every SM and the loop holds little but the arithmetic:
//   * a WARP takes AT_HG = 2 heads and a run of rows, two rows per step. Its lanes own the columns (lane l the kvl / 32
//     consecutive latent columns from l * kvl / 32; kvl 384 differs), q and the output sums of the heads stay in registers, and a cached
//     row is decoded once and used for both heads, once as key and once as value. AT_RING rows per warp are in flight as
//     asynchronous copies into the warp's own slots of shared memory (16 bytes per lane and row at kvl 512): loads into
//     registers a step ahead were waited for on the spot, at the register limit (1,700 of 2,900 cycles per step);
//   * products are the packed form (fma.rn.f32x2: two f32 multiply-adds per issued instruction, each rounded as usual);
//   * the four scores of a step (2 rows x 2 heads) are summed over the warp with six shuffles, after which each group
//     of eight lanes holds one of them: one exponential per lane and step;
//   * the sums are rescaled when a score leaves its head's reference maximum AT_LAG behind, and only then;
//   * the rows of a head pair are split over the warps of a CTA and the up to eight CTAs of a thread-block cluster,
//     which merge their (maximum, sum, output) through shared and distributed shared memory (plain loads of mapped
//     addresses): no partials in global memory and no second launch. Two CTAs share an SM, so that a cluster needs four
//     SMs and all clusters of a launch are resident at once.
// A warp resolves the addresses of 32 rows at a time (token -> page -> pool row -> scale), lane by lane.
// Measured at 64 heads x 2,048 of 8,193 rows, one sequence: 23 us; one CTA for all heads per 256 rows (eight
// CTAs), rows dequantised into shared memory and a combine launch took 1,098 us.
#include <cooperative_groups.h>

#include "codec.cuh"
#include "common.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

constexpr int AT_HG = 2;             // heads per warp (the reduction below is written for two)
constexpr int AT_WARPS = 6;          // two CTAs of six warps per SM: 170 registers per thread
constexpr int AT_THREADS = AT_WARPS * 32;
constexpr float AT_LAG = 8.0f;
constexpr int AT_MAX_CLUSTER = 8;
constexpr int AT_MAX_SPLITS = 16;    // sizes the scratch of the reference's operator (attn.hip:67); this kernel needs none

constexpr int AT_RING = 8;           // rows in flight per warp (64 rope columns: the model's shape)
// Shared memory per warp: a row in flight is its latent codes, its rope columns and (slab) one scale per lane; the same
// bytes hold the warp's outputs afterwards.
__host__ __device__ constexpr int at_row_bytes(bool paged, int kvl) { return kvl + (paged ? 64 : 256); }
__host__ __device__ constexpr int at_warp_bytes(bool paged, int kvl) {
    return AT_RING * at_row_bytes(paged, kvl) > AT_HG * kvl * 4 ? AT_RING * at_row_bytes(paged, kvl) : AT_HG * kvl * 4;
}
__device__ __forceinline__ void at_cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// Column of word k (four columns) of lane `lane`, NL columns per lane.
template <int NL>
__device__ __forceinline__ int at_col(int lane, int k) { return NL == 12 ? 128 * k + 4 * lane : lane * NL + 4 * k; }

// Two f32 in a register pair, and the packed multiply-add.
typedef unsigned long long at_f2;
__device__ __forceinline__ at_f2 at_pack(float lo, float hi) {
    at_f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 at_unpack(at_f2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ at_f2 at_fma2(at_f2 a, at_f2 b, at_f2 c) {
    at_f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

struct AttSlab {
    const float* qabs; const float* qrope; const unsigned char* lc8; const float* lscale;
    const unsigned short* rc; const unsigned int* rows; int n_blocks; float* clat;
};
struct AttPaged {
    const uint16_t* q; const uint8_t* pool; const float* pscale; const int32_t* block_table;
    const uint32_t* rows; long long row_stride; const int32_t* n_rows; int page_tokens; int max_pages;
    int n_pool_pages; uint16_t* out; float* out_m; float* out_lse;
    int rows_lo, rows_hi;   // the launch serves sequences with rows_lo <= n_rows < rows_hi only (others are left untouched)
};

// WIDE: the slab's rows and q allow wide loads. At kvl 384 a run of 12 columns would straddle the slab's scale blocks:
// there a lane owns four columns of each block instead (at_col) and the slab's values are scaled as they are decoded. NL = kvl / 32 latent columns per lane (4, 8, 12, 16). ROPE64: 64 rope columns, a neighbouring pair per lane; otherwise
// up to 128, lane + 32 k. Grid (cluster size, head pairs, sequences), clusters along x.
template <bool PAGED, bool WIDE, int NL, bool ROPE64>
__global__ void __launch_bounds__(AT_THREADS, 2)
attend_simt_kernel(AttSlab sp, AttPaged pp, int H, int rope, float scale, int nr_single) {
    constexpr int KVL = NL * 32, HG = AT_HG, N2 = NL / 2, NR = ROPE64 ? 1 : 4;   // NR: rope words per lane
    constexpr bool RING = WIDE && ROPE64;
    constexpr int ROW_BYTES = at_row_bytes(PAGED, KVL), WARP_FLOATS = at_warp_bytes(PAGED, KVL) / 4;
    extern __shared__ __align__(16) float at_smem[];           // per warp: rows in flight, then its outputs [HG][KVL]
    __shared__ float s_m[AT_WARPS][HG], s_l[AT_WARPS][HG];      // their reference maxima and sums
    __shared__ float s_top[AT_WARPS][HG], c_top[HG];            // the largest scores, of warps and of the CTA (out_m)
    __shared__ float s_w[AT_MAX_CLUSTER][HG];                    // weights in the merge, of warps and then of CTAs
    __shared__ float c_m[HG], c_l[HG];                          // the CTA's, read by its cluster
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned char* at_warp_smem = reinterpret_cast<unsigned char*>(at_smem + (size_t)warp * WARP_FLOATS);
    const int n_cta = gridDim.x, rank = blockIdx.x, head0 = blockIdx.y * HG, b = blockIdx.z;
    const int W = KVL + rope;
    rv_grid_dep_trigger();             // a dependent kernel may set itself up; it waits for this grid before reading
    rv_grid_dep_wait();                // the counts, rows and q may come from the kernel before
    int nr = nr_single;
    if (PAGED) {  // clamp device-side counts so a bad entry can never index past a table
        nr = pp.n_rows[b];
        // a row list whose first entry is the dense marker stands for "row j = token j" over the first n_rows tokens
        if (pp.rows && pp.rows[(size_t)b * pp.row_stride] == 0xffffffffu) pp.rows = nullptr;
        const long long cap = pp.rows ? pp.row_stride : (long long)pp.max_pages * pp.page_tokens;
        nr = (int)max(0LL, min((long long)nr, cap));
        if (nr < pp.rows_lo || nr >= pp.rows_hi) return;   // another kernel of the same call serves this sequence (uniform over the cluster)
    }

    // q of the warp's heads (a head past H repeats the last one; it is not stored)
    at_f2 ql[HG][N2];
    float qr[HG][ROPE64 ? 2 : 4];
#pragma unroll
    for (int j = 0; j < HG; ++j) {
        const int h = min(head0 + j, H - 1);
        if (PAGED) {
            const uint16_t* q = pp.q + ((size_t)b * H + h) * W;
#pragma unroll
            for (int k = 0; k < N2; k += 2) {
                const uint16_t* c = q + at_col<NL>(lane, k / 2);
                const uint2 v = WIDE ? *reinterpret_cast<const uint2*>(c)
                                           : make_uint2((uint32_t)c[0] | (uint32_t)c[1] << 16, (uint32_t)c[2] | (uint32_t)c[3] << 16);
                ql[j][k] = at_pack(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u));
                ql[j][k + 1] = at_pack(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
            }
            if (ROPE64) {
                qr[j][0] = rv_bf16_to_f32(q[KVL + 2 * lane]); qr[j][1] = rv_bf16_to_f32(q[KVL + 2 * lane + 1]);
            } else {
#pragma unroll
                for (int k = 0; k < NR; ++k) qr[j][k] = lane + 32 * k < rope ? rv_bf16_to_f32(q[KVL + lane + 32 * k]) : 0.0f;
            }
        } else {
            const float* q = sp.qabs + (size_t)h * KVL;
            if (WIDE) {
#pragma unroll
                for (int k = 0; k < N2; k += 2) {
                    const float4 v = *reinterpret_cast<const float4*>(q + at_col<NL>(lane, k / 2));
                    ql[j][k] = at_pack(v.x, v.y); ql[j][k + 1] = at_pack(v.z, v.w);
                }
            } else {
#pragma unroll
                for (int k = 0; k < N2; ++k) { const float* c = q + at_col<NL>(lane, k / 2) + 2 * (k & 1); ql[j][k] = at_pack(c[0], c[1]); }
            }
            const float* r = sp.qrope + (size_t)h * rope;
            if (ROPE64) { qr[j][0] = r[2 * lane]; qr[j][1] = r[2 * lane + 1]; }
            else {
#pragma unroll
                for (int k = 0; k < NR; ++k) qr[j][k] = lane + 32 * k < rope ? r[lane + 32 * k] : 0.0f;
            }
        }
    }

    // this warp's rows: an even share of nr over the cluster's warps
    const int n_shares = n_cta * AT_WARPS, share = rank * AT_WARPS + warp;
    const int r_begin = (int)((long long)nr * share / n_shares), r_end = (int)((long long)nr * (share + 1) / n_shares);

    at_f2 acc[HG][N2];
    const int my_row = lane >> 4, my_head = (lane >> 3) & 1;      // the score this lane's group of eight ends up with
    float m = -INFINITY, l = 0.0f;                                // reference maximum of my_head, sum of its rows of parity my_row
    float top = -INFINITY;                                        // their largest score, which m follows at a distance
#pragma unroll
    for (int j = 0; j < HG; ++j)
#pragma unroll
        for (int k = 0; k < N2; ++k) acc[j][k] = 0ull;

    constexpr int NS = !PAGED && NL == 12 ? 3 : 1;               // scales per lane and row
    struct Raw { uint32_t c[NL / 4]; uint32_t r[NR]; float s[NS]; };
    const int my_blk = NS == 3 ? lane % 3 : lane * NL / 128;     // slab: scale block of this lane's columns (three blocks: the one it fetches)
    unsigned char* ring = at_warp_smem;                          // RING: [AT_RING rows][latent codes | rope | scales (slab)]
    for (int t0 = r_begin; t0 < r_end; t0 += 32) {
        const int tn = min(32, r_end - t0);
        // lane i locates row t0 + i
        uint32_t where = 0u;
        float tok_s = 0.0f;
        if (lane < tn) {
            const uint32_t* list = PAGED ? pp.rows ? pp.rows + (size_t)b * pp.row_stride : nullptr : sp.rows;
            const uint32_t t = list ? list[t0 + lane] : (uint32_t)(t0 + lane);
            if (PAGED) {
                const int lp = (int)(t / (uint32_t)pp.page_tokens);
                int page = lp < pp.max_pages ? pp.block_table[(size_t)b * pp.max_pages + lp] : -1;
                if (page < 0 || page >= pp.n_pool_pages) page = 0;  // guarded: never read outside the pool
                where = (uint32_t)page * (uint32_t)pp.page_tokens + (t & (uint32_t)(pp.page_tokens - 1));
                tok_s = pp.pscale[where];
            } else {
                where = t;
            }
        }
        auto fetch = [&](int i, Raw& v) {                         // row t0 + i, waited for where it is used
            const size_t r = __shfl_sync(0xffffffffu, where, i);
            const unsigned char* row = PAGED ? pp.pool + r * W : sp.lc8 + r * KVL;
#pragma unroll
            for (int k = 0; k < NL / 4; ++k) {
                const unsigned char* c = row + at_col<NL>(lane, k);
                v.c[k] = PAGED || WIDE ? *reinterpret_cast<const uint32_t*>(c)
                                       : (uint32_t)c[0] | (uint32_t)c[1] << 8 | (uint32_t)c[2] << 16 | (uint32_t)c[3] << 24;
            }
#pragma unroll
            for (int k = 0; k < NR; ++k)
                v.r[k] = lane + 32 * k >= rope ? 0u : PAGED ? pp.pool[r * W + KVL + lane + 32 * k] : sp.rc[r * rope + lane + 32 * k];
#pragma unroll
            for (int k = 0; k < NS; ++k) v.s[k] = PAGED ? __shfl_sync(0xffffffffu, tok_s, i) : sp.lscale[r * sp.n_blocks + (NS == 3 ? k : my_blk)];
        };
        // RING: a row's pieces go to this warp's slots in shared memory (every lane copies what it will read itself, but
        // for the paged rope codes, two lanes' in one word, and the scales of three blocks)
        auto request = [&](int i) {
            const uint32_t r = __shfl_sync(0xffffffffu, where, i);
            const uint32_t dst = tc::smem_u32(ring + (i % AT_RING) * ROW_BYTES);
            const unsigned char* row = PAGED ? pp.pool + (size_t)r * W : sp.lc8 + (size_t)r * KVL;
            if constexpr (NL == 16) tc::cp_async16(dst + lane * 16, row + lane * 16);
            else {
#pragma unroll
                for (int k = 0; k < NL / 4; ++k) at_cp_async4(dst + at_col<NL>(lane, k), row + at_col<NL>(lane, k));
            }
            if (PAGED) {
                if (lane < 16) at_cp_async4(dst + KVL + lane * 4, row + KVL + lane * 4);
            } else {
                at_cp_async4(dst + KVL + lane * 4, sp.rc + (size_t)r * 64 + 2 * lane);
                at_cp_async4(dst + KVL + 128 + lane * 4, sp.lscale + (size_t)r * sp.n_blocks + my_blk);
            }
        };
        auto take = [&](int i, Raw& v) {
            const unsigned char* row = ring + (i % AT_RING) * ROW_BYTES;
            if constexpr (NL == 16) {
                const uint4 p = *reinterpret_cast<const uint4*>(row + lane * 16);
                v.c[0] = p.x; v.c[1] = p.y; v.c[2] = p.z; v.c[3] = p.w;
            } else {
#pragma unroll
                for (int k = 0; k < NL / 4; ++k) v.c[k] = *reinterpret_cast<const uint32_t*>(row + at_col<NL>(lane, k));
            }
            v.r[0] = PAGED ? *reinterpret_cast<const uint16_t*>(row + KVL + lane * 2) : *reinterpret_cast<const uint32_t*>(row + KVL + lane * 4);
#pragma unroll
            for (int k = 0; k < NS; ++k) v.s[k] = PAGED ? __shfl_sync(0xffffffffu, tok_s, i) : *reinterpret_cast<const float*>(row + KVL + 128 + (NS == 3 ? k : lane) * 4);
        };
        if (RING) {
#pragma unroll
            for (int g = 0; g < AT_RING; g += 2) {
                if (g < tn) { request(g); request(min(g + 1, tn - 1)); }
                tc::cp_async_commit();
            }
        }
        for (int i = 0; i < tn; i += 2) {
            const bool live = i + my_row < tn;                   // the second row of the last step may not exist
            Raw now[2];
            if (RING) {
                tc::cp_async_wait<AT_RING / 2 - 1>();
                if (PAGED || NS == 3) __syncwarp();
                take(i, now[0]);
                if (i + 1 < tn) take(i + 1, now[1]); else now[1] = now[0];
                if (PAGED || NS == 3) __syncwarp();
            } else {
                fetch(i, now[0]);
                fetch(min(i + 1, tn - 1), now[1]);
            }
            at_f2 lv[2][N2];                                     // the codes' values; the lane's columns share one scale
            float rv[2][ROPE64 ? 2 : 4], rs[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int k = 0; k < NL / 4; ++k) {
                    float2 x = rv_e4m3x2_to_f32x2((uint16_t)now[u].c[k]), y = rv_e4m3x2_to_f32x2((uint16_t)(now[u].c[k] >> 16));
                    if (NS == 3) { const float sk = now[u].s[k % NS]; x.x *= sk; x.y *= sk; y.x *= sk; y.y *= sk; }
                    lv[u][2 * k] = at_pack(x.x, x.y);
                    lv[u][2 * k + 1] = at_pack(y.x, y.y);
                }
                if (ROPE64) {
                    if (PAGED) { const float2 x = rv_e4m3x2_to_f32x2((uint16_t)now[u].r[0]); rv[u][0] = x.x; rv[u][1] = x.y; }
                    else { rv[u][0] = __uint_as_float(now[u].r[0] << 16); rv[u][1] = __uint_as_float(now[u].r[0] & 0xffff0000u); }
                } else {
#pragma unroll
                    for (int k = 0; k < NR; ++k) rv[u][k] = PAGED ? rv_e4m3_to_f32((uint8_t)now[u].r[k]) : rv_bf16_to_f32((uint16_t)now[u].r[k]);
                }
                rs[u] = NS == 3 ? 1.0f : now[u].s[0];
            }
            if (RING) {                                          // the slots just read take the rows AT_RING further on
                if (i + AT_RING < tn) { request(i + AT_RING); request(min(i + AT_RING + 1, tn - 1)); }
                tc::cp_async_commit();
            }
            float part[2][HG];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int j = 0; j < HG; ++j) {
                    at_f2 p2 = 0ull;
                    float pr = 0.0f;
#pragma unroll
                    for (int k = 0; k < N2; ++k) p2 = at_fma2(ql[j][k], lv[u][k], p2);
#pragma unroll
                    for (int k = 0; k < (ROPE64 ? 2 : 4); ++k) pr = fmaf(qr[j][k], rv[u][k], pr);
                    const float2 p = at_unpack(p2);
                    // the rope columns have the token's scale in the paged cache, none in the slab
                    part[u][j] = PAGED ? (p.x + p.y + pr) * rs[u] : fmaf(p.x + p.y, rs[u], pr);
                }
            // four sums over the warp
            float a0 = my_row ? part[1][0] : part[0][0], a1 = my_row ? part[1][1] : part[0][1];
            a0 += __shfl_xor_sync(0xffffffffu, my_row ? part[0][0] : part[1][0], 16);
            a1 += __shfl_xor_sync(0xffffffffu, my_row ? part[0][1] : part[1][1], 16);
            float s = my_head ? a1 : a0;
            s += __shfl_xor_sync(0xffffffffu, my_head ? a0 : a1, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s = live ? s * scale : -INFINITY;
            if (PAGED) top = fmaxf(top, s);
            // the reference m follows the maximum at a distance: a weight may reach e^AT_LAG, which f32 holds as well as
            // 1, and the sums are rescaled at a warp's first rows and then hardly ever
            if (__any_sync(0xffffffffu, s > m + AT_LAG)) {
                const float m_new = fmaxf(m, fmaxf(s, __shfl_xor_sync(0xffffffffu, s, 16)));
                const float corr = m_new == m ? 1.0f : expf(m - m_new);
                m = m_new;
                l *= corr;
#pragma unroll
                for (int j = 0; j < HG; ++j) {
                    const float cj = __shfl_sync(0xffffffffu, corr, 8 * j);
#pragma unroll
                    for (int k = 0; k < N2; ++k) { const float2 o = at_unpack(acc[j][k]); acc[j][k] = at_pack(o.x * cj, o.y * cj); }
                }
            }
            const float p = expf(s - m);
            l += p;
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int j = 0; j < HG; ++j) {
                    const float w = __shfl_sync(0xffffffffu, p, 16 * u + 8 * j) * rs[u];
                    const at_f2 w2 = at_pack(w, w);
#pragma unroll
                    for (int k = 0; k < N2; ++k) acc[j][k] = at_fma2(w2, lv[u][k], acc[j][k]);
                }
        }
    }
    l += __shfl_xor_sync(0xffffffffu, l, 16);                    // both row parities
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
    if (RING) tc::cp_async_wait<0>();                            // (nothing is in flight; the slots become the output buffer)

    // ---- the CTA's warps meet in shared memory (a warp without rows has m = -inf, l = 0) ----
    if ((lane & 23) == 0) { s_m[warp][my_head] = m; s_l[warp][my_head] = l; s_top[warp][my_head] = top; }
    if (r_begin < r_end) {
#pragma unroll
        for (int j = 0; j < HG; ++j)
#pragma unroll
            for (int k = 0; k < N2; k += 2) {
                const float2 x = at_unpack(acc[j][k]), y = at_unpack(acc[j][k + 1]);
                *reinterpret_cast<float4*>(at_smem + (size_t)warp * WARP_FLOATS + j * KVL + at_col<NL>(lane, k / 2)) = make_float4(x.x, x.y, y.x, y.y);
            }
    }
    __syncthreads();
    auto store = [&](int h, int c, float v) {
        if (PAGED) pp.out[((size_t)b * H + h) * KVL + c] = rv_f32_to_bf16(v);
        else sp.clat[(size_t)h * KVL + c] = v;
    };
    auto stats = [&](int h, float most, float mg, float lg) {
        if (PAGED) {
            if (pp.out_m) pp.out_m[(size_t)b * H + h] = most;
            if (pp.out_lse) pp.out_lse[(size_t)b * H + h] = lg > 0.0f ? mg + logf(lg) : -INFINITY;
        }
    };
    // the CTA's maximum and sum per head, and the weight of each warp's outputs at that maximum. A sum of exactly 0 says that
    // there were no rows (the weight of the maximum is 1); one that is NaN goes on to the denominator and makes the head NaN.
    if (tid < AT_WARPS * HG) {
        const int j = tid % HG, w = tid / HG;
        float mx = -INFINITY, sum = 0.0f;
#pragma unroll
        for (int v = 0; v < AT_WARPS; ++v) mx = fmaxf(mx, s_m[v][j]);
#pragma unroll
        for (int v = 0; v < AT_WARPS; ++v)
            if (s_l[v][j] != 0.0f) sum += s_l[v][j] * expf(s_m[v][j] - mx);
        s_w[w][j] = s_l[w][j] != 0.0f ? expf(s_m[w][j] - mx) : 0.0f;
        if (w == 0) {
            c_m[j] = mx; c_l[j] = sum;
            float most = -INFINITY;
#pragma unroll
            for (int v = 0; v < AT_WARPS; ++v) most = fmaxf(most, s_top[v][j]);
            c_top[j] = most;
        }
    }
    __syncthreads();
    auto cta_sum = [&](int j, int c) {                            // column c of head j over the CTA's warps
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < AT_WARPS; ++w)
            if (s_w[w][j] != 0.0f) v = fmaf(at_smem[(size_t)w * WARP_FLOATS + j * KVL + c], s_w[w][j], v);
        return v;
    };
    if (n_cta == 1) {
        for (int e = tid; e < HG * KVL; e += AT_THREADS) {
            const int j = e / KVL, c = e - j * KVL;
            if (head0 + j < H) store(head0 + j, c, c_l[j] != 0.0f ? cta_sum(j, c) * (1.0f / c_l[j]) : 0.0f);
        }
        if (tid < HG && head0 + tid < H) stats(head0 + tid, c_top[tid], c_m[tid], c_l[tid]);
        return;
    }
    // ---- and the cluster's CTAs through distributed shared memory ----
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int PER = (HG * KVL + AT_THREADS - 1) / AT_THREADS;
    float mine[PER];
#pragma unroll
    for (int e = 0; e < PER; ++e) { const int c = tid + e * AT_THREADS; mine[e] = c < HG * KVL ? cta_sum(c / KVL, c % KVL) : 0.0f; }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < PER; ++e) if (tid + e * AT_THREADS < HG * KVL) at_smem[tid + e * AT_THREADS] = mine[e];
    cluster.sync();                                               // every CTA's (m, l, output)
    if (tid < 32) {                                               // weight of each CTA's outputs, normalised: lane = (CTA, head)
        const int j = lane % HG, q = lane / HG;
        static_assert(HG * AT_MAX_CLUSTER <= 32, "one lane per (CTA, head)");
        const float mq = q < n_cta ? cluster.map_shared_rank(c_m, q)[j] : -INFINITY, lq = q < n_cta ? cluster.map_shared_rank(c_l, q)[j] : 0.0f;
        float mg = mq, most = q < n_cta ? cluster.map_shared_rank(c_top, q)[j] : -INFINITY;
#pragma unroll
        for (int o = HG; o < HG * AT_MAX_CLUSTER; o <<= 1) {
            mg = fmaxf(mg, __shfl_xor_sync(0xffffffffu, mg, o));
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
        }
        const float wq = lq != 0.0f ? expf(mq - mg) : 0.0f;
        float lg = lq * wq;
#pragma unroll
        for (int o = HG; o < HG * AT_MAX_CLUSTER; o <<= 1) lg += __shfl_xor_sync(0xffffffffu, lg, o);
        if (q < AT_MAX_CLUSTER) s_w[q][j] = lq != 0.0f ? wq / lg : 0.0f;
        if (q == 0 && rank == 0 && head0 + j < H) stats(head0 + j, most, mg, lg);
    }
    __syncthreads();
    const int c_lo = HG * KVL * rank / n_cta, c_hi = HG * KVL * (rank + 1) / n_cta;   // this CTA merges and stores these columns
    for (int e = c_lo + tid; e < c_hi; e += AT_THREADS) {
        const int j = e / KVL;
        float v = 0.0f, o[AT_MAX_CLUSTER];
#pragma unroll
        for (int q = 0; q < AT_MAX_CLUSTER; ++q) o[q] = q < n_cta ? cluster.map_shared_rank(at_smem, q)[e] : 0.0f;   // all in flight
#pragma unroll
        for (int q = 0; q < AT_MAX_CLUSTER; ++q)
            if (q < n_cta && s_w[q][j] != 0.0f) v = fmaf(o[q], s_w[q][j], v);   // (a CTA without rows left its array unwritten)
        if (head0 + j < H) store(head0 + j, e - j * KVL, v);
    }
    cluster.sync();                                               // nobody reads this CTA's memory any more
}

// CTAs per (sequence, head group): enough that the grid covers the SMs about twice over, at most one cluster of eight,
// and no more than leave every warp about two rows (rows_most: what the host knows of the longest sequence).
static int simt_cluster(int B, int groups, long long rows_most) {
    int n = 1;
    while (n < AT_MAX_CLUSTER && (long long)B * groups * n * 2 <= 2 * rv_sm_count() && (long long)n * AT_WARPS * 2 < rows_most) n *= 2;
    return n;
}

template <bool PAGED>
static int launch_attend_simt(const AttSlab& sp, const AttPaged& pp, bool wide, int H, int kvl, int rope, float scale,
                              int nr_single, int B, long long rows_most, cudaStream_t st) {
    const int groups = (H + AT_HG - 1) / AT_HG, n = simt_cluster(B, groups, rows_most);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n, (unsigned)groups, (unsigned)B); cfg.blockDim = dim3(AT_THREADS);
    cfg.dynamicSmemBytes = (size_t)AT_WARPS * at_warp_bytes(PAGED, kvl); cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)n; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = n > 1 ? 2 : 1;
    rv_drain_error();
#define RV_ATT(WIDE, NL, R64)                                                                             \
    do {                                                                                                  \
        rv_allow_smem<attend_simt_kernel<PAGED, WIDE, NL, R64>>(AT_WARPS * at_warp_bytes(PAGED, NL * 32)); \
        (void)cudaLaunchKernelEx(&cfg, attend_simt_kernel<PAGED, WIDE, NL, R64>, sp, pp, H, rope, scale, nr_single); \
    } while (0)
#define RV_ATT2(NL)                                                                                       \
    do {                                                                                                  \
        if (!wide) RV_ATT(false, NL, false);                                                              \
        else if (rope == 64) RV_ATT(true, NL, true);                                                      \
        else RV_ATT(true, NL, false);                                                                     \
    } while (0)
    if (kvl == 512) RV_ATT2(16);
    else if (kvl == 384) RV_ATT2(12);
    else if (kvl == 256) RV_ATT2(8);
    else RV_ATT2(4);
#undef RV_ATT2
#undef RV_ATT
    return rv_launch_status();
}

RIVOLI_API size_t rivoli_mla_attend_scratch_floats(int H, int kvl) {
    if (H <= 0 || kvl <= 0) return 0;
    return (size_t)AT_MAX_SPLITS * (size_t)H * ((size_t)kvl + 2);
}

static int mla_attend_guard(int H, int nr, int kvl, int rope, int n_blocks) {
    if (H <= 0 || nr <= 0 || kvl <= 0 || rope <= 0 || n_blocks <= 0) return 1001;
    // The reference's staging bound and width rule, kept so the same shapes are rejected
    // with the same codes (attn.hip:285-293).
    if (((size_t)16 * kvl + (size_t)16 * rope) * sizeof(float) > 65536) return 1002;
    if (kvl > 512 || (kvl % 128) != 0) return 1004;
    if (rope > 128) return 1002;
    return 0;
}

RIVOLI_API int rivoli_mla_attend(const float* qabs, const float* qrope, const unsigned char* Lc8,
                                 const float* Lscale, const unsigned short* Rc, const unsigned int* rows,
                                 int H, int nr, int kvl, int rope, int n_blocks, float scale, float* clat,
                                 float* partial) {
    if (int e = mla_attend_guard(H, nr, kvl, rope, n_blocks)) return e;
    // `partial` is the reference's scratch for a split: this library merges the splits on the chip and leaves it alone,
    // so the result does not depend on whether it was lent.
    (void)partial;
    AttSlab sp{qabs, qrope, Lc8, Lscale, Rc, rows, n_blocks, clat};
    const bool wide = ((((uintptr_t)Lc8 | (uintptr_t)qabs) & 15) | ((uintptr_t)Rc & 3)) == 0;
    return launch_attend_simt<false>(sp, AttPaged{}, wide, H, kvl, rope, scale, nr, 1, nr, 0);
}

// rivoli_mla_attend for callers that have no device memory to lend (everything carved into their own arenas, a decode
// thread that must not wait for the allocator, a plugin contract that forbids it). The kernel needs no scratch, so this
// is the same launch. More than 64 heads stay refused, as the entry point's contract has it: a host may rely on the code.
constexpr int NA_MAX_H = 64;

RIVOLI_API int rivoli_mla_attend_static(const float* qabs, const float* qrope, const unsigned char* Lc8,
                                        const float* Lscale, const unsigned short* Rc, const unsigned int* rows,
                                        int H, int nr, int kvl, int rope, int n_blocks, float scale, float* clat) {
    if (int e = mla_attend_guard(H, nr, kvl, rope, n_blocks)) return e;
    if (H > NA_MAX_H) return 1002;
    return rivoli_mla_attend(qabs, qrope, Lc8, Lscale, Rc, rows, H, nr, kvl, rope, n_blocks, scale, clat, nullptr);
}

// None: the splits merge on the chip.
RIVOLI_API size_t rivoli_attend_simt_scratch_bytes(const DsaGeom*, int) { return 0; }

// Paged bf16 attention on CUDA cores. Same contract as rivoli_mla_attend_paged_bf16.
RIVOLI_API int rivoli_attend_simt_paged_bf16(const DsaGeom* g, const uint16_t* q, const uint8_t* latent_pool,
                                             const float* latent_scale, const int32_t* block_table,
                                             const uint32_t* rows, int row_stride, const int32_t* n_rows,
                                             int B, uint16_t* out, float* out_m, float* out_lse,
                                             void* scratch, void* stream) {
    if (int e = rv_check_geom(g)) return e;
    if (B <= 0 || !q || !latent_pool || !latent_scale || !block_table || !n_rows || !out) return 1001;
    if (rows && row_stride <= 0) return 1001;
    if (((uintptr_t)latent_pool & 15) || ((g->kv_lora + g->rope_dim) % 16) != 0) return 1005;
    (void)scratch;   // the splits merge on the chip
    AttPaged pp{q, latent_pool, latent_scale, block_table, rows, row_stride, n_rows, g->page_tokens,
                g->max_pages_per_seq, g->n_pool_pages, out, out_m, out_lse, 0, 0x7fffffff};
    const long long most = rows ? row_stride : (long long)g->max_pages_per_seq * g->page_tokens;
    return launch_attend_simt<true>(AttSlab{}, pp, ((uintptr_t)q & 7) == 0, g->n_heads, g->kv_lora, g->rope_dim, g->softmax_scale, 0, B, most,
                                    (cudaStream_t)stream);
}

// The sequences of a batch with rows_lo <= n_rows < rows_hi on the CUDA-core kernel: the short-context arm of
// rivoli_mla_attend_paged_bf16, launched in front of the tensor-core kernel as a programmatic dependent of whatever
// precedes it in the stream. rows_lo = 0: the caller knows that no sequence reaches rows_hi, and none is left out.
extern "C" int rivoli_attend_simt_short_rows(const DsaGeom* g, const uint16_t* q, const uint8_t* latent_pool,
                                             const float* latent_scale, const int32_t* block_table,
                                             const uint32_t* rows, int row_stride, const int32_t* n_rows, int B,
                                             uint16_t* out, float* out_m, float* out_lse, int rows_lo,
                                             int rows_hi, cudaStream_t st) {
    AttPaged pp{q, latent_pool, latent_scale, block_table, rows, row_stride, n_rows, g->page_tokens,
                g->max_pages_per_seq, g->n_pool_pages, out, out_m, out_lse, rows_lo, rows_lo ? rows_hi : 0x7fffffff};
    return launch_attend_simt<true>(AttSlab{}, pp, ((uintptr_t)q & 7) == 0, g->n_heads, g->kv_lora, g->rope_dim, g->softmax_scale, 0, B, rows_hi, st);
}
