// Exact top-k selection over the tensor-core scorer's approximate scores: one thread-block CLUSTER per
// sequence, so a sequence's tokens are spread over up to 8 SMs whatever the batch size is.
//
// Input: a_t (approximate score of token t, without the key scale) from index_score_mma_kernel, with
// |a_t * s_k[t] - o_t| <= eps for the exact score o_t. With A_k the k-th largest approximate score,
// a_t > A_k + 2 eps implies "selected" and a_t < A_k - 2 eps implies "not selected" (|A_k - E_k| <= eps for
// the exact k-th value E_k); the band in between is re-scored in the exact fold order of
// rivoli_index_score_paged and ranked exactly (ties -> lower index). The rows written are therefore
// IDENTICAL to exact scoring + exact top-k (contract and tie rule: crates/backend/kernels/indexer.hip:143-257,
// crates/core/src/routing.rs:42-61).
//
// Layout: CTAs of 1024 threads; CTA `r` of a cluster of C owns the CH consecutive tokens [r * CH, (r + 1) * CH), CH <= 16,384;
// thread t the four tokens from (it * 1024 + t) * 4 of each of the CTA's up to four steps `it`, keys in shared memory. So every
// load is a whole line, and the loops over the steps stay loops: a kernel whose code runs once per launch waits for its own
// instructions (keys in registers, 32 consecutive tokens per thread and everything unrolled: 5.3 warps per issue slot stalled
// without an instruction, and 16-byte loads 128 bytes apart).
// What the CTAs of a cluster exchange goes through distributed shared memory, and is PUSHED into the reader's memory before a
// cluster barrier: no CTA waits for a remote load except in the histogram's reduction.
//
//   1. keys; cluster-wide min / max key and max key scale (eps). What does not depend on the scores (page table, key scales,
//      query) is loaded before the wait for the scorer.
//   2. ONE histogram pass over 4096 bins spread linearly in value between the smallest and the largest score:
//      the distribution decides the bin width, so the bin of the k-th value holds a handful of tokens on
//      score-like data. Histograms are all-reduced slice by slice, the k-th bin is found by a suffix scan.
//   3. classification against the band [lower edge of that bin - 2 eps, upper edge + 2 eps]; band tokens
//      are listed per CTA.
//   4. exact re-score of the CTA's own band tokens (a warp takes 4 at a time, lane = head), the lists are
//      pushed cluster-wide, band tokens are ranked against all of them.
//   5. ascending write-out: each CTA compacts its own contiguous token range.
//
// A lone CTA (a batch that fills the chip by itself, or few tokens): the exchanges, the cluster barriers and the list copies
// are compiled out (SOLO below).
//
// VALUES: the same selection over given scores (rivoli_index_topk and its batched form): no error band (eps = 0), no key
// scales and no re-score - the band is the k-th value's bin itself and its tokens are ranked by the scores as they are.
//
// If the band does not fit the list (tie-dominated scores: thousands of tokens at the cut) the cluster takes
// the slow path instead: every band token is re-scored chunk by chunk, the exact keys replace the approximate
// ones, and an exact 4 x 8-bit radix selection runs over the whole cluster.
//
// A whole step, us, with keys in registers and with them here, when that was changed: 4 sequences of 131,072 tokens 85.5 -> 64.2; 32
// of up to 32,768 88.3 -> 80.5; 64 of 16,384 104.7 -> 92.3; 128 of 16,384 149.0 -> 138.6; 16 of 16,384 65.8 -> 56.9; one of 4,099
// 42.4 -> 38.0. Other kernels of the step have changed since, and this one: 52.5 for 4 of 131,072, 129 for 128 of 16,384, 29.3 for one of 4,099 now.
#include <cooperative_groups.h>

#include "codec.cuh"
#include "common.cuh"
#include "index_rescore.cuh"
#include "index_select.hpp"
#include "topk_core.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int SEL_NT = 1024, SEL_NW = SEL_NT / 32;
constexpr int SEL_STEP = SEL_NT * 4;                    // tokens of one step
constexpr int SEL_STEPS = 4, SEL_CH = SEL_STEP * SEL_STEPS;   // most tokens per CTA
constexpr int SEL_BINS = 4096;
static_assert(SEL_BINS == SEL_NT * 4, "a thread scans four bins");
constexpr int SEL_LIST = 2048;     // band tokens per SEQUENCE the fast path holds (and per chunk on the slow path)
constexpr int SEL_RANK_ALL = SEL_NT;  // up to this many entries of the gathered list every CTA ranks them all, one per thread, instead of one more exchange
constexpr int SEL_HD = RS_HD;      // index dim (one code word per lane)

struct SelXc {                     // per-CTA exchange block; slot q of an array is written by rank q
    uint32_t kmin[SEL_MAX_CLUSTER], kmax[SEL_MAX_CLUSTER], skmax[SEL_MAX_CLUSTER];
    uint32_t n_in[SEL_MAX_CLUSTER], n_band[SEL_MAX_CLUSTER];
    uint32_t n_out[SEL_MAX_CLUSTER];
    uint32_t cnt_gt[SEL_MAX_CLUSTER], cnt_eq[SEL_MAX_CLUSTER];
    uint32_t red[2][SEL_NW];
    uint32_t red3[3][SEL_NW];
    uint32_t wcnt[SEL_NW];
    uint32_t pre[2][SEL_NW];
    uint32_t list_n, lower;
    uint32_t bstar;
    uint32_t pivot, need;
};

// Sum over the block, one barrier (double-buffered partials).
__device__ __forceinline__ uint32_t sel_block_sum(uint32_t v, SelXc& xc, int& buf) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) xc.red[buf][warp] = v;
    __syncthreads();
    const uint32_t t = __reduce_add_sync(0xffffffffu, xc.red[buf][lane]);
    buf ^= 1;
    return t;
}

// Exclusive prefix of `v` over the block in thread order (one barrier).
__device__ __forceinline__ uint32_t sel_block_excl(uint32_t v, SelXc& xc) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) xc.wcnt[warp] = incl;
    __syncthreads();
    return __reduce_add_sync(0xffffffffu, lane < warp ? xc.wcnt[lane] : 0u) + incl - v;
}

// For a mask of 4 bits per step: how many bits of tokens before this thread's are set, per step (token order: step, then
// thread). One barrier; two steps share a word (a step holds at most 4,096 tokens).
__device__ __forceinline__ void sel_token_excl(uint32_t mask, SelXc& xc, uint32_t (&before)[SEL_STEPS]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t c[2], incl[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        c[u] = (uint32_t)__popc(mask & (0xfu << (8 * u))) | ((uint32_t)__popc(mask & (0xf0u << (8 * u))) << 16);
        incl[u] = c[u];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl[u], o);
            if (lane >= o) incl[u] += t;
        }
    if (lane == 31) { xc.pre[0][warp] = incl[0]; xc.pre[1][warp] = incl[1]; }
    __syncthreads();
    uint32_t run = 0u;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const uint32_t w = xc.pre[u][lane];
        const uint32_t tot = __reduce_add_sync(0xffffffffu, w);
        const uint32_t ex = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + incl[u] - c[u];
        before[2 * u] = run + (ex & 0xffffu);
        run += tot & 0xffffu;
        before[2 * u + 1] = run + (ex >> 16);
        run += tot >> 16;
    }
}

// VEC: the score rows allow 16-byte loads (a kernel of its own: both forms in one cost the clusters' kernel a spill of 8 bytes, and
// given scores, which take the loop further below instead, four predicated steps for the one or two that hold scores). us a step or
// pass with both in one -> apart: 1 x 4,099 30.2 -> 29.3, 2 x 15,001 34.0 -> 33.6, 1 x 1,024 23.8 -> 22.5, operators at 8,193 123.0 -> 122.7.
template <bool VALUES, bool SOLO, bool VEC>
__global__ void __launch_bounds__(SEL_NT, 1)
index_select_cluster_kernel(SelArgs A, int CH) {
    cg::cluster_group cluster = cg::this_cluster();
    const int C = SOLO ? 1 : (int)cluster.dim_blocks().x, r = SOLO ? 0 : (int)cluster.block_rank();
    if constexpr (!SOLO) cluster.barrier_arrive();                        // [0] every CTA runs: its memory may be written
    extern __shared__ __align__(16) uint32_t sel_smem[];
    __shared__ SelXc xc;
    uint32_t* keys = sel_smem;                                            // [CH]
    uint32_t* hist = keys + CH;                                           // [SEL_BINS]; later `dec`
    uint32_t* l_tok = hist + SEL_BINS;                                    // [SEL_LIST] this CTA's band tokens
    uint64_t* l_cmp = reinterpret_cast<uint64_t*>(l_tok + SEL_LIST);      // [SEL_LIST] their exact keys, ~token below: larger = ranked higher
    uint32_t* l_row = l_tok + 3 * SEL_LIST;                               // [SEL_LIST] their pool rows (the lookup is done where the token is listed)
    uint32_t* red = l_row + SEL_LIST;                                  // [SEL_BINS] reduced histogram, before the re-score
    float* kfw = reinterpret_cast<float*>(red);                           // [warps][SEL_HD][4] key rows as f32
    uint32_t* qf = red + SEL_NW * SEL_HD * 4;                             // [RS_QWORDS] packed q codes
    uint64_t* a_cmp = reinterpret_cast<uint64_t*>(VALUES ? red + SEL_BINS : qf + RS_QWORDS);   // [SEL_LIST] the cluster's band (clusters only)

    const DsaGeom& g = A.g;
    const int nh = g.index_heads, P = g.page_tokens;
    const int b = (int)blockIdx.x / C, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    rv_grid_dep_trigger();   // the next kernel may set itself up; it waits for this grid before reading rows
    // The scorer is launched only when all before it is complete and starts this kernel only then, so everything but its
    // scores may be read before the wait. Given scores come with no such promise.
    if constexpr (VALUES) rv_grid_dep_wait();
    // (requested before the sequence's length is known: nothing here waits for another load)
    const int c0 = r * CH, pshift = VALUES ? 0 : 31 - __clz(P);
    const int32_t* bt = A.block_table + (size_t)b * g.max_pages_per_seq;
    uint32_t qw = 0u;
    int pgs[SEL_STEPS];
    float my_sq = 0.0f, my_wh = 0.0f, cb = 0.0f;                          // head constants of the re-score (nh <= 32); error constant
    if constexpr (!VALUES) {
        static_assert(RS_QWORDS == SEL_NT, "a word per thread");
        qw = rv_rescore_q_word(A.qcodes + (size_t)b * nh * SEL_HD, nh, tid);
#pragma unroll
        for (int it = 0; it < SEL_STEPS; ++it) {                          // (the score rows are no longer than the page table)
            const int i = c0 + it * SEL_STEP + tid * 4;
            pgs[it] = it * SEL_STEP + tid * 4 < CH && i < A.score_stride ? bt[i >> pshift] : 0;
        }
        if (lane < nh) { my_sq = A.qscales[(size_t)b * nh + lane]; my_wh = __fmul_rn(A.w[(size_t)b * nh + lane], g.index_wscale); }
        cb = A.cb[b];
    }
    const int nt = min(VALUES && !A.seq_len ? A.nt_single : A.seq_len[b], A.score_stride);
    const int kk = min(A.k, nt);
    uint32_t* out = A.rows + (size_t)b * A.k;
    const int nloc = max(0, min(CH, nt - c0));                            // this CTA's tokens: [c0, c0 + nloc)
    if (kk == nt || kk <= 0) {                                            // everything (or nothing) is selected: the identity
        if constexpr (!VALUES) rv_grid_dep_wait();
        if (r == 0 && tid == 0 && (!VALUES || A.n_sel)) A.n_sel[b] = kk > 0 ? kk : 0;
        for (int i = tid; i < nloc; i += SEL_NT) out[c0 + i] = (uint32_t)(c0 + i);
        if (r == 0 && tid == 0 && A.stats && kk > 0) { A.stats[b * 2] = 0; A.stats[b * 2 + 1] = (unsigned)nt; }
        if constexpr (!VALUES) {                                              // nobody scored these tokens: look at their pages here
            for (int lp = r * SEL_NT + tid; lp * P < nt; lp += C * SEL_NT) {
                const int pg = lp < g.max_pages_per_seq ? bt[lp] : 0;
                if (pg < 0 || pg >= g.n_pool_pages) atomicCAS(A.err, 0, 1005);
            }
        }
        if constexpr (!SOLO) cluster.barrier_wait();
        return;
    }

    // ---- 1. approximate keys: (unscaled tensor-core score) * key scale of the token --------------------------
    const float* s = A.scores + (size_t)b * (VALUES ? (size_t)A.value_stride : (size_t)A.score_stride);
    const int steps = (nloc + SEL_STEP - 1) / SEL_STEP;
    auto scale_row = [&](int i, int pg) {
        pg = (pg < 0 || pg >= g.n_pool_pages) ? 0 : pg;
        return ((size_t)pg << pshift) + (i & (P - 1));
    };
    auto page_of = [&](int it) { return it < 2 ? (it ? pgs[1] : pgs[0]) : (it == 2 ? pgs[2] : pgs[3]); };   // of this thread's tokens of step `it` (P % 4 == 0)
    auto row_of_bit = [&](int bit, int i) {                                   // pool row of token c0 + i, bit = 4 * step + e
        return A.vec_ok ? (uint32_t)scale_row(c0 + i, page_of(bit >> 2)) : rv_pool_row(g, bt, (uint32_t)(c0 + i));
    };
    uint32_t kmin = 0xffffffffu, kmax = 0u;
    float skm = 0.0f;
    auto take4 = [&](int i4, const float (&v)[4]) {                       // four keys of the token vector at local index i4
        uint32_t k[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            k[e] = topk_key(v[e]);
            if (i4 + e < nloc) { kmin = min(kmin, k[e]); kmax = max(kmax, k[e]); }
        }
        *reinterpret_cast<uint4*>(keys + i4) = make_uint4(k[0], k[1], k[2], k[3]);
    };
    for (int i = tid; i < SEL_BINS / 4; i += SEL_NT) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (!SOLO)                                                  // empty slots of the gathered list rank below every token
        for (int i = tid; i < SEL_LIST; i += SEL_NT) a_cmp[i] = 0ull;
    if constexpr (!VALUES) qf[tid] = qw;
    if (tid == 0) { xc.list_n = 0; xc.lower = 0; }
    if (VALUES ? VEC : A.vec_ok != 0) {
        float4 sk[SEL_STEPS], sc[SEL_STEPS];
        if constexpr (!VALUES) {
#pragma unroll
            for (int it = 0; it < SEL_STEPS; ++it) {
                const int i4 = it * SEL_STEP + tid * 4;
                sk[it] = i4 < nloc ? *reinterpret_cast<const float4*>(A.index_scale + scale_row(c0 + i4, pgs[it])) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            rv_grid_dep_wait();
        }
        // (rows of any length: the same tokens, a score at a time, two steps in flight; all four cost a spill of 16 bytes. Given scores:
        // two steps of a loop that ends with the scores, as one or two is what most rows have: 8 x 4,096 of the 16-head layer 20.8 us a
        // step with four unrolled, 20.6 so; 2 x 16,384 23.2 both)
        constexpr int AHEAD = VEC && !VALUES ? SEL_STEPS : 2;
#pragma unroll (VALUES ? 1 : SEL_STEPS)
        for (int it0 = 0; it0 < SEL_STEPS; it0 += AHEAD) {
            if (VALUES && it0 * SEL_STEP >= nloc) break;
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int i4 = (it0 + u) * SEL_STEP + tid * 4;
                const float* p = s + c0 + i4;
                if constexpr (VEC) sc[u] = i4 < nloc ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
                else sc[u] = make_float4(i4 < nloc ? p[0] : 0.f, i4 + 1 < nloc ? p[1] : 0.f, i4 + 2 < nloc ? p[2] : 0.f, i4 + 3 < nloc ? p[3] : 0.f);
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int it = it0 + u, i4 = it * SEL_STEP + tid * 4;
                if (i4 < nloc) {
                    float v[4] = {sc[u].x, sc[u].y, sc[u].z, sc[u].w};
                    if constexpr (!VALUES) {
                        const float k4[4] = {sk[it].x, sk[it].y, sk[it].z, sk[it].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            v[e] *= k4[e];
                            if (i4 + e < nloc) skm = fmaxf(skm, k4[e]);
                        }
                    }
                    take4(i4, v);
                }
            }
        }
    } else {
        if constexpr (!VALUES) rv_grid_dep_wait();
#pragma unroll 1
        for (int it = 0; it < steps; ++it) {
            const int i4 = it * SEL_STEP + tid * 4;
            if (i4 >= nloc) break;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[e] = 0.0f;
                if (i4 + e < nloc) {
                    v[e] = s[c0 + i4 + e];
                    if constexpr (!VALUES) {
                        const float k1 = A.index_scale[scale_row(c0 + i4 + e, bt[(c0 + i4 + e) >> pshift])];
                        v[e] *= k1;
                        skm = fmaxf(skm, k1);
                    }
                }
            }
            take4(i4, v);
        }
    }
    if (r == 0 && tid == 0 && (!VALUES || A.n_sel)) A.n_sel[b] = kk;
    // keys of this thread's four tokens of step `it` (only this thread reads and writes them until the slow path's end)
    auto for_keys = [&](auto f) {                                          // f(step, e, key)
#pragma unroll 1
        for (int it = 0; it < steps; ++it) {
            const int i4 = it * SEL_STEP + tid * 4;
            if (i4 < nloc) {
                const uint4 k = *reinterpret_cast<const uint4*>(keys + i4);
                f(it, 0, k.x);
                if (i4 + 4 <= nloc) {
                    f(it, 1, k.y);
                    f(it, 2, k.z);
                    f(it, 3, k.w);
                } else {
                    if (i4 + 1 < nloc) f(it, 1, k.y);
                    if (i4 + 2 < nloc) f(it, 2, k.z);
                }
            }
        }
    };
    int buf = 0;
    float sk_max;
    {
        uint32_t sm = __reduce_max_sync(0xffffffffu, __float_as_uint(skm));    // scales are >= 0: bit order = value order
        kmin = __reduce_min_sync(0xffffffffu, kmin);
        kmax = __reduce_max_sync(0xffffffffu, kmax);
        if (lane == 0) { xc.red3[0][warp] = kmin; xc.red3[1][warp] = kmax; xc.red3[2][warp] = sm; }
        __syncthreads();                                                       // (also orders the zeroing above before the histogram)
        kmin = __reduce_min_sync(0xffffffffu, xc.red3[0][lane]);
        kmax = __reduce_max_sync(0xffffffffu, xc.red3[1][lane]);
        sm = __reduce_max_sync(0xffffffffu, xc.red3[2][lane]);
        if constexpr (!SOLO) {
            cluster.barrier_wait();                                            // [0]
            if (tid < C) {
                SelXc* dst = cluster.map_shared_rank(&xc, tid);
                dst->kmin[r] = kmin; dst->kmax[r] = kmax; dst->skmax[r] = sm;
            }
            cluster.sync();                                                    // [1] everybody's extremes
            const int q = lane < C ? lane : 0;
            kmin = __reduce_min_sync(0xffffffffu, xc.kmin[q]);
            kmax = __reduce_max_sync(0xffffffffu, xc.kmax[q]);
            sm = __reduce_max_sync(0xffffffffu, xc.skmax[q]);
        }
        sk_max = __uint_as_float(sm);
    }
    const float eps = VALUES ? 0.0f : sk_max * cb;

    // ---- 2. one histogram pass: 4096 bins spread linearly IN VALUE between the smallest and the largest score ----
    // bin(v) = min(4095, int((v - vmin) * inv_w)) is monotone in v, which is all the selection needs: tokens in
    // higher bins than the k-th value's are above it, tokens in lower bins below. (Bins linear in the key BITS
    // would be logarithmic in value: 6 % wide around 1.0.) A degenerate range (all scores equal, or a span
    // that overflows; given scores may also hold infinities and NaNs) gives inv_w = 0 and one bin, all of it band.
    const float vmin = topk_unkey(kmin), vmax = topk_unkey(kmax);
    float inv_w = (float)SEL_BINS / (vmax - vmin);
    if (!(inv_w > 0.0f) || !(inv_w < 3.0e38f)) inv_w = 0.0f;
    if (inv_w > 0.0f)
        for_keys([&](int, int, uint32_t k) {
            atomicAdd(&hist[(uint32_t)fminf((topk_unkey(k) - vmin) * inv_w, (float)(SEL_BINS - 1))], 1u);
        });
    else if (tid == 0) hist[0] = (uint32_t)nloc;
    const uint32_t* all = hist;
    if constexpr (!SOLO) {
        cluster.sync();                                                       // [2] every CTA's histogram is complete
        const int SL4 = SEL_BINS / 4 / C;                                     // rank r reduces its share and pushes it to everybody
        for (int i = tid; i < SL4; i += SEL_NT) {
            uint4 h[SEL_MAX_CLUSTER], v = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int q = 0; q < SEL_MAX_CLUSTER; ++q)                         // (all remote loads in flight at once)
                h[q] = q < C ? reinterpret_cast<const uint4*>(cluster.map_shared_rank(hist, q < C ? q : 0))[r * SL4 + i] : v;
#pragma unroll
            for (int q = 0; q < SEL_MAX_CLUSTER; ++q) { v.x += h[q].x; v.y += h[q].y; v.z += h[q].z; v.w += h[q].w; }
            for (int q = 0; q < C; ++q) reinterpret_cast<uint4*>(cluster.map_shared_rank(red, q))[r * SL4 + i] = v;
        }
        cluster.sync();                                                       // [3] the whole reduced histogram
        all = red;
    } else {
        __syncthreads();
    }
    {
        // suffix scan: thread t owns the bins 4 t .. 4 t + 3
        const uint4 h = reinterpret_cast<const uint4*>(all)[tid];
        const uint32_t mine = h.x + h.y + h.z + h.w, before = sel_block_excl(mine, xc);
        uint32_t acc = (uint32_t)nt - before - mine;                          // tokens in bins above this thread's
        const uint32_t hb[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int j = 3; j >= 0; --j) {
            if (acc < (uint32_t)kk && (uint32_t)kk <= acc + hb[j]) xc.bstar = (uint32_t)(tid * 4 + j);
            acc += hb[j];
        }
    }
    __syncthreads();

    // ---- 3. classification: surely selected / band (re-scored exactly) / surely not -------------------------
    // The k-th approximate score is one of the tokens of bin `bstar`: it lies between the bin's edges. Their slack covers
    // every rounding of bin_of and of the edges (a few 2^-24 of the larger of |vmin|, |vmax|); it only widens the band.
    uint32_t k_lo = 0u, k_hi = 0xffffffffu;
    if (inv_w > 0.0f) {
        const float w = (vmax - vmin) * (1.0f / (float)SEL_BINS), fb = (float)xc.bstar;
        const float slack = 2.0f * eps + (fabsf(vmin) + fabsf(vmax)) * 1.9073486328125e-6f;   // 2^-19
        const float lo_f = vmin + fb * w - slack, hi_f = (xc.bstar == SEL_BINS - 1 ? vmax : vmin + (fb + 1.0f) * w) + slack;
        if (xc.bstar > 0 && lo_f == lo_f) k_lo = topk_key(lo_f);
        if (hi_f == hi_f) k_hi = topk_key(hi_f);
    }
    // the histogram is dead (its remote readers passed [3]): counters of the ranking; a lone CTA's list ends in empty slots
    static_assert(SEL_LIST + SEL_RANK_ALL <= SEL_BINS, "dec and cnt take the histogram's place");
    hist[SEL_LIST + tid] = 0u;
    uint32_t m_in = 0u, m_band = 0u;                                          // bit 4 * step + e
    {
        uint32_t ge = 0u;                                                     // in the band or above it
        for_keys([&](int it, int e, uint32_t k) {
            m_in |= (k > k_hi ? 1u << e : 0u) << (4 * it);
            ge |= (k >= k_lo ? 1u << e : 0u) << (4 * it);
        });
        m_band = ge & ~m_in;
    }
    auto local_of = [&](int bit) { return ((bit >> 2) * SEL_NT + tid) * 4 + (bit & 3); };
    {   // this CTA's count of surely selected tokens: the warp sums meet at the barrier that closes the list
        const uint32_t v = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(m_in));
        if (lane == 0) xc.red[buf][warp] = v;
    }
    uint32_t my_pos;                                                          // list position of this thread's first band token
    {
        const uint32_t cnt = (uint32_t)__popc(m_band);
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        uint32_t wbase = 0u;
        if (lane == 31 && incl) wbase = atomicAdd(&xc.list_n, incl);          // order inside the list is irrelevant
        wbase = __shfl_sync(0xffffffffu, wbase, 31);
        my_pos = wbase + incl - cnt;
        uint32_t pos = my_pos;
        for (uint32_t m = m_band; m && pos < SEL_LIST; m &= m - 1u, ++pos) {
            const int bit = __ffs(m) - 1, i = local_of(bit);
            l_tok[pos] = (uint32_t)(c0 + i);
            if (!VALUES) l_row[pos] = row_of_bit(bit, i);
            if (VALUES) l_cmp[pos] = ((uint64_t)keys[i] << 32) | ~(uint32_t)(c0 + i);
        }
    }
    __syncthreads();
    const uint32_t n_in_mine = __reduce_add_sync(0xffffffffu, xc.red[buf][lane]);
    buf ^= 1;
    const uint32_t n_band_mine = xc.list_n;
    if (SOLO && tid < 8 && n_band_mine + tid < (uint32_t)SEL_LIST) l_cmp[n_band_mine + tid] = 0ull;

    // Exact key of the first `ln` listed tokens -> l_cmp[position] (0 and ~0 are reserved for "surely out" / "surely in").
    auto rescore = [&](uint32_t ln) {
        rv_rescore_listed<SEL_NW>([&](uint32_t i) { return l_row[i]; }, ln, qf, kfw + warp * (SEL_HD * 4), g, A.index_pool, A.index_scale, my_sq, my_wh,
                                  [&](uint32_t pos, float score) {
            uint32_t ku = topk_key(score);
            ku = ku == 0xffffffffu ? 0xfffffffeu : (ku == 0u ? 1u : ku);
            l_cmp[pos] = ((uint64_t)ku << 32) | ~l_tok[pos];
        });
    };
    // ascending write-out of this CTA's tokens whose bit is set in `sel`, from slot `base` on (one barrier)
    auto write_out = [&](uint32_t sel, uint32_t base) {
        uint32_t before[SEL_STEPS];
        sel_token_excl(sel, xc, before);
#pragma unroll
        for (int it = 0; it < SEL_STEPS; ++it) {
            uint32_t pos = base + before[it];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (sel & (1u << (4 * it + e))) out[pos++] = (uint32_t)(c0 + it * SEL_STEP + tid * 4 + e);
        }
    };

    // ---- 4. exact keys of the band -------------------------------------------------------------------------
    if constexpr (!VALUES)
        if (n_band_mine <= (uint32_t)SEL_LIST) rescore(n_band_mine);
    __syncthreads();
    uint32_t n_in = n_in_mine, n_band = n_band_mine;
    const uint32_t RG = SEL_LIST / C;                                         // entries of one rank in everybody's gathered list
    uint32_t n_all = n_band_mine;                                             // gathered entries, empty slots included
    if constexpr (!SOLO) {
        {   // a warp serves one destination; entry i of rank r goes to slot i * C + r, so that the lists end close together
            const int q = warp & (C - 1);
            uint64_t* dst = cluster.map_shared_rank(a_cmp, q) + r;
            for (uint32_t i = (warp / C) * 32 + lane; i < min(n_band_mine, RG); i += (SEL_NW / C) * 32) dst[i * C] = l_cmp[i];
            if (tid < C) {
                SelXc* dx = cluster.map_shared_rank(&xc, tid);
                dx->n_in[r] = n_in_mine; dx->n_band[r] = n_band_mine;
            }
        }
        cluster.sync();                                                       // [4] counts and lists
        const uint32_t nb = lane < C ? xc.n_band[lane] : 0u;
        n_in = __reduce_add_sync(0xffffffffu, lane < C ? xc.n_in[lane] : 0u);
        n_band = __reduce_add_sync(0xffffffffu, nb);
        n_all = __reduce_max_sync(0xffffffffu, nb) * C;
    }

    if (n_band <= (uint32_t)SEL_LIST) {
        // ---- common case: the whole band fits the list ------------------------------------------------------
        const uint64_t* all_cmp = SOLO ? l_cmp : a_cmp;
        const uint32_t take = (uint32_t)kk - n_in;   // >= 1: fewer than kk tokens lie above the band
        uint32_t* dec = hist;                                                 // per own list entry: selected
        uint32_t base = 0u;
        // Band tokens are ranked among ALL of them by (exact key descending, index ascending).
        const bool rank_all = n_all <= (uint32_t)SEL_RANK_ALL;
        if (rank_all) {
            // `parts` threads per entry, each against its share of the list in batches of eight (one pair of entries at a
            // time costs a shared-memory round trip a pair: 320 entries 8,800 cycles); their counts meet in `cnt`. The
            // selected entries of the lower ranks say where this CTA's rows begin.
            uint32_t* cnt = hist + SEL_LIST;                                  // [SEL_RANK_ALL], zeroed with the list
            const int sh = n_all <= SEL_NT / 8 ? 3 : (n_all <= SEL_NT / 4 ? 2 : (n_all <= SEL_NT / 2 ? 1 : 0));
            const uint32_t e = (uint32_t)tid & ((SEL_NT >> sh) - 1), per = (((n_all + 7) / 8 + (1u << sh) - 1) >> sh) * 8;
            const uint64_t mine = e < n_all ? all_cmp[e] : 0ull;
            if (e < n_all) {
                const uint32_t j0 = ((uint32_t)tid >> (10 - sh)) * per, j1 = min(j0 + per, (n_all + 7) / 8 * 8);
                uint32_t c = 0;
#pragma unroll 1
                for (uint32_t j = j0; j < j1; j += 8) {                       // (broadcast reads; the list ends in empty slots)
                    ulonglong2 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = reinterpret_cast<const ulonglong2*>(all_cmp + j)[u];
#pragma unroll
                    for (int u = 0; u < 4; ++u) c += (v[u].x > mine ? 1u : 0u) + (v[u].y > mine ? 1u : 0u);
                }
                if (c) atomicAdd(&cnt[e], c);
            }
            __syncthreads();
            if (tid < (int)n_all) {
                const bool win = cnt[tid] < take;
                const int q = SOLO ? 0 : tid & (C - 1);
                if (q == r) dec[SOLO ? tid : tid / C] = win ? 1u : 0u;        // (an empty slot's entry is never looked at)
                else if (q < r && win && mine != 0ull) atomicAdd(&xc.lower, 1u);
            }
        } else {
            if (!SOLO && n_all > (uint32_t)SEL_LIST) {                        // one rank's share alone exceeds its slots: pull instead
                cluster.sync();                                               // nobody writes our gathered list any more
                uint32_t off = 0u;
                for (int q = 0; q < C; ++q) {
                    const uint32_t nq = xc.n_band[q];
                    const uint64_t* src = cluster.map_shared_rank(l_cmp, q);
                    for (uint32_t i = tid; i < nq; i += SEL_NT) a_cmp[off + i] = src[i];
                    off += nq;
                }
                n_all = n_band;
                cluster.sync();
            }
#pragma unroll 1
            for (uint32_t i = warp; i < n_band_mine; i += SEL_NW) {           // a warp per own entry
                const uint64_t mine = l_cmp[i];
                uint32_t c = 0;
#pragma unroll 4
                for (uint32_t j = lane; j < n_all; j += 32) c += all_cmp[j] > mine ? 1u : 0u;
                c = __reduce_add_sync(0xffffffffu, c);
                if (lane == 0) dec[i] = c < take ? 1u : 0u;
            }
        }
        __syncthreads();
        uint32_t sel = m_in;
        {
            uint32_t pos = my_pos;
            for (uint32_t m = m_band; m; m &= m - 1u, ++pos)
                if (dec[pos]) sel |= m & (0u - m);
        }
        if constexpr (!SOLO) {
            if (rank_all) {
                base = __reduce_add_sync(0xffffffffu, lane < r ? xc.n_in[lane] : 0u) + xc.lower;
            } else {
                const uint32_t n_out_mine = sel_block_sum((uint32_t)__popc(sel), xc, buf);
                if (tid < C) cluster.map_shared_rank(&xc, tid)->n_out[r] = n_out_mine;
                cluster.sync();
                for (int q = 0; q < r; ++q) base += xc.n_out[q];
            }
        }
        write_out(sel, base);
        if (r == 0 && tid == 0 && A.stats) { A.stats[b * 2] = n_band; A.stats[b * 2 + 1] = n_in; }
        return;
    }

    // ---- slow path (tie-dominated scores): the band does not fit the list --------------------------------------
    // Exact keys replace the approximate ones: surely-in -> all ones, surely-out -> 0, band -> exact key (re-scored in chunks
    // of SEL_LIST consecutive tokens, so a chunk's band always fits the list).
    if constexpr (!VALUES) {
#pragma unroll 1
        for (int ch = 0; ch < nloc; ch += SEL_LIST) {
            __syncthreads();
            if (tid == 0) xc.list_n = 0;
            __syncthreads();
            // a thread's four tokens of a step lie in one chunk: which of its bits are in this one
            const int it = ch / SEL_STEP;
            const bool mine = (it * SEL_NT + tid) * 4 / SEL_LIST == ch / SEL_LIST;
            const uint32_t bits = mine ? (m_band >> (4 * it)) & 0xfu : 0u;
            const int i4 = (it * SEL_NT + tid) * 4;
            uint32_t pos0 = bits ? atomicAdd(&xc.list_n, (uint32_t)__popc(bits)) : 0u;
            {
                uint32_t pos = pos0;
                for (uint32_t m = bits; m; m &= m - 1u, ++pos) {
                    const int e = __ffs(m) - 1;
                    l_tok[pos] = (uint32_t)(c0 + i4 + e);
                    l_row[pos] = row_of_bit(4 * it + e, i4 + e);
                }
            }
            __syncthreads();
            rescore(xc.list_n);
            __syncthreads();
            for (uint32_t m = bits; m; m &= m - 1u) keys[i4 + __ffs(m) - 1] = (uint32_t)(l_cmp[pos0++] >> 32);
        }
#pragma unroll 1
        for (int bit = 0; bit < 4 * steps; ++bit) {
            const int i = local_of(bit);
            if (i < nloc && !((m_band >> bit) & 1u)) keys[i] = ((m_in >> bit) & 1u) ? 0xffffffffu : 0u;
        }
    }
    // exact cluster-wide radix selection, four 8-bit digits, MSB first; per-warp histograms so that ties never
    // serialise a CTA on one bin; whist takes the place of `hist` and both lists, the CTA's digit histogram goes to red[0 .. 256)
    uint32_t pivot = 0u, mask = 0u, need = (uint32_t)kk;
    uint32_t* whist = hist;                                                   // [warps][256]
    static_assert(SEL_NW * 256 <= SEL_BINS + 3 * SEL_LIST, "the digit histograms fit");
    uint32_t* dig = red;
    uint32_t* sum = red + 256;
    if constexpr (!SOLO) cluster.sync();                                      // nobody reads our lists any more
#pragma unroll 1
    for (int sh2 = 24; sh2 >= 0; sh2 -= 8) {
        __syncthreads();
        for (int i = tid; i < SEL_NW * 256; i += SEL_NT) whist[i] = 0u;
        __syncthreads();
        for_keys([&](int, int, uint32_t k) {
            if ((k & mask) == pivot) atomicAdd(&whist[warp * 256 + ((k >> sh2) & 0xffu)], 1u);
        });
        __syncthreads();
        if (tid < 256) {
            uint32_t t = 0;
#pragma unroll 8
            for (int w2 = 0; w2 < SEL_NW; ++w2) t += whist[w2 * 256 + tid];
            dig[tid] = t;
        }
        __syncthreads();
        if constexpr (!SOLO) cluster.sync();                                  // every CTA's digit histogram
        if (tid < 256) {
            uint32_t t = 0;
            for (int q = 0; q < C; ++q) t += SOLO ? dig[tid] : cluster.map_shared_rank(dig, q)[tid];
            sum[tid] = t;
        }
        __syncthreads();
        if (warp == 0) {
            // lane owns bins 8 * lane .. 8 * lane + 7; acc = entries in strictly higher bins
            uint32_t h[8], tot = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) { h[j] = sum[lane * 8 + j]; tot += h[j]; }
            uint32_t incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_down_sync(0xffffffffu, incl, o);
                if (lane + o < 32) incl += v;
            }
            uint32_t acc = incl - tot;
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                if (acc < need && need <= acc + h[j]) {
                    xc.pivot = pivot | ((uint32_t)(lane * 8 + j) << sh2);
                    xc.need = need - acc;
                }
                acc += h[j];
            }
        }
        __syncthreads();
        pivot = xc.pivot;
        need = xc.need;
        mask |= 0xffu << sh2;
        if constexpr (!SOLO) cluster.sync();                                  // dig may be rewritten by the next digit
    }
    // `need` of the tokens tied at the pivot are taken, in ascending global index = ascending rank, then token order
    uint32_t sel_gt = 0u, sel_eq = 0u;
    for_keys([&](int it, int e, uint32_t k) {
        if (k > pivot) sel_gt |= 1u << (4 * it + e);
        else if (k == pivot) sel_eq |= 1u << (4 * it + e);
    });
    uint32_t base = 0u, eq_lower = 0u;
    if constexpr (!SOLO) {
        const uint32_t gt_mine = sel_block_sum((uint32_t)__popc(sel_gt), xc, buf);
        const uint32_t eq_mine = sel_block_sum((uint32_t)__popc(sel_eq), xc, buf);
        if (tid < C) {
            SelXc* dst = cluster.map_shared_rank(&xc, tid);
            dst->cnt_gt[r] = gt_mine; dst->cnt_eq[r] = eq_mine;
        }
        cluster.sync();
        for (int q = 0; q < r; ++q) {
            const uint32_t left = need > eq_lower ? need - eq_lower : 0u;
            base += xc.cnt_gt[q] + min(xc.cnt_eq[q], left);
            eq_lower += xc.cnt_eq[q];
        }
    }
    const uint32_t need_mine = need > eq_lower ? need - eq_lower : 0u;          // ties this CTA may still take
    uint32_t ties[SEL_STEPS];
    sel_token_excl(sel_eq, xc, ties);
    uint32_t sel = sel_gt;
#pragma unroll
    for (int it = 0; it < SEL_STEPS; ++it) {
        uint32_t e0 = ties[it];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (sel_eq & (1u << (4 * it + e))) { if (e0 < need_mine) sel |= 1u << (4 * it + e); ++e0; }
    }
    __syncthreads();                                                          // (the prefix partials are written again)
    write_out(sel, base);
    if (r == 0 && tid == 0 && A.stats) { A.stats[b * 2] = n_band; A.stats[b * 2 + 1] = 0; }
}

// ---------------------------------------------------------------------------------------------
// The same selection over at most 768 given scores: a thread per score, one CTA per sequence. The k-th largest key is found bit
// by bit from the top, a barrier that counts per bit; ties at it go to the lower indices. Bound by its 32 barriers (1 us with nine
// warps; they take longer the more warps meet at them). It reads the scores once and keeps nothing but a key per thread. us a step of
// the 16-head layer, the kernel above -> this one: one sequence of 100 tokens 16.7 -> 14.8, 257 16.6 -> 15.3, 512 16.7 -> 15.8, 768 16.8
// both, 1,024 16.8 -> 17.6; four of 640 18.2 -> 17.7, 1,024 18.2 -> 21.2; eight of 768 19.4 -> 19.1, 896 19.3 -> 19.4. So up to 768.
// ---------------------------------------------------------------------------------------------
constexpr int SEL_SMALL = 768;

__global__ void __launch_bounds__(SEL_SMALL)
index_select_small_kernel(const float* __restrict__ scores, long long stride, const int32_t* __restrict__ seq_len, int nt_single,
                          int max_nt, int k, uint32_t* __restrict__ rows, int32_t* __restrict__ n_sel) {
    __shared__ uint32_t w_eq[32], w_sel[32];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    const int nt = min(seq_len ? seq_len[b] : nt_single, max_nt), kk = min(k, nt);
    const float v = tid < nt ? scores[(size_t)b * stride + tid] : 0.0f;
    uint32_t* out = rows + (size_t)b * k;
    if (tid == 0 && n_sel) n_sel[b] = kk > 0 ? kk : 0;
    if (kk == nt || kk <= 0) {                              // everything (or nothing) is selected: the identity
        if (tid < nt) out[tid] = (uint32_t)tid;
        return;
    }
    const uint32_t key = topk_key(v);
    const bool live = tid < nt;
    uint32_t pivot = 0u;                                    // the largest value that kk keys reach
#pragma unroll 1
    for (uint32_t bit = 0x80000000u; bit; bit >>= 1)
        if (__syncthreads_count(live && key >= (pivot | bit)) >= kk) pivot |= bit;
    const int above = __syncthreads_count(live && key > pivot);
    // ties at the pivot, in index order, then the slots of the selected
    const unsigned below = (1u << lane) - 1u, eq = __ballot_sync(0xffffffffu, live && key == pivot);
    if (lane == 0) w_eq[warp] = (uint32_t)__popc(eq);
    __syncthreads();
    const uint32_t eq_before = __reduce_add_sync(0xffffffffu, lane < warp ? w_eq[lane] : 0u) + (uint32_t)__popc(eq & below);
    const bool take = live && (key > pivot || (key == pivot && above + (int)eq_before < kk));
    const unsigned sel = __ballot_sync(0xffffffffu, take);
    if (lane == 0) w_sel[warp] = (uint32_t)__popc(sel);
    __syncthreads();
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? w_sel[lane] : 0u) + (uint32_t)__popc(sel & below);
    if (take) out[before] = (uint32_t)tid;
}

}  // namespace

namespace rivoli {

static std::atomic<int> g_sel_cluster_override{0};

// CTAs per sequence: a lone CTA up to 8,192 tokens at any batch (what the tokens cost is less than the cluster barriers), else
// two or four while each has an SM of its own, and at least enough for 16,384 tokens each. (Eight only when the tokens need
// them: their barriers cost what the shorter steps give, and at one CTA per SM sixteen such clusters do not fit the chip at
// once: 16 sequences of 16,384 tokens 61 us per step with four, 80 with eight.)
static bool select_cluster_plan(int B, int score_stride, int* cluster, int* ch) {
    int C = 1;
    if (score_stride > 8192)
        while (C < 4 && (long long)B * C * 2 <= rv_sm_count()) C *= 2;
    if (const int forced = g_sel_cluster_override.load(std::memory_order_relaxed)) C = forced;
    while (C < SEL_MAX_CLUSTER && (long long)C * SEL_CH < score_stride) C *= 2;
    *cluster = C;
    *ch = ((score_stride + C - 1) / C + 3) / 4 * 4;
    return *ch <= SEL_CH;
}

}  // namespace rivoli

// Test hook: force the cluster size of the following selection launches (1, 2, 4 or 8; 0 = the plan's own choice),
// so that every cluster size can be exercised at any batch size.
extern "C" __attribute__((visibility("default"))) void rivoli_index_select_test_cluster(int cluster) {
    rivoli::g_sel_cluster_override = (cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8) ? cluster : 0;
}

namespace rivoli {

template <bool VALUES, bool SOLO, bool VEC>
static int launch_select(const SelArgs& a, int B, int C, int ch, cudaStream_t st) {
    constexpr size_t fixed = SEL_BINS + 4 * SEL_LIST + (VALUES ? SEL_BINS : SEL_NW * SEL_HD * 4 + RS_QWORDS) + (SOLO ? 0 : 2 * SEL_LIST);
    static_assert((fixed + SEL_CH) * 4 + sizeof(SelXc) + 1024 <= 232448, "shared memory budget");
    const size_t smem = (fixed + (size_t)ch) * 4;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(B * C)); cfg.blockDim = dim3(SEL_NT); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)C; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 2;
    rv_drain_error();
    rv_allow_smem<index_select_cluster_kernel<VALUES, SOLO, VEC>>((int)((fixed + SEL_CH) * 4));
    (void)cudaLaunchKernelEx(&cfg, index_select_cluster_kernel<VALUES, SOLO, VEC>, a, ch);
    return rv_launch_status();
}

int launch_index_select_cluster(const SelArgs& a, int B, cudaStream_t st) {
    int C = 1, ch = 0;
    if (!select_cluster_plan(B, a.score_stride, &C, &ch)) return 1002;
    if (a.vec_scores) return C == 1 ? launch_select<false, true, true>(a, B, C, ch, st) : launch_select<false, false, true>(a, B, C, ch, st);
    return C == 1 ? launch_select<false, true, false>(a, B, C, ch, st) : launch_select<false, false, false>(a, B, C, ch, st);
}

int launch_topk_values(const float* scores, long long stride, const int32_t* seq_len, int nt_single, int B, int k,
                       uint32_t* rows, int32_t* n_sel, int max_nt, cudaStream_t st) {
    if (max_nt > SEL_MAX_CLUSTER * SEL_CH || stride > 0x7fffffff) return 1002;
    if (max_nt <= SEL_SMALL) {
        rv_drain_error();
        rv_launch_dependent(index_select_small_kernel, dim3((unsigned)B), dim3((unsigned)((max_nt + 31) / 32 * 32)), 0, st, scores, stride, seq_len,
                            nt_single, max_nt, k, rows, n_sel);
        return rv_launch_status();
    }
    SelArgs a{};
    a.scores = scores; a.score_stride = max_nt; a.value_stride = stride; a.seq_len = seq_len; a.nt_single = nt_single;
    a.rows = rows; a.n_sel = n_sel; a.k = k;
    a.vec_scores = ((uintptr_t)scores & 15) == 0 && stride % 4 == 0 && stride >= max_nt;   // (whole vectors are read)
    // no re-score to spread: a lone CTA up to 16,384 scores (no exchanges between CTAs; 8,193 scores: 9.7 us,
    // four radix passes over shared memory took 14.2), beyond that clusters of eight
    const int C = max_nt <= SEL_CH ? 1 : SEL_MAX_CLUSTER, ch = ((max_nt + C - 1) / C + 3) / 4 * 4;
    if (a.vec_scores) return C == 1 ? launch_select<true, true, true>(a, B, C, ch, st) : launch_select<true, false, true>(a, B, C, ch, st);
    return C == 1 ? launch_select<true, true, false>(a, B, C, ch, st) : launch_select<true, false, false>(a, B, C, ch, st);
}

}  // namespace rivoli
