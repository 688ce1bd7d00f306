// Lightning-indexer selection on the tensor cores, with an exactness guarantee.
//
// The indexer reads 132 bytes per cached token and spends 8192 FLOP on them (~62 FLOP/B),
// so only tensor cores keep it HBM-bound. But an MMA does not accumulate in the fixed
// order the reference's score is defined in, so its scores can differ from the exact ones
// in the last bits, which would move top-k indices at the cut. This file therefore does:
//
//   1. index_q_prepare_kernel   q -> e4m3 codes + per-head scale (bit-exact codec), plus one
//                               error-bound constant per sequence. On the fused decode path
//                               (rivoli_dsa_append_select_paged) the same work runs in
//                               step_prologue_kernel, whose extra blocks append the step's tokens.
//   2. index_score_mma_kernel   approximate scores a_t for every cached token: fp8 keys are
//                               streamed page by page by TMA (one 2-D box per page) into swizzled
//                               shared memory and consumed by tcgen05.mma kind::f8f6f4
//                               (tokens = M 128, heads = N 32, dims = K 128), accumulators
//                               in TMEM, scale/ReLU/head-weight epilogue from TMEM.
//   3. index_select_cluster_kernel (index_select.cu)  per sequence, one thread-block cluster: locate
//                               the bin of the k-th approximate score A_k with one histogram pass;
//                               every token within 2*eps of that bin is re-scored in
//                               the exact order (sequential f32 fold, identical to
//                               rivoli_index_score_paged); tokens above the band are in,
//                               below are out; the final exact top-k (ties -> lower index)
//                               is emitted ascending.
//
// Why this yields the exact top-k set: with |a_t - o_t| <= eps for the exact scores o_t,
// the k-th largest values satisfy |A_k - E_k| <= eps, so a_t > A_k + 2 eps implies
// o_t > E_k (selected) and a_t < A_k - 2 eps implies o_t < E_k (not selected); everything
// else is decided on exact scores. eps per sequence = max key scale * sum_h |w_h ws| ds
// s_q[h] ||qcode_h||_1 * 448 * 2^-16: a bound on sum |q_d k_d| (no key code exceeds 448; with the
// 2-norms of both it was a quarter wider, and the band with it) times 2^-16 relative error. The sequential fold's own worst case is hd * 2^-24 = 2^-17
// of sum |q_d k_d|; the tensor core measured 2^-21.9 on full-range random codes.
#include "codec.cuh"
#include "common.cuh"
#include "quant.cuh"
#include "tc_common.cuh"
#include "index_select.hpp"
#include "tmap.hpp"

namespace {

constexpr int IM_TILE = 128;       // tokens per MMA tile (M)
constexpr int IM_HD = 128;         // index dim = one 128-byte swizzle row
constexpr int IM_NPAD = 32;        // heads padded to N = 32
constexpr int IM_NS = 6;           // key-tile stages in flight
constexpr int IM_NACC = 4;         // TMEM accumulators (32 columns each)
constexpr int IM_TPI = 16;         // most tiles per work item
constexpr int IM_THREADS = 192;    // warps 0-3 epilogue, 4 producer, 5 MMA
constexpr int IM_STAGE_BYTES = IM_TILE * IM_HD;   // 16 KiB
constexpr int IM_Q_BYTES = IM_NPAD * IM_HD;       // 4 KiB
constexpr float IM_EPS_REL = 1.52587890625e-05f;  // 2^-16
constexpr int IM_ERR_BAD_PAGE = 1005;             // error word: a block-table entry inside seq_len lies outside the pool

struct IndexMmaArgs {
    DsaGeom g;
    const uint8_t* qcodes; const float* qscales; const float* w;
    const uint8_t* index_pool; const float* index_scale; const int32_t* block_table; const int32_t* seq_len;
    float* scores; int score_stride; int B;
    int* err;              // device error word (0 = ok)
};

// ---------------------------------------------------------------------------------------------
// 1. q quantisation + per-sequence error-bound constant. One CTA per sequence, one warp per head.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void
index_q_prepare_block(int b, const uint16_t* __restrict__ q, const float* __restrict__ w, int nh, int hd, float wscale,
                      float dscale, uint8_t* __restrict__ codes, float* __restrict__ scales, float* __restrict__ cb,
                      int* __restrict__ err, float* term) {
    const int h = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (h < nh) {
        const size_t v = (size_t)b * nh + h;
        // same codec path as rivoli_index_q_quant (index_dim is 128 here): eight values per lane, sixteen lanes
        const bool act = lane < IM_HD / 8;
        const uint4 x = act ? *reinterpret_cast<const uint4*>(q + v * IM_HD + lane * 8) : make_uint4(0u, 0u, 0u, 0u);
        const float wv = w[v];
        uint32_t m = rv_absmax8(x);
#pragma unroll
        for (int o = IM_HD / 16; o > 0; o >>= 1) m = rv_max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, o));
        const QuantScale qs = rv_quant_scale(__uint_as_float(m << 16));
        float n1 = 0.0f;
        if (act) {
            uint32_t redo = qs.r == 0.0f ? RV_REDO : 0u;
            uint2 c = rv_codes8(x, qs, redo);
            if (redo & RV_REDO) c = rv_codes8_exact(x, qs.s);
            *reinterpret_cast<uint2*>(codes + v * IM_HD + lane * 8) = c;
            const uint32_t cc[2] = {c.x, c.y};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float2 lo = rv_e4m3x2_to_f32x2((uint16_t)(cc[i] & 0xffff)), hi = rv_e4m3x2_to_f32x2((uint16_t)(cc[i] >> 16));
                n1 += fabsf(lo.x) + fabsf(lo.y) + fabsf(hi.x) + fabsf(hi.y);
            }
        }
#pragma unroll
        for (int o = IM_HD / 16; o > 0; o >>= 1) n1 += __shfl_xor_sync(0xffffffffu, n1, o);
        if (lane == 0) {
            scales[v] = qs.s;
            term[h] = fabsf(wv * wscale) * dscale * qs.s * n1;
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const float sum = rv_warp_sum(lane < nh ? term[lane] : 0.0f);
        // no key code is larger than 448; 1.01 covers the roundings of this very sum
        if (lane == 0) {
            cb[b] = sum * 448.0f * IM_EPS_REL * 1.01f;
            if (b == 0) *err = 0;   // the scorer's error word starts clean on every call
        }
    }
}

__global__ void __launch_bounds__(1024)
index_q_prepare_kernel(const uint16_t* __restrict__ q, const float* __restrict__ w, int nh, int hd, float wscale,
                       float dscale, uint8_t* __restrict__ codes, float* __restrict__ scales, float* __restrict__ cb,
                       int* __restrict__ err) {
    __shared__ float term[32];
    rv_grid_dep_wait();
    rv_grid_dep_trigger();   // the scorer may set itself up while this runs; it waits before reading these outputs
    index_q_prepare_block(blockIdx.x, q, w, nh, hd, wscale, dscale, codes, scales, cb, err, term);
}

// Decode-step prologue in one launch: blocks [0, B) prepare the indexer query of sequence b,
// the blocks behind them append the step's new token of PROLOGUE_ROWS sequences each (one warp per row).
// The two halves touch disjoint memory.
struct AppendArgs {
    const uint16_t* latent; const uint16_t* index_key; const int32_t* row_pos; const int32_t* block_table;
    uint8_t* latent_pool; float* latent_scale; uint8_t* index_pool; float* index_scale; int32_t* status;
};

// Rows appended by a block: 4, or 8 or 16 where only so every block has an SM of its own, else 32. 32 -> 4 rows, us a step: 32 sequences
// of 4,096 45.7 -> 44.7, of up to 32,768 61.8 -> 61.0, 64 of 8,192 68.8 -> 68.2, 90 of 2,000 - 4,000 38.1 -> 37.2. At 128 sequences of 900 /
// 4,000 - 8,000 tokens: 4 rows 36.5 / 59.8, 32 rows 35.9 / 59.2, 8 rows (144 blocks) 35.4 / 58.6; 119 of 900: 35.6, 35.9, 34.6.
constexpr int PROLOGUE_ROWS_FEW = 4, PROLOGUE_ROWS_MOST = 32;
__global__ void __launch_bounds__(1024)
step_prologue_kernel(DsaGeom g, AppendArgs ap, int B, int per_block, const uint16_t* __restrict__ q, const float* __restrict__ w,
                     uint8_t* __restrict__ codes, float* __restrict__ scales, float* __restrict__ cb,
                     int* __restrict__ err) {
    __shared__ float term[32];
    rv_grid_dep_wait();
    rv_grid_dep_trigger();   // the scorer may set itself up while this runs; it waits before reading these outputs
    if ((int)blockIdx.x < B) {
        index_q_prepare_block(blockIdx.x, q, w, g.index_heads, g.index_dim, g.index_wscale, g.index_dscale, codes, scales,
                              cb, err, term);
        return;
    }
    const int row = ((int)blockIdx.x - B) * per_block + (threadIdx.x >> 5);
    if (row >= B || (int)(threadIdx.x >> 5) >= per_block) return;
    AppendRow<3> a;
    append_row_load<3>(a, g, ap.latent, ap.index_key, row, row, ap.row_pos[row], ap.block_table, threadIdx.x & 31);
    append_row_store<3>(a, g, ap.latent_pool, ap.latent_scale, ap.index_pool, ap.index_scale, ap.status, threadIdx.x & 31);
}

// The prologue of geometries whose scores come from the CUDA-core kernel: a warp per query vector, then a warp per row to
// append.
__global__ void __launch_bounds__(256)
step_quant_kernel(DsaGeom g, AppendArgs ap, int B, const uint16_t* __restrict__ q, uint8_t* __restrict__ codes,
                  float* __restrict__ scales) {
    const int lane = threadIdx.x & 31, id = blockIdx.x * 8 + (threadIdx.x >> 5), n_vec = B * g.index_heads;
    rv_grid_dep_wait();
    rv_grid_dep_trigger();
    if (id < n_vec) {
        const float s = quant_vec(q + (size_t)id * g.index_dim, g.index_dim, codes + (size_t)id * g.index_dim, lane);
        if (lane == 0) scales[id] = s;
    } else if (id < n_vec + B) {
        const int row = id - n_vec;
        AppendRow<3> a;
        append_row_load<3>(a, g, ap.latent, ap.index_key, row, row, ap.row_pos[row], ap.block_table, lane);
        append_row_store<3>(a, g, ap.latent_pool, ap.latent_scale, ap.index_pool, ap.index_scale, ap.status, lane);
    }
}

// A batch whose every sequence fits top_k (the score rows are no longer than that) selects everything: no query, no score
// and no cut are needed. Blocks [0, B) write the identity rows of a sequence, block B checks the sequences' pages as the
// scorer does when it reads them, blocks from B + 1 on append the step's tokens (a warp per row). One launch takes the
// place of prologue, scorer and selection: 32 sequences of 2,048 tokens 41.7 -> 32.2 us per step.
constexpr int SD_THREADS = 256;
__global__ void __launch_bounds__(SD_THREADS)
step_dense_kernel(DsaGeom g, AppendArgs ap, int B, const int32_t* __restrict__ block_table, const int32_t* __restrict__ seq_len,
                  int score_stride, uint32_t* __restrict__ rows, int32_t* __restrict__ n_sel, unsigned int* __restrict__ stats,
                  int* __restrict__ err) {
    rv_grid_dep_wait();
    rv_grid_dep_trigger();   // (after the wait: the attention behind this reads its q, the lengths and all pool rows but the new ones at once)
    const int tid = threadIdx.x, blk = (int)blockIdx.x;
    if (blk < B) {
        const int n = min(min(seq_len[blk], score_stride), g.top_k);
        uint32_t* out = rows + (size_t)blk * g.top_k;
        for (int i = tid; i < n; i += SD_THREADS) out[i] = (uint32_t)i;
        if (tid == 0) {
            n_sel[blk] = n > 0 ? n : 0;
            stats[blk * 2] = 0; stats[blk * 2 + 1] = (unsigned)max(n, 0);
        }
    } else if (blk == B) {
        const int per = (score_stride + g.page_tokens - 1) / g.page_tokens;
        bool bad = false;
#pragma unroll 8
        for (int e = tid; e < B * per; e += SD_THREADS) {   // (the stride is within the table, so every lp is)
            const int b = e / per, lp = e - b * per, pg = block_table[(size_t)b * g.max_pages_per_seq + lp];
            bad |= lp * g.page_tokens < min(seq_len[b], score_stride) && (pg < 0 || pg >= g.n_pool_pages);
        }
        bad = __syncthreads_or(bad);
        if (tid == 0) *err = bad ? IM_ERR_BAD_PAGE : 0;
    } else {
        const int row = (blk - B - 1) * (SD_THREADS / 32) + (tid >> 5);
        if (row >= B) return;
        AppendRow<3> a;
        append_row_load<3>(a, g, ap.latent, ap.index_key, row, row, ap.row_pos[row], ap.block_table, tid & 31);
        append_row_store<3>(a, g, ap.latent_pool, ap.latent_scale, ap.index_pool, ap.index_scale, ap.status, tid & 31);
    }
}

// ---------------------------------------------------------------------------------------------
// 2. approximate scores on the tensor cores (persistent CTAs, warp specialised)
// ---------------------------------------------------------------------------------------------
struct ImBarriers {
    uint64_t full[IM_NS], empty[IM_NS], tfull[IM_NACC], tempty[IM_NACC], qfree[2];
};

// Tiles of sequence b that need a score: none if the selection takes all its tokens anyway.
__device__ __forceinline__ int scored_tokens(const IndexMmaArgs& A, int b) {
    const int nt = min(A.seq_len[b], A.score_stride);
    return nt <= A.g.top_k ? 0 : nt;
}
__device__ __forceinline__ int scored_tiles(const IndexMmaArgs& A, int b) { return (scored_tokens(A, b) + IM_TILE - 1) / IM_TILE; }

// A CTA's share: the tiles of all sequences in one row, split evenly over the grid (a ragged batch in equal items of 16 tiles
// left some CTAs twice the work of others: 32 sequences of 512 to 32,768 tokens 28 us, 19 now). It is walked in items
// of at most IM_TPI tiles of one sequence; every role of the CTA walks the same items.
struct ImShare {
    int b, t, left;        // next tile: tile t of sequence b; tiles left
    int nt, t1;            // of the current item: the sequence's tokens, its end
    __device__ __forceinline__ bool next(const IndexMmaArgs& A) {   // advances to the item [t, t1) of sequence b
        if (left <= 0) return false;
        for (;; ++b, t = 0) {
            if (b >= A.B) return false;
            nt = scored_tokens(A, b);
            if (t < (nt + IM_TILE - 1) / IM_TILE) break;
        }
        t1 = min(min(t + IM_TPI, (nt + IM_TILE - 1) / IM_TILE), t + left);
        left -= t1 - t;
        return true;
    }
};
// The share of this CTA, by one warp (two passes over the lengths: all tiles, then where the share begins).
__device__ __forceinline__ ImShare im_share(const IndexMmaArgs& A) {
    const int lane = threadIdx.x & 31;
    int total = 0;
    for (int b0 = 0; b0 < A.B; b0 += 32) total += __reduce_add_sync(0xffffffffu, b0 + lane < A.B ? scored_tiles(A, b0 + lane) : 0);
    const int lo = (int)((long long)total * blockIdx.x / gridDim.x), hi = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
    ImShare r{0, 0, hi - lo, 0, 0};
    int before = 0;
    for (int b0 = 0; b0 < A.B && hi > lo; b0 += 32) {
        const int n = b0 + lane < A.B ? scored_tiles(A, b0 + lane) : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        const unsigned hit = __ballot_sync(0xffffffffu, before + incl > lo);
        if (hit) {
            const int l = __ffs(hit) - 1;
            r.b = b0 + l;
            r.t = lo - (before + __shfl_sync(0xffffffffu, incl - n, l));
            break;
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    return r;
}

__global__ void __launch_bounds__(IM_THREADS)
index_score_mma_kernel(IndexMmaArgs A, const __grid_constant__ CUtensorMap tm_keys,
                       const __grid_constant__ CUtensorMap tm_q) {
    extern __shared__ __align__(1024) uint8_t im_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(im_smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* s_keys = smem;                                   // IM_NS x 16 KiB
    uint8_t* s_q = smem + IM_NS * IM_STAGE_BYTES;             // 2 x 4 KiB
    __shared__ ImBarriers bars;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;
    __shared__ float s_wh[IM_NPAD];
    __shared__ int s_pg[IM_TPI * (IM_TILE / 16)];
    __shared__ ImShare s_share;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const DsaGeom& g = A.g;
    const int nh = g.index_heads, P = g.page_tokens;

    if (tid == 0) {
        for (int i = 0; i < IM_NS; ++i) { tc::mbar_init(&bars.full[i], 1); tc::mbar_init(&bars.empty[i], 1); }
        for (int i = 0; i < IM_NACC; ++i) { tc::mbar_init(&bars.tfull[i], 1); tc::mbar_init(&bars.tempty[i], 4); }
        tc::mbar_init(&bars.qfree[0], 1); tc::mbar_init(&bars.qfree[1], 1);
        tc::mbar_init_fence();
        abort_flag = 0;
    }
    // q tiles start zeroed: rows >= nh are never loaded and must contribute exact zeros
    for (int i = tid; i < 2 * IM_Q_BYTES / 16; i += IM_THREADS) reinterpret_cast<uint4*>(s_q)[i] = make_uint4(0, 0, 0, 0);
    if (warp == 5) tc::tmem_alloc<IM_NACC * 32>(&tmem_base_s);
    // (the lengths are an input of the call whose first kernel is the one before this: complete before that kernel's trigger)
    if (warp == 4) { const ImShare sh = im_share(A); if (lane == 0) s_share = sh; }
    tc::fence_proxy_async();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    rv_grid_dep_wait();      // query codes, head scales and this step's appended keys come from the kernel before
    rv_grid_dep_trigger();   // the selection kernel may start (after the wait: it reads all but the scores at once)

    ImShare sh = s_share;
    if (warp == 4) {
        // ------------------------------ producer: TMA page loads ----------------------------------
        // A page is P rows x 128 bytes, contiguous in the pool; one 2-D TMA box per page lands it in
        // shared memory already in the 128-byte-swizzled K-major form the MMA consumes. The whole
        // warp fetches an item's page ids once; lane 0 then issues one instruction per page.
        int it = 0, items_done = 0;
        bool ok = true;
        const int ppt = IM_TILE / P;  // pages per tile (16 <= P <= 128)
        for (; ok && sh.next(A); sh.t = sh.t1) {
            const int b = sh.b, nt = sh.nt;
            const int first_lp = sh.t * ppt;
            __syncwarp();
            for (int j = lane; j < (sh.t1 - sh.t) * ppt; j += 32) {
                const int lp = first_lp + j;
                int pg = -1;
                const bool live = lp < g.max_pages_per_seq && lp * P < nt;
                if (live) pg = A.block_table[(size_t)b * g.max_pages_per_seq + lp];
                const bool bad = pg < 0 || pg >= g.n_pool_pages;
                // A page inside the sequence that the table does not map into the pool is never loaded (its
                // tokens get scores of whatever the stage held) and the call is flagged, as the append does.
                if (live && bad) atomicCAS(A.err, 0, IM_ERR_BAD_PAGE);
                s_pg[j] = bad ? -1 : pg;
            }
            __syncwarp();
            const int qb = items_done & 1;
            for (int tile = sh.t; tile < sh.t1 && ok; ++tile) {
                const int s = it % IM_NS;
                ok = tc::mbar_wait_warp(&bars.empty[s], ((it / IM_NS) & 1) ^ 1, &abort_flag, 11);
                if (!ok) break;
                const bool first = tile == sh.t;
                if (first) {
                    ok = tc::mbar_wait_warp(&bars.qfree[qb], ((items_done >> 1) & 1) ^ 1, &abort_flag, 12);
                    if (!ok) break;
                }
                if (lane == 0) {
                    const int pbase = (tile - sh.t) * ppt;
                    uint32_t bytes = first ? (uint32_t)nh * IM_HD : 0u;
                    for (int p2 = 0; p2 < ppt; ++p2) bytes += s_pg[pbase + p2] >= 0 ? (uint32_t)P * IM_HD : 0u;
                    tc::mbar_arrive_expect_tx(&bars.full[s], bytes);
                    if (first)  // this sequence's q codes ride the first tile's barrier
                        tc::tma_load_2d(tc::smem_u32(s_q + qb * IM_Q_BYTES), &tm_q, 0, b * nh, &bars.full[s]);
                    for (int p2 = 0; p2 < ppt; ++p2) {
                        const int pg = s_pg[pbase + p2];
                        if (pg >= 0)
                            tc::tma_load_2d(tc::smem_u32(s_keys + s * IM_STAGE_BYTES + p2 * P * IM_HD), &tm_keys, 0,
                                            pg * P, &bars.full[s]);
                    }
                }
                __syncwarp();
                ++it;
            }
            ++items_done;
        }
    } else if (warp == 5) {
        // ------------------------------ MMA issuer ------------------------------------------------
        int it = 0, items_done = 0;
        bool ok = true;
        const uint32_t idesc = tc::idesc_e4m3(IM_TILE, IM_NPAD, 0, 0);
        for (; ok && sh.next(A); sh.t = sh.t1) {
            const int qb = items_done & 1;
            for (int tile = sh.t; tile < sh.t1 && ok; ++tile) {
                const int s = it % IM_NS, a = it % IM_NACC;
                ok = tc::mbar_wait_warp(&bars.full[s], (it / IM_NS) & 1, &abort_flag, 21) &&
                     tc::mbar_wait_warp(&bars.tempty[a], ((it / IM_NACC) & 1) ^ 1, &abort_flag, 22);
                if (!ok) break;
                tc::tc_fence_after();
                if (tc::elect_one()) {
                    const uint32_t ka = tc::smem_u32(s_keys + s * IM_STAGE_BYTES), qa = tc::smem_u32(s_q + qb * IM_Q_BYTES);
#pragma unroll
                    for (int k = 0; k < IM_HD / 32; ++k)
                        tc::mma_f8(tmem + a * 32, tc::smem_desc_sw128(ka + k * 32, 16, 1024),
                                   tc::smem_desc_sw128(qa + k * 32, 16, 1024), idesc, k > 0);
                    tc::mma_commit(&bars.empty[s]);
                    tc::mma_commit(&bars.tfull[a]);
                    if (tile == sh.t1 - 1) tc::mma_commit(&bars.qfree[qb]);
                }
                __syncwarp();
                ++it;
            }
            ++items_done;
        }
    } else {
        // ------------------------------ epilogue: TMEM -> scores --------------------------------
        int it = 0;
        bool ok = true;
        for (; sh.next(A); sh.t = sh.t1) {
            const int b = sh.b, nt = sh.nt;
            if (tc::barrier_any(1, 128, !ok)) break;   // previous item's constants are no longer read
            if (tid < IM_NPAD) {
                // a_t / s_k = sum_h (w_h ws s_q[h] ds) * max(cd_h, 0): the exact formula up to a few
                // roundings (s_q, s_k, ds > 0 commute with the ReLU); the band covers them
                s_wh[tid] = tid < nh ? A.w[(size_t)b * nh + tid] * g.index_wscale * A.qscales[(size_t)b * nh + tid] *
                                           g.index_dscale : 0.0f;
            }
            tc::named_barrier(1, 128);
            for (int tile = sh.t; tile < sh.t1 && ok; ++tile) {
                const int a = it % IM_NACC;
                const int t = tile * IM_TILE + tid;
                ok = tc::mbar_wait_warp(&bars.tfull[a], (it / IM_NACC) & 1, &abort_flag, 31);
                if (!ok) break;
                tc::tc_fence_after();
                uint32_t r[32];
                tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + a * 32, r);
                tc::tmem_ld_wait();
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&bars.tempty[a]);
                if (t < nt) {
                    float acc = 0.0f;
#pragma unroll
                    for (int h = 0; h < IM_NPAD; ++h) acc = fmaf(s_wh[h], fmaxf(__uint_as_float(r[h]), 0.0f), acc);
                    A.scores[(size_t)b * A.score_stride + t] = acc;   // the key scale s_k[t] is applied by the selector
                }
                ++it;
            }
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc::settle(abort_flag);
        tc::tmem_dealloc<IM_NACC * 32>(tmem);
    }
    if (tid == 0 && abort_flag) atomicCAS(A.err, 0, abort_flag);
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct SelectScratch {
    uint8_t* qcodes; float* qscales; float* cb; int* err; unsigned int* stats; float* scores;
};

SelectScratch carve(const DsaGeom* g, int B, int score_stride, void* scratch, size_t* total) {
    uint8_t* p = static_cast<uint8_t*>(scratch);
    size_t off = 0;
    SelectScratch s;
    auto take = [&](size_t n) { uint8_t* r = p ? p + off : nullptr; off += align_up(n, 256); return r; };
    s.qcodes = take((size_t)B * g->index_heads * g->index_dim);
    s.qscales = reinterpret_cast<float*>(take((size_t)B * g->index_heads * 4));
    s.cb = reinterpret_cast<float*>(take((size_t)B * 4));
    s.err = reinterpret_cast<int*>(take(4));
    s.stats = reinterpret_cast<unsigned int*>(take((size_t)B * 8));
    s.scores = reinterpret_cast<float*>(take((size_t)B * score_stride * 4));
    *total = off;
    return s;
}

constexpr int SEL_MAX_NT = 8 * 16384;   // what one cluster of the selection kernel covers

bool mma_geometry_ok(const DsaGeom* g, int score_stride) {
    return g->index_dim == IM_HD && g->index_heads <= IM_NPAD && g->page_tokens >= 16 && g->page_tokens <= IM_TILE &&
           score_stride <= SEL_MAX_NT;
}

}  // namespace

RIVOLI_API size_t rivoli_index_select_scratch_bytes(const DsaGeom* g, int B, int score_stride) {
    if (!g || B <= 0 || score_stride <= 0) return 0;
    size_t total = 0;
    carve(g, B, score_stride, nullptr, &total);
    return total;
}

// 1 if rivoli_index_select_paged takes the tensor-core path for this geometry, else 0.
RIVOLI_API int rivoli_index_select_uses_mma(const DsaGeom* g, int score_stride) {
    return (g && mma_geometry_ok(g, score_stride)) ? 1 : 0;
}

RIVOLI_API int rivoli_kv_append_paged(const DsaGeom* g, const uint16_t* latent, const uint16_t* index_key,
                                      const int32_t* row_seq, const int32_t* row_pos, int n_rows,
                                      const int32_t* block_table, uint8_t* latent_pool, float* latent_scale,
                                      uint8_t* index_pool, float* index_scale, int32_t* status, void* stream);

// Whether the score rows are no longer than top_k and one launch takes the place of prologue, scorer and selection.
extern "C" bool rivoli_index_select_takes_all(const DsaGeom* g, int score_stride) {
    return score_stride <= g->top_k && rv_append_chunks(*g) <= 3 * 32;
}

// `ap` != NULL: the step's append (one new token per sequence) rides in the same launch as the
// query preparation.
static int select_impl(const DsaGeom* g, const AppendArgs* ap, const uint16_t* index_q, const float* w,
                       const uint8_t* index_pool, const float* index_scale,
                       const int32_t* block_table, const int32_t* seq_len, int B,
                       int score_stride, uint32_t* rows, int32_t* n_sel, void* scratch,
                       void* stream) {
    if (int e = rv_check_geom(g)) return e;
    if (B <= 0 || score_stride <= 0 || !index_q || !w || !index_pool || !index_scale || !block_table || !seq_len ||
        !rows || !n_sel || !scratch)
        return 1001;
    if ((((uintptr_t)index_pool | (uintptr_t)index_q | (uintptr_t)scratch) & 15)) return 1005;
    if ((long long)score_stride > (long long)g->max_pages_per_seq * g->page_tokens) return 1002;
    cudaStream_t st = (cudaStream_t)stream;
    size_t total = 0;
    SelectScratch s = carve(g, B, score_stride, scratch, &total);
    const int nh = g->index_heads, hd = g->index_dim;
    const bool narrow = rv_append_chunks(*g) <= 3 * 32;   // what the append inside a prologue launch covers

    if (rivoli_index_select_takes_all(g, score_stride)) {
        rv_drain_error();
        rv_stage_event(0, st);
        // (the query codes stay part of the operator's scratch: the sharded step reads them after it)
        if (!ap)
            if (int e = rivoli_index_q_quant(index_q, B * nh, hd, s.qcodes, s.qscales, stream)) return e;
        const dim3 grid((unsigned)(B + 1 + (ap ? (B + SD_THREADS / 32 - 1) / (SD_THREADS / 32) : 0)));
        const AppendArgs aa = ap ? *ap : AppendArgs{};
        rv_launch_dependent(step_dense_kernel, grid, dim3(SD_THREADS), 0, st, *g, aa, B, block_table, seq_len, score_stride, rows, n_sel,
                            s.stats, s.err);
        rv_stage_event(1, st);
        rv_stage_event(2, st);
        return rv_launch_status();
    }

    if (!mma_geometry_ok(g, score_stride)) {
        // geometries outside the tensor-core kernel: the exact CUDA-core scorer + exact top-k
        int e = 0;
        if (ap && narrow) {
            if ((hd % 16) != 0 || hd > 512) return 1004;
            rv_drain_error();
            rv_launch_dependent(step_quant_kernel, dim3((unsigned)((B * nh + B + 7) / 8)), dim3(256), 0, st, *g, *ap, B, index_q, s.qcodes, s.qscales);
            e = rv_launch_status();
        } else {
            if (ap)
                e = rivoli_kv_append_paged(g, ap->latent, ap->index_key, nullptr, ap->row_pos, B, ap->block_table,
                                           ap->latent_pool, ap->latent_scale, ap->index_pool, ap->index_scale,
                                           ap->status, stream);
            if (!e) e = rivoli_index_q_quant(index_q, B * nh, hd, s.qcodes, s.qscales, stream);
        }
        if (e) return e;
        e = rivoli_index_score_paged(g, s.qcodes, s.qscales, w, index_pool, index_scale, block_table, seq_len, B,
                                     s.scores, score_stride, stream);
        if (e) return e;
        return rivoli_index_topk_batched(s.scores, score_stride, seq_len, B, g->top_k, rows, n_sel, stream);
    }

    rv_drain_error();
    rv_stage_event(0, st);
    if (ap) {
        int per_block = PROLOGUE_ROWS_FEW;
        while (per_block < PROLOGUE_ROWS_MOST && B + (B + per_block - 1) / per_block > rv_sm_count()) per_block *= 2;
        rv_launch_dependent(step_prologue_kernel, dim3((unsigned)(B + (B + per_block - 1) / per_block)), dim3(1024), 0, st, *g, *ap, B, per_block, index_q, w, s.qcodes,
                            s.qscales, s.cb, s.err);
    } else
        rv_launch_dependent(index_q_prepare_kernel, dim3((unsigned)B), dim3(32 * nh), 0, st, index_q, w, nh, hd, g->index_wscale,
                            g->index_dscale, s.qcodes, s.qscales, s.cb, s.err);
    if (int e = rv_launch_status()) return e;

    IndexMmaArgs ma{*g, s.qcodes, s.qscales, w, index_pool, index_scale, block_table, seq_len,
                    s.scores, score_stride, B, s.err};
    constexpr size_t smem1 = (size_t)IM_NS * IM_STAGE_BYTES + 2 * IM_Q_BYTES + 1024;
    rv_allow_smem<index_score_mma_kernel>((int)smem1);
    const int sms = rv_sm_count();
    // two persistent CTAs per SM; a batch with fewer tiles at most gets as many CTAs
    const long long most = (long long)B * ((score_stride + IM_TILE - 1) / IM_TILE);
    const int grid = most < 2 * sms ? (int)most : 2 * sms;
    CUtensorMap tm_keys, tm_q;
    if (int e = rivoli::make_tmap_rows_sw128(&tm_keys, index_pool, (uint64_t)g->n_pool_pages * g->page_tokens, IM_HD,
                                             (uint32_t)g->page_tokens))
        return e;
    if (int e = rivoli::make_tmap_rows_sw128(&tm_q, s.qcodes, (uint64_t)B * nh, IM_HD, (uint32_t)nh)) return e;
    rv_stage_event(1, st);
    rv_launch_dependent(index_score_mma_kernel, dim3(grid), dim3(IM_THREADS), smem1, st, ma, tm_keys, tm_q);
    if (int e = rv_launch_status()) return e;
    rv_stage_event(2, st);

    const SelArgs ra{*g, s.scores, score_stride, seq_len, s.qcodes, s.qscales, w, s.cb,
                     index_pool, index_scale, block_table, rows, n_sel, g->top_k, s.stats,
                     (((uintptr_t)index_scale & 15) == 0 && g->page_tokens % 4 == 0) ? 1 : 0, score_stride % 4 == 0 ? 1 : 0, s.err};
    return rivoli::launch_index_select_cluster(ra, B, st);
}

RIVOLI_API int rivoli_index_select_paged(const DsaGeom* g, const uint16_t* index_q, const float* w,
                                         const uint8_t* index_pool, const float* index_scale,
                                         const int32_t* block_table, const int32_t* seq_len, int B,
                                         int score_stride, uint32_t* rows, int32_t* n_sel, void* scratch,
                                         void* stream) {
    return select_impl(g, nullptr, index_q, w, index_pool, index_scale, block_table, seq_len, B, score_stride, rows,
                       n_sel, scratch, stream);
}

// Decode step, first half: append the step's token of every sequence (row b belongs to sequence
// b, position row_pos[b]) AND select the attended rows, with the append riding in the launch
// that prepares the indexer query. Same results as rivoli_kv_append_paged followed by
// rivoli_index_select_paged.
RIVOLI_API int rivoli_dsa_append_select_paged(const DsaGeom* g, const uint16_t* latent, const uint16_t* index_key,
                                              const int32_t* row_pos, const int32_t* block_table,
                                              uint8_t* latent_pool, float* latent_scale, uint8_t* index_pool,
                                              float* index_scale, int32_t* status, const uint16_t* index_q,
                                              const float* w, const int32_t* seq_len, int B, int score_stride,
                                              uint32_t* rows, int32_t* n_sel, void* scratch, void* stream) {
    if (int e = rv_check_geom(g)) return e;
    if (B <= 0 || !latent || !index_key || !row_pos || !block_table || !latent_pool || !latent_scale || !index_pool ||
        !index_scale)
        return 1001;
    if ((g->rope_dim % 4) != 0 || ((g->kv_lora + g->rope_dim) % 16) != 0) return 1004;
    if ((((uintptr_t)latent | (uintptr_t)index_key | (uintptr_t)latent_pool | (uintptr_t)index_pool) & 15) ||
        ((uintptr_t)latent_scale & 3))
        return 1005;
    const AppendArgs ap{latent, index_key, row_pos, block_table, latent_pool, latent_scale, index_pool, index_scale, status};
    return select_impl(g, &ap, index_q, w, index_pool, index_scale, block_table, seq_len, B, score_stride, rows, n_sel,
                       scratch, stream);
}

// Where the last rivoli_index_select_paged call on `scratch` left the query codes and their scales (both paths
// of that call fill them): read by the page-range shard step, which re-scores its candidates exactly.
extern "C" void rivoli_index_select_query_codes(const DsaGeom* g, int B, int score_stride, void* scratch,
                                                const uint8_t** qcodes, const float** qscales) {
    size_t total = 0;
    SelectScratch s = carve(g, B, score_stride, scratch, &total);
    *qcodes = s.qcodes;
    *qscales = s.qscales;
}

// Reads back the tensor-core scorer's error word and clears it: 1005 = a block-table entry inside a
// sequence's length pointed outside the pool (rows undefined), 1008 = a bounded wait gave up.
// Synchronises the stream.
RIVOLI_API int rivoli_index_select_status(const DsaGeom* g, int B, int score_stride, void* scratch, void* stream) {
    if (!g || !scratch) return 1001;
    size_t total = 0;
    SelectScratch s = carve(g, B, score_stride, scratch, &total);
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, s.err, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return -(int)e;
    if (h) cudaMemsetAsync(s.err, 0, sizeof(int), (cudaStream_t)stream);
    return h == IM_ERR_BAD_PAGE ? 1005 : (h ? 1008 : 0);
}

// Diagnostics: copies the per-sequence band sizes of the last call (tokens re-scored
// exactly) to host memory. Synchronises the stream.
RIVOLI_API int rivoli_index_select_band_stats(const DsaGeom* g, int B, int score_stride, void* scratch,
                                              uint32_t* host_band, void* stream) {
    if (!g || !scratch || !host_band || B <= 0) return 1001;
    size_t total = 0;
    SelectScratch s = carve(g, B, score_stride, scratch, &total);
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaMemcpy2D(host_band, 4, s.stats, 8, 4, (size_t)B, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? 0 : -(int)e;
}

