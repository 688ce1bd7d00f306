// V4 cousin of the decode path, part 2: MQA sparse attention over one shared entry per position, gathered by an
// explicit index list, with a per-head sink in the softmax denominator.
// Reference behaviour: crates/backend/kernels/attn.hip:358-465.
#include <atomic>

#include "o_merge.cuh"
#include "tc_common.cuh"
#include "v4_common.cuh"

namespace {

// ---------------------------------------------------------------------------------------------------
// sparse attention, CUDA cores: any shape, f32 or bf16 storage. One CTA per (query row, head).
// ---------------------------------------------------------------------------------------------------
constexpr int GA_THREADS = 256;
constexpr int GA_ACC = 4;

__device__ __forceinline__ void v4_store_out(float* o, size_t i, float v) { o[i] = v4_rbf16(v); }
__device__ __forceinline__ void v4_store_out(uint16_t* o, size_t i, float v) { o[i] = rv_f32_to_bf16(v); }

template <class T>
__global__ void __launch_bounds__(GA_THREADS) v4_gather_attn_kernel(const T* __restrict__ q, const T* __restrict__ kv,
                                                                    size_t kv_row_stride_per_t,
                                                                    const float* __restrict__ sink,
                                                                    const int* __restrict__ idxs, int h, int d,
                                                                    int topk, float scale, T* __restrict__ o) {
    extern __shared__ __align__(16) float ga_smem[];
    float* qs = ga_smem;      // [d]
    float* lg = ga_smem + d;  // [topk] logits, then softmax weights
    __shared__ float red[GA_THREADS / 32];
    __shared__ float bc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int head = blockIdx.x, t = blockIdx.y;
    const T* kvt = kv + (size_t)t * kv_row_stride_per_t;
    const int* ix = idxs + (size_t)t * topk;
    for (int i = tid; i < d; i += GA_THREADS) qs[i] = v4_load_f32(q, ((size_t)t * h + head) * d + i);
    __syncthreads();
    // logits: one warp per slot, lanes across the row
    float mx = -INFINITY;
    for (int j = warp; j < topk; j += GA_THREADS / 32) {
        const int p = ix[j];
        float l = -INFINITY;
        if (p >= 0) {
            float a = 0.0f;
            for (int i = lane; i < d; i += 32) a = fmaf(qs[i], v4_load_f32(kvt, (size_t)p * d + i), a);
            l = rv_warp_sum(a) * scale;
        }
        if (lane == 0) lg[j] = l;
        mx = fmaxf(mx, l);
    }
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int i = 1; i < GA_THREADS / 32; ++i) mx = fmaxf(mx, red[i]);
    __syncthreads();
    float ps = 0.0f;
    for (int j = tid; j < topk; j += GA_THREADS) {
        const float e = ix[j] >= 0 ? expf(lg[j] - mx) : 0.0f;
        lg[j] = e;
        ps += e;
    }
    ps = rv_warp_sum(ps);
    if (lane == 0) red[warp] = ps;
    __syncthreads();
    if (tid == 0) {
        float s = 0.0f;
        for (int i = 0; i < GA_THREADS / 32; ++i) s += red[i];
        // a query with every slot masked is made loud, not zero
        bc = isfinite(mx) ? s + expf(sink[head] - mx) : NAN;
    }
    __syncthreads();
    const float denom = bc;
    float acc[GA_ACC];
#pragma unroll
    for (int c = 0; c < GA_ACC; ++c) acc[c] = 0.0f;
    for (int j = 0; j < topk; ++j) {
        const int p = ix[j];
        if (p < 0) continue;
        const float e = lg[j];
#pragma unroll
        for (int c = 0; c < GA_ACC; ++c) {
            const int i = tid + c * GA_THREADS;
            if (i < d) acc[c] = fmaf(e, v4_load_f32(kvt, (size_t)p * d + i), acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < GA_ACC; ++c) {
        const int i = tid + c * GA_THREADS;
        if (i < d) v4_store_out(o, ((size_t)t * h + head) * d + i, acc[c] / denom);
    }
}

// ---------------------------------------------------------------------------------------------------
// sparse attention, 5th-generation tensor cores: 64 heads x 512 dims, bf16 rows as they lie in the cache.
//
// A tile is 64 gathered rows (64 KiB: eight 64-dim chunks of [64 rows][128 B], 128-byte swizzle), two tiles in flight; it
// serves every head twice, as K and as V:
//   S^T[64 rows x 64 heads]   = K_tile . Q^T            32 MMAs (M = 64, N = 64, K = 16), tile K-major, Q from shared memory
//   O^T[512 dims x 64 heads] += K_tile^T . P             4 x 4 MMAs (M = 128, N = 64), the same tile read MN-major
// Rows of S^T are tokens, so a thread of the softmax holds one token's scores: P leaves as 16-byte pieces of a token's 64
// heads (MN-major B operand), a head's sum stays in the token's registers until the end, and only the reference maximum
// needs an exchange: it LAGS (one barrier-with-OR per tile) until a score exceeds it by more than SA_LAG (log2), then the
// exact maxima are taken and O^T is rescaled in tensor memory. Weights are bf16, the sum is the sum of the rounded weights.
// TMEM (512 columns): O^T 4 x 64, S^T 2 x 64 (M = 64: row i in lane 32 (i / 16) + i % 16).
// 12 warps: 0-7 softmax + epilogue (lane quarter = warp % 4, head half = warp / 4), 8 QK issue, 9 PV issue, 10 and 11 gather
// (32 rows of every tile each, cp.async; masked slots are zero rows).
// One CTA per sequence; a batch that leaves SMs idle gets a thread-block cluster per sequence (tiles split evenly, at most
// eight CTAs), or several that share its heads, merged as o_merge.cuh says: O^T rows are pushed as they are to the CTA that
// writes the head, which weighs them.
// Bound by the rows an SM can take in (18 bytes a clock): 640 rows x 128 sequences 57 us with mma.sync (operand reloads from
// shared memory), 29.7 us now; 3 sequences 55 us on three SMs, 12.9 us now.
// All waits are bounded (tc_common.cuh); one that gives up makes the sequence's output NaN and sets g_sa_err.
// ---------------------------------------------------------------------------------------------------
constexpr int SA_H = 64, SA_D = 512, SA_TILE = 64;
constexpr int SA_SW = 8, SA_QKW = 8, SA_PVW = 9, SA_GW0 = 10, SA_GW = 2;
constexpr int SA_THREADS = (SA_GW0 + SA_GW) * 32, SA_ST = SA_SW * 32;      // threads, softmax threads
constexpr int SA_MAX_SPLITS = om::MAX_N;
constexpr float SA_LAG = 3.0f;
constexpr int SA_KSTAGE = SA_TILE * SA_D * 2, SA_CHUNK = SA_TILE * 128;
constexpr int SA_SQ = 2 * SA_KSTAGE;                       // q: [8 chunks][64 heads][128 B]
constexpr int SA_SP = SA_SQ + SA_H * SA_D * 2;             // P: 2 x [64 tokens][64 heads] bf16
constexpr int SA_PBUF = SA_TILE * SA_H * 2;
constexpr int SA_WMAX = SA_SP + 2 * SA_PBUF;               // f32 [4][64] exchange between the lane quarters
constexpr int SA_REF = SA_WMAX + 4 * SA_H * 4;             // f32 [64] reference maxima
constexpr int SA_FAC = SA_REF + SA_H * 4;                  // f32 [64] rescale of O^T; 1 / denominator in the epilogue
constexpr int SA_ML = SA_FAC + SA_H * 4;                   // float2 [n][hpc] (reference, sum) of this CTA's heads, from the cluster
constexpr int SA_BARS = SA_ML + (SA_H + SA_MAX_SPLITS) * 8;
constexpr int SA_MISC = SA_BARS + 128;
constexpr int SA_TOTAL = SA_MISC + 16;
constexpr int SA_TMO = 0, SA_TMS = 256;                    // tensor memory columns
static_assert(SA_TOTAL <= 232448, "shared memory budget");
static_assert(om::H == SA_H && om::D == SA_D && om::recv_floats(SA_MAX_SPLITS) * 4 <= SA_SP, "the merge buffers fit the tiles and q");
__device__ int g_sa_err;

struct SaBars { uint64_t k_full[2], k_empty[2], s_full[2], s_empty[2], p_full[2], q_full; };
static_assert(sizeof(SaBars) <= 128, "barrier block");

struct SaArgs {
    const uint16_t* q; const uint16_t* kv; size_t kv_rows; const float* sink; const int32_t* sel;
    int cols, n_splits, q_early;      // q_early: q was complete before the preceding kernel was launched
    float scale_log2; uint16_t* out;
};

__device__ __forceinline__ float v4_ex2(float x) {   // 2^x, -inf -> 0; relative error 2^-22
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// bf16 x bf16 -> f32
__device__ __forceinline__ uint32_t sa_idesc(int M, int N, uint32_t a_mn, uint32_t b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn << 15) | (b_mn << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void sa_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// Sixteen values per lane -> lane i of each half-warp holds the half-warp's maximum (or sum) of value i.
template <bool SUM>
__device__ __forceinline__ float sa_fold16(const float (&v)[16], int lane) {
    float m[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) m[i] = v[i];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < o) {
                const bool up = lane & o;
                const float keep = up ? m[i + o] : m[i], got = __shfl_xor_sync(0xffffffffu, up ? m[i] : m[i + o], o);
                m[i] = SUM ? keep + got : fmaxf(keep, got);
            }
    return m[0];
}

__global__ void __launch_bounds__(SA_THREADS, 1) v4_sparse_attend_kernel(SaArgs A) {
    extern __shared__ __align__(1024) unsigned char sa_smem[];
    SaBars& bars = *reinterpret_cast<SaBars*>(sa_smem + SA_BARS);
    float* s_wmax = reinterpret_cast<float*>(sa_smem + SA_WMAX);
    float* s_ref = reinterpret_cast<float*>(sa_smem + SA_REF);
    float* s_fac = reinterpret_cast<float*>(sa_smem + SA_FAC);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sa_smem + SA_MISC);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sa_smem + SA_MISC + 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x / A.n_splits, split = blockIdx.x - b * A.n_splits;
    const int32_t* ix = A.sel + (size_t)b * A.cols;
    const int tiles_all = (A.cols + SA_TILE - 1) / SA_TILE, tps = (tiles_all + A.n_splits - 1) / A.n_splits;
    const int t0 = split * tps, ntiles = max(0, min(tiles_all, t0 + tps) - t0);
    float2 my_ml = make_float2(-INFINITY, 0.0f);         // a split's reference maximum and weight sum of head tid

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(&bars.k_full[s], SA_GW * 32); tc::mbar_init(&bars.k_empty[s], 1);
            tc::mbar_init(&bars.s_full[s], 1); tc::mbar_init(&bars.s_empty[s], SA_SW);
            tc::mbar_init(&bars.p_full[s], SA_ST);
        }
        tc::mbar_init(&bars.q_full, SA_ST);
        tc::mbar_init_fence();
        *abort_flag = 0;
    }
    if (tid < SA_H) s_ref[tid] = -INFINITY;
    if (warp == SA_QKW) tc::tmem_alloc<512>(tmem_slot);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot, TM_O = tmem + SA_TMO, TM_S = tmem + SA_TMS;

    // Under a programmatic dependent launch the kernel before this one may still be running: nothing it may have written is
    // read before the dependency wait.
    rv_grid_dep_trigger();   // the next kernel may be scheduled as CTAs leave; it waits for this grid first
    if (!A.q_early) rv_grid_dep_wait();
    if (warp < SA_SW) {   // q of this sequence: 64 rows of 64 16-byte pieces, swizzled; the copies signal the barrier
#pragma unroll
        for (int it = 0; it < SA_H * SA_D / 8 / SA_ST; ++it) {
            const int e = it * SA_ST + tid, row = e >> 6, c = e & 63;
            tc::cp_async16(tc::smem_u32(sa_smem + SA_SQ + (c >> 3) * SA_CHUNK + tc::sw128_chunk(row, c & 7)),
                           A.q + ((size_t)b * SA_H + row) * SA_D + c * 8);
        }
        tc::cp_async_mbar_arrive_noinc(&bars.q_full);
    }
    rv_grid_dep_wait();

    if (warp >= SA_GW0) {
        // ---- gather: warp g fills the rows 32 g .. 32 g + 31 of every tile, half a row (512 bytes) per instruction
        const int g = warp - SA_GW0;
        const uint16_t* kvb = A.kv + (size_t)b * A.kv_rows * SA_D;
        auto slot = [&](int t) -> int {      // of row 32 g + lane
            const int j = (t0 + t) * SA_TILE + 32 * g + lane;
            return t < ntiles && j < A.cols ? ix[j] : -1;
        };
        int next = slot(0);
        bool ok = true;
        for (int t = 0; t < ntiles; ++t) {
            const int s = t & 1, mine = next;
            next = slot(t + 1);
            ok = tc::mbar_wait_warp(&bars.k_empty[s], ((t >> 1) & 1) ^ 1, abort_flag, 91);
            if (!ok) break;
            uint8_t* tile = sa_smem + s * SA_KSTAGE;
#pragma unroll 8
            for (int r = 0; r < 32; ++r) {
                const int p = __shfl_sync(0xffffffffu, mine, r), row = 32 * g + r;
                const uint16_t* src = kvb + (size_t)(p >= 0 ? p : 0) * SA_D + lane * 8;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = h * 32 + lane;
                    tc::cp_async16_zfill(tc::smem_u32(tile + (c >> 3) * SA_CHUNK + tc::sw128_chunk(row, c & 7)), src + h * 256, p >= 0 ? 16u : 0u);
                }
            }
            tc::cp_async_mbar_arrive_noinc(&bars.k_full[s]);
        }
        tc::cp_async_commit();
        tc::cp_async_wait<0>();              // (an aborted CTA leaves no copy in flight)
    } else if (warp == SA_QKW) {
        if (ntiles > 0) {
            const uint32_t id = sa_idesc(SA_TILE, SA_H, 0, 0);
            const uint64_t dq = tc::smem_desc_sw128(tc::smem_u32(sa_smem + SA_SQ), 16, 1024);
            bool ok = tc::mbar_wait_warp(&bars.q_full, 0, abort_flag, 92);
            for (int t = 0; t < ntiles && ok; ++t) {
                const int s = t & 1;
                ok = tc::mbar_wait_warp(&bars.k_full[s], (t >> 1) & 1, abort_flag, 93) &&
                     tc::mbar_wait_warp(&bars.s_empty[s], ((t >> 1) & 1) ^ 1, abort_flag, 94);
                if (!ok) break;
                tc::fence_proxy_async();     // the copies wrote through the generic proxy, the MMAs read through the async one
                tc::tc_fence_after();
                const uint64_t dk = tc::smem_desc_sw128(tc::smem_u32(sa_smem + s * SA_KSTAGE), 16, 1024);
                if (tc::elect_one()) {
#pragma unroll
                    for (int k = 0; k < SA_D / 16; ++k) {   // four steps of 32 bytes per chunk; address fields count 16-byte units
                        const uint64_t off = (uint64_t)(((k >> 2) * SA_CHUNK + (k & 3) * 32) >> 4);
                        sa_mma(TM_S + s * SA_H, dk + off, dq + off, id, k != 0);
                    }
                    tc::mma_commit(&bars.s_full[s]);
                }
                __syncwarp();
            }
        }
    } else if (warp == SA_PVW) {
        if (ntiles > 0) {
            const uint32_t id = sa_idesc(128, SA_H, 1, 1);
            bool ok = true;
            for (int t = 0; t < ntiles && ok; ++t) {
                const int s = t & 1;
                ok = tc::mbar_wait_warp(&bars.p_full[s], (t >> 1) & 1, abort_flag, 95);
                if (!ok) break;
                tc::fence_proxy_async();
                tc::tc_fence_after();
                const uint64_t dv = tc::smem_desc_sw128(tc::smem_u32(sa_smem + s * SA_KSTAGE), SA_CHUNK, 1024);
                const uint64_t dp = tc::smem_desc_sw128(tc::smem_u32(sa_smem + SA_SP + s * SA_PBUF), 16, 1024);
                if (tc::elect_one()) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < SA_TILE / 16; ++k)   // sixteen tokens = two groups of eight rows
                            sa_mma(TM_O + c * SA_H, dv + (uint64_t)((2 * c * SA_CHUNK + k * 2048) >> 4), dp + (uint64_t)((k * 2048) >> 4), id, (t | k) != 0);
                    tc::mma_commit(&bars.k_empty[s]);
                }
                __syncwarp();
            }
        }
    } else {
        // ---- softmax. After the exchange below lane l of warp (sq, th) holds token 16 sq + l % 16 of the tile and the
        // sixteen heads hb .. hb + 15 (the scores of the upper sixteen columns come from the lane sixteen below).
        const int sq = warp & 3, th = warp >> 2, tok = 16 * sq + (lane & 15), hb = 32 * th + 16 * (lane >> 4);
        const uint32_t lane_base = ((uint32_t)(sq * 32)) << 16;
        const bool up = lane >= 16;
        float l_acc[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) l_acc[j] = 0.0f;
        auto live_slot = [&](int t) { const int j = (t0 + t) * SA_TILE + tok; return t < ntiles && j < A.cols && ix[j] >= 0; };
        bool next_live = live_slot(0), ok = ntiles > 0;
        // A warp whose wait gave up brings the others to the slow path of the tile that they are in or come to next, where all
        // agree to leave.
        auto give_up = [&]() { (void)tc::barrier_any(1, SA_ST, true); (void)tc::barrier_any(2, SA_ST, true); };
        for (int t = 0; t < ntiles; ++t) {
            const int s = t & 1;
            const bool live = next_live;
            next_live = live_slot(t + 1);
            ok = tc::mbar_wait_warp(&bars.s_full[s], (t >> 1) & 1, abort_flag, 96);
            if (!ok) { give_up(); break; }
            tc::tc_fence_after();
            float s2[16], dmax = -INFINITY;
            {
                uint32_t r[32];
                tc::tmem_ld32(TM_S + s * SA_H + lane_base + 32 * th, r);
                tc::tmem_ld_wait();
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&bars.s_empty[s]);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const uint32_t other = __shfl_sync(0xffffffffu, r[16 + j], lane & 15);
                    s2[j] = live ? __uint_as_float(up ? other : r[j]) * A.scale_log2 : -INFINITY;
                }
            }
            float ref[16];
#pragma unroll
            for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(ref + j) = *reinterpret_cast<const float4*>(s_ref + hb + j);
#pragma unroll
            for (int j = 0; j < 16; ++j) dmax = fmaxf(dmax, s2[j] - ref[j]);   // (a masked slot before any reference: NaN, ignored)
            if (tc::barrier_any(1, SA_ST, dmax > SA_LAG)) {
                s_wmax[sq * SA_H + 32 * th + lane] = sa_fold16<false>(s2, lane);
                if (tc::barrier_any(2, SA_ST, false)) { ok = false; break; }
                if (tid < SA_H) {
                    const float old = s_ref[tid];
                    const float m = fmaxf(fmaxf(fmaxf(s_wmax[tid], s_wmax[SA_H + tid]), fmaxf(s_wmax[2 * SA_H + tid], s_wmax[3 * SA_H + tid])), old);
                    s_ref[tid] = m;
                    s_fac[tid] = m == -INFINITY ? 1.0f : v4_ex2(old - m);
                }
                tc::named_barrier(2, SA_ST);
                if (t > 0) {   // O^T to the new references, once the values of the tile before have landed
                    ok = tc::mbar_wait_warp(&bars.k_empty[(t - 1) & 1], ((t - 1) >> 1) & 1, abort_flag, 97);
                    if (!ok) { if (t + 1 < ntiles) give_up(); break; }
                    tc::tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t r[32];
                        tc::tmem_ld32(TM_O + c * SA_H + lane_base + 32 * th, r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int h = 0; h < 32; ++h) r[h] = __float_as_uint(__uint_as_float(r[h]) * s_fac[32 * th + h]);
                        tc::tmem_st32(TM_O + c * SA_H + lane_base + 32 * th, r);
                    }
                    tc::tmem_st_wait();
                    tc::tc_fence_before();
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) { ref[j] = s_ref[hb + j]; l_acc[j] *= s_fac[hb + j]; }
            }
            uint32_t pk[8];
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                // (no reference yet: every score so far is -inf and weighs 0)
                const float p0 = v4_ex2(s2[j] - (ref[j] == -INFINITY ? 0.0f : ref[j])), p1 = v4_ex2(s2[j + 1] - (ref[j + 1] == -INFINITY ? 0.0f : ref[j + 1]));
                asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(pk[j >> 1]) : "f"(p1), "f"(p0));
                l_acc[j] += __uint_as_float(pk[j >> 1] << 16);      // the sum of what the value product sees
                l_acc[j + 1] += __uint_as_float(pk[j >> 1] & 0xffff0000u);
            }
            uint8_t* pb = sa_smem + SA_SP + s * SA_PBUF;            // (the values of tile t - 2 are done: its stage was refilled)
            *reinterpret_cast<uint4*>(pb + tc::sw128_chunk(tok, hb / 8)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            *reinterpret_cast<uint4*>(pb + tc::sw128_chunk(tok, hb / 8 + 1)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
            tc::fence_proxy_async();
            tc::mbar_arrive(&bars.p_full[s]);
        }
        tc::named_barrier(1, SA_ST);
        s_wmax[sq * SA_H + 32 * th + lane] = sa_fold16<true>(l_acc, lane);
        tc::named_barrier(1, SA_ST);
        if (tid < SA_H) {
            const float l = (s_wmax[tid] + s_wmax[SA_H + tid]) + (s_wmax[2 * SA_H + tid] + s_wmax[3 * SA_H + tid]), m = s_ref[tid];
            my_ml = make_float2(m, l);
            // the sink joins the denominator only, shifted by the same maximum; a query with every slot masked is loud
            s_fac[tid] = m == -INFINITY ? NAN : 1.0f / (l + v4_ex2(A.sink[tid] * 1.4426950408889634f - m));
        }
        if (ok) ok = tc::mbar_wait_warp(&bars.k_empty[(ntiles - 1) & 1], ((ntiles - 1) >> 1) & 1, abort_flag, 98);
        tc::tc_fence_after();
        tc::named_barrier(1, SA_ST);
        // O^T: lane = dim of each 128-dim block. The output is staged in the idle tiles, eight heads at a time, and leaves as
        // 8 KiB bulk copies. (A split sequence is merged in its cluster below.)
        if (A.n_splits == 1) {
            uint16_t* stage = reinterpret_cast<uint16_t*>(sa_smem);
            const bool have = *abort_flag == 0;
#pragma unroll 1
            for (int g = 0; g < 4; ++g) {
                const int hg = 32 * th + g * 8;
                uint32_t r[4][8];
#pragma unroll
                for (int c = 0; c < 4; ++c) tc::tmem_ld8(TM_O + lane_base + c * SA_H + hg, r[c]);
                tc::tmem_ld_wait();
                uint16_t* sp = stage + hg * SA_D + sq * 32 + lane;
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        const float x = have ? __uint_as_float(r[c][i]) * s_fac[hg + i] : NAN, y = have ? __uint_as_float(r[c][i + 1]) * s_fac[hg + i + 1] : NAN;
                        uint32_t w2;
                        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w2) : "f"(y), "f"(x));
                        sp[i * SA_D + c * 128] = (uint16_t)w2;
                        sp[(i + 1) * SA_D + c * 128] = (uint16_t)(w2 >> 16);
                    }
                tc::fence_proxy_async();
                tc::named_barrier(4 + th, SA_ST / 2);
                if (sq == 0 && lane == 0) {
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                 ::"l"(A.out + ((size_t)b * SA_H + hg) * SA_D), "r"(tc::smem_u32(stage + hg * SA_D)), "r"(8 * SA_D * 2) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            if (sq == 0 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    }

    if (A.n_splits > 1) {
        // ---- merge inside the cluster (o_merge.cuh). Every thread of every CTA takes part in both cluster barriers; a CTA that
        // gave up sends sums that make the output NaN.
        const om::Share S(A.n_splits, split, (int)gridDim.y, (int)blockIdx.y);
        float* recv = reinterpret_cast<float*>(sa_smem);                      // [n][hpc][512]
        float2* ml = reinterpret_cast<float2*>(sa_smem + SA_ML);              // [n][hpc]: (maximum, sum) of rank q
        float* wts = reinterpret_cast<float*>(sa_smem + SA_SP);               // [hpc][8]: what rank q's row counts
        om::cluster_arrive();
        om::cluster_wait();                                                   // [1] every CTA's MMAs have read their tiles and q
        if (warp < SA_SW) {
            if (tid < SA_H) om::push_stats(S, ml, tid, *abort_flag ? make_float2(0.0f, NAN) : my_ml);
            om::push_rows(S, TM_O, recv, ntiles > 0, warp, lane);
        }
        om::cluster_arrive();
        om::cluster_wait();                                                   // [2] every CTA's share of this CTA's heads
        static_assert(om::MAX_N == 8 && SA_H / 2 * 8 <= SA_THREADS, "eight lanes a head, at most half of the heads");
        const int wh = tid >> 3, wq = tid & 7;
        const bool told = wh < S.heads && wq < S.n;
        const float2 part = told ? ml[wq * S.hpc + wh] : make_float2(-INFINITY, 0.0f);
        const float mg = om::fold8<false>(part.x), w = part.x > -INFINITY ? v4_ex2(part.x - mg) : 0.0f, L = om::fold8<true>(part.y * w);
        if (told) {
            const float sink = A.sink[S.hz0 + S.lo + wh] * 1.4426950408889634f;
            wts[wh * om::MAX_N + wq] = mg == -INFINITY ? NAN : w / (L + v4_ex2(sink - mg));
        }
        __syncthreads();
        om::write_rows(S, recv, wts, A.out + (size_t)b * SA_H * SA_D, tid, SA_THREADS);
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == SA_QKW) {
        tc::settle(*abort_flag);
        tc::tmem_dealloc<512>(tmem);
    }
    if (tid == 0 && *abort_flag) atomicCAS(&g_sa_err, 0, *abort_flag);
}

// CTAs per sequence: as many as leave all clusters resident at once (at most eight), and no more than there are tiles to
// share out evenly; then the clusters that share its heads.
struct SaPlan { int splits, shares; };
int sa_resident(int n_seqs, int n) {           // clusters of n CTAs that are resident at once
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n * n_seqs)); cfg.blockDim = dim3(SA_THREADS); cfg.dynamicSmemBytes = SA_TOTAL;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)n; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, v4_sparse_attend_kernel, &cfg) == cudaSuccess) return active;
    (void)cudaGetLastError();
    return 0;
}
SaPlan sa_plan(int n_seqs, int tiles) {
    constexpr int MOST = 128;
    static std::atomic<int> cache[MOST + 1];   // largest resident cluster size by batch; 0 = not asked yet
    static std::atomic<int> room[SA_MAX_SPLITS + 1];   // resident clusters by size, plus 1
    const int sms = rv_sm_count();
    if (n_seqs > MOST || 2 * n_seqs > sms) return {1, 1};
    int most = cache[n_seqs].load(std::memory_order_relaxed);
    if (!most) {
        for (most = sms / n_seqs < SA_MAX_SPLITS ? sms / n_seqs : SA_MAX_SPLITS; most > 1; --most)
            if (sa_resident(n_seqs, most) >= n_seqs) break;
        if (most < 1) most = 1;
        cache[n_seqs].store(most, std::memory_order_relaxed);
    }
    const int tps = (tiles + most - 1) / most, n = (tiles + tps - 1) / tps;
    if (n < 2) return {1, 1};
    int active = room[n].load(std::memory_order_relaxed) - 1;
    if (active < 0) {
        active = sa_resident(n_seqs, n);
        room[n].store(active + 1, std::memory_order_relaxed);
    }
    return {n, om::shares(n, n_seqs, active)};
}

}  // namespace


RIVOLI_API int rivoli_gather_attn_shared_kv(const float* q, const float* kv, const float* sink, const int* idxs, int m,
                                            int h, int d, int topk, float scale, float* o, void* stream) {
    if (m <= 0 || h <= 0 || d <= 0 || topk <= 0) return 1001;
    if (d > GA_THREADS * GA_ACC) return 1002;   // dims past the per-thread accumulators would never be written
    const size_t smem = ((size_t)d + (size_t)topk) * sizeof(float);
    if (smem + sizeof(float) * (GA_THREADS + 2) > 65536) return 1006;
    rv_drain_error();
    rv_allow_smem<v4_gather_attn_kernel<float>>(65536);
    v4_gather_attn_kernel<float><<<dim3((unsigned)h, (unsigned)m), GA_THREADS, smem, (cudaStream_t)stream>>>(
        q, kv, 0, sink, idxs, h, d, topk, scale, o);
    return rv_launch_status();
}

// q_early: q was complete before the kernel in front of this call was launched.
int rivoli_v4_sparse_attend_launch(const V4Geom* g, int n_seqs, const uint16_t* q, const uint16_t* kv_cache, const float* sink,
                                   const int32_t* sel, int cols, uint16_t* out, int force_simt, int q_early, cudaStream_t st) {
    if (int rc = v4_check_geom(g, n_seqs)) return rc;
    if (cols <= 0) return 1001;
    if (g->head_dim > GA_THREADS * GA_ACC) return 1002;
    const size_t kv_rows = (size_t)g->window + (size_t)g->max_comp;
    rv_drain_error();
    if (!force_simt && g->n_heads == SA_H && g->head_dim == SA_D) {
        rv_allow_smem<v4_sparse_attend_kernel>(SA_TOTAL);
        const SaPlan plan = sa_plan(n_seqs, (cols + SA_TILE - 1) / SA_TILE);
        const int n = plan.splits;
        const SaArgs a{q, kv_cache, kv_rows, sink, sel, cols, n, q_early, g->softmax_scale * 1.4426950408889634f, out};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)n_seqs * (unsigned)n, (unsigned)plan.shares); cfg.blockDim = dim3(SA_THREADS);
        cfg.dynamicSmemBytes = (size_t)SA_TOTAL; cfg.stream = st;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        at[1].id = cudaLaunchAttributeClusterDimension;
        at[1].val.clusterDim.x = (unsigned)n; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = n > 1 ? 2 : 1;
        (void)cudaLaunchKernelEx(&cfg, v4_sparse_attend_kernel, a);
        return rv_launch_status();
    }
    const size_t smem = ((size_t)g->head_dim + (size_t)cols) * sizeof(float);
    if (smem > 200 * 1024) return 1006;
    if (n_seqs > 65535) return 1002;
    rv_allow_smem<v4_gather_attn_kernel<uint16_t>>(200 * 1024);
    v4_gather_attn_kernel<uint16_t><<<dim3((unsigned)g->n_heads, (unsigned)n_seqs), GA_THREADS, smem, st>>>(
        q, kv_cache, kv_rows * (size_t)g->head_dim, sink, sel, g->n_heads, g->head_dim, cols, g->softmax_scale, out);
    return rv_launch_status();
}

RIVOLI_API int rivoli_v4_sparse_attend_bf16(const V4Geom* g, int n_seqs, const uint16_t* q, const uint16_t* kv_cache,
                                            const float* sink, const int32_t* sel, int cols, uint16_t* out,
                                            int force_simt, void* stream) {
    return rivoli_v4_sparse_attend_launch(g, n_seqs, q, kv_cache, sink, sel, cols, out, force_simt, 0, (cudaStream_t)stream);
}

// Synchronises the stream; 1008 if a bounded wait of the sparse attention gave up since the last call.
RIVOLI_API int rivoli_v4_sparse_attend_status(void* stream) {
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return -(int)e;
    int h = 0;
    e = cudaMemcpyFromSymbol(&h, g_sa_err, sizeof(int));
    if (e != cudaSuccess) return -(int)e;
    if (h) { const int z = 0; cudaMemcpyToSymbol(g_sa_err, &z, sizeof(int)); }
    return h ? 1008 : 0;
}
