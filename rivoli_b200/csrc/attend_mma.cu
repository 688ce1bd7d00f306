// Absorbed MLA decode attention on the 5th-generation tensor cores, all operands fp8.
//
//     out_h = sum_t softmax_t((q_h . [L_t | R_t]) * scale) * L_t        (H = 64, 512 + 64 dims)
//
// The cache rows are e4m3 codes with one f32 scale per token, and tcgen05 kind::f8f6f4
// takes e4m3 operands directly, so the gathered rows are consumed AS THEY LIE in HBM: no
// dequantisation pass and half the shared memory of a 16-bit staging. The two operands that
// are not fp8 by nature are split into two e4m3 terms each (x ~ hi + lo, relative error
// ~2^-8, bf16-like):
//   * q (bf16 in)  -> q_hi and q_lo as 128 "virtual heads" along M, per-head scales;
//   * P (softmax)  -> p_hi, p_lo issued as two MMAs accumulating into the same columns.
// The per-token scale folds into the softmax: with s2 = log2(e) * scale * (q.k) and
// s2' = s2 + log2(s_tok), P' = 2^(s2' - m) = weight * s_tok, so P' x (raw V codes) is already
// the dequantised product and P' is bounded by 2^8 whatever the scales are.
//
// What bounds this kernel is how many gathered rows an SM keeps in flight, so the tile is SMALL and the ring is
// DEEP: 64 tokens per tile, SIX tiles (6 x 36 KiB) in flight. The room comes from keeping q out of shared memory: its
// 512 latent columns live in TENSOR MEMORY as the A operand of the QK MMAs (128 lanes = hi|lo heads, 128 columns of
// four e4m3 codes), which also spares the shared-memory pipe 64 KiB of operand reads per tile; only the 64 rope
// columns of q stay in shared memory. Tokens are the MMA N dimension, which may be 64 while every instruction keeps
// the full M = 128:
//   S[128 (hi|lo heads) x 64 tok] = Qcat . K_tile^T                         2 (rope, A in smem) + 16 (A in TMEM) MMAs, K = 32
//   O^T[512 dims x 64 heads]     += V^T (the SAME shared tile, read MN-major) . P'
//                                   4 blocks x 2 K-steps x {hi, lo} = 16 MMAs (N = 64)
// TMEM (512 columns): S double buffered (2 x 64) + q (128) + O^T (4 x 64).
//
// One CTA per (sequence, split), 14 warps: 0-7 softmax + epilogue, 8 QK issue, 9 PV issue, 10-13 gather (sixteen
// rows each of the first four tiles, then a tile per warp, in plain program order; no warp waits for its copies: the copies signal the
// stage's barrier themselves, so a warp goes straight on to its next tile as soon as that tile's stage is free; a lane
// locates two rows, copies go row by row with 32 lanes on 32 consecutive 16-byte chunks (cp.async into the swizzled
// tile); the row address chain (token -> page -> pool row -> scale) is software-pipelined in register queues).
// A softmax thread is one TMEM lane = one virtual head, and the q rows are ordered so that the hi and lo terms of a
// head sit 16 lanes apart in the SAME warp: lanes 0-15 of warp s hold the hi rows of heads 16 s .. 16 s + 15, lanes
// 16-31 their lo rows. One shuffle per score adds the two terms and leaves each lane with HALF the tokens of its
// head: thread = (head, 32 tokens of the tile). Two groups of four warps take the tiles in turn. A head's
// running sum and its q scale are registers, its reference maximum is handed from tile to tile through shared memory, and P'
// leaves as 16-byte stores (heads are the rows of the K-major P' operand, tokens its bytes).
// q arrives as bf16 (bulk copies) and is split into its two e4m3 terms by the softmax warps inside the kernel while the
// first tiles are gathered; the output leaves through the idle ring as 8 KiB bulk copies.
// Where only the step's new tokens can be changing under this kernel (a step that selects everything, a layer that shares a
// selection), it gathers beside the append in front of it and waits only where it comes to a new token's row: 32 sequences of
// 2,048 rows 28.3 -> 25.7 us a step, with the other changes noted below.
// Online softmax with a LAGGING reference max: as long as no score of a tile exceeds its head's
// reference by more than 3 (log2) the references stand (one barrier-with-OR per tile, no exchange);
// otherwise the exact per-head maxima are taken and O is rescaled through TMEM. P' carries 2^5, so
// it stays <= 256 < 448 and typical weights keep both e4m3 terms in the normal range.
// A batch too small to fill the chip is split: the CTAs of a sequence form one thread-block cluster (up to 8), each takes
// a contiguous range of tiles, and they merge their (maximum, sum, O) through distributed shared memory inside the kernel.
// All waits are bounded (tc_common.cuh).
#include "codec.cuh"
#include "common.cuh"
#include "o_merge.cuh"
#include "quant.cuh"
#include "tc_common.cuh"

namespace {

constexpr int AM_TILE = 64;
constexpr int AM_STAGES = 6;             // K ring depth
constexpr int AM_ROPES = 3;              // rope tiles: released right after the two rope MMAs of a tile, so fewer than stages
constexpr int AM_SBUF = 2;               // S accumulators
constexpr int AM_GW = 4;                 // gather warps
// A CTA of at most this many tiles has every tile filled by all gather warps. Eight against four, us a step: CTAs of five to eight tiles
// 26.2 -> 25.4 (32 x 2,048), 24.2 -> 23.8 (24 x 2,048), 23.5 -> 22.8 (128 x 500), 19.4 -> 18.6 (128 x 300); of one to four the same within 0.7 %.
constexpr int AM_JOINT = 8;
constexpr int AM_H = 64, AM_KVL = 512, AM_ROPE = 64, AM_W = AM_KVL + AM_ROPE;
constexpr int AM_SW = 8;                 // softmax + epilogue warps: TMEM lane quarter = warp % 4, token / head half = warp / 4
constexpr int AM_HPT = 32;               // head columns of O^T a thread owns in the rescale and the epilogue
constexpr int AM_SOFTMAX_THREADS = AM_SW * 32;
constexpr int AM_QKW = AM_SW, AM_PVW = AM_SW + 1, AM_GW0 = AM_SW + 2;   // warp roles: QK issue, PV issue, first gather warp
constexpr int AM_THREADS = (AM_GW0 + AM_GW) * 32;
constexpr int AM_MAX_SPLITS = om::MAX_N;     // CTAs per sequence = thread-block cluster size
// P'' = 2^(s2' - m_ref + AM_POFF) with m_ref lagging the true maximum by at most AM_LAG, so
// P'' <= 2^(AM_POFF + AM_LAG) = 256 < 448 while typical weights (a few binades below the maximum)
// land where BOTH e4m3 terms are normal numbers. In the code s2 carries the offset (s2 = s2' + AM_POFF)
// and the reference is kept WITHOUT it (m_ref = max s2'), so that the difference s2 - m_ref is the
// exponent of P'' directly.
constexpr float AM_POFF = 5.0f, AM_LAG = 3.0f;

// tensor memory map (columns)
constexpr int TMC_S = 0, TMC_Q = AM_SBUF * AM_TILE, TMC_O = TMC_Q + AM_KVL / 4;
static_assert(TMC_O + 4 * AM_H == 512, "tensor memory budget");

// shared memory map (bytes); every operand tile is 1024-byte aligned
constexpr int SM_K0 = 0;                 // 6 stages x (4 latent chunks x [64 rows][128 B]), 128-byte swizzle
constexpr int SM_KSTAGE = 32768, SM_KCHUNK = 8192;
constexpr int SM_ROPE = SM_K0 + AM_STAGES * SM_KSTAGE;       // 3 x [64 rows][64 B], 64-byte swizzle
constexpr int SM_ROPEBUF = 4096;
constexpr int SM_QR = SM_ROPE + AM_ROPES * SM_ROPEBUF;       // rope columns of q: [128 virtual heads][64 B], 64-byte swizzle
constexpr int SM_P = SM_QR + 8192;       // hi [64 heads][64 tokens], lo the same: K-major, 64-byte swizzle
constexpr int SM_PTERM = 4096;
constexpr int SM_TOK = SM_P + 2 * SM_PTERM;   // f32 [3][6 stages][64 tokens]: scale | log2(scale) + AM_POFF | 1 / scale
constexpr int SM_TOKPLANE = AM_STAGES * AM_TILE * 4;
constexpr int SM_AHI = SM_TOK + 3 * SM_TOKPLANE;   // f32 [64] per-head q scale * softmax scale * log2(e)
constexpr int SM_WMAX = SM_AHI + 256;    // f32 [2][64] exchange between the two token halves
constexpr int SM_FAC = SM_WMAX + 512;    // f32 [64] rescale factor of the current tile; 1 / l in the epilogue
constexpr int SM_BARS = SM_FAC + 256;    // mbarriers
constexpr int SM_MISC = SM_BARS + 320;
constexpr int SM_MREF = SM_MISC + 64;   // f32 [64] reference maximum per head, as the last tile decided it
constexpr int SM_TOTAL = SM_MREF + 256;
constexpr int SM_ZQ = SM_K0 + 3 * SM_KSTAGE;   // q as it arrives: ring stages 3 .. 5 before their first tile
constexpr int SM_ZROW = AM_W * 2 + 16;
static_assert(SM_ZQ + AM_H * SM_ZROW <= SM_K0 + AM_STAGES * SM_KSTAGE, "q fits the last stages");
constexpr int SM_STAGE = SM_K0;          // epilogue (the ring is idle by then): bf16 [64 heads][512 dims], or f32 [splits][heads][512 dims] received from the cluster
static_assert(om::H == AM_H && om::D == AM_KVL && om::recv_floats(AM_MAX_SPLITS) * 4 <= AM_STAGES * SM_KSTAGE, "the O staging fits the ring");

struct AmBars {
    uint64_t k_full[AM_STAGES], k_empty[AM_STAGES], s_full[AM_SBUF], s_empty[AM_SBUF], rope_free[AM_ROPES],
        p_full, pv_done[2], dec[2], q_full, q_raw[4];
};
static_assert(sizeof(AmBars) <= 320, "barrier block");
static_assert(SM_TOTAL <= 232448, "shared memory budget");
static_assert(SM_QR % 1024 == 0 && SM_P % 1024 == 0 && SM_ROPE % 1024 == 0, "operand tiles are 1024-byte aligned");


struct AttendMmaArgs {
    const uint16_t* q;       // [B][64][576] bf16: absorbed query, latent part then rope part
    float softmax_scale;
    const uint8_t* pool; const float* pscale; const int32_t* block_table;
    const uint32_t* rows; long long row_stride; const int32_t* n_rows;
    int page_tokens, max_pages, n_pool_pages, n_splits;
    uint16_t* out; float* out_m; float* out_lse;
    int* err;
    int min_rows;      // sequences with 0 < n_rows < min_rows are served by the CUDA-core kernel of the same call
    int q_early;       // 1: q was complete before the preceding kernel was launched, so it may be read before the grid-dependency wait
    int max_polls;     // poll limit of every bounded wait
    // The token of sequence b' at fresh_pos[b'], b' < n_fresh, is appended by the kernel before this one; all else that this one reads
    // was complete before that kernel started, so that its rows may be fetched beside it. NULL: no such promise.
    const int32_t* fresh_pos; int n_fresh;
    int row_cap;       // most rows of a sequence without a row list (beside its page table)
    int withhold;      // self-test: one gather warp never signals its part of the first tile (the waits on it must run out cleanly)
};

__device__ __forceinline__ uint32_t sw64_chunk(uint32_t row, uint32_t chunk) { return row * 64u + ((chunk ^ ((row >> 1) & 3u)) << 4); }

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)layout << 61;   // 2 = 128-byte swizzle, 4 = 64-byte swizzle
    return d;
}

// ---------------------------------------------------------------------------------------------
// main kernel
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(AM_THREADS, 1)
attend_mma_kernel(AttendMmaArgs A) {
    extern __shared__ __align__(1024) uint8_t smem[];
    AmBars& bars = *reinterpret_cast<AmBars*>(smem + SM_BARS);
    float* s_tok = reinterpret_cast<float*>(smem + SM_TOK);   // three planes of SM_TOKPLANE bytes
    float* s_ahi = reinterpret_cast<float*>(smem + SM_AHI);
    float* s_wmax = reinterpret_cast<float*>(smem + SM_WMAX);
    float* s_fac = reinterpret_cast<float*>(smem + SM_FAC);
    float* s_mref = reinterpret_cast<float*>(smem + SM_MREF);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + SM_MISC);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM_MISC + 4);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = blockIdx.x, b = blockIdx.y;
    const int P = A.page_tokens;

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < AM_STAGES; ++s) { tc::mbar_init(&bars.k_full[s], AM_GW * (32 + 1)); tc::mbar_init(&bars.k_empty[s], 1); }
#pragma unroll
        for (int s = 0; s < AM_SBUF; ++s) { tc::mbar_init(&bars.s_full[s], 2); tc::mbar_init(&bars.s_empty[s], AM_SW / 2); }
#pragma unroll
        for (int s = 0; s < AM_ROPES; ++s) tc::mbar_init(&bars.rope_free[s], 1);
        tc::mbar_init(&bars.p_full, AM_SOFTMAX_THREADS / 2);
#pragma unroll
        for (int s = 0; s < 2; ++s) { tc::mbar_init(&bars.pv_done[s], 1); tc::mbar_init(&bars.dec[s], AM_SW / 2); }
        tc::mbar_init(&bars.q_full, AM_SOFTMAX_THREADS);
#pragma unroll
        for (int s = 0; s < 4; ++s) tc::mbar_init(&bars.q_raw[s], 1);
        tc::mbar_init_fence();
        *abort_flag = 0;
    }
    if (tid < AM_H) s_mref[tid] = -INFINITY;
    if (warp == AM_QKW) tc::tmem_alloc<512>(tmem_base_s);

    tc::fence_proxy_async();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_base_s;
    const uint32_t TM_S0 = tmem + TMC_S, TM_Q = tmem + TMC_Q, TM_O = tmem + TMC_O;

    // q -> two e4m3 terms per head (once per CTA):
    //   hi = e4m3(q / s), s = absmax / 448;  lo = e4m3(q / s - hi)   =>  q ~ s * (hi + lo)
    // (the residual of a value of typical size is a normal e4m3 number; below 2^-6 it is kept to 2^-10 absolute,
    // 2^-19 of the head's largest value).
    // The sequence's 72 KiB of q arrive as one bulk copy per head in ring stages 3 to 5, which the gather leaves alone until q_full;
    // a head's row is 16 bytes longer there than its 1,152, so that the rows of eight heads lie in different banks.
    // Lane l of warp w converts the values of head 16 (w % 4) + l % 16 that the half w / 4 of the row has on its side l / 16: 128
    // latent and 16 rope values, both terms; one shuffle a word then gives each lane one term of both sides, which is a run of
    // the row of its OWN tensor-memory lane (virtual head): column c = codes 4c .. 4c + 3, lowest byte first, which is the
    // layout the MMA expects of an 8-bit A operand. The rope codes go to the shared operand tile.
    // (Converted a row per warp, staged in shared memory and read back by the rows' lanes it took 6,800 cycles behind the copy.)
    // The QK issuer waits for q_full before its first MMA.
    // Under a programmatic dependent launch the kernel before this one may still be running. Unless the
    // caller vouches that q was complete before that kernel was even launched (q_early: the fused decode
    // step), q may be that kernel's output and is read only after the dependency wait.
    rv_grid_dep_trigger();   // the next kernel may be scheduled as CTAs leave; it waits for this grid first
    if (!A.q_early) rv_grid_dep_wait();
    if (warp < AM_SW) {
        uint8_t* zq = smem + SM_ZQ;
        const int sq = warp & 3, half = warp >> 2, term = lane >> 4, h = 16 * sq + (lane & 15);
        if (half == 0) {
            if (lane == 0) tc::mbar_arrive_expect_tx(&bars.q_raw[sq], 16 * AM_W * 2);
            __syncwarp();
            if (lane < 16)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(tc::smem_u32(zq + h * SM_ZROW)), "l"(A.q + ((size_t)b * AM_H + h) * AM_W), "r"(AM_W * 2), "r"(tc::smem_u32(&bars.q_raw[sq])) : "memory");
            __syncwarp();
        }
        tc::mbar_wait_warp(&bars.q_raw[sq], 0, abort_flag, 55, A.max_polls);
        const uint4* src = reinterpret_cast<const uint4*>(zq + h * SM_ZROW + half * AM_KVL + term * (AM_KVL / 2));
        const uint4* rsrc = reinterpret_cast<const uint4*>(zq + h * SM_ZROW + AM_KVL * 2 + half * AM_ROPE + term * (AM_ROPE / 2));
        float inv;
        {
            uint32_t m = rv_max_bf16x2(rv_absmax8(rsrc[0]), rv_absmax8(rsrc[1]));
#pragma unroll 4
            for (int c = 0; c < 16; ++c) m = rv_max_bf16x2(m, rv_absmax8(src[c]));
            m = rv_max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, 16));
            if (term == 0) s_wmax[half * 64 + h] = __uint_as_float(m << 16);
            tc::named_barrier(3, AM_SOFTMAX_THREADS);
            const float amax = fmaxf(s_wmax[h], s_wmax[64 + h]);
            const float sc = amax > 0.0f ? amax / 448.0f : 1.0f;
            inv = 1.0f / sc;
            if (half == 0 && term == 0) s_ahi[h] = sc * A.softmax_scale * 1.4426950408889634f;
        }
        // 8 values -> their 8 hi codes and 8 lo codes
        auto codes8 = [&](const uint4 v, uint2& hi, uint2& lo) {
            const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
            uint16_t ch[4], cl[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float x0 = __uint_as_float(ww[i] << 16) * inv, x1 = __uint_as_float(ww[i] & 0xffff0000u) * inv;
                asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(ch[i]) : "f"(x1), "f"(x0));
                const float2 xh = rv_e4m3x2_to_f32x2(ch[i]);
                asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(cl[i]) : "f"(x1 - xh.y), "f"(x0 - xh.x));
            }
            hi = make_uint2((uint32_t)ch[0] | ((uint32_t)ch[1] << 16), (uint32_t)ch[2] | ((uint32_t)ch[3] << 16));
            lo = make_uint2((uint32_t)cl[0] | ((uint32_t)cl[1] << 16), (uint32_t)cl[2] | ((uint32_t)cl[3] << 16));
        };
        // a converted chunk -> this lane's term of the first and of the second side
        auto exchange = [&](const uint2 hi, const uint2 lo, uint32_t* first, uint32_t* second) {
            const uint2 keep = term ? lo : hi, give = term ? hi : lo;
            const uint2 got = make_uint2(__shfl_xor_sync(0xffffffffu, give.x, 16), __shfl_xor_sync(0xffffffffu, give.y, 16));
            first[0] = term ? got.x : keep.x; first[1] = term ? got.y : keep.y;
            second[0] = term ? keep.x : got.x; second[1] = term ? keep.y : got.y;
        };
        const uint32_t dst = TM_Q + (((uint32_t)(sq * 32)) << 16) + half * 64;
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {                  // (a loop: code that runs once is waited for)
            uint32_t r0[8], r1[8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint2 hi, lo;
                codes8(src[g * 4 + c], hi, lo);
                exchange(hi, lo, r0 + 2 * c, r1 + 2 * c);
            }
            tc::tmem_st8(dst + g * 8, r0);
            tc::tmem_st8(dst + 32 + g * 8, r1);
        }
        {
            uint32_t r0[4], r1[4];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint2 hi, lo;
                codes8(rsrc[c], hi, lo);
                exchange(hi, lo, r0 + 2 * c, r1 + 2 * c);
            }
            *reinterpret_cast<uint4*>(smem + SM_QR + sw64_chunk(sq * 32 + lane, 2 * half)) = make_uint4(r0[0], r0[1], r0[2], r0[3]);
            *reinterpret_cast<uint4*>(smem + SM_QR + sw64_chunk(sq * 32 + lane, 2 * half + 1)) = make_uint4(r1[0], r1[1], r1[2], r1[3]);
        }
        tc::tmem_st_wait();
        tc::fence_proxy_async();
        tc::tc_fence_before();
        tc::mbar_arrive(&bars.q_full);
        tc::named_barrier(3, AM_SOFTMAX_THREADS);   // the head scales are read by other warps than the ones that wrote them
    }

    // With q_early everything above read only inputs that predate the preceding kernel, so it overlapped
    // that kernel's tail; the selected rows and their counts are read below (of a call that appends and selects nothing
    // they predate it as well: the gather below waits where it comes to a row that may be new).
    const bool fresh = A.fresh_pos != nullptr;
    if (!fresh) rv_grid_dep_wait();
    int nr = A.n_rows[b];
    // a row list whose first entry is the dense marker stands for "row j = token j" over the first n_rows tokens
    const bool listed = A.rows && A.rows[(size_t)b * A.row_stride] != 0xffffffffu;
    {
        const long long cap = listed ? A.row_stride : min((long long)A.row_cap, (long long)A.max_pages * P);
        nr = (int)max(0LL, min((long long)nr, cap));
    }
    // Short contexts belong to the CUDA-core kernel launched by the same call: this CTA touches no output.
    const bool skip = nr > 0 && nr < A.min_rows;
    if (skip) nr = 0;
    const int ntiles_all = (nr + AM_TILE - 1) / AM_TILE;
    const bool clustered = A.n_splits > 1;   // the CTAs of a sequence form one thread-block cluster and merge through its shared memory
    const int tps = (ntiles_all + A.n_splits - 1) / A.n_splits;
    const int r_begin = split * tps * AM_TILE;
    const int r_end = min(nr, r_begin + tps * AM_TILE);
    const int ntiles = r_end > r_begin ? (r_end - r_begin + AM_TILE - 1) / AM_TILE : 0;
    float2 my_ml = make_float2(-INFINITY, 0.0f);   // a split's reference maximum and weight sum of a head (one thread per head)
    const bool publishes = warp < AM_SW / 2 && lane < 16;                 // that thread
    const int ph = 16 * (warp & 3) + (lane & 15);                         // and its head

    if (warp >= AM_GW0 && ntiles > 0) {
        // ------------------------------ gather producers ------------------------------------------
        // The first four tiles, or all of a CTA that has at most eight, are filled together, sixteen rows of each by every warp:
        // the first is there after a quarter of the time that a tile per warp would take. Then warp g fills the tiles g + 4,
        // g + 8, ... (ring stage = tile % 6), a tile per warp: sixteen rows of every tile throughout held the latent copies of all
        // warps back at the next tile's rope buffer (batch 128: 59.4 -> 63.5 us), and four tiles that land together leave the
        // MMAs waiting for 3,500 cycles where eight are all there is. All in plain program order, and never waiting for
        // a copy to land: a thread's copies signal the stage's barrier themselves when they are complete
        // (cp.async.mbarrier.arrive), so the warp goes straight on to its next tile as soon as that tile's stage is
        // free. A lane resolves the addresses of two rows of its warp's tile.
        const int g = warp - AM_GW0;
        bool ok = true;
        // The address chain of a row (selected token -> page -> pool row -> scale) is three dependent global loads, and
        // under load each of them comes back only after the tens of kilobytes of copies queued in front of it. It
        // therefore runs as a software pipeline AM_LOOK of the warp's tiles deep PER LEVEL that keeps the raw loaded
        // words in register queues and touches a word only AM_LOOK iterations after it was requested (the warp issues
        // in order: a use right behind its load would stall every copy after it). For row u of the lane:
        //   tk[u][k]               token of the warp's tile i + 2 AM_LOOK + k, being loaded
        //   tok[u][k], pg[u][k]    token of its tile i + AM_LOOK + k and its page-table entry, being loaded
        //   row[u][k], scl[u][k]   pool row of its tile i + k (NONE: write zeros) and its scale; k = 0 is the current tile
        constexpr uint32_t NONE = 0xffffffffu;
        constexpr int AM_LOOK = 2;
        const uint32_t* rowp = listed ? A.rows + (size_t)b * A.row_stride : nullptr;
        const int32_t* btp = A.block_table + (size_t)b * A.max_pages;
        const int pshift = 31 - __clz(P);                  // page sizes are powers of two (checked by the host entry)
        static_assert(AM_GW * 16 == AM_TILE, "sixteen rows per warp of the first four tiles");
        const int n_joint = ntiles <= AM_JOINT ? AM_JOINT / AM_GW : 1;      // the warp's steps that are shared tiles
        auto load_tok = [&](int n, int u) -> uint32_t {     // this lane's u-th row of the warp's step n
            const int ri = r_begin + n * AM_GW * AM_TILE +
                           (n < n_joint ? (2 * u + (lane >> 4)) * AM_TILE + 16 * g + (lane & 15) : g * AM_TILE + u * 32 + lane);
            if (ri >= r_end) return NONE;
            return rowp ? rowp[ri] : (uint32_t)ri;
        };
        auto load_pg = [&](uint32_t t) -> int32_t {
            if (t == NONE) return -1;
            const uint32_t lp = t >> pshift;
            return lp < (uint32_t)A.max_pages ? btp[lp] : -1;
        };
        auto pool_row = [&](uint32_t t, int32_t pg) -> uint32_t {
            return (t != NONE && pg >= 0 && pg < A.n_pool_pages) ? (uint32_t)pg * (uint32_t)P + (t & (uint32_t)(P - 1)) : NONE;
        };
        // (not through L1: a line that holds an older scale of a new token may have been read beside the append)
        auto load_scl = [&](uint32_t r) -> float { return r != NONE ? __ldcg(A.pscale + r) : 0.0f; };
        uint32_t tk[2][AM_LOOK], tok[2][AM_LOOK], row[2][AM_LOOK];
        int32_t pg[2][AM_LOOK];
        float scl[2][AM_LOOK];
        // prologue: all token loads at once, then the page entries, then the scales of the first tiles
        // Rows that the kernel before may still be writing are marked in a bitmap by a hash of the pool row (in the P' tile, which
        // is not in use before the first QK): a tile of the first four that holds a marked row waits for that kernel, and so
        // does everything behind them. A hash that two rows share only makes a tile wait.
        uint32_t* marks = reinterpret_cast<uint32_t*>(smem + SM_P);
        constexpr int MARK_BITS = 2 * SM_PTERM * 8, AM_GT = AM_GW * 32;
        auto mark_of = [](uint32_t r) { return (r * 2654435761u) >> 16; };
        static_assert(MARK_BITS == 1 << 16, "sixteen hash bits");
        const int gt = g * 32 + lane;
        int fp[2] = {-1, -1};
        if (fresh) {
#pragma unroll
            for (int v = 0; v < 2; ++v)
                if (gt + v * AM_GT < A.n_fresh) fp[v] = A.fresh_pos[gt + v * AM_GT];
#pragma unroll
            for (int v = 0; v < MARK_BITS / 128 / AM_GT; ++v) reinterpret_cast<uint4*>(marks)[gt + v * AM_GT] = make_uint4(0u, 0u, 0u, 0u);
        }
        uint32_t t0[2][AM_LOOK];
        int32_t p0[2][AM_LOOK];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int k = 0; k < AM_LOOK; ++k) {
                t0[u][k] = load_tok(k, u); tok[u][k] = load_tok(AM_LOOK + k, u);
                tk[u][k] = load_tok(2 * AM_LOOK + k, u);
            }
        uint32_t hits[2] = {0u, 0u};   // lanes whose row of the first four tiles is marked
        uint32_t fr[2] = {NONE, NONE};
        if (fresh) {
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const uint32_t lp = (uint32_t)fp[v] >> pshift;
                const int32_t fpg = fp[v] >= 0 && lp < (uint32_t)A.max_pages ? A.block_table[(size_t)(gt + v * AM_GT) * A.max_pages + lp] : -1;
                fr[v] = pool_row((uint32_t)fp[v], fpg);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int k = 0; k < AM_LOOK; ++k) { p0[u][k] = load_pg(t0[u][k]); pg[u][k] = load_pg(tok[u][k]); }
        if (fresh) {
            tc::named_barrier(2, AM_GT);
#pragma unroll
            for (int v = 0; v < 2; ++v)
                if (fr[v] != NONE) atomicOr(marks + (mark_of(fr[v]) >> 5), 1u << (mark_of(fr[v]) & 31));
            tc::named_barrier(2, AM_GT);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
            for (int k = 0; k < AM_LOOK; ++k) { row[u][k] = pool_row(t0[u][k], p0[u][k]); scl[u][k] = load_scl(row[u][k]); }
            if (fresh) hits[u] = __ballot_sync(0xffffffffu, row[u][0] != NONE && ((marks[mark_of(row[u][0]) >> 5] >> (mark_of(row[u][0]) & 31)) & 1u));
        }
        bool waited = !fresh;
        auto wait_fresh = [&]() {
            rv_grid_dep_wait();
            waited = true;
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int k = 0; k < AM_LOOK; ++k) scl[u][k] = load_scl(row[u][k]);
        };
        // Each lane owns the addresses of two rows, but the COPIES are issued row by row with the 32 lanes of
        // the warp on 32 consecutive 16-byte chunks (the pool row travels by shuffle): one warp
        // instruction then reads 512 contiguous bytes instead of 32 scattered 16-byte pieces. A row past the end
        // (or on an unmapped page) is written as exact zeros by the same instruction with a source size of 0:
        // 0 x (stale NaN code) would poison O.
        auto token_words = [&](int s, int slot, uint32_t r, float sc) {   // scale, log2 and reciprocal of a token of stage s
            const bool live = r != NONE && sc > 0.0f;
            float* tp = s_tok + s * AM_TILE + slot;
            tp[0] = live ? sc : 0.0f;
            tp[SM_TOKPLANE / 4] = live ? __log2f(sc) + AM_POFF : -INFINITY;
            tp[2 * (SM_TOKPLANE / 4)] = live ? __frcp_rn(sc) : 0.0f;
        };
        auto copy_latent = [&](uint8_t* kbuf, uint32_t r, int slot) {     // chunk = lane
            tc::cp_async16_zfill(tc::smem_u32(kbuf + (lane >> 3) * SM_KCHUNK + tc::sw128_chunk(slot, lane & 7)),
                                 A.pool + (r != NONE ? (size_t)r * AM_W + lane * 16 : 0), r != NONE ? 16u : 0u);
        };
        auto copy_rope = [&](uint8_t* rope, uint32_t r, int slot) {       // 8 rows per instruction, 4 chunks each
            tc::cp_async16_zfill(tc::smem_u32(rope + sw64_chunk(slot, lane & 3)),
                                 A.pool + (r != NONE ? (size_t)r * AM_W + 512 + (lane & 3) * 16 : 0), r != NONE ? 16u : 0u);
        };
        // advance the chain past the warp's step n: every value consumed here was requested AM_LOOK iterations ago
        auto advance = [&](int n) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t row_new = pool_row(tok[u][0], pg[u][0]);
                const uint32_t tok_new = tk[u][0];
#pragma unroll
                for (int k = 0; k + 1 < AM_LOOK; ++k) {
                    row[u][k] = row[u][k + 1]; scl[u][k] = scl[u][k + 1]; tok[u][k] = tok[u][k + 1]; pg[u][k] = pg[u][k + 1]; tk[u][k] = tk[u][k + 1];
                }
                row[u][AM_LOOK - 1] = row_new; scl[u][AM_LOOK - 1] = load_scl(row_new);
                tok[u][AM_LOOK - 1] = tok_new; pg[u][AM_LOOK - 1] = load_pg(tok_new);
                tk[u][AM_LOOK - 1] = load_tok(n + 3 * AM_LOOK, u);
            }
        };
        // A stage is full when every copy has landed (the lanes' arrivals by the copies themselves: 32 from each of the four
        // warps, or four times 32 from the one that fills it) and the token words are written (plain arrivals, four in all,
        // which also publish those stores).
        const int n_steps = ntiles <= n_joint * AM_GW ? n_joint : (ntiles - 1 - g + AM_GW) / AM_GW;
#pragma unroll 1
        for (int n = 0; n < n_steps && ok; ++n) {
            const bool joint = n < n_joint;
#pragma unroll 1
            for (int t = joint ? 0 : g; ; ++t) {
                const int j = n * AM_GW + t, s = j % AM_STAGES, rb = j % AM_ROPES;
                const bool last = t >= (joint ? AM_GW : g + 1) || j >= ntiles;
                const int l0 = (t & 1) * 16;                   // (joint) the lanes that hold this tile's rows
                if (!waited && (last || (((t < 2 ? hits[0] : hits[1]) >> l0) & 0xffffu))) wait_fresh();
                if (last) break;
                if (j >= AM_STAGES) ok = tc::mbar_wait_warp(&bars.k_empty[s], ((j / AM_STAGES) & 1) ^ 1, abort_flag, 41, A.max_polls);
                else if (j >= AM_ROPES) ok = tc::mbar_wait_warp(&bars.q_full, 0, abort_flag, 43, A.max_polls);   // stages 3 to 5 held q
                if (!ok) break;
                uint8_t* kbuf = smem + SM_K0 + s * SM_KSTAGE;
                if (joint) {
                    const uint32_t src = t < 2 ? row[0][0] : row[1][0];
#pragma unroll 8
                    for (int it = 0; it < 16; ++it) copy_latent(kbuf, __shfl_sync(0xffffffffu, src, l0 + it), 16 * g + it);
                } else {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
#pragma unroll 8
                        for (int it = 0; it < 32; ++it) copy_latent(kbuf, __shfl_sync(0xffffffffu, row[u][0], it), u * 32 + it);
                    }
                }
                // a rope tile is free as soon as the two rope MMAs of the tile that used it last are done
                ok = tc::mbar_wait_warp(&bars.rope_free[rb], ((j / AM_ROPES) & 1) ^ 1, abort_flag, 42, A.max_polls);
                if (!ok) break;
                uint8_t* rope = smem + SM_ROPE + rb * SM_ROPEBUF;
                const int own = joint ? 1 : AM_GW;             // arrivals: this warp's share of the stage's
                if (joint) {
#pragma unroll
                    for (int it = 0; it < 2; ++it) {
                        const int rl = it * 8 + (lane >> 2);
                        copy_rope(rope, __shfl_sync(0xffffffffu, t < 2 ? row[0][0] : row[1][0], l0 + rl), 16 * g + rl);
                    }
                    tc::cp_async_mbar_arrive_noinc(&bars.k_full[s]);
                    if ((lane >> 4) == (t & 1)) token_words(s, 16 * g + (lane & 15), t < 2 ? row[0][0] : row[1][0], t < 2 ? scl[0][0] : scl[1][0]);
                } else {
#pragma unroll
                    for (int it = 0; it < 8; ++it) {
                        const int rl = it * 8 + (lane >> 2);
                        copy_rope(rope, __shfl_sync(0xffffffffu, row[it >> 2][0], rl & 31), rl);
                    }
#pragma unroll
                    for (int it = 0; it < AM_GW; ++it) tc::cp_async_mbar_arrive_noinc(&bars.k_full[s]);
#pragma unroll
                    for (int u = 0; u < 2; ++u) token_words(s, u * 32 + lane, row[u][0], scl[u][0]);
                }
                __syncwarp();
                if (lane < own && !(A.withhold && j == 0 && g == 0)) tc::mbar_arrive(&bars.k_full[s]);
            }
            advance(n);
        }
    } else if (warp == AM_QKW) {
        // ------------------------------ QK issuer -------------------------------------------------
        // The two MMA streams, QK(0..n-1) and PV(0..n-1), are each in order and are issued by ONE thread each, from two
        // warps: a warp blocks on the barriers of its own next instruction group only, so neither stream's control
        // latency (barrier observed -> fence -> issue -> commit) sits in the other's way and the tensor pipe takes
        // whichever group arrives first. QK runs ahead of the softmax by the two S buffers.
        if (ntiles > 0) {
            const uint32_t id_qk = tc::idesc_e4m3(128, AM_TILE, 0, 0);
            const uint64_t d_qr = smem_desc(tc::smem_u32(smem + SM_QR), 16, 512, 4);
            bool ok = tc::mbar_wait_warp(&bars.q_full, 0, abort_flag, 51, A.max_polls);
            for (int i = 0; i < ntiles && ok; ++i) {   // S(i) = Qcat . K(i)^T
                const int s = i % AM_STAGES, use = i / AM_STAGES, rb = i % AM_ROPES, sb = i % AM_SBUF, suse = i / AM_SBUF;
                ok = tc::mbar_wait_warp(&bars.k_full[s], use & 1, abort_flag, 52, A.max_polls) &&
                     tc::mbar_wait_warp(&bars.s_empty[sb], (suse & 1) ^ 1, abort_flag, 53, A.max_polls);
                if (!ok) break;
                tc::fence_proxy_async();   // the copies wrote through the generic proxy, the MMAs read through the async one
                tc::tc_fence_after();
                const uint64_t d_k = smem_desc(tc::smem_u32(smem + SM_K0 + s * SM_KSTAGE), 16, 1024, 2);
                const uint64_t d_rope = smem_desc(tc::smem_u32(smem + SM_ROPE + rb * SM_ROPEBUF), 16, 512, 4);
                const uint32_t d = TM_S0 + sb * AM_TILE;
                if (tc::elect_one()) {
                    // rope columns first (A from shared memory): their tile is released as soon as these two are done
#pragma unroll
                    for (int k = 0; k < 2; ++k) tc::mma_f8(d, d_qr + (uint64_t)(k * 2), d_rope + (uint64_t)(k * 2), id_qk, k != 0);
                    tc::mma_commit(&bars.rope_free[rb]);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < 4; ++k)   // A from tensor memory: 32 codes = 8 columns per step; descriptor address fields count 16-byte units
                            tc::mma_f8_ta(d, TM_Q + (uint32_t)(c * 32 + k * 8), d_k + (uint64_t)((c * SM_KCHUNK + k * 32) >> 4), id_qk, 1);
                    tc::mma_commit(&bars.s_full[sb]);
                    tc::mbar_arrive(&bars.s_full[sb]);   // hands the token words on: this thread has seen k_full
                }
                __syncwarp();
            }
        }
    } else if (warp == AM_PVW) {
        // ------------------------------ PV issuer -------------------------------------------------
        if (ntiles > 0) {
            const uint32_t id_pv = tc::idesc_e4m3(128, AM_H, 1, 0);
            const uint64_t d_phi = smem_desc(tc::smem_u32(smem + SM_P), 16, 512, 4);
            const uint64_t d_plo = smem_desc(tc::smem_u32(smem + SM_P + SM_PTERM), 16, 512, 4);
            bool ok = true;
            for (int j = 0; j < ntiles && ok; ++j) {   // O^T += V(j)^T . P'(j)
                const int s = j % AM_STAGES;
                ok = tc::mbar_wait_warp(&bars.p_full, j & 1, abort_flag, 54, A.max_polls);
                if (!ok) break;
                tc::fence_proxy_async();
                tc::tc_fence_after();
                const uint64_t d_v = smem_desc(tc::smem_u32(smem + SM_K0 + s * SM_KSTAGE), SM_KCHUNK, 1024, 2);
                if (tc::elect_one()) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
#pragma unroll
                        for (int k = 0; k < 2; ++k)   // p_hi
                            tc::mma_f8(TM_O + c * 64, d_v + (uint64_t)((c * SM_KCHUNK + k * 4096) >> 4), d_phi + (uint64_t)(k * 2), id_pv, (j | k) != 0);
#pragma unroll
                        for (int k = 0; k < 2; ++k)   // p_lo, same accumulator
                            tc::mma_f8(TM_O + c * 64, d_v + (uint64_t)((c * SM_KCHUNK + k * 4096) >> 4), d_plo + (uint64_t)(k * 2), id_pv, 1);
                    }
                    tc::mma_commit(&bars.k_empty[s]);
                    tc::mma_commit(&bars.pv_done[j & 1]);
                }
                __syncwarp();
            }
        }
    } else if (warp < AM_SW) {
        // ------------------------------ softmax + epilogue ---------------------------------------
        // S: TMEM lane = virtual head; lane quarter sq = warp % 4 (heads 16 sq .. 16 sq + 15, hi terms in lanes 0-15 and lo terms in
        // lanes 16-31). The warps are two groups of four that take the tiles in turn, so that the round trips of one tile (to
        // tensor memory, to its barriers, through the shuffles) run beside those of the other: eight warps on one tile spent
        // 2,000 - 2,300 cycles in a row on it, whatever the order, and that was the loop's period (batch 128 x 2,048 rows:
        // 1.32 us a tile, 1.27 so in a step; alone and from cold caches 1.34).
        // (A lone tile shared by both groups, a half of its tokens each, was 0.3 - 4 % slower: 1 x 256 rows 10.8 -> 11.1 us a step.)
        // After the hi + lo exchange lane l keeps the tokens 32 hf + 16 (l / 16) .. + 15 of each half hf of the tile, of head
        // 16 sq + l % 16.
        // O^T: TMEM lane = latent dim 32 sq + lane of each 128-dim block; in the epilogue th = warp / 4 is the half of the heads.
        const int sq = warp & 3, th = warp >> 2, tb = lane >> 4;
        const int hd = 16 * sq + (lane & 15);
        const int row = sq * 32 + lane;
        const uint32_t lane_base = ((uint32_t)(sq * 32)) << 16;
        const int h0 = th * AM_HPT;
        constexpr int AM_GROUP_THREADS = AM_SOFTMAX_THREADS / 2;
        const float a_h = s_ahi[hd];
        float l_acc = 0.0f;                                // sum of this thread's weights of head hd, at the reference m_ref
        float m_ref = -INFINITY;                           // reference max of head hd
        bool ok = ntiles > 0;
        // A warp whose wait gave up brings the others of its group to the slow path of the tile that they are in or come to next,
        // where all agree to leave.
        auto give_up = [&]() { (void)tc::barrier_any(6 + th, AM_GROUP_THREADS, true); (void)tc::barrier_any(8 + th, AM_GROUP_THREADS, true); };
        for (int i = th; i < ntiles; i += 2) {
            const int s = i % AM_STAGES;
            ok = tc::mbar_wait_warp(&bars.s_full[th], (i >> 1) & 1, abort_flag, 62, A.max_polls);
            if (!ok) { give_up(); break; }
            tc::tc_fence_after();
            // this thread's 32 tokens: 16-byte loads per plane (the two half-warps read 64 bytes apart: no bank conflict)
            const float4* ti = reinterpret_cast<const float4*>(s_tok + s * AM_TILE + 16 * tb);
            float s2[32];
            float mx = -INFINITY;                 // max over this thread's tokens of s2
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint32_t r[32];
                tc::tmem_ld32(TM_S0 + th * AM_TILE + lane_base + 32 * hf, r);
                tc::tmem_ld_wait();
                if (hf == 1) {
                    tc::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&bars.s_empty[th]);
                }
#pragma unroll
                for (int j4 = 0; j4 < 4; ++j4) {
                    const float4 ts = ti[8 * hf + j4], tc2 = ti[SM_TOKPLANE / 16 + 8 * hf + j4];
                    const float sc4[4] = {ts.x, ts.y, ts.z, ts.w}, c24[4] = {tc2.x, tc2.y, tc2.z, tc2.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = 4 * j4 + e;
                        const float mine = __uint_as_float(tb ? r[16 + j] : r[j]);
                        const float give = __uint_as_float(tb ? r[j] : r[16 + j]);
                        const float raw = mine + __shfl_xor_sync(0xffffffffu, give, 16);
                        // rows past the end are exact zeros in shared memory, so their raw scores are 0 and an
                        // additive -inf makes every weight of theirs exactly 0 without a select per element
                        s2[16 * hf + j] = fmaf(raw, a_h * sc4[e], c24[e]);
                        mx = fmaxf(mx, s2[16 * hf + j]);
                    }
                }
            }
            // The references as tile i - 1 left them (the other group's tile)
            if (i > 0) {
                ok = tc::mbar_wait_warp(&bars.dec[th ^ 1], ((i - 1) >> 1) & 1, abort_flag, 65, A.max_polls);
                if (!ok) { give_up(); break; }
                const float m_now = s_mref[hd];
                if (m_now != m_ref) { l_acc *= exp2f(m_ref - m_now); m_ref = m_now; }
            }
            // asked ahead (a look at a barrier takes 200 cycles beside the MMAs, one whose phase is complete as well)
            const bool pv_ready = i == 0 || tc::mbar_test(&bars.pv_done[th ^ 1], ((i - 1) >> 1) & 1);   // PV(i - 1) has read the P' tile

            // Fast path: no score of the tile exceeds its head's reference by more than AM_LAG, so the
            // references stand and nothing has to be exchanged. One barrier-with-OR decides for the group, and the other group
            // for its tile then.
            // (before the first live tile the reference is -inf; s2 carries AM_POFF, the reference does not)
            if (tc::barrier_any(6 + th, AM_GROUP_THREADS, mx - m_ref > AM_LAG + AM_POFF)) {
                // exact per-head tile max: this thread's tokens and its partner lane's
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                float fac = 1.0f;
                {
                    const float tm = mx - AM_POFF;
                    if (m_ref == -INFINITY) { if (tm > -INFINITY) m_ref = tm; }          // first live tile of this head
                    else if (tm > m_ref) { fac = exp2f(m_ref - tm); m_ref = tm; }          // any growth is taken now
                    if (lane < 16) { s_fac[hd] = fac; s_mref[hd] = m_ref; }
                }
                if (tc::barrier_any(8 + th, AM_GROUP_THREADS, false)) { ok = false; break; }
                // bring O^T and l to the new references. PV(i-1) must have landed first.
                if (i >= 1) ok = tc::mbar_wait_warp(&bars.pv_done[th ^ 1], ((i - 1) >> 1) & 1, abort_flag, 63, A.max_polls);
                if (!ok) { if (i + 2 < ntiles) give_up(); break; }
                tc::tc_fence_after();
                if (i >= 1) {
                    uint32_t r[32];
#pragma unroll 1
                    for (int c = 0; c < 8; ++c) {   // this thread's dim lane, half the head columns of a block at a time
                        tc::tmem_ld32(TM_O + lane_base + c * 32, r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int h = 0; h < 32; ++h) r[h] = __float_as_uint(__uint_as_float(r[h]) * s_fac[(c & 1) * 32 + h]);
                        tc::tmem_st32(TM_O + lane_base + c * 32, r);
                    }
                    tc::tmem_st_wait();
                }
                l_acc *= fac;
                tc::tc_fence_before();
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&bars.dec[th]);     // the other group may decide on its tile
            // P'' = 2^(s2' - m) = weight * s_tok * 2^AM_POFF as two e4m3 terms (via f16: p <= 256 and the
            // residual p - hi are exact enough in half precision); l accumulates the plain weight.
            // A head that has seen no live token yet has no reference: its scores are all -inf and weigh 0.
            const float m_use = m_ref == -INFINITY ? 0.0f : m_ref;
            uint32_t hi_w[8], lo_w[8];
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 ti4 = ti[2 * (SM_TOKPLANE / 16) + 8 * (j >> 4) + ((j & 15) >> 2)];
                const float inv4[4] = {ti4.x, ti4.y, ti4.z, ti4.w};
                uint32_t chs[2], cls[2];
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    float p0, p1;
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p0) : "f"(s2[j + e] - m_use));
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p1) : "f"(s2[j + e + 1] - m_use));
                    l_acc = fmaf(p0, inv4[e], l_acc);
                    l_acc = fmaf(p1, inv4[e + 1], l_acc);
                    const __half2 ph = __floats2half2_rn(p0, p1);
                    const uint32_t phb = *reinterpret_cast<const uint32_t*>(&ph);
                    uint16_t ch, cl;
                    uint32_t hfb;
                    asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(ch) : "r"(phb));
                    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(hfb) : "h"(ch));
                    const __half2 res = __hsub2(ph, *reinterpret_cast<const __half2*>(&hfb));
                    asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(cl) : "r"(*reinterpret_cast<const uint32_t*>(&res)));
                    chs[e >> 1] = ch; cls[e >> 1] = cl;
                }
                hi_w[j >> 2] = chs[0] | (chs[1] << 16);
                lo_w[j >> 2] = cls[0] | (cls[1] << 16);
            }
            if (!__all_sync(0xffffffffu, pv_ready)) ok = tc::mbar_wait_warp(&bars.pv_done[th ^ 1], ((i - 1) >> 1) & 1, abort_flag, 64, A.max_polls);
            if (!ok) { if (i + 2 < ntiles) give_up(); break; }
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                // row = head, bytes = tokens: this thread's 16 tokens of a half are the 16-byte chunk 2 hf + tb of its head's row
                uint8_t* prow = smem + SM_P + sw64_chunk(hd, 2 * hf + tb);
                *reinterpret_cast<uint4*>(prow) = make_uint4(hi_w[4 * hf], hi_w[4 * hf + 1], hi_w[4 * hf + 2], hi_w[4 * hf + 3]);
                *reinterpret_cast<uint4*>(prow + SM_PTERM) = make_uint4(lo_w[4 * hf], lo_w[4 * hf + 1], lo_w[4 * hf + 2], lo_w[4 * hf + 3]);
            }
            tc::fence_proxy_async();
            tc::mbar_arrive(&bars.p_full);
        }

        // ---- epilogue ----
        rv_grid_dep_wait();   // (the grid is not to be complete before the kernel in front of it)
        // l per head: its four threads (two lanes 16 apart in a warp of each group) meet at the last reference by one shuffle
        // and one exchange through shared memory.
        tc::named_barrier(1, AM_SOFTMAX_THREADS);
        {
            const float m_now = s_mref[hd];
            if (m_now != m_ref) { l_acc *= exp2f(m_ref - m_now); m_ref = m_now; }
            const float mine = l_acc + __shfl_xor_sync(0xffffffffu, l_acc, 16);
            if (lane < 16) s_wmax[th * 64 + hd] = mine;
        }
        tc::named_barrier(1, AM_SOFTMAX_THREADS);
        if (th == 0 && lane < 16) {
            const int h = hd;
            const float l = s_wmax[h] + s_wmax[64 + h];
            const float m_nat = (m_ref - AM_POFF) * 0.6931471805599453f;   // natural-log units (l and O carry 2^AM_POFF)
            if (clustered) {
                my_ml = (l > 0.0f && ok) ? make_float2(m_ref, l) : make_float2(-INFINITY, 0.0f);
            } else if (skip) {
                // nothing: the sequence's output and statistics are written by the CUDA-core kernel
            } else {
                if (A.out_m) A.out_m[(size_t)b * AM_H + h] = l > 0.0f ? m_nat : -INFINITY;
                if (A.out_lse) A.out_lse[(size_t)b * AM_H + h] = l > 0.0f ? m_nat + logf(l) : -INFINITY;
            }
            s_fac[h] = l > 0.0f ? 1.0f / l : 0.0f;
        }
        if (ok && ntiles > 0) ok = tc::mbar_wait_warp(&bars.pv_done[(ntiles - 1) & 1], ((ntiles - 1) >> 1) & 1, abort_flag, 66, A.max_polls);
        tc::tc_fence_after();
        tc::named_barrier(1, AM_SOFTMAX_THREADS);
        // O^T: this thread's TMEM lane is one latent dim of each 128-dim block; its head columns. Every MMA of the CTA has
        // read its operands, so the idle ring takes the bf16 output, eight heads of a token half at a time (all 512 dims:
        // four accumulator blocks), and each group leaves as one 8 KiB bulk copy while the next is converted. (A split
        // sequence is merged inside its cluster instead, below.)
        // 2-byte stores from the registers to global memory took 6,700 cycles for the epilogue, 4,400 this way.
        if (!skip && !clustered) {
            uint16_t* stage = reinterpret_cast<uint16_t*>(smem + SM_STAGE);
            const bool have = ntiles > 0 && ok;
#pragma unroll 1
            for (int g = 0; g < AM_HPT / 8; ++g) {
                const int hg = h0 + g * 8;
                uint32_t r[4][8];
#pragma unroll
                for (int c = 0; c < 4; ++c) tc::tmem_ld8(TM_O + lane_base + c * 64 + hg, r[c]);
                tc::tmem_ld_wait();
                const float4 i0 = *reinterpret_cast<const float4*>(s_fac + hg), i1 = *reinterpret_cast<const float4*>(s_fac + hg + 4);
                const float inv_l[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
                uint16_t* sp = stage + hg * AM_KVL + row;
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        const float x = have ? __uint_as_float(r[c][i]) * inv_l[i] : 0.0f, y = have ? __uint_as_float(r[c][i + 1]) * inv_l[i + 1] : 0.0f;
                        uint32_t w2;
                        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w2) : "f"(y), "f"(x));
                        sp[i * AM_KVL + c * 128] = (uint16_t)w2;
                        sp[(i + 1) * AM_KVL + c * 128] = (uint16_t)(w2 >> 16);
                    }
                tc::fence_proxy_async();
                tc::named_barrier(4 + th, AM_SOFTMAX_THREADS / 2);
                if (sq == 0 && lane == 0) {
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                 ::"l"(A.out + ((size_t)b * AM_H + hg) * AM_KVL), "r"(tc::smem_u32(stage + hg * AM_KVL)), "r"(8 * AM_KVL * 2) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            if (sq == 0 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    }

    if (clustered) {
        // ---- merge of a sequence's splits inside its thread-block cluster (o_merge.cuh) ----
        // All threads of all CTAs take part in both cluster barriers, whatever a bounded wait did before: a CTA that gave up
        // sends weight sums of zero.
        const om::Share S(A.n_splits, split, (int)gridDim.z, (int)blockIdx.z);
        float* recv = reinterpret_cast<float*>(smem + SM_STAGE);              // [n][hpc][512]
        float2* ml = reinterpret_cast<float2*>(smem + SM_QR);                 // [n][hpc]: (maximum, sum) of rank q
        float* wts = reinterpret_cast<float*>(smem + SM_P);                   // [hpc][8]: what rank q's row counts
        const bool live = ntiles > 0 && *abort_flag == 0;
        om::cluster_arrive();
        om::cluster_wait();                                                   // [1] every CTA's MMAs have read their ring and q
        if (warp < AM_SW) {
            if (publishes) om::push_stats(S, ml, ph, live ? my_ml : make_float2(-INFINITY, 0.0f));
            om::push_rows(S, TM_O, recv, live, warp, lane);
        }
        om::cluster_arrive();
        om::cluster_wait();                                                   // [2] every CTA's share of this CTA's heads
        // eight lanes a head (a lane per rank) work out what each rank's row counts
        static_assert(om::MAX_N == 8 && AM_H / 2 * 8 <= AM_THREADS, "eight lanes a head, at most half of the heads");
        const int wh = tid >> 3, wq = tid & 7;
        const bool told = wh < S.heads && wq < S.n;
        const float2 part = told ? ml[wq * S.hpc + wh] : make_float2(-INFINITY, 0.0f);
        const float mg = om::fold8<false>(part.x), w = part.y > 0.0f ? exp2f(part.x - mg) : 0.0f, L = om::fold8<true>(part.y * w);
        if (told) wts[wh * om::MAX_N + wq] = L > 0.0f ? w / L : 0.0f;
        __syncthreads();
        if (!skip) {
            om::write_rows(S, recv, wts, A.out + (size_t)b * AM_H * AM_KVL, tid, AM_THREADS);
            if (wq == 0 && told) {
                const size_t at = (size_t)b * AM_H + S.hz0 + S.lo + wh;
                const float m_nat = (mg - AM_POFF) * 0.6931471805599453f;
                if (A.out_m) A.out_m[at] = L > 0.0f ? m_nat : -INFINITY;
                if (A.out_lse) A.out_lse[at] = L > 0.0f ? m_nat + logf(L) : -INFINITY;
            }
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == AM_QKW) {
        tc::settle(*abort_flag);
        tc::tmem_dealloc<512>(tmem);
    }
    if (tid == 0 && *abort_flag) atomicCAS(A.err, 0, *abort_flag);
}

// A CTA takes a whole SM (shared memory), and the CTAs of a sequence form one thread-block cluster (co-scheduled
// inside a GPC). A batch is split only as far as all its clusters are resident at once: the largest cluster size
// (<= 8) for which the device reports room for B clusters; anything more would run as a second wave. What room is left then
// goes to clusters that share a sequence's heads.
// The split follows the batch alone: cut to two tiles per CTA where the list is short, the same rows gave other bits in a list of
// another length, 1.2 % further from their 64-bit value (each CTA has reference maxima of its own, and fewer of them serve the
// same rows); steps of one to four sequences of 256 - 1,024 tokens took 2 - 12 % longer so, of eight to twenty 4 - 12 % less.
struct MmaPlan { int splits, shares; };
int mma_resident(int B, int n) {           // clusters of n CTAs that are resident at once
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n, (unsigned)B); cfg.blockDim = dim3(AM_THREADS); cfg.dynamicSmemBytes = SM_TOTAL;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)n; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, attend_mma_kernel, &cfg) == cudaSuccess) return active;
    (void)cudaGetLastError();
    return 0;
}
MmaPlan mma_plan(int B) {
    constexpr int MOST = 128;
    static std::atomic<int> cache[MOST + 1];            // largest resident cluster size by batch; 0 = not asked yet
    static std::atomic<int> room[AM_MAX_SPLITS + 1];    // resident clusters by size, plus 1
    const int sms = rv_sm_count();
    if (B <= 0 || B > MOST || 2 * B > sms) return {1, 1};
    int n = cache[B].load(std::memory_order_relaxed);
    if (!n) {
        for (n = sms / B < AM_MAX_SPLITS ? sms / B : AM_MAX_SPLITS; n > 1; --n)
            if (mma_resident(B, n) >= B) break;
        if (n < 1) n = 1;
        cache[B].store(n, std::memory_order_relaxed);
    }
    if (n < 2) return {1, 1};
    int active = room[n].load(std::memory_order_relaxed) - 1;
    if (active < 0) {
        active = mma_resident(B, n);
        room[n].store(active + 1, std::memory_order_relaxed);
    }
    return {n, om::shares(n, B, active)};
}

}  // namespace

extern "C" bool rivoli_attend_mma_supported(const DsaGeom* g) {
    return g->n_heads == AM_H && g->kv_lora == AM_KVL && g->rope_dim == AM_ROPE;
}

// scratch layout: [err 256 B]. The error word is sticky: it keeps the first failure
// until rivoli_attend_mma_status reads and clears it, so it must be zero before the first call.

extern "C" int rivoli_attend_simt_short_rows(const DsaGeom* g, const uint16_t* q, const uint8_t* latent_pool,
                                             const float* latent_scale, const int32_t* block_table,
                                             const uint32_t* rows, int row_stride, const int32_t* n_rows, int B,
                                             uint16_t* out, float* out_m, float* out_lse, int rows_lo,
                                             int rows_hi, cudaStream_t st);

// Below this many attended rows a sequence is served by the f32 CUDA-core kernel instead: with one tile
// or less the two-term fp8 operands of the tensor-core kernel (bf16-class, ~2^-9) no longer average out
// against the 1e-3 absolute tolerance on near-zero outputs.
constexpr int AM_MIN_ROWS = 128;

// Self-test state (rivoli_attend_mma_test_hook): overrides of the next launches, host side only.
static std::atomic<int> g_am_min_rows_override{-1}, g_am_withhold_once{0}, g_am_max_polls{tc::kMaxPolls};

// Test hook, not for production callers. min_rows >= 0 replaces AM_MIN_ROWS until reset with -1 (0 sends every
// sequence to the tensor-core kernel); withhold != 0 makes the NEXT launch leave out one barrier arrival so that
// its bounded waits run out (the launch returns, the status call reports 1008 and later launches are unaffected);
// max_polls > 0 sets the poll limit of the bounded waits (<= 0 restores the default).
extern "C" __attribute__((visibility("default"))) void rivoli_attend_mma_test_hook(int min_rows, int withhold,
                                                                                    int max_polls) {
    g_am_min_rows_override = min_rows;
    g_am_withhold_once = withhold;
    g_am_max_polls = max_polls > 0 ? max_polls : tc::kMaxPolls;
}

// q_early != 0: the caller guarantees q was complete before the kernel preceding this call in the stream
// was launched (the fused decode step), so the query conversion may overlap that kernel's tail.
// min_rows_hint: a lower bound the caller knows for n_rows over the batch (0 = unknown). With a bound of
// AM_MIN_ROWS or more no sequence needs the CUDA-core arm and its launch is left out. max_rows: an upper bound; below
// AM_MIN_ROWS no sequence needs this kernel and the CUDA-core arm serves them all, the empty ones too.
// fresh_pos (with q_early): the launch before this call's first appends ONE token per sequence, at these positions, and writes nothing
// else that the attention reads, but rows and n_rows if dense_len is given: they are then the first min(dense_len[b], max_rows)
// tokens of each sequence.
extern "C" int rivoli_attend_mma_paged_bf16(const DsaGeom* g, const uint16_t* q, const uint8_t* latent_pool,
                                            const float* latent_scale, const int32_t* block_table,
                                            const uint32_t* rows, int row_stride, const int32_t* n_rows, int B,
                                            uint16_t* out, float* out_m, float* out_lse, void* scratch,
                                            int q_early, int min_rows_hint, long long max_rows, const int32_t* fresh_pos,
                                            const int32_t* dense_len, void* stream) {
    if (!scratch) return 1001;
    if (((uintptr_t)latent_pool | (uintptr_t)scratch | (uintptr_t)q | (uintptr_t)out) & 15) return 1005;
    cudaStream_t st = (cudaStream_t)stream;
    int* err = reinterpret_cast<int*>(scratch);
    rv_allow_smem<attend_mma_kernel>(SM_TOTAL);
    const int forced = g_am_min_rows_override.load(std::memory_order_relaxed);
    int min_rows = forced >= 0 ? forced : AM_MIN_ROWS;
    if (min_rows_hint >= min_rows) min_rows = 0;          // the caller vouches that no sequence is that short
    const int withhold = g_am_withhold_once.load(std::memory_order_relaxed) ? g_am_withhold_once.exchange(0) : 0;

    // short contexts first (a programmatic dependent of whatever precedes this call; its CTAs leave at once
    // for every other sequence), then the tensor-core kernel as a dependent of that launch
    long long cap = (long long)g->max_pages_per_seq * g->page_tokens;
    if (rows && row_stride > cap) cap = row_stride;   // (a row list may name a row twice)
    const bool only_short = (cap < max_rows ? cap : max_rows) < min_rows;
    const MmaPlan plan = mma_plan(B);
    if (min_rows > 1)
        if (int e = rivoli_attend_simt_short_rows(g, q, latent_pool, latent_scale, block_table, rows, row_stride, n_rows,
                                                  B, out, out_m, out_lse, only_short ? 0 : 1, min_rows, st))
            return e;
    if (only_short) return 0;
    rv_drain_error();
    if (B > 2 * AM_GW * 32) fresh_pos = dense_len = nullptr;   // (two marked rows per gather thread)
    AttendMmaArgs a{q, g->softmax_scale, latent_pool, latent_scale, block_table, dense_len ? nullptr : rows, row_stride, dense_len ? dense_len : n_rows,
                    g->page_tokens, g->max_pages_per_seq, g->n_pool_pages, plan.splits,
                    out, out_m, out_lse, err,
                    min_rows, q_early ? 1 : 0, g_am_max_polls.load(std::memory_order_relaxed),
                    fresh_pos, B, dense_len ? (int)max_rows : 0x7fffffff, withhold};
    // one CTA per (sequence, split); the splits of a sequence are one thread-block cluster and merge inside the kernel
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.splits, (unsigned)B, (unsigned)plan.shares); cfg.blockDim = dim3(AM_THREADS);
    cfg.dynamicSmemBytes = (size_t)SM_TOTAL; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)plan.splits; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = plan.splits > 1 ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, attend_mma_kernel, a);
    return rv_launch_status();
}

// Synchronises `stream`; 1008 if a bounded device-side wait of the last call gave up.
extern "C" int rivoli_attend_mma_status(void* scratch, void* stream) {
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, scratch, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return -(int)e;
    if (h) cudaMemsetAsync(scratch, 0, sizeof(int), (cudaStream_t)stream);
    return h ? 1008 : 0;
}

