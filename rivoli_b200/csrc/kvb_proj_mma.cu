// Batched kv_b projections on the tensor cores (tcgen05, kind::f16: bf16 x bf16 -> f32).
//
// kv_b holds e4m3 codes with one f32 scale per 128 x 128 block. An e4m3 code is exactly a bf16
// number, so the codes go to shared memory as bf16 (converted on the way in) and the activations
// stay bf16: every product in the MMA is exact. The block scale cannot ride inside the MMA, so each
// run of the contraction with ONE scale gets its own TMEM accumulator and the epilogue adds the
// runs in f32: out = sum_run scale_run * D_run.
//
//   absorb: q_abs[b][h][i] = sum_d q[b][h][d] * kvb[448 h + d][i]         M = 128 sequences, N = 128 of the
//           512 latent columns (one scale column), K = nope = 192 = two runs (the head's rows straddle one
//           block boundary); CTA = (column block, head); weights are the MN-major B operand.
//   value:  ctx[b][h][j]  = sum_i o[b][h][i] * kvb[448 h + 192 + j][i]     M = 128 sequences, N = 128 of the 256
//           value rows (two scale rows, one per 64 columns), K = kvl = 512 = four runs (one per scale
//           column); CTA = (row block, head) - 128 CTAs, one wave; weights are the K-major B operand.
// Geometry outside these shapes takes the CUDA-core kernels of kvb_proj.cu.
// All waits are bounded (tc_common.cuh); a wait that gives up sets g_kp_err (rivoli_kvb_proj_status).
#include "codec.cuh"
#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int KP_THREADS = 256;   // warps 0-7 request, convert and store (epilogue by (lane quadrant, column half))
constexpr int KP_LAUNCH = KP_THREADS + 32;   // warp 8 issues the MMAs: by one of the converting warps that took half of a chunk's time
__device__ int g_kp_err;

__device__ __forceinline__ uint64_t kp_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;   // 128-byte swizzle
    return d;
}
// Instruction descriptor, kind::f16: bf16 x bf16 -> f32.
__device__ __forceinline__ uint32_t kp_idesc(int M, int N, int b_mn_major) {
    uint32_t d = 0;
    d |= 1u << 4;                      // accumulator f32
    d |= 1u << 7;                      // A = bf16
    d |= 1u << 10;                     // B = bf16
    d |= (uint32_t)b_mn_major << 16;   // A is always K-major here
    d |= (uint32_t)(N >> 3) << 17;
    d |= (uint32_t)(M >> 4) << 24;
    return d;
}
__device__ __forceinline__ void kp_mma(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// 8 e4m3 codes -> 8 bf16 (exact), as one 16-byte chunk.
__device__ __forceinline__ uint4 kp_codes_to_bf16(uint2 c) {
    uint32_t o[4];
    const uint32_t w[2] = {c.x, c.y};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint16_t pair = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
        const float2 f = rv_e4m3x2_to_f32x2(pair);
        o[i] = (__float_as_uint(f.x) >> 16) | (__float_as_uint(f.y) & 0xffff0000u);   // exact: 3 mantissa bits
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

__device__ __forceinline__ uint32_t kp_pack(float a, float b) {   // two f32 -> bf16x2, round to nearest even
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}

struct KpArgs {
    const uint16_t* x;      // activations [B][H][xs] bf16 (xs = row pitch per head)
    const uint8_t* kvb; const float* scale;
    int H, xs, nope, vh, kvl, rope, block, B;
    uint16_t* out;
};

// The contraction in chunks of 64, one cp.async group each (activations, raw codes), all requested ahead. A chunk's codes are
// converted (two tile buffers) and its MMAs issued while later chunks are on their way; they stay for the next batch tile. The
// result is staged in the idle converted tiles and leaves as whole rows.
// 128 sequences, us, each behind itself with cold weights: absorb 16.4 -> 8.9, value 15.9 -> 9.9 (before: loads into registers,
// one conversion pass, two halves of the value contraction one after the other, 16-byte stores to 32 rows at a time); bound by
// what an SM takes in (192 KiB at 18 bytes a clock in the value kernel), a launch's ramp and the epilogue. Three chunks of the value contraction in
// flight, with which a value CTA can start beside an absorb CTA, are slower in every order of the launches: absorb and value of
// 128 / 8 sequences back to back 18.2 / 16.2 us, 17.5 / 15.4 so; with a layer's attention between them 88.5 / 38.0 and 87.3 / 36.9.
constexpr int KP_ACHUNK = 16384, KP_WCHUNK = 8192, KP_CONV = 16384;
static_assert(2 * KP_CONV == 128 * 256, "the result fits the converted tiles");

// Requests activation chunk c (128 sequences from b0 x 64 bf16, swizzled K-major; rows past B are zeros) into `dst`.
__device__ __forceinline__ void kp_request_acts(const KpArgs& A, int h, int b0, int c, uint8_t* dst) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = threadIdx.x + i * KP_THREADS, row = e >> 3, j = e & 7;
        const bool live = b0 + row < A.B;
        tc::cp_async16_zfill(tc::smem_u32(dst + tc::sw128_chunk(row, j)),
                             A.x + ((size_t)(live ? b0 + row : 0) * A.H + h) * A.xs + c * 64 + j * 8, live ? 16u : 0u);
    }
}
// Asks L2 for `n` runs of `bytes` bytes, `pitch` apart (whole CTA, lines of 128 bytes). Under a programmatic dependent launch a
// CTA may sit here while the kernel before it finishes; a prefetch into L2 may precede the dependency wait, whoever writes.
__device__ __forceinline__ void kp_prefetch(const void* base, size_t pitch, int n, int bytes) {
    const int lines = (bytes + 127) / 128;
    for (int e = threadIdx.x; e < n * lines; e += KP_LAUNCH) {
        const int r = e / lines;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint8_t*>(base) + (size_t)r * pitch + (e - r * lines) * 128));
    }
}
// Sixteen e4m3 codes of a raw piece -> two 16-byte bf16 chunks.
__device__ __forceinline__ void kp_convert16(const uint8_t* raw, uint8_t* d0, uint8_t* d1) {
    const uint4 v = *reinterpret_cast<const uint4*>(raw);
    *reinterpret_cast<uint4*>(d0) = kp_codes_to_bf16(make_uint2(v.x, v.y));
    *reinterpret_cast<uint4*>(d1) = kp_codes_to_bf16(make_uint2(v.z, v.w));
}
constexpr int KP_ACHUNKS = 4, KP_VCHUNKS = 8;      // most chunks of a contraction (rivoli_kvb_mma_supported: nope <= 256, kvl <= 512)
// Waits until at most `left` of this thread's copy groups are pending (left < KP_ACHUNKS).
__device__ __forceinline__ void kp_wait_groups(int left) {
    switch (left) {
        case 0: tc::cp_async_wait<0>(); break;
        case 1: tc::cp_async_wait<1>(); break;
        case 2: tc::cp_async_wait<2>(); break;
        default: tc::cp_async_wait<KP_ACHUNKS - 1>(); break;
    }
}
// The 128 x 128 bf16 result staged as [128 rows][256 B], 16-byte chunks XORed with the row: chunk k of row r.
__device__ __forceinline__ uint32_t kp_stage(int r, int k) { return (uint32_t)(r * 256 + ((k ^ (r & 7)) << 4)); }
// ... and stored: sixteen lanes a row.
__device__ __forceinline__ void kp_store_rows(const uint8_t* stage, uint16_t* out, size_t pitch, int rows) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = threadIdx.x + i * KP_THREADS, r = e >> 4, k = e & 15;
        if (r < rows) *reinterpret_cast<uint4*>(out + (size_t)r * pitch + k * 8) = *reinterpret_cast<const uint4*>(stage + kp_stage(r, k));
    }
}

// ---------------------------------------------------------------------------------------------
// absorb: grid (kvl / 128, H). Shared: activation chunks [nope/64][128 rows][128 B] | raw codes [nope/64][64 rows][128 B] |
// two converted tiles [2 column halves][64 rows][128 B] (MN-major).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(KP_LAUNCH)
kvb_absorb_mma_kernel(KpArgs A) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar[2], full[2];   // MMAs of a converted tile done | its conversion done
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int iblk = blockIdx.x, h = blockIdx.y;
    const int nope = A.nope, kvl = A.kvl, W = A.kvl + A.rope, nch = nope / 64;
    uint8_t* sA = smem;
    uint8_t* sW = sA + nch * KP_ACHUNK;
    uint8_t* sB = sW + nch * KP_WCHUNK;
    const size_t rbase = (size_t)h * (nope + A.vh);
    const int sc_cols = kvl / 128;
    // runs of d with one scale: [0, cut) and [cut, nope); cut = distance to the next block boundary
    const int cut = min(nope, (int)(128 - (rbase & 127)));
    const bool two_runs = cut < nope;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { tc::mbar_init(&bar[i], 1); tc::mbar_init(&full[i], KP_THREADS); }
        tc::mbar_init_fence();
        abort_word = 0;
    }
    if (warp == 8) tc::tmem_alloc<256>(&tmem_slot);
    kp_prefetch(A.kvb + rbase * kvl + iblk * 128, (size_t)kvl, nope, 128);
    kp_prefetch(A.x + (size_t)h * A.xs, (size_t)A.H * A.xs * 2, min(128, A.B), nope * 2);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    // Behind the allocation, which waits for its columns without a limit: a dependent that is already on the SM could take them
    // and then wait for this grid.
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    if (warp < 8) for (int c = 0; c < nch; ++c) {
        kp_request_acts(A, h, 0, c, sA + c * KP_ACHUNK);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = tid + i * KP_THREADS, d = e >> 3, j = e & 7;
            tc::cp_async16(tc::smem_u32(sW + c * KP_WCHUNK + d * 128 + j * 16), A.kvb + (rbase + c * 64 + d) * kvl + iblk * 128 + j * 16);
        }
        tc::cp_async_commit();
    }
    const float s0 = A.scale[(rbase >> 7) * sc_cols + iblk];
    const float s1 = two_runs ? A.scale[((rbase + cut) >> 7) * sc_cols + iblk] : 0.0f;
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = kp_idesc(128, 128, 1);
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;   // TMEM lane quadrant of this warp
    const int erow = (warp & 3) * 32 + lane, chalf = warp >> 2;      // epilogue: sequence row, column half
    bool ok = true;
    int done[2] = {0, 0};
    for (int b0 = 0; b0 < A.B; b0 += 128) {                  // (after a wait that gave up too: the barriers stay matched)
        if (warp == 8) {
            for (int c = 0; c < nch && ok; ++c) {
                const int wb = c & 1, run = c * 64 >= cut ? 1 : 0;       // (a run boundary is a multiple of 64)
                ok = tc::mbar_wait_warp(&full[wb], done[wb]++ & 1, abort_flag, 75);
                if (!ok) break;
                tc::tc_fence_after();
                const uint64_t da = kp_desc(tc::smem_u32(sA + c * KP_ACHUNK), 16, 1024), db = kp_desc(tc::smem_u32(sB + wb * KP_CONV), 8192, 1024);
                const uint32_t fresh = (c == 0 || c * 64 == cut) ? 0u : 1u;
                if (tc::elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) kp_mma(tmem + run * 128, da + 2 * k, db + 128 * k, idesc, k ? 1u : fresh);   // address fields count 16-byte units
                    tc::mma_commit(&bar[wb]);
                }
                __syncwarp();
            }
            __syncthreads();
            __syncthreads();
            continue;
        }
        if (b0 > 0)
            for (int c = 0; c < nch; ++c) { kp_request_acts(A, h, b0, c, sA + c * KP_ACHUNK); tc::cp_async_commit(); }
        // the rope segment of q rides along (column block 0 only)
        const int rope16 = A.rope / 8;
        uint4 rope_v[4];
        if (iblk == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = tid + i * KP_THREADS, r = rope16 > 0 ? e / rope16 : 128, j = e - r * rope16;
                if (r < 128 && b0 + r < A.B) rope_v[i] = *reinterpret_cast<const uint4*>(A.x + ((size_t)(b0 + r) * A.H + h) * A.xs + nope + j * 8);
            }
        }
        for (int c = 0; c < nch && ok; ++c) {
            const int wb = c & 1;
            if (done[wb] > 0) ok = tc::mbar_wait_warp(&bar[wb], (done[wb] - 1) & 1, abort_flag, 71);
            if (!ok) break;
            kp_wait_groups(nch - 1 - c);   // (a thread converts the codes that it requested itself)
            uint8_t* sb = sB + wb * KP_CONV;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int e = tid + i * KP_THREADS, d = e >> 3, j = e & 7;
                uint8_t* half = sb + (j >> 2) * 8192;
                kp_convert16(sW + c * KP_WCHUNK + d * 128 + j * 16, half + tc::sw128_chunk(d, (j & 3) * 2), half + tc::sw128_chunk(d, (j & 3) * 2 + 1));
            }
            tc::fence_proxy_async();
            tc::mbar_arrive(&full[wb]);
            ++done[wb];
        }
        if (iblk == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = tid + i * KP_THREADS, r = rope16 > 0 ? e / rope16 : 128, j = e - r * rope16;
                if (r < 128 && b0 + r < A.B) *reinterpret_cast<uint4*>(A.out + ((size_t)(b0 + r) * A.H + h) * W + kvl + j * 8) = rope_v[i];
            }
        }
        for (int wb = 0; wb < 2 && ok; ++wb)
            if (done[wb] > 0) ok = tc::mbar_wait_warp(&bar[wb], (done[wb] - 1) & 1, abort_flag, 72);
        tc::tc_fence_after();
        if (ok) {
#pragma unroll
            for (int c = chalf * 2; c < chalf * 2 + 2; ++c) {
                uint32_t r0[32], r1[32];
                tc::tmem_ld32(tmem + lane_base + c * 32, r0);
                tc::tmem_ld32(tmem + lane_base + 128 + c * 32, r1);
                tc::tmem_ld_wait();
                if (!two_runs) {   // the second accumulator was never written
#pragma unroll
                    for (int e = 0; e < 32; ++e) r1[e] = 0u;
                }
                uint32_t o[16];
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    const float v0 = fmaf(__uint_as_float(r1[e]), s1, __uint_as_float(r0[e]) * s0);
                    const float v1 = fmaf(__uint_as_float(r1[e + 1]), s1, __uint_as_float(r0[e + 1]) * s0);
                    o[e >> 1] = kp_pack(v0, v1);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    *reinterpret_cast<uint4*>(sB + kp_stage(erow, c * 4 + e)) = make_uint4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]);
            }
        }
        tc::tc_fence_before();
        __syncthreads();
        if (ok) kp_store_rows(sB, A.out + ((size_t)b0 * A.H + h) * W + iblk * 128, (size_t)A.H * W, min(128, A.B - b0));
        __syncthreads();   // TMEM and the A tiles are free for the next batch tile
    }
    tc::cp_async_wait<0>();
    if (warp == 8) {
        tc::settle(abort_word);
        tc::tmem_dealloc<256>(tmem);
    }
    if (tid == 0 && abort_word) atomicCAS(&g_kp_err, 0, abort_word);
}

// ---------------------------------------------------------------------------------------------
// value: grid (vh / 128, H), N = 128 value rows = two 64-row scale rows. Shared: activation chunks [kvl/64][128 rows][128 B] |
// raw codes [kvl/64][128 rows][64 B] (room for eight of each) | two converted tiles [128 rows][128 B] (K-major).
// TMEM: one 128-column accumulator per scale column (kvl / 128 <= 4 runs).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(KP_LAUNCH)
kvb_value_mma_kernel(KpArgs A) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar[2], full[2];   // MMAs of a converted tile done | its conversion done
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    __shared__ float s_sc[2][4];
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int jblk = blockIdx.x, h = blockIdx.y;
    const int kvl = A.kvl, vh = A.vh, nch = kvl / 64;
    uint8_t* sA = smem;
    uint8_t* sW = sA + KP_VCHUNKS * KP_ACHUNK;
    uint8_t* sB = sW + KP_VCHUNKS * KP_WCHUNK;
    const size_t row0 = (size_t)h * (A.nope + vh) + A.nope + (size_t)jblk * 128;   // 128 value rows = 2 scale rows
    const int sc_cols = kvl / 128;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { tc::mbar_init(&bar[i], 1); tc::mbar_init(&full[i], KP_THREADS); }
        tc::mbar_init_fence();
        abort_word = 0;
    }
    if (warp == 8) tc::tmem_alloc<512>(&tmem_slot);
    kp_prefetch(A.kvb + row0 * kvl, (size_t)kvl, 128, kvl);
    kp_prefetch(A.x + (size_t)h * A.xs, (size_t)A.H * A.xs * 2, min(128, A.B), kvl * 2);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    rv_grid_dep_trigger();   // (behind the allocation: see the absorb kernel)
    rv_grid_dep_wait();
    // (a group per chunk that there could be, so that the waits below have constant counts)
    if (warp < 8)
#pragma unroll 1
        for (int c = 0; c < KP_VCHUNKS; ++c) {
            if (c < nch) {
                kp_request_acts(A, h, 0, c, sA + c * KP_ACHUNK);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int e = tid + i * KP_THREADS, r = e >> 2, j = e & 3;
                    tc::cp_async16(tc::smem_u32(sW + c * KP_WCHUNK + r * 64 + j * 16), A.kvb + (row0 + r) * kvl + c * 64 + j * 16);
                }
            }
            tc::cp_async_commit();
        }
    if (tid < 2 * sc_cols) s_sc[tid / sc_cols][tid % sc_cols] = A.scale[((row0 + (tid / sc_cols) * 64) >> 7) * sc_cols + tid % sc_cols];
    __syncthreads();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = kp_idesc(128, 128, 0);
    const uint32_t lane_base = ((uint32_t)((warp & 3) * 32)) << 16;   // TMEM lane quadrant of this warp
    const int erow = (warp & 3) * 32 + lane, chalf = warp >> 2;      // epilogue: sequence row, 64-column half
    bool ok = true;
    int done[2] = {0, 0};
    for (int b0 = 0; b0 < A.B; b0 += 128) {                  // (after a wait that gave up too: the barriers stay matched)
        if (warp == 8) {
            for (int c = 0; c < nch && ok; ++c) {
                const int wb = c & 1;
                ok = tc::mbar_wait_warp(&full[wb], done[wb]++ & 1, abort_flag, 76);
                if (!ok) break;
                tc::tc_fence_after();
                const uint64_t da = kp_desc(tc::smem_u32(sA + c * KP_ACHUNK), 16, 1024), db = kp_desc(tc::smem_u32(sB + wb * KP_CONV), 16, 1024);
                if (tc::elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) kp_mma(tmem + (c >> 1) * 128, da + 2 * k, db + 2 * k, idesc, ((c & 1) | k) ? 1u : 0u);
                    tc::mma_commit(&bar[wb]);
                }
                __syncwarp();
            }
            __syncthreads();
            __syncthreads();
            continue;
        }
        if (b0 > 0)
            for (int c = 0; c < KP_VCHUNKS; ++c) {
                if (c < nch) kp_request_acts(A, h, b0, c, sA + c * KP_ACHUNK);
                tc::cp_async_commit();
            }
        for (int c = 0; c < nch && ok; ++c) {
            const int wb = c & 1;
            if (done[wb] > 0) ok = tc::mbar_wait_warp(&bar[wb], (done[wb] - 1) & 1, abort_flag, 73);
            if (!ok) break;
            if (c > 0) tc::cp_async_commit();             // (empty: the group of chunk c stays KP_VCHUNKS - 1 from the newest)
            tc::cp_async_wait<KP_VCHUNKS - 1>();          // (a thread converts the codes that it requested itself)
            uint8_t* sb = sB + wb * KP_CONV;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int e = tid + i * KP_THREADS, r = e >> 2, j = e & 3;
                kp_convert16(sW + c * KP_WCHUNK + r * 64 + j * 16, sb + tc::sw128_chunk(r, 2 * j), sb + tc::sw128_chunk(r, 2 * j + 1));
            }
            tc::fence_proxy_async();
            tc::mbar_arrive(&full[wb]);
            ++done[wb];
        }
        for (int wb = 0; wb < 2 && ok; ++wb)
            if (done[wb] > 0) ok = tc::mbar_wait_warp(&bar[wb], (done[wb] - 1) & 1, abort_flag, 74);
        tc::tc_fence_after();
        if (ok) {
#pragma unroll
            for (int c = chalf * 2; c < chalf * 2 + 2; ++c) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {                 // sixteen columns: all runs of them in flight together
                    uint32_t r[4][16];
#pragma unroll
                    for (int run = 0; run < 4; ++run)
                        if (run < sc_cols) tc::tmem_ld16(tmem + lane_base + run * 128 + c * 32 + q * 16, r[run]);
                    tc::tmem_ld_wait();
                    float acc[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[e] = __uint_as_float(r[0][e]) * s_sc[chalf][0];
#pragma unroll
                    for (int run = 1; run < 4; ++run)
                        if (run < sc_cols) {
                            const float sc = s_sc[chalf][run];
#pragma unroll
                            for (int e = 0; e < 16; ++e) acc[e] = fmaf(__uint_as_float(r[run][e]), sc, acc[e]);
                        }
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        *reinterpret_cast<uint4*>(sB + kp_stage(erow, c * 4 + q * 2 + e)) =
                            make_uint4(kp_pack(acc[8 * e], acc[8 * e + 1]), kp_pack(acc[8 * e + 2], acc[8 * e + 3]),
                                       kp_pack(acc[8 * e + 4], acc[8 * e + 5]), kp_pack(acc[8 * e + 6], acc[8 * e + 7]));
                }
            }
        }
        tc::tc_fence_before();
        __syncthreads();
        if (ok) kp_store_rows(sB, A.out + ((size_t)b0 * A.H + h) * vh + jblk * 128, (size_t)A.H * vh, min(128, A.B - b0));
        __syncthreads();
    }
    tc::cp_async_wait<0>();
    if (warp == 8) {
        tc::settle(abort_word);
        tc::tmem_dealloc<512>(tmem);
    }
    if (tid == 0 && abort_word) atomicCAS(&g_kp_err, 0, abort_word);
}

}  // namespace

// The tensor-core kernels cover: 128 x 128 scale blocks; kvl 256 or 512; nope a multiple of 64 up to 256
// whose rows straddle at most one block boundary; vh a multiple of 128; the head's row count a multiple
// of 64; 16-byte aligned activation rows; rope <= 64.
extern "C" int rivoli_kvb_mma_supported(int H, int qh, int nope, int vh, int kvl, int rope, int block) {
    if (block != 128 || kvl % 256 || kvl > KP_VCHUNKS * 64 || nope % 64 || nope > KP_ACHUNKS * 64 || vh % 128 || (nope + vh) % 64) return 0;
    if (qh % 8 || rope % 8 || rope > 64 || H <= 0) return 0;
    for (int h = 0; h < 2 && h < H; ++h) {          // the straddle pattern repeats with period <= 2 heads
        const int off = (h * (nope + vh)) & 127;
        if (nope > (128 - off) + 128) return 0;       // would need a third run
    }
    return 1;
}

extern "C" int rivoli_kvb_absorb_mma(const uint16_t* q, const uint8_t* kvb, const float* scale, int H, int qh, int nope,
                                     int vh, int kvl, int rope, int block, int B, uint16_t* q_abs, cudaStream_t st) {
    const KpArgs a{q, kvb, scale, H, qh, nope, vh, kvl, rope, block, B, q_abs};
    const size_t smem = (size_t)(nope / 64) * (KP_ACHUNK + KP_WCHUNK) + 2 * KP_CONV;
    rv_allow_smem<kvb_absorb_mma_kernel>(KP_ACHUNKS * (KP_ACHUNK + KP_WCHUNK) + 2 * KP_CONV);
    rv_drain_error();
    rv_launch_dependent(kvb_absorb_mma_kernel, dim3(kvl / 128, H), dim3(KP_LAUNCH), smem, st, a);
    return rv_launch_status();
}

extern "C" int rivoli_kvb_value_mma(const uint16_t* clat, const uint8_t* kvb, const float* scale, int H, int nope, int vh,
                                    int kvl, int block, int B, uint16_t* ctx, cudaStream_t st) {
    const KpArgs a{clat, kvb, scale, H, kvl, nope, vh, kvl, 0, block, B, ctx};
    // (never two on an SM: each takes all of its tensor memory)
    constexpr int smem = KP_VCHUNKS * (KP_ACHUNK + KP_WCHUNK) + 2 * KP_CONV;
    rv_allow_smem<kvb_value_mma_kernel>(smem);
    rv_drain_error();
    rv_launch_dependent(kvb_value_mma_kernel, dim3(vh / 128, H), dim3(KP_LAUNCH), (size_t)smem, st, a);
    return rv_launch_status();
}

// Synchronises the stream; 1008 if a bounded wait of a tensor-core projection gave up since the last call.
RIVOLI_API int rivoli_kvb_proj_status(void* stream) {
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return -(int)e;
    int h = 0;
    e = cudaMemcpyFromSymbol(&h, g_kp_err, sizeof(int));
    if (e != cudaSuccess) return -(int)e;
    if (h) { const int z = 0; cudaMemcpyToSymbol(g_kp_err, &z, sizeof(int)); }
    return h ? 1008 : 0;
}

