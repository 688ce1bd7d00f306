// Indexer front end: the operators that produce what the lightning indexer consumes,
//   k   = rope(layernorm(wk . x))            index key    (crates/backend/kernels/indexer.hip:1-13)
//   q_h = rope((wq_b . q_resid)[h])           index queries
//   w   = weights_proj . x                    head weights
// with wk / wq_b / weights_proj fp8-e4m3 block-scaled.
//
//   rivoli_gemv_fp8, rivoli_layernorm, rivoli_rope_interleave : the reference's single-token f32
//       operators (linalg.hip:324-342, indexer.hip:22-50,259-266, activation.hip:337-371,551-559), same
//       arguments and guards. The GEMV folds in the order of the reference's host arithmetic
//       (crates/artifact/src/quant/fp8.rs:32-42), bit for bit.
//   rivoli_index_frontend_bf16 : the batched decode form - three block-scaled GEMMs over the batch
//       written as split-K partial sums (deterministic: a fixed split, summed in order), then one
//       per-sequence epilogue kernel that reduces the partials, applies LayerNorm to the key, rotates
//       key and queries at the sequence's position and stores bf16 - the rows rivoli_kv_append_paged and
//       rivoli_index_select_paged take.
#include "codec.cuh"
#include "common.cuh"
#include "fold_gemv.cuh"
#include "tc_common.cuh"

namespace {

// One block; sums in f64 (the reference's host test removes the summation-order error the same way),
// then the reference's f32 formula with var = E[x^2] - mean^2.
__global__ void __launch_bounds__(256)
layernorm_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, int n,
                 float eps, float* __restrict__ y) {
    __shared__ double ss[256], sq[256];
    const int t = threadIdx.x;
    rv_grid_dep_trigger();
    rv_grid_dep_wait();
    double s = 0.0, q = 0.0;
    for (int i = t; i < n; i += 256) { const double v = (double)x[i]; s += v; q += v * v; }
    ss[t] = s; sq[t] = q;
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if (t < st) { ss[t] += ss[t + st]; sq[t] += sq[t + st]; }
        __syncthreads();
    }
    const float mean = (float)(ss[0] / (double)n);
    const float var = __fsub_rn((float)(sq[0] / (double)n), __fmul_rn(mean, mean));
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(var, eps)));
    for (int i = t; i < n; i += 256) y[i] = __fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(x[i], mean), inv), w[i]), b[i]);
}

__global__ void rope_interleave_kernel(float* __restrict__ base, int stride, int seg, int pos, double theta) {
    const int s = blockIdx.x, j = threadIdx.x, half = seg / 2;
    float* v = base + (size_t)s * stride;
    rv_grid_dep_trigger();
    // the angle (f64) needs nothing from the kernel before
    const double ang = (double)pos * pow(theta, -2.0 * (double)j / (double)seg);
    const float cs = (float)cos(ang), sn = (float)sin(ang);
    rv_grid_dep_wait();
    const float a = v[2 * j], b = v[2 * j + 1];
    __syncthreads();   // every pair is read before any element is written: in place, race free
    v[j] = __fsub_rn(__fmul_rn(a, cs), __fmul_rn(b, sn));
    v[half + j] = __fadd_rn(__fmul_rn(b, cs), __fmul_rn(a, sn));
}

// ---------------------------------------------------------------------------------------------
// Batched front end.
// ---------------------------------------------------------------------------------------------
struct FrontMat { const uint8_t* w; const float* scale; int n; };   // weights e4m3 [n][K], block scales
struct FrontJob {            // Y[b][o] = sum over a K range of X[b][i] * W[o][i] * scale
    const uint16_t* x; int K;                         // activations bf16 [B][K]
    FrontMat m[2]; int N;                             // the outputs are m[0]'s rows, then m[1]'s (n = 0: none); N = both
    float* partial;                                   // f32 [k_splits][n_tiles][B][tile_n]
    int n_tiles, k_splits, k_chunks, cta0, tile_n;    // output tiles of tile_n columns, splits of k_chunks x 64 values, first CTA
    int mask;                                         // 16-byte pieces of a partial row are XORed with (row & mask)
};
struct FrontArgs { FrontJob job[3]; int n_jobs, B, block, n_cta; };

// CUDA-core split-K GEMM: CTA = (job, 64-output tile, K split), 256 threads = 64 outputs x 4 sequence
// groups; thread (o, g) folds its K range for sequences g, g + 4, ... (32 accumulators per pass of 128
// sequences). The weights of a 128-wide K chunk are staged dequantised in shared memory once per CTA;
// activations stream from L2. Works for any geometry.
constexpr int FT_N = 64, FT_KC = 128;
__global__ void __launch_bounds__(256)
front_gemm_simt_kernel(FrontArgs A) {
    __shared__ float ws[FT_KC][FT_N + 1];
    int jid = 0;
    while (jid < A.n_jobs - 1 && (int)blockIdx.x >= A.job[jid + 1].cta0) ++jid;
    const FrontJob& J = A.job[jid];
    const int local = blockIdx.x - J.cta0;
    const int tile = local % J.n_tiles, split = local / J.n_tiles;
    const int k0 = split * J.k_chunks * 64, k1 = min(J.K, k0 + J.k_chunks * 64);
    const int bq = threadIdx.x >> 6;   // this kernel always plans tile_n == FT_N and one matrix per job
    const int bsh = rv_log2(A.block), sc_cols = (J.K + A.block - 1) / A.block;
    rv_grid_dep_wait();
    rv_grid_dep_trigger();
    // sequences bq, bq + 4, ... ; at most 32 accumulators per thread per pass
    for (int b0 = 0; b0 < A.B; b0 += 128) {
        float acc[32];
#pragma unroll
        for (int r = 0; r < 32; ++r) acc[r] = 0.0f;
        for (int kc = k0; kc < k1; kc += FT_KC) {
            __syncthreads();
            for (int e = threadIdx.x; e < FT_KC * FT_N; e += 256) {
                const int kk = e % FT_KC, oo = e / FT_KC, i = kc + kk, og = tile * FT_N + oo;
                float v = 0.0f;
                if (i < k1 && og < J.N) v = __fmul_rn(rv_e4m3_to_f32(J.m[0].w[(size_t)og * J.K + i]), J.m[0].scale[(size_t)(og >> bsh) * sc_cols + (i >> bsh)]);
                ws[kk][oo] = v;
            }
            __syncthreads();
            const int kn = min(FT_KC, k1 - kc);
#pragma unroll
            for (int r = 0; r < 32; ++r) {
                const int b = b0 + bq + 4 * r;
                if (b < A.B) {
                    const uint16_t* xr = J.x + (size_t)b * J.K + kc;
                    float a = acc[r];
                    for (int kk = 0; kk < kn; ++kk) a = __fadd_rn(a, __fmul_rn(ws[kk][threadIdx.x & 63], rv_bf16_to_f32(xr[kk])));
                    acc[r] = a;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            const int b = b0 + bq + 4 * r;
            if (b < A.B) J.partial[(((size_t)split * J.n_tiles + tile) * A.B + b) * FT_N + (threadIdx.x & 63)] = acc[r];
        }
    }
}


// ---------------------------------------------------------------------------------------------
// The same split-K GEMM on the tensor cores (tcgen05 kind::f16). CTA = (job, output tile, K split), one per SM; M = 128
// sequences, N = the tile (128, the whole of a narrower matrix, or the key and head-weight matrices together: they share
// their activations, up to 160 columns), K in chunks of 64 through six shared-memory stages, all requested at once.
// A thread converts the 16 codes that it requested itself to bf16(code * block scale) (one rounding, 2^-9 relative; a
// 64-wide chunk of a 128-aligned tile lies inside ONE scale block), so a chunk takes one CTA barrier. The accumulator leaves
// as the f32 split partial: staged in the idle stages, one bulk copy (a CTA's partial rows are contiguous).
// Bound by what an SM takes in (192 KiB at 18 bytes a clock = 5.4 us at the 64-head model's sizes, activations being read by
// 32 tiles) and the launch's ramp. 128 sequences: 19 us with three stages, two barriers a chunk and 16-byte stores to 32 rows
// at a time, then 12.5 us for the epilogue below; 20.6 us together after that (31.8). The MMAs have a warp of their own: one of
// the converting warps issued them between two chunks, behind a CTA barrier, 18.4 us together for one sequence; 17.3 now, and
// 20 for 128 with cold weights.
// ---------------------------------------------------------------------------------------------
constexpr int FM_THREADS = 256;                             // warps 0-7 request, convert and store
constexpr int FM_LAUNCH = FM_THREADS + 32;                  // warp 8 issues the MMAs
constexpr int FM_NMAX = 160;                                // widest tile
constexpr int FM_NST = 6;                                   // stages of (activations 16 KiB | raw codes) in flight
constexpr int FM_STAGE = 16384 + FM_NMAX * 64;
constexpr int FM_BOFF = FM_NST * FM_STAGE;                  // two converted weight tiles (bf16) follow the stages
constexpr int FM_SMEM = FM_BOFF + 2 * FM_NMAX * 128;
static_assert(FM_BOFF % 1024 == 0 && FM_STAGE % 1024 == 0 && (FM_NMAX * 128) % 1024 == 0, "operand tiles are 1024-byte aligned");
static_assert(128 * FM_NMAX * 4 <= FM_BOFF, "the partial fits the stages");

__device__ __forceinline__ uint64_t fm_desc(uint32_t saddr) {     // K-major, 128-byte swizzle, 8-row groups 1024 B apart
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ void fm_mma(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ int g_front_err;

// (two CTAs' worth of registers, 96 a thread: nine warps leave one of the four register files three of them, beside which
// three of the epilogue's fit only up to here; 128 and 150 registers cost the epilogue its early start, 19.4 -> 21 us)
__global__ void __launch_bounds__(FM_LAUNCH, 2)
front_gemm_mma_kernel(FrontArgs A) {
    extern __shared__ __align__(1024) uint8_t fm_smem[];
    __shared__ uint64_t bar[2], full[2];   // MMAs of a converted tile done | its conversion done
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int jid = 0;
    while (jid < A.n_jobs - 1 && (int)blockIdx.x >= A.job[jid + 1].cta0) ++jid;
    const FrontJob& J = A.job[jid];
    const int local = blockIdx.x - J.cta0;
    const int tile = local % J.n_tiles, split = local / J.n_tiles;
    const int TN = J.tile_n, K = J.K, n0 = J.n_tiles > 1 ? TN : J.m[0].n;   // (columns of the tile from m[0])
    const int k0 = split * J.k_chunks * 64, nch = min(J.k_chunks, K / 64 - split * J.k_chunks);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { tc::mbar_init(&bar[i], 1); tc::mbar_init(&full[i], FM_THREADS); }
        tc::mbar_init_fence();
        abort_word = 0;
    }
    if (warp == 8) tc::tmem_alloc<256>(&tmem_slot);
    // (a prefetch into L2 may precede the wait, whoever writes)
    for (int e = tid; e < TN * ((nch * 64 + 127) / 128); e += FM_LAUNCH) {
        const int row = e % TN, line = e / TN;
        const uint8_t* w = row < n0 ? J.m[0].w + (size_t)(tile * TN + row) * K : J.m[1].w + (size_t)(row - n0) * K;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(w + k0 + line * 128));
    }
    rv_grid_dep_wait();
    // this thread's weight pieces: row e / 4, codes 16 (e % 4) .. + 15 of each chunk
    const uint8_t* pw[3];
    uint32_t dw[3];
    bool lw[3], second[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int e = tid + i * FM_THREADS, row = e >> 2, j = e & 3;
        lw[i] = row < TN && warp < 8;
        second[i] = row >= n0;
        const int r = lw[i] ? row : 0;
        pw[i] = (r < n0 ? J.m[0].w + (size_t)(tile * TN + r) * K : J.m[1].w + (size_t)(r - n0) * K) + k0 + j * 16;
        dw[i] = 16384 + row * 64 + j * 16;
    }
    const float* sc0 = J.m[0].scale + (size_t)(tile * TN / 128) * (K / 128);
    const float* sc1 = J.m[1].n ? J.m[1].scale : sc0;
    const uint32_t smem0 = tc::smem_u32(fm_smem);
    bool ok = true;
    int done[2] = {0, 0};                                   // commits issued per weight buffer so far
    uint32_t tmem = 0;
    // instruction descriptor: bf16 x bf16 -> f32, both K-major, M = 128, N = TN
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    for (int b0 = 0; b0 < A.B; b0 += 128) {                  // (after a wait that gave up too: the barriers stay matched)
        const uint16_t* pa[4]; uint32_t da[4]; uint32_t la[4];   // 4 activation pieces a thread; rows past B are zeros
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + i * FM_THREADS, row = e >> 3, j = e & 7;
            la[i] = b0 + row < A.B && warp < 8 ? 16u : 0u;
            pa[i] = J.x + (size_t)(la[i] ? b0 + row : 0) * K + k0 + j * 8;
            da[i] = tc::sw128_chunk(row, j);
        }
        auto request = [&](int c) {                          // one cp.async group per call, with or without a chunk
            if (c < nch) {
                const uint32_t st = smem0 + (c % FM_NST) * FM_STAGE;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (lw[i]) tc::cp_async16(st + dw[i], pw[i] + c * 64);
#pragma unroll
                for (int i = 0; i < 4; ++i) tc::cp_async16_zfill(st + da[i], pa[i] + c * 64, la[i]);
            }
            tc::cp_async_commit();
        };
        if (warp < 8)
#pragma unroll 1
            for (int c = 0; c < FM_NST; ++c) request(c);
        float s0 = sc0[k0 >> 7], s1 = sc1[k0 >> 7];
        if (b0 == 0) {
            tc::tc_fence_before();
            __syncthreads();
            tc::tc_fence_after();
            tmem = tmem_slot;
            // Behind the wait: the epilogue kernel may then read inputs of this call before its own. Behind the allocation, which
            // waits for its columns without a limit: a dependent could take them and then wait for this grid.
            rv_grid_dep_trigger();
        }
        if (warp == 8) {
            for (int c = 0; c < nch && ok; ++c) {
                const int wb = c & 1;
                ok = tc::mbar_wait_warp(&full[wb], done[wb]++ & 1, abort_flag, 85);
                if (!ok) break;
                tc::tc_fence_after();
                const uint64_t d_a = fm_desc(smem0 + (c % FM_NST) * FM_STAGE), d_b = fm_desc(smem0 + FM_BOFF + wb * FM_NMAX * 128);
                if (tc::elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) fm_mma(tmem, d_a + 2 * k, d_b + 2 * k, idesc, (c | k) ? 1u : 0u);   // +32 bytes = +2 in the address field
                    tc::mma_commit(&bar[wb]);
                }
                __syncwarp();
            }
            __syncthreads();
            if (b0 + 128 < A.B) __syncthreads();
            continue;
        }
        for (int c = 0; c < nch && ok; ++c) {
            const int wb = c & 1;
            // weight buffer wb and stage (c - 2) % 6 were read by the MMAs of chunk c - 2 (or of the batch tile before)
            if (done[wb] > 0) ok = tc::mbar_wait_warp(&bar[wb], (done[wb] - 1) & 1, abort_flag, 81);
            if (!ok) break;
            if (c >= 2) request(c - 2 + FM_NST);
            if (c == 0) tc::cp_async_wait<5>(); else tc::cp_async_wait<4>();   // this thread's part of chunk c has landed
            const float n0s = sc0[(k0 + min(c + 1, nch - 1) * 64) >> 7], n1s = sc1[(k0 + min(c + 1, nch - 1) * 64) >> 7];
            uint8_t* st = fm_smem + (c % FM_NST) * FM_STAGE;
            uint8_t* sB = fm_smem + FM_BOFF + wb * FM_NMAX * 128;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                if (lw[i]) {
                    const uint4 cw = *reinterpret_cast<const uint4*>(st + dw[i]);
                    const float sc = second[i] ? s1 : s0;
                    const uint32_t w4[4] = {cw.x, cw.y, cw.z, cw.w};
                    uint32_t o[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float2 f = rv_e4m3x2_to_f32x2((uint16_t)(w4[k >> 1] >> (16 * (k & 1))));
                        const __nv_bfloat162 h = __floats2bfloat162_rn(f.x * sc, f.y * sc);   // finite values: plain RNE
                        o[k] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    const int e = tid + i * FM_THREADS, row = e >> 2, j = e & 3;
                    *reinterpret_cast<uint4*>(sB + tc::sw128_chunk(row, 2 * j)) = make_uint4(o[0], o[1], o[2], o[3]);
                    *reinterpret_cast<uint4*>(sB + tc::sw128_chunk(row, 2 * j + 1)) = make_uint4(o[4], o[5], o[6], o[7]);
                }
            s0 = n0s; s1 = n1s;
            tc::fence_proxy_async();
            tc::mbar_arrive(&full[wb]);
            ++done[wb];
        }
        tc::cp_async_wait<0>();
        // all MMAs of this batch tile: wait for the last commit of each weight buffer
        for (int st = 0; st < 2 && ok; ++st)
            if (done[st] > 0) ok = tc::mbar_wait_warp(&bar[st], (done[st] - 1) & 1, abort_flag, 83 + st);
        tc::tc_fence_after();
        if (ok) {
            const int row = (warp & 3) * 32 + lane;
            for (int c = warp >> 2; c < TN / 16; c += 2) {   // 16-column chunks; warps 0-3 take the even ones, 4-7 the odd
                uint32_t r[16];
                tc::tmem_ld16(tmem + (((uint32_t)((warp & 3) * 32)) << 16) + c * 16, r);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    *reinterpret_cast<uint4*>(fm_smem + row * TN * 4 + (((c * 4 + e) ^ (row & J.mask)) << 4)) =
                        make_uint4(r[4 * e], r[4 * e + 1], r[4 * e + 2], r[4 * e + 3]);
            }
        }
        tc::fence_proxy_async();
        tc::tc_fence_before();
        __syncthreads();
        if (ok && tid == 0) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                         ::"l"(J.partial + (((size_t)split * J.n_tiles + tile) * A.B + b0) * TN), "r"(smem0), "r"(min(128, A.B - b0) * TN * 4) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
        if (b0 + 128 < A.B) __syncthreads();                 // the stages are free for the next batch tile
    }
    if (warp == 8) {
        tc::settle(abort_word);
        tc::tmem_dealloc<256>(tmem_slot);
    }
    if (tid == 0 && abort_word) atomicCAS(&g_front_err, 0, abort_word);
}

struct EpiPart {             // where the split partials of some outputs lie
    const float* p; int splits, n_tiles, tile_n, col0, mask;
    __device__ __forceinline__ const float* at(int s, int B, int b, int n) const {   // split s, output n (a float4 may be read where n % 4 == 0)
        n += col0;
        const int tile = n / tile_n, c = n - tile * tile_n;
        return p + (((size_t)s * n_tiles + tile) * B + b) * tile_n + ((((c >> 2) ^ (b & mask)) << 2) | (c & 3));
    }
};
struct EpiArgs {
    EpiPart k, q, w;
    const float* kn_w; const float* kn_b; const int32_t* pos;
    int B, nh, hd, rope_off, rope_seg; double theta; float eps;
    uint16_t* index_key; uint16_t* index_q; float* index_w;
};

// One CTA per sequence: reduce the split partials in split order, LayerNorm the key, rotate key and queries at the
// sequence's position, store bf16 (and the f32 head weights). Eight warps fold the queries, four the key and the weights meanwhile (a CTA of this size fits beside one of the GEMM's, so
// its f64 work is done before the GEMM ends). The rotation angles depend only on (position, pair index): rope_seg / 2 (cos, sin) pairs are computed once in
// f64, while the GEMM still runs.
constexpr int FE_Q = 256, FE_K = 128, FE_THREADS = FE_Q + FE_K;
__global__ void __launch_bounds__(FE_THREADS)
front_epilogue_kernel(EpiArgs A) {
    extern __shared__ __align__(16) float fe_smem[];          // (nh + 1) * hd values: queries then key
    __shared__ double s_red[2][FE_K / 32];
    __shared__ float s_cs[512], s_sn[512];
    const int b = blockIdx.x, t = threadIdx.x, nh = A.nh, hd = A.hd;
    float* kv = fe_smem + (size_t)nh * hd;
    rv_grid_dep_trigger();
    const int half = A.rope_seg / 2, pos = A.pos[b];
    for (int j = t; j < half; j += FE_THREADS) {
        const double ang = (double)pos * pow(A.theta, -2.0 * (double)j / (double)A.rope_seg);
        s_cs[j] = (float)cos(ang); s_sn[j] = (float)sin(ang);
    }
    rv_grid_dep_wait();
    if (t < FE_Q) {
        const int nq4 = nh * hd / 4;                 // index_dim is a multiple of 4 (checked by the launcher)
        for (int e0 = t; e0 < nq4; e0 += FE_Q * 2) {     // two elements x four splits of loads in flight per thread
            float4 a[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int s0 = 0; s0 < A.q.splits; s0 += 4) {
                float4 p[2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const int e = e0 + u * FE_Q;
                        p[u][s] = (e < nq4 && s0 + s < A.q.splits) ? *reinterpret_cast<const float4*>(A.q.at(s0 + s, A.B, b, e * 4))
                                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        if (s0 + s < A.q.splits) {            // split order; the guard keeps "+ 0" out of the fold
                            a[u].x = __fadd_rn(a[u].x, p[u][s].x); a[u].y = __fadd_rn(a[u].y, p[u][s].y);
                            a[u].z = __fadd_rn(a[u].z, p[u][s].z); a[u].w = __fadd_rn(a[u].w, p[u][s].w);
                        }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (e0 + u * FE_Q < nq4) *reinterpret_cast<float4*>(fe_smem + (e0 + u * FE_Q) * 4) = a[u];
        }
    } else {
        const int kt = t - FE_Q, lane = t & 31, kw = kt >> 5;
        auto fold = [&](const EpiPart& P, int n) {       // sixteen loads in flight, folded in split order
            float a = 0.0f;
            for (int s0 = 0; s0 < P.splits; s0 += 16) {
                float p[16];
#pragma unroll
                for (int s = 0; s < 16; ++s) p[s] = s0 + s < P.splits ? *P.at(s0 + s, A.B, b, n) : 0.0f;
#pragma unroll
                for (int s = 0; s < 16; ++s)
                    if (s0 + s < P.splits) a = __fadd_rn(a, p[s]);
            }
            return a;
        };
        double s1 = 0.0, s2 = 0.0;
        for (int e = kt; e < hd; e += FE_K) {
            const float a = fold(A.k, e);
            kv[e] = a;
            s1 += (double)a; s2 += (double)a * (double)a;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { s1 += __shfl_xor_sync(0xffffffffu, s1, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); }
        if (lane == 0) { s_red[0][kw] = s1; s_red[1][kw] = s2; }
        tc::named_barrier(1, FE_K);
        s1 = s2 = 0.0;
#pragma unroll
        for (int i = 0; i < FE_K / 32; ++i) { s1 += s_red[0][i]; s2 += s_red[1][i]; }
        const float mean = (float)(s1 / (double)hd);
        const float var = __fsub_rn((float)(s2 / (double)hd), __fmul_rn(mean, mean));
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(var, A.eps)));
        for (int e = kt; e < hd; e += FE_K)
            kv[e] = __fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(kv[e], mean), inv), A.kn_w[e]), A.kn_b[e]);
        for (int h = kt; h < nh; h += FE_K) A.index_w[(size_t)b * nh + h] = fold(A.w, h);
    }
    __syncthreads();
    // output i of a vector: rotated pairs inside [rope_off, rope_off + rope_seg), the value itself elsewhere
    auto value = [&](const float* v, int i) {
        const int r = i - A.rope_off;
        if (r < 0 || r >= A.rope_seg) return v[i];
        const int j = r < half ? r : r - half;
        const float a = v[A.rope_off + 2 * j], c = v[A.rope_off + 2 * j + 1];
        return r < half ? __fsub_rn(__fmul_rn(a, s_cs[j]), __fmul_rn(c, s_sn[j])) : __fadd_rn(__fmul_rn(c, s_cs[j]), __fmul_rn(a, s_sn[j]));
    };
    for (int p = t; p < (nh + 1) * (hd / 2); p += FE_THREADS) {
        const int vec = p / (hd / 2), i = 2 * (p - vec * (hd / 2));
        const float* v = fe_smem + (size_t)vec * hd;
        const uint16_t x = rv_f32_to_bf16(value(v, i)), y = rv_f32_to_bf16(value(v, i + 1));
        if (vec < nh) {
            *reinterpret_cast<uint32_t*>(A.index_q + ((size_t)b * nh + vec) * hd + i) = (uint32_t)x | ((uint32_t)y << 16);
        } else {
            A.index_key[(size_t)b * hd + i] = x;
            A.index_key[(size_t)b * hd + i + 1] = y;
        }
    }
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

}  // namespace

RIVOLI_API int rivoli_gemv_fp8(const float* x, const unsigned char* packed, const float* scale, int o_dim, int i_dim,
                               int block, int nrow, float* y) {
    if (o_dim <= 0 || i_dim <= 0 || block <= 0) return 1001;
    if (block & (block - 1)) return 1003;
    if (nrow != 1 && nrow != 2) return 1004;
    rv_drain_error();
    return launch_fold_gemv(FoldGemv{x, (size_t)i_dim, 0, packed, 0, 0, scale, rv_log2(block), ceil_div(i_dim, block), i_dim, o_dim,
                                     y, (size_t)o_dim, 0, 0, 0}, 1, nrow, 0);
}

// The reference switches to a split-K kernel for long rows (linalg.hip:296-321); here both names run the
// same fold, so their results are identical.
RIVOLI_API int rivoli_gemv_fp8_splitk(const float* x, const unsigned char* packed, const float* scale, int o_dim,
                                      int i_dim, int block, int nrow, float* y) {
    return rivoli_gemv_fp8(x, packed, scale, o_dim, i_dim, block, nrow, y);
}

RIVOLI_API int rivoli_layernorm(const float* x, const float* w, const float* b, int n, float eps, float* y) {
    if (n <= 0) return 1001;
    rv_drain_error();
    rv_launch_dependent(layernorm_kernel, dim3(1), dim3(256), 0, (cudaStream_t)0, x, w, b, n, eps, y);
    return rv_launch_status();
}

RIVOLI_API int rivoli_rope_interleave(float* base, int count, int stride, int seg, int pos, double theta) {
    if (count <= 0 || seg <= 0 || (seg & 1) || (seg / 2) > 1024) return 1001;
    if (count > 1 && stride < seg) return 1001;
    rv_drain_error();
    rv_launch_dependent(rope_interleave_kernel, dim3((unsigned)count), dim3((unsigned)(seg / 2)), 0, (cudaStream_t)0, base, stride, seg, pos, theta);
    return rv_launch_status();
}

// The tensor-core GEMM covers: 128-blocks, contraction lengths that are multiples of 128, output counts that
// are multiples of 128 (tiled) or of 16 up to 128 (one tile), 16-byte aligned rows.
static bool front_mma_ok(const IndexFrontGeom* g) {
    const int N[3] = {g->index_dim, g->index_heads * g->index_dim, g->index_heads};
    const int K[3] = {g->hidden, g->q_lora, g->hidden};
    if (g->block != 128) return false;
    for (int j = 0; j < 3; ++j) {
        if (K[j] % 128) return false;
        if (N[j] % 16 || (N[j] > 128 && N[j] % 128)) return false;
    }
    return true;
}

// The jobs of a call and the floats of their partials. Tensor cores: the key and head-weight matrices share their activations
// and take one tile where that is at most FM_NMAX wide; the split is the chunk count L with the shortest critical path, waves x
// (L + 4), a launch's ramp and a partial's way out counting as four chunks (a function of geometry and batch alone: it sizes the
// caller's scratch). CUDA cores: enough CTAs to fill the machine, at
// least 256 contraction values per split, at most 32 splits.
static void plan_jobs(const IndexFrontGeom* g, int B, bool mma, FrontArgs* fa, size_t* floats) {
    const int N[3] = {g->index_dim, g->index_heads * g->index_dim, g->index_heads};
    const int K[3] = {g->hidden, g->q_lora, g->hidden};
    const bool joint = mma && N[0] <= 128 && N[0] + N[2] <= FM_NMAX;
    fa->n_jobs = joint ? 2 : 3; fa->B = B; fa->block = g->block;
    for (int j = 0; j < fa->n_jobs; ++j) {
        FrontJob& J = fa->job[j];
        J.m[0].n = N[j]; J.m[1].n = joint && j == 0 ? N[2] : 0;
        J.N = J.m[0].n + J.m[1].n; J.K = K[j];
        J.tile_n = !mma ? FT_N : (J.N <= 128 || J.m[1].n ? J.N : 128);
        J.n_tiles = ceil_div(J.N, J.tile_n);
        J.mask = !mma ? 0 : (J.tile_n % 32 == 0 ? 7 : 3);
        int splits = ceil_div(296, J.n_tiles * 3);
        if (splits > K[j] / 256) splits = K[j] / 256;
        if (splits > 32) splits = 32;
        if (splits < 1) splits = 1;
        J.k_chunks = ceil_div(ceil_div(K[j], splits), 128) * 2;
    }
    if (mma) {
        long long best = -1;
        int pick = 2;
        for (int L = 2; L <= 64; ++L) {
            long long ctas = 0;
            for (int j = 0; j < fa->n_jobs; ++j) ctas += (long long)fa->job[j].n_tiles * ceil_div(fa->job[j].K / 64, L);
            const long long cost = (ctas + RV_SMS - 1) / RV_SMS * (L + 4);
            if (best < 0 || cost < best) { best = cost; pick = L; }
        }
        for (int j = 0; j < fa->n_jobs; ++j) fa->job[j].k_chunks = pick;
    }
    int cta = 0;
    size_t off = 0;
    for (int j = 0; j < fa->n_jobs; ++j) {
        FrontJob& J = fa->job[j];
        J.k_splits = ceil_div(ceil_div(J.K, 64), J.k_chunks);
        J.cta0 = cta;
        cta += J.n_tiles * J.k_splits;
        J.partial = reinterpret_cast<float*>(off);   // offset for now, rebased by the caller
        off += (size_t)J.k_splits * J.n_tiles * B * J.tile_n;
    }
    fa->n_cta = cta;
    *floats = off;
}

RIVOLI_API size_t rivoli_index_frontend_scratch_bytes(const IndexFrontGeom* g, int B) {
    if (!g || B <= 0) return 0;
    FrontArgs fa;
    size_t simt = 0, mma = 0;                        // a call may take either path
    plan_jobs(g, B, false, &fa, &simt);
    if (front_mma_ok(g)) plan_jobs(g, B, true, &fa, &mma);
    return (simt > mma ? simt : mma) * sizeof(float);
}

RIVOLI_API int rivoli_index_frontend_bf16(const IndexFrontGeom* g, const uint16_t* x, const uint16_t* q_resid,
                                          const int32_t* pos, int B, const unsigned char* wk, const float* wk_scale,
                                          const float* knorm_w, const float* knorm_b, const unsigned char* wq_b,
                                          const float* wq_b_scale, const unsigned char* wproj,
                                          const float* wproj_scale, uint16_t* index_key, uint16_t* index_q,
                                          float* index_w, void* scratch, int force_simt, void* stream) {
    if (!g || B <= 0 || !x || !q_resid || !pos || !wk || !wk_scale || !knorm_w || !knorm_b || !wq_b || !wq_b_scale ||
        !wproj || !wproj_scale || !index_key || !index_q || !index_w || !scratch)
        return 1001;
    if (g->hidden <= 0 || g->q_lora <= 0 || g->index_heads <= 0 || g->index_dim <= 0 || g->block <= 0) return 1001;
    if (g->block & (g->block - 1)) return 1003;
    if (g->rope_seg <= 0 || (g->rope_seg & 1) || g->rope_off < 0 || g->rope_off + g->rope_seg > g->index_dim) return 1002;
    if (g->index_heads > 256 || (size_t)(g->index_heads + 1) * g->index_dim * 4 > 200 * 1024) return 1002;
    if ((g->index_heads + 1) * (g->rope_seg / 2) > 8 * 256 || g->rope_seg > 1024 || (g->index_dim & 3)) return 1002;
    cudaStream_t st = (cudaStream_t)stream;
    const bool mma = !force_simt && front_mma_ok(g) && (((uintptr_t)x | (uintptr_t)q_resid | (uintptr_t)wk | (uintptr_t)wq_b |
                                                         (uintptr_t)wproj | (uintptr_t)scratch) & 15) == 0;
    FrontArgs fa;
    size_t floats = 0;
    plan_jobs(g, B, mma, &fa, &floats);
    float* base = static_cast<float*>(scratch);
    const uint16_t* xs[3] = {x, q_resid, x};
    const FrontMat mats[3] = {{wk, wk_scale, g->index_dim}, {wq_b, wq_b_scale, g->index_heads * g->index_dim}, {wproj, wproj_scale, g->index_heads}};
    for (int j = 0; j < fa.n_jobs; ++j) {
        fa.job[j].x = xs[j]; fa.job[j].m[0] = mats[j];
        if (fa.job[j].m[1].n) fa.job[j].m[1] = mats[2];
        fa.job[j].partial = base + reinterpret_cast<size_t>(fa.job[j].partial);
    }
    rv_drain_error();
    if (mma) {
        rv_allow_smem<front_gemm_mma_kernel>(FM_SMEM);
        rv_launch_dependent(front_gemm_mma_kernel, dim3((unsigned)fa.n_cta), dim3(FM_LAUNCH), (size_t)FM_SMEM, st, fa);
    } else {
        rv_launch_dependent(front_gemm_simt_kernel, dim3((unsigned)fa.n_cta), dim3(256), 0, st, fa);
    }
    if (int e = rv_launch_status()) return e;
    auto part = [&](int j, int col0) {
        const FrontJob& J = fa.job[j];
        return EpiPart{J.partial, J.k_splits, J.n_tiles, J.tile_n, col0, J.mask};
    };
    EpiArgs ea{part(0, 0), part(1, 0), fa.n_jobs == 3 ? part(2, 0) : part(0, g->index_dim), knorm_w, knorm_b, pos, B, g->index_heads,
               g->index_dim, g->rope_off, g->rope_seg, g->theta, g->eps, index_key, index_q, index_w};
    const size_t smem = (size_t)(g->index_heads + 1) * g->index_dim * sizeof(float);
    rv_allow_smem<front_epilogue_kernel>(200 * 1024);
    rv_launch_dependent(front_epilogue_kernel, dim3((unsigned)B), dim3(FE_THREADS), smem, st, ea);
    return rv_launch_status();
}

// Synchronises the stream; 1008 if a bounded wait of the tensor-core front end gave up since the last call.
RIVOLI_API int rivoli_index_frontend_status(void* stream) {
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return -(int)e;
    int h = 0;
    e = cudaMemcpyFromSymbol(&h, g_front_err, sizeof(int));
    if (e != cudaSuccess) return -(int)e;
    if (h) { const int z = 0; cudaMemcpyToSymbol(g_front_err, &z, sizeof(int)); }
    return h ? 1008 : 0;
}

