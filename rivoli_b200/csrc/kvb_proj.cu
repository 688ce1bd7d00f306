// The two contractions through kv_b either side of MLA attention.
//
//   rivoli_mla_absorb_fp8 / rivoli_mla_value_fp8 : the reference's single-token f32 operators
//       (crates/backend/kernels/mla.hip:12-231): same symbols, arguments, guard codes. The
//       reference's fold order (d, resp. i, ascending; q * (e4m3 * scale)), no
//       contraction - bit-identical to the host references of its tests
//       (crates/engine/tests/kernel_attend.rs:361-390).
//   rivoli_mla_absorb_batched_bf16 / rivoli_mla_value_batched_bf16 : the batched decode form
//       (bf16 activations [B][H][..]); CUDA-core kernels here for any geometry, tensor-core
//       kernels in kvb_proj_mma.cu for the model geometry.
//
// kv_b: e4m3 codes [H*(nope+vh) rows][kvl cols], scale[(row / block) * ceil(kvl/block) + col / block].
#include "codec.cuh"
#include "common.cuh"
#include "fold_gemv.cuh"
#include "tc_common.cuh"

namespace {

// One output column per pair of lanes' 16-bit word: thread t owns the columns 2t, 2t + 1 of the CTA's 128, for R query
// rows, and folds over d. What bounds it: 6.3 MB of codes (1 us) and a chain of nope additions; the codes of up to
// AB_DCH rows are requested at once (16-byte copies into shared memory, 24 KB of the CTA's 128 columns) so that the
// chain never waits for memory. 64 threads per 128 columns keep every scheduler of 148 SMs busy with 64 heads x 4
// blocks. One thread per column with byte loads from global memory took 81 us at 64 x 512 x 192; this takes 5.1.
constexpr int AB_COLS = 128, AB_THREADS = 64, AB_DCH = 192;

template <int R, bool VEC>
__global__ void __launch_bounds__(AB_THREADS)
absorb_f32_kernel(const float* __restrict__ q, const uint8_t* __restrict__ kvb, const float* __restrict__ scale, int H,
                  int qh, int nope, int vh, int kvl, int block, float* __restrict__ qabs) {
    __shared__ __align__(16) uint8_t codes[AB_DCH][AB_COLS];
    __shared__ float qs[R][AB_DCH];
    const int tid = threadIdx.x, head = blockIdx.y, c0 = blockIdx.x * AB_COLS, i = c0 + 2 * tid;
    const int bsh = rv_log2(block), sc_cols = (kvl + block - 1) / block;
    const size_t rbase = (size_t)head * (nope + vh);
    const int cols = min(AB_COLS, kvl - c0);
    rv_grid_dep_trigger();
    for (int d = tid; d < nope; d += AB_THREADS)              // (a prefetch returns no data: safe before the wait)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(kvb + (rbase + d) * kvl + c0));
    rv_grid_dep_wait();
    float acc[R][2];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = 0.0f;
    for (int d0 = 0; d0 < nope; d0 += AB_DCH) {
        const int dn = min(AB_DCH, nope - d0);
        __syncthreads();
        if (VEC) {
            for (int e = tid; e < dn * (AB_COLS / 16); e += AB_THREADS) {
                const int d = e >> 3, c = (e & 7) * 16;
                if (c < cols) tc::cp_async16(tc::smem_u32(&codes[d][c]), kvb + (rbase + d0 + d) * kvl + c0 + c);
            }
            tc::cp_async_commit();
        } else {
            for (int e = tid; e < dn * AB_COLS; e += AB_THREADS) {
                const int d = e >> 7, c = e & 127;
                if (c < cols) codes[d][c] = kvb[(rbase + d0 + d) * kvl + c0 + c];
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            for (int d = tid; d < dn; d += AB_THREADS) qs[r][d] = q[(size_t)r * H * qh + (size_t)head * qh + d0 + d];
        if (VEC) tc::cp_async_wait<0>();
        __syncthreads();
        if (2 * tid >= cols) continue;
        for (int d = 0; d < dn;) {
            // rows up to the next scale block share their scales
            const size_t row = rbase + d0 + d;
            const int stop = min(dn, d + (int)(block - (row & (size_t)(block - 1))));
            const float* srow = scale + (row >> bsh) * sc_cols;
            const float s0 = srow[i >> bsh], s1 = i + 1 < kvl ? srow[(i + 1) >> bsh] : 0.0f;
#pragma unroll 8
            for (; d < stop; ++d) {
                const float2 f = rv_e4m3x2_to_f32x2(*reinterpret_cast<const uint16_t*>(&codes[d][2 * tid]));
                const float w0 = __fmul_rn(f.x, s0), w1 = __fmul_rn(f.y, s1);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    acc[r][0] = __fadd_rn(acc[r][0], __fmul_rn(qs[r][d], w0));
                    acc[r][1] = __fadd_rn(acc[r][1], __fmul_rn(qs[r][d], w1));
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (i + e < kvl) qabs[((size_t)r * H + head) * kvl + i + e] = acc[r][e];
}

// Batched bf16, any geometry: one thread per (sequence, head, output), the same folds.
__global__ void __launch_bounds__(256)
absorb_batched_simt_kernel(const uint16_t* __restrict__ q, const uint8_t* __restrict__ kvb,
                           const float* __restrict__ scale, int H, int qh, int nope, int vh, int kvl, int rope,
                           int block, int B, uint16_t* __restrict__ q_abs) {
    const int W = kvl + rope;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)B * H * W) return;
    const int i = (int)(idx % W);
    const size_t bh = idx / W;
    const int head = (int)(bh % H);
    const uint16_t* qr = q + bh * qh;
    if (i >= kvl) { q_abs[idx] = qr[nope + (i - kvl)]; return; }   // the rope segment rides along, bit for bit
    const int bsh = rv_log2(block), sc_cols = (kvl + block - 1) / block;
    const size_t rbase = (size_t)head * (nope + vh);
    float acc = 0.0f;
    for (int d = 0; d < nope; ++d) {
        const size_t row = rbase + d;
        const float ws = __fmul_rn(rv_e4m3_to_f32(kvb[row * kvl + i]), scale[(row >> bsh) * sc_cols + (i >> bsh)]);
        acc = __fadd_rn(acc, __fmul_rn(rv_bf16_to_f32(qr[d]), ws));
    }
    q_abs[idx] = rv_f32_to_bf16(acc);
}

__global__ void __launch_bounds__(256)
value_batched_simt_kernel(const uint16_t* __restrict__ clat, const uint8_t* __restrict__ kvb,
                          const float* __restrict__ scale, int H, int nope, int vh, int kvl, int block, int B,
                          uint16_t* __restrict__ ctx) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)B * H * vh) return;
    const int j = (int)(idx % vh);
    const size_t bh = idx / vh;
    const int head = (int)(bh % H);
    const int bsh = rv_log2(block), sc_cols = (kvl + block - 1) / block;
    const size_t row = (size_t)head * (nope + vh) + nope + j;
    const uint8_t* w = kvb + row * kvl;
    const float* srow = scale + (row >> bsh) * sc_cols;
    const uint16_t* cr = clat + bh * kvl;
    float acc = 0.0f;
    for (int i = 0; i < kvl; ++i)
        acc = __fadd_rn(acc, __fmul_rn(rv_bf16_to_f32(cr[i]), __fmul_rn(rv_e4m3_to_f32(w[i]), srow[i >> bsh])));
    ctx[idx] = rv_f32_to_bf16(acc);
}

int guard_dims(int H, int qh, int nope, int vh, int kvl, int block) {
    if (H <= 0 || qh <= 0 || nope <= 0 || vh <= 0 || kvl <= 0 || block <= 0) return 1001;
    if (block & (block - 1)) return 1003;   // the block index is a shift
    return 0;
}

}  // namespace

RIVOLI_API int rivoli_mla_absorb_fp8(const float* q, const unsigned char* kvb, const float* kvb_scale, int H, int qh,
                                     int nope, int vh, int kvl, int block, int nrow, float* qabs) {
    if (int e = guard_dims(H, qh, nope, vh, kvl, block)) return e;
    if (nrow != 1 && nrow != 2) return 1004;
    const dim3 grid((unsigned)((kvl + AB_COLS - 1) / AB_COLS), (unsigned)H);
    const bool vec = kvl % 16 == 0 && ((uintptr_t)kvb & 15) == 0;
    rv_drain_error();
#define RV_AB(RR, VV)                                                                                                     \
    rv_launch_dependent(absorb_f32_kernel<RR, VV>, grid, dim3(AB_THREADS), 0, (cudaStream_t)0, q, kvb, kvb_scale, H, qh,  \
                        nope, vh, kvl, block, qabs)
    if (nrow == 2) { if (vec) RV_AB(2, true); else RV_AB(2, false); }
    else { if (vec) RV_AB(1, true); else RV_AB(1, false); }
#undef RV_AB
    return rv_launch_status();
}

RIVOLI_API int rivoli_mla_value_fp8(const float* clat, const unsigned char* kvb, const float* kvb_scale, int H,
                                    int nope, int vh, int kvl, int block, int nrow, float* ctx) {
    if (int e = guard_dims(H, 1, nope, vh, kvl, block)) return e;
    if (nrow != 1 && nrow != 2) return 1004;
    if (kvl & 3) return 1002;   // the reference's value kernel loads weights as words (mla.hip:216-225)
    rv_drain_error();
    return launch_fold_gemv(FoldGemv{clat, (size_t)H * kvl, (size_t)kvl, kvb, (size_t)(nope + vh), (size_t)nope, kvb_scale, rv_log2(block),
                                     (kvl + block - 1) / block, kvl, vh, ctx, (size_t)H * vh, (size_t)vh, 0, 0}, H, nrow, 0);
}

// Defined in kvb_proj_mma.cu: 0 if the geometry is outside the tensor-core kernels.
extern "C" int rivoli_kvb_mma_supported(int H, int qh, int nope, int vh, int kvl, int rope, int block);
extern "C" int rivoli_kvb_absorb_mma(const uint16_t* q, const uint8_t* kvb, const float* scale, int H, int qh, int nope,
                                     int vh, int kvl, int rope, int block, int B, uint16_t* q_abs, cudaStream_t st);
extern "C" int rivoli_kvb_value_mma(const uint16_t* clat, const uint8_t* kvb, const float* scale, int H, int nope, int vh,
                                    int kvl, int block, int B, uint16_t* ctx, cudaStream_t st);

RIVOLI_API int rivoli_mla_absorb_batched_bf16(const uint16_t* q, const unsigned char* kvb, const float* kvb_scale, int H,
                                              int qh, int nope, int vh, int kvl, int rope, int block, int B,
                                              uint16_t* q_abs, int force_simt, void* stream) {
    if (int e = guard_dims(H, qh, nope, vh, kvl, block)) return e;
    if (B <= 0 || rope < 0 || !q || !kvb || !kvb_scale || !q_abs) return 1001;
    if (nope + rope > qh) return 1002;
    cudaStream_t st = (cudaStream_t)stream;
    if (!force_simt && rivoli_kvb_mma_supported(H, qh, nope, vh, kvl, rope, block)) {
        if (((uintptr_t)q | (uintptr_t)kvb | (uintptr_t)q_abs) & 15) return 1005;
        return rivoli_kvb_absorb_mma(q, kvb, kvb_scale, H, qh, nope, vh, kvl, rope, block, B, q_abs, st);
    }
    const size_t total = (size_t)B * H * (kvl + rope);
    rv_drain_error();
    absorb_batched_simt_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(q, kvb, kvb_scale, H, qh, nope, vh, kvl,
                                                                                rope, block, B, q_abs);
    return rv_launch_status();
}

RIVOLI_API int rivoli_mla_value_batched_bf16(const uint16_t* clat, const unsigned char* kvb, const float* kvb_scale,
                                             int H, int nope, int vh, int kvl, int block, int B, uint16_t* ctx,
                                             int force_simt, void* stream) {
    if (int e = guard_dims(H, 1, nope, vh, kvl, block)) return e;
    if (B <= 0 || !clat || !kvb || !kvb_scale || !ctx) return 1001;
    cudaStream_t st = (cudaStream_t)stream;
    if (!force_simt && rivoli_kvb_mma_supported(H, nope, nope, vh, kvl, 0, block)) {
        if (((uintptr_t)clat | (uintptr_t)kvb | (uintptr_t)ctx) & 15) return 1005;
        return rivoli_kvb_value_mma(clat, kvb, kvb_scale, H, nope, vh, kvl, block, B, ctx, st);
    }
    const size_t total = (size_t)B * H * vh;
    rv_drain_error();
    value_batched_simt_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(clat, kvb, kvb_scale, H, nope, vh, kvl,
                                                                               block, B, ctx);
    return rv_launch_status();
}
