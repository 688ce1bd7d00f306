// Matrix-vector products whose every output is ONE left fold in f32,
//     y[r][o] = ((..((0 + p_0) + p_1)..) + p_{K-1}),   p_i = (e4m3(W[o][i]) * scale[..]) * x[r][i],
// each operation rounded on its own (the reference's host arithmetic, bit for bit): rivoli_gemv_fp8 and
// rivoli_mla_value_fp8.
//
// The additions of one output depend on each other (4 cycles each: 6,144 of them take 13 us whatever else the chip
// does), so that chain is what bounds the kernel and everything else is kept off it. Eight warps load codes with the
// lanes along a row (128 contiguous bytes per warp load), decode, scale and multiply, and leave the products in shared
// memory; warp 0 does nothing but add, lane = output, four products per shared-memory load, while the others prepare
// the next CH columns. A CTA takes as many rows as leave one CTA per SM (at most one per lane of warp 0), so a matrix
// of few rows is spread over as many SMs as it has rows. Rows are padded by 16 bytes: the eight lanes of a 16-byte
// load phase fall in different banks.
// The weights are requested into L2 before the dependency wait of a programmatic dependent launch (a prefetch
// returns no data, so it cannot see an old value); everything is READ after it.
// One thread per output with byte loads took 636 us for 128 x 6,144 and 305 us for 4,096 x 2,048; this form takes
// 17.4 and 9.3 us (launches back to back, weights in L2).
#pragma once

#include "codec.cuh"
#include "common.cuh"

struct FoldGemv {
    const float* x; size_t x_row, x_head;                 // pitch between the R rows, between heads
    const uint8_t* w; size_t w_head_rows, w_off;          // head h owns weight rows [h * w_head_rows + w_off, + n_out)
    const float* scale; int bsh, sc_cols;                 // log2 of the scale block, scale columns
    int K, n_out;                                         // contraction length, outputs per head
    float* y; size_t y_row, y_head;
    int opc, blocks;                                      // outputs per CTA, CTAs per head
};

constexpr int FG_SLACK = 128;   // bytes past the last row that the adding warp may read ahead
constexpr int FG_LOADERS = 256;      // a multiple of every chunk's columns: a thread keeps its columns
// Warp 0 adds. With the wide chunk (one CTA per SM) warps 1-3, 5-7, 9 and 10 load, and 4 and 8 do nothing but keep the
// adding warp's scheduler free of other issue (128 x 6,144: 22.4 -> 17.4 us); with the narrow one several CTAs share an
// SM and warps 1-8 load.
__host__ __device__ constexpr int fg_threads(int ch) { return (ch == 512 ? 11 : 9) * 32; }

template <int R, int CH, bool VEC>
__global__ void __launch_bounds__(fg_threads(CH))
fold_gemv_kernel(FoldGemv a) {
    extern __shared__ __align__(16) float fg_smem[];      // 2 x [R * opc][CH + 4] products
    constexpr int LD = CH + 4;
    const int tid = threadIdx.x, head = blockIdx.x / a.blocks, o0 = (blockIdx.x - head * a.blocks) * a.opc;
    const int n = min(a.opc, a.n_out - o0), K = a.K;
    const size_t row0 = (size_t)head * a.w_head_rows + a.w_off + o0;
    const uint8_t* w = a.w + row0 * K;
    rv_grid_dep_trigger();
    {
        const size_t bytes = (size_t)n * K;
        for (size_t i = (size_t)tid * 128; i < bytes; i += (size_t)fg_threads(CH) * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(w + i));
    }
    rv_grid_dep_wait();
    const float* x = a.x + (size_t)head * a.x_head;
    const int nch = (K + CH - 1) / CH;
    const int buf_floats = R * a.opc * LD;

    // Products of columns [c * CH, ..) by the loader threads. A thread keeps its PER columns and walks the rows, ROWS
    // apart; the codes of a step are requested one step before they are used (load), behind the barrier of the step between.
    constexpr int PER = VEC ? 4 : 1, COLS = CH / PER, ROWS = FG_LOADERS / COLS, UN = 32 / ROWS;
    static_assert(FG_LOADERS % COLS == 0 && 32 % ROWS == 0, "a thread keeps its columns");
    const int warp = tid >> 5;
    const bool loader = CH == 512 ? (warp & 3) != 0 : warp > 0;
    const int lt = (CH == 512 ? warp - 1 - (warp >> 2) : warp - 1) * 32 + (tid & 31), col = (lt % COLS) * PER, ob = lt / COLS;
    uint32_t code[UN];
    float sc[UN], xv[R][PER];
    auto load = [&](int c) {
        const int i = c * CH + col;
        if (i >= K) return;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (VEC) *reinterpret_cast<float4*>(xv[r]) = *reinterpret_cast<const float4*>(x + r * a.x_row + i);
            else xv[r][0] = x[r * a.x_row + i];
        }
        const float* scol = a.scale + (i >> a.bsh);
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int o = ob + u * ROWS;
            if (o < n) {
                const uint8_t* p = w + (size_t)o * K + i;
                code[u] = VEC ? *reinterpret_cast<const uint32_t*>(p) : (uint32_t)*p;
                sc[u] = scol[((row0 + o) >> a.bsh) * a.sc_cols];
            }
        }
    };
    auto store = [&](int c) {
        if (c * CH + col >= K) return;
        float* dst = fg_smem + (c & 1) * buf_floats + col;
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int o = ob + u * ROWS;
            if (o < n) {
                float f[4];
                const float2 lo = rv_e4m3x2_to_f32x2((uint16_t)code[u]);
                f[0] = lo.x; f[1] = lo.y;
                if (VEC) { const float2 hi = rv_e4m3x2_to_f32x2((uint16_t)(code[u] >> 16)); f[2] = hi.x; f[3] = hi.y; }
#pragma unroll
                for (int e = 0; e < PER; ++e) f[e] = __fmul_rn(f[e], sc[u]);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float* d = dst + (r * a.opc + o) * LD;
                    if (VEC)
                        *reinterpret_cast<float4*>(d) = make_float4(__fmul_rn(f[0], xv[r][0]), __fmul_rn(f[1], xv[r][VEC ? 1 : 0]),
                                                                    __fmul_rn(f[2], xv[r][VEC ? 2 : 0]), __fmul_rn(f[3], xv[r][VEC ? 3 : 0]));
                    else d[0] = __fmul_rn(f[0], xv[r][0]);
                }
            }
        }
    };

    if (loader) {
        load(0);
        store(0);
        if (nch > 1) load(1);
    }
    __syncthreads();
    float acc = 0.0f;
    const int r = R == 1 ? 0 : tid / a.opc, o = R == 1 ? tid : tid - r * a.opc;   // this lane's output (warp 0)
    const bool mine = tid < 32 && r < R && o < n;
    auto add4 = [&](const float4& v) {
        acc = __fadd_rn(acc, v.x); acc = __fadd_rn(acc, v.y); acc = __fadd_rn(acc, v.z); acc = __fadd_rn(acc, v.w);
    };
    for (int c = 0; c < nch; ++c) {
        if (loader) {
            if (c + 1 < nch) store(c + 1);
            if (c + 2 < nch) load(c + 2);
        } else if (mine) {
            // eight 16-byte loads are on their way while eight are added; a load past the row's end stays inside the
            // allocation (FG_SLACK) and is not added
            const float4* p = reinterpret_cast<const float4*>(fg_smem + (c & 1) * buf_floats + (r * a.opc + o) * LD);
            const int kn = min(CH, K - c * CH), n4 = kn >> 2;
            float4 v[8], u[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = p[j];
            int i = 0;
            for (; i + 16 <= n4; i += 16) {
#pragma unroll
                for (int j = 0; j < 8; ++j) u[j] = p[i + 8 + j];
#pragma unroll
                for (int j = 0; j < 8; ++j) add4(v[j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = p[i + 16 + j];
#pragma unroll
                for (int j = 0; j < 8; ++j) add4(u[j]);
            }
            for (; i < n4; ++i) add4(p[i]);
            for (int e = i * 4; e < kn; ++e) acc = __fadd_rn(acc, reinterpret_cast<const float*>(p)[e]);
        }
        __syncthreads();
    }
    if (mine) a.y[r * a.y_row + head * a.y_head + o0 + o] = acc;
}

// Rows per CTA: one CTA per SM where the matrix has that many rows, at most 32 / R (the lanes of the adding warp).
// CH: 512 columns per step keep the barrier to 2 % of a long chain; contractions of at most 1,024 take 128 (34 KB of
// shared memory at 32 rows: several CTAs per SM, and the first addition starts early).
static inline int launch_fold_gemv(FoldGemv a, int heads, int R, cudaStream_t st) {
    const int total = heads * a.n_out, most = 32 / R;
    const int sms = rv_sm_count();
    a.opc = (total + sms - 1) / sms;
    if (a.opc > most) a.opc = most;
    if (a.opc > a.n_out) a.opc = a.n_out;
    a.blocks = (a.n_out + a.opc - 1) / a.opc;
    const bool vec = a.K % 4 == 0 && a.bsh >= 2 && (((uintptr_t)a.w & 3) == 0) && (((uintptr_t)a.x & 15) == 0) &&
                     a.x_row % 4 == 0 && a.x_head % 4 == 0;
    const int ch = vec && a.K > 1024 ? 512 : 128;
    const size_t smem = (size_t)2 * R * a.opc * (ch + 4) * sizeof(float) + FG_SLACK;
    const dim3 grid((unsigned)(heads * a.blocks));
#define RV_FG(RR, CC, VV)                                                                                                  \
    do {                                                                                                                   \
        rv_allow_smem<fold_gemv_kernel<RR, CC, VV>>(2 * 32 * (CC + 4) * 4 + FG_SLACK);                                                \
        rv_launch_dependent(fold_gemv_kernel<RR, CC, VV>, grid, dim3(fg_threads(CC)), smem, st, a);                            \
    } while (0)
#define RV_FG2(RR)                                                                                                         \
    do {                                                                                                                   \
        if (ch == 512) RV_FG(RR, 512, true);                                      \
        else if (vec) RV_FG(RR, 128, true);                                                                                \
        else RV_FG(RR, 128, false);                                                                                        \
    } while (0)
    if (R == 2) RV_FG2(2); else RV_FG2(1);
#undef RV_FG2
#undef RV_FG
    return rv_launch_status();
}
