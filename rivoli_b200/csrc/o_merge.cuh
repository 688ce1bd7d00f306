// Merge of the attention kernels' splits inside a thread-block cluster: 64 heads x 512 dims of O^T per CTA, in tensor memory
// (lane = dim of a 128-dim block, column 64 c + h = block c of head h), held by eight warps (lane quarter warp % 4).
//
// Each CTA PUSHES its O^T, as it is, head by head into idle memory of the CTA that writes that head (CTA r: the heads
// [HZ r / n, HZ (r + 1) / n) of the cluster's HZ), and its reference maximum and weight sum of the head beside it; that CTA brings
// the n contributions to the common reference and the total sum while it adds them from its own memory. So nothing has to be
// exchanged before the push (maxima and sums first, and O^T scaled by its sender, cost two more barriers and 2 us), and remote
// stores need no answer. Distributed shared memory takes 21 bytes a clock, whatever the width of the stores; a CTA's own share
// does not go through it.
// A batch of a few sequences leaves SMs idle even so: then 64 / HZ clusters attend over the same rows, and each pushes and writes
// HZ of the heads (the push and the sums are what a small batch waits for: 5,500 + 2,000 of the 16,000 cycles behind the last
// score of one sequence; 32.9 -> 30.5 us a step).
// The loops are short: code that runs once per launch comes in from L2, at a tenth of the rate that it issues at.
#pragma once

#include "tc_common.cuh"

namespace om {

constexpr int H = 64, D = 512, MAX_N = 8;

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

struct Share {
    int n, split;          // CTAs of the cluster, this one's rank
    int lgz, hz, hz0;      // the cluster's heads: hz = 1 << lgz of them from hz0 on
    int hpc;               // most heads of a CTA
    int lo, heads;         // this CTA's: from the cluster's head lo on
    __device__ __forceinline__ Share(int n_, int split_, int shares, int z)
        : n(n_), split(split_), lgz(shares == 1 ? 6 : shares == 2 ? 5 : shares == 4 ? 4 : 3), hz(1 << lgz), hz0(z << lgz),
          hpc((hz + n - 1) / n), lo(split * hz / n), heads((split + 1) * hz / n - lo) {}
    __device__ __forceinline__ int owner(int i) const { return ((i + 1) * n - 1) >> lgz; }               // of the cluster's head i
    __device__ __forceinline__ int slot(int i, int o) const { return split * hpc + i - o * hz / n; }     // of this CTA's row of head i at its owner o
};
constexpr int recv_floats(int max_n) { return (H + max_n) * D; }                                     // [n][hpc][512]

__device__ __forceinline__ uint32_t map_rank(uint32_t smem, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(rank));
    return r;
}

// (maximum, sum) of head `head` to the CTA that writes it; ml = [n][hpc] there.
__device__ __forceinline__ void push_stats(const Share& S, float2* ml, int head, float2 v) {
    const int i = head - S.hz0;
    if (i < 0 || i >= S.hz) return;
    const int o = S.owner(i);
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(map_rank(tc::smem_u32(ml + S.slot(i, o)), o)), "f"(v.x), "f"(v.y) : "memory");
}

// This CTA's O^T rows of the cluster's heads, by the eight warps that hold them; recv = [n][hpc][512] at every owner.
__device__ __forceinline__ void push_rows(const Share& S, uint32_t tm_o, float* recv, bool live, int warp, int lane) {
    const int sq = warp & 3, th = warp >> 2, hz = S.hz;
    // a warp takes 32 heads: its th's half of them and all dims, or the half that holds the cluster's heads and th's half of the
    // dims; lane l: where this CTA's row of head win + l goes
    const int win = hz == H ? 32 * th : S.hz0 & 32;
    const int i = min(max(win + lane - S.hz0, 0), hz - 1), o = S.owner(i);
    const uint32_t own = tc::smem_u32(recv + S.slot(i, o) * D);
    const uint32_t remote = map_rank(own, o), to = o == S.split ? own : remote;   // (an address of this CTA's own window)
    const int c0 = hz == H ? 0 : 2 * th, c1 = hz == H ? 4 : c0 + 2;
#pragma unroll 1
    for (int c = c0; c < c1; ++c) {
        const uint32_t off = (uint32_t)(c * 128 + sq * 32 + lane) * 4u;
        uint32_t r[32];
        if (live) {
            tc::tmem_ld32(tm_o + (((uint32_t)(sq * 32)) << 16) + c * H + win, r);
            tc::tmem_ld_wait();
        } else {
#pragma unroll
            for (int h = 0; h < 32; ++h) r[h] = 0u;
        }
#pragma unroll
        for (int h8 = 0; h8 < 32; h8 += 8)
            if (win + h8 >= S.hz0 && win + h8 < S.hz0 + hz)
#pragma unroll
                for (int h = h8; h < h8 + 8; ++h) {   // lanes = consecutive dims: 128 bytes per warp store
                    const uint32_t d = __shfl_sync(0xffffffffu, to, h);
                    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(d + off), "r"(r[h]) : "memory");
                }
    }
}

// The weighted sums of this CTA's heads as bf16 rows; wts = [hpc][8], out = the sequence's [64][512].
__device__ __forceinline__ void write_rows(const Share& S, const float* recv, const float* wts, uint16_t* out, int tid, int n_threads) {
    const int hb = S.hz0 + S.lo, heads = S.heads, hpc = S.hpc, n = S.n;
#pragma unroll 1
    for (int e = tid; e < heads * (D / 4); e += n_threads) {
        const int hl = e / (D / 4), d4 = e % (D / 4);
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
        for (int q0 = 0; q0 < n; q0 += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(wts + hl * MAX_N + q0);
            const float w[4] = {w4.x, w4.y, w4.z, w4.w};
            float4 v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q0 + q < n) v[q] = *reinterpret_cast<const float4*>(recv + ((q0 + q) * hpc + hl) * D + d4 * 4);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q0 + q < n) {
                    acc.x = fmaf(v[q].x, w[q], acc.x); acc.y = fmaf(v[q].y, w[q], acc.y);
                    acc.z = fmaf(v[q].z, w[q], acc.z); acc.w = fmaf(v[q].w, w[q], acc.w);
                }
        }
        uint2 w;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w.x) : "f"(acc.y), "f"(acc.x));
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w.y) : "f"(acc.w), "f"(acc.z));
        *reinterpret_cast<uint2*>(out + (size_t)(hb + hl) * D + d4 * 4) = w;
    }
}

// Maximum or sum over the eight lanes of a head's group.
template <bool SUM>
__device__ __forceinline__ float fold8(float v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const float t = __shfl_xor_sync(0xffffffffu, v, o);
        v = SUM ? v + t : fmaxf(v, t);
    }
    return v;
}

// Clusters that share a sequence's heads, given n CTAs per sequence and room for `active` clusters of that size: a power of two of
// them, with eight heads or more and a head per CTA each.
inline int shares(int n, int n_seqs, int active) {
    int z = 1;
    while (n > 1 && z < 8 && H / (2 * z) >= n && 2 * z * n_seqs <= active) z *= 2;
    return z;
}

}  // namespace om
