// The end of a decode whose CTAs merge their shares themselves: a cluster of CTAs serves one (batch, KV head) pair, each CTA a
// share of its tokens, and the shares meet in distributed shared memory instead of a partial buffer and a second launch.
// Every CTA stores its share into the shared memory of all (the stores travel while the cluster's barrier is on its way, and
// nothing is read from a neighbour afterwards, so one barrier is enough), merges all rows and applies its slice of V's
// rotation: 128 / cluster output dims.
#pragma once
#ifndef BGTQ_JIT
#include "bgtq_decode_params.cuh"
#endif

namespace bgtq {

// A CTA's shared memory may be written once that CTA runs: each says so as it starts, and who stores looks first.
__device__ __forceinline__ void cluster_started() { asm volatile("barrier.cluster.arrive.relaxed.aligned;"); }
__device__ __forceinline__ void cluster_all_started() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_cluster2(uint32_t addr, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_cluster4(uint32_t addr, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float exp2_approx(float x) {      // see fast_exp2
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint16_t f16_bits(float x) {
    unsigned short h;
    asm("cvt.rn.f16.f32 %0, %1;" : "=h"(h) : "f"(x));
    return h;
}

// This CTA's slice of V's rotation, [128][width], asynchronously into shared memory (behind the dependency wait: what is in
// front of the launch may have made the matrix).
__device__ __forceinline__ void merge_prefetch(const DecParams& P, uint8_t* smem, int h, int rank) {
    constexpr int kWidth = kHD / kClusterN, kPieces = kWidth / 4;      // 16-byte pieces of a row
    if (!P.m.v_rot) return;
    const int tid = threadIdx.x;
    const uint32_t to = smem_u32(smem + P.m.rot_off);
    const float* R = P.m.v_rot + (size_t)h * kHD * kHD + rank * kWidth;
    if ((reinterpret_cast<uintptr_t>(P.m.v_rot) & 15u) == 0) {
#pragma unroll
        for (int i = tid; i < kHD * kPieces; i += kDecThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * 16), "l"(R + (i / kPieces) * kHD + (i % kPieces) * 4) : "memory");
    } else {
#pragma unroll 1
        for (int i = tid; i < kHD * kWidth; i += kDecThreads)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + i * 4), "l"(R + (i / kWidth) * kHD + i % kWidth) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The sixteen warps' (O, m, l) of a CTA -> its share, sent to every CTA of the cluster.  One pass through shared memory: a
// warp with tokens leaves its sums as rows [query][128], thread (query, four dims) adds them up in warp order.  (The split
// form's tree of levels has a barrier per level and keeps the states in few registers, which a run of many tiles needs; here
// a CTA's share is a tile or two: the merge took 3200 cycles that way.)  16-byte chunk c of row q lies at c ^ (q / 2): the four
// lanes of a quad hold different rows of the same dims.  `buf`: kMergeRowsBytes of shared memory nobody else uses any more.
// `live`: warps that had tokens.  Called by all threads.
constexpr uint32_t kMergeRowsBytes = kDecWarps * (8 * kHD * 4 + 8 * 8);
__device__ __forceinline__ void merge_share(const DecParams& P, uint8_t* smem, uint8_t* buf, const float (&O)[8][4], float m0, float m1,
                                            float l0, float l1, int live, int rank) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, j = lane & 3;
    float2* const ml = reinterpret_cast<float2*>(buf + kDecWarps * 8 * kHD * 4);      // [warp][query]
    if (warp < live) {
        float4* const rows = reinterpret_cast<float4*>(buf) + warp * (8 * kHD / 4);
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (2 * j + e < P.gqa) {
                float4* const row = rows + (2 * j + e) * (kHD / 4);
#pragma unroll
                for (int i = 0; i < 8; i += 2) row[(4 * r + i / 2) ^ j] = make_float4(O[i][e], O[i][e + 2], O[i + 1][e], O[i + 1][e + 2]);
                if (r == 0) ml[warp * 8 + 2 * j + e] = e ? make_float2(m1, l1) : make_float2(m0, l0);
            }
    }
    __syncthreads();
    const int q = warp, c = lane;
    if (q >= P.gqa || q >= 8) return;
    // lane w looks at warp w's maximum and sum
    const float2 s = lane < live ? ml[lane * 8 + q] : make_float2(-BGTQ_INF, 0.f);
    float M = s.x;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    M = __shfl_sync(0xffffffffu, M, 0);         // (lanes 16 and up hold nothing)
    const float a = exp2_approx(s.x - (M == -BGTQ_INF ? 0.f : M));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4* row = reinterpret_cast<const float4*>(buf) + q * (kHD / 4) + (c ^ (q >> 1));
#pragma unroll 4
    for (int w = 0; w < live; ++w) {
        const float4 v = row[w * (8 * kHD / 4)];
        const float aw = __shfl_sync(0xffffffffu, a, w);
        acc.x = fmaf(v.x, aw, acc.x); acc.y = fmaf(v.y, aw, acc.y); acc.z = fmaf(v.z, aw, acc.z); acc.w = fmaf(v.w, aw, acc.w);
    }
    float L = s.y * a;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    L = __shfl_sync(0xffffffffu, L, 0);
    if (!(L > 0.f)) {       // no tokens, or a score that is no number: nothing, as the split form's partial of such a run
        M = -BGTQ_INF;
        L = 0.f;
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint32_t mine = smem_u32(smem + P.m.share_off + rank * kShareBytes);
#pragma unroll
    for (int k = 0; k < kClusterN; ++k) {
        const uint32_t to = cluster_addr(mine, k);
        st_cluster4(to + 4u * (q * kHD + 4 * c), acc);
        if (c == 0) st_cluster2(to + 8u * kHD * 4u + 8u * q, M, L);
    }
}

// A row's value and log-sum-exp with the other partial's, as the merge launch does it (launch_combine).
__device__ __forceinline__ void merge_other(float& y, float& lse, float other, float other_lse) {
    const float m = fmaxf(lse, other_lse);
    if (m > -BGTQ_INF) {
        const float wy = lse == -BGTQ_INF ? 0.f : expf(lse - m), wo = other_lse == -BGTQ_INF ? 0.f : expf(other_lse - m);
        y = (wy * y + wo * other) / (wy + wo);
        lse = m + logf(wy + wo);
    }
}

// merge_finish of shares that are all empty: this CTA's slice of the other partial, or zeros.
__device__ __forceinline__ void merge_none(const DecParams& P, int h, int b, int rank) {
    constexpr int kWidth = kHD / kClusterN;
    const MergeParams& F = P.m;
    for (int i = threadIdx.x; i < P.gqa * kWidth; i += kDecThreads) {
        const int q = i / kWidth, dim = rank * kWidth + i % kWidth, hq = h * P.gqa + q;
        const int64_t row = (int64_t)b * P.n_q + hq;
        float y = 0.f, lse = -BGTQ_INF;
        if (F.buf_o) merge_other(y, lse, F.buf_o[row * kHD + dim], F.buf_lse[row]);
        F.out[b * F.o_sb + hq * F.o_sh + dim] = f16_bits(y);
        if (F.out_f32) F.out_f32[row * kHD + dim] = y;
        if (F.lse_out && dim == 0) F.lse_out[row] = lse;
    }
}

// The cluster's shares -> this CTA's slice of the pair's output rows.  `buf`: shared memory that this CTA no longer uses (21 KB).
// Called by all threads of the cluster, their shares on their way.
__device__ __forceinline__ void merge_finish(const DecParams& P, uint8_t* smem, uint8_t* buf, int h, int b, int rank) {
    constexpr int kWidth = kHD / kClusterN, kParts = kDecThreads / kWidth, kPer = kHD / kParts;
    static_assert(!kMerges || (kPer % 4 == 0 && 8 * kWidth <= kDecThreads), "clusters of 2, 4 and 8");
    constexpr int kShare = kWidth < 32 ? 32 / kWidth : 1;       // parts in a warp
    constexpr int kSums = kParts / kShare;
    const MergeParams& F = P.m;
    const int tid = threadIdx.x;
    const int dl = tid % kWidth, pt = tid / kWidth;             // output dim of the slice, kPer rows of the rotation
    // this thread's value of the other partial, requested ahead
    const int64_t row0 = (int64_t)b * P.n_q + h * P.gqa;
    float bo = 0.f, bl = -BGTQ_INF;
    if (F.buf_o && tid < P.gqa * kWidth) {
        bo = F.buf_o[(row0 + tid / kWidth) * kHD + rank * kWidth + dl];
        bl = F.buf_lse[row0 + tid / kWidth];
    }
    if (F.v_rot) asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_sync();
    const uint8_t* shares = smem + F.share_off;
    float* const merged = reinterpret_cast<float*>(buf);
    float* const red = merged + 8 * kHD;        // [query][warp or part][dim of the slice]
    float* const lse = red + 8 * kDecThreads;
#pragma unroll 1
    for (int i = tid; i < P.gqa * kHD; i += kDecThreads) {
        const int q = i >> 7;
        float2 ml[kClusterN];
        float o[kClusterN];
#pragma unroll
        for (int c = 0; c < kClusterN; ++c) {
            ml[c] = *reinterpret_cast<const float2*>(shares + c * kShareBytes + 8 * kHD * 4 + q * 8);
            o[c] = *reinterpret_cast<const float*>(shares + c * kShareBytes + i * 4);
        }
        float M = ml[0].x;
#pragma unroll
        for (int c = 1; c < kClusterN; ++c) M = fmaxf(M, ml[c].x);
        const float Z = M == -BGTQ_INF ? 0.f : M;
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int c = 0; c < kClusterN; ++c) {
            const float wc = exp2_approx(ml[c].x - Z);
            den = fmaf(ml[c].y, wc, den);
            num = fmaf(o[c], wc, num);
        }
        merged[i] = den > 0.f ? num / den : 0.f;
        if ((i & 127) == 0) lse[q] = den > 0.f ? (M + log2f(den)) * 0.6931471805599453f : -BGTQ_INF;
    }
    __syncthreads();
    if (F.v_rot) {
        const float* rot = reinterpret_cast<const float*>(smem + F.rot_off) + pt * kPer * kWidth + dl;
        float r[kPer];
#pragma unroll
        for (int i = 0; i < kPer; ++i) r[i] = rot[i * kWidth];
        float* to = red + (pt / kShare) * kWidth + dl;
        const float* m = merged + pt * kPer;
#pragma unroll 2
        for (int g = 0; g < P.gqa; ++g, m += kHD, to += kSums * kWidth) {
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < kPer; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(m + i);
                acc = fmaf(v.x, r[i], acc); acc = fmaf(v.y, r[i + 1], acc); acc = fmaf(v.z, r[i + 2], acc); acc = fmaf(v.w, r[i + 3], acc);
            }
#pragma unroll
            for (int o = kWidth; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (pt % kShare == 0) *to = acc;
        }
        __syncthreads();
    }
    if (tid < P.gqa * kWidth) {
        const int q = tid / kWidth, dim = rank * kWidth + dl, hq = h * P.gqa + q;
        float y;
        if (F.v_rot) {
            const float* from = red + q * kSums * kWidth + dl;
            float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < kSums; ++s) s4[s & 3] += from[s * kWidth];
            y = (s4[0] + s4[1]) + (s4[2] + s4[3]);
        } else {
            y = merged[q * kHD + dim];
        }
        const int64_t row = row0 + q;
        float tot = lse[q];
        if (F.buf_o) merge_other(y, tot, bo, bl);
        F.out[b * F.o_sb + hq * F.o_sh + dim] = f16_bits(y);
        if (F.out_f32) F.out_f32[row * kHD + dim] = y;
        if (F.lse_out && dim == 0) F.lse_out[row] = tot;
    }
}

}  // namespace bgtq
