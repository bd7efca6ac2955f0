// Launch parameters and shared-memory layout of the decode kernel (compiled ahead of time and at run time, see
// bgtq_decode_kernel.cuh).
#pragma once
#ifndef BGTQ_JIT
#include "bgtq_common.cuh"
#include "bgtq_plan.h"
#endif

namespace bgtq {

constexpr int kDecWarps = 16;
constexpr int kDecThreads = 32 * kDecWarps;
constexpr int kDecStages = 2;
constexpr int kMergeSlot = 9 * 32;   // float4 per warp in the end-of-run merge buffer: 8 of O and (m, l), per lane
// shared-memory layout (byte offsets from the start of dynamic shared memory)
// [barriers | query fragments | pad | lookup tables | stages (merge buffer at run end)]
// The lookup tables start at the first address past kOffMisc whose ABSOLUTE shared-window address is a
// multiple of kLutAlign (table bases are OR-ed into addresses); the stages follow at a fixed offset that
// leaves room for the worst-case pad.
constexpr uint32_t kOffQf = 1024, kOffMisc = kOffQf + kMaxSteps * 32 * 8;
constexpr uint32_t kOffStagesMin = kOffMisc + kLutAlign;     // + lut_bytes = P.stage_off
static_assert(kOffMisc % 128 == 0, "layout");
// two regions the tree merge alternates between: 8 slots (first level) and 4 (second); later levels fit in them
constexpr uint32_t kMergeBytes = (kDecWarps / 2 + kDecWarps / 4) * kMergeSlot * 16;
constexpr uint32_t kQuadBytes = 256u * 16u * 8u;      // V quad table of the specialised kernel
#define BGTQ_INF __int_as_float(0x7f800000)

// CTAs per (batch, KV head) pair of the form that merges a pair's shares itself (bgtq_decode_cluster.cuh): the cluster size.
// 0: the split form, whose partials a second launch merges (and all that is compiled ahead of time).
#ifdef BGTQ_JIT
constexpr int kCluster = BGTQ_JIT_CLUSTER;
#else
constexpr int kCluster = 0;
#endif
constexpr bool kMerges = kCluster > 0;
constexpr int kClusterN = kMerges ? kCluster : 1;
constexpr uint32_t kShareBytes = 8 * kHD * 4 + 8 * 8;       // a CTA's share of a pair: sums [8][128], (maximum, sum) [8]

// Where the merged rows go.
struct MergeParams {
    const float* v_rot;             // optional: R per KV head
    uint16_t* out;                  // fp16, element strides
    int64_t o_sb, o_sh;
    float* out_f32;                 // optional, (n_batch, n_q, 128)
    float* lse_out;                 // optional, (n_batch, n_q)
    const float* buf_o;             // optional: another partial of every row, (n_batch, n_q, 128) with its log-sum-exp
    const float* buf_lse;
    uint32_t share_off, rot_off;    // shared memory: the cluster's shares, the CTA's slice of the rotation
};

struct DecParams {
    const uint16_t* q_rot;  // fp16 bit patterns
    const uint8_t* kp;
    const uint8_t* kn;  // byte pointers; strides below are in bytes
    const uint8_t* vp;
    const uint8_t* vn;
    int64_t kp_sb, kp_sh, kn_sb, kn_sh, vp_sb, vp_sh, vn_sb, vn_sh;
    int32_t kp_st, kn_st, vp_st, vn_st;  // bytes per token
    int32_t n_batch, n_q, n_kv, gqa;
    int32_t t_begin, t_end, n_splits;
    const int32_t* pos_dev;
    int32_t pos_add;
    float scale_log2;
    float* part_o;
    float* part_lse;
    int32_t* status;
    uint32_t stage_off, stage_bytes, off_kn, off_v, off_vn;  // shared-memory layout
    MergeParams m;
    DecPlanDev plan;
};

}  // namespace bgtq
