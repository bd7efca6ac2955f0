// Launch parameters and helpers shared by the encoder kernels, and the launches that bgtq_step.cu puts together.
#pragma once
#include "bgtq_common.cuh"

namespace bgtq {

struct EncParams {
    const BgtqHeadDesc* desc;
    const float* rot_k;
    const float* rot_v;
    const __half* k;
    const __half* v;
    int64_t k_sb, k_sh, k_ss, v_sb, v_sh, v_ss;
    int32_t n_batch, n_kv, n_tok, t0;
    const int32_t* pos_dev;
    uint8_t* kp; int64_t kp_sb, kp_sh, kp_st; int32_t kp_row_bytes;
    void* kn; int64_t kn_sb, kn_sh, kn_st; int32_t kn_count;
    uint8_t* vp; int64_t vp_sb, vp_sh, vp_st;
    __half* vn; int64_t vn_sb, vn_sh, vn_st;
    uint8_t* k_codes;
    uint8_t* v_codes;
    int32_t flags;
    int32_t capacity;   // token slots per (batch, head) in the destination arrays, 0 = unknown
    int32_t* status;    // optional device word for kStatusOverflow
};

// With a device-side position the host cannot check the destination range: a launch whose rows would land
// outside [0, capacity) stores nothing and reports it.  Uniform over the launch (every thread sees the same slot).
__device__ __forceinline__ bool enc_range_ok(const EncParams& P, int t0, int n_tok) {
    if (P.capacity > 0 && (t0 < 0 || t0 + n_tok > P.capacity)) {
        if (P.status && threadIdx.x == 0) atomicExch(P.status, kStatusOverflow);
        return false;
    }
    return true;
}

// Tensor-core bulk path (bgtq_encode_tc.cu).  Rows must be 16-byte aligned.
int launch_encode_tc(const EncParams& P, cudaStream_t stream);

// tcgen05 bulk path (bgtq_encode_t5.cu): same requirements, n_tok >= 16.
int launch_encode_t5(const EncParams& P, cudaStream_t stream);

// Query rotation alone (the query items of the step-preparation kernel), optionally as a programmatic dependent.
int launch_rotate_q(const BgtqHeadDesc* desc, const float* rot_k, const void* q, int64_t q_sb, int64_t q_sh, void* q_rot,
                    int32_t n_batch, int32_t n_q, int32_t n_kv, bool programmatic, cudaStream_t stream);

// bgtq_decode with the plan's early fetch as it is or off for this launch; with `merge` (a plan of
// clusters) the merged rows come out of that launch and part_o and part_lse are null (bgtq_decode.cu).
struct MergeParams;
int launch_decode_plan(const BgtqDecodePlan* plan_host, const void* q_rot, const uint8_t* k_packed, int64_t kp_sb, int64_t kp_sh,
                       int64_t kp_st, const void* k_norms, int64_t kn_sb, int64_t kn_sh, int64_t kn_st, const uint8_t* v_packed,
                       int64_t vp_sb, int64_t vp_sh, int64_t vp_st, const void* v_norms, int64_t vn_sb, int64_t vn_sh, int64_t vn_st,
                       int32_t n_batch, int32_t n_q, int32_t n_kv, int32_t t_begin, int32_t t_end, int32_t n_splits, float scale,
                       float* part_o, float* part_lse, int32_t* status, const int32_t* pos_dev, int32_t pos_add, bool early_fetch,
                       const MergeParams* merge, void* stream);

}  // namespace bgtq
