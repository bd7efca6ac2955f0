// One call for the launches of a layer's decode step, and one for those of an attention over cached tokens.
//
// A decode step of a short sequence is bounded by the host: the two or three (one more with fp16 regions) launches of a
// layer take the GPU 9 to 15 us, and passing their forty-odd arguments one launch at a time, or staging the step's inputs
// for a captured graph (three copies and a graph launch per layer), took the host 36 us.  Everything that does not
// change from step to step is filled in once (BgtqLayerStep); a step then costs one call, and the kernels read the
// caller's query, key and value rows where they lie.
#include "bgtq_common.cuh"
#include "bgtq_decode_params.cuh"
#include "bgtq_encode_params.cuh"

using namespace bgtq;

// The query rows of (n_batch, n_q) heads lie one behind the other; the stride of a dim of one element says nothing.
static bool contiguous_rows(int32_t n_batch, int32_t n_q, int64_t q_sb, int64_t q_sh) {
    return (n_q == 1 || q_sh == kHD) && (n_batch == 1 || q_sb == (int64_t)n_q * kHD);
}

extern "C" __attribute__((visibility("default"))) int bgtq_layer_step_size(void) { return (int)sizeof(BgtqLayerStep); }

extern "C" __attribute__((visibility("default"))) int bgtq_layer_step(
    const BgtqLayerStep* s, const void* q, int64_t q_sb, int64_t q_sh, const void* k, int64_t k_sb, int64_t k_sh,
    const void* v, int64_t v_sb, int64_t v_sh, const void* rope_cos, const void* rope_sin, int64_t rope_sb, void* stream) {
    if (!s || !q || !k || !v || !s->pos_dev) return BGTQ_E_BADARG;
    const bool ring = s->k_buf != nullptr;
    if (ring && rope_cos) return BGTQ_E_UNSUPPORTED;
    const void* q_dec = s->q_rot;
    const bool rotate = !(s->flags & BGTQ_STEP_Q_ROTATED);
    if (!rotate) {      // the queries arrive in the packed-K basis: the decode reads them where they are
        if (!contiguous_rows(s->n_batch, s->n_q, q_sb, q_sh)) return BGTQ_E_UNSUPPORTED;
        q_dec = q;
    }
    int rc;
    if (ring)
        rc = bgtq_step_prepare_ring(s->desc, s->rot_k, s->rot_v, rotate ? q : nullptr, q_sb, q_sh, s->q_rot, s->n_q, k, k_sb, k_sh, v,
                                    v_sb, v_sh, s->n_batch, s->n_kv, 0, s->k_packed, s->kp_sb, s->kp_sh, s->kp_st, s->kp_row_bytes,
                                    s->k_norms, s->kn_sb, s->kn_sh, s->kn_st, s->kn_count, s->v_packed, s->vp_sb, s->vp_sh, s->vp_st,
                                    s->v_norms, s->vn_sb, s->vn_sh, s->vn_st, s->enc_flags, s->pos_dev, s->t_capacity, s->status,
                                    s->k_buf, s->v_buf, s->kb_sb, s->kb_sh, s->n_sink, s->window, stream);
    else if (rope_cos)
        rc = bgtq_step_prepare_rope(s->desc, s->rot_k, s->rot_v, rotate ? q : nullptr, q_sb, q_sh, s->q_rot, s->n_q, k, k_sb, k_sh, v,
                                    v_sb, v_sh, s->n_batch, s->n_kv, 0, s->k_packed, s->kp_sb, s->kp_sh, s->kp_st, s->kp_row_bytes,
                                    s->k_norms, s->kn_sb, s->kn_sh, s->kn_st, s->kn_count, s->v_packed, s->vp_sb, s->vp_sh, s->vp_st,
                                    s->v_norms, s->vn_sb, s->vn_sh, s->vn_st, s->enc_flags, s->pos_dev, s->t_capacity, s->status,
                                    rope_cos, rope_sin, rope_sb, stream);
    else
        rc = bgtq_step_prepare(s->desc, s->rot_k, s->rot_v, rotate ? q : nullptr, q_sb, q_sh, s->q_rot, s->n_q, k, k_sb, k_sh, v, v_sb,
                               v_sh, s->n_batch, s->n_kv, 0, s->k_packed, s->kp_sb, s->kp_sh, s->kp_st, s->kp_row_bytes, s->k_norms,
                               s->kn_sb, s->kn_sh, s->kn_st, s->kn_count, s->v_packed, s->vp_sb, s->vp_sh, s->vp_st, s->v_norms,
                               s->vn_sb, s->vn_sh, s->vn_st, s->enc_flags, s->pos_dev, s->t_capacity, s->status, stream);
    if (rc != BGTQ_OK) return rc;
    auto regions = [&]() {      // the fp16 sink and window
        return bgtq_buffer_attn_pos(q, q_sb, q_sh, s->k_buf, s->v_buf, s->kb_sb, s->kb_sh, 0, 0, s->n_sink, 0, s->window + 1, s->n_batch,
                                    s->n_q, s->n_kv, s->scale, s->buf_o, s->buf_lse, s->pos_dev, stream);
    };
    bool regions_done = false;
    if (bgtq_decode_plan_cluster(s->plan)) {
        if (ring) {     // its partial comes first here: the decode merges it too.  (The decode's early fetch stays sound: the append
                        // lets its dependents start behind its own wait, and so this one the decode.)
            rc = regions();
            if (rc != BGTQ_OK) return rc;
            regions_done = true;
        }
        const MergeParams M = {s->v_rot, static_cast<uint16_t*>(s->out), s->o_sb, s->o_sh, nullptr, nullptr, ring ? s->buf_o : nullptr,
                               ring ? s->buf_lse : nullptr, 0, 0};
        rc = launch_decode_plan(s->plan, q_dec, s->k_packed, s->kp_sb, s->kp_sh, s->kp_st, s->k_norms, s->kn_sb, s->kn_sh, s->kn_st,
                                s->v_packed, s->vp_sb, s->vp_sh, s->vp_st, s->v_norms, s->vn_sb, s->vn_sh, s->vn_st, s->n_batch, s->n_q,
                                s->n_kv, 0, s->t_capacity, s->n_splits, s->scale, nullptr, nullptr, s->status, s->pos_dev, s->pos_add, true, &M,
                                stream);
        if (rc != BGTQ_E_UNSUPPORTED) return rc;
    }
    rc = bgtq_decode(s->plan, s->desc, q_dec, s->k_packed, s->kp_sb, s->kp_sh, s->kp_st, s->k_norms, s->kn_sb, s->kn_sh, s->kn_st,
                     s->v_packed, s->vp_sb, s->vp_sh, s->vp_st, s->v_norms, s->vn_sb, s->vn_sh, s->vn_st, s->n_batch, s->n_q, s->n_kv,
                     0, s->t_capacity, s->n_splits, s->scale, s->part_o, s->part_lse, s->status, s->pos_dev, s->pos_add, stream);
    if (rc != BGTQ_OK) return rc;
    if (ring && !regions_done) {
        rc = regions();
        if (rc != BGTQ_OK) return rc;
    }
    return bgtq_combine(s->part_o, s->part_lse, s->n_splits, s->v_rot, ring ? s->buf_o : nullptr, ring ? s->buf_lse : nullptr,
                        s->n_batch, s->n_q, s->n_kv, s->out, s->o_sb, s->o_sh, nullptr, nullptr, s->combine_flags, stream);
}

extern "C" __attribute__((visibility("default"))) int bgtq_layer_encode(const BgtqLayerStep* s, const void* k, int64_t k_sb, int64_t k_sh,
                                                                        int64_t k_ss, const void* v, int64_t v_sb, int64_t v_sh,
                                                                        int64_t v_ss, int32_t n_tok, int32_t t0, int32_t flags, void* stream) {
    if (!s) return BGTQ_E_BADARG;
    return bgtq_encode(s->desc, s->rot_k, s->rot_v, k, k_sb, k_sh, k_ss, v, v_sb, v_sh, v_ss, s->n_batch, s->n_kv, n_tok, t0, s->k_packed,
                       s->kp_sb, s->kp_sh, s->kp_st, s->kp_row_bytes, s->k_norms, s->kn_sb, s->kn_sh, s->kn_st, s->kn_count, s->v_packed,
                       s->vp_sb, s->vp_sh, s->vp_st, s->v_norms, s->vn_sb, s->vn_sh, s->vn_st, nullptr, nullptr,
                       (s->enc_flags & ~BGTQ_ENC_PROGRAMMATIC) | flags, nullptr, s->t_capacity, nullptr, stream);
}

extern "C" __attribute__((visibility("default"))) int64_t bgtq_attend_scratch_bytes(int32_t n_batch, int32_t n_q, int32_t n_splits) {
    if (n_batch < 1 || n_q < 1 || n_splits < 1) return 0;
    const int64_t rows = (int64_t)n_batch * n_q;
    return rows * kHD * 2 + rows * n_splits * (kHD + 1) * 4;
}

extern "C" __attribute__((visibility("default"))) int bgtq_attend(
    const BgtqDecodePlan* plan, const BgtqHeadDesc* desc, const float* rot_k, const void* q, int64_t q_sb, int64_t q_sh,
    const uint8_t* k_packed, int64_t kp_sb, int64_t kp_sh, int64_t kp_st, const void* k_norms, int64_t kn_sb, int64_t kn_sh,
    int64_t kn_st, const uint8_t* v_packed, int64_t vp_sb, int64_t vp_sh, int64_t vp_st, const void* v_norms, int64_t vn_sb,
    int64_t vn_sh, int64_t vn_st, int32_t n_batch, int32_t n_q, int32_t n_kv, int32_t t_begin, int32_t t_end, int32_t n_splits,
    float scale, const float* v_rot, const float* buf_o, const float* buf_lse, void* scratch, void* out, float* out_f32,
    float* lse_out, int32_t* status, void* stream) {
    if (!plan || !q || !out || n_batch < 1 || n_q < 1 || n_splits < 1) return BGTQ_E_BADARG;
    if (!scratch && (rot_k || !bgtq_decode_plan_cluster(plan))) return BGTQ_E_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(scratch) & 15u) return BGTQ_E_ALIGN;
    const int64_t rows = (int64_t)n_batch * n_q;
    float* const part_o = static_cast<float*>(scratch);
    float* const part_lse = part_o + rows * n_splits * kHD;
    __half* const q_rot = reinterpret_cast<__half*>(part_lse + rows * n_splits);
    const void* q_dec = q;
    if (rot_k) {
        const int rc = launch_rotate_q(desc, rot_k, q, q_sb, q_sh, q_rot, n_batch, n_q, n_kv, true, static_cast<cudaStream_t>(stream));
        if (rc != BGTQ_OK) return rc;
        q_dec = q_rot;
    } else if (!contiguous_rows(n_batch, n_q, q_sb, q_sh)) {
        return BGTQ_E_UNSUPPORTED;
    }
    // No early fetch here, whatever the plan says: what is in front of this call may be a bulk encode of the very rows
    // that are attended, and it lets its dependents start while it runs.  (A layer step is different: there the launch in
    // front of the decode is its own append.)
    if ((buf_o == nullptr) == (buf_lse == nullptr) && bgtq_decode_plan_cluster(plan)) {
        const MergeParams M = {v_rot, static_cast<uint16_t*>(out), (int64_t)n_q * kHD, kHD, out_f32, lse_out, buf_o, buf_lse, 0, 0};
        const int rc = launch_decode_plan(plan, q_dec, k_packed, kp_sb, kp_sh, kp_st, k_norms, kn_sb, kn_sh, kn_st, v_packed, vp_sb, vp_sh,
                                          vp_st, v_norms, vn_sb, vn_sh, vn_st, n_batch, n_q, n_kv, t_begin, t_end, n_splits, scale, nullptr,
                                          nullptr, status, nullptr, 0, false, &M, stream);
        if (rc != BGTQ_E_UNSUPPORTED || !scratch) return rc;
    }
    const int rc = launch_decode_plan(plan, q_dec, k_packed, kp_sb, kp_sh, kp_st, k_norms, kn_sb, kn_sh, kn_st, v_packed, vp_sb, vp_sh,
                                      vp_st, v_norms, vn_sb, vn_sh, vn_st, n_batch, n_q, n_kv, t_begin, t_end, n_splits, scale, part_o,
                                      part_lse, status, nullptr, 0, false, nullptr, stream);
    if (rc != BGTQ_OK) return rc;
    return bgtq_combine(part_o, part_lse, n_splits, v_rot, buf_o, buf_lse, n_batch, n_q, n_kv, out, (int64_t)n_q * kHD, kHD, out_f32,
                        lse_out, BGTQ_COMBINE_PROGRAMMATIC, stream);
}
