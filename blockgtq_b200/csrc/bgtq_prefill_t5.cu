// Packed-cache prefill attention on the fifth-generation tensor cores (tcgen05) with accumulators in tensor
// memory, in two launches (three when the cache is split):
//
//   unpack  every 128-token tile of the cache is dequantised ONCE into a workspace, in the tensor cores' operand
//           layout: khat = fp16 centroid * fp16 norm held exactly as a high and a low fp16 tile [token][dim], vhat =
//           fp16(centroid * norm) transposed [dim][token]; 32 KB each, stored with one bulk copy.  (A kernel that
//           dequantised inside the attention repeated it for every 256 query rows, between the products: 6.40 ms for
//           16384 tokens x 32 heads, the tensor cores 22 % busy.)
//   attend  one CTA owns 256 query rows of one (batch, KV head) as two blocks of 128 = the M of every product (row =
//           position * gqa + head of the group, whatever gqa is) and walks the tiles.  Eighteen warps with three jobs:
//             * one thread streams the tiles into a ring of five 32 KB slots (khat low, khat high, vhat, ...);
//             * one thread issues S_m = Q_m . Khat_lo^T + Q_m . Khat_hi^T (16 tcgen05.mma, M = N = 128) and O_m += P_m .
//               Vhat (8 tcgen05.mma, P read from tensor memory) for the two blocks in turn, so that the tensor cores
//               work on one block while the other block's softmax runs;
//             * 512 threads, two per query row (64 columns each), read their part of S with tcgen05.ld, apply the causal
//               limit and put P (fp16) over S in tensor memory.  The value a row scales by moves, and O is rescaled, only
//               when the row's maximum grew by more than 2^8 since it was set: whether any row's did is one barrier with
//               an OR, and only then the two threads of a row exchange their maxima.  (With one thread per row, 128
//               columns in a chain, a block's softmax outlasted the other block's products: a quarter of the tensor pipe's time.)
//           The normalised rows meet V's rotation on the tensor cores too (row and rotation as high + low fp16 parts,
//           three products: the missing low x low part is 2^-22 of a value): O . R leaves as fp16, and no fp32 copy of
//           the output is written.
//   merge   the cache of a launch with few query rows is cut among several CTAs; their (O, log-sum-exp) partials are
//           added up per row.
//
// What bounds attend: the tensor pipe.  A tile costs a CTA 2 x 16 products for S and 2 x 8 for O, 64 cycles each at the
// nominal rate: 3072 cycles, two thirds of them for S because khat takes two passes (its product of two fp16 numbers
// has 22 significant bits, all of which the reference's fp32 scaling keeps); the exponentials of the tile take the
// special-function pipe 2048.  Measured for 16384 causal positions x 32 heads over 8 KV heads: 2.41 to 2.50 ms in single
// launches (about 900 TFLOP/s of attention, 1340 of products; tensor pipe 65 % active, special functions 43 %, issue slots
// 34 %), 2.72 ms where launches follow each other for seconds, at the power limit; unthrottled a tile takes 4070 cycles.
// Every wait is bounded: a wait that gives up is recorded in a sticky status word and in shared memory, where the
// other warps' waits see it; the CTA then drains its copies and products, releases its tensor memory and returns.
#include "bgtq_prefill_common.cuh"
#include "bgtq_tcgen05.cuh"

namespace bgtq {

__device__ int g_pf5_status = 0;

namespace {

constexpr int kT5Tok = 128;                     // cache tokens per tile = N of the S product, K of the O product
constexpr int kT5Rows = 128;                    // M of every product
constexpr int kT5Blocks = 2;                    // 128-row blocks per CTA
constexpr int kPart = kT5Tok * kHD * 2;         // bytes of one operand tile (32 KB)
constexpr int kTileBytes = 3 * kPart;           // khat low, khat high, vhat of a tile, in the order the ring takes them
constexpr float kRotScale = 64.0f;              // rotations are stored times this, so that their low parts stay normal fp16 numbers

// ------------------------------------------------------------------------------------------------------------------
// unpack
// ------------------------------------------------------------------------------------------------------------------
constexpr int kUpThreads = 512;
constexpr int kPtWords = BGTQ_MAX_SEGMENTS * 256 + 256;

// Operand layout (no swizzle, K-major): 8 x 8 core matrices of 128 B (8 rows of 16 B); along K they follow each
// other 128 B apart, 8-row groups are 2048 B apart: element (row, k) at
//     (row / 8) * 2048 + (k / 8) * 128 + (row % 8) * 16 + (k % 8) * 2.
struct UpSmem {
    __align__(128) uint8_t kl[kPart];
    __align__(128) uint8_t kh[kPart];
    __align__(128) uint8_t vt[kPart];
    __align__(16) uint32_t pt[kPtWords];            // pair tables: (code, code) -> fp16x2, per K segment of <= 4 stored bits, then V
    uint16_t seg_pt[BGTQ_MAX_SEGMENTS + 1];         // first word of each segment's pair table; last entry: V's
    uint16_t cb[528];                               // 512 K entries + 16 V entries (fp16 bits)
    uint2 ktask[kPfMaxTasks];
    uint2 vtask[16];
    int32_t n_ktask, n_vtask;
};

struct UpRaw {      // byte offsets of the tile's packed rows behind UpSmem (each region 16-byte aligned, + 4 bytes of phase)
    uint32_t k, kn, v, vn, total;
};

__device__ __forceinline__ void up_stage(uint8_t* dst, const uint8_t* src, int n_bytes, int tid) {
    // dst[(src & 3) + i] = src[i]: whole 32-bit words asynchronously, the ragged tail byte by byte
    const uint32_t ph = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3u);
    const uint8_t* s4 = src - ph;
    const uint32_t d4 = smem_u32(dst);
    const int n_words = (int)((ph + n_bytes) >> 2);
    for (int i = tid; i < n_words; i += kUpThreads)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d4 + 4u * i), "l"(s4 + 4 * i) : "memory");
    const int tail = (int)((ph + n_bytes) & 3u);
    if (tid < tail) dst[4 * n_words + tid] = s4[4 * n_words + tid];
}

// The 32 (or, for raw-byte codes, 64) bits that start at byte p, from aligned 32-bit loads.  Reads up to 11
// bytes past p + 4: inside the staging buffer (its regions carry that much slack or are followed by another).
__device__ __forceinline__ void up_words(const uint8_t* p, bool two, uint32_t& w0, uint32_t& w1) {
    const uint32_t a = smem_u32(p), al = a & ~3u, sh = (a & 3u) * 8u;
    const uint32_t x0 = lds32(al), x1 = lds32(al + 4u);
    w0 = __funnelshift_r(x0, x1, sh);
    w1 = 0u;
    if (two) w1 = __funnelshift_r(x1, lds32(al + 8u), sh);
}

// One K task of TWO tokens (lane and lane + 32 of the tile: two independent chains per lane): up to 8 codes of SB
// stored bits at src[e] -> khat = centroid * norm as a high and a low fp16 tile.  hi = fp16(centroid * norm);
// lo = fp16(centroid * norm - hi) with one rounding (fused), i.e. the two fp16 numbers the exact fp32 product
// splits into.  A token past the tile's end stores zeros.
// FAST: a full task (8 codes) of two live tokens whose low part is kept: no per-pair checks.
template <int SB, bool FAST>
__device__ __forceinline__ void up_k_task(uint8_t* kh, uint8_t* kl, const uint8_t* const (&src)[2], const uint32_t* pt,
                                          const uint16_t* cb, const __half2 (&n2)[2], bool round16, int first, int n,
                                          const uint32_t (&trow)[2], uint32_t rot, const bool (&live)[2]) {
    uint32_t w0[2] = {0u, 0u}, w1[2] = {0u, 0u};
#pragma unroll
    for (int e = 0; e < 2; ++e)
        if (FAST || live[e]) up_words(src[e], SB == 8, w0[e], w1[e]);
#pragma unroll
    for (int pi0 = 0; pi0 < 4; ++pi0) {
        const uint32_t c = 2u * ((pi0 + rot) & 3u);
        if (FAST || (int)c < n) {
            const int dd = first + (int)c;
            const uint32_t doff = (uint32_t)((dd >> 3) * 128 + (dd & 7) * 2);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t cc;       // the two centroids as fp16x2
                if constexpr (SB == 8) {
                    const uint32_t two = (c < 4u ? w0[e] : w1[e]) >> ((c & 2u) * 8u);
                    cc = (uint32_t)cb[two & 0xFFu] | (uint32_t)cb[(two >> 8) & 0xFFu] << 16;
                } else {
                    cc = pt[(w0[e] >> (c * SB)) & ((1u << (2 * SB)) - 1u)];
                }
                const __half2 c2 = *reinterpret_cast<const __half2*>(&cc);
                const __half2 h2 = __hmul2(c2, n2[e]);
                const __half2 l2 = __hfma2(c2, n2[e], __hneg2(h2));
                uint32_t hi = *reinterpret_cast<const uint32_t*>(&h2), lo = *reinterpret_cast<const uint32_t*>(&l2);
                if (!FAST) {
                    if (round16) lo = 0u;
                    if (!live[e]) hi = lo = 0u;
                }
                *reinterpret_cast<uint32_t*>(kh + trow[e] + doff) = hi;
                *reinterpret_cast<uint32_t*>(kl + trow[e] + doff) = lo;
            }
        }
    }
}
// One V task of two tokens: 8 codes each -> vhat = fp16(centroid * norm), stored down each token's column of the
// transposed tile (`col` = the task's first dim, token `lane`; token lane + 32 sits 4 k-chunks = 512 B further).
template <int SB, bool FAST>
__device__ __forceinline__ void up_v_task(uint8_t* col, const uint8_t* const (&src)[2], const uint32_t* vpt, const __half2 (&n2)[2],
                                          uint32_t rot, const bool (&live)[2]) {
    uint32_t w0[2] = {0u, 0u}, w1 = 0u;
#pragma unroll
    for (int e = 0; e < 2; ++e)
        if (FAST || live[e]) up_words(src[e], false, w0[e], w1);
#pragma unroll
    for (int pi0 = 0; pi0 < 4; ++pi0) {
        const uint32_t c = 2u * ((pi0 + rot) & 3u);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t cc = vpt[(w0[e] >> (c * SB)) & ((1u << (2 * SB)) - 1u)];
            const __half2 v2 = __hmul2(*reinterpret_cast<const __half2*>(&cc), n2[e]);
            uint32_t v = *reinterpret_cast<const uint32_t*>(&v2);
            if (!FAST && !live[e]) v = 0u;
            *reinterpret_cast<uint16_t*>(col + e * 512 + c * 16u) = (uint16_t)v;
            *reinterpret_cast<uint16_t*>(col + e * 512 + (c + 1u) * 16u) = (uint16_t)(v >> 16);
        }
    }
}

__device__ __forceinline__ void bulk_s2g(void* dst_gmem, const void* src_smem, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_gmem), "r"(smem_u32(src_smem)), "r"(bytes)
                 : "memory");
}

// grid: (CTAs per pair, KV head, batch), each CTA walks `per_cta` consecutive tiles; with a rotation the last
// blockIdx.x (of batch 0) makes the head's rotation operand instead.
__global__ void __launch_bounds__(kUpThreads, 1) pf_unpack_kernel(const PfParams P, const UpRaw R, uint8_t* tiles, uint8_t* rots,
                                                                  const float* v_rot, int per_cta) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    UpSmem& S = *reinterpret_cast<UpSmem*>(smem_raw);
    uint8_t* const raw0 = smem_raw + sizeof(UpSmem);      // two staging buffers of R.total bytes
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.y, b = blockIdx.z;
    const int n_tiles = (P.n_tok + kT5Tok - 1) / kT5Tok;
    grid_launch_dependents();
    if (v_rot && blockIdx.x == gridDim.x - 1) {      // rotation operand: element (n, k) = R[k][n], as high and low fp16 parts
        grid_dependency_wait();
        if (b != 0) return;
        const float* W = v_rot + (size_t)h * kHD * kHD;
        for (int i = tid; i < kHD * kHD / 8; i += kUpThreads) {
            const int n = i & (kHD - 1), k8 = i >> 7;
            __align__(16) __half hi[8], lo[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float w = W[(size_t)(8 * k8 + e) * kHD + n] * kRotScale;        // (may have been converted right in front)
                hi[e] = __float2half_rn(w);
                lo[e] = __float2half_rn(w - __half2float(hi[e]));
            }
            uint8_t* o = rots + (size_t)h * 2 * kPart + (n >> 3) * 2048 + k8 * 128 + (n & 7) * 16;
            *reinterpret_cast<uint4*>(o) = *reinterpret_cast<uint4*>(hi);
            *reinterpret_cast<uint4*>(o + kPart) = *reinterpret_cast<uint4*>(lo);
        }
        return;
    }
    const BgtqHeadDesc& d = P.desc[h];
    const int first_tile = blockIdx.x * per_cta, last_tile = min(n_tiles, first_tile + per_cta);      // never empty

    for (int i = tid; i < 528; i += kUpThreads) S.cb[i] = i < 512 ? d.codebook[i] : d.v_lut[i - 512];
    if (tid == 0) pf_build_tasks(P, d, S.ktask, S.vtask, &S.n_ktask, &S.n_vtask);
    // pair tables: entry i of a table for `sb` stored bits = (centroid[i & m], centroid[(i >> sb) & m])
    {
        const bool mixed = P.flags & BGTQ_DEC_K_MIXED;
        int base = 0;
        for (int sg = 0; sg <= d.n_seg; ++sg) {
            const bool is_v = sg == d.n_seg;
            const int bw = is_v ? d.v_bits : d.seg_bw[sg];
            const int sb = is_v ? ((P.flags & BGTQ_DEC_V_NIBBLE) ? 4 : d.v_bits) : (mixed ? (bw <= 4 ? 4 : 8) : (bw <= 4 ? bw : 8));
            if (tid == 0) S.seg_pt[is_v ? BGTQ_MAX_SEGMENTS : sg] = (uint16_t)base;
            if (sb <= 4) {
                const uint32_t m = (1u << sb) - 1u;
                const uint16_t* src = is_v ? d.v_lut : d.codebook + d.seg_lut_off[sg];
                for (int i = tid; i < (1 << (2 * sb)); i += kUpThreads)
                    S.pt[base + i] = (uint32_t)src[i & m] | (uint32_t)src[(i >> sb) & m] << 16;
                base += 1 << (2 * sb);
            }
        }
    }
    const size_t bh_kp = (size_t)b * P.kp_sb + (size_t)h * P.kp_sh, bh_kn = (size_t)b * P.kn_sb + (size_t)h * P.kn_sh;
    const size_t bh_vp = (size_t)b * P.vp_sb + (size_t)h * P.vp_sh, bh_vn = (size_t)b * P.vn_sb + (size_t)h * P.vn_sh;
    auto stage_tile = [&](int tile) {
        uint8_t* const raw = raw0 + (size_t)(tile & 1) * R.total;
        const int t0 = tile * kT5Tok, nt = min(kT5Tok, P.n_tok - t0);
        up_stage(raw + R.k, P.kp + bh_kp + (size_t)t0 * P.kp_st, nt * P.kp_st, tid);
        up_stage(raw + R.kn, P.kn + bh_kn + (size_t)t0 * P.kn_st, nt * P.kn_st, tid);
        up_stage(raw + R.v, P.vp + bh_vp + (size_t)t0 * P.vp_st, nt * P.vp_st, tid);
        up_stage(raw + R.vn, P.vn + bh_vn + (size_t)t0 * P.vn_st, nt * P.vn_st, tid);
    };
    grid_dependency_wait();          // the cache rows come from earlier work in the stream
    stage_tile(first_tile);
    for (int tile = first_tile; tile < last_tile; ++tile) {
        const int t0 = tile * kT5Tok, nt = min(kT5Tok, P.n_tok - t0);
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");     // the previous tile has left the operand buffers
        __syncthreads();
        if (tile + 1 < last_tile) stage_tile(tile + 1);
        const uint8_t* const raw = raw0 + (size_t)(tile & 1) * R.total;
        const uint8_t* rk = raw + R.k + (reinterpret_cast<uintptr_t>(P.kp + bh_kp + (size_t)t0 * P.kp_st) & 3u);
        const uint8_t* rn = raw + R.kn + (reinterpret_cast<uintptr_t>(P.kn + bh_kn + (size_t)t0 * P.kn_st) & 3u);
        const uint8_t* rv = raw + R.v + (reinterpret_cast<uintptr_t>(P.vp + bh_vp + (size_t)t0 * P.vp_st) & 3u);
        const uint8_t* rw = raw + R.vn + (reinterpret_cast<uintptr_t>(P.vn + bh_vn + (size_t)t0 * P.vn_st) & 3u);
        // One warp per (task, 64-token half): the task's fields are uniform; lane l dequantises tokens l and l + 32.  The
        // four 8-token groups of a warp walk a task's four pairs in different order, so that their stores (same banks,
        // 2048 / 128 B apart) do not collide.
        const uint32_t rot = (uint32_t)lane >> 3;
        const uint32_t* vpt = S.pt + S.seg_pt[BGTQ_MAX_SEGMENTS];
        const uint32_t vsb = (S.vtask[0].x >> 12) & 0xF;
        const int n_k = 2 * S.n_ktask, n_all = n_k + 2 * S.n_vtask;
        for (int u = warp; u < n_all; u += kUpThreads / 32) {
            const bool is_v = u >= n_k;
            const int ti = (is_v ? u - n_k : u) >> 1;
            const int tb = (u & 1) * 64 + lane;                            // this lane's tokens: tb and tb + 32   (n_k is even)
            const bool live[2] = {tb < nt, tb + 32 < nt};
            if (is_v) {
                const uint2 tk = S.vtask[ti];
                const int first = tk.x & 0xFF;
                uint8_t* const col = S.vt + (first >> 3) * 2048 + (tb >> 3) * 128 + (tb & 7) * 2;
                const uint8_t* const src[2] = {rv + tb * P.vp_st + (tk.y & 0xFFFFu), rv + (tb + 32) * P.vp_st + (tk.y & 0xFFFFu)};
                const __half2 n2[2] = {__half2half2(__ushort_as_half(*reinterpret_cast<const uint16_t*>(rw + tb * P.vn_st))),
                                       __half2half2(__ushort_as_half(*reinterpret_cast<const uint16_t*>(rw + (tb + 32) * P.vn_st)))};
                if (nt == kT5Tok) {
                    switch (vsb) {
                        case 1: up_v_task<1, true>(col, src, vpt, n2, rot, live); break;
                        case 2: up_v_task<2, true>(col, src, vpt, n2, rot, live); break;
                        case 3: up_v_task<3, true>(col, src, vpt, n2, rot, live); break;
                        default: up_v_task<4, true>(col, src, vpt, n2, rot, live); break;
                    }
                } else {
                    switch (vsb) {
                        case 1: up_v_task<1, false>(col, src, vpt, n2, rot, live); break;
                        case 2: up_v_task<2, false>(col, src, vpt, n2, rot, live); break;
                        case 3: up_v_task<3, false>(col, src, vpt, n2, rot, live); break;
                        default: up_v_task<4, false>(col, src, vpt, n2, rot, live); break;
                    }
                }
                continue;
            }
            const uint2 tk = S.ktask[ti];
            const int first = tk.x & 0xFF, n = (tk.x >> 8) & 0xF, sg = (tk.x >> 16) & 0xF;
            const uint32_t sb = (tk.x >> 12) & 0xF;
            const bool round16 = (tk.x >> 20) & 1u;
            const uint32_t trow[2] = {(uint32_t)((tb >> 3) * 2048 + (tb & 7) * 16), (uint32_t)(((tb >> 3) + 4) * 2048 + (tb & 7) * 16)};
            const uint8_t* const src[2] = {rk + tb * P.kp_st + (tk.y & 0xFFFFu), rk + (tb + 32) * P.kp_st + (tk.y & 0xFFFFu)};
            const __half2 n2[2] = {
                __half2half2(__ushort_as_half(*reinterpret_cast<const uint16_t*>(rn + tb * P.kn_st + 2 * sg))),
                __half2half2(__ushort_as_half(*reinterpret_cast<const uint16_t*>(rn + (tb + 32) * P.kn_st + 2 * sg)))};
            const uint32_t* pt = S.pt + S.seg_pt[sg];
            const uint16_t* cb = S.cb + (tk.y >> 16);
            if (nt == kT5Tok && n == 8 && !round16) {       // (uniform over the warp)
                switch (sb) {
                    case 1: up_k_task<1, true>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    case 2: up_k_task<2, true>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    case 3: up_k_task<3, true>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    case 4: up_k_task<4, true>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    default: up_k_task<8, true>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                }
            } else {
                switch (sb) {
                    case 1: up_k_task<1, false>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    case 2: up_k_task<2, false>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    case 3: up_k_task<3, false>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    case 4: up_k_task<4, false>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                    default: up_k_task<8, false>(S.kh, S.kl, src, pt, cb, n2, round16, first, n, trow, rot, live); break;
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {         // kl, kh and vt lie one behind the other
            bulk_s2g(tiles + (((size_t)b * P.n_kv + h) * n_tiles + tile) * kTileBytes, S.kl, kTileBytes);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ------------------------------------------------------------------------------------------------------------------
// attend
// ------------------------------------------------------------------------------------------------------------------
constexpr int kAtThreads = 576;         // warps 0-7: rows of block 0 (columns 0..63, then 64..127), 8-15: block 1, 16: products, 17: copies
constexpr int kWarpMma = 16, kWarpCopy = 17;
constexpr int kSlots = 5;
constexpr uint32_t kTmemCols = 512;     // S (and P) of block m: columns [128 m, 128 m + 128); O of block m: [256 + 128 m, 384 + 128 m)
constexpr uint32_t kColS = 0, kColO = 256;
constexpr float kLazyLog2 = 8.0f;       // a row rescales O only when its maximum grew by more than 2^8

struct AtSmem {
    __align__(128) uint8_t q[kT5Blocks][kPart];
    __align__(128) uint8_t ring[kSlots][kPart];
    __align__(8) uint64_t full[kSlots], empty[kSlots], s_ready[kT5Blocks], p_ready[kT5Blocks], o_ready[kT5Blocks];
    float xch[kT5Blocks][2][kT5Rows];       // the two threads of a row: maxima, at the end denominators
    uint32_t tmem_base;
    volatile int32_t failed;
};
static_assert(sizeof(AtSmem) <= 227 * 1024, "fits an SM");

struct AtParams {
    const __half* q;
    int64_t q_sb, q_sh, q_ss;
    const uint8_t* tiles;       // operand tiles of the cache
    const uint8_t* rots;        // rotation operands (high, low) per KV head, or null: the output stays in V's rotated basis
    int32_t n_q, n_kv, gqa, s_q, n_tok, q_pos_offset, causal, n_splits, n_qblk;
    float scale_log2;
    __half* out16;              // (batch, n_q, s_q, 128) fp16, or null
    float* out32;               // the same in fp32; with n_splits > 1 (split, batch, n_q, s_q, 128) partials
    float* lse2;                // n_splits > 1: (split, batch, n_q, s_q) log2 of the partials' denominators
};

__device__ __forceinline__ float at_exp2(float x) {      // hardware 2^x; ex2(-inf) = 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 16 consecutive 32-bit columns of this thread's tensor-memory lane from registers
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// 8 consecutive fp32 columns of this thread's lane times a factor, in place
__device__ __forceinline__ void tmem_scale8(uint32_t taddr, float f) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Barrier over the 256 threads of one block's rows; returns whether any of them says so.
__device__ __forceinline__ bool bar_or(uint32_t id, bool flag) {
    uint32_t out;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.or.pred p, %2, 256, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(out)
        : "r"((uint32_t)flag), "r"(id)
        : "memory");
    return out != 0;
}
// Bounded wait that also ends when another warp of the CTA gave up.
__device__ __forceinline__ bool at_wait(AtSmem& S, uint64_t* bar, uint32_t parity) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 63u && S.failed) return false;
    }
    S.failed = 1;
    return false;
}

__global__ void __launch_bounds__(kAtThreads, 1) pf_attend_kernel(const AtParams P) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    AtSmem& S = *reinterpret_cast<AtSmem*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // block index: query block fastest (latest positions, with the most tiles under the causal mask, first), so that
    // CTAs that run at the same time read the same head's tiles from L2
    const int blk = P.n_qblk - 1 - (int)(blockIdx.x / P.n_splits), sp = (int)(blockIdx.x % P.n_splits);
    const int h = blockIdx.y, b = blockIdx.z;
    const int n_rows = P.s_q * P.gqa, row0 = blk * kT5Rows * kT5Blocks;
    const int last_pos = (min(n_rows, row0 + kT5Rows * kT5Blocks) - 1) / P.gqa;
    const int t_max = P.causal ? min(P.n_tok, P.q_pos_offset + last_pos + 1) : P.n_tok;
    const int n_all = (t_max + kT5Tok - 1) / kT5Tok;
    const int tile0 = (int)((int64_t)n_all * sp / P.n_splits), n_t = (int)((int64_t)n_all * (sp + 1) / P.n_splits) - tile0;

    grid_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(&S.full[i], 1);
            mbar_init(&S.empty[i], 1);
        }
        for (int m = 0; m < kT5Blocks; ++m) {
            mbar_init(&S.s_ready[m], 1);
            mbar_init(&S.p_ready[m], 2 * kT5Rows);
            mbar_init(&S.o_ready[m], 1);
        }
        mbar_fence_init();
        S.failed = 0;
    }
    if (warp == kWarpMma) tmem_alloc(&S.tmem_base, kTmemCols);
    grid_dependency_wait();
    // the CTA's query rows -> the A operands (16-byte chunks of 8 dims, all requested before the first is waited for);
    // rows past the end are zero
    const bool q16 = ((reinterpret_cast<uintptr_t>(P.q) | (uint64_t)(2 * P.q_sb) | (uint64_t)(2 * P.q_sh) | (uint64_t)(2 * P.q_ss)) & 15u) == 0;
    for (int i = tid; i < kT5Rows * kT5Blocks * 16; i += kAtThreads) {
        const int row = i >> 4, kc = i & 15, g = row0 + row;
        uint8_t* const dst = S.q[row >> 7] + ((row & 127) >> 3) * 2048 + kc * 128 + (row & 7) * 16;
        const int pos = g < n_rows ? g / P.gqa : 0, hq = h * P.gqa + (g < n_rows ? g - pos * P.gqa : 0);
        const __half* src = P.q + b * P.q_sb + hq * P.q_sh + (int64_t)pos * P.q_ss + kc * 8;
        if (q16) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(g < n_rows ? 16 : 0) : "memory");
        } else {
            const uint32_t* s32 = reinterpret_cast<const uint32_t*>(src);
            *reinterpret_cast<uint4*>(dst) =
                g < n_rows ? make_uint4(s32[0], s32[1], s32[2], s32[3]) : make_uint4(0, 0, 0, 0);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // Q: generic-proxy stores -> tensor-core reads
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = S.tmem_base;
    bool ok = true;

    if (warp == kWarpCopy) {
        // ---- copies: tile parts in ring order, then the rotation operands ----
        if (lane == 0) {
            const uint8_t* src = P.tiles + (((size_t)b * P.n_kv + h) * ((P.n_tok + kT5Tok - 1) / kT5Tok) + tile0) * kTileBytes;
            const int n_tile_parts = 3 * n_t, n_parts = n_tile_parts + (P.rots && n_t > 0 ? 2 : 0);
            int n = 0;
            for (; n < n_parts; ++n) {
                const int slot = n % kSlots;
                if (n >= kSlots && !at_wait(S, &S.empty[slot], (uint32_t)(n / kSlots - 1) & 1u)) { ok = false; break; }
                mbar_arrive_expect_tx(&S.full[slot], kPart);
                const uint8_t* from = n < n_tile_parts ? src + (size_t)n * kPart : P.rots + ((size_t)h * 2 + (n - n_tile_parts)) * kPart;
                bulk_g2s(S.ring[slot], from, kPart, &S.full[slot]);
            }
            if (!ok)        // the copies in flight land before the CTA leaves
                for (int i = max(0, n - kSlots); i < n; ++i) mbar_wait_bounded(&S.full[i % kSlots], (uint32_t)(i / kSlots) & 1u);
        }
    } else if (warp == kWarpMma) {
        // ---- products (the whole warp walks the tiles; one lane issues) ----
        if (n_t > 0) {
            const uint32_t lead = elect_one();
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint64_t q_desc = op_desc(smem_u32(S.q[0])), ring_desc = op_desc(smem_u32(S.ring[0]));
            auto wait_part = [&](int n) { return (bool)__all_sync(0xffffffffu, at_wait(S, &S.full[n % kSlots], (uint32_t)(n / kSlots) & 1u)); };
            auto part_desc = [&](int n) { return ring_desc + (uint32_t)(n % kSlots) * (kPart >> 4); };
            auto commit = [&](uint64_t* bar) {
                if (lead) umma_commit(bar);
                __syncwarp();
            };
            // A in tensor memory, k-step ks: the first four steps lie in columns 0..31 of S, the others in 64..95
            auto a_of = [](uint32_t base, int ks) { return base + 64u * (uint32_t)(ks >> 2) + 8u * (uint32_t)(ks & 3); };
            auto issue_s = [&](int i, int m) {
                const uint64_t qa = q_desc + (uint32_t)m * (kPart >> 4), lo = part_desc(3 * i), hi = part_desc(3 * i + 1);
                const uint32_t dst = tm + kColS + 128u * m;
#pragma unroll
                for (int ks = 0; ks < kHD / 16; ++ks) mma_ss(dst, qa + 16u * ks, lo + 16u * ks, ks > 0, lead);
#pragma unroll
                for (int ks = 0; ks < kHD / 16; ++ks) mma_ss(dst, qa + 16u * ks, hi + 16u * ks, 1u, lead);
                commit(&S.s_ready[m]);
                if (m == kT5Blocks - 1) {
                    commit(&S.empty[(3 * i) % kSlots]);
                    commit(&S.empty[(3 * i + 1) % kSlots]);
                }
            };
            ok = wait_part(0) && wait_part(1);
            if (ok) {
                issue_s(0, 0);
                issue_s(0, 1);
            }
            for (int i = 0; i < n_t && ok; ++i) {
#pragma unroll
                for (int m = 0; m < kT5Blocks; ++m) {
                    if (m == 0 && !wait_part(3 * i + 2)) { ok = false; break; }
                    if (!__all_sync(0xffffffffu, at_wait(S, &S.p_ready[m], (uint32_t)i & 1u))) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint64_t vt = part_desc(3 * i + 2);
                    const uint32_t a = tm + kColS + 128u * m, dst = tm + kColO + 128u * m;
#pragma unroll
                    for (int ks = 0; ks < kT5Tok / 16; ++ks) mma_ts(dst, a_of(a, ks), vt + 16u * ks, (i > 0 || ks > 0) ? 1u : 0u, lead);
                    commit(&S.o_ready[m]);
                    if (m == kT5Blocks - 1) commit(&S.empty[(3 * i + 2) % kSlots]);
                    if (i + 1 < n_t) {      // (products of one thread execute in order: S replaces the P that was just read)
                        if (m == 0 && !(wait_part(3 * i + 3) && wait_part(3 * i + 4))) { ok = false; break; }
                        issue_s(i + 1, m);
                    }
                }
            }
            if (P.rots && ok) {     // O . R: A = the row's high part and, 32 columns further, its low part
                const int n = 3 * n_t;
                ok = wait_part(n) && wait_part(n + 1);
                for (int m = 0; m < kT5Blocks && ok; ++m) {
                    if (!__all_sync(0xffffffffu, at_wait(S, &S.p_ready[m], (uint32_t)n_t & 1u))) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint64_t rh = part_desc(n), rl = part_desc(n + 1);
                    const uint32_t a = tm + kColS + 128u * m, dst = tm + kColO + 128u * m;
#pragma unroll
                    for (int ks = 0; ks < kHD / 16; ++ks) mma_ts(dst, a_of(a, ks) + 32u, rh + 16u * ks, ks > 0, lead);
#pragma unroll
                    for (int ks = 0; ks < kHD / 16; ++ks) mma_ts(dst, a_of(a, ks), rl + 16u * ks, 1u, lead);
#pragma unroll
                    for (int ks = 0; ks < kHD / 16; ++ks) mma_ts(dst, a_of(a, ks), rh + 16u * ks, 1u, lead);
                    commit(&S.o_ready[m]);
                }
            }
            if (!ok) {              // products in flight end before the tensor memory is released
                commit(&S.s_ready[0]);
                mbar_wait_bounded(&S.s_ready[0], 0u);
                mbar_wait_bounded(&S.s_ready[0], 1u);
            }
        }
    } else {
        // ---- softmax: two threads per query row ----
        const int mb = warp >> 3, hf = (warp >> 2) & 1, r128 = (warp & 3) * 32 + lane;
        const int g = row0 + kT5Rows * mb + r128;
        const bool rok = g < n_rows;
        const int pos = g / P.gqa;
        const int lim = !rok ? 0 : (P.causal ? min(P.n_tok, P.q_pos_offset + pos + 1) : P.n_tok);
        const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);   // this warp's quarter of the lanes
        const uint32_t colS = tlane + kColS + 128u * mb, colO = tlane + kColO + 128u * mb + 64u * hf;
        float m_used = -INFINITY, lsum = 0.f;    // the maximum this row scales by (log2 domain), this half's denominator
        const uint64_t sc2 = pack_f2(P.scale_log2, P.scale_log2);
        for (int i = 0; i < n_t; ++i) {
            if (!__all_sync(0xffffffffu, at_wait(S, &S.s_ready[mb], (uint32_t)i & 1u))) ok = false;
            tc_fence_after_sync();
            // 32 columns at a time, the second half of them read again for the exponentials: two chains of few registers
            // instead of 64 logits held across the barrier (which spilled)
            const uint32_t sS = colS + 64u * hf;
            const int t0 = (tile0 + i) * kT5Tok + 64 * hf;
            const bool cut = !__all_sync(0xffffffffu, t0 + 64 <= lim);     // only tiles that reach a row's causal limit
            float sv[32];
            auto load = [&](int c0) {
                tmem_ld32(sS + (uint32_t)c0, sv);
                tmem_ld_wait();
                if (cut) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) sv[c] = t0 + c0 + c < lim ? sv[c] : -INFINITY;
                }
            };
            auto top = [&]() {
                float a = max3(sv[0], sv[1], sv[2]), c = max3(sv[3], sv[4], sv[5]);
#pragma unroll
                for (int e = 6; e < 30; e += 4) {
                    a = max3(a, sv[e], sv[e + 1]);
                    c = max3(c, sv[e + 2], sv[e + 3]);
                }
                return max3(max3(a, c, c), sv[30], sv[31]);
            };
            load(32);
            float m_half = top();
            load(0);
            m_half = fmaxf(m_half, top()) * P.scale_log2;
            const bool move = bar_or(1 + mb, m_half > m_used + kLazyLog2 || (m_used == -INFINITY && m_half > -INFINITY) || !ok);
            if (move) {
                S.xch[mb][hf][r128] = m_half;
                const bool all_ok = bar_and(3 + mb, 256, ok);
                if (!all_ok) { ok = false; break; }              // (the same verdict for the whole block)
                const float m_new = fmaxf(m_used, fmaxf(m_half, S.xch[mb][hf ^ 1][r128]));
                float alpha = 1.f;
                if (m_used == -INFINITY) m_used = m_new;         // nothing accumulated for this row yet
                else if (m_new > m_used + kLazyLog2) {
                    alpha = at_exp2(m_used - m_new);
                    m_used = m_new;
                }
                lsum *= alpha;
                if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                    // O is at rest between the previous tile's product and this tile's
                    if (!__all_sync(0xffffffffu, at_wait(S, &S.o_ready[mb], (uint32_t)(i - 1) & 1u))) ok = false;   // (ends at the next tile)
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int ch = 0; ch < 8; ++ch) tmem_scale8(colO + 8u * ch, alpha);      // (few registers: the row's logits are live)
                }
            }
            const float z = m_used == -INFINITY ? 0.f : m_used;
            const uint64_t nz2 = pack_f2(-z, -z);
            uint64_t ps[2] = {0ull, 0ull};
            auto put = [&](uint32_t c0) {       // P of the columns in sv -> 16 columns of the half's own part of S
                uint32_t pk[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float x0, x1;
                    unpack_f2(fma_f2(pack_f2(sv[2 * e], sv[2 * e + 1]), sc2, nz2), x0, x1);
                    const float p0 = at_exp2(x0), p1 = at_exp2(x1);
                    ps[e & 1] = add_f2(ps[e & 1], pack_f2(p0, p1));
                    pk[e] = pack_half2(p0, p1);
                }
                tmem_st16(sS + c0, pk);
            };
            put(0u);
            load(32);
            put(16u);
            float a0, a1;
            unpack_f2(add_f2(ps[0], ps[1]), a0, a1);
            lsum += a0 + a1;
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(&S.p_ready[mb]);
        }
        // ---- normalise, rotate, write ----
        if (n_t > 0 && ok) {
            ok = __all_sync(0xffffffffu, at_wait(S, &S.o_ready[mb], (uint32_t)(n_t - 1) & 1u));
            tc_fence_after_sync();
        }
        S.xch[mb][hf][r128] = lsum;
        if (!bar_and(3 + mb, 256, ok)) ok = false;
        lsum += S.xch[mb][hf ^ 1][r128];
        const float inv = lsum > 0.f ? 1.0f / lsum : 0.f;
        float out_scale = inv;
        if (P.rots && n_t > 0 && ok) {
#pragma unroll 1
            for (int ch = 0; ch < 2; ++ch) {
                float o[32];
                uint32_t hi[16], lo[16];
                tmem_ld32(colO + 32u * ch, o);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float x0 = o[2 * e] * inv, x1 = o[2 * e + 1] * inv;
                    const __half2 h2 = __floats2half2_rn(x0, x1);
                    const float2 hf2 = __half22float2(h2);
                    hi[e] = *reinterpret_cast<const uint32_t*>(&h2);
                    lo[e] = pack_half2(x0 - hf2.x, x1 - hf2.y);
                }
                tmem_st16(colS + 64u * hf + 16u * ch, hi);
                tmem_st16(colS + 64u * hf + 32u + 16u * ch, lo);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(&S.p_ready[mb]);
            ok = __all_sync(0xffffffffu, at_wait(S, &S.o_ready[mb], (uint32_t)n_t & 1u));
            tc_fence_after_sync();
            out_scale = 1.0f / kRotScale;
        }
        if (ok) {
            const int hq = h * P.gqa + g - pos * P.gqa;
            const size_t orow = ((size_t)b * P.n_q + hq) * P.s_q + pos;
            const size_t srow = P.n_splits > 1 ? (size_t)sp * gridDim.z * P.n_q * P.s_q + orow : orow;
#pragma unroll 1
            for (int ch = 0; ch < 2; ++ch) {
                float o[32];
                if (n_t > 0) {
                    tmem_ld32(colO + 32u * ch, o);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int c = 0; c < 32; ++c) o[c] = 0.f;
                }
                const int d0 = 64 * hf + 32 * ch;
                if (rok && P.out32) {
                    float4* dst = reinterpret_cast<float4*>(P.out32 + srow * kHD + d0);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        dst[c] = make_float4(o[4 * c] * out_scale, o[4 * c + 1] * out_scale, o[4 * c + 2] * out_scale, o[4 * c + 3] * out_scale);
                }
                if (rok && P.out16) {
                    uint4* dst = reinterpret_cast<uint4*>(P.out16 + orow * kHD + d0);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        dst[c] = make_uint4(pack_half2(o[8 * c] * out_scale, o[8 * c + 1] * out_scale),
                                            pack_half2(o[8 * c + 2] * out_scale, o[8 * c + 3] * out_scale),
                                            pack_half2(o[8 * c + 4] * out_scale, o[8 * c + 5] * out_scale),
                                            pack_half2(o[8 * c + 6] * out_scale, o[8 * c + 7] * out_scale));
                }
            }
            if (rok && hf == 0 && P.lse2) P.lse2[srow] = lsum > 0.f ? m_used + log2f(lsum) : -INFINITY;
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kWarpMma) tmem_dealloc(tmem, kTmemCols);
    if (tid == 0 && S.failed) atomicExch(&g_pf5_status, kStatusWaitTimeout);
}

// ------------------------------------------------------------------------------------------------------------------
// merge: one warp per output row adds the splits' partials (each normalised, with the log2 of its denominator).
// ------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) pf_merge_kernel(const float* part, const float* lse2, int64_t n_rows, int n_splits, __half* out16,
                                                       float* out32) {
    grid_dependency_wait();
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= n_rows) return;
    float mx = -INFINITY;
    for (int s = 0; s < n_splits; ++s) mx = fmaxf(mx, lse2[s * n_rows + row]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float den = 0.f;
    if (mx > -INFINITY) {
        for (int s = 0; s < n_splits; ++s) {
            const float w = at_exp2(lse2[s * n_rows + row] - mx);
            const float4 v = reinterpret_cast<const float4*>(part + (s * n_rows + row) * kHD)[lane];
            den += w;
            acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
        }
    }
    const float inv = den > 0.f ? 1.0f / den : 0.f;
    acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
    if (out32) reinterpret_cast<float4*>(out32 + row * kHD)[lane] = acc;
    if (out16) reinterpret_cast<uint2*>(out16 + row * kHD)[lane] = make_uint2(pack_half2(acc.x, acc.y), pack_half2(acc.z, acc.w));
}

// ------------------------------------------------------------------------------------------------------------------
// rotate: many query rows of one KV head into the packed-K basis, q_rot[p] = sum_d q[d] . W[d][p] with W's rows in the
// order of the query's own dims (the permutation moves rows of the small matrix instead of columns of the large one).
// W is held as high + low fp16 parts (x is fp16 already): two products per 128 rows, fp32 accumulation, what is dropped is
// 2^-22 of a value.  A CTA keeps W in shared memory and works with two groups of four warps, each on its own tiles:
// rows arrive by cp.async one tile ahead, leave through the tile's own buffer as whole 16-byte chunks.  Bound: memory,
// 512 bytes per row (a gather, an fp32 copy, an fp32 GEMM and a conversion of 16384 x 32 rows took 965 us).
// ------------------------------------------------------------------------------------------------------------------
constexpr int kRotThreads = 256;
struct RotSmem {
    __align__(128) uint8_t w[2][kPart];             // high, low
    __align__(128) uint8_t a[2][2][kPart];          // per group: two row tiles
    __align__(8) uint64_t bar[2];
    uint32_t tmem_base;
    uint8_t inv[kHD];
};
static_assert(sizeof(RotSmem) > 114 * 1024 && sizeof(RotSmem) <= 227 * 1024, "one CTA per SM");

__global__ void __launch_bounds__(kRotThreads, 1) rotate_rows_kernel(const BgtqHeadDesc* desc, const float* rot_k, const __half* q,
                                                                     int64_t q_sb, int64_t q_sh, int64_t q_ss, __half* out, int n_q,
                                                                     int gqa, int n_pos) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    RotSmem& S = *reinterpret_cast<RotSmem*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, grp = warp >> 2, gt = tid & 127;
    const int h = blockIdx.y, b = blockIdx.z;
    const int n_rows = gqa * n_pos, n_tiles = (n_rows + 127) / 128;       // row = head of the group * n_pos + position
    grid_launch_dependents();
    if (tid == 0) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&S.tmem_base, 256);
    if (tid < kHD) S.inv[desc[h].head_perm[tid]] = (uint8_t)tid;
    grid_dependency_wait();
    const __half* const src = q + b * q_sb + (int64_t)h * gqa * q_sh;
    __half* const dst = out + ((size_t)b * n_q + (size_t)h * gqa) * n_pos * kHD;
    auto fetch = [&](int tile, int buf) {
        const uint32_t base = smem_u32(S.a[grp][buf]);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int row = i * 8 + (gt >> 4), kc = gt & 15, g = tile * 128 + row;
            const int head = g < n_rows ? g / n_pos : 0, pos = g < n_rows ? g - head * n_pos : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (row >> 3) * 2048 + kc * 128 + (row & 7) * 16),
                         "l"(src + head * q_sh + pos * q_ss + kc * 8), "r"(g < n_rows ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int step = 2 * gridDim.x;
    int tile = 2 * blockIdx.x + grp;
    if (tile < n_tiles) fetch(tile, 0);
    __syncthreads();
    // operand (n, k) = W[k][n], 16 bytes = eight k of one n
    const float* W = rot_k + (size_t)h * kHD * kHD;
#pragma unroll 2
    for (int i = tid; i < kHD * kHD / 8; i += kRotThreads) {
        const int n = i & (kHD - 1), k8 = i >> 7;
        __align__(16) __half hi[8], lo[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float w = __ldg(W + (size_t)S.inv[8 * k8 + e] * kHD + n) * kRotScale;
            hi[e] = __float2half_rn(w);
            lo[e] = __float2half_rn(w - __half2float(hi[e]));
        }
        const uint32_t o = (n >> 3) * 2048 + k8 * 128 + (n & 7) * 16;
        *reinterpret_cast<uint4*>(S.w[0] + o) = *reinterpret_cast<uint4*>(hi);
        *reinterpret_cast<uint4*>(S.w[1] + o) = *reinterpret_cast<uint4*>(lo);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t acc = S.tmem_base + 128u * grp, tlane = acc + ((uint32_t)((warp & 3) * 32) << 16);
    bool ok = true;
    for (int it = 0; tile < n_tiles; tile += step, ++it) {
        uint8_t* const a = S.a[grp][it & 1];
        if (tile + step < n_tiles) {
            fetch(tile + step, (it + 1) & 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before_sync();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
        if ((warp & 3) == 0) {
            tc_fence_after_sync();
            const uint32_t lead = elect_one();
            const uint64_t ad = op_desc(smem_u32(a)), w0 = op_desc(smem_u32(S.w[0])), w1 = op_desc(smem_u32(S.w[1]));
#pragma unroll
            for (int ks = 0; ks < kHD / 16; ++ks) mma_ss(acc, ad + 16u * ks, w1 + 16u * ks, ks > 0, lead);
#pragma unroll
            for (int ks = 0; ks < kHD / 16; ++ks) mma_ss(acc, ad + 16u * ks, w0 + 16u * ks, 1u, lead);
            if (lead) umma_commit(&S.bar[grp]);
            __syncwarp();
        }
        ok = bar_and(3 + grp, 128, mbar_wait_bounded(&S.bar[grp], it & 1));      // one verdict for the group
        if (!ok) break;
        tc_fence_after_sync();
        // row gt of the tile -> its buffer (chunk c of row r at chunk c ^ (r & 7)), then whole chunks out
#pragma unroll
        for (int ch = 0; ch < kHD / 32; ++ch) {
            float o[32];
            tmem_ld32(tlane + 32u * ch, o);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                constexpr float s = 1.0f / kRotScale;
                *reinterpret_cast<uint4*>(a + gt * 256 + (((4 * ch + c) ^ (gt & 7)) << 4)) =
                    make_uint4(pack_half2(o[8 * c] * s, o[8 * c + 1] * s), pack_half2(o[8 * c + 2] * s, o[8 * c + 3] * s),
                               pack_half2(o[8 * c + 4] * s, o[8 * c + 5] * s), pack_half2(o[8 * c + 6] * s, o[8 * c + 7] * s));
            }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
#pragma unroll 4
        for (int i = gt; i < 128 * 16; i += 128) {
            const int row = i >> 4, c = i & 15;
            if (tile * 128 + row < n_rows)
                *reinterpret_cast<uint4*>(dst + ((size_t)tile * 128 + row) * kHD + c * 8) =
                    *reinterpret_cast<const uint4*>(a + row * 256 + ((c ^ (row & 7)) << 4));
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");        // the buffer is refilled two tiles on
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(S.tmem_base, 256);
    if (!ok && gt == 0) atomicExch(&g_pf5_status, kStatusWaitTimeout);
}

int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
}

UpRaw raw_layout(const PfParams& P) {
    auto r16 = [](uint32_t x) { return (x + 15u) & ~15u; };
    UpRaw R;
    R.k = 0;
    R.kn = R.k + r16((uint32_t)kT5Tok * P.kp_st + 8u);
    R.v = R.kn + r16((uint32_t)kT5Tok * P.kn_st + 8u);
    R.vn = R.v + r16((uint32_t)kT5Tok * P.vp_st + 8u);
    R.total = R.vn + r16((uint32_t)kT5Tok * P.vn_st + 8u);
    return R;
}

}  // namespace

// Into how many pieces the cache of each query block is cut: as many as make the launch shortest.  A CTA costs its
// tiles and about three tiles' time for its queries and output.  Where all blocks have the same tiles (few positions
// behind a long cache) the launch takes whole waves of CTAs; where their number falls from the last block to the first
// (causal, no cache) the hardware's own scheduling, longest first, evens them out and the average decides.
int prefill_t5_splits(int n_batch, int n_kv, int gqa, int s_q, int n_tok, int q_pos_offset, bool causal) {
    const int64_t rows = (int64_t)s_q * gqa, per_pair = (rows + 255) / 256, blocks = per_pair * n_kv * n_batch;
    const int sms = sm_count();
    auto tiles_of = [&](int64_t pos) {
        const int64_t t = causal && pos < n_tok ? pos : n_tok;
        return (double)((t + kT5Tok - 1) / kT5Tok);
    };
    const double most = tiles_of((int64_t)q_pos_offset + s_q), least = tiles_of((int64_t)q_pos_offset + (255 / gqa < s_q ? 255 / gqa : s_q));
    const double avg = 0.5 * (most + least), even = most > 0 ? least / most : 1.0;
    int best = 1;
    double cost = 0;
    for (int s = 1; s <= 16 && s <= (most + 1) / 2 && (s == 1 || blocks * (s - 1) < 2 * (int64_t)sms); ++s) {
        const double waves = (double)((blocks * s + sms - 1) / sms) * (most / s + 3);
        const double fill = blocks * s * (avg / s + 3) / sms, longest = most / s + 3;
        const double c = even * waves + (1 - even) * (fill > longest ? fill : longest) + (s > 1 ? 1 : 0);
        if (s == 1 || c < 0.97 * cost) {
            best = s;
            cost = c;
        }
    }
    return best;
}

int64_t prefill_t5_workspace(int n_batch, int n_q, int n_kv, int s_q, int n_tok, int q_pos_offset, bool causal, bool rot) {
    const int64_t tiles = (n_tok + kT5Tok - 1) / kT5Tok;
    const int splits = prefill_t5_splits(n_batch, n_kv, n_q / n_kv, s_q, n_tok, q_pos_offset, causal);
    int64_t n = (int64_t)n_batch * n_kv * tiles * kTileBytes + (rot ? (int64_t)n_kv * 2 * kPart : 0);
    if (splits > 1) n += (int64_t)splits * n_batch * n_q * s_q * (kHD + 1) * 4;
    return n;
}

// P.out is ignored: the result goes to out16 and / or out32.
cudaError_t launch_prefill_t5(const PfParams& P, int n_batch, const float* v_rot, uint8_t* ws, __half* out16, float* out32,
                              cudaStream_t stream) {
    const UpRaw R = raw_layout(P);
    const size_t smem_up = sizeof(UpSmem) + 2u * (size_t)R.total;
    const int n_tiles = (P.n_tok + kT5Tok - 1) / kT5Tok, sms = sm_count();
    uint8_t* const tiles = ws;
    uint8_t* const rots = ws + (size_t)n_batch * P.n_kv * n_tiles * kTileBytes;
    // a few tiles per CTA when there are many (its tables are made once), one each otherwise
    const int64_t all = (int64_t)n_tiles * P.n_kv * n_batch;
    const int per_cta = (int)(all > 2 * sms ? (all + 2 * sms - 1) / (2 * sms) : 1);
    const int ctas = (n_tiles + per_cta - 1) / per_cta;
    cudaError_t e = cudaFuncSetAttribute(pf_unpack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_up);
    if (e == cudaSuccess && n_tiles > 0)
        e = launch_kernel(pf_unpack_kernel, dim3(ctas + (v_rot ? 1 : 0), P.n_kv, n_batch), dim3(kUpThreads), smem_up, stream, true, P, R,
                          tiles, rots, v_rot, per_cta);
    if (e != cudaSuccess) return e;

    AtParams A;
    A.q = P.q; A.q_sb = P.q_sb; A.q_sh = P.q_sh; A.q_ss = P.q_ss;
    A.tiles = tiles; A.rots = v_rot ? rots : nullptr;
    A.n_q = P.n_q; A.n_kv = P.n_kv; A.gqa = P.gqa; A.s_q = P.s_q; A.n_tok = P.n_tok; A.q_pos_offset = P.q_pos_offset;
    A.causal = P.causal; A.scale_log2 = P.scale_log2;
    A.n_splits = prefill_t5_splits(n_batch, P.n_kv, P.gqa, P.s_q, P.n_tok, P.q_pos_offset, P.causal != 0);
    A.n_qblk = (int)(((int64_t)P.s_q * P.gqa + 255) / 256);
    const int64_t rows = (int64_t)n_batch * P.n_q * P.s_q;
    float* const part = reinterpret_cast<float*>(rots + (v_rot ? (size_t)P.n_kv * 2 * kPart : 0));
    const bool split = A.n_splits > 1;
    A.out16 = split ? nullptr : out16;
    A.out32 = split ? part : out32;
    A.lse2 = split ? part + (size_t)A.n_splits * rows * kHD : nullptr;
    e = cudaFuncSetAttribute(pf_attend_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AtSmem));
    if (e != cudaSuccess) return e;
    e = launch_kernel(pf_attend_kernel, dim3((unsigned)A.n_qblk * A.n_splits, P.n_kv, n_batch), dim3(kAtThreads), sizeof(AtSmem), stream,
                      true, A);
    if (e != cudaSuccess || !split) return e;
    return launch_kernel(pf_merge_kernel, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, stream, true, (const float*)part,
                         (const float*)A.lse2, rows, (int)A.n_splits, out16, out32);
}

}  // namespace bgtq

extern "C" __attribute__((visibility("default"))) int bgtq_prefill_tcgen05_status(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, bgtq::g_pf5_status, sizeof(v)) != cudaSuccess) {
        cudaGetLastError();
        return BGTQ_E_LAUNCH;
    }
    return v;
}

extern "C" __attribute__((visibility("default"))) int bgtq_rotate_q_rows(const BgtqHeadDesc* desc, const float* rot_k, const void* q,
                                                                         int64_t q_sb, int64_t q_sh, int64_t q_ss, void* q_rot,
                                                                         int32_t n_batch, int32_t n_q, int32_t n_kv, int32_t n_pos,
                                                                         void* stream) {
    using namespace bgtq;
    if (!desc || !rot_k || !q || !q_rot || n_batch < 1 || n_kv < 1 || n_q < n_kv || n_q % n_kv || n_pos < 1) return BGTQ_E_BADARG;
    const int64_t rows = (int64_t)(n_q / n_kv) * n_pos, tiles = (rows + 127) / 128;
    if (rows > (1LL << 30) || n_batch > 65535 || n_kv > 65535) return BGTQ_E_TOOBIG;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(q_rot) | (uint64_t)(2 * q_sb) | (uint64_t)(2 * q_sh) |
         (uint64_t)(2 * q_ss)) & 15u)
        return BGTQ_E_ALIGN;
    // one CTA per SM, two tiles of it at a time
    int64_t per = sm_count() / ((int64_t)n_kv * n_batch);
    if (per < 1) per = 1;
    if (per > (tiles + 1) / 2) per = (tiles + 1) / 2;
    if (cudaFuncSetAttribute(rotate_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RotSmem)) != cudaSuccess ||
        launch_kernel(rotate_rows_kernel, dim3((unsigned)per, n_kv, n_batch), dim3(kRotThreads), sizeof(RotSmem),
                      static_cast<cudaStream_t>(stream), true, desc, rot_k, static_cast<const __half*>(q), q_sb, q_sh, q_ss,
                      static_cast<__half*>(q_rot), n_q, n_q / n_kv, n_pos) != cudaSuccess) {
        cudaGetLastError();
        return BGTQ_E_LAUNCH;
    }
    return BGTQ_OK;
}
