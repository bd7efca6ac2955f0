// Bulk (prefill) encoder: rotation on tcgen05, then one pass of a thread over its part of a row.
//
//   * a CTA of 16 warps works on tiles of 128 rows of one (KV head, K or V); the rotation W is staged once as
//     hi = fp16(W), lo = fp16((W - hi) * 2^10) in the tensor cores' operand layout;
//   * the warps form two groups of eight, which run out of phase, each on its own tiles (a CTA with a single tile: all sixteen
//     on it): rows arrive by cp.async a tile ahead (V: straight into the operand's swizzled layout; K: and move on into packed
//     order, the two dims of a RoPE pair as one word), two warps issue 8 tcgen05.mma each (x . hi and x . lo into 2 x 128
//     tensor-memory columns), and meanwhile all warps sum the rows' group norms;
//   * then thread (row, half or quarter) takes its part of the row's columns eight at a time straight from tensor memory
//     (tcgen05.ld of one lane): the row is the thread's own, so everything that depends on the column (segment, bin grid, code
//     width, byte position) is uniform over the warp and comes ready made from a list (E5Rec), codes never leave registers, two
//     values share an instruction where they can (f32x2), and whole 32-bit words of the packed row go to a staging image of the
//     tile that leaves as coalesced words.
// Bound: instruction issue and its latencies with 16 warps per SM (all registers and shared memory are taken): 1 048 576 K and
// as many V rows take 374 us (451 with every thread working out each task's control; K rows alone 219 and 286, V rows 162 and
// 164), where the bytes alone would take 100; 777 tokens of 8 heads, a tile per CTA, 8.5 us (10.8 with half of the warps on it).
// The sums that decide a code (group norms, products) keep the order they had: the packed bytes are bit for bit the same.
// Every wait is bounded; tensor memory is released on every path out of the kernel.
#include <atomic>
#include <cstddef>
#include <type_traits>

#include "bgtq_common.cuh"
#include "bgtq_encode_params.cuh"
#include "bgtq_tcgen05.cuh"

namespace bgtq {
// Sticky error word of this kernel: set when a wait for the tensor cores ran out.
__device__ int g_enc5_status = 0;

namespace {

constexpr int kThreads = 512;
constexpr int kGroup = 256;                     // threads of a group
constexpr int kTileRows = 128;                  // = tensor-memory lanes
constexpr int kTile = kTileRows * kHD * 2;      // bytes of a row tile
constexpr int kMaxTasks = 40;           // 128 / 4 + one remainder per segment
constexpr int kLevelOff = kTileRows * (kHD + 4) + 16;       // past the widest staged rows
static_assert(kLevelOff + 2 * BGTQ_MAX_SEGMENTS * kTileRows * 4 <= kTile, "staged rows and level sums fit the operand tile");
constexpr float kLoScale = 1024.0f;
constexpr uint32_t kTmemCols = 512;             // per group: hi accumulator 128 columns + lo accumulator 128 columns
constexpr int kSeg = BGTQ_MAX_SEGMENTS;
constexpr int kLutLd = BGTQ_N_BINS + 4;

// What the packing of a task (E5Smem::tasks) needs, ready made: read by all lanes at one address, in two 16-byte loads.
struct __align__(16) E5Rec {
    uint32_t col;       // first column to load | 2 (first column of the task - that) << 8: a last short task loads from column 120
    uint32_t mask;      // the valid bits of its code word
    uint32_t lut;       // shared address of its segment's code table
    uint32_t part;      // byte offset of its segment's row factors
    float off, scale;   // bin = (y + off) * scale, in units of 256 bins
    uint32_t mul;       // 2^(stored bits)
    uint32_t ctl;       // bit position in its first word | 256 where it completes that word | byte offset of the word in the row << 16
};
struct E5Smem {
    __align__(128) uint8_t w_hi[kTile];
    __align__(128) uint8_t w_lo[kTile];
    // Row tiles of each group, in the tensor cores' 128-byte-swizzle layout: 16-byte chunk c of row r at
    // (c / 8) * 16384 + r * 128 + ((c % 8) ^ (r % 8)) * 16.  V: two operand tiles, used in turn.  K: [0] = rows as they come,
    // [1] = operand, columns in packed order.  After the product the operand tile holds the staged packed rows.
    __align__(1024) uint8_t buf[2][2][kTile];
    // per group: the two partial sums of squares of a (segment, row), replaced by its group norm and by 1 / norm (or 1
    // where the norm is below the floor)
    float part[2][2][kSeg][kTileRows];
    float vtab[32];                                 // V: boundaries, levels (sixteen neighbouring words: lookups never collide)
    float kcent[512];
    uint8_t code_lut[kSeg][kLutLd];                 // K: entry 256 = entry 255
    float2 grid[kSeg];                              // K, in units of 256 bins: {offset, 1 / range}
    // Up to eight consecutive codes of one segment, at most 32 bits: first column | count << 8 | stored bits << 12 | segment << 16
    // | bytes << 20.  A K row's tasks follow each other in its bytes; its threads take equal numbers of them.
    uint32_t tasks[kMaxTasks];
    E5Rec rec[kMaxTasks];
    int32_t cut[5], cut_byte[5];                    // K: first task of each quarter of the tasks, and its first byte
    int32_t row_bytes, n_seg, paired, v_sb, v_bits;
    int32_t seg_start[kSeg], seg_len[kSeg], seg_bw[kSeg], seg_lut_off[kSeg];
    __align__(16) uint16_t to[kHD];                 // K: operand offset (row 0) of an input column, its packed position's place
    __align__(8) uint64_t mma_bar[2];
    uint32_t tmem_base;
};
static_assert(sizeof(E5Rec) == 32 && offsetof(E5Smem, rec) % 16 == 0 && offsetof(E5Smem, to) % 16 == 0, "loaded 16 bytes at a time");
static_assert(sizeof(E5Smem) > 114 * 1024 && sizeof(E5Smem) <= 227 * 1024, "exactly one CTA per SM (it takes all tensor memory)");

// Shared addresses of entries trunc(256 v) of a byte table at `table`, for two values already saturated to [0, 1].  An
// address is an integer, and as the bits of a float a multiple of the smallest subnormal: 256 v added to it in those units and
// rounded toward zero is the entry's address.  v = 1 reads entry 256, a copy of entry 255.
__device__ __forceinline__ void bin_addr2(float v0, float v1, uint32_t table, uint32_t& a0, uint32_t& a1) {
    const float t = __uint_as_float(table), step = __uint_as_float(256u);
    float b0, b1;
    unpack_f2(fma_rz_f2(pack_f2(v0, v1), pack_f2(step, step), pack_f2(t, t)), b0, b1);
    a0 = __float_as_uint(b0);
    a1 = __float_as_uint(b1);
}
__device__ __forceinline__ uint32_t lds8(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float lds_f(uint32_t addr) {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
// eight fp32 columns of this thread's tensor-memory lane (no wait)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void group_sync(int grp) { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kGroup) : "memory"); }

// eight codes, LSB first, `m` = 2^(stored bits); what does not fit 32 bits is zero
__device__ __forceinline__ uint32_t squeeze8(const uint32_t (&c)[8], uint32_t m) {
    uint32_t w = c[7];
#pragma unroll
    for (int e = 6; e >= 0; --e) w = w * m + c[e];
    return w;
}

// The same of 4 x the codes (stored bits at most 4).
__device__ __forceinline__ uint32_t squeeze8_4(const uint32_t (&c)[8], uint32_t m) {
    uint32_t w = c[7];
#pragma unroll
    for (int e = 6; e >= 1; --e) w = w * m + c[e];
    return (w >> 2) * m + (c[0] >> 2);
}

// A thread's part of a packed row on its way into the staging image: bytes are appended, whole words stored.  Staged rows
// start on word boundaries, so that the position inside a word is the same for every row and all control is uniform.
struct ByteStream {
    uint32_t addr;      // shared address of the word being filled
    uint32_t acc, pos;  // its bits so far
    uint32_t skip;      // bits of the first word that belong to the part before
    __device__ __forceinline__ void open(uint32_t row_addr, uint32_t byte) {
        addr = row_addr + (byte & ~3u);
        pos = skip = (byte & 3u) * 8u;
        acc = 0u;
    }
    __device__ __forceinline__ void bytes(uint32_t lo, uint32_t hi) {
#pragma unroll 1
        for (uint32_t b = lo; b < hi; b += 8u) asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr + (b >> 3)), "r"(acc >> b) : "memory");
    }
    __device__ __forceinline__ void put(uint32_t w, uint32_t n_bits) {      // n_bits a multiple of 8, at most 32; w has no bits past them
        acc |= w << pos;
        const uint32_t old = pos;
        pos += n_bits;
        if (pos >= 32u) {
            if (skip) {
                bytes(skip, 32u);
                skip = 0u;
            } else {
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(acc) : "memory");
            }
            addr += 4u;
            acc = __funnelshift_rc(w, 0u, 32u - old);       // what did not fit (old = 0: nothing)
            pos -= 32u;
        }
    }
    // a task's code word (see E5Rec::ctl)
    __device__ __forceinline__ void word(uint32_t w, uint32_t ctl, uint32_t row_addr) {
        const uint32_t at = ctl & 31u;
        acc |= w << at;
        if (ctl & 256u) {
            addr = row_addr + (ctl >> 16);
            if (skip) {
                bytes(skip, 32u);
                skip = 0u;
            } else {
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(acc) : "memory");
            }
            acc = __funnelshift_rc(w, 0u, 32u - at);       // what did not fit (position 0: nothing)
        }
    }
    __device__ __forceinline__ void end_at(uint32_t row_addr, uint32_t byte) {
        addr = row_addr + (byte & ~3u);
        pos = (byte & 3u) * 8u;
    }
    __device__ __forceinline__ void close() { bytes(skip, pos); }
};

// Per-CTA tables: rotation split into the operand layout, bin tables, tasks.  (A few microseconds of every launch: descriptor
// fields come to shared memory first, all loads at once, and the lists are made by a warp, not by one thread.)
__device__ void e5_setup(E5Smem& S, const EncParams& P, const BgtqHeadDesc& d, bool is_v, int h) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < kSeg) {
        S.seg_start[tid] = d.seg_start[tid];
        S.seg_len[tid] = d.seg_len[tid];
        S.seg_bw[tid] = d.seg_bw[tid];
        S.seg_lut_off[tid] = d.seg_lut_off[tid];
        if (!is_v) S.grid[tid] = make_float2(d.lut_off[tid], d.lut_inv[tid] * (1.0f / 256.0f));      // (a power of two: exact)
    }
    if (tid == 32) {
        S.n_seg = is_v ? 1 : d.n_seg;
        S.v_sb = (P.flags & BGTQ_ENC_V_NIBBLE) ? 4 : d.v_bits;
        S.v_bits = d.v_bits;
    }
    if (tid < kHD) S.to[d.head_perm[tid] & (kHD - 1)] = (uint16_t)((tid >> 6) * 16384 + ((tid >> 3) & 7) * 16 + (tid & 7) * 2);
    if (is_v) {
        if (tid < 32) S.vtab[tid] = tid < 16 ? d.v_bounds[tid] : d.v_cents[tid - 16];
    } else {
        *reinterpret_cast<uint32_t*>(&S.code_lut[tid >> 6][4 * (tid & 63)]) = reinterpret_cast<const uint32_t*>(&d.code_lut[0][0])[tid];
        S.kcent[tid] = d.k_cents[tid];
    }
    // operand row n (output position), eight k at a time: W[k][n] is coalesced over n, 16 bytes go to shared memory
    const float* W = (is_v ? P.rot_v : P.rot_k) + (size_t)h * kHD * kHD;
#pragma unroll
    for (int u = 0; u < kHD * kHD / 8 / kThreads; ++u) {
        const int i = tid + u * kThreads, n = i & (kHD - 1), k8 = i >> 7;
        __align__(16) __half hi[8], lo[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float w = __ldg(W + (size_t)(8 * k8 + e) * kHD + n);
            hi[e] = __float2half_rn(w);
            lo[e] = __float2half_rn((w - __half2float(hi[e])) * kLoScale);
        }
        const uint32_t o = (uint32_t)((n >> 3) * 2048 + k8 * 128 + (n & 7) * 16);
        *reinterpret_cast<uint4*>(S.w_hi + o) = *reinterpret_cast<uint4*>(hi);
        *reinterpret_cast<uint4*>(S.w_lo + o) = *reinterpret_cast<uint4*>(lo);
    }
    // RoPE pairs (dims i, i + 64) side by side in packed order, as the reference's calibration lays every head out
    const bool pair = tid >= kHD / 2 || (d.head_perm[2 * tid] < kHD / 2 && d.head_perm[2 * tid + 1] == d.head_perm[2 * tid] + kHD / 2);
    const int paired = __syncthreads_and(is_v || pair);
    if (is_v) {
        if (tid == 0) S.row_bytes = seg_storage_bytes(S.v_sb, kHD);
    } else {
        if (tid < kSeg) S.code_lut[tid][BGTQ_N_BINS] = S.code_lut[tid][BGTQ_N_BINS - 1];
        const int n_seg = S.n_seg;
        if (warp == 0) {        // lane = segment: its tasks behind those of the segments before
            const bool live = lane < n_seg;
            const int st = live ? S.seg_start[lane] : 0, len = live ? S.seg_len[lane] : 0, bw = live ? S.seg_bw[lane] : 1;
            const int sb = (P.flags & BGTQ_ENC_K_MIXED) ? (bw <= 4 ? 4 : 8) : (bw <= 4 ? bw : 8), per = sb == 8 ? 4 : 8;
            auto n_bytes = [&](int n) { return sb == 3 ? 3 : (n * sb + 7) >> 3; };
            const int nt = (len + per - 1) / per;
            int t_at = nt;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const int tu = __shfl_up_sync(0xffffffffu, t_at, o);
                if (lane >= o) t_at += tu;
            }
            const int n_tasks = __shfl_sync(0xffffffffu, t_at, n_seg - 1);
            t_at -= nt;
#pragma unroll 1
            for (int c = 0; c < nt; ++c) {
                const int first = st + per * c, n = min(per, len - per * c);
                S.tasks[t_at + c] = (uint32_t)first | (uint32_t)n << 8 | (uint32_t)sb << 12 | (uint32_t)lane << 16 | (uint32_t)n_bytes(n) << 20;
            }
            __syncwarp();
            int at = 0;
#pragma unroll 1
            for (int base = 0; base < n_tasks; base += 32) {        // lane = task
                const int t = base + lane;
                const uint32_t task = t < n_tasks ? S.tasks[t] : 0u;
                const int nb = (int)(task >> 20);
                int end = nb;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xffffffffu, end, o);
                    if (lane >= o) end += x;
                }
                const int byte = at + end - nb;
                at += __shfl_sync(0xffffffffu, end, 31);
                if (t < n_tasks) {
                    const int first = task & 0xFF, bits = (int)((task >> 8) & 15u) * (int)((task >> 12) & 15u), seg = (task >> 16) & 15u;
                    const int col = min(first, kHD - 8), pos = 8 * (byte & 3);
                    E5Rec r;
                    r.col = (uint32_t)col | (uint32_t)(first - col) << 8;
                    r.mask = bits >= 32 ? ~0u : (1u << bits) - 1u;
                    r.lut = smem_u32(S.code_lut[seg]);
                    r.part = (uint32_t)(seg * kTileRows * 4);
                    r.off = -S.grid[seg].x;
                    r.scale = S.grid[seg].y;
                    r.mul = 1u << ((task >> 12) & 15u);
                    r.ctl = (uint32_t)pos | (pos + 8 * nb >= 32 ? 256u : 0u) | (uint32_t)(byte & ~3) << 16;
                    S.rec[t] = r;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (t == (n_tasks * k + 2) / 4) {
                            S.cut[k] = t;
                            S.cut_byte[k] = byte;
                        }
                }
            }
            if (lane == 0) {
                S.cut[4] = n_tasks;
                S.cut_byte[4] = at;
                S.row_bytes = P.kp_row_bytes;
                S.paired = paired;
#pragma unroll 1
                for (int k = 1; k < 4; ++k)         // (fewer than two tasks: empty quarters)
                    if ((n_tasks * k + 2) / 4 >= n_tasks) {
                        S.cut[k] = n_tasks;
                        S.cut_byte[k] = at;
                    }
            }
        }
    }
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// acc + x0^2 + x1^2 of two fp16 values, in that order (fp16 -> fp32 is exact: the same bits as converting first)
__device__ __forceinline__ float square2(float acc, uint32_t w) {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tfma.rn.f32.f16 %0, l, l, %0;\n\tfma.rn.f32.f16 %0, h, h, %0;\n\t}" : "+f"(acc) : "r"(w));
    return acc;
}

// Columns [first, first + 8 N) of a V row, of one thread's tensor-memory lane -> its bytes in the staged row; returns the sum
// of the squared levels (added up quarter by quarter).  A code counts the boundaries below a value: the upper halvings of
// the search are compares with boundaries in registers, the last one (of 4 bits: two) looks its boundary up: few lookups, as the
// other group's K tile shares their pipe (with a table of 256 bins K and V rows together take 380 us, so 374).
template <int BITS, bool CODES, int N>
__device__ __forceinline__ float e5_cols_v(E5Smem& S, uint32_t lane_base, int first, float r, uint32_t row_addr, uint8_t* codes) {
    const char* const vt = reinterpret_cast<const char*>(S.vtab);       // byte 4 c: boundary c, 64 + 4 c: level c
    auto entry = [&](uint32_t at) { return *reinterpret_cast<const float*>(vt + at); };
    constexpr int kMid = (1 << (BITS - 1)) - 1;
    const float mid = S.vtab[kMid], low = BITS > 2 ? S.vtab[kMid / 2] : 0.f, high = BITS > 2 ? S.vtab[kMid + 1 + kMid / 2] : 0.f;
    const uint32_t sb = (uint32_t)S.v_sb, mul = 1u << sb;
    const uint32_t col = lane_base + (uint32_t)first;
    uint32_t addr = row_addr + sb * (uint32_t)first / 8u, acc = 0u, pos = 0u;
    const uint64_t r2 = pack_f2(r, r), scale2 = pack_f2(1.0f / kLoScale, 1.0f / kLoScale);
    uint64_t csq2 = 0ull;
    float csq = 0.f;
    float hi[2][8], lo[2][8];
    tmem_ld8(col, hi[0]);
    tmem_ld8(col + kHD, lo[0]);
#pragma unroll
    for (int t2 = 0; t2 < N; t2 += 2) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int ti = t2 + u;
            tmem_ld_wait();
            if (ti + 1 < N) {       // the next columns come while these are worked on
                tmem_ld8(col + 8u * (ti + 1), hi[u ^ 1]);
                tmem_ld8(col + kHD + 8u * (ti + 1), lo[u ^ 1]);
            }
            uint32_t c[8];          // 4 x codes
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                float y[2], cv[2];
                unpack_f2(mul_f2(fma_f2(pack_f2(lo[u][e], lo[u][e + 1]), scale2, pack_f2(hi[u][e], hi[u][e + 1])), r2), y[0], y[1]);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const bool up = y[k] > mid;
                    uint32_t cc = up ? 4u << (BITS - 1) : 0u;
                    if (BITS > 2 && y[k] > (up ? high : low)) cc += 2u << (BITS - 1);
                    if (BITS > 3 && y[k] > entry(cc + 4u)) cc += 8u;
                    if (BITS > 1 && y[k] > entry(cc)) cc += 4u;
                    c[e + k] = cc;
                    cv[k] = entry(64u + cc);
                }
                const uint64_t cv2 = pack_f2(cv[0], cv[1]);
                csq2 = fma_f2(cv2, cv2, csq2);
            }
            if (CODES && codes) {
#pragma unroll
                for (int e = 0; e < 8; ++e) codes[first + 8 * ti + e] = (uint8_t)(c[e] >> 2);
            }
            const uint32_t w = squeeze8_4(c, mul);
            acc |= w << pos;
            if (pos + 8u * sb >= 32u) {
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(acc) : "memory");
                addr += 4u;
                acc = __funnelshift_rc(w, 0u, 32u - pos);
            }
            pos = (pos + 8u * sb) & 31u;
        }
        if ((t2 & 3) == 2) {        // a quarter ends
            float s0, s1;
            unpack_f2(csq2, s0, s1);
            csq += s0 + s1;
            csq2 = 0ull;
        }
    }
    return csq;
}

// Sums of squares of segments first, first + step, .. of a K row: of its pairs 0, 2, .. and of its pairs 1, 3, .., each in
// order.  A 16-byte load brings four pairs, even and odd positions into a sum of their own; what belongs to a neighbour in a
// segment's first and last chunk counts as zero.  (4 x 32768 tokens x 8 heads of K rows: with E5Rec 286 -> 229 us.)
__device__ __forceinline__ void e5_norms_k(E5Smem& S, int grp, uint32_t tile, int row, int first, int step) {
    const uint32_t xr = tile + (uint32_t)row * 128u, sw = (uint32_t)(row & 7) << 4;
    const int n_seg = S.n_seg;
#pragma unroll 1
    for (int s = first; s < n_seg; s += step) {
        const int p0 = S.seg_start[s] >> 1, p1 = p0 + (S.seg_len[s] >> 1), c0 = p0 >> 2, c1 = (p1 - 1) >> 2;
        auto chunk = [&](int c) { return lds128(xr + (uint32_t)(c >> 3) * 16384u + (((uint32_t)(c & 7) << 4) ^ sw)); };
        float even = 0.f, odd = 0.f;        // of positions
        auto add = [&](const uint4& v) {
            even = square2(even, v.x);
            odd = square2(odd, v.y);
            even = square2(even, v.z);
            odd = square2(odd, v.w);
        };
        auto cut = [&](uint4 v, int c) {
            const uint32_t lo = (uint32_t)(p0 - 4 * c), n = (uint32_t)(p1 - p0);
            v.x = 0u - lo < n ? v.x : 0u;
            v.y = 1u - lo < n ? v.y : 0u;
            v.z = 2u - lo < n ? v.z : 0u;
            v.w = 3u - lo < n ? v.w : 0u;
            return v;
        };
        add(cut(chunk(c0), c0));
#pragma unroll 4
        for (int c = c0 + 1; c < c1; ++c) add(chunk(c));
        if (c1 > c0) add(cut(chunk(c1), c1));
        S.part[grp][0][s][row] = p0 & 1 ? odd : even;
        S.part[grp][1][s][row] = p0 & 1 ? even : odd;
    }
}

// operand descriptor of a tile in the 128-byte-swizzle layout; k-step ks of 16: see tile_step
__device__ __forceinline__ uint64_t tile_desc(uint32_t smem_addr) {
    return (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61) | (uint64_t)(smem_addr >> 4);
}
__device__ __forceinline__ uint32_t tile_step(int ks) { return (uint32_t)(ks >> 2) * (16384u >> 4) + (uint32_t)(ks & 3) * 2u; }
// Tiles [lo, hi) of one (head, K or V).  `n_mma`: products this thread's group has issued so far (the barrier's phase).
// ONE: the CTA's only tile, on which all sixteen warps work, a thread on a quarter of its row (a second group would have
// nothing to do, and the launch takes as long as one tile).
template <bool IS_V, bool MIXED, bool CODES, bool ONE>
__device__ __forceinline__ bool e5_role(E5Smem& S, const EncParams& P, const int h, const int lo_tile, const int hi_tile, int& n_mma,
                                        bool& waited) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kThr = ONE ? kThreads : kGroup, kWrp = kThr / 32;
    const int grp = ONE ? 0 : tid >> 8, gt = ONE ? tid : tid & (kGroup - 1);
    constexpr int kParts = kThr / kTileRows;                 // threads of a row: 2 or 4
    const int qf = (warp >> 2) & (kParts - 1), hf = qf & 1, row = (warp & 3) * 32 + lane;      // (a warp reads tensor-memory lanes 32 (warp % 4) .. + 31)
    const int n_rows = P.n_batch * P.n_tok;                  // the launcher checks that this fits
    const int t0 = P.pos_dev ? *P.pos_dev : P.t0;
    const uint32_t acc_hi = S.tmem_base + 256u * grp;
    const uint32_t lane_base = acc_hi + ((uint32_t)((warp & 3) * 32) << 16);
    uint64_t* const bar = &S.mma_bar[grp];
    const int n_seg = S.n_seg, rb = S.row_bytes;
    constexpr bool mixed = !IS_V && MIXED;
    const bool f16n = P.flags & BGTQ_ENC_K_NORMS_F16;
    const __half* const src_base = IS_V ? P.v + h * P.v_sh : P.k + h * P.k_sh;
    const int64_t s_sb = IS_V ? P.v_sb : P.k_sb, s_ss = IS_V ? P.v_ss : P.k_ss;
    uint8_t* const out_base = IS_V ? P.vp + h * P.vp_sh : P.kp + h * P.kp_sh;
    const int64_t o_sb = IS_V ? P.vp_sb : P.kp_sb, o_st = IS_V ? P.vp_st : P.kp_st;
    const uint32_t magic = ((1u << 24) + (uint32_t)rb - 1u) / (uint32_t)rb;      // x / rb = x * magic >> 24 below 128 rows
    const int stage_ld = 4 * (((rb + 3) >> 2) | 1);       // bytes between staged rows: an odd number of words
    const int q_lo = qf * (4 / kParts);                      // this thread's first quarter
    const int task_lo = S.cut[q_lo], task_hi = S.cut[q_lo + 4 / kParts], task_mid = S.cut[q_lo + 1];
    auto tile_sync = [&]() {
        if (ONE) __syncthreads();
        else group_sync(grp);
    };
    uint8_t* const codes_out = IS_V ? P.v_codes : P.k_codes;

    // K: where the pairs of the chunks that this lane moves into the operand go (dims 8 (4 j + lane / 8) .. + 7 and 64 above, of
    // rows = lane mod 8: eight rows and four chunks per access keep the scattered stores few to a bank)
    uint32_t koff[IS_V ? 1 : 2][8];
    if constexpr (!IS_V) {
        const uint32_t rows = smem_u32(S.buf[grp][1]) + ((gt >> 5) * (kTileRows / kWrp) + (lane & 7)) * 128;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint4 o = *reinterpret_cast<const uint4*>(&S.to[(4 * j + (lane >> 3)) * 8]);
            const uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) koff[j][e] = rows + (((w[e >> 1] >> (16 * (e & 1))) & 0xFFFFu) ^ ((uint32_t)(lane & 7) << 4));
        }
    }
    // Rows of a tile -> a buffer, asynchronously: thread -> chunk (gt & 15) of rows (gt >> 4) + kStep q; rows past the end are
    // zero-filled.
    constexpr int kStep = kThr / 16, kRowsEach = kTileRows / kStep;
    const int fr = gt >> 4, fc = gt & 15;
    const uint32_t fetch_off = (uint32_t)((fc >> 3) * 16384 + fr * 128 + (((fc & 7) ^ (fr & 7)) << 4));
    auto prefetch = [&](int tl, int b0, int s0, uint8_t* to) {
        const uint32_t dst = smem_u32(to) + fetch_off;
        auto copy = [](uint32_t d, const __half* s, int bytes) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(s), "r"(bytes) : "memory");
        };
        if (s0 + kTileRows <= P.n_tok && (tl + 1) * kTileRows <= n_rows) {
            const __half* src = src_base + b0 * s_sb + (s0 + fr) * s_ss + fc * 8;
            const int64_t inc = kStep * s_ss;
#pragma unroll
            for (int q = 0; q < kRowsEach; ++q, src += inc) copy(dst + q * (128u * kStep), src, 16);
            return;
        }
        int b = b0, s = s0 + fr;
#pragma unroll 1
        for (int q = 0; q < kRowsEach; ++q) {
            while (s >= P.n_tok) { s -= P.n_tok; ++b; }
            const bool valid = tl * kTileRows + fr + kStep * q < n_rows;
            copy(dst + q * (128u * kStep), valid ? src_base + b * s_sb + s * s_ss + fc * 8 : src_base, valid ? 16 : 0);
            s += kStep;
        }
    };
    // (b0, s0) = first row of tile tl
    const int step_b = (int)((uint32_t)(2 * kTileRows) / (uint32_t)P.n_tok), step_s = 2 * kTileRows - step_b * P.n_tok;
    int tl = lo_tile + grp;
    int b0 = (int)((uint32_t)(tl * kTileRows) / (uint32_t)P.n_tok), s0 = tl * kTileRows - b0 * P.n_tok;
    if (ONE && !waited) {
        grid_dependency_wait();
        waited = true;
    }
    if (tl < hi_tile) prefetch(tl, b0, s0, S.buf[grp][0]);
    for (int it = 0, nb0, ns0; tl < hi_tile; tl += 2, ++it, b0 = nb0, s0 = ns0) {
        const int n0 = tl * kTileRows, n_valid = n_rows - n0 < kTileRows ? n_rows - n0 : kTileRows;
        nb0 = b0 + step_b;
        ns0 = s0 + step_s;
        if (ns0 >= P.n_tok) { ns0 -= P.n_tok; ++nb0; }
        uint8_t* const a = S.buf[grp][IS_V ? it & 1 : 1];       // the operand tile
        // sums of squared levels per (part, segment, row), behind the staged rows in the (by then dead) operand tile, or in the
        // other group's buffer
        auto level = [&](int part, int s, int r) -> float& {
            return reinterpret_cast<float*>(ONE ? S.buf[1][0] : a + kLevelOff)[(part * kSeg + s) * kTileRows + r];
        };
        // ---- the prefetched rows; K: their columns into packed order ----
        asm volatile("cp.async.wait_all;" ::: "memory");
        if constexpr (!IS_V) {
            tile_sync();
            const uint32_t raw = smem_u32(S.buf[grp][0]);
            if (S.paired) {
#pragma unroll
                for (int rg = 0; rg < kTileRows / kWrp / 8; ++rg)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int chunk = 4 * j + (lane >> 3), r = (gt >> 5) * (kTileRows / kWrp) + 8 * rg + (lane & 7);
                        const uint32_t from = raw + (uint32_t)(r * 128 + ((chunk ^ (lane & 7)) << 4));
                        const uint4 v = lds128(from), v2 = lds128(from + 16384u);
                        const uint32_t w[4] = {v.x, v.y, v.z, v.w}, w2[4] = {v2.x, v2.y, v2.z, v2.w};
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            asm volatile("st.shared.u32 [%0], %1;" ::"r"(koff[j][c] + rg * 1024u), "r"(__byte_perm(w[c >> 1], w2[c >> 1], c & 1 ? 0x7632 : 0x5410)) : "memory");
                    }
            } else {            // any other order, element by element
                const uint32_t op = smem_u32(a);
#pragma unroll 1
                for (int i = gt; i < kTileRows * kHD / 2; i += kThr) {
                    const int r = i >> 6, c2 = (i & 63) * 2;
                    const uint32_t sw = (uint32_t)(r & 7) << 4, v = lds32(raw + (uint32_t)((c2 >> 6) * 16384 + r * 128) + (((uint32_t)(c2 & 63) * 2u) ^ sw));
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(op + (uint32_t)(r * 128) + (S.to[c2 + e] ^ sw)), "h"((unsigned short)(v >> (16 * e))) : "memory");
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // these rows -> tensor-core reads
        tc_fence_before_sync();     // also orders this thread's tensor-memory reads of the previous tile
        tile_sync();
        // ---- product: one warp issues x . hi, another x . lo ----
        if (ONE ? warp < 2 : (warp & 7) < 2) {
            tc_fence_after_sync();
            const uint32_t lead = elect_one();
            const uint32_t which = warp & 1;
            const uint32_t dst = __shfl_sync(0xffffffffu, acc_hi, 0) + which * kHD;
            const uint64_t xd = tile_desc(smem_u32(a)), w = op_desc(smem_u32(which ? S.w_lo : S.w_hi));
#pragma unroll
            for (int ks = 0; ks < kHD / 16; ++ks) mma_ss(dst, xd + tile_step(ks), w + 16u * ks, ks > 0, lead);
            if (lead) umma_commit(bar);
            __syncwarp();
        }
        if (!ONE && tl + 2 < hi_tile) prefetch(tl + 2, nb0, ns0, S.buf[grp][IS_V ? (it + 1) & 1 : 0]);     // arrives during this tile's work
        // ---- group norms.  K: a thread per segment; V: two threads take alternate element pairs ----
        if constexpr (!IS_V) {
            e5_norms_k(S, grp, smem_u32(a), row, qf, kParts);
        } else if (qf < 2) {
            const uint32_t xr = smem_u32(a) + (uint32_t)row * 128u, sw = (uint32_t)(row & 7) << 4;
            float acc = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {       // four chunks requested together
                uint4 w[4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    w[c] = lds128(xr + (uint32_t)(q >> 1) * 16384u + (((uint32_t)(4 * (q & 1) + c) << 4) ^ sw));
                if (hf == 0) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc = square2(square2(acc, w[c].x), w[c].z);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc = square2(square2(acc, w[c].y), w[c].w);
                }
            }
            S.part[grp][hf][0][row] = acc;
        }
        const int n = n0 + row;
        int b = b0, t = s0 + row;                   // this thread's row
        while (t >= P.n_tok) { t -= P.n_tok; ++b; }
        tile_sync();
        // part q finishes segments 2 q, 2 q + 1 and, of two, 2 q + 4, 2 q + 5 (norm rows are written two values at a time)
#pragma unroll
        for (int u = 0; u < 8 / kParts; ++u) {
            const int s = 2 * qf + (u & 1) + 4 * (u >> 1);
            if (s >= n_seg) continue;
            const float nr = sqrtf((S.part[grp][0][s][row] + S.part[grp][1][s][row]) + 1e-30f);
            S.part[grp][0][s][row] = nr;
            S.part[grp][1][s][row] = nr > (IS_V ? 1e-8f : 1e-10f) ? 1.0f / nr : 1.0f;
        }
        if (!bar_and(3 + grp, kThr, mbar_wait_bounded(bar, n_mma++ & 1))) {      // same verdict for the whole group
            if (gt == 0) atomicExch(&g_enc5_status, kStatusWaitTimeout);
            asm volatile("cp.async.wait_all;" ::: "memory");
            return false;
        }
        tc_fence_after_sync();
        // ---- quantise and pack this thread's part of its row ----
        const uint32_t row_addr = smem_u32(a) + (uint32_t)(row * stage_ld);
        uint8_t* const cd = CODES && codes_out && n < n_rows ? codes_out + (((size_t)b * P.n_kv + h) * P.n_tok + t) * kHD : nullptr;
        float csq = 0.f;
        ByteStream out;
        if (IS_V) {
            constexpr int kCols = kHD / kParts;
            const float r = S.part[grp][1][0][row];
            auto cols = [&](auto bits) { return e5_cols_v<decltype(bits)::value, CODES, kCols / 8>(S, lane_base, kCols * qf, r, row_addr, cd); };
            switch (S.v_bits) {
                case 1: csq = cols(std::integral_constant<int, 1>{}); break;
                case 2: csq = cols(std::integral_constant<int, 2>{}); break;
                case 3: csq = cols(std::integral_constant<int, 3>{}); break;
                default: csq = cols(std::integral_constant<int, 4>{}); break;
            }
            level(qf, 0, row) = csq;
        } else {
            out.open(row_addr, (uint32_t)S.cut_byte[q_lo]);
            if (mixed) {                // (a part without tasks of a segment adds nothing)
                for (int s = 0; s < n_seg; ++s) level(qf, s, row) = 0.f;
            }
            float before = 0.f;         // the segment's sum in this thread's first quarter
            int seg_now = -1;
            const uint64_t scale2 = pack_f2(1.0f / kLoScale, 1.0f / kLoScale);
            const uint32_t factors = smem_u32(&S.part[grp][1][0][row]), recs = smem_u32(S.rec);
            // Two tasks at a time: their table lookups overlap.  An odd count repeats the last task and packs it once.
            float hi[2][8], lo[2][8];
            auto fetch = [&](int ti, int u) {
                const uint32_t col = lane_base + (lds32(recs + (uint32_t)min(ti, task_hi - 1) * (uint32_t)sizeof(E5Rec)) & 0xFFu);
                tmem_ld8(col, hi[u]);
                tmem_ld8(col + kHD, lo[u]);
            };
            if (task_lo < task_hi) {
                fetch(task_lo, 0);
                fetch(task_lo + 1, 1);
            }
            for (int ti = task_lo; ti < task_hi; ti += 2) {
                uint32_t c[2][8];
                uint4 ra[2], rb[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t at = recs + (uint32_t)min(ti + u, task_hi - 1) * (uint32_t)sizeof(E5Rec);
                    ra[u] = lds128(at);
                    rb[u] = lds128(at + 16);
                }
                __syncwarp();
                tmem_ld_wait();
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t off = ra[u].x >> 8;      // 0, 2, 4 or 6
                    if (off) {
                        if (off & 2u) {
#pragma unroll
                            for (int e = 0; e < 6; ++e) { hi[u][e] = hi[u][e + 2]; lo[u][e] = lo[u][e + 2]; }
                        }
                        if (off & 4u) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) { hi[u][e] = hi[u][e + 4]; lo[u][e] = lo[u][e + 4]; }
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float r = lds_f(factors + ra[u].w), g = __uint_as_float(rb[u].y), o = __uint_as_float(rb[u].x);
                    const uint64_t r2 = pack_f2(r, r), off2 = pack_f2(o, o);
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const uint64_t x2 = fma_f2(pack_f2(lo[u][e], lo[u][e + 1]), scale2, pack_f2(hi[u][e], hi[u][e + 1]));
                        float y0, y1;
                        unpack_f2(fma_f2(x2, r2, off2), y0, y1);
                        uint32_t a0, a1;
                        bin_addr2(__saturatef(y0 * g), __saturatef(y1 * g), ra[u].z, a0, a1);
                        c[u][e] = lds8(a0);
                        c[u][e + 1] = lds8(a1);
                    }
                }
                if (ti + 2 < task_hi) {       // the next tasks' columns come while this pair is packed
                    fetch(ti + 2, 0);
                    fetch(ti + 3, 1);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (ti + u >= task_hi) break;
                    if (mixed || CODES) {
                        const uint32_t task = S.tasks[ti + u];
                        const int cnt = (task >> 8) & 0xF, seg = (task >> 16) & 0xF;
                        if (mixed) {        // squared norm of the chosen levels, per segment
                            if (seg != seg_now) {
                                if (seg_now >= 0) level(qf, seg_now, row) = before + csq;
                                csq = before = 0.f;
                                seg_now = seg;
                            } else if (!ONE && ti + u == task_mid) {
                                before = csq;
                                csq = 0.f;
                            }
                            const uint32_t cent = smem_u32(S.kcent + S.seg_lut_off[seg]);
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const float cv = e < cnt ? lds_f(cent + 4u * c[u][e]) : 0.f;
                                csq = fmaf(cv, cv, csq);
                            }
                        }
                        if (CODES && cd) {
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                if (e < cnt) cd[(task & 0xFFu) + e] = (uint8_t)c[u][e];
                        }
                    }
                    out.word(squeeze8(c[u], rb[u].z) & ra[u].y, rb[u].w, row_addr);
                }
            }
            out.end_at(row_addr, (uint32_t)S.cut_byte[q_lo + 4 / kParts]);
            if (mixed && seg_now >= 0) level(qf, seg_now, row) = before + csq;
            if (qf == kParts - 1)
#pragma unroll 1
                for (int p = S.cut_byte[4]; p < rb; p += 4) out.put(0u, 8u * min(4, rb - p));      // rows of a head with fewer bytes than the widest
            out.close();
        }
        tc_fence_before_sync();
        tile_sync();
        // ---- norms out ----
        if (n < n_rows) {
            if (!IS_V) {
                const size_t o = b * P.kn_sb + h * P.kn_sh + (size_t)(t0 + t) * P.kn_st;
#pragma unroll
                for (int u = 0; u < 8 / kParts; ++u) {
                    const int s = 2 * qf + (u & 1) + 4 * (u >> 1);
                    if (s >= P.kn_count) continue;
                    float val = s < n_seg ? S.part[grp][0][s][row] : 0.f;
                    if (mixed && s < n_seg) {       // (a segment on both sides of a cut has several sums)
                        const float q = ONE ? (level(0, s, row) + level(1, s, row)) + (level(2, s, row) + level(3, s, row))
                                            : level(0, s, row) + level(1, s, row);
                        val = val / fmaxf(sqrtf(q), 1e-10f);
                    }
                    if (f16n) static_cast<__half*>(P.kn)[o + s] = __float2half_rn(val);
                    else static_cast<float*>(P.kn)[o + s] = val;
                }
            } else if (qf == 0) {
                const float sum = ONE ? (level(0, 0, row) + level(1, 0, row)) + (level(2, 0, row) + level(3, 0, row)) : level(0, 0, row) + level(1, 0, row);
                const float cnorm = sqrtf(sum + 1e-20f);
                P.vn[b * P.vn_sb + h * P.vn_sh + (size_t)(t0 + t) * P.vn_st] =
                    __float2half_rn(S.part[grp][0][0][row] / (cnorm > 1e-10f ? cnorm : 1.0f));
            }
        }
        // ---- rows out: where the tile's rows are one run of bytes in the cache, as its aligned words ----
        if (o_st == rb && s0 + n_valid <= P.n_tok) {
            uint8_t* const dst0 = out_base + b0 * o_sb + (int64_t)(t0 + s0) * o_st;
            const int total = n_valid * rb, head = min((int)((4u - (uint32_t)(reinterpret_cast<uintptr_t>(dst0) & 3u)) & 3u), total);
            const int words = (total - head) >> 2, tail = total - head - 4 * words;
            const uint32_t stage = smem_u32(a);
            auto row_of = [&](int x) { return (int)(((uint32_t)x * magic) >> 24); };     // x / rb, exact below 128 rows
            if (head == 0 && (rb & 3) == 0) {
#pragma unroll 4
                for (int i = gt; i < words; i += kThr) {
                    const int r = row_of(4 * i);
                    *reinterpret_cast<uint32_t*>(dst0 + 4 * i) = lds32(stage + (uint32_t)(r * (stage_ld - rb) + 4 * i));
                }
                continue;
            }
            if (gt < head) dst0[gt] = a[gt];                                                   // (inside row 0: rb >= 4)
            if (gt < tail) {
                const int x = total - tail + gt, r = row_of(x);
                dst0[x] = a[r * stage_ld + x - r * rb];
            }
            for (int i = gt; i < words; i += kThr) {
                const int x = head + 4 * i, r = row_of(x), p = x - r * rb;
                const uint32_t at = stage + (uint32_t)(r * stage_ld + (p & ~3));
                uint32_t w = lds32(at);
                if (p & 3) w = __funnelshift_r(w, lds32(at + 4), (uint32_t)(p & 3) * 8u);
                const int left = rb - p;            // bytes of this row from here
                if (left < 4) w = (w & ((1u << (8 * left)) - 1u)) | lds32(stage + (uint32_t)((r + 1) * stage_ld)) << (8 * left);
                *reinterpret_cast<uint32_t*>(dst0 + x) = w;
            }
        } else {
            for (int i = gt; i < n_valid * rb; i += kThr) {
                const int r = i / rb, p = i - r * rb;
                const int nn = n0 + r, bb = (int)((uint32_t)nn / (uint32_t)P.n_tok), tt = nn - bb * P.n_tok;
                out_base[bb * o_sb + (int64_t)(t0 + tt) * o_st + p] = a[r * stage_ld + p];
            }
        }
    }
    return true;
}

// One CTA per SM.  The tiles of all (KV head, K or V) form one list, a K tile kUnitsK units long and a V tile kUnitsV (what
// they take, 219 and 162 us for a million rows: 374 us for both so; with 13 to 7 a sixth more); CTA i works on the tiles that begin in its share of the units,
// and loads the tables again where its share crosses into the next (head, role).  With few tiles per CTA whole tiles count, not
// units: see slowest_share.
constexpr int kUnitsK = 11, kUnitsV = 8, kUnitsK2 = 13, kUnitsV2 = 7;
template <bool MIXED, bool CODES, bool ONE>
__global__ void __launch_bounds__(kThreads, 1) encode_t5_kernel(const EncParams P, const int units_k, const int units_v) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    E5Smem& S = *reinterpret_cast<E5Smem*>(smem_raw);
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&S.mma_bar[0], 2);
        mbar_init(&S.mma_bar[1], 2);
        mbar_fence_init();
    }
    if (tid < 32) tmem_alloc(&S.tmem_base, kTmemCols);
    const int n_tiles = (P.n_batch * P.n_tok + kTileRows - 1) / kTileRows;
    // What follows may start once every CTA is at its last (head, role).  From the start of the launch, its CTAs (and those of
    // the launch behind it) all settle on the first SMs to be free, while this launch holds the others, and share them to the
    // end: encode, rotation and prefill of 5192 tokens of 4 KV heads x 2 took 187.3 us, 182.7 so (10000 x 1: 293.6, 288.1).  With
    // more than 32 tiles per CTA the few that begin their last range late would hold up the next launch's tables more than
    // that costs (1 048 576 K and as many V rows, again and again: 373.7 us from the start, 375.0 so); with one tile each all end
    // together (K, then V, of 2000 rows of 8 heads: 18.5, 19.1).
    if (ONE || n_tiles * P.n_kv > 16 * (int)gridDim.x) grid_launch_dependents();
    const int64_t len_k = (int64_t)units_k * n_tiles, len_v = (int64_t)units_v * n_tiles, len = len_k + len_v, all = len * P.n_kv;
    const int64_t u0 = all * blockIdx.x / gridDim.x, u1 = all * (blockIdx.x + 1) / gridDim.x;
    bool waited = false, in_range = true;
    int n_mma = 0;
    for (int64_t u = u0; u < u1 && in_range;) {
        const int h = (int)(u / len);
        const bool is_v = u - h * len >= len_k;
        const int64_t base = h * len + (is_v ? len_k : 0), end = base + (is_v ? len_v : len_k);
        const int w = is_v ? units_v : units_k;
        const int lo = (int)((u - base + w - 1) / w), hi = (int)((min(u1, end) - base + w - 1) / w);
        u = end;
        if (!ONE && u >= u1) grid_launch_dependents();
        if (lo >= hi) continue;
        e5_setup(S, P, P.desc[h], is_v, h);
        // The rows, and what this launch overwrites, belong to earlier work in the stream.  (The one-tile form waits where it
        // asks for its rows; with many tiles that costs the loop registers.)
        if (!waited && (!ONE || P.pos_dev)) {
            grid_dependency_wait();
            waited = true;
            if (P.pos_dev) in_range = enc_range_ok(P, *P.pos_dev, P.n_tok);      // (uniform over the launch: else nothing is stored)
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");          // W operand: generic stores -> tensor-core reads
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        if (!in_range) break;
        const bool ok = is_v ? e5_role<true, MIXED, CODES, ONE>(S, P, h, lo, hi, n_mma, waited) : e5_role<false, MIXED, CODES, ONE>(S, P, h, lo, hi, n_mma, waited);
        if (!__syncthreads_and(ok ? 1 : 0) || ONE) break;      // (also: everyone is done with this range's tables)
    }
    if (!waited) grid_dependency_wait();
    tc_fence_before_sync();
    __syncthreads();
    if (tid < 32) tmem_dealloc(S.tmem_base, kTmemCols);
}

}  // namespace

// The slowest CTA's time, in tenths of a unit, for K and V tiles that count uk and uv: the two row groups of a CTA work side by
// side, so an odd tile takes about 1.3 of its units instead of half a pair's two, and a (head, role) begun takes four.
static int slowest_share(int n_tiles, int n_kv, int uk, int uv, int sms) {
    const int len_k = uk * n_tiles, len = len_k + uv * n_tiles, all = len * n_kv;
    int worst = 0;
    for (int i = 0; i < sms; ++i) {
        const int u1 = all * (i + 1) / sms;
        int t = 0;
        for (int u = all * i / sms; u < u1;) {
            const int at = u / len * len, base = u - at >= len_k ? at + len_k : at;
            const bool is_v = base != at;
            const int end = is_v ? at + len : at + len_k, w = is_v ? uv : uk, top = u1 < end ? u1 : end;
            const int n = (top - base + w - 1) / w - (u - base + w - 1) / w;
            if (n > 0) t += (n / 2 * 20 + n % 2 * 13) * (is_v ? kUnitsV : kUnitsK) + 40;
            u = end;
        }
        worst = t > worst ? t : worst;
    }
    return worst;
}

// Whether K and V tiles are better weighed 13 : 7 than 11 : 8.  Working it out takes 2.5 us, more than the launch: the answers for
// the latest shapes are kept (a model's layers ask with the same one), each in one word: shape | valid | answer.
static bool second_weights(int n_tiles, int n_kv, int sms) {
    static std::atomic<uint64_t> kept[64];
    const uint64_t shape = (uint64_t)n_tiles | (uint64_t)n_kv << 20 | (uint64_t)sms << 40;
    std::atomic<uint64_t>& slot = kept[(n_tiles * 5 + n_kv) & 63];
    const uint64_t have = slot.load(std::memory_order_relaxed);
    if (have >> 2 == shape) return have & 1u;
    const bool second = slowest_share(n_tiles, n_kv, kUnitsK2, kUnitsV2, sms) < slowest_share(n_tiles, n_kv, kUnitsK, kUnitsV, sms);
    slot.store(shape << 2 | 2u | (second ? 1u : 0u), std::memory_order_relaxed);
    return second;
}

// The launcher's caller checks: every input row 16-byte aligned and n_tok >= 16 (as for the warp-MMA bulk path).
int launch_encode_t5(const EncParams& P, cudaStream_t stream) {
    const int64_t n_rows = (int64_t)P.n_batch * P.n_tok;
    if (n_rows > (1LL << 30)) return BGTQ_E_TOOBIG;
    const bool do_k = !(P.flags & BGTQ_ENC_SKIP_K), do_v = !(P.flags & BGTQ_ENC_SKIP_V);
    if (!do_k && !do_v) return BGTQ_OK;
    const int n_tiles = (int)((n_rows + kTileRows - 1) / kTileRows);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t all = (int64_t)n_tiles * P.n_kv * ((do_k ? 1 : 0) + (do_v ? 1 : 0));
    const bool few = all <= sms;                // one tile per CTA (the code written out for it: ONE)
    int units_k = do_k ? (few ? 1 : kUnitsK) : 0, units_v = do_v ? (few ? 1 : kUnitsV) : 0;
    // With up to eight tiles per CTA the better of two weightings: 4 KV heads at 6144 tokens 28 and 22 us with 11 : 8 and
    // 13 : 7, at 5120 19 and 22, at 10000 (11 : 8) 29 and 33.
    if (do_k && do_v && !few && all <= 8 * sms && second_weights(n_tiles, P.n_kv, sms)) {
        units_k = kUnitsK2;
        units_v = kUnitsV2;
    }
    const int smem = (int)sizeof(E5Smem);
    const bool mixed = P.flags & BGTQ_ENC_K_MIXED, codes = P.k_codes != nullptr || P.v_codes != nullptr;
    auto kern = mixed ? (codes ? encode_t5_kernel<true, true, false> : few ? encode_t5_kernel<true, false, true> : encode_t5_kernel<true, false, false>)
                      : (codes ? encode_t5_kernel<false, true, false> : few ? encode_t5_kernel<false, false, true> : encode_t5_kernel<false, false, false>);
    // the attribute is per device: set it on every launch (cheap, and legal under stream capture)
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
        cudaGetLastError();
        return BGTQ_E_LAUNCH;
    }
    return launch_kernel(kern, dim3((unsigned)(few ? all : sms)), dim3(kThreads), smem, stream, true, P, units_k,
                         units_v) == cudaSuccess ? BGTQ_OK : BGTQ_E_LAUNCH;
}

}  // namespace bgtq

extern "C" __attribute__((visibility("default"))) int bgtq_encode_tcgen05_status(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, bgtq::g_enc5_status, sizeof(v)) != cudaSuccess) {
        cudaGetLastError();
        return BGTQ_E_LAUNCH;
    }
    return v;
}
