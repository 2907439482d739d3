// chunk_tc5.cuh -- fp32 products on the bf16 tensor cores, as the chunked recurrence uses them.
//
// A float is the sum of three bf16 numbers (its rounding to 8 bits, that of the rest, and what is left: exact), and a product of two
// floats is six of the nine products of their parts: what is left out is below 2^-25 of it (Henry, Tang, Heinecke, "Leveraging the bfloat16
// artificial intelligence datatype for higher-precision computations", 2019).  (Parts by truncation instead of rounding
// take as many instructions and are all of one sign: errors a third higher.)  Products of parts are exact in fp32, but
// the tensor core truncates its accumulator at every instruction, so the leading parts' products have an accumulator of their own, which
// takes one addition per 16 entries, or the small products come first.  Sums of 128 products of normal numbers against 64 bits, relative to
// the result's norm: 1.2e-7 with two accumulators, 0.8e-7 with one per 64 entries and the small products first, 8.2e-7 with one for all;
// a chain of 128 FMAs 2.0e-7.  Of 64 products: 7.0e-8 with one leading accumulator, 5.1e-8 with two in turns, 4.7e-8 with four; FMAs 1.4e-7.
// Cutting off draws every result towards zero (4.5e-8 of it with one accumulator, 2.3e-8 with two), so more of them help twice.
//
// Operands are tiles of 128-byte rows in the 128-byte swizzle: rows of 64 entries of the summed index (K-major), or rows of 64 entries of
// the result's index, a row per summed index (MN-major).
#pragma once
#include "b2_act.cuh"
#include "b2_tc5.cuh"

#ifdef __CUDACC__
namespace chunk_tc5 {
using namespace b2tc;

// two floats -> their parts, packed
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = b2::pack_bf16x2(x, y);
    x -= __uint_as_float(hi << 16);
    y -= __uint_as_float(hi & 0xffff0000u);
    mid = b2::pack_bf16x2(x, y);
    lo = b2::pack_bf16x2(x - __uint_as_float(mid << 16), y - __uint_as_float(mid & 0xffff0000u));
}
struct Split8 { uint4 hi, mid, lo; };
// eight floats -> their parts, packed in order
__device__ __forceinline__ Split8 split8(const float (&x)[8]) {
    Split8 s;
    split2(x[0], x[1], s.hi.x, s.mid.x, s.lo.x);
    split2(x[2], x[3], s.hi.y, s.mid.y, s.lo.y);
    split2(x[4], x[5], s.hi.z, s.mid.z, s.lo.z);
    split2(x[6], x[7], s.hi.w, s.mid.w, s.lo.w);
    return s;
}
// four floats -> 8 bytes of each part, `part_bytes` apart
__device__ __forceinline__ void store_parts4(unsigned char* dst, int part_bytes, const float4& x) {
    uint2 hi, mid, lo;
    split2(x.x, x.y, hi.x, mid.x, lo.x);
    split2(x.z, x.w, hi.y, mid.y, lo.y);
    *reinterpret_cast<uint2*>(dst) = hi;
    *reinterpret_cast<uint2*>(dst + part_bytes) = mid;
    *reinterpret_cast<uint2*>(dst + 2 * part_bytes) = lo;
}
__device__ __forceinline__ void store_parts(unsigned char* dst, int part_bytes, const Split8& s) {
    *reinterpret_cast<uint4*>(dst) = s.hi;
    *reinterpret_cast<uint4*>(dst + part_bytes) = s.mid;
    *reinterpret_cast<uint4*>(dst + 2 * part_bytes) = s.lo;
}
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }
// An infinity, and what rounds to one in bf16, has no parts that add up to it: a product with it is NaN.  Kernels find such results and sum
// them again in plain fp32, as the scan token by token would.
__device__ __forceinline__ bool splits(float x) { return fabsf(x) < __uint_as_float(0x7f7f8000u); }
// four floats -> 8 bytes of each part, from which joined() gives back any float: parts by truncation where rounding would overflow, infinities and NaN
// in the first part alone
__device__ __forceinline__ void store_any4(unsigned char* dst, int part_bytes, const float4& x) {
    if (splits(x.x) && splits(x.y) && splits(x.z) && splits(x.w)) {
        store_parts4(dst, part_bytes, x);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float v = e == 0 ? x.x : e == 1 ? x.y : e == 2 ? x.z : x.w;
        const uint32_t bits = __float_as_uint(v);
        uint32_t hi, mid, lo;
        split2(v, 0.f, hi, mid, lo);
        if (!splits(v)) {
            uint32_t none;
            hi = v == v ? bits >> 16 : 0x7fffu;
            split2(finite(v) ? v - __uint_as_float(bits & 0xffff0000u) : 0.f, 0.f, mid, lo, none);
        }
        reinterpret_cast<uint16_t*>(dst)[e] = (uint16_t)hi;
        reinterpret_cast<uint16_t*>(dst + part_bytes)[e] = (uint16_t)mid;
        reinterpret_cast<uint16_t*>(dst + 2 * part_bytes)[e] = (uint16_t)lo;
    }
}
__device__ __forceinline__ float joined(const unsigned char* src, int part_bytes) {
    float p[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) p[u] = __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t*>(src + u * part_bytes) << 16);
    return finite(p[0]) ? p[0] + p[1] + p[2] : p[0];
}
// 16-byte vector `c` (eight entries) of row `r`, in sub-tiles of 64 entries x `rows` rows
__device__ __forceinline__ int tile_at(int r, int c, int rows) { return (c >> 3) * rows * 128 + r * 128 + (((c & 7) ^ (r & 7)) << 4); }

// 8192 floats of a row-major matrix in registers, twice eight neighbours a thread of 512: 64 rows x 128 columns or 128 x 64.  Rows
// and columns outside are zeros.
template <int COLS>
struct Fetch {
    static constexpr int VECS = COLS / 8, STEP = 512 / VECS;         // STEP: rows from one vector of a thread to the next, a multiple of 8
    float x[2][8];
    static __device__ __forceinline__ int row(int i) { return threadIdx.x / VECS + i * STEP; }
    static __device__ __forceinline__ int col() { return threadIdx.x % VECS * 8; }
    __device__ __forceinline__ void load(const float* base, int64_t stride, int rows, int cols) {
        const float* p = base + row(0) * stride + col();
        if (rows >= 2 * STEP && cols >= COLS) {
#pragma unroll
            for (int i = 0; i < 2; ++i, p += STEP * stride) {
                const float4 u = *reinterpret_cast<const float4*>(p), v = *reinterpret_cast<const float4*>(p + 4);
                x[i][0] = u.x; x[i][1] = u.y; x[i][2] = u.z; x[i][3] = u.w; x[i][4] = v.x; x[i][5] = v.y; x[i][6] = v.z; x[i][7] = v.w;
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i, p += STEP * stride)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (row(i) < rows && col() + 4 * h < cols) v = *reinterpret_cast<const float4*>(p + 4 * h);
                x[i][4 * h] = v.x; x[i][4 * h + 1] = v.y; x[i][4 * h + 2] = v.z; x[i][4 * h + 3] = v.w;
            }
    }
    // parts `part_bytes` apart
    __device__ __forceinline__ void store(unsigned char* dst, int part_bytes) const {
        dst += tile_at(row(0), col() / 8, 8192 / COLS);
#pragma unroll
        for (int i = 0; i < 2; ++i) store_parts(dst + i * STEP * 128, part_bytes, split8(x[i]));
    }
};

// D (two accumulators of 128 columns) = A B over a first slice of `ksteps` times 16 entries, or += over a second one.  The first accumulator
// takes the first slice's leading products, the other one the small ones of both and behind these the second's leading ones, so none is cut
// off eight times at full size.  The parts of A and B are PART bytes apart, those of B neighbours in N.  AK, BK: bytes >> 4
// from one k-step to the next.
constexpr int PART = 64 * 256;
constexpr uint32_t kAmn = 1u << 15, kBmn = 1u << 16;              // operand is MN-major
template <int AK, int BK>
__device__ __forceinline__ void mma_parts(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t majors, int ksteps, bool second) {
    const uint32_t n128 = idesc_bf16(128, 128, 0) | majors, n256 = idesc_bf16(128, 256, 0) | majors;
#pragma unroll 1
    for (int k = 0; k < ksteps; ++k) {
        const uint64_t a = desc_join(a_lo + k * AK), a1 = desc_join(a_lo + k * AK + (PART >> 4)), a2 = desc_join(a_lo + k * AK + (2 * PART >> 4));
        const uint64_t b = desc_join(b_lo + k * BK), b1 = desc_join(b_lo + k * BK + (PART >> 4)), b2 = desc_join(b_lo + k * BK + (2 * PART >> 4));
        if (second) mma_ss(d + 128, a, b1, n128, true);
        else mma_ss(d, a, b, n256, k > 0);           // the leading parts' and a b1
        mma_ss(d + 128, a, b2, n128, true);
        mma_ss(d + 128, a1, b, n128, true);
        mma_ss(d + 128, a1, b1, n128, true);
        mma_ss(d + 128, a2, b, n128, true);
    }
    if (second)
#pragma unroll 1
        for (int k = 0; k < ksteps; ++k) mma_ss(d + 128, desc_join(a_lo + k * AK), desc_join(b_lo + k * BK), n128, true);
}

// The same over 64 entries at once, and nothing in D before: both accumulators take leading products, every other k-step each, and the first of
// them all others before these, where what the tensor core cuts off is small.
template <int AK, int BK>
__device__ __forceinline__ void mma_parts64(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t majors) {
    const uint32_t id = idesc_bf16(128, 128, 0) | majors;
    constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
#pragma unroll 1
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int p = 0; p < 5; ++p)
            mma_ss(d, desc_join(a_lo + k * AK + (A[p] * PART >> 4)), desc_join(b_lo + k * BK + (B[p] * PART >> 4)), id, p > 0 || k > 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) mma_ss(d + 128 * (k & 1), desc_join(a_lo + k * AK), desc_join(b_lo + k * BK), id, k != 1);
}

// The same with 64 columns: D (accumulators of 64 columns: LEAD that take the leading parts' products in turns, then products of the parts'
// order 1 and 2) += A B over `ksteps` times 16 entries, at least LEAD of them.  The parts of B are side by side as 192 columns, 8192 bytes
// apart.  A_PART: bytes from one part of A to the next.
template <int LEAD, int A_PART, int AK, int BK>
__device__ __forceinline__ void mma_orders(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t majors, int ksteps, bool acc) {
    static_assert(LEAD == 1 || LEAD == 2, "");
    const uint32_t n64 = idesc_bf16(128, 64, 0) | majors, n128 = idesc_bf16(128, 128, 0) | majors, n192 = idesc_bf16(128, 192, 0) | majors;
    const uint32_t order1 = d + 64 * LEAD;
#pragma unroll 1
    for (int k = 0; k < ksteps; ++k) {
        const uint64_t a = desc_join(a_lo + k * AK), b = desc_join(b_lo + k * BK);
        if (LEAD == 2 && (k & 1)) {
            mma_ss(d, a, b, n64, acc || k > 1);
            mma_ss(order1, a, desc_join(b_lo + k * BK + (8192 >> 4)), n128, true);
        } else {
            mma_ss(order1 - 64, a, b, n192, acc || k > 0);
        }
        mma_ss(order1, desc_join(a_lo + k * AK + (A_PART >> 4)), b, n128, true);
        mma_ss(order1 + 64, desc_join(a_lo + k * AK + (2 * A_PART >> 4)), b, n64, true);
    }
}

// 32 lanes x 8 columns
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "r"(taddr));
}
// the sum of the two accumulators' columns c .. c + 7 in this thread's lane
__device__ __forceinline__ void read_parts(uint32_t d, float (&s)[8]) {
    float r[8];
    tmem_ld8(d, s);
    tmem_ld8(d + 128, r);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] += r[i];
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
                   "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void read_parts(uint32_t d, float (&s)[16]) {
    float r[16];
    tmem_ld16(d, s);
    tmem_ld16(d + 128, r);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] += r[i];
}
// The same with one accumulator for all small products behind two leading ones: fewer columns to read, more MMAs
template <int A_PART, int AK, int BK>
__device__ __forceinline__ void mma_orders3(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t majors, int ksteps, bool acc) {
    const uint32_t n64 = idesc_bf16(128, 64, 0) | majors;
    constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
#pragma unroll 1
    for (int k = 0; k < ksteps; ++k) {
        const uint64_t a = desc_join(a_lo + k * AK), b = desc_join(b_lo + k * BK);
        mma_ss(d + 64 * (k & 1), a, b, n64, acc || k > 1);
#pragma unroll
        for (int p = 0; p < 5; ++p)
            mma_ss(d + 128, desc_join(a_lo + k * AK + (A[p] * A_PART >> 4)), desc_join(b_lo + k * BK + (B[p] * 8192 >> 4)), n64, acc || p > 0 || k > 0);
    }
}
__device__ __forceinline__ void read_orders3(uint32_t d, float (&s)[16]) {
    float r[16], q[16];
    tmem_ld16(d + 128, s);
    tmem_ld16(d + 64, r);
    tmem_ld16(d, q);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = (s[i] + r[i]) + q[i];
}
template <int LEAD>
__device__ __forceinline__ void read_orders(uint32_t d, float (&s)[16]) {         // the accumulators of mma_orders, the smallest first
    float r[16], q[16];
    tmem_ld16(d + 64 * LEAD + 64, s);
    tmem_ld16(d + 64 * LEAD, r);
    tmem_ld16(d + 64 * LEAD - 64, q);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = (s[i] + r[i]) + q[i];
    if (LEAD == 2) {
        tmem_ld16(d, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) s[i] += r[i];
    }
}
// Which of a CTA's items have results that are not finite: once it is through, it looks at those from the first to the last of them again
struct Again {
    int first, last;
    __device__ __forceinline__ void none() { first = 0x7fffffff; last = -1; }
    __device__ __forceinline__ void add(int item) { atomicMin(&first, item); atomicMax(&last, item); }
};

struct Args {
    const float *qkv, *decay;
    int H, G, dk, dv, n_seq, blocks, items;          // blocks of 128 columns; items = chunks of this piece (an upper bound) x heads x blocks
    int first, chunks;                               // the piece: chunks first .. first + chunks - 1 of the batch, whose scratch ws holds
    const int32_t *cu_q, *ctx_start, *state_slot;
    float *state, *o, *ws;
    const float* carry_in;                           // [H][dk][dv]: state of the sequence that the piece before cut, and of the one that this one cuts
    float* carry_out;
};

// Loads that a thread of a state kernel has in flight: eight (72 registers, seven CTAs an SM), or sixteen (128, four) where the chains are longer than that,
// but not where eight would keep all CTAs resident and sixteen would not.  Scans of 16 heads of 128 x 128, eight / sixteen: one sequence of 4096 tokens
// 123.5 / 120.8 us, of 2000 63.9 / 62.7, of 500 33.4 / 34.0; 2 x 4096 229.7 / 239.0, 4 x 2000 214.5 / 211.3, 4 x 200 36.8 / 40.2, 8 x 500 119.8 / 125.8; channel
// decays 1 x 4096 294.2 / 290.8, 2 x 2048 296.5 / 305.4, 3 x 1000 226.9 / 224.1, 8 x 200 146.2 / 153.1.
inline bool long_chains(const Args& a, int ctas) { return a.chunks > 9 * a.n_seq && (ctas <= 4 * b2_sm_count() || ctas > 7 * b2_sm_count()); }

// A sequence's chunks in this piece.  What goes on after the piece, and into it, is the one sequence that its border cuts.
struct Portion {
    int begin, count;                                // first one in the scratch, and how many (0: none)
    bool starts, ends;                               // the sequence's first and last chunk are among them
};
template <int TILE>
__device__ __forceinline__ Portion portion(const Args& a, int seq) {
    int base = -a.first;
    for (int s = 0; s < seq; ++s)
        if (a.ctx_start[s] >= 0) base += (a.cu_q[s + 1] - a.cu_q[s] + TILE - 1) / TILE;
    const int n = a.ctx_start[seq] < 0 ? 0 : (a.cu_q[seq + 1] - a.cu_q[seq] + TILE - 1) / TILE, lo = max(base, 0), hi = min(base + n, a.chunks);
    return {lo, max(hi - lo, 0), base >= 0, base + n <= a.chunks};
}
// where a head's state comes from and goes to: the sequence's slot (none: null), or the carried state
__device__ __forceinline__ const float* state_from(const Args& a, const Portion& p, int slot, int head, int ctx) {
    const float* src = p.starts ? (slot >= 0 && ctx > 0 ? a.state + (size_t)slot * a.H * a.dk * a.dv : nullptr) : a.carry_in;
    return src ? src + (size_t)head * a.dk * a.dv : nullptr;
}
__device__ __forceinline__ float* state_to(const Args& a, const Portion& p, int slot, int head) {
    float* dst = p.ends ? (slot >= 0 ? a.state + (size_t)slot * a.H * a.dk * a.dv : nullptr) : a.carry_out;
    return dst ? dst + (size_t)head * a.dk * a.dv : nullptr;
}

// Where an item lies.  The whole warp works.
struct At {
    int row, nt, chunk, head, block, fresh;          // first row, rows (0: none, and none follow), chunk of the piece, fresh: the state before it is zero
};
template <int TILE>
__device__ __forceinline__ At locate(const Args& a, int item) {
    At at{0, 0, 0, 0, 0, 0};
    if (item >= a.items) return at;
    const int lane = threadIdx.x & 31, hz = a.H * a.blocks;
    at.chunk = item / hz;
    at.head = (item - at.chunk * hz) / a.blocks;
    at.block = (item - at.chunk * hz) % a.blocks;
    int want = a.first + at.chunk;
    for (int s0 = 0; s0 < a.n_seq; s0 += 32) {
        int lo = 0, len = 0, ctx = -1;
        if (s0 + lane < a.n_seq) {
            lo = a.cu_q[s0 + lane];
            ctx = a.ctx_start[s0 + lane];
            len = ctx < 0 ? 0 : a.cu_q[s0 + lane + 1] - lo;
        }
        const int own = (len + TILE - 1) / TILE;
        int c = own;                                 // chunks up to this sequence's last
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, c, d);
            if (lane >= d) c += u;
        }
        const unsigned has = __ballot_sync(0xffffffffu, want < c);
        if (has) {
            const int src = __ffs(has) - 1, in = want - __shfl_sync(0xffffffffu, c - own, src);
            at.row = __shfl_sync(0xffffffffu, lo, src) + in * TILE;
            at.nt = min(TILE, __shfl_sync(0xffffffffu, len, src) - in * TILE);
            at.fresh = in == 0 && __shfl_sync(0xffffffffu, ctx, src) == 0;
            return at;
        }
        want -= __shfl_sync(0xffffffffu, c, 31);
    }
    return at;
}

// Products of neighbours in a warp: up to the lane, from the lane on, of all.  In 64 bits: a tree of products squares its rounding errors
// where the decays are alike (a fixed decay per head: 0.9961^128 off by 2e-6, the state of 4096 tokens by 6.8e-7; 1.5e-7 so, 4.1e-7 with chains)
__device__ __forceinline__ double product_up_to(double g) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, g, d);
        if ((threadIdx.x & 31) >= d) g *= u;
    }
    return g;
}
__device__ __forceinline__ double product_from(double g) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double u = __shfl_down_sync(0xffffffffu, g, d);
        if ((threadIdx.x & 31) + d < 32) g *= u;
    }
    return g;
}
__device__ __forceinline__ double product_of_all(double g) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) g *= __shfl_xor_sync(0xffffffffu, g, d);
    return g;
}

// What this warp wrote to shared memory and read from TMEM is handed over; true (in all lanes) in the last of the CTA's warps to do so
__device__ __forceinline__ bool hand_over(unsigned* count) {
    b2::fence_proxy_async();
    tc_fence_before();
    __syncwarp();
    unsigned before = 0;
    if ((threadIdx.x & 31) == 0) asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(b2::smem_u32(count)) : "memory");
    const bool last = (__shfl_sync(0xffffffffu, before, 0) & 15) == 15;
    if (last) tc_fence_after();
    return last;
}
__device__ __forceinline__ uint32_t tmem_alloc(uint32_t* at, int warp) {         // all 512 columns; the whole CTA
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(b2::smem_u32(at)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return *at;
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, int warp) {
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

}  // namespace chunk_tc5
#endif
