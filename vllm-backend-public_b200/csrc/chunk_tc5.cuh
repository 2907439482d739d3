// chunk_tc5.cuh -- fp32 products on the bf16 tensor cores, as the chunked recurrence uses them.
//
// A float is the sum of three bf16 numbers (its leading 8 bits, the next 8, the last 8: truncation, so exact), and a product of two
// floats is six of the nine products of their parts: what is left out is below 2^-22 of it.  Products of parts are exact in fp32, but
// the tensor core truncates its accumulator at every instruction, so the leading parts' products have an accumulator of their own, which
// takes one addition per 16 entries, or the small products come first.  Sums of 128 products of normal numbers against 64 bits, relative to
// the result's norm: 1.6e-7 with two accumulators, 1.3e-7 with one per 64 entries and the small products first, 9.8e-7 with one for all;
// a chain of 128 FMAs 2.0e-7.
//
// Operands are tiles of 128-byte rows in the 128-byte swizzle: rows of 64 entries of the summed index (K-major), or rows of 64 entries of
// the result's index, a row per summed index (MN-major).
#pragma once
#include "b2_act.cuh"
#include "b2_tc5.cuh"

#ifdef __CUDACC__
namespace chunk_tc5 {
using namespace b2tc;

// two floats' leading 16 bits
__device__ __forceinline__ uint32_t tops(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }
// what x's leading part leaves, and what that one's leaves; the leading parts are the upper halves of x and m
__device__ __forceinline__ void split(float x, uint32_t& m, uint32_t& l) {
    const float r = x - __uint_as_float(__float_as_uint(x) & 0xffff0000u);
    m = __float_as_uint(r);
    l = __float_as_uint(r - __uint_as_float(m & 0xffff0000u));
}
struct Split8 { uint4 hi, mid, lo; };
// eight floats -> their parts, packed in order
__device__ __forceinline__ Split8 split8(const float (&x)[8]) {
    uint32_t m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split(x[i], m[i], l[i]);
    auto x2 = [&](int i) { return tops(__float_as_uint(x[i]), __float_as_uint(x[i + 1])); };
    return {make_uint4(x2(0), x2(2), x2(4), x2(6)), make_uint4(tops(m[0], m[1]), tops(m[2], m[3]), tops(m[4], m[5]), tops(m[6], m[7])),
            make_uint4(tops(l[0], l[1]), tops(l[2], l[3]), tops(l[4], l[5]), tops(l[6], l[7]))};
}
__device__ __forceinline__ void store_parts(unsigned char* dst, int part_bytes, const Split8& s) {
    *reinterpret_cast<uint4*>(dst) = s.hi;
    *reinterpret_cast<uint4*>(dst + part_bytes) = s.mid;
    *reinterpret_cast<uint4*>(dst + 2 * part_bytes) = s.lo;
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

// D (two accumulators of 128 columns: the leading parts' products, and the five others) += A B over `ksteps` times 16 entries.  The parts
// of A and B are PART bytes apart, those of B neighbours in N.  AK, BK: bytes >> 4 from one k-step to the next.
constexpr int PART = 64 * 256;
constexpr uint32_t kAmn = 1u << 15, kBmn = 1u << 16;              // operand is MN-major
template <int AK, int BK>
__device__ __forceinline__ void mma_parts(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t majors, int ksteps, bool acc) {
    const uint32_t n128 = idesc_bf16(128, 128, 0) | majors, n256 = idesc_bf16(128, 256, 0) | majors;
#pragma unroll 1
    for (int k = 0; k < ksteps; ++k) {
        const uint64_t a = desc_join(a_lo + k * AK), a1 = desc_join(a_lo + k * AK + (PART >> 4)), a2 = desc_join(a_lo + k * AK + (2 * PART >> 4));
        const uint64_t b = desc_join(b_lo + k * BK), b1 = desc_join(b_lo + k * BK + (PART >> 4)), b2 = desc_join(b_lo + k * BK + (2 * PART >> 4));
        mma_ss(d, a, b, n256, acc || k > 0);
        mma_ss(d + 128, a, b2, n128, true);
        mma_ss(d + 128, a1, b, n128, true);
        mma_ss(d + 128, a1, b1, n128, true);
        mma_ss(d + 128, a2, b, n128, true);
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
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

}  // namespace chunk_tc5
#endif
