// prompt_tc5.cuh -- what the two tcgen05 prompt kernels share: prompt_tc5.cu (a CTA a tile) and prompt_turns_tc5.cu (a CTA that takes
// tiles in turns).
#pragma once
#include "b2_mask.cuh"
#include "b2_tc5.cuh"

#ifdef __CUDACC__
namespace b2prompt {

constexpr int BM = 128, BN = 128;                    // rows of a slot, keys of a tile
constexpr int SUB = 128 * 128;                       // bytes of a [128 rows][64 el] sub-tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float FLOOR = -1e30f;                      // a row that has seen no key yet: exp2(-inf - FLOOR) = 0, not NaN
enum { KIND_SOFTMAX = 0, KIND_CAPPED = 1, KIND_SIGMOID = 2 };

// 16 bytes, or zeros without reading `src` (no branch: a divergent one would serialise the copies of a warp)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
// bits 0..31 of the columns [lo, hi) of a 32-column group that starts at column 0
__device__ __forceinline__ uint32_t col_bits(int lo, int hi) {
    lo = min(max(lo, 0), 32);
    hi = min(max(hi, 0), 32);
    return hi > lo ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
}
// what a query row sees of the compact key order: c <= hi and (c >= low or block <= c < keep)
struct RowRange {
    int hi, low, block;
};
template <class Span>
__device__ __forceinline__ RowRange range_of(const Span& span, int i, int chunk, int window) {
    RowRange r;
    r.hi = span.index(i);
    r.block = 0;
    if (chunk > 0) r.block = span.index((i / chunk) * chunk);
    r.low = r.block;
    if (window > 0) r.low = max(r.block, span.index(i - window + 1));
    return r;
}

}  // namespace b2prompt
#endif
