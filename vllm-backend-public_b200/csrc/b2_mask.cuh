// b2_mask.cuh -- which cached keys a query sees (mask blocks, sliding window, kept first tokens), and what happens to a score and
// to a head's output; shared by the kernels of b2_masked_attention and b2_window_attention.
#pragma once
#include "b2_act.cuh"

#ifdef __CUDACC__
// The keys a query at position `pos` may see, as one compact index range [0, n): first the kept keys lo .. lo+nfirst-1
// (the sequence's first tokens that lie before the window), then wlo .. pos.  Without a window nfirst = 0 and wlo = lo.
struct KeySpan {
    int lo, nfirst, wlo, n;
    __device__ __forceinline__ int key(int c) const { return c < nfirst ? lo + c : wlo + (c - nfirst); }
    // compact index of the first key at or behind position j
    __device__ __forceinline__ int index(int j) const { return j < wlo ? min(max(j - lo, 0), nfirst) : nfirst + (j - wlo); }
};
__device__ __forceinline__ KeySpan key_span(int pos, int last, int chunk, int window, int keep_first) {
    KeySpan s;
    s.lo = chunk > 0 ? (pos / chunk) * chunk : 0;
    s.wlo = window > 0 ? max(s.lo, pos - window + 1) : s.lo;
    s.nfirst = (window > 0 && keep_first > s.lo) ? max(0, min(keep_first, s.wlo) - s.lo) : 0;
    s.n = s.nfirst + (last - s.wlo + 1);
    return s;
}
// what the masks leave of key j for the query at position i
__device__ __forceinline__ bool key_visible(int i, int j, int lo_i, int window, int keep_first) {
    return j <= i && j >= lo_i && (window <= 0 || i - j < window || j < keep_first);
}

// sigmoid of a score that is already in the exponent of 2
__device__ __forceinline__ float sigmoid2_f(float x2) { return __fdividef(1.f, 1.f + b2::fast_exp2(-x2)); }

// What happens to a score before its weight is taken, and to a head's output after the values are summed.
struct HeadShape {
    float cap;               // > 0: scores become cap * tanh(score / cap)
    float lambda;            // two maps: output = a1 - lambda * a2 ...
    float eps, out_scale;    // ... / sqrt(mean(output^2) + eps) * out_scale
};
// cap * tanh(s / cap); tanh x = 1 - 2 / (1 + e^2x), whose absolute error (times cap) is that of one fp32 rounding
__device__ __forceinline__ float cap_score(float s, float cap, float e_scale) {
    return fmaf(-cap, __fdividef(2.f, 1.f + b2::fast_exp2(s * e_scale)), cap);
}
__device__ __forceinline__ float cap_score_exact(float s, float cap) { return cap * tanhf(s / cap); }
#endif
