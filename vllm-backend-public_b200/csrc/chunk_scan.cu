// chunk_scan.cu -- the scan of delta_rule.cu for prompts: S <- g S, u = beta (v - S^T k) (or u = v), S <- S + k u^T, o = S^T q, in
// chunks of 64 tokens instead of token after token, everything in fp32 on the FMA pipe.
//
// With G_t the product of the chunk's decays up to token t (per head, or per key channel), S_0 the state before the chunk and
// every ratio G_t / G_s taken as the product g_{s+1} .. g_t (decays are only ever multiplied, nothing is divided by a product that
// may have underflowed):
//   A[t, s] = beta_t sum_i k_t k_s G_t/G_s  (s < t),    T = (I + A)^-1 diag(beta),     P[t, s] = sum_i q_t k_s G_t/G_s  (s <= t)
//   U = T (V - (G K) S_0)   (no delta: U = V),   S = G_C S_0 + (G_C/G K)^T U,   O = (G Q) S_0 + P U
// Nothing above a diagonal is multiplied: a product that counts no later token must not become NaN by an infinity or NaN in one, so zeros
// there are selected or left out, and a token's output depends on it and earlier ones alone, as in the scan token by token.
// It is the same recurrence summed in another order (the WY form of Yang et al., "Parallelizing linear transformers with the
// delta rule over sequence length", 2024).  One decay per head without delta goes to chunk_tc5.cu; the others are three kernels, only the
// second of which is a chain:
//   chunk_prep_kernel    P, T and the decay products; without delta also F = (G_C/G K)^T V: a CTA per (chunk, head)
//   chunk_state_kernel   without delta: S <- G_C S + F over the chunks, element by element (memory bound)
//   chunk_delta_kernel   with delta: U and S over the chunks, a CTA per (sequence, head, 16 columns of S)
//   chunk_out_kernel     O of every chunk from its S_0: a CTA per (chunk, head, 128 columns)
// What bounds them: the first and last are products on the FMA pipe with 8 x 8 / 4 x 8 tiles a thread (shared-memory reads cost
// about 0.7 of the FMA cycles); the delta chain is a chain of 64-token steps of [64 x dk][dk x 16], [64 x 64][64 x 16] and
// [dk x 64][64 x 16], bound by shared-memory reads and their latency.  Sixteen columns a CTA fill the chip with one sequence of 16
// heads of 128.  The scan token by token waited 200 - 400 cycles a token for shuffles and shared memory whatever the shape.
#include "b2_act.cuh"

#include <float.h>
#include <math.h>
#include <type_traits>

namespace {

constexpr int C = 64, NC = 16, NT = 256, JB = 128, LP = C + 4;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(b2::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Scratch of one (chunk, head), in floats: P | T (delta) | products | S_0 (first F) | U (delta)
struct Scratch {
    int t, dec, s0, u, total;
    __host__ __device__ Scratch(int dk, int dv, bool ch, bool delta) {
        t = C * C;
        dec = t + (delta ? C * C : 0);
        s0 = dec + (ch ? 3 * C * dk + dk : 2 * C);   // per channel: G K | G Q | G_C/G K | G_C; per head: G | G_C/G
        u = s0 + dk * dv;
        total = u + (delta ? C * dv : 0);
    }
};

struct ChunkArgs {
    const float *qkv, *beta, *decay;
    int H, G, dk, dv, n_seq;
    const int32_t *cu_q, *ctx_start, *state_slot;
    float *state, *o, *ws;
};

// chunk number -> first batch row and number of rows (row < 0: a spare CTA)
__device__ __forceinline__ void find_chunk(const ChunkArgs& a, int want, int* at) {
    at[0] = -1;
    for (int s = 0; s < a.n_seq; ++s) {
        if (a.ctx_start[s] < 0) continue;
        const int len = a.cu_q[s + 1] - a.cu_q[s], nc = (len + C - 1) / C;
        if (want < nc) {
            at[0] = a.cu_q[s] + want * C;
            at[1] = min(C, len - want * C);
            return;
        }
        want -= nc;
    }
}
__device__ __forceinline__ int first_chunk(const ChunkArgs& a, int seq) {
    int base = 0;
    for (int s = 0; s < seq; ++s)
        if (a.ctx_start[s] >= 0) base += (a.cu_q[s + 1] - a.cu_q[s] + C - 1) / C;
    return base;
}
// Two FMAs an instruction on register pairs: the rate is that of two (73 TFLOP/s either way), but half the issue slots, which the
// shared-memory reads need.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t dup(float x) {
    pair_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void fma2(pair_t& acc, pair_t x, pair_t y) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y)); }
__device__ __forceinline__ float2 halves(pair_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ ulonglong2 pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ float4 unpack(pair_t lo, pair_t hi) {
    const float2 a = halves(lo), b = halves(hi);
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 scaled(const float4& v, float f) { return make_float4(v.x * f, v.y * f, v.z * f, v.w * f); }

// ---------------------------------------------------------------------------------------------------------------- prep
template <bool CH, bool DELTA>
__global__ void __launch_bounds__(NT)
chunk_prep_kernel(const ChunkArgs a) {
    static_assert(CH || DELTA, "chunk_tc5.cu");
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_at[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, hh = blockIdx.y;
    const int dk = a.dk, dv = a.dv, LD = dk + 4, per = dk / 4;
    if (tid == 0) find_chunk(a, blockIdx.x, s_at);
    __syncthreads();
    const int r0 = s_at[0], nt = s_at[1];
    if (r0 < 0) return;
    float* ks = sm;                                  // [C][LD]
    float* qs = ks + C * LD;                         // [C][LD]; later (no delta) the columns of V
    float* Ps = qs + (DELTA ? C * LD : max(C * LD, C * JB));        // [C][C + 1]
    float* As = Ps + C * (C + 1);                    // [C][C + 1] (delta)
    float* gs = As + (DELTA ? C * (C + 1) : 0);      // [C], per channel [C][LD]
    float* bs = gs + (CH ? C * LD : C);              // [C] beta; per head 4 + C more
    const int Cq = 2 * a.G * dk + a.H * dv, kvh = hh / (a.H / a.G);
    const float* qrow = a.qkv + (size_t)r0 * Cq + (size_t)kvh * dk;
    const float* krow = qrow + (size_t)a.G * dk;
    for (int idx = tid; idx < C * per; idx += NT) {
        const int t = idx / per, c = (idx - t * per) * 4;
        float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k, g = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t < nt) {
            k = *reinterpret_cast<const float4*>(krow + (size_t)t * Cq + c);
            q = *reinterpret_cast<const float4*>(qrow + (size_t)t * Cq + c);
            if (CH) g = *reinterpret_cast<const float4*>(a.decay + ((size_t)(r0 + t) * a.H + hh) * dk + c);
        }
        *reinterpret_cast<float4*>(ks + t * LD + c) = k;
        *reinterpret_cast<float4*>(qs + t * LD + c) = q;
        if (CH) *reinterpret_cast<float4*>(gs + t * LD + c) = g;
    }
    if (tid < C) {
        if (!CH) gs[tid] = tid < nt ? a.decay[(size_t)(r0 + tid) * a.H + hh] : 1.f;
        if (DELTA) bs[tid] = tid < nt ? a.beta[(size_t)(r0 + tid) * a.H + hh] : 0.f;
    }
    const Scratch sc(dk, dv, CH, DELTA);
    float* out = a.ws + ((size_t)blockIdx.x * a.H + hh) * sc.total;
    float* dec = out + sc.dec;
    __syncthreads();
    // sums over dk of rows x (q, and with delta k) times columns k_s: 16 x 16 threads, rows rg + 16 rr, columns cg + 16 cc
    const int rg = tid >> 4, cg = tid & 15;
    if (CH) {
        // inside a half of 32 tokens a warp takes a column s: k_s times the running product of the decays, dotted with every later row
        for (int s = wid; s < C; s += NT / 32) {
            float w[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) w[m] = lane + 32 * m < dk ? ks[s * LD + lane + 32 * m] : 0.f;
            for (int t = lane; t < s; t += 32) {
                Ps[t * (C + 1) + s] = 0.f;
                if (DELTA) As[t * (C + 1) + s] = 0.f;
            }
            for (int t = s; t < (s < 32 ? 32 : C); ++t) {
                float dq = 0.f, dd = 0.f;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int i = lane + 32 * m;
                    if (i < dk) {
                        if (t > s) w[m] *= gs[t * LD + i];
                        dq = fmaf(w[m], qs[t * LD + i], dq);
                        if (DELTA) dd = fmaf(w[m], ks[t * LD + i], dd);
                    }
                }
                if (DELTA) {                         // both sums in one butterfly: the lower half carries the first, the upper the second
                    const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? dd : dq, 16);
                    float v = (lane < 16 ? dq : dd) + other;
#pragma unroll
                    for (int x = 8; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
                    if (lane == 0) Ps[t * (C + 1) + s] = v;
                    if (lane == 16) As[t * (C + 1) + s] = t > s ? bs[t] * v : 0.f;
                } else {
                    dq = b2::warp_sum(dq);
                    if (lane == 0) Ps[t * (C + 1) + s] = dq;
                }
            }
        }
        __syncthreads();
        // across the halves: rows 32 .. 63 decayed from the boundary, columns 0 .. 31 decayed to it, then a plain product; the copies
        // for the chain are written on the way
        const int i = tid & 127;
        if (i < dk) {
            if (tid < 128) {
                float run = 1.f;
                for (int t = 0; t < 32; ++t) {
                    run *= gs[t * LD + i];
                    dec[t * dk + i] = run * ks[t * LD + i];
                    dec[(C + t) * dk + i] = run * qs[t * LD + i];
                }
                float half = 1.f;
                for (int t = 32; t < C; ++t) {
                    half *= gs[t * LD + i];
                    const float k = half * ks[t * LD + i], q = half * qs[t * LD + i];
                    dec[t * dk + i] = run * k;
                    dec[(C + t) * dk + i] = run * q;
                    qs[t * LD + i] = q;              // this thread's channel: nobody else reads it before the barrier
                }
                dec[3 * C * dk + i] = run * half;
            }
        }
        __syncthreads();                             // the later half's keys are still as they came: their copy to the chunk's end
        if (i < dk && tid >= 128) {
            float run = 1.f;
            for (int t = C - 1; t >= 32; --t) {
                const float k = ks[t * LD + i], g = gs[t * LD + i];
                dec[(2 * C + t) * dk + i] = run * k;
                run *= g;
            }
            float half = 1.f;
            for (int t = 31; t >= 0; --t) {
                const float k = half * ks[t * LD + i];
                dec[(2 * C + t) * dk + i] = run * k;
                ks[t * LD + i] = k;
                half *= gs[t * LD + i];
            }
            if (DELTA) {                             // keys 32 .. 63 decayed from the boundary
                float from = 1.f;
                for (int t = 32; t < C; ++t) {
                    from *= gs[t * LD + i];
                    ks[t * LD + i] *= from;
                }
            }
        }
        __syncthreads();
        float acc[DELTA ? 4 : 2][2];
#pragma unroll
        for (int r = 0; r < (DELTA ? 4 : 2); ++r) acc[r][0] = acc[r][1] = 0.f;
        for (int x = 0; x < dk; x += 4) {
            const float4 k0 = *reinterpret_cast<const float4*>(ks + cg * LD + x), k1 = *reinterpret_cast<const float4*>(ks + (cg + 16) * LD + x);
#pragma unroll
            for (int r = 0; r < (DELTA ? 4 : 2); ++r) {
                const float4 v = *reinterpret_cast<const float4*>((r < 2 ? qs : ks) + (32 + rg + 16 * (r & 1)) * LD + x);
                acc[r][0] = fmaf(v.x, k0.x, acc[r][0]); acc[r][0] = fmaf(v.y, k0.y, acc[r][0]);
                acc[r][0] = fmaf(v.z, k0.z, acc[r][0]); acc[r][0] = fmaf(v.w, k0.w, acc[r][0]);
                acc[r][1] = fmaf(v.x, k1.x, acc[r][1]); acc[r][1] = fmaf(v.y, k1.y, acc[r][1]);
                acc[r][1] = fmaf(v.z, k1.z, acc[r][1]); acc[r][1] = fmaf(v.w, k1.w, acc[r][1]);
            }
        }
#pragma unroll
        for (int r = 0; r < (DELTA ? 4 : 2); ++r) {
            const int t = 32 + rg + 16 * (r & 1);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (r < 2) Ps[t * (C + 1) + cg + 16 * c] = acc[r][c];
                else As[t * (C + 1) + cg + 16 * c] = bs[t] * acc[r][c];
            }
        }
    } else {
        // the decay ratios of all (t, s), and the products from the chunk's start and to its end: by segments of 16 tokens, a chain of
        // 16 + 16 products instead of 64
        float* seg = As + (DELTA ? C * (C + 1) : 0) + 2 * C;         // behind g and beta: [4] segments | [C] from s + 1 to the end of its segment
        float* tail = seg + 4;
        const int col = tid & (C - 1), sg = tid >> 6, own = col >> 4;
        if (tid < C) {
            float run = 1.f;
            for (int r = tid + 1; r < (tid | 15) + 1; ++r) run *= gs[r];
            tail[tid] = run;
            if ((tid & 15) == 0) seg[tid >> 4] = run * gs[tid];
        }
        __syncthreads();
        {
            float run = tail[col];
            for (int m = own + 1; m < sg; ++m) run *= seg[m];
            if (sg == own) run = 1.f;
#pragma unroll 4
            for (int t = sg * 16; t < sg * 16 + 16; ++t) {
                if (t > col) run *= gs[t];
                Ps[t * (C + 1) + col] = t >= col ? run : 0.f;
            }
        }
        if (tid < C) {
            float to = tail[tid], from = 1.f;
            for (int m = own + 1; m < 4; ++m) to *= seg[m];
            for (int m = 0; m < own; ++m) from *= seg[m];
            for (int r = own * 16; r <= tid; ++r) from *= gs[r];
            dec[tid] = from;
            dec[C + tid] = to;
        }
        __syncthreads();
        pair_t acc[8][4];                            // sums over even and odd entries; blocks above the diagonal are left out
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0;
        for (int i = 0; i < dk; i += 4) {
            ulonglong2 kc[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) kc[c] = pairs(ks + (cg + 16 * c) * LD + i);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const ulonglong2 x = pairs((r < 4 ? qs : ks) + (rg + 16 * (r & 3)) * LD + i);
#pragma unroll
                for (int c = 0; c <= (r & 3); ++c) {
                    fma2(acc[r][c], x.x, kc[c].x);
                    fma2(acc[r][c], x.y, kc[c].y);
                }
            }
        }
#pragma unroll
        for (int r = 7; r >= 0; --r) {          // the k rows still need the ratios that the q rows overwrite (same thread)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int t = rg + 16 * (r & 3), x = cg + 16 * c;
                const float2 h = halves(acc[r][c]);
                const float v = t >= x ? (h.x + h.y) * Ps[t * (C + 1) + x] : 0.f;
                if (r < 4) Ps[t * (C + 1) + x] = v;
                else As[t * (C + 1) + x] = t > x ? bs[t] * v : 0.f;
            }
        }
    }
    __syncthreads();
    for (int idx = tid; idx < C * C; idx += NT) out[idx] = Ps[(idx / C) * (C + 1) + idx % C];
    if (DELTA) {
        // the inverse of I + A by halves: forward substitution on the diagonal blocks (a warp each, a lane per column), then
        // T21 = -T22 A21 T11; Ps is free and takes T
        if (wid >= 6) {
            const int o = wid == 6 ? 0 : 32;
            float T[32];
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                float v = t == lane ? 1.f : 0.f;
#pragma unroll
                for (int s = 0; s < t; ++s) v = fmaf(-As[(o + t) * (C + 1) + o + s], T[s], v);
                T[t] = v;
            }
            __syncwarp();
            asm volatile("bar.sync 1, 64;" ::: "memory");            // both warps are done reading A's diagonal blocks ...
#pragma unroll
            for (int t = 0; t < 32; ++t) As[(o + t) * (C + 1) + o + lane] = T[t];        // ... whose place T takes
        }
        __syncthreads();
        float* x = Ps;                               // A21 T11, [32][C + 1]
        const int row = tid >> 3, c4 = (tid & 7) * 4;
        {
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            for (int s = 0; s < 32; ++s) {
                const float l = As[(32 + row) * (C + 1) + s];
#pragma unroll
                for (int c = 0; c < 4; ++c) v[c] = fmaf(l, As[s * (C + 1) + c4 + c], v[c]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) x[row * (C + 1) + c4 + c] = v[c];
        }
        __syncthreads();
        {
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            for (int s = 0; s <= row; ++s) {
                const float l = As[(32 + row) * (C + 1) + 32 + s];
#pragma unroll
                for (int c = 0; c < 4; ++c) v[c] = fmaf(-l, x[s * (C + 1) + c4 + c], v[c]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) As[(32 + row) * (C + 1) + c4 + c] = v[c];        // A21 was read before the last barrier
        }
        __syncthreads();
        float* to = out + sc.t;
        for (int idx = tid; idx < C * C; idx += NT) {
            const int t = idx / C, s = idx % C;
            to[idx] = s <= t ? As[t * (C + 1) + s] * bs[s] : 0.f;
        }
    } else {
        // F = (G_C/G K)^T V, 128 columns at a time, 8 x 8 results a thread: rows 8 ti .., columns 4 tj .. and 64 + 4 tj ..
        const int ti = tid >> 4, tj = tid & 15;
        const float* vrow = a.qkv + (size_t)r0 * Cq + (size_t)2 * a.G * dk + (size_t)hh * dv;
        float* f0 = out + sc.s0;
        for (int idx = tid; idx < C * per; idx += NT) {              // the keys decayed to the chunk's end, from where they were just written
            const int t = idx / per, c = (idx - t * per) * 4;
            *reinterpret_cast<float4*>(ks + t * LD + c) = *reinterpret_cast<const float4*>(dec + (2 * C + t) * dk + c);
        }
        float* vs = qs;
        for (int j0 = 0; j0 < dv; j0 += JB) {
            __syncthreads();
            for (int idx = tid; idx < C * (JB / 4); idx += NT) {
                const int t = idx / (JB / 4), c = (idx % (JB / 4)) * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t < nt && j0 + c < dv) v = *reinterpret_cast<const float4*>(vrow + (size_t)t * Cq + j0 + c);
                *reinterpret_cast<float4*>(vs + t * JB + c) = v;
            }
            __syncthreads();
            if (ti * 8 < dk) {
                pair_t acc[8][4];
#pragma unroll
                for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0;
                const int hi = min(ti * 8 + 4, dk - 4);              // heads of 4 (mod 8) entries: a second look at the last four
#pragma unroll 4
                for (int t = 0; t < C; ++t) {
                    const float4 x0 = *reinterpret_cast<const float4*>(ks + t * LD + ti * 8), x1 = *reinterpret_cast<const float4*>(ks + t * LD + hi);
                    const ulonglong2 y0 = pairs(vs + t * JB + tj * 4), y1 = pairs(vs + t * JB + 64 + tj * 4);
                    const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const pair_t xx = dup(x[r]);
                        fma2(acc[r][0], xx, y0.x);
                        fma2(acc[r][1], xx, y0.y);
                        fma2(acc[r][2], xx, y1.x);
                        fma2(acc[r][3], xx, y1.y);
                    }
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int i = r < 4 ? ti * 8 + r : hi + r - 4;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const int j = j0 + b * 64 + tj * 4;
                        if (j < dv) *reinterpret_cast<float4*>(f0 + (size_t)i * dv + j) = unpack(acc[r][2 * b], acc[r][2 * b + 1]);
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------- state, no delta
__global__ void __launch_bounds__(NT)
chunk_state_kernel(const ChunkArgs a) {
    const int seq = blockIdx.x, hh = blockIdx.y;
    const int ctx = a.ctx_start[seq];
    if (ctx < 0) return;
    const int dk = a.dk, dv = a.dv, e = (blockIdx.z * blockDim.x + threadIdx.x) * 4;
    if (e >= dk * dv) return;
    const int nchunks = (a.cu_q[seq + 1] - a.cu_q[seq] + C - 1) / C;
    if (nchunks == 0) return;
    const Scratch sc(dk, dv, true, false);
    const size_t step = (size_t)a.H * sc.total;
    float* w = a.ws + ((size_t)first_chunk(a, seq) * a.H + hh) * sc.total;
    const float* g = w + sc.dec + 3 * C * dk + e / dv;        // the chunk's whole product
    float* f = w + sc.s0 + e;
    const int slot = a.state_slot[seq];
    float* sp = slot >= 0 ? a.state + ((size_t)slot * a.H + hh) * dk * dv + e : nullptr;
    float4 s = sp && ctx > 0 ? *reinterpret_cast<const float4*>(sp) : make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int AHEAD = 6;                         // loads in flight: they do not depend on the chain
    float4 x[AHEAD];
    float d[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
        if (u < nchunks) {
            x[u] = *reinterpret_cast<const float4*>(f + u * step);
            d[u] = g[u * step];
        }
    for (int c0 = 0; c0 < nchunks; c0 += AHEAD) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int c = c0 + u;
            if (c < nchunks) {
                *reinterpret_cast<float4*>(f + c * step) = s;
                s = make_float4(fmaf(s.x, d[u], x[u].x), fmaf(s.y, d[u], x[u].y), fmaf(s.z, d[u], x[u].z), fmaf(s.w, d[u], x[u].w));
                if (c + AHEAD < nchunks) {
                    x[u] = *reinterpret_cast<const float4*>(f + (c + AHEAD) * step);
                    d[u] = g[(c + AHEAD) * step];
                }
            }
        }
    }
    if (sp) *reinterpret_cast<float4*>(sp) = s;
}

// ---------------------------------------------------------------------------------------------------------------- state, delta
__host__ __device__ constexpr int delta_stage(int dk, bool ch) { return (ch ? 2 : 1) * C * (dk + 4) + C * NC + C * LP + (ch ? dk : 2 * C); }
__host__ __device__ constexpr int delta_fixed(int dk) { return dk * NC + 2 * 4 * C * NC + 2 * C * NC; }

template <bool CH>
__global__ void __launch_bounds__(NT)
chunk_delta_kernel(const ChunkArgs a, int stages) {
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    // CTAs start in the order of their sequences' lengths, the longest first: 3 sequences of 16 heads are 384 chains on
    // 296 places (1500 + 1000 + 501 tokens, whole scan: 393 us in the order of the batch, 342 so)
    __shared__ int s_seq;
    for (int i = tid; i < a.n_seq; i += NT) {
        const int len = a.cu_q[i + 1] - a.cu_q[i];
        int rank = 0;
        for (int j = 0; j < a.n_seq; ++j) {
            const int other = a.cu_q[j + 1] - a.cu_q[j];
            rank += other > len || (other == len && j < i);
        }
        if (rank == blockIdx.z) s_seq = i;
    }
    __syncthreads();
    const int seq = s_seq, hh = blockIdx.y, j0 = blockIdx.x * NC;
    const int ctx = a.ctx_start[seq];
    if (ctx < 0) return;
    const int dk = a.dk, dv = a.dv, H = a.H, LD = dk + 4, per = dk / 4;
    const int r0 = a.cu_q[seq], n = a.cu_q[seq + 1] - r0, nchunks = (n + C - 1) / C, base = first_chunk(a, seq);
    const int Cq = 2 * a.G * dk + H * dv, kvh = hh / (H / a.G);
    const int slot = a.state_slot[seq];
    const int cols = min(NC, dv - j0);               // a multiple of 4
    const Scratch sc(dk, dv, CH, true);
    float* S = sm;                                   // [dk][NC]
    float* redA = S + dk * NC;                       // [4][C][NC]: partial products with the state
    float* redB = redA + 4 * C * NC;                 // [4][C][NC]: partial products with T
    float* Rm = redB + 4 * C * NC;                   // [C][NC] V - (G K) S
    float* Ud = Rm + C * NC;                         // [C][NC] U, times the decay to the chunk's end (decay per head)
    float* st0 = Ud + C * NC;
    const int stage_floats = delta_stage(dk, CH);

    auto issue = [&](int c, int buf) {
        float* ks = st0 + (size_t)buf * stage_floats;
        float* ku = ks + C * LD;                     // per channel only
        float* vs = ku + (CH ? C * LD : 0);
        float* ts = vs + C * NC;
        float* de = ts + C * LP;
        const int t0 = c * C, nt = min(C, n - t0);
        const float* ws = a.ws + ((size_t)(base + c) * H + hh) * sc.total;
        const float* dec = ws + sc.dec;
        const float* krow = a.qkv + (size_t)(r0 + t0) * Cq + (size_t)(a.G + kvh) * dk;
        const float* vrow = a.qkv + (size_t)(r0 + t0) * Cq + (size_t)2 * a.G * dk + (size_t)hh * dv + j0;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int idx = tid; idx < C * per; idx += NT) {
            const int t = idx / per, x = (idx - t * per) * 4;
            if (CH) {                                // the decayed copies; rows past the end are zeros there
                cp_async16(ks + t * LD + x, dec + t * dk + x);
                cp_async16(ku + t * LD + x, dec + (2 * C + t) * dk + x);
            } else if (t < nt) {
                cp_async16(ks + t * LD + x, krow + (size_t)t * Cq + x);
            } else {
                *reinterpret_cast<float4*>(ks + t * LD + x) = zero;
            }
        }
        {
            const int t = tid / (NC / 4), x = (tid % (NC / 4)) * 4;  // 64 rows x 4 vectors
            if (t < nt && x < cols) cp_async16(vs + t * NC + x, vrow + (size_t)t * Cq + x);
            else *reinterpret_cast<float4*>(vs + t * NC + x) = zero;
        }
        for (int idx = tid; idx < C * (C / 4); idx += NT) cp_async16(ts + (idx / (C / 4)) * LP + (idx % (C / 4)) * 4, ws + sc.t + idx * 4);
        const int nd = CH ? per : 2 * C / 4;
        if (tid < nd) cp_async16(de + tid * 4, dec + (CH ? 3 * C * dk : 0) + tid * 4);
        cp_commit();
    };

    // this thread's part of the state: rows i0 .. i0 + 3, columns jc, jc + 1
    const int i0 = (tid >> 3) * 4, jc = (tid & 7) * 2;
    const bool mine = i0 < dk, in_cols = jc < cols;
    float* sp = slot >= 0 ? a.state + ((size_t)slot * H + hh) * dk * dv + j0 + jc : nullptr;
    float2 s[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        s[r] = make_float2(0.f, 0.f);
        if (mine && in_cols && sp && ctx > 0) s[r] = *reinterpret_cast<const float2*>(sp + (size_t)(i0 + r) * dv);
        if (mine) *reinterpret_cast<float2*>(S + (i0 + r) * NC + jc) = s[r];
    }
    const int rg = lane >> 2, cg = lane & 3;         // products: rows 32 (w / 4) + rg + 8 rr, columns 4 cg .. 4 cg + 3
    const int half = w >> 2, kq = w & 3;
    if (nchunks > 0) issue(0, 0);
    for (int c = 0; c < nchunks; ++c) {
        const int buf = stages == 2 ? c & 1 : 0;
        cp_wait<0>();
        __syncthreads();                             // the chunk's operands and S are there; the last chunk's stage is read
        if (stages == 2 && c + 1 < nchunks) issue(c + 1, buf ^ 1);
        const float* ks = st0 + (size_t)buf * stage_floats;
        const float* ku = CH ? ks + C * LD : ks;
        const float* vs = ks + (CH ? 2 : 1) * C * LD;
        const float* ts = vs + C * NC;
        const float* de = ts + C * LP;
        const int nt = min(C, n - c * C);
        float* ws = a.ws + ((size_t)(base + c) * H + hh) * sc.total;
        if (mine && in_cols) {
            float* s0 = ws + sc.s0 + (size_t)i0 * dv + j0 + jc;
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float2*>(s0 + (size_t)r * dv) = s[r];
        }
        {   // K S, a quarter of dk a warp
            const float* rows = ks + (half * 32 + rg) * LD;
            const int span = (per + 3) / 4 * 4, k0 = kq * span, k1 = min(k0 + span, dk);
            pair_t acc[4][2];
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0;
#pragma unroll 2
            for (int i = k0; i < k1; i += 4) {
                float4 x[4];
                ulonglong2 y[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(rows + r * 8 * LD + i);
#pragma unroll
                for (int q = 0; q < 4; ++q) y[q] = pairs(S + (i + q) * NC + cg * 4);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float xv[4] = {x[r].x, x[r].y, x[r].z, x[r].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const pair_t xx = dup(xv[q]);
                        fma2(acc[r][0], xx, y[q].x);
                        fma2(acc[r][1], xx, y[q].y);
                    }
                }
            }
            float* dst = redA + (kq * C + half * 32 + rg) * NC + cg * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(dst + r * 8 * NC) = unpack(acc[r][0], acc[r][1]);
        }
        __syncthreads();
        const int t = tid >> 2, x4 = (tid & 3) * 4;  // the small matrices: four columns of a row a thread
        bool bad;
        {
            const float f = CH ? 1.f : de[t];
            const float4 v = *reinterpret_cast<const float4*>(vs + t * NC + x4);
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 y = *reinterpret_cast<const float4*>(redA + (q * C + t) * NC + x4);
                p = make_float4(p.x + y.x, p.y + y.y, p.z + y.z, p.w + y.w);
            }
            p = make_float4(fmaf(-f, p.x, v.x), fmaf(-f, p.y, v.y), fmaf(-f, p.z, v.z), fmaf(-f, p.w, v.w));
            *reinterpret_cast<float4*>(Rm + t * NC + x4) = p;
            bad = !(fabsf(p.x) + fabsf(p.y) + fabsf(p.z) + fabsf(p.w) <= FLT_MAX);
        }
        bad = __syncthreads_or(bad);                 // only then T's zeros above the diagonal have to be left out
        {   // T R, columns 16 it + 4 kq of T
            pair_t acc[4][2];
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0;
            auto product = [&](auto select) {
                for (int it = 0; it < (half == 0 ? 2 : 4); ++it) {
                    const int s0 = it * 16 + kq * 4;
                    float4 x[4];
                    ulonglong2 y[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(ts + (half * 32 + rg + 8 * r) * LP + s0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) y[q] = pairs(Rm + (s0 + q) * NC + cg * 4);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float xv[4] = {x[r].x, x[r].y, x[r].z, x[r].w};
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            if (decltype(select)::value && s0 + q > half * 32 + rg + 8 * r) continue;
                            const pair_t xx = dup(xv[q]);
                            fma2(acc[r][0], xx, y[q].x);
                            fma2(acc[r][1], xx, y[q].y);
                        }
                    }
                }
            };
            if (bad) product(std::true_type());
            else product(std::false_type());
            float* dst = redB + (kq * C + half * 32 + rg) * NC + cg * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(dst + r * 8 * NC) = unpack(acc[r][0], acc[r][1]);
        }
        __syncthreads();
        {
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 y = *reinterpret_cast<const float4*>(redB + (q * C + t) * NC + x4);
                p = make_float4(p.x + y.x, p.y + y.y, p.z + y.z, p.w + y.w);
            }
            if (x4 < cols) *reinterpret_cast<float4*>(ws + sc.u + (size_t)t * dv + j0 + x4) = p;
            *reinterpret_cast<float4*>(Ud + t * NC + x4) = CH ? p : scaled(p, de[C + t]);
        }
        __syncthreads();
        if (mine) {                                  // S = G_C S + (decayed K)^T U
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float f = CH ? de[i0 + r] : de[C - 1];
                s[r].x *= f;
                s[r].y *= f;
            }
#pragma unroll 8
            for (int u = 0; u < nt; ++u) {
                const float4 k = *reinterpret_cast<const float4*>(ku + u * LD + i0);
                const float2 x = *reinterpret_cast<const float2*>(Ud + u * NC + jc);
                s[0].x = fmaf(k.x, x.x, s[0].x); s[0].y = fmaf(k.x, x.y, s[0].y);
                s[1].x = fmaf(k.y, x.x, s[1].x); s[1].y = fmaf(k.y, x.y, s[1].y);
                s[2].x = fmaf(k.z, x.x, s[2].x); s[2].y = fmaf(k.z, x.y, s[2].y);
                s[3].x = fmaf(k.w, x.x, s[3].x); s[3].y = fmaf(k.w, x.y, s[3].y);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float2*>(S + (i0 + r) * NC + jc) = s[r];
        }
        if (stages == 1 && c + 1 < nchunks) {
            __syncthreads();                         // the single stage is read
            issue(c + 1, 0);
        }
    }
    if (sp && mine && in_cols && nchunks > 0) {
#pragma unroll
        for (int r = 0; r < 4; ++r) *reinterpret_cast<float2*>(sp + (size_t)(i0 + r) * dv) = s[r];
    }
}

// ---------------------------------------------------------------------------------------------------------------- output
// [64 x (dk + 64)] times [(dk + 64) x 128]: the rows [ G Q | P ] stay in shared memory, the rows of S_0 and of U (or V) stream through
// two stages of 32.  Rows 4 rg .., columns 4 tj .. and 64 + 4 tj .. a thread.
template <bool CH, bool DELTA>
__global__ void __launch_bounds__(NT, 2)
chunk_out_kernel(const ChunkArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_at[2];
    const int tid = threadIdx.x, hh = blockIdx.y, j0 = blockIdx.z * JB;
    const int dk = a.dk, dv = a.dv, LD = dk + 4, per = dk / 4;
    if (tid == 0) find_chunk(a, blockIdx.x, s_at);
    __syncthreads();
    const int r0 = s_at[0], nt = s_at[1];
    if (r0 < 0) return;
    float* qs = sm;                                  // [C][LD]
    float* ps = qs + C * LD;                         // [C][LP]
    float* bsm = ps + C * LP;                        // [2][32][JB]
    const int Cq = 2 * a.G * dk + a.H * dv, kvh = hh / (a.H / a.G);
    const Scratch sc(dk, dv, CH, DELTA);
    const float* ws = a.ws + ((size_t)blockIdx.x * a.H + hh) * sc.total;
    const float* dec = ws + sc.dec;
    const float* vrow = a.qkv + (size_t)r0 * Cq + (size_t)2 * a.G * dk + (size_t)hh * dv;
    const int n1 = (dk + 31) / 32, n2 = (nt + 31) / 32;              // slices of S_0, slices of U
    auto issue = [&](int sl, int buf) {
        const bool second = sl >= n1;
        const int k0 = (second ? sl - n1 : sl) * 32, rows = second ? nt : dk;
        for (int idx = tid; idx < 32 * (JB / 4); idx += NT) {
            const int r = idx / (JB / 4), c = (idx % (JB / 4)) * 4;
            float* dst = bsm + ((size_t)buf * 32 + r) * JB + c;
            const float* src = !second ? ws + sc.s0 + (size_t)(k0 + r) * dv + j0 + c
                             : DELTA ? ws + sc.u + (size_t)(k0 + r) * dv + j0 + c : vrow + (size_t)(k0 + r) * Cq + j0 + c;
            if (k0 + r < rows && j0 + c < dv) cp_async16(dst, src);
            else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        cp_commit();
    };
    issue(0, 0);
    for (int idx = tid; idx < C * per; idx += NT) {
        const int t = idx / per, c = (idx - t * per) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (CH) q = *reinterpret_cast<const float4*>(dec + (C + t) * dk + c);
        else if (t < nt) q = scaled(*reinterpret_cast<const float4*>(a.qkv + (size_t)(r0 + t) * Cq + (size_t)kvh * dk + c), dec[t]);
        *reinterpret_cast<float4*>(qs + t * LD + c) = q;
    }
    for (int idx = tid; idx < C * (C / 4); idx += NT)
        *reinterpret_cast<float4*>(ps + (idx / (C / 4)) * LP + (idx % (C / 4)) * 4) = *reinterpret_cast<const float4*>(ws + idx * 4);
    const int rg = tid >> 4, tj = tid & 15;
    pair_t acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0;
    for (int sl = 0; sl < n1 + n2; ++sl) {
        cp_wait<0>();
        __syncthreads();                             // slice sl is there, the other stage is read
        if (sl + 1 < n1 + n2) issue(sl + 1, (sl + 1) & 1);
        const bool second = sl >= n1;
        const int k0 = (second ? sl - n1 : sl) * 32;
        const int ld = second ? LP : LD;
        const float* rows = (second ? ps : qs) + (size_t)(rg * 4) * ld + k0;
        const float* b = bsm + (size_t)(sl & 1) * 32 * JB + tj * 4;
        auto block = [&](int k, auto diagonal) {     // four columns; on P's diagonal a row takes those up to its own
            float4 x[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(rows + r * ld + k);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2 y0 = pairs(b + (k + q) * JB), y1 = pairs(b + (k + q) * JB + 64);
#pragma unroll
                for (int r = decltype(diagonal)::value ? q : 0; r < 4; ++r) {
                    const pair_t xx = dup(q == 0 ? x[r].x : q == 1 ? x[r].y : q == 2 ? x[r].z : x[r].w);
                    fma2(acc[r][0], xx, y0.x);
                    fma2(acc[r][1], xx, y0.y);
                    fma2(acc[r][2], xx, y1.x);
                    fma2(acc[r][3], xx, y1.y);
                }
            }
        };
        const int kn = second ? min(32, rg * 4 - k0) : min(32, dk - k0);     // of P nothing above the diagonal
#pragma unroll 2
        for (int k = 0; k < kn; k += 4) block(k, std::false_type());
        if (second && kn >= 0 && kn < 32) block(kn, std::true_type());
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int t = rg * 4 + r;
        if (t < nt) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int j = j0 + b * 64 + tj * 4;
                if (j < dv)
                    *reinterpret_cast<float4*>(a.o + ((size_t)(r0 + t) * a.H + hh) * dv + j) = unpack(acc[r][2 * b], acc[r][2 * b + 1]);
            }
        }
    }
}

template <typename K>
int allow(K kern, size_t bytes) {
    if (bytes > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return B2_OK;
}

template <bool CH, bool DELTA>
int launch(const ChunkArgs& a, int total_rows, cudaStream_t st) {
    const int n_sm = b2_sm_count();
    const int chunks = total_rows / C + a.n_seq;     // upper bound on sum(ceil(len / C)); spare CTAs leave at once
    const size_t LD = a.dk + 4, rows = C * LD;
    const size_t psm = sizeof(float) * (rows + (DELTA ? rows : (rows > C * JB ? rows : C * JB)) + (DELTA ? 2 : 1) * C * (C + 1) + (CH ? rows : 2 * C + 4) + C);
    int rc = allow(chunk_prep_kernel<CH, DELTA>, psm);
    if (rc != B2_OK) return rc;
    chunk_prep_kernel<CH, DELTA><<<dim3(chunks, a.H), NT, psm, st>>>(a);
    if constexpr (DELTA) {
        const dim3 grid((a.dv + NC - 1) / NC, a.H, a.n_seq);
        const size_t stage = sizeof(float) * (size_t)delta_stage(a.dk, CH), fixed = sizeof(float) * (size_t)delta_fixed(a.dk);
        // two CTAs an SM cover each other's copies when there are enough of them; a lone one prefetches
        const int stages = (long)grid.x * grid.y * grid.z > n_sm || fixed + 2 * stage > 227 * 1024 ? 1 : 2;
        rc = allow(chunk_delta_kernel<CH>, fixed + stages * stage);
        if (rc != B2_OK) return rc;
        chunk_delta_kernel<CH><<<grid, NT, fixed + stages * stage, st>>>(a, stages);
    } else {
        chunk_state_kernel<<<dim3(a.n_seq, a.H, (a.dk * a.dv / 4 + 127) / 128), 128, 0, st>>>(a);
    }
    const size_t osm = sizeof(float) * (rows + C * LP + 2 * 32 * JB);
    rc = allow(chunk_out_kernel<CH, DELTA>, osm);
    if (rc != B2_OK) return rc;
    chunk_out_kernel<CH, DELTA><<<dim3(chunks, a.H, (a.dv + JB - 1) / JB), NT, osm, st>>>(a);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

}  // namespace

// Scratch (floats) of the chunked form; 0 for sizes it is not built for and for scratch above 2 GiB
int64_t b2_internal_chunk_scan_floats(int total_rows, int n_seq, int H, int dk, int dv, bool ch, bool delta) {
    if (dk % 4 || dv % 4 || dk > 128 || n_seq <= 0 || total_rows <= 0) return 0;
    const int64_t n = !ch && !delta ? b2_internal_chunk_tc5_floats(total_rows, n_seq, H, dk, dv)
                                    : (int64_t)(total_rows / C + n_seq) * H * Scratch(dk, dv, ch, delta).total;
    return n <= (int64_t)1 << 29 ? n : 0;
}

// Where the chunked form is the faster one.  Both times are estimated in us from what they measured for heads of 128 x 128 on
// one B200 (w = dk dv / 16384 scales the products); the host knows the rows and the number of sequences, so the longest of several is taken to be 1.25 times the mean:
//   tokens   a chain of 0.20 (delta 0.285, per channel 0.235 / 0.31) a token, or, with several sequences, 5.2 (7.1 / 10.6 / 12.4) ns a
//            token and head, down to 5.0 (6.3 / 6.8 / 8.3) from 64 sequences on; keys of other sizes than 32, 64, 128 run as the next one, a third slower
//   chunks   one decay per head without delta (chunk_tc5.cu): 20, 0.2 a chunk of 128 and head for the products (0.14 at 64 x 64) and 0.03 a
//            sequence and head for its state; at least 33 (29 to dk = 64): three launches
//            else 0.16 (per channel 0.55 / 0.70) a chunk of 64 and head for the products, 0.11 a sequence and head for its state, with delta
//            4.8 a step of the chain and SM's share of CTAs; at least 40 (80 per channel, 110 with delta too)
// Measured, tokens -> chunks: 1 x 4096 tokens, 16 heads: 804 -> 121, 1160 -> 470, 963 -> 572, 1254 -> 1006; 1 x 500: 102 -> 34,
// 146 -> 74, 121 -> 82, 158 -> 144; 16 x 100: 121 -> 74 the first; 64 x 64: 330 -> 258, 413 -> 567: the second is left to the tokens, as are 64 x 24: 148 -> 250,
// 147 -> 317, and 1 x 130: 29 -> 33 the first.
bool b2_internal_chunk_scan_pays(int total_rows, int n_seq, int H, int dk, int dv, bool ch, bool delta) {
    if (total_rows < 2 * n_seq) return false;
    const float len = (float)total_rows / n_seq, w = dk * dv / 16384.f, steps = ceilf(len / C), heads = (float)n_seq * H;
    const int kind = (ch ? 2 : 0) + (delta ? 1 : 0), run_as = dk <= 32 ? 32 : dk <= 64 ? 64 : 128;
    const float chain_tok[4] = {0.20f, 0.285f, 0.235f, 0.31f}, rate_few[4] = {5.2e-3f, 7.1e-3f, 10.6e-3f, 12.4e-3f}, rate_many[4] = {5.0e-3f, 6.3e-3f, 6.8e-3f, 8.3e-3f};
    const float per_chunk[4] = {0.f, 0.16f, 0.55f, 0.70f}, least[4] = {dk <= 64 ? 29.f : 33.f, 40.f, 80.f, 110.f};
    const float many = fminf(1.f, fmaxf(0.f, log2f(n_seq / 4.f) / 4.f)), rate = rate_few[kind] + (rate_many[kind] - rate_few[kind]) * many;
    const float longest = len * (n_seq > 1 ? 1.25f : 1.f);
    const float tokens = (run_as == dk ? 1.f : 1.33f) * fmaxf(chain_tok[kind] * (dk <= 64 ? 0.75f : 1.f) * longest, rate * (float)total_rows * H * run_as * dv / 16384.f);
    float chunks;
    if (kind == 0) {
        chunks = 20.f + (0.2f * (0.6f + 0.4f * w) * ceilf(len / 128) + 0.03f * w) * heads;
    } else {
        chunks = (per_chunk[kind] * (0.35f + 0.65f * w) * steps + 0.11f * w) * heads;
        if (delta) chunks += (3.4f + 1.4f * w) * fmaxf(ceilf(longest / C), steps * heads * ((dv + NC - 1) / NC) / b2_sm_count());
    }
    return tokens >= fmaxf(chunks, least[kind]);
}

int b2_internal_chunk_scan(const float* qkv, const float* beta, const float* decay, int total_rows, int H, int G, int dk, int dv,
                           bool ch, bool delta, const int32_t* cu_q, const int32_t* ctx_start, const int32_t* state_slot, int n_seq,
                           float* state, float* o, float* ws, void* stream) {
    const ChunkArgs a{qkv, beta, decay, H, G, dk, dv, n_seq, cu_q, ctx_start, state_slot, state, o, ws};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (ch) return delta ? launch<true, true>(a, total_rows, st) : launch<true, false>(a, total_rows, st);
    if (!delta) return b2_internal_chunk_tc5(qkv, decay, total_rows, H, G, dk, dv, cu_q, ctx_start, state_slot, n_seq, state, o, ws, stream);
    return launch<false, true>(a, total_rows, st);
}
