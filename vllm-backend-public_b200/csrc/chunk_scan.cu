// chunk_scan.cu -- the scan of delta_rule.cu for prompts: S <- g S, u = beta (v - S^T k) (or u = v), S <- S + k u^T, o = S^T q, in
// chunks instead of token after token.  With G_t the product of the chunk's decays up to token t (per head, or per key channel), S_0 the
// state before the chunk and every ratio G_t / G_s taken as the product g_{s+1} .. g_t (decays are only ever multiplied, nothing is
// divided by a product that may have underflowed):
//   A[t, s] = beta_t sum_i k_t k_s G_t/G_s  (s < t),    T = (I + A)^-1 diag(beta),     P[t, s] = sum_i q_t k_s G_t/G_s  (s <= t)
//   U = T (V - (G K) S_0)   (no delta: U = V),   S = G_C S_0 + (G_C/G K)^T U,   O = (G Q) S_0 + P U
// Nothing above a diagonal is multiplied: a product that counts no later token must not become NaN by an infinity or NaN in one, so zeros
// there are selected or left out, and a token's output depends on it and earlier ones alone, as in the scan token by token.
// It is the same recurrence summed in another order (the WY form of Yang et al., "Parallelizing linear transformers with the
// delta rule over sequence length", 2024).
//
// One decay per head without delta is all in chunk_tc5.cu, chunks of 128 tokens.  For the others chunk_prep_kernel here computes P, T and the
// decay products of every chunk of 64 tokens, a CTA per (chunk, head), on the FMA pipe; the rest is delta_tc5.cu's.  Per head: tiles of
// 8 x 8 / 4 x 8 a thread (shared-memory reads cost about 0.7 of the FMA cycles).  Per channel the decays stand between k and q, so
// pairs of tokens of a segment of 16 are taken one by one, and those of different segments as products of rows decayed to and
// from a boundary between them.  A warp per column with its sums in butterflies, over segments of 32, took 350 us of 4096 tokens'
// scan (16 heads of 128), this one about 110: a third of the pairs, and one transposing sum for 16 of them.  Keys and queries come four vectors in flight, P and T
// leave as vectors, and the triangular solve takes two rows at a time: 76 -> 66 us per head (3001 tokens, delta).  Products of queries and keys are
// sums of 16 entries and of these, for one more us: as one chain P was 1.1e-7 off, now 0.7e-7, and it is half of the squared error of the
// outputs.  Products of decays are taken in 64 bits.  The choice between chunks and tokens is at the end.
#include "chunk_tc5.cuh"

#include <math.h>

namespace {

constexpr int C = 64;

struct ChunkArgs {
    const float *qkv, *beta, *decay;
    int H, G, dk, dv, n_seq;
    const int32_t *cu_q, *ctx_start, *state_slot;
    float* ws;
    int first, chunks;                               // the chunks of this piece: first .. first + chunks - 1, whose scratch ws holds
    int t_at, dec_at, total;                         // scratch of a (chunk, head) in floats: P at 0, T, the decays (delta_tc5.cu)
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
// Two FMAs an instruction on register pairs: the rate is that of two (73 TFLOP/s either way), but half the issue slots, which the
// shared-memory reads need.
typedef unsigned long long pair_t;
__device__ __forceinline__ void fma2(pair_t& acc, pair_t x, pair_t y) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y)); }
__device__ __forceinline__ float2 halves(pair_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ ulonglong2 pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
// ---------------------------------------------------------------------------------------------------------------- prep
template <bool CH, bool DELTA>
__global__ void __launch_bounds__(CH ? 512 : 256)
chunk_prep_kernel(const ChunkArgs a) {
    constexpr int NT = CH ? 512 : 256;
    static_assert(CH || DELTA, "chunk_tc5.cu");
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_at[2];
    __shared__ double s_tail[CH ? 1 : C], s_seg[4];  // per head: the decays from s + 1 to the end of its segment; segments
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, hh = blockIdx.y;
    const int dk = a.dk, dv = a.dv, LD = dk + 4, per = dk / 4;
    if (tid == 0) find_chunk(a, a.first + blockIdx.x, s_at);
    __syncthreads();
    const int r0 = s_at[0], nt = s_at[1];
    if (r0 < 0) return;
    float* ks = sm;                                  // [C][LD]
    float* qs = ks + C * LD;                         // [C][LD]
    float* Ps = qs + C * LD;                         // [C][C + 1]
    float* As = Ps + C * (C + 1);                    // [C][C + 1] (delta)
    float* gs = As + (DELTA ? C * (C + 1) : 0);      // [C], per channel [C][LD]
    float* bs = gs + (CH ? C * LD : C);              // [C] beta
    const int Cq = 2 * a.G * dk + a.H * dv, kvh = hh / (a.H / a.G);
    const float* qrow = a.qkv + (size_t)r0 * Cq + (size_t)kvh * dk;
    const float* krow = qrow + (size_t)a.G * dk;
    for (int base = tid; base < C * per; base += 4 * NT) {           // four vectors a thread in flight
        float4 k[4], q[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int idx = base + u * NT, t = idx / per, c = (idx - t * per) * 4;
            k[u] = q[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            g[u] = make_float4(1.f, 1.f, 1.f, 1.f);
            if (t < nt) {
                k[u] = *reinterpret_cast<const float4*>(krow + (size_t)t * Cq + c);
                q[u] = *reinterpret_cast<const float4*>(qrow + (size_t)t * Cq + c);
                if (CH) g[u] = *reinterpret_cast<const float4*>(a.decay + ((size_t)(r0 + t) * a.H + hh) * dk + c);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int idx = base + u * NT, t = idx / per, c = (idx - t * per) * 4;
            if (t >= C) break;
            *reinterpret_cast<float4*>(ks + t * LD + c) = k[u];
            *reinterpret_cast<float4*>(qs + t * LD + c) = q[u];
            if (CH) *reinterpret_cast<float4*>(gs + t * LD + c) = g[u];
        }
    }
    if (tid < C) {
        if (!CH) gs[tid] = tid < nt ? a.decay[(size_t)(r0 + tid) * a.H + hh] : 1.f;
        if (DELTA) bs[tid] = tid < nt ? a.beta[(size_t)(r0 + tid) * a.H + hh] : 0.f;
    }
    float* out = a.ws + ((size_t)blockIdx.x * a.H + hh) * a.total;
    float* dec = out + a.dec_at;
    __syncthreads();
    // sums over dk of rows x (q, and with delta k) times columns k_s: 16 x 16 threads, rows rg + 16 rr, columns cg + 16 cc
    const int rg = tid >> 4, cg = tid & 15;
    if (CH) {
        // Inside a segment of 16 tokens: a lane takes a column s and eight channels (4 l .. and 64 + 4 l ..), and multiplies k_s by one
        // decay after the other on its way to the later rows; 16 lanes' parts of the 16 rows are then summed, a row a lane.
        for (int idx = tid; idx < C * (C + 1); idx += NT) {
            Ps[idx] = 0.f;
            if (DELTA) As[idx] = 0.f;
        }
        __syncthreads();
        {
            const int l = lane & 15;
            const bool in0 = 4 * l < dk, in1 = 64 + 4 * l < dk;
            auto row8 = [&](const float* m, int t, float fill, float (&x)[8]) {
                const float* p = m + t * LD + 4 * l;
                const float4 none = make_float4(fill, fill, fill, fill);
                const float4 u = in0 ? *reinterpret_cast<const float4*>(p) : none, v = in1 ? *reinterpret_cast<const float4*>(p + 64) : none;
                x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
            };
#pragma unroll 1
            for (int s0 = wid * 2; s0 < C; s0 += NT / 16) {
                const int s = s0 + (lane >> 4), tb = s & ~15, from = s0 & 15;
                float w[8], sq[16], sk[16];
                row8(ks, s, 0.f, w);
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    sq[t] = sk[t] = 0.f;
                    if (t < from) continue;
                    float x[8];
                    if (t > from) {                  // (the second half's s is one more: it starts a step later)
                        row8(gs, tb + t, 1.f, x);
                        const bool step = tb + t > s;
#pragma unroll
                        for (int e = 0; e < 8; ++e) w[e] = step ? w[e] * x[e] : w[e];
                    }
                    if (tb + t < s) continue;
                    row8(qs, tb + t, 0.f, x);
#pragma unroll
                    for (int e = 0; e < 8; ++e) sq[t] = fmaf(w[e], x[e], sq[t]);
                    if (DELTA) {
                        row8(ks, tb + t, 0.f, x);
#pragma unroll
                        for (int e = 0; e < 8; ++e) sk[t] = fmaf(w[e], x[e], sk[t]);
                    }
                }
                __syncwarp();
                auto gather = [&](float (&v)[16]) {  // lane l: the sum of row l
#pragma unroll
                    for (int d = 8; d > 0; d >>= 1)
#pragma unroll
                        for (int i = 0; i < d; ++i) {
                            const bool up = l & d;
                            const float send = up ? v[i] : v[i + d], keep = up ? v[i + d] : v[i];
                            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
                        }
                    return v[0];
                };
                const int t = tb + l;
                const float vq = gather(sq);
                if (t >= s) Ps[t * (C + 1) + s] = vq;
                if (DELTA) {
                    const float vk = gather(sk);
                    if (t > s) As[t * (C + 1) + s] = bs[t] * vk;
                }
            }
        }
        __syncthreads();
        // A thread takes a channel of a segment: its decays from the segment's start and to its end, then the copies for delta_tc5.cu.
        // Rows decayed from their segment's start replace q and (in the decays' place) k, k decayed to its segment's end replaces k.
        double* total = reinterpret_cast<double*>(bs + C);           // [4][128] the segments' whole products
        {
            const int i = tid & 127, b = tid >> 7, t0 = b * 16;
            double f[16];
            if (i < dk) {
                double run = 1.;
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    run *= gs[(t0 + t) * LD + i];
                    f[t] = run;
                }
                total[b * 128 + i] = run;
            }
            __syncthreads();
            if (i < dk) {
                double before = 1., after = 1.;
                for (int m = 0; m < b; ++m) before *= total[m * 128 + i];
                for (int m = 3; m > b; --m) after *= total[m * 128 + i];
                if (b == 3) dec[3 * C * dk + i] = before * f[15];
                double run = 1.;
#pragma unroll
                for (int t = 15; t >= 0; --t) {
                    const int at = (t0 + t) * LD + i;
                    const float k = ks[at], q = qs[at], g = gs[at], here = f[t], from = before * f[t];
                    if (DELTA) dec[(t0 + t) * dk + i] = from * k;
                    dec[(C + t0 + t) * dk + i] = from * q;
                    dec[(2 * C + t0 + t) * dk + i] = (float)(after * run) * k;
                    ks[at] = (float)run * k;
                    if (DELTA) gs[at] = here * k;
                    qs[at] = here * q;
                    run *= g;
                }
            }
        }
        __syncthreads();
        // a block of 4 rows x 2 columns a thread, all channels; `rows` of q and, with delta, of k
        auto block = [&](int t0, int s0, const float* rows, float* to, bool scale) {
            float sum[4][2] = {};
            for (int x0 = 0; x0 < dk; x0 += 16) {    // sums of 16, and of these: a chain over all channels has twice the error
                float acc[4][2] = {};
#pragma unroll
                for (int x = x0; x < x0 + 16; x += 4) {
                    if (x >= dk) break;
                    const float4 k0 = *reinterpret_cast<const float4*>(ks + s0 * LD + x), k1 = *reinterpret_cast<const float4*>(ks + (s0 + 1) * LD + x);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float4 v = *reinterpret_cast<const float4*>(rows + (t0 + r) * LD + x);
                        acc[r][0] = fmaf(v.x, k0.x, acc[r][0]); acc[r][0] = fmaf(v.y, k0.y, acc[r][0]);
                        acc[r][0] = fmaf(v.z, k0.z, acc[r][0]); acc[r][0] = fmaf(v.w, k0.w, acc[r][0]);
                        acc[r][1] = fmaf(v.x, k1.x, acc[r][1]); acc[r][1] = fmaf(v.y, k1.y, acc[r][1]);
                        acc[r][1] = fmaf(v.z, k1.z, acc[r][1]); acc[r][1] = fmaf(v.w, k1.w, acc[r][1]);
                    }
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    sum[r][0] += acc[r][0];
                    sum[r][1] += acc[r][1];
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) to[(t0 + r) * (C + 1) + s0 + c] = scale ? bs[t0 + r] * sum[r][c] : sum[r][c];
        };
        // neighbouring segments of a half: 16 x 16 results, 32 threads; [half][q, k]
        if (wid < (DELTA ? 4 : 2)) {
            const int h = wid & 1, t0 = 32 * h + 16 + (lane & 3) * 4, s0 = 32 * h + (lane >> 2) * 2;
            if (wid < 2) block(t0, s0, qs, Ps, false);
            else block(t0, s0, gs, As, true);
        }
        __syncthreads();
        // across the halves: on to the boundary, and from it
        if (tid < 128 && tid < dk) {
            const float to = (float)total[128 + tid], from = (float)total[2 * 128 + tid];
#pragma unroll 4
            for (int t = 0; t < 16; ++t) {
                ks[t * LD + tid] *= to;
                qs[(48 + t) * LD + tid] *= from;
                if (DELTA) gs[(48 + t) * LD + tid] *= from;
            }
        }
        __syncthreads();
        if (wid < (DELTA ? 8 : 4)) {                 // 32 x 32 results, 128 threads
            const int u = tid & 127, t0 = 32 + (u & 7) * 4, s0 = (u >> 3) * 2;
            if (wid < 4) block(t0, s0, qs, Ps, false);
            else block(t0, s0, gs, As, true);
        }
    } else {
        // the decay ratios of all (t, s), and the products from the chunk's start and to its end: by segments of 16 tokens, a chain of
        // 16 + 16 products instead of 64, in 64 bits
        const int col = tid & (C - 1), sg = tid >> 6, own = col >> 4;
        if (tid < C) {
            double run = 1.;
            for (int r = tid + 1; r < (tid | 15) + 1; ++r) run *= gs[r];
            s_tail[tid] = run;
            if ((tid & 15) == 0) s_seg[tid >> 4] = run * gs[tid];
        }
        __syncthreads();
        {
            double run = s_tail[col];
            for (int m = own + 1; m < sg; ++m) run *= s_seg[m];
            if (sg == own) run = 1.;
#pragma unroll 4
            for (int t = sg * 16; t < sg * 16 + 16; ++t) {
                if (t > col) run *= gs[t];
                Ps[t * (C + 1) + col] = t >= col ? (float)run : 0.f;
            }
        }
        if (tid < C) {
            double to = s_tail[tid], from = 1.;
            for (int m = own + 1; m < 4; ++m) to *= s_seg[m];
            for (int m = 0; m < own; ++m) from *= s_seg[m];
            for (int r = own * 16; r <= tid; ++r) from *= gs[r];
            dec[tid] = (float)from;
            dec[C + tid] = (float)to;
        }
        __syncthreads();
        // sums over the even and odd ones of 16 entries, and of these; blocks above the diagonal are left out
        float sum[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) sum[r][0] = sum[r][1] = sum[r][2] = sum[r][3] = 0.f;
#pragma unroll 1
        for (int i0 = 0; i0 < dk; i0 += 16) {
            pair_t acc[8][4];
#pragma unroll
            for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0;
#pragma unroll
            for (int i = i0; i < i0 + 16; i += 4) {
                if (i >= dk) break;
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
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int c = 0; c <= (r & 3); ++c) {
                    const float2 h = halves(acc[r][c]);
                    sum[r][c] += h.x + h.y;
                }
        }
#pragma unroll
        for (int r = 7; r >= 0; --r) {          // the k rows still need the ratios that the q rows overwrite (same thread)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int t = rg + 16 * (r & 3), x = cg + 16 * c;
                const float v = t >= x ? sum[r][c] * Ps[t * (C + 1) + x] : 0.f;
                if (r < 4) Ps[t * (C + 1) + x] = v;
                else As[t * (C + 1) + x] = t > x ? bs[t] * v : 0.f;
            }
        }
    }
    __syncthreads();
    for (int idx = tid * 4; idx < C * C; idx += NT * 4) {
        const float* p = Ps + (idx / C) * (C + 1) + idx % C;
        *reinterpret_cast<float4*>(out + idx) = make_float4(p[0], p[1], p[2], p[3]);
    }
    if (DELTA) {
        // the inverse of I + A by halves: forward substitution on the diagonal blocks (a warp each, a lane per column), then
        // T21 = -T22 A21 T11; Ps is free and takes T
        if (wid == 6 || wid == 7) {
            const int o = wid == 6 ? 0 : 32;
            float T[32];
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                float v = t == lane ? 1.f : 0.f, v1 = 0.f;           // two chains
#pragma unroll
                for (int s = 0; s < t; ++s) (s & 1 ? v1 : v) = fmaf(-As[(o + t) * (C + 1) + o + s], T[s], s & 1 ? v1 : v);
                T[t] = v + v1;
            }
            __syncwarp();
            asm volatile("bar.sync 1, 64;" ::: "memory");            // both warps are done reading A's diagonal blocks ...
#pragma unroll
            for (int t = 0; t < 32; ++t) As[(o + t) * (C + 1) + o + lane] = T[t];        // ... whose place T takes
        }
        __syncthreads();
        float* x = Ps;                               // A21 T11, [32][C + 1]
        const int row = tid >> 3, c4 = (tid & 7) * 4;                // 256 threads
        if (tid < 256) {
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
        if (tid < 256) {
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
        float* to = out + a.t_at;
        for (int idx = tid * 4; idx < C * C; idx += NT * 4) {
            const int t = idx / C, s = idx % C;
            const float* p = As + t * (C + 1) + s;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = s + e <= t ? p[e] * bs[s + e] : 0.f;
            *reinterpret_cast<float4*>(to + idx) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

template <typename K>
int allow(K kern, size_t bytes) {
    if (bytes > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return B2_OK;
}

template <bool CH, bool DELTA>
int launch_prep(const ChunkArgs& a, cudaStream_t st) {
    const size_t LD = a.dk + 4, rows = C * LD;
    const size_t psm = sizeof(float) * (2 * rows + (DELTA ? 2 : 1) * C * (C + 1) + (CH ? rows + 2 * 4 * 128 : C) + C);
    int rc = allow(chunk_prep_kernel<CH, DELTA>, psm);
    if (rc != B2_OK) return rc;
    chunk_prep_kernel<CH, DELTA><<<dim3(a.chunks, a.H), CH ? 512 : 256, psm, st>>>(a);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

// Scratch of one chunk of all heads, and the tokens that it takes
int64_t chunk_floats(int H, int dk, int dv, bool ch, bool delta, int* tokens) {
    *tokens = !ch && !delta ? 128 : C;
    if (!ch && !delta) return (int64_t)H * b2_internal_chunk_tc5_layout(dk, dv);
    int t, dec, total;
    b2_internal_delta_tc5_layout(dk, dv, ch, delta, &t, &dec, &total);
    return (int64_t)H * total;
}
// Scratch is at most this many floats (512 MiB), or what one chunk takes: longer batches go through it in pieces, one after another, and the
// state of a sequence that a border cuts is carried.  Cost, all at once -> in pieces: 32 heads of 128 x 128, 8192 tokens with delta
// 1296 us (1356 MiB) -> 1419, gated channels 1106 (1292 MiB) -> 1238; 16 heads, 32768 tokens 3246 (2697 MiB) -> 3478.
constexpr int64_t kMostScratch = 1 << 27;

}  // namespace

// Scratch (floats) of the chunked form: grows with rows and sequences up to the limit; 0 for sizes it is not built for
int64_t b2_internal_chunk_scan_floats(int total_rows, int n_seq, int H, int dk, int dv, bool ch, bool delta) {
    if (dk % 4 || dv % 4 || dk > 128 || n_seq <= 0 || total_rows <= 0) return 0;
    int tokens;
    const int64_t one = chunk_floats(H, dk, dv, ch, delta, &tokens), all = (total_rows / tokens + n_seq) * one, carry = (int64_t)2 * H * dk * dv;
    return all <= kMostScratch ? all : one + carry > kMostScratch ? one + carry : kMostScratch;
}

// Where the chunked form is taken.  Both times are estimated in us from what they measured for heads of 128 x 128 on one B200
// (w = dk dv / 16384 scales the products); the host knows the rows and the number of sequences, so the longest of several is taken to be 1.25 times the mean:
//   tokens   a chain of 0.20 (delta 0.285, per channel 0.235 / 0.31) a token, or, with several sequences, 5.2 (7.1 / 10.6 / 12.4) ns a
//            token and head, down to 5.0 (6.3 / 6.8 / 8.3) from 64 sequences on; without delta keys of other sizes than 32, 64, 128 run
//            as the next one, a third slower
//   chunks   one decay per head without delta (chunk_tc5.cu): 20, 0.2 a chunk of 128 and head for the products (0.14 at 64 x 64) and 0.03 a
//            sequence and head for its state; at least 33 (29 to dk = 64): three launches
//            a decay per channel without delta: 20, 0.27 a chunk of 64 and head for the products, 0.11 a sequence and head for its
//            state; at least 39 (33 to dk = 64): four launches
//            delta: 0.16 (per channel 0.70) a chunk and head for the products, 0.11 a sequence and head for its state, 4.8 a step of the chain
//            and SM's share of CTAs; at least 40 (110).  That is more than the chunks take (table), and the line lies there for their
//            error: nearer, 700 to 3100 rows in several sequences would take 10 to 37 % less time, but their outputs would be 1.05 times as far from
//            64 bits as token by token (28 pairs of sizes and inputs, 0.88 to 1.13; their states 0.92 times).
// Measured, tokens -> chunks: 1 x 4096 tokens, 16 heads: 804 -> 121, 1160 -> 434, 963 -> 288, 1255 -> 575; 1 x 500: 102 -> 34,
// 146 -> 70, 121 -> 43, 158 -> 88; 1500 + 1000 + 501: 411 -> 92, 573 -> 279, 503 -> 225, 631 -> 400; 16 x 100: 121 -> 74, 181 -> 160, but 160 -> 196 and
// 223 -> 274 with delta, which are left to the tokens, as are 64 x 24: 148 -> 250, 180 -> 415, 193 -> 379, and 1 x 130: 29 -> 33, 41 -> 58, 35 -> 40.
bool b2_internal_chunk_scan_pays(int total_rows, int n_seq, int H, int dk, int dv, bool ch, bool delta) {
    if (total_rows < 2 * n_seq) return false;
    const float len = (float)total_rows / n_seq, w = dk * dv / 16384.f, steps = ceilf(len / C), heads = (float)n_seq * H;
    const int kind = (ch ? 2 : 0) + (delta ? 1 : 0), run_as = delta ? dk : dk <= 32 ? 32 : dk <= 64 ? 64 : 128;
    const float chain_tok[4] = {0.20f, 0.285f, 0.235f, 0.31f}, rate_few[4] = {5.2e-3f, 7.1e-3f, 10.6e-3f, 12.4e-3f}, rate_many[4] = {5.0e-3f, 6.3e-3f, 6.8e-3f, 8.3e-3f};
    const float many = fminf(1.f, fmaxf(0.f, log2f(n_seq / (delta ? 4.f : 2.5f)) / 4.f)), rate = rate_few[kind] + (rate_many[kind] - rate_few[kind]) * many;
    const float longest = len * (n_seq > 1 ? 1.25f : 1.f);
    const float tokens = (run_as == dk ? 1.f : 1.33f) * fmaxf(chain_tok[kind] * (dk <= 64 ? 0.75f : 1.f) * longest, rate * (float)total_rows * H * run_as * dv / 16384.f);
    float chunks, least;
    if (kind == 0) {
        chunks = 20.f + (0.2f * (0.6f + 0.4f * w) * ceilf(len / 128) + 0.03f * w) * heads;
        least = dk <= 64 ? 29.f : 33.f;
    } else if (kind == 2) {
        chunks = 20.f + (0.27f * (0.55f + 0.45f * w) * steps + 0.11f * w) * heads;
        least = dk <= 64 ? 33.f : 39.f;
    } else {
        chunks = ((ch ? 0.70f : 0.16f) * (0.35f + 0.65f * w) * steps + 0.11f * w) * heads +
                 (3.4f + 1.4f * w) * fmaxf(ceilf(longest / C), steps * heads * ((dv + 15) / 16) / b2_sm_count());
        least = ch ? 110.f : 40.f;
    }
    return tokens >= fmaxf(chunks, least);
}

int b2_internal_chunk_scan(const float* qkv, const float* beta, const float* decay, int total_rows, int H, int G, int dk, int dv,
                           bool ch, bool delta, const int32_t* cu_q, const int32_t* ctx_start, const int32_t* state_slot, int n_seq,
                           float* state, float* o, float* ws, void* stream) {
    // upper bound on sum(ceil(len / tokens)): spare CTAs leave at once.  In pieces the scratch starts with the carried states, of which a piece
    // reads one and writes the other.
    int tokens;
    const int64_t one = chunk_floats(H, dk, dv, ch, delta, &tokens), most = b2_internal_chunk_scan_floats(total_rows, n_seq, H, dk, dv, ch, delta);
    const int chunks = total_rows / tokens + n_seq, blocks = (dv + 127) / 128;
    const bool whole = chunks * one <= most;
    const int64_t carry = whole ? 0 : (int64_t)H * dk * dv;
    const int fit = whole ? chunks : (int)((most - 2 * carry) / one), pieces = (chunks + fit - 1) / fit, piece = (chunks + pieces - 1) / pieces;
    for (int first = 0, turn = 0; first < chunks; first += piece, turn ^= 1) {
        const int n = chunks - first < piece ? chunks - first : piece;
        const chunk_tc5::Args a{qkv, decay, H, G, dk, dv, n_seq, blocks, n * H * blocks, first, n, cu_q, ctx_start, state_slot, state, o, ws + 2 * carry,
                                ws + turn * carry, ws + (turn ^ 1) * carry};
        int rc;
        if (!ch && !delta) {
            rc = b2_internal_chunk_tc5(a, stream);
        } else {
            ChunkArgs p{qkv, beta, decay, H, G, dk, dv, n_seq, cu_q, ctx_start, state_slot, a.ws, first, n, 0, 0, 0};
            b2_internal_delta_tc5_layout(dk, dv, ch, delta, &p.t_at, &p.dec_at, &p.total);
            cudaStream_t st = static_cast<cudaStream_t>(stream);
            rc = !ch ? launch_prep<false, true>(p, st) : delta ? launch_prep<true, true>(p, st) : launch_prep<true, false>(p, st);
            if (rc == B2_OK) rc = b2_internal_delta_tc5(a, ch, delta, stream);
        }
        if (rc != B2_OK) return rc;
    }
    return B2_OK;
}
