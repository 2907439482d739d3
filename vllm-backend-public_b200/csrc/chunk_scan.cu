// chunk_scan.cu -- the scan of delta_rule.cu for prompts: S <- g S, u = beta (v - S^T k) (or u = v), S <- S + k u^T, o = S^T q, in
// chunks of C tokens instead of token after token, everything in fp32 on the FMA pipe.
//
// With G_t the product of the chunk's decays up to token t (per head, or per key channel), S_0 the state before the chunk and
// every ratio G_t / G_s taken as the product g_{s+1} .. g_t (numbers in [0, 1] are only ever multiplied, nothing is divided by a
// product that may have underflowed):
//   A[t, s] = beta_t sum_i k_t k_s G_t/G_s  (s < t),    T = (I + A)^-1 diag(beta),     P[t, s] = sum_i q_t k_s G_t/G_s  (s <= t)
//   R = V - (G K) S_0,   U = T R  (no delta: U = V),   O = (G Q) S_0 + P U,   S = G_C S_0 + (G_C/G K)^T U
// which is the same recurrence, summed in another order (the WY form of Yang et al., "Parallelizing linear transformers with the
// delta rule over sequence length", 2024).  Two kernels:
//   chunk_prep_kernel   A, T, P and the decay products: a CTA per (chunk, head), all chunks at once, into the caller's scratch
//   chunk_scan_kernel   the chain over a sequence's chunks: a CTA per (sequence, head, 16 columns of S), the next chunk's operands
//                       in flight by cp.async; three products per chunk of [2C x dk][dk x 16], [C x C][C x 16], [dk x C][C x 16]
// What bounds it: the chain.  A CTA needs C/32 x 0.23 M FMAs a chunk (1.8k cycles of its SM for C = 32), plus a few barriers; the
// token-by-token scan it replaces waited 200 - 400 cycles a token for shuffles and shared memory whatever the shape.  Sixteen columns
// a CTA fill the chip with one sequence of 16 heads of 128; wider slices would halve the reads of K and Q but leave SMs idle.
// C = 64 without delta and with a decay per head (half the barriers), else 32 (T is C x C and the products per channel cost C dk).
#include "b2_act.cuh"

namespace {

constexpr int NC = 16, NT = 256;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(b2::smem_u32(dst)), "l"(src) : "memory");
}

// floats of scratch per (chunk, head): P | T | decay products
__host__ __device__ constexpr int scratch_floats(int C, int dk, bool ch, bool delta) {
    return C * C * (delta ? 2 : 1) + (ch ? 3 * C * dk + dk : 2 * C);
}

struct ChunkArgs {
    const float *qkv, *beta, *decay;
    int H, G, dk, dv, n_seq;
    const int32_t *cu_q, *ctx_start, *state_slot;
    float *state, *o, *ws;
};

// ---------------------------------------------------------------------------------------------------------------- prep
template <int C, bool CH, bool DELTA>
__global__ void __launch_bounds__(NT)
chunk_prep_kernel(const ChunkArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_at[3];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, hh = blockIdx.y;
    const int dk = a.dk, LD = dk + 4;
    if (tid == 0) {
        int want = blockIdx.x;
        s_at[0] = -1;
        for (int s = 0; s < a.n_seq; ++s) {
            if (a.ctx_start[s] < 0) continue;
            const int len = a.cu_q[s + 1] - a.cu_q[s], nc = (len + C - 1) / C;
            if (want < nc) {
                s_at[0] = a.cu_q[s] + want * C;
                s_at[1] = min(C, len - want * C);
                break;
            }
            want -= nc;
        }
    }
    __syncthreads();
    const int r0 = s_at[0], nt = s_at[1];
    if (r0 < 0) return;
    float* ks = sm;                                  // [C][LD]
    float* qs = ks + C * LD;                         // [C][LD]
    float* As = qs + C * LD;                         // [C][C + 1]
    float* Ps = As + C * (C + 1);                    // [C][C + 1]
    float* gs = Ps + C * (C + 1);                    // [C], CH: [C][LD]
    float* bs = gs + (CH ? C * LD : C);              // [C]
    const int Cq = 2 * a.G * dk + a.H * a.dv, kvh = hh / (a.H / a.G);
    const float* qrow = a.qkv + (size_t)r0 * Cq + (size_t)kvh * dk;
    const float* krow = qrow + (size_t)a.G * dk;
    const int per = dk / 4;
    for (int idx = tid; idx < C * per; idx += NT) {
        const int t = idx / per, c = (idx % per) * 4;
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
    float* out = a.ws + ((size_t)blockIdx.x * a.H + hh) * scratch_floats(C, dk, CH, DELTA);
    float* dec = out + C * C * (DELTA ? 2 : 1);
    __syncthreads();
    if (CH) {
        // a warp per column s: k_s times the running product of the decays, dotted with every later row
        for (int s = wid; s < C; s += NT / 32) {
            float w[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) w[m] = lane + 32 * m < dk ? ks[s * LD + lane + 32 * m] : 0.f;
            if (lane < s) Ps[lane * (C + 1) + s] = As[lane * (C + 1) + s] = 0.f;         // C = 32: one lane a row above the diagonal
            for (int t = s; t < C; ++t) {
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
        // decayed copies of the rows: from the chunk's start (k, q) and to its end (k); the whole chunk's product
        const int i = tid & 127;
        if (i < dk) {
            float run = 1.f;
            if (tid < 128) {
                for (int t = 0; t < C; ++t) {
                    run *= gs[t * LD + i];
                    dec[t * dk + i] = run * ks[t * LD + i];
                    dec[(C + t) * dk + i] = run * qs[t * LD + i];
                }
                dec[3 * C * dk + i] = run;
            } else {
                for (int t = C - 1; t >= 0; --t) {
                    dec[(2 * C + t) * dk + i] = run * ks[t * LD + i];
                    run *= gs[t * LD + i];
                }
            }
        }
    } else {
        if (tid < C) {                               // column s of the decay ratios, and the products from the start / to the end
            float run = 1.f;
            for (int t = 0; t < tid; ++t) Ps[t * (C + 1) + tid] = 0.f;
            Ps[tid * (C + 1) + tid] = 1.f;
            for (int t = tid + 1; t < C; ++t) {
                run *= gs[t];
                Ps[t * (C + 1) + tid] = run;
            }
            dec[C + tid] = run;
            float from = 1.f;
            for (int t = 0; t <= tid; ++t) from *= gs[t];
            dec[tid] = from;
        }
        __syncthreads();
        // rows (q, and with delta k) against the columns k_s: 16 x 16 threads, rows rg + 16 rr, columns cg + 16 cc
        constexpr int RR = (DELTA ? 2 : 1) * C / 16, CC = C / 16;
        const int rg = tid >> 4, cg = tid & 15;
        float acc[RR][CC];
#pragma unroll
        for (int r = 0; r < RR; ++r)
#pragma unroll
            for (int c = 0; c < CC; ++c) acc[r][c] = 0.f;
        for (int i = 0; i < dk; i += 4) {
            float4 kc[CC];
#pragma unroll
            for (int c = 0; c < CC; ++c) kc[c] = *reinterpret_cast<const float4*>(ks + (cg + 16 * c) * LD + i);
#pragma unroll
            for (int r = 0; r < RR; ++r) {
                const int row = rg + 16 * r;         // q rows first, then k rows
                const float4 x = *reinterpret_cast<const float4*>((row < C ? qs + row * LD : ks + (row - C) * LD) + i);
#pragma unroll
                for (int c = 0; c < CC; ++c) {
                    acc[r][c] = fmaf(x.x, kc[c].x, acc[r][c]);
                    acc[r][c] = fmaf(x.y, kc[c].y, acc[r][c]);
                    acc[r][c] = fmaf(x.z, kc[c].z, acc[r][c]);
                    acc[r][c] = fmaf(x.w, kc[c].w, acc[r][c]);
                }
            }
        }
#pragma unroll
        for (int r = RR - 1; r >= 0; --r) {          // the k rows still need the ratios that the q rows overwrite
#pragma unroll
            for (int c = 0; c < CC; ++c) {
                const int row = rg + 16 * r, s = cg + 16 * c, t = row < C ? row : row - C;
                const float ratio = Ps[t * (C + 1) + s];
                if (row < C) Ps[t * (C + 1) + s] = acc[r][c] * ratio;                    // 0 above the diagonal
                else As[t * (C + 1) + s] = t > s ? bs[t] * acc[r][c] * ratio : 0.f;
            }
        }
    }
    __syncthreads();
    for (int idx = tid; idx < C * C; idx += NT) out[idx] = Ps[(idx / C) * (C + 1) + idx % C];
    if (DELTA && wid == 7) {                         // forward substitution, a lane per column of T
        float T[C];
        float* to = out + C * C;
#pragma unroll
        for (int t = 0; t < C; ++t) {
            float v = t == lane ? bs[t] : 0.f;
#pragma unroll
            for (int s = 0; s < t; ++s) v = fmaf(-As[t * (C + 1) + s], T[s], v);
            T[t] = v;
            to[t * C + lane] = v;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------- scan
template <int C, bool CH, bool DELTA>
struct ScanSmem {
    static constexpr int RB = DELTA ? 2 : C / 32;    // 32-row blocks of the product with the state
    static constexpr int KS = 8 / RB;                // slices of dk, one a warp
    static constexpr int LP = C + 4;                 // padded rows of P and T
    static constexpr int VLD = NC;
    __host__ __device__ static constexpr int stage(int dk) {
        return (CH ? 3 : 2) * C * (dk + 4) + C * VLD + (DELTA ? 2 : 1) * C * LP + (CH ? dk : 2 * C);
    }
    __host__ __device__ static constexpr int fixed(int dk) { return dk * NC + 2 * 8 * 32 * NC + 3 * C * NC; }
};

template <int C, bool CH, bool DELTA>
__global__ void __launch_bounds__(NT)
chunk_scan_kernel(const ChunkArgs a, int stages) {
    using L = ScanSmem<C, CH, DELTA>;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int seq = blockIdx.x, hh = blockIdx.y, j0 = blockIdx.z * NC;
    const int ctx = a.ctx_start[seq];
    if (ctx < 0) return;
    const int dk = a.dk, dv = a.dv, H = a.H, LD = dk + 4, per = dk / 4;
    const int r0 = a.cu_q[seq], n = a.cu_q[seq + 1] - r0, nchunks = (n + C - 1) / C;
    int base = 0;                                    // this sequence's first chunk
    for (int s = 0; s < seq; ++s)
        if (a.ctx_start[s] >= 0) base += (a.cu_q[s + 1] - a.cu_q[s] + C - 1) / C;
    const int Cq = 2 * a.G * dk + H * dv, kvh = hh / (H / a.G);
    const int slot = a.state_slot[seq];
    const int cols = min(NC, dv - j0);               // a multiple of 4
    float* S = sm;                                   // [dk][NC]
    float* redA = S + dk * NC;                       // [KS][32 RB][NC]: partial products with the state
    float* redB = redA + 8 * 32 * NC;                // partial products with T, then with P
    float* Rm = redB + 8 * 32 * NC;                  // [C][NC] R (delta)
    float* U = Rm + C * NC;                          // [C][NC]
    float* Ud = U + C * NC;                          // [C][NC] U times the decay to the chunk's end (decay per head)
    float* st0 = Ud + C * NC;
    const int stage_floats = L::stage(dk);

    auto issue = [&](int c, int buf) {
        float* ks = st0 + (size_t)buf * stage_floats;
        float* qs = ks + C * LD;
        float* ku = qs + C * LD;                     // CH only
        float* vs = ku + (CH ? C * LD : 0);
        float* ps = vs + C * L::VLD;
        float* ts = ps + C * L::LP;
        float* de = ts + (DELTA ? C * L::LP : 0);
        const int t0 = c * C, nt = min(C, n - t0);
        const float* ws = a.ws + ((size_t)(base + c) * H + hh) * scratch_floats(C, dk, CH, DELTA);
        const float* dec = ws + C * C * (DELTA ? 2 : 1);
        const float* qrow = a.qkv + (size_t)(r0 + t0) * Cq + (size_t)kvh * dk;
        const float* krow = qrow + (size_t)a.G * dk;
        const float* vrow = a.qkv + (size_t)(r0 + t0) * Cq + (size_t)2 * a.G * dk + (size_t)hh * dv + j0;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int idx = tid; idx < C * per; idx += NT) {
            const int t = idx / per, x = (idx - t * per) * 4;
            if (CH) {                                // the decayed copies; rows past the end are zeros there
                if (DELTA) cp_async16(ks + t * LD + x, dec + t * dk + x);
                cp_async16(qs + t * LD + x, dec + (C + t) * dk + x);
                cp_async16(ku + t * LD + x, dec + (2 * C + t) * dk + x);
            } else if (t < nt) {
                cp_async16(ks + t * LD + x, krow + (size_t)t * Cq + x);
                cp_async16(qs + t * LD + x, qrow + (size_t)t * Cq + x);
            } else {
                *reinterpret_cast<float4*>(ks + t * LD + x) = zero;
                *reinterpret_cast<float4*>(qs + t * LD + x) = zero;
            }
        }
        for (int idx = tid; idx < C * (NC / 4); idx += NT) {
            const int t = idx / (NC / 4), x = (idx % (NC / 4)) * 4;
            if (t < nt && x < cols) cp_async16(vs + t * L::VLD + x, vrow + (size_t)t * Cq + x);
            else *reinterpret_cast<float4*>(vs + t * L::VLD + x) = zero;
        }
        for (int idx = tid; idx < (DELTA ? 2 : 1) * C * (C / 4); idx += NT) {            // P, then T behind it
            const int row = idx / (C / 4), x = (idx % (C / 4)) * 4;
            cp_async16(ps + row * L::LP + x, ws + row * C + x);
        }
        if (CH) { for (int idx = tid; idx < per; idx += NT) cp_async16(de + idx * 4, dec + 3 * C * dk + idx * 4); }
        else { for (int idx = tid; idx < 2 * C / 4; idx += NT) cp_async16(de + idx * 4, dec + idx * 4); }
        asm volatile("cp.async.commit_group;" ::: "memory");
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
    const int rg = lane >> 2, cg = lane & 3;         // products: rows rg + 8 rr of a 32-row block, columns 4 cg .. 4 cg + 3
    if (nchunks > 0) issue(0, 0);
    for (int c = 0; c < nchunks; ++c) {
        const int buf = stages == 2 ? c & 1 : 0;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                             // the chunk's operands and S are there; the last chunk's stage and sums are read
        if (stages == 2 && c + 1 < nchunks) issue(c + 1, buf ^ 1);
        const float* ks = st0 + (size_t)buf * stage_floats;
        const float* qs = ks + C * LD;
        const float* ku = CH ? qs + C * LD : ks;
        const float* vs = qs + C * LD + (CH ? C * LD : 0);
        const float* ps = vs + C * L::VLD;
        const float* ts = ps + C * L::LP;
        const float* de = ts + (DELTA ? C * L::LP : 0);
        const int t0 = c * C, nt = min(C, n - t0);
        {   // rows times the state: block rb (delta: k rows, q rows; else q rows 0 - 31, 32 - 63), slice kq of dk
            const int rb = w / L::KS, kq = w % L::KS;
            const float* rows = (DELTA ? (rb == 0 ? ks : qs) : qs + rb * 32 * LD) + rg * LD;
            const int span = (per + L::KS - 1) / L::KS * 4, k0 = kq * span, k1 = min(k0 + span, dk);
            float acc[4][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll 2
            for (int i = k0; i < k1; i += 4) {
                float4 x[4], y[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(rows + r * 8 * LD + i);
#pragma unroll
                for (int q = 0; q < 4; ++q) y[q] = *reinterpret_cast<const float4*>(S + (i + q) * NC + cg * 4);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float xv[4] = {x[r].x, x[r].y, x[r].z, x[r].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc[r][0] = fmaf(xv[q], y[q].x, acc[r][0]);
                        acc[r][1] = fmaf(xv[q], y[q].y, acc[r][1]);
                        acc[r][2] = fmaf(xv[q], y[q].z, acc[r][2]);
                        acc[r][3] = fmaf(xv[q], y[q].w, acc[r][3]);
                    }
                }
            }
            float* dst = redA + ((size_t)kq * 32 * L::RB + rb * 32 + rg) * NC + cg * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(dst + r * 8 * NC) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
        if (!DELTA && !CH) {                         // U = V: its decayed copy while the products settle
            for (int idx = tid; idx < C * NC / 4; idx += NT) {
                const float f = de[C + idx / (NC / 4)];
                const float4 v = *reinterpret_cast<const float4*>(vs + idx * 4);
                *reinterpret_cast<float4*>(Ud + idx * 4) = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
            }
        }
        __syncthreads();
        // partial products of a [C x C] lower-triangular matrix with a [C x NC] one into redB: C = 32: slice w of 4 columns; C = 64:
        // row half w / 4, columns 16 it + 4 (w % 4)
        auto tri = [&](const float* m, const float* b) {
            float acc[4][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
            const int half = C == 32 ? 0 : w >> 2;
            const int its = C == 32 ? 1 : (half == 0 ? 2 : 4);          // nothing above the diagonal
            for (int it = 0; it < its; ++it) {
                const int s0 = C == 32 ? w * 4 : it * 16 + (w & 3) * 4;
                float4 x[4], y[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(m + (half * 32 + rg + 8 * r) * L::LP + s0);
#pragma unroll
                for (int q = 0; q < 4; ++q) y[q] = *reinterpret_cast<const float4*>(b + (s0 + q) * NC + cg * 4);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float xv[4] = {x[r].x, x[r].y, x[r].z, x[r].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc[r][0] = fmaf(xv[q], y[q].x, acc[r][0]);
                        acc[r][1] = fmaf(xv[q], y[q].y, acc[r][1]);
                        acc[r][2] = fmaf(xv[q], y[q].z, acc[r][2]);
                        acc[r][3] = fmaf(xv[q], y[q].w, acc[r][3]);
                    }
                }
            }
            float* dst = redB + ((size_t)(C == 32 ? w * 32 : (w & 3) * 64 + half * 32) + rg) * NC + cg * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(dst + r * 8 * NC) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        };
        constexpr int NS = C == 32 ? 8 : 4;          // partial products in redB
        if (DELTA) {
            {
                const int t = tid >> 3, x = (tid & 7) * 2;           // C = 32: a pair of columns a thread
                float2 v = make_float2(0.f, 0.f);
#pragma unroll
                for (int kq = 0; kq < L::KS; ++kq) {
                    const float2 p = *reinterpret_cast<const float2*>(redA + (kq * 32 * L::RB + t) * NC + x);
                    v.x += p.x;
                    v.y += p.y;
                }
                const float f = CH ? 1.f : de[t];
                const float2 vv = *reinterpret_cast<const float2*>(vs + t * L::VLD + x);
                *reinterpret_cast<float2*>(Rm + t * NC + x) = make_float2(fmaf(-f, v.x, vv.x), fmaf(-f, v.y, vv.y));
            }
            __syncthreads();
            tri(ts, Rm);
            __syncthreads();
            {
                const int t = tid >> 3, x = (tid & 7) * 2;
                float2 v = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < NS; ++q) {
                    const float2 p = *reinterpret_cast<const float2*>(redB + (q * C + t) * NC + x);
                    v.x += p.x;
                    v.y += p.y;
                }
                *reinterpret_cast<float2*>(U + t * NC + x) = v;
                if (!CH) {
                    const float f = de[C + t];
                    *reinterpret_cast<float2*>(Ud + t * NC + x) = make_float2(v.x * f, v.y * f);
                }
            }
            __syncthreads();
        }
        const float* u = DELTA ? U : vs;
        const float* ud = CH ? u : Ud;
        if (mine) {                                  // S = G_C S + (decayed K)^T U
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float f = CH ? de[i0 + r] : de[C - 1];
                s[r].x *= f;
                s[r].y *= f;
            }
#pragma unroll 8
            for (int t = 0; t < C; ++t) {
                const float4 k = *reinterpret_cast<const float4*>(ku + t * LD + i0);
                const float2 x = *reinterpret_cast<const float2*>(ud + t * NC + jc);
                s[0].x = fmaf(k.x, x.x, s[0].x); s[0].y = fmaf(k.x, x.y, s[0].y);
                s[1].x = fmaf(k.y, x.x, s[1].x); s[1].y = fmaf(k.y, x.y, s[1].y);
                s[2].x = fmaf(k.z, x.x, s[2].x); s[2].y = fmaf(k.z, x.y, s[2].y);
                s[3].x = fmaf(k.w, x.x, s[3].x); s[3].y = fmaf(k.w, x.y, s[3].y);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) *reinterpret_cast<float2*>(S + (i0 + r) * NC + jc) = s[r];
        }
        tri(ps, u);
        __syncthreads();
        for (int idx = tid; idx < nt * (NC / 2); idx += NT) {        // O = G (Q S_0) + P U
            const int t = idx >> 3, x = (idx & 7) * 2;
            float2 v = make_float2(0.f, 0.f);
#pragma unroll
            for (int kq = 0; kq < L::KS; ++kq) {
                const float2 p = *reinterpret_cast<const float2*>(redA + (kq * 32 * L::RB + (DELTA ? 32 : 0) + t) * NC + x);
                v.x += p.x;
                v.y += p.y;
            }
            if (!CH) {
                v.x *= de[t];
                v.y *= de[t];
            }
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                const float2 p = *reinterpret_cast<const float2*>(redB + (q * C + t) * NC + x);
                v.x += p.x;
                v.y += p.y;
            }
            if (x < cols) *reinterpret_cast<float2*>(a.o + ((size_t)(r0 + t0 + t) * H + hh) * dv + j0 + x) = v;
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

template <int C, bool CH, bool DELTA>
int launch(const ChunkArgs& a, int total_rows, cudaStream_t st) {
    const int chunks = total_rows / C + a.n_seq;     // upper bound on sum(ceil(len / C)); spare CTAs leave at once
    const int LD = a.dk + 4;
    const size_t psm = sizeof(float) * (size_t)(2 * C * LD + 2 * C * (C + 1) + (CH ? C * LD : C) + C);
    auto prep = chunk_prep_kernel<C, CH, DELTA>;
    if (psm > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psm));
    prep<<<dim3(chunks, a.H), NT, psm, st>>>(a);
    using L = ScanSmem<C, CH, DELTA>;
    const size_t stage = sizeof(float) * (size_t)L::stage(a.dk), fixed = sizeof(float) * (size_t)L::fixed(a.dk);
    const int stages = fixed + 2 * stage <= 227 * 1024 ? 2 : 1;
    const size_t ssm = fixed + stages * stage;
    auto scan = chunk_scan_kernel<C, CH, DELTA>;
    if (ssm > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm));
    scan<<<dim3(a.n_seq, a.H, (a.dv + NC - 1) / NC), NT, ssm, st>>>(a, stages);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

int chunk_of(bool ch, bool delta) { return ch || delta ? 32 : 64; }

}  // namespace

// Scratch (floats) of the chunked form, 0 where the token-by-token scan is the one to run: head sizes it is not built for, and
// batches of short portions -- below about 24 tokens a sequence a chunk's products cost more than the tokens' chain
// (measured at 64 sequences of 16 heads of 128: 1 token 41 us there, 100+ here).
int64_t b2_internal_chunk_scan_floats(int total_rows, int n_seq, int H, int dk, int dv, bool ch, bool delta) {
    if (dk % 4 || dv % 4 || dk > 128 || n_seq <= 0 || total_rows < 24 * n_seq) return 0;
    const int C = chunk_of(ch, delta);
    return (int64_t)(total_rows / C + n_seq) * H * scratch_floats(C, dk, ch, delta);
}

int b2_internal_chunk_scan(const float* qkv, const float* beta, const float* decay, int total_rows, int H, int G, int dk, int dv,
                           bool ch, bool delta, const int32_t* cu_q, const int32_t* ctx_start, const int32_t* state_slot, int n_seq,
                           float* state, float* o, float* ws, void* stream) {
    const ChunkArgs a{qkv, beta, decay, H, G, dk, dv, n_seq, cu_q, ctx_start, state_slot, state, o, ws};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (ch) return delta ? launch<32, true, true>(a, total_rows, st) : launch<32, true, false>(a, total_rows, st);
    return delta ? launch<32, false, true>(a, total_rows, st) : launch<64, false, false>(a, total_rows, st);
}
