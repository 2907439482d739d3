// chunk_tc5.cu -- the chunked scan of chunk_scan.cu with one decay per head and without the delta correction, S <- g S + k v^T,
// o = S^T q, on the 5th-gen tensor cores: fp32 products as six products of bf16 parts (chunk_tc5.cuh).
//
//   kv_kernel      F = (G_C/G K)^T V of every chunk of 128 tokens
//   state_kernel   S <- G_C S + F over the chunks, element by element; the state before a chunk is written as parts
//   out_kernel     O^T = G (S_0^T Q^T) + V^T P^T with P = Q K^T G_t/G_s
// The first and last take a chunk, a head and 128 columns at a time, one persistent CTA of 16 warps an SM: all of them load, split into parts
// and read the results back; whichever hands over its share of a tile last issues the tile's MMAs.  The features lie on the tensor core's lanes, the tokens on its columns.  Ratios of decays
// are products of the decays between (nothing is divided), scanned within each warp.
// Nothing runs backwards in time: P above its diagonal is selected to zero, and if a result is not finite, the values without parts are
// taken out of V, the product is repeated (so earlier tokens get the very numbers that they get without them) and
// their columns become NaN from their tokens on.  When a CTA is through with its items, it sums what is not finite again in plain fp32: infinities
// stay infinities.
//
// 4096 tokens, 16 heads of 128 x 128 in a graph: 124 us (with the products on the FMA pipe 243, token by token 804); 500 tokens 35 (41, 102).  Under
// ncu, cold: kv 35, state 20, out 75.
// out_kernel's item takes 30e3 cycles, of which the MMAs are 9e3: splitting into parts, the copies of S_0 (20 bytes a cycle and SM when all
// ask at once) and the read-back follow one another in the one CTA that an SM's shared memory holds.  Two CTAs of 64 tokens an SM took 89 us
// instead of the 72 that this one took then (twice the instructions), a warp of its own for the MMAs 78 - 90 (the registers it costs the others spill).
#include "chunk_tc5.cuh"

namespace {
using namespace chunk_tc5;

constexpr int CS = 128, NT = 512, SMEM = 12 * PART + 1024;

// Scratch of a (chunk, head), in floats: G_C | F | S_0 as out_kernel's operand: the parts of 64 rows x 128 columns after one another, per
// block of the columns and slice of the rows.  All three start on 128 bytes.
constexpr int F_AT = 32;
__host__ __device__ constexpr int image(int dk, int dv) { return F_AT + (dk * dv + 31) / 32 * 32; }
__host__ __device__ constexpr int scratch(int dk, int dv) { return image(dk, dv) + (dk + 63) / 64 * ((dv + 127) / 128) * (3 * PART / 4); }

// Results that are not finite, summed again from the inputs (and the state's parts) in plain fp32, as far as they are no NaN.  It is for broken inputs: 4096
// tokens of 16 heads take 2 ms with one infinite value, 3 with states of NaN, 5 with values of NaN.
__device__ __noinline__ void again_sums(const Args& a, const Again& again) {
    const int tid = threadIdx.x, dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv, group = a.H / a.G;
    for (int m = again.first; m <= again.last; ++m) {
        const At t = locate<CS>(a, blockIdx.x + m * gridDim.x);
        const float* base = a.qkv + (size_t)t.row * Cq, *k = base + (a.G + t.head / group) * dk, *v = base + 2 * a.G * dk + t.head * dv;
        const float* g = a.decay + (size_t)t.row * a.H + t.head;
        float* f = a.ws + ((size_t)t.chunk * a.H + t.head) * scratch(dk, dv) + F_AT;
        for (int e = tid; e < 128 * dk; e += NT) {
            const int i = e >> 7, j = t.block * 128 + (e & 127);
            if (j >= dv || finite(f[(size_t)i * dv + j])) continue;
            double to = 1.;
            float sum = 0.f;
            for (int s = t.nt - 1; s >= 0 && sum == sum; --s) {
                sum = fmaf(k[(size_t)s * Cq + i], (float)to * v[(size_t)s * Cq + j], sum);
                to *= g[(size_t)s * a.H];
            }
            f[(size_t)i * dv + j] = sum;
        }
    }
}
// P: shared memory for P, row after row, and the decays from the chunk's start
__device__ __noinline__ void again_outputs(const Args& a, const Again& again, float* P) {
    const int tid = threadIdx.x, dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv, group = a.H / a.G;
    float* const from = P + CS * CS;
    for (int m = again.first; m <= again.last; ++m) {
        const At t = locate<CS>(a, blockIdx.x + m * gridDim.x);
        const float* base = a.qkv + (size_t)t.row * Cq, *q = base + (t.head / group) * dk, *k = q + a.G * dk, *v = base + 2 * a.G * dk + t.head * dv;
        const float* g = a.decay + (size_t)t.row * a.H + t.head;
        __syncthreads();
        for (int e = tid; e < CS * CS; e += NT) {
            const int r = e / CS, s = e % CS;
            if (s > r || r >= t.nt) continue;
            double run = 1.;
            for (int u = s + 1; u <= r; ++u) run *= g[(size_t)u * a.H];
            float p = 0.f;
            for (int i = 0; i < dk; ++i) p = fmaf(q[(size_t)r * Cq + i], k[(size_t)s * Cq + i], p);
            P[e] = p * (float)run;
            if (s == 0) from[r] = run * g[0];
        }
        __syncthreads();
        const unsigned char* s0 = reinterpret_cast<const unsigned char*>(a.ws + ((size_t)t.chunk * a.H + t.head) * scratch(dk, dv) + image(dk, dv)) +
                                  t.block * (dk > 64 ? 2 : 1) * (3 * PART);
        for (int e = tid; e < 128 * t.nt; e += NT) {
            const int r = e >> 7, c = e & 127, j = t.block * 128 + c;
            float* o = a.o + ((size_t)(t.row + r) * a.H + t.head) * dv + j;
            if (j >= dv || finite(*o)) continue;
            float sum = 0.f;
            for (int i = 0; i < dk && !t.fresh && sum == sum; ++i)
                sum = fmaf(from[r] * q[(size_t)r * Cq + i], joined(s0 + (i >> 6) * (3 * PART) + tile_at(i & 63, c >> 3, 64) + (c & 7) * 2, PART), sum);
            for (int s = 0; s <= r && sum == sum; ++s) sum = fmaf(P[r * CS + s], v[(size_t)s * Cq + j], sum);
            *o = sum;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------- F
// Two slices of 64 tokens, each with its own tiles of V and K and its own accumulator; while one is multiplied, the next is split,
// the one after it is on its way, and the accumulators of two items alternate.
__global__ void __launch_bounds__(NT, 1)
kv_kernel(const __grid_constant__ Args a) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t s_done[2];
    __shared__ unsigned s_full[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    __shared__ Again s_again;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    At at = locate<CS>(a, blockIdx.x);
    if (at.nt == 0) return;
    const uint32_t sm = (b2::smem_u32(sm_raw) + 1023u) & ~1023u;
    unsigned char* const gen = sm_raw + (sm - b2::smem_u32(sm_raw));
    auto done = [&](int u) { return b2::smem_u32(&s_done[u]); };
    if (tid == 0) {
        s_failed = 0;
        s_again.none();
        for (int u = 0; u < 2; ++u) {
            s_full[u] = 0;
            b2::mbar_init(done(u), 1);
        }
        b2::fence_mbar_init();
    }
    const uint32_t tmem = tmem_alloc(&s_tmem, warp);
    const int dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv, group = a.H / a.G;
    int n = 0;                                       // items of this CTA so far
    Fetch<128> v, k;
    auto load = [&](const At& t, int u) {
        const float* base = a.qkv + (size_t)(t.row + 64 * u) * Cq;
        v.load(base + 2 * a.G * dk + t.head * dv + t.block * 128, Cq, t.nt - 64 * u, dv - t.block * 128);
        k.load(base + (a.G + t.head / group) * dk, Cq, t.nt - 64 * u, dk);
    };
    float g[4];
    auto load_g = [&](const At& t) {                 // four tokens a lane
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] = 4 * lane + i < t.nt ? a.decay[(size_t)(t.row + 4 * lane + i) * a.H + t.head] : 1.f;
    };
    load(at, 0);
    load_g(at);
    At before{};
    auto finish = [&]() {                            // the results of the item before: lane a column of F, registers its rows
        wait(done(1), (n - 1) & 1, &s_failed);
        tc_fence_after();
        const int q = warp & 3, i0 = (warp >> 2) * 32, j = before.block * 128 + q * 32 + lane;
        if (i0 >= dk) return;
        const uint32_t src = tmem + ((uint32_t)(q * 32) << 16) + 256 * ((n - 1) & 1) + i0;
        float* f = a.ws + ((size_t)before.chunk * a.H + before.head) * scratch(dk, dv) + F_AT + (size_t)i0 * dv + j;
        const bool bad = *(volatile int*)&s_failed != 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float x[16];
            read_parts(src + 16 * h, x);             // the two slices' sums
            if (j < dv) {
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < 16; ++i, f += dv)
                    if (i0 + 16 * h + i < dk) {
                        *f = bad ? __int_as_float(0x7fc00000) : x[i];
                        sum += fabsf(x[i]);
                    }
                if (!finite(sum)) s_again.add(n - 1);
            }
        }
    };
#pragma unroll 1
    for (int item = blockIdx.x; at.nt > 0; ++n) {
        At next;
        // from s + 1 to the chunk's end: four tokens a lane, then the lanes behind
        const double g23 = (double)g[2] * g[3], all = product_from((double)g[0] * g[1] * g23);
        double to3 = __shfl_down_sync(0xffffffffu, all, 1);
        if (lane == 31) to3 = 1.;
        const double to2 = g[3] * to3;
        const float even = warp & 1 ? to2 : g[1] * g23 * to3, odd = warp & 1 ? to3 : g23 * to3;
        if (tid == 0 && at.block == 0) a.ws[((size_t)at.chunk * a.H + at.head) * scratch(dk, dv)] = all;
#pragma unroll 1
        for (int u = 0; u < 2; ++u) {
            if (n > 0) wait(done(u), (n - 1) & 1, &s_failed);
#pragma unroll
            for (int i = 0; i < 2; ++i) {            // a warp's rows are 64 u + 32 i + 2 warp and the one after it
                const int src = (64 * u + 32 * i + 2 * warp) >> 2;
                const float x = __shfl_sync(0xffffffffu, even, src), y = __shfl_sync(0xffffffffu, odd, src), to = lane < 16 ? x : y;
#pragma unroll
                for (int e = 0; e < 8; ++e) v.x[i][e] *= to;
            }
            v.store(gen + u * 6 * PART, PART);
            k.store(gen + (u * 6 + 3) * PART, PART);
            if (hand_over(&s_full[u]) && elect_one()) {
                const uint32_t id = idesc_bf16(128, (dk + 15) & ~15, 1) | kAmn;
                const uint32_t vl = desc_lo(sm + u * 6 * PART, PART / 2), kl = desc_lo(sm + (u * 6 + 3) * PART, PART / 2);
                constexpr int A[6] = {2, 0, 1, 1, 0, 0}, B[6] = {0, 2, 1, 0, 1, 0};      // the smallest products first
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        mma_ss(tmem + 256 * (n & 1) + 128 * u, desc_join(vl + ((A[p] * PART + kk * 2048) >> 4)),
                               desc_join(kl + ((B[p] * PART + kk * 2048) >> 4)), id, p > 0 || kk > 0);
                mma_commit(done(u));
            }
            __syncwarp();
            if (u == 0) {
                load(at, 1);
                next = locate<CS>(a, item += gridDim.x);
                if (n > 0) finish();
            } else if (next.nt > 0) {
                load(next, 0);
                load_g(next);
            }
        }
        before = at;
        at = next;
    }
    // (within the loop the next item's first slice waits for it; commits of different threads promise no order among one another)
    wait(done(0), (n - 1) & 1, &s_failed);
    finish();
    if (*(volatile int*)&s_failed)
        for (int u = 0; u < 2; ++u) drain(done(u), (n - 1) & 1);
    tmem_free(tmem, warp);
    if (!*(volatile int*)&s_failed) again_sums(a, s_again);
}

// ---------------------------------------------------------------------------------------------------------------- state
template <int AHEAD>
__global__ void __launch_bounds__(128)
state_kernel(const Args a) {
    const int seq = blockIdx.x, hh = blockIdx.y;
    // four columns of a row; rows up to the next multiple of 16 are zeros
    const int dk = a.dk, dv = a.dv, e = (blockIdx.z * blockDim.x + threadIdx.x) * 4, row = e / dv, col = e - row * dv;
    const Portion part = portion<CS>(a, seq);
    const int nchunks = part.count;
    if (row >= ((dk + 15) & ~15) || nchunks == 0) return;
    const size_t step = (size_t)a.H * scratch(dk, dv);
    float* ws = a.ws + ((size_t)part.begin * a.H + hh) * scratch(dk, dv);
    const float *g = ws, *f = ws + F_AT + e;            // the chunk's whole product; F
    unsigned char* to = reinterpret_cast<unsigned char*>(ws + image(dk, dv)) + ((col >> 7) * ((dk + 63) / 64) + (row >> 6)) * (3 * PART) +
                        tile_at(row & 63, (col & 127) >> 3, 64) + (col & 4) * 2;
    const bool pad = row >= dk;
    const float* from = pad ? nullptr : state_from(a, part, a.state_slot[seq], hh, a.ctx_start[seq]);
    float4 s = from ? *reinterpret_cast<const float4*>(from + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 x[AHEAD];                                 // they do not depend on the chain
    float d[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
        if (u < nchunks && !pad) {
            x[u] = *reinterpret_cast<const float4*>(f + u * step);
            d[u] = g[u * step];
        }
    for (int c0 = 0; c0 < nchunks; c0 += AHEAD) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int c = c0 + u;
            if (c < nchunks) {
                store_any4(to + (size_t)c * step * 4, PART, s);
                if (pad) continue;
                s = make_float4(fmaf(s.x, d[u], x[u].x), fmaf(s.y, d[u], x[u].y), fmaf(s.z, d[u], x[u].z), fmaf(s.w, d[u], x[u].w));
                if (c + AHEAD < nchunks) {
                    x[u] = *reinterpret_cast<const float4*>(f + (c + AHEAD) * step);
                    d[u] = g[(c + AHEAD) * step];
                }
            }
        }
    }
    float* dst = pad ? nullptr : state_to(a, part, a.state_slot[seq], hh);
    if (dst) *reinterpret_cast<float4*>(dst + e) = s;
}

// ---------------------------------------------------------------------------------------------------------------- output
// Shared memory: two tiles X for S_0, then K, then V, a slice of 64 features or tokens each, and Q, whose place P takes.  TMEM: S_0^T Q^T,
// and K Q^T, whose place V^T P^T takes.
__global__ void __launch_bounds__(NT, 1)
out_kernel(const __grid_constant__ Args a) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t s_done[2], s_copied;
    __shared__ unsigned s_full[4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed, s_repeat;               // s_repeat: number of the last item (from 1) with a result that was not finite
    __shared__ Again s_again;
    __shared__ int s_bad_from[128];                  // first token whose value in this column has no parts
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    At at = locate<CS>(a, blockIdx.x);
    if (at.nt == 0) return;
    const uint32_t sm = (b2::smem_u32(sm_raw) + 1023u) & ~1023u, q_sm = sm + 6 * PART;
    unsigned char* const gen = sm_raw + (sm - b2::smem_u32(sm_raw)), * const qb = gen + 6 * PART;
    auto done = [&](int u) { return b2::smem_u32(&s_done[u]); };
    const uint32_t copied = b2::smem_u32(&s_copied);
    if (tid == 0) {
        s_failed = s_repeat = 0;
        s_again.none();
        for (int u = 0; u < 4; ++u) s_full[u] = 0;
        for (int u = 0; u < 2; ++u) b2::mbar_init(done(u), 1);
        b2::mbar_init(copied, 1);
        b2::fence_mbar_init();
    }
    const uint32_t tmem = tmem_alloc(&s_tmem, warp);
    const int dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv, group = a.H / a.G;
    const int slices = dk > 64 ? 2 : 1, k_last = (dk - (slices - 1) * 64 + 15) / 16;     // of the features; 16-steps of the last
    const int qd = warp & 3, cg = warp >> 2;         // this thread's lanes and its 32 columns
    const uint32_t mine = tmem + ((uint32_t)(qd * 32) << 16) + cg * 32;
    unsigned copies = 0, turns0 = 0, turns1 = 0;     // phases so far of `copied` and done[u]
    auto settled = [&](int u) {                      // the tile's product is complete
        wait(done(u), (u ? turns1++ : turns0++) & 1, &s_failed);
        tc_fence_after();
    };
    Fetch<64> q0, q1;
    float dec[4];                                    // decays: a token of each group of 32 a lane
    auto load_q = [&](const At& t) {
        const float* q = a.qkv + (size_t)t.row * Cq + (t.head / group) * dk;
        q0.load(q, Cq, t.nt, dk);
        if (slices == 2) q1.load(q + 64, Cq, t.nt, dk - 64);
#pragma unroll
        for (int m = 0; m < 4; ++m) dec[m] = m * 32 + lane < t.nt ? a.decay[(size_t)(t.row + m * 32 + lane) * a.H + t.head] : 1.f;
    };
    load_q(at);
    auto state_parts = [&](const At& t) {
        return a.ws + ((size_t)t.chunk * a.H + t.head) * scratch(dk, dv) + image(dk, dv) + t.block * slices * (3 * PART / 4);
    };
    int n = 0;
#pragma unroll 1
    for (int item = blockIdx.x; at.nt > 0; ++n) {
        const bool two = at.nt > 64;
        if (!at.fresh && tid == 0 && !*(volatile int*)&s_failed) {
            const float* s0 = state_parts(at);
            b2::mbar_arrive_expect_tx(copied, slices * 3 * PART);
            for (int u = 0; u < slices; ++u) b2::bulk_load(sm + u * 3 * PART, s0 + u * (3 * PART / 4), 3 * PART, copied);
        }
        q0.store(qb, PART);
        if (slices == 2) q1.store(qb + 3 * PART, PART);
        if (hand_over(&s_full[0]) && !at.fresh) {
            wait(copied, copies & 1, &s_failed);
            tc_fence_after();
            if (elect_one())
                for (int u = 0; u < slices; ++u) {
                    mma_parts<128, 2>(tmem, desc_lo(sm + u * 3 * PART, PART / 2), desc_lo(q_sm + u * 3 * PART, 16), kAmn, u + 1 < slices ? 4 : k_last, u > 0);
                    mma_commit(done(u));
                }
            __syncwarp();
        }
        if (!at.fresh) ++copies;
        Fetch<64> k0, k1;
        {
            const float* k = a.qkv + (size_t)at.row * Cq + (a.G + at.head / group) * dk;
            k0.load(k, Cq, at.nt, dk);
            if (slices == 2) k1.load(k + 64, Cq, at.nt, dk - 64);
        }
        // decays: from s + 1 to the end of the key's group and on to the start of the tokens' group; from the chunk's start to a token
        double from_s = 1., upto = 1.;
        float g = dec[0];
#pragma unroll
        for (int m = 0; m < 3; ++m)
            if (m < cg) {
                const double x = product_of_all(dec[m]);
                upto *= x;
                if (m > qd) from_s *= x;
                g = dec[m + 1];
            }
        const double in_group = product_up_to(g);
        const float to_t = upto * in_group;
        {
            const double x = __shfl_down_sync(0xffffffffu, product_from(qd == 0 ? dec[0] : qd == 1 ? dec[1] : qd == 2 ? dec[2] : dec[3]), 1);
            if (lane < 31) from_s *= x;
        }
        auto scores = [&](int u) {
            if (elect_one()) {
                mma_parts<2, 2>(tmem + 256, desc_lo(sm + u * 3 * PART, 16), desc_lo(q_sm + u * 3 * PART, 16), 0, u + 1 < slices ? 4 : k_last, u > 0);
                mma_commit(done(u));
            }
            __syncwarp();
        };
        if (!at.fresh) settled(0);
        k0.store(gen, PART);
        if (hand_over(&s_full[1])) scores(0);
        const float* v = a.qkv + (size_t)at.row * Cq + 2 * a.G * dk + at.head * dv + at.block * 128;
        Fetch<128> v0, v1;
        v0.load(v, Cq, at.nt, dv - at.block * 128);
        if (slices == 2) {
            if (!at.fresh) settled(1);
            k1.store(gen + 3 * PART, PART);
            if (hand_over(&s_full[2])) scores(1);
        }
        if (two) v1.load(v + (size_t)64 * Cq, Cq, at.nt - 64, dv - at.block * 128);
        settled(0);
        v0.store(gen, PART);
        if (slices == 2) settled(1);
        if (two || qd < 2) {                         // lane: key s; registers: its weight in the tokens' results; takes Q's place
            const int s = qd * 32 + lane;
            unsigned char* to = qb + (s >> 6) * 3 * PART;
            float run = qd < cg ? from_s : 1.;       // (diagonal: one chain, of at most 31 products)
#pragma unroll 1
            for (int h = 0; h < 4; ++h) {
                if (h > 0) {                         // below it chains of eight
                    const double x = __shfl_sync(0xffffffffu, in_group, 8 * h - 1);
                    if (qd < cg) run = from_s * x;
                }
                float p[8];
                if (qd <= cg) read_parts(mine + 256 + 8 * h, p);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int t = cg * 32 + 8 * h + i;
                    const float gt = __shfl_sync(0xffffffffu, g, 8 * h + i);
                    if (t > s) run *= gt;
                    p[i] = t >= s && s < at.nt ? p[i] * run : 0.f;
                }
                store_parts(to + tile_at(s & 63, cg * 4 + h, 64), PART, split8(p));
            }
        }
        if (two) v1.store(gen + 3 * PART, PART);
        auto values = [&]() {
            if (elect_one()) {
                for (int u = 0; u < (two ? 2 : 1); ++u)
                    mma_parts<128, 128>(tmem + 256, desc_lo(sm + u * 3 * PART, PART / 2), desc_lo(q_sm + u * 3 * PART, PART / 2), kAmn | kBmn, 4, u > 0);
                mma_commit(done(0));
            }
            __syncwarp();
        };
        if (hand_over(&s_full[3])) values();
        const At next = locate<CS>(a, item += gridDim.x);
        if (next.nt > 0) load_q(next);
        const int j = at.block * 128 + qd * 32 + lane;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            settled(0);
            const bool failed = *(volatile int*)&s_failed != 0;
            const int nan_from = pass ? s_bad_from[qd * 32 + lane] : CS;
            const float nan = __int_as_float(0x7fc00000);
            bool bad = false;
            float* to = a.o + ((size_t)(at.row + cg * 32) * a.H + at.head) * dv + j;
#pragma unroll 1
            for (int h = 0; h < 4; ++h) {
                float x[8];
                read_parts(mine + 256 + 8 * h, x);
                if (!at.fresh) {
                    float y[8];
                    read_parts(mine + 8 * h, y);
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = fmaf(y[i], __shfl_sync(0xffffffffu, to_t, 8 * h + i), x[i]);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i, to += a.H * dv) {
                    const int t = cg * 32 + 8 * h + i;
                    if (t < at.nt && j < dv) {
                        bad |= !finite(x[i]);
                        *to = failed || t >= nan_from ? nan : x[i];
                    }
                }
            }
            if (pass) break;
            if (bad) s_repeat = n + 1;
            tc_fence_before();
            __syncthreads();                         // (and a volatile flag: __syncthreads_or spills 48 bytes here)
            if (*(volatile int*)&s_repeat != n + 1) break;
            // some result is not finite: the values without what has no parts
            if (tid == 0) s_again.add(n);
            if (tid < 128) s_bad_from[tid] = CS;
            __syncthreads();
#pragma unroll 1
            for (int u = 0; u < (two ? 2 : 1); ++u) {
                Fetch<128> x;
                x.load(v + (size_t)64 * u * Cq, Cq, at.nt - 64 * u, dv - at.block * 128);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (!splits(x.x[i][e])) {
                            atomicMin(&s_bad_from[x.col() + e], u * 64 + x.row(i));
                            x.x[i][e] = 0.f;
                        }
                x.store(gen + u * 3 * PART, PART);
            }
            __syncthreads();
            if (hand_over(&s_full[3])) values();
        }
        at = next;
    }
    if (*(volatile int*)&s_failed) {
        if (turns0) drain(done(0), (turns0 - 1) & 1);
        if (turns1) drain(done(1), (turns1 - 1) & 1);
        if (copies) drain(copied, (copies - 1) & 1);
    }
    tmem_free(tmem, warp);
    if (!*(volatile int*)&s_failed) again_outputs(a, s_again, reinterpret_cast<float*>(gen));
}

}  // namespace

int b2_internal_chunk_tc5_layout(int dk, int dv) { return scratch(dk, dv); }

int b2_internal_chunk_tc5(const chunk_tc5::Args& a, void* stream) {
    const int n_seq = a.n_seq, H = a.H, dk = a.dk, dv = a.dv, items = a.items;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    B2_CUDA_OK(cudaFuncSetAttribute(kv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    B2_CUDA_OK(cudaFuncSetAttribute(out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    const int ctas = items < b2_sm_count() ? items : b2_sm_count();
    kv_kernel<<<ctas, NT, SMEM, st>>>(a);
    const dim3 grid(n_seq, H, (((dk + 15) & ~15) * dv / 4 + 127) / 128);
    if (long_chains(a, grid.x * grid.y * grid.z)) state_kernel<16><<<grid, 128, 0, st>>>(a);
    else state_kernel<8><<<grid, 128, 0, st>>>(a);
    out_kernel<<<ctas, NT, SMEM, st>>>(a);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}
