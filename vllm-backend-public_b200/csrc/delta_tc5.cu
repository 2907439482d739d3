// delta_tc5.cu -- the chunked scan of chunk_scan.cu with the delta correction, or with a decay per key channel, on the 5th-gen tensor
// cores: fp32 products as six products of bf16 parts (chunk_tc5.cuh).  chunk_scan.cu prepares P, T and the decays of every chunk of 64
// tokens; what is left is put so that the chain over the chunks is one product a chunk:
//   wy_kernel       W = T (G K), U_0 = T V (no delta: U_0 = V), and from them
//                   M = (G_C/G K)^T W, F = (G_C/G K)^T U_0, Q' = G Q - P W, and P U_0 straight to the outputs
//   chain_kernel    S <- G_C S + F - M S over the chunks (no delta: without M); S before each chunk is kept
//   read_kernel     O = P U_0 + Q' S_0
// M, Q' and S are written as the parts of the products that read them, so these two only copy them to shared memory.
// Nothing runs backwards in time: rows of G K, V, W and U_0 that hold something without parts enter the products that multiply them
// with T's and P's zeros without it, and what they reach -- a row of G K all of the later tokens, a value its column -- becomes NaN.  When a
// CTA is through with its items, it sums what is not finite of F and the outputs again in plain fp32 from P, T and V: infinities stay infinities.
#include "chunk_tc5.cuh"

namespace {
using namespace chunk_tc5;

constexpr int C = 64;
constexpr float kNaN = __builtin_nanf("");

// Scratch of a (chunk, head) in floats.  Images are the operands' parts, slice after slice of 64 features.
struct Layout {
    int p, t, dec, m, f, q, s, total;
    int slices, zs;                                  // slices of 64 key features; of 64 columns of the state
    __host__ __device__ Layout(int dk, int dv, bool ch, bool delta) {
        slices = dk > 64 ? 2 : 1;
        zs = (dv + 63) / 64;
        p = 0;
        t = p + C * C;
        dec = t + (delta ? C * C : 0);               // per head: G | G_C/G; per channel: G K | G Q | G_C/G K | G_C
        m = (dec + (ch ? 3 * C * dk + dk : 2 * C) + 31) / 32 * 32;
        f = m + (delta ? slices * (3 * PART / 4) : 0);               // [part][128 rows][64 features]
        q = f + (dk * dv + 31) / 32 * 32;            // F: delta [column][key feature], else [key feature][column]
        s = q + slices * (3 * 8192 / 4);             // [part][64 features][64 tokens]
        total = s + zs * slices * (3 * 8192 / 4);    // a slice of columns: [part][64 features][64 columns]
    }
};

// eight entries without those that have no parts; `bad` is told their places
template <typename F>
__device__ __forceinline__ void clean(float (&x)[8], F&& bad) {
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s += fabsf(x[e]);
    if (splits(s)) return;
#pragma unroll 1
    for (int e = 0; e < 8; ++e) {
        float v = x[0];
#pragma unroll
        for (int u = 1; u < 8; ++u) v = e == u ? x[u] : v;
        if (splits(v)) continue;
        bad(e);
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = e == u ? 0.f : x[u];
    }
}

// U_0 of a column: 64 tokens in fp32 (no T: V)
__device__ __forceinline__ void plain_u(const float* T, const float* v, int stride, int nt, float (&u)[C]) {
#pragma unroll 1
    for (int t = 0; t < C; ++t) {
        float sum = t < nt ? v[(size_t)t * stride] : 0.f;
        if (T) {
            sum = 0.f;
            for (int s = 0; s <= t && s < nt; ++s) sum = fmaf(T[t * C + s], v[(size_t)s * stride], sum);
        }
        u[t] = sum;
    }
}
// Results of wy_kernel that are not finite, summed again
template <bool CH, bool DELTA>
__device__ __noinline__ void again_wy(const Args& a, const Again& again) {
    const int tid = threadIdx.x, dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv, c = tid & 127, part = tid >> 7;
    const Layout L(dk, dv, CH, DELTA);
    for (int m = again.first; m <= again.last; ++m) {
        const At at = locate<C>(a, blockIdx.x + m * gridDim.x);
        const int j = at.block * 128 + c;
        if (j >= dv) continue;
        float* ws = a.ws + ((size_t)at.chunk * a.H + at.head) * L.total;
        const float* k = CH ? ws + L.dec + 2 * C * dk : a.qkv + (size_t)at.row * Cq + (a.G + at.head / (a.H / a.G)) * dk;
        float u[C];
        plain_u(DELTA ? ws + L.t : nullptr, a.qkv + (size_t)at.row * Cq + 2 * a.G * dk + at.head * dv + j, Cq, at.nt, u);
        for (int t = part; t < at.nt; t += 4) {
            float* o = a.o + ((size_t)(at.row + t) * a.H + at.head) * dv + j;
            if (finite(*o)) continue;
            float sum = 0.f;
            for (int s = 0; s <= t && sum == sum; ++s) sum = fmaf(ws[L.p + t * C + s], u[s], sum);
            *o = sum;
        }
        for (int i = part; i < dk; i += 4) {
            float* f = ws + L.f + (DELTA ? (size_t)j * dk + i : (size_t)i * dv + j);
            if (finite(*f)) continue;
            float sum = 0.f;
            for (int t = 0; t < at.nt && sum == sum; ++t) sum = fmaf(CH ? k[(size_t)t * dk + i] : ws[L.dec + C + t] * k[(size_t)t * Cq + i], u[t], sum);
            *f = sum;
        }
    }
}
// ... of read_kernel without the correction: P V + G Q S_0
__device__ __noinline__ void again_read(const Args& a, const Again& again) {
    const int dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv;
    const Layout L(dk, dv, true, false);
    for (int m = again.first; m <= again.last; ++m) {
        const At at = locate<C>(a, blockIdx.x + m * gridDim.x);
        const float* ws = a.ws + ((size_t)at.chunk * a.H + at.head) * L.total, *v = a.qkv + (size_t)at.row * Cq + 2 * a.G * dk + at.head * dv;
        for (int e = threadIdx.x; e < 128 * at.nt; e += blockDim.x) {
            const int t = e >> 7, j = at.block * 128 + (e & 127);
            float* o = a.o + ((size_t)(at.row + t) * a.H + at.head) * dv + j;
            if (j >= dv || finite(*o)) continue;
            const unsigned char* s0 = reinterpret_cast<const unsigned char*>(ws + L.s) + (j >> 6) * L.slices * (3 * 8192) + (j & 7) * 2;
            float sum = 0.f;
            for (int i = 0; i < dk && sum == sum; ++i)
                sum = fmaf(ws[L.dec + (C + t) * dk + i], joined(s0 + (i >> 6) * (3 * 8192) + tile_at(i & 63, (j & 63) >> 3, 64), 8192), sum);
            for (int s = 0; s <= t && sum == sum; ++s) sum = fmaf(ws[L.p + t * C + s], v[(size_t)s * Cq + j], sum);
            *o = sum;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------- W, U_0 and their products
// Tiles in shared memory: X0 for G K and later G_C/G K, X1 for V and later U_0, Y for W, T and P; in the end 16 KB and X0 for F, X1 and Y
// for M, T and P for Q'.
// Bound by its own phases: with 208 KB of tiles and copies one CTA fits an SM, and an item of 64 tokens goes through ten of them (loads, split,
// product, read back, split ...), 33e3 cycles, 7e3 of which the copies out take (29 bytes a cycle).  784 items (1119 + 779 + 1103 tokens, 16 heads of
// 128 x 128) 111 us (ncu, cold; 1024 items of 4096 tokens 131): 122 with the keys read where they are needed instead of an item ahead, 115 with
// the decays read per token.  U_0 and P U_0 have two leading accumulators, for 3 us: with one their outputs are 1.02 times as far from 64 bits.
// 128 registers spill 28 bytes per head and 8 per channel, once an item.
template <bool CH, bool DELTA>
__global__ void __launch_bounds__(512, 1)
wy_kernel(const __grid_constant__ Args a) {
    extern __shared__ unsigned char sm_raw[];
    enum { OUT_Q, OUT_M, OUT_F };
    __shared__ __align__(8) uint64_t s_done[2], s_out[3];
    __shared__ unsigned s_full[6], s_staged[3];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    __shared__ Again s_again;
    __shared__ int s_row[2], s_col[2][128];          // first token with a bad G K; first bad value of a column
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    At at = locate<C>(a, blockIdx.x);
    if (at.nt == 0) return;
    const uint32_t sm = (b2::smem_u32(sm_raw) + 1023u) & ~1023u, x0 = sm + PART, x1 = x0 + 3 * PART, y = x1 + 3 * PART, tb = y + 3 * PART, pb = tb + 3 * 8192;
    unsigned char* const gen = sm_raw + (sm - b2::smem_u32(sm_raw));
    auto at_sm = [&](uint32_t p) { return gen + (p - sm); };
    auto done = [&](int u) { return b2::smem_u32(&s_done[u]); };
    auto out = [&](int u) { return b2::smem_u32(&s_out[u]); };
    if (tid == 0) {
        s_failed = 0;
        s_again.none();
        for (int u = 0; u < 6; ++u) s_full[u] = 0;
        for (int u = 0; u < 3; ++u) {
            s_staged[u] = 0;
            b2::mbar_init(out(u), 1);
        }
        for (int u = 0; u < 2; ++u) {
            b2::mbar_init(done(u), 1);
            s_row[u] = C;
        }
        b2::fence_mbar_init();
    }
    if (tid < 256) s_col[tid >> 7][tid & 127] = C;
    const uint32_t tmem = tmem_alloc(&s_tmem, warp);
    const int dk = a.dk, dv = a.dv, Cq = 2 * a.G * dk + a.H * dv, group = a.H / a.G;
    const Layout L(dk, dv, CH, DELTA);
    const int qd = warp & 3, cg = warp >> 2, feature = qd * 32 + lane, t0 = cg * 16;         // this thread's lane; its 16 tokens (or 32 features)
    const uint32_t ra = tmem + ((uint32_t)(qd * 32) << 16), rb = ra + 256;
    unsigned turns0 = 0, turns1 = 0, outs_q = 0, outs_f = 0, mine = 0;       // phases of done[] and out[]; copies that this warp issued
    auto settled = [&](int u) {
        wait(done(u), (u ? turns1++ : turns0++) & 1, &s_failed);
        tc_fence_after();
    };
    auto copy_out = [](float* dst, uint32_t src, uint32_t bytes) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
    };
    // a square of 64 in registers: eight neighbours a thread
    auto load64 = [&](const float* m, float (&x)[8]) {
        const float4 u = *reinterpret_cast<const float4*>(m + tid * 8), v = *reinterpret_cast<const float4*>(m + tid * 8 + 4);
        x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    };
    auto store64 = [&](uint32_t dst, const float (&x)[8]) { store_parts(at_sm(dst) + tile_at(tid >> 3, tid & 7, 64), 8192, split8(x)); };
    auto scratch = [&](const At& t) { return a.ws + ((size_t)t.chunk * a.H + t.head) * L.total; };
    // an item ahead: V, P, T, keys (per channel their decayed copies: rows past the end are zeros there) and, per head, the decays of
    // this thread's two rows to the chunk's start and end, and of a lane's token
    Fetch<128> k, v;
    float tm[8], pm[8], from[2], to[2], from_t = 0.f;
    auto load_ahead = [&](const At& t) {
        const float* ws = scratch(t);
        v.load(a.qkv + (size_t)t.row * Cq + 2 * a.G * dk + t.head * dv + t.block * 128, Cq, t.nt, dv - t.block * 128);
        load64(ws + L.p, pm);
        if (DELTA) {
            load64(ws + L.t, tm);
            if (CH) k.load(ws + L.dec, dk, C, dk);
            else k.load(a.qkv + (size_t)t.row * Cq + (a.G + t.head / group) * dk, Cq, t.nt, dk);
        }
        if (!CH) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                from[i] = ws[L.dec + k.row(i)];
                to[i] = ws[L.dec + C + k.row(i)];
            }
            from_t = ws[L.dec + t0 + (lane & 15)];
        }
    };
    load_ahead(at);
    int n = 0;
    bool was_first = false;                          // the item before had M and Q'
#pragma unroll 1
    for (int item = blockIdx.x; at.nt > 0; ++n) {
        float* ws = scratch(at);
        int* const col = s_col[n & 1];
        int* const row = &s_row[n & 1];
        const bool first = at.block == 0;            // M and Q' are the same for every block of columns
        // the item before is copied out of its places: Q' of T's and P's, M of X1 and Y ...
        if (mine) {
            if (lane == 0) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                for (int u = 0; u < 3; ++u)
                    if (mine >> u & 1) b2::mbar_arrive(out(u));
            }
            mine = 0;
            __syncwarp();
        }
        if (was_first) {
            wait(out(OUT_Q), outs_q & 1, &s_failed);
            if (DELTA) wait(out(OUT_M), outs_q & 1, &s_failed);
            ++outs_q;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) clean(v.x[i], [&](int e) { atomicMin(&col[v.col() + e], v.row(i)); });
        v.store(at_sm(x1), PART);
        store64(pb, pm);
        if (DELTA) store64(tb, tm);
        if (hand_over(&s_full[1])) {
            if (elect_one()) {
                mma_orders<2, PART, 128, 2>(tmem + 256, desc_lo(x1, 8192), desc_lo(DELTA ? tb : pb, 16), kAmn, 4, false);
                mma_commit(done(1));
            }
            __syncwarp();
        }
        if (n > 0) wait(out(OUT_F), outs_f++ & 1, &s_failed);        // ... F of X0's; every warp has read its marks
        if (tid < 128) s_col[(n + 1) & 1][tid] = C;
        if (tid == 128) s_row[(n + 1) & 1] = C;
        Fetch<128> kd;
        if (CH) kd.load(ws + L.dec + 2 * C * dk, dk, C, dk);
        else kd.load(a.qkv + (size_t)at.row * Cq + (a.G + at.head / group) * dk, Cq, at.nt, dk);
        if (DELTA) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (!CH)
#pragma unroll
                    for (int e = 0; e < 8; ++e) k.x[i][e] *= from[i];
                clean(k.x[i], [&](int) { atomicMin(row, k.row(i)); });
            }
            k.store(at_sm(x0), PART);
            if (hand_over(&s_full[0]) && elect_one()) {
                mma_orders<1, PART, 128, 2>(tmem, desc_lo(x0, 8192), desc_lo(tb, 16), kAmn, 4, false);
                mma_commit(done(0));
            }
            __syncwarp();
        }
        float q[16];                                 // G Q: lane a key feature, registers tokens
        {
            const float* src = CH ? ws + L.dec + C * dk + (size_t)t0 * dk + feature : a.qkv + (size_t)(at.row + t0) * Cq + (at.head / group) * dk + feature;
            const int rows = !first || feature >= dk ? 0 : CH ? C : at.nt - t0;
#pragma unroll
            for (int i = 0; i < 16; ++i) q[i] = i < rows ? src[(size_t)i * (CH ? dk : Cq)] : 0.f;
        }
        // U_0 takes the place of V, W that of Y: without what is not finite
        float w[16];
        auto store_rows = [&](uint32_t dst, int* mark) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float e8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) e8[e] = w[8 * h + e];
                clean(e8, [&](int e) { atomicMin(mark, t0 + h * 8 + e); });
                store_parts(at_sm(dst) + tile_at(feature, cg * 2 + h, 128), PART, split8(e8));
            }
        };
        if (DELTA) {
            settled(1);
            read_orders<2>(rb + cg * 16, w);
            store_rows(x1, &col[feature]);
            if (hand_over(&s_full[3]) && elect_one()) {
                mma_orders<2, PART, 2, 2>(tmem + 256, desc_lo(x1, 16), desc_lo(pb, 16), 0, 4, false);
                mma_commit(done(1));
            }
            __syncwarp();
            settled(0);
        }
        if (!CH)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 8; ++e) kd.x[i][e] *= to[i];
        kd.store(at_sm(x0), PART);                   // (its products M and F take all tokens: nothing is kept out)
        if (DELTA) {
            read_orders<1>(ra + cg * 16, w);
            store_rows(y, row);
            if (hand_over(&s_full[2]) && elect_one()) {
                mma_orders<1, PART, 2, 2>(tmem, desc_lo(y, 16), desc_lo(pb, 16), 0, 4, false);
                mma_commit(done(0));
            }
            __syncwarp();
        }
        if (!CH)
#pragma unroll
            for (int i = 0; i < 16; ++i) q[i] *= __shfl_sync(0xffffffffu, from_t, i);
        if (DELTA) {                                 // Q'
            settled(0);                              // (after it, W's marks are final)
            read_orders<1>(ra + cg * 16, w);
            if (first) {                             // M
                if (hand_over(&s_full[4]) && elect_one()) {
                    mma_parts64<128, 2>(tmem, desc_lo(x0, 8192), desc_lo(y, 16), kAmn);
                    mma_commit(done(0));
                }
                __syncwarp();
            }
            const int bad = *(volatile int*)row;
#pragma unroll
            for (int i = 0; i < 16; ++i) q[i] = t0 + i >= bad ? kNaN : q[i] - w[i];
        }
        settled(1);                                  // P U_0: lane a column
        read_orders<2>(rb + cg * 16, w);
        if (hand_over(&s_full[5]) && elect_one()) {  // F: lane a key feature (no delta: a column), registers the others
            if (DELTA) mma_parts64<128, 2>(tmem + 256, desc_lo(x0, 8192), desc_lo(x1, 16), kAmn);
            else mma_parts64<128, 128>(tmem + 256, desc_lo(x1, 8192), desc_lo(x0, 8192), kAmn | kBmn);
            mma_commit(done(1));
        }
        __syncwarp();
        const bool failed = *(volatile int*)&s_failed != 0, all_bad = *(volatile int*)row < C;
        {
            const int j = at.block * 128 + feature, bad = min(*(volatile int*)row, *(volatile int*)&col[feature]);
            if (j < dv) {
                float* dst = a.o + ((size_t)(at.row + t0) * a.H + at.head) * dv + j;
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < 16; ++i, dst += a.H * dv)
                    if (t0 + i < at.nt) {
                        *dst = failed || t0 + i >= bad ? kNaN : w[i];
                        sum += fabsf(w[i]);
                    }
                if (!finite(sum) || bad < C) s_again.add(n);
            }
        }
        // the results go through shared memory, which copies them out as they lie there: Q' where T and P were
        if (first) {
            if (feature < L.slices * 64)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float e8[8] = {q[8 * h], q[8 * h + 1], q[8 * h + 2], q[8 * h + 3], q[8 * h + 4], q[8 * h + 5], q[8 * h + 6], q[8 * h + 7]};
                    store_parts(at_sm(tb) + (feature >> 6) * (3 * 8192) + tile_at(feature & 63, cg * 2 + h, 64), 8192, split8(e8));
                }
            if (hand_over(&s_staged[OUT_Q])) {
                if (lane == 0) {
                    copy_out(ws + L.q, tb, L.slices * 3 * 8192);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                mine |= 1 << OUT_Q;
                __syncwarp();
            }
        }
        const At next = locate<C>(a, item += gridDim.x);
        if (next.nt > 0) load_ahead(next);
        if (DELTA && first) settled(0);
        settled(1);
        if (DELTA && first) {
            if ((cg >> 1) < L.slices)
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    float m[8];
                    read_parts(ra + cg * 32 + 8 * h, m);
                    if (all_bad) m[0] = m[1] = m[2] = m[3] = m[4] = m[5] = m[6] = m[7] = kNaN;
                    store_parts(at_sm(x1) + (cg >> 1) * (3 * PART) + tile_at(feature, (cg & 1) * 4 + h, 128), PART, split8(m));
                }
            if (hand_over(&s_staged[OUT_M])) {
                if (lane == 0) {
                    copy_out(ws + L.m, x1, L.slices * 3 * PART);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                mine |= 1 << OUT_M;
                __syncwarp();
            }
        }
        {
            const int cols = min(128, dv - at.block * 128), wide = DELTA ? dk : cols;        // floats a row
            float* f = reinterpret_cast<float*>(at_sm(x0) - PART) + (size_t)(cg * 32) * wide + feature, sum = 0.f;
            const bool bad = failed || all_bad || (!DELTA && *(volatile int*)&col[feature] < C);
            // DELTA: a register is a column, and 32 lanes look at 32 marks
            const unsigned bad_cols = DELTA ? __ballot_sync(0xffffffffu, *(volatile int*)&col[cg * 32 + lane] < C) : 0u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float x[16];
                read_parts(rb + cg * 32 + 16 * h, x);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (feature < wide) {
                        f[(16 * h + i) * wide] = bad || (bad_cols >> (16 * h + i) & 1) ? kNaN : x[i];
                        sum += fabsf(x[i]);
                    }
            }
            if (bad_cols || bad || !finite(sum)) s_again.add(n);
            if (hand_over(&s_staged[OUT_F])) {
                if (lane == 0) {
                    if (DELTA) copy_out(ws + L.f + (size_t)at.block * 128 * dk, x0 - PART, cols * dk * 4);
                    else if (cols == dv) copy_out(ws + L.f, x0 - PART, cols * dk * 4);
                    else
                        for (int i = 0; i < dk; ++i) copy_out(ws + L.f + (size_t)i * dv + at.block * 128, x0 - PART + i * cols * 4, cols * 4);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                mine |= 1 << OUT_F;
                __syncwarp();
            }
        }
        was_first = first;
        at = next;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
    if (*(volatile int*)&s_failed) {
        if (turns0) drain(done(0), (turns0 - 1) & 1);
        if (turns1) drain(done(1), (turns1 - 1) & 1);
    }
    b2::fence_proxy_async();                         // F was copied out
    tmem_free(tmem, warp);
    if (!*(volatile int*)&s_failed) again_wy<CH, DELTA>(a, s_again);
}

// ---------------------------------------------------------------------------------------------------------------- the chain
// A CTA per 64 columns of a head's state.  Eight warps keep it in registers, in fp32 (lane a key feature, 32 columns a thread), and
// write its parts; one warp copies M ahead, three slices of 64 features in a ring; one multiplies and copies the parts out.
// Bound by a step's own phases, one after another: split, store, product, read back; 2.9 us a step (64 chunks of one sequence, 16 heads of
// 128 x 128, 185 us; 18 chunks at most, 1119 + 779 + 1103 tokens, 61 us, where W and U on the FMA pipe within the chain took 196).  Its 96 KB
// of M a step come a ring ahead, at a quarter of what an SM can take in.
template <bool CH>
__global__ void __launch_bounds__(320, 1)
chain_kernel(const Args a) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t s_full, s_done, s_stored, s_here[3], s_free[3];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed, s_seq;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    // CTAs start in the order of their sequences' lengths, the longest first
    for (int i = tid; i < a.n_seq; i += 320) {
        const int len = a.cu_q[i + 1] - a.cu_q[i];
        int rank = 0;
        for (int j = 0; j < a.n_seq; ++j) {
            const int other = a.cu_q[j + 1] - a.cu_q[j];
            rank += other > len || (other == len && j < i);
        }
        if (rank == blockIdx.z) s_seq = i;
    }
    if (tid == 0) {
        s_failed = 0;
        b2::mbar_init(b2::smem_u32(&s_full), 8);
        b2::mbar_init(b2::smem_u32(&s_done), 1);
        b2::mbar_init(b2::smem_u32(&s_stored), 1);
        for (int u = 0; u < 3; ++u) {
            b2::mbar_init(b2::smem_u32(&s_here[u]), 1);
            b2::mbar_init(b2::smem_u32(&s_free[u]), 1);
        }
        b2::fence_mbar_init();
    }
    __syncthreads();
    const int seq = s_seq, hh = blockIdx.y, z = blockIdx.x;
    const Portion part = portion<C>(a, seq);
    const int nchunks = part.count;
    if (nchunks == 0) return;
    const int dk = a.dk, dv = a.dv;
    const Layout L(dk, dv, CH, true);
    const uint32_t sm = (b2::smem_u32(sm_raw) + 1023u) & ~1023u, tile = sm + 9 * PART;
    unsigned char* const gen = sm_raw + (sm - b2::smem_u32(sm_raw));
    const size_t step = (size_t)a.H * L.total;
    float* const ws = a.ws + ((size_t)part.begin * a.H + hh) * L.total;
    const uint32_t full = b2::smem_u32(&s_full), done = b2::smem_u32(&s_done), stored = b2::smem_u32(&s_stored);
    auto here = [&](int b) { return b2::smem_u32(&s_here[b]); };
    auto free_ = [&](int b) { return b2::smem_u32(&s_free[b]); };
    const uint32_t tmem = tmem_alloc(&s_tmem, warp);
    const int total = nchunks * L.slices;
    int sent = 0;                                    // slices of M that this thread has asked for
    if (warp == 8) {
        if (lane == 0) {
#pragma unroll 1
            for (int i = 0; i < total; ++i) {
                const int b = i % 3;
                if (i >= 3 && !wait(free_(b), (i / 3 - 1) & 1, &s_failed)) break;
                sent = i + 1;
                b2::mbar_arrive_expect_tx(here(b), 3 * PART);
                b2::bulk_load(sm + b * 3 * PART, ws + (i / L.slices) * step + L.m + (i % L.slices) * (3 * PART / 4), 3 * PART, here(b));
            }
        }
    } else if (warp == 9) {
        const int k_last = (dk - (L.slices - 1) * 64 + 15) / 16;
#pragma unroll 1
        for (int c = 0; c < nchunks; ++c) {
            wait(full, c & 1, &s_failed);
            tc_fence_after();
            if (lane == 0) {
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                             ::"l"(ws + c * step + L.s + z * L.slices * (3 * 8192 / 4)), "r"(tile), "r"(L.slices * 3 * 8192) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                for (int u = 0; u < L.slices; ++u) {
                    const int i = c * L.slices + u, b = i % 3;
                    wait(here(b), (i / 3) & 1, &s_failed);
                    mma_orders<1, PART, 2, 128>(tmem, desc_lo(sm + b * 3 * PART, 16), desc_lo(tile + u * 3 * 8192, 8192), kBmn, u + 1 < L.slices ? 4 : k_last, u > 0);
                    mma_commit(free_(b));
                }
                mma_commit(done);
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                b2::mbar_arrive(stored);
            }
            __syncwarp();
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        __syncwarp();
    } else {
        const int qd = warp & 3, cg = warp >> 2, i0 = qd * 32 + lane, j0 = z * 64 + cg * 32;
        const uint32_t mine = tmem + ((uint32_t)(qd * 32) << 16) + cg * 32;
        float s[32], f[32];
        auto row32 = [&](const float* p, bool there, float (&x)[32]) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (there && j0 + e < dv) v = *reinterpret_cast<const float4*>(p + e);
                x[e] = v.x; x[e + 1] = v.y; x[e + 2] = v.z; x[e + 3] = v.w;
            }
        };
        const float* from = state_from(a, part, a.state_slot[seq], hh, a.ctx_start[seq]);
        row32(from && i0 < dk ? from + (size_t)i0 * dv + j0 : nullptr, from && i0 < dk, s);
        float gc = 0.f;
        const bool pad = i0 >= L.slices * 64;
#pragma unroll 1
        for (int c = 0; c < nchunks; ++c) {
            if (c > 0) wait(stored, (c - 1) & 1, &s_failed);
            if (!pad)
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float e8[8] = {s[8 * h], s[8 * h + 1], s[8 * h + 2], s[8 * h + 3], s[8 * h + 4], s[8 * h + 5], s[8 * h + 6], s[8 * h + 7]};
                    store_parts(gen + 9 * PART + (i0 >> 6) * (3 * 8192) + tile_at(i0 & 63, cg * 4 + h, 64), 8192, split8(e8));
                }
            b2::fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) b2::mbar_arrive(full);
            const float* w = ws + c * step;
#pragma unroll
            for (int e = 0; e < 32; ++e) f[e] = i0 < dk && j0 + e < dv ? w[L.f + (size_t)(j0 + e) * dk + i0] : 0.f;
            if (i0 < dk) gc = w[L.dec + (CH ? 3 * C * dk + i0 : C - 1)];
#pragma unroll
            for (int e = 0; e < 32; ++e) s[e] = fmaf(gc, s[e], f[e]);
            wait(done, c & 1, &s_failed);
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float d[16];
                read_orders<1>(mine + 16 * h, d);
#pragma unroll
                for (int e = 0; e < 16; ++e) s[16 * h + e] -= d[e];
            }
        }
        float* dst = state_to(a, part, a.state_slot[seq], hh);
        if (dst && i0 < dk) {
            dst += (size_t)i0 * dv + j0;
            const bool bad = *(volatile int*)&s_failed != 0;
#pragma unroll
            for (int e = 0; e < 32; e += 4)
                if (j0 + e < dv)
                    *reinterpret_cast<float4*>(dst + e) = bad ? make_float4(kNaN, kNaN, kNaN, kNaN) : make_float4(s[e], s[e + 1], s[e + 2], s[e + 3]);
        }
    }
    __syncthreads();
    if (*(volatile int*)&s_failed) {                 // what nobody has waited for: every role is done now
        drain(done, (nchunks - 1) & 1);
        for (int back = 1; back <= min(3, sent); ++back) drain(here((sent - back) % 3), ((sent - back) / 3) & 1);
    }
    __syncwarp();
    tmem_free(tmem, warp);
}

// Without the correction: element by element, four columns of a row a thread; rows up to the end of a slice are zeros
template <bool CH, int AHEAD>
__global__ void __launch_bounds__(128)
state_kernel(const Args a) {
    const int seq = blockIdx.x, hh = blockIdx.y, dk = a.dk, dv = a.dv;
    const int e = (blockIdx.z * blockDim.x + threadIdx.x) * 4, row = e / dv, col = e - row * dv;
    const Portion part = portion<C>(a, seq);
    const int nchunks = part.count;
    const Layout L(dk, dv, CH, false);
    if (nchunks == 0 || row >= L.slices * 64) return;
    const size_t step = (size_t)a.H * L.total;
    float* ws = a.ws + ((size_t)part.begin * a.H + hh) * L.total;
    const bool pad = row >= dk;
    const float *g = ws + L.dec + (CH ? 3 * C * dk + row : C - 1), *f = ws + L.f + e;
    unsigned char* to = reinterpret_cast<unsigned char*>(ws + L.s) + ((col >> 6) * L.slices + (row >> 6)) * (3 * 8192) +
                        tile_at(row & 63, (col & 63) >> 3, 64) + (col & 4) * 2;
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
                store_any4(to + (size_t)c * step * 4, 8192, s);
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

// ---------------------------------------------------------------------------------------------------------------- read-out
// O^T += S_0^T Q'^T: both operands are copied as they are, three stages of a slice of 64 features (72 KB); two accumulators alternate.
// Bound by the copies: 3001 tokens, 16 heads of 128 x 128, 29 us for 116 MB of images and twice 25 MB of outputs, part of them in L2 (the FMA pipe
// took 84).  Two leading accumulators for Q' S_0, which is a sum over up to 128 features.
template <bool CH, bool DELTA>
__global__ void __launch_bounds__(320, 1)
read_kernel(const __grid_constant__ Args a) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t s_here[3], s_free[3], s_done[2], s_read[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    __shared__ Again s_again;
    constexpr int STAGE = 9 * 8192;                  // two slices of S_0's columns, and Q'
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    At at = locate<C>(a, blockIdx.x);
    if (at.nt == 0) return;
    const uint32_t sm = (b2::smem_u32(sm_raw) + 1023u) & ~1023u;
    auto bar = [&](uint64_t* b, int i) { return b2::smem_u32(&b[i]); };
    if (tid == 0) {
        s_failed = 0;
        s_again.none();
        for (int u = 0; u < 3; ++u) {
            b2::mbar_init(bar(s_here, u), 1);
            b2::mbar_init(bar(s_free, u), 1);
        }
        for (int u = 0; u < 2; ++u) {
            b2::mbar_init(bar(s_done, u), 1);
            b2::mbar_init(bar(s_read, u), 8);
        }
        b2::fence_mbar_init();
    }
    const uint32_t tmem = tmem_alloc(&s_tmem, warp);
    const int dk = a.dk, dv = a.dv;
    const Layout L(dk, dv, CH, DELTA);
    int n = 0, sent = 0;                             // items with a state so far; slices that this thread has asked for
    if (warp == 8) {
        int i = 0;
#pragma unroll 1
        for (int item = blockIdx.x; at.nt > 0; at = locate<C>(a, item += gridDim.x)) {
            if (at.fresh) continue;
            const float* ws = a.ws + ((size_t)at.chunk * a.H + at.head) * L.total;
            const int zn = min(2, L.zs - 2 * at.block);
            for (int u = 0; u < L.slices; ++u, ++i) {
                const int b = i % 3;
                if (i >= 3) wait(bar(s_free, b), (i / 3 - 1) & 1, &s_failed);
                if (lane == 0 && !*(volatile int*)&s_failed) {
                    sent = i + 1;
                    b2::mbar_arrive_expect_tx(bar(s_here, b), (zn + 1) * 3 * 8192);
                    for (int z = 0; z < zn; ++z)
                        b2::bulk_load(sm + b * STAGE + z * 3 * 8192, ws + L.s + ((2 * at.block + z) * L.slices + u) * (3 * 8192 / 4), 3 * 8192, bar(s_here, b));
                    b2::bulk_load(sm + b * STAGE + 6 * 8192, ws + L.q + u * (3 * 8192 / 4), 3 * 8192, bar(s_here, b));
                }
                __syncwarp();
            }
        }
    } else if (warp == 9) {
        const int k_last = max(2, (dk - (L.slices - 1) * 64 + 15) / 16);           // past dk there are zeros
        int i = 0;
#pragma unroll 1
        for (int item = blockIdx.x; at.nt > 0; at = locate<C>(a, item += gridDim.x)) {
            if (at.fresh) continue;
            if (n >= 2) wait(bar(s_read, n & 1), (n / 2 - 1) & 1, &s_failed);
            tc_fence_after();
            for (int u = 0; u < L.slices; ++u, ++i) {
                const int b = i % 3;
                wait(bar(s_here, b), (i / 3) & 1, &s_failed);
                if (elect_one()) {
                    const uint32_t st = sm + b * STAGE;
                    mma_orders3<8192, 128, 128>(tmem + 256 * (n & 1), desc_lo(st, 3 * 8192), desc_lo(st + 6 * 8192, 8192), kAmn | kBmn, u + 1 < L.slices ? 4 : k_last, u > 0);
                    mma_commit(bar(s_free, b));
                    if (u + 1 == L.slices) mma_commit(bar(s_done, n & 1));
                }
                __syncwarp();
            }
            ++n;
        }
    } else {
        const int qd = warp & 3, cg = warp >> 2;
#pragma unroll 1
        for (int item = blockIdx.x; at.nt > 0;) {
            const At next = locate<C>(a, item += gridDim.x);
            if (!at.fresh) {
                const int j = at.block * 128 + qd * 32 + lane, t0 = cg * 32, rows = j < dv ? at.nt - t0 : 0;
                const size_t stride = (size_t)a.H * dv;
                float* o = a.o + ((size_t)(at.row + t0) * a.H + at.head) * dv + j;
                float x[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) x[i] = i < rows ? o[i * stride] : 0.f;
                wait(bar(s_done, n & 1), (n / 2) & 1, &s_failed);
                tc_fence_after();
                const uint32_t src = tmem + ((uint32_t)(qd * 32) << 16) + 256 * (n & 1) + t0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float d[16];
                    read_orders3(src + 16 * h, d);
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[16 * h + i] += d[i];
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) b2::mbar_arrive(bar(s_read, n & 1));
                const bool bad = *(volatile int*)&s_failed != 0;
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i < rows) {
                        o[i * stride] = bad ? kNaN : x[i];
                        if (!DELTA) sum += fabsf(x[i]);
                    }
                if (!DELTA && !finite(sum)) s_again.add((item - (int)gridDim.x - (int)blockIdx.x) / (int)gridDim.x);
                ++n;
            }
            at = next;
        }
    }
    __syncthreads();
    if (*(volatile int*)&s_failed) {                 // what nobody has waited for: every role is done now
        if (n > 0) drain(bar(s_done, (n - 1) & 1), ((n - 1) / 2) & 1);
        for (int back = 1; back <= min(3, sent); ++back) drain(bar(s_here, (sent - back) % 3), ((sent - back) / 3) & 1);
    }
    __syncwarp();
    tmem_free(tmem, warp);
    if (!DELTA && !*(volatile int*)&s_failed) again_read(a, s_again);
}

template <bool CH, bool DELTA>
int launch(const Args& a, cudaStream_t st) {
    const Layout L(a.dk, a.dv, CH, DELTA);
    constexpr int WY = 10 * PART + 6 * 8192 + 1024, CHAIN = 9 * PART + 6 * 8192 + 1024, READ = 27 * 8192 + 1024;
    B2_CUDA_OK(cudaFuncSetAttribute(wy_kernel<CH, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, WY));
    B2_CUDA_OK(cudaFuncSetAttribute(chain_kernel<CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN));
    B2_CUDA_OK(cudaFuncSetAttribute(read_kernel<CH, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, READ));
    const int ctas = a.items < b2_sm_count() ? a.items : b2_sm_count();
    wy_kernel<CH, DELTA><<<ctas, 512, WY, st>>>(a);
    if constexpr (DELTA) {
        chain_kernel<CH><<<dim3(L.zs, a.H, a.n_seq), 320, CHAIN, st>>>(a);
    } else {
        const dim3 grid(a.n_seq, a.H, (L.slices * 64 * a.dv / 4 + 127) / 128);
        if (long_chains(a, grid.x * grid.y * grid.z)) state_kernel<CH, 16><<<grid, 128, 0, st>>>(a);
        else state_kernel<CH, 8><<<grid, 128, 0, st>>>(a);
    }
    read_kernel<CH, DELTA><<<ctas, 320, READ, st>>>(a);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

}  // namespace

void b2_internal_delta_tc5_layout(int dk, int dv, bool ch, bool delta, int* t, int* dec, int* total) {
    const Layout L(dk, dv, ch, delta);
    *t = L.t;
    *dec = L.dec;
    *total = L.total;
}

int b2_internal_delta_tc5(const chunk_tc5::Args& a, bool ch, bool delta, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (ch) return delta ? launch<true, true>(a, st) : launch<true, false>(a, st);
    return launch<false, true>(a, st);
}
