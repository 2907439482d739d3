// latent_tc5.cu -- decode rows of b2_latent_attention in bf16 on the 5th-gen tensor cores (as many rows as sequences, R a multiple
// of 128): out[t, h] = sum_j softmax_j(qa[t, h] . c_j) c_j[0..R) over the cached rows c_j of R + dr numbers.
//
// A CTA takes one token, up to 32 heads and one share of its keys, 64 keys at a time.  The keys are the M side of the scores and the
// latent's columns the M side of the output, the heads the N side of both: S^T[64 keys, heads] = C Q^T, O^T[R, heads] += C^T P^T, with C
// read from shared memory twice and from memory once.  One ring of two halves holds C as sub-tiles of 128 rows x 64 columns: a half's
// scores are computed on all 128 rows and read from its own 64 lanes.  Warps 0, 1 and 2, 3 do the softmax of the halves in turn (a lane
// a key), warp 4 issues the MMAs, warps 5 - 8 fetch: whole tiles by TMA boxes of 16 rows, tiles with an end (or pages whose size is no
// multiple of 16) by cp.async with zeros outside.
// The softmax needs no running maximum: weights are taken against a reference m per head, the maximum of the share's first tile (and the sink), and
// bf16 and fp32 keep their relative precision for every weight from 2^-100 to 2^60.  If a later score exceeds m by more than 60 (in
// powers of two), the share is computed again with the maxima found.  A weight is two bf16 numbers, its rounding and what that left
// over, side by side in the 128 bytes of a key's row of P: with one, the largest weights, which a running maximum makes exactly one,
// are rounded too (error against 64 bits 0.00210, 0.00206 with a running maximum, 0.0018 with both halves).
// Bound: the bytes of the cached rows (74 KB a tile and SM).  64 sequences x 32 heads x 2560 keys of 576 in a graph, merge of two shares a
// row included: 137 us on mma.sync (its own chain of ldmatrix, MMA and barriers, two warps a scheduler), 60 here (on 128 SMs: a tile's
// load, scores, softmax and output follow one another in each half of the ring).  An output goes before the next scores whenever those
// still wait for their tile: always behind them, it took 88.  Start and end take 13 us with a single tile; they took 20 with the queries
// loaded one after another in front of the first tile, row sums by one warp and a branch around every store.
#include "b2_act.cuh"
#include "b2_tc5.cuh"

namespace {
using namespace b2tc;
using bf16 = __nv_bfloat16;

constexpr int KT = 64, HEADS = 32, SUB = 128 * 128, NTHREADS = 288;      // keys a tile; bytes of a sub-tile of 128 rows x 64 columns
constexpr int Q_SUB = HEADS * 128;
constexpr float kLog2e = 1.4426950408889634f, kRedo = 60.f;

struct LatentArgs {
    CUtensorMap map;                                 // the pool as rows of Dc numbers, boxes of 16 rows x 64 columns
    const bf16 *qa, *cache;
    const int32_t *block_tables, *cu_q, *ctx_start;
    int n_seq, max_nb, H, dr, bs, window, tma;
    float scale_log2;
    const float* sink_logits;
    const bf16* gate;
    int64_t gate_stride;
    bf16* out;
    float *ws_o, *ws_ml;
};

// what two floats lose when they are rounded to the pair `hi` of bf16, as bf16
__device__ __forceinline__ uint32_t left_over(float a, float b, uint32_t hi) {
    return b2::pack_bf16x2(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}
// order of floats as order of ints (its own inverse)
__device__ __forceinline__ int ordered(int bits) { return bits ^ ((bits >> 31) & 0x7fffffff); }

template <int RT>                                    // R = 128 RT
__global__ void __launch_bounds__(NTHREADS, 1)
latent_tc5_kernel(const __grid_constant__ LatentArgs p) {
    constexpr int R = 128 * RT, COLS = RT == 4 ? 512 : RT == 2 ? 256 : 128;      // TMEM: S of the halves at 0 and 32, O^T at 64
    extern __shared__ unsigned char lat_sm_raw[];
    __shared__ __align__(8) uint64_t s_bar[10];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed, s_redo;
    __shared__ int s_max[HEADS];                     // ordered(): maxima found
    __shared__ __align__(16) float s_ref[HEADS];
    __shared__ __align__(16) float s_f[HEADS];
    __shared__ float s_sum[4][HEADS];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // a CTA belongs to a row: as many rows as sequences is one row each as a rule, but [2, 0] is as many too
    const int tok = blockIdx.x, guess = p.ctx_start[tok];            // asked for beside the row's sequence: nearly always its own
    const int seq = b2::seq_of_row(p.cu_q, p.n_seq, tok), h0 = blockIdx.y * HEADS, nh = min(HEADS, p.H - h0);
    const int nsplit = gridDim.z, zs = blockIdx.z, ctx = seq == tok ? guess : p.ctx_start[seq], bs = p.bs;
    const int pos = ctx + tok - p.cu_q[seq], klo = p.window > 0 ? max(pos - p.window + 1, 0) : 0, kbase = klo & ~15;
    const int all_tiles = ctx < 0 ? 0 : (pos - kbase) / KT + 1, per = (all_tiles + nsplit - 1) / nsplit;
    const int t0 = zs * per, nt = min(all_tiles, t0 + per) - t0;
    if (nt <= 0) {                                   // padding, or a share without keys
        if (nsplit > 1) {
            for (int h = tid; h < nh; h += NTHREADS) {
                float* ml = p.ws_ml + (((size_t)tok * p.H + h0 + h) * nsplit + zs) * 2;
                ml[0] = -INFINITY;
                ml[1] = 0.f;
            }
        } else {
            for (int idx = tid; idx < nh * (R / 8); idx += NTHREADS)
                *reinterpret_cast<uint4*>(p.out + ((size_t)tok * p.H + h0) * R + idx * 8) = make_uint4(0, 0, 0, 0);
        }
        return;
    }
    const int Dc = R + p.dr, NS = (Dc + 63) / 64;
    const uint32_t ring = (b2::smem_u32(lat_sm_raw) + 1023u) & ~1023u, q_sm = ring + NS * SUB, p_sm = q_sm + NS * Q_SUB;
    unsigned char* gen = lat_sm_raw + (ring - b2::smem_u32(lat_sm_raw));
    volatile int* failed = &s_failed;
    auto bar = [&](int i) { return b2::smem_u32(&s_bar[i]); };
    enum { FULL = 0, EMPTY = 2, SC = 4, PR = 6, END = 8, QUERY = 9 };
    if (tid == 0) {
        s_failed = s_redo = 0;
        for (int s = 0; s < 2; ++s) {
            b2::mbar_init(bar(FULL + s), 4);         // one arrive per fetching warp
            b2::mbar_init(bar(EMPTY + s), 1);
            b2::mbar_init(bar(SC + s), 1);
            b2::mbar_init(bar(PR + s), 2);           // ... per softmax warp of the half
        }
        b2::mbar_init(bar(END), 1);
        b2::mbar_init(bar(QUERY), 5);                // one arrive per warp that loads queries
        b2::fence_mbar_init();
    }
    // the sink counts among the scores the reference is taken from: a sum is at least one and finite, which the merge relies on
    if (tid < HEADS) s_max[tid] = ordered(__float_as_int(p.sink_logits && zs == 0 ? p.sink_logits[h0 + min(tid, nh - 1)] * kLog2e : -INFINITY));
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(b2::smem_u32(&s_tmem)), "n"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int32_t* bt = p.block_tables + (size_t)seq * p.max_nb;
    float l[HEADS], mx[HEADS];
    if (warp < 5) {                                  // the queries, five loads in flight, while the other warps fetch the first tiles
        const int qc = Dc / 8;
        const bf16* q = p.qa + ((size_t)tok * p.H + h0) * Dc;
        for (int first = tid; first < HEADS * qc; first += 5 * 160) {
            uint4 v[5];
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                const int idx = first + u * 160;
                v[u] = make_uint4(0, 0, 0, 0);
                if (idx < nh * qc) v[u] = *reinterpret_cast<const uint4*>(q + idx * 8);
            }
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                const int idx = first + u * 160, r = idx / qc, c = idx - r * qc;
                if (idx < HEADS * qc) *reinterpret_cast<uint4*>(gen + (q_sm - ring) + (c >> 3) * Q_SUB + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = v[u];
            }
        }
        b2::fence_proxy_async();
        __syncwarp();
        if (lane == 0) b2::mbar_arrive(bar(QUERY));
    }
#pragma unroll
    for (int h = 0; h < HEADS; ++h) mx[h] = -INFINITY;

    for (int pass = 0, it0 = 0; pass < 2; ++pass, it0 += nt) {           // `it` counts the tiles of both passes: half it & 1
        if (warp >= 5) {
            // ---------------------------------------------- fetch
            const int cw = warp - 5;
            int row_a = 0, row_b = 0;                // pool rows of this lane's boxes of the tile to come
            auto pool_row = [&](int j) {
                const int pg = j / bs;
                return bt[pg] * bs + j - pg * bs;
            };
            auto whole = [&](int t) {
                const int kv0 = kbase + (t0 + t) * KT;
                return p.tma && kv0 >= klo && kv0 + KT - 1 <= pos;
            };
            auto lookup = [&](int t) {
                if (cw != 0 || t >= nt || !whole(t)) return;
                const int kv0 = kbase + (t0 + t) * KT;
                row_a = pool_row(kv0 + (lane / NS) * 16 * (lane < 4 * NS));
                if (lane + 32 < 4 * NS) row_b = pool_row(kv0 + (lane + 32) / NS * 16);
            };
            lookup(0);
#pragma unroll 1
            for (int t = 0; t < nt; ++t) {
                const int it = it0 + t, s = it & 1, kv0 = kbase + (t0 + t) * KT;
                const uint32_t base = ring + s * (KT * 128), full = bar(FULL + s);
                if (it >= 2 && !__all_sync(0xffffffffu, wait(bar(EMPTY + s), ((it >> 1) - 1) & 1, failed))) break;
                if (whole(t)) {
                    if (cw == 0) {
                        if (lane == 0) b2::mbar_arrive_expect_tx(full, (uint32_t)NS * KT * 128);      // columns past Dc are zero-filled and count
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int idx = lane + 32 * u, sub = idx % NS, pg = idx / NS;
                            if (idx < 4 * NS) tma_load_2d(base + sub * SUB + pg * 2048, &p.map, full, sub * 64, u ? row_b : row_a);
                        }
                        __syncwarp();
                    } else if (lane == 0) {
                        b2::mbar_arrive(full);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int r = cw * 16 + (lane >> 3) + 4 * u, j = kv0 + r;
                        const bool there = j >= klo && j <= pos;         // others are zeros: 0 * NaN must not reach an accumulator
                        const bf16* src = p.cache + (there ? (size_t)pool_row(j) * Dc : 0);
#pragma unroll 1
                        for (int sub = 0; sub < NS; ++sub) {
                            const int col = sub * 64 + (lane & 7) * 8;
                            const bool ok = there && col < Dc;
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                                         ::"r"(base + sub * SUB + r * 128 + (((lane & 7) ^ (r & 7)) << 4)), "l"(ok ? src + col : p.cache), "r"(ok ? 16 : 0)
                                         : "memory");
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    b2::fence_proxy_async();         // this lane's copies, before the MMAs that read them
                    __syncwarp();
                    if (lane == 0) b2::mbar_arrive(full);
                }
                lookup(t + 1);
            }
        } else if (warp == 4) {
            // ---------------------------------------------- MMA issuer
            constexpr uint32_t ID_S = idesc_bf16(128, HEADS, 0), ID_O = idesc_bf16(128, 2 * HEADS, 1) | (1u << 15);  // O^T: A MN-major too
            const int ksteps = Dc / 16;
            auto scores = [&](int t) {
                const int it = it0 + t, s = it & 1;
                wait(bar(FULL + s), (it >> 1) & 1, failed);
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t kl = desc_lo(ring, 16), ql = desc_lo(q_sm, 16);
#pragma unroll 4
                    for (int kk = 0; kk < ksteps; ++kk)
                        mma_ss(tmem + 32 * s, desc_join(kl + (((kk >> 2) * SUB + (kk & 3) * 32) >> 4)),
                               desc_join(ql + (((kk >> 2) * Q_SUB + (kk & 3) * 32) >> 4)), ID_S, kk > 0);
                    mma_commit(bar(SC + s));
                }
                __syncwarp();
            };
            wait(bar(QUERY), 0, failed);
            scores(0);
#pragma unroll 1
            for (int t = 0; t < nt; ++t) {
                const int it = it0 + t, s = it & 1;
                // The next scores go first if their tile is there, else behind this output.  Lanes may see a phase end at different
                // probes, and both branches hold instructions of the whole warp: every answer is the warp's vote, not the lane's.
                bool ahead = t + 1 < nt;
                for (uint32_t spins = 0; !__all_sync(0xffffffffu, b2::mbar_try_wait(bar(PR + s), (it >> 1) & 1));) {
                    if (ahead && __all_sync(0xffffffffu, b2::mbar_try_wait(bar(FULL + (s ^ 1)), ((it + 1) >> 1) & 1))) {
                        scores(t + 1);
                        ahead = false;
                    }
                    if (__any_sync(0xffffffffu, *failed || ++spins > (1u << 22))) { *failed = 1; break; }
                }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t vl = desc_lo(ring + s * (KT * 128), SUB), pl = desc_lo(p_sm + s * (KT * 128), 16);
#pragma unroll
                    for (int m = 0; m < RT; ++m)
#pragma unroll
                        for (int kk = 0; kk < KT / 16; ++kk)
                            mma_ss(tmem + 64 + 64 * m, desc_join(vl + ((m * 2 * SUB + kk * 2048) >> 4)), desc_join(pl + (kk * 2048 >> 4)), ID_O,
                                   t > 0 || kk > 0);
                    mma_commit(bar(EMPTY + s));
                    if (t + 1 == nt) mma_commit(bar(END));
                }
                __syncwarp();
                if (ahead) scores(t + 1);
            }
            if (!wait(bar(END), pass, failed)) drain(bar(END), pass);
        } else {
            // ---------------------------------------------- softmax: lane = key; warps 0, 1 the first half of the ring, 2, 3 the second
#pragma unroll
            for (int h = 0; h < HEADS; ++h) l[h] = 0.f;
            auto publish = [&]() {                   // s_max: the maxima over this warp's lanes
#pragma unroll
                for (int h = 0; h < HEADS; ++h) {
                    const int m = __reduce_max_sync(0xffffffffu, ordered(__float_as_int(mx[h])));
                    if (lane == h) atomicMax(&s_max[h], m);
                }
            };
            auto settle = [&]() {                    // the four warps: references from s_max
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (tid < HEADS) {
                    const float m = __int_as_float(ordered(s_max[tid]));
                    s_ref[tid] = m == -INFINITY ? 0.f : m;
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            };
            if (pass == 1) publish();                // all the maxima found
            if (pass == 1 || warp >= 2) settle();
#pragma unroll 1
            for (int t = (it0 ^ (warp >> 1)) & 1; t < nt; t += 2) {
                const int it = it0 + t, s = it & 1, r = (warp & 1) * 32 + lane, j = kbase + (t0 + t) * KT + r;
                const bool in = j >= klo && j <= pos;
                wait(bar(SC + s), (it >> 1) & 1, failed);
                tc_fence_after();
                uint32_t acc[32], rest[16];
                tmem_ld32(tmem + 32 * s + ((uint32_t)(warp * 32) << 16), acc);
                tmem_wait_ld();
#pragma unroll
                for (int h = 0; h < HEADS; ++h) {
                    const float x = in ? __uint_as_float(acc[h]) * p.scale_log2 : -INFINITY;
                    mx[h] = fmaxf(mx[h], x);
                    acc[h] = __float_as_uint(x);
                }
                if (pass == 0 && t == 0) {           // warps 0 and 1
                    publish();
                    settle();
                }
#pragma unroll
                for (int h = 0; h < HEADS; h += 4) {
                    const float4 m = *reinterpret_cast<const float4*>(s_ref + h);
                    const float e0 = b2::fast_exp2(__uint_as_float(acc[h]) - m.x), e1 = b2::fast_exp2(__uint_as_float(acc[h + 1]) - m.y);
                    const float e2 = b2::fast_exp2(__uint_as_float(acc[h + 2]) - m.z), e3 = b2::fast_exp2(__uint_as_float(acc[h + 3]) - m.w);
                    l[h] += e0;
                    l[h + 1] += e1;
                    l[h + 2] += e2;
                    l[h + 3] += e3;
                    acc[h / 2] = b2::pack_bf16x2(e0, e1);
                    acc[h / 2 + 1] = b2::pack_bf16x2(e2, e3);
                    rest[h / 2] = left_over(e0, e1, acc[h / 2]);
                    rest[h / 2 + 1] = left_over(e2, e3, acc[h / 2 + 1]);
                }
                unsigned char* prow = gen + (p_sm - ring) + (s * KT + r) * 128;      // [key][heads, heads' rests], as C's sub-tiles
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    *reinterpret_cast<uint4*>(prow + ((c ^ (r & 7)) << 4)) = make_uint4(acc[4 * c], acc[4 * c + 1], acc[4 * c + 2], acc[4 * c + 3]);
                    *reinterpret_cast<uint4*>(prow + (((4 + c) ^ (r & 7)) << 4)) = make_uint4(rest[4 * c], rest[4 * c + 1], rest[4 * c + 2], rest[4 * c + 3]);
                }
                b2::fence_proxy_async();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) b2::mbar_arrive(bar(PR + s));
            }
            if (pass == 0) {
                bool far = false;
#pragma unroll
                for (int h = 0; h < HEADS; ++h) far |= mx[h] > s_ref[h] + kRedo;
                if (__any_sync(0xffffffffu, far) && lane == 0) s_redo = 1;
            }
        }
        __syncthreads();                             // every tile is consumed, O^T is complete
        if (!s_redo) break;
    }
    wait(bar(END), s_redo ? 1 : 0, failed);
    tc_fence_after();
    // row sums: lanes' parts through the ring, which nothing reads any more
    float* part = reinterpret_cast<float*>(gen);     // [128][33]
    if (warp < 4)
#pragma unroll
        for (int h = 0; h < HEADS; ++h) part[tid * (HEADS + 1) + h] = l[h];
    __syncthreads();
    if (warp < 4) {                                  // a quarter of the lanes' parts a warp
        float sum = 0.f;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) sum += part[(warp * 32 + r) * (HEADS + 1) + lane];
        s_sum[warp][lane] = sum;
    }
    __syncthreads();
    if (tid < HEADS) {
        float sum = (s_sum[0][tid] + s_sum[1][tid]) + (s_sum[2][tid] + s_sum[3][tid]);
        const int h = h0 + min(tid, nh - 1);
        if (p.sink_logits && zs == 0) sum += b2::fast_exp2(p.sink_logits[h] * kLog2e - s_ref[tid]);
        if (s_failed) sum = __int_as_float(0x7fc00000);
        float f = 1.f;
        if (nsplit > 1) {
            if (tid < nh) {
                float* ml = p.ws_ml + (((size_t)tok * p.H + h) * nsplit + zs) * 2;
                ml[0] = s_ref[tid];
                ml[1] = sum;
            }
        } else {
            f = sum > 0.f ? 1.f / sum : sum == 0.f ? 0.f : sum;          // NaN stays NaN
            if (p.gate) f *= b2::sigmoid_f(__bfloat162float(p.gate[(size_t)tok * p.gate_stride + h]));
        }
        s_f[tid] = f;
    }
    __syncthreads();
    if (warp < 4) {
#pragma unroll 1
        for (int m = 0; m < RT; ++m) {
            uint32_t acc[32], rest[32];
            tmem_ld32(tmem + 64 + 64 * m + ((uint32_t)(warp * 32) << 16), acc);
            tmem_ld32(tmem + 96 + 64 * m + ((uint32_t)(warp * 32) << 16), rest);
            tmem_wait_ld();
            const size_t row = (size_t)tok * p.H + h0;
            if (nsplit > 1) {
                float* o = p.ws_o + (row * nsplit + zs) * R + 128 * m + tid;
                const size_t step = (size_t)nsplit * R;
#pragma unroll
                for (int h = 0; h < HEADS; ++h)
                    if (h < nh) o[h * step] = __uint_as_float(acc[h]) + __uint_as_float(rest[h]);
            } else {
                bf16* o = p.out + row * R + 128 * m + tid;
#pragma unroll
                for (int h = 0; h < HEADS; h += 4) {
                    const float4 f4 = *reinterpret_cast<const float4*>(s_f + h);
                    const float f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (h + u < nh) o[(h + u) * R] = __float2bfloat16_rn((__uint_as_float(acc[h + u]) + __uint_as_float(rest[h + u])) * f[u]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 4) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS) : "memory");
    if (*failed && lane == 0) {                      // boxes that nobody has waited for: every role is done now
        const int n = s_redo ? 2 * nt : nt;          // (a tile that was never begun takes the whole millisecond, which is as good)
        for (int it = max(0, n - 2); it < n; ++it) drain(bar(FULL + (it & 1)), (it >> 1) & 1);
    }
}

size_t smem_bytes(int Dc) { return (size_t)((Dc + 63) / 64) * (SUB + Q_SUB) + SUB + 1024; }

}  // namespace

// R = 128, 256 or 512, dr a multiple of 16; pointers and rows of 16 bytes
bool b2_internal_latent_tc5_ok(int R, int dr) {
    return (R == 128 || R == 256 || R == 512) && dr % 16 == 0 && smem_bytes(R + dr) <= 226 * 1024;
}
int b2_internal_latent_tc5_heads(void) { return HEADS; }

int b2_internal_latent_tc5(void* out, const void* qa, const void* cache, const int32_t* block_tables, int max_nb, const int32_t* cu_q,
                           const int32_t* ctx_start, int n_seq, int T, int H, int R, int dr, int bs, float scale, int window, const float* sink_logits,
                           const void* gate, int64_t gate_stride, int nsplit, float* ws_o, float* ws_ml, void* stream) {
    LatentArgs p{};
    const int Dc = R + dr;
    p.qa = static_cast<const bf16*>(qa);
    p.cache = static_cast<const bf16*>(cache);
    p.block_tables = block_tables; p.cu_q = cu_q; p.ctx_start = ctx_start; p.n_seq = n_seq; p.max_nb = max_nb;
    p.H = H; p.dr = dr; p.bs = bs; p.window = window; p.scale_log2 = scale * kLog2e;
    p.sink_logits = sink_logits;
    p.gate = static_cast<const bf16*>(gate);
    p.gate_stride = gate_stride;
    p.out = static_cast<bf16*>(out);
    p.ws_o = ws_o; p.ws_ml = ws_ml;
    p.tma = bs % 16 == 0;                            // a box of 16 rows never leaves its page
    if (p.tma) {                                     // rows of the pool: the caller's pages, of which 2^31 tokens are the limit
        const uint64_t dims[2] = {(uint64_t)Dc, (uint64_t)1 << 31}, st[1] = {(uint64_t)Dc * 2};
        const uint32_t box[2] = {64, 16};
        const int rc = b2_internal_encode_bf16_sw128(&p.map, cache, 2, dims, st, box);
        if (rc != B2_OK) return rc;
    }
    const size_t smem = smem_bytes(Dc);
    const dim3 grid(T, (H + HEADS - 1) / HEADS, nsplit);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto kern = R == 512 ? latent_tc5_kernel<4> : R == 256 ? latent_tc5_kernel<2> : latent_tc5_kernel<1>;
    B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, NTHREADS, smem, s>>>(p);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}
