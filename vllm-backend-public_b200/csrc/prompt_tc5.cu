// prompt_tc5.cu -- masked prompt attention on the 5th-gen tensor cores: the prompt rows of b2_masked_attention (paged pools per
// kv head) and of b2_window_attention (keys and values rebuilt per head in gathered buffers), with every option of those entry
// points: sliding window with kept first tokens, mask blocks, sinks, capped scores, sigmoid weights, two maps per head, gates.
//
// A CTA takes one tile: 128 query rows of a head in one slot, or two slots: two heads of a kv head on the same rows, two row tiles of a head, or
// its two maps on the same rows (differential attention: slot x multiplies the keys of map x).  Warps 0-3 / 4-7 are the softmax of slot 0 / 1 (a
// thread per row = TMEM lane), warp 9 issues the MMAs, warps 8 and 11 copy K tiles, warp 10 V tiles (all three Q), 128 keys at a time.  Launches
// of more tiles are prompt_turns_tc5.cu's.
// Keys are walked in the compact order of KeySpan (kept first keys, then the union of the rows' windows), so a window costs no
// tiles between its parts and neither page size nor alignment shows: the copies are 16-byte cp.async gathers with a page lookup
// per key row, written in the 128-byte swizzle that the MMA descriptors name (gathered rows: TMA boxes).  A mask is tested per
// score only in tiles that the slot's rows see in part.
// S = Q K^T and O += P V are tcgen05.mma 128x128x16 (bf16 -> fp32 in TMEM); P replaces S in TMEM and is the A operand of the
// second product.  The online softmax takes a row's weights against its maximum so far, whatever that costs in rescales of O: the largest
// weight is exactly one then and loses nothing in bf16.  (A row that kept its maximum until the true one exceeded it by 2^8 saved 7 us of
// 124 at 4096 capped rows, and its error against 64 bits was 0.0029 instead of 0.0028.)
//
// Bound: tensor pipe (2 (dk + dv) flops per visible pair) and, for the exponentials, the XU pipe, 16 a clock and SM.  A capped
// score would need two more XU operations (the exponential and the division of tanh): where a whole warp's scores are below 3/16
// of the cap, tanh is its Taylor polynomial to x^7 on the packed FMA pipe instead (remainder below 7e-9; the exponential form's
// error is one fp32 rounding, 6e-8).
// Attention alone in a graph: 300 rows x 16 heads of 128 on 4 kv heads, causal, 12.9 us; 1000 rows 23.3; 1200 gathered rows x 16 heads of
// 128 + 64 / 128, causal, 24.4 (25.4 with one V stage, which the second slot's Q once cost the form of one).  A step of 128 keys is the softmax of the tile (0.5k cycles for the maximum, 0.6k to bring O along, 1.4k for the
// weights) and the MMAs behind it, one after the other.
// What cost most on the way: code size (95 - 145 KB with everything unrolled: every warp waited for instructions, 10.9k cycles per
// tile; loops are rolled wherever registers are not indexed), and a divergent branch per row in the copies (~100 cycles an
// instruction, serialised; zero-filling copies need none).
#include "prompt_tc5.cuh"

#include <algorithm>

namespace {

using namespace b2tc;
using namespace b2prompt;

constexpr int NTHREADS = 384;

// NH: 64-column sub-tiles of a slot's Q and K; DVH: of V.  Three sub-tiles of two slots leave room for one V stage beside two of K.
template <int NH, int DVH, bool TWO_MAPS, bool PAIRS>
struct Shape {
    static constexpr int SLOTS = TWO_MAPS || PAIRS ? 2 : 1;
    static constexpr int VST = SLOTS * NH <= 4 ? 2 : 1, KST = 2;
    static constexpr int KSUBS = TWO_MAPS ? 2 : NH;
    static constexpr int Q_BYTES = SLOTS * NH * SUB, K_STAGE = KSUBS * SUB, V_STAGE = DVH * SUB;
    static constexpr int BAR_Q = 0, BAR_K = 1, BAR_V = BAR_K + KST, BAR_KE = BAR_V + VST, BAR_VE = BAR_KE + KST, BAR_S = BAR_VE + VST,
                         BAR_P = BAR_S + 2, BAR_P2 = BAR_P + 2, BAR_PV = BAR_P2 + 2, BAR_END = BAR_PV + 2, BARS = BAR_END + 1;
    static constexpr int SMEM = Q_BYTES + KST * K_STAGE + VST * V_STAGE + 256;
    static_assert(BARS * 8 <= 256, "barrier area");
};

struct Params {
    b2_prompt_args a;
    int rows_per_cta, heads_per_cta;
    int bs_shift;                                    // log2 of the page size, or -1
    float scale_log2;
    int tma;                                         // gathered form: whole key tiles come by TMA boxes of 128 rows x 64 columns
    CUtensorMap map_k0, map_k1, map_v;
};

// (s0, s1) (1 + z a1 + z^2 a2 + z^3 a3), z = s^2, on the packed pipe: s tanh(x) / x of a score s = x / c, a_i = t_i c^2i with the
// Taylor coefficients -1/3, 2/15, -17/315
__device__ __forceinline__ void tanh_small_x2(uint32_t& s0, uint32_t& s1, float a1, float a2, float a3) {
    asm("{\n\t.reg .b64 s, z, p, c1, c2, c3;\n\t"
        "mov.b64 s, {%0, %1};\n\tmov.b64 c1, {%2, %2};\n\tmov.b64 c2, {%3, %3};\n\tmov.b64 c3, {%4, %4};\n\t"
        "mul.rn.f32x2 z, s, s;\n\tfma.rn.f32x2 p, z, c3, c2;\n\tfma.rn.f32x2 p, z, p, c1;\n\tmul.rn.f32x2 p, z, p;\n\t"
        "fma.rn.f32x2 s, s, p, s;\n\tmov.b64 {%0, %1}, s;\n\t}"
        : "+r"(s0), "+r"(s1) : "f"(a1), "f"(a2), "f"(a3));
}
// what one thread works out for the CTA
struct Plan {
    KeySpan span;
    int keep;                                        // compact index below which keys are kept for every row of their mask block
    int first_row[2], rows[2];                       // position of a slot's first row, number of rows
    int t0[2], t1[2];                                // a slot works on the key tiles t0 .. t1 - 1
    int all_hi[2], all_low[2];                       // keys all_low .. all_hi are visible to every row of the slot
};

template <int NH, int DVH, int KIND, bool TWO_MAPS, bool GATHERED, bool PAIRS>
__global__ void __launch_bounds__(NTHREADS, 1)
prompt_tc5_kernel(const __grid_constant__ Params prm) {
    using L = Shape<NH, DVH, TWO_MAPS, PAIRS>;
    using bf16 = __nv_bfloat16;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ Plan s_plan;
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    __shared__ float s_inv[TWO_MAPS ? BM : 1];
    const b2_prompt_args& a = prm.a;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);          // warp-uniform for the compiler too
    const uint32_t q_smem = b2::smem_u32(smem_raw);
    const uint32_t k_ring = q_smem + L::Q_BYTES, v_ring = k_ring + L::KST * L::K_STAGE, bars = v_ring + L::VST * L::V_STAGE;
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile int* failed = &s_failed;

    // This CTA's tile: counted from the batch's last row backwards (late rows see more keys, and the spare CTAs of a grid that is an
    // upper bound come behind all tiles), by every warp for itself, 32 sequences at a time, so that a spare CTA leaves at once.
    const int hpc = PAIRS ? prm.heads_per_cta : 1, rows_per_cta = PAIRS ? prm.rows_per_cta : BM;
    const bool two_rows = rows_per_cta > BM;
    const int groups = a.H / hpc, group = blockIdx.x % groups;
    int seq = -1, q0 = 0, len = 0;
    {
        int want = blockIdx.x / groups;
#pragma unroll 1
        for (int top = a.n_seq - 1; top >= 0; top -= 32) {
            const int s = top - lane, n = s >= 0 ? a.cu_q[s + 1] - a.cu_q[s] : 0;
            const int nt = n >= a.min_rows ? (n + rows_per_cta - 1) / rows_per_cta : 0;
            int upto = nt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += below;
            }
            const uint32_t hit = __ballot_sync(0xffffffffu, want < upto);
            if (hit) {
                const int who = __ffs(hit) - 1;
                seq = top - who;
                len = __shfl_sync(0xffffffffu, n, who);
                q0 = (__shfl_sync(0xffffffffu, upto, who) - 1 - want) * rows_per_cta;
                break;
            }
            want -= __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (seq < 0) return;
    const int ctx = a.ctx_start[seq], row0 = a.cu_q[seq] + q0;
    if (ctx < 0) {                                                   // padding: zero rows (the paged form's are another kernel's)
        const int rows = GATHERED ? min(len - q0, rows_per_cta) : 0, v8 = a.dv / 8;
        for (int idx = tid; idx < rows * v8; idx += NTHREADS)
            *reinterpret_cast<uint4*>(static_cast<bf16*>(a.out) + (size_t)(row0 + idx / v8) * a.out_stride + (size_t)group * a.dv + (idx % v8) * 8) =
                make_uint4(0, 0, 0, 0);
        return;
    }

    if (tid == 0) {
        s_failed = 0;
        Plan& pl = s_plan;
        pl.rows[0] = pl.rows[1] = pl.t0[0] = pl.t0[1] = pl.t1[0] = pl.t1[1] = 0;
        {
            const int left = len - q0, p0 = ctx + q0, p_last = p0 + min(left, rows_per_cta) - 1;
            KeySpan span = key_span(p0, p_last, a.chunk, a.window, a.keep_first);
            if (GATHERED && span.wlo < a.k_lo[seq]) {                // the gathered rows begin at k_lo
                span.wlo = span.lo = a.k_lo[seq];
                span.n = p_last - span.lo + 1;
            }
            pl.span = span;
            pl.keep = a.window > 0 ? span.index(a.keep_first) : 0;
            pl.rows[0] = min(BM, left);
            pl.rows[1] = two_rows ? min(BM, max(0, left - BM)) : (TWO_MAPS || hpc == 2) ? pl.rows[0] : 0;
#pragma unroll 1
            for (int x = 0; x < 2; ++x) {
                if (pl.rows[x] == 0) continue;
                const int pf = p0 + (two_rows && x ? BM : 0);
                const RowRange f = range_of(span, pf, a.chunk, a.window), l = range_of(span, pf + pl.rows[x] - 1, a.chunk, a.window);
                pl.first_row[x] = pf;
                pl.t0[x] = (f.block < pl.keep ? f.block : f.low) / BN;
                pl.t1[x] = l.hi / BN + 1;
                pl.all_hi[x] = f.hi;
                pl.all_low[x] = l.low;
            }
        }
        b2::mbar_init(bar(L::BAR_Q), 3);                             // one arrive per copying warp
        for (int s = 0; s < L::KST; ++s) { b2::mbar_init(bar(L::BAR_K + s), 2); b2::mbar_init(bar(L::BAR_KE + s), 1); }
        for (int s = 0; s < L::VST; ++s) { b2::mbar_init(bar(L::BAR_V + s), 1); b2::mbar_init(bar(L::BAR_VE + s), 1); }
        for (int x = 0; x < 2; ++x) {
            b2::mbar_init(bar(L::BAR_S + x), 1);
            b2::mbar_init(bar(L::BAR_P + x), 4);                     // one arrive per softmax warp: keys 0-63 of P are in TMEM
            b2::mbar_init(bar(L::BAR_P2 + x), 4);                    // ... keys 64-127
            b2::mbar_init(bar(L::BAR_PV + x), 1);
        }
        b2::mbar_init(bar(L::BAR_END), 1);
        b2::fence_mbar_init();
    }
    if (warp == 9) {                                                 // all 512 columns: one CTA per SM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(b2::smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int n_tiles = max(s_plan.t1[0], s_plan.t1[1]), n_keys = s_plan.span.n;
    const int kvh = (group * hpc) / (a.H / a.G);                     // kv head of the paged pools

    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp != 9) {
            // ------------------------------------------ copies: warps 8 and 11 the even and odd groups of K rows, warp 10 V
            // Eight lanes copy the 128 bytes of a row and sub-tile, four rows (a group) an instruction.  The pool rows of a tile's
            // 128 keys (four a lane, through the page table) are looked up before the stage is free: a lookup in front of its
            // copies would put its latency on the path of every tile.
            const int c8 = lane & 7, rsub = lane >> 3;
            const bool is_v = warp == 10;
            const int odd = warp == 11;
            const int32_t* bt = GATHERED ? nullptr : a.block_tables + (int64_t)seq * a.max_nb;
            const uint32_t g0 = GATHERED ? (uint32_t)a.cu_k[seq] - (uint32_t)a.k_lo[seq] : 0u;
            constexpr uint32_t NONE = 0xffffffffu;
            const uint32_t heads = (uint32_t)(TWO_MAPS && !is_v ? 2 * a.G : a.G), head0 = (uint32_t)(TWO_MAPS && !is_v ? 2 * kvh : kvh);
            const KeySpan span = s_plan.span;
            uint32_t rows[4];
            auto lookup = [&](int it) {                              // pool rows (of this head) of keys it * 128 + lane + 32 q
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int c = it * BN + q * 32 + lane;
                    rows[q] = NONE;
                    if (c < n_keys) {
                        const int j = span.key(c);
                        if (GATHERED) {
                            rows[q] = g0 + (uint32_t)j;
                        } else {
                            int pg = j >> (prm.bs_shift & 31);
                            if (prm.bs_shift < 0) pg = j / a.bs;
                            rows[q] = ((uint32_t)bt[pg] * heads + head0) * (uint32_t)a.bs + (uint32_t)(j - pg * a.bs);
                        }
                    }
                }
            };
            // row r = 4 group + rsub: the swizzled column of even and odd groups; a group is 512 bytes
            const uint32_t sw_even = (uint32_t)(rsub * 128 + ((c8 ^ rsub) << 4)), sw_odd = (uint32_t)(rsub * 128 + ((c8 ^ (4 + rsub)) << 4));
            {                                                        // Q, by all three warps: rows past the tile are zeros
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    const int hh = group * hpc + (hpc == 2 ? x : 0), nrows = s_plan.rows[x];
                    const int rbase = row0 + (two_rows && x ? BM : 0);
                    if (nrows == 0) continue;
                    const int col0 = TWO_MAPS ? x * a.dk : 0;
                    const char* qh = reinterpret_cast<const char*>(static_cast<const bf16*>(a.q0) + (size_t)rbase * a.q0_row + (size_t)hh * a.q0_head + col0 + c8 * 8);
                    const char* q1 = GATHERED ? reinterpret_cast<const char*>(static_cast<const bf16*>(a.q1) + (size_t)rbase * a.q1_row + (size_t)hh * a.q1_head + c8 * 8) - 2 * a.dk0 : qh;
#pragma unroll 4
                    for (int rg = is_v ? 2 : odd; rg < BM / 4; rg += 3) {
                        const int r = rg * 4 + rsub, rr = min(r, nrows - 1);
                        const char* s0 = qh + (size_t)rr * (2 * a.q0_row);
                        const char* s1 = GATHERED ? q1 + (size_t)rr * (2 * a.q1_row) : nullptr;
#pragma unroll
                        for (int h = 0; h < NH; ++h) {
                            const int col = h * 64 + c8 * 8;
                            const char* sp = (GATHERED && col >= a.dk0 ? s1 : s0) + h * 128;
                            const bool ok = r < nrows && col < a.dk;
                            cp_async16(q_smem + (x * NH + h) * SUB + rg * 512 + (rg & 1 ? sw_odd : sw_even), ok ? sp : s0, ok);
                        }
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            lookup(0);
            const int nst = is_v ? L::VST : L::KST;
            const int n_sub = is_v ? DVH : L::KSUBS, width = is_v ? a.dv : a.dk, split = GATHERED && !is_v ? a.dk0 : width;
            const uint32_t ld = 2u * (uint32_t)(GATHERED ? a.H * split : width), ld1 = 2u * (uint32_t)a.k1_row;    // bytes between pool rows
            const char* p0 = reinterpret_cast<const char*>(static_cast<const bf16*>(is_v ? a.v : a.k0) + (GATHERED ? (size_t)group * split : 0) + c8 * 8);
            const char* p1 = GATHERED && !is_v ? reinterpret_cast<const char*>(static_cast<const bf16*>(a.k1) + c8 * 8) - 2 * split : p0;
            const uint32_t map2 = 2u * (uint32_t)a.bs * (uint32_t)a.dk;                  // the second map's rows lie a page of the first behind
#pragma unroll 1
            for (int it = 0; it < n_tiles; ++it) {
                const int s = it % nst, ph = (it / nst) & 1;
                if (!__all_sync(0xffffffffu, wait(bar((is_v ? L::BAR_VE : L::BAR_KE) + s), ph ^ 1, failed))) break;
                const uint32_t base = is_v ? v_ring + s * L::V_STAGE : k_ring + s * L::K_STAGE;
                const uint32_t full = bar((is_v ? L::BAR_V : L::BAR_K) + s);
                const bool whole = GATHERED && prm.tma && (it + 1) * BN <= n_keys;      // all 128 rows are this sequence's
                if (whole && !odd) {
                    if (lane == 0) {
                        const int row = (int)g0 + span.wlo + it * BN, hh = group;
                        b2::mbar_arrive_expect_tx(full, (uint32_t)n_sub * SUB);          // columns past the head are zero-filled and count
#pragma unroll 1
                        for (int h = 0; h < n_sub; ++h) {
                            if (!is_v && h * 64 >= split) tma_load_2d(base + h * SUB, &prm.map_k1, full, h * 64 - split, row);
                            else tma_load_3d(base + h * SUB, is_v ? &prm.map_v : &prm.map_k0, full, h * 64, hh, row);
                        }
                    }
                    __syncwarp();
                }
#pragma unroll 1
                for (int q = 0; q < (whole ? 0 : is_v ? 8 : 4); ++q) {           // four groups each: K every second group, V every one
                    const int first = is_v ? q * 4 : q * 8 + odd, gs = is_v ? 1 : 2;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int g = first + u * gs;
                        const uint32_t pr = __shfl_sync(0xffffffffu, rows[0], (g & 7) * 4 + rsub);
                        const uint32_t dst = base + g * 512 + (g & 1 ? sw_odd : sw_even);
                        const bool there = pr != NONE;               // rows past the keys are zeros: 0 * NaN must not reach an accumulator
                        const char* src = p0 + (size_t)pr * ld;
                        const char* src1 = GATHERED ? p1 + (size_t)pr * ld1 : nullptr;
#pragma unroll
                        for (int h = 0; h < (L::KSUBS > DVH ? L::KSUBS : DVH); ++h) {
                            if (h < n_sub) {                         // warp-uniform
                                const int col = (TWO_MAPS && !is_v ? 0 : h * 64) + c8 * 8;
                                const char* sp = src + (TWO_MAPS && !is_v ? h * map2 : h * 128u);
                                if (GATHERED) sp = col >= split ? src1 + h * 128 : sp;
                                const bool ok = there && col < width;
                                cp_async16(dst + h * SUB, ok ? sp : p0, ok);
                            }
                        }
                    }
                    if (!is_v || (q & 1)) {
                        rows[0] = rows[1];
                        rows[1] = rows[2];
                        rows[2] = rows[3];
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                lookup(it + 1);
                if (it == 0) {                                       // Q has been in flight under the first keys' copies
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    b2::fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) b2::mbar_arrive(bar(L::BAR_Q));
                }
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                b2::fence_proxy_async();                             // this thread's copies, before the MMAs that read them
                __syncwarp();
                if (lane == 0 && !(whole && !odd)) b2::mbar_arrive(full);
            }
        } else {
            // ------------------------------------------ MMA issuer: the whole warp, warp-uniform operands, one elected lane
            // step j: P_0 V(j), Q_0 K(j+1), P_1 V(j), Q_1 K(j+1) -- the softmax of one slot runs under the MMAs of the other
            constexpr uint32_t ID_QK = idesc_bf16(128, 128, 0), ID_PV = idesc_bf16(128, 64 * DVH, 1);
            const uint32_t q_lo = desc_lo(q_smem, 16), k_lo = desc_lo(k_ring, 16), v_lo = desc_lo(v_ring, SUB);
            const int ksteps_qk = a.dk >> 4;
            const int t00 = s_plan.t0[0], t01 = s_plan.t0[1], t10 = s_plan.t1[0], t11 = s_plan.t1[1];
            wait(bar(L::BAR_Q), 0, failed);
#pragma unroll 1
            for (int j = -1; j < n_tiles; ++j) {
                const int s = j < 0 ? 0 : j % L::VST, sk = (j + 1) % L::KST;
                if (j >= 0) wait(bar(L::BAR_V + s), (j / L::VST) & 1, failed);
                if (j + 1 < n_tiles) wait(bar(L::BAR_K + sk), ((j + 1) / L::KST) & 1, failed);
                tc_fence_after();
                const int ksteps = min(8, (n_keys - j * BN + 15) >> 4);
                const uint32_t vl = v_lo + (uint32_t)s * (L::V_STAGE >> 4);
                const uint32_t kl0 = k_lo + (uint32_t)sk * (L::K_STAGE >> 4);
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    const int tb = x ? t01 : t00, te = x ? t11 : t10, i = j - tb;
                    const uint32_t tx = tmem + x * 128;
                    if (i >= 0 && j < te) {
                        wait(bar(L::BAR_P + x), i & 1, failed);      // keys 0-63 of P_x are in TMEM, O_x rescaled if needed
                        tc_fence_after();
                        if (elect_one()) {                           // O_x += P_x V(j): k-steps of 16 keys
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                if (t < ksteps) mma_ts(tx + 256, tx + t * 8, desc_join(vl + t * (2048 >> 4)), ID_PV, i > 0 || t > 0);
                        }
                        __syncwarp();
                        wait(bar(L::BAR_P2 + x), i & 1, failed);     // keys 64-127
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int t = 4; t < 8; ++t)
                                if (t < ksteps) mma_ts(tx + 256, tx + t * 8, desc_join(vl + t * (2048 >> 4)), ID_PV, true);
                            mma_commit(bar(L::BAR_PV + x));
                        }
                        __syncwarp();
                    }
                    if (x == 1 && j >= 0) {
                        if (elect_one()) mma_commit(bar(L::BAR_VE + s));     // V(j) consumed: its stage refills under the Q K^T below
                        __syncwarp();
                    }
                    if (j + 1 >= tb && j + 1 < te) {                 // S_x = Q_x K(j+1)^T
                        const uint32_t kl = kl0 + (TWO_MAPS ? (uint32_t)x * (SUB >> 4) : 0u), ql = q_lo + (uint32_t)x * (NH * SUB >> 4);
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < 4 * NH; ++kk) {
                                const uint32_t off16 = (uint32_t)(((kk >> 2) * SUB + (kk & 3) * 32) >> 4);
                                if (kk < ksteps_qk) mma_ss(tx, desc_join(ql + off16), desc_join(kl + off16), ID_QK, kk > 0);
                            }
                            mma_commit(bar(L::BAR_S + x));
                        }
                        __syncwarp();
                    }
                }
                if (j + 1 < n_tiles) {
                    if (elect_one()) mma_commit(bar(L::BAR_KE + sk));        // K(j+1) consumed
                    __syncwarp();
                }
            }
            if (elect_one()) mma_commit(bar(L::BAR_END));            // nothing in flight when the TMEM is given back
            __syncwarp();
            if (!wait(bar(L::BAR_END), 0, failed)) drain(bar(L::BAR_END), 0);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int x = warp >> 2, wq = warp & 3;
        const int tb = s_plan.t0[x], te = s_plan.t1[x], nrows = s_plan.rows[x];
        if (te > tb) {
            // ------------------------------------------ softmax of slot x
            const int row = wq * 32 + lane;                          // query row of the slot = TMEM lane
            const uint32_t lane_off = (uint32_t)(wq * 32) << 16;
            const uint32_t s_addr = tmem + lane_off + x * 128, o_addr = tmem + lane_off + 256 + x * 128;
            const int hh = group * hpc + (hpc == 2 ? x : 0);
            const RowRange mine = range_of(s_plan.span, s_plan.first_row[x] + min(row, nrows - 1), a.chunk, a.window);
            const int all_hi = s_plan.all_hi[x], all_low = s_plan.all_low[x], keep = s_plan.keep;
            const float sl2 = prm.scale_log2;
            const float cap2 = a.cap * LOG2E, cx = a.cap > 0.f ? a.scale / a.cap : 0.f, cap_e = a.cap > 0.f ? 2.f / a.cap : 0.f;
            const float cz = cx * cx, a1 = cz * (-1.f / 3.f), a2 = cz * cz * (2.f / 15.f), a3 = cz * cz * cz * (-17.f / 315.f);
            const float bias2 = KIND == KIND_SIGMOID && a.head_bias ? a.head_bias[hh] * LOG2E : 0.f;
            float m = a.sink > 0.f ? (a.sink_logits ? a.sink_logits[hh] : a.sink_logit) * LOG2E : -INFINITY, l = a.sink;
#pragma unroll 1
            for (int j = tb; j < te; ++j) {
                const int i = j - tb;
                wait(bar(L::BAR_S + x), i & 1, failed);
                tc_fence_after();
                uint32_t sr[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + c * 32, sr[c]);
                tmem_wait_ld();
                const int c0 = j * BN;
                const bool partial = c0 + BN - 1 > all_hi || c0 < all_low;
                float eff = sl2;                                     // the exponent of 2 is sr * eff
                float mp[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};     // short chains: one warp a scheduler and slot hides nothing
                auto reduce = [&]() {
                    return fmaxf(fmaxf(fmaxf(mp[0], mp[1]), fmaxf(mp[2], mp[3])), fmaxf(fmaxf(mp[4], mp[5]), fmaxf(mp[6], mp[7])));
                };
                bool small = false;
                uint32_t see[4] = {~0u, ~0u, ~0u, ~0u};
                if (KIND == KIND_CAPPED) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < 32; ++k) mp[k & 7] = fmaxf(mp[k & 7], fabsf(__uint_as_float(sr[c][k])));
                    const float am = reduce();
                    small = __all_sync(0xffffffffu, cx > 0.f && am * cx <= 0.1875f);
                    if (small) {
#pragma unroll
                        for (int c = 0; c < 4; ++c)
#pragma unroll
                            for (int k = 0; k < 32; k += 2) tanh_small_x2(sr[c][k], sr[c][k + 1], a1, a2, a3);
                    } else {                                         // any score, any scale: through TMEM, a rolled loop
                        eff = 1.f;
#pragma unroll 1
                        for (int c = 0; c < 4; ++c) {
                            uint32_t r[32];
                            tmem_ld32(s_addr + c * 32, r);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 32; ++k) {
                                float y = __uint_as_float(r[k]) * sl2;
                                if (a.cap > 0.f) y = cap_score(y, cap2, cap_e);
                                r[k] = __float_as_uint(y);
                            }
                            tmem_st32(s_addr + c * 32, r);
                        }
                        tmem_wait_st();
#pragma unroll
                        for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + c * 32, sr[c]);
                        tmem_wait_ld();
                    }
                }
                if (partial) {
                    const int hi = mine.hi + 1 - c0, low = mine.low - c0, k0 = mine.block - c0, k1 = keep - c0;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        see[c] = col_bits(low - c * 32, hi - c * 32) | col_bits(k0 - c * 32, min(k1, hi) - c * 32);
                        if (KIND != KIND_SIGMOID) {
#pragma unroll
                            for (int k = 0; k < 32; ++k)
                                if (!(see[c] >> k & 1)) sr[c][k] = 0xff800000u;          // -inf
                        }
                    }
                }
                if (KIND != KIND_SIGMOID) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) mp[k] = -INFINITY;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < 32; ++k) mp[k & 7] = fmaxf(mp[k & 7], __uint_as_float(sr[c][k]));
                    const float m_new = fmaxf(fmaxf(m, reduce() * eff), FLOOR), alpha = b2::fast_exp2(m - m_new);
                    l *= alpha;                                      // at first the sink's share, if any; exp2(-inf) = 0
                    if (i > 0) {
                        if (__any_sync(0xffffffffu, m_new > m)) {    // else every factor is one
                            wait(bar(L::BAR_PV + x), (i - 1) & 1, failed);
                            tc_fence_after();
#pragma unroll 1
                            for (int c = 0; c < 2 * DVH; ++c) {
                                uint32_t o[32];
                                tmem_ld32(o_addr + c * 32, o);
                                tmem_wait_ld();
#pragma unroll
                                for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                                tmem_st32(o_addr + c * 32, o);
                            }
                        }
                    }
                    m = m_new;
                }
                float sum[4] = {0.f, 0.f, 0.f, 0.f};                 // the denominator sums the fp32 weights
#pragma unroll
                for (int c = 0; c < 2; ++c) {                        // 64 keys -> 32 packed pairs
                    uint32_t pk[32];
#pragma unroll
                    for (int k = 0; k < 32; ++k) {
                        const int cc = 2 * c + (k >> 4), ii = (2 * k) & 31;
                        float w0, w1;
                        if (KIND == KIND_SIGMOID) {
                            fma_x2(w0, w1, __uint_as_float(sr[cc][ii]), __uint_as_float(sr[cc][ii + 1]), sl2, bias2);
                            w0 = sigmoid2_f(w0);
                            w1 = sigmoid2_f(w1);
                            w0 = see[cc] >> ii & 1 ? w0 : 0.f;
                            w1 = see[cc] >> (ii + 1) & 1 ? w1 : 0.f;
                        } else {
                            fma_x2(w0, w1, __uint_as_float(sr[cc][ii]), __uint_as_float(sr[cc][ii + 1]), eff, -m);
                            w0 = b2::fast_exp2(w0);
                            w1 = b2::fast_exp2(w1);
                            add_x2(sum[2 * (k & 1)], sum[2 * (k & 1) + 1], w0, w1);
                        }
                        pk[k] = b2::pack_bf16x2(w0, w1);
                    }
                    tmem_st32(s_addr + c * 32, pk);                  // P overwrites the first 64 columns of S_x
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) b2::mbar_arrive(bar((c == 0 ? L::BAR_P : L::BAR_P2) + x));     // the P V of 64 keys runs under the next 64
                }
                if (KIND != KIND_SIGMOID) l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            }
            // ------------------------------------------ output rows
            const int n = te - tb;
            const bool valid = row < nrows;
            const size_t brow = (size_t)row0 + (two_rows && x ? BM : 0) + row;
            wait(bar(L::BAR_PV + x), (n - 1) & 1, failed);
            float inv = KIND == KIND_SIGMOID ? 1.f : (l > 0.f ? 1.f / l : 0.f);
            if (*failed) inv = __int_as_float(0x7fc00000);           // behind the last wait, which may be the one that gave up
            if (TWO_MAPS && x == 1) {                                // slot 0 writes: it reads both outputs from its own TMEM lane
                s_inv[TWO_MAPS ? row : 0] = inv;
                tc_fence_after();
                tc_fence_before();
                asm volatile("bar.arrive 1, 256;" ::: "memory");
            } else {
                if (TWO_MAPS) asm volatile("bar.sync 1, 256;" ::: "memory");
                tc_fence_after();
                const float inv2 = TWO_MAPS ? -a.map_lambda * s_inv[TWO_MAPS ? row : 0] : 0.f;
                const bf16* gp = static_cast<const bf16*>(a.gate);
                bf16* orow = static_cast<bf16*>(a.out) + brow * a.out_stride + (size_t)hh * a.dv;
                float f = inv, f2 = inv2;
                if (TWO_MAPS) {                                      // the difference's own norm
                    float ss = 0.f;
#pragma unroll 1
                    for (int c = 0; c < 2 * DVH; ++c) {
                        if (c * 32 < a.dv) {
                            uint32_t o[32], o2[32];
                            tmem_ld32(o_addr + c * 32, o);
                            tmem_ld32(o_addr + 128 + c * 32, o2);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 32; ++k) {
                                const float d = fmaf(__uint_as_float(o2[k]), inv2, __uint_as_float(o[k]) * inv);
                                if (c * 32 + k < a.dv) ss = fmaf(d, d, ss);
                            }
                        }
                    }
                    const float r = rsqrtf(ss / (float)a.dv + a.map_eps) * a.map_scale;
                    f *= r;
                    f2 *= r;
                }
                if (gp && !a.gate_channels && valid) {
                    const float z = b2::sigmoid_f(__bfloat162float(gp[brow * a.gate_stride + hh]));
                    f *= z;
                    f2 *= z;
                }
#pragma unroll 1
                for (int c = 0; c < 2 * DVH; ++c) {
                    if (c * 32 < a.dv) {                             // uniform
                        uint32_t o[32], o2[TWO_MAPS ? 32 : 1];
                        tmem_ld32(o_addr + c * 32, o);
                        if constexpr (TWO_MAPS) tmem_ld32(o_addr + 128 + c * 32, o2);
                        tmem_wait_ld();
                        if (valid) {
                            float r[32];
#pragma unroll
                            for (int k = 0; k < 32; ++k) {
                                r[k] = __uint_as_float(o[k]) * f;
                                if (TWO_MAPS) r[k] = fmaf(__uint_as_float(o2[TWO_MAPS ? k : 0]), f2, r[k]);
                            }
                            if (GATHERED && gp && a.gate_channels) {
                                const bf16* g = gp + brow * a.gate_stride + (size_t)hh * a.dv + c * 32;
#pragma unroll
                                for (int k = 0; k < 32; k += 2) {
                                    if (c * 32 + k < a.dv) {
                                        const uint32_t z = *reinterpret_cast<const uint32_t*>(g + k);
                                        r[k] *= b2::sigmoid_as<bf16>(__uint_as_float(z << 16));
                                        r[k + 1] *= b2::sigmoid_as<bf16>(__uint_as_float(z & 0xffff0000u));
                                    }
                                }
                            }
#pragma unroll
                            for (int k = 0; k < 32; k += 8) {
                                if (c * 32 + k < a.dv) {
                                    uint4 v;
                                    v.x = b2::pack_bf16x2(r[k], r[k + 1]);
                                    v.y = b2::pack_bf16x2(r[k + 2], r[k + 3]);
                                    v.z = b2::pack_bf16x2(r[k + 4], r[k + 5]);
                                    v.w = b2::pack_bf16x2(r[k + 6], r[k + 7]);
                                    *reinterpret_cast<uint4*>(orow + c * 32 + k) = v;
                                }
                            }
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
    if (GATHERED && *failed && lane == 0 && (warp == 8 || warp == 10)) {     // boxes that nobody has waited for: every role is done now
        const int nst = warp == 10 ? L::VST : L::KST;                // (a tile that was never begun takes the whole millisecond, which is as good)
        for (int it = max(0, n_tiles - nst); it < n_tiles; ++it) drain(bar((warp == 10 ? L::BAR_V : L::BAR_K) + it % nst), (it / nst) & 1);
    }
}

template <int NH, int DVH, int KIND, bool TWO_MAPS, bool GATHERED>
int launch(const Params& p, dim3 grid, cudaStream_t st) {
    auto kern = prompt_tc5_kernel<NH, DVH, KIND, TWO_MAPS, GATHERED, false>;
    int smem = Shape<NH, DVH, TWO_MAPS, false>::SMEM;
    if constexpr (!TWO_MAPS)
        if (p.rows_per_cta > BM || p.heads_per_cta > 1) {
            kern = prompt_tc5_kernel<NH, DVH, KIND, TWO_MAPS, GATHERED, true>;
            smem = Shape<NH, DVH, TWO_MAPS, true>::SMEM;
        }
    B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kern<<<grid, NTHREADS, smem, st>>>(p);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

// A tile a CTA, of one slot, of two heads of a kv head or of two row tiles; or CTAs that take tiles in turns (prompt_turns_tc5.cu), whose first
// scores come 1.3 us later.  Times below: in a graph, this kernel / turns.
enum Form { ONE_SLOT, HEAD_PAIRS, ROW_PAIRS, TURNS };

int64_t longs_of(const b2_prompt_args& a) { return std::min(a.n_seq, a.T / a.min_rows); }      // most sequences of min_rows rows or more

Form form_of(const b2_prompt_args& a) {
    const int64_t n_sm = b2_sm_count(), longs = longs_of(a);
    if (longs == 0) return ONE_SLOT;
    // One slot to one and a half waves: 300 rows x 16 heads 15.0 / 15.4 us, 1000 x 16 22.2 / 23.6, 1200 gathered x 16 40.7 / 41.8, 1300 x 16 (176 tiles)
    // 27.4 / 27.1, 4 x 146 x 32 (256) 26.6 / 25.2.  The count is a bound: every sequence may begin a tile more.
    int64_t tiles = (int64_t)a.T / BM + longs;
    // Where most sequences must be decode rows it is far too large: if those of one or two portions are one wave, capped scores and two maps, whose
    // start in turns is the longer one, stay here.  64 decode rows and a prompt of 200, with the decode kernel: 16 heads, capped 61.2 / 70.4, two maps
    // 63.7 / 68.2, but ten prompts of 20 x 32 heads, capped, 83.4 / 81.3; other weights 73.1 / 73.6 and 81.6 / 77.4 (32 heads).
    const bool rows_of_few = a.T < (int64_t)a.min_rows * a.n_seq;
    if (rows_of_few && (a.cap > 0.f || a.maps == 2) && ((a.T - a.n_seq) / BM + 2) * a.H <= n_sm) return ONE_SLOT;
    // Tiles of two rows, where they are the form in turns too, leave fewer tiles: 85 + 58 + 83 + 148 gathered rows behind 555 x 32, 128 CTAs of two and
    // 160 of one, 18.7 against 26.4.
    const bool row_pairs = a.maps == 1 && (a.cu_k || (a.H / a.G) % 2) && ((int64_t)a.T / (2 * BM) + longs) * a.H >= n_sm;
    if (tiles * a.H <= n_sm * 3 / 2) return row_pairs ? ROW_PAIRS : ONE_SLOT;
    // One causal portion without context is as long as its longest tile, which turns do not shorten.  One slot: 1792 gathered rows x 16 heads (224
    // tiles) 32.4 / 34.1 us, 1800 x 16 (240) 36.3 / 34.9, 871 x 32 (224) 23.8 / 22.1; past 16 steps 3584 x 8 (224) 56.6 / 59.0, 4000 x 8 (256) 62.6 /
    // 65.0.  Two row tiles past 16 steps: 2400 x 16 (160 CTAs) 46.2 / 47.4, 3584 x 16 (224) 66.0 / 68.4, 4000 x 16 (256) 76.6 / 75.8, 1792 x 32 (14
    // steps, 224) 41.2 / 39.3; 2000 x 16, which would leave SMs without a CTA, 42.5 / 38.1.
    if (a.cu_k && a.n_seq == 1 && a.window == 0 && a.k_rows == a.T) {
        const int64_t one = ((int64_t)a.T + BM - 1) / BM * a.H, two = ((int64_t)a.T + 2 * BM - 1) / (2 * BM) * a.H;
        const bool longer = a.T > 16 * BM;
        if (longer ? one * 4 <= n_sm * 7 : a.T > 12 * BM && one * 5 <= n_sm * 8) return ONE_SLOT;
        if (longer && two >= n_sm && two * 5 <= n_sm * 8) return ROW_PAIRS;
    }
    if (a.cu_k || a.maps == 2 || rows_of_few) return TURNS;
    const bool heads = (a.H / a.G) % 2 == 0;
    // Capped scores of which a mask cuts most key tiles, up to two waves: such a step takes 6k cycles in turns.  Windows of 150: 4096 rows x 16 heads on 4
    // kv heads 37.2 / 40.6, 16 on 16 40.7 / 44.1, 8 on 8 25.9 / 32.4, 2000 x 16 20.4 / 24.1; of 500: 50.7 / 52.4, 54.3 / 61.3, 34.7 / 41.9, 26.9 / 31.8;
    // of 1024 75.1 / 70.0, and of 500 in 3.4 waves (4096 x 32) 97.5 / 93.0; three waves of row tiles (600 + 417 + 591 + 1055 x 28) 54.3 / 59.3 but
    // 52.0 / 45.7 with windows of 150.  The tiles of 1.1 to 1.4 waves go either way (600 + 417 + 591 + 1055 x 16, 150, 500 and 850: 30.8 / 30.7, 35.4 /
    // 30.2, 36.2 / 37.4).
    const int reach = a.chunk > 0 && (a.window == 0 || a.chunk < a.window) ? a.chunk : a.window;
    if (a.cap > 0.f && reach > 0 && reach <= 7 * BN) {
        const Form form = heads ? HEAD_PAIRS : row_pairs ? ROW_PAIRS : ONE_SLOT;
        const int64_t ctas = form == ROW_PAIRS ? ((int64_t)a.T / (2 * BM) + longs) * a.H : (a.T + longs * (BM / 2)) * (heads ? a.H / 2 : a.H) / BM;
        return ctas <= (form == ROW_PAIRS && reach > 2 * BN ? 3 : 2) * n_sm ? form : TURNS;
    }
    // Two heads a CTA, if that is one wave with remainders of half a tile (the host does not have the lengths) and short: 8 x 200 rows x 16 heads
    // 13.7 / 15.4, 4 x 400 17.0 / 18.9, 2 x 900 (8 steps) 25.2 / 26.6, 1000 x 32 26.6 / 27.2.  Not at 9 steps (1750 x 16, window 1024, 30.2 / 29.6),
    // beyond one wave (4 x 600 x 16, 160 CTAs, 23.7 / 21.6; 830 + 577 + 817 x 16 in blocks of 510, 152 CTAs, 26.7 / 23.0), with capped scores
    // (1000 + 800 x 16 34.9 / 32.3) or heads of 96 (570 + 396 x 32, window 152, 19.8 / 18.9).  The ragged 187 + 750 + 187 + 375 x 16 take 22.7 in
    // either, and would take 20.0 in one slot each.
    // Not two row tiles: 66 + 101 + 257 + 94 + 97 + 30 + 32 + 137 gathered rows x 16 13.1 / 13.6, but 292 + 211 + 298 x 32 22.9 / 20.1.
    if (!heads || a.cap > 0.f || a.dk % 64) return TURNS;
    const int64_t pairs = (a.T + longs * (BM / 2)) * (a.H / 2) / BM;
    int64_t steps = ((int64_t)a.max_nb * a.bs + BN - 1) / BN;                 // of the longest tile, at most
    if (a.window > 0) steps = std::min<int64_t>(steps, (a.window + BM) / BN + 1);
    if (a.chunk > 0) steps = std::min<int64_t>(steps, a.chunk / BN + 2);
    return pairs <= n_sm && steps <= 8 ? HEAD_PAIRS : TURNS;
}

}  // namespace

bool b2_internal_prompt_tc5_ok(const b2_prompt_args& a) {
    if (a.dk <= 0 || a.dv <= 0 || a.dk % 16 || a.dv % 8 || a.dv > 128) return false;
    if (a.cu_k && !(a.scale > 0.f)) return false;
    if (a.maps == 2) return a.dk <= 64;              // two maps' keys of 128 leave no room for two stages
    return a.dk <= (a.cu_k ? 192 : 128);
}

int b2_internal_prompt_tc5(const b2_prompt_args& a, void* stream) {
    const Form form = form_of(a);
    if (form == TURNS) return b2_internal_prompt_turns(a, stream);
    Params p;
    p.rows_per_cta = form == ROW_PAIRS ? 2 * BM : BM;
    p.heads_per_cta = form == HEAD_PAIRS ? 2 : 1;
    const int64_t tiles = (int64_t)a.T / p.rows_per_cta + longs_of(a);       // upper bound on sum(ceil(len / rows)); spare CTAs leave at once
    if (tiles == 0) return B2_OK;
    const int64_t ctas = tiles * (a.H / p.heads_per_cta);
    B2_REQUIRE(ctas <= 0x7fffffff, B2_EUNSUPPORTED, "prompt attention: %lld row tiles exceed the grid", (long long)tiles);
    p.a = a;
    p.scale_log2 = a.scale * LOG2E;
    p.bs_shift = -1;
    for (int b = 0; b < 16; ++b)
        if (a.bs == 1 << b) p.bs_shift = b;
    const bool gathered = a.cu_k != nullptr;
    // Gathered rows are consecutive: a whole key tile is one TMA box a sub-tile (a lane issues five instructions where the gather
    // takes 112 warp-wide copies; with one stage of V the time of its copy is on every tile's path: 6.5k -> 3.3k cycles a tile).
    // The maps have no row limit -- a box is only taken where all its 128 rows are the sequence's.  A sub-tile must lie on one side
    // of dk0.
    p.tma = gathered && (a.dk0 % 64 == 0 || a.dk0 >= a.dk) && (a.k1_row * 2) % 16 == 0;
    if (p.tma) {
        const uint64_t many = 0x7fffffff;
        const int dr = a.dk - a.dk0;
        const uint32_t box3[3] = {64, 1, BN}, box2[2] = {64, BN};
        int rc = B2_OK;
        if (a.dk0 > 0) {
            const uint64_t dims[3] = {(uint64_t)a.dk0, (uint64_t)a.H, many}, st[2] = {(uint64_t)a.dk0 * 2, (uint64_t)a.H * a.dk0 * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_k0, a.k0, 3, dims, st, box3);
        }
        if (rc == B2_OK && dr > 0) {
            const uint64_t dims[2] = {(uint64_t)dr, many}, st[1] = {(uint64_t)a.k1_row * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_k1, a.k1, 2, dims, st, box2);
        }
        if (rc == B2_OK) {
            const uint64_t dims[3] = {(uint64_t)a.dv, (uint64_t)a.H, many}, st[2] = {(uint64_t)a.dv * 2, (uint64_t)a.H * a.dv * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_v, a.v, 3, dims, st, box3);
        }
        if (rc != B2_OK) return rc;
    }
    const dim3 grid((unsigned)ctas);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nh = (a.dk + 63) / 64, dvh = (a.dv + 63) / 64;
    const bool one_by_one = a.cap > 0.f || !(a.scale > 0.f);         // the capped form takes any score and any sign of the scale
#define B2_PT(NH, DVH, KIND, MAPS2, GATH) return launch<NH, DVH, KIND, MAPS2, GATH>(p, grid, st)
    if (gathered) {
        if (nh == 1) { if (dvh == 1) B2_PT(1, 1, KIND_SOFTMAX, false, true); B2_PT(1, 2, KIND_SOFTMAX, false, true); }
        if (nh == 2) { if (dvh == 1) B2_PT(2, 1, KIND_SOFTMAX, false, true); B2_PT(2, 2, KIND_SOFTMAX, false, true); }
        if (dvh == 1) B2_PT(3, 1, KIND_SOFTMAX, false, true);
        B2_PT(3, 2, KIND_SOFTMAX, false, true);
    }
    if (a.maps == 2) {
        if (one_by_one) { if (dvh == 1) B2_PT(1, 1, KIND_CAPPED, true, false); B2_PT(1, 2, KIND_CAPPED, true, false); }
        if (dvh == 1) B2_PT(1, 1, KIND_SOFTMAX, true, false);
        B2_PT(1, 2, KIND_SOFTMAX, true, false);
    }
#define B2_PK(KIND)                                                                                                         \
    do {                                                                                                                    \
        if (nh == 1) { if (dvh == 1) B2_PT(1, 1, KIND, false, false); B2_PT(1, 2, KIND, false, false); }                     \
        if (dvh == 1) B2_PT(2, 1, KIND, false, false);                                                                      \
        B2_PT(2, 2, KIND, false, false);                                                                                    \
    } while (0)
    if (a.sigmoid) B2_PK(KIND_SIGMOID);
    if (one_by_one) B2_PK(KIND_CAPPED);
    B2_PK(KIND_SOFTMAX);
#undef B2_PK
#undef B2_PT
}
