// prompt_turns_tc5.cu -- masked prompt attention where the tiles are more than the SMs: what prompt_tc5.cu computes, by CTAs that stay on their
// SM and take tiles in turns, so that one tile's start and end lie under the work of others, longest tiles first.
//
// A tile is two slots of 128 query rows.  The 16 warps:
//   0-3, 4-7   softmax of slot 0 / 1: a thread a row = TMEM lane
//   8-11       outputs: bring O to a new maximum while the softmax takes its weights, and write it out under the next tile's first steps
//   12         issues the MMAs          13, 14   copy K / V, 128 keys at a time          15   plans the next tile and copies its Q
// The slots are
//   two query heads of one kv head on the same rows   where a kv head serves an even number of heads: both see the same keys, a
//                                                     window of W keys costs W + 127 rounded up to tiles instead of W + 255
//   two row tiles of one head                         otherwise
//   the two maps of a head on the same rows           differential attention: slot x multiplies the keys of map x
//   one slot                                          where two would leave SMs idle
// Keys are walked in the compact order of TileSpan (kept first keys, then the union of the rows' windows), so a window costs no
// tiles between its parts.  K, V and Q come by TMA, a box a page or 128 gathered rows; where a page is no box, by 16-byte cp.async gathers
// with a page lookup per key row, in the 128-byte swizzle that the MMA descriptors name.  A mask is tested per score only in tiles that
// the slot's rows see in part.
// S = Q K^T and O += P V are tcgen05.mma 128x128x16 (bf16 -> fp32 in TMEM); P replaces S in TMEM and is the A operand of the second
// product.  The weights are taken against the row's maximum so far, as in prompt_tc5.cu and for its reason.
//
// Bound: tensor pipe (2 (dk + dv) flops per visible pair) and, for the exponentials, the XU pipe, 16 a clock and SM.  Where a whole warp's
// scores are below 3/16 of the cap, the cap is a Taylor polynomial (prompt_tc5.cu) in one pass with the exponent; it rises with the score, so a
// row's largest capped score is that of its largest score and needs no pass.
// Measured with clock64, 128 keys x two slots: 3.3 - 3.9k cycles with heads of 192 / 128 (softmax 0.5k for the maximum and 1.5 - 2k for the
// weights, then the P V of its last 64 keys and the next Q K^T one after another, 1.3k), 4.4k with capped scores.
// A CTA a tile needs 7.5 - 9k cycles to its first scores and 5k to write its rows, and takes tiles in the order of the rows: with 16 heads of
// 128 + 64 / 128 and 4096 ragged causal rows the SMs ended between 29 and 56 us.  Attention alone in a graph, a CTA a tile -> here: 4096 rows x 32
// heads of 128, window 1024, capped 122 -> 107 us, not capped 93.6 -> 77.2; those causal rows 52.8 -> 42.6; 4 x 625 rows x 16 heads of two maps 37.0 ->
// 30.2; 3500 gathered rows x 16 heads in windows of 300 39.0 -> 34.5; 1000 rows x 32 heads of sigmoid weights 30.8 -> 22.6.
// What is left of the first steps is fetching code, 9 - 12k cycles to the first scores: which launches are prompt_tc5.cu's, and why, stands there.
// The forms of two maps spill 12 - 60 bytes a thread, the others nothing.
// What cost most on the way: an MMA loop with the slot as a variable, whose operands are not uniform to the compiler (3.6k cycles between a
// softmax and the next instead of 1.3k); the weights in a rolled loop over 32 keys (2.3k cycles instead of 1.5k); stores by a thread a row
// (32 lines each) and gates per column in the same kernel (10k cycles a tile's output instead of 3k).
#include "prompt_tc5.cuh"

#include <algorithm>

namespace {

using namespace b2tc;
using namespace b2prompt;

constexpr int NTHREADS = 512;
constexpr int W_OUT = 8, W_MMA = 12, W_K = 13, W_V = 14, W_PLAN = 15;      // first warps of the roles; warps 0-7 are the softmax

// NH: 64-column sub-tiles of a slot's Q and K; DVH: of V.  Behind Q lies a ring of 16-KB units, filled in the order they are read:
// the K sub-tiles of a step (128 keys x 64 columns), then its V in halves (64 keys x all columns; of 64 columns both in one).
template <int NH, int DVH, bool TWO_MAPS>
struct Shape {
    static constexpr int Q_BYTES = 2 * NH * SUB, NK = TWO_MAPS ? 2 : NH, NS = NK + DVH;
    static constexpr int FIT = (232448 - 3072 - Q_BYTES) / SUB;      // 227 KB, the static part rounded up to the alignment of the ring
    static constexpr int UNITS = FIT < 3 * NS ? FIT : 3 * NS;        // never four steps ahead: a barrier a step of four
    static constexpr int BAR_Q = 0, BAR_QE = 2, BAR_PLAN = 4, BAR_PLANE = 6, BAR_K = 8, BAR_V = 12, BAR_KE = 16, BAR_VE = 20, BAR_S = 24, BAR_P = 26,
                         BAR_P2 = 28, BAR_PV = 30, BAR_A = 32, BAR_E = 34, BAR_END = 36, BARS = 37;
    static constexpr int SMEM = Q_BYTES + UNITS * SUB;
};

struct Params {
    b2_prompt_args a;
    int rows_per_cta, heads_per_cta;
    int bs_shift;                                    // log2 of the page size, or -1
    int align;                                       // the two parts of the keys begin on multiples of it (positions)
    int k_box, v_box;                                // log2 of the rows of a box
    float scale_log2;
    int tma, tma_q;                                  // K and V / Q come by TMA boxes
    CUtensorMap map_q0, map_q1, map_k0, map_k1, map_v;
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// y = s (e + z (a1 + z (a2 + z a3))) - m, z = s^2, on the packed pipe: the exponent e s tanh(x) / x - m of a score s = x / c, a_i = e t_i c^2i with
// the Taylor coefficients -1/3, 2/15, -17/315
__device__ __forceinline__ void tanh_small_exponent_x2(float& y0, float& y1, uint32_t s0, uint32_t s1, float e, float a1, float a2, float a3, float m) {
    asm("{\n\t.reg .b64 s, z, p, c0, c1, c2, c3, mm;\n\t"
        "mov.b64 s, {%2, %3};\n\tmov.b64 c0, {%4, %4};\n\tmov.b64 c1, {%5, %5};\n\tmov.b64 c2, {%6, %6};\n\tmov.b64 c3, {%7, %7};\n\t"
        "mov.b64 mm, {%8, %8};\n\tmul.rn.f32x2 z, s, s;\n\tfma.rn.f32x2 p, z, c3, c2;\n\tfma.rn.f32x2 p, z, p, c1;\n\t"
        "fma.rn.f32x2 p, z, p, c0;\n\tfma.rn.f32x2 s, s, p, mm;\n\tmov.b64 {%0, %1}, s;\n\t}"
        : "=f"(y0), "=f"(y1) : "r"(s0), "r"(s1), "f"(e), "f"(a1), "f"(a2), "f"(a3), "f"(-m));
}
// KeySpan with its parts widened to whole boxes: positions f0 .. f0 + nf - 1 (the kept first keys, nf may be 0), then w0 ..; compact
// indices in order.  What the widening adds, [0, z0) and [z1, z2), is hidden by the masks like any other key a row does not see.
struct TileSpan {
    int f0, nf, w0, n, z0, z1, z2;
    __device__ __forceinline__ int key(int c) const { return c < nf ? f0 + c : w0 + (c - nf); }
    // compact index of the first key at or behind position j
    __device__ __forceinline__ int index(int j) const { return j < w0 ? min(max(j - f0, 0), nf) : nf + (j - w0); }
};
__device__ __forceinline__ TileSpan tile_span(const KeySpan& k, int last, int align) {
    const int end = k.lo + k.nfirst, f1 = (end + align - 1) & -align;
    TileSpan s;
    s.f0 = k.lo & -align;
    s.w0 = k.wlo & -align;
    s.nf = 0;
    s.z1 = s.z2 = 0;
    if (k.nfirst == 0) {
        s.z0 = k.wlo - s.w0;
    } else {
        if (f1 < s.w0) s.nf = f1 - s.f0;
        else s.w0 = s.f0;                            // the parts meet
        s.z0 = k.lo - s.f0;
        s.z1 = end - s.f0;
        s.z2 = s.nf + k.wlo - s.w0;
    }
    s.n = s.nf + last - s.w0 + 1;
    return s;
}
// What the plan warp works out for one tile: two slots of rows of one (sequence, head group).
struct Plan {
    TileSpan span;
    int keep;                                        // compact index below which keys are kept for every row of their mask block
    int first_row[2], rows[2];                       // position of a slot's first row, number of rows
    int t0[2], t1[2];                                // a slot works on the key tiles t0 .. t1 - 1
    int all_hi[2], all_low[2];                       // keys all_low .. all_hi are visible to every row of the slot
    int n_tiles;                                     // key tiles of the slots together; 0: no more tiles for this CTA
    int seq, row0, head;                             // row0: first row in q and out; head: slot 0's
};

// The order of the tiles: by the number of key tiles they walk, most first, so that the CTAs, which take tiles in boustrophedon
// turns, end together.  No list is made: how many row tiles have at least L steps is a closed form per sequence, so the tile of a
// rank is a binary search over L.  The prompts lie in the lanes of the warp; more than 32 are taken in the order of the batch, which one walk
// through it gives: to search among 256 would take as long as a short tile.
struct Prompt {
    int seq, row, len, ctx;                          // first row in q, rows (0: not this kernel's), first position (< 0: padding)
};
// In mask blocks a tile's steps go up and down with its place in the block: then they are listed, for as many row tiles as the list holds (more
// average out).  In the order of their positions, which is none, two long tiles could meet in a CTA; order of positions -> list (a CTA a tile), heads
// of 128 behind 2000 keys: 666 + 1593 rows x 16, blocks of 1273, 49.4 -> 36.4 us (37.1); 3309 x 16, 1649, 52.8 -> 44.2 (45.0); 3860 x 16, 463, 33.4 -> 27.9
// (35.5); 298 + 891 x 32, 1946, 45.6 -> 28.7 (27.6); three long portions behind 0, blocks of 947, 29.3 -> 30.4 (33.0).
constexpr int LISTED = 256;
template <bool BLOCKS>
struct TileOrder {
    const b2_prompt_args* a;
    uint8_t* list;                                   // steps of the row tiles in the order of the batch (at most 255)
    int n_list, ahead;                               // row tiles listed (0: none are); of the prompts before this lane's
    int shift, cap;                                  // log2 of the rows per tile; windows and mask blocks: steps beyond which tiles cost the same
    int lane, n_long, max_level;
    int from, before;                                // more prompts than lanes: batch of 32 at which the search goes on, row tiles before it
    Prompt mine;                                     // this lane's, if all fit

    __device__ __forceinline__ int batches() const { return n_long <= 32 ? 1 : (a->n_seq + 31) / 32; }
    __device__ __forceinline__ Prompt read(int s) const {
        Prompt p = {s, 0, 0, 0};
        if (s < a->n_seq) {
            p.row = a->cu_q[s];
            p.len = a->cu_q[s + 1] - p.row;
            p.ctx = a->ctx_start[s];
            if (p.len < a->min_rows) p.len = 0;
        }
        return p;
    }
    __device__ __forceinline__ Prompt load(int b) const { return n_long <= 32 ? mine : read(b * 32 + lane); }
    // first of a prompt's row tiles that walks at least L key tiles (their number, if none does)
    __device__ __forceinline__ int first_at(int L, const Prompt& p) const {
        const int nt = (p.len + (1 << shift) - 1) >> shift, need = (L - 1) * BN + 1 - max(p.ctx, 0);
        if (L > cap || need > p.len) return nt;
        return min(max(((need + (1 << shift) - 1) >> shift) - 1, 0), max(nt - 1, 0));
    }
    __device__ __forceinline__ int total(int L) const {
        return __reduce_add_sync(0xffffffffu, ((mine.len + (1 << shift) - 1) >> shift) - first_at(L, mine));
    }
    // rows, heads: of a tile; both become those of one slot where the batch turns out to hold no more tiles of one slot than there are CTAs
    __device__ __forceinline__ void init(const b2_prompt_args& args, uint8_t* s_list, int& rows, int& heads, int ln) {
        a = &args;
        list = s_list;
        lane = ln;
        n_list = 0;
        n_long = 0;
        mine = {0, 0, 0, 0};
        int level = 1;
#pragma unroll 1
        for (int s0 = 0; s0 < a->n_seq && n_long <= 32; s0 += 32) {
            const Prompt p = read(s0 + lane);
            uint32_t longs = __ballot_sync(0xffffffffu, p.len > 0);
            if (p.len > 0) level = max(level, (max(p.ctx, 0) + p.len + BN - 1) / BN);
            if (a->n_seq <= 32) {
                mine = p;
                break;
            }
#pragma unroll 1
            while (longs && n_long <= 32) {
                const int who = __ffs(longs) - 1;
                const Prompt o = {s0 + who, __shfl_sync(0xffffffffu, p.row, who), __shfl_sync(0xffffffffu, p.len, who), __shfl_sync(0xffffffffu, p.ctx, who)};
                if (lane == n_long) mine = o;
                longs &= longs - 1;
                ++n_long;                            // 33: more than the lanes hold
            }
        }
        if (n_long <= 32 && __reduce_add_sync(0xffffffffu, (mine.len + BM - 1) / BM) * a->H <= (int)gridDim.x) {
            rows = BM;
            heads = 1;
        }
        shift = rows == BM ? 7 : 8;
        cap = 0x7fffff;
        if (a->window > 0) cap = min(cap, (a->window + rows) / BN + 1);
        if (a->chunk > 0) cap = min(cap, a->chunk / BN + 2);
        max_level = min(cap, (int)__reduce_max_sync(0xffffffffu, level));
        from = before = 0;
        if (n_long > 32) cap = max_level = 1;        // one level: in the order of the batch
        else if (total(1) * (a->H / heads) <= (int)gridDim.x) cap = max_level = 1;       // a tile a CTA in any order
        else if (BLOCKS && total(1) <= LISTED) make_list();
    }
    __device__ __forceinline__ int scan(int n) const {               // inclusive sum over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, n, d);
            if (lane >= d) n += below;
        }
        return n;
    }
    __device__ __forceinline__ void make_list() {
        const int nt = (mine.len + (1 << shift) - 1) >> shift, upto = scan(nt), prompts = 32 - __clz(__ballot_sync(0xffffffffu, nt > 0));
        ahead = upto - nt;
        n_list = __shfl_sync(0xffffffffu, upto, 31);
        max_level = min(max_level, 255);
#pragma unroll 1
        for (int u0 = 0; u0 < n_list; u0 += 32) {
            int k = 0, ctx = 0, len = 0;             // of the last prompt that begins at or before this lane's tile
#pragma unroll 1
            for (int s = 0; s < prompts; ++s) {
                const int b = __shfl_sync(0xffffffffu, ahead, s), c = __shfl_sync(0xffffffffu, mine.ctx, s), l = __shfl_sync(0xffffffffu, mine.len, s);
                if (u0 + lane >= b) { k = u0 + lane - b; ctx = max(c, 0); len = l; }
            }
            const int q0 = k << shift;
            if (u0 + lane < n_list) list[u0 + lane] = (uint8_t)min(max_level, ((ctx + q0) % a->chunk + min(len - q0, 1 << shift) + BN - 1) / BN);
        }
        __syncwarp();
    }
    __device__ __forceinline__ int listed(int L) const {             // row tiles of at least L steps
        int n = 0;
#pragma unroll 1
        for (int u = lane; u < n_list; u += 32) n += list[u] >= L;
        return __reduce_add_sync(0xffffffffu, n);
    }
    __device__ __forceinline__ bool find_listed(int r, Prompt& at, int& q0) const {
        if (r >= n_list) return false;
        int lo = 1, hi = max_level + 1;              // listed(lo) > r >= listed(hi) = 0
#pragma unroll 1
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (listed(mid) > r) lo = mid;
            else hi = mid;
        }
        r -= listed(lo + 1);
        int u = 0;
#pragma unroll 1
        for (;; u += 32) {
            const uint32_t bits = __ballot_sync(0xffffffffu, u + lane < n_list && list[u + lane] == lo);
            if (r < __popc(bits)) {
                u += __ffs(__ballot_sync(0xffffffffu, (bits >> lane & 1) && __popc(bits & ((1u << lane) - 1)) == r)) - 1;
                break;
            }
            r -= __popc(bits);
        }
        const int nt = (mine.len + (1 << shift) - 1) >> shift;
        const int who = __ffs(__ballot_sync(0xffffffffu, u >= ahead && u < ahead + nt)) - 1;
        at = {__shfl_sync(0xffffffffu, mine.seq, who), __shfl_sync(0xffffffffu, mine.row, who), __shfl_sync(0xffffffffu, mine.len, who),
              __shfl_sync(0xffffffffu, mine.ctx, who)};
        q0 = (u - __shfl_sync(0xffffffffu, ahead, who)) << shift;
        return true;
    }
    // row tile of rank r: its prompt and first row in it (false: there are no more)
    __device__ __forceinline__ bool find(int r, Prompt& at, int& q0) {
        if (BLOCKS && n_list > 0) return find_listed(r, at, q0);
        int lo = 1, hi = max_level + 1;              // total(lo) > r >= total(hi) = 0
        if (n_long <= 32) {
            if (r >= total(1)) return false;
#pragma unroll 1
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (total(mid) > r) lo = mid;
                else hi = mid;
            }
            r -= total(lo + 1);
        } else {
            r -= before;                             // a CTA's ranks rise
        }
#pragma unroll 1
        for (int b = from; b < batches(); ++b) {
            const Prompt p = load(b);
            const int first = first_at(lo, p), n = first_at(lo + 1, p) - first;
            const int upto = scan(n);
            const uint32_t hit = __ballot_sync(0xffffffffu, r < upto);
            if (hit) {
                const int who = __ffs(hit) - 1;
                at = {__shfl_sync(0xffffffffu, p.seq, who), __shfl_sync(0xffffffffu, p.row, who), __shfl_sync(0xffffffffu, p.len, who),
                      __shfl_sync(0xffffffffu, p.ctx, who)};
                q0 = __shfl_sync(0xffffffffu, first + r - (upto - n), who) << shift;
                return true;
            }
            const int all = __shfl_sync(0xffffffffu, upto, 31);
            r -= all;
            if (n_long > 32) {
                before += all;
                from = b + 1;
            }
        }
        return false;
    }
};
// the t-th tile of this CTA: forwards and backwards through the CTAs in turn
__device__ __forceinline__ uint32_t tile_rank(uint32_t t) {
    return t * gridDim.x + (t & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}

// Four column groups of a row, a pair of entries in each of the quad's lanes (tcgen05.ld 16x256b) -> lane q holds group q whole.
__device__ __forceinline__ uint4 quad_transpose(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, int lane) {
    const bool odd = lane & 1, up = lane & 2;
    const uint32_t a = __shfl_xor_sync(0xffffffffu, odd ? w0 : w1, 1), b = __shfl_xor_sync(0xffffffffu, odd ? w2 : w3, 1);
    if (odd) { w0 = a; w2 = b; }
    else { w1 = a; w3 = b; }
    const uint32_t c = __shfl_xor_sync(0xffffffffu, up ? w0 : w2, 2), d = __shfl_xor_sync(0xffffffffu, up ? w1 : w3, 2);
    return up ? make_uint4(c, d, w2, w3) : make_uint4(w0, w1, c, d);
}
// 16 TMEM lanes x 32 columns: register 4 i + e of lane l is column 8 i + 2 (l % 4) + e % 2 of TMEM lane l / 4 + 8 (e / 2)
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}

// 32 TMEM lanes x 16 columns, a thread a lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                   "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}

template <int NH, int DVH, int KIND, bool TWO_MAPS, bool GATHERED, bool GATE_COLUMNS, bool BLOCKS>
__global__ void __launch_bounds__(NTHREADS, 1)
prompt_turns_kernel(const __grid_constant__ Params prm) {
    using L = Shape<NH, DVH, TWO_MAPS>;
    using bf16 = __nv_bfloat16;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ uint64_t s_bars[L::BARS];
    __shared__ Plan s_plan[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    __shared__ uint8_t s_list[BLOCKS ? LISTED : 1];
    __shared__ float s_alpha[2][BM], s_inv[2][BM];                   // softmax -> output warps: factor of O, 1 / denominator
    const b2_prompt_args& a = prm.a;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);          // warp-uniform for the compiler too
    const uint32_t q_smem = b2::smem_u32(smem_raw);
    const uint32_t ring = q_smem + L::Q_BYTES, bars = b2::smem_u32(s_bars);
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile int* failed = &s_failed;

    if (tid == 0) {
        s_failed = 0;
        for (int s = 0; s < 2; ++s) { b2::mbar_init(bar(L::BAR_PLAN + s), 1); b2::mbar_init(bar(L::BAR_PLANE + s), 15); }   // every warp but the plan's reads it
        for (int s = 0; s < 16; ++s) b2::mbar_init(bar(L::BAR_K + s), 1);    // K, V full and taken, four steps each
        for (int x = 0; x < 2; ++x) {
            b2::mbar_init(bar(L::BAR_Q + x), 1);
            b2::mbar_init(bar(L::BAR_QE + x), 1);
            b2::mbar_init(bar(L::BAR_S + x), 1);
            b2::mbar_init(bar(L::BAR_P + x), 8);                     // softmax warps: keys 0-63 of P are in TMEM; output warps: O is at this step's maximum
            b2::mbar_init(bar(L::BAR_P2 + x), 4);                    // keys 64-127
            b2::mbar_init(bar(L::BAR_PV + x), 1);
            b2::mbar_init(bar(L::BAR_A + x), 4);                     // s_alpha of a step behind the tile's first
            b2::mbar_init(bar(L::BAR_E + x), 4);                     // s_inv of a tile
        }
        b2::mbar_init(bar(L::BAR_END), 1);
        b2::fence_mbar_init();
    }
    if (warp == W_MMA) {                                             // all 512 columns: one CTA per SM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(b2::smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    TileOrder<BLOCKS> order;
    // The plan warp comes to this barrier with its first plan in hand, made while the others set up what it does not need.
    auto meet = [] { asm volatile("bar.sync 2, 512;" ::: "memory"); };
    static_assert(NTHREADS == 512, "the barrier's threads");
    if (warp != W_PLAN) {
        tc_fence_before();
        meet();
        tc_fence_after();
    }
    const uint32_t tmem = warp != W_PLAN ? s_tmem : 0u;
    int sent0 = 0, sent1 = 0;                                        // Q tiles of the slots that the plan warp has asked for; key tiles of a copying warp
    const bool two_rows = prm.rows_per_cta > BM, two_heads = prm.heads_per_cta == 2;     // slot 1's rows or head, where it is not empty
    // the plan of tile t: its place, which stays the tile's until every warp has said that it is done with it
    auto plan_of = [&](int t) -> const Plan* {
        const bool ok = wait(bar(L::BAR_PLAN + (t & 1)), (t >> 1) & 1, failed);
        return __all_sync(0xffffffffu, ok) && s_plan[t & 1].n_tiles > 0 ? &s_plan[t & 1] : nullptr;
    };
    auto plan_done = [&](int t) {
        __syncwarp();
        if (lane == 0) b2::mbar_arrive(bar(L::BAR_PLANE + (t & 1)));
    };

    if (warp >= W_MMA) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        const int c8 = lane & 7, rsub = lane >> 3;
        // row r = 4 group + rsub: the swizzled column of even and odd groups; a group is 512 bytes
        const uint32_t sw_even = (uint32_t)(rsub * 128 + ((c8 ^ rsub) << 4)), sw_odd = (uint32_t)(rsub * 128 + ((c8 ^ (4 + rsub)) << 4));
        if (warp == W_PLAN) {
            // ------------------------------------------ plans, one tile ahead of their use, and Q
            if (prm.tma_q && lane == 0) {
                if (!GATHERED || a.dk0 > 0) b2::tma_prefetch_desc(&prm.map_q0);
                if (GATHERED && a.dk0 < a.dk) b2::tma_prefetch_desc(&prm.map_q1);
            }
            int tile_rows = prm.rows_per_cta, hpc = prm.heads_per_cta;
            order.init(a, s_list, tile_rows, hpc, lane);
            const uint32_t groups = (uint32_t)(a.H / hpc);
            int t = 0;                                               // tiles published
#pragma unroll 1
            for (uint32_t turn = 0;; ++turn) {
                const uint32_t rank = tile_rank(turn);
                const int head = (int)(rank % groups) * hpc;
                Prompt at = {0, 0, 0, 0};
                int q0 = 0;
                const bool more = order.find((int)(rank / groups), at, q0);
                const int seq = at.seq, len = at.len, ctx = at.ctx, row0 = at.row + q0;
                if (more && ctx < 0) {                               // padding: zero rows (the paged form's are another kernel's)
                    const int rows = GATHERED ? min(len - q0, tile_rows) : 0, v8 = a.dv / 8;
#pragma unroll 1
                    for (int idx = lane; idx < rows * v8; idx += 32)
                        *reinterpret_cast<uint4*>(static_cast<bf16*>(a.out) + (size_t)(row0 + idx / v8) * a.out_stride + (size_t)head * a.dv + (idx % v8) * 8) =
                            make_uint4(0, 0, 0, 0);
                    continue;
                }
                const int nrows0 = min(BM, len - q0), nrows1 = tile_rows > BM ? min(BM, max(0, len - q0 - BM)) : (TWO_MAPS || hpc == 2) ? nrows0 : 0;
                auto q_boxes = [&](int x) {                          // rows behind the tile are the next ones' (zeros behind the last): their results go nowhere
                    if (lane == 0) {
                        const int hh = head + (two_heads ? x : 0), rb = row0 + (two_rows && x ? BM : 0);
                        b2::mbar_arrive_expect_tx(bar(L::BAR_Q + x), NH * SUB);
#pragma unroll 1
                        for (int h = 0; h < NH; ++h) {
                            const uint32_t dst = q_smem + (x * NH + h) * SUB;
                            if (GATHERED && h * 64 >= a.dk0) tma_load_4d(dst, &prm.map_q1, bar(L::BAR_Q + x), h * 64 - a.dk0, 0, hh, rb);
                            else tma_load_4d(dst, &prm.map_q0, bar(L::BAR_Q + x), h * 64, TWO_MAPS ? x : 0, hh, rb);
                        }
                    }
                    __syncwarp();
                };
                if (t >= 2 && !__all_sync(0xffffffffu, wait(bar(L::BAR_PLANE + (t & 1)), ((t >> 1) & 1) ^ 1, failed))) break;
                Plan& pl = s_plan[t & 1];
                int tiles = 0;
                if (lane < 2 && more) {                              // a lane a slot
                    const int x = lane, rows = x ? nrows1 : nrows0;
                    const int p0 = ctx + q0, p_last = p0 + min(len - q0, tile_rows) - 1;
                    KeySpan keys = key_span(p0, p_last, a.chunk, a.window, a.keep_first);
                    if (GATHERED && keys.wlo < a.k_lo[seq]) keys.wlo = keys.lo = a.k_lo[seq];     // the gathered rows begin at k_lo
                    const TileSpan span = tile_span(keys, p_last, prm.align);
                    const int kept = a.window > 0 ? span.index(a.keep_first) : 0;
                    pl.rows[x] = rows;
                    pl.t0[x] = pl.t1[x] = 0;
                    if (rows > 0) {
                        const int pf = p0 + (two_rows && x ? BM : 0);
                        const RowRange f = range_of(span, pf, a.chunk, a.window), l = range_of(span, pf + rows - 1, a.chunk, a.window);
                        pl.first_row[x] = pf;
                        pl.t0[x] = (f.block < kept ? f.block : f.low) / BN;
                        pl.t1[x] = tiles = l.hi / BN + 1;
                        pl.all_hi[x] = f.hi;
                        pl.all_low[x] = l.low;
                    }
                    if (x == 0) {
                        pl.span = span;
                        pl.keep = kept;
                        pl.seq = seq;
                        pl.row0 = row0;
                        pl.head = head;
                    }
                }
                tiles = max(tiles, __shfl_sync(0xffffffffu, tiles, 1));
                if (t == 0) meet();
                __syncwarp();                                        // lane 0's word covers what lane 1 wrote: a shuffle orders no memory
                if (lane == 0) {
                    pl.n_tiles = tiles;
                    b2::mbar_arrive(bar(L::BAR_PLAN + (t & 1)));
                }
                if (!more) break;
                // Q, when the last product with the tile before it has been taken
                bool ok = true;
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    if ((x ? nrows1 : nrows0) == 0) continue;
                    ok = __all_sync(0xffffffffu, wait(bar(L::BAR_QE + x), ((x ? sent1 : sent0) & 1) ^ 1, failed));
                    if (!ok) break;
                    if (x) ++sent1;
                    else ++sent0;
                    if (prm.tma_q) {
                        q_boxes(x);
                        continue;
                    }
                    {                                                // rows past the tile are zeros
                        const int hh = head + (two_heads ? x : 0), nrows = x ? nrows1 : nrows0;
                        const int rbase = row0 + (two_rows && x ? BM : 0);
                        const int col0 = TWO_MAPS ? x * a.dk : 0;
                        const char* qh = reinterpret_cast<const char*>(static_cast<const bf16*>(a.q0) + (size_t)rbase * a.q0_row + (size_t)hh * a.q0_head + col0 + c8 * 8);
                        const char* q1 = GATHERED ? reinterpret_cast<const char*>(static_cast<const bf16*>(a.q1) + (size_t)rbase * a.q1_row + (size_t)hh * a.q1_head + c8 * 8) - 2 * a.dk0 : qh;
#pragma unroll 1
                        for (int rg = 0; rg < BM / 4; ++rg) {
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
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    b2::fence_proxy_async();                         // this thread's copies, before the MMAs that read them
                    __syncwarp();
                    if (lane == 0) b2::mbar_arrive(bar(L::BAR_Q + x));
                }
                if (!ok) break;
                ++t;
            }
        } else if (warp != W_MMA) {
            // ------------------------------------------ copies: K tiles / V tiles, on through all tiles of the CTA
            // By TMA, a box a page and 64 columns (gathered rows: 128 rows), a lane each.  Forms without boxes -- pages that do not lie on a
            // tile's eight-row groups, gathered rows at an end that the host does not know -- are cp.async gathers: eight lanes copy the 128 bytes of a row
            // and sub-tile, four rows (a group) an instruction, the pool rows of a tile's 128 keys (four a lane) looked up before the
            // stage is free: a lookup in front of its copies would put its latency on the path of every tile.
            const bool is_v = warp == W_V;
            const int n_sub = is_v ? DVH : L::NK, width = is_v ? a.dv : a.dk, split = GATHERED && !is_v ? a.dk0 : width;
            const uint32_t ld = 2u * (uint32_t)(GATHERED ? a.H * split : width), ld1 = 2u * (uint32_t)a.k1_row;    // bytes between pool rows
            const char* p1 = GATHERED && !is_v ? reinterpret_cast<const char*>(static_cast<const bf16*>(a.k1) + c8 * 8) - 2 * split : nullptr;
            const uint32_t map2 = 2u * (uint32_t)a.bs * (uint32_t)a.dk;                  // the second map's rows lie a page of the first behind
            constexpr uint32_t NONE = 0xffffffffu;
            const uint32_t heads = (uint32_t)(TWO_MAPS && !is_v ? 2 * a.G : a.G);
            const int box_shift = is_v ? prm.v_box : prm.k_box, n_box = (BN >> box_shift) * n_sub;     // boxes of a tile, their rows (log2)
            if (prm.tma && lane == 0) {
                if (is_v) b2::tma_prefetch_desc(&prm.map_v);
                else if (!GATHERED || a.dk0 > 0) b2::tma_prefetch_desc(&prm.map_k0);
                if (GATHERED && !is_v && a.dk0 < a.dk) b2::tma_prefetch_desc(&prm.map_k1);
            }
            int& g = sent0;                                          // key tiles of this CTA so far
            int unit = is_v ? L::NK : 0;                             // first of this one's units
            bool going = true;
            // A box of gathered rows must not read behind the last one, which the device knows (cu_k[n_seq]) whatever the host was told: where both
            // agree the maps end there and zeros come behind, else the box has to end before either.
            int box_end = -1;
            if (GATHERED && prm.tma) {
                const int last = a.cu_k[a.n_seq];
                if (a.k_rows != last) box_end = a.k_rows > 0 && a.k_rows < last ? (int)a.k_rows : last;
            }
#pragma unroll 1
            for (int t = 0; going; ++t) {
                const Plan* pl = plan_of(t);
                if (!pl) break;
                const TileSpan span = pl->span;
                const int n_tiles = pl->n_tiles, n_keys = span.n, seq = pl->seq, head = pl->head;
                plan_done(t);
                const int kvh = head / (a.H / a.G);                  // kv head of the paged pools
                const int32_t* bt = GATHERED ? nullptr : a.block_tables + (int64_t)seq * a.max_nb;
                const uint32_t g0 = GATHERED ? (uint32_t)a.cu_k[seq] - (uint32_t)a.k_lo[seq] : 0u;
                const uint32_t head0 = (uint32_t)(TWO_MAPS && !is_v ? 2 * kvh : kvh);
                const char* p0 = reinterpret_cast<const char*>(static_cast<const bf16*>(is_v ? a.v : a.k0) + (GATHERED ? (size_t)head * split : 0) + c8 * 8);
                const char* p1g = GATHERED && !is_v ? p1 : p0;
                const int in_boxes = !prm.tma ? 0 : GATHERED && box_end >= 0 ? (box_end - (int)g0 - span.w0) / BN : n_tiles;     // the first key tiles
                uint32_t rows[4];
                auto lookup = [&](int it) {
                    if (!GATHERED && prm.tma) {                      // rows[0], rows[1]: page of this lane's box, row in it
                        const int c = it * BN + ((lane % (BN >> box_shift)) << box_shift);
                        rows[0] = NONE;
                        if (c < n_keys) {
                            const int j = span.key(c), pg = j >> prm.bs_shift;
                            rows[0] = (uint32_t)bt[pg];
                            rows[1] = (uint32_t)(j - (pg << prm.bs_shift));
                        }
                        return;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {                    // pool rows (of this head) of keys it * 128 + lane + 32 q
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
                lookup(0);
#pragma unroll 1
                for (int it = 0; it < n_tiles; ++it, ++g, unit = (unit + L::NS) % L::UNITS) {
                    // what lay in the last of these units a lap ago has been taken (units are given back in the order of the ring)
                    const int lap = g * L::NS + (is_v ? L::NS : L::NK) - 1 - L::UNITS, before = lap / L::NS;
                    const int taken = lap % L::NS < L::NK ? L::BAR_KE : L::BAR_VE;
                    if (lap >= 0 && !__all_sync(0xffffffffu, wait(bar(taken + (before & 3)), (before >> 2) & 1, failed))) {
                        going = false;
                        break;
                    }
                    const uint32_t full = bar((is_v ? L::BAR_V : L::BAR_K) + (g & 3));
                    const int left = n_keys - it * BN;
                    // sub-tile h of rows r ..: K sub-tiles are a unit each; V lies in halves of 64 keys, each with its columns side by side
                    auto place = [&](int h, int r) {
                        if (!is_v) return ring + (uint32_t)((unit + h) % L::UNITS) * SUB + (uint32_t)r * 128;
                        const int half = r >> 6;
                        return (DVH == 2 ? ring + (uint32_t)((unit + half) % L::UNITS) * SUB : ring + (uint32_t)unit * SUB + half * (SUB / 2)) +
                               h * (SUB / 2) + (uint32_t)(r & 63) * 128;
                    };
                    if (it < in_boxes) {
                        // columns past the head are zero-filled and count; so do rows past the last one of a gathered buffer
                        const int there = GATHERED ? BN >> box_shift : min(BN >> box_shift, (left + (1 << box_shift) - 1) >> box_shift);
                        if (lane == 0) b2::mbar_arrive_expect_tx(full, (uint32_t)(there * n_sub) << (box_shift + 7));
                        __syncwarp();
#pragma unroll 1
                        for (int b = lane; b < n_box; b += 32) {     // 32 lanes: a multiple of the boxes across, or all boxes
                            const int i = b % (BN >> box_shift), h = b / (BN >> box_shift), r = i << box_shift;
                            if (i >= there) continue;
                            const uint32_t dst = place(h, r);
                            if (GATHERED) {
                                const int row = (int)g0 + span.key(it * BN + r);
                                if (!is_v && h * 64 >= split) tma_load_2d(dst, &prm.map_k1, full, h * 64 - split, row);
                                else tma_load_3d(dst, is_v ? &prm.map_v : &prm.map_k0, full, h * 64, head, row);
                            } else {
                                const bool second = TWO_MAPS && !is_v;
                                tma_load_4d(dst, is_v ? &prm.map_v : &prm.map_k0, full, second ? 0 : h * 64, (int)rows[1], (int)head0 + (second ? h : 0), (int)rows[0]);
                            }
                        }
                        __syncwarp();
                        lookup(it + 1);
                        continue;
                    }
#pragma unroll 1
                    for (int q = 0; q < 8; ++q) {                    // four groups each
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int gr = q * 4 + u;
                            const uint32_t pr = __shfl_sync(0xffffffffu, rows[0], (gr & 7) * 4 + rsub);
                            const bool there = pr != NONE;           // rows past the keys are zeros: 0 * NaN must not reach an accumulator
                            const char* src = p0 + (size_t)pr * ld;
                            const char* src1 = GATHERED ? p1g + (size_t)pr * ld1 : nullptr;
#pragma unroll
                            for (int h = 0; h < (L::NK > DVH ? L::NK : DVH); ++h) {
                                if (h < n_sub) {                     // warp-uniform
                                    const int col = (TWO_MAPS && !is_v ? 0 : h * 64) + c8 * 8;
                                    const char* sp = src + (TWO_MAPS && !is_v ? h * map2 : h * 128u);
                                    if (GATHERED) sp = col >= split ? src1 + h * 128 : sp;
                                    const bool ok = there && col < width;
                                    cp_async16(place(h, gr * 4) + (gr & 1 ? sw_odd : sw_even), ok ? sp : p0, ok);
                                }
                            }
                        }
                        if (q & 1) {
                            rows[0] = rows[1];
                            rows[1] = rows[2];
                            rows[2] = rows[3];
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    lookup(it + 1);
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    b2::fence_proxy_async();                         // this thread's copies, before the MMAs that read them
                    __syncwarp();
                    if (lane == 0) b2::mbar_arrive(full);
                }
            }
        } else {
            // ------------------------------------------ MMA issuer: the whole warp, warp-uniform operands, one elected lane
            // A turn is P_0 V, Q_0 K', P_1 V, Q_1 K': the outputs of a step and the scores of the next one -- of the next tile's first,
            // behind a tile's last -- so that the softmax of one slot runs under the MMAs of the other.
            constexpr uint32_t ID_QK = idesc_bf16(128, 128, 0), ID_PV = idesc_bf16(128, 64 * DVH, 1);
            const uint32_t q_lo = desc_lo(q_smem, 16), ring_k = desc_lo(ring, 16), ring_v = desc_lo(ring, SUB / 2);
            const int ksteps_qk = a.dk >> 4;
            auto uwait = [&](int b, int parity) { __all_sync(0xffffffffu, wait(bar(b), parity, failed)); };
            // rows r0 .. r1 - 1 of the V tile are not keys of this CTA's: zeros, since 0 * NaN must not reach an accumulator
            auto zero_rows = [&](int unit, int r0, int r1) {
#pragma unroll 1
                for (int i = r0 * 8 * DVH + lane; i < r1 * 8 * DVH; i += 32) {
                    const int r = i / (8 * DVH), h = i / 8 % DVH, half = r >> 6;
                    const uint32_t at = (DVH == 2 ? ring + (uint32_t)((unit + half) % L::UNITS) * SUB : ring + (uint32_t)unit * SUB + half * (SUB / 2)) +
                                        h * (SUB / 2) + (uint32_t)(r & 63) * 128 + (uint32_t)(i & 7) * 16;
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(0) : "memory");
                }
                b2::fence_proxy_async();
                __syncwarp();
            };
            auto commit = [&](int b) {
                if (elect_one()) mma_commit(bar(b));
                __syncwarp();
            };
            int t = 0, g = 0, unit = 0;                              // tile; key tiles before this step, first unit of its K
            int c0 = 0, c1 = 0;                                      // steps of the slots in the tiles before it
            int q0 = 0, q1 = 0;                                      // Q tiles of the slots so far
            struct { int t0[2], t1[2], n_tiles, n_keys, z0, z1, z2; } cur = {}, nxt = {};
            auto fetch = [&](int which) {
                const Plan* pl = plan_of(which);
                nxt.n_tiles = 0;
                if (pl) {
                    nxt.t0[0] = pl->t0[0];
                    nxt.t0[1] = pl->t0[1];
                    nxt.t1[0] = pl->t1[0];
                    nxt.t1[1] = pl->t1[1];
                    nxt.n_tiles = pl->n_tiles;
                    nxt.n_keys = pl->span.n;
                    nxt.z0 = pl->span.z0;
                    nxt.z1 = pl->span.z1;
                    nxt.z2 = pl->span.z2;
                    plan_done(which);
                }
            };
            // g, unit: of the step whose scores are next; the outputs are one step behind
            int jo = -1, vu = 0, gv = 0;                             // output step in its tile (-1: none yet), first unit and number of its V
#pragma unroll 1
            for (;;) {
                const bool out = jo >= 0, last = !out || jo + 1 == cur.n_tiles;
                if (last) fetch(t);
                const bool scores = !last || nxt.n_tiles > 0;
                if (!out && !scores) break;
                const int js = last ? 0 : jo + 1, r0 = jo * BN, ksteps = out ? min(8, (cur.n_keys - r0 + 15) >> 4) : 0;
                if (out) {
                    uwait(L::BAR_V + (gv & 3), (gv >> 2) & 1);
                    if (r0 < cur.z0) zero_rows(vu, 0, min(BN, cur.z0 - r0));
                    if (cur.z1 < cur.z2 && r0 < cur.z2 && r0 + BN > cur.z1) zero_rows(vu, max(0, cur.z1 - r0), min(BN, cur.z2 - r0));
                    if (cur.n_keys - r0 < BN) zero_rows(vu, cur.n_keys - r0, ksteps * 16);
                }
                const uint32_t va = ring_v + (uint32_t)vu * (SUB >> 4);
                const uint32_t vb = DVH == 2 ? ring_v + (uint32_t)((vu + 1) % L::UNITS) * (SUB >> 4) : va + (SUB / 2 >> 4);
                const int kf = L::BAR_K + (g & 3), kp = (g >> 2) & 1;
                auto issue_qk = [&](int x) {                         // S_x = Q_x K^T
                    const int tb = last ? nxt.t0[x] : cur.t0[x], te = last ? nxt.t1[x] : cur.t1[x];
                    if (js < tb || js >= te) return;
                    if (js == tb) { uwait(L::BAR_Q + x, (x ? q1 : q0) & 1); if (x) ++q1; else ++q0; }
                    uwait(kf, kp);
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int h = 0; h < NH; ++h) {
                            const uint32_t kl = ring_k + (uint32_t)((unit + (TWO_MAPS ? x : h)) % L::UNITS) * (SUB >> 4);
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                if (h * 4 + kk < ksteps_qk)
                                    mma_ss(tmem + x * 128, desc_join(q_lo + (((x * NH + h) * SUB + kk * 32) >> 4)), desc_join(kl + (kk * 32 >> 4)), ID_QK, h + kk > 0);
                        }
                        mma_commit(bar(L::BAR_S + x));
                        if (js + 1 == te) mma_commit(bar(L::BAR_QE + x));        // the last keys of this Q
                    }
                    __syncwarp();
                };
                // a next tile whose Q is still on its way is not worth holding the other slot's output back
                bool early = scores;
                if (scores && last && out)
                    early = __all_sync(0xffffffffu, b2::mbar_try_wait(bar(L::BAR_Q), q0 & 1) && b2::mbar_try_wait(bar(kf), kp));
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int tb = cur.t0[x], te = cur.t1[x], i = jo - tb, k = (x ? c1 : c0) + i;
                    const uint32_t tx = tmem + x * 128;
                    if (out && i >= 0 && jo < te) {                  // O_x += P_x V: k-steps of 16 keys
                        uwait(L::BAR_P + x, k & 1);                  // keys 0-63 of P_x are in TMEM, O_x is free (first step) or rescaled
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                if (u < ksteps) mma_ts(tx + 256, tx + u * 8, desc_join(va + u * (2048 >> 4)), ID_PV, i > 0 || u > 0);
                        }
                        __syncwarp();
                        uwait(L::BAR_P2 + x, k & 1);                 // keys 64-127
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                if (u + 4 < ksteps) mma_ts(tx + 256, tx + 32 + u * 8, desc_join(vb + u * (2048 >> 4)), ID_PV, true);
                            mma_commit(bar(L::BAR_PV + x));
                        }
                        __syncwarp();
                    }
                    if (x == 1 && out) commit(L::BAR_VE + (gv & 3));         // V consumed: its units refill under the Q K^T below
                    if (x == 1 && scores && !early) issue_qk(0);
                    if (x == 1 ? scores : early) issue_qk(x);
                }
                if (!scores) break;
                commit(L::BAR_KE + (g & 3));                         // K consumed
                if (last) {
                    if (out) {
                        c0 += max(0, cur.t1[0] - cur.t0[0]);
                        c1 += max(0, cur.t1[1] - cur.t0[1]);
                    }
                    cur = nxt;
                    ++t;
                }
                jo = js;
                gv = g++;
                vu = (unit + L::NK) % L::UNITS;
                unit = (unit + L::NS) % L::UNITS;
            }
            commit(L::BAR_END);                                      // nothing in flight when the TMEM is given back
            if (!__all_sync(0xffffffffu, wait(bar(L::BAR_END), 0, failed))) drain(bar(L::BAR_END), 0);
        }
    } else if (warp >= W_OUT) {
        // ------------------------------------------ output warps: O to a new maximum while the softmax takes its weights, and out
        // A quarter of the TMEM lanes each, of both slots.  BAR_P of a tile's first step is the word that O of the tile before it
        // has been read; the very first is given here.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        const int wq = warp - W_OUT, row = wq * 32 + lane;
        const uint32_t lane_off = (uint32_t)(wq * 32) << 16;
        if (lane < 2) b2::mbar_arrive(bar(L::BAR_P + lane));
        int steps0 = 0, steps1 = 0;                                  // of the slots in the tiles so far
        uint32_t alphas = 0, ends = 0;                               // phases of BAR_A and BAR_E, a bit a slot
#pragma unroll 1
        for (int t = 0;; ++t) {
            const Plan* pl = plan_of(t);
            if (!pl) break;
            const int n_tiles = pl->n_tiles, head = pl->head, row0 = pl->row0;
            const int tb0 = pl->t0[0], tb1 = pl->t0[1], te0 = pl->t1[0], te1 = pl->t1[1], nrows0 = pl->rows[0], nrows1 = pl->rows[1];
            plan_done(t);
#pragma unroll 1
            for (int j = 0; j < n_tiles; ++j) {
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    const int i = j - (x ? tb1 : tb0);
                    if (i > 0 && j < (x ? te1 : te0)) {
                        const uint32_t o_addr = tmem + lane_off + 256 + x * 128;
                        wait(bar(L::BAR_A + x), alphas >> x & 1, failed);
                        alphas ^= 1u << x;
                        if (KIND != KIND_SIGMOID) {
                            const float alpha = s_alpha[x][row];
                            if (__any_sync(0xffffffffu, alpha != 1.f)) {
                                wait(bar(L::BAR_PV + x), ((x ? steps1 : steps0) + i - 1) & 1, failed);
                                __syncwarp();
                                tc_fence_after();
#pragma unroll 1
                                for (int c = 0; c < 2 * DVH; c += 2) {
                                    uint32_t o[32], o2[32];
                                    tmem_ld32(o_addr + c * 32, o);
                                    tmem_ld32(o_addr + c * 32 + 32, o2);
                                    tmem_wait_ld();
#pragma unroll
                                    for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                                    tmem_st32(o_addr + c * 32, o);
#pragma unroll
                                    for (int k = 0; k < 32; ++k) o2[k] = __float_as_uint(__uint_as_float(o2[k]) * alpha);
                                    tmem_st32(o_addr + c * 32 + 32, o2);
                                }
                                tmem_wait_st();
                                tc_fence_before();
                            }
                        }
                        __syncwarp();
                        if (lane == 0) b2::mbar_arrive(bar(L::BAR_P + x));
                    }
                }
#pragma unroll 1
                for (int x = 0; x < 2; ++x) {
                    const int i = j - (x ? tb1 : tb0);
                    if (i < 0 || j + 1 != (x ? te1 : te0)) continue;
                    const uint32_t o_addr = tmem + lane_off + 256 + x * 128;
                    // ------------------------------ the slot's rows of this tile
                    wait(bar(L::BAR_E + x), ends >> x & 1, failed);
                    ends ^= 1u << x;
                    if (TWO_MAPS && x == 0) continue;                // the maps' difference is written when both are there
                    if (TWO_MAPS) wait(bar(L::BAR_PV), (steps0 + i) & 1, failed);
                    wait(bar(L::BAR_PV + x), ((x ? steps1 : steps0) + i) & 1, failed);
                    __syncwarp();
                    tc_fence_after();
                    const int hh = head + (two_heads ? x : 0);
                    const uint32_t out0 = TWO_MAPS ? tmem + lane_off + 256 : o_addr;
                    const int brow0 = row0 + (two_rows && x ? BM : 0) + wq * 32, left = (x ? nrows1 : nrows0) - wq * 32;      // the warp's rows
                    float f = s_inv[TWO_MAPS ? 0 : x][row], f2 = TWO_MAPS ? -a.map_lambda * s_inv[1][row] : 0.f;
                    const bf16* gp = static_cast<const bf16*>(a.gate);
                    if (TWO_MAPS) {                                  // the difference's own norm
                        float ss = 0.f;
#pragma unroll 1
                        for (int c = 0; c < 4 * DVH; ++c) {
                            if (c * 16 < a.dv) {
                                uint32_t o[16], o2[16];
                                tmem_ld_32x16(out0 + c * 16, o);
                                tmem_ld_32x16(out0 + 128 + c * 16, o2);
                                tmem_wait_ld();
#pragma unroll
                                for (int k = 0; k < 16; ++k) {
                                    const float d = fmaf(__uint_as_float(o2[k]), f2, __uint_as_float(o[k]) * f);
                                    if (c * 16 + k < a.dv) ss = fmaf(d, d, ss);
                                }
                            }
                        }
                        const float r = rsqrtf(ss / (float)a.dv + a.map_eps) * a.map_scale;
                        f *= r;
                        f2 *= r;
                    }
                    if (!GATE_COLUMNS && gp && lane < left) {
                        const float z = b2::sigmoid_f(__bfloat162float(gp[(size_t)(brow0 + lane) * a.gate_stride + hh]));
                        f *= z;
                        f2 *= z;
                    }
                    // 32 columns at a time; a lane stores 16 bytes of a row, its quad 64: a thread a row would spread each store over 32 lines
                    float fr[4], fr2[TWO_MAPS ? 4 : 1];
                    bf16* rp[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {                    // rows 8 g + lane / 4
                        const int r = g * 8 + (lane >> 2);
                        fr[g] = __shfl_sync(0xffffffffu, f, r);
                        if (TWO_MAPS) fr2[TWO_MAPS ? g : 0] = __shfl_sync(0xffffffffu, f2, r);
                        rp[g] = r < left ? static_cast<bf16*>(a.out) + (size_t)(brow0 + r) * a.out_stride + (size_t)hh * a.dv + 8 * (lane & 3) : nullptr;
                    }
#pragma unroll 1
                    for (int c = 0; c * 32 < a.dv; ++c) {
                        uint32_t o[2][16], o2[2][TWO_MAPS ? 16 : 1];
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            tmem_ld_16x32(out0 + ((uint32_t)(half * 16) << 16) + c * 32, o[half]);
                            if constexpr (TWO_MAPS) tmem_ld_16x32(out0 + 128 + ((uint32_t)(half * 16) << 16) + c * 32, o2[half]);
                        }
                        tmem_wait_ld();
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const int half = g >> 1, u = g & 1;
                            uint32_t w[4];
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                float v0 = __uint_as_float(o[half][4 * b + 2 * u]) * fr[g], v1 = __uint_as_float(o[half][4 * b + 2 * u + 1]) * fr[g];
                                if constexpr (TWO_MAPS) {
                                    v0 = fmaf(__uint_as_float(o2[half][4 * b + 2 * u]), fr2[g], v0);
                                    v1 = fmaf(__uint_as_float(o2[half][4 * b + 2 * u + 1]), fr2[g], v1);
                                }
                                if (GATE_COLUMNS && rp[g]) {
                                    const int r = g * 8 + (lane >> 2), col = c * 32 + b * 8 + 2 * (lane & 3);
                                    if (col < a.dv) {
                                        const uint32_t z = *reinterpret_cast<const uint32_t*>(gp + (size_t)(brow0 + r) * a.gate_stride + (size_t)hh * a.dv + col);
                                        v0 *= b2::sigmoid_as<bf16>(__uint_as_float(z << 16));
                                        v1 *= b2::sigmoid_as<bf16>(__uint_as_float(z & 0xffff0000u));
                                    }
                                }
                                w[b] = b2::pack_bf16x2(v0, v1);
                            }
                            const uint4 v = quad_transpose(w[0], w[1], w[2], w[3], lane);
                            if (rp[g] && c * 32 + 8 * (lane & 3) < a.dv) *reinterpret_cast<uint4*>(rp[g] + c * 32) = v;
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (TWO_MAPS ? lane < 2 : lane == 0) b2::mbar_arrive(bar(L::BAR_P + (TWO_MAPS ? lane : x)));
                }
            }
            steps0 += max(0, te0 - tb0);
            steps1 += max(0, te1 - tb1);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
        // ------------------------------------------ softmax of slot x
        const int x = warp >> 2, wq = warp & 3;
        const int row = wq * 32 + lane;                              // query row of the slot = TMEM lane
        const uint32_t s_addr = tmem + ((uint32_t)(wq * 32) << 16) + x * 128;
        const float sl2 = prm.scale_log2;
        const float cap2 = a.cap * LOG2E, cx = a.cap > 0.f ? a.scale / a.cap : 0.f, cap_e = a.cap > 0.f ? 2.f / a.cap : 0.f;
        const float cz = cx * cx, e1 = sl2 * cz * (-1.f / 3.f), e2 = sl2 * cz * cz * (2.f / 15.f), e3 = sl2 * cz * cz * cz * (-17.f / 315.f);
        int steps = 0;                                               // of this slot in the tiles so far
#pragma unroll 1
        for (int t = 0;; ++t) {
            const Plan* pl = plan_of(t);
            if (!pl) break;
            const int tb = pl->t0[x], te = pl->t1[x], nrows = pl->rows[x], head = pl->head;
            const int all_hi = pl->all_hi[x], all_low = pl->all_low[x], keep = pl->keep;
            RowRange mine = {0, 0, 0};
            if (te > tb) mine = range_of(pl->span, pl->first_row[x] + min(row, nrows - 1), a.chunk, a.window);
            plan_done(t);
            if (te <= tb) continue;
            const int hh = head + (two_heads ? x : 0);
            const float bias2 = KIND == KIND_SIGMOID && a.head_bias ? a.head_bias[hh] * LOG2E : 0.f;
            float m = a.sink > 0.f ? (a.sink_logits ? a.sink_logits[hh] : a.sink_logit) * LOG2E : -INFINITY, l = a.sink;
#pragma unroll 1
            for (int j = tb; j < te; ++j, ++steps) {
                wait(bar(L::BAR_S + x), steps & 1, failed);
                __syncwarp();
                tc_fence_after();
                const int c0 = j * BN;
                const bool partial = c0 + BN - 1 > all_hi || c0 < all_low;
                // which of a group's 32 keys the row sees
                auto seen = [&](int c) {
                    const int b = c0 + c * 32;
                    return col_bits(mine.low - b, mine.hi + 1 - b) | col_bits(mine.block - b, min(keep, mine.hi + 1) - b);
                };
                uint32_t sr[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + c * 32, sr[c]);
                tmem_wait_ld();
                bool small = false;                                  // capped: the polynomial will do for every score of the warp
                if (KIND != KIND_SIGMOID) {
                    // The largest score the row sees (capped: the smallest too; the cap rises with the score, so it is taken of these two
                    // alone), in short chains: one warp a scheduler and slot hides nothing.
                    float hi[8], lo[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) { hi[k] = -INFINITY; lo[k] = INFINITY; }
                    if (partial) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t see = seen(c);
                            if (KIND == KIND_CAPPED || !__all_sync(0xffffffffu, see == ~0u)) {
#pragma unroll
                                for (int k = 0; k < 32; ++k) {
                                    const bool ok = see >> k & 1;
                                    if (KIND == KIND_CAPPED) lo[k & 7] = fminf(lo[k & 7], ok ? __uint_as_float(sr[c][k]) : INFINITY);
                                    sr[c][k] = ok ? sr[c][k] : 0xff800000u;              // -inf
                                }
                            }
                        }
                    } else if (KIND == KIND_CAPPED) {
#pragma unroll
                        for (int c = 0; c < 4; ++c)
#pragma unroll
                            for (int k = 0; k < 32; k += 2) lo[(k >> 1) & 7] = min3(lo[(k >> 1) & 7], __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 1]));
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < 32; k += 2) hi[(k >> 1) & 7] = max3(hi[(k >> 1) & 7], __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 1]));
                    const float mx = max3(max3(hi[0], hi[1], hi[2]), max3(hi[3], hi[4], hi[5]), fmaxf(hi[6], hi[7]));
                    float top = mx * sl2;                            // in the exponent of 2
                    if (KIND == KIND_CAPPED) {
                        const float mn = min3(min3(lo[0], lo[1], lo[2]), min3(lo[3], lo[4], lo[5]), fminf(lo[6], lo[7]));
                        small = __all_sync(0xffffffffu, cx > 0.f && fmaxf(mx, -mn) * cx <= 0.1875f);
                        if (mn > mx) {                               // the row sees none of these keys
                            top = -INFINITY;
                        } else if (small) {
                            float y1;
                            tanh_small_exponent_x2(top, y1, __float_as_uint(mx), __float_as_uint(mx), sl2, e1, e2, e3, 0.f);
                        } else {
                            top = (sl2 < 0.f ? mn : mx) * sl2;       // any score, any sign of the scale
                            if (a.cap > 0.f) top = cap_score(top, cap2, cap_e);
                        }
                    }
                    const float m_new = max3(m, top, FLOOR), alpha = b2::fast_exp2(m - m_new);
                    l *= alpha;                                      // at first the sink's share, if any; exp2(-inf) = 0
                    m = m_new;
                    if (j > tb) s_alpha[x][row] = alpha;             // the output warps bring O along while the weights are taken
                }
                if (j > tb) {
                    __syncwarp();
                    if (lane == 0) b2::mbar_arrive(bar(L::BAR_A + x));
                }
                // P overwrites the first 64 columns of S_x; the P V of 64 keys runs under the next 64
                auto handed = [&](int c) {
                    if (c & 1) {
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) b2::mbar_arrive(bar((c == 1 ? L::BAR_P : L::BAR_P2) + x));
                    }
                };
                float sum[4] = {0.f, 0.f, 0.f, 0.f};                 // the denominator sums the fp32 weights
                if (KIND == KIND_CAPPED && (partial || !small)) {
                    // the rare tiles: masks behind the cap, any score; from TMEM once more, so that the loop can be rolled
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t r[32], pk[16];
                        float y[32];
                        tmem_ld32(s_addr + c * 32, r);
                        tmem_wait_ld();
                        const uint32_t see = partial ? seen(c) : ~0u;
                        if (small) {
#pragma unroll
                            for (int k = 0; k < 32; k += 2) tanh_small_exponent_x2(y[k], y[k + 1], r[k], r[k + 1], sl2, e1, e2, e3, m);
                        } else {
#pragma unroll
                            for (int k = 0; k < 32; ++k) {
                                y[k] = __uint_as_float(r[k]) * sl2;
                                if (a.cap > 0.f) y[k] = cap_score(y[k], cap2, cap_e);
                                y[k] -= m;
                            }
                        }
                        if (!__all_sync(0xffffffffu, see == ~0u)) {
#pragma unroll
                            for (int k = 0; k < 32; ++k) y[k] = see >> k & 1 ? y[k] : -INFINITY;
                        }
#pragma unroll
                        for (int k = 0; k < 32; k += 2) {
                            const float w0 = b2::fast_exp2(y[k]), w1 = b2::fast_exp2(y[k + 1]);
                            add_x2(sum[k & 2], sum[(k & 2) + 1], w0, w1);
                            pk[k >> 1] = b2::pack_bf16x2(w0, w1);
                        }
                        tmem_st16(s_addr + c * 16, pk);
                        handed(c);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t pk[16];
                        const uint32_t see = KIND == KIND_SIGMOID && partial ? seen(c) : ~0u;
#pragma unroll
                        for (int k = 0; k < 32; k += 2) {
                            float w0, w1;
                            if (KIND == KIND_SIGMOID) {
                                fma_x2(w0, w1, __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 1]), sl2, bias2);
                                w0 = sigmoid2_f(w0);
                                w1 = sigmoid2_f(w1);
                                w0 = see >> k & 1 ? w0 : 0.f;
                                w1 = see >> (k + 1) & 1 ? w1 : 0.f;
                            } else {
                                if (KIND == KIND_CAPPED) tanh_small_exponent_x2(w0, w1, sr[c][k], sr[c][k + 1], sl2, e1, e2, e3, m);
                                else fma_x2(w0, w1, __uint_as_float(sr[c][k]), __uint_as_float(sr[c][k + 1]), sl2, -m);
                                w0 = b2::fast_exp2(w0);
                                w1 = b2::fast_exp2(w1);
                                add_x2(sum[k & 2], sum[(k & 2) + 1], w0, w1);
                            }
                            pk[k >> 1] = b2::pack_bf16x2(w0, w1);
                        }
                        tmem_st16(s_addr + c * 16, pk);
                        handed(c);
                    }
                }
                if (KIND != KIND_SIGMOID) l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            }
            // s_inv is one tile deep: of a tile with one step nothing else says that the output warps have read the one before it
            if (te - tb == 1) wait(bar(L::BAR_PV + x), (steps - 1) & 1, failed);
            s_inv[x][row] = KIND == KIND_SIGMOID ? 1.f : (l > 0.f ? 1.f / l : 0.f);
            __syncwarp();
            if (lane == 0) b2::mbar_arrive(bar(L::BAR_E + x));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
    if (*failed && lane == 0) {                                      // boxes that nobody has waited for, whichever wait gave up: every role is done now
        if (warp == W_PLAN) {
            if (sent0 > 0) drain(bar(L::BAR_Q), (sent0 - 1) & 1);
            if (sent1 > 0) drain(bar(L::BAR_Q + 1), (sent1 - 1) & 1);
        } else if (warp == W_K || warp == W_V) {
            for (int back = 1; back <= min(4, sent0); ++back) drain(bar((warp == W_V ? L::BAR_V : L::BAR_K) + ((sent0 - back) & 3)), ((sent0 - back) >> 2) & 1);
        }
    }
    if (*failed) {                                                   // a wait gave up: every row of this CTA's tiles is NaN
        int tile_rows = prm.rows_per_cta, hpc = prm.heads_per_cta;
        order.init(a, s_list, tile_rows, hpc, lane);
        const uint32_t groups = (uint32_t)(a.H / hpc);
#pragma unroll 1
        for (uint32_t turn = 0;; ++turn) {
            const uint32_t rank = tile_rank(turn);
            Prompt at = {0, 0, 0, 0};
            int q0 = 0;
            if (!order.find((int)(rank / groups), at, q0)) break;
            if (at.ctx < 0) continue;
            const int rows = min(at.len - q0, tile_rows), wide = hpc * a.dv;
#pragma unroll 1
            for (int idx = tid; idx < rows * wide; idx += NTHREADS)
                static_cast<bf16*>(a.out)[(size_t)(at.row + q0 + idx / wide) * a.out_stride + (size_t)(rank % groups) * wide + idx % wide] =
                    __float2bfloat16(__int_as_float(0x7fc00000));
        }
    }
}

template <int NH, int DVH, int KIND, bool TWO_MAPS, bool GATHERED, bool GATE_COLUMNS = false>
int launch(const Params& p, dim3 grid, cudaStream_t st) {
    auto kern = prompt_turns_kernel<NH, DVH, KIND, TWO_MAPS, GATHERED, GATE_COLUMNS, false>;
    if constexpr (!GATHERED)                         // instances of their own: the list's code would cost all others 0.3 us
        if (p.a.chunk > 0) kern = prompt_turns_kernel<NH, DVH, KIND, TWO_MAPS, GATHERED, GATE_COLUMNS, true>;
    constexpr int smem = Shape<NH, DVH, TWO_MAPS>::SMEM;
    B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kern<<<grid, NTHREADS, smem, st>>>(p);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

}  // namespace

int b2_internal_prompt_turns(const b2_prompt_args& a, void* stream) {
    const int n_sm = b2_sm_count();
    Params p;
    p.a = a;
    p.scale_log2 = a.scale * LOG2E;
    p.bs_shift = -1;
    for (int b = 0; b < 16; ++b)
        if (a.bs == 1 << b) p.bs_shift = b;
    const bool gathered = a.cu_k != nullptr;
    // Boxes: gathered rows are consecutive, 128 (V: 64) of them one a sub-tile; a page is one, if it fills whole groups of eight rows of a
    // tile.  A head's columns from two tensors (dk0) have to change between sub-tiles.  Pages: no limit, the tables' entries are the
    // caller's; gathered rows: k_rows, behind which zeros come, or none where it is not known (the kernel looks at their number itself).
    const uint64_t many = 0x7fffffff;
    const bool sides = !gathered || a.dk0 % 64 == 0 || a.dk0 >= a.dk;
    const int dr = a.dk - a.dk0;
    p.tma = gathered ? sides && (a.k1_row * 2) % 16 == 0 : p.bs_shift >= 3;
    p.k_box = gathered ? 7 : std::min(std::max(p.bs_shift, 0), 7);
    p.v_box = std::min(p.k_box, 6);
    p.align = !gathered && p.tma ? 1 << p.k_box : 1;
    p.tma_q = sides && (a.q0_row % 8 == 0) && (a.q0_head % 8 == 0) && b2_aligned16(a.q0) &&
              (!gathered || dr == 0 || (a.q1_row % 8 == 0 && a.q1_head % 8 == 0 && b2_aligned16(a.q1)));
    int rc = B2_OK;
    if (p.tma && gathered) {
        const uint64_t rows = a.k_rows > 0 && (uint64_t)a.k_rows < many ? (uint64_t)a.k_rows : many;
        const uint32_t box3[3] = {64, 1, BN}, box2[2] = {64, BN}, boxv[3] = {64, 1, 64};
        if (a.dk0 > 0) {
            const uint64_t dims[3] = {(uint64_t)a.dk0, (uint64_t)a.H, rows}, st[2] = {(uint64_t)a.dk0 * 2, (uint64_t)a.H * a.dk0 * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_k0, a.k0, 3, dims, st, box3);
        }
        if (rc == B2_OK && dr > 0) {
            const uint64_t dims[2] = {(uint64_t)dr, rows}, st[1] = {(uint64_t)a.k1_row * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_k1, a.k1, 2, dims, st, box2);
        }
        if (rc == B2_OK) {
            const uint64_t dims[3] = {(uint64_t)a.dv, (uint64_t)a.H, rows}, st[2] = {(uint64_t)a.dv * 2, (uint64_t)a.H * a.dv * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_v, a.v, 3, dims, st, boxv);
        }
    } else if (p.tma) {
        const uint64_t bs = (uint64_t)a.bs, gk = (uint64_t)a.G * a.maps, gv = (uint64_t)a.G, dk = (uint64_t)a.dk, dv = (uint64_t)a.dv;
        const uint32_t boxk[4] = {64, 1u << p.k_box, 1, 1}, boxv[4] = {64, 1u << p.v_box, 1, 1};
        const uint64_t dk4[4] = {dk, bs, gk, many}, sk3[3] = {dk * 2, bs * dk * 2, gk * bs * dk * 2};
        const uint64_t dv4[4] = {dv, bs, gv, many}, sv3[3] = {dv * 2, bs * dv * 2, gv * bs * dv * 2};
        rc = b2_internal_encode_bf16_sw128(&p.map_k0, a.k0, 4, dk4, sk3, boxk);
        if (rc == B2_OK) rc = b2_internal_encode_bf16_sw128(&p.map_v, a.v, 4, dv4, sv3, boxv);
    }
    if (rc == B2_OK && p.tma_q) {
        const uint32_t box[4] = {64, 1, 1, BM};
        const int d0 = gathered ? a.dk0 : a.dk;
        if (d0 > 0) {
            const uint64_t dims[4] = {(uint64_t)d0, (uint64_t)a.maps, (uint64_t)a.H, (uint64_t)a.T};
            const uint64_t st[3] = {(uint64_t)d0 * 2, (uint64_t)a.q0_head * 2, (uint64_t)a.q0_row * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_q0, a.q0, 4, dims, st, box);
        }
        if (rc == B2_OK && gathered && dr > 0) {
            const uint64_t dims[4] = {(uint64_t)dr, 1, (uint64_t)a.H, (uint64_t)a.T};
            const uint64_t st[3] = {(uint64_t)dr * 2, (uint64_t)a.q1_head * 2, (uint64_t)a.q1_row * 2};
            rc = b2_internal_encode_bf16_sw128(&p.map_q1, a.q1, 4, dims, st, box);
        }
    }
    if (rc != B2_OK) return rc;
    // Two slots a CTA share the copies of a key tile and cover each other's softmax; row tiles, whose later one sees more keys, only where they
    // fill the SMs (2000 gathered rows x 16 heads: 42.8 us in pairs, 38.1 one by one).  Two heads of a kv head before two row tiles: see above.
    // These counts are bounds, far too large where most sequences are decode rows: TileOrder::init counts, and takes one slot a tile where
    // that is all in one wave (64 decode rows and a prompt of 300, 16 heads of sigmoid weights: 67.3 us in pairs, 64.4 one by one).
    const int64_t longs = std::min(a.n_seq, a.T / a.min_rows);       // sequences of min_rows rows or more
    const int64_t tiles128 = (int64_t)a.T / BM + longs, tiles256 = (int64_t)a.T / (2 * BM) + longs;
    p.rows_per_cta = BM;
    p.heads_per_cta = 1;
    if (a.maps == 1) {
        const bool pair = !gathered && (a.H / a.G) % 2 == 0;
        if (pair) p.heads_per_cta = 2;
        else if (tiles256 * a.H >= n_sm) p.rows_per_cta = 2 * BM;
    }
    B2_REQUIRE(tiles128 * a.H <= 0x7fffffff, B2_EUNSUPPORTED, "prompt attention: %lld row tiles exceed the grid", (long long)tiles128);
    const dim3 grid((unsigned)n_sm);                 // CTAs without a tile leave at once; a grid of fewer leaves the kernel behind it unevenly spread
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nh = (a.dk + 63) / 64, dvh = (a.dv + 63) / 64;
    const bool one_by_one = a.cap > 0.f || !(a.scale > 0.f);         // the capped form takes any score and any sign of the scale
#define B2_PT(NH, DVH, KIND, MAPS2, GATH) return launch<NH, DVH, KIND, MAPS2, GATH>(p, grid, st)
#define B2_PG(NH, DVH)                                                                              \
    do {                                                                                            \
        if (a.gate && a.gate_channels) return launch<NH, DVH, KIND_SOFTMAX, false, true, true>(p, grid, st); \
        return launch<NH, DVH, KIND_SOFTMAX, false, true>(p, grid, st);                             \
    } while (0)
    if (gathered) {
        if (nh == 1) { if (dvh == 1) B2_PG(1, 1); B2_PG(1, 2); }
        if (nh == 2) { if (dvh == 1) B2_PG(2, 1); B2_PG(2, 2); }
        if (dvh == 1) B2_PG(3, 1);
        B2_PG(3, 2);
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
#undef B2_PG
#undef B2_PT
}
