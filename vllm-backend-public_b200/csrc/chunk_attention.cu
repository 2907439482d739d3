// chunk_attention.cu -- attention over a paged cache of keys and values per kv head, with parameters that designs set
// independently of each other:
//   * per-head RMS norm of queries and keys (a plain weight of size dk shared by the heads),
//   * a block-local causal mask: position i sees j <= i with floor(j / chunk) == floor(i / chunk), blocks counted from
//     position 0 of the sequence (chunk = 0: plain causal),
//   * a sink: `sink` is added to the softmax denominator as exp(sink_logit - max), a key with no value (sink = 0: none;
//     sink = 1 with logit 0 gives p_j = exp(s_j) / (1 + sum exp(s))); the logit may also be one learned number per
//     query head (sink_logits [H], not scaled),
//   * a sliding window that keeps the first tokens: position i sees j <= i with i - j < window or j < keep_first
//     (window = 0: no window).  A query then reads the kept keys and its window's keys and nothing between them,
//   * a sigmoid gate per (token, head) on the head's output,
//   * the weight of a visible key: its share of the softmax, or (B2_WEIGHT_SIGMOID) sigmoid(score + head_bias[h]), a number
//     of its own that no other key changes -- no maximum, no denominator, and a sink has no meaning,
//   * a cap on the scores: s <- cap * tanh(s / cap) before the mask and the softmax (cap = 0: none),
//   * two maps per head (differential attention): a head holds two queries and two keys of size dk, each pair of them is a
//     softmax attention of its own over the head's values, and the head's output is a1 - lambda * a2, divided by its own root
//     mean square over dv (eps inside the root) and multiplied by a constant.  The two maps of a head are neighbours in q
//     [T, H, maps, dk] and in the K pool; they are walked together, so a value row is read once for both.
// Key size dk and value size dv are independent; K and V live in separate paged pools
//   k_cache [num_blocks, G * maps, bs, dk],  v_cache [num_blocks, G, bs, dv]      (activation type).
//
//   b2_qknorm_cache      per token: q heads normalised into q_out; k heads normalised and written to the K pool, v copied
//                        to the V pool, through the token's slot (slot < 0 skips the write).
//   b2_qk_prep_cache     the same pass with the norm optional and a query temperature: the query of the token at position p
//                        is multiplied by 1 + coef * ln(floor((p + 1) / every) + 1) (fp32), so queries sharpen as the
//                        context grows in steps of `every` positions (coef = 0: none).
//   b2_qk_rope_cache     rows [q | k] or [q | k | v]: the first rot_dims entries of every q and k head are rotated by the
//                        token's position (pairs (i, i + rot_dims/2) or (2i, 2i + 1); fp32 table [max_pos, rot_dims] =
//                        cos | sin halves), q to q_out, rotated k to the K pool; the V pool receives v, or, for designs
//                        whose values ARE the keys, the k heads as projected (before the rotation).  The value heads may be
//                        fewer than the key heads (two key maps over one set of values).
//   b2_qk_norm_rope_cache  rows [q | k | v]: all of q (H * dk numbers) and all of k (G * dk) are RMS-normed as one row each,
//                        before the split into heads (fp32 weights of those sizes), then rotated and written as above; the
//                        numbers stay in fp32 between the norm and the rotation.
//   b2_chunk_attention   prompt rows of bf16 models: prompt_tc5.cu (tcgen05), or mma.sync tiles of 64 rows for the head sizes that
//                        one does not take; decode rows and short portions of bf16 models on mma.sync with the keys (up to eight
//                        query heads a kv head) or the query heads as operand rows, or (head sizes the tensor cores do not
//                        take) one CTA per (row, kv head) on fp32 FMAs; fp32 and odd sizes one warp per (token, head). Scores, softmax state and accumulators are fp32 in all of them.  With a mask a query
//                        touches only the keys it sees, wherever it stands; a decode row is a sequence with one query.
// Sequences are described like everywhere in this library: rows cu_q[i] .. cu_q[i+1]-1, ctx_start[i] cached tokens
// before them (< 0: padding, output rows are zeroed), block_tables[i, :].
#include "b2_mask.cuh"
#include "b2_tc5.cuh"

namespace {

constexpr int kMaxDvPerLane = 16;                    // dv <= 512

// 1 / rms of nq and of nk numbers whose squares the threads of the block have summed up in parts
__device__ __forceinline__ void block_scales(float sq, float sk, int nq, int nk, float eps, float* red, float& inv_q, float& inv_k) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    sq = b2::warp_sum(sq);
    sk = b2::warp_sum(sk);
    if (lane == 0) {
        red[2 * wid] = sq;
        red[2 * wid + 1] = sk;
    }
    __syncthreads();
    sq = sk = 0.f;
    for (int x = 0; x < nw; ++x) {                   // at most eight warps: every thread adds them up itself
        sq += red[2 * x];
        sk += red[2 * x + 1];
    }
    inv_q = rsqrtf(sq / (float)nq + eps);
    inv_k = rsqrtf(sk / (float)nk + eps);
}

// 1 / rms of all H * dk numbers of q and of all G * dk of k, which lie one after the other at `src` (block-wide)
template <typename T, int W>
__device__ __forceinline__ void qk_row_scales(const T* src, int nq, int nk, float eps, float* red, float& inv_q, float& inv_k) {
    float sq = 0.f, sk = 0.f;
    for (int i = threadIdx.x * W; i < nq + nk; i += blockDim.x * W) {
        float v[4] = {0.f, 0.f, 0.f, 0.f}, ss = 0.f;
        if (W == 4) b2::ld4(src + i, v); else v[0] = b2::ld(src + i);
#pragma unroll
        for (int c = 0; c < W; ++c) ss = fmaf(v[c], v[c], ss);
        if (i < nq) sq += ss; else sk += ss;
    }
    block_scales(sq, sk, nq, nk, eps, red, inv_q, inv_k);
}

// Rows [q | k] (+ [v]): partial rotation of the q and k heads, K (rotated) and V pool writes; see the file comment.  NORM:
// q and k are first normed over their whole rows.
template <typename T, bool NORM>
__global__ void qk_rope_cache_kernel(const T* __restrict__ qkv, int64_t qkv_stride, int H, int G, int Gv, int dk, int dv, bool v_from_k,
                                     int rot_dims, bool interleaved, const int32_t* __restrict__ positions,
                                     const float* __restrict__ cos_sin, int max_pos, const int64_t* __restrict__ slots, int bs,
                                     const float* __restrict__ q_w, const float* __restrict__ k_w, float eps,
                                     T* __restrict__ q_out, T* __restrict__ k_cache, T* __restrict__ v_cache) {
    __shared__ float red[16];
    const int row = blockIdx.x;
    const T* src = qkv + (size_t)row * qkv_stride;
    float inv_q = 1.f, inv_k = 1.f;
    if (NORM) qk_row_scales<T, 1>(src, H * dk, G * dk, eps, red, inv_q, inv_k);
    int pos = positions[row];
    pos = pos < 0 ? 0 : (pos >= max_pos ? max_pos - 1 : pos);
    const float* cs = cos_sin + (size_t)pos * rot_dims;
    const int half = rot_dims / 2;
    const int64_t slot = slots[row];
    const int64_t blk = slot >= 0 ? slot / bs : 0;
    const int off = slot >= 0 ? (int)(slot % bs) : 0;
    // q and k heads: element i of a head
    for (int idx = threadIdx.x; idx < (H + G) * dk; idx += blockDim.x) {
        const int hd = idx / dk, i = idx % dk;
        if (hd >= H && slot < 0) continue;
        const T* v = src + (size_t)hd * dk;
        const float* w = NORM ? (hd < H ? q_w + (size_t)hd * dk : k_w + (size_t)(hd - H) * dk) : nullptr;
        const float inv = hd < H ? inv_q : inv_k;
        float x = b2::ld(v + i);
        if (NORM) x *= inv * w[i];
        if (i < rot_dims) {
            int pr, partner;
            bool second;
            if (interleaved) { pr = i >> 1; partner = i ^ 1; second = i & 1; }
            else { second = i >= half; pr = second ? i - half : i; partner = second ? i - half : i + half; }
            const float c = cs[pr], sn = cs[half + pr], other = b2::ld(v + partner) * (NORM ? inv * w[partner] : 1.f);
            x = second ? fmaf(x, c, other * sn) : fmaf(x, c, -other * sn);
        }
        T* dst = hd < H ? q_out + ((size_t)row * H + hd) * dk : k_cache + (((size_t)blk * G + (hd - H)) * bs + off) * dk;
        b2::st(dst + i, x);
    }
    if (slot < 0) return;
    const T* vsrc = v_from_k ? src + (size_t)H * dk : src + (size_t)(H + G) * dk;
    for (int idx = threadIdx.x; idx < Gv * dv; idx += blockDim.x) {
        const int g = idx / dv, i = idx % dv;
        v_cache[(((size_t)blk * Gv + g) * bs + off) * dv + i] = vsrc[idx];
    }
}

// The same with four entries per access (8 or 16 bytes): every size a multiple of four, the rotated entries a multiple of
// eight in the (i, i + rot_dims/2) layout so that a group of four and its partners never straddle the halves.
// A thread takes two groups of four of a head, where they rotate one another the two partners, and the same two in every head it
// visits: their cosines and sines stay in registers.  `held`: at most kRopeHeld heads a thread, whose inputs it keeps in registers
// from the row's sums to the stores, so a row is read once.
// Bound: memory, and the instructions around it.  With one group a thread, its partner read again beside it, the table entry by entry
// and the row read a second time behind the norm, 4096 rows of 32 + 8 heads of 128 with NORM took 56 us, this one 40; the bytes need 14.
// 64 registers and four CTAs an SM: with 120 registers it took 54.
constexpr int kRopeHeld = 4;

template <typename T> struct Raw4;
template <> struct Raw4<float> { using type = float4; };
template <> struct Raw4<__nv_bfloat16> { using type = uint2; };

template <typename T, bool NORM>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 4 : 3)
qk_rope_cache_vec_kernel(const T* __restrict__ qkv, int64_t qkv_stride, int H, int G, int Gv, int dk, int dv, bool v_from_k, int rot_dims,
                         bool interleaved, const int32_t* __restrict__ positions, const float* __restrict__ cos_sin, int max_pos,
                         const int64_t* __restrict__ slots, int bs, const float* __restrict__ q_w, const float* __restrict__ k_w,
                         float eps, T* __restrict__ q_out, T* __restrict__ k_cache, T* __restrict__ v_cache) {
    using Raw = typename Raw4<T>::type;
    __shared__ float red[16];
    const int row = blockIdx.x;
    const T* src = qkv + (size_t)row * qkv_stride;
    const int64_t slot = slots[row];
    int pos = positions[row];
    const int half = rot_dims / 2, per = (dk + 7) / 8, heads = slot >= 0 ? H + G : H;
    // heads of at most 256 groups of eight: a thread keeps its place in the head; larger ones step through it
    const int step = per < (int)blockDim.x ? blockDim.x / per : 1, wide = per < (int)blockDim.x ? step * per : blockDim.x;
    const bool held = per <= wide && H + G <= kRopeHeld * step;
    const int hd0 = per < (int)blockDim.x ? threadIdx.x / per : 0, jt = threadIdx.x - hd0 * per;
    const bool in = (int)threadIdx.x < wide;
    auto place = [&](int j, int& i, int& i2) {
        const bool pairs = !interleaved && j < half / 4;
        i = pairs ? 4 * j : interleaved ? 8 * j : rot_dims + 8 * (j - half / 4);
        i2 = pairs ? i + half : i + 4;
        return pairs;
    };
    auto load = [&](int hd, int i, int i2, Raw& a, Raw& b) {
        const T* v = src + (size_t)hd * dk;
        a = *reinterpret_cast<const Raw*>(v + i);
        b = i2 < dk ? *reinterpret_cast<const Raw*>(v + i2) : Raw{};
    };
    Raw ra[kRopeHeld], rb[kRopeHeld];
    float inv_q = 1.f, inv_k = 1.f;
    if (held) {
        int i, i2;
        place(jt, i, i2);
#pragma unroll
        for (int u = 0; u < kRopeHeld; ++u) {
            ra[u] = rb[u] = Raw{};
            if (in && hd0 + u * step < heads) load(hd0 + u * step, i, i2, ra[u], rb[u]);
        }
    }
    pos = pos < 0 ? 0 : (pos >= max_pos ? max_pos - 1 : pos);
    const float* cs = cos_sin + (size_t)pos * rot_dims;
    int64_t blk = 0;
    int off = 0;
    if (slot >= 0) {                                 // a 64-bit division only where it has to be one
        if (slot >> 31) { blk = slot / bs; off = (int)(slot % bs); }
        else { blk = (int)slot / bs; off = (int)slot - (int)blk * bs; }
    }
    if (NORM) {
        if (held) {
            float sq = 0.f, sk = 0.f;
#pragma unroll
            for (int u = 0; u < kRopeHeld; ++u) {
                float x[4], y[4];
                b2::ld4(reinterpret_cast<const T*>(&ra[u]), x);
                b2::ld4(reinterpret_cast<const T*>(&rb[u]), y);
                float s = 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) s = fmaf(x[c], x[c], fmaf(y[c], y[c], s));
                if (hd0 + u * step < H) sq += s; else sk += s;
            }
            block_scales(sq, sk, H * dk, G * dk, eps, red, inv_q, inv_k);
        } else {
            qk_row_scales<T, 4>(src, H * dk, G * dk, eps, red, inv_q, inv_k);
        }
    }
    for (int j0 = 0; j0 < per; j0 += wide) {
        const int j = j0 + jt;
        if (!in || j >= per) continue;
        int i, i2;
        const bool pairs = place(j, i, i2), two = i2 < dk;
        float co[4], si[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) { co[c] = 1.f; si[c] = 0.f; }
        if (pairs) {
#pragma unroll
            for (int c = 0; c < 4; ++c) { co[c] = cs[i + c]; si[c] = cs[half + i + c]; }
        } else if (interleaved) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (i + 2 * c < rot_dims) { co[c] = cs[i / 2 + c]; si[c] = cs[half + i / 2 + c]; }
        }
        auto turn = [&](int hd, const Raw& a0, const Raw& b0) {
            float x[4], y[4];
            b2::ld4(reinterpret_cast<const T*>(&a0), x);
            b2::ld4(reinterpret_cast<const T*>(&b0), y);
            if (NORM) {
                const float* w = hd < H ? q_w + (size_t)hd * dk : k_w + (size_t)(hd - H) * dk;
                const float inv = hd < H ? inv_q : inv_k;
                float wx[4], wy[4] = {0.f, 0.f, 0.f, 0.f};
                b2::ld4(w + i, wx);
                if (two) b2::ld4(w + i2, wy);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    x[c] *= inv * wx[c];
                    y[c] *= inv * wy[c];
                }
            }
            if (pairs) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float a = x[c], b = y[c];
                    x[c] = fmaf(a, co[c], -b * si[c]);
                    y[c] = fmaf(b, co[c], a * si[c]);
                }
            } else if (interleaved && i < rot_dims) {
#pragma unroll
                for (int c = 0; c < 4; c += 2) {
                    const float a = x[c], b = x[c + 1], a2 = y[c], b2_ = y[c + 1];
                    x[c] = fmaf(a, co[c / 2], -b * si[c / 2]);
                    x[c + 1] = fmaf(b, co[c / 2], a * si[c / 2]);
                    if (i2 < rot_dims) {
                        y[c] = fmaf(a2, co[2 + c / 2], -b2_ * si[2 + c / 2]);
                        y[c + 1] = fmaf(b2_, co[2 + c / 2], a2 * si[2 + c / 2]);
                    }
                }
            }
            T* dst = hd < H ? q_out + ((size_t)row * H + hd) * dk : k_cache + (((size_t)blk * G + (hd - H)) * bs + off) * dk;
            b2::st4(dst + i, x);
            if (two) b2::st4(dst + i2, y);
        };
        if (held) {
#pragma unroll
            for (int u = 0; u < kRopeHeld; ++u)
                if (hd0 + u * step < heads) turn(hd0 + u * step, ra[u], rb[u]);
        } else {
            for (int hd = hd0; hd < heads; hd += step) {
                Raw a0, b0;
                load(hd, i, i2, a0, b0);
                turn(hd, a0, b0);
            }
        }
    }
    if (slot < 0) return;
    const T* vsrc = v_from_k ? src + (size_t)H * dk : src + (size_t)(H + G) * dk;
    const int pv = dv / 4;
    for (int idx = threadIdx.x; idx < Gv * pv; idx += blockDim.x) {
        const int g = idx / pv, i = (idx - g * pv) * 4;
        *reinterpret_cast<Raw*>(v_cache + (((size_t)blk * Gv + g) * bs + off) * dv + i) = *reinterpret_cast<const Raw*>(vsrc + (size_t)idx * 4);
    }
}

// The same in bf16 with sixteen entries a thread: every size a multiple of sixteen, at most 1024 threads a row.  A thread keeps its
// head, its place in it and its norm weights; with the rotation in halves its entries are 8 j .. and their partners.
// RING: a CTA goes over rows gridDim.x apart, which come with their cosines and sines by bulk copies, kRopeStages ahead; without, a CTA
// takes one row and loads it itself (a decode step has too few rows for the copies to run ahead).
// Bound: memory, and the norm, which needs a whole row before its first result.  4096 rows of 32 + 8 heads of 128 with NORM (92 MB): kernel
// above 39 us, this one 31; without NORM 16 + 4 heads 20.6 -> 10.4, 32 + 8 in neighbours 33 -> 27; a row ahead in registers instead of
// the ring took 36 with NORM.  380 instructions a warp and row are half of the issue slots.  1024 threads a CTA hold it to 64 registers, of
// which the ring with NORM spills 48 bytes.
constexpr int kRopeStages = 6;
struct RopeArgs {
    const __nv_bfloat16* qkv;
    int64_t qkv_stride;
    int rows, H, G, Gv, dk, dv, v_from_k, rot_dims;
    const int32_t* positions;
    const float* cos_sin;
    int max_pos;
    const int64_t* slots;
    int bs, bs_log2;                                 // bs_log2 < 0: bs is no power of two
    const float *q_w, *k_w;
    float eps;
    __nv_bfloat16 *q_out, *k_cache, *v_cache;
    __host__ __device__ int width() const { return (H + G) * dk + (v_from_k ? 0 : Gv * dv); }
    __host__ __device__ int stage_bytes() const { return (width() * 2 + rot_dims * 4 + 127) / 128 * 128; }
};

template <bool NORM, bool INTERLEAVED, bool RING>
__global__ void __launch_bounds__(1024)
qk_rope_cache_rows_kernel(const RopeArgs p) {
    extern __shared__ __align__(128) unsigned char rope_sm[];
    __shared__ __align__(8) uint64_t s_full[kRopeStages];
    __shared__ float red[2][2][32];                  // [row's parity][q, k][warp]
    __shared__ int s_failed;
    using bf16 = __nv_bfloat16;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, dk = p.dk, per = dk / 16, half = p.rot_dims / 2;
    const bool mine = tid < (p.H + p.G) * per;
    const int hd = mine ? tid / per : 0, j = tid - (tid / per) * per;
    const bool pairs = !INTERLEAVED && j < half / 8, is_q = hd < p.H;
    const int ia = pairs ? 8 * j : INTERLEAVED ? 16 * j : p.rot_dims + 16 * (j - half / 8), ib = pairs ? ia + half : ia + 8;
    const bool turns = mine && (INTERLEAVED ? ia < p.rot_dims : pairs);
    const int count = RING ? (p.rows - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 1, stage = p.stage_bytes(), row_bytes = p.width() * 2;
    auto position = [&](int row) {
        const int pos = p.positions[row];
        return pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
    };
    auto full = [&](int s) { return b2::smem_u32(&s_full[s]); };
    auto fetch = [&](int n, int pos) {               // one thread
        const uint32_t dst = b2::smem_u32(rope_sm) + n % kRopeStages * stage, bar = full(n % kRopeStages);
        b2::mbar_arrive_expect_tx(bar, row_bytes + p.rot_dims * 4);
        b2::bulk_load(dst, p.qkv + (size_t)(blockIdx.x + n * gridDim.x) * p.qkv_stride, row_bytes, bar);
        if (p.rot_dims) b2::bulk_load(dst + row_bytes, p.cos_sin + (size_t)pos * p.rot_dims, p.rot_dims * 4, bar);
    };
    int ahead_pos = 0;                               // thread 0: position of the next row to be fetched
    if (NORM && tid < 128) red[tid >> 6][(tid >> 5) & 1][lane] = 0.f;
    if (RING && tid == 0) {
        s_failed = 0;
        for (int s = 0; s < kRopeStages; ++s) b2::mbar_init(full(s), 1);
        b2::fence_mbar_init();
        for (int n = 0; n < min(count, kRopeStages); ++n) fetch(n, position(blockIdx.x + n * gridDim.x));
        if (count > kRopeStages) ahead_pos = position(blockIdx.x + kRopeStages * gridDim.x);
    }
    if (RING || NORM) __syncthreads();
    float wa[8], wb[8];
    if (NORM && mine) {
        const float* w = is_q ? p.q_w + (size_t)hd * dk : p.k_w + (size_t)(hd - p.H) * dk;
#pragma unroll
        for (int c = 0; c < 8; c += 4) {
            const float4 u = *reinterpret_cast<const float4*>(w + ia + c), v = *reinterpret_cast<const float4*>(w + ib + c);
            wa[c] = u.x; wa[c + 1] = u.y; wa[c + 2] = u.z; wa[c + 3] = u.w;
            wb[c] = v.x; wb[c + 1] = v.y; wb[c + 2] = v.z; wb[c + 3] = v.w;
        }
    }
    const bool some_q = __any_sync(0xffffffffu, mine && is_q), some_k = __any_sync(0xffffffffu, mine && !is_q);
    int64_t next_slot = p.slots[blockIdx.x];
    for (int n = 0; n < count; ++n) {
        const int row = blockIdx.x + n * gridDim.x;
        const int64_t slot = next_slot;
        if (RING && n + 1 < count) next_slot = p.slots[row + gridDim.x];
        const unsigned char* src = RING ? rope_sm + n % kRopeStages * stage : reinterpret_cast<const unsigned char*>(p.qkv + (size_t)row * p.qkv_stride);
        const float* cs = RING ? reinterpret_cast<const float*>(src + row_bytes) : p.cos_sin + (turns ? (size_t)position(row) * p.rot_dims : 0);
        if (RING) b2tc::wait(full(n % kRopeStages), n / kRopeStages & 1, &s_failed);
        const bf16* head = reinterpret_cast<const bf16*>(src) + hd * dk;
        uint4 ra = make_uint4(0, 0, 0, 0), rb = ra, rv = ra;
        if (mine) {
            ra = *reinterpret_cast<const uint4*>(head + ia);
            rb = *reinterpret_cast<const uint4*>(head + ib);
        }
        const bool own_v = !p.v_from_k && tid < p.Gv * p.dv / 8;
        if (own_v) rv = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(src) + (p.H + p.G) * dk + tid * 8);
        float co[8], si[8];
        if (turns)
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
                const float4 u = *reinterpret_cast<const float4*>(cs + 8 * j + c), v = *reinterpret_cast<const float4*>(cs + half + 8 * j + c);
                co[c] = u.x; co[c + 1] = u.y; co[c + 2] = u.z; co[c + 3] = u.w;
                si[c] = v.x; si[c + 1] = v.y; si[c + 2] = v.z; si[c + 3] = v.w;
            }
        float x[8], y[8];
        {
            const uint32_t u[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                x[2 * c] = __uint_as_float(u[c] << 16);
                x[2 * c + 1] = __uint_as_float(u[c] & 0xffff0000u);
                y[2 * c] = __uint_as_float(u[4 + c] << 16);
                y[2 * c + 1] = __uint_as_float(u[4 + c] & 0xffff0000u);
            }
        }
        float (&part)[2][32] = red[n & 1];
        if (NORM) {
            float s = 0.f;
#pragma unroll
            for (int c = 0; c < 8; ++c) s = fmaf(x[c], x[c], fmaf(y[c], y[c], s));
            if (some_q) {
                const float t = b2::warp_sum(is_q ? s : 0.f);
                if (lane == 0) part[0][wid] = t;
            }
            if (some_k) {
                const float t = b2::warp_sum(is_q ? 0.f : s);
                if (lane == 0) part[1][wid] = t;
            }
        }
        if (NORM || RING) __syncthreads();           // the row is read; its sums are there (two sets of them: the next row's are not these)
        if (RING && tid == 0 && n + kRopeStages < count && !*(volatile int*)&s_failed) {
            fetch(n + kRopeStages, ahead_pos);
            if (n + kRopeStages + 1 < count) ahead_pos = position(row + (kRopeStages + 1) * gridDim.x);
        }
        if (NORM) {
            float t = 0.f;
            if (some_q) t = b2::warp_sum(part[0][lane]);
            if (some_k) {
                const float tk = b2::warp_sum(part[1][lane]);
                if (!is_q) t = tk;
            }
            const float inv = rsqrtf(t / (float)((is_q ? p.H : p.G) * dk) + p.eps);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                x[c] *= inv * wa[c];
                y[c] *= inv * wb[c];
            }
        }
        if (turns) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (!INTERLEAVED) {
                    const float u = x[c], v = y[c];
                    x[c] = fmaf(u, co[c], -v * si[c]);
                    y[c] = fmaf(v, co[c], u * si[c]);
                } else if (c % 2 == 0) {
                    const float u = x[c], v = x[c + 1], u2 = y[c], v2 = y[c + 1];
                    x[c] = fmaf(u, co[c / 2], -v * si[c / 2]);
                    x[c + 1] = fmaf(v, co[c / 2], u * si[c / 2]);
                    y[c] = fmaf(u2, co[4 + c / 2], -v2 * si[4 + c / 2]);
                    y[c + 1] = fmaf(v2, co[4 + c / 2], u2 * si[4 + c / 2]);
                }
            }
        }
        if (RING && *(volatile int*)&s_failed) {
#pragma unroll
            for (int c = 0; c < 8; ++c) x[c] = y[c] = __int_as_float(0x7fc00000);
        }
        int64_t blk = 0;
        int off = 0;
        if (slot >= 0) {
            if (p.bs_log2 >= 0) { blk = slot >> p.bs_log2; off = (int)slot & (p.bs - 1); }
            else { blk = slot / p.bs; off = (int)(slot % p.bs); }
        }
        if (mine && (is_q || slot >= 0)) {
            const size_t pool = ((size_t)blk * p.G + (hd - p.H)) * p.bs + off;
            bf16* dst = is_q ? p.q_out + ((size_t)row * p.H + hd) * dk : p.k_cache + pool * dk;
            b2::st8(dst + ia, x);
            b2::st8(dst + ib, y);
            if (p.v_from_k && !is_q) {               // a value head per key head, of its size
                *reinterpret_cast<uint4*>(p.v_cache + pool * p.dv + ia) = ra;
                *reinterpret_cast<uint4*>(p.v_cache + pool * p.dv + ib) = rb;
            }
        }
        if (own_v && slot >= 0) {
            const int g = tid * 8 / p.dv, i = tid * 8 - g * p.dv;
            *reinterpret_cast<uint4*>(p.v_cache + (((size_t)blk * p.Gv + g) * p.bs + off) * p.dv + i) = rv;
        }
    }
    if (RING && *(volatile int*)&s_failed)           // what is still on its way to this CTA's memory
        for (int n = max(0, count - kRopeStages); n < count; ++n) b2tc::drain(full(n % kRopeStages), n / kRopeStages & 1);
}

template <typename T>
__global__ void qknorm_cache_kernel(const T* __restrict__ qkv, int64_t qkv_stride, int H, int G, int dk, int dv,
                                    const float* __restrict__ q_w, const float* __restrict__ k_w, float eps,
                                    const int64_t* __restrict__ slots, int bs, T* __restrict__ q_out,
                                    T* __restrict__ k_cache, T* __restrict__ v_cache, bool norm,
                                    const int32_t* __restrict__ positions, float temp_coef, int temp_every) {
    const int row = blockIdx.x;
    float q_factor = 1.f;
    if (positions && temp_coef != 0.f) q_factor = 1.f + temp_coef * logf((float)((positions[row] + 1) / temp_every + 1));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const T* src = qkv + (size_t)row * qkv_stride;
    const int64_t slot = slots[row];
    const int64_t blk = slot >= 0 ? slot / bs : 0;
    const int off = slot >= 0 ? (int)(slot % bs) : 0;
    for (int hd = wid; hd < H + 2 * G; hd += nw) {
        if (hd < H + G) {                            // q or k head: x / sqrt(mean(x^2) + eps) * w
            const T* v = src + (size_t)hd * dk;
            float inv = hd < H ? q_factor : 1.f;
            if (norm) {
                float ss = 0.f;
                for (int i = lane; i < dk; i += 32) {
                    const float x = b2::ld(v + i);
                    ss = fmaf(x, x, ss);
                }
                inv = rsqrtf(b2::warp_sum(ss) / (float)dk + eps) * (hd < H ? q_factor : 1.f);
            }
            T* dst;
            const float* w;
            if (hd < H) {
                dst = q_out + ((size_t)row * H + hd) * dk;
                w = q_w;
            } else {
                if (slot < 0) continue;
                dst = k_cache + (((size_t)blk * G + (hd - H)) * bs + off) * dk;
                w = k_w;
            }
            for (int i = lane; i < dk; i += 32) b2::st(dst + i, b2::ld(v + i) * inv * (w ? w[i] : 1.f));
        } else {
            if (slot < 0) continue;
            const int g = hd - H - G;
            const T* v = src + (size_t)(H + G) * dk + (size_t)g * dv;
            T* dst = v_cache + (((size_t)blk * G + g) * bs + off) * dv;
            for (int i = lane; i < dv; i += 32) dst[i] = v[i];
        }
    }
}

template <typename T, bool SIG, int MAPS>
__global__ void chunk_attention_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                                       const int32_t* __restrict__ block_tables, int max_nb,
                                       const int32_t* __restrict__ cu_q, const int32_t* __restrict__ ctx_start, int n_seq,
                                       int rows, int H, int G, int dk, int dv, int bs, float scale, int chunk, int window,
                                       int keep_first, float sink, float sink_logit, const float* __restrict__ sink_logits,
                                       const float* __restrict__ head_bias, const T* __restrict__ gate, int64_t gate_stride,
                                       HeadShape hs, int skip_rows_from, T* __restrict__ out, int64_t out_stride) {
    extern __shared__ float q_sm[];                  // [warps, dk]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int item = blockIdx.x * (blockDim.x >> 5) + wid;       // (row, head)
    if (item >= rows * H) return;
    const int row = item / H, hh = item % H;
    const int seq = b2::seq_of_row(cu_q, n_seq, row);
    const int ctx = ctx_start[seq];
    T* dst = out + (size_t)row * out_stride + (size_t)hh * dv;
    if (skip_rows_from > 0 && ctx >= 0 && cu_q[seq + 1] - cu_q[seq] >= skip_rows_from) return;    // the tile kernel's
    if (ctx < 0) {
        for (int i = lane; i < dv; i += 32) b2::st(dst + i, 0.f);
        return;
    }
    const int pos = ctx + row - cu_q[seq];
    const KeySpan span = key_span(pos, pos, chunk, window, keep_first);
    const int g = hh / (H / G);
    float* qs = q_sm + (size_t)wid * dk;
    const int32_t* bt = block_tables + (size_t)seq * max_nb;
    const float bias = SIG && head_bias ? head_bias[hh] : 0.f;
    float first[MAPS > 1 ? kMaxDvPerLane : 1];       // the first map's output
    float acc[kMaxDvPerLane];
    float inv = 1.f;
#pragma unroll
    for (int mp = 0; mp < MAPS; ++mp) {
        const T* qv = q + ((size_t)item * MAPS + mp) * dk;
        __syncwarp();
        for (int i = lane; i < dk; i += 32) qs[i] = b2::ld(qv + i) * scale;
        __syncwarp();
        float m = sink > 0.f ? (sink_logits ? sink_logits[hh] : sink_logit) : -INFINITY, l = sink;      // the sink seeds the running maximum and denominator
#pragma unroll
        for (int c = 0; c < kMaxDvPerLane; ++c) acc[c] = 0.f;
        for (int c0 = 0; c0 < span.n; c0 += 32) {
            const bool in = c0 + lane < span.n;
            const int j = span.key(c0 + lane);
            float s = -INFINITY;
            size_t vbase = 0;
            if (in) {
                const size_t page = bt[j / bs];
                const T* kr = k_cache + ((page * (G * MAPS) + g * MAPS + mp) * bs + (j % bs)) * dk;
                vbase = ((page * G + g) * bs + (j % bs)) * dv;
                float d = 0.f;
                for (int i = 0; i < dk; ++i) d = fmaf(qs[i], b2::ld(kr + i), d);
                s = hs.cap > 0.f ? cap_score_exact(d, hs.cap) : d;
            }
            float p;
            if (SIG) {
                p = in ? b2::sigmoid_f(s + bias) : 0.f;
            } else {
                const float m_new = fmaxf(m, b2::warp_max(s));
                const float corr = m == -INFINITY ? 0.f : __expf(m - m_new);
                p = in ? __expf(s - m_new) : 0.f;
                l = l * corr + b2::warp_sum(p);
                m = m_new;
#pragma unroll
                for (int c = 0; c < kMaxDvPerLane; ++c) acc[c] *= corr;
            }
            const int nk = min(32, span.n - c0);
            for (int kk = 0; kk < nk; ++kk) {
                const float pk = __shfl_sync(0xffffffffu, p, kk);
                const size_t vb = __shfl_sync(0xffffffffu, (unsigned long long)vbase, kk);
                const T* vr = v_cache + vb;
#pragma unroll
                for (int c = 0; c < kMaxDvPerLane; ++c) {
                    const int i = lane + 32 * c;
                    if (i < dv) acc[c] = fmaf(pk, b2::ld(vr + i), acc[c]);
                }
            }
        }
        inv = SIG ? 1.f : (l > 0.f ? 1.f / l : 0.f);
        if (MAPS > 1 && mp == 0) {
#pragma unroll
            for (int c = 0; c < kMaxDvPerLane; ++c) first[MAPS > 1 ? c : 0] = acc[c] * inv;
        }
    }
    if (MAPS > 1) {
        float ss = 0.f;
#pragma unroll
        for (int c = 0; c < kMaxDvPerLane; ++c) {
            acc[c] = first[MAPS > 1 ? c : 0] - hs.lambda * (acc[c] * inv);
            ss = fmaf(acc[c], acc[c], ss);           // columns past dv hold zeros
        }
        inv = rsqrtf(b2::warp_sum(ss) / (float)dv + hs.eps) * hs.out_scale;
    }
    if (gate) inv *= b2::sigmoid_f(b2::ld(gate + (size_t)row * gate_stride + hh));
#pragma unroll
    for (int c = 0; c < kMaxDvPerLane; ++c) {
        const int i = lane + 32 * c;
        if (i < dv) b2::st(dst + i, acc[c] * inv);
    }
}

// ------------------------------------------------------------------------------------------------- grouped decode kernel
// bf16 rows that neither tensor-core kernel takes (decode rows and short portions of other head sizes): one CTA per (row, kv head) serves ALL the
// query heads of that kv head, so K and V are read once per group instead of once per head.  Four warps share the visible
// keys 32 at a time (a lane per key, 16-byte loads of its K row, one dot product per query head), keep an online softmax
// per head, accumulate P.V with a lane per pair of value columns, and merge through shared memory; the sink enters
// through warp 0's initial state.  Up to kGroupMaxHeads query heads per pass (more: further passes over the keys).  With two
// maps the pass holds the heads' maps one after the other (an even number) and a key's two halves lie side by side in the tile.
constexpr int kGroupMaxHeads = 8, kGroupMaxPairs = 4;      // dv <= 256

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(b2::smem_u32(dst)), "l"(src) : "memory");
}

template <bool SIG, int MAPS>
__global__ void __launch_bounds__(128)
chunk_attention_group_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_cache,
                             const __nv_bfloat16* __restrict__ v_cache, const int32_t* __restrict__ block_tables, int max_nb,
                             const int32_t* __restrict__ cu_q, const int32_t* __restrict__ ctx_start, int n_seq, int H, int G,
                             int dk, int dv, int bs, float scale, int chunk, int window, int keep_first, float sink,
                             float sink_logit, const float* __restrict__ sink_logits, const float* __restrict__ head_bias,
                             const __nv_bfloat16* __restrict__ gate, int64_t gate_stride, HeadShape hs, int skip_rows_from,
                             __nv_bfloat16* __restrict__ out, int64_t out_stride) {
    // q [QH][dk] | per warp: m [QH], l [QH], acc [QH][dv] | per warp: K tile [32][MAPS * dk + 8], V tile [32][dv] (bf16)
    extern __shared__ __align__(16) float grp_sm[];
    const int row = blockIdx.x, g = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int seq = b2::seq_of_row(cu_q, n_seq, row);
    const int ctx = ctx_start[seq];
    const int QHall = H / G;                               // query heads of this key head
    const int VHall = QHall * MAPS;                        // ... each with its maps
    if (skip_rows_from > 0 && ctx >= 0 && cu_q[seq + 1] - cu_q[seq] >= skip_rows_from) return;    // the tile kernel's
    if (ctx < 0) {
        for (int i = tid; i < QHall * dv; i += 128)
            out[(size_t)row * out_stride + (size_t)g * QHall * dv + i] = __float2bfloat16_rn(0.f);
        return;
    }
    const int pos = ctx + row - cu_q[seq];
    const KeySpan span = key_span(pos, pos, chunk, window, keep_first);
    const int32_t* bt = block_tables + (size_t)seq * max_nb;
    const int npairs = dv / 2;
    for (int h0 = 0; h0 < VHall; h0 += kGroupMaxHeads) {
        const int QH = min(kGroupMaxHeads, VHall - h0);
        float* qs = grp_sm;
        float* part = grp_sm + kGroupMaxHeads * dk;
        const int ldk = MAPS * dk + 8;                     // 16 bytes of padding: the lanes' rows spread over the banks
        __nv_bfloat16* kt = reinterpret_cast<__nv_bfloat16*>(part + 4 * kGroupMaxHeads * (2 + dv)) + (size_t)w * 32 * (ldk + dv);
        __nv_bfloat16* vt = kt + 32 * ldk;
        __syncthreads();                                   // a previous pass is done with the shared memory
        for (int i = tid; i < QH * dk; i += 128)
            qs[i] = __bfloat162float(q[((size_t)row * H * MAPS + (size_t)g * VHall + h0) * dk + i]) * scale;
        __syncthreads();
        float m[kGroupMaxHeads], l[kGroupMaxHeads], acc[kGroupMaxHeads][kGroupMaxPairs][2];
#pragma unroll
        for (int h = 0; h < kGroupMaxHeads; ++h) {
            m[h] = (w == 0 && sink > 0.f) ? (sink_logits ? sink_logits[g * QHall + (h0 + min(h, QH - 1)) / MAPS] : sink_logit) : -INFINITY;
            l[h] = w == 0 ? sink : 0.f;
            if (SIG) m[h] = head_bias ? head_bias[g * QHall + (h0 + min(h, QH - 1)) / MAPS] : 0.f;      // holds the head's bias instead
#pragma unroll
            for (int c = 0; c < kGroupMaxPairs; ++c) acc[h][c][0] = acc[h][c][1] = 0.f;
        }
        for (int c0 = w * 32; c0 < span.n; c0 += 128) {
            const bool valid = c0 + lane < span.n;
            float sc[kGroupMaxHeads];
#pragma unroll
            for (int h = 0; h < kGroupMaxHeads; ++h) sc[h] = 0.f;
            // the warp's 32 keys: K and V rows gathered from the pages with every 16-byte copy in flight at once
            const int nk = min(32, span.n - c0);
            __syncwarp();                                  // the previous tile has been read
            for (int idx = lane; idx < nk * MAPS * (dk / 8); idx += 32) {
                const int part_ = idx / (dk / 8), c = (idx % (dk / 8)) * 8, key = part_ / MAPS, mp = part_ % MAPS, jk = span.key(c0 + key);
                cp_async16(kt + key * ldk + mp * dk + c,
                           k_cache + (((size_t)bt[jk / bs] * (G * MAPS) + g * MAPS + mp) * bs + jk % bs) * dk + c);
            }
            for (int idx = lane; idx < nk * (dv / 8); idx += 32) {
                const int key = idx / (dv / 8), c = (idx % (dv / 8)) * 8, jk = span.key(c0 + key);
                cp_async16(vt + key * dv + c, v_cache + (((size_t)bt[jk / bs] * G + g) * bs + jk % bs) * dv + c);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();
            if (valid) {
#pragma unroll
                for (int mp = 0; mp < MAPS; ++mp) {
                    const __nv_bfloat16* kr = kt + lane * ldk + mp * dk;
                    for (int c = 0; c < dk; c += 8) {
                        const uint4 raw = *reinterpret_cast<const uint4*>(kr + c);
                        const uint32_t wds[4] = {raw.x, raw.y, raw.z, raw.w};
                        float kf[8];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            kf[2 * e] = __uint_as_float(wds[e] << 16);
                            kf[2 * e + 1] = __uint_as_float(wds[e] & 0xffff0000u);
                        }
#pragma unroll
                        for (int h = mp; h < kGroupMaxHeads; h += MAPS) {
                            if (h < QH) {
                                const float4 qa = *reinterpret_cast<const float4*>(qs + h * dk + c);
                                const float4 qb = *reinterpret_cast<const float4*>(qs + h * dk + c + 4);
                                sc[h] = fmaf(qa.x, kf[0], sc[h]); sc[h] = fmaf(qa.y, kf[1], sc[h]);
                                sc[h] = fmaf(qa.z, kf[2], sc[h]); sc[h] = fmaf(qa.w, kf[3], sc[h]);
                                sc[h] = fmaf(qb.x, kf[4], sc[h]); sc[h] = fmaf(qb.y, kf[5], sc[h]);
                                sc[h] = fmaf(qb.z, kf[6], sc[h]); sc[h] = fmaf(qb.w, kf[7], sc[h]);
                            }
                        }
                    }
                }
                if (hs.cap > 0.f) {
                    const float e_scale = 2.8853900817779268f / hs.cap;         // 2 log2(e) / cap
#pragma unroll
                    for (int h = 0; h < kGroupMaxHeads; ++h) sc[h] = cap_score(sc[h], hs.cap, e_scale);
                }
            }
            float pr[kGroupMaxHeads];
#pragma unroll
            for (int h = 0; h < kGroupMaxHeads; ++h) {
                pr[h] = 0.f;
                if (SIG) {
                    if (h < QH && valid) pr[h] = b2::sigmoid_f(sc[h] + m[h]);
                } else if (h < QH) {
                    const float x = valid ? sc[h] : -INFINITY;
                    const float mn = fmaxf(m[h], b2::warp_max(x));          // finite: the tile has at least one key
                    const float corr = m[h] == -INFINITY ? 0.f : __expf(m[h] - mn);
                    pr[h] = valid ? __expf(x - mn) : 0.f;
                    l[h] = l[h] * corr + b2::warp_sum(pr[h]);
                    m[h] = mn;
#pragma unroll
                    for (int c = 0; c < kGroupMaxPairs; ++c) {
                        acc[h][c][0] *= corr;
                        acc[h][c][1] *= corr;
                    }
                }
            }
            for (int kk = 0; kk < nk; ++kk) {
                float vx[kGroupMaxPairs], vy[kGroupMaxPairs];
#pragma unroll
                for (int c = 0; c < kGroupMaxPairs; ++c) {
                    const int pi = lane + 32 * c;
                    vx[c] = vy[c] = 0.f;
                    if (pi < npairs) {
                        const uint32_t wd = *reinterpret_cast<const uint32_t*>(vt + kk * dv + 2 * pi);
                        vx[c] = __uint_as_float(wd << 16);
                        vy[c] = __uint_as_float(wd & 0xffff0000u);
                    }
                }
#pragma unroll
                for (int h = 0; h < kGroupMaxHeads; ++h) {
                    if (h < QH) {
                        const float ph = __shfl_sync(0xffffffffu, pr[h], kk);
#pragma unroll
                        for (int c = 0; c < kGroupMaxPairs; ++c) {
                            acc[h][c][0] = fmaf(ph, vx[c], acc[h][c][0]);
                            acc[h][c][1] = fmaf(ph, vy[c], acc[h][c][1]);
                        }
                    }
                }
            }
        }
        // merge the four warps
        float* mine = part + (size_t)w * kGroupMaxHeads * (2 + dv);
#pragma unroll
        for (int h = 0; h < kGroupMaxHeads; ++h) {
            if (h < QH) {
                if (lane == 0) {
                    mine[h * (2 + dv)] = m[h];
                    mine[h * (2 + dv) + 1] = l[h];
                }
#pragma unroll
                for (int c = 0; c < kGroupMaxPairs; ++c) {
                    const int pi = lane + 32 * c;
                    if (pi < npairs) {
                        mine[h * (2 + dv) + 2 + 2 * pi] = acc[h][c][0];
                        mine[h * (2 + dv) + 3 + 2 * pi] = acc[h][c][1];
                    }
                }
            }
        }
        __syncthreads();
        // output of (virtual) head h at column col
        auto merged = [&](int h, int col) {
            float M = -INFINITY, L = 0.f, O = 0.f;
            if (SIG) {
                L = 1.f;
                for (int x = 0; x < 4; ++x) O += part[((size_t)x * kGroupMaxHeads + h) * (2 + dv) + 2 + col];
            } else {
                for (int x = 0; x < 4; ++x) M = fmaxf(M, part[((size_t)x * kGroupMaxHeads + h) * (2 + dv)]);
            }
            if (!SIG && M > -INFINITY) {
                for (int x = 0; x < 4; ++x) {
                    const float* px = part + ((size_t)x * kGroupMaxHeads + h) * (2 + dv);
                    const float f = px[0] == -INFINITY ? 0.f : __expf(px[0] - M);
                    L = fmaf(px[1], f, L);
                    O = fmaf(px[2 + col], f, O);
                }
            }
            return L > 0.f ? O / L : 0.f;
        };
        if (MAPS == 1) {
            for (int i = tid; i < QH * dv; i += 128) {
                const int h = i / dv, col = i % dv;
                float res = merged(h, col);
                if (gate) res *= b2::sigmoid_f(__bfloat162float(gate[(size_t)row * gate_stride + (size_t)g * QHall + h0 + h]));
                out[(size_t)row * out_stride + ((size_t)g * QHall + h0 + h) * dv + col] = __float2bfloat16_rn(res);
            }
        } else {
            for (int h = w; h < QH / MAPS; h += 4) {           // a warp per head: the norm runs over its dv columns
                const size_t head = (size_t)g * QHall + h0 / MAPS + h;
                float v[2 * kGroupMaxPairs], ss = 0.f;
#pragma unroll
                for (int c = 0; c < 2 * kGroupMaxPairs; ++c) {
                    const int col = lane + 32 * c;
                    v[c] = col < dv ? merged(h * MAPS, col) - hs.lambda * merged(h * MAPS + MAPS - 1, col) : 0.f;
                    ss = fmaf(v[c], v[c], ss);
                }
                float inv = rsqrtf(b2::warp_sum(ss) / (float)dv + hs.eps) * hs.out_scale;
                if (gate) inv *= b2::sigmoid_f(__bfloat162float(gate[(size_t)row * gate_stride + head]));
#pragma unroll
                for (int c = 0; c < 2 * kGroupMaxPairs; ++c) {
                    const int col = lane + 32 * c;
                    if (col < dv) out[(size_t)row * out_stride + head * dv + col] = __float2bfloat16_rn(v[c] * inv);
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------- head-tile decode kernel
// The same rows for head sizes the tensor cores take (dk a multiple of 32, dv one of the prompt kernel's sizes): one CTA per
// (row, kv head), the query heads of that kv head as the rows of a 16-row operand (two maps: rows 0 - 7 hold the first maps of
// eight heads, rows 8 - 15 their second), so a K or V row is read once and multiplied for all of them at once.  NW warps take
// 16 visible keys at a time each, gather their K and V rows from the pages with cp.async (four lanes a row, one page lookup per
// key, a tile ahead), run S = Q K^T and O += P V on mma.sync with the softmax in the accumulator registers, and merge through shared
// memory, which by then no longer holds tiles.  The keys a single row sees are one exact range: nothing to mask but its end.
// Bound: the bytes of K and V.  A warp has one buffer for K and one for V and refills each as soon as it is multiplied, so one of the
// two is always in flight under the other's arithmetic; 16 keys a tile and 128 registers let 16 warps share an SM.  With 32 keys
// copied and then multiplied, three CTAs of four warps an SM, 64 rows x 8 kv heads x 1028 keys of 128 took 73 us: two waves, each
// warp idle while its tile arrived (62 us with this form, 60 with the keys as rows, below).  NW is 16, 8 or 4 so that a small batch's rows are still shared by 16 warps an SM.
constexpr int kHeadRows = 16, kHeadKeys = 16;

// At most eight query heads a kv head (and one map, dk <= 128): the keys are the 16 rows of the operand and the heads its 8 columns,
// S^T = K Q^T and O^T += V^T P^T.  No half of the tile is padding: half the products, scores, rescales and accumulators of the form
// below, Q in registers, and P^T turns into an operand by 8 x 8 transpositions.  Keys of 64
// numbers and less go 32 at a time: the same bytes in flight as 16 of 128, and the weights' rounding is that of tiles of 32, which these
// sizes always had (a router behind such a layer may stand within it of another choice).  128 rows x 8 kv heads x 2000 keys of 64: 92 us,
// 108 in tiles of 16.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
    uint32_t y;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}

constexpr int kFewHeads = 8, kFewDk = 128, kShortDk = 64;

template <int DVT, bool SIG, int NW, int KEYS>
__global__ void __launch_bounds__(32 * NW, DVT <= 8 && NW < 16 && KEYS == kHeadKeys ? 20 / NW : 16 / NW)
chunk_attention_few_heads_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_cache,
                             const __nv_bfloat16* __restrict__ v_cache, const int32_t* __restrict__ block_tables, int max_nb,
                             const int32_t* __restrict__ cu_q, const int32_t* __restrict__ ctx_start, int n_seq, int H, int G,
                             int dk, int bs, float scale_log2, int chunk, int window, int keep_first, float sink,
                             float sink_logit, const float* __restrict__ sink_logits, const float* __restrict__ head_bias,
                             const __nv_bfloat16* __restrict__ gate, int64_t gate_stride, HeadShape hs, int skip_rows_from, bool by_seq,
                             __nv_bfloat16* __restrict__ out, int64_t out_stride) {
    constexpr int DV = 16 * DVT, LDV = DV + 8, PW = 2 + DV, NTH = 32 * NW, MAXDK = KEYS > kHeadKeys ? kShortDk : kFewDk;
    constexpr float kLog2e = 1.4426950408889634f;
    // q [8][dk + 8], then per warp: K tile [KEYS][dk + 8], V tile [KEYS][DV + 8]; the merge reuses the tiles' place
    extern __shared__ __align__(16) unsigned char head_sm[];
    const int g = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int QHall = H / G;
    // by_seq: a batch with prompt portions for the tile kernel -- the CTAs are the up to skip_rows_from - 1 rows of every short sequence
    const int per = skip_rows_from - 1;
    const int seq = by_seq ? blockIdx.x / per : b2::seq_of_row(cu_q, n_seq, blockIdx.x);
    const int r0 = cu_q[seq], len = cu_q[seq + 1] - r0;
    int row = by_seq ? r0 + blockIdx.x % per : blockIdx.x;
    const int ctx = ctx_start[seq];
    if (by_seq && row >= r0 + len) return;
    if (skip_rows_from > 0 && ctx >= 0 && len >= skip_rows_from) return;         // the tile kernel's
    if (ctx < 0) {
        do {
            for (int i = tid; i < QHall * DV; i += NTH)
                out[(size_t)row * out_stride + (size_t)g * QHall * DV + i] = __float2bfloat16_rn(0.f);
        } while (by_seq && (row += per) < r0 + len);
        return;
    }
    const int pos = ctx + row - r0;
    const KeySpan span = key_span(pos, pos, chunk, window, keep_first);
    const int32_t* bt = block_tables + (size_t)seq * max_nb;
    const int ldq = dk + 8, ldk = dk + 8;
    __nv_bfloat16* q_sm = reinterpret_cast<__nv_bfloat16*>(head_sm);
    __nv_bfloat16* tiles = q_sm + kFewHeads * ldq;
    __nv_bfloat16* kt = tiles + (size_t)w * KEYS * (ldk + LDV);
    __nv_bfloat16* vt = kt + KEYS * ldk;
    float* part = reinterpret_cast<float*>(tiles);       // [NW][8][m, l, O (DV)]
    const uint32_t q_base = b2::smem_u32(q_sm), k_base = b2::smem_u32(kt), v_base = b2::smem_u32(vt);
    const int gq = lane >> 2, tq = lane & 3;
    const float cap_log2 = hs.cap * kLog2e, cap_e = hs.cap > 0.f ? 2.f / hs.cap : 0.f;
    constexpr int STEP = NW * KEYS;

    // keys past the end repeat the last one: finite numbers that the mask drops
    auto key_at = [&](int c) { return span.key(min(c + (lane & (KEYS - 1)), span.n - 1)); };
    auto page_of = [&](int j, int& off) {
        const int pg = j / bs;
        off = j - pg * bs;
        return bt[pg];
    };
    int off, page, next_off = 0, next_page = 0;      // of the tile in flight, and of the one behind it
    auto issue_k = [&]() {
#pragma unroll
        for (int kq = 0; kq < KEYS / 8; ++kq) {
            const int key = kq * 8 + (lane >> 2), c = (lane & 3) * 8;
            const size_t pg = __shfl_sync(0xffffffffu, page, key);
            const int of = __shfl_sync(0xffffffffu, off, key);
            const __nv_bfloat16* ks = k_cache + ((pg * G + g) * bs + of) * dk + c;
            __nv_bfloat16* kd = kt + key * ldk + c;
#pragma unroll
            for (int t = 0; t < MAXDK; t += 32)
                if (t < dk) cp_async16(kd + t, ks + t);
        }
    };
    auto issue_v = [&]() {
#pragma unroll
        for (int kq = 0; kq < KEYS / 8; ++kq) {
            const int key = kq * 8 + (lane >> 2), c = (lane & 3) * 8;
            const size_t pg = __shfl_sync(0xffffffffu, page, key);
            const int of = __shfl_sync(0xffffffffu, off, key);
            const __nv_bfloat16* vs = v_cache + ((pg * G + g) * bs + of) * DV + c;
            __nv_bfloat16* vd = vt + key * LDV + c;
#pragma unroll
            for (int t = 0; t < DV; t += 32) cp_async16(vd + t, vs + t);
        }
    };
    const int first = w * KEYS;
    if (first < span.n) {
        page = page_of(key_at(first), off);
        issue_k();
        asm volatile("cp.async.commit_group;" ::: "memory");
        issue_v();
        asm volatile("cp.async.commit_group;" ::: "memory");
        next_page = page_of(key_at(first + STEP), next_off);
    }
    for (int idx = tid; idx < kFewHeads * (dk / 8); idx += NTH) {
        const int r = idx / (dk / 8), c = (idx % (dk / 8)) * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < QHall) v = *reinterpret_cast<const uint4*>(q + ((size_t)row * H + (size_t)g * QHall + r) * dk + c);
        *reinterpret_cast<uint4*>(q_sm + r * ldq + c) = v;
    }
    __syncthreads();
    uint32_t qf[MAXDK / 16][2];
#pragma unroll
    for (int kk = 0; kk < MAXDK / 16; kk += 2) {
        qf[kk][0] = qf[kk][1] = qf[kk + 1][0] = qf[kk + 1][1] = 0u;
        if (kk * 16 < dk) b2::ldmatrix_x4(q_base + 2u * ((lane & 7) * ldq + kk * 16 + (lane >> 3) * 8), qf[kk][0], qf[kk][1], qf[kk + 1][0], qf[kk + 1][1]);
    }
    // this thread's two heads (of S^T and O^T columns 2 tq and 2 tq + 1)
    const int ha = g * QHall + min(2 * tq, QHall - 1), hb = g * QHall + min(2 * tq + 1, QHall - 1);
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f, ba = 0.f, bb = 0.f;
    if (w == 0 && sink > 0.f) {                      // the sink enters once, through the first warp
        m0 = (sink_logits ? sink_logits[ha] : sink_logit) * kLog2e;
        m1 = (sink_logits ? sink_logits[hb] : sink_logit) * kLog2e;
        l0 = l1 = gq == 0 ? sink : 0.f;
    }
    if (SIG && head_bias) {
        ba = head_bias[ha] * kLog2e;
        bb = head_bias[hb] * kLog2e;
    }
    float o[DVT][4];
#pragma unroll
    for (int n = 0; n < DVT; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

    for (int c0 = first; c0 < span.n; c0 += STEP) {
        const bool more = c0 + STEP < span.n;
        asm volatile("cp.async.wait_group 1;" ::: "memory");     // K is there, V may still be on its way
        __syncwarp();
        float sc[KEYS / 16][4][4];                   // four chains
#pragma unroll
        for (int n = 0; n < KEYS / 16; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) sc[n][c][0] = sc[n][c][1] = sc[n][c][2] = sc[n][c][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < MAXDK / 16; ++kk) {
            if (kk * 16 >= dk) break;
#pragma unroll
            for (int n = 0; n < KEYS / 16; ++n) {
                uint32_t a0, a1, a2, a3;
                b2::ldmatrix_x4(k_base + 2u * ((n * 16 + (lane & 15)) * ldk + kk * 16 + (lane >> 4) * 8), a0, a1, a2, a3);
                b2::mma_bf16_16816(sc[n][kk & 3], a0, a1, a2, a3, qf[kk][0], qf[kk][1]);
            }
        }
        __syncwarp();                                // the K tile is multiplied: the next one takes its place
        if (more) {
            page = next_page;
            off = next_off;
            issue_k();
            next_page = page_of(key_at(c0 + 2 * STEP), next_off);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        float p[KEYS / 4], mx0 = -INFINITY, mx1 = -INFINITY;     // of every 16 keys gq (0, 1) and gq + 8 (2, 3), heads ha and hb
#pragma unroll
        for (int e = 0; e < KEYS / 4; ++e) {
            const float(&s4)[4][4] = sc[e / 4];
            float x = ((s4[0][e & 3] + s4[1][e & 3]) + (s4[2][e & 3] + s4[3][e & 3])) * scale_log2;
            const bool in = c0 + e / 4 * 16 + gq + (e & 2 ? 8 : 0) < span.n;
            if (SIG) {
                x = in ? sigmoid2_f(x + (e & 1 ? bb : ba)) : 0.f;
            } else {
                if (hs.cap > 0.f) x = cap_score(x, cap_log2, cap_e);
                if (!in) x = -INFINITY;
                if (e & 1) mx1 = fmaxf(mx1, x); else mx0 = fmaxf(mx0, x);
            }
            p[e] = x;
        }
        if (!SIG) {
            if (__any_sync(0xffffffffu, mx0 > m0 || mx1 > m1)) {            // a lane's keys exceed the maximum: else every factor is one
#pragma unroll
                for (int x = 4; x < 32; x <<= 1) {
                    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, x));
                    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, x));
                }
                const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);     // finite: the tile has at least one key
                const float f0 = b2::fast_exp2(m0 - mn0), f1 = b2::fast_exp2(m1 - mn1);
                m0 = mn0;
                m1 = mn1;
                l0 *= f0;
                l1 *= f1;
#pragma unroll
                for (int n = 0; n < DVT; ++n) {
                    o[n][0] *= f0;
                    o[n][1] *= f1;
                    o[n][2] *= f0;
                    o[n][3] *= f1;
                }
            }
#pragma unroll
            for (int e = 0; e < KEYS / 4; e += 4) {
                p[e] = b2::fast_exp2(p[e] - m0);
                p[e + 1] = b2::fast_exp2(p[e + 1] - m1);
                p[e + 2] = b2::fast_exp2(p[e + 2] - m0);
                p[e + 3] = b2::fast_exp2(p[e + 3] - m1);
                l0 += p[e] + p[e + 2];
                l1 += p[e + 1] + p[e + 3];
            }
        }
        uint32_t pt[KEYS / 8];
#pragma unroll
        for (int n = 0; n < KEYS / 8; ++n) pt[n] = transpose_8x8(b2::pack_bf16x2(p[2 * n], p[2 * n + 1]));
        asm volatile("cp.async.wait_group 1;" ::: "memory");     // V is there, the next K may still be on its way
        __syncwarp();
#pragma unroll
        for (int n = 0; n < DVT; ++n) {
            const int key = (lane >> 4) * 8 + (lane & 7), col = n * 16 + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int ks = 0; ks < KEYS / 16; ++ks) {
                uint32_t a0, a1, a2, a3;
                b2::ldmatrix_x4_trans(v_base + 2u * ((ks * 16 + key) * LDV + col), a0, a1, a2, a3);
                b2::mma_bf16_16816(o[n], a0, a1, a2, a3, pt[2 * ks], pt[2 * ks + 1]);
            }
        }
        __syncwarp();                                // the V tile is multiplied
        if (more) issue_v();
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, x);
        l1 += __shfl_xor_sync(0xffffffffu, l1, x);
    }
    __syncthreads();                                 // every warp is done with its tiles: the partial results take their place
    const int used = min(NW, (span.n + KEYS - 1) / KEYS);        // warps that had a tile: NW follows the width of the table, not this row
    if (w < used) {
        float* pa = part + (size_t)(w * kFewHeads + 2 * tq) * PW;
        float* pb = pa + PW;
        if (gq == 0) {
            pa[0] = m0; pa[1] = l0;
            pb[0] = m1; pb[1] = l1;
        }
#pragma unroll
        for (int n = 0; n < DVT; ++n) {
            const int col = 2 + n * 16 + gq;
            pa[col] = o[n][0];
            pb[col] = o[n][1];
            pa[col + 8] = o[n][2];
            pb[col + 8] = o[n][3];
        }
    }
    __syncthreads();
    for (int h = w; h < QHall; h += NW) {            // a warp per head
        const size_t head = (size_t)g * QHall + h;
        const float* px = part + (size_t)h * PW;
        float v[DV / 32], M = -INFINITY, L = 0.f;
#pragma unroll
        for (int c = 0; c < DV / 32; ++c) v[c] = 0.f;
#pragma unroll
        for (int x = 0; x < NW; ++x)
            if (x < used) M = fmaxf(M, px[(size_t)x * kFewHeads * PW]);
#pragma unroll
        for (int x = 0; x < NW; ++x) {
            if (x >= used) break;
            const float* pw = px + (size_t)x * kFewHeads * PW;
            const float f = SIG ? 1.f : (pw[0] == -INFINITY ? 0.f : b2::fast_exp2(pw[0] - M));
            L = fmaf(pw[1], f, L);
#pragma unroll
            for (int c = 0; c < DV / 32; ++c) v[c] = fmaf(pw[2 + lane + 32 * c], f, v[c]);
        }
        float inv = SIG ? 1.f : (L > 0.f ? 1.f / L : 0.f);
        if (gate) inv *= b2::sigmoid_f(__bfloat162float(gate[(size_t)row * gate_stride + head]));
#pragma unroll
        for (int c = 0; c < DV / 32; ++c)
            out[(size_t)row * out_stride + head * DV + lane + 32 * c] = __float2bfloat16_rn(v[c] * inv);
    }
}

template <int DVT, bool SIG, int MAPS, int NW>
__global__ void __launch_bounds__(32 * NW, DVT <= 8 ? 16 / NW : (NW < 8 ? 8 / NW : 1))
chunk_attention_heads_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_cache,
                             const __nv_bfloat16* __restrict__ v_cache, const int32_t* __restrict__ block_tables, int max_nb,
                             const int32_t* __restrict__ cu_q, const int32_t* __restrict__ ctx_start, int n_seq, int H, int G,
                             int dk, int bs, float scale_log2, int chunk, int window, int keep_first, float sink,
                             float sink_logit, const float* __restrict__ sink_logits, const float* __restrict__ head_bias,
                             const __nv_bfloat16* __restrict__ gate, int64_t gate_stride, HeadShape hs, int skip_rows_from, bool by_seq,
                             __nv_bfloat16* __restrict__ out, int64_t out_stride) {
    constexpr int DV = 16 * DVT, LDV = DV + 8, PASS = kHeadRows / MAPS, PW = 2 + DV, NTH = 32 * NW;
    constexpr float kLog2e = 1.4426950408889634f;
    // q [16][dk + 8], then per warp: K tile [16][MAPS * dk + 8], V tile [16][DV + 8]; the merge reuses the tiles' place
    extern __shared__ __align__(16) unsigned char head_sm[];
    const int g = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int QHall = H / G;
    // by_seq: a batch with prompt portions for the tile kernel -- the CTAs are the up to skip_rows_from - 1 rows of every short sequence
    const int per = skip_rows_from - 1;
    const int seq = by_seq ? blockIdx.x / per : b2::seq_of_row(cu_q, n_seq, blockIdx.x);
    const int r0 = cu_q[seq], len = cu_q[seq + 1] - r0;
    int row = by_seq ? r0 + blockIdx.x % per : blockIdx.x;
    const int ctx = ctx_start[seq];
    if (by_seq && row >= r0 + len) return;
    if (skip_rows_from > 0 && ctx >= 0 && len >= skip_rows_from) return;         // the tile kernel's
    if (ctx < 0) {
        do {
            for (int i = tid; i < QHall * DV; i += NTH)
                out[(size_t)row * out_stride + (size_t)g * QHall * DV + i] = __float2bfloat16_rn(0.f);
        } while (by_seq && (row += per) < r0 + len);
        return;
    }
    const int pos = ctx + row - r0;
    const KeySpan span = key_span(pos, pos, chunk, window, keep_first);
    const int32_t* bt = block_tables + (size_t)seq * max_nb;
    const int ldq = dk + 8, ldk = MAPS * dk + 8;
    __nv_bfloat16* q_sm = reinterpret_cast<__nv_bfloat16*>(head_sm);
    __nv_bfloat16* tiles = q_sm + kHeadRows * ldq;
    __nv_bfloat16* kt = tiles + (size_t)w * kHeadKeys * (ldk + LDV);
    __nv_bfloat16* vt = kt + kHeadKeys * ldk;
    float* part = reinterpret_cast<float*>(tiles);       // [NW][16][m, l, O (DV)]
    const uint32_t q_base = b2::smem_u32(q_sm), k_base = b2::smem_u32(kt), v_base = b2::smem_u32(vt);
    const int gq = lane >> 2, tq = lane & 3;
    const float cap_log2 = hs.cap * kLog2e, cap_e = hs.cap > 0.f ? 2.f / hs.cap : 0.f;
    constexpr int STEP = NW * kHeadKeys;

    for (int h0 = 0; h0 < QHall; h0 += PASS) {
        const int QH = min(PASS, QHall - h0);
        // keys past the end repeat the last one: finite numbers that the mask drops
        auto key_at = [&](int c) { return span.key(min(c + (lane & 15), span.n - 1)); };
        auto page_of = [&](int j, int& off) {
            const int pg = j / bs;
            off = j - pg * bs;
            return bt[pg];
        };
        int off, page, next_off = 0, next_page = 0;      // of the tile in flight, and of the one behind it
        auto issue_k = [&]() {
#pragma unroll
            for (int kq = 0; kq < kHeadKeys / 8; ++kq) {
                const int key = kq * 8 + (lane >> 2), c = (lane & 3) * 8;
                const size_t pg = __shfl_sync(0xffffffffu, page, key);
                const int of = __shfl_sync(0xffffffffu, off, key);
#pragma unroll
                for (int mp = 0; mp < MAPS; ++mp) {
                    const __nv_bfloat16* ks = k_cache + ((pg * (G * MAPS) + g * MAPS + mp) * bs + of) * dk + c;
                    __nv_bfloat16* kd = kt + key * ldk + mp * dk + c;
                    for (int t = 0; t < dk; t += 32) cp_async16(kd + t, ks + t);
                }
            }
        };
        auto issue_v = [&]() {
#pragma unroll
            for (int kq = 0; kq < kHeadKeys / 8; ++kq) {
                const int key = kq * 8 + (lane >> 2), c = (lane & 3) * 8;
                const size_t pg = __shfl_sync(0xffffffffu, page, key);
                const int of = __shfl_sync(0xffffffffu, off, key);
                const __nv_bfloat16* vs = v_cache + ((pg * G + g) * bs + of) * DV + c;
                __nv_bfloat16* vd = vt + key * LDV + c;
#pragma unroll
                for (int t = 0; t < DV; t += 32) cp_async16(vd + t, vs + t);
            }
        };
        const int first = w * kHeadKeys;
        __syncthreads();                                 // a previous pass is done with the shared memory
        if (first < span.n) {
            page = page_of(key_at(first), off);
            issue_k();
            asm volatile("cp.async.commit_group;" ::: "memory");
            issue_v();
            asm volatile("cp.async.commit_group;" ::: "memory");
            next_page = page_of(key_at(first + STEP), next_off);
        }
        for (int idx = tid; idx < kHeadRows * (dk / 8); idx += NTH) {
            const int r = idx / (dk / 8), c = (idx % (dk / 8)) * 8, h = r % PASS, mp = r / PASS;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (h < QH) v = *reinterpret_cast<const uint4*>(q + (((size_t)row * H + (size_t)g * QHall + h0 + h) * MAPS + mp) * dk + c);
            *reinterpret_cast<uint4*>(q_sm + r * ldq + c) = v;
        }
        __syncthreads();
        // this thread's two rows and the heads they belong to
        const int ha = g * QHall + h0 + min(gq, QH - 1), hb = MAPS > 1 ? ha : g * QHall + h0 + min(gq + 8, QH - 1);
        float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f, ba = 0.f, bb = 0.f;
        if (w == 0 && sink > 0.f) {                      // the sink enters once, through the first warp
            m0 = (sink_logits ? sink_logits[ha] : sink_logit) * kLog2e;
            m1 = (sink_logits ? sink_logits[hb] : sink_logit) * kLog2e;
            l0 = l1 = tq == 0 ? sink : 0.f;
        }
        if (SIG && head_bias) {
            ba = head_bias[ha] * kLog2e;
            bb = head_bias[hb] * kLog2e;
        }
        float o[2 * DVT][4];
#pragma unroll
        for (int n = 0; n < 2 * DVT; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

        for (int c0 = first; c0 < span.n; c0 += STEP) {
            const bool more = c0 + STEP < span.n;
            asm volatile("cp.async.wait_group 1;" ::: "memory");     // K is there, V may still be on its way
            __syncwarp();
            float sc[2][4], sd[MAPS > 1 ? 2 : 1][4];
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
                if (MAPS > 1) sd[MAPS > 1 ? n : 0][0] = sd[MAPS > 1 ? n : 0][1] = sd[MAPS > 1 ? n : 0][2] = sd[MAPS > 1 ? n : 0][3] = 0.f;
            }
#pragma unroll 4
            for (int kk = 0; kk < dk; kk += 16) {
                uint32_t a0, a1, a2, a3, b0, b1, b2_, b3;
                b2::ldmatrix_x4(q_base + 2u * ((lane & 15) * ldq + kk + (lane >> 4) * 8), a0, a1, a2, a3);
                const int key = (lane >> 4) * 8 + (lane & 7), dim = kk + ((lane >> 3) & 1) * 8;
                b2::ldmatrix_x4(k_base + 2u * (key * ldk + dim), b0, b1, b2_, b3);
                b2::mma_bf16_16816(sc[0], a0, a1, a2, a3, b0, b1);
                b2::mma_bf16_16816(sc[1], a0, a1, a2, a3, b2_, b3);
                if (MAPS > 1) {                          // rows 8 - 15 belong to the second maps and take their keys
                    b2::ldmatrix_x4(k_base + 2u * (key * ldk + dk + dim), b0, b1, b2_, b3);
                    b2::mma_bf16_16816(sd[0], a0, a1, a2, a3, b0, b1);
                    b2::mma_bf16_16816(sd[MAPS > 1 ? 1 : 0], a0, a1, a2, a3, b2_, b3);
                }
            }
            if (MAPS > 1) {
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    sc[n][2] = sd[MAPS > 1 ? n : 0][2];
                    sc[n][3] = sd[MAPS > 1 ? n : 0][3];
                }
            }
            __syncwarp();                                // the K tile is multiplied: the next one takes its place
            if (more) {
                page = next_page;
                off = next_off;
                issue_k();
                next_page = page_of(key_at(c0 + 2 * STEP), next_off);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            const bool whole = c0 + kHeadKeys <= span.n;
            float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float x = sc[n][e] * scale_log2;
                    const bool in = whole || c0 + n * 8 + 2 * tq + (e & 1) < span.n;
                    if (SIG) {
                        x = in ? sigmoid2_f(x + (e < 2 ? ba : bb)) : 0.f;
                    } else {
                        if (hs.cap > 0.f) x = cap_score(x, cap_log2, cap_e);
                        if (!in) x = -INFINITY;
                        if (e < 2) mx0 = fmaxf(mx0, x); else mx1 = fmaxf(mx1, x);
                    }
                    sc[n][e] = x;
                }
            }
            if (!SIG) {
#pragma unroll
                for (int x = 1; x < 4; x <<= 1) {
                    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, x));
                    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, x));
                }
                const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);         // finite: the tile has at least one key
                const float f0 = b2::fast_exp2(m0 - mn0), f1 = b2::fast_exp2(m1 - mn1);
                m0 = mn0;
                m1 = mn1;
                l0 *= f0;
                l1 *= f1;
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    sc[n][0] = b2::fast_exp2(sc[n][0] - mn0);
                    sc[n][1] = b2::fast_exp2(sc[n][1] - mn0);
                    sc[n][2] = b2::fast_exp2(sc[n][2] - mn1);
                    sc[n][3] = b2::fast_exp2(sc[n][3] - mn1);
                    l0 += sc[n][0] + sc[n][1];
                    l1 += sc[n][2] + sc[n][3];
                }
#pragma unroll
                for (int n = 0; n < 2 * DVT; ++n) {
                    o[n][0] *= f0;
                    o[n][1] *= f0;
                    o[n][2] *= f1;
                    o[n][3] *= f1;
                }
            }
            asm volatile("cp.async.wait_group 1;" ::: "memory");     // V is there, the next K may still be on its way
            __syncwarp();
            {
                const uint32_t a0 = b2::pack_bf16x2(sc[0][0], sc[0][1]), a1 = b2::pack_bf16x2(sc[0][2], sc[0][3]);
                const uint32_t a2 = b2::pack_bf16x2(sc[1][0], sc[1][1]), a3 = b2::pack_bf16x2(sc[1][2], sc[1][3]);
#pragma unroll
                for (int n2 = 0; n2 < DVT; ++n2) {
                    uint32_t b0, b1, b2_, b3;
                    const int key = ((lane >> 3) & 1) * 8 + (lane & 7), col = n2 * 16 + (lane >> 4) * 8;
                    b2::ldmatrix_x4_trans(v_base + 2u * (key * LDV + col), b0, b1, b2_, b3);
                    b2::mma_bf16_16816(o[2 * n2], a0, a1, a2, a3, b0, b1);
                    b2::mma_bf16_16816(o[2 * n2 + 1], a0, a1, a2, a3, b2_, b3);
                }
            }
            __syncwarp();                                // the V tile is multiplied
            if (more) issue_v();
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, x);
            l1 += __shfl_xor_sync(0xffffffffu, l1, x);
        }
        __syncthreads();                                 // every warp is done with its tiles: the partial results take their place
        const int used = min(NW, (span.n + kHeadKeys - 1) / kHeadKeys);  // warps that had a tile
        if (w < used) {
            float* pa = part + (size_t)(w * kHeadRows + gq) * PW;
            float* pb = pa + 8 * PW;
            if (tq == 0) {
                pa[0] = m0; pa[1] = l0;
                pb[0] = m1; pb[1] = l1;
            }
#pragma unroll
            for (int n = 0; n < 2 * DVT; ++n) {
                const int col = 2 + n * 8 + 2 * tq;
                *reinterpret_cast<float2*>(pa + col) = make_float2(o[n][0], o[n][1]);
                *reinterpret_cast<float2*>(pb + col) = make_float2(o[n][2], o[n][3]);
            }
        }
        __syncthreads();
        // a warp per head: merged output of operand row r at column col
        for (int h = w; h < QH; h += NW) {
            const size_t head = (size_t)g * QHall + h0 + h;
            float v[DV / 32], ss = 0.f;
#pragma unroll
            for (int c = 0; c < DV / 32; ++c) v[c] = 0.f;
#pragma unroll
            for (int mp = 0; mp < MAPS; ++mp) {
                const float* px = part + (size_t)(h + mp * PASS) * PW;
                float M = -INFINITY, L = 0.f;
#pragma unroll
                for (int x = 0; x < NW; ++x)
                    if (x < used) M = fmaxf(M, px[(size_t)x * kHeadRows * PW]);
                auto weight = [&](int x) {
                    const float mx = px[(size_t)x * kHeadRows * PW];
                    return SIG ? 1.f : (mx == -INFINITY ? 0.f : b2::fast_exp2(mx - M));
                };
#pragma unroll
                for (int x = 0; x < NW; ++x)
                    if (x < used) L = fmaf(px[(size_t)x * kHeadRows * PW + 1], weight(x), L);
                const float inv = (SIG ? 1.f : (L > 0.f ? 1.f / L : 0.f)) * (mp == 0 ? 1.f : -hs.lambda);
#pragma unroll
                for (int x = 0; x < NW; ++x) {
                    if (x >= used) break;
                    const float f = weight(x) * inv;
#pragma unroll
                    for (int c = 0; c < DV / 32; ++c) v[c] = fmaf(px[(size_t)x * kHeadRows * PW + 2 + lane + 32 * c], f, v[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < DV / 32; ++c) ss = fmaf(v[c], v[c], ss);
            float inv = MAPS > 1 ? rsqrtf(b2::warp_sum(ss) / (float)DV + hs.eps) * hs.out_scale : 1.f;
            if (gate) inv *= b2::sigmoid_f(__bfloat162float(gate[(size_t)row * gate_stride + head]));
#pragma unroll
            for (int c = 0; c < DV / 32; ++c)
                out[(size_t)row * out_stride + head * DV + lane + 32 * c] = __float2bfloat16_rn(v[c] * inv);
        }
    }
}

template <int DVT, bool SIG, int MAPS, int NW, bool FEW, int KEYS>
int launch_heads_nw(const void* q, const void* k_cache, const void* v_cache, const int32_t* block_tables, int max_nb,
                    const int32_t* cu_q, const int32_t* ctx_start, int n_seq, int ctas, int H, int G, int dk, int bs, float scale, int chunk,
                    int window, int keep_first, float sink, float sink_logit, const float* sink_logits, const float* head_bias,
                    const void* gate, int64_t gate_stride, const HeadShape& hs, int skip_from, bool by_seq, void* out, int64_t out_stride,
                    cudaStream_t st) {
    constexpr int DV = 16 * DVT;
    constexpr int ROWS = FEW ? kFewHeads : kHeadRows;
    const size_t tiles = (size_t)NW * KEYS * (MAPS * dk + 8 + DV + 8) * sizeof(__nv_bfloat16);
    const size_t merge = (size_t)NW * ROWS * (2 + DV) * sizeof(float);
    const size_t smem = (size_t)ROWS * (dk + 8) * sizeof(__nv_bfloat16) + (tiles > merge ? tiles : merge);
    auto kern = [] {
        if constexpr (FEW) return chunk_attention_few_heads_kernel<DVT, SIG, NW, KEYS>;
        else return chunk_attention_heads_kernel<DVT, SIG, MAPS, NW>;
    }();
    if (smem > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<dim3(ctas, G), 32 * NW, smem, st>>>(static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k_cache),
                                              static_cast<const __nv_bfloat16*>(v_cache), block_tables, max_nb, cu_q, ctx_start, n_seq, H,
                                              G, dk, bs, scale * 1.4426950408889634f, chunk, window, keep_first, sink, sink_logit, sink_logits,
                                              head_bias, static_cast<const __nv_bfloat16*>(gate), gate_stride, hs, skip_from, by_seq,
                                              static_cast<__nv_bfloat16*>(out), out_stride);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

template <int DVT, bool SIG, int MAPS>
int launch_heads(const void* q, const void* k_cache, const void* v_cache, const int32_t* block_tables, int max_nb,
                 const int32_t* cu_q, const int32_t* ctx_start, int n_seq, int T, int H, int G, int dk, int bs, float scale, int chunk,
                 int window, int keep_first, float sink, float sink_logit, const float* sink_logits, const float* head_bias,
                 const void* gate, int64_t gate_stride, const HeadShape& hs, int skip_from, void* out, int64_t out_stride,
                 cudaStream_t st) {
    // beside the tile kernel only the rows of sequences below skip_from are left, at most skip_from - 1 a sequence: a CTA for each of
    // those and not for every row of the batch (4096 rows x 8 kv heads of CTAs that leave at once took 31 us)
    const bool by_seq = skip_from > 1 && (int64_t)n_seq * (skip_from - 1) < T;
    const int ctas = by_seq ? n_seq * (skip_from - 1) : T;
    // warps a CTA: 16 an SM together, as long as each still has a few tiles of keys
    int64_t keys = (int64_t)max_nb * bs;
    if (chunk > 0 && chunk < keys) keys = chunk;
    if (window > 0 && window + keep_first < keys) keys = window + keep_first;
    const int64_t items = (int64_t)ctas * G;
    const int nw = items <= b2_sm_count() && keys >= 512 ? 16 : items <= 2 * b2_sm_count() && keys >= 256 ? 8 : 4;
#define B2_HEADS_NW(NW, FEW)                                                                                                      \
    return (FEW && dk <= kShortDk ? launch_heads_nw<DVT, SIG, MAPS, NW, FEW, FEW ? 2 * kHeadKeys : kHeadKeys>                     \
                                  : launch_heads_nw<DVT, SIG, MAPS, NW, FEW, kHeadKeys>)(q, k_cache, v_cache, block_tables, max_nb, cu_q, ctx_start, n_seq, ctas, H, G, dk, bs, scale, \
                                               chunk, window, keep_first, sink, sink_logit, sink_logits, head_bias, gate, gate_stride, hs, \
                                               skip_from, by_seq, out, out_stride, st)
    if constexpr (MAPS == 1) {
        if (H / G <= kFewHeads && dk <= kFewDk) {
            if constexpr (DVT <= 8) {                    // else 16 warps would not have the shared memory
                if (nw == 16) B2_HEADS_NW(16, true);
            }
            if (nw >= 8) B2_HEADS_NW(8, true);
            B2_HEADS_NW(4, true);
        }
    }
    if (nw >= 8) B2_HEADS_NW(8, false);
    B2_HEADS_NW(4, false);
#undef B2_HEADS_NW
}

// ------------------------------------------------------------------------------------------------- tiled prompt kernel
// What the tcgen05 prompt kernel does not take: two maps of more than 64 numbers, and values of 192 or 256.
// bf16, dk and dv multiples of 16, softmax weights: one CTA = 64 consecutive query rows of one sequence x one head, four warps of 16 rows.
// Keys are walked 64 at a time from the first row's block start to the last row's position (at most chunk + 63 keys
// with a mask, the whole prefix without): K and V tiles are gathered from the pages into shared memory (cp.async, two
// threads per key row with one page lookup each, the next tile in flight while this one is multiplied), S = Q K^T and
// O += P V run on mma.sync m16n8k16 with ldmatrix operands, the online softmax lives in the accumulator registers
// (exp2 with the scale folded in, the sink seeding the running maximum and denominator).  A warp tests the mask per score
// only in tiles that its rows see in part.  Sequences with fewer than kTileMinRows rows (decode rows) are left to the warp
// kernel above.
constexpr int kTQ = 64, kTK = 64, kTileMinRows = 16;

template <int DKT, int DVT, int MAPS>
__global__ void __launch_bounds__(128)
chunk_attention_tile_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_cache,
                            const __nv_bfloat16* __restrict__ v_cache, const int32_t* __restrict__ block_tables, int max_nb,
                            const int32_t* __restrict__ cu_q, const int32_t* __restrict__ ctx_start, int n_seq, int H, int G,
                            int bs, float scale_log2, int chunk, int window, int keep_first, float sink,
                            float sink_logit_log2, const float* __restrict__ sink_logits,
                            const __nv_bfloat16* __restrict__ gate, int64_t gate_stride, HeadShape hs, __nv_bfloat16* __restrict__ out,
                            int64_t out_stride) {
    constexpr int DK = 16 * DKT, DV = 16 * DVT, LDK = MAPS * DK + 8, LDV = DV + 8;
    extern __shared__ __align__(16) unsigned char tile_smem[];
    __nv_bfloat16* q_sm = reinterpret_cast<__nv_bfloat16*>(tile_smem);      // [64][LDK]
    __nv_bfloat16* k_sm = q_sm + kTQ * LDK;                                 // [2][64][LDK]
    __nv_bfloat16* v_sm = k_sm + 2 * kTK * LDK;                             // [2][64][LDV]
    __shared__ int s_info[2];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) {
        int want = blockIdx.x, found = -1, t0 = 0;
        for (int s = 0; s < n_seq; ++s) {
            const int len = cu_q[s + 1] - cu_q[s];
            if (len < kTileMinRows || ctx_start[s] < 0) continue;
            const int nt = (len + kTQ - 1) / kTQ;
            if (want < nt) { found = s; t0 = want * kTQ; break; }
            want -= nt;
        }
        s_info[0] = found;
        s_info[1] = t0;
    }
    __syncthreads();
    const int seq = s_info[0], t0 = s_info[1];
    if (seq < 0) return;
    const int hh = blockIdx.y, g = hh / (H / G);
    const int r0 = cu_q[seq] + t0;
    const int rows = min(kTQ, cu_q[seq + 1] - r0);
    const int p0 = ctx_start[seq] + t0, p_last = p0 + rows - 1;
    // the union of what the tile's rows see, as one compact range: kept first keys, then the first row's window .. p_last
    const KeySpan span = key_span(p0, p_last, chunk, window, keep_first);
    const int32_t* bt = block_tables + (size_t)seq * max_nb;

    for (int idx = tid; idx < kTQ * (MAPS * DK / 8); idx += 128) {
        const int r = idx / (MAPS * DK / 8), c = (idx % (MAPS * DK / 8)) * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < rows) v = *reinterpret_cast<const uint4*>(q + ((size_t)(r0 + r) * H + hh) * (MAPS * DK) + c);
        *reinterpret_cast<uint4*>(q_sm + r * LDK + c) = v;
    }
    const int gq = lane >> 2, tq = lane & 3;
    const int i0 = p0 + w * 16 + gq, i1 = i0 + 8;                           // positions of this thread's two rows
    const int lo0 = chunk > 0 ? (i0 / chunk) * chunk : 0, lo1 = chunk > 0 ? (i1 / chunk) * chunk : 0;
    const int w_first = p0 + w * 16, w_last = w_first + 15;
    const int w_clo = chunk > 0 ? (w_first / chunk) * chunk : 0;
    const int w_lo = window > 0 ? max(w_clo, w_first - window + 1) : w_clo;   // the lowest key of the warp's rows' windows
    if (sink_logits) sink_logit_log2 = sink_logits[hh] * 1.4426950408889634f;
    float m0[MAPS], m1[MAPS], l0[MAPS], l1[MAPS];                           // partial sums per lane; the sink counted once
    float o[MAPS][2 * DVT][4];
#pragma unroll
    for (int mp = 0; mp < MAPS; ++mp) {
        m0[mp] = m1[mp] = sink > 0.f ? sink_logit_log2 : -INFINITY;
        l0[mp] = l1[mp] = tq == 0 ? sink : 0.f;
#pragma unroll
        for (int n = 0; n < 2 * DVT; ++n) o[mp][n][0] = o[mp][n][1] = o[mp][n][2] = o[mp][n][3] = 0.f;
    }
    const float cap_log2 = hs.cap * 1.4426950408889634f, cap_e = hs.cap > 0.f ? 2.f / hs.cap : 0.f;
    const uint32_t q_base = b2::smem_u32(q_sm), k_base0 = b2::smem_u32(k_sm), v_base0 = b2::smem_u32(v_sm);

    const int ld_key = tid >> 1, ld_half = tid & 1;
    auto issue = [&](int kv0, int buf) {                                    // kv0: compact key index of the tile's first key
        const int j = span.key(kv0 + ld_key);
        __nv_bfloat16* kd = k_sm + (buf * kTK + ld_key) * LDK;
        __nv_bfloat16* vd = v_sm + (buf * kTK + ld_key) * LDV;
        if (j <= p_last) {
            const int page = j / bs;
            const size_t blk = bt[page], off = j - page * bs;
            const __nv_bfloat16* vs = v_cache + ((blk * G + g) * bs + off) * DV;
#pragma unroll
            for (int mp = 0; mp < MAPS; ++mp) {
                const __nv_bfloat16* ks = k_cache + ((blk * (G * MAPS) + g * MAPS + mp) * bs + off) * DK;
#pragma unroll
                for (int c = 0; c < DKT; ++c) cp_async16(kd + mp * DK + (2 * c + ld_half) * 8, ks + (2 * c + ld_half) * 8);
            }
#pragma unroll
            for (int c = 0; c < DVT; ++c) cp_async16(vd + (2 * c + ld_half) * 8, vs + (2 * c + ld_half) * 8);
        } else {
#pragma unroll
            for (int c = 0; c < MAPS * DKT; ++c) *reinterpret_cast<uint4*>(kd + (2 * c + ld_half) * 8) = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int c = 0; c < DVT; ++c) *reinterpret_cast<uint4*>(vd + (2 * c + ld_half) * 8) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0, 0);
    for (int kv0 = 0, buf = 0; kv0 < span.n; kv0 += kTK, buf ^= 1) {
        if (kv0 + kTK < span.n) {
            issue(kv0 + kTK, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();                                                    // the tile (and, first time, Q) is in shared memory
        const uint32_t k_base = k_base0 + (uint32_t)(buf * kTK * LDK) * 2u, v_base = v_base0 + (uint32_t)(buf * kTK * LDV) * 2u;
        const int j_min = span.key(kv0), j_max = span.key(min(kv0 + kTK, span.n) - 1);
        // nothing in this tile is visible to the warp's rows: all keys after them, or all before their windows and not kept
        const bool none = j_min > w_last || (j_max < w_lo && (window <= 0 || j_min >= keep_first));
        // all of it is visible to all of them
        const bool full = kv0 + kTK <= span.n && j_max <= w_first && (chunk <= 0 || j_min >= (w_last / chunk) * chunk) &&
                          (window <= 0 || w_last - j_min < window || j_max < keep_first);
        if (!none) {
#pragma unroll
            for (int mp = 0; mp < MAPS; ++mp) {
                float sc[8][4];
#pragma unroll
                for (int n = 0; n < 8; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
#pragma unroll
                for (int kk = 0; kk < DKT; ++kk) {
                    uint32_t a0, a1, a2, a3;
                    b2::ldmatrix_x4(q_base + 2u * ((w * 16 + (lane & 15)) * LDK + mp * DK + kk * 16 + (lane >> 4) * 8), a0, a1, a2, a3);
#pragma unroll
                    for (int n2 = 0; n2 < 4; ++n2) {
                        uint32_t b0, b1, b2_, b3;
                        const int key = n2 * 16 + (lane >> 4) * 8 + (lane & 7), dim = mp * DK + kk * 16 + ((lane >> 3) & 1) * 8;
                        b2::ldmatrix_x4(k_base + 2u * (key * LDK + dim), b0, b1, b2_, b3);
                        b2::mma_bf16_16816(sc[2 * n2], a0, a1, a2, a3, b0, b1);
                        b2::mma_bf16_16816(sc[2 * n2 + 1], a0, a1, a2, a3, b2_, b3);
                    }
                }
                float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) sc[n][e] *= scale_log2;
                }
                if (hs.cap > 0.f) {
#pragma unroll
                    for (int n = 0; n < 8; ++n) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) sc[n][e] = cap_score(sc[n][e], cap_log2, cap_e);
                    }
                }
                if (!full) {
#pragma unroll
                    for (int n = 0; n < 8; ++n) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int j = span.key(kv0 + n * 8 + 2 * tq + (e & 1));
                            const bool ok = e < 2 ? key_visible(i0, j, lo0, window, keep_first) : key_visible(i1, j, lo1, window, keep_first);
                            if (!ok) sc[n][e] = -INFINITY;
                        }
                    }
                }
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    mx0 = fmaxf(mx0, fmaxf(sc[n][0], sc[n][1]));
                    mx1 = fmaxf(mx1, fmaxf(sc[n][2], sc[n][3]));
                }
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
                const float mn0 = fmaxf(m0[mp], mx0), mn1 = fmaxf(m1[mp], mx1);
                const float mu0 = mn0 == -INFINITY ? 0.f : mn0, mu1 = mn1 == -INFINITY ? 0.f : mn1;
                const float c0 = b2::fast_exp2(m0[mp] - mu0), c1 = b2::fast_exp2(m1[mp] - mu1);             // exp2(-inf) = 0: nothing accumulated yet
                m0[mp] = mn0;
                m1[mp] = mn1;
                float s0 = 0.f, s1 = 0.f;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    sc[n][0] = b2::fast_exp2(sc[n][0] - mu0);
                    sc[n][1] = b2::fast_exp2(sc[n][1] - mu0);
                    sc[n][2] = b2::fast_exp2(sc[n][2] - mu1);
                    sc[n][3] = b2::fast_exp2(sc[n][3] - mu1);
                    s0 += sc[n][0] + sc[n][1];
                    s1 += sc[n][2] + sc[n][3];
                }
                l0[mp] = l0[mp] * c0 + s0;
                l1[mp] = l1[mp] * c1 + s1;
#pragma unroll
                for (int n = 0; n < 2 * DVT; ++n) {
                    o[mp][n][0] *= c0;
                    o[mp][n][1] *= c0;
                    o[mp][n][2] *= c1;
                    o[mp][n][3] *= c1;
                }
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    const uint32_t a0 = b2::pack_bf16x2(sc[2 * ks][0], sc[2 * ks][1]), a1 = b2::pack_bf16x2(sc[2 * ks][2], sc[2 * ks][3]);
                    const uint32_t a2 = b2::pack_bf16x2(sc[2 * ks + 1][0], sc[2 * ks + 1][1]),
                                   a3 = b2::pack_bf16x2(sc[2 * ks + 1][2], sc[2 * ks + 1][3]);
#pragma unroll
                    for (int n2 = 0; n2 < DVT; ++n2) {
                        uint32_t b0, b1, b2_, b3;
                        const int key = ks * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), col = n2 * 16 + (lane >> 4) * 8;
                        b2::ldmatrix_x4_trans(v_base + 2u * (key * LDV + col), b0, b1, b2_, b3);
                        b2::mma_bf16_16816(o[mp][2 * n2], a0, a1, a2, a3, b0, b1);
                        b2::mma_bf16_16816(o[mp][2 * n2 + 1], a0, a1, a2, a3, b2_, b3);
                    }
                }
            }
        }
        __syncthreads();                                                    // the tile is consumed: its buffer may be refilled
    }
    float inv0 = 1.f, inv1 = 1.f;
#pragma unroll
    for (int mp = 0; mp < MAPS; ++mp) {
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
            l0[mp] += __shfl_xor_sync(0xffffffffu, l0[mp], x);
            l1[mp] += __shfl_xor_sync(0xffffffffu, l1[mp], x);
        }
        inv0 = l0[mp] > 0.f ? 1.f / l0[mp] : 0.f;
        inv1 = l1[mp] > 0.f ? 1.f / l1[mp] : 0.f;
        if (MAPS > 1) {
            const float f0 = mp == 0 ? inv0 : -hs.lambda * inv0, f1 = mp == 0 ? inv1 : -hs.lambda * inv1;
#pragma unroll
            for (int n = 0; n < 2 * DVT; ++n) {
                o[mp][n][0] *= f0;
                o[mp][n][1] *= f0;
                o[mp][n][2] *= f1;
                o[mp][n][3] *= f1;
            }
        }
    }
    const int ra = w * 16 + gq, rb = ra + 8;
    if (MAPS > 1) {                                                         // the difference and its norm over the head's columns
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int n = 0; n < 2 * DVT; ++n) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[0][n][e] += o[MAPS - 1][n][e];
                if (e < 2) s0 = fmaf(o[0][n][e], o[0][n][e], s0);
                else s1 = fmaf(o[0][n][e], o[0][n][e], s1);
            }
        }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, x);
            s1 += __shfl_xor_sync(0xffffffffu, s1, x);
        }
        inv0 = rsqrtf(s0 / (float)DV + hs.eps) * hs.out_scale;
        inv1 = rsqrtf(s1 / (float)DV + hs.eps) * hs.out_scale;
    }
    if (gate) {
        if (ra < rows) inv0 *= b2::sigmoid_f(__bfloat162float(gate[(size_t)(r0 + ra) * gate_stride + hh]));
        if (rb < rows) inv1 *= b2::sigmoid_f(__bfloat162float(gate[(size_t)(r0 + rb) * gate_stride + hh]));
    }
#pragma unroll
    for (int n = 0; n < 2 * DVT; ++n) {
        const int col = n * 8 + 2 * tq;
        if (ra < rows)
            *reinterpret_cast<uint32_t*>(out + (size_t)(r0 + ra) * out_stride + hh * DV + col) = b2::pack_bf16x2(o[0][n][0] * inv0, o[0][n][1] * inv0);
        if (rb < rows)
            *reinterpret_cast<uint32_t*>(out + (size_t)(r0 + rb) * out_stride + hh * DV + col) = b2::pack_bf16x2(o[0][n][2] * inv1, o[0][n][3] * inv1);
    }
}

template <int DKT, int DVT, int MAPS>
int launch_tile(const void* q, const void* k_cache, const void* v_cache, const int32_t* block_tables, int max_nb,
                const int32_t* cu_q, const int32_t* ctx_start, int n_seq, int T, int H, int G, int bs, float scale, int chunk,
                int window, int keep_first, float sink, float sink_logit, const float* sink_logits,
                const void* gate, int64_t gate_stride, const HeadShape& hs, void* out, int64_t out_stride, cudaStream_t st) {
    constexpr int DK = 16 * DKT, DV = 16 * DVT;
    const size_t smem = (size_t)(kTQ * (MAPS * DK + 8) + 2 * kTK * (MAPS * DK + 8) + 2 * kTK * (DV + 8)) * sizeof(__nv_bfloat16);
    auto kern = chunk_attention_tile_kernel<DKT, DVT, MAPS>;
    if (smem > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int tiles = (T + kTQ - 1) / kTQ + n_seq;          // upper bound on sum(ceil(len / 64)); spare CTAs leave at once
    kern<<<dim3(tiles, H), 128, smem, st>>>(static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k_cache),
                                           static_cast<const __nv_bfloat16*>(v_cache), block_tables, max_nb, cu_q, ctx_start,
                                           n_seq, H, G, bs, scale * 1.4426950408889634f, chunk, window, keep_first, sink,
                                           sink_logit * 1.4426950408889634f, sink_logits,
                                           static_cast<const __nv_bfloat16*>(gate), gate_stride, hs, static_cast<__nv_bfloat16*>(out),
                                           out_stride);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

}  // namespace

extern "C" int b2_qknorm_cache(const void* qkv, int64_t qkv_stride, int act_dtype, int T, int H, int G, int dk, int dv,
                               const float* q_w, const float* k_w, float eps, const int64_t* slots, int bs, void* q_out,
                               void* k_cache, void* v_cache, void* stream) {
    B2_REQUIRE(T >= 0 && H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0 && bs > 0, B2_EINVAL, "qknorm_cache: bad sizes");
    if (T == 0) return B2_OK;
    B2_REQUIRE(qkv && slots && q_out && k_cache && v_cache, B2_EINVAL, "qknorm_cache: null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int warps = H + 2 * G < 8 ? H + 2 * G : 8;
    B2_DISPATCH_ACT(act_dtype, A, (qknorm_cache_kernel<A><<<T, warps * 32, 0, st>>>(
        static_cast<const A*>(qkv), qkv_stride, H, G, dk, dv, q_w, k_w, eps, slots, bs, static_cast<A*>(q_out),
        static_cast<A*>(k_cache), static_cast<A*>(v_cache), true, nullptr, 0.f, 1)));
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

extern "C" int b2_qk_prep_cache(const void* qkv, int64_t qkv_stride, int act_dtype, int T, int H, int G, int dk, int dv,
                                int norm, const float* q_w, const float* k_w, float eps, const int32_t* positions,
                                float temp_coef, int temp_every, const int64_t* slots, int bs, void* q_out, void* k_cache,
                                void* v_cache, void* stream) {
    B2_REQUIRE(T >= 0 && H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0 && bs > 0, B2_EINVAL, "qk_prep_cache: bad sizes");
    B2_REQUIRE(temp_coef == 0.f || (positions && temp_every >= 1), B2_EINVAL,
               "qk_prep_cache: a query temperature needs positions and a period of at least 1");
    if (T == 0) return B2_OK;
    B2_REQUIRE(qkv && slots && q_out && k_cache && v_cache, B2_EINVAL, "qk_prep_cache: null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int warps = H + 2 * G < 8 ? H + 2 * G : 8;
    B2_DISPATCH_ACT(act_dtype, A, (qknorm_cache_kernel<A><<<T, warps * 32, 0, st>>>(
        static_cast<const A*>(qkv), qkv_stride, H, G, dk, dv, q_w, k_w, eps, slots, bs, static_cast<A*>(q_out),
        static_cast<A*>(k_cache), static_cast<A*>(v_cache), norm != 0, positions, temp_coef, temp_every > 0 ? temp_every : 1)));
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

extern "C" int b2_qk_rope_cache(const void* qkv, int64_t qkv_stride, int act_dtype, int T, int H, int G, int dk, int dv,
                                int v_from_k, int rot_dims, int interleaved, const int32_t* positions, const float* cos_sin,
                                int max_pos, const int64_t* slots, int bs, void* q_out, void* k_cache, void* v_cache,
                                void* stream) {
    return b2_qk_norm_rope_cache(qkv, qkv_stride, act_dtype, T, H, G, G, dk, dv, v_from_k, nullptr, nullptr, 0.f, rot_dims, interleaved,
                                 positions, cos_sin, max_pos, slots, bs, q_out, k_cache, v_cache, stream);
}

extern "C" int b2_qk_norm_rope_cache(const void* qkv, int64_t qkv_stride, int act_dtype, int T, int H, int G, int Gv, int dk, int dv,
                                     int v_from_k, const float* q_w, const float* k_w, float eps, int rot_dims, int interleaved,
                                     const int32_t* positions, const float* cos_sin, int max_pos, const int64_t* slots, int bs,
                                     void* q_out, void* k_cache, void* v_cache, void* stream) {
    B2_REQUIRE(T >= 0 && H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0 && bs > 0, B2_EINVAL, "qk_rope_cache: bad sizes");
    B2_REQUIRE(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dk, B2_EINVAL,
               "qk_rope_cache: %d rotated entries in heads of %d", rot_dims, dk);
    B2_REQUIRE(Gv > 0 && Gv <= G, B2_EINVAL, "qk_rope_cache: %d value heads beside %d key heads", Gv, G);
    B2_REQUIRE(!v_from_k || (dv == dk && Gv == G), B2_EINVAL, "qk_rope_cache: values taken from the keys need dv == dk and a value head per key head");
    B2_REQUIRE(rot_dims == 0 || max_pos > 0, B2_EINVAL, "qk_rope_cache: empty rotation table");
    B2_REQUIRE(!q_w == !k_w, B2_EINVAL, "qk_rope_cache: the norm needs the weights of both q and k");
    if (T == 0) return B2_OK;
    B2_REQUIRE(qkv && slots && q_out && k_cache && v_cache && positions && (cos_sin || rot_dims == 0), B2_EINVAL,
               "qk_rope_cache: null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t esz = act_dtype == B2_ACT_BF16 ? 2 : 4;
    auto al = [&](const void* p) { return reinterpret_cast<uintptr_t>(p) % (4 * esz) == 0; };
    const bool vec = dk % 4 == 0 && dv % 4 == 0 && qkv_stride % 4 == 0 && rot_dims % (interleaved ? 4 : 8) == 0 && al(qkv) && al(q_out) &&
                     al(k_cache) && al(v_cache) && b2_aligned16(q_w) && b2_aligned16(k_w);
    const int work = (H + G) * (vec ? (dk + 7) / 8 : dk);
    const int threads = work >= 256 ? 256 : (work >= 128 ? 128 : 64);
#define B2_ROPE(KERN, NORM)                                                                                                     \
    KERN<A, NORM><<<T, threads, 0, st>>>(static_cast<const A*>(qkv), qkv_stride, H, G, Gv, dk, dv, v_from_k != 0, rot_dims,         \
                                         interleaved != 0, positions, cos_sin, max_pos > 0 ? max_pos : 1, slots, bs, q_w, k_w, eps, \
                                         static_cast<A*>(q_out), static_cast<A*>(k_cache), static_cast<A*>(v_cache))
    const int row_threads = ((H + G) * (dk / 16) + 31) / 32 * 32;
    if (act_dtype == B2_ACT_BF16 && dk % 16 == 0 && rot_dims % 16 == 0 && dv % 8 == 0 && qkv_stride % 8 == 0 && row_threads <= 1024 && row_threads >= 128 &&
        (v_from_k || Gv * dv / 8 <= row_threads) && b2_aligned16(qkv) && b2_aligned16(q_out) && b2_aligned16(k_cache) && b2_aligned16(v_cache) &&
        b2_aligned16(q_w) && b2_aligned16(k_w) && b2_aligned16(cos_sin)) {
        const RopeArgs a{static_cast<const __nv_bfloat16*>(qkv), qkv_stride, T, H, G, Gv, dk, dv, v_from_k != 0, rot_dims, positions, cos_sin,
                         max_pos > 0 ? max_pos : 1, slots, bs, bs & (bs - 1) ? -1 : __builtin_ctz(bs), q_w, k_w, eps,
                         static_cast<__nv_bfloat16*>(q_out), static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache)};
        // the ring where every CTA has several rows: 64 rows 4.2 us without it, and its copies could not run ahead
        const int smem = kRopeStages * a.stage_bytes(), per_sm = 1024 / row_threads, fit = 216 * 1024 / (smem + 2048);
        const int ctas = (fit < per_sm ? fit : per_sm) * b2_sm_count();
        const bool ring = ctas > 0 && T >= 2 * ctas;
#define B2_ROPE_ROWS(NORM, IL)                                                                                                  \
    do {                                                                                                                        \
        if (ring) {                                                                                                             \
            auto kern = qk_rope_cache_rows_kernel<NORM, IL, true>;                                                                \
            B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));                           \
            kern<<<ctas, row_threads, smem, st>>>(a);                                                                             \
        } else {                                                                                                                \
            qk_rope_cache_rows_kernel<NORM, IL, false><<<T, row_threads, 0, st>>>(a);                                             \
        }                                                                                                                       \
    } while (0)
        if (q_w) { if (interleaved) B2_ROPE_ROWS(true, true); else B2_ROPE_ROWS(true, false); }
        else if (interleaved) B2_ROPE_ROWS(false, true);
        else B2_ROPE_ROWS(false, false);
#undef B2_ROPE_ROWS
        B2_CUDA_OK(cudaGetLastError());
        return B2_OK;
    }
    B2_DISPATCH_ACT(act_dtype, A, {
        if (vec && q_w) B2_ROPE(qk_rope_cache_vec_kernel, true);
        else if (vec) B2_ROPE(qk_rope_cache_vec_kernel, false);
        else if (q_w) B2_ROPE(qk_rope_cache_kernel, true);
        else B2_ROPE(qk_rope_cache_kernel, false);
    });
#undef B2_ROPE
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

extern "C" int b2_chunk_attention(void* out, const void* q, const void* k_cache, const void* v_cache, int act_dtype,
                                  const int32_t* block_tables, int max_nb, const int32_t* cu_q, const int32_t* ctx_start,
                                  int n_seq, int T, int H, int G, int dk, int dv, int bs, float scale, int chunk, float sink,
                                  float sink_logit, void* stream) {
    return b2_masked_attention(out, q, k_cache, v_cache, act_dtype, block_tables, max_nb, cu_q, ctx_start, n_seq, T, H, G, dk, dv,
                               bs, scale, chunk, 0, 0, sink, sink_logit, nullptr, B2_WEIGHT_SOFTMAX, nullptr, nullptr, 0, 0.f, 1, 0.f,
                               0.f, 1.f, (int64_t)H * dv, stream);
}

extern "C" int b2_masked_attention(void* out, const void* q, const void* k_cache, const void* v_cache, int act_dtype,
                                   const int32_t* block_tables, int max_nb, const int32_t* cu_q, const int32_t* ctx_start,
                                   int n_seq, int T, int H, int G, int dk, int dv, int bs, float scale, int chunk, int window,
                                   int keep_first, float sink, float sink_logit, const float* sink_logits, int weight_kind,
                                   const float* head_bias, const void* gate, int64_t gate_stride, float softcap, int maps,
                                   float map_lambda, float map_eps, float map_scale, int64_t out_stride, void* stream) {
    B2_REQUIRE(T >= 0 && H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0 && bs > 0 && chunk >= 0 && sink >= 0.f && window >= 0 &&
               keep_first >= 0, B2_EINVAL, "masked_attention: bad sizes");
    B2_REQUIRE(!gate || gate_stride >= H, B2_EINVAL, "masked_attention: gate rows shorter than the heads");
    B2_REQUIRE(weight_kind == B2_WEIGHT_SOFTMAX || weight_kind == B2_WEIGHT_SIGMOID, B2_EINVAL,
               "masked_attention: unknown weight kind %d", weight_kind);
    const bool sig = weight_kind == B2_WEIGHT_SIGMOID;
    B2_REQUIRE(sig ? sink == 0.f : !head_bias, B2_EINVAL,
               "masked_attention: sigmoid weights have no sink, and only they take a bias per head");
    B2_REQUIRE(maps == 1 || maps == 2, B2_EINVAL, "masked_attention: %d maps per head", maps);
    B2_REQUIRE(!sig || (maps == 1 && softcap == 0.f), B2_EINVAL, "masked_attention: sigmoid weights have one map and no cap");
    B2_REQUIRE(softcap >= 0.f, B2_EINVAL, "masked_attention: negative cap");
    B2_REQUIRE(out_stride >= (int64_t)H * dv, B2_EINVAL, "masked_attention: output rows shorter than the heads");
    B2_REQUIRE(dv <= 32 * kMaxDvPerLane, B2_EUNSUPPORTED, "chunk_attention: value size %d above %d", dv, 32 * kMaxDvPerLane);
    if (T == 0 || n_seq == 0) return B2_OK;
    B2_REQUIRE(out && q && k_cache && v_cache && block_tables && cu_q && ctx_start, B2_EINVAL, "chunk_attention: null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const HeadShape hs{softcap, map_lambda, map_eps, map_scale};
    const int warps = 4;
    const size_t smem = (size_t)warps * dk * sizeof(float);
    B2_REQUIRE(smem <= 48 * 1024, B2_EUNSUPPORTED, "chunk_attention: key size %d too large", dk);
    const int items = T * H, blocks = (items + warps - 1) / warps;
    // prompt chunks of bf16 models with tensor-core friendly head sizes go to the tiled kernel (a sequence needs at least
    // kTileMinRows rows, so a batch of T rows over n_seq sequences can only hold one when T - n_seq >= kTileMinRows - 1)
    int skip_from = 0;
    const bool wide = dv == 192 || dv == 256;                // one softmax map only: the accumulators of two would not fit
    if (act_dtype == B2_ACT_BF16 && T - n_seq >= kTileMinRows - 1 && dk % 32 == 0 && dv % 32 == 0 && dk <= 128 &&
        (dv <= 128 || (wide && maps == 1 && !sig)) &&
        b2_aligned16(q) && b2_aligned16(k_cache) && b2_aligned16(v_cache) && b2_aligned16(out) && out_stride % 8 == 0) {
        skip_from = kTileMinRows;
        int rc = B2_OK;
        b2_prompt_args pa{};
        pa.q0 = q;
        pa.q0_row = (int64_t)H * maps * dk;
        pa.q0_head = maps * dk;
        pa.k0 = k_cache;
        pa.v = v_cache;
        pa.block_tables = block_tables;
        pa.max_nb = max_nb; pa.bs = bs; pa.cu_q = cu_q; pa.ctx_start = ctx_start; pa.n_seq = n_seq; pa.T = T;
        pa.H = H; pa.G = G; pa.dk0 = pa.dk = dk; pa.dv = dv; pa.maps = maps; pa.min_rows = kTileMinRows;
        pa.scale = scale; pa.chunk = chunk; pa.window = window; pa.keep_first = keep_first;
        pa.sink = sink; pa.sink_logit = sink_logit; pa.sink_logits = sink_logits; pa.head_bias = head_bias; pa.sigmoid = sig;
        pa.cap = softcap; pa.map_lambda = map_lambda; pa.map_eps = map_eps; pa.map_scale = map_scale;
        pa.gate = gate; pa.gate_stride = gate_stride; pa.out = out; pa.out_stride = out_stride;
        if (b2_internal_prompt_tc5_ok(pa)) {
            rc = b2_internal_prompt_tc5(pa, stream);
        } else {
#define B2_TILE(a, b, MAPS)                                                                                               \
    if (dk == 16 * a && dv == 16 * b)                                                                                     \
        rc = launch_tile<a, b, MAPS>(q, k_cache, v_cache, block_tables, max_nb, cu_q, ctx_start, n_seq, T, H, G, bs, scale, \
                                            chunk, window, keep_first, sink, sink_logit, sink_logits, gate, gate_stride, \
                                            hs, out, out_stride, st);
            if (maps == 2) {
                B2_TILE(6, 2, 2) B2_TILE(6, 4, 2) B2_TILE(6, 6, 2) B2_TILE(6, 8, 2)
                B2_TILE(8, 2, 2) B2_TILE(8, 4, 2) B2_TILE(8, 6, 2) B2_TILE(8, 8, 2)
            } else {
                B2_TILE(2, 12, 1) B2_TILE(4, 12, 1) B2_TILE(6, 12, 1) B2_TILE(8, 12, 1)
                B2_TILE(2, 16, 1) B2_TILE(4, 16, 1) B2_TILE(6, 16, 1) B2_TILE(8, 16, 1)
            }
#undef B2_TILE
        }
        if (rc != B2_OK) return rc;
    }
    if (act_dtype == B2_ACT_BF16 && dk % 32 == 0 && dk <= 256 && b2_aligned16(q) && b2_aligned16(k_cache) && b2_aligned16(v_cache)) {
        int rc = B2_EUNSUPPORTED;
#define B2_HEADS_RUN(b, SIG, MAPS)                                                                                        \
    launch_heads<b, SIG, MAPS>(q, k_cache, v_cache, block_tables, max_nb, cu_q, ctx_start, n_seq, T, H, G, dk, bs, scale, chunk, \
                               window, keep_first, sink, sink_logit, sink_logits, head_bias, gate, gate_stride, hs, skip_from, out, \
                               out_stride, st)
#define B2_HEADS(b) if (dv == 16 * b) rc = sig ? B2_HEADS_RUN(b, true, 1) : (maps == 2 ? B2_HEADS_RUN(b, false, 2) : B2_HEADS_RUN(b, false, 1));
        B2_HEADS(2) B2_HEADS(4) B2_HEADS(6) B2_HEADS(8) B2_HEADS(12) B2_HEADS(16)
#undef B2_HEADS
#undef B2_HEADS_RUN
        if (rc != B2_EUNSUPPORTED) return rc;
    }
    if (act_dtype == B2_ACT_BF16 && dk % 8 == 0 && dv % 8 == 0 && dv <= 64 * kGroupMaxPairs && b2_aligned16(q) &&
        b2_aligned16(k_cache) && b2_aligned16(v_cache) && b2_aligned16(out)) {
        const size_t gsm = (size_t)(kGroupMaxHeads * dk + 4 * kGroupMaxHeads * (2 + dv)) * sizeof(float) +
                           (size_t)4 * 32 * (maps * dk + 8 + dv) * sizeof(__nv_bfloat16);
        if (gsm <= 200 * 1024) {
            auto kern = sig ? chunk_attention_group_kernel<true, 1>
                            : (maps == 2 ? chunk_attention_group_kernel<false, 2> : chunk_attention_group_kernel<false, 1>);
            if (gsm > 48 * 1024) B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm));
            kern<<<dim3(T, G), 128, gsm, st>>>(static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k_cache),
                                               static_cast<const __nv_bfloat16*>(v_cache), block_tables, max_nb, cu_q, ctx_start,
                                               n_seq, H, G, dk, dv, bs, scale, chunk, window, keep_first, sink, sink_logit,
                                               sink_logits, head_bias, static_cast<const __nv_bfloat16*>(gate), gate_stride, hs,
                                               skip_from, static_cast<__nv_bfloat16*>(out), out_stride);
            B2_CUDA_OK(cudaGetLastError());
            return B2_OK;
        }
    }
#define B2_WARP_ATTENTION(SIG, MAPS)                                                                                          \
    chunk_attention_kernel<A, SIG, MAPS><<<blocks, warps * 32, smem, st>>>(                                                   \
        static_cast<const A*>(q), static_cast<const A*>(k_cache), static_cast<const A*>(v_cache), block_tables, max_nb, cu_q, \
        ctx_start, n_seq, T, H, G, dk, dv, bs, scale, chunk, window, keep_first, sink, sink_logit, sink_logits, head_bias,    \
        static_cast<const A*>(gate), gate_stride, hs, skip_from, static_cast<A*>(out), out_stride)
    B2_DISPATCH_ACT(act_dtype, A, {
        if (sig) B2_WARP_ATTENTION(true, 1);
        else if (maps == 2) B2_WARP_ATTENTION(false, 2);
        else B2_WARP_ATTENTION(false, 1);
    });
#undef B2_WARP_ATTENTION
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}
