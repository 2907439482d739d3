// moe_tc5.cu -- the two grouped products of moe.cu in bf16 on the 5th-gen tensor cores: per tile of 32 sorted (token, choice) rows,
// act = glu(h W_gate[e]^T, h W_up[e]^T) and rows = act W_down[e]^T.
//
// The weights are the M side of the product and the tile's rows the N side (32), so no weight row is padding however few tokens an
// expert has.  A CTA takes 128 weight rows of one row tile's expert -- 64 of W_gate and the same 64 of W_up, or 128 of W_up / W_down
// -- and runs over all of K in steps of 64 columns: one thread asks for the 16 KB of weights by TMA, a warp copies the 32 gathered
// rows with cp.async, one thread issues the MMAs into 32 columns of TMEM, and all four warps apply the activation and store.
// Bound: the weights' bytes, read once per row tile of their expert (more than one only above 32 rows an expert, from L2 then).
// Three CTAs of three stages share an SM: 144 KB of weights in flight, and one CTA's start and end lie under the others' streams.
#include "b2_act.cuh"
#include "b2_tc5.cuh"

namespace {
using namespace b2tc;
using bf16 = __nv_bfloat16;

constexpr int ROWS = 32, WROWS = 128, KSTEP = 64, NT = 128;
constexpr int W_STAGE = WROWS * KSTEP * 2, A_STAGE = ROWS * KSTEP * 2;

struct ExpertArgs {
    CUtensorMap map0, map1;                          // weight rows 0 - 63 and 64 - 127 of a CTA: W_gate | W_up, or the same matrix twice
    const bf16* a;                                   // GATHER: h, row of pair s / top; else the tile's own rows
    int64_t a_stride;
    const int32_t *sorted, *tile_expert;
    int top, K, N;                                   // weights [E, N, K]
    const float* in_w;
    void* out;                                       // act bf16 [cap, N], or rows fp32 [cap, N]
    int glu;
    float alpha, limit;
};

enum { PAIR, SINGLE, DOWN };                         // glu of two products; relu^2 of one; one product in fp32

template <int KIND, int ST>
__global__ void __launch_bounds__(NT)
moe_tc5_kernel(const __grid_constant__ ExpertArgs p) {
    extern __shared__ unsigned char moe_sm_raw[];
    __shared__ __align__(8) uint64_t s_full[ST], s_empty[ST], s_end;
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    const int e = p.tile_expert[blockIdx.x];
    if (e < 0) return;
    constexpr int OUT = KIND == PAIR ? 64 : 128;     // output columns of a CTA
    const int m0 = blockIdx.x * ROWS, n0 = blockIdx.y * OUT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sm = (b2::smem_u32(moe_sm_raw) + 1023u) & ~1023u, rows_sm = sm + ST * W_STAGE;
    volatile int* failed = &s_failed;
    auto full = [&](int s) { return b2::smem_u32(&s_full[s]); };
    auto empty = [&](int s) { return b2::smem_u32(&s_empty[s]); };
    if (tid == 0) {
        s_failed = 0;
        for (int s = 0; s < ST; ++s) {
            b2::mbar_init(full(s), 2);               // the weights' bytes, and the row warp
            b2::mbar_init(empty(s), 1);
        }
        b2::mbar_init(b2::smem_u32(&s_end), 1);
        b2::fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;" ::"r"(b2::smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int nk = (p.K + KSTEP - 1) / KSTEP;

    int sent = 0;                                    // k-steps whose weights this thread has asked for
    if (warp == 0) {
        if (lane == 0) {
#pragma unroll 1
            for (int it = 0; it < nk; ++it) {
                const int s = it % ST;
                if (it >= ST && !wait(empty(s), (it / ST - 1) & 1, failed)) break;
                sent = it + 1;
                b2::mbar_arrive_expect_tx(full(s), W_STAGE);         // columns and rows past the matrix are zero-filled and count
                tma_load_3d(sm + s * W_STAGE, &p.map0, full(s), it * KSTEP, n0, e);
                tma_load_3d(sm + s * W_STAGE + W_STAGE / 2, &p.map1, full(s), it * KSTEP, KIND == PAIR ? n0 : n0 + 64, e);
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t ID = idesc_bf16(WROWS, ROWS, 0);
        const uint32_t w_lo = desc_lo(sm, 16), r_lo = desc_lo(rows_sm, 16);
#pragma unroll 1
        for (int it = 0; it < nk; ++it) {
            const int s = it % ST;
            wait(full(s), (it / ST) & 1, failed);
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < KSTEP / 16; ++kk)
                    mma_ss(tmem, desc_join(w_lo + s * (W_STAGE >> 4) + kk * 2), desc_join(r_lo + s * (A_STAGE >> 4) + kk * 2), ID, it > 0 || kk > 0);
                mma_commit(it + 1 < nk ? empty(s) : b2::smem_u32(&s_end));
            }
            __syncwarp();
        }
    } else if (warp == 2) {
        // lane: 16-byte column lane & 7 of rows lane / 8 + 4 i; a padding row (no pair) is zeros
        constexpr int LAG = ST - 2;                  // k-steps whose copies are in flight when a step is handed over
        const char* src[8];
        uint32_t there = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = (lane >> 3) + 4 * i, pair = p.sorted[m0 + r];
            if (pair >= 0) there |= 1u << i;
            const int64_t row = KIND == DOWN ? m0 + r : (pair >= 0 ? pair / p.top : 0);
            src[i] = reinterpret_cast<const char*>(p.a + row * p.a_stride + (lane & 7) * 8);
        }
        auto hand_over = [&](int it) {
            b2::fence_proxy_async();                 // this lane's copies, before the MMAs that read them
            __syncwarp();
            if (lane == 0) b2::mbar_arrive(full(it % ST));
        };
#pragma unroll 1
        for (int it = 0; it < nk; ++it) {
            const int s = it % ST;
            if (it >= ST) wait(empty(s), (it / ST - 1) & 1, failed);
            const bool in = it * KSTEP + (lane & 7) * 8 < p.K;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = (lane >> 3) + 4 * i;
                const uint32_t dst = rows_sm + s * A_STAGE + r * 128 + (((lane & 7) ^ (r & 7)) << 4);
                const bool ok = in && ((there >> i) & 1);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                             ::"r"(dst), "l"(ok ? src[i] + (size_t)it * KSTEP * 2 : reinterpret_cast<const char*>(p.a)), "r"(ok ? 16 : 0) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (it >= LAG) {
                asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                hand_over(it - LAG);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        for (int it = nk > LAG ? nk - LAG : 0; it < nk; ++it) hand_over(it);
    }
    __syncwarp();
    wait(b2::smem_u32(&s_end), 0, failed);
    tc_fence_after();
    uint32_t acc[ROWS];
    tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16), acc);            // this thread's weight row against the tile's 32 rows
    tmem_wait_ld();
    const bool bad = *failed != 0;
    if constexpr (KIND == DOWN) {
        const int n = n0 + tid;
        float* o = static_cast<float*>(p.out) + (size_t)m0 * p.N + n;
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
            if (n < p.N && p.sorted[m0 + r] >= 0) o[(size_t)r * p.N] = bad ? __int_as_float(0x7fc00000) : __uint_as_float(acc[r]);
    } else {
        float* c_sm = reinterpret_cast<float*>(moe_sm_raw + (sm - b2::smem_u32(moe_sm_raw)));      // [32][128]: every MMA has read its stage
#pragma unroll
        for (int r = 0; r < ROWS; ++r) c_sm[r * WROWS + tid] = __uint_as_float(acc[r]);
        __syncthreads();
        for (int idx = tid; idx < ROWS * OUT; idx += NT) {
            const int r = idx / OUT, c = idx % OUT, pair = p.sorted[m0 + r];
            if (n0 + c >= p.N || pair < 0) continue;
            const float wt = p.in_w ? p.in_w[pair] : 1.f;            // weight on the expert's input: W (wt h) = wt (W h)
            float v;
            if constexpr (KIND == SINGLE) {
                v = b2::relu_sq_f(wt * c_sm[r * WROWS + c]);
            } else {
                const float g = wt * c_sm[r * WROWS + c], u = wt * c_sm[r * WROWS + 64 + c];
                v = p.glu == B2_GLU_CLAMPED ? b2::glu_clamped_f(g, u, p.alpha, p.limit) : b2::silu_f(g) * u;
            }
            b2::st(static_cast<bf16*>(p.out) + (size_t)(m0 + r) * p.N + n0 + c, bad ? __int_as_float(0x7fc00000) : v);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*failed) {                                   // what nobody has waited for: every role is done now
        drain(b2::smem_u32(&s_end), 0);
        for (int back = 1; back <= min(ST, sent); ++back) drain(full((sent - back) % ST), ((sent - back) / ST) & 1);
        __syncwarp();
    }
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;" ::"r"(tmem) : "memory");
}

// weights [experts, N, K], experts `stride` elements apart; the expert ids are the caller's, 65536 only has to be above them
int encode(CUtensorMap* map, const void* w, int64_t stride, int N, int K) {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, 65536}, st[2] = {(uint64_t)K * 2, (uint64_t)stride * 2};
    const uint32_t box[3] = {KSTEP, 64, 1};
    return b2_internal_encode_bf16_sw128(map, w, 3, dims, st, box);
}

template <int KIND>
int launch(const ExpertArgs& p, int tiles, cudaStream_t st) {
    constexpr int ST = 3, OUT = KIND == PAIR ? 64 : 128, SMEM = ST * (W_STAGE + A_STAGE) + 1024;
    auto kern = moe_tc5_kernel<KIND, ST>;
    B2_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    kern<<<dim3(tiles, (p.N + OUT - 1) / OUT), NT, SMEM, st>>>(p);
    B2_CUDA_OK(cudaGetLastError());
    return B2_OK;
}

}  // namespace

bool b2_internal_moe_tc5_ok(const void* h, int64_t h_stride, const void* w_gate, const void* w_up, const void* w_down,
                            int64_t w13_expert_stride, int D, int F, const void* act) {
    // 16-byte rows and at least one whole box of each matrix
    return D % 8 == 0 && F % 8 == 0 && D >= 64 && F >= 64 && h_stride % 8 == 0 && w13_expert_stride % 8 == 0 && b2_aligned16(h) &&
           b2_aligned16(w_gate) && b2_aligned16(w_up) && b2_aligned16(w_down) && b2_aligned16(act) && w13_expert_stride < (int64_t)1 << 38;
}

int b2_internal_moe_gate_up_tc5(const void* h, int64_t h_stride, const void* w_gate, const void* w_up, int64_t w13_expert_stride,
                                const int32_t* sorted, const int32_t* tile_expert, int tiles, int top, int D, int F, int glu, float alpha,
                                float limit, const float* in_w, void* act, void* stream) {
    const bool gated = glu != B2_FF_RELU_SQ;
    ExpertArgs p{};
    int rc = encode(&p.map0, gated ? w_gate : w_up, w13_expert_stride, F, D);
    if (rc == B2_OK) rc = encode(&p.map1, w_up, w13_expert_stride, F, D);
    if (rc != B2_OK) return rc;
    p.a = static_cast<const bf16*>(h);
    p.a_stride = h_stride;
    p.sorted = sorted; p.tile_expert = tile_expert; p.top = top; p.K = D; p.N = F; p.in_w = in_w; p.out = act;
    p.glu = glu; p.alpha = alpha; p.limit = limit;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return gated ? launch<PAIR>(p, tiles, st) : launch<SINGLE>(p, tiles, st);
}

int b2_internal_moe_down_tc5(const void* act, const void* w_down, const int32_t* sorted, const int32_t* tile_expert, int tiles, int D,
                             int F, float* rows, void* stream) {
    ExpertArgs p{};
    int rc = encode(&p.map0, w_down, (int64_t)D * F, D, F);
    if (rc != B2_OK) return rc;
    p.map1 = p.map0;
    p.a = static_cast<const bf16*>(act);
    p.a_stride = F;
    p.sorted = sorted; p.tile_expert = tile_expert; p.top = 1; p.K = F; p.N = D; p.out = rows;
    return launch<DOWN>(p, tiles, static_cast<cudaStream_t>(stream));
}
