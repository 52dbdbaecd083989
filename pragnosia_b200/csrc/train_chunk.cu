// Training through the chunked scan on the tensor cores: the backward of the plain and the delta rule as a few
// chunk-parallel kernels around the one thing that is sequential, the gradient G_c on the state entering each chunk.
// (Reference: src/assoc_kernel.py:75-126 _bwd_chunk, 206-221 _prefix_bwd, 390-459 _delta_loop_bwd, 626-656 _inv_bwd.)
//
//   o_t = sum_{s<=t} P_ts dec_ts W_s + e^{L_t} q_t S,   S' = e^{L_C} S + sum_s w_s k_s W_s^T,   dec_ts = e^{L_t-L_s}, w_s = e^{L_C-L_s}
//   plain: W = V.   delta: W = X beta (V - e^L K S),  X = (I + N)^-1,  N_ts = beta_t (k_t.k_s) dec_ts for s < t.
//
//   1. train_pre_kernel (a CTA per chunk):   D_c = (Q e^L)^T dO;  delta: dW0 = A^T dO as well (A = P dec)
//   2. plain: state_grad_scan_kernel, elementwise over the chunks backwards:  G_c = e^{L_C} G_{c+1} + D_c
//      delta: delta_walk_kernel<D, true>:  dW = dW0 + w K G,  dR = X^T dW,  G_c = e^{L_C} G_{c+1} + D_c - (K beta e^L)^T dR
//   3. train_post_kernel (a CTA per chunk): everything else, as two groups of products with one pass over registers between.
//
// The unfused operators (split_ops_bwd.cu) form the gradient of X and pull it back through the inverse; here
// dN = -X^T dX X^T collapses to -dR W^T, because dX = dW rhs^T and X rhs = W.
//
// Operands that are fp32 (A, dP = dA dec, dR, G, Q e^L) enter the tensor cores as bf16 head and tail; q, k, v, do, the saved
// states and W are bf16 as the operators hand them on.
//
// The chunk kernels are bound by latency and by the shared-memory passes between their two groups of products; several CTAs
// share an SM at D = 64. At B4 H11 T2048 D64 (1408 chunks): plain pre 13 + scan 10 + post 40 us, where the FFMA operators
// took 698 + 641 us (assoc_out_bwd, prefix_scan_bwd); delta pre 21 + walk 93 + post 47 us against 3134 + 696 + 411 us
// (delta_loop_bwd, assoc_out_bwd, delta_inv_bwd).
#include "delta_walk.cuh"

namespace pgb {

constexpr int TR_NT = 256;
constexpr float TR_LOG2E = 1.4426950408889634f;

struct TrainMaps { CUtensorMap q, k, v, dout, s, g, dr; };            // v: W under the delta rule
struct TrainParams {
    const float *la, *beta;
    const __nv_bfloat16 *v;                                           // delta, post: V itself
    const float *dsent;
    float *Dc, *dW0, *Ltot;                                           // pre out
    __nv_bfloat16 *dq, *dk, *dv;
    float *dla, *dbeta;
    int BH, T;
};

// The chunk's statistics by warp 0: L, e^L, w = e^{L_C - L} (0 past T), beta; a lane owns tokens l and l + 32.
__device__ __forceinline__ void tr_stats(const float *la, const float *beta, int t0, int T, int lane, float *Ls, float *eLs, float *wts, float *bes) {
    const int a = t0 + lane, b = a + 32;
    float sl = a < T ? la[a] : 0.f, sh = b < T ? la[b] : 0.f;
    if (beta != nullptr) { bes[lane] = a < T ? beta[a] : 0.f; bes[lane + 32] = b < T ? beta[b] : 0.f; }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float nl = __shfl_up_sync(0xffffffffu, sl, o), nh = __shfl_up_sync(0xffffffffu, sh, o);
        if (lane >= o) { sl += nl; sh += nh; }
    }
    sh += __shfl_sync(0xffffffffu, sl, 31);
    const float tot = __shfl_sync(0xffffffffu, sh, 31);
    Ls[lane] = sl; Ls[lane + 32] = sh;
    eLs[lane] = expf(sl); eLs[lane + 32] = expf(sh);
    wts[lane] = a < T ? expf(fminf(tot - sl, 0.f)) : 0.f;
    wts[lane + 32] = b < T ? expf(fminf(tot - sh, 0.f)) : 0.f;
}

// the products, issued by a whole converged warp (one elected lane). K-major step k of a tile of 64-column sub-tiles
// `sub_bytes` apart; rows of 16 for an operand whose rows are the contraction
__device__ __forceinline__ uint32_t tr_ko(int k, uint32_t sub_bytes) { return ((uint32_t)(k >> 2) * sub_bytes + (uint32_t)(k & 3) * 32u) >> 4; }

// ------------------------------------------------------------------------------------------------ 1. before the sequential part
template <int D, bool DELTA>
struct PreSmem {
    static constexpr int QK = TC_C * D * 2, SQ = TC_C * TC_C * 2;
    static constexpr int o_q = 0, o_do = QK, o_qh = 2 * QK, o_ql = 3 * QK, o_k = 4 * QK, o_ah = o_k + (DELTA ? QK : 0), o_al = o_ah + (DELTA ? SQ : 0);
    static constexpr int off_misc = o_al + (DELTA ? SQ : 0), bytes = off_misc + 64 + 4 * 256 + 1024;
    static constexpr int TMC = (D == 64 ? 64 : 128) + (DELTA ? 64 + D : 0), TM_COLS = TMC <= 64 ? 64 : TMC <= 128 ? 128 : TMC <= 256 ? 256 : 512;
};

template <int D, bool DELTA>
__global__ void __launch_bounds__(TR_NT) train_pre_kernel(const __grid_constant__ TrainMaps m, TrainParams p) {
    using SM = PreSmem<D, DELTA>;
    constexpr int SUB = D / 64, HALF = D / 2, NSG = D / 64;
    constexpr uint32_t TM_D = 0, TM_P = D, TM_W = D + 64;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    uint8_t *misc = sm + SM::off_misc;
    const uint32_t bar_t = base + SM::off_misc, bar_1 = bar_t + 8, bar_2 = bar_t + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + 32);
    float *Ls = reinterpret_cast<float *>(misc + 64), *eLs = Ls + 64, *wts = eLs + 64, *bes = wts + 64;
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5), wg = warp >> 2, sub = warp & 3;
    const int c = blockIdx.x, bh = blockIdx.y, NC = gridDim.x, T = p.T, t0 = c * TC_C;
    if (tid == 0) {
        mbar_init(bar_t, 1); mbar_init(bar_1, 1); mbar_init(bar_2, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(bar_t, (DELTA ? 3 : 2) * SM::QK);
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            tma_load_3d(base + SM::o_q + s * 8192, &m.q, bar_t, 64 * s, t0, bh);
            tma_load_3d(base + SM::o_do + s * 8192, &m.dout, bar_t, 64 * s, t0, bh);
            if (DELTA) tma_load_3d(base + SM::o_k + s * 8192, &m.k, bar_t, 64 * s, t0, bh);
        }
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), SM::TM_COLS);
    if (warp == 0) tr_stats(p.la + (size_t)bh * T, nullptr, t0, T, lane, Ls, eLs, wts, bes);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    pdl_launch_dependents();                                          // this CTA has its tensor memory
    if (tid == 0) p.Ltot[(size_t)bh * NC + c] = Ls[TC_C - 1];
    bool ok = mbar_wait_warp(bar_t, 0, 21);
    if (DELTA && warp == 2 && ok) {
        const uint64_t dq = smem_desc(base + SM::o_q, 16, 1024), dk = smem_desc(base + SM::o_k, 16, 1024);
        constexpr uint32_t I_P = idesc_bf16(64, 64, 0, 0);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) mma_bf16_elect(tmem + TM_P, dq + tr_ko(k, 8192), dk + tr_ko(k, 8192), I_P, k > 0);
        mma_commit_elect(bar_1);
    }
    if (ok) {                                                         // Q e^L, head and tail, in Q's own layout
        for (int idx = tid; idx < TC_C * (D / 8); idx += TR_NT) {
            const int r = idx / (D / 8), jj = idx % (D / 8);
            const uint32_t off = (uint32_t)(jj >> 3) * 8192u + swz(r, jj & 7);
            const uint4 raw = *reinterpret_cast<const uint4 *>(sm + SM::o_q + off);
            const __nv_bfloat162 *b2 = reinterpret_cast<const __nv_bfloat162 *>(&raw);
            const float e = eLs[r];
            float x[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(b2[i]); x[2 * i] = f.x * e; x[2 * i + 1] = f.y * e; }
            uint4 hi, lo;
            split8(x, hi, lo);
            *reinterpret_cast<uint4 *>(sm + SM::o_qh + off) = hi;
            *reinterpret_cast<uint4 *>(sm + SM::o_ql + off) = lo;
        }
    }
    const int fr = lane >> 2, fq = lane & 3, row0 = 16 * sub + fr, row1 = row0 + 8;
    const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16);
    if (DELTA && ok) {                                                // A = P dec, head and tail
        ok = mbar_wait_warp(bar_1, 0, 22);
        tc_fence_after();
        float pv[16];
        tmem_ld_frag4(lb + TM_P + 32 * wg, pv);
        const float L0 = Ls[row0] * TR_LOG2E, L1 = Ls[row1] * TR_LOG2E;
        float2 Lc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { Lc[j] = *reinterpret_cast<const float2 *>(Ls + 32 * wg + 8 * j + 2 * fq); Lc[j].x *= TR_LOG2E; Lc[j].y *= TR_LOG2E; }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int s = 32 * wg + 8 * j + 2 * fq;
            const float a00 = s <= row0 ? pv[4 * j] * fast_exp2(fminf(L0 - Lc[j].x, 0.f)) : 0.f, a01 = s + 1 <= row0 ? pv[4 * j + 1] * fast_exp2(fminf(L0 - Lc[j].y, 0.f)) : 0.f;
            const float a10 = s <= row1 ? pv[4 * j + 2] * fast_exp2(fminf(L1 - Lc[j].x, 0.f)) : 0.f, a11 = s + 1 <= row1 ? pv[4 * j + 3] * fast_exp2(fminf(L1 - Lc[j].y, 0.f)) : 0.f;
            const uint32_t o0 = swz(row0, 4 * wg + j) + 4 * fq, o1 = swz(row1, 4 * wg + j) + 4 * fq;
            uint32_t hi, lo;
            split2(a00, a01, hi, lo);
            *reinterpret_cast<uint32_t *>(sm + SM::o_ah + o0) = hi; *reinterpret_cast<uint32_t *>(sm + SM::o_al + o0) = lo;
            split2(a10, a11, hi, lo);
            *reinterpret_cast<uint32_t *>(sm + SM::o_ah + o1) = hi; *reinterpret_cast<uint32_t *>(sm + SM::o_al + o1) = lo;
        }
    }
    fence_proxy_async();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (warp == 2 && ok) {
        constexpr uint32_t I_D = idesc_bf16(D, D, 1, 1), I_W = idesc_bf16(64, D, 1, 1);
        const uint64_t dh = smem_desc(base + SM::o_qh, 8192, 1024), dl = smem_desc(base + SM::o_ql, 8192, 1024), dd = smem_desc(base + SM::o_do, 8192, 1024);
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem + TM_D, (half ? dl : dh) + k * 128, dd + k * 128, I_D, half | (k > 0));
        if constexpr (DELTA) {
            const uint64_t ah = smem_desc(base + SM::o_ah, 8192, 1024), al = smem_desc(base + SM::o_al, 8192, 1024);
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem + TM_W, (half ? al : ah) + k * 128, dd + k * 128, I_W, half | (k > 0));
        }
        mma_commit_elect(bar_2);
    }
    if (ok) ok = mbar_wait_warp(bar_2, 0, 23);
    tc_fence_after();
    if (ok) {
        float *dst = p.Dc + ((size_t)bh * NC + c) * D * D;
        const float *ds = p.dsent != nullptr ? p.dsent + ((size_t)bh * NC + c) * D * D : nullptr;
#pragma unroll
        for (int g = 0; g < NSG; ++g)
#pragma unroll
            for (int cb = 0; cb < HALF; cb += 32) {
                float x[16];
                tmem_ld_frag4(lb + ((uint32_t)(16 * g) << 16) + TM_D + HALF * wg + cb, x);
                tmem_ld_wait();
#pragma unroll
                for (int hi8 = 0; hi8 < 2; ++hi8) {
                    const size_t off = (size_t)((D == 128 ? 32 * sub + 16 * g : 16 * sub) + fr + 8 * hi8) * D + HALF * wg + cb + 2 * fq;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float2 y = make_float2(x[4 * j + 2 * hi8], x[4 * j + 2 * hi8 + 1]);
                        if (ds != nullptr) { const float2 a = *reinterpret_cast<const float2 *>(ds + off + 8 * j); y.x += a.x; y.y += a.y; }
                        *reinterpret_cast<float2 *>(dst + off + 8 * j) = y;
                    }
                }
            }
        if constexpr (DELTA) {
#pragma unroll
            for (int cb = 0; cb < HALF; cb += 32) {
                float x[16];
                tmem_ld_frag4(lb + TM_W + HALF * wg + cb, x);
                tmem_ld_wait();
#pragma unroll
                for (int hi8 = 0; hi8 < 2; ++hi8) {
                    const int t = t0 + (hi8 ? row1 : row0);
                    if (t < T)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            *reinterpret_cast<float2 *>(p.dW0 + ((size_t)bh * T + t) * D + HALF * wg + cb + 8 * j + 2 * fq) =
                                make_float2(x[4 * j + 2 * hi8], x[4 * j + 2 * hi8 + 1]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, SM::TM_COLS);
}

// ------------------------------------------------------------------------------------------------ 2. plain rule: G over the chunks
// A thread owns four adjacent elements of one chain's state: 16-byte loads, four chunks requested ahead of the recurrence.
// G [BH][NC][2][D*D]: the gradient on the state LEAVING chunk c, head and tail. dS: gradient on the final state or NULL.
__global__ void __launch_bounds__(256) state_grad_scan_kernel(const float *__restrict__ Dc, const float *__restrict__ Ltot, const float *__restrict__ dS,
                                                              __nv_bfloat16 *__restrict__ G, float *__restrict__ dS0, int NC, int DD) {
    const int e = (blockIdx.x * 256 + threadIdx.x) * 4, bh = blockIdx.y;
    pdl_launch_dependents();
    if (e >= DD) return;
    pdl_wait();
    float4 g = dS != nullptr ? *reinterpret_cast<const float4 *>(dS + (size_t)bh * DD + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float *src = Dc + (size_t)bh * NC * DD + e;
    const float *lt = Ltot + (size_t)bh * NC;
    for (int c1 = NC; c1 > 0; c1 -= 4) {
        float4 d[4];
        float a[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = c1 - 1 - j;
            if (c >= 0) { d[j] = *reinterpret_cast<const float4 *>(src + (size_t)c * DD); a[j] = expf(lt[c]); }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = c1 - 1 - j;
            if (c < 0) break;
            uint2 hi, lo;
            split2(g.x, g.y, hi.x, lo.x);
            split2(g.z, g.w, hi.y, lo.y);
            __nv_bfloat16 *dst = G + ((size_t)bh * NC + c) * 2 * DD + e;
            *reinterpret_cast<uint2 *>(dst) = hi;
            *reinterpret_cast<uint2 *>(dst + DD) = lo;
            g.x = fmaf(a[j], g.x, d[j].x); g.y = fmaf(a[j], g.y, d[j].y); g.z = fmaf(a[j], g.z, d[j].z); g.w = fmaf(a[j], g.w, d[j].w);
        }
    }
    if (dS0 != nullptr) *reinterpret_cast<float4 *>(dS0 + (size_t)bh * DD + e) = g;
}

// ------------------------------------------------------------------------------------------------ 3. after it
template <int D, bool DELTA>
struct PostSmem {
    static constexpr int QK = TC_C * D * 2, SQ = TC_C * TC_C * 2, ST = D * D * 2;
    static constexpr int o_q = 0, o_k = QK, o_v = 2 * QK, o_do = 3 * QK, o_gh = 4 * QK, o_gl = o_gh + ST, o_drh = o_gl + ST,
                         o_drl = o_drh + (DELTA ? QK : 0), o_s = o_drl + (DELTA ? QK : 0);
    // the operands of the second group: dP, and A (plain) or C (delta). At D = 128 under the delta rule they take the place
    // of S, which the first group is through with (224 KB of tiles otherwise)
    static constexpr bool alias = DELTA && D == 128;
    static constexpr int o_ph = alias ? o_s : o_s + ST, o_pl = o_ph + SQ, o_ah = o_pl + SQ, o_al = o_ah + SQ;
    static constexpr int off_misc = alias ? o_s + ST : o_al + SQ;
    static constexpr int bytes = off_misc + 64 + 4 * 256 + 5 * 512 + 5 * 256 + 64 + 1024;    // statistics, row and column sums, <G, S>
    static constexpr int LOADED = 4 * QK + 3 * ST + (DELTA ? 2 * QK : 0);
    static constexpr int TM_COLS = D == 64 ? 256 : 512;
};

// At D = 64 half of the tensor memory has to do, so that two CTAs share an SM (delta, B4 H11 T2048: 57 -> 47 us). The delta rule's first group
// then leaves out R and R2, which follow into the columns of P and E once those have been read, under the pass over registers.
template <int D, bool DELTA>
__global__ void __launch_bounds__(TR_NT, D == 64 ? 2 : 1) train_post_kernel(const __grid_constant__ TrainMaps m, TrainParams p) {
    using SM = PostSmem<D, DELTA>;
    constexpr int SUB = D / 64, HALF = D / 2, NB = D / 64;            // NB: 32-column blocks of this warp's half of a D-wide accumulator
    // first group: P, dA, R = dO S^T (all); plain: VG = V G^T; delta: KK, E = dR W^T, R2 = dR S^T
    constexpr uint32_t TM_P = 0, TM_DA = 64, TM_KK = 128, TM_E = 192, TM_R = DELTA ? (D == 64 ? 0 : 256) : 128, TM_VG = DELTA && D == 64 ? 192 : TM_R + D;   // delta: R2 in VG's place
    constexpr bool TIGHT = DELTA && D == 64;
    // second group: dQ = dP K, dK = dP^T Q (+ C K + C^T K); plain: dV = A^T dO, KG = K G; delta: WG = W G^T
    constexpr uint32_t TM_DK = DELTA ? D : (D == 64 ? 64 : 384), TM_DV = 0, TM_DQ = DELTA ? 0 : TM_R, TM_KG = DELTA ? (D == 64 ? 128 : TM_R) : TM_VG;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    uint8_t *misc = sm + SM::off_misc;
    const uint32_t bar_t = base + SM::off_misc, bar_1 = bar_t + 8, bar_2 = bar_t + 16, bar_r = bar_t + 24;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + 32);
    float *Ls = reinterpret_cast<float *>(misc + 64), *eLs = Ls + 64, *wts = eLs + 64, *bes = wts + 64;
    float *rr = bes + 64;                                             // row sums [quantity][column half][64]: gm, q.R, k.VG, dbeta part, k.R2
    float *cs = rr + 5 * 128;                                         // column sums of gm [row quarter][64]
    float *gs = cs + 320;                                             // (cs[256..]: dR . V per row), <G, S> per warp
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5), wg = warp >> 2, sub = warp & 3;
    const int c = blockIdx.x, bh = blockIdx.y, NC = gridDim.x, T = p.T, t0 = c * TC_C;
    pdl_wait();
    if (tid == 0) {
        mbar_init(bar_t, 1); mbar_init(bar_1, 1); mbar_init(bar_2, 1); mbar_init(bar_r, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(bar_t, SM::LOADED);
        const int ci = bh * NC + c;
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            tma_load_3d(base + SM::o_q + s * 8192, &m.q, bar_t, 64 * s, t0, bh);
            tma_load_3d(base + SM::o_k + s * 8192, &m.k, bar_t, 64 * s, t0, bh);
            tma_load_3d(base + SM::o_v + s * 8192, &m.v, bar_t, 64 * s, t0, bh);
            tma_load_3d(base + SM::o_do + s * 8192, &m.dout, bar_t, 64 * s, t0, bh);
            tma_load_3d(base + SM::o_gh + s * D * 128, &m.g, bar_t, 64 * s, 0, 2 * ci);
            tma_load_3d(base + SM::o_gl + s * D * 128, &m.g, bar_t, 64 * s, 0, 2 * ci + 1);
            tma_load_3d(base + SM::o_s + s * D * 128, &m.s, bar_t, 64 * s, 0, ci);
            if (DELTA) {
                tma_load_3d(base + SM::o_drh + s * 8192, &m.dr, bar_t, 64 * s, t0, bh);
                tma_load_3d(base + SM::o_drl + s * 8192, &m.dr, bar_t, 64 * s, t0, p.BH + bh);
            }
        }
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), SM::TM_COLS);
    if (warp == 0) tr_stats(p.la + (size_t)bh * T, DELTA ? p.beta + (size_t)bh * T : nullptr, t0, T, lane, Ls, eLs, wts, bes);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    bool ok = mbar_wait_warp(bar_t, 0, 31);
    const uint64_t q_k = smem_desc(base + SM::o_q, 16, 1024), k_k = smem_desc(base + SM::o_k, 16, 1024), v_k = smem_desc(base + SM::o_v, 16, 1024),
                   do_k = smem_desc(base + SM::o_do, 16, 1024), s_k = smem_desc(base + SM::o_s, 16, 1024), gh_k = smem_desc(base + SM::o_gh, 16, 1024),
                   gl_k = smem_desc(base + SM::o_gl, 16, 1024), drh_k = smem_desc(base + SM::o_drh, 16, 1024), drl_k = smem_desc(base + SM::o_drl, 16, 1024);
    constexpr uint32_t I_SQ = idesc_bf16(64, 64, 0, 0), I_RD = idesc_bf16(64, D, 0, 0);
    // rows of a tile times rows of a tile (contraction over the D columns); B's sub-tiles sub_b bytes apart
    auto rows_rows = [&](uint32_t acc, uint64_t a, uint64_t b, uint32_t sub_b, uint32_t idesc, uint32_t onto) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k) mma_bf16_elect(tmem + acc, a + tr_ko(k, 8192), b + tr_ko(k, sub_b), idesc, onto | (k > 0));
    };
    auto states = [&]() {                                             // R = dO S^T, R2 = dR S^T
        if constexpr (DELTA) {
            rows_rows(TM_VG, drh_k, s_k, D * 128, I_RD, 0);
            rows_rows(TM_VG, drl_k, s_k, D * 128, I_RD, 1);
        }
        rows_rows(TM_R, do_k, s_k, D * 128, I_RD, 0);
    };
    if (warp == 2 && ok) {
        rows_rows(TM_P, q_k, k_k, 8192, I_SQ, 0);
        rows_rows(TM_DA, do_k, v_k, 8192, I_SQ, 0);
        if constexpr (DELTA) {
            rows_rows(TM_KK, k_k, k_k, 8192, I_SQ, 0);
            rows_rows(TM_E, drh_k, v_k, 8192, I_SQ, 0);
            rows_rows(TM_E, drl_k, v_k, 8192, I_SQ, 1);
        } else {
            rows_rows(TM_VG, v_k, gh_k, D * 128, I_RD, 0);
            rows_rows(TM_VG, v_k, gl_k, D * 128, I_RD, 1);
        }
        if constexpr (!TIGHT) states();
        mma_commit_elect(bar_1);
    }
    // <G, S> while they run: the same bytes of two tiles of one layout
    {
        float part = 0.f;
        if (ok)
            for (int idx = tid; idx < SM::ST / 16; idx += TR_NT) {
                const uint4 a = *reinterpret_cast<const uint4 *>(sm + SM::o_s + idx * 16), h = *reinterpret_cast<const uint4 *>(sm + SM::o_gh + idx * 16),
                            l = *reinterpret_cast<const uint4 *>(sm + SM::o_gl + idx * 16);
                const __nv_bfloat162 *a2 = reinterpret_cast<const __nv_bfloat162 *>(&a), *h2 = reinterpret_cast<const __nv_bfloat162 *>(&h),
                                     *l2 = reinterpret_cast<const __nv_bfloat162 *>(&l);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 s = __bfloat1622float2(a2[i]), x = __bfloat1622float2(h2[i]), y = __bfloat1622float2(l2[i]);
                    part = fmaf(s.x, x.x + y.x, fmaf(s.y, x.y + y.y, part));
                }
            }
        part = warp_sum(part);
        if (lane == 0) gs[warp] = part;
    }
    if (ok) ok = mbar_wait_warp(bar_1, 0, 32);
    ok = __syncthreads_and(ok);                                       // every read of S ahead of what may take its place
    tc_fence_after();
    const int fr = lane >> 2, fq = lane & 3, row0 = 16 * sub + fr, row1 = row0 + 8;
    const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16);
    auto row_out = [&](int which, float a, float b) {                 // this thread's share of two row sums -> the quad -> [which][wg][row]
        a += __shfl_xor_sync(0xffffffffu, a, 1); a += __shfl_xor_sync(0xffffffffu, a, 2);
        b += __shfl_xor_sync(0xffffffffu, b, 1); b += __shfl_xor_sync(0xffffffffu, b, 2);
        if (fq == 0) { rr[which * 128 + wg * 64 + row0] = a; rr[which * 128 + wg * 64 + row1] = b; }
    };
    // x[16]: this thread's fragment of columns cb.. of a 64 x D product; dot with the same places of a bf16 tile, per row
    auto row_dot = [&](int o_tile, int cb, const float *x, float &a, float &b) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = cb + 8 * j;
            const uint8_t *t = sm + o_tile + (col >> 6) * 8192 + 4 * fq;
            const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(t + swz(row0, (col & 63) >> 3)));
            const float2 w = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(t + swz(row1, (col & 63) >> 3)));
            a = fmaf(u.x, x[4 * j], fmaf(u.y, x[4 * j + 1], a));
            b = fmaf(w.x, x[4 * j + 2], fmaf(w.y, x[4 * j + 3], b));
        }
    };
    float R[NB][16], VG[DELTA ? 1 : NB][16];
    if (ok) {
        const int col0 = 32 * wg;
        float pv[16], da[16], kk[DELTA ? 16 : 1], ev[DELTA ? 16 : 1];
        tmem_ld_frag4(lb + TM_P + col0, pv);
        tmem_ld_frag4(lb + TM_DA + col0, da);
        if constexpr (DELTA) { tmem_ld_frag4(lb + TM_KK + col0, kk); tmem_ld_frag4(lb + TM_E + col0, ev); }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            if constexpr (!TIGHT) tmem_ld_frag4(lb + TM_R + HALF * wg + 32 * b, R[b]);
            if constexpr (!DELTA) tmem_ld_frag4(lb + TM_VG + HALF * wg + 32 * b, VG[b]);
        }
        const float L0 = Ls[row0] * TR_LOG2E, L1 = Ls[row1] * TR_LOG2E, be0 = DELTA ? bes[row0] : 0.f, be1 = DELTA ? bes[row1] : 0.f;
        float2 Lc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { Lc[j] = *reinterpret_cast<const float2 *>(Ls + col0 + 8 * j + 2 * fq); Lc[j].x *= TR_LOG2E; Lc[j].y *= TR_LOG2E; }
        tmem_ld_wait();
        if constexpr (TIGHT) {
            tc_fence_before();
            __syncthreads();                                          // every warp has its fragments (ok is the same for the whole CTA)
            tc_fence_after();
            if (warp == 2) { states(); mma_commit_elect(bar_r); }
        }
        float g0 = 0.f, g1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t hp[2], lp[2], ha[2], la2[2];
            float gc[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float av[2], dp[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int s = col0 + 8 * j + 2 * fq + e, row = r ? row1 : row0, i = 4 * j + 2 * r + e;
                    const float dec = fast_exp2(fminf((r ? L1 : L0) - (e ? Lc[j].y : Lc[j].x), 0.f));
                    float g, second;
                    dp[e] = s <= row ? da[i] * dec : 0.f;
                    g = dp[e] * pv[i];                                // dA A = dA dec P
                    if constexpr (DELTA) {
                        const float dn = s < row ? -ev[i] * dec : 0.f;                // dN dec
                        const float bt = r ? be1 : be0;
                        second = dn * bt;                             // C = dN beta dec
                        (r ? b1 : b0) += dn * kk[i];
                        g = fmaf(second, kk[i], g);
                    } else second = s <= row ? pv[i] * dec : 0.f;     // A
                    av[e] = second;
                    (r ? g1 : g0) += g;
                    if (r == 0) gc[e] = g; else gc[e] += g;
                }
                split2(dp[0], dp[1], hp[r], lp[r]);
                split2(av[0], av[1], ha[r], la2[r]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {                             // column sums over this warp's 16 rows
                gc[e] += __shfl_xor_sync(0xffffffffu, gc[e], 4); gc[e] += __shfl_xor_sync(0xffffffffu, gc[e], 8); gc[e] += __shfl_xor_sync(0xffffffffu, gc[e], 16);
                if (fr == 0) cs[sub * 64 + col0 + 8 * j + 2 * fq + e] = gc[e];
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t o = swz(r ? row1 : row0, 4 * wg + j) + 4 * fq;
                *reinterpret_cast<uint32_t *>(sm + SM::o_ph + o) = hp[r]; *reinterpret_cast<uint32_t *>(sm + SM::o_pl + o) = lp[r];
                *reinterpret_cast<uint32_t *>(sm + SM::o_ah + o) = ha[r]; *reinterpret_cast<uint32_t *>(sm + SM::o_al + o) = la2[r];
            }
        }
        row_out(0, g0, g1);
        if (DELTA) row_out(3, b0, b1);
        if constexpr (TIGHT) {
            ok = mbar_wait_warp(bar_r, 0, 34);
            tc_fence_after();
            tmem_ld_frag4(lb + TM_R + HALF * wg, R[0]);
            tmem_ld_wait();
        }
        float a = 0.f, b = 0.f, x = 0.f, y = 0.f;
#pragma unroll
        for (int bl = 0; bl < NB; ++bl) {
            row_dot(SM::o_q, HALF * wg + 32 * bl, R[bl], a, b);
            if constexpr (!DELTA) row_dot(SM::o_k, HALF * wg + 32 * bl, VG[bl], x, y);
        }
        row_out(1, a, b);
        if (!DELTA) row_out(2, x, y);
    }
    fence_proxy_async();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (warp == 2 && ok) {
        constexpr uint32_t I_TD = idesc_bf16(64, D, 1, 1), I_ND = idesc_bf16(64, D, 0, 1);
        const uint64_t q_m = smem_desc(base + SM::o_q, 8192, 1024), k_m = smem_desc(base + SM::o_k, 8192, 1024), do_m = smem_desc(base + SM::o_do, 8192, 1024);
        const uint32_t ph = base + SM::o_ph, ah = base + SM::o_ah;
        // M^T tile (transposed: contraction over M's rows) and M tile (over its columns), M in head and tail
        auto trans = [&](uint32_t acc, uint32_t mt, uint64_t b, uint32_t onto) {
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem + acc, smem_desc(mt + half * SM::SQ, 8192, 1024) + k * 128, b + k * 128, I_TD, onto | half | (k > 0));
        };
        auto plain = [&](uint32_t acc, uint32_t mt, uint64_t b, uint32_t onto) {
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem + acc, smem_desc(mt + half * SM::SQ, 16, 1024) + k * 2, b + k * 128, I_ND, onto | half | (k > 0));
        };
        plain(TM_DQ, ph, k_m, 0);                                     // dQ = dP K
        trans(TM_DK, ph, q_m, 0);                                     // dK = dP^T Q
        if constexpr (DELTA) {
            plain(TM_DK, ah, k_m, 1);                                 //  + C K + C^T K
            trans(TM_DK, ah, k_m, 1);
            rows_rows(TM_KG, v_k, gh_k, D * 128, I_RD, 0);            // W G^T
            rows_rows(TM_KG, v_k, gl_k, D * 128, I_RD, 1);
        } else {
            trans(TM_DV, ah, do_m, 0);                                // dV = A^T dO
#pragma unroll
            for (int half = 0; half < 2; ++half)                      // K G: rows of G (keys) are the contraction
#pragma unroll
                for (int k = 0; k < D / 16; ++k)
                    mma_bf16_elect(tmem + TM_KG, k_k + tr_ko(k, 8192), smem_desc(base + (half ? SM::o_gl : SM::o_gh), D * 128, 1024) + k * 128, I_ND, half | (k > 0));
        }
        mma_commit_elect(bar_2);
    }
    if constexpr (DELTA) {
        // dV = beta dR and dR . V, while they run: a thread per (row, 16-byte piece), eight or sixteen threads a row
        constexpr int PC = D / 8;
        for (int idx = tid; idx < TC_C * PC; idx += TR_NT) {
            const int r = idx / PC, jj = idx % PC;
            const uint32_t off = (uint32_t)(jj >> 3) * 8192u + swz(r, jj & 7);
            const uint4 h = *reinterpret_cast<const uint4 *>(sm + SM::o_drh + off), l = *reinterpret_cast<const uint4 *>(sm + SM::o_drl + off);
            const __nv_bfloat162 *h2 = reinterpret_cast<const __nv_bfloat162 *>(&h), *l2 = reinterpret_cast<const __nv_bfloat162 *>(&l);
            const bool live = t0 + r < T;
            const size_t g = ((size_t)bh * T + t0 + r) * D + 8 * jj;
            uint4 vr = make_uint4(0u, 0u, 0u, 0u), outv;
            if (live) vr = *reinterpret_cast<const uint4 *>(p.v + g);
            const __nv_bfloat162 *v2 = reinterpret_cast<const __nv_bfloat162 *>(&vr);
            __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&outv);
            float dot = 0.f;
            const float be = bes[r];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 a = __bfloat1622float2(h2[i]), b = __bfloat1622float2(l2[i]), v = __bfloat1622float2(v2[i]);
                const float x = a.x + b.x, y = a.y + b.y;
                dot = fmaf(x, v.x, fmaf(y, v.y, dot));
                o2[i] = __floats2bfloat162_rn(be * x, be * y);
            }
            if (live) *reinterpret_cast<uint4 *>(p.dv + g) = outv;
#pragma unroll
            for (int o = 1; o < PC; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            if (jj == 0) cs[256 + r] = dot;
        }
    }
    if (ok) ok = mbar_wait_warp(bar_2, 0, 33);
    tc_fence_after();
    const float e0 = eLs[row0], e1 = eLs[row1], w0 = wts[row0], w1 = wts[row1];
    auto store = [&](__nv_bfloat16 *dst, int cb, const float *x) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = t0 + (r ? row1 : row0);
            if (t < T)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<__nv_bfloat162 *>(dst + ((size_t)bh * T + t) * D + cb + 8 * j + 2 * fq) = __floats2bfloat162_rn(x[4 * j + 2 * r], x[4 * j + 2 * r + 1]);
        }
    };
    if (ok) {
        float x = 0.f, y = 0.f, u = 0.f, w = 0.f;
#pragma unroll
        for (int bl = 0; bl < NB; ++bl) {
            const int cb = HALF * wg + 32 * bl;
            float a[16], b[16], z[DELTA ? 16 : 1];
            tmem_ld_frag4(lb + TM_DQ + cb, a);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = fmaf((j & 2) ? e1 : e0, R[bl][j], a[j]);
            store(p.dq, cb, a);
            tmem_ld_frag4(lb + TM_DK + cb, a);
            if constexpr (DELTA) {
                tmem_ld_frag4(lb + TM_KG + cb, b);
                tmem_ld_frag4(lb + TM_VG + cb, z);
                tmem_ld_wait();
                row_dot(SM::o_k, cb, b, x, y);                        // dw = k . (G W)
                row_dot(SM::o_k, cb, z, u, w);                        // k . R2
                const float f0 = -bes[row0] * e0, f1 = -bes[row1] * e1;
#pragma unroll
                for (int j = 0; j < 16; ++j) a[j] = fmaf((j & 2) ? f1 : f0, z[j], fmaf((j & 2) ? w1 : w0, b[j], a[j]));
                store(p.dk, cb, a);
            } else {
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) a[j] = fmaf((j & 2) ? w1 : w0, VG[bl][j], a[j]);
                store(p.dk, cb, a);
                tmem_ld_frag4(lb + TM_DV + cb, a);
                tmem_ld_frag4(lb + TM_KG + cb, b);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) a[j] = fmaf((j & 2) ? w1 : w0, b[j], a[j]);
                store(p.dv, cb, a);
            }
        }
        if (DELTA) { row_out(2, x, y); row_out(4, u, w); }
    }
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (warp == 0 && ok) {
        // dL of a lane's two tokens, dbeta, then dla as the reverse cumulative sum
        float dl[2], wd[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = lane + 32 * i;
            auto row = [&](int which) { return rr[which * 128 + t] + rr[which * 128 + 64 + t]; };
            const float gcol = (cs[t] + cs[64 + t]) + (cs[128 + t] + cs[192 + t]);
            wd[i] = wts[t] * row(2);
            dl[i] = row(0) - gcol + eLs[t] * row(1) - wd[i];
            if (DELTA) {
                const float kr = eLs[t] * row(4);
                dl[i] -= bes[t] * kr;
                if (t0 + t < T) p.dbeta[(size_t)bh * T + t0 + t] = row(3) + cs[256 + t] - kr;
            }
        }
        float tot = warp_sum(wd[0] + wd[1]);                          // sum of w dw
        float gsum = 0.f;
#pragma unroll
        for (int i = 0; i < TR_NT / 32; ++i) gsum += gs[i];
        tot = fmaf(eLs[TC_C - 1], gsum, tot);
        if (lane == 31) dl[1] += tot;
        float hi = dl[1], lo = dl[0];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float nh = __shfl_down_sync(0xffffffffu, hi, o), nl = __shfl_down_sync(0xffffffffu, lo, o);
            if (lane + o < 32) { hi += nh; lo += nl; }
        }
        lo += __shfl_sync(0xffffffffu, hi, 0);
        if (t0 + lane < T) p.dla[(size_t)bh * T + t0 + lane] = lo;
        if (t0 + lane + 32 < T) p.dla[(size_t)bh * T + t0 + lane + 32] = hi;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, SM::TM_COLS);
}

// ------------------------------------------------------------------------------------------------ host side
namespace {

struct TrainScratch {                                                 // one buffer, cut up; every piece a multiple of 256 bytes
    size_t dc, g, lt, dw0, dr, bytes;
    TrainScratch(long long BH, long long T, int D, bool delta) {
        const long long NC = (T + TC_C - 1) / TC_C;
        auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
        dc = 0;
        g = dc + up((size_t)BH * NC * D * D * 4);
        lt = g + up((size_t)BH * NC * D * D * 4);
        dw0 = lt + up((size_t)BH * NC * 4);
        dr = dw0 + (delta ? up((size_t)BH * T * D * 4) : 0);
        bytes = dr + (delta ? up((size_t)BH * T * D * 4) : 0);
    }
};

template <typename K> int tr_attr(K kern, int smem, const char *what) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) { set_cuda_error(e, what); return PGB_ERR_CUDA; }
    return PGB_OK;
}

template <int D, bool DELTA>
int train_bwd_go(const TrainBwdArgs &a, cudaStream_t st) {
    const long long BH = (long long)a.B * a.H, TD = (long long)a.T * D;
    const int NC = (a.T + TC_C - 1) / TC_C;
    const TrainScratch sc(BH, a.T, D, DELTA);
    uint8_t *buf = (uint8_t *)a.scratch;
    __nv_bfloat16 *G = (__nv_bfloat16 *)(buf + sc.g), *dR = (__nv_bfloat16 *)(buf + sc.dr);
    TrainMaps m{};
    bool made = tc_make_map(&m.q, a.q, BH, a.T, D, D, TD) && tc_make_map(&m.k, a.k, BH, a.T, D, D, TD) &&
                tc_make_map(&m.v, DELTA ? a.W : a.v, BH, a.T, D, D, TD) && tc_make_map(&m.dout, a.dout, BH, a.T, D, D, TD) &&
                tc_make_map(&m.s, a.sent, BH * NC, D, D, D, (long long)D * D, D) && tc_make_map(&m.g, G, BH * NC * 2, D, D, D, (long long)D * D, D);
    DwMaps w{};
    if (made && DELTA)
        made = tc_make_map(&m.dr, dR, 2 * BH, a.T, D, D, TD) && tc_make_map(&w.x, a.X, BH * NC * 2, TC_C, TC_C, TC_C, TC_C * TC_C) &&
               tc_make_store_map(&w.g, G, false, BH * NC * 2, D, D, 32, D / 2) && tc_make_store_map(&w.dr, dR, false, 2 * BH, a.T, D, 32, 32);
    if (!made) { set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled"); return PGB_ERR_CUDA; }
    TrainParams p{};
    p.la = a.la; p.beta = a.beta; p.v = (const __nv_bfloat16 *)a.v; p.dsent = a.dsent;
    p.Dc = (float *)(buf + sc.dc); p.dW0 = (float *)(buf + sc.dw0); p.Ltot = (float *)(buf + sc.lt);
    p.dq = (__nv_bfloat16 *)a.dq; p.dk = (__nv_bfloat16 *)a.dk; p.dv = (__nv_bfloat16 *)a.dv; p.dla = a.dla; p.dbeta = a.dbeta;
    p.BH = (int)BH; p.T = a.T;
    auto pre = train_pre_kernel<D, DELTA>;
    auto post = train_post_kernel<D, DELTA>;
    int rc = tr_attr(pre, PreSmem<D, DELTA>::bytes, "train_pre smem attribute");
    if (rc == PGB_OK) rc = tr_attr(post, PostSmem<D, DELTA>::bytes, "train_post smem attribute");
    if (rc != PGB_OK) return rc;
    const dim3 grid((unsigned)NC, (unsigned)BH);
    pre<<<grid, TR_NT, PreSmem<D, DELTA>::bytes, st>>>(m, p);
    if ((rc = check_launch("train_pre_kernel")) != PGB_OK) return rc;
    // the rest as programmatic dependents: set-up (barriers, tensor memory) under the tail of the kernel ahead
    cudaError_t e = cudaSuccess;
    if constexpr (DELTA) {
        auto walk = delta_walk_kernel<D, true>;
        if ((rc = tr_attr(walk, DwSmem<D, true>::bytes, "delta_walk backward smem attribute")) != PGB_OK) return rc;
        w.k = m.k;
        DwParams d{};
        d.la = a.la; d.beta = a.beta; d.S0 = a.dS; d.S_out = a.dS0; d.dW0 = p.dW0; d.Dc = p.Dc; d.H = a.H; d.T = a.T;
        e = pdl_launch(walk, dim3((unsigned)BH), dim3(DW_NT), (size_t)DwSmem<D, true>::bytes, st, w, d);
    } else {
        e = pdl_launch(state_grad_scan_kernel, dim3((unsigned)(D * D / 1024), (unsigned)BH), dim3(256), (size_t)0, st, (const float *)p.Dc, (const float *)p.Ltot,
                       a.dS, G, a.dS0, NC, D * D);
    }
    if (e == cudaSuccess) e = pdl_launch(post, grid, dim3(TR_NT), (size_t)PostSmem<D, DELTA>::bytes, st, m, p);
    if (e != cudaSuccess) { set_cuda_error(e, "train backward launch"); return PGB_ERR_CUDA; }
    return check_launch("train_post_kernel");
}

}  // namespace

size_t train_bwd_scratch_bytes(int B, int H, int T, int D, bool delta) { return TrainScratch((long long)B * H, T, D, delta).bytes; }

int train_bwd_launch(const TrainBwdArgs &a, int D, cudaStream_t st) {
    if (a.beta != nullptr) return D == 64 ? train_bwd_go<64, true>(a, st) : train_bwd_go<128, true>(a, st);
    return D == 64 ? train_bwd_go<64, false>(a, st) : train_bwd_go<128, false>(a, st);
}

int tc_train_error_flag(int *out) { return tc_read_error_flag(out); }

}  // namespace pgb
