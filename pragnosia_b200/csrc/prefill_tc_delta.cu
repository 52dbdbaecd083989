// Delta-rule chunked prefill on the tensor cores (tcgen05.mma, TMEM accumulators, TMA-fed tiles): two kernels.
//
// The delta rule writes v minus what the memory already returns for the key: S_t = a_t S_{t-1} + k_t [b_t (v_t - a_t S_{t-1}^T k_t)]^T.
// In a 64-token chunk the residuals actually written, W, solve (I + N) W = rhs with
//     N = diag(beta) strictly_lower((K K^T) * dec),   rhs = diag(beta) (V - e^{L} K S_entering),
// (reference src/assoc.py:207-251). N does not depend on the state, so
//
//   delta_inv_kernel   (chunk-parallel, one CTA per (sequence-head, chunk)): K K^T on the tensor core, N in fp32, then
//                      X = (I + N)^-1 by blocked forward substitution to fp32's precision, every intermediate bounded (the
//                      reduced-precision Neumann doubling the reference warns about at src/assoc_kernel.py:577-582 is
//                      never formed). X goes to a scratch buffer as bf16 head + tail.
//   delta_walk_kernel  (delta_walk.cuh; one CTA per (sequence, head), walking the chunks): W = X rhs, the state update and o.
//
// Everything fp32 that re-enters the tensor core (S, rhs, X, A, W) is split into bf16 head + tail and multiplied as
// head*head + head*tail + tail*head. Every mbarrier wait is bounded.
//
// Measured, B8 H16 T8192 D128 (1.1 GB of operands): walk 396 us, inverse 166.
#include "delta_walk.cuh"

namespace pgb {

constexpr float TD_LOG2E = 1.4426950408889634f;

// decay statistics of one 64-token chunk by warps 0 and 1 (tid < 64): L (inclusive cumulative log-decay) and beta (0 past T)
__device__ __forceinline__ void chunk_stats(const float *la, const float *beta, int t0, int T, int tid, int lane, int warp, float *Ls, float *bes) {
    const int t = t0 + tid, tx = t0 + (tid ^ 32);
    const float own = t < T ? la[t] : 0.f, other = tx < T ? la[tx] : 0.f;
    float sc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, sc, o);
        if (lane >= o) sc += n;
    }
    const float sum_other = warp_sum(other);
    Ls[tid] = sc + (warp == 1 ? sum_other : 0.f);
    bes[tid] = t < T ? beta[t] : 0.f;
}

// ------------------------------------------------------------------------------------------------ X = (I + N)^-1
// One column of X per thread is a chain of 2016 dependent multiply-adds on half the threads. The blocked form keeps the chain to 16 steps: the four
// 16 x 16 diagonal blocks are inverted side by side (half a warp each, a lane per column), then twice X21 = -X22 (N21 X11) joins neighbouring blocks, 16
// and 32 wide, as warp-level products (m16n8k8, too small for the tensor-memory kind) of factors split into three tf32 parts, which are all of fp32.
// One array holds all of it, in the K tile's place once that is consumed: N below the diagonal; X transposed above it, a diagonal block of X over N's own
// once its columns are done; T = N21 X11, transposed, in the quarter that X21 would take (X21 itself goes from registers to memory). 20 KB a CTA where
// N, X and T side by side were 43: eight CTAs an SM (the tensor memory's limit, too) instead of five.
// B8 H16 T8192 D128: 194 us with the joins as fp32 register tiles, whose 16-byte shared loads filled the load unit, 166 so; B64 H12 T512 D64 77 and 67. Two
// parts a factor took 137 and 55, but X21's error against 64 bits rose by 10 to 15 % where keys resemble one another (2.9e-6 -> 3.2e-6 of it, 3.7e-6 -> 4.3e-6
// for keys that all but repeat); with three it is the register tiles', 0.3 % below to 0.7 % above, X's as a whole 0.02 % below to 0.07 % above. What bounds it: issue slots.
struct InvSmem {
    static constexpr int P = 68;                                      // row pitch, in floats (16-byte aligned, four banks on)
    static constexpr int off_misc = TC_C * P * 4;                     // not below a K tile of 64 x 128 bf16
    static constexpr int bytes = off_misc + 1024 + 1024;
};
static_assert(InvSmem::off_misc >= TC_C * 128 * 2, "the K tile lies in the array's place");

// P = A B for 16 rows and NT tiles of eight columns over the K blocks k0 <= k < k1 of eight, by a warp. A element (m, k) lies at A[m ra + k ka], an
// element (k, n) of B at B[n P + k]. Lane l of the accumulator has rows l / 4 and l / 4 + 8, columns 2 (l % 4) and the next of each tile. Of the products of
// the factors' three parts all are added but those below 2^-33 of the whole. The heads' products of a block are added by an addition that rounds:
// accumulated in the tensor core, which cuts off, X was off by 0.1 % more where nothing decays (162 us).
template <int NT>
__device__ __forceinline__ void inv_product(float (&acc)[NT][4], const float *A, int ra, int ka, const float *B, int k0, int k1, int lane) {
    const float *ap = A + (lane >> 2) * ra + (lane & 3) * ka, *bp = B + (lane >> 2) * InvSmem::P + (lane & 3);
    float low[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = low[n][i] = 0.f;
#pragma unroll 2
    for (int k = k0; k < k1; ++k) {
        uint32_t ah[4], am[4], al[4];
        tf32_split(ap[8 * k * ka], ah[0], am[0], al[0]);
        tf32_split(ap[8 * ra + 8 * k * ka], ah[1], am[1], al[1]);
        tf32_split(ap[(8 * k + 4) * ka], ah[2], am[2], al[2]);
        tf32_split(ap[8 * ra + (8 * k + 4) * ka], ah[3], am[3], al[3]);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            uint32_t bh[2], bm[2], bl[2];
            tf32_split(bp[8 * n * InvSmem::P + 8 * k], bh[0], bm[0], bl[0]);
            tf32_split(bp[8 * n * InvSmem::P + 8 * k + 4], bh[1], bm[1], bl[1]);
            mma_tf32(low[n], al, bh);
            mma_tf32(low[n], ah, bl);
            mma_tf32(low[n], am, bm);
            mma_tf32(low[n], am, bh);
            mma_tf32(low[n], ah, bm);
            float hh[4] = {0.f, 0.f, 0.f, 0.f};
            mma_tf32(hh, ah, bh);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] += hh[i];
        }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] += low[n][i];
}
// such an accumulator (or its negative) transposed: element (m, n) to at[n P + m]
template <int NT, bool NEG>
__device__ __forceinline__ void inv_put(float *at, const float (&acc)[NT][4], int lane) {
    float *p = at + 2 * (lane & 3) * InvSmem::P + (lane >> 2);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) p[(8 * n + (i & 1)) * InvSmem::P + 8 * (i >> 1)] = NEG ? -acc[n][i] : acc[n][i];
}

template <int D>
__global__ void __launch_bounds__(128, 8) delta_inv_kernel(const __grid_constant__ CUtensorMap mk, const float *__restrict__ la_all,
                                                        const float *__restrict__ beta_all, __nv_bfloat16 *__restrict__ X, int T,
                                                        int with_tail) {
    using SM = InvSmem;
    constexpr int P = SM::P;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    float *M = reinterpret_cast<float *>(sm);                         // the array: N[t][s] at M[t P + s], s < t; X[t][s] at M[s P + t]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + SM::off_misc + 32);
    float *Ls = reinterpret_cast<float *>(sm + SM::off_misc + 64), *bes = Ls + 64;
    const uint32_t bar_k = base + SM::off_misc, bar_m = bar_k + 8;

    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    const int c = blockIdx.x, bh = blockIdx.y, NC = gridDim.x, t0 = c * TC_C;

    if (tid == 0) {
        mbar_init(bar_k, 1); mbar_init(bar_m, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(bar_k, TC_C * D * 2);
#pragma unroll
        for (int s = 0; s < D / 64; ++s) tma_load_3d(base + s * 8192, &mk, bar_k, 64 * s, t0, bh);
    }
    if (warp == 3) tmem_alloc(smem_u32(tmem_slot), 64);
    if (warp < 2) chunk_stats(la_all + (size_t)bh * T, beta_all + (size_t)bh * T, t0, T, tid, lane, warp, Ls, bes);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    bool ok = mbar_wait_warp(bar_k, 0, 11);
    if (warp == 2 && ok) {
        constexpr uint32_t I_KK = idesc_bf16(64, 64, 0, 0);
        const uint64_t dk = smem_desc(base, 16, 1024);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            const uint32_t ko = ((uint32_t)(k >> 2) * 8192u + (uint32_t)(k & 3) * 32u) >> 4;
            mma_bf16_elect(tmem, dk + ko, dk + ko, I_KK, k > 0);
        }
        mma_commit_elect(bar_m);
    }
    if (ok) ok = mbar_wait_warp(bar_m, 0, 12);
    tc_fence_after();
    // ---- over K, which the finished product has consumed: N = beta_t (k_t . k_s) exp(min(L_t - L_s, 0)) for s < t.   Each warp: its 16 rows, the columns up to its
    //      diagonal block's end (beyond lies X's place).
    {
        const int fr = lane >> 2, fq = lane & 3, r0 = 16 * warp + fr, r1 = r0 + 8;
        float kk[32];
        tmem_ld_frag8(tmem + ((uint32_t)(32 * warp) << 16), kk);
        const float L0 = Ls[r0] * TD_LOG2E, L1 = Ls[r1] * TD_LOG2E, b0 = bes[r0], b1 = bes[r1];
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j > 2 * warp + 1) break;
            const int s = 8 * j + 2 * fq;
            const float2 Lp = *reinterpret_cast<const float2 *>(Ls + s);
            const float La = Lp.x * TD_LOG2E, Lb = Lp.y * TD_LOG2E;
            float2 n0, n1;
            n0.x = (s < r0) ? b0 * kk[4 * j] * fast_exp2(fminf(L0 - La, 0.f)) : 0.f;
            n0.y = (s + 1 < r0) ? b0 * kk[4 * j + 1] * fast_exp2(fminf(L0 - Lb, 0.f)) : 0.f;
            n1.x = (s < r1) ? b1 * kk[4 * j + 2] * fast_exp2(fminf(L1 - La, 0.f)) : 0.f;
            n1.y = (s + 1 < r1) ? b1 * kk[4 * j + 3] * fast_exp2(fminf(L1 - Lb, 0.f)) : 0.f;
            *reinterpret_cast<float2 *>(M + r0 * P + s) = n0;
            *reinterpret_cast<float2 *>(M + r1 * P + s) = n1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 3) tmem_dealloc(tmem, 64);
    // ---- diagonal blocks: lane j of a half warp owns column j of a block;  x_t = [t == j] - sum_{s<t} N[t][s] x_s
    if (warp < 2) {
        const int j = lane & 15, blk = 2 * warp + (lane >> 4);
        float *Mb = M + 16 * blk * (P + 1);
        float x[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            float a0 = t == j ? 1.f : 0.f, a1 = 0.f;
#pragma unroll
            for (int s4 = 0; s4 < (t + 3) / 4; ++s4) {
                const float4 n = *reinterpret_cast<const float4 *>(Mb + t * P + 4 * s4);   // the same address for every lane of a half: a broadcast
                if (4 * s4 + 0 < t) a0 = fmaf(-n.x, x[4 * s4 + 0], a0);
                if (4 * s4 + 1 < t) a1 = fmaf(-n.y, x[4 * s4 + 1], a1);
                if (4 * s4 + 2 < t) a0 = fmaf(-n.z, x[4 * s4 + 2], a0);
                if (4 * s4 + 3 < t) a1 = fmaf(-n.w, x[4 * s4 + 3], a1);
            }
            x[t] = a0 + a1;
        }
        __syncwarp();                                                 // nobody needs N's block any more: X's takes its place, zeros and all
#pragma unroll
        for (int t = 0; t < 16; t += 4) *reinterpret_cast<float4 *>(Mb + j * P + t) = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
    }
    __syncthreads();
    // ---- join 16 x 16 blocks, two warps a pair of blocks, eight columns each
    {
        const int pair = warp >> 1, g = 32 * pair, c0 = 8 * (warp & 1);            // the pair's first row
        float *Tt = M + 16 * pair * P + 32 + c0 * P, acc[1][4];
        inv_product<1>(acc, M + (g + 16) * P + g, P, 1, M + (g + c0) * P + g, 0, 2, lane);
        inv_put<1, false>(Tt, acc, lane);
        __syncwarp();                                                 // a warp reads its own columns only
        inv_product<1>(acc, M + (g + 16) * P + g + 16, 1, P, Tt, 0, 2, lane);
        inv_put<1, true>(M + (g + c0) * P + g + 16, acc, lane);
    }
    __syncthreads();
    // ---- join the 32 x 32 blocks: T = N21 X11, X21 = -X22 T. A warp has 16 rows by 16 columns of each; blocks of zeros are left out (X11 and X22 are
    //      lower triangular; N lies in their place).
    const int m16 = 16 * (warp & 1), n16 = 16 * (warp >> 1);
    float acc[2][4];
    inv_product<2>(acc, M + (32 + m16) * P, P, 1, M + n16 * P, n16 / 8, 4, lane);
    inv_put<2, false>(M + n16 * P + 32 + m16, acc, lane);
    __syncthreads();
    inv_product<2>(acc, M + 32 * P + 32 + m16, 1, P, M + n16 * P + 32, 0, m16 / 8 + 2, lane);
    // ---- head then tail, 8 KB each, to the scratch buffer; or the head alone, densely packed (the stand-alone operator). The last block from the
    //      registers, neighbouring lanes trading column pairs so that a row's quad stores a whole 32-byte sector.
    uint4 *dst = reinterpret_cast<uint4 *>(X + ((size_t)bh * NC + c) * ((with_tail ? 2 : 1) * TC_C * TC_C));
    {
        const int fr = lane >> 2, fq = lane & 3;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            uint32_t h[2], l[2];
#pragma unroll
            for (int n = 0; n < 2; ++n) split2(-acc[n][2 * r], -acc[n][2 * r + 1], h[n], l[n]);
            const uint32_t gh = __shfl_xor_sync(0xffffffffu, (fq & 1) ? h[0] : h[1], 1), gl = __shfl_xor_sync(0xffffffffu, (fq & 1) ? l[0] : l[1], 1);
            const int at = (32 + m16 + fr + 8 * r) * 16 + (n16 + 8 * (fq & 1)) / 4 + (fq >> 1);       // in pieces of four columns
            uint2 *d2 = reinterpret_cast<uint2 *>(dst);
            d2[at] = (fq & 1) ? make_uint2(gh, h[1]) : make_uint2(h[0], gh);
            if (with_tail) d2[1024 + at] = (fq & 1) ? make_uint2(gl, l[1]) : make_uint2(l[0], gl);
        }
    }
    // the two blocks on the diagonal, eight columns a thread and time, of which the upper block's upper quarter is zero (N lies there)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = (tid >> 2) + 32 * i, piece = (tid & 3) + 4 * i, rr = row & 31;
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = M[(8 * piece + e) * P + row];
        if (rr < 16 && (tid & 2))
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = 0.f;
        uint4 hi, lo;
        split8(x, hi, lo);
        dst[row * 8 + piece] = hi;
        if (with_tail) dst[512 + row * 8 + piece] = lo;
        if (i == 0) {                                                 // the block above the diagonal: zero
            dst[row * 8 + piece + 4] = make_uint4(0u, 0u, 0u, 0u);
            if (with_tail) dst[512 + row * 8 + piece + 4] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

// ------------------------------------------------------------------------------------------------ host side
template <int D>
static int delta_inverse_go(const PrefillArgs &a, void *x_scratch, cudaStream_t stream) {
    const int BH = a.B * a.H, NC = (a.T + TC_C - 1) / TC_C;
    CUtensorMap mk;
    if (!tc_make_map(&mk, a.k, BH, a.T, D, D, (long long)a.T * D)) { set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled"); return PGB_ERR_CUDA; }
    auto inv = delta_inv_kernel<D>;
    const cudaError_t e = cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, InvSmem::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_inv smem attribute"); return PGB_ERR_CUDA; }
    inv<<<dim3(NC, BH), 128, InvSmem::bytes, stream>>>(mk, a.la, a.beta, (__nv_bfloat16 *)x_scratch, a.T, 1);
    return check_launch("delta_inv_kernel");
}
// the inverses of the chunks of `a` into x_scratch
int delta_inverse_launch(const PrefillArgs &a, int D, void *x_scratch, cudaStream_t stream) {
    return D == 64 ? delta_inverse_go<64>(a, x_scratch, stream) : delta_inverse_go<128>(a, x_scratch, stream);
}

template <int D>
static int delta_go(const PrefillArgs &a, int o_dtype, void *x_scratch, cudaStream_t stream) {
    const int BH = a.B * a.H, NC = (a.T + TC_C - 1) / TC_C;
    const bool f32 = o_dtype == PGB_F32;
    DwMaps m{};
    if (!tc_make_map(&m.q, a.q, BH, a.T, D, D, (long long)a.T * D) || !tc_make_map(&m.k, a.k, BH, a.T, D, D, (long long)a.T * D) ||
        !tc_make_map(&m.v, a.v, BH, a.T, D, D, (long long)a.T * D) ||
        !tc_make_map(&m.x, x_scratch, (long long)BH * NC * 2, TC_C, TC_C, TC_C, TC_C * TC_C) ||
        !tc_make_store_map(&m.o, a.o, f32, BH, a.T, D, 32, 32) ||
        (a.W_out != nullptr && !tc_make_store_map(&m.w, a.W_out, false, BH, a.T, D, 32, 32)) ||
        (a.sent != nullptr && !tc_make_store_map(&m.sent, a.sent, false, (long long)BH * NC, D, D, 32, D / 2))) {
        set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled");
        return PGB_ERR_CUDA;
    }
    auto walk = delta_walk_kernel<D, false>;
    cudaError_t e = cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, DwSmem<D, false>::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_walk smem attribute"); return PGB_ERR_CUDA; }
    const int rc = delta_inverse_go<D>(a, x_scratch, stream);
    if (rc != PGB_OK) return rc;
    DwParams p{};
    p.la = a.la; p.beta = a.beta; p.S0 = a.S0; p.theta = a.theta; p.shift_dev = a.shift_dev; p.shift_host = a.shift_host;
    p.S_out = a.S_out; p.want_sent = a.sent != nullptr; p.want_w = a.W_out != nullptr; p.H = a.H; p.T = a.T; p.o_is_f32 = f32;
    p.rebase_chunks = a.rebase_chunks; p.rebase_shift = (float)(a.rebase_chunks * TC_C);
    walk<<<(unsigned)BH, DW_NT, DwSmem<D, false>::bytes, stream>>>(m, p);
    return check_launch("delta_walk_kernel");
}

// bytes of scratch the delta path needs for X (head and tail, 64 x 64 bf16 each, per (sequence-head, chunk))
size_t prefill_tc_delta_scratch_bytes(int B, int H, int T) {
    return (size_t)B * H * ((T + TC_C - 1) / TC_C) * 2 * TC_C * TC_C * sizeof(__nv_bfloat16);
}

int prefill_tc_delta_launch(const PrefillArgs &a, int o_dtype, int D, void *x_scratch, cudaStream_t stream) {
    return D == 64 ? delta_go<64>(a, o_dtype, x_scratch, stream) : delta_go<128>(a, o_dtype, x_scratch, stream);
}

int tc_delta_error_flag(int *out) { return tc_read_error_flag(out); }

// The inverse alone, as the reference's stand-alone operator returns it (src/assoc_kernel.py:658-667 membrae::delta_inv):
// X [B*H][NC][64][64] bf16, the rounded heads only.
template <int D>
static int delta_inv_go(const void *k, const float *la, const float *beta, void *X, int BH, int T, cudaStream_t stream) {
    const int NC = (T + TC_C - 1) / TC_C;
    CUtensorMap mk;
    if (!tc_make_map(&mk, k, BH, T, D, D, (long long)T * D)) { set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled"); return PGB_ERR_CUDA; }
    auto inv = delta_inv_kernel<D>;
    cudaError_t e = cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, InvSmem::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_inv smem attribute"); return PGB_ERR_CUDA; }
    inv<<<dim3(NC, BH), 128, InvSmem::bytes, stream>>>(mk, la, beta, (__nv_bfloat16 *)X, T, 0);
    return check_launch("delta_inv_kernel");
}
int delta_inv_launch(const void *k, const float *la, const float *beta, void *X, int BH, int T, int D, cudaStream_t stream) {
    return D == 64 ? delta_inv_go<64>(k, la, beta, X, BH, T, stream) : delta_inv_go<128>(k, la, beta, X, BH, T, stream);
}

// ------------------------------------------------------------------------------------------------ built-in scratch
// The same delta prefill for callers that have no way to hand over a scratch buffer. The chunk inverses then live in
// this file-scope device array: PGB_STATIC_SCRATCH_BYTES of device memory that every GPU which loads the library keeps
// reserved until the process exits. In host code the array's name is only a stand-in for the device object, so its
// device address is asked for once per device (cudaGetSymbolAddress, with that device current) and cached.
constexpr size_t PGB_STATIC_SCRATCH_BYTES = 32u << 20;                 // 2048 (sequence-head, chunk) pairs of 16 KiB
static __device__ __align__(256) unsigned char g_static_scratch[PGB_STATIC_SCRATCH_BYTES];

static void *static_scratch_ptr() {
    constexpr int MAX_DEV = 64;
    static void *cache[MAX_DEV] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) return nullptr;
    void *ptr = __atomic_load_n(&cache[dev], __ATOMIC_ACQUIRE);
    if (ptr == nullptr) {
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || ptr == nullptr) { set_cuda_error(e, "cudaGetSymbolAddress(static scratch)"); return nullptr; }
        __atomic_store_n(&cache[dev], ptr, __ATOMIC_RELEASE);         // the same value whoever gets here first
    }
    return ptr;
}

long long prefill_tc_delta_static_capacity() { return (long long)PGB_STATIC_SCRATCH_BYTES; }

int prefill_tc_delta_static_launch(const PrefillArgs &a, int o_dtype, int D, cudaStream_t stream) {
    if (prefill_tc_delta_scratch_bytes(a.B, a.H, a.T) > PGB_STATIC_SCRATCH_BYTES) return PGB_ERR_TOO_LARGE;
    void *scratch = static_scratch_ptr();
    if (scratch == nullptr) return PGB_ERR_CUDA;
    return prefill_tc_delta_launch(a, o_dtype, D, scratch, stream);
}

}  // namespace pgb
