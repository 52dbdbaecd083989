// Delta-rule chunked prefill on the tensor cores (tcgen05.mma, TMEM accumulators, TMA-fed tiles): two kernels.
//
// The delta rule writes v minus what the memory already returns for the key: S_t = a_t S_{t-1} + k_t [b_t (v_t - a_t S_{t-1}^T k_t)]^T.
// In a 64-token chunk the residuals actually written, W, solve (I + N) W = rhs with
//     N = diag(beta) strictly_lower((K K^T) * dec),   rhs = diag(beta) (V - e^{L} K S_entering),
// (reference src/assoc.py:207-251). N does not depend on the state, so
//
//   delta_inv_kernel   (chunk-parallel, one CTA per (sequence-head, chunk)): K K^T on the tensor core, N in fp32, then
//                      X = (I + N)^-1 by blocked forward substitution in true fp32 FFMA, every intermediate bounded (the
//                      reduced-precision Neumann doubling the reference warns about at src/assoc_kernel.py:577-582 is
//                      never formed). X goes to a scratch buffer as bf16 head + tail.
//   delta_walk_kernel  (delta_walk.cuh; one CTA per (sequence, head), walking the chunks): W = X rhs, the state update and o.
//
// Everything fp32 that re-enters the tensor core (S, rhs, X, A, W) is split into bf16 head + tail and multiplied as
// head*head + head*tail + tail*head. Every mbarrier wait is bounded.
//
// Measured, B8 H16 T8192 D128 (1.1 GB of operands): walk 396 us, inverse 170.
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
// One column of X per thread is a chain of 2016 dependent multiply-adds on half the threads. The blocked form keeps the chain to 16 steps: the four 16 x 16
// diagonal blocks are inverted side by side (half a warp each, a lane per column), then twice X21 = -X22 (N21 X11) joins neighbouring blocks, 16 and 32 wide, as fp32
// products in register tiles of two by four and four by four, read 16 bytes at a time. Bound by the passes of the shared-memory loads; five CTAs share an SM.
// B8 H16 T8192 D128: 193 us with tiles of two by four throughout, 170 so; B64 H12 T512 D64 76 and 68.
// Products on the tensor cores instead (m16n8k8, one array of 20 KB a CTA): factors in two tf32 parts 135 us, but X21's error against 64 bits rises by 10 to 15 % where keys resemble
// one another (2.9e-6 -> 3.2e-6 of it, 3.7e-6 -> 4.3e-6 for keys that all but repeat) and X's as a whole by 1 %; in three parts, which are all of fp32, 158 to 166.
template <int D>
struct InvSmem {
    static constexpr int NP = 68, TP = 36;                            // row pitches of N / X and of the product T, in floats (16-byte aligned)
    static constexpr int XB = TC_C * NP * 4;
    static constexpr int off_k = 0;                                   // K tile, TC_C x D bf16; then X fp32 [64][NP] in its place
    static constexpr int off_n = XB > TC_C * D * 2 ? (XB + 1023) / 1024 * 1024 : TC_C * D * 2;
    static constexpr int off_t = off_n + XB;                          // T fp32 [32][TP]
    static constexpr int off_misc = off_t + 32 * TP * 4;
    static constexpr int bytes = off_misc + 1024 + 1024;
};

// rows r0, r0 + 1 and columns c0..c0+3 of P = A B for K-long rows of A (pitch pa) and rows of B (pitch pb); K a multiple of 4
template <int K>
__device__ __forceinline__ void inv_product(float (&acc)[2][4], const float *A, int pa, const float *B, int pb, int r0, int c0) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
#pragma unroll
    for (int k = 0; k < K; k += 4) {
        const float4 a0 = *reinterpret_cast<const float4 *>(A + r0 * pa + k), a1 = *reinterpret_cast<const float4 *>(A + (r0 + 1) * pa + k);
        const float f0[4] = {a0.x, a0.y, a0.z, a0.w}, f1[4] = {a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 b = *reinterpret_cast<const float4 *>(B + (k + i) * pb + c0);
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) { acc[0][c] = fmaf(f0[i], bv[c], acc[0][c]); acc[1][c] = fmaf(f1[i], bv[c], acc[1][c]); }
        }
    }
}

// rows r0 + RS i and columns c0..c0+3 of P = A B, i < 4, over k0 <= k < K: eight loads of 16 bytes for 64 products, and rows RS apart so
// that the rows a warp reads at once lie in different banks
template <int K, int RS>
__device__ __forceinline__ void inv_product4(float (&acc)[4][4], const float *A, int pa, const float *B, int pb, int r0, int c0, int k0) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
#pragma unroll 2
    for (int k = k0; k < K; k += 4) {
        float f[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 a = *reinterpret_cast<const float4 *>(A + (r0 + RS * r) * pa + k);
            f[r][0] = a.x; f[r][1] = a.y; f[r][2] = a.z; f[r][3] = a.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 b = *reinterpret_cast<const float4 *>(B + (k + i) * pb + c0);
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(f[r][i], bv[c], acc[r][c]);
        }
    }
}

template <int D>
__global__ void __launch_bounds__(128) delta_inv_kernel(const __grid_constant__ CUtensorMap mk, const float *__restrict__ la_all,
                                                        const float *__restrict__ beta_all, __nv_bfloat16 *__restrict__ X, int T,
                                                        int with_tail) {
    using SM = InvSmem<D>;
    constexpr int NP = SM::NP, TP = SM::TP;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    float *Nf = reinterpret_cast<float *>(sm + SM::off_n), *Xf = reinterpret_cast<float *>(sm + SM::off_k), *Tf = reinterpret_cast<float *>(sm + SM::off_t);
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
        for (int s = 0; s < D / 64; ++s) tma_load_3d(base + SM::off_k + s * 8192, &mk, bar_k, 64 * s, t0, bh);
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
        const uint64_t dk = smem_desc(base + SM::off_k, 16, 1024);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            const uint32_t ko = ((uint32_t)(k >> 2) * 8192u + (uint32_t)(k & 3) * 32u) >> 4;
            mma_bf16_elect(tmem, dk + ko, dk + ko, I_KK, k > 0);
        }
        mma_commit_elect(bar_m);
    }
    if (ok) ok = mbar_wait_warp(bar_m, 0, 12);
    tc_fence_after();
    // ---- N = beta_t (k_t . k_s) exp(min(L_t - L_s, 0)) for s < t, else 0.   Each warp: its 16 rows, all 64 columns.
    {
        const int fr = lane >> 2, fq = lane & 3, r0 = 16 * warp + fr, r1 = r0 + 8;
        float kk[32];
        tmem_ld_frag8(tmem + ((uint32_t)(32 * warp) << 16), kk);
        const float L0 = Ls[r0] * TD_LOG2E, L1 = Ls[r1] * TD_LOG2E, b0 = bes[r0], b1 = bes[r1];
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int s = 8 * j + 2 * fq;
            const float2 Lp = *reinterpret_cast<const float2 *>(Ls + s);
            const float La = Lp.x * TD_LOG2E, Lb = Lp.y * TD_LOG2E;
            float2 n0, n1;
            n0.x = (s < r0) ? b0 * kk[4 * j] * fast_exp2(fminf(L0 - La, 0.f)) : 0.f;
            n0.y = (s + 1 < r0) ? b0 * kk[4 * j + 1] * fast_exp2(fminf(L0 - Lb, 0.f)) : 0.f;
            n1.x = (s < r1) ? b1 * kk[4 * j + 2] * fast_exp2(fminf(L1 - La, 0.f)) : 0.f;
            n1.y = (s + 1 < r1) ? b1 * kk[4 * j + 3] * fast_exp2(fminf(L1 - Lb, 0.f)) : 0.f;
            *reinterpret_cast<float2 *>(Nf + r0 * NP + s) = n0;
            *reinterpret_cast<float2 *>(Nf + r1 * NP + s) = n1;
        }
    }
    tc_fence_before();
    __syncthreads();                                                  // K is consumed (the product is complete): X takes its place
    if (warp == 3) tmem_dealloc(tmem, 64);
    // ---- diagonal blocks: lane j of a half warp owns column j of a block;  x_t = [t == j] - sum_{s<t} N[t][s] x_s
    if (warp < 2) {
        const int j = lane & 15, blk = 2 * warp + (lane >> 4);
        const float *Nb = Nf + 16 * blk * (NP + 1);
        float *Xb = Xf + 16 * blk * (NP + 1);
        float x[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            float a0 = t == j ? 1.f : 0.f, a1 = 0.f;
#pragma unroll
            for (int s4 = 0; s4 < (t + 3) / 4; ++s4) {
                const float4 n = *reinterpret_cast<const float4 *>(Nb + t * NP + 4 * s4);   // the same address for every lane of a half: a broadcast
                if (4 * s4 + 0 < t) a0 = fmaf(-n.x, x[4 * s4 + 0], a0);
                if (4 * s4 + 1 < t) a1 = fmaf(-n.y, x[4 * s4 + 1], a1);
                if (4 * s4 + 2 < t) a0 = fmaf(-n.z, x[4 * s4 + 2], a0);
                if (4 * s4 + 3 < t) a1 = fmaf(-n.w, x[4 * s4 + 3], a1);
            }
            x[t] = a0 + a1;
            Xb[t * NP + j] = x[t];
        }
    } else {                                                          // the two blocks above the diagonal that the joins below read: zero
        const int g = 32 * (warp & 1), r = 2 * (lane >> 2), cc = 4 * (lane & 3);
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<float4 *>(Xf + (g + r + i) * NP + g + 16 + cc) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // ---- join 16 x 16 blocks, a warp per pair of blocks, whose lanes cover the new block as two rows by four columns each
    if (warp < 2) {
        float acc[2][4];
        const int g = 32 * warp, r = 2 * (lane >> 2), cc = 4 * (lane & 3);         // the pair's first row
        float *Tb = Tf + warp * 16 * TP;
        inv_product<16>(acc, Nf + (g + 16) * NP + g, NP, Xf + g * NP + g, NP, r, cc);
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<float4 *>(Tb + (r + i) * TP + cc) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        __syncwarp();
        inv_product<16>(acc, Xf + (g + 16) * NP + g + 16, NP, Tb, TP, r, cc);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            *reinterpret_cast<float4 *>(Xf + (g + 16 + r + i) * NP + g + cc) = make_float4(-acc[i][0], -acc[i][1], -acc[i][2], -acc[i][3]);
    }
    __syncthreads();
    // ---- join the 32 x 32 blocks by two warps, which store the new block from their registers; the other two store the rest meanwhile.
    //      Head then tail, 8 KB each, to the scratch buffer; or the head alone, densely packed (the stand-alone operator).
    uint4 *dst = reinterpret_cast<uint4 *>(X + ((size_t)bh * NC + c) * ((with_tail ? 2 : 1) * TC_C * TC_C));
    if (warp < 2) {
        float acc[4][4];
        {   // T = N21 X11, 16 columns a warp: X11 is lower triangular, so the right half's products begin at its row 16
            const int r = lane >> 2, cc = 16 * warp + 4 * (lane & 3);
            inv_product4<32, 8>(acc, Nf + 32 * NP, NP, Xf, NP, r, cc, 16 * warp);
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4 *>(Tf + (r + 8 * i) * TP + cc) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        named_sync(1, 64);
        // X21 = -X22 T, 16 rows a warp: the upper half's products end at column 16
        const int r = 16 * warp + (lane >> 3), cc = 4 * (lane & 7);
        if (warp == 0) inv_product4<16, 4>(acc, Xf + 32 * NP + 32, NP, Tf, TP, r, cc, 0);
        else inv_product4<32, 4>(acc, Xf + 32 * NP + 32, NP, Tf, TP, r, cc, 0);
        uint2 *d2 = reinterpret_cast<uint2 *>(dst);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t h0, l0, h1, l1;
            split2(-acc[i][0], -acc[i][1], h0, l0);
            split2(-acc[i][2], -acc[i][3], h1, l1);
            d2[(32 + r + 4 * i) * 16 + (lane & 7)] = make_uint2(h0, h1);
            if (with_tail) d2[1024 + (32 + r + 4 * i) * 16 + (lane & 7)] = make_uint2(l0, l1);
        }
    } else {
        auto store = [&](int row, int piece) {                        // eight columns
            const float4 a = *reinterpret_cast<const float4 *>(Xf + row * NP + 8 * piece), b = *reinterpret_cast<const float4 *>(Xf + row * NP + 8 * piece + 4);
            const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            uint4 hi, lo;
            split8(x, hi, lo);
            dst[row * 8 + piece] = hi;
            if (with_tail) dst[512 + row * 8 + piece] = lo;
            if (row < 32) {                                           // the block above the diagonal: zero
                dst[row * 8 + piece + 4] = make_uint4(0u, 0u, 0u, 0u);
                if (with_tail) dst[512 + row * 8 + piece + 4] = make_uint4(0u, 0u, 0u, 0u);
            }
        };
        const int t = tid - 64;
#pragma unroll
        for (int i = 0; i < 2; ++i) store((t >> 2) + 16 * i, t & 3);
#pragma unroll
        for (int i = 0; i < 2; ++i) store(32 + (t >> 2) + 16 * i, 4 + (t & 3));
    }
}

// ------------------------------------------------------------------------------------------------ host side
template <int D>
static int delta_inverse_go(const PrefillArgs &a, void *x_scratch, cudaStream_t stream) {
    const int BH = a.B * a.H, NC = (a.T + TC_C - 1) / TC_C;
    CUtensorMap mk;
    if (!tc_make_map(&mk, a.k, BH, a.T, D, D, (long long)a.T * D)) { set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled"); return PGB_ERR_CUDA; }
    auto inv = delta_inv_kernel<D>;
    const cudaError_t e = cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, InvSmem<D>::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_inv smem attribute"); return PGB_ERR_CUDA; }
    inv<<<dim3(NC, BH), 128, InvSmem<D>::bytes, stream>>>(mk, a.la, a.beta, (__nv_bfloat16 *)x_scratch, a.T, 1);
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
    cudaError_t e = cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, InvSmem<D>::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_inv smem attribute"); return PGB_ERR_CUDA; }
    inv<<<dim3(NC, BH), 128, InvSmem<D>::bytes, stream>>>(mk, la, beta, (__nv_bfloat16 *)X, T, 0);
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
