// Delta-rule chunked prefill on the tensor cores (tcgen05.mma, TMEM accumulators, TMA-fed tiles): two kernels.
//
// The delta rule writes v minus what the memory already returns for the key: S_t = a_t S_{t-1} + k_t [b_t (v_t - a_t S_{t-1}^T k_t)]^T.
// In a 64-token chunk the residuals actually written, W, solve (I + N) W = rhs with
//     N = diag(beta) strictly_lower((K K^T) * dec),   rhs = diag(beta) (V - e^{L} K S_entering),
// (reference src/assoc.py:207-251). N does not depend on the state, so
//
//   delta_inv_kernel   (chunk-parallel, one CTA per (sequence-head, chunk)): K K^T on the tensor core, N in fp32, then
//                      X = (I + N)^-1 by forward substitution in true fp32 FFMA -- one thread per column of X, every
//                      intermediate bounded (the reduced-precision Neumann doubling the reference warns about at
//                      src/assoc_kernel.py:577-582 is never formed). X goes to a scratch buffer as bf16 head + tail.
//   delta_walk_kernel  (delta_walk.cuh; one CTA per (sequence, head), walking the chunks): W = X rhs, the state update and o.
//
// Everything fp32 that re-enters the tensor core (S, rhs, X, A, W) is split into bf16 head + tail and multiplied as
// head*head + head*tail + tail*head. Every mbarrier wait is bounded.
//
// Measured, B8 H16 T8192 D128 (1.1 GB of operands): walk 1311 -> 407 us, the whole call 1640 -> 750 us.
#include "delta_walk.cuh"

namespace pgb {

constexpr float TD_LOG2E = 1.4426950408889634f;

// decay statistics of one 64-token chunk by warps 0 and 1 (tid < 64): L (inclusive cumulative log-decay), e^L,
// w = e^{L_C - L} (0 past T) and beta (0 past T)
__device__ __forceinline__ void chunk_stats(const float *la, const float *beta, int t0, int T, int tid, int lane, int warp,
                                            float *Ls, float *eLs, float *wts, float *bes) {
    const int t = t0 + tid, tx = t0 + (tid ^ 32);
    const float own = t < T ? la[t] : 0.f, other = tx < T ? la[tx] : 0.f;
    float sc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, sc, o);
        if (lane >= o) sc += n;
    }
    const float sum_other = warp_sum(other), sum_own = __shfl_sync(0xffffffffu, sc, 31);
    const float L = sc + (warp == 1 ? sum_other : 0.f), Ltot = sum_own + sum_other;
    Ls[tid] = L;
    if (eLs != nullptr) eLs[tid] = expf(L);
    if (wts != nullptr) wts[tid] = t < T ? expf(fminf(Ltot - L, 0.f)) : 0.f;
    bes[tid] = t < T ? beta[t] : 0.f;
}

// ------------------------------------------------------------------------------------------------ X = (I + N)^-1
template <int D>
struct InvSmem {
    static constexpr int off_k = 0;                                   // K tile, TC_C x D bf16
    static constexpr int NP = 68;                                     // row pitch of N in floats (16-byte aligned, spreads banks)
    static constexpr int off_n = TC_C * D * 2;                        // N fp32 [64][NP]
    static constexpr int off_x = off_n + TC_C * NP * 4;               // X head, X tail: [64][64] bf16 each
    static constexpr int off_misc = off_x + 2 * TC_C * TC_C * 2;
    static constexpr int bytes = off_misc + 1024 + 1024;
};

template <int D>
__global__ void __launch_bounds__(128) delta_inv_kernel(const __grid_constant__ CUtensorMap mk, const float *__restrict__ la_all,
                                                        const float *__restrict__ beta_all, __nv_bfloat16 *__restrict__ X, int T,
                                                        int with_tail) {
    using SM = InvSmem<D>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    float *Nf = reinterpret_cast<float *>(sm + SM::off_n);
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
    if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 64);
    if (warp < 2) chunk_stats(la_all + (size_t)bh * T, beta_all + (size_t)bh * T, t0, T, tid, lane, warp, Ls, nullptr, nullptr, bes);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    bool ok = mbar_wait(bar_k, 0, 11);
    if (tid == 0 && ok) {
        constexpr uint32_t I_KK = idesc_bf16(64, 64, 0, 0);
        const uint64_t dk = smem_desc(base + SM::off_k, 16, 1024);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            const uint32_t ko = ((uint32_t)(k >> 2) * 8192u + (uint32_t)(k & 3) * 32u) >> 4;
            mma_bf16(tmem, dk + ko, dk + ko, I_KK, k > 0);
        }
        mma_commit(bar_m);
    }
    if (ok && !mbar_wait(bar_m, 0, 12)) ok = false;
    tc_fence_after();
    // ---- N = beta_t (k_t . k_s) exp(min(L_t - L_s, 0)) for s < t, else 0.   Each warp: its 16 rows, all 64 columns.
    {
        const int fr = lane >> 2, fq = lane & 3, r0 = 16 * warp + fr, r1 = r0 + 8;
        float kk[32];
        tmem_ld_frag8(tmem + ((uint32_t)(32 * warp) << 16), kk);
        tmem_ld_wait();
        const float L0 = Ls[r0] * TD_LOG2E, L1 = Ls[r1] * TD_LOG2E, b0 = bes[r0], b1 = bes[r1];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int s = 8 * j + 2 * fq + e;
                const float Lsv = Ls[s] * TD_LOG2E;
                Nf[r0 * SM::NP + s] = (s < r0) ? b0 * kk[4 * j + e] * exp2f(fminf(L0 - Lsv, 0.f)) : 0.f;
                Nf[r1 * SM::NP + s] = (s < r1) ? b1 * kk[4 * j + 2 + e] * exp2f(fminf(L1 - Lsv, 0.f)) : 0.f;
            }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 64);
    // ---- column j of X: x_t = [t == j] - sum_{s<t} N[t][s] x_s   (x_s = 0 above the diagonal, so one code path for all j)
    __nv_bfloat16 *Xh = reinterpret_cast<__nv_bfloat16 *>(sm + SM::off_x), *Xl = Xh + TC_C * TC_C;
    if (tid < TC_C) {
        float x[TC_C];
#pragma unroll
        for (int t = 0; t < TC_C; ++t) {
            float acc0 = (t == tid) ? 1.f : 0.f, acc1 = 0.f;
            const float4 *row = reinterpret_cast<const float4 *>(Nf + t * SM::NP);
#pragma unroll
            for (int s4 = 0; s4 < (t + 3) / 4; ++s4) {
                const float4 n = row[s4];                             // the same address for every thread: a broadcast
                if (4 * s4 + 0 < t) acc0 = fmaf(-n.x, x[4 * s4 + 0], acc0);
                if (4 * s4 + 1 < t) acc1 = fmaf(-n.y, x[4 * s4 + 1], acc1);
                if (4 * s4 + 2 < t) acc0 = fmaf(-n.z, x[4 * s4 + 2], acc0);
                if (4 * s4 + 3 < t) acc1 = fmaf(-n.w, x[4 * s4 + 3], acc1);
            }
            x[t] = acc0 + acc1;
            __nv_bfloat16 hi, lo;
            split_bf16(x[t], hi, lo);
            Xh[t * 64 + tid] = hi;
            Xl[t * 64 + tid] = lo;
        }
    }
    __syncthreads();
    // ---- head then tail, 8 KB each, to the scratch buffer; or the head alone, densely packed (the stand-alone operator)
    {
        uint4 *dst = reinterpret_cast<uint4 *>(X + ((size_t)bh * NC + c) * ((with_tail ? 2 : 1) * TC_C * TC_C));
        const uint4 *src = reinterpret_cast<const uint4 *>(Xh);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (with_tail || i < 4) dst[tid + 128 * i] = src[tid + 128 * i];
    }
}

// ------------------------------------------------------------------------------------------------ host side
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
    auto inv = delta_inv_kernel<D>;
    auto walk = delta_walk_kernel<D, false>;
    cudaError_t e = cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, InvSmem<D>::bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, DwSmem<D, false>::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_walk smem attribute"); return PGB_ERR_CUDA; }
    inv<<<dim3(NC, BH), 128, InvSmem<D>::bytes, stream>>>(m.k, a.la, a.beta, (__nv_bfloat16 *)x_scratch, a.T, 1);
    int rc = check_launch("delta_inv_kernel");
    if (rc != PGB_OK) return rc;
    DwParams p{};
    p.la = a.la; p.beta = a.beta; p.S0 = a.S0; p.theta = a.theta; p.shift_dev = a.shift_dev; p.shift_host = a.shift_host;
    p.S_out = a.S_out; p.want_sent = a.sent != nullptr; p.want_w = a.W_out != nullptr; p.H = a.H; p.T = a.T; p.o_is_f32 = f32;
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
