// The plain rule's prefill in full fp32 (FFMA), chunk-parallel: the precise mode for callers that hand over scratch.
//
// The walk of prefill_fp32.cu gives a chain to one CTA (two at head dim 128), and two sequences of twelve heads then occupy
// 24 of 148 SMs for the whole sequence. Only S_{c+1} = e^{L_C} S_c + U_c is sequential, so here
//   1. fp32_outer_kernel   a CTA per (chain, chunk, 64 x 64 tile of the state):  U_c = (K w)^T V,  w_s = e^{L_C - L_s}
//   2. fp32_states_kernel  elementwise over the chunks, in place of U:           S_c, and the final state
//   3. fp32_out_kernel     a CTA per (chain, chunk, 64 value columns):           o = ((Q K^T) dec) V + e^L (Q S_c)
// Every product is 64 x 64 outputs by 256 threads, a 4 x 4 tile each, with both operands contraction-major in shared memory
// (two 16-byte loads per 16 multiply-adds). Same masking as the walk: rows
// past T are zero tokens with log-decay 0. The three are programmatic dependents of one another: the output kernel's scores need no state, so its
// CTAs load and multiply while the two before it run. What bounds the output kernel is instruction issue and the latency of 8 to 24 warps an SM
// (17 us at B2 H12 T512 D64); 8 x 8 outputs a thread (fewer loads, half the warps) and halves of a chunk per CTA took the same or longer.
// B2 H12 T512 D64: 131 us as a walk, 26 behind one another, 21 so; a call of one chunk 15 -> 11.
#include "common.cuh"

namespace pgb {

constexpr int PC_C = 64, PC_NT = 256, PC_P = 68;                      // chunk, threads, row pitch in floats (16-byte aligned)

// acc[i][j] += sum_k A[k][4 ty + i] B[k][4 tx + j]
template <int K>
__device__ __forceinline__ void pc_product(float (&acc)[4][4], const float *A, const float *B, int ty, int tx) {
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
        const float4 a = *reinterpret_cast<const float4 *>(A + k * PC_P + 4 * ty), b = *reinterpret_cast<const float4 *>(B + k * PC_P + 4 * tx);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
}
// Operands travel in two steps, all of a thread's loads first and its stores to shared memory behind them (the compiler moves no load across
// such a store, so written as one step every piece waits for the one before it).
// rows t0.. of a (T x D) matrix, columns c0..c0+63, as they lie: dst[row][col]
__device__ __forceinline__ void pc_load(float4 (&x)[4], const float *src, int t0, int T, int D, int c0, int tid) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = tid + PC_NT * i, r = idx >> 4, c = 4 * (idx & 15);
        x[i] = t0 + r < T ? *reinterpret_cast<const float4 *>(src + (size_t)(t0 + r) * D + c0 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__device__ __forceinline__ void pc_put(float *dst, const float4 (&x)[4], int tid) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = tid + PC_NT * i;
        *reinterpret_cast<float4 *>(dst + (idx >> 4) * PC_P + 4 * (idx & 15)) = x[i];
    }
}
// the same transposed: dst[col][row], D columns. A thread takes one row's four adjacent columns; lanes run over rows, so the
// four stores of a warp hit consecutive banks
template <int D>
__device__ __forceinline__ void pc_cols_load(float4 (&x)[D / 16], const float *src, int t0, int T, int tid) {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
        const int idx = tid + PC_NT * i, r = idx & 63, c = 4 * (idx >> 6);
        x[i] = t0 + r < T ? *reinterpret_cast<const float4 *>(src + (size_t)(t0 + r) * D + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
template <int D>
__device__ __forceinline__ void pc_cols_put(float *dst, const float4 (&x)[D / 16], int tid) {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
        const int idx = tid + PC_NT * i, r = idx & 63, c = 4 * (idx >> 6);
        dst[c * PC_P + r] = x[i].x; dst[(c + 1) * PC_P + r] = x[i].y; dst[(c + 2) * PC_P + r] = x[i].z; dst[(c + 3) * PC_P + r] = x[i].w;
    }
}
// L (inclusive cumulative log-decay of the chunk) by warp 0, two tokens a lane; returns nothing, the caller synchronises
__device__ __forceinline__ void pc_decay(const float *la, int t0, int T, int lane, float *L) {
    float sl = t0 + lane < T ? la[t0 + lane] : 0.f, sh = t0 + lane + 32 < T ? la[t0 + lane + 32] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float nl = __shfl_up_sync(0xffffffffu, sl, o), nh = __shfl_up_sync(0xffffffffu, sh, o);
        if (lane >= o) { sl += nl; sh += nh; }
    }
    sh += __shfl_sync(0xffffffffu, sl, 31);
    L[lane] = sl; L[lane + 32] = sh;
}

struct PcParams {
    const float *q, *k, *v, *la;
    float *U, *Ltot;                                                  // [BH][NC][D][D] (then the entering states), [BH][NC]
    void *o; int o_is_bf16;
    int T, NC;
};

template <int D>
__global__ void __launch_bounds__(PC_NT) fp32_outer_kernel(PcParams p) {
    __shared__ __align__(16) float Ks[PC_C * PC_P], Vs[PC_C * PC_P], L[64], w[64];
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, c = blockIdx.x, bh = blockIdx.y, t0 = c * PC_C, T = p.T;
    const int i0 = 64 * (blockIdx.z % (D / 64)), j0 = 64 * (blockIdx.z / (D / 64));
    float4 kx[4], vx[4];
    pc_load(kx, p.k + (size_t)bh * T * D, t0, T, D, i0, tid);
    pc_load(vx, p.v + (size_t)bh * T * D, t0, T, D, j0, tid);
    pdl_launch_dependents();
    if (tid < 32) {
        pc_decay(p.la + (size_t)bh * T, t0, T, tid, L);
        __syncwarp();
        const float end = L[63];
        w[tid] = expf(fminf(end - L[tid], 0.f)); w[tid + 32] = expf(fminf(end - L[tid + 32], 0.f));
        if (tid == 0 && blockIdx.z == 0) p.Ltot[(size_t)bh * p.NC + c] = end;
    }
    pc_put(Vs, vx, tid);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float f = w[(tid + PC_NT * i) >> 4]; kx[i].x *= f; kx[i].y *= f; kx[i].z *= f; kx[i].w *= f; }
    pc_put(Ks, kx, tid);
    __syncthreads();
    float acc[4][4] = {};
    pc_product<PC_C>(acc, Ks, Vs, ty, tx);
    float *dst = p.U + (((size_t)bh * p.NC + c) * D + i0 + 4 * ty) * D + j0 + 4 * tx;
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float4 *>(dst + (size_t)i * D) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// a thread owns two value columns of one pair of key rows (the rebase of the entering state rotates pairs of rows)
__global__ void __launch_bounds__(256) fp32_states_kernel(float *__restrict__ U, const float *__restrict__ Ltot, const float *__restrict__ S0,
                                                          const float *__restrict__ theta, const float *__restrict__ shift_dev, float shift_host,
                                                          __nv_bfloat16 *__restrict__ sent, float *__restrict__ S_out, int NC, int H, int D) {
    const int e = blockIdx.x * 256 + threadIdx.x, bh = blockIdx.y, i = e / (D / 2), j = 2 * (e % (D / 2));
    pdl_launch_dependents();
    const size_t DD = (size_t)D * D, at = (size_t)(2 * i) * D + j;
    float2 a = make_float2(0.f, 0.f), b = a;
    if (S0 != nullptr) {
        a = *reinterpret_cast<const float2 *>(S0 + bh * DD + at);
        b = *reinterpret_cast<const float2 *>(S0 + bh * DD + at + D);
        const float shift = theta == nullptr ? 0.f : (shift_dev != nullptr ? *shift_dev : shift_host);
        if (shift != 0.f) {
            float sn, cs;
            sincosf(-shift * theta[(size_t)(bh % H) * (D / 2) + i], &sn, &cs);
            const float2 ra = make_float2(a.x * cs - b.x * sn, a.y * cs - b.y * sn), rb = make_float2(a.x * sn + b.x * cs, a.y * sn + b.y * cs);
            a = ra; b = rb;
        }
    }
    pdl_wait();                                                       // U and the chunks' decays
    for (int c0 = 0; c0 < NC; c0 += 8) {                              // eight chunks' additions requested ahead of the recurrence
        float2 ua[8], ub[8];
        float d[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c0 + k < NC) {
                const size_t base = ((size_t)bh * NC + c0 + k) * DD + at;
                ua[k] = *reinterpret_cast<const float2 *>(U + base);
                ub[k] = *reinterpret_cast<const float2 *>(U + base + D);
                d[k] = expf(Ltot[(size_t)bh * NC + c0 + k]);
            }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c0 + k < NC) {
                const size_t base = ((size_t)bh * NC + c0 + k) * DD + at;
                *reinterpret_cast<float2 *>(U + base) = a;
                *reinterpret_cast<float2 *>(U + base + D) = b;
                if (sent != nullptr) {
                    *reinterpret_cast<__nv_bfloat162 *>(sent + base) = __floats2bfloat162_rn(a.x, a.y);
                    *reinterpret_cast<__nv_bfloat162 *>(sent + base + D) = __floats2bfloat162_rn(b.x, b.y);
                }
                a = make_float2(fmaf(d[k], a.x, ua[k].x), fmaf(d[k], a.y, ua[k].y));
                b = make_float2(fmaf(d[k], b.x, ub[k].x), fmaf(d[k], b.y, ub[k].y));
            }
    }
    *reinterpret_cast<float2 *>(S_out + bh * DD + at) = a;
    *reinterpret_cast<float2 *>(S_out + bh * DD + at + D) = b;
}

template <int D>
struct PcOut {
    static constexpr int off_q = 0, off_k = D * PC_P, off_a = 2 * D * PC_P, off_v = off_a + PC_C * PC_P, off_l = off_v + PC_C * PC_P;
    static constexpr size_t bytes = (size_t)(off_l + 64) * sizeof(float);
};

template <int D>
__global__ void __launch_bounds__(PC_NT) fp32_out_kernel(PcParams p) {
    using SM = PcOut<D>;
    extern __shared__ __align__(16) float pc_smem[];
    float *Qt = pc_smem + SM::off_q, *Kt = pc_smem + SM::off_k, *At = pc_smem + SM::off_a, *Vs = pc_smem + SM::off_v, *L = pc_smem + SM::off_l;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, c = blockIdx.x, bh = blockIdx.y, j0 = 64 * blockIdx.z, t0 = c * PC_C, T = p.T;
    const size_t base = (size_t)bh * T * D;
    {
        float4 qx[D / 16], kx[D / 16], vx[4];
        pc_cols_load<D>(qx, p.q + base, t0, T, tid);
        pc_cols_load<D>(kx, p.k + base, t0, T, tid);
        pc_load(vx, p.v + base, t0, T, D, j0, tid);
        if (tid < 32) pc_decay(p.la + (size_t)bh * T, t0, T, tid, L);
        pc_cols_put<D>(Qt, qx, tid);
        pc_cols_put<D>(Kt, kx, tid);
        pc_put(Vs, vx, tid);
    }
    __syncthreads();
    float acc[4][4] = {};
    pc_product<D>(acc, Qt, Kt, ty, tx);
    __syncthreads();                                                  // K is consumed: the state's columns take its place
#pragma unroll
    for (int j = 0; j < 4; ++j) {                                     // A = (Q K^T) dec, transposed
        const int s = 4 * tx + j;
        float x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { const int t = 4 * ty + i; x[i] = s <= t ? acc[i][j] * expf(fminf(L[t] - L[s], 0.f)) : 0.f; }
        *reinterpret_cast<float4 *>(At + s * PC_P + 4 * ty) = make_float4(x[0], x[1], x[2], x[3]);
    }
    pdl_wait();                                                       // the entering states
    {
        const float *src = p.U + ((size_t)bh * p.NC + c) * D * D + j0;
        float4 x[D / 16];
#pragma unroll
        for (int i = 0; i < D / 16; ++i) { const int idx = tid + PC_NT * i; x[i] = *reinterpret_cast<const float4 *>(src + (size_t)(idx >> 4) * D + 4 * (idx & 15)); }
#pragma unroll
        for (int i = 0; i < D / 16; ++i) { const int idx = tid + PC_NT * i; *reinterpret_cast<float4 *>(Kt + (idx >> 4) * PC_P + 4 * (idx & 15)) = x[i]; }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    pc_product<D>(acc, Qt, Kt, ty, tx);                               // Q S
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float e = expf(L[4 * ty + i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] *= e;
    }
    pc_product<PC_C>(acc, At, Vs, ty, tx);                            // + A V
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = t0 + 4 * ty + i;
        if (t < T) {
            const size_t off = base + (size_t)t * D + j0 + 4 * tx;
            if (p.o_is_bf16) {
                __nv_bfloat162 *d = reinterpret_cast<__nv_bfloat162 *>((__nv_bfloat16 *)p.o + off);
                d[0] = __floats2bfloat162_rn(acc[i][0], acc[i][1]); d[1] = __floats2bfloat162_rn(acc[i][2], acc[i][3]);
            } else *reinterpret_cast<float4 *>((float *)p.o + off) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
    }
}

size_t prefill_fp32_chunk_scratch_bytes(int B, int H, int T, int D) {
    const size_t n = (size_t)B * H * ((T + PC_C - 1) / PC_C);
    return n * ((size_t)D * D + 1) * sizeof(float);
}

template <int D>
static int prefill_fp32_chunk_go(const PrefillArgs &a, int o_dtype, float *scratch, cudaStream_t st) {
    const int BH = a.B * a.H, NC = (a.T + PC_C - 1) / PC_C;
    float *Ltot = scratch + (size_t)BH * NC * D * D;
    const PcParams p{(const float *)a.q, (const float *)a.k, (const float *)a.v, a.la, scratch, Ltot, a.o, o_dtype == PGB_BF16, a.T, NC};
    // Output CTAs that come while the first kernel's are still there go wherever there is room, three to an SM beside SMs with none: where they
    // all fit one or two to an SM, as many bytes of shared memory as leave room for no more keep them there (192 CTAs on 148 SMs: 30.7 us the call without, 20.7 with).
    // The size is the launch's; the limit belongs to the function, which threads with calls of other sizes share, so it is the same at every call.
    constexpr size_t ONE_PER_SM = 116 * 1024, TWO_PER_SM = 78 * 1024;
    static_assert(PcOut<D>::bytes <= ONE_PER_SM, "the function's limit is the largest size of all calls");
    const long long ctas = (long long)BH * NC * (D / 64), sms = sm_count();
    const size_t least = ctas <= sms ? ONE_PER_SM : ctas <= 2 * sms ? TWO_PER_SM : 0, out_bytes = PcOut<D>::bytes > least ? PcOut<D>::bytes : least;
    const cudaError_t e = cudaFuncSetAttribute(fp32_out_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ONE_PER_SM);
    if (e != cudaSuccess) { set_cuda_error(e, "fp32_out smem attribute"); return PGB_ERR_CUDA; }
    fp32_outer_kernel<D><<<dim3((unsigned)NC, (unsigned)BH, (D / 64) * (D / 64)), PC_NT, 0, st>>>(p);
    int rc = check_launch("fp32_outer_kernel");
    if (rc != PGB_OK) return rc;
    cudaError_t le = pdl_launch(fp32_states_kernel, dim3(D * D / 4 / 256, (unsigned)BH), dim3(256), (size_t)0, st, scratch, (const float *)Ltot, a.S0, a.theta,
                                a.shift_dev, a.shift_host, a.sent, a.S_out, NC, a.H, D);
    if (le == cudaSuccess) le = pdl_launch(fp32_out_kernel<D>, dim3((unsigned)NC, (unsigned)BH, D / 64), dim3(PC_NT), out_bytes, st, p);
    if (le != cudaSuccess) { set_cuda_error(le, "fp32 prefill launch"); return PGB_ERR_CUDA; }
    return check_launch("fp32_out_kernel");
}

int prefill_fp32_chunk_launch(const PrefillArgs &a, int o_dtype, int D, void *scratch, cudaStream_t st) {
    return D == 64 ? prefill_fp32_chunk_go<64>(a, o_dtype, (float *)scratch, st) : prefill_fp32_chunk_go<128>(a, o_dtype, (float *)scratch, st);
}

}  // namespace pgb
