// The plain rule's prefill in full fp32 (FFMA), chunk-parallel: the precise mode for callers that hand over scratch.
//
// The walk of prefill_fp32.cu gives a chain to one CTA (two at head dim 128), and two sequences of twelve heads then occupy
// 24 of 148 SMs for the whole sequence. Only S_{c+1} = e^{L_C} S_c + U_c is sequential, so here
//   1. fp32_outer_kernel   a CTA per (chain, chunk, 64 x 64 tile of the state):  U_c = (K w)^T V,  w_s = e^{L_C - L_s}
//   2. fp32_states_kernel  elementwise over the chunks, in place of U:           S_c, and the final state
//   3. fp32_out_kernel     a CTA per (chain, chunk, 64 value columns):           o = ((Q K^T) dec) V + e^L (Q S_c)
// Every product is 64 x 64 outputs by 256 threads, a 4 x 4 tile each, with both operands contraction-major in shared memory
// (two 16-byte loads per 16 multiply-adds), which puts the FFMA pipe ahead of shared memory. Same masking as the walk: rows
// past T are zero tokens with log-decay 0. B2 H12 T512 D64: 131 us as a walk -> 27 us (states 6.5,
// prefix 3.2, outputs 17.4).
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
// rows t0.. of a (T x D) matrix, columns c0..c0+63, as they lie: dst[row][col]
__device__ __forceinline__ void pc_rows(float *dst, const float *src, int t0, int T, int D, int c0, int tid, const float *scale) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = tid + PC_NT * i, r = idx >> 4, c = 4 * (idx & 15);
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + r < T) x = *reinterpret_cast<const float4 *>(src + (size_t)(t0 + r) * D + c0 + c);
        if (scale != nullptr) { const float w = scale[r]; x.x *= w; x.y *= w; x.z *= w; x.w *= w; }
        *reinterpret_cast<float4 *>(dst + r * PC_P + c) = x;
    }
}
// the same transposed: dst[col][row], D columns. A thread takes one row's four adjacent columns; lanes run over rows, so the
// four stores of a warp hit consecutive banks
template <int D>
__device__ __forceinline__ void pc_cols(float *dst, const float *src, int t0, int T, int tid) {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
        const int idx = tid + PC_NT * i, r = idx & 63, c = 4 * (idx >> 6);
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + r < T) x = *reinterpret_cast<const float4 *>(src + (size_t)(t0 + r) * D + c);
        dst[c * PC_P + r] = x.x; dst[(c + 1) * PC_P + r] = x.y; dst[(c + 2) * PC_P + r] = x.z; dst[(c + 3) * PC_P + r] = x.w;
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
    if (tid < 32) pc_decay(p.la + (size_t)bh * T, t0, T, tid, L);
    pc_rows(Vs, p.v + (size_t)bh * T * D, t0, T, D, j0, tid, nullptr);
    __syncthreads();
    if (tid < 64) w[tid] = expf(fminf(L[63] - L[tid], 0.f));
    if (tid == 0 && blockIdx.z == 0) p.Ltot[(size_t)bh * p.NC + c] = L[63];
    __syncthreads();
    pc_rows(Ks, p.k + (size_t)bh * T * D, t0, T, D, i0, tid, w);
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
    pc_cols<D>(Qt, p.q + base, t0, T, tid);
    pc_cols<D>(Kt, p.k + base, t0, T, tid);
    pc_rows(Vs, p.v + base, t0, T, D, j0, tid, nullptr);
    if (tid < 32) pc_decay(p.la + (size_t)bh * T, t0, T, tid, L);
    __syncthreads();
    float acc[4][4] = {};
    pc_product<D>(acc, Qt, Kt, ty, tx);
    __syncthreads();                                                  // K is consumed: the state's columns take its place
    {
        const float *src = p.U + ((size_t)bh * p.NC + c) * D * D + j0;
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            const int idx = tid + PC_NT * i, r = idx >> 4, cc = 4 * (idx & 15);
            *reinterpret_cast<float4 *>(Kt + r * PC_P + cc) = *reinterpret_cast<const float4 *>(src + (size_t)r * D + cc);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {                                 // A = (Q K^T) dec, transposed
            const int s = 4 * tx + j;
            float x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { const int t = 4 * ty + i; x[i] = s <= t ? acc[i][j] * expf(fminf(L[t] - L[s], 0.f)) : 0.f; }
            *reinterpret_cast<float4 *>(At + s * PC_P + 4 * ty) = make_float4(x[0], x[1], x[2], x[3]);
        }
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
    const cudaError_t e = cudaFuncSetAttribute(fp32_out_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PcOut<D>::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "fp32_out smem attribute"); return PGB_ERR_CUDA; }
    fp32_outer_kernel<D><<<dim3((unsigned)NC, (unsigned)BH, (D / 64) * (D / 64)), PC_NT, 0, st>>>(p);
    int rc = check_launch("fp32_outer_kernel");
    if (rc != PGB_OK) return rc;
    fp32_states_kernel<<<dim3(D * D / 4 / 256, (unsigned)BH), 256, 0, st>>>(scratch, Ltot, a.S0, a.theta, a.shift_dev, a.shift_host, a.sent, a.S_out, NC, a.H, D);
    if ((rc = check_launch("fp32_states_kernel")) != PGB_OK) return rc;
    fp32_out_kernel<D><<<dim3((unsigned)NC, (unsigned)BH, D / 64), PC_NT, PcOut<D>::bytes, st>>>(p);
    return check_launch("fp32_out_kernel");
}

int prefill_fp32_chunk_launch(const PrefillArgs &a, int o_dtype, int D, void *scratch, cudaStream_t st) {
    return D == 64 ? prefill_fp32_chunk_go<64>(a, o_dtype, (float *)scratch, st) : prefill_fp32_chunk_go<128>(a, o_dtype, (float *)scratch, st);
}

}  // namespace pgb
