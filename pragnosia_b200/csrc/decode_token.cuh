// What the two kernels that take a whole decode step as one launch share (decode_token.cu, decode_flow.cu): the layer table, the
// staging of weights, roundings.
#pragma once
#include "decode_step.cuh"

namespace pgb {

constexpr int DT_THREADS = DEC_THREADS;                               // 256: what decode_step_body is written for
constexpr int DT_WARPS = DT_THREADS / 32;
constexpr unsigned DT_SPIN_LIMIT = 1u << 20;                          // polls of about a microsecond each

// One layer's pointers and norm settings; the host lays the table out as 18 64-bit words per layer.
struct DtLayer {
    const __nv_bfloat16 *Wc, *bc, *ln_w, *ln_b, *ow, *n_w, *n_b, *a_w, *a_b, *b_w, *b_b;
    const float *theta, *A, *on_w;
    float *S;
    int ln_kind, n_kind;
    float ln_eps, n_eps;
    float on_eps;                                                     // of the per-head RMS norm on the read
    int pad;
};
static_assert(sizeof(DtLayer) == 18 * 8, "the host writes 18 words per layer");

__device__ __forceinline__ void dt_unpack8(const uint4 &raw, float (&f)[8]) {
    const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(b[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ uint4 dt_pack8(const float (&f)[8]) {
    uint4 raw;
    __nv_bfloat162 *b = reinterpret_cast<__nv_bfloat162 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    return raw;
}
__device__ __forceinline__ float dt_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ void dt_cp_async16(void *smem_dst, const void *gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void dt_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void dt_cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

constexpr int DT_PIECES = 12;                                         // 128-bit pieces of weights a lane has in flight per item
constexpr int DT_DEPTH = 3;                                           // items a warp has in flight or in use
constexpr int DT_STAGE_U4 = DT_DEPTH * DT_PIECES * 32;                // a warp's staging buffers, in uint4

}  // namespace pgb
