// prep_bwd: the gradient of the normalise / gate / rotate plumbing (reference: src/assoc_kernel.py:774-826 _prep_bwd), for
// callers that train through it: with u = x / |x|, r = R(ang) u and g the gradient on r: du = R^T g,
// dx = (du - u (u . du)) / |x|, d ang = g2 r1 - g1 r2 per pair; theta's gradient is the sum of pos * d ang over batch and time,
// written as one partial per CTA and summed by the caller.
#include "common.cuh"

namespace pgb {

// ---------------------------------------------------------------------------------------------------- prep backward
constexpr int PB_WARPS = 8;                                           // consecutive tokens of one (sequence, head) per partial of theta's gradient
constexpr int PB_TOK = 32;                                            // ... and per CTA of the 16-byte form: their sum, and zeros in the other three places the callers' buffers have

template <typename T_, int PER>
__device__ __forceinline__ void pb_ld(float (&d)[PER], const T_ *p) {
#pragma unroll
    for (int i = 0; i < PER; ++i) d[i] = to_f32(p[i]);
}
template <typename T_, int PER>
__device__ __forceinline__ void pb_st(T_ *p, const float (&d)[PER]) {
#pragma unroll
    for (int i = 0; i < PER; ++i) from_f32(p[i], d[i]);
}

// qp, kp, vp: TIN views (B,T,H,D) with element strides (sb, st, sh);  dq, dk, dv: TG, contiguous (B,H,T,D)
// dqp, dkp, dvp: TIN, contiguous (B,T,H,D);  dgl fp32 (B,T,H);  dth_part fp32 [B * NT][H][D/2], NT = ceil(T / PB_WARPS); dth_part NULL: theta's gradient is not wanted
template <typename TIN, typename TG, int D>
__global__ void __launch_bounds__(PB_WARPS * 32)
prep_bwd_kernel(const TIN *__restrict__ qp, const TIN *__restrict__ kp, const TIN *__restrict__ vp, long long sb, long long st, long long sh,
                const TIN *__restrict__ gate, long long gsb, long long gst, const float *__restrict__ theta, const long long *__restrict__ pos,
                const TG *__restrict__ dq, const TG *__restrict__ dk, const TG *__restrict__ dv, TIN *__restrict__ dqp, TIN *__restrict__ dkp,
                TIN *__restrict__ dvp, float *__restrict__ dgl, float *__restrict__ dth_part, int T, int H, int NT) {
    constexpr int PER = D / 32, NP = PER / 2;
    __shared__ float part[PB_WARPS][D / 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pt = blockIdx.x, bh = blockIdx.y, b = bh / H, h = bh % H;
    const int t = pt * PB_WARPS + warp;
    float dang[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) dang[i] = 0.f;
    float p = 0.f;
    if (t < T) {
        const size_t in_off = (size_t)b * sb + (size_t)t * st + (size_t)h * sh + lane * PER;
        const size_t g_off = ((size_t)bh * T + t) * D + lane * PER;
        const size_t o_off = (((size_t)b * T + t) * H + h) * D + lane * PER;
        p = (float)pos[t];
        float cs[NP], sn[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) sincosf(p * theta[(size_t)h * (D / 2) + lane * NP + i], &sn[i], &cs[i]);
        float x[PER], gr[PER], out[PER];
        // ---- q and k: normalise, (gate,) rotate
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            pb_ld<TIN, PER>(x, (which ? kp : qp) + in_off);
            pb_ld<TG, PER>(gr, (which ? dk : dq) + g_off);
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) ss = fmaf(x[i], x[i], ss);
            const float inv = 1.0f / fmaxf(sqrtf(warp_sum(ss)), 1e-12f);
            float r1[NP], r2[NP], u1[NP], u2[NP];
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                u1[i] = x[2 * i] * inv; u2[i] = x[2 * i + 1] * inv;
                r1[i] = u1[i] * cs[i] - u2[i] * sn[i]; r2[i] = u1[i] * sn[i] + u2[i] * cs[i];
            }
            if (which == 1 && gate != nullptr) {
                const float sg = sigmoidf_(to_f32(gate[(size_t)b * gsb + (size_t)t * gst + h]));
                float dsg = 0.f;
#pragma unroll
                for (int i = 0; i < NP; ++i) dsg += gr[2 * i] * r1[i] + gr[2 * i + 1] * r2[i];
                dsg = warp_sum(dsg);
                if (lane == 0) dgl[((size_t)b * T + t) * H + h] = dsg * sg * (1.0f - sg);
#pragma unroll
                for (int i = 0; i < PER; ++i) gr[i] *= sg;
            }
            float du1[NP], du2[NP], dot = 0.f;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                dang[i] += gr[2 * i + 1] * r1[i] - gr[2 * i] * r2[i];
                du1[i] = gr[2 * i] * cs[i] + gr[2 * i + 1] * sn[i];
                du2[i] = gr[2 * i + 1] * cs[i] - gr[2 * i] * sn[i];
                dot += u1[i] * du1[i] + u2[i] * du2[i];
            }
            dot = warp_sum(dot);
#pragma unroll
            for (int i = 0; i < NP; ++i) { out[2 * i] = (du1[i] - u1[i] * dot) * inv; out[2 * i + 1] = (du2[i] - u2[i] * dot) * inv; }
            pb_st<TIN, PER>((which ? dkp : dqp) + o_off, out);
        }
        // ---- v: normalise only
        pb_ld<TIN, PER>(x, vp + in_off);
        pb_ld<TG, PER>(gr, dv + g_off);
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) ss = fmaf(x[i], x[i], ss);
        const float inv = 1.0f / fmaxf(sqrtf(warp_sum(ss)), 1e-12f);
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) dot = fmaf(x[i] * inv, gr[i], dot);
        dot = warp_sum(dot);
#pragma unroll
        for (int i = 0; i < PER; ++i) out[i] = (gr[i] - x[i] * inv * dot) * inv;
        pb_st<TIN, PER>(dvp + o_off, out);
    }
    if (dth_part == nullptr) return;
    // ---- theta: this CTA's share of the sum over batch and time, tokens added in a fixed order
#pragma unroll
    for (int i = 0; i < NP; ++i) part[warp][lane * NP + i] = dang[i] * p;
    __syncthreads();
    if (threadIdx.x < D / 2) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < PB_WARPS; ++w) s += part[w][threadIdx.x];
        dth_part[(((size_t)b * NT + pt) * H + h) * (D / 2) + threadIdx.x] = s;
    }
}

// The same for bf16 operands and gradients with 16-byte aligned rows: D/8 lanes share a row, 8 channels (four pairs) each, so a
// warp takes four rows (D = 64) or two: 16-byte accesses, a shuffle tree of three or four steps per sum instead of five, and a
// quarter of the instructions a row. Bound by instruction issue before HBM (four sincosf a lane). 90112 rows of 64:
// 54 -> 30-34 us; three CTAs an SM (80 registers, a few of them spilled in sincosf's slow path) instead of two: with a
// flushed L2 41.5 -> 34.9.
template <int D>
__global__ void __launch_bounds__(PB_WARPS * 32, 3)
prep8_bwd_kernel(const __nv_bfloat16 *__restrict__ qp, const __nv_bfloat16 *__restrict__ kp, const __nv_bfloat16 *__restrict__ vp, long long sb, long long st,
                 long long sh, const __nv_bfloat16 *__restrict__ gate, long long gsb, long long gst, const float *__restrict__ theta,
                 const long long *__restrict__ pos, const __nv_bfloat16 *__restrict__ dq, const __nv_bfloat16 *__restrict__ dk,
                 const __nv_bfloat16 *__restrict__ dv, __nv_bfloat16 *__restrict__ dqp, __nv_bfloat16 *__restrict__ dkp, __nv_bfloat16 *__restrict__ dvp,
                 float *__restrict__ dgl, float *__restrict__ dth_part, int T, int H, int NT) {
    constexpr int LPR = D / 8, RPC = PB_WARPS * 32 / LPR;
    __shared__ float part[PB_WARPS][D / 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, li = threadIdx.x % LPR;
    const int pt = blockIdx.x, bh = blockIdx.y, b = bh / H, h = bh % H;
    const unsigned mask = (LPR == 32 ? 0xffffffffu : ((1u << LPR) - 1u)) << (lane / LPR * LPR);
    auto row_sum = [&](float x) {
#pragma unroll
        for (int m = 1; m < LPR; m <<= 1) x += __shfl_xor_sync(mask, x, m);
        return x;
    };
    const float4 th = *reinterpret_cast<const float4 *>(theta + (size_t)h * (D / 2) + 4 * li);
    const float ang[4] = {th.x, th.y, th.z, th.w};
    float dsum[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t = pt * PB_TOK + threadIdx.x / LPR; t < min(T, (pt + 1) * PB_TOK); t += RPC) {
        const size_t in = (size_t)b * sb + (size_t)t * st + (size_t)h * sh + 8 * li, gr = ((size_t)bh * T + t) * D + 8 * li,
                     out = (((size_t)b * T + t) * H + h) * D + 8 * li;
        const uint4 xr[3] = {*reinterpret_cast<const uint4 *>(qp + in), *reinterpret_cast<const uint4 *>(kp + in), *reinterpret_cast<const uint4 *>(vp + in)};
        const uint4 gv[3] = {*reinterpret_cast<const uint4 *>(dq + gr), *reinterpret_cast<const uint4 *>(dk + gr), *reinterpret_cast<const uint4 *>(dv + gr)};
        const float p = (float)pos[t];
        const float sg = gate != nullptr ? sigmoidf_(__bfloat162float(gate[(size_t)b * gsb + (size_t)t * gst + h])) : 1.f;
        float cs[4], sn[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) sincosf(p * ang[i], &sn[i], &cs[i]);
#pragma unroll
        for (int w = 0; w < 3; ++w) {
            const __nv_bfloat162 *x2 = reinterpret_cast<const __nv_bfloat162 *>(&xr[w]), *g2 = reinterpret_cast<const __nv_bfloat162 *>(&gv[w]);
            float2 x[4], g[4];
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) { x[i] = __bfloat1622float2(x2[i]); g[i] = __bfloat1622float2(g2[i]); ss = fmaf(x[i].x, x[i].x, fmaf(x[i].y, x[i].y, ss)); }
            const float inv = 1.0f / fmaxf(sqrtf(row_sum(ss)), 1e-12f);
            float2 du[4];
            float dot = 0.f, dsg = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float u1 = x[i].x * inv, u2 = x[i].y * inv;
                if (w < 2) {
                    const float r1 = u1 * cs[i] - u2 * sn[i], r2 = u1 * sn[i] + u2 * cs[i];
                    if (w == 1) { dsg += g[i].x * r1 + g[i].y * r2; g[i].x *= sg; g[i].y *= sg; }
                    dsum[i] = fmaf(p, g[i].y * r1 - g[i].x * r2, dsum[i]);
                    du[i] = make_float2(g[i].x * cs[i] + g[i].y * sn[i], g[i].y * cs[i] - g[i].x * sn[i]);
                } else du[i] = g[i];
                dot += u1 * du[i].x + u2 * du[i].y;
            }
            dot = row_sum(dot);
            if (w == 1 && gate != nullptr) {
                dsg = row_sum(dsg);
                if (li == 0) dgl[((size_t)b * T + t) * H + h] = dsg * sg * (1.0f - sg);
            }
            uint4 res;
            __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&res);
#pragma unroll
            for (int i = 0; i < 4; ++i) o2[i] = __floats2bfloat162_rn((du[i].x - x[i].x * inv * dot) * inv, (du[i].y - x[i].y * inv * dot) * inv);
            *reinterpret_cast<uint4 *>((w == 0 ? dqp : w == 1 ? dkp : dvp) + out) = res;
        }
    }
    if (dth_part == nullptr) return;
    // theta: the warp's rows, then the warps, in a fixed order
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int m = LPR; m < 32; m <<= 1) dsum[i] += __shfl_xor_sync(0xffffffffu, dsum[i], m);
        if (lane < LPR) part[warp][4 * li + i] = dsum[i];
    }
    __syncthreads();
    if (threadIdx.x < D / 2) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < PB_WARPS; ++w) s += part[w][threadIdx.x];
        for (int k = 0; k < PB_TOK / PB_WARPS && 4 * pt + k < NT; ++k)
            dth_part[(((size_t)b * NT + 4 * pt + k) * H + h) * (D / 2) + threadIdx.x] = k == 0 ? s : 0.f;
    }
}

int prep_bwd_tiles(int T) { return (T + PB_WARPS - 1) / PB_WARPS; }

template <typename TIN, typename TG>
static int prep_bwd_go(const void *qp, const void *kp, const void *vp, long long sb, long long st, long long sh, const void *gate,
                       long long gsb, long long gst, const float *theta, const long long *pos, const void *dq, const void *dk,
                       const void *dv, void *dqp, void *dkp, void *dvp, float *dgl, float *dth_part, int B, int T, int H, int D,
                       cudaStream_t stream) {
    const int NT = prep_bwd_tiles(T);
    auto go = [&](auto kern) {
        kern<<<dim3(NT, B * H), PB_WARPS * 32, 0, stream>>>((const TIN *)qp, (const TIN *)kp, (const TIN *)vp, sb, st, sh, (const TIN *)gate,
                                                           gsb, gst, theta, pos, (const TG *)dq, (const TG *)dk, (const TG *)dv, (TIN *)dqp,
                                                           (TIN *)dkp, (TIN *)dvp, dgl, dth_part, T, H, NT);
    };
    if (D == 64) go(prep_bwd_kernel<TIN, TG, 64>); else go(prep_bwd_kernel<TIN, TG, 128>);
    return check_launch("prep_bwd_kernel");
}

int prep_bwd_launch(const void *qp, const void *kp, const void *vp, int in_dtype, long long sb, long long st, long long sh, const void *gate,
                    long long gsb, long long gst, const float *theta, const long long *pos, const void *dq, const void *dk, const void *dv,
                    int g_dtype, void *dqp, void *dkp, void *dvp, float *dgl, float *dth_part, int B, int T, int H, int D,
                    cudaStream_t stream) {
    const void *rows[] = {qp, kp, vp, dq, dk, dv, dqp, dkp, dvp, theta};
    bool wide = in_dtype == PGB_BF16 && g_dtype == PGB_BF16 && sb % 8 == 0 && st % 8 == 0 && sh % 8 == 0;
    for (const void *r : rows) wide = wide && aligned(r, 16);
    if (wide) {
        typedef const __nv_bfloat16 *In;
        typedef __nv_bfloat16 *Out;
        const int NT = prep_bwd_tiles(T);
        auto go = [&](auto kern) {
            kern<<<dim3((T + PB_TOK - 1) / PB_TOK, B * H), PB_WARPS * 32, 0, stream>>>((In)qp, (In)kp, (In)vp, sb, st, sh, (In)gate, gsb, gst, theta, pos, (In)dq, (In)dk, (In)dv,
                                                               (Out)dqp, (Out)dkp, (Out)dvp, dgl, dth_part, T, H, NT);
        };
        if (D == 64) go(prep8_bwd_kernel<64>); else go(prep8_bwd_kernel<128>);
        return check_launch("prep8_bwd_kernel");
    }
#define PB_ARGS qp, kp, vp, sb, st, sh, gate, gsb, gst, theta, pos, dq, dk, dv, dqp, dkp, dvp, dgl, dth_part, B, T, H, D, stream
    if (in_dtype == PGB_F32) return g_dtype == PGB_F32 ? prep_bwd_go<float, float>(PB_ARGS) : prep_bwd_go<float, __nv_bfloat16>(PB_ARGS);
    return g_dtype == PGB_F32 ? prep_bwd_go<__nv_bfloat16, float>(PB_ARGS) : prep_bwd_go<__nv_bfloat16, __nv_bfloat16>(PB_ARGS);
#undef PB_ARGS
}

}  // namespace pgb
