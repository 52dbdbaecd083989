// The delta rule with few chains (head dim 64): segments of a chain side by side. A chunk's update is linear in the state it is entered with, so over a
// segment entered with E
//     o_t = oB_t + E^T a_t,      S_end = A E + B
// where oB, B come of the segment entered with zero, and a_t = (map to t)^T q_t, A of its linear map alone (V = 0, entered with the identity). The walk
// forms both at once in the lanes that head dim 64 leaves idle (delta_walk.cuh, WITH_MAP). Then
//   delta_chain_kernel   E_{i+1} = A_i E_i + B_i over the segments of a chain, value columns side by side;
//   delta_join_kernel    o = oB + E^T a to fp32's precision, a CTA per chunk; then what the walk's caller does with the read (the per-head RMS norm and the token-major
//                        layout of the layer, or neither).
// The chain of a sequence is a segment long instead of a sequence: 36 chains of 21 chunks: 55 us -> 24 for
// the walk of four segments of six, 6 and 13 (a language model's pass of three sequences of 1333 tokens, six layers, 958 -> 847 us); 12 chains of 63 chunks
// 175 -> 62 with their inverses (12 of it), 2 of 32 88 -> 36. Error against 64 bits, segments to whole chains, over decays and keys of seven kinds and four shapes: S (5e-6 where
// keys are drawn alike) 0.97 to 1.06 times, 1.00 on the mean; o (5.1e-6, read in fp32) 1.00 to 1.02 times, 1.004 on the mean: oB and E^T a round apart. The read in bf16, the
// default, rounds to 300 times that.
#include "delta_walk.cuh"

namespace pgb {

constexpr int DS_P = 68, DS_PE = 72;                                  // pitches of a and E in shared memory: conflict-free as operands
constexpr long long DS_SCRATCH_MOST = 256ll << 20;

struct DeltaSegs { int n, chunks; };
// How many segments: at most what fills the chip at one CTA an SM, where that shortens a chain by more than it costs. Microseconds: a chunk of the walk 2.6 and 5 for its start,
// with the map 3.0 and 7 for its start; a step of the chain kernel 0.8; 0.19 a thousand rows joined; 10 for the two launches.
DeltaSegs delta_segment_plan(int B, int H, int T, int D) {
    const int NC = (T + TC_C - 1) / TC_C, sms = sm_count();
    const long long BH = (long long)B * H;
    DeltaSegs best{1, NC};
    double cost = 2.6 * NC + 5.0;
    if (D != 64) return best;
    for (int n = 2; n * BH <= sms && n <= NC; ++n) {
        const int len = (NC + n - 1) / n;
        const double c = 3.0 * len + 0.8 * n + 17.0 + 0.19e-3 * BH * T;
        if (c + 1.0 < cost && (NC + len - 1) / len == n) { cost = c - 1.0; best = {n, len}; }
    }
    return BH * ((long long)T * 2 * 64 + best.n * 2ll * 64 * 64) * 4 <= DS_SCRATCH_MOST ? best : DeltaSegs{1, NC};
}
struct DeltaSegScratch {                                              // fp32: oB, a [BH][T][64] each; B, A [n][BH][64][64] each
    size_t oB, a, B, A, bytes;
    DeltaSegScratch(long long BH, long long T, int n) {
        oB = 0; a = (size_t)BH * T * 256; B = 2 * a; A = B + (size_t)n * BH * 64 * 64 * 4; bytes = A + (size_t)n * BH * 64 * 64 * 4;
    }
};
size_t delta_segment_scratch_bytes(int B, int H, int T, int D) {
    const DeltaSegs s = delta_segment_plan(B, H, T, D);
    return s.n < 2 ? 0 : DeltaSegScratch((long long)B * H, T, s.n).bytes;
}

// a load that stays where it is written: the compiler would otherwise move a row's loads to their uses, a round trip each (13 us a step of the chain)
__device__ __forceinline__ float4 ds_ld(const float *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// E_{i+1} = A_i E_i + B_i: a CTA takes 16 value columns of a chain, a thread eight of them in one key row; the next segment's A and B are on their way
// meanwhile. B_i's place takes E_{i+1}, the state entering segment i + 1; the last goes to S_out. Rolled loops: with A's row in registers and all 64
// steps of a product unrolled the kernel waited 9 us for its instructions, whatever the segments.
__global__ void __launch_bounds__(128) delta_chain_kernel(const float *__restrict__ A, float *__restrict__ B, float *__restrict__ S_out, int n, int BH) {
    __shared__ __align__(16) float E[64][16], As[64 * DS_P];
    const int tid = threadIdx.x, bh = blockIdx.x, c0 = 16 * blockIdx.y, r = tid >> 1, c = 8 * (tid & 1);
    const size_t step = (size_t)BH * 4096, at = (size_t)bh * 4096, mine = at + (size_t)r * 64 + c0 + c;
    pdl_launch_dependents();
    float4 x[2], b[2], a[8];
    auto fetch = [&](int i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = ds_ld(A + i * step + at + 4 * (tid + 128 * j));
#pragma unroll
        for (int j = 0; j < 2; ++j) b[j] = ds_ld(B + i * step + mine + 4 * j);
    };
#pragma unroll
    for (int j = 0; j < 2; ++j) x[j] = ds_ld(B + mine + 4 * j);
    fetch(1);
#pragma unroll 1
    for (int i = 1; i < n; ++i) {
#pragma unroll
        for (int j = 0; j < 2; ++j) *reinterpret_cast<float4 *>(&E[r][c + 4 * j]) = x[j];
#pragma unroll
        for (int j = 0; j < 8; ++j) *reinterpret_cast<float4 *>(As + ((tid >> 4) + 8 * j) * DS_P + 4 * (tid & 15)) = a[j];
        float acc[8] = {b[0].x, b[0].y, b[0].z, b[0].w, b[1].x, b[1].y, b[1].z, b[1].w};
        __syncthreads();
        if (i + 1 < n) fetch(i + 1);
#pragma unroll 2
        for (int k = 0; k < 64; k += 4) {
            const float4 av = *reinterpret_cast<const float4 *>(As + r * DS_P + k);
            const float f[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 e0 = *reinterpret_cast<const float4 *>(&E[k + q][c]), e1 = *reinterpret_cast<const float4 *>(&E[k + q][c + 4]);
                acc[0] = fmaf(f[q], e0.x, acc[0]); acc[1] = fmaf(f[q], e0.y, acc[1]); acc[2] = fmaf(f[q], e0.z, acc[2]); acc[3] = fmaf(f[q], e0.w, acc[3]);
                acc[4] = fmaf(f[q], e1.x, acc[4]); acc[5] = fmaf(f[q], e1.y, acc[5]); acc[6] = fmaf(f[q], e1.z, acc[6]); acc[7] = fmaf(f[q], e1.w, acc[7]);
            }
        }
        x[0] = make_float4(acc[0], acc[1], acc[2], acc[3]); x[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        float *dst = i + 1 < n ? B + i * step + mine : S_out + mine;
#pragma unroll
        for (int j = 0; j < 2; ++j) *reinterpret_cast<float4 *>(dst + 4 * j) = x[j];
        __syncthreads();                                              // E and A have been read
    }
}

struct DjParams {
    const float *oB, *a, *E; void *o; const float *w; float eps;      // E: [n][BH][64][64], entering segment i + 1; w: the norm's weight (NULL: no norm)
    int T, H, BH, seg_chunks, o_is_f32, token_major;
};

// A CTA per chunk of 64 tokens; warp w has tokens 16 (w % 4) .. and columns 32 (w / 4) .. Factors as two tf32 parts, tail by tail left out: 2^-21 of a product at most (the walk's own products keep 2^-16).
// 756 chunks: 13 us, as fp32 register tiles 17.
__global__ void __launch_bounds__(256) delta_join_kernel(const __grid_constant__ DjParams p) {
    __shared__ __align__(16) float as[64 * DS_P], es[64 * DS_PE], red[2][64];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H, seg = c / p.seg_chunks, t0 = c * TC_C, live = min(64, p.T - t0);
    const int m = 16 * (warp & 3), n0 = 32 * (warp >> 2), row[2] = {m + g, m + g + 8};
    const size_t first = (size_t)bh * p.T + t0;                       // the chunk's first row
    pdl_wait();
    if (seg > 0) {
        const float *E = p.E + ((size_t)(seg - 1) * p.BH + bh) * 4096;
        float4 x[4], e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = (tid >> 4) + 16 * i, col = 4 * (tid & 15);
            x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < live) x[i] = ds_ld(p.a + (first + r) * 64 + col);
            e[i] = ds_ld(E + r * 64 + col);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = (tid >> 4) + 16 * i, col = 4 * (tid & 15);
            *reinterpret_cast<float4 *>(as + r * DS_P + col) = x[i];
            *reinterpret_cast<float4 *>(es + r * DS_PE + col) = e[i];
        }
    }
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float2 x = make_float2(0.f, 0.f);
            if (row[r] < live) x = *reinterpret_cast<const float2 *>(p.oB + (first + row[r]) * 64 + n0 + 8 * j + 2 * t4);
            acc[j][2 * r] = x.x; acc[j][2 * r + 1] = x.y;
        }
    if (seg > 0) {
        __syncthreads();
#pragma unroll 2
        for (int k = 0; k < 64; k += 8) {
            uint32_t ah[4], al[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) tf32_split(as[row[i & 1] * DS_P + k + t4 + 4 * (i >> 1)], ah[i], al[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t eh[2], el[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) tf32_split(es[(k + t4 + 4 * i) * DS_PE + n0 + 8 * j + g], eh[i], el[i]);
                mma_tf32(acc[j], al, eh);
                mma_tf32(acc[j], ah, el);
                mma_tf32(acc[j], ah, eh);
            }
        }
    }
    float sc[2] = {1.f, 1.f};
    if (p.w != nullptr) {                                             // of the read as the walk alone would hand it on, in bf16
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float ss = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float &x = acc[j][2 * r + i];
                    x = __bfloat162float(__float2bfloat16_rn(x));
                    ss = fmaf(x, x, ss);
                }
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            ss += __shfl_xor_sync(0xffffffffu, ss, 2);
            if (t4 == 0) red[warp >> 2][row[r]] = ss;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; ++r) sc[r] = rsqrtf((red[0][row[r]] + red[1][row[r]]) * (1.f / 64.f) + p.eps);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool in = row[r] < live;
        const size_t dst = (p.token_major ? ((size_t)b * p.T + t0 + row[r]) * p.H + h : first + row[r]) * 64 + n0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (p.w != nullptr) {
                acc[j][2 * r] *= sc[r] * p.w[n0 + 8 * j + 2 * t4];
                acc[j][2 * r + 1] *= sc[r] * p.w[n0 + 8 * j + 2 * t4 + 1];
            }
        if (p.o_is_f32) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (in) *reinterpret_cast<float2 *>((float *)p.o + dst + 8 * j + 2 * t4) = make_float2(acc[j][2 * r], acc[j][2 * r + 1]);
        } else {
            // neighbouring lanes trade column pairs, so that a row's quad stores whole 32-byte sectors
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const __nv_bfloat162 ev2 = __floats2bfloat162_rn(acc[j][2 * r], acc[j][2 * r + 1]), od2 = __floats2bfloat162_rn(acc[j + 1][2 * r], acc[j + 1][2 * r + 1]);
                const uint32_t ev = *reinterpret_cast<const uint32_t *>(&ev2), od = *reinterpret_cast<const uint32_t *>(&od2);
                const uint32_t got = __shfl_xor_sync(0xffffffffu, (t4 & 1) ? ev : od, 1);
                if (in) *reinterpret_cast<uint2 *>((__nv_bfloat16 *)p.o + dst + 8 * (j + (t4 & 1)) + 4 * (t4 >> 1)) = (t4 & 1) ? make_uint2(got, od) : make_uint2(ev, got);
            }
        }
    }
}

int delta_inverse_launch(const PrefillArgs &a, int D, void *x_scratch, cudaStream_t stream);

// The prefill `a` (plain outputs; with a.rms_w the layer's: norm and token-major bf16) in the planned segments; scratch: delta_segment_scratch_bytes
int delta_segments_launch(const PrefillArgs &a, int o_dtype, void *x_scratch, void *scratch, cudaStream_t stream) {
    constexpr int D = 64;
    const int BH = a.B * a.H, NC = (a.T + TC_C - 1) / TC_C;
    const DeltaSegs s = delta_segment_plan(a.B, a.H, a.T, D);
    const DeltaSegScratch sc(BH, a.T, s.n);
    uint8_t *buf = (uint8_t *)scratch;
    float *oB = (float *)(buf + sc.oB), *ap = (float *)(buf + sc.a), *Bp = (float *)(buf + sc.B), *Ap = (float *)(buf + sc.A);
    DwMaps m{};
    if (!tc_make_map(&m.q, a.q, BH, a.T, D, D, (long long)a.T * D) || !tc_make_map(&m.k, a.k, BH, a.T, D, D, (long long)a.T * D) ||
        !tc_make_map(&m.v, a.v, BH, a.T, D, D, (long long)a.T * D) ||
        !tc_make_map(&m.x, x_scratch, (long long)BH * NC * 2, TC_C, TC_C, TC_C, TC_C * TC_C) ||
        !tc_make_store_map(&m.o, oB, true, BH, a.T, D, 32, 32) || !tc_make_store_map(&m.w, ap, true, BH, a.T, D, 32, 32)) {
        set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled");
        return PGB_ERR_CUDA;
    }
    auto walk = delta_walk_kernel<D, false, true>;
    cudaError_t e = cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, DwSmem<D, false>::bytes);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_walk smem attribute"); return PGB_ERR_CUDA; }
    int rc = delta_inverse_launch(a, D, x_scratch, stream);
    if (rc != PGB_OK) return rc;
    DwParams p{};
    p.la = a.la; p.beta = a.beta; p.S0 = a.S0; p.theta = a.theta; p.shift_dev = a.shift_dev; p.shift_host = a.shift_host;
    p.S_out = Bp; p.S_map = Ap; p.H = a.H; p.T = a.T; p.o_is_f32 = 1;
    p.rebase_chunks = a.rebase_chunks; p.rebase_shift = (float)(a.rebase_chunks * TC_C);
    p.BH = BH; p.seg_chunks = s.chunks;
    walk<<<(unsigned)(BH * s.n), DW_NT, DwSmem<D, false>::bytes, stream>>>(m, p);
    if ((rc = check_launch("delta_walk_kernel")) != PGB_OK) return rc;
    // launched plainly: as a programmatic dependent of the walk it took 18.8 us instead of 6.2 (36 chains of four segments)
    delta_chain_kernel<<<dim3((unsigned)BH, 4), 128, 0, stream>>>((const float *)Ap, Bp, a.S_out, s.n, BH);
    if ((rc = check_launch("delta_chain_kernel")) != PGB_OK) return rc;
    const DjParams j{oB, ap, Bp, a.o, a.rms_w, a.rms_eps, a.T, a.H, BH, s.chunks, o_dtype == PGB_F32, a.o_token_major};
    e = pdl_launch(delta_join_kernel, dim3((unsigned)NC, (unsigned)BH), dim3(256), (size_t)0, stream, j);
    if (e != cudaSuccess) { set_cuda_error(e, "delta_segments launch"); return PGB_ERR_CUDA; }
    return check_launch("delta_join_kernel");
}

int delta_segments_error_flag(int *out) { return tc_read_error_flag(out); }

}  // namespace pgb
