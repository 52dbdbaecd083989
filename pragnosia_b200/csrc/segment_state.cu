// The states entering the segments of a sequence, for the plain rule at head dim 64, so that the segments of one sequence can run
// side by side instead of one behind the other (the reference walks them in order, src/model.py:857-863). RAW: the windows of a
// long sequence, on the layer's raw projections. Else: a long prepared sequence cut so that its chains fill the chip.
//
//   segment_state_kernel    a CTA per (segment but the last, sequence, head): what the segment adds to the state by its end,
//                               U = sum_s e^{L_end - L_s} k_s v_s^T,
//                           one long product over the segment's tokens. With the decay taken to the segment's END (every
//                           exponent <= 0) nothing in it is sequential: the chunks stream through the plumbing (RAW: normalise,
//                           gate, rotate; the same arithmetic and roundings as the prefill kernel's) and accumulate in
//                           tensor memory.
//   segment_combine_kernel  E_{w+1} = e^{L_w} R E_w + U_w over the segments, elementwise, in place of U; R rotates by -len theta
//                           where the segments are windows, else only the sequence's own entering state is rebased.
//
// prefill_tc_ws_kernel then takes every segment with its own entering state. Bound by the tiles' latency (K and V are read a
// second time: 16 KB a chunk, three stages ahead of the product); with 12 chains of 8192 tokens the walk of a layer is 12 CTAs of
// 128 chunks without it and 192 CTAs of 8 with it. Prepared
// operands, whole call: B1 H12 T8192 174 -> 36 us, B1 H12 T2048 47 -> 19, B4 H16 T4096 93 -> 77.
#include "tc_common.cuh"

namespace pgb {

constexpr int SG_NT = 256, SG_D = 64, SG_ST = 3;                      // threads; head dim; stages
constexpr int SG_MAX = 1024, SG_MAX_PREPARED = 4096;                  // tokens of a segment at most

template <bool RAW, bool FINE> struct SgSmem {
    static constexpr int TILE = 8192, STAGE = (FINE ? 4 : 3) * TILE;  // K (then heads of K w), V, tails of K w, their rest
    static constexpr int MAX = RAW ? SG_MAX : SG_MAX_PREPARED;
    static constexpr int off_w = SG_ST * STAGE, off_g = off_w + MAX * 4, off_misc = off_g + (RAW ? MAX * 4 : 0), bytes = off_misc + 256 + 1024;
};
struct SgParams {
    const __nv_bfloat16 *decay, *gate; long long sb, st;              // logits (gate NULL: write everything), token and batch strides
    const float *decay_A; const float2 *rot; int rot_T;
    const float *la; int T;                                           // prepared operands: log-decays [BH][T]
    float *U, *Lend;                                                  // [nseg - 1][BH][D][D], [nseg - 1][BH]
    int BH, H; SegCut seg;
};

template <bool RAW, bool FINE>
__global__ void __launch_bounds__(SG_NT, FINE ? 1 : 2) segment_state_kernel(const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv,
                                                                 SgParams p) {
    using SM = SgSmem<RAW, FINE>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    float *ws = reinterpret_cast<float *>(sm + SM::off_w), *gs = reinterpret_cast<float *>(sm + SM::off_g);
    uint8_t *misc = sm + SM::off_misc;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + 64);
    float *part = reinterpret_cast<float *>(misc + 96);
    auto full = [&](int s) { return base + SM::off_misc + 8 * s; };
    auto done = [&](int s) { return base + SM::off_misc + 24 + 8 * s; };
    const uint32_t bar_end = base + SM::off_misc + 48;
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5), wg = warp >> 2, sub = warp & 3;
    const int seg = blockIdx.x / p.BH, bh = blockIdx.x - seg * p.BH, h = bh % p.H, b = bh / p.H;
    int tb, t_in, tokens;
    p.seg.at(seg, tb, t_in, tokens);
    const int NC = tokens / TC_C;
    auto load = [&](int c) {
        const uint32_t sb = base + (c % SG_ST) * SM::STAGE, bar = full(c % SG_ST);
        mbar_expect_tx(bar, 2 * SM::TILE);
        tma_load_3d(sb, &mk, bar, RAW ? h * SG_D : 0, tb + c * TC_C, RAW ? b : bh);
        tma_load_3d(sb + SM::TILE, &mv, bar, RAW ? h * SG_D : 0, tb + c * TC_C, RAW ? b : bh);
    };
    if (tid == 0) {
        for (int s = 0; s < SG_ST; ++s) { mbar_init(full(s), 1); mbar_init(done(s), 1); }
        mbar_init(bar_end, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 64);
    pdl_wait();
    if (tid == 0)
        for (int c = 0; c < 2 && c < NC; ++c) load(c);
    // ---- decay to the end of the segment and key gate of its tokens: a thread owns a few consecutive ones
    {
        constexpr int PER = SM::MAX / SG_NT;
        const float expA = RAW ? expf(p.decay_A[h]) : 1.f;
        float la[PER], g[RAW ? PER : 1], s = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int t = PER * tid + i;
            la[i] = 0.f;
            if constexpr (RAW) {
                g[i] = 1.f;
                if (t < tokens) {
                    const size_t off = (size_t)b * p.sb + (size_t)(tb + t) * p.st + h;
                    la[i] = -fast_softplus(__bfloat162float(p.decay[off])) * expA;
                    if (p.gate != nullptr) g[i] = fast_sigmoid(__bfloat162float(p.gate[off]));
                }
            } else if (t < tokens) la[i] = p.la[(size_t)bh * p.T + tb + t];
            s += la[i]; la[i] = s;                                    // running sum inside the thread
        }
        float sc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) sc += n;
        }
        if (lane == 31) part[warp] = sc;
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        float before = sc - s, total = 0.f;
#pragma unroll
        for (int w = 0; w < SG_NT / 32; ++w) { total += part[w]; if (w < warp) before += part[w]; }
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (PER * tid + i < tokens) {
                ws[PER * tid + i] = expf(fminf(total - (before + la[i]), 0.f));
                if constexpr (RAW) gs[PER * tid + i] = g[i];
            }
        if (tid == 0) p.Lend[(size_t)seg * p.BH + bh] = total;
        __syncthreads();
    }
    const uint32_t tmem = warp_uniform(*tmem_slot);
    pdl_launch_dependents();
    bool ok = true;
    for (int c = 0; c < NC; ++c) {
        const int st = c % SG_ST;
        uint8_t *kt = sm + st * SM::STAGE, *vt = kt + SM::TILE, *lt = vt + SM::TILE;
        ok = mbar_wait_warp(full(st), (c / SG_ST) & 1, 11);
        if (!RAW && ok) {                                             // K w, head and tail; V as it came
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int row = 32 * pass + 4 * warp + (lane >> 3);
                const uint32_t off = swz(row, lane & 7);
                const uint4 raw = *reinterpret_cast<const uint4 *>(kt + off);
                const __nv_bfloat162 *b2 = reinterpret_cast<const __nv_bfloat162 *>(&raw);
                const float w = ws[c * TC_C + row];
                float kw[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(b2[i]); kw[2 * i] = f.x * w; kw[2 * i + 1] = f.y * w; }
                uint4 hi, lo;
                if constexpr (FINE) {
                    uint4 rest;
                    split8(kw, hi, lo, rest);
                    *reinterpret_cast<uint4 *>(lt + SM::TILE + off) = rest;
                } else split8(kw, hi, lo);
                *reinterpret_cast<uint4 *>(kt + off) = hi;
                *reinterpret_cast<uint4 *>(lt + off) = lo;
            }
        }
        if (RAW && ok) {
            const int cp = lane & 7;
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int row = 32 * pass + 4 * warp + (lane >> 3), t = c * TC_C + row;
                const uint32_t off = swz(row, cp);
                uint4 raw[2] = {*reinterpret_cast<const uint4 *>(kt + off), *reinterpret_cast<const uint4 *>(vt + off)};
                const float4 *rt = reinterpret_cast<const float4 *>(p.rot + ((size_t)h * p.rot_T + t_in + t) * (SG_D / 2) + cp * 4);
                const float4 r01 = rt[0], r23 = rt[1];
                const float cs[4] = {r01.x, r01.z, r23.x, r23.z}, sn[4] = {r01.y, r01.w, r23.y, r23.w};
                const float w = ws[t], g = gs[t];
                uint4 hi, lo, vo;
#pragma unroll
                for (int which = 0; which < 2; ++which) {
                    const __nv_bfloat162 *b2 = reinterpret_cast<const __nv_bfloat162 *>(&raw[which]);
                    float x[8], ss = 0.f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(b2[i]);
                        x[2 * i] = f.x; x[2 * i + 1] = f.y;
                        ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
                    }
                    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                    ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                    ss += __shfl_xor_sync(0xffffffffu, ss, 4);
                    const float inv = rsqrtf(fmaxf(ss, 1e-24f)) * (which == 0 ? g : 1.f);
                    __nv_bfloat162 o2[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        o2[i] = which == 0 ? __floats2bfloat162_rn((x[2 * i] * cs[i] - x[2 * i + 1] * sn[i]) * inv, (x[2 * i] * sn[i] + x[2 * i + 1] * cs[i]) * inv)
                                           : __floats2bfloat162_rn(x[2 * i] * inv, x[2 * i + 1] * inv);
                    if (which == 0) {                                 // K w from the ROUNDED k, as the prefill kernel forms it
                        float kw[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(o2[i]); kw[2 * i] = f.x * w; kw[2 * i + 1] = f.y * w; }
                        split8(kw, hi, lo);
                    } else vo = *reinterpret_cast<const uint4 *>(o2);
                }
                *reinterpret_cast<uint4 *>(kt + off) = hi;
                *reinterpret_cast<uint4 *>(lt + off) = lo;
                *reinterpret_cast<uint4 *>(vt + off) = vo;
            }
        }
        fence_proxy_async();
        ok = __syncthreads_and(ok);
        if (!ok) break;
        if (warp == 0) {
            constexpr uint32_t I_U = idesc_bf16(64, 64, 1, 1);
            const uint32_t sb = base + st * SM::STAGE;
            const uint64_t dh = smem_desc(sb, 8192, 1024), dv = smem_desc(sb + SM::TILE, 8192, 1024), dl = smem_desc(sb + 2 * SM::TILE, 8192, 1024);
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem, dh + k * 128, dv + k * 128, I_U, (c > 0) | (k > 0));
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem, dl + k * 128, dv + k * 128, I_U, 1);
            if constexpr (FINE)
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_bf16_elect(tmem, dl + (SM::TILE >> 4) + k * 128, dv + k * 128, I_U, 1);
            mma_commit_elect(done(st));
            if (c + 1 == NC) mma_commit_elect(bar_end);
            if (c + 2 < NC) {                                         // into the stage of chunk c - 1, whose product is an iteration old
                if (c > 0 && !mbar_wait_warp(done((c - 1) % SG_ST), ((c - 1) / SG_ST) & 1, 12)) ok = false;
                if (ok && lane == 0) load(c + 2);
            }
        }
    }
    if (ok) ok = mbar_wait_warp(bar_end, 0, 13);
    tc_fence_after();
    if (ok) {
        const int fr = lane >> 2, fq = lane & 3;
        float x[16];
        tmem_ld_frag4(tmem + ((uint32_t)(32 * sub) << 16) + 32 * wg, x);
        tmem_ld_wait();
#pragma unroll
        for (int hi8 = 0; hi8 < 2; ++hi8) {
            float *dst = p.U + ((size_t)blockIdx.x * SG_D + 16 * sub + fr + 8 * hi8) * SG_D + 32 * wg + 2 * fq;
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<float2 *>(dst + 8 * j) = make_float2(x[4 * j + 2 * hi8], x[4 * j + 2 * hi8 + 1]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 64);
}

// A thread owns COLS value columns of a pair of key rows; AHEAD segments' additions are requested ahead of the recurrence, the first ones also ahead of the factors,
// which the CTA forms side by side. Up to four segments: two columns a thread, four CTAs of 256 a chain; more: one column, 16 CTAs of 128, sixteen segments ahead. The whole
// call, us, the first form at any number / the second behind its factors / these: 44 chains of 2048 tokens (training) 34.5 / 35.9 / 33.9, 36 of 1333 22.7 / 23.1 / 22.3,
// 12 of 8192 35.3 / 33.1 / 32.9, 2 of 4096 18.1 / 14.3 / 14.3, 1 of 8192 22.9 / 16.5 / 16.2.
constexpr int SC_SEGS = 128, SC_FEW = 4;
template <int COLS, int AHEAD, int NT>
__global__ void __launch_bounds__(NT) segment_combine_kernel(float *__restrict__ E, const float *__restrict__ Lend, const float *__restrict__ S0,
                                                             const float *__restrict__ theta, const float *__restrict__ shift_dev, int n, int BH, int H,
                                                             float shift_host, bool windows, SegCut seg) {
    __shared__ float2 fac[SC_SEGS];                                   // e^{L}; not zero: the segment begins a window
    auto get = [](float (&v)[COLS], const float *p) {
        if constexpr (COLS == 2) { const float2 t = *reinterpret_cast<const float2 *>(p); v[0] = t.x; v[1] = t.y; }
        else v[0] = *p;
    };
    auto put = [](float *p, const float (&v)[COLS]) {
        if constexpr (COLS == 2) *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
        else *p = v[0];
    };
    pdl_wait();
    const int e = blockIdx.x * NT + threadIdx.x, bh = blockIdx.y, i = e / (SG_D / COLS), j = COLS * (e % (SG_D / COLS));
    const size_t step = (size_t)BH * SG_D * SG_D;
    float *at = E + ((size_t)bh * SG_D + 2 * i) * SG_D + j;
    float a[COLS], b[COLS], ua[AHEAD][COLS], ub[AHEAD][COLS];         // rows 2i, 2i + 1
    auto request = [&](const float *from, int m) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (k < m) { get(ua[k], from + k * step); get(ub[k], from + k * step + SG_D); }
    };
    request(at, n);
#pragma unroll
    for (int c = 0; c < COLS; ++c) a[c] = b[c] = 0.f;
    if (S0 != nullptr) {
        const float *src = S0 + ((size_t)bh * SG_D + 2 * i) * SG_D + j;
        get(a, src); get(b, src + SG_D);
    }
    float sn = 0.f, cs = 1.f;
    const float shift = theta == nullptr ? 0.f : (shift_dev != nullptr ? *shift_dev : shift_host);
    if (shift != 0.f) sincosf(-shift * theta[(size_t)(bh % H) * (SG_D / 2) + i], &sn, &cs);
    auto rotate = [&]() {
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const float ra = a[c] * cs - b[c] * sn;
            b[c] = a[c] * sn + b[c] * cs; a[c] = ra;
        }
    };
    if (!windows) rotate();
    for (int s0 = 0; s0 < n; s0 += SC_SEGS) {
        if (s0 > 0) __syncthreads();
        if (threadIdx.x < SC_SEGS && s0 + threadIdx.x < n) {
            int begin, in_piece, tokens;
            seg.at(s0 + threadIdx.x, begin, in_piece, tokens);
            fac[threadIdx.x] = make_float2(expf(Lend[(size_t)(s0 + threadIdx.x) * BH + bh]), in_piece == 0 ? 1.f : 0.f);
        }
        __syncthreads();
        const int m = min(n - s0, SC_SEGS);
        for (int w0 = 0; w0 < m; w0 += AHEAD) {
            float *here = at + (size_t)(s0 + w0) * step;
            if (s0 + w0 > 0) request(here, m - w0);
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
                if (w0 + k < m) {
                    const float2 f = fac[w0 + k];
                    // the state enters a window rotated back by the previous one's length, the sequence's own (S0) too
                    if (windows && f.y != 0.f) rotate();
#pragma unroll
                    for (int c = 0; c < COLS; ++c) { a[c] = fmaf(f.x, a[c], ua[k][c]); b[c] = fmaf(f.x, b[c], ub[k][c]); }
                    put(here + k * step, a); put(here + k * step + SG_D, b);
                }
        }
    }
}

size_t segment_scratch_bytes(int B, int H, int T, const SegCut &seg) {
    const size_t n = (size_t)seg.count(T) - 1;
    return n * B * H * (SG_D * SG_D + 1) * sizeof(float);
}

// Which prepared chains of T tokens are cut, and into how long segments. Where all chains leave SMs idle, all of them: a chunk costs its walk
// 1.3 us and the state pass 0.9, the two launches before the walk about 7 (train of 44 chains of 32 chunks: 45 us whole). Where they fill the
// SMs more than once, those of the last round, as whole rows of the batch, so that the round is as short as the SMs can make it instead of a whole
// chain long (9 us more for the launches and the round's ragged start; at 4 us more 200 chains of 64 chunks and 640 of 24 were taken and lost 0 to 2 %).
// Whole and cut, us: 64 x 12 chains of 64 chunks 477 and 451, 64 x 7 315 and 268, 25 x 12 of 63 232 and 188, 13 x 12 of 128 303 and 197, 16 x 12 of 32 84 and 79.
SegPlan segment_plan(int B, int H, int T) {
    const int NC = (T + TC_C - 1) / TC_C, sms = sm_count();
    const long long BH = (long long)B * H;
    if (NC < 16) return {0, 0};
    SegPlan best{0, 0};
    int rows = B;
    double cost = 1.3 * NC, extra = 7.0;                              // of the part that could be cut
    if (BH > sms) {
        const long long rounds = (BH + sms - 1) / sms;
        const long long rest = BH - (rounds - 1) * sms;              // chains of the last round
        rows = (int)((rest + H - 1) / H);
        extra = 16.0;
    }
    const long long chains = (long long)rows * H;
    if (rows > B || chains * 2 > sms) return best;
    for (int n = 2; n * chains <= sms; ++n) {
        const int len = (NC + n - 1) / n;
        if (len < 2) break;
        if (len * TC_C <= SG_MAX_PREPARED && len * 2.2 + extra < cost) { cost = len * 2.2 + extra; best = {rows, len * TC_C}; }
    }
    return best;
}

// How the windows of a sequence are dealt to the SMs, one segment a CTA and an SM. Whole windows come in rounds of equal length, so a last round that is
// not full costs as much as a full one: its windows are cut into parts that just fill the chip, their entering states a few more segments of the same
// pass. A segment costs its chunks and about one and a half to fill the pipeline. B1 H12 T8192, 192 windows of eight chunks on 148 SMs:
// 144 whole and 48 in thirds; the walk 47 -> 38 us a layer, the states 20 -> 18, their combination 9 -> 7, the whole pass 2254 -> 2164.
SegCut windows_cut(int B, int H, int T, int window) {
    SegCut best;
    best.win = window;
    const int sms = sm_count(), wl = window / TC_C, NW = (T + window - 1) / window;
    const long long BH = (long long)B * H;
    if (NW < 2 || BH * NW > 0x7fffffffLL) return best;
    const double fill = 1.5;
    double cost = (double)((BH * NW + sms - 1) / sms) * (wl + fill) - 1.0;
    for (long long r = 0; r * sms < BH * NW; ++r) {
        const int whole = (int)(r * sms / BH);
        if (whole >= NW) break;
        for (int len = 1; len < wl; ++len) {
            const long long parts = (wl + len - 1) / len;
            if ((NW - whole) * parts * BH > sms) continue;
            const double c = r * (wl + fill) + len + fill;
            if (c < cost) { cost = c; best.whole = whole; best.len = len * TC_C; }
            break;                                                    // the shortest parts that fit
        }
    }
    return best;
}

// the states entering segments 1, 2, ... of the prefill `a` (head dim 64, a.seg set) into scratch
int segment_states_launch(const PrefillArgs &a, float *scratch, cudaStream_t stream) {
    const int BH = a.B * a.H, nseg = a.seg.count(a.T);
    CUtensorMap mk, mv;
    const bool made = a.raw ? tc_make_map(&mk, a.k, a.B, a.T, (long long)a.H * SG_D, a.raw_st, a.raw_sb) && tc_make_map(&mv, a.v, a.B, a.T, (long long)a.H * SG_D, a.raw_st, a.raw_sb)
                            : tc_make_map(&mk, a.k, BH, a.T, SG_D, SG_D, (long long)a.T * SG_D) && tc_make_map(&mv, a.v, BH, a.T, SG_D, SG_D, (long long)a.T * SG_D);
    if (!made) { set_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled"); return PGB_ERR_CUDA; }
    float *Lend = scratch + (size_t)(nseg - 1) * BH * SG_D * SG_D;
    SgParams p{(const __nv_bfloat16 *)a.la_raw, (const __nv_bfloat16 *)a.gate_raw, a.la_sb, a.la_st, a.decay_A, (const float2 *)a.rot, a.rot_T, a.la, a.T,
               scratch, Lend, BH, a.H, a.seg};
    auto go = [&](auto kern, int smem) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        return e != cudaSuccess ? e : pdl_launch(kern, dim3((unsigned)(BH * (nseg - 1))), dim3(SG_NT), (size_t)smem, stream, mk, mv, p);
    };
    cudaError_t e = a.raw    ? go(segment_state_kernel<true, false>, SgSmem<true, false>::bytes)
                    : a.fine ? go(segment_state_kernel<false, true>, SgSmem<false, true>::bytes)
                             : go(segment_state_kernel<false, false>, SgSmem<false, false>::bytes);
    auto combine = [&](auto kern, int cols, int threads) {
        return pdl_launch(kern, dim3((unsigned)(SG_D * SG_D / 2 / cols / threads), (unsigned)BH), dim3((unsigned)threads), (size_t)0, stream, scratch,
                          (const float *)Lend, a.S0, a.theta, a.shift_dev, nseg - 1, BH, a.H, a.shift_host, (bool)a.seg_rotates, a.seg);
    };
    if (e == cudaSuccess)
        e = nseg - 1 <= SC_FEW ? combine(segment_combine_kernel<2, 4, 256>, 2, 256) : combine(segment_combine_kernel<1, 16, 128>, 1, 128);
    if (e != cudaSuccess) { set_cuda_error(e, "segment_state launch"); return PGB_ERR_CUDA; }
    return check_launch("segment_state_kernel");
}

int tc_segment_error_flag(int *out) { return tc_read_error_flag(out); }

}  // namespace pgb
