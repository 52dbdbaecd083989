// The delta rule's walk over 64-token chunks on the tensor cores, forward and backward, with everything transposed so that
// what is sequential never leaves tensor memory and registers.
//
// One CTA walks one (sequence, head). Forward, per chunk (X = (I + N)^-1 comes from delta_inv_kernel):
//     KS  = K S_c                rhs = beta (V - e^L KS)         W = X rhs           S_{c+1} = e^{L_C} S_c + K^T (w W)
//     o   = (P . dec) W + e^L Q S_c,   P = Q K^T
// Backward, the chunks in reverse with G = dLoss/dS_{c+1} in place of the state (dW0 = A^T do and D_c = (Q e^L)^T do are
// formed chunk-parallel beforehand):
//     KG  = K G                  dW  = dW0 + w KG                dR = X^T dW         G <- e^{L_C} G + D_c + K^T (-beta e^L dR)
// Both are the same chain of three products, so one kernel does both.
//
// Value columns are the M side of every product (lane = value column), tokens or keys the N side: S^T, rhs^T, W^T and
// (w W)^T are A operands read from TENSOR MEMORY, where the thread that owns the lane writes them as bf16 head and tail, and
// the B operands -- K, Q, X and the score matrix -- are the tiles as TMA delivers them (K serves K-major for K S and
// MN-major for the state update). A link of the chain is then: accumulator -> registers -> a few FMAs -> tensor memory; no
// shared-memory round trip, no proxy fence, no CTA barrier. The row scale w goes on W instead of K, which leaves K exact and
// drops one of the three head/tail products of the state update.
//
// Roles: 8 math warps (2 per 32-lane quarter, each half of the columns) run the chain; 4 score warps form the decayed scores
// (the only operand that goes through shared memory); 4 output warps scale Q S by e^L where it lies, so that A W accumulates
// onto it, and store o; one warp issues the MMAs in chain order; one loads tiles and prepares the decay statistics ahead.
// They meet only at mbarriers, every wait bounded.
//
// What bounds it: the latency of the chain. At D = 128 the products of a chunk are 2.6 k cycles of tensor pipe, of which
// 1.4 k (KS, W, U) are on the chain; at D = 64 the upper 64 lanes idle (an M = 64 product takes as long as an M = 128 one).
// Instruction fetch came next: with the state in registers and every loop unrolled the warps spent a third of their time
// waiting for instructions (five roles share the caches), so the state lives in tensor memory, where the update accumulates
// onto it, and every phase is a rolled loop over blocks of columns.
#pragma once
#include "tc_common.cuh"

namespace pgb {

constexpr int DW_MATH = 8, DW_OUT = 4, DW_SCORE = 4;
constexpr int DW_LOADER = DW_MATH + DW_OUT + DW_SCORE;
constexpr int DW_ISSUER = DW_LOADER + 2;                              // on a scheduler that has no math warps at D = 64 (warp % 4 = 2)
constexpr int DW_NT = (DW_ISSUER + 1) * 32;                           // 608 threads
constexpr float DW_LOG2E = 1.4426950408889634f;

struct DwParams {
    const float *la, *beta, *S0, *theta, *shift_dev;                  // S0: entering state (forward) or gradient on the final state
    float shift_host;
    float *S_out;                                                     // final state, or gradient on the entering one
    const float *dW0, *Dc;                                            // backward inputs
    int H, T, o_is_f32, want_sent, want_w, rebase_chunks;                               // rebase_chunks > 0: the state is rotated by -shift theta every so many chunks
    float rebase_shift;
    int BH, seg_chunks;                                               // WITH_MAP: chains, chunks of a segment; S_out and S_map are [segment][BH][D][D]
    float *S_map;
};

// tensor maps: tiles in, and what a warp stores 32 value columns at a time (a lane owns a column; its rows are staged in
// shared memory and leave in one bulk store -- stored directly, two bytes a lane, they took twice as long as the chain)
struct DwMaps {
    CUtensorMap q, k, v, x;                                           // in
    CUtensorMap o, sent, w;                                           // forward out: o; [BH*NC][D][D] bf16; [BH][T][D] bf16
    CUtensorMap g, dr;                                                // backward out, head and tail: [BH*NC*2][D][D], [2*BH][T][D] bf16
};

template <int D, bool BWD>
struct DwSmem {
    static constexpr int QK = TC_C * D * 2, SQ = TC_C * TC_C * 2;
    static constexpr int o_k = 0, o_x = QK, o_q = o_x + 2 * SQ, o_v = o_q + QK;       // K, X head, X tail, then (forward) Q, V
    // Backward, dW0 and (at D = 64) D_c of the chunk, fp32, come with its tiles. Loaded by the math warps where they are used, a round trip to
    // the L2 or two of every chunk were on the chain: B4 H11 T2048 D64 132 -> 93 us, B4 H8 T2048 D128 210 -> 177. At D = 128 D_c does not fit
    // beside them: its loads run a block of keys ahead.
    static constexpr bool FETCH_DC = BWD && D == 64;
    static constexpr int o_dw0 = o_q, o_dc = o_dw0 + TC_C * D * 4;
    static constexpr int STAGE = FETCH_DC ? o_dc + D * D * 4 : BWD ? o_dc : o_v + QK;
    static constexpr int NST = D == 128 ? 2 : 3;
    static constexpr int off_a = NST * STAGE;                         // decayed scores, two slots of head and tail (forward)
    static constexpr int off_out = off_a + (BWD ? 0 : 4 * SQ);        // staging of the stores, a slot per warp: math, then output
    static constexpr int MSLOT = (D / 2 > 32 ? D / 2 : 32) * 64, TSLOT = BWD ? 0 : 4096;
    static constexpr int off_rot = off_out + (BWD ? 2 : 1) * DW_MATH * MSLOT + DW_OUT * TSLOT;       // (cos, sin) of the rebase, D/2 pairs
    static constexpr int off_misc = off_rot + 512;
    static constexpr int bytes = off_misc + 5120 + 256 + 1024;
    static constexpr int b_full = 0, b_empty = 32, b_s = 64, b_ks = 72, b_r = 80, b_w = 88, b_ww = 96, b_u = 104, b_p = 112, b_a = 120,
                         b_qs = 128, b_qread = 136, b_oread = 152, b_stats = 160, b_done = 192, tmem_slot = 224, b_w2 = 232, stats = 256;
};

// 16 fp32 in registers -> 8 + 8 packed bf16 pairs (heads, tails) at columns hi / lo of this thread's lane
__device__ __forceinline__ void dw_put16(uint32_t hi, uint32_t lo, const float *x) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split2(x[2 * i], x[2 * i + 1], h[i], l[i]);
    tmem_st8(hi, h);
    tmem_st8(lo, l);
}
// the stores of a warp: rows of 32 columns (a lane each) staged in shared memory, then one bulk store by lane 0
struct DwStore {
    uint8_t *slot; uint32_t addr; int lane;
    __device__ __forceinline__ void begin() const {
        if (lane == 0) tma_store_source_free();
        __syncwarp();
    }
    __device__ __forceinline__ void put(int row, __nv_bfloat16 x) const { *reinterpret_cast<__nv_bfloat16 *>(slot + row * 64 + lane * 2) = x; }
    __device__ __forceinline__ void put(int row, float x) const { *reinterpret_cast<float *>(slot + row * 128 + lane * 4) = x; }
    __device__ __forceinline__ void end(const CUtensorMap *map, int c0, int c1, int c2) const {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) tma_store_3d(map, addr, c0, c1, c2);
    }
};

// WITH_MAP (forward, head dim 64): a CTA walks one SEGMENT of a chain, entered with S0 by the first segment and with zero by the others, and in the 64 lanes that
// the value columns leave idle (a product of 128 rows takes as long as one of 64) the segment's linear map of the state: the same walk with V = 0 and the
// identity as the entering state. Its outputs q_t^T (map to t) go to m.w, the map to the segment's end to S_map; what S adds to the outputs and to
// the state behind the segment is then a product each (delta_segments.cu), and the segments of a chain need not wait for one another.
template <int D, bool BWD, bool WITH_MAP = false>
__global__ void __launch_bounds__(DW_NT, 1) delta_walk_kernel(const __grid_constant__ DwMaps m, DwParams p) {
    using SM = DwSmem<D, BWD>;
    static_assert(!WITH_MAP || (D == 64 && !BWD), "the map lies in the lanes that head dim 64 leaves idle");
    constexpr int SUB = D / 64, NMATH = WITH_MAP ? DW_MATH : 2 * (D / 32), KH = D / 2;     // math warps with live lanes; keys a math thread owns
    constexpr uint32_t TM_S = 0, TM_SH = D, TM_SL = TM_SH + D / 2;    // S^T in fp32; its heads and tails
    constexpr uint32_t TM_WWH = TM_SH, TM_WWL = TM_SH + 32;           // (w W)^T reuses their columns: consumed by then
    constexpr uint32_t TM_KS = 2 * D, TM_QS = TM_KS + 64, TM_RH = TM_QS + 64, TM_RL = TM_RH + 32, TM_P = TM_RL + 32, TM_COLS = 512;
    constexpr uint32_t I_N64 = idesc_bf16(128, 64, 0, 0), I_N64T = idesc_bf16(128, 64, 0, 1), I_U = idesc_bf16(128, D, 0, 1),
                       I_P = idesc_bf16(64, 64, 0, 0);

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - smem_u32(smem_raw));
    uint8_t *misc = sm + SM::off_misc;
    const uint32_t mb = base + SM::off_misc;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + SM::tmem_slot);
    float *stats = reinterpret_cast<float *>(misc + SM::stats);       // [4 chunks][L, e^L, w, beta, -beta e^L][64]
    float2 *rot = reinterpret_cast<float2 *>(sm + SM::off_rot);
    auto full = [&](int s) { return mb + SM::b_full + 8 * s; };
    auto empty = [&](int s) { return mb + SM::b_empty + 8 * s; };
    auto bst = [&](int s) { return mb + SM::b_stats + 8 * s; };
    auto bdone = [&](int s) { return mb + SM::b_done + 8 * s; };

    // warp index and tensor-memory base through a shuffle: values the compiler then knows to be uniform over the warp, so the
    // MMA's operands stay in uniform registers (an MMA issued every 34 cycles instead of every 110)
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5), sub = warp & 3;
    const int seg = WITH_MAP ? blockIdx.x / p.BH : 0, bh = WITH_MAP ? blockIdx.x - seg * p.BH : blockIdx.x, h = bh % p.H;
    const int T = p.T, NCT = (T + TC_C - 1) / TC_C, c_first = WITH_MAP ? seg * p.seg_chunks : 0, NC = WITH_MAP ? min(p.seg_chunks, NCT - c_first) : NCT;
    auto chunk = [&](int i) { return BWD ? NC - 1 - i : c_first + i; };

    if (tid == 0) {
        for (int s = 0; s < 4; ++s) {
            mbar_init(full(s), 1); mbar_init(empty(s), 1); mbar_init(bst(s), 1);
            mbar_init(bdone(s), BWD ? NMATH : DW_OUT);
        }
        const int single[] = {SM::b_ks, SM::b_w, SM::b_u, SM::b_p, SM::b_qs};
        for (int b : single) mbar_init(mb + b, 1);
        mbar_init(mb + SM::b_s, NMATH); mbar_init(mb + SM::b_r, NMATH); mbar_init(mb + SM::b_ww, NMATH);
        mbar_init(mb + SM::b_w2, NMATH);
        mbar_init(mb + SM::b_a, DW_SCORE); mbar_init(mb + SM::b_qread, DW_OUT); mbar_init(mb + SM::b_oread, DW_OUT);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == DW_ISSUER) tmem_alloc(smem_u32(tmem_slot), TM_COLS);
    pdl_wait();                                                       // launched as a programmatic dependent: the set-up above overlaps the kernel ahead
    if (!BWD && p.rebase_chunks > 0 && tid < D / 2) {
        float sn, cs;
        sincosf(-p.rebase_shift * p.theta[(size_t)h * (D / 2) + tid], &sn, &cs);
        rot[tid] = make_float2(cs, sn);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    pdl_launch_dependents();                                          // not before the tensor memory is this CTA's: a dependent must not take it first. (The forward walk is launched plainly: under the inverse's tail it cost 8 us of 590.)

    if (warp < DW_MATH) {
        // ====================================================================================================== math
        if (WITH_MAP || sub * 32 < D) {
            const bool map = WITH_MAP && sub >= 2;                    // this warp's lanes hold the map's columns
            const int v = 32 * (WITH_MAP ? sub & 1 : sub) + lane, g = warp >> 2;      // value column; which half of the tokens / keys
            const int k0 = g * KH;
            const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16);
            const size_t sbase = (size_t)bh * D * D + (size_t)k0 * D + v;
            auto told = [&](uint32_t bar) {                           // this warp's columns are written
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar);
            };
            {
                const float shift = (BWD || map || seg > 0 || p.S0 == nullptr || p.theta == nullptr) ? 0.f : (p.shift_dev != nullptr ? *p.shift_dev : p.shift_host);
#pragma unroll 1
                for (int b = 0; b < KH; b += 16) {
                    float x[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) x[k] = map ? (k0 + b + k == v ? 1.f : 0.f) : p.S0 != nullptr && seg == 0 ? p.S0[sbase + (size_t)(b + k) * D] : 0.f;
                    if (shift != 0.f) {
#pragma unroll
                        for (int k = 0; k < 16; k += 2) {
                            float sn, cs;
                            sincosf(-shift * p.theta[(size_t)h * (D / 2) + ((k0 + b + k) >> 1)], &sn, &cs);
                            const float a = x[k], c = x[k + 1];
                            x[k] = a * cs - c * sn; x[k + 1] = a * sn + c * cs;
                        }
                    }
                    tmem_st16(lb + TM_S + k0 + b, reinterpret_cast<const uint32_t (&)[16]>(x));
                }
                tmem_st_wait();
            }
            const DwStore out{sm + SM::off_out + warp * SM::MSLOT, base + SM::off_out + warp * SM::MSLOT, lane};
            const DwStore out2{out.slot + DW_MATH * SM::MSLOT, out.addr + DW_MATH * SM::MSLOT, lane};
            bool ok = true;
            for (int i = 0; i < NC; ++i) {
                const int c = chunk(i), st = i % SM::NST, t0 = c * TC_C;
                const float *Ls = stats + (i & 3) * 320, *wts = Ls + 128, *bes = wts + 64, *bws = bes + 64;
                // ---- 1. the state as the A operand (the columns' last reader, the previous chunk's state update, is through)
                if (!BWD && p.rebase_chunks > 0 && c > 0 && c % p.rebase_chunks == 0) {
#pragma unroll 1
                    for (int b = 0; b < KH; b += 16) {
                        float x[16];
                        tmem_ld16_nowait(lb + TM_S + k0 + b, x);
                        tmem_ld_wait();
#pragma unroll
                        for (int k = 0; k < 16; k += 2) {
                            const float2 r = rot[(k0 + b + k) >> 1];
                            const float y = x[k], z = x[k + 1];
                            x[k] = y * r.x - z * r.y; x[k + 1] = y * r.y + z * r.x;
                        }
                        tmem_st16(lb + TM_S + k0 + b, reinterpret_cast<const uint32_t (&)[16]>(x));
                    }
                    tmem_st_wait();
                }
#pragma unroll 1
                for (int b = 0; b < KH; b += 32) {
                    float x[32];
                    tmem_ld32_nowait(lb + TM_S + k0 + b, x);
                    tmem_ld_wait();
                    dw_put16(lb + TM_SH + (k0 + b) / 2, lb + TM_SL + (k0 + b) / 2, &x[0]);
                    dw_put16(lb + TM_SH + (k0 + b) / 2 + 8, lb + TM_SL + (k0 + b) / 2 + 8, &x[16]);
                }
                told(mb + SM::b_s);
                if (!(ok = mbar_wait_warp(bst(i & 3), (i >> 2) & 1, 11))) break;
                // ---- 2. right-hand side. What does not wait for the chain is at hand before: beta V (forward), A^T do (backward)
                const uint8_t *vt = sm + st * SM::STAGE + SM::o_v + (v >> 6) * 8192 + (v & 7) * 2;
                const int vj = (v & 63) >> 3;
                float d0[32];
                float d[BWD ? 16 : 1];                                // D_c, a block of keys
                const float *dc = !BWD ? nullptr : SM::FETCH_DC ? reinterpret_cast<const float *>(sm + st * SM::STAGE + SM::o_dc) + k0 * D + v
                                                                : p.Dc + (((size_t)bh * NC + c) * D + k0) * D + v;
                if constexpr (BWD) {
                    if constexpr (!SM::FETCH_DC) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) d[k] = dc[k * D];
                    }
                    if (!(ok = mbar_wait_warp(full(st), (i / SM::NST) & 1, 12))) break;
                    const float *dw = reinterpret_cast<const float *>(sm + st * SM::STAGE + SM::o_dw0) + 32 * g * D + v;
#pragma unroll
                    for (int j = 0; j < 32; ++j) d0[j] = t0 + 32 * g + j < T ? dw[j * D] : 0.f;
                } else {
                    if (!(ok = mbar_wait_warp(full(st), (i / SM::NST) & 1, 12))) break;
#pragma unroll
                    for (int j = 0; j < 32; ++j) d0[j] = map ? 0.f : __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t *>(vt + swz(32 * g + j, vj)) << 16);
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 bb = *reinterpret_cast<const float4 *>(bes + 32 * g + j);
                        d0[j] *= bb.x; d0[j + 1] *= bb.y; d0[j + 2] *= bb.z; d0[j + 3] *= bb.w;
                    }
                }
                const float *rs = (BWD ? wts : bws) + 32 * g;         // factor of the state's product: w, or -beta e^L
                if (!(ok = mbar_wait_warp(mb + SM::b_ks, i & 1, 13))) break;
                tc_fence_after();
#pragma unroll
                for (int b = 0; b < 32; b += 16) {
                    float x[16];
                    tmem_ld16_nowait(lb + TM_KS + 32 * g + b, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        const float4 f = *reinterpret_cast<const float4 *>(rs + b + j);
                        x[j] = fmaf(f.x, x[j], d0[b + j]); x[j + 1] = fmaf(f.y, x[j + 1], d0[b + j + 1]);
                        x[j + 2] = fmaf(f.z, x[j + 2], d0[b + j + 2]); x[j + 3] = fmaf(f.w, x[j + 3], d0[b + j + 3]);
                    }
                    dw_put16(lb + TM_RH + 16 * g + b / 2, lb + TM_RL + 16 * g + b / 2, x);
                }
                told(mb + SM::b_r);
                // ---- while W is formed: the decay of the state for the accumulating update, and what is stored of it
                const float aC = expf(Ls[TC_C - 1]);
                const bool keep = BWD || p.want_sent;
                if (keep) out.begin();
#pragma unroll 1
                for (int b = 0; b < KH; b += 16) {
                    float x[16], dn[BWD ? 16 : 1];
                    if constexpr (SM::FETCH_DC) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) d[k] = dc[(b + k) * D];
                    } else if constexpr (BWD) {
                        const int nb = b + 16 < KH ? b + 16 : b;
#pragma unroll
                        for (int k = 0; k < 16; ++k) dn[k] = dc[(nb + k) * D];
                    }
                    tmem_ld16_nowait(lb + TM_S + k0 + b, x);
                    tmem_ld_wait();
                    if (keep) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            __nv_bfloat16 hi, lo;
                            split_bf16(x[k], hi, lo);
                            out.put(b + k, hi);
                            if constexpr (BWD) out2.put(b + k, lo);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 16; ++k) { if constexpr (BWD) x[k] = fmaf(aC, x[k], d[k]); else x[k] *= aC; }
                    tmem_st16(lb + TM_S + k0 + b, reinterpret_cast<const uint32_t (&)[16]>(x));
                    if constexpr (BWD && !SM::FETCH_DC) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) d[k] = dn[k];
                    }
                }
                if (BWD) {
                    out.end(&m.g, 32 * sub, k0, (bh * NCT + c) * 2);
                    out2.end(&m.g, 32 * sub, k0, (bh * NCT + c) * 2 + 1);
                } else if (keep) out.end(&m.sent, 32 * sub, k0, bh * NCT + c);
                // ---- 3. W (or dR), scaled, as the operand of the state update; then W itself, which only O1 waits for
                if (!(ok = mbar_wait_warp(mb + SM::b_w, i & 1, 14))) break;
                tc_fence_after();
#pragma unroll 1
                for (int b = 0; b < 32; b += 16) {
                    float x[16];
                    tmem_ld16_nowait(lb + TM_KS + 32 * g + b, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        const int t = 32 * g + b + j;
                        const float4 f = *reinterpret_cast<const float4 *>((BWD ? bws : wts) + t);
                        x[j] *= f.x; x[j + 1] *= f.y; x[j + 2] *= f.z; x[j + 3] *= f.w;
                    }
                    dw_put16(lb + TM_WWH + 16 * g + b / 2, lb + TM_WWL + 16 * g + b / 2, x);
                }
                told(mb + SM::b_ww);
                const bool keep_w = BWD || p.want_w;
                if (keep_w) out.begin();
#pragma unroll 1
                for (int b = 0; b < 32; b += 16) {
                    float x[16];
                    tmem_ld16_nowait(lb + TM_KS + 32 * g + b, x);
                    tmem_ld_wait();
                    if constexpr (!BWD) dw_put16(lb + TM_RH + 16 * g + b / 2, lb + TM_RL + 16 * g + b / 2, x);
                    if (keep_w) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            __nv_bfloat16 hi, lo;
                            split_bf16(x[j], hi, lo);
                            out.put(b + j, hi);
                            if constexpr (BWD) out2.put(b + j, lo);
                        }
                    }
                }
                if constexpr (!BWD) told(mb + SM::b_w2);
                if (BWD) {
                    out.end(&m.dr, 32 * sub, t0 + 32 * g, bh);
                    out2.end(&m.dr, 32 * sub, t0 + 32 * g, bh + (int)gridDim.x);
                } else if (keep_w) out.end(&m.w, 32 * sub, t0 + 32 * g, bh);
                // ---- 4. the state leaving the chunk has been accumulated
                if (!(ok = mbar_wait_warp(mb + SM::b_u, i & 1, 15))) break;
                tc_fence_after();
                if constexpr (BWD) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bdone(i & 3));
                }
            }
            if (lane == 0) tma_store_done();
            if (ok && p.S_out != nullptr) {
#pragma unroll 1
                for (int b = 0; b < KH; b += 16) {
                    float x[16];
                    tmem_ld16_nowait(lb + TM_S + k0 + b, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int k = 0; k < 16; ++k) (map ? p.S_map : p.S_out)[(size_t)seg * (WITH_MAP ? p.BH : 0) * D * D + sbase + (size_t)(b + k) * D] = x[k];
                }
            }
        }
    } else if (warp < DW_MATH + DW_OUT) {
        // ====================================================================================================== output
        if constexpr (!BWD) {
            const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16);
            const bool mine = WITH_MAP ? sub < 2 || seg > 0 : 32 * sub < D;   // this warp's lanes hold value columns, or the map's where it is wanted
            const CUtensorMap *to = WITH_MAP && sub >= 2 ? &m.w : &m.o;
            const int col = 32 * (WITH_MAP ? sub & 1 : sub);
            const uint32_t slot = SM::off_out + DW_MATH * SM::MSLOT + sub * SM::TSLOT;
            const DwStore out{sm + slot, base + slot, lane};
            const DwStore half2{out.slot + 2048, out.addr + 2048, lane};
            for (int i = 0; i < NC; ++i) {
                const float *eLs = stats + (i & 3) * 320 + 64;
                if (!(mbar_wait_warp(bst(i & 3), (i >> 2) & 1, 31) && mbar_wait_warp(mb + SM::b_qs, i & 1, 33))) break;
                tc_fence_after();
                if (mine) {
#pragma unroll 1
                    for (int b = 0; b < 64; b += 16) {                // e^{L_t} Q S where it lies: O1 accumulates onto it
                        float x[16];
                        tmem_ld16_nowait(lb + TM_QS + b, x);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j += 4) {
                            const float4 e = *reinterpret_cast<const float4 *>(eLs + b + j);
                            x[j] *= e.x; x[j + 1] *= e.y; x[j + 2] *= e.z; x[j + 3] *= e.w;
                        }
                        tmem_st16(lb + TM_QS + b, reinterpret_cast<const uint32_t (&)[16]>(x));
                    }
                    tmem_st_wait();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(mb + SM::b_qread);
                if (!mbar_wait_warp(empty(i % SM::NST), (i / SM::NST) & 1, 34)) break;    // A W has accumulated
                tc_fence_after();
                float y[64];
                if (mine) {
                    tmem_ld32_nowait(lb + TM_QS, *reinterpret_cast<float (*)[32]>(&y[0]));
                    tmem_ld32_nowait(lb + TM_QS + 32, *reinterpret_cast<float (*)[32]>(&y[32]));
                    tmem_ld_wait();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(mb + SM::b_oread); mbar_arrive(bdone(i & 3)); }
                if (mine) {
                    out.begin();
                    if (p.o_is_f32) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) out.put(j, y[j]);
                        out.end(to, col, chunk(i) * TC_C, bh);
                        out.begin();
#pragma unroll
                        for (int j = 0; j < 32; ++j) out.put(j, y[32 + j]);
                        out.end(to, col, chunk(i) * TC_C + 32, bh);
                    } else {
#pragma unroll
                        for (int j = 0; j < 64; ++j) out.put(j, __float2bfloat16_rn(y[j]));
                        out.end(to, col, chunk(i) * TC_C, bh);
                        half2.end(to, col, chunk(i) * TC_C + 32, bh);
                    }
                }
            }
            if (lane == 0) tma_store_done();
        }
    } else if (warp < DW_LOADER) {
        // ====================================================================================================== scores
        if constexpr (!BWD) {
            const int fr = lane >> 2, fq = lane & 3, row0 = 16 * sub + fr, row1 = row0 + 8;
            const uint32_t lb = tmem + ((uint32_t)(32 * sub) << 16);
            for (int i = 0; i < NC; ++i) {
                const float *Ls = stats + (i & 3) * 320;
                uint8_t *ah = sm + SM::off_a + (i & 1) * 2 * SM::SQ, *al = ah + SM::SQ;
                // the slot's last reader, the A W product of chunk i - 2, is through (its output has been read)
                if (!(mbar_wait_warp(bst(i & 3), (i >> 2) & 1, 41) && mbar_wait_warp(mb + SM::b_p, i & 1, 42) &&
                      (i < 2 || mbar_wait_warp(bdone((i - 2) & 3), ((i - 2) >> 2) & 1, 43)))) break;
                tc_fence_after();
                const float Lt0 = Ls[row0] * DW_LOG2E, Lt1 = Ls[row1] * DW_LOG2E;
#pragma unroll 1
                for (int b = 0; b < 64; b += 16) {
                    float pv[8];
                    tmem_ld_frag2(lb + TM_P + b, pv);
                    const float2 L0 = *reinterpret_cast<const float2 *>(Ls + b + 2 * fq), L1 = *reinterpret_cast<const float2 *>(Ls + b + 8 + 2 * fq);
                    const float Lc[4] = {L0.x * DW_LOG2E, L0.y * DW_LOG2E, L1.x * DW_LOG2E, L1.y * DW_LOG2E};
                    tmem_ld_wait();
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int s = b + 8 * j + 2 * fq;
                        const float a00 = (s <= row0) ? pv[4 * j] * fast_exp2(fminf(Lt0 - Lc[2 * j], 0.f)) : 0.f;
                        const float a01 = (s + 1 <= row0) ? pv[4 * j + 1] * fast_exp2(fminf(Lt0 - Lc[2 * j + 1], 0.f)) : 0.f;
                        const float a10 = (s <= row1) ? pv[4 * j + 2] * fast_exp2(fminf(Lt1 - Lc[2 * j], 0.f)) : 0.f;
                        const float a11 = (s + 1 <= row1) ? pv[4 * j + 3] * fast_exp2(fminf(Lt1 - Lc[2 * j + 1], 0.f)) : 0.f;
                        split2(a00, a01, hi[2 * j], lo[2 * j]);
                        split2(a10, a11, hi[2 * j + 1], lo[2 * j + 1]);
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t o0 = swz(row0, (b >> 3) + j) + 4 * fq, o1 = swz(row1, (b >> 3) + j) + 4 * fq;
                        *reinterpret_cast<uint32_t *>(ah + o0) = hi[2 * j];     *reinterpret_cast<uint32_t *>(al + o0) = lo[2 * j];
                        *reinterpret_cast<uint32_t *>(ah + o1) = hi[2 * j + 1]; *reinterpret_cast<uint32_t *>(al + o1) = lo[2 * j + 1];
                    }
                }
                tc_fence_before();
                warp_arrive(mb + SM::b_a, lane);
            }
        }
    } else if (warp == DW_ISSUER) {
        // ====================================================================================================== issuer
        // the whole warp runs this, converged, and one elected lane issues: the descriptors then stay in uniform registers
        // (a lone thread under a branch issues an MMA only every 65-100 cycles, slower than the tensor pipe runs them)
        {
            auto score = [&](int i) {                                 // P = Q K^T of chunk i (its tiles have landed)
                const uint32_t sb = base + (i % SM::NST) * SM::STAGE;
                const uint64_t dq = smem_desc(sb + SM::o_q, 16, 1024), dk = smem_desc(sb + SM::o_k, 16, 1024);
#pragma unroll
                for (int k = 0; k < D / 16; ++k) {
                    const uint32_t ko = ((uint32_t)(k >> 2) * 8192u + (uint32_t)(k & 3) * 32u) >> 4;
                    mma_bf16_elect(tmem + TM_P, dq + ko, dk + ko, I_P, k > 0);
                }
                mma_commit_elect(mb + SM::b_p);
            };
            // (S^T) B^T with B the K or Q tile: heads, then tails of S^T
            auto state_product = [&](uint32_t acc, uint32_t tile) {
                const uint64_t db = smem_desc(tile, 16, 1024);
#pragma unroll
                for (int j = 0; j < 2 * SUB; ++j) {                   // half (heads, tails) x 64 keys
                    const uint32_t a = tmem + TM_SH + 32 * j;         // the tails lie behind the heads
                    const uint64_t d = db + (uint32_t)(j % SUB) * (8192u >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k) mma_bf16_ts_elect(tmem + acc, a + 8 * k, d + 2 * k, I_N64, (j > 0) | (k > 0));
                }
            };
            // (R^T)(M^T) over 64 tokens, head*head + head*tail + tail*head; step: descriptor advance per 16 tokens
            auto square_product = [&](uint32_t acc, uint64_t dh, uint64_t dl, uint32_t idesc, uint32_t step, uint32_t onto) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const uint32_t a = tmem + (j == 2 ? TM_RL : TM_RH);
                    const uint64_t d = j == 1 ? dl : dh;
#pragma unroll
                    for (int k = 0; k < 4; ++k) mma_bf16_ts_elect(tmem + acc, a + 8 * k, d + k * step, idesc, onto | (j > 0) | (k > 0));
                }
            };
            auto outputs = [&](int i) {                               // A W of chunk i onto e^L Q S; then its tiles are free
                const uint32_t ab = base + SM::off_a + (i & 1) * 2 * SM::SQ;
                square_product(TM_QS, smem_desc(ab, 16, 1024), smem_desc(ab + SM::SQ, 16, 1024), I_N64, 2, 1);
                mma_commit_elect(empty(i % SM::NST));
            };
            // Order: whatever the chain waits for goes out on an idle pipe; the rest fills the pipe while the math warps convert
            // (Q S behind K S, the next chunk's scores behind W, A W behind the state update).
            bool ok = mbar_wait_warp(full(0), 0, 51);
            if (!BWD && ok) score(0);
            for (int i = 0; i < NC && ok; ++i) {
                const int st = i % SM::NST;
                const uint32_t sb = base + st * SM::STAGE;
                if (!(ok = mbar_wait_warp(mb + SM::b_s, i & 1, 52))) break;
                if (BWD && !(ok = mbar_wait_warp(full(st), (i / SM::NST) & 1, 58))) break;
                tc_fence_after();
                state_product(TM_KS, sb + SM::o_k);
                mma_commit_elect(mb + SM::b_ks);
                if constexpr (!BWD) {
                    if (i > 0 && !(ok = mbar_wait_warp(mb + SM::b_oread, (i - 1) & 1, 53))) break;
                    tc_fence_after();
                    state_product(TM_QS, sb + SM::o_q);
                    mma_commit_elect(mb + SM::b_qs);
                }
                if (!(ok = mbar_wait_warp(mb + SM::b_r, i & 1, 54))) break;
                tc_fence_after();
                // forward: W = X rhs, so N = rows of X, K-major;  backward: dR = X^T dW, N = columns of X, MN-major
                square_product(TM_KS, smem_desc(sb + SM::o_x, BWD ? 8192 : 16, 1024), smem_desc(sb + SM::o_x + SM::SQ, BWD ? 8192 : 16, 1024),
                               BWD ? I_N64T : I_N64, BWD ? 128 : 2, 0);
                mma_commit_elect(mb + SM::b_w);
                if (!BWD && i + 1 < NC) {
                    if (!(ok = mbar_wait_warp(full((i + 1) % SM::NST), ((i + 1) / SM::NST) & 1, 60) && mbar_wait_warp(mb + SM::b_a, i & 1, 55))) break;
                    tc_fence_after();
                    score(i + 1);
                }
                if (!(ok = mbar_wait_warp(mb + SM::b_ww, i & 1, 55))) break;
                tc_fence_after();
                const uint64_t dk = smem_desc(sb + SM::o_k, 8192, 1024);
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mma_bf16_ts_elect(tmem + TM_S, tmem + (half ? TM_WWL : TM_WWH) + 8 * k, dk + k * 128, I_U, 1);
                mma_commit_elect(mb + SM::b_u);
                if constexpr (BWD) mma_commit_elect(empty(st));
                else {
                    if (i + 1 == NC && !(ok = mbar_wait_warp(mb + SM::b_a, i & 1, 56))) break;
                    if (!(ok = mbar_wait_warp(mb + SM::b_w2, i & 1, 59) && mbar_wait_warp(mb + SM::b_qread, i & 1, 57))) break;
                    tc_fence_after();
                    outputs(i);
                }
            }
        }
    } else if (warp == DW_LOADER) {
        // ====================================================================================================== loader, statistics
        const float *la = p.la + (size_t)bh * T, *beta = p.beta + (size_t)bh * T;
        auto fetch = [&](const float *src, int t) { return t < T ? src[t] : 0.f; };
        float a_lo = fetch(la, chunk(0) * TC_C + lane), a_hi = fetch(la, chunk(0) * TC_C + lane + 32);
        float b_lo = fetch(beta, chunk(0) * TC_C + lane), b_hi = fetch(beta, chunk(0) * TC_C + lane + 32);
        for (int i = 0; i < NC; ++i) {
            const int c = chunk(i), t0 = c * TC_C, st = i % SM::NST;
            if (i >= SM::NST && !mbar_wait_warp(empty(st), ((i / SM::NST) + 1) & 1, 61)) break;
            if (lane == 0) {
                const uint32_t sb = base + st * SM::STAGE, bar = full(st);
                const uint32_t dw0 = BWD ? (uint32_t)(T - t0 < TC_C ? T - t0 : TC_C) * D * 4 : 0, dcb = SM::FETCH_DC ? D * D * 4 : 0;
                mbar_expect_tx(bar, BWD ? SM::o_dw0 + dw0 + dcb : SM::STAGE);
                if constexpr (BWD) bulk_load_1d(sb + SM::o_dw0, p.dW0 + ((size_t)bh * T + t0) * D, dw0, bar);
                if constexpr (SM::FETCH_DC) bulk_load_1d(sb + SM::o_dc, p.Dc + ((size_t)bh * NC + c) * D * D, dcb, bar);
#pragma unroll
                for (int s = 0; s < SUB; ++s) tma_load_3d(sb + SM::o_k + s * 8192, &m.k, bar, 64 * s, t0, bh);
                tma_load_3d(sb + SM::o_x, &m.x, bar, 0, 0, (bh * NCT + c) * 2);
                tma_load_3d(sb + SM::o_x + SM::SQ, &m.x, bar, 0, 0, (bh * NCT + c) * 2 + 1);
                if constexpr (!BWD) {
#pragma unroll
                    for (int s = 0; s < SUB; ++s) {
                        tma_load_3d(sb + SM::o_q + s * 8192, &m.q, bar, 64 * s, t0, bh);
                        tma_load_3d(sb + SM::o_v + s * 8192, &m.v, bar, 64 * s, t0, bh);
                    }
                }
            }
            if (i >= 4 && !mbar_wait_warp(bdone(i & 3), ((i >> 2) + 1) & 1, 62)) break;
            float *Ls = stats + (i & 3) * 320, *eLs = Ls + 64, *wts = eLs + 64, *bes = wts + 64, *bws = bes + 64;
            float sl = a_lo, sh = a_hi;
            const float bl = b_lo, bh2 = b_hi;
            bes[lane] = bl; bes[lane + 32] = bh2;
            if (i + 1 < NC) {
                const int n0 = chunk(i + 1) * TC_C;
                a_lo = fetch(la, n0 + lane); a_hi = fetch(la, n0 + lane + 32);
                b_lo = fetch(beta, n0 + lane); b_hi = fetch(beta, n0 + lane + 32);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float nl = __shfl_up_sync(0xffffffffu, sl, o), nh = __shfl_up_sync(0xffffffffu, sh, o);
                if (lane >= o) { sl += nl; sh += nh; }
            }
            sh += __shfl_sync(0xffffffffu, sl, 31);
            const float tot = __shfl_sync(0xffffffffu, sh, 31);
            Ls[lane] = sl; Ls[lane + 32] = sh;
            const float el = expf(sl), eh = expf(sh);
            eLs[lane] = el; eLs[lane + 32] = eh;
            bws[lane] = -bl * el; bws[lane + 32] = -bh2 * eh;
            wts[lane] = t0 + lane < T ? expf(fminf(tot - sl, 0.f)) : 0.f;
            wts[lane + 32] = t0 + lane + 32 < T ? expf(fminf(tot - sh, 0.f)) : 0.f;
            __syncwarp();
            if (lane == 0) mbar_arrive(bst(i & 3));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == DW_ISSUER) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace pgb
