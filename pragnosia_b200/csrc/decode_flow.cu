// One decode step of the whole language model as ONE launch, for a few sequences (batch <= 4, bf16 weights, fp32 state), without
// barriers between its phases: every value that one CTA hands to another carries the mark of the launch it belongs to.
//
// The phases are those of decode_token.cu -- per layer projection, state step, output projection, MLP up, MLP down; the tied head
// at the end -- and so are the roundings, and the order of every sum but one kind's: rows of the output projection or the MLP's second layer
// that are few and long (the latter at K 3072, N 768) are shared across a CTA's eight warps, whose fp32 sums are added in warp order. A
// bf16 rounding may then fall the other way. There, a phase ends with a grid-wide barrier: the results are
// made visible (a release), counted (148 additions to one word), the count is seen (a round trip), and only then are the
// results fetched (another): 3.7 us a phase, 61 phases a token. Here an exchanged value is a 32-bit word, the bf16
// value in the low half and the launch's mark in the high half, written and read with relaxed accesses of that size or vectors of them. A consumer
// reads the words it wants, 16 bytes at a time, and reads those again whose mark is not this launch's: one round trip once the producer's
// store has landed, nothing to order, nothing to count. Every phase of every layer has words of its own, so within a launch nothing is
// written twice; the next launch has another mark, and a launch ends before the next begins.
//
// What is left on the way of a token is the latency of each phase: from a store to the load that finds it about a microsecond, the rows
// 0.4 us, the products and their sum over a warp 0.7 (stamped per phase at batch 1). Everything else is off it: the residual stream stays in each CTA's
// shared memory (every CTA forms the same sums), the state slice and the head's constants are requested a phase early, and
// weights do not stop at a phase's end: the CTA's runs of rows are one list over the whole token, three of 48 KB in flight at any time, one bulk
// copy each, so HBM is asked for the coming phases' weights while this one's values travel.
//
// d 768, 12 layers, vocabulary 8192, microseconds a token with barriers and without: batch 1 231 -> 172, batch 2 251 -> 190, batch 4 307 -> 216
// (28 us is what the weights' bytes take).
//
// Waits are bounded: a thread that gives up raises a word beside the launch counter that every other one looks at, the CTA's threads agree on
// it at their next barrier, and the kernel winds down; the last CTA takes the word back, so launches behind it, and those of other models,
// never see it. All CTAs are resident (a cooperative launch), and a phase only waits for earlier ones.
#include "decode_token.cuh"
#include "tc_common.cuh"

#include <stddef.h>

namespace pgb {

static __device__ int g_fl_error = 0;

struct FlArgs {
    const DtLayer *layers;
    const __nv_bfloat16 *E, *P, *fn_w, *fn_b;
    const long long *tok;
    long long *pos;
    float *shift;
    unsigned *words;                                                  // [L] x ([B][NP] y, [B][d] o, [B][d] d1, [B][d] d2, [B][dff] hmid)
    float *logits;
    unsigned long long *sync;                                         // [0] CTAs that have come to the head so far, over all launches; [1] not zero
                                                                      // while a launch winds down
    int L, B, d, H, NP, dff, V, ctx, fn_kind, window;
    float fn_eps;
};

__device__ __forceinline__ void fl_put(unsigned *at, float v, unsigned mark) {
    const unsigned w = (unsigned)__bfloat16_as_ushort(__float2bfloat16_rn(v)) | mark;
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(at), "r"(w) : "memory");
}
__device__ __forceinline__ uint4 fl_ld4(const unsigned *at) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(at) : "memory");
    return v;
}
__device__ __forceinline__ unsigned fl_ld1(const unsigned *at) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(at) : "memory");
    return v;
}
// what a wait is for, and what ends it
struct FlWait {
    unsigned mark;
    unsigned *given_up;                                               // sync[1]
    unsigned limit = DT_SPIN_LIMIT;
};
// the 64th look, 128th, ... at something: true: the wait ran out, here or at another thread of the launch (out of line: rarely called, and the
// kernel's code is fetched once a token)
__device__ __noinline__ bool fl_gone(unsigned spins, unsigned limit, unsigned *given_up) {
    if (spins < limit && *reinterpret_cast<volatile unsigned *>(given_up) == 0u) return false;
    atomicExch(given_up, 1u);
    atomicExch(&g_fl_error, 82);
    return true;
}
__device__ __forceinline__ bool fl_again(unsigned &spins, const FlWait &wt) {
    return (++spins & 63u) != 0u || !fl_gone(spins, wt.limit, wt.given_up);
}
// N vectors of four words each, those of `want` (a bit each): read until all of them carry the mark. A whole warp calls it. While
// something is missing one lane looks for the first of it: a line that the whole chip reads again and again takes microseconds to be
// written. Batch 1: all lanes on their own words 212 us a token where one lane a warp took 181; every CTA another word first 176 where
// all on the same took 172; eight words a load 187; a line of its own to wait on, written behind the values, 190: a round trip more.
template <int N>
__device__ __forceinline__ bool fl_take4(const unsigned *(&at)[N], unsigned want, const FlWait &wt, uint4 (&v)[N]) {
    const unsigned mark = wt.mark;
    constexpr unsigned FULL = 0xffffffffu;
    while (true) {
#pragma unroll
        for (int i = 0; i < N; ++i) if (want >> i & 1u) v[i] = fl_ld4(at[i]);
#pragma unroll
        for (int i = 0; i < N; ++i)
            if ((want >> i & 1u) && ((v[i].x ^ mark) | (v[i].y ^ mark) | (v[i].z ^ mark) | (v[i].w ^ mark)) < 0x10000u) want &= ~(1u << i);
        const unsigned missing = __ballot_sync(FULL, want != 0u);
        if (missing == 0u) return true;
        const int leader = __ffs(missing) - 1;
        int found = 1;
        if ((threadIdx.x & 31) == leader) {
            const unsigned *p = at[0];
#pragma unroll
            for (int i = N - 1; i > 0; --i) if (want >> i & 1u) p = at[i];
            if (want & 1u) p = at[0];
            unsigned spins = 0;
            while (found != 0 && (fl_ld1(p) ^ mark) >= 0x10000u) found = fl_again(spins, wt);
        }
        if (__shfl_sync(FULL, found, leader) == 0) return false;
    }
}
template <int N>
__device__ __forceinline__ bool fl_take1(const unsigned *(&at)[N], const FlWait &wt, float (&x)[N]) {
    unsigned spins = 0, v[N];
    while (true) {
        unsigned off = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = fl_ld1(at[i]);
#pragma unroll
        for (int i = 0; i < N; ++i) { off |= v[i] ^ wt.mark; x[i] = __uint_as_float(v[i] << 16); }
        if (off < 0x10000u) return true;
        if (!fl_again(spins, wt)) return false;
    }
}
// the values of four words as two pairs of bf16
__device__ __forceinline__ uint2 fl_pairs(const uint4 &v) { return make_uint2(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410)); }

// the state step's projection and read as marked words (decode_step.cuh)
template <int D>
struct FlRows {
    const unsigned *y;                                                // the sequence's row
    unsigned *o;                                                      // the head's words
    int d, H, h;
    const FlWait &wt;
    bool &lost, &alive;
    __device__ __forceinline__ bool between() const { return true; }
    __device__ __forceinline__ void vec(int which, int lane, float (&x)[D / 32]) const {
        const unsigned *at[D / 32];
#pragma unroll
        for (int i = 0; i < D / 32; ++i) at[i] = y + which * d + h * D + lane + 32 * i;
        if (!fl_take1(at, wt, x)) lost = true;
    }
    __device__ __forceinline__ void scalars(float &dec, float &g) const {
        const unsigned *at[2] = {y + 3 * d + h, y + 3 * d + H + h};
        float x[2];
        if (!fl_take1(at, wt, x)) lost = true;
        dec = x[0]; g = x[1];
    }
    __device__ __forceinline__ bool sync() const { alive = __syncthreads_or(lost) == 0; return alive; }
    __device__ __forceinline__ void put(int j, float v) const { fl_put(o + j, v, wt.mark); }
};

// rows of z in shared memory as they were exchanged; false: the wait ran out (the same for the whole CTA)
__device__ __forceinline__ bool fl_rows(const unsigned *src, int n, const FlWait &wt, uint4 *zs, bool lost) {
    for (int base = 0; base < n / 4 && !lost; base += 4 * DT_THREADS) {
        const unsigned *at[4];
        unsigned want = 0;
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            at[i] = src + 4 * (base + i * DT_THREADS + threadIdx.x);
            if (base + i * DT_THREADS + threadIdx.x < n / 4) want |= 1u << i;
        }
        lost = !fl_take4(at, want, wt, v);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (want >> i & 1u) reinterpret_cast<uint2 *>(zs)[base + i * DT_THREADS + threadIdx.x] = fl_pairs(v[i]);
    }
    return __syncthreads_or(lost) == 0;
}

struct FlNorm { int kind; float eps; const __nv_bfloat16 *w, *b; };

// The residual stream xs += what src holds (first: xs = E[tok] + P[pos]), rounded, and z = norm(xs); warps are dealt to the rows as in
// decode_token.cu and every sum is formed in its order. A thread only meets its own pieces of xs.
__device__ __forceinline__ bool fl_norm_rows(const FlArgs &a, const unsigned *src, const FlNorm &nm, const FlWait &wt, uint4 *xs, uint4 *zs,
                                             float (*part)[DT_WARPS], bool lost) {
    const int K = a.d, K8 = K >> 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wpr = a.B == 1 ? DT_WARPS : (a.B == 2 ? DT_WARPS / 2 : DT_WARPS / 4);
    const int b = warp / wpr, li = (warp % wpr) * 32 + lane, stride = wpr * 32;
    const bool live = b < a.B;
    uint4 pnw[2], pnb[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        pnw[i] = pnb[i] = make_uint4(0u, 0u, 0u, 0u);
        if (live && li + stride * i < K8) {
            pnw[i] = reinterpret_cast<const uint4 *>(nm.w)[li + stride * i];
            if (nm.kind == 2) pnb[i] = reinterpret_cast<const uint4 *>(nm.b)[li + stride * i];
        }
    }
    const uint4 *er = nullptr, *pr = nullptr;
    if (src == nullptr && live) {
        long long t = a.tok[b], p = a.pos[0];
        t = t < 0 ? 0 : (t >= a.V ? a.V - 1 : t);                     // ids outside the table are clamped, never dereferenced
        p = p < 0 ? 0 : (p >= a.ctx ? a.ctx - 1 : p);
        er = reinterpret_cast<const uint4 *>(a.E + (size_t)t * K);
        pr = reinterpret_cast<const uint4 *>(a.P + (size_t)p * K);
    }
    float s1 = 0.f, s2 = 0.f;
    auto add = [&](int k8, const uint4 &xr, const uint4 &dr) {
        float t[8], dd[8];
        dt_unpack8(xr, t);
        dt_unpack8(dr, dd);
#pragma unroll
        for (int j = 0; j < 8; ++j) { t[j] = dt_round(t[j] + dd[j]); s1 += t[j]; s2 = fmaf(t[j], t[j], s2); }
        xs[b * K8 + k8] = dt_pack8(t);
    };
    if (live)
        for (int base = li - lane; base < K8 && !lost; base += 2 * stride) {          // a whole warp together
            const int k0 = base + lane, k1 = k0 + stride;
            if (src == nullptr) {
                if (k0 < K8) add(k0, er[k0], pr[k0]);
                if (k1 < K8) add(k1, er[k1], pr[k1]);
            } else {
                const unsigned *r0 = src + (size_t)b * K + 8 * k0, *r1 = r0 + 8 * stride;
                const unsigned *at[4] = {r0, r0 + 4, r1, r1 + 4};
                uint4 v[4];
                lost = !fl_take4(at, (k0 < K8 ? 3u : 0u) | (k1 < K8 ? 12u : 0u), wt, v);
                if (k0 < K8) {
                    const uint2 lo = fl_pairs(v[0]), hi = fl_pairs(v[1]);
                    add(k0, xs[b * K8 + k0], make_uint4(lo.x, lo.y, hi.x, hi.y));
                }
                if (k1 < K8) {
                    const uint2 lo = fl_pairs(v[2]), hi = fl_pairs(v[3]);
                    add(k1, xs[b * K8 + k1], make_uint4(lo.x, lo.y, hi.x, hi.y));
                }
            }
        }
    // a row's sum: its warps' partials, added in warp order by every thread of the row
    auto row_sum = [&](float x, int slot) {
        x = warp_sum(x);
        if (lane == 0) part[slot][warp] = x;
        __syncthreads();
        float tot = 0.f;
        for (int w = 0; w < wpr; ++w) tot += part[slot][(live ? b : 0) * wpr + w];
        return tot;
    };
    float mean = 0.f, rstd;
    if (nm.kind == 1) {
        rstd = rsqrtf(row_sum(s2, 0) / (float)K + nm.eps);
    } else {
        mean = row_sum(s1, 0) / (float)K;
        float sv = 0.f;
        if (live)
            for (int k8 = li; k8 < K8; k8 += stride) {
                float t[8];
                dt_unpack8(xs[b * K8 + k8], t);
#pragma unroll
                for (int j = 0; j < 8; ++j) { const float c = t[j] - mean; sv = fmaf(c, c, sv); }
            }
        rstd = rsqrtf(row_sum(sv, 1) / (float)K + nm.eps);
    }
    if (live) {
        int i = 0;
        for (int k8 = li; k8 < K8; k8 += stride, ++i) {
            const uint4 wraw = i == 0 ? pnw[0] : (i == 1 ? pnw[1] : reinterpret_cast<const uint4 *>(nm.w)[k8]);
            float t[8], w[8], o[8];
            dt_unpack8(xs[b * K8 + k8], t);
            dt_unpack8(wraw, w);
            if (nm.kind == 2) {
                float bb[8];
                dt_unpack8(i == 0 ? pnb[0] : (i == 1 ? pnb[1] : reinterpret_cast<const uint4 *>(nm.b)[k8]), bb);
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = (t[j] - mean) * rstd * w[j] + bb[j];
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = t[j] * rstd * w[j];
            }
            zs[b * K8 + k8] = dt_pack8(o);
        }
    }
    return __syncthreads_or(lost) == 0;
}

// The five kinds of linear phase: projection, output projection, MLP up, MLP down, head. Output rows are dealt to the CTAs in runs
// of `run` consecutive ones, run after run round the grid; a run's weights are one contiguous piece of the matrix and come as one bulk copy.
//   R > 0  each warp takes R rows of the run (run = 8 R; R at most four, and about what gives every warp of the grid one set of rows)
//   R = 0  few long rows: every warp takes an eighth of K of all rows of the run, so a piece of z meets all of them, and all CTAs have work
struct FlKind { int N, K8, R, run, W, bias; };                        // W, bias: offsets of the pointers in the layer's record (bias < 0: none)
constexpr int FL_STAGE_U4 = DT_WARPS * DT_PIECES * 32;                // weights of a run at most, in pieces of 16 bytes: 48 KB
constexpr int FL_ACROSS = 6;                                          // rows of a run shared across the warps

// The CTA's place in its list of runs, (phase, round), over the whole token. Thread 0 requests up to three ahead of their use, whatever
// phase they belong to; run i of the list lies in stage i mod 3. A stage is free at the CTA's first barrier after its use.
struct FlQueue {
    int ip, base, rq;                                                 // next run to request: phase, first row; its stage
    int open, used, freed;                                            // runs requested and not used; used since the last barrier; free stages
    int buf; unsigned parity;                                         // the run used next: its stage; the stages' parities, a bit each
    uint32_t stage, bars;                                             // shared-memory addresses of the stages and their barriers
};

__device__ __forceinline__ void fl_request(const FlArgs &a, const DtLayer *layers, const FlKind *kinds, FlQueue &q) {
    const int last = 4 * a.L;
    const FlKind *kp = &kinds[q.ip == last ? 4 : q.ip & 3];
    while (q.ip <= last && q.base >= kp->N) {
        ++q.ip;
        kp = &kinds[q.ip == last ? 4 : q.ip & 3];
        q.base = blockIdx.x * kp->run;
    }
    if (q.ip > last) return;
    const char *ly = reinterpret_cast<const char *>(layers + (q.ip >> 2));           // behind the last layer's record: the head's
    const char *W = *reinterpret_cast<const char *const *>(ly + kp->W);
    const uint32_t bar = q.bars + 8 * q.rq, bytes = (uint32_t)(min(kp->run, kp->N - q.base) * kp->K8) * 16u;
    mbar_expect_tx(bar, bytes);
    bulk_load_1d(q.stage + q.rq * (FL_STAGE_U4 * 16), W + (size_t)q.base * kp->K8 * 16, bytes, bar);
    if (kp->bias >= 0) {                                              // into the L2: a token's weights have pushed it out
        const __nv_bfloat16 *bias = *reinterpret_cast<const __nv_bfloat16 *const *>(ly + kp->bias);
        if (bias != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(bias + q.base));
    }
    q.base += gridDim.x * kp->run;
    q.rq = q.rq + 1 == DT_DEPTH ? 0 : q.rq + 1;
    ++q.open;
}

__device__ __forceinline__ unsigned fl_bias(const __nv_bfloat16 *at, bool want) {
    unsigned raw = 0;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.global.u16 %0, [%1];\n\t}" : "+r"(raw) : "l"(at), "r"((unsigned)want));
    return raw;
}
// the bias (raw) of the output that this thread finishes in the run that begins at row n0
template <int NB>
__device__ __forceinline__ unsigned fl_my_bias(const FlKind &k, const __nv_bfloat16 *bias, int n0) {
    const int tid = threadIdx.x, mine = k.R == 0 ? tid : tid & 31, row = (k.R == 0 ? 0 : (tid >> 5) * k.R) + mine / NB;
    return fl_bias(bias + n0 + row, bias != nullptr && mine < (k.R == 0 ? k.run : k.R) * NB && n0 + row < k.N);
}

// A run's products: out[b][n] = act(sum_k W[n][k] z[b][k] + bias[n]), as marked words, or as fp32 (the logits). NB: rows of z
// the instantiation multiplies (>= the batch; the surplus is computed on whatever shared memory holds and never written).
template <int R, int NB, bool HEAD>
__device__ __forceinline__ void fl_products(const FlArgs &a, const FlKind &k, int n0, unsigned bias_raw, bool gelu, unsigned *out, unsigned mark,
                                            const uint4 *zs, const uint4 *stage) {
    constexpr int AT_ONCE = R + NB <= 2 ? 3 : (R + NB <= 4 ? 2 : 1);  // pieces of K read ahead of their products
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = n0 + warp * R, cnt = (k.K8 - lane + 31) >> 5;
    if (r0 >= k.N) return;
    float acc[R][NB];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[r][b] = 0.f;
    const uint4 *wp = stage + warp * R * k.K8 + lane, *zp = zs + lane;
#pragma unroll 1
    for (int u = 0; u < cnt; u += AT_ONCE) {
        uint4 w[AT_ONCE][R], z[AT_ONCE][NB];
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j)
            if (j == 0 || u + j < cnt) {
#pragma unroll
                for (int r = 0; r < R; ++r) w[j][r] = wp[r * k.K8 + (u + j) * 32];
#pragma unroll
                for (int b = 0; b < NB; ++b) z[j][b] = zp[b * k.K8 + (u + j) * 32];
            }
#pragma unroll
        for (int j = 0; j < AT_ONCE; ++j)
            if (j == 0 || u + j < cnt) {
                float wf[R][8];
#pragma unroll
                for (int r = 0; r < R; ++r) dt_unpack8(w[j][r], wf[r]);
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    float zf[8];
                    dt_unpack8(z[j][b], zf);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int r = 0; r < R; ++r) acc[r][b] = fmaf(wf[r][i], zf[i], acc[r][b]);
                }
            }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[r][b] = warp_sum(acc[r][b]);
    // lane (r * NB + b) finishes and writes output (b, r0 + r): pick the value with selects, finish it once
    float mine = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b)
            if (lane == r * NB + b) mine = acc[r][b];
    const int r_ = lane / NB, b_ = lane % NB;
    if (lane < R * NB && b_ < a.B && r0 + r_ < k.N) {
        float v = dt_round(mine + __uint_as_float(bias_raw << 16));   // the linear layer's bf16 output
        if (gelu) v = 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
        if constexpr (HEAD) a.logits[(size_t)b_ * k.N + r0 + r_] = v;
        else fl_put(out + (size_t)b_ * k.N + r0 + r_, v, mark);
    }
}

// The same with the run's rows shared across the warps, whose sums meet in `red` and are added in warp order.
template <int NB>
__device__ __forceinline__ void fl_across(const FlArgs &a, const FlKind &k, int n0, unsigned bias_raw, unsigned *out, unsigned mark, const uint4 *zs,
                                          const uint4 *stage, float (*red)[FL_ACROSS * NB]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rows = min(k.run, k.N - n0);
    const int k1 = (warp + 1) * k.K8 / DT_WARPS;
    float acc[FL_ACROSS][NB];
#pragma unroll
    for (int r = 0; r < FL_ACROSS; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[r][b] = 0.f;
#pragma unroll 1
    for (int u = warp * k.K8 / DT_WARPS + lane; u < k1; u += 32) {
        uint4 w[FL_ACROSS], z[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) z[b] = zs[b * k.K8 + u];
#pragma unroll
        for (int r = 0; r < FL_ACROSS; ++r) w[r] = stage[min(r, rows - 1) * k.K8 + u];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            float zf[8];
            dt_unpack8(z[b], zf);
#pragma unroll
            for (int r = 0; r < FL_ACROSS; ++r) {
                float wf[8];
                dt_unpack8(w[r], wf);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[r][b] = fmaf(wf[i], zf[i], acc[r][b]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < FL_ACROSS; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[r][b] = warp_sum(acc[r][b]);
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < FL_ACROSS; ++r)
#pragma unroll
            for (int b = 0; b < NB; ++b) red[warp][r * NB + b] = acc[r][b];
    }
    __syncthreads();
    if (tid < rows * NB && tid % NB < a.B) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < DT_WARPS; ++w) v += red[w][tid];
        fl_put(out + (size_t)(tid % NB) * k.N + n0 + tid / NB, dt_round(v + __uint_as_float(bias_raw << 16)), mark);
    }
}

template <int D, bool DELTA, int NB>
__global__ void __launch_bounds__(DT_THREADS, 1) decode_flow_kernel(FlArgs a) {
    extern __shared__ uint4 fl_smem[];                                // weight staging, the phases' rows in turn, the residual stream, the layer table
    const int d8 = a.d >> 3, z8 = (a.dff > a.d ? a.dff : a.d) >> 3;
    uint4 *zeven = fl_smem + DT_DEPTH * FL_STAGE_U4, *zodd = zeven + NB * d8, *xs = zodd + NB * z8;
    DtLayer *layers = reinterpret_cast<DtLayer *>(xs + NB * d8);
    __shared__ float part[2][2][DT_WARPS];
    __shared__ FlKind kinds[5];
    __shared__ float red[DT_WARPS][FL_ACROSS * NB];
    __shared__ unsigned s_mark;
    __shared__ __align__(8) unsigned long long bars[DT_DEPTH];
    const int tid = threadIdx.x;
    {
        const uint2 *src = reinterpret_cast<const uint2 *>(a.layers);
        uint2 *dst = reinterpret_cast<uint2 *>(layers);
        for (int i = tid; i < a.L * (int)(sizeof(DtLayer) / 8); i += DT_THREADS) dst[i] = src[i];
        if (tid == 96) layers[a.L].Wc = a.E;                          // the head's weights, where a layer's would be
    }
    if (tid < 5) {
        const int grid = gridDim.x, N = tid == 0 ? a.NP : (tid == 2 ? a.dff : (tid == 4 ? a.V : a.d)), K8 = tid == 3 ? a.dff >> 3 : d8;
        const int at[5] = {(int)offsetof(DtLayer, Wc), (int)offsetof(DtLayer, ow), (int)offsetof(DtLayer, a_w), (int)offsetof(DtLayer, b_w), (int)offsetof(DtLayer, Wc)};
        const int bias[5] = {(int)offsetof(DtLayer, bc), -1, (int)offsetof(DtLayer, a_b), (int)offsetof(DtLayer, b_b), -1};
        const int want = (N + grid * DT_WARPS - 1) / (grid * DT_WARPS), most = (N + grid - 1) / grid;
        int R = min(min(want, 4), FL_STAGE_U4 / (DT_WARPS * K8));     // 0: not even a row a warp fits a stage
        // rows shared across the warps (a layer's phases without activation): where a warp a row would leave CTAs idle and K is long enough for it
        if ((tid == 1 || tid == 3) && (R == 0 || (N < grid * DT_WARPS && K8 >= 32 * DT_WARPS))) R = 0;
        kinds[tid] = FlKind{N, K8, R, R > 0 ? DT_WARPS * R : min(min(most, FL_ACROSS), FL_STAGE_U4 / K8), at[tid], bias[tid]};
    } else if (tid == 64) {
        for (int i = 0; i < DT_DEPTH; ++i) mbar_init(smem_u32(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (tid == 32) {
        // the launch's number: a CTA adds itself below, so the count cannot complete the next multiple before this one has
        unsigned long long c;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(a.sync) : "memory");
        s_mark = ((unsigned)((c / gridDim.x) % 65535u) + 1u) << 16;
    }
    __syncthreads();
    const unsigned mark = s_mark;
    const FlWait wt{mark, reinterpret_cast<unsigned *>(a.sync + 1)};
    FlQueue q{0, (int)blockIdx.x * kinds[0].run, 0, 0, 0, 0, 0, 0u, smem_u32(fl_smem), smem_u32(bars)};
    if (tid == 0)
#pragma unroll 1
        for (int i = 0; i < DT_DEPTH; ++i) fl_request(a, layers, kinds, q);

    const int per = a.B * (a.NP + 3 * a.d + a.dff);
    bool alive = true, lost = false;                                  // lost: this thread gave a wait up; the CTA agrees on it at its next barrier
    DecodeHeld<D> held;
#pragma unroll 1
    for (int p = 0; p < 4 * a.L && alive; ++p) {
        const int kd = p & 3;
        const DtLayer &ly = layers[p >> 2];
        unsigned *y = a.words + (size_t)(p >> 2) * per, *o = y + a.B * a.NP, *d1 = o + a.B * a.d, *d2 = d1 + a.B * a.d, *hm = d2 + a.B * a.d;
        uint4 *zs = kd & 1 ? zodd : zeven;
        unsigned *out;
        const __nv_bfloat16 *bias = kd == 0 ? ly.bc : (kd == 2 ? ly.a_b : (kd == 3 ? ly.b_b : nullptr));
        const FlKind k = kinds[kd];
        int n0 = blockIdx.x * k.run;
        const bool works = n0 < k.N;                                  // this CTA has rows of the phase
        unsigned bias_raw = fl_my_bias<NB>(k, bias, works ? n0 : k.N);   // arrives while the exchange is waited for
        const DecodeArgs da{nullptr, nullptr, nullptr, 0, 1, a.E, 0, 1, nullptr, 0, ly.A, ly.theta, a.shift, 0.f, ly.S, ly.S, ly.on_w, ly.on_eps,
                            nullptr, 0, a.B, a.H};
        if (kd & 1) {                                                 // the coming phase's norm: into the L2 (a token's weights have pushed it out)
            const DtLayer &ln = layers[min((p + 1) >> 2, a.L - 1)];
            const __nv_bfloat16 *w = kd == 1 ? ln.n_w : (p + 1 == 4 * a.L ? a.fn_w : ln.ln_w), *nb = kd == 1 ? ln.n_b : (p + 1 == 4 * a.L ? a.fn_b : ln.ln_b);
            for (int i = 64 * tid; i < a.d; i += 64 * DT_THREADS) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(w + i));
                if (nb != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(nb + i));
            }
        }
        if (kd == 0) {
            out = y;
            // the state of this CTA's (sequence, head) is on its way while the projection is formed (at head dim 128 it is 64 registers a thread: not held)
            if (D == 64 && blockIdx.x < a.B * a.H) held.request(da, blockIdx.x / a.H, blockIdx.x % a.H);
            alive = fl_norm_rows(a, p == 0 ? nullptr : d2 - per, FlNorm{ly.ln_kind, ly.ln_eps, ly.ln_w, ly.ln_b}, wt, xs, zs, part[0], lost);
        } else if (kd == 1) {
            // the recurrent state step, one (sequence, head) per CTA
            out = d1;
#pragma unroll 1
            for (int bh = blockIdx.x; bh < a.B * a.H && alive; bh += gridDim.x) {
                const int b = bh / a.H, h = bh % a.H;
                if (D != 64 || bh != blockIdx.x) held.request(da, b, h);
                held.constants();
                decode_step_body<D, DELTA>(da, b, h, held, FlRows<D>{y + (size_t)b * a.NP, o + (size_t)b * a.d + h * D, a.d, a.H, h, wt, lost, alive});
                __syncthreads();
            }
            if (alive && works) alive = fl_rows(o, a.B * a.d, wt, zs, lost);
        } else if (kd == 2) {
            out = hm;
            alive = fl_norm_rows(a, d1, FlNorm{ly.n_kind, ly.n_eps, ly.n_w, ly.n_b}, wt, xs, zs, part[1], lost);
        } else {
            out = d2;
            if (works) alive = fl_rows(hm, a.B * a.dff, wt, zs, lost);
        }
        if (alive) {
            if (works) { q.freed += q.used; q.used = 0; }             // the rows' barriers are behind every warp's last run
#pragma unroll 1
            while (n0 < k.N) {
                if (!mbar_wait_tries(q.bars + 8 * q.buf, q.parity >> q.buf & 1u)) lost = true;
                q.parity ^= 1u << q.buf;
                const uint4 *stage = fl_smem + q.buf * FL_STAGE_U4;
                if (k.R == 0) fl_across<NB>(a, k, n0, bias_raw, out, mark, zs, stage, red);
                else if (k.R == 1) fl_products<1, NB, false>(a, k, n0, bias_raw, kd == 2, out, mark, zs, stage);
                else if (k.R == 2) fl_products<2, NB, false>(a, k, n0, bias_raw, kd == 2, out, mark, zs, stage);
                else if (k.R == 3) fl_products<3, NB, false>(a, k, n0, bias_raw, kd == 2, out, mark, zs, stage);
                else fl_products<4, NB, false>(a, k, n0, bias_raw, kd == 2, out, mark, zs, stage);
                q.buf = q.buf + 1 == DT_DEPTH ? 0 : q.buf + 1;
                --q.open; ++q.used;
                n0 += gridDim.x * k.run;
                if (n0 < k.N) {                                       // another round
                    bias_raw = fl_my_bias<NB>(k, bias, n0);
                    __syncthreads();
                    q.freed += q.used; q.used = 0;
                }
                if (tid == 0)
                    for (; q.freed > 0; --q.freed) fl_request(a, layers, kinds, q);
                q.freed = 0;
            }
        }
    }
    // ---- final norm and the tied head
    if (alive) {
        const unsigned *d2 = a.words + (size_t)(a.L - 1) * per + a.B * (a.NP + 2 * a.d);
        alive = fl_norm_rows(a, d2, FlNorm{a.fn_kind, a.fn_eps, a.fn_w, a.fn_b}, wt, xs, zeven, part[0], lost);
    }
    if (tid == 0) {
        // this CTA has read the position and the shift for the last time, and waits for no more words; the last one to say so leaves them as
        // the next token needs them
        if (!alive) {                                                 // a wait for weights may have run out unseen by the other CTAs
            atomicExch(wt.given_up, 1u);
            __threadfence();
        }
        const unsigned long long c = atomicAdd(a.sync, 1ull) + 1ull;
        if (c % gridDim.x == 0ull) {
            if (alive && a.window > 0) {
                a.pos[0] = (a.pos[0] + 1) % a.window;
                a.shift[0] = 1.f;
            }
            __threadfence();
            atomicExch(wt.given_up, 0u);
        }
    }
    if (alive) {
        const FlKind k = kinds[4];
        q.freed += q.used; q.used = 0;
#pragma unroll 1
        for (int n0 = blockIdx.x * k.run; n0 < k.N; n0 += gridDim.x * k.run) {
            if (!mbar_wait_tries(q.bars + 8 * q.buf, q.parity >> q.buf & 1u)) lost = true;
            q.parity ^= 1u << q.buf;
            const uint4 *stage = fl_smem + q.buf * FL_STAGE_U4;
            if (k.R == 1) fl_products<1, NB, true>(a, k, n0, 0u, false, nullptr, mark, zeven, stage);
            else if (k.R == 2) fl_products<2, NB, true>(a, k, n0, 0u, false, nullptr, mark, zeven, stage);
            else if (k.R == 3) fl_products<3, NB, true>(a, k, n0, 0u, false, nullptr, mark, zeven, stage);
            else fl_products<4, NB, true>(a, k, n0, 0u, false, nullptr, mark, zeven, stage);
            q.buf = q.buf + 1 == DT_DEPTH ? 0 : q.buf + 1;
            --q.open;
            __syncthreads();                                          // every warp is through with the stage
            ++q.freed;
            if (tid == 0)
                for (; q.freed > 0; --q.freed) fl_request(a, layers, kinds, q);
            q.freed = 0;
        }
    }
    if (lost) atomicExch(&g_fl_error, 82);
    if (tid == 0)                                                     // nothing may land behind the block's end (a healthy launch has used all it asked for)
        for (; q.open > 0; --q.open) {
            mbar_wait_tries(q.bars + 8 * q.buf, q.parity >> q.buf & 1u);
            q.parity ^= 1u << q.buf;
            q.buf = q.buf + 1 == DT_DEPTH ? 0 : q.buf + 1;
        }
}

// The waits' failure path on its own: one CTA as the first launch of a pair. Its first warp looks for 128 words, `limit` times or up to 63 more;
// its second writes them `late` cycles from the start (late < 0: never), and the kernel returns normally either way.
__global__ void __launch_bounds__(64) decode_flow_wait_selftest_kernel(unsigned *words, unsigned long long *sync, unsigned limit, long long late) {
    const int lane = threadIdx.x & 31;
    const FlWait wt{1u << 16, reinterpret_cast<unsigned *>(sync + 1), limit};
    if (threadIdx.x < 32) {
        const unsigned *at[1] = {words + 4 * lane};
        uint4 v[1];
        fl_take4(at, 1u, wt, v);
    } else if (late >= 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < late) {}
        for (int i = 0; i < 4; ++i) fl_put(words + 4 * lane + i, (float)i, wt.mark);
    }
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(sync, 1ull);
}

int decode_flow_wait_selftest_launch(unsigned *words, unsigned long long *sync, unsigned limit, long long late, cudaStream_t stream) {
    decode_flow_wait_selftest_kernel<<<1, 64, 0, stream>>>(words, sync, limit, late);
    return check_launch("decode_flow_wait_selftest_kernel");
}

int decode_flow_error_flag(int *out) {
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(out, g_fl_error, sizeof(int));
    if (e == cudaSuccess && *out != 0) e = cudaMemcpyToSymbol(g_fl_error, &zero, sizeof(int));
    if (e != cudaSuccess) { set_cuda_error(e, "decode_flow error flag"); return PGB_ERR_CUDA; }
    return PGB_OK;
}

// dynamic shared memory at most, beside 7 KB of the kernel's own; also the function's limit at every call, whatever the call's model needs (other
// threads may be launching the same function for other models)
constexpr size_t FL_SMEM_MOST = 220 * 1024;

static size_t decode_flow_smem(int NB, int L, int d, int dff) {
    return (size_t)DT_DEPTH * FL_STAGE_U4 * sizeof(uint4) + (size_t)NB * (2 * (size_t)d + (dff > d ? dff : d)) * sizeof(__nv_bfloat16) + (size_t)(L + 1) * sizeof(DtLayer);
}
// bytes of marked words; 0: the shapes need more shared memory than a CTA has, or have rows of which not
// even one a warp (the MLP's second layer: one) fits a stage
size_t decode_flow_work_bytes(int L, int B, int d, int NP, int dff) {
    if (d / 8 > FL_STAGE_U4 / DT_WARPS || dff / 8 > FL_STAGE_U4 || decode_flow_smem(B <= 2 ? B : 4, L, d, dff) > FL_SMEM_MOST) return 0;
    return (size_t)L * B * ((size_t)NP + 3 * d + dff) * sizeof(unsigned);
}

template <int D, bool DELTA, int NB>
static int decode_flow_go(const FlArgs &a, cudaStream_t stream) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = decode_flow_smem(NB, a.L, a.d, a.dff);
    auto kern = decode_flow_kernel<D, DELTA, NB>;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FL_SMEM_MOST);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, DT_THREADS, smem);
    if (e != cudaSuccess || sms <= 0 || per_sm <= 0) {
        set_cuda_error(e == cudaSuccess ? cudaErrorLaunchOutOfResources : e, "decode_flow set-up");
        return PGB_ERR_CUDA;
    }
    FlArgs args = a;
    void *params[] = {&args};
    // cooperative: either every CTA is resident at once (the waits need it) or the launch fails
    e = cudaLaunchCooperativeKernel((const void *)kern, dim3((unsigned)sms), dim3(DT_THREADS), params, smem, stream);
    if (e != cudaSuccess) { set_cuda_error(e, "decode_flow launch"); return PGB_ERR_CUDA; }
    return check_launch("decode_flow_kernel");
}

template <int D, bool DELTA>
static int decode_flow_nb(const FlArgs &a, cudaStream_t stream) {
    if (a.B == 1) return decode_flow_go<D, DELTA, 1>(a, stream);
    if (a.B == 2) return decode_flow_go<D, DELTA, 2>(a, stream);
    return decode_flow_go<D, DELTA, 4>(a, stream);
}

int decode_flow_launch(const void *layers, int L, const void *E, const void *P, const void *fn_w, const void *fn_b, int fn_kind,
                       float fn_eps, const long long *tok, long long *pos, float *shift, void *work, float *logits,
                       unsigned long long *sync, int B, int d, int H, int D, int NP, int dff, int V, int ctx, int delta,
                       int window, cudaStream_t stream) {
    const FlArgs a{(const DtLayer *)layers, (const __nv_bfloat16 *)E, (const __nv_bfloat16 *)P, (const __nv_bfloat16 *)fn_w, (const __nv_bfloat16 *)fn_b,
                   tok, pos, shift, (unsigned *)work, logits, sync, L, B, d, H, NP, dff, V, ctx, fn_kind, window, fn_eps};
    if (D == 64) return delta ? decode_flow_nb<64, true>(a, stream) : decode_flow_nb<64, false>(a, stream);
    return delta ? decode_flow_nb<128, true>(a, stream) : decode_flow_nb<128, false>(a, stream);
}

}  // namespace pgb
