// Per-token complex recurrence h_t = lambda_t h_{t-1} + u_t as a chunked parallel scan, and its adjoint.
//
// Layout in HBM: u, logmag, y are [B][T][D] fp32 with D contiguous: 12 B read (8 B when the angle is one value per
// channel) and 4 B written per (b,t,d) element. What bounds it is the SM's arithmetic: a tile's loads fly under the arithmetic of the one
// before, and pairs of channels (e^x, sin, cos and the recurrence, scan_math.cuh: 68 instructions an element, 50 with one angle per channel) keep
// the FMA pipe two cycles each, so the time goes with the SM clock. B64 T4096 D768: 660 us at 1965 MHz (4.9 TB/s, 0.74 of a copy; the adjoint, nine
// streams, 5.2), 735 to 760 once the chip's power limit has taken the clock to 1610 - 1690 MHz, which some 50 ms of such calls do (one angle per
// channel 440 and 500). At the full clock, with loads ahead of their use but inside the tile 760, with the slots below 660 (one angle per
// channel 587 -> 447); B16 T4096 D768 253 -> 200 (199 -> 141).
//
// Work split. A lane owns VEC adjacent channels (4 where D, pointers and strides allow: one 128-bit access; else 2 or 1). A warp is TS time-segments x CQ
// channel groups (TS * CQ = 32): lanes of one segment read 16*CQ contiguous bytes of one time row, so every 128-byte
// line is used whole. A tile is TS*SEG consecutive time steps; per tile each lane
//   1. takes its SEG steps, requested two tiles ahead, and forms c_t = |l_t| cos, s_t = |l_t| sin,
//   2. folds them into the segment's affine map h -> A h + Bv (complex A, Bv), starting from (1, 0),
//   3. combines the maps of the segments before it with a shuffle scan over the TS segment lanes
//      ((A2,B2) o (A1,B1) = (A2 A1, A2 B1 + B2)), which gives the state entering its segment,
//   4. replays the recurrence over its SEG steps from that state in the reference's operation order
//      (src/scan_kernel.py:42-48) and stores Re h.
// The state leaving the tile is broadcast from the last segment lane. With TS = 1 the kernel is the literal sequential
// recurrence; with TS > 1 only the state at segment boundaries is reassociated (fp32 rounding, no other difference).
#include <math.h>

#include <type_traits>

#include "scan_math.cuh"

namespace pgb {

constexpr int LS_WARPS = 2;
// Where a lane owns four channels, its steps of the coming two tiles travel global -> shared memory by asynchronous copies into slots
// that only this lane reads, so no registers are held while they fly and nobody synchronises: a tile is read out of its slot,
// the slot is requested again, and the arithmetic of the tile runs under the copy. 16 warps an SM are enough then (a tile of loads ahead of
// its use needed 24, B64 T4096 D768 760 us against 660, one angle per channel 590 against 480; spills are poison next to this much shared
// memory, which leaves the L1 no room: 1010 us with 24 warps and 70 bytes spilled). Narrower lanes request the next tile into
// registers: a copy of 4 or 8 bytes costs an instruction more than it saves (B13 T1111 D510: 44 against 54 us).
// So does BRIEF, for walks of a few tiles, with two steps a lane and tile: what counts there is the way of a tile through a lane (1.3 us, of four
// steps through slots 1.9), and the slots' extra step through shared memory (one sequence of 64 tokens: 3.2 us against 3.8; of 700: 15.9 and 13.3).
template <int VEC, bool BRIEF = false> struct LsForm {
    static constexpr bool staged = VEC == 4 && !BRIEF;
    static constexpr int slots = staged ? 2 : 1, seg = BRIEF ? 2 : 4;
};
constexpr int LS_SEG = LsForm<4>::seg;                                // steps a lane takes of a tile
constexpr int LS_CTAS_PER_SM = 8;                                     // the same for the adjoint, whose slots make room for two warps more an SM

// VEC adjacent channels of one row as pairs (the last one half empty when VEC is 1)
template <int VEC> struct LsVec { static constexpr int NP = (VEC + 1) / 2; };
template <int VEC>
__device__ __forceinline__ void ls_ld(f2 (&d)[LsVec<VEC>::NP], const float *p) {
    if constexpr (VEC == 4) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(p);
        d[0] = t.x; d[1] = t.y;
    } else if constexpr (VEC == 2) d[0] = *reinterpret_cast<const f2 *>(p);
    else d[0] = f2_pack(*p, 0.f);
}
template <int VEC>
__device__ __forceinline__ void ls_st(float *p, const f2 (&d)[LsVec<VEC>::NP]) {
    if constexpr (VEC == 4) __stcs(reinterpret_cast<ulonglong2 *>(p), make_ulonglong2(d[0], d[1]));
    else if constexpr (VEC == 2) *reinterpret_cast<f2 *>(p) = d[0];
    else { float a, b; f2_unpack(d[0], a, b); *p = a; }
}
// one step's channels of this lane into its slot; false: zeros (nothing is read)
template <int VEC>
__device__ __forceinline__ void ls_cp(float *slot, const float *src, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(slot);
    const int n = live ? 4 * VEC : 0;
    if constexpr (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else if constexpr (VEC == 2) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void ls_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void ls_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }
// a complex pair product and sum: (ar + i ai)(br + i bi) + (cr + i ci)
__device__ __forceinline__ void ls_cfma(f2 &outr, f2 &outi, f2 ar, f2 ai, f2 br, f2 bi, f2 cr, f2 ci) {
    const f2 nai = f2_neg(ai);
    outr = f2_fma(ar, br, f2_fma(nai, bi, cr));
    outi = f2_fma(ai, br, f2_fma(ar, bi, ci));
}
// exclusive scan of the segments' affine maps over the TS segment lanes (lanes CQ apart): the map of everything before this one
template <int TS, int CQ>
__device__ __forceinline__ void ls_scan_maps(f2 &Ar, f2 &Ai, f2 &Br, f2 &Bi, int seg) {
    constexpr unsigned FULL = 0xffffffffu;
#pragma unroll
    for (int off = 1; off < TS; off <<= 1) {
        const f2 par = __shfl_up_sync(FULL, Ar, off * CQ), pai = __shfl_up_sync(FULL, Ai, off * CQ), pbr = __shfl_up_sync(FULL, Br, off * CQ),
                 pbi = __shfl_up_sync(FULL, Bi, off * CQ);
        if (seg >= off) {
            f2 nbr, nbi, nar, nai;
            ls_cfma(nbr, nbi, Ar, Ai, pbr, pbi, Br, Bi);
            ls_cfma(nar, nai, Ar, Ai, par, pai, 0ull, 0ull);
            Ar = nar; Ai = nai; Br = nbr; Bi = nbi;
        }
    }
    Ar = __shfl_up_sync(FULL, Ar, CQ); Ai = __shfl_up_sync(FULL, Ai, CQ); Br = __shfl_up_sync(FULL, Br, CQ); Bi = __shfl_up_sync(FULL, Bi, CQ);
    if (seg == 0) { Ar = f2_both(1.f); Ai = 0ull; Br = 0ull; Bi = 0ull; }
}

template <int VEC, int TS, bool ANG_BCAST, bool KEEP, bool BRIEF>
__global__ void __launch_bounds__(LS_WARPS * 32, LS_CTAS_PER_SM)
lambda_scan_kernel(const float *__restrict__ u, const float *__restrict__ lm, const float *__restrict__ an,
                   long long an_sb, long long an_st, const float *__restrict__ h0r, const float *__restrict__ h0i,
                   float *__restrict__ y, float *__restrict__ hr_out, float *__restrict__ hi_out, float *__restrict__ hi_all,
                   int B, int T, int D) {
    using Form = LsForm<VEC, BRIEF>;
    constexpr int CQ = 32 / TS, SEG = Form::seg, NST = Form::slots, NP = LsVec<VEC>::NP;
    constexpr int NA = ANG_BCAST ? 2 : 3;                          // u, logmag, angle
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ __align__(16) float slots[Form::staged ? NST : 1][NA][SEG][Form::staged ? LS_WARPS * 32 * VEC : 1];
    const int lane = threadIdx.x & 31;
    const int ngroups = D / VEC;
    const int wpb = (ngroups + CQ - 1) / CQ;                       // warps per batch row
    const long long wg = (long long)blockIdx.x * LS_WARPS + (threadIdx.x >> 5);
    if (wg >= (long long)B * wpb) return;                          // a whole warp leaves together
    const int b = (int)(wg / wpb);
    const int cq = lane % CQ;
    const int seg = lane / CQ;
    const int grp = (int)(wg % wpb) * CQ + cq;
    const bool live = grp < ngroups;
    const int d0 = live ? grp * VEC : 0;

    f2 hr[NP], hi[NP];                                             // state entering the current tile
#pragma unroll
    for (int v = 0; v < NP; ++v) { hr[v] = 0ull; hi[v] = 0ull; }
    if (h0r != nullptr && live) {
        ls_ld<VEC>(hr, h0r + (size_t)b * D + d0);
        ls_ld<VEC>(hi, h0i + (size_t)b * D + d0);
    }
    f2 acs[NP], asn[NP];                                           // cos / sin of a per-channel angle
    if constexpr (ANG_BCAST) {
        f2 a[NP];
#pragma unroll
        for (int v = 0; v < NP; ++v) a[v] = 0ull;
        if (live) ls_ld<VEC>(a, an + d0);
#pragma unroll
        for (int v = 0; v < NP; ++v) { float a0, a1; f2_unpack(a[v], a0, a1); f2_sincos(a0, a1, asn[v], acs[v]); }
    }

    const size_t row0 = (size_t)b * T;
    const int my = (int)threadIdx.x * VEC;
    auto request = [&](int tb, int slot) {                             // one group of copies: a lane's steps of one tile
        if constexpr (!Form::staged) return;
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = tb + i;
            const bool ok = live && t < T;
            const size_t off = ok ? (row0 + t) * D + d0 : 0;
            ls_cp<VEC>(&slots[slot][0][i][my], u + off, ok);
            ls_cp<VEC>(&slots[slot][1][i][my], lm + off, ok);
            if constexpr (!ANG_BCAST) ls_cp<VEC>(&slots[slot][NA - 1][i][my], ok ? an + (size_t)b * an_sb + (size_t)t * an_st + d0 : an, ok);
        }
        ls_cp_commit();
    };
    auto fetch = [&](int tb, f2 (&c)[SEG][NP], f2 (&s)[SEG][NP], f2 (&x)[SEG][NP]) {       // the same into registers
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = tb + i;
            if (live && t < T) {
                const size_t off = (row0 + t) * D + d0;
                ls_ld<VEC>(x[i], u + off);
                ls_ld<VEC>(c[i], lm + off);
                if constexpr (!ANG_BCAST) ls_ld<VEC>(s[i], an + (size_t)b * an_sb + (size_t)t * an_st + d0);
            } else {
#pragma unroll
                for (int v = 0; v < NP; ++v) { x[i][v] = 0ull; c[i][v] = 0ull; s[i][v] = 0ull; }
            }
        }
    };
    constexpr int NREG = Form::staged ? 1 : SEG;
    f2 nc[NREG][NP], ns[NREG][NP], nx[NREG][NP];
    if constexpr (Form::staged) {
#pragma unroll
        for (int k = 0; k < NST; ++k) request((k * TS + seg) * SEG, k);
    } else fetch(seg * SEG, nc, ns, nx);
    for (int t0 = 0, slot = 0; t0 < T; t0 += TS * SEG, slot = slot + 1 == NST ? 0 : slot + 1) {
        const int tb = t0 + seg * SEG;
        f2 c[SEG][NP], s[SEG][NP], x[SEG][NP];
        // 1. the tile out of its slot (or the registers it was requested into), and a later one requested in its place
        if constexpr (Form::staged) {
            ls_cp_wait<NST - 1>();
#pragma unroll
            for (int i = 0; i < SEG; ++i) {
                ls_ld<VEC>(x[i], &slots[slot][0][i][my]);
                ls_ld<VEC>(c[i], &slots[slot][1][i][my]);
                if constexpr (!ANG_BCAST) ls_ld<VEC>(s[i], &slots[slot][NA - 1][i][my]);
            }
            request(tb + NST * TS * SEG, slot);
        } else {
#pragma unroll
            for (int i = 0; i < SEG; ++i)
#pragma unroll
                for (int v = 0; v < NP; ++v) { c[i][v] = nc[i][v]; s[i][v] = ns[i][v]; x[i][v] = nx[i][v]; }
            if (t0 + TS * SEG < T) fetch(tb + TS * SEG, nc, ns, nx);
        }
        // lambda of every step; steps past the end keep log-magnitude and angle 0, the identity map
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const bool ok = live && (tb + i) < T;
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                float l0, l1;
                f2_unpack(c[i][v], l0, l1);
                const f2 mag = f2_exp(l0, l1);
                f2 cs, sn;
                if constexpr (ANG_BCAST) { cs = ok ? acs[v] : f2_both(1.f); sn = ok ? asn[v] : 0ull; }
                else { float a0, a1; f2_unpack(s[i][v], a0, a1); f2_sincos(a0, a1, sn, cs); }
                c[i][v] = f2_mul(mag, cs);
                s[i][v] = f2_mul(mag, sn);
            }
        }
        f2 hsr[NP], hsi[NP];                                       // state entering this lane's segment
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            hsr[v] = hr[v]; hsi[v] = hi[v];
            if constexpr (TS > 1) {
                // 2. the segment's affine map, 3. the map of the segments before it
                f2 Ar = c[0][v], Ai = s[0][v], Br = x[0][v], Bi = 0ull;
#pragma unroll
                for (int i = 1; i < SEG; ++i) {
                    f2 nbr, nbi, nar, nai;
                    ls_cfma(nbr, nbi, c[i][v], s[i][v], Br, Bi, x[i][v], 0ull);
                    ls_cfma(nar, nai, c[i][v], s[i][v], Ar, Ai, 0ull, 0ull);
                    Ar = nar; Ai = nai; Br = nbr; Bi = nbi;
                }
                ls_scan_maps<TS, CQ>(Ar, Ai, Br, Bi, seg);
                ls_cfma(hsr[v], hsi[v], Ar, Ai, hr[v], hi[v], Br, Bi);
            }
        }
        // 4. replay in order and store Re h (and, for a backward pass, Im h)
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = tb + i;
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                f2 nr, ni;
                ls_cfma(nr, ni, c[i][v], s[i][v], hsr[v], hsi[v], x[i][v], 0ull);
                hsr[v] = nr; hsi[v] = ni;
            }
            if (live && t < T) {
                ls_st<VEC>(y + (row0 + t) * D + d0, hsr);
                if constexpr (KEEP) ls_st<VEC>(hi_all + (row0 + t) * D + d0, hsi);
            }
        }
        // state leaving the tile: the last segment's final state
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            if constexpr (TS > 1) {
                hr[v] = __shfl_sync(FULL, hsr[v], (TS - 1) * CQ + cq);
                hi[v] = __shfl_sync(FULL, hsi[v], (TS - 1) * CQ + cq);
            } else {
                hr[v] = hsr[v]; hi[v] = hsi[v];
            }
        }
    }
    ls_cp_wait<0>();                                                   // nothing may land in the slots behind the block's end
    if (live && seg == 0) {
        ls_st<VEC>(hr_out + (size_t)b * D + d0, hr);
        ls_st<VEC>(hi_out + (size_t)b * D + d0, hi);
    }
}

// The adjoint, a_{t-1} = conj(lambda_t) a_t + g_{t-1}, as the same scan over the reversed sequence (reference:
// src/scan_kernel.py:54-101, wired at :121-140); with R_t h_{t-1} = h_t - (u_t, 0) the per-token gradients are
//   du_t = Re a_t,   dlogmag_t = a_t . (h_t - u_t),   dang_t = a_t . i (h_t - u_t).
// One lane per four channels; its loads go through slots as in the forward kernel: maps (g, logmag, angle) a tile ahead, states and u
// requested when the tile before is done, so that the registers hold the maps only (128, 16 warps an SM; 168 and 12 before).
// B64 T4096 D768 1563 -> 1310 us, one angle per channel 1347 -> 1090; B16 T512 D704: 58 -> 47.
template <int VEC, int TS, bool ANG_BCAST>
__global__ void __launch_bounds__(LS_WARPS * 32, LS_CTAS_PER_SM)
lambda_scan_bwd_kernel(const float *__restrict__ g, const float *__restrict__ u, const float *__restrict__ lm, const float *__restrict__ an,
                       long long an_sb, long long an_st, const float *__restrict__ hr_all, const float *__restrict__ hi_all,
                       const float *__restrict__ gli, float *__restrict__ du, float *__restrict__ dlm, float *__restrict__ dan,
                       float *__restrict__ dh0r, float *__restrict__ dh0i, int B, int T, int D) {
    constexpr int CQ = 32 / TS, SEG = LS_SEG, NP = LsVec<VEC>::NP, NA = ANG_BCAST ? 2 : 3;
    constexpr unsigned FULL = 0xffffffffu;
    // g, logmag, angle: free again before the tile's arithmetic; Re h, Im h, u: read step by step in the replay
    __shared__ __align__(16) float slots[NA + 3][SEG][LS_WARPS * 32 * VEC];
    const int lane = threadIdx.x & 31;
    const int ngroups = D / VEC;
    const int wpb = (ngroups + CQ - 1) / CQ;
    const long long wg = (long long)blockIdx.x * LS_WARPS + (threadIdx.x >> 5);
    if (wg >= (long long)B * wpb) return;
    const int b = (int)(wg / wpb), cq = lane % CQ, seg = lane / CQ;
    const int grp = (int)(wg % wpb) * CQ + cq;
    const bool live = grp < ngroups;
    const int d0 = live ? grp * VEC : 0;
    const size_t row0 = (size_t)b * T;
    f2 ar[NP], ai[NP];                                             // adjoint state entering the tile (from later times)
#pragma unroll
    for (int v = 0; v < NP; ++v) { ar[v] = 0ull; ai[v] = 0ull; }
    if (live && gli != nullptr) ls_ld<VEC>(ai, gli + (size_t)b * D + d0);
    auto lambda = [&](const f2 (&l)[NP], const f2 (&a)[NP], f2 (&c)[NP], f2 (&s)[NP]) {
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            float x0, x1;
            f2_unpack(l[v], x0, x1);
            const f2 mag = f2_exp(x0, x1);
            f2 cs, sn;
            f2_unpack(a[v], x0, x1);
            f2_sincos(x0, x1, sn, cs);
            c[v] = f2_mul(mag, cs); s[v] = f2_mul(mag, sn);
        }
    };
    f2 acs[NP], asn[NP];
    if constexpr (ANG_BCAST) {
        f2 a[NP];
#pragma unroll
        for (int v = 0; v < NP; ++v) a[v] = 0ull;
        if (live) ls_ld<VEC>(a, an + d0);
#pragma unroll
        for (int v = 0; v < NP; ++v) { float a0, a1; f2_unpack(a[v], a0, a1); f2_sincos(a0, a1, asn[v], acs[v]); }
    }
    const int my = (int)threadIdx.x * VEC;
    auto request_map = [&](int rb) {                                   // steps past either end: zeros, the identity map
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = T - 1 - (rb + i);
            const bool ok = live && t >= 0, next = ok && t + 1 < T;
            ls_cp<VEC>(&slots[0][i][my], ok ? g + (row0 + t) * D + d0 : g, ok);
            ls_cp<VEC>(&slots[1][i][my], next ? lm + (row0 + t + 1) * D + d0 : lm, next);
            if constexpr (!ANG_BCAST) ls_cp<VEC>(&slots[NA - 1][i][my], next ? an + (size_t)b * an_sb + (size_t)(t + 1) * an_st + d0 : an, next);
        }
        ls_cp_commit();
    };
    auto request_states = [&](int rb) {
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = T - 1 - (rb + i);
            const bool ok = live && t >= 0;
            const size_t off = ok ? (row0 + t) * D + d0 : 0;
            ls_cp<VEC>(&slots[NA][i][my], hr_all + off, ok);
            ls_cp<VEC>(&slots[NA + 1][i][my], hi_all + off, ok);
            ls_cp<VEC>(&slots[NA + 2][i][my], u + off, ok);
        }
        ls_cp_commit();
    };
    request_map(seg * SEG);
    request_states(seg * SEG);
    for (int r0 = 0; r0 < T; r0 += TS * SEG) {
        const int rb = r0 + seg * SEG;                             // reversed step index; time t = T - 1 - r
        f2 c[SEG][NP], s[SEG][NP], x[SEG][NP];
        ls_cp_wait<1>();                                           // the tile's maps are here, its states may still be on their way
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            ls_ld<VEC>(x[i], &slots[0][i][my]);
            ls_ld<VEC>(c[i], &slots[1][i][my]);
            if constexpr (!ANG_BCAST) ls_ld<VEC>(s[i], &slots[NA - 1][i][my]);
        }
        request_map(rb + TS * SEG);
        // conj(lambda_{t+1}); the latest step and steps before time 0 have log-magnitude and angle 0: the identity
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = T - 1 - (rb + i);
            const bool ok = live && t >= 0 && t + 1 < T;
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                float x0, x1;
                f2_unpack(c[i][v], x0, x1);
                const f2 mag = f2_exp(x0, x1);
                f2 cs, sn;
                if constexpr (ANG_BCAST) { cs = ok ? acs[v] : f2_both(1.f); sn = ok ? asn[v] : 0ull; }
                else { f2_unpack(s[i][v], x0, x1); f2_sincos(x0, x1, sn, cs); }
                c[i][v] = f2_mul(mag, cs);
                s[i][v] = f2_neg(f2_mul(mag, sn));
            }
        }
        f2 hsr[NP], hsi[NP];
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            hsr[v] = ar[v]; hsi[v] = ai[v];
            if constexpr (TS > 1) {
                f2 Ar = c[0][v], Ai = s[0][v], Br = x[0][v], Bi = 0ull;
#pragma unroll
                for (int i = 1; i < SEG; ++i) {
                    f2 nbr, nbi, nar, nai;
                    ls_cfma(nbr, nbi, c[i][v], s[i][v], Br, Bi, x[i][v], 0ull);
                    ls_cfma(nar, nai, c[i][v], s[i][v], Ar, Ai, 0ull, 0ull);
                    Ar = nar; Ai = nai; Br = nbr; Bi = nbi;
                }
                ls_scan_maps<TS, CQ>(Ar, Ai, Br, Bi, seg);
                ls_cfma(hsr[v], hsi[v], Ar, Ai, ar[v], ai[v], Br, Bi);
            }
        }
        ls_cp_wait<1>();                                           // the tile's states are here, the next one's maps may still be on their way
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = T - 1 - (rb + i);
            f2 dl[NP], da[NP], rr[NP], ri[NP], uu[NP];             // lambda_t h_{t-1} = h_t - (u_t, 0)
            ls_ld<VEC>(rr, &slots[NA][i][my]);
            ls_ld<VEC>(ri, &slots[NA + 1][i][my]);
            ls_ld<VEC>(uu, &slots[NA + 2][i][my]);
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                rr[v] = f2_add(rr[v], f2_neg(uu[v]));
                f2 nr, ni;
                ls_cfma(nr, ni, c[i][v], s[i][v], hsr[v], hsi[v], x[i][v], 0ull);
                hsr[v] = nr; hsi[v] = ni;
                dl[v] = f2_fma(nr, rr[v], f2_mul(ni, ri[v]));
                da[v] = f2_fma(ni, rr[v], f2_neg(f2_mul(nr, ri[v])));
            }
            if (live && t >= 0) {
                const size_t off = (row0 + t) * D + d0;
                ls_st<VEC>(du + off, hsr);
                ls_st<VEC>(dlm + off, dl);
                ls_st<VEC>(dan + off, da);
            }
        }
        request_states(rb + TS * SEG);
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            if constexpr (TS > 1) {
                ar[v] = __shfl_sync(FULL, hsr[v], (TS - 1) * CQ + cq);
                ai[v] = __shfl_sync(FULL, hsi[v], (TS - 1) * CQ + cq);
            } else {
                ar[v] = hsr[v]; ai[v] = hsi[v];
            }
        }
    }
    ls_cp_wait<0>();                                                   // nothing may land in the slots behind the block's end
    if (live && seg == 0 && dh0r != nullptr) {                     // a_{-1} = conj(lambda_0) a_0
        f2 l[NP], a[NP], c[NP], s[NP], outr[NP], outi[NP];
        ls_ld<VEC>(l, lm + row0 * D + d0);
        ls_ld<VEC>(a, an + (size_t)b * an_sb + d0);
        lambda(l, a, c, s);
#pragma unroll
        for (int v = 0; v < NP; ++v) ls_cfma(outr[v], outi[v], c[v], f2_neg(s[v]), ar[v], ai[v], 0ull, 0ull);
        ls_st<VEC>(dh0r + (size_t)b * D + d0, outr);
        ls_st<VEC>(dh0i + (size_t)b * D + d0, outi);
    }
}

namespace {

struct LsArgs {
    const float *u, *lm, *an; long long sb, st; const float *h0r, *h0i; float *y, *hro, *hio, *hia;
    int B, T, D;
    bool brief;
};
struct LsBwdArgs {
    const float *g, *u, *lm, *an; long long sb, st; const float *hr_all, *hi_all, *gli; float *du, *dlm, *dan, *dh0r, *dh0i;
    int B, T, D;
};

template <int VEC, int TS>
long long ls_ctas(int B, int D) {
    constexpr int CQ = 32 / TS;
    const long long warps = (long long)B * ((D / VEC + CQ - 1) / CQ);
    return (warps + LS_WARPS - 1) / LS_WARPS;
}

template <int VEC, int TS>
int launch_ts(const LsArgs &a, cudaStream_t stream) {
    const long long ctas = ls_ctas<VEC, TS>(a.B, a.D);
    if (ctas > 0x7fffffffLL) return PGB_ERR_TOO_LARGE;
    auto go = [&](auto kern) {
        kern<<<(unsigned)ctas, LS_WARPS * 32, 0, stream>>>(a.u, a.lm, a.an, a.sb, a.st, a.h0r, a.h0i, a.y, a.hro, a.hio, a.hia, a.B, a.T, a.D);
    };
    const bool bc = a.sb == 0 && a.st == 0, keep = a.hia != nullptr;
    auto form = [&](auto brief) {
        constexpr bool BRIEF = decltype(brief)::value;
        if (keep) { if (bc) go(lambda_scan_kernel<VEC, TS, true, true, BRIEF>); else go(lambda_scan_kernel<VEC, TS, false, true, BRIEF>); }
        else { if (bc) go(lambda_scan_kernel<VEC, TS, true, false, BRIEF>); else go(lambda_scan_kernel<VEC, TS, false, false, BRIEF>); }
    };
    if constexpr (VEC == 4) {
        if (a.brief) form(std::true_type{}); else form(std::false_type{});
    } else form(std::false_type{});
    return check_launch("lambda_scan_kernel");
}
template <int VEC, int TS>
int launch_ts(const LsBwdArgs &a, cudaStream_t stream) {
    const long long ctas = ls_ctas<VEC, TS>(a.B, a.D);
    if (ctas > 0x7fffffffLL) return PGB_ERR_TOO_LARGE;
    auto go = [&](auto kern) {
        kern<<<(unsigned)ctas, LS_WARPS * 32, 0, stream>>>(a.g, a.u, a.lm, a.an, a.sb, a.st, a.hr_all, a.hi_all, a.gli, a.du, a.dlm, a.dan, a.dh0r, a.dh0i,
                                                          a.B, a.T, a.D);
    };
    if (a.sb == 0 && a.st == 0) go(lambda_scan_bwd_kernel<VEC, TS, true>); else go(lambda_scan_bwd_kernel<VEC, TS, false>);
    return check_launch("lambda_scan_bwd_kernel");
}

template <int VEC, typename A>
int launch_vec(int ts, const A &a, cudaStream_t stream) {
    switch (ts) {
        case 1:  return launch_ts<VEC, 1>(a, stream);
        case 2:  return launch_ts<VEC, 2>(a, stream);
        case 4:  return launch_ts<VEC, 4>(a, stream);
        case 8:  return launch_ts<VEC, 8>(a, stream);
        case 16: return launch_ts<VEC, 16>(a, stream);
        default: return launch_ts<VEC, 32>(a, stream);
    }
}
template <typename A>
int launch_any(int vec, int ts, const A &a, cudaStream_t stream) {
    return vec == 4 ? launch_vec<4>(ts, a, stream) : vec == 2 ? launch_vec<2>(ts, a, stream) : launch_vec<1>(ts, a, stream);
}
// channels a lane takes: as many as D and every pointer and stride allow
template <typename... P>
int ls_vec(int D, long long sb, long long st, P... ptrs) {
    for (int v = 4; v > 1; v >>= 1)
        if (D % v == 0 && sb % v == 0 && st % v == 0 && (... && aligned(ptrs, 4 * v))) return v;
    return 1;
}

}  // namespace

// Number of time segments per warp, the power of two with the smallest estimate. A launch takes (i) the walk of a warp -- its
// tiles, 1.2 us each (the adjoint's 1.75) and a little for every round of the scan over the segments, times
// warps / resident warps where that is more than one -- and (ii) the bytes at 5 (the adjoint 6) TB/s and, for narrow lanes, their
// instructions; more segments shorten (i), but make the rows a warp reads narrower: the adjoint with rows of 256, 128, 64, 32 and 16 bytes takes
// 1231, 1315, 1410, 1744 and 3241 us at B64 T4096 D768, the scan forward without a copy of the state 886, 642, 662, 725 and 1300. The two overlap:
// root of the sum of squares (B16 T4096 D768, 2 to 16 segments: 652, 362, 259, 201 us; the estimate says 645, 370, 258, 209).
struct LsCost { double tile_us, ps, narrow_ps; bool adjoint; int seg; };   // per tile; per element: the bytes' time, the instructions' of lanes with one channel
struct LsPick { int ts; double cost; };
static LsPick ls_pick(int B, int T, int D, int vec, const LsCost &k, int sms) {
    static const double width[7] = {1.0, 1.0, 1.08, 1.4, 2.3, 3.5, 6.0};        // rows of 256, 128, ... 4 bytes
    const int ngroups = D / vec;
    const double cap = (double)sms * LS_CTAS_PER_SM * LS_WARPS;                 // resident warps
    LsPick best{1, 0.0};
    for (int ts = 1, lg = 0; ts <= 32; ts <<= 1, ++lg) {
        if (ts > 1 && (ts / 2) * k.seg >= T) break;                             // the sequence has no more pieces to hand out
        const int cq = 32 / ts;
        const long long warps = (long long)B * ((ngroups + cq - 1) / cq), tiles = (T + ts * k.seg - 1) / (ts * k.seg);
        int w = 0;
        for (int row = 4 * vec * cq; row < 256; row <<= 1) ++w;
        double f = width[w < 6 ? w : 6];
        if (!k.adjoint && w <= 4) f = sqrt(f);
        if (ts == 32 && warps <= 8LL * sms && f > 1.4) f = 1.4;                 // few warps do not load the memory: a narrow row costs no more than another
        const double walk = (double)tiles * (k.tile_us + 0.1 * lg) * (warps > cap ? (double)warps / cap : 1.0);
        const double move = (double)B * (k.adjoint ? T : tiles * ts * k.seg) * D * 1e-6 * (k.ps * f + (vec == 1 ? k.narrow_ps : 0.0));
        const double cost = walk * walk + move * move;
        if (ts == 1 || cost < best.cost) best = {ts, cost};
    }
    return best;
}
// brief: half the steps a tile, requested a tile ahead into registers, at four fifths of the slots' pace once the memory is loaded
static LsCost ls_cost_fwd(bool bcast, bool brief) {
    const double ps = bcast ? 2.4 : 3.2;
    return brief ? LsCost{bcast ? 0.45 : 0.6, 1.25 * ps, 3.0, false, 2} : LsCost{1.2, ps, 3.0, false, LS_SEG};
}
// Segments and form of a forward call: from its sizes and the angle's form only. A pass that also writes Im h for a backward moves a quarter
// more bytes, for which another choice would now and then be the estimate's best (7 % of shapes, 0.3 % of the time on average, 11 to 19 at most),
// but it takes the same one, so that a sequence gives the same bits in training and in inference.
struct LsForward { int ts; bool brief; };
static LsForward ls_choose_fwd(int B, int T, int D, int vec, bool bcast, int sms) {
    const LsPick slots = ls_pick(B, T, D, vec, ls_cost_fwd(bcast, false), sms);
    if (vec != 4) return {slots.ts, false};
    const LsPick brief = ls_pick(B, T, D, vec, ls_cost_fwd(bcast, true), sms);
    return brief.cost < slots.cost ? LsForward{brief.ts, true} : LsForward{slots.ts, false};
}
// the number to ask for by force_ts, whose segments have LS_SEG steps: an angle per token, rows aligned as D allows
int lambda_scan_pick_ts(int B, int T, int D, int sms) { return ls_pick(B, T, D, ls_vec(D, 0, 0), ls_cost_fwd(false, false), sms).ts; }

int lambda_scan_launch(const float *u, const float *lm, const float *an, long long sb, long long st, const float *h0r,
                       const float *h0i, float *y, float *hro, float *hio, float *hia, int B, int T, int D, int force_ts,
                       cudaStream_t stream) {
    const int vec = ls_vec(D, sb, st, u, lm, an, y, hia, hro, hio, h0r, h0i);
    const LsForward f = force_ts > 0 ? LsForward{force_ts, false} : ls_choose_fwd(B, T, D, vec, sb == 0 && st == 0, sm_count());
    return launch_any(vec, f.ts, LsArgs{u, lm, an, sb, st, h0r, h0i, y, hro, hio, hia, B, T, D, f.brief}, stream);
}

int lambda_scan_bwd_launch(const float *g, const float *u, const float *lm, const float *an, long long sb, long long st,
                           const float *hr_all, const float *hi_all, const float *gli, float *du, float *dlm, float *dan,
                           float *dh0r, float *dh0i, int B, int T, int D, cudaStream_t stream) {
    const int vec = ls_vec(D, sb, st, g, u, lm, an, hr_all, hi_all, gli, du, dlm, dan, dh0r, dh0i);
    const int ts = ls_pick(B, T, D, vec, LsCost{1.75, sb == 0 && st == 0 ? 5.1 : 6.1, 4.5, true, LS_SEG}, sm_count()).ts;
    return launch_any(vec, ts, LsBwdArgs{g, u, lm, an, sb, st, hr_all, hi_all, gli, du, dlm, dan, dh0r, dh0i, B, T, D}, stream);
}

}  // namespace pgb
