// Per-token complex recurrence h_t = lambda_t h_{t-1} + u_t as a chunked parallel scan, and its adjoint.
//
// Layout in HBM: u, logmag, y are [B][T][D] fp32 with D contiguous: 12 B read (8 B when the angle is one value per
// channel) and 4 B written per (b,t,d) element. What bounds it is the wait for a tile's loads at the warps that the registers
// allow: 80 a thread leave 24 warps an SM, 19 active; issue slots are 55 % busy and HBM runs at 0.64 of a copy. e^x, sin, cos and
// the recurrence run on pairs of channels (scan_math.cuh): 90 -> 68 instructions an element, B64 T1024 D768 214 -> 197 us (one angle
// per channel 56 -> 50, 177 -> 155). Rows of 64 or 128 bytes a warp (four time segments or eight) take the same time.
//
// Work split. A lane owns VEC adjacent channels (4 where D, pointers and strides allow: one 128-bit access; else 2 or 1). A warp is TS time-segments x CQ
// channel groups (TS * CQ = 32): lanes of one segment read 16*CQ contiguous bytes of one time row, so every 128-byte
// line is used whole. A tile is TS*SEG consecutive time steps; per tile each lane
//   1. loads its SEG steps (all loads issued before any is used) and forms c_t = |l_t| cos, s_t = |l_t| sin,
//   2. folds them into the segment's affine map h -> A h + Bv (complex A, Bv), starting from (1, 0),
//   3. combines the maps of the segments before it with a shuffle scan over the TS segment lanes
//      ((A2,B2) o (A1,B1) = (A2 A1, A2 B1 + B2)), which gives the state entering its segment,
//   4. replays the recurrence over its SEG steps from that state in the reference's operation order
//      (src/scan_kernel.py:42-48) and stores Re h.
// The state leaving the tile is broadcast from the last segment lane. With TS = 1 the kernel is the literal sequential
// recurrence; with TS > 1 only the state at segment boundaries is reassociated (fp32 rounding, no other difference).
#include "scan_math.cuh"

namespace pgb {

constexpr int LS_WARPS = 2;
// Two forms of the forward kernel. WIDE fills the chip with warps: 24 an SM (80 registers a thread), every load of a tile ahead
// of its use, four steps a lane and tile (two with one angle per channel, whose cosines take the registers, and with Im h kept). AHEAD is for
// launches with fewer warps than that, which cannot hide a tile's loads behind one another: two steps a lane and tile (four
// with narrow vectors) and the next tile requested before this one is worked on, 16 warps an SM (12 with 32 segments).
// B64 T4096 D768: wide 785-830 us (577 with one angle per channel; with Im h 930 and 719), ahead 1291; B4 T2048 D768, one angle
// per channel: 63 and 52; B16 T512 D704, one angle per channel, with Im h: 53 and 35.
template <int VEC, bool AHEAD, bool FEW> struct LsSeg { static constexpr int n = VEC < 4 ? 4 : (AHEAD || FEW ? 2 : 4); };
constexpr int LS_WIDE_CTAS = 12, LS_AHEAD_CTAS = 8, LS_AHEAD_CTAS_TS32 = 6;
constexpr int LS_BWD_CTAS_PER_SM = 6;                                 // the adjoint: 168 registers, it holds the states of its steps as well

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
    if constexpr (VEC == 4) *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(d[0], d[1]);
    else if constexpr (VEC == 2) *reinterpret_cast<f2 *>(p) = d[0];
    else { float a, b; f2_unpack(d[0], a, b); *p = a; }
}
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

template <int VEC, int TS, bool ANG_BCAST, bool KEEP, bool AHEAD>
__global__ void __launch_bounds__(LS_WARPS * 32, !AHEAD ? LS_WIDE_CTAS : TS == 32 ? LS_AHEAD_CTAS_TS32 : LS_AHEAD_CTAS)
lambda_scan_kernel(const float *__restrict__ u, const float *__restrict__ lm, const float *__restrict__ an,
                   long long an_sb, long long an_st, const float *__restrict__ h0r, const float *__restrict__ h0i,
                   float *__restrict__ y, float *__restrict__ hr_out, float *__restrict__ hi_out, float *__restrict__ hi_all,
                   int B, int T, int D) {
    constexpr int CQ = 32 / TS, SEG = LsSeg<VEC, AHEAD, ANG_BCAST || KEEP>::n, NP = LsVec<VEC>::NP;
    constexpr unsigned FULL = 0xffffffffu;
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
    auto fetch = [&](int tb, f2 (&c)[SEG][NP], f2 (&s)[SEG][NP], f2 (&x)[SEG][NP]) {       // every load of a lane's steps
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
    f2 nc[AHEAD ? SEG : 1][NP], ns[AHEAD ? SEG : 1][NP], nx[AHEAD ? SEG : 1][NP];
    if constexpr (AHEAD) fetch(seg * SEG, nc, ns, nx);
    for (int t0 = 0; t0 < T; t0 += TS * SEG) {
        const int tb = t0 + seg * SEG;
        f2 c[SEG][NP], s[SEG][NP], x[SEG][NP];
        // 1. loads first
        if constexpr (AHEAD) {
#pragma unroll
            for (int i = 0; i < SEG; ++i)
#pragma unroll
                for (int v = 0; v < NP; ++v) { c[i][v] = nc[i][v]; s[i][v] = ns[i][v]; x[i][v] = nx[i][v]; }
            if (t0 + TS * SEG < T) fetch(tb + TS * SEG, nc, ns, nx);
        } else fetch(tb, c, s, x);
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
    if (live && seg == 0) {
        ls_st<VEC>(hr_out + (size_t)b * D + d0, hr);
        ls_st<VEC>(hi_out + (size_t)b * D + d0, hi);
    }
}

// The adjoint, a_{t-1} = conj(lambda_t) a_t + g_{t-1}, as the same scan over the reversed sequence (reference:
// src/scan_kernel.py:54-101, wired at :121-140); with R_t h_{t-1} = h_t - (u_t, 0) the per-token gradients are
//   du_t = Re a_t,   dlogmag_t = a_t . (h_t - u_t),   dang_t = a_t . i (h_t - u_t).
// One lane per four channels instead of one, the state's rows requested before the scan over the segments. B64 T4096 D768, one
// angle per channel: 5716 -> 1430-1670 us (4.3-4.5 TB/s); B16 T512 D704: 123 -> 63 us.
template <int VEC, int TS, bool ANG_BCAST>
__global__ void __launch_bounds__(LS_WARPS * 32, LS_BWD_CTAS_PER_SM)
lambda_scan_bwd_kernel(const float *__restrict__ g, const float *__restrict__ u, const float *__restrict__ lm, const float *__restrict__ an,
                       long long an_sb, long long an_st, const float *__restrict__ hr_all, const float *__restrict__ hi_all,
                       const float *__restrict__ gli, float *__restrict__ du, float *__restrict__ dlm, float *__restrict__ dan,
                       float *__restrict__ dh0r, float *__restrict__ dh0i, int B, int T, int D) {
    constexpr int CQ = 32 / TS, SEG = 4, NP = LsVec<VEC>::NP;
    constexpr unsigned FULL = 0xffffffffu;
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
    for (int r0 = 0; r0 < T; r0 += TS * SEG) {
        const int rb = r0 + seg * SEG;                             // reversed step index; time t = T - 1 - r
        f2 c[SEG][NP], s[SEG][NP], x[SEG][NP], rr[SEG][NP], ri[SEG][NP];
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = T - 1 - (rb + i);
#pragma unroll
            for (int v = 0; v < NP; ++v) { c[i][v] = 0ull; s[i][v] = 0ull; x[i][v] = 0ull; rr[i][v] = 0ull; ri[i][v] = 0ull; }
            if (live && t >= 0) {
                const size_t off = (row0 + t) * D + d0;
                ls_ld<VEC>(x[i], g + off);
                if (t + 1 < T) {
                    ls_ld<VEC>(c[i], lm + off + D);
                    if constexpr (!ANG_BCAST) ls_ld<VEC>(s[i], an + (size_t)b * an_sb + (size_t)(t + 1) * an_st + d0);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < SEG; ++i) {                            // lambda_t h_{t-1} = h_t - (u_t, 0)
            const int t = T - 1 - (rb + i);
            if (live && t >= 0) {
                const size_t off = (row0 + t) * D + d0;
                f2 uu[NP];
                ls_ld<VEC>(rr[i], hr_all + off);
                ls_ld<VEC>(uu, u + off);
                ls_ld<VEC>(ri[i], hi_all + off);
#pragma unroll
                for (int v = 0; v < NP; ++v) rr[i][v] = f2_add(rr[i][v], f2_neg(uu[v]));
            }
        }
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
#pragma unroll
        for (int i = 0; i < SEG; ++i) {
            const int t = T - 1 - (rb + i);
            f2 dl[NP], da[NP];
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                f2 nr, ni;
                ls_cfma(nr, ni, c[i][v], s[i][v], hsr[v], hsi[v], x[i][v], 0ull);
                hsr[v] = nr; hsi[v] = ni;
                dl[v] = f2_fma(nr, rr[i][v], f2_mul(ni, ri[i][v]));
                da[v] = f2_fma(ni, rr[i][v], f2_neg(f2_mul(nr, ri[i][v])));
            }
            if (live && t >= 0) {
                const size_t off = (row0 + t) * D + d0;
                ls_st<VEC>(du + off, hsr);
                ls_st<VEC>(dlm + off, dl);
                ls_st<VEC>(dan + off, da);
            }
        }
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
    bool wide;
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
    if constexpr (VEC == 4 && TS < 32)
        if (a.wide) {
            if (keep) { if (bc) go(lambda_scan_kernel<VEC, TS, true, true, false>); else go(lambda_scan_kernel<VEC, TS, false, true, false>); }
            else { if (bc) go(lambda_scan_kernel<VEC, TS, true, false, false>); else go(lambda_scan_kernel<VEC, TS, false, false, false>); }
            return check_launch("lambda_scan_kernel");
        }
    if (keep) { if (bc) go(lambda_scan_kernel<VEC, TS, true, true, true>); else go(lambda_scan_kernel<VEC, TS, false, true, true>); }
    else { if (bc) go(lambda_scan_kernel<VEC, TS, true, false, true>); else go(lambda_scan_kernel<VEC, TS, false, false, true>); }
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

// Number of time segments per warp. Every warp walks its whole time axis and all warps of a launch take the same time, so the
// launch lasts rounds x tiles-per-warp x tile cost with rounds = ceil(warps / resident warps). More segments shorten a warp's
// walk but cost shuffle-scan rounds and, past the resident capacity, a whole extra round; and 32 segments leave each row access
// 16 bytes wide, half a memory sector, which costs as much again once there are warps enough to load memory (B52 T1579
// D240: 143 us with 32, 102 with 16). Take the power of two with the smallest estimate. `force_ts` > 0 overrides (tests).
static int ls_pick(int B, int T, int D, int vec, int seg, int sms, int ctas_per_sm) {
    const int ngroups = D / vec;
    const long long cap = (long long)sms * ctas_per_sm * LS_WARPS;              // resident warps
    int best = 1;
    double best_cost = 0.0;
    for (int ts = 1, lg = 0; ts <= 32; ts <<= 1, ++lg) {
        if (ts > 1 && (ts / 2) * seg >= T) break;                               // the sequence has no more pieces to hand out
        const int cq = 32 / ts;
        const long long warps = (long long)B * ((ngroups + cq - 1) / cq);
        const long long rounds = (warps + cap - 1) / cap;
        const long long tiles = (T + ts * seg - 1) / (ts * seg);
        const double tile = seg * 60.0 + lg * 14.0 + 12.0;                      // per lane and channel: steps, scan rounds, hand-over
        const double cost = (double)rounds * (double)tiles * tile * (ts == 32 && warps > 8LL * sms ? 2.0 : 1.0);
        if (ts == 1 || cost < best_cost) { best = ts; best_cost = cost; }
    }
    return best;
}
int lambda_scan_pick_ts(int B, int T, int D, int vec, int sms, int force_ts) {
    return force_ts > 0 ? force_ts : ls_pick(B, T, D, vec, LsSeg<4, false, false>::n, sms, LS_WIDE_CTAS);
}

int lambda_scan_launch(const float *u, const float *lm, const float *an, long long sb, long long st, const float *h0r,
                       const float *h0i, float *y, float *hro, float *hio, float *hia, int B, int T, int D, int force_ts,
                       cudaStream_t stream) {
    const int sms = sm_count();
    const int vec = ls_vec(D, sb, st, u, lm, an, y, hia, hro, hio, h0r, h0i);
    int ts = lambda_scan_pick_ts(B, T, D, vec, sms, force_ts);
    // the wide form where its warps outnumber what the form that loads ahead can keep resident
    const int cq = 32 / ts;
    const bool wide = vec == 4 && ts < 32 && (long long)B * ((D / vec + cq - 1) / cq) > (long long)sms * LS_AHEAD_CTAS * LS_WARPS;
    if (!wide && force_ts <= 0) ts = ls_pick(B, T, D, vec, LsSeg<4, true, false>::n, sms, LS_AHEAD_CTAS);
    return launch_any(vec, ts, LsArgs{u, lm, an, sb, st, h0r, h0i, y, hro, hio, hia, B, T, D, wide}, stream);
}

int lambda_scan_bwd_launch(const float *g, const float *u, const float *lm, const float *an, long long sb, long long st,
                           const float *hr_all, const float *hi_all, const float *gli, float *du, float *dlm, float *dan,
                           float *dh0r, float *dh0i, int B, int T, int D, cudaStream_t stream) {
    const int vec = ls_vec(D, sb, st, g, u, lm, an, hr_all, hi_all, gli, du, dlm, dan, dh0r, dh0i);
    const int ts = ls_pick(B, T, D, vec, 4, sm_count(), LS_BWD_CTAS_PER_SM);
    return launch_any(vec, ts, LsBwdArgs{g, u, lm, an, sb, st, hr_all, hi_all, gli, du, dlm, dan, dh0r, dh0i, B, T, D}, stream);
}

}  // namespace pgb
