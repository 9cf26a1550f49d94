// forces64_dev.cuh — pair loops of the FP64 force stages.
//
// A GB300 SM issues one FP64 warp instruction about every 16 cycles (64 times
// slower than FP32), so these passes are bound by the number of FP64
// operations per pair, and, for systems that do not fill the GPU, by how many
// SMs have a warp at all. Hence:
//  - comparisons of squared distances, interval indices and conversions run
//    on the integer and FP32 pipes (exact on the FP64 bits);
//  - an FP32 screen picks the entries that can be inside the cutoff, so each
//    lane walks in-range pairs only (walk64);
//  - 1/r and 1/r^2 come from an FP32 hardware estimate refined by one
//    third-order (Householder) step in FP64, five and three FP64 operations,
//    in place of a square root and two divisions (about thirty);
//  - table pieces are cubics in x = r - r_n with coefficients made on the
//    host, W = V'r - V as one cubic (no cancellation of V'r against V);
//  - a pair across a periodic face takes its image by one addition per axis,
//    in the one walk over the list;
//  - G lanes share an atom's list where one thread per atom would leave SMs
//    without work (kFewAtoms64).
// EAM Cu 389,344 atoms: force pass 0.90 ms (27 FP64 operations per in-range
// pair, FP64 pipe 86% active), density 0.65 ms (18, 83%). EAM Cu 1,000,188
// atoms: 13.1 -> 3.87 ms per step; LJ argon 4,000 atoms 0.45 -> 0.05 ms.
#pragma once

#include <cuda_runtime.h>

#include "forces_dev.cuh"

namespace mdg {

// Lanes per atom of the FP64 passes, launched (with_lanes64) or by a grid's
// team, whose sums over lanes then have the same order: 32 below 2,000 atoms,
// 16 below 12,500 with EAM tables and 24,000 without, 4 below 100,000, else
// one. Fewer atoms than about 100,000 threads' worth leave SMs with too few
// warps to keep their FP64 pipe busy; more lanes than that cost the sums over
// lanes and lanes without a pair. Measured per launched FP64 step, 4 / 16 / 32
// lanes: LJ argon 500 atoms - / 30.3 / 26.4 us, 8,788 74 / 62 / 72, 19,652
// 118 / 101 / 126; EAM Cu 500 - / 42.1 / 32.9, 8,788 - / 98.7 / 103.9, 13,500
// 113 / 131 / 141; 1 / 4 lanes: EAM Cu 108,000 560 / 565, 1,000,188 3,870 /
// 4,540.
constexpr size_t kFewAtoms64 = 2000;
inline size_t some_atoms64(bool eam) { return eam ? 12500 : 24000; }

// The FP32 number nearest below a positive double (2^-126 <= x), by integer
// operations; beyond FP32's range it saturates. NaN gives a finite number.
__device__ __forceinline__ float to_float_rz(double x) {
    const int hi = min(__double2hiint(x), 0x47efffff);
    return __int_as_float((int)__funnelshift_l((unsigned)__double2loint(x), (unsigned)(hi - 0x38000000), 3));
}

// A positive (or zero: then 2^-127) FP32 number as a double, by integer operations.
__device__ __forceinline__ double widen(float f) {
    const int b = __float_as_int(f);
    return __hiloint2double((b >> 3) + 0x38000000, b << 29);
}

// 1/sqrt(x) in FP64: y0 from FP32 (|e| = |1 - x y0^2| < 2^-20), then the
// third-order Householder step y0 (1 + e/2 + 3 e^2 / 8), whose remainder
// 5 e^3 / 16 is below 2^-61. rf gets sqrt(x) in FP32.
__device__ __forceinline__ double rsqrt64(double x, float& rf) {
    const float xf = to_float_rz(x);
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
    rf = xf * yf;
    const double y0 = widen(yf);
    const double e = fma(-(x * y0), y0, 1.0);
    return fma(y0 * e, fma(0.375, e, 0.5), y0);
}

// 1/x in FP64: y0 from FP32, then y0 (1 + e + e^2), e = 1 - x y0; the
// remainder e^3 is below 2^-60.
__device__ __forceinline__ double rcp64(double x) {
    float yf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(to_float_rz(x)));
    const double y0 = widen(yf);
    const double e = fma(-x, y0, 1.0);
    return fma(y0, fma(e, e, e), y0);
}

__device__ __forceinline__ void load_row64(const double* p, double c[4]) {
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(c[0]), "=d"(c[1]), "=d"(c[2]), "=d"(c[3]) : "l"(p));
}

__device__ __forceinline__ double cubic64(const double c[4], double x) {
    return fma(x, fma(x, fma(x, c[3], c[2]), c[1]), c[0]);
}

// Interval of r = r2 ri on a table's grid and x = r - r_n; false past the
// table (N1 >= Nr1). The index comes from FP32 (rf = r to 2^-21) and is moved
// by one where x shows it a neighbour's; near the table's end it is the
// reference's trunc(r / dr) in FP64, which decides whether the table ends.
__device__ __forceinline__ bool interval64(const PotParams& P, double r2, double ri, float rf, int& nn, double& x) {
    nn = (int)(rf * P.inv_dr_f);
    if (nn >= P.Nr1 - 1) {
        nn = (int)trunc(r2 * ri * P.dr1);
        if (nn >= P.Nr1) return false;
        nn = max(nn, 0);  // r = NaN: any row, x is NaN
        x = fma(r2, ri, -__ldg(P.rn64 + nn));
        return true;
    }
    x = fma(r2, ri, -__ldg(P.rn64 + nn));
    const long long xb = __double_as_longlong(x);
    if (xb < 0 || xb >= __double_as_longlong(P.dr)) {
        nn += xb >= 0 ? 1 : nn > 0 ? -1 : 0;
        x = fma(r2, ri, -__ldg(P.rn64 + nn));
    }
    return true;
}

// Force over r of a tabulated pair, AdF rho' + (V'r - V)/r^2 over r
// (EAM.cxx:417-463; the tabulated Pair has zero rho rows, pair.cxx:316-346),
// and V/(2r), its energy term.
template <bool EAM, bool ENERGY>
__device__ __forceinline__ double table_ff64(const PotParams& P, double r2, double AdF, double& E) {
    float rf;
    const double ri = rsqrt64(r2, rf);
    int nn;
    double x;
    E = 0.0;
    if (!interval64(P, r2, ri, rf, nn, x)) return 0.0;
    double w[4];
    load_row64(P.wd64 + 8 * (size_t)nn, w);
    double ff = cubic64(w, x) * (ri * ri);
    if (EAM) {
        double d[4];
        load_row64(P.wd64 + 8 * (size_t)nn + 4, d);
        ff = fma(AdF, fma(x, fma(x, d[2], d[1]), d[0]), ff);
    }
    if (ENERGY) {
        double v[4];
        load_row64(P.v64 + 4 * (size_t)nn, v);
        E = 0.5 * cubic64(v, x) * ri;
    }
    return ff * ri;
}

// rho(r) of an EAM pair (EAM.cxx:533-560).
__device__ __forceinline__ double table_rho64(const PotParams& P, double r2) {
    float rf;
    const double ri = rsqrt64(r2, rf);
    int nn;
    double x;
    if (!interval64(P, r2, ri, rf, nn, x)) return 0.0;
    double c[4];
    load_row64(P.rho64 + 4 * (size_t)nn, c);
    return cubic64(c, x);
}

// LJsCut force over r (LJs-cut.cxx:35-47) and energy term (LJs-cut.cxx:105).
template <bool ENERGY>
__device__ __forceinline__ double ljcut_ff64(const PotParams& P, double r2, double& E) {
    const double r2i = rcp64(r2);
    const double r6i = r2i * r2i * r2i;
    if (ENERGY) {
        const double t = P.s6 * r6i;
        E = 2.0 * P.a * t * (t - 1.0);
    }
    return fma(P.mhf_lj1, r6i, P.hf_lj2) * (r6i * r2i);
}

// LJs force over r and energy term (LJs.cxx:90-101, 153-166).
template <bool ENERGY>
__device__ __forceinline__ double ljs_pair64(const PotParams& P, double r2, double& E) {
    const double X = fma(P.ljs_rVr1, r2, -1.2599210498948732);
    const double FV = P.ljs_rVr2 * rcp64(r2);
    const double Ur = FV * FV * FV;
    if (ENERGY) E = P.ljs_aVr * (Ur * (Ur - 1.0) - (P.ljs_aLJ3 + P.ljs_bLJ2 * X) * X * X);
    return P.ljs_aVr2 * (Ur * (Ur - 0.5) * FV + (P.ljs_aLJ + P.ljs_bLJ * X) * X);
}

// r2 <= R2cut and not r2 < 1e-15, on the bits of a non-negative r2; NaN of
// either sign passes (unsigned, its bits are above infinity's), as it fails
// both of the reference's tests (its force is flagged).
__device__ __forceinline__ bool in_cut64(double r2, double R2cut) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(r2);
    return b >= 0x3cd203af9ee75616ULL /* 1e-15 */ &&
           (b <= (unsigned long long)__double_as_longlong(R2cut) || b > 0x7ff0000000000000ULL);
}

// Any double as FP32 by integer operations, truncated; NaN from 2^128 up.
__device__ __forceinline__ float screen_float(double x) {
    const int hi = __double2hiint(x);
    const int m = max(min(hi & 0x7fffffff, 0x47ffffff), 0x38000000);
    return __int_as_float((int)__funnelshift_l((unsigned)__double2loint(x), (unsigned)(m - 0x38000000), 3) |
                          (hi & (int)0x80000000));
}

struct Pair64 {
    double dx, dy, dz, r2;
};
// (Where a sum of products could be contracted in more than one way, these
// passes spell the fma out: a grid's team gives the launched passes' bits.)
__device__ __forceinline__ double norm64(double x, double y, double z) { return fma(x, x, fma(y, y, z * z)); }

// The Periodic boundary's ghost of a listed pair (boundary/periodic.cxx:
// 36-102), for an atom near a periodic face: a pair whose raw distance is at
// least max(rns) counts again through its shortest image. False when the
// reference makes none.
__device__ __forceinline__ bool ghost64(const FArgs& A, double rni, uint32_t j, const Pair64& p, Pair64& q) {
    const double rnj = A.rns[j];
    const double rn = rnj < rni ? rni : rnj;
    const double r2rns = rn * rn;
    if (p.r2 < r2rns) return false;
    q.dx = shortest1(p.dx, A.L[0], A.periodic[0]);
    q.dy = shortest1(p.dy, A.L[1], A.periodic[1]);
    q.dz = shortest1(p.dz, A.L[2], A.periodic[2]);
    q.r2 = norm64(q.dx, q.dy, q.dz);
    return !(q.r2 > r2rns);
}

// What FP32 tells of the pairs of atom i before any FP64 work: the box as
// seen from it and the screen's threshold.
struct Screen64 {
    float x, y, z;     // the atom's position
    float L[3], il[3]; // periodic edges and their inverses (0: open)
    float thr;         // (rc + error)^2
    float rc, Lmin;    // the largest cutoff; the smallest periodic edge, 0: images by FP64

    template <bool MULTI>
    __device__ __forceinline__ void set(const FArgs& A, const PotSet* __restrict__ ps, int ki, double xi, double yi,
                                        double zi) {
        x = screen_float(xi);
        y = screen_float(yi);
        z = screen_float(zi);
        float far = 0.f, rc2 = 0.f;
        Lmin = 3e38f;
        for (int a = 0; a < 3; ++a) {
            const float l = (float)A.L[a];
            far = fmaxf(far, l);
            const bool per = A.periodic[a] && l > 0.f;
            L[a] = per ? l : 0.f;
            il[a] = per ? 1.0f / l : 0.f;
            if (per) Lmin = fminf(Lmin, l);
        }
        for (int b = 0; b < (MULTI ? ps->nkinds : 1); ++b) rc2 = fmaxf(rc2, ps->p[ki][b].r2cut_f);
        rc = sqrtf(rc2) * 1.00001f;
        // each FP32 coordinate difference is off by less than 2^-21 of the
        // largest coordinate an atom within reach can have
        const float reach = fmaf(fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)) + far + rc, 9.5367431640625e-7f, rc);
        thr = reach * reach;
        // nor does an FP32 difference tell the image of a pair in range where
        // the shorter way round is not longer by that error: no edge will do
        if (!(Lmin > 2.0f * reach)) Lmin = 0.f;
    }
};

// Walks the entries k = lane, lane + G, ... of atom i's list, 64 a turn.
// SCREEN: a first pass in FP32 marks the entries whose shortest image may lie
// inside the cutoff (a superset: its threshold covers the FP32 error), and
// only those are visited in FP64, so that the lanes of a warp spend their
// FP64 work on nearly the same number of pairs rather than on the union of
// their in-range entries (EAM Cu: 42 of 54 listed pairs are in range).
// A pair is what the reference visits (Pair::* then Periodic::*_one): the raw
// difference and, for atoms near a periodic face (bc), its ghost. Where every
// periodic edge is above 2 rns, and above twice the cutoff by more than the
// FP32 error at these coordinates, and rns above the cutoff, a pair is one or
// the other by the sign and size of its FP32 difference, and the image is one
// addition per axis; otherwise ghost64 decides in FP64, and with rns below
// the cutoff both can count.
// For every visit: seen(P, kj, k, ghost) (without SCREEN, which skips
// visits); for those inside the cutoff: use(P, kj, j, pair, ghost).
template <bool MULTI, int G, bool SCREEN, bool RO, typename Seen, typename Use>
__device__ __forceinline__ void walk64(const FArgs& A, const PotSet* __restrict__ ps, int i, int ki, int lane,
                                       Seen&& seen, Use&& use) {
    const double xi = A.rx[i], yi = A.ry[i], zi = A.rz[i];
    const int cnt = A.ncnt[i];
    const bool bc = A.bc[i] != 0;
    const double rni = A.rns[i];
    const long long rni2 = __double_as_longlong(rni * rni);
    Screen64 S;
    S.set<MULTI>(A, ps, ki, xi, yi, zi);
    const float rnf = screen_float(rni);
    for (int k0 = lane; k0 < cnt; k0 += 64 * G) {
        const int turn = min((cnt - k0 + G - 1) / G, 64);
        unsigned long long todo = turn == 64 ? ~0ull : (1ull << turn) - 1ull;
        if (SCREEN) {
            todo = 0;
#pragma unroll 4
            for (int m = 0; m < turn; ++m) {
                const uint32_t j = ld_ro<RO>(A.nbr + nidx(k0 + m * G, i, A.np)) & kJMask;
                float dx = screen_float(ld_ro<RO>(A.rx + j)) - S.x;
                float dy = screen_float(ld_ro<RO>(A.ry + j)) - S.y;
                float dz = screen_float(ld_ro<RO>(A.rz + j)) - S.z;
                dx = fmaf(-S.L[0], rintf(dx * S.il[0]), dx);
                dy = fmaf(-S.L[1], rintf(dy * S.il[1]), dy);
                dz = fmaf(-S.L[2], rintf(dz * S.il[2]), dz);
                const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                todo |= (unsigned long long)(!(r2 > S.thr) && j != (uint32_t)i) << m;
            }
        }
        while (todo) {
            const int k = k0 + (__ffsll((long long)todo) - 1) * G;
            todo &= todo - 1ull;
            const uint32_t j = ld_ro<RO>(A.nbr + nidx(k, i, A.np)) & kJMask;
            const int kj = MULTI ? (A.kind[j] & 3) : 0;
            const PotParams& P = ps->p[ki][kj];
            Pair64 p, s;
            const double xj = ld_ro<RO>(A.rx + j), yj = ld_ro<RO>(A.ry + j), zj = ld_ro<RO>(A.rz + j);
            p.dx = xj - xi;
            p.dy = yj - yi;
            p.dz = zj - zi;
            bool ghost = false, exact = false;
            if (bc) {
                const float rn = fmaxf(rnf, screen_float(A.rns[j])) * 1.00001f;
                exact = !SCREEN || !(S.Lmin > 2.0f * rn && rn * 0.9999f > S.rc);
                if (!exact) {
                    // the image the reference's Domain::shortest picks, L / 2
                    // apart being out of range
                    const float tx = rintf((screen_float(xj) - S.x) * S.il[0]);
                    const float ty = rintf((screen_float(yj) - S.y) * S.il[1]);
                    const float tz = rintf((screen_float(zj) - S.z) * S.il[2]);
                    ghost = tx != 0.f || ty != 0.f || tz != 0.f;
                    if (ghost) {
                        p.dx = dadd(p.dx, tx > 0.f ? -A.L[0] : tx < 0.f ? A.L[0] : 0.0);
                        p.dy = dadd(p.dy, ty > 0.f ? -A.L[1] : ty < 0.f ? A.L[1] : 0.0);
                        p.dz = dadd(p.dz, tz > 0.f ? -A.L[2] : tz < 0.f ? A.L[2] : 0.0);
                    }
                }
            }
            p.r2 = norm64(p.dx, p.dy, p.dz);
            if (!SCREEN) seen(P, kj, k, false);
            bool in = in_cut64(p.r2, P.R2cut), both = false;
            if (exact && __double_as_longlong(p.r2) >= rni2 && ghost64(A, rni, j, p, s)) {
                if (!SCREEN) seen(P, kj, k, true);
                both = in;  // rns below the cutoff: the raw pair and its ghost both count
                if (!in) {
                    p = s;
                    ghost = true;
                    in = in_cut64(p.r2, P.R2cut);
                }
            }
            for (;;) {
                if (in) use(P, kj, j, p, ghost);
                if (!both) break;
                both = false;
                p = s;
                ghost = true;
                in = in_cut64(p.r2, P.R2cut);
            }
        }
    }
}

// Sum over the G lanes of an atom (every lane gets it).
template <int G>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void eam_embed64(const PotParams& P, double nr, double* EF, double* dF,
                                            DevStatus* st) {
    double RN = nr * P.drh1;
    int N1 = (int)trunc(RN);
    double dF0 = 0.0;  // the reference's output array is zero-initialised
    if (RN >= 0.0 && N1 < P.Nrh1) {
        if (N1 == P.Nrh1 - 1) atomicOr(&st->flags, FLAG_TABLE);
        double VR = N1;
        double DV = RN - VR;
        RN = fma(-VR, P.drh, nr);
        VR = (P.Femb[N1 + 1] - P.Femb[N1]) * P.drh1;
        const double aa = (P.dFemb[N1 + 1] - VR) - (VR - P.dFemb[N1]);
        const double bb = aa - (VR - P.dFemb[N1]);
        *EF = fma(RN, fma(DV, fma(aa, DV, -bb), P.dFemb[N1]), P.Femb[N1]);
        *dF = fma(2.0 * DV, fma(1.5 * aa, DV, -bb), P.dFemb[N1]);
    } else {
        atomicOr(&st->flags, FLAG_TABLE);
        if (N1 >= P.Nrh1) {
            *EF = P.Femb[P.Nrh1] + P.dFemb[P.Nrh1] * (dF0 - P.Nrh1 * P.drh);
            *dF = P.dFemb[P.Nrh1];
        } else {
            *EF = P.Femb[0] - P.dFemb[0] * dF0;
            *dF = P.dFemb[0];
        }
    }
}

// The force of atom i by G lanes (every lane of a warp calls this; `live`
// false: none); on all of them. FORM: the potential of every pair where there
// is one (POT_LJCUT, POT_EAM; Single), 0 = by kind pair. HALF also pushes the
// pair-type terms onto the neighbours.
template <bool MULTI, int FORM, bool HALF, int G, bool RO = true>
__device__ __forceinline__ void forces64_lanes(const FArgs& A, const PotSet* __restrict__ ps, bool live, int i,
                                               int lane, double f[3]) {
    f[0] = f[1] = f[2] = 0.0;
    if (live) {
        const int ki = MULTI ? (A.kind[i] & 3) : 0;
        walk64<MULTI, G, true, RO>(A, ps, i, ki, lane, [](const PotParams&, int, int, bool) {},
                         [&](const PotParams& P, int kj, uint32_t j, const Pair64& p, bool ghost) {
            const int type = FORM ? FORM : P.type;
            double pref, E;
            if (type == POT_LJCUT) {
                pref = ljcut_ff64<false>(P, p.r2, E);
            } else if (type == POT_EAM) {
                const double AdF = A.Fp64[(size_t)ki * A.np + j] + A.Fp64[(size_t)kj * A.np + i];
                pref = table_ff64<true, false>(P, p.r2, AdF, E);
            } else if (type == POT_TAB) {
                pref = table_ff64<false, false>(P, p.r2, 0.0, E);
            } else if (type == POT_LJS) {
                pref = ljs_pair64<false>(P, p.r2, E);
            } else {
                return;
            }
            f[0] = fma(p.dx, pref, f[0]);
            f[1] = fma(p.dy, pref, f[1]);
            f[2] = fma(p.dz, pref, f[2]);
            if (HALF && !ghost && type != POT_EAM) {
                atomicAdd(&A.fx[j], -(p.dx * pref));
                atomicAdd(&A.fy[j], -(p.dy * pref));
                atomicAdd(&A.fz[j], -(p.dz * pref));
            }
        });
    }
    for (int a = 0; a < 3; ++a) f[a] = lane_sum<G>(f[a]);
    if (live && lane == 0 && !(isfinite(f[0]) && isfinite(f[1]) && isfinite(f[2])))
        atomicOr(&A.st->flags, FLAG_NONFINITE);
}

// The EAM density of atom i (where `in`) by G lanes, and F' of it.
template <bool MULTI, int G, bool RO = true>
__device__ __forceinline__ void density64_lanes(const FArgs& A, const PotSet* __restrict__ ps, bool in, int i,
                                                int lane) {
    if (!in) i = 0;
    const int ki = MULTI && in ? (A.kind[i] & 3) : 0;
    const bool live = in && A.tag[i] != 0;
    double rho = 0.0;
    if (live)
        walk64<MULTI, G, true, RO>(A, ps, i, ki, lane, [](const PotParams&, int, int, bool) {},
                         [&](const PotParams& P, int, uint32_t, const Pair64& p, bool) {
            if (!MULTI || P.type == POT_EAM) rho += table_rho64(P, p.r2);
        });
    rho = lane_sum<G>(rho);
    if (!in || lane) return;
    // an atom with tag 0 is untouched by the reference's charge stage; its F' is still defined
    if (live) A.nc[i] = rho;
    else rho = A.nc[i];
    for (int b = 0; b < ps->nkinds; ++b) {
        const PotParams& P = ps->p[ki][b];
        double EF = 0, dF = 0;
        if (P.type == POT_EAM) eam_embed64(P, rho, &EF, &dF, A.st);
        A.Fp64[(size_t)b * A.np + i] = dF;
    }
}

}  // namespace mdg
