// forces_dev.cuh — per-atom bodies of the mixed-precision force stages,
// shared by the per-stage kernels (forces.cu) and the fused per-system loop
// (solo.cu), so both give the same forces bit for bit.
//
// LJsCut::compute / EAM::charge and forces (mdcraft/solver/potential/
// LJs-cut.cxx:22-131, EAM.cxx:141-601) in FP32 pair arithmetic on pair
// vectors taken exactly from fixed-point cell-centred offsets, with
// compensated per-atom sums.
#pragma once

#include <cuda_runtime.h>

#include "mdg_internal.cuh"

namespace mdg {

// A group of four list entries: streamed once per pass, so kept out of L1
// (the gathers of neighbour records and table rows keep it).
// RO (here and below): the data is read-only while the kernel runs, so the
// read-only path may serve it; the fused loops (solo.cu), whose own passes
// write it, take ordinary loads.
template <bool RO>
__device__ __forceinline__ uint4 ldg_list(const uint4* p) {
    uint4 v;
    if (RO)
        asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
            : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
            : "l"(p));
    else
        asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "l"(p));
    return v;
}
template <bool RO, typename T>
__device__ __forceinline__ T ld_ro(const T* p) {
    return RO ? __ldg(p) : *p;
}


struct FArgs {
    int n, np;
    const double *rx, *ry, *rz, *rns;
    const uint32_t *nbr, *ncnt;
    const uint16_t *kind, *tag;
    const uint8_t* bc;
    double L[3];
    int periodic[3];
    float uf[3];  // length of one fixed-point offset unit per axis, cs / 2^29 in FP32
    // outputs / intermediate
    double *fx, *fy, *fz;
    float *gx, *gy, *gz;  // mixed forces
    double* nc;
    double* Fp64;
    float* Fp32;
    const int4* pos32;  // fixed-point offsets (mdg_internal.cuh)
    int4* pos32b;       // the same offsets with w = bits of the FP32 F'(rho) (EAM)
    uint32_t* cutbits;  // null, or the density pass's FP64 decisions of band pairs (mdg_system::cutbits)
    double *Ep, *Em;
    double* V[9];
    DevStatus* st;
    // second half-kick fused into the force pass (mixed form): v += g * hdt / m
    const double* m;
    double *vx, *vy, *vz;
    float kick_hdt;  // 0.5f * (float)dt
};

// Stores the atom's FP32 force and, with KICK, applies the second half-kick
// exactly as kick_mixed_one does (same FP32 product, same rounding).
template <bool KICK>
__device__ __forceinline__ void store_force(const FArgs& A, int i, float fx, float fy, float fz) {
    A.gx[i] = fx;
    A.gy[i] = fy;
    A.gz[i] = fz;
    if (KICK) {
        const float hm = A.kick_hdt * __frcp_rn((float)A.m[i]);
        A.vx[i] += (double)(fx * hm);
        A.vy[i] += (double)(fy * hm);
        A.vz[i] += (double)(fz * hm);
    }
}

// ---------------------------------------------------------------------------
// mixed precision
// ---------------------------------------------------------------------------
__device__ __forceinline__ float ksum_add(float& s, float& c, float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
    return s;
}

// The pair vectors r_j - r_i of N list entries and their
// squares: from the fixed-point cell-centred offsets an exact integer
// difference (modulo 2^32; the true value is within +-2^31 units), one
// rounding to FP32, one scaling by the unit. The passes are bound by the
// instructions they issue (LJ liquid: 79% of the slots) or, with tables, by L1
// and those; so the FP32 arithmetic takes two pairs an instruction (the same
// roundings), and the own offsets come with one cell less (own_units), which
// makes an entry's image one shifted and masked word. With the cut test's one
// branch for several pairs (cut_pairs) and the bare hardware estimates
// (rcp_approx, rsqrt_approx): LJ liquid 4,000,000 atoms 0.675 -> 0.525 ms,
// EAM Cu 1,000,188 density 0.153 -> 0.135 (force: kForceStepThreads), NiAl
// 1,018,880 density 0.356 -> 0.332 and force 0.551 -> 0.506.
template <int N>
struct PairVecs {
    float x[N], y[N], z[N], r2[N];
};
__device__ __forceinline__ int4 own_units(const int4& p) {
    const uint32_t cell = 1u << kOffBits;
    return make_int4((int)((uint32_t)p.x + cell), (int)((uint32_t)p.y + cell), (int)((uint32_t)p.z + cell), p.w);
}
template <int N>
__device__ __forceinline__ PairVecs<N> pair_vecs(const uint32_t e[N], const int4& pi, const int4 pj[N],
                                                 const float uf[3]) {
    PairVecs<N> v;
#pragma unroll
    for (int q = 0; q < N; q += 2) {
        unsigned long long d[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const uint32_t i = a == 0 ? pi.x : a == 1 ? pi.y : pi.z;
            const uint32_t j0 = a == 0 ? pj[q].x : a == 1 ? pj[q].y : pj[q].z;
            const uint32_t j1 = a == 0 ? pj[q + 1].x : a == 1 ? pj[q + 1].y : pj[q + 1].z;
            d[a] = mul2(pack2(__int2float_rn((int)(j0 - i + image_units(e[q], a))),
                              __int2float_rn((int)(j1 - i + image_units(e[q + 1], a)))),
                        pack2(uf[a], uf[a]));
        }
        unpack2(d[0], v.x[q], v.x[q + 1]);
        unpack2(d[1], v.y[q], v.y[q + 1]);
        unpack2(d[2], v.z[q], v.z[q + 1]);
        unpack2(fma2(d[0], d[0], fma2(d[1], d[1], mul2(d[2], d[2]))), v.r2[q], v.r2[q + 1]);
    }
    return v;
}

// Hardware estimates of 1/x and 1/sqrt(x), x a normal number: all that a
// squared distance of at least 1e-12 needs (__fdividef and rsqrtf, the same
// bits there, also carry subnormal numbers).
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 1/sqrt(x) for x >= 1e-12: the hardware estimate refined by one Newton step, so
// r = x * rinv and 1/r are nearly correctly rounded (pair forces near an
// equilibrium lattice cancel, which magnifies their relative errors).
__device__ __forceinline__ float rsqrt_nr(float x) {
    const float y = rsqrt_approx(x);
    return y * fmaf(-0.5f * x * y, y, 1.5f);
}
// Of a pair of numbers.
__device__ __forceinline__ unsigned long long rsqrt_nr2(unsigned long long x, unsigned long long y) {
    return mul2(y, fma2(mul2(mul2(pack2(-0.5f, -0.5f), x), y), y, pack2(1.5f, 1.5f)));
}

// Both force rows (W, D) of one interval: 32 bytes, one 256-bit load
// (measured: EAM Cu 1M force pass 0.208 ms, against 0.216 ms with separate
// tables and 0.245 ms with two 128-bit loads of the interleaved rows).
__device__ __forceinline__ void load_rv(const float4* rv, int nn, float4& cw, float4& cd) {
    const float4* p = rv + 2 * nn;
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(cw.x), "=f"(cw.y), "=f"(cw.z), "=f"(cw.w), "=f"(cd.x), "=f"(cd.y), "=f"(cd.z), "=f"(cd.w)
        : "l"(p));
}

__device__ __forceinline__ float cubic(const float4 c, float u) {
    return fmaf(u, fmaf(u, fmaf(u, c.w, c.z), c.y), c.x);
}
__device__ __forceinline__ float dcubic(const float4 c, float u) {
    return fmaf(u, fmaf(u, 3.0f * c.w, 2.0f * c.z), c.y);
}

// Pair entries whose image crossed a periodic face contribute only with
// the Periodic boundary (without it the reference's raw distance is beyond
// the cutoff); bit 31 marks them.
constexpr uint32_t kWrapBit = 1u << 31;

// Cutoff membership of a pair. The FP32 r^2 decides unless it lies within
// 1e-5 (relative) of rc^2; those rare pairs are decided on the FP64
// positions, so the mixed form cuts exactly the pairs the FP64 form cuts
// (the potentials are discontinuous at rc, so a flipped pair would change
// forces by a whole pair term).
__device__ __forceinline__ bool cut_in(const FArgs& A, int i, uint32_t j, float r2, float r2c, double R2cut) {
    if (r2 < 1e-15f) return false;
    float band = 1e-5f * r2c;
    if (r2 < r2c - band) return true;
    if (r2 > r2c + band) return false;
    double dx = shortest1(A.rx[j] - A.rx[i], A.L[0], A.periodic[0]);
    double dy = shortest1(A.ry[j] - A.ry[i], A.L[1], A.periodic[1]);
    double dz = shortest1(A.rz[j] - A.rz[i], A.L[2], A.periodic[2]);
    return dx * dx + dy * dy + dz * dz <= R2cut;
}

// Cutoff membership from the FP32 r^2, with the rare pairs inside the
// 1e-5 band around rc^2 (and entries that crossed a periodic face when the
// solver has no Periodic boundary) settled exactly.
// (R2c() gives the FP64 cutoff, read only for those).
template <typename Cut>
__device__ __forceinline__ bool pair_in(const FArgs& A, int i, uint32_t e, float r2, float r2c, Cut&& R2c,
                                        bool per) {
    bool in = r2 >= 1e-15f && r2 <= r2c;
    if (fabsf(r2 - r2c) <= 1e-5f * r2c) in = cut_in(A, i, e & kJMask, r2, r2c, R2c());
    return in && (per || !(e & kWrapBit));
}

// pair_in for the density pass of a step whose force pass moves atoms: the
// FP64 decisions of the band pairs (entry k of atom i) are also collected in
// *bits, one bit per entry, and *band notes that the word has one.
template <typename Cut>
__device__ __forceinline__ bool pair_in_rec(const FArgs& A, int i, uint32_t e, float r2, float r2c, Cut&& R2c,
                                            bool per, int k, uint32_t* bits, bool* band) {
    bool in = r2 >= 1e-15f && r2 <= r2c;
    if (fabsf(r2 - r2c) <= 1e-5f * r2c) {
        in = cut_in(A, i, e & kJMask, r2, r2c, R2c());
        *bits |= (uint32_t)in << (k & 31);
        *band = true;
    }
    return in && (per || !(e & kWrapBit));
}

// pair_in for such a force pass: a band pair takes the density pass's FP64
// decision (the same FP32 r^2 puts it in the band there), so the pass reads
// no neighbour's FP64 position.
__device__ __forceinline__ bool pair_in_bits(const FArgs& A, int i, uint32_t e, float r2, float r2c, bool per,
                                             int k) {
    bool in = r2 >= 1e-15f && r2 <= r2c;
    if (fabsf(r2 - r2c) <= 1e-5f * r2c) in = (A.cutbits[(size_t)(k >> 5) * A.np + i] >> (k & 31)) & 1u;
    return in && (per || !(e & kWrapBit));
}

// pair_in of N pairs of one potential, with one branch for the
// rare band pairs: exact(q) settles pair q. [lo, hi] are the FP32 numbers
// within 1e-5 of rc^2 (cut_band).
__device__ __forceinline__ void cut_band(float r2c, float& lo, float& hi) {
    const float band = 1e-5f * r2c;
    lo = fminf(__fsub_ru(r2c, band), r2c);
    hi = __fadd_rd(r2c, band);
}
template <int N, typename Exact>
__device__ __forceinline__ void cut_pairs(const uint32_t e[N], const float r2[N], float lo, float hi, bool per,
                                          bool in[N], Exact&& exact) {
    bool band = false;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        in[q] = r2[q] >= 1e-15f && r2[q] < lo;
        band = band || (r2[q] >= lo && r2[q] <= hi);
    }
    if (band) {
#pragma unroll
        for (int q = 0; q < N; ++q)
            if (r2[q] >= lo && r2[q] <= hi) in[q] = exact(q);
    }
    if (!per) {
#pragma unroll
        for (int q = 0; q < N; ++q) in[q] = in[q] && !(e[q] & kWrapBit);
    }
}

// The pair loops below read four list entries with one 16-byte load, then
// the four neighbour records, so the loads of a group overlap; the four
// contributions are summed in FP32 and the group sum enters a Kahan sum, in
// the order of the groups. A body's state and its group are a struct
// (LjGroup, PairGroup, RhoGroup, EamGroup), walked by one thread per atom
// (group_sums) or by eight lanes per atom (lane_sums); both add the same
// group sums in the same order, so they give the same bits.

// One thread per atom: the sums of NC components over the atom's groups.
template <int NC, typename Group>
__device__ __forceinline__ void group_sums(const FArgs& A, int i, int ng, Group& grp, float out[NC]) {
    float s[NC], c[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) s[k] = c[k] = 0.f;
    const uint4* row = reinterpret_cast<const uint4*>(A.nbr) + i;
    uint4 e4n = ng > 0 ? ldg_list<Group::kRO>(row) : make_uint4(0, 0, 0, 0);
    for (int g = 0; g < ng; ++g) {
        // the next group's entries are requested before this group's work
        const uint4 e4 = e4n;
        if (g + 1 < ng) e4n = ldg_list<Group::kRO>(row + (size_t)(g + 1) * A.np);
        float f[NC];
        grp(A, i, g, e4, f);
#pragma unroll
        for (int k = 0; k < NC; ++k) ksum_add(s[k], c[k], f[k]);
        grp.word(A, i, g, ng);
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) out[k] = s[k];
}

// Eight lanes per atom (lane = threadIdx.x & 7; `live` false: no atom): lane l
// evaluates groups l, l + 8, ...; after each round of eight groups lane k adds
// the eight sums of component k in group order (through sh, 32 NC floats per
// warp, read by 16-byte words: on a kLaneAlign boundary, as every row of
// [warps][32 NC] is when the first is). Every lane of the warp calls this; out
// is the atom's sums, on all eight lanes. A group's sums take about 100
// instructions and the ordered additions 4 a group and component, so the eight
// lanes run about six times as fast as one where the GPU is not full.
constexpr int kLaneAlign = 16;
template <int NC, typename Group>
__device__ __forceinline__ void lane_sums(const FArgs& A, bool live, int i, int ng, Group& grp, float* sh,
                                          float out[NC]) {
    const int lane = threadIdx.x & 31, sub = lane & 7;
    if (!live) ng = 0;
    const uint4* row = reinterpret_cast<const uint4*>(A.nbr) + i;
    const int rounds = (__reduce_max_sync(0xffffffffu, (unsigned)ng) + 7) >> 3;
    uint4 e4n = sub < ng ? ldg_list<Group::kRO>(row + (size_t)sub * A.np) : make_uint4(0, 0, 0, 0);
    float s = 0.f, c = 0.f;  // component `sub` of this lane's atom
    for (int r = 0; r < rounds; ++r) {
        const int g = 8 * r + sub;
        const uint4 e4 = e4n;
        if (g + 8 < ng) e4n = ldg_list<Group::kRO>(row + (size_t)(g + 8) * A.np);
        float f[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) f[k] = 0.f;
        if (g < ng) grp(A, i, g, e4, f);
        grp.word8(A, i, r, g < ng);
#pragma unroll
        for (int k = 0; k < NC; ++k) sh[32 * k + lane] = f[k];
        __syncwarp();
        const float4* col = reinterpret_cast<const float4*>(sh + 32 * (sub < NC ? sub : 0) + (lane & ~7));
        const float4 lo = col[0], hi = col[1];
        const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (8 * r + q < ng) ksum_add(s, c, v[q]);
        __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) out[k] = __shfl_sync(0xffffffffu, s, (lane & ~7) + k);
}

template <bool MULTI, bool RO = true>
struct LjGroup {
    static constexpr bool kRO = RO;
    const PotSet* ps;
    int4 pi;
    int ki;
    bool per;
    float uf[3], lo, hi;
    unsigned long long l1, ml2, mh;  // Single: the potential's constants, twice each

    __device__ __forceinline__ LjGroup(const FArgs& A, const PotSet* __restrict__ p, int i) : ps(p) {
        pi = own_units(A.pos32[i]);
        ki = MULTI ? (A.kind[i] & 3) : 0;
        per = ps->periodic;
        for (int a = 0; a < 3; ++a) uf[a] = A.uf[a];
        if (MULTI) return;
        const PotParams& P0 = ps->p[ki][0];
        cut_band(P0.r2cut_f, lo, hi);
        l1 = pack2(P0.lj1_f, P0.lj1_f);
        ml2 = pack2(-P0.lj2_f, -P0.lj2_f);
        mh = pack2(P0.mhf_f, P0.mhf_f);
    }
    __device__ __forceinline__ void operator()(const FArgs& A, int i, int, const uint4& e4, float f[3]) {
        const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
        int4 pj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) pj[q] = ld_ro<RO>(A.pos32 + (e[q] & kJMask));
        const PairVecs<4> v = pair_vecs<4>(e, pi, pj, uf);
        float pref[4];
        if (MULTI) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const PotParams& P = ps->p[ki][pj[q].w & 3];
                const bool in = pair_in(A, i, e[q], v.r2[q], P.r2cut_f, [&] { return P.R2cut; }, per);
                const float r2inv = rcp_approx(fmaxf(v.r2[q], 1e-12f));
                const float r6inv = r2inv * r2inv * r2inv;
                pref[q] = in ? P.mhf_f * fmaf(P.lj1_f, r6inv, -P.lj2_f) * r6inv * r2inv : 0.f;
            }
        } else {
            bool in[4];
            cut_pairs<4>(e, v.r2, lo, hi, per, in, [&](int q) {
                const PotParams& P = ps->p[0][0];
                return cut_in(A, i, e[q] & kJMask, v.r2[q], P.r2cut_f, P.R2cut);
            });
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                const unsigned long long r2inv =
                    pack2(rcp_approx(fmaxf(v.r2[q], 1e-12f)), rcp_approx(fmaxf(v.r2[q + 1], 1e-12f)));
                const unsigned long long r6inv = mul2(mul2(r2inv, r2inv), r2inv);
                unpack2(mul2(mul2(mul2(mh, fma2(l1, r6inv, ml2)), r6inv), r2inv), pref[q], pref[q + 1]);
                pref[q] = in[q] ? pref[q] : 0.f;
                pref[q + 1] = in[q + 1] ? pref[q + 1] : 0.f;
            }
        }
        f[0] = f[1] = f[2] = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            f[0] = fmaf(v.x[q], pref[q], f[0]);
            f[1] = fmaf(v.y[q], pref[q], f[1]);
            f[2] = fmaf(v.z[q], pref[q], f[2]);
        }
    }
    __device__ __forceinline__ void word(const FArgs&, int, int, int) {}
    __device__ __forceinline__ void word8(const FArgs&, int, int, bool) {}
};

// The forces of atom i by a thread of its own; false for an atom with tag 0.
template <typename Group>
__device__ __forceinline__ bool thread_forces(const FArgs& A, const PotSet* __restrict__ ps, int i, float f[3]) {
    if (A.tag[i] == 0) return false;
    Group grp(A, ps, i);
    group_sums<3>(A, i, A.ncnt[i] >> 2, grp, f);
    return true;
}

// By eight lanes (every lane of the warp calls this; i < n where `in`).
template <typename Group>
__device__ __forceinline__ bool lane_forces(const FArgs& A, const PotSet* __restrict__ ps, bool in, int i, float* sh,
                                            float f[3]) {
    const bool live = in && A.tag[i] != 0;
    Group grp(A, ps, i);
    lane_sums<3>(A, live, i, live ? A.ncnt[i] >> 2 : 0, grp, sh, f);
    return live;
}

template <bool MULTI, bool KICK = false>
__device__ __forceinline__ void lj_mixed_one(const FArgs& A, const PotSet* __restrict__ ps, int i) {
    float f[3];
    if (thread_forces<LjGroup<MULTI>>(A, ps, i, f)) store_force<KICK>(A, i, f[0], f[1], f[2]);
}

// Force / r of a tabulated Pair term (pair.cxx:316-346) in FP32 from the
// cubic coefficients of its r*phi table: d(r phi)/dr * r - r phi, over r^3.
__device__ __forceinline__ float tab_ff32(const PotParams& P, float r2, bool& in) {
    const float rinv = rsqrt_nr(fmaxf(r2, 1e-12f));
    const float r = r2 * rinv;
    const float t = r * P.inv_dr_f;
    int nn = (int)t;
    in = in && nn < P.Nr1;
    nn = in ? nn : 0;
    const float u = t - (float)nn;
    const float4 cv = __ldg(P.v_c + nn);
    const float V = cubic(cv, u);
    const float dV = dcubic(cv, u) * P.inv_dr_f;
    return (dV * r - V) * (rinv * rinv) * rinv;
}

__device__ __forceinline__ float lj_ff32(const PotParams& P, float r2) {
    const float r2inv = rcp_approx(fmaxf(r2, 1e-12f));
    const float r6inv = r2inv * r2inv * r2inv;
    return P.mhf_f * fmaf(P.lj1_f, r6inv, -P.lj2_f) * r6inv * r2inv;
}

// Force / r of an LJs pair (LJs.cxx:153-166) in FP32.
__device__ __forceinline__ float ljs_ff32(const PotParams& P, float r2) {
    const float XX = fmaf(P.ljs_rVr1_f, r2, -1.2599210498948732f);
    const float FV = P.ljs_rVr2_f * rcp_approx(fmaxf(r2, 1e-12f));
    const float Ur = FV * FV * FV;
    return P.ljs_aVr2_f * fmaf(Ur * (Ur - 0.5f), FV, fmaf(P.ljs_bLJ_f, XX, P.ljs_aLJ_f) * XX);
}

// Force / r of an analytic pair potential by type (LJsCut or LJs).
__device__ __forceinline__ float analytic_ff32(const PotParams& P, float r2) {
    return P.type == POT_LJS ? ljs_ff32(P, r2) : lj_ff32(P, r2);
}

// Pair-type forces (no EAM term) beyond the plain LJsCut kernel: FORM 3 =
// every pair a tabulated Pair, 4 = every pair LJs, 0 = chosen per kind pair
// among LJsCut, Pair and LJs.
template <bool MULTI, int FORM, bool RO = true>
struct PairGroup {
    static constexpr bool kRO = RO;
    const PotSet* ps;
    int4 pi;
    int ki;
    bool per;
    float uf[3];

    __device__ __forceinline__ PairGroup(const FArgs& A, const PotSet* __restrict__ p, int i) : ps(p) {
        pi = own_units(A.pos32[i]);
        ki = MULTI ? (A.kind[i] & 3) : 0;
        per = ps->periodic;
        for (int a = 0; a < 3; ++a) uf[a] = A.uf[a];
    }
    __device__ __forceinline__ void operator()(const FArgs& A, int i, int, const uint4& e4, float f[3]) {
        const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
        int4 pj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) pj[q] = ld_ro<RO>(A.pos32 + (e[q] & kJMask));
        const PairVecs<4> v = pair_vecs<4>(e, pi, pj, uf);
        float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const PotParams& P = ps->p[ki][MULTI ? (pj[q].w & 3) : 0];
            const float dx = v.x[q], dy = v.y[q], dz = v.z[q], r2 = v.r2[q];
            bool in = pair_in(A, i, e[q], r2, P.r2cut_f, [&] { return P.R2cut; }, per);
            float FF;
            if (FORM == 3 || (FORM == 0 && P.type == POT_TAB)) {
                FF = tab_ff32(P, r2, in);
            } else if (FORM == 4) {
                FF = ljs_ff32(P, r2);
            } else {
                in = in && (P.type == POT_LJCUT || P.type == POT_LJS);
                FF = analytic_ff32(P, r2);
            }
            FF = in ? FF : 0.f;
            fx = fmaf(dx, FF, fx);
            fy = fmaf(dy, FF, fy);
            fz = fmaf(dz, FF, fz);
        }
        f[0] = fx;
        f[1] = fy;
        f[2] = fz;
    }
    __device__ __forceinline__ void word(const FArgs&, int, int, int) {}
    __device__ __forceinline__ void word8(const FArgs&, int, int, bool) {}
};

template <bool MULTI, int FORM, bool KICK = false>
__device__ __forceinline__ void pair_mixed_one(const FArgs& A, const PotSet* __restrict__ ps, int i) {
    float f[3];
    if (thread_forces<PairGroup<MULTI, FORM>>(A, ps, i, f)) store_force<KICK>(A, i, f[0], f[1], f[2]);
}

__device__ __forceinline__ void embed32(const PotParams& P, float rho, float* F, float* dF,
                                        DevStatus* st) {
    float t = rho * P.inv_drh_f;
    if (!(t >= 0.0f) || t >= (float)(P.Nrh1 - 1)) {
        atomicOr(&st->flags, FLAG_TABLE);
        t = fminf(fmaxf(t, 0.0f), (float)(P.Nrh1 - 1) - 1e-3f);
    }
    int nn = (int)t;
    float u = t - (float)nn;
    float4 c = __ldg(P.f_c + nn);
    *F = cubic(c, u);
    *dF = dcubic(c, u) * P.inv_drh_f;
}

// What the EAM passes need of a pair's potential, by the partner's kind.
// KINDS = 0: Single (read once per atom); 2: two kinds, both read once per
// atom and selected per pair; 4: read from the PotSet per pair. (The Multi
// passes are bound by L1 as well, and the five reads per pair took as many
// wavefronts as the pair's own gathers: NiAl B2 1M force pass 0.687 ->
// 0.551 ms, density 0.421 -> 0.355 ms.)
struct PairPot {
    float r2c, idr;
    int Nr1;
    const float4* tab;
    bool eam, lj;
};
template <int KINDS, bool FORCE>
struct KindPots {
    float r2c[2], idr[2];
    int Nr1[2];
    const float4* tab[2];
    unsigned eam, lj;  // bit per kind

    static __device__ __forceinline__ const float4* table(const PotParams& P) { return FORCE ? P.rv_c : P.rho_c; }
    // a tabulated Pair has zero rho rows: the EAM force arithmetic reduces to
    // its pair term exactly
    static __device__ __forceinline__ bool is_eam(int type) {
        return type == POT_EAM || (FORCE && type == POT_TAB);
    }
    static __device__ __forceinline__ bool is_lj(int type) {
        return FORCE && (type == POT_LJCUT || type == POT_LJS);
    }
    __device__ __forceinline__ void set(const PotSet* ps, int ki) {
        eam = lj = 0;
        if (KINDS == 4) return;
        for (int b = 0; b < (KINDS ? 2 : 1); ++b) {
            const PotParams& P = ps->p[KINDS ? ki : 0][b];
            r2c[b] = P.r2cut_f;
            idr[b] = P.inv_dr_f;
            Nr1[b] = P.Nr1;
            tab[b] = table(P);
            if (KINDS) {
                eam |= is_eam(P.type) ? 1u << b : 0u;
                lj |= is_lj(P.type) ? 1u << b : 0u;
            }
        }
    }
    __device__ __forceinline__ PairPot get(const PotSet* ps, int ki, int kj) const {
        if (KINDS == 4) {
            const PotParams& P = ps->p[ki][kj];
            return PairPot{P.r2cut_f, P.inv_dr_f, P.Nr1, table(P), is_eam(P.type), is_lj(P.type)};
        }
        if (KINDS == 2) {
            const bool one = kj & 1;  // a kind beyond the two has no potential (its bits are clear)
            return PairPot{one ? r2c[1] : r2c[0], one ? idr[1] : idr[0], one ? Nr1[1] : Nr1[0],
                           one ? tab[1] : tab[0], ((eam >> kj) & 1u) != 0u, FORCE && ((lj >> kj) & 1u) != 0u};
        }
        return PairPot{r2c[0], idr[0], Nr1[0], tab[0], true, false};
    }
};

// REC: also record the FP64 decisions of the band pairs in A.cutbits, for a
// force pass that moves atoms (pair_in_rec): one bit per entry, a word of 32
// stored when it has a band pair.
template <int KINDS, bool REC, bool RO = true>
struct RhoGroup {
    static constexpr bool kRO = RO;
    static constexpr bool MULTI = KINDS != 0;
    const PotSet* ps;
    int4 pi;
    int ki;
    bool per, band = false;
    float uf[3], lo, hi;
    KindPots<KINDS, false> pots;
    uint32_t bits = 0;  // FP64 cut decisions of this word's band entries

    __device__ __forceinline__ RhoGroup(const FArgs& A, const PotSet* __restrict__ p, int i) : ps(p) {
        pi = own_units(A.pos32[i]);
        ki = MULTI ? (A.kind[i] & 3) : 0;
        per = ps->periodic;
        for (int a = 0; a < 3; ++a) uf[a] = A.uf[a];
        pots.set(ps, ki);
        if (!MULTI) cut_band(pots.r2c[0], lo, hi);
    }
    __device__ __forceinline__ void operator()(const FArgs& A, int i, int g, const uint4& e4, float f[1]) {
        const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
        int4 pj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) pj[q] = ld_ro<RO>(A.pos32 + (e[q] & kJMask));
        const PairVecs<4> v = pair_vecs<4>(e, pi, pj, uf);
        bool in[4];
        if (!MULTI)
            cut_pairs<4>(e, v.r2, lo, hi, per, in, [&](int q) {
                const PotParams& P = ps->p[0][0];
                const bool settled = cut_in(A, i, e[q] & kJMask, v.r2[q], P.r2cut_f, P.R2cut);
                if (REC) {
                    bits |= (uint32_t)settled << ((4 * g + q) & 31);
                    band = true;
                }
                return settled;
            });
        float part = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            float t[2];
            if (!MULTI) {
                const float x0 = fmaxf(v.r2[q], 1e-12f), x1 = fmaxf(v.r2[q + 1], 1e-12f);
                const unsigned long long rinv = rsqrt_nr2(pack2(x0, x1), pack2(rsqrt_approx(x0), rsqrt_approx(x1)));
                unpack2(mul2(mul2(pack2(v.r2[q], v.r2[q + 1]), rinv), pack2(pots.idr[0], pots.idr[0])), t[0], t[1]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int o = q + h;
                const int kj = MULTI ? pj[o].w & 3 : 0;  // the partner's kind rides in its offsets' w
                const PairPot P = pots.get(ps, ki, kj);
                if (MULTI) {
                    auto R2c = [&] { return ps->p[ki][kj].R2cut; };
                    if (REC)  // every pair's band decision, whatever its potential
                        in[o] = pair_in_rec(A, i, e[o], v.r2[o], P.r2c, R2c, per, 4 * g + o, &bits, &band) && P.eam;
                    else
                        in[o] = P.eam && pair_in(A, i, e[o], v.r2[o], P.r2c, R2c, per);
                    t[h] = v.r2[o] * rsqrt_nr(fmaxf(v.r2[o], 1e-12f)) * P.idr;
                }
                int nn = (int)t[h];
                in[o] = in[o] && nn < P.Nr1;
                nn = in[o] ? nn : 0;
                const float u = t[h] - (float)nn;
                part += in[o] ? cubic(__ldg(P.tab + nn), u) : 0.f;
            }
        }
        f[0] = part;
    }
    __device__ __forceinline__ void word(const FArgs& A, int i, int g, int ng) {
        if (REC && ((g & 7) == 7 || g + 1 == ng)) {
            if (band) A.cutbits[(size_t)(g >> 3) * A.np + i] = bits;
            bits = 0;
            band = false;
        }
    }
    // eight lanes hold the word of round r
    __device__ __forceinline__ void word8(const FArgs& A, int i, int r, bool) {
        if (REC && __any_sync(0xffffffffu, band)) {
            unsigned any = band;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                bits |= __shfl_xor_sync(0xffffffffu, bits, o);
                any |= __shfl_xor_sync(0xffffffffu, any, o);
            }
            if (any && (threadIdx.x & 7) == 0) A.cutbits[(size_t)r * A.np + i] = bits;
            bits = 0;
            band = false;
        }
    }
};

// The atom's density rho from its sum, F'(rho) for its partners' kinds, and
// the record the force pass gathers.
template <bool MULTI>
__device__ __forceinline__ void store_density(const FArgs& A, const PotSet* __restrict__ ps, int i, const int4& pi,
                                              int ki, float rho) {
    // the atom's density as the reference's charge stage leaves it (FP32 sum here)
    if (A.tag[i] != 0) A.nc[i] = (double)rho;
    float Fp0 = 0.f;
    for (int b = 0; b < ps->nkinds; ++b) {
        const PotParams& P = ps->p[ki][b];
        float F = 0.f, dF = 0.f;
        if (P.type == 2) embed32(P, rho, &F, &dF, A.st);
        if (b == 0) Fp0 = dF;
        if (MULTI) A.Fp32[(size_t)b * A.np + i] = dF;
    }
    // Multi: the two lowest mantissa bits of F' (relative 2^-22, below the
    // FP32 sums' own rounding) carry the atom's kind for the force pass
    const int w = MULTI ? ((__float_as_int(Fp0) & ~3) | ki) : __float_as_int(Fp0);
    A.pos32b[i] = make_int4(pi.x, pi.y, pi.z, w);
}

template <typename Group>
__device__ __forceinline__ void density_one(const FArgs& A, const PotSet* __restrict__ ps, int i) {
    float rho[1] = {0.f};
    Group grp(A, ps, i);
    if (A.tag[i] != 0) group_sums<1>(A, i, A.ncnt[i] >> 2, grp, rho);
    store_density<Group::MULTI>(A, ps, i, A.pos32[i], grp.ki, rho[0]);
}

// BITS: a pair in the 1e-5 band around the cutoff takes the density pass's
// FP64 decision (A.cutbits) rather than testing the FP64 positions itself;
// the force pass then reads no FP64 position of a neighbour (what a force
// pass that moves its atoms needs).
template <int KINDS, bool BITS, bool RO = true>
struct EamGroup {
    static constexpr bool kRO = RO;
    static constexpr bool MULTI = KINDS != 0;
    const PotSet* ps;
    int4 pi;
    int ki;
    bool per;
    float uf[3], lo, hi;
    KindPots<KINDS, true> pots;
    // Multi: F' of atom i for the kinds 1..3 of its partners, read once (the
    // density pass's Fp32 rows; kind 0's is the record's w, with the atom's
    // kind in its two lowest bits)
    float fpi1 = 0.f, fpi2 = 0.f, fpi3 = 0.f;

    __device__ __forceinline__ EamGroup(const FArgs& A, const PotSet* __restrict__ p, int i) : ps(p) {
        pi = own_units(A.pos32b[i]);
        ki = MULTI ? (A.kind[i] & 3) : 0;
        per = ps->periodic;
        for (int a = 0; a < 3; ++a) uf[a] = A.uf[a];
        pots.set(ps, ki);
        if (!MULTI) cut_band(pots.r2c[0], lo, hi);
        if (MULTI) {
            const int nk = ps->nkinds;
            if (nk > 1) fpi1 = A.Fp32[A.np + i];
            if (KINDS == 4 && nk > 2) fpi2 = A.Fp32[2 * (size_t)A.np + i];
            if (KINDS == 4 && nk > 3) fpi3 = A.Fp32[3 * (size_t)A.np + i];
        }
    }
    __device__ __forceinline__ void operator()(const FArgs& A, int i, int g, const uint4& e4, float f[3]) {
        const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
        int4 pj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) pj[q] = ld_ro<RO>(A.pos32b + (e[q] & kJMask));
        float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            const PairVecs<2> v = pair_vecs<2>(e + q, pi, pj + q, uf);
            bool in[2];
            if (!MULTI)
                cut_pairs<2>(e + q, v.r2, lo, hi, per, in, [&](int h) {
                    const int k = 4 * g + q + h;
                    if (BITS) return ((A.cutbits[(size_t)(k >> 5) * A.np + i] >> (k & 31)) & 1u) != 0u;
                    const PotParams& P = ps->p[0][0];
                    return cut_in(A, i, e[q + h] & kJMask, v.r2[h], P.r2cut_f, P.R2cut);
                });
            // one reciprocal square root gives both r and 1/r
            const float x0 = fmaxf(v.r2[0], 1e-12f), x1 = fmaxf(v.r2[1], 1e-12f);
            // (with one table the pass is bound by L1, and the longer way to the
            // same estimate spaces its gathers: kForceStepThreads)
            const unsigned long long est = MULTI ? pack2(rsqrt_approx(x0), rsqrt_approx(x1))
                                                 : pack2(rsqrtf(x0), rsqrtf(x1));
            const unsigned long long rinv = rsqrt_nr2(pack2(x0, x1), est);
            const unsigned long long r = mul2(pack2(v.r2[0], v.r2[1]), rinv);
            float t[2], W[2], D[2], Fp[2], FF[2];
            if (MULTI) unpack2(r, t[0], t[1]);
            else unpack2(mul2(r, pack2(pots.idr[0], pots.idr[0])), t[0], t[1]);
            bool lj[2] = {false, false};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int o = q + h;
                float Fpi = __int_as_float(MULTI ? pi.w & ~3 : pi.w), Fpj = __int_as_float(MULTI ? pj[o].w & ~3 : pj[o].w);
                const int kj = MULTI ? pj[o].w & 3 : 0;
                const PairPot P = pots.get(ps, ki, kj);
                if (MULTI) {
                    // j's F' for i's kind (kind 0's is in j's record)
                    if (ki != 0) Fpj = A.Fp32[(size_t)ki * A.np + (e[o] & kJMask)];
                    Fpi = kj == 0 ? Fpi : KINDS == 2 || kj == 1 ? fpi1 : kj == 2 ? fpi2 : fpi3;
                    if (BITS)
                        in[h] = (P.eam || P.lj) && pair_in_bits(A, i, e[o], v.r2[h], P.r2c, per, 4 * g + o);
                    else
                        in[h] = (P.eam || P.lj) &&
                                pair_in(A, i, e[o], v.r2[h], P.r2c, [&] { return ps->p[ki][kj].R2cut; }, per);
                    t[h] *= P.idr;
                    lj[h] = P.lj;
                }
                int nn = (int)t[h];
                in[h] = in[h] && (P.lj || nn < P.Nr1);
                nn = in[h] && !P.lj ? nn : 0;
                const float u = t[h] - (float)nn;
                float4 cw, cd;
                load_rv(P.tab, nn, cw, cd);
                // W = V'r - V and D = rho' on the interval (force_rows)
                W[h] = cubic(cw, u);
                D[h] = fmaf(u, fmaf(u, cd.z, cd.y), cd.x);
                Fp[h] = Fpi + Fpj;
            }
            unpack2(mul2(fma2(pack2(Fp[0], Fp[1]), pack2(D[0], D[1]), mul2(pack2(W[0], W[1]), mul2(rinv, rinv))), rinv),
                    FF[0], FF[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int o = q + h;
                if (MULTI && lj[h]) FF[h] = analytic_ff32(ps->p[ki][pj[o].w & 3], v.r2[h]);
                FF[h] = in[h] ? FF[h] : 0.f;
                fx = fmaf(FF[h], v.x[h], fx);
                fy = fmaf(FF[h], v.y[h], fy);
                fz = fmaf(FF[h], v.z[h], fz);
            }
        }
        f[0] = fx;
        f[1] = fy;
        f[2] = fz;
    }
    __device__ __forceinline__ void word(const FArgs&, int, int, int) {}
    __device__ __forceinline__ void word8(const FArgs&, int, int, bool) {}
};

template <int KINDS, bool KICK = false>
__device__ __forceinline__ void eam_mixed_one(const FArgs& A, const PotSet* __restrict__ ps, int i) {
    float f[3];
    if (thread_forces<EamGroup<KINDS, false>>(A, ps, i, f)) store_force<KICK>(A, i, f[0], f[1], f[2]);
}

}  // namespace mdg

struct mdg_system;

namespace mdg {
// Argument block of a system's force stages (forces.cu).
FArgs force_args(mdg_system* sys);
}  // namespace mdg
