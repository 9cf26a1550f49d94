// thermo_dev.cuh — the Langevin thermostat of one atom, shared by the
// thermostat pass (forces.cu) and the fused step loop (solo.cu).
#pragma once

#include <cuda_runtime.h>

#include "forces64_dev.cuh"
#include "mdg_internal.cuh"

namespace mdg {

// ---- Langevin thermostat (langevin.cxx:29-42) ----------------------------------
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11): ten rounds of two
// 32x32->64 multiplications, key bumped by the Weyl constants.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r > 0) {
            k.x += 0x9E3779B9u;
            k.y += 0xBB67AE85u;
        }
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    }
    return c;
}

// The thermostat needs two logarithms, two square roots, two cosines and a
// sine of 64 bits per atom; as library calls they are some 200 FP64
// instructions at 16 cycles each (EAM Cu 32,000 atoms: 14 us of a 64 us step).
// The arguments are 32-bit integers, so the ranges are reduced exactly by
// integer operations, and tables of 128 nodes with short series do the rest
// (P. T. P. Tang, Table-driven implementation of the logarithm function in
// IEEE floating-point arithmetic, ACM TOMS 16, 1990; the angle addition
// theorems for the other two). Errors are one or two units in the last place.

// log((b + 1/2) / 2^32): the number is 2^e m, its nearest node c = 1 + j / 128,
// log = e log 2 + log c + log1p(m / c - 1). Nodes from sqrt(2) up are halved
// (e one more), so that near 1 nothing cancels.
__device__ __forceinline__ double log_u32(const ThermoTables& T, uint32_t b) {
    const unsigned long long n = 2ull * b + 1ull;  // (b + 1/2) / 2^32 = n / 2^33
    const int lead = 63 - __clzll((long long)n);   // 0 .. 32
    const unsigned long long frac = n << (52 - lead) & 0xfffffffffffffull;
    const unsigned long long round = frac + (1ull << 44);  // to the nearest node; may carry to 2
    const int carry = (int)(round >> 52), j = (int)(round >> 45) & 127;
    // m in units of the node's power of two: [1, 2), or [1/2, 1) after a carry
    const double m = __longlong_as_double((long long)((unsigned long long)(1023 - carry) << 52 | frac));
    const int e = lead - 33 + carry + (j >= 53 ? 1 : 0);
    const double r = fma(m, __ldg(T.inv + j), -1.0);  // |r| <= 2^-8
    double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
    p = fma(r, p, 1.0 / 5.0);
    p = fma(r, p, -1.0 / 4.0);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -1.0 / 2.0);
    p = fma(r * r, p, r);
    return fma((double)e, 0.693147180559945309417, __ldg(T.log + j) + p);
}

// cos and sin of 2 pi (b + 1/2) / 2^32: the nearest node 2 pi j / 128 plus
// d = n 2 pi / 2^33, |d| <= pi / 128.
__device__ __forceinline__ void cos_sin_u32(const ThermoTables& T, uint32_t b, double& c, double& s) {
    const unsigned long long n = 2ull * b + 1ull;
    const uint32_t j = (uint32_t)((n + (1ull << 25)) >> 26);  // 0 .. 128
    const double d = (double)(int)((long long)n - ((long long)j << 26)) * 7.314590396335798e-10;  // 2 pi / 2^33
    const double2 node = __ldg(reinterpret_cast<const double2*>(T.cs[j & 127]));
    const double q = d * d;
    const double sd = fma(d * q, fma(q, fma(q, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), d);
    const double c1 = q * fma(q, fma(q, -1.0 / 720.0, 1.0 / 24.0), -0.5);  // cos d - 1
    c = node.x + fma(node.x, c1, -(node.y * sd));
    s = node.y + fma(node.y, c1, node.x * sd);
}

struct ThermoArgs {
    int n;
    const double *rx, *vx, *vy, *vz, *m;
    const uint32_t* orig;
    double *fx, *fy, *fz;  // FP64 form
    float *gx, *gy, *gz;   // mixed form
    const DevStatus* st;
};

// f += heat * (sqrt(m) * sigma * z - (v - U) * beta * m) for every term whose
// x range holds the atom; z = three Box-Muller normals of one Philox block
// with counter {caller index, call, term, 0}; call = the applications before
// this one (DevStatus::therm_calls).
template <bool MIXED>
__device__ __forceinline__ void langevin_one(const ThermoArgs& A, const ThermoDev* __restrict__ th, int i,
                                             uint32_t call) {
    const int nt = th->n;
    if (nt == 0) return;
    const double x = A.rx[i], m = A.m[i];
    const double v[3] = {A.vx[i], A.vy[i], A.vz[i]};
    const double sqrt_mass = sqrt(m);
    double f[3] = {0.0, 0.0, 0.0};
    if (!MIXED) {
        f[0] = A.fx[i];
        f[1] = A.fy[i];
        f[2] = A.fz[i];
    }
    const uint32_t atom = A.orig[i];
    for (int q = 0; q < nt && q < kMaxThermo; ++q) {
        const LangevinTerm& L = th->t[q];
        if (x < L.xmin || x > L.xmax) continue;
        const uint4 b = philox4x32_10(make_uint4(atom, call, (uint32_t)q, 0u),
                                      make_uint2((uint32_t)L.seed, (uint32_t)(L.seed >> 32)));
        const double xa = -2.0 * log_u32(th->tab, b.x), xb = -2.0 * log_u32(th->tab, b.z);
        float rf;
        const double ra = xa * rsqrt64(xa, rf), rb = xb * rsqrt64(xb, rf);
        double ca, sa, cb, sb;
        cos_sin_u32(th->tab, b.y, ca, sa);
        cos_sin_u32(th->tab, b.w, cb, sb);
        const double z[3] = {ra * ca, ra * sa, rb * cb};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double tf = __dmul_rn(__dadd_rn(__dmul_rn(z[k], L.sigma), 0.0), sqrt_mass);
            tf = __dsub_rn(tf, __dmul_rn(__dmul_rn(__dsub_rn(v[k], L.U[k]), L.beta), m));
            tf = __dmul_rn(tf, L.heat[k]);
            f[k] = __dadd_rn(f[k], tf);
        }
    }
    if (MIXED) {
        A.gx[i] += (float)f[0];
        A.gy[i] += (float)f[1];
        A.gz[i] += (float)f[2];
    } else {
        A.fx[i] = f[0];
        A.fy[i] = f[1];
        A.fz[i] = f[2];
    }
}

}  // namespace mdg

struct mdg_system;

namespace mdg {
// Argument block of a system's thermostat pass (forces.cu).
ThermoArgs thermo_args(mdg_system* sys);
}  // namespace mdg
