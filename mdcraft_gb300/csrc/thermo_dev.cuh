// thermo_dev.cuh — the Langevin thermostat of one atom, shared by the
// thermostat pass (forces.cu) and the fused step loop (solo.cu).
#pragma once

#include <cuda_runtime.h>

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
        const double k32 = 2.3283064365386962890625e-10;  // 2^-32
        const double two_pi = 6.283185307179586476925;
        const double ra = sqrt(-2.0 * log(((double)b.x + 0.5) * k32));
        const double rb = sqrt(-2.0 * log(((double)b.z + 0.5) * k32));
        const double a1 = two_pi * (((double)b.y + 0.5) * k32);
        const double a3 = two_pi * (((double)b.w + 0.5) * k32);
        const double z[3] = {ra * cos(a1), ra * sin(a1), rb * cos(a3)};
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
