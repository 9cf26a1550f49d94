// forces.cu — LJsCut and two-pass EAM force stages on the Verlet list.
//
// FP64 form: the reference's sums (LJs-cut.cxx:22-131, EAM.cxx:141-601) in FP64,
// with an arithmetic of fewer operations a pair (forces64_dev.cuh; the arrays' and
// single atoms' calls keep the reference's), including the Periodic boundary's ghost pass
// (boundary/periodic.cxx:36-102): listed pairs contribute with the raw
// difference r_j - r_i; for atoms flagged by Periodic::prepare_one, listed
// pairs at raw distance >= max(rns) contribute again through the shortest
// periodic image, as ghost copies at r_i + shortest(d).
//
// Mixed form: pair vectors come from FP32 offsets to the cell centres plus
// the image's cell offset stored in the list entry (minimum image, which is
// what the ghost pass produces whenever every periodic box edge is at least
// 2*rns), pair math and splines in FP32 (cubic coefficients per table
// interval), and per-atom sums with Kahan compensation.
//
// One thread or several lanes per atom over the ELL list (entry k of atom i at
// nbr[k*np+i]); an atom's sum is the one thread's, or its lanes' in a fixed order,
// so the per-atom sums need no atomics and are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "mdg_host.h"
#include "forces64_dev.cuh"
#include "forces_dev.cuh"
#include "integrate_dev.cuh"
#include "thermo_dev.cuh"

namespace mdg {

constexpr int kBlock64 = 128;  // threads per block of the FP64 pair passes

// ---------------------------------------------------------------------------
// FP64 spline pieces (EAM.cxx, same operation order)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double eam_rho64(const PotParams& P, double R1) {
    double RN = R1 * P.dr1;
    int N1 = (int)trunc(RN);
    if (N1 < P.Nr1) {
        double VR = N1;
        double DV = RN - VR;
        RN = R1 - VR * P.dr;
        VR = (P.Rho[N1 + 1] - P.Rho[N1]) * P.dr1;
        double aa = (P.dRho[N1 + 1] - VR) - (VR - P.dRho[N1]);
        double bb = aa - (VR - P.dRho[N1]);
        return P.Rho[N1] + RN * (P.dRho[N1] + DV * (DV * aa - bb));
    }
    return 0.0;
}

// Force(r)/r of one pair and the pair energy term V(r) (EAM.cxx:417-463).
__device__ __forceinline__ double eam_ff64(const PotParams& P, double R2, double AdF, double* Vr) {
    double R1 = sqrt(R2);
    double RN = R1 * P.dr1;
    int N1 = (int)trunc(RN);
    double FF, VR, DV;
    if (N1 < P.Nr1) {
        VR = N1;
        DV = RN - VR;
        RN = R1 - VR * P.dr;
        VR = (P.Rho[N1 + 1] - P.Rho[N1]) * P.dr1;
        double aa = (P.dRho[N1 + 1] - VR) - (VR - P.dRho[N1]);
        double bb = aa - (VR - P.dRho[N1]);
        FF = P.dRho[N1] + 2.0 * DV * (1.5 * DV * aa - bb);
        VR = (P.Vpar[N1 + 1] - P.Vpar[N1]) * P.dr1;
        aa = (P.dVpar[N1 + 1] - VR) - (VR - P.dVpar[N1]);
        bb = aa - (VR - P.dVpar[N1]);
        aa = aa * DV;
        VR = P.Vpar[N1] + RN * (P.dVpar[N1] + DV * (aa - bb));
        DV = P.dVpar[N1] + 2.0 * DV * (1.5 * aa - bb);
    } else {
        FF = 0.0;
        VR = 0.0;
        DV = 0.0;
    }
    if (Vr) *Vr = 0.5 * VR / R1;
    return (AdF * FF + (DV * R1 - VR) / R2) / R1;
}

// Force(r)/r of a tabulated Pair and its energy term V(r)/(2r)
// (pair.cxx:316-346, 228-314).
__device__ __forceinline__ double tab_ff64(const PotParams& P, double R2, double* Vr) {
    double R1 = sqrt(R2);
    double RN = R1 * P.dr1;
    int N1 = (int)trunc(RN);
    double VR = 0.0, DV = 0.0;
    if (N1 < P.Nr1) {
        VR = N1;
        DV = RN - VR;
        RN = R1 - VR * P.dr;
        VR = (P.Vpar[N1 + 1] - P.Vpar[N1]) * P.dr1;
        double aa = (P.dVpar[N1 + 1] - VR) - (VR - P.dVpar[N1]);
        double bb = aa - (VR - P.dVpar[N1]);
        aa = aa * DV;
        VR = P.Vpar[N1] + RN * (P.dVpar[N1] + DV * (aa - bb));
        DV = P.dVpar[N1] + 2.0 * DV * (1.5 * aa - bb);
    }
    if (Vr) *Vr = 0.5 * VR / R1;
    return ((DV * R1 - VR) / R2) / R1;
}

// LJs force / r (LJs.cxx:153-166) and energy term (LJs.cxx:90-101).
__device__ __forceinline__ double ljs_ff64(const PotParams& P, double r2, double* E) {
    const double X2min = 1.2599210498948732;
    double XX = P.ljs_rVr1 * r2 - X2min;
    double FV = P.ljs_rVr2 / r2;
    double Ur = FV * FV * FV;
    if (E) *E = P.ljs_aVr * (Ur * (Ur - 1.0) - (P.ljs_aLJ3 + P.ljs_bLJ2 * XX) * XX * XX);
    return P.ljs_aVr2 * (Ur * (Ur - 0.5) * FV + (P.ljs_aLJ + P.ljs_bLJ * XX) * XX);
}

__device__ __forceinline__ double lj_pref64(const PotParams& P, double r2) {
    double r2inv = 1.0 / r2;
    double r6inv = r2inv * r2inv * r2inv;
    return -0.5 * P.factor * (P.lj1 * r6inv - P.lj2) * r6inv * r2inv;
}

// ---- F'(nc) of the current densities, FP64 -----------------------------------
// The reference's force pass evaluates the embedding derivative from each
// atom's nc as it is (EAM.cxx:465-497); the FP64 force kernel reads it from
// Fp64, which the density pass writes. When nc changed since (prepare clears
// it, an upload replaces it, a rebuild permutes the atoms), this pass brings
// Fp64 back in line before a force pass.
template <bool MULTI>
__global__ void __launch_bounds__(kBlock) k_embed64(FArgs A, const PotSet* __restrict__ ps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const double nci = A.nc[i];
    const int ki = MULTI ? (A.kind[i] & 3) : 0;
    for (int b = 0; b < ps->nkinds; ++b) {
        const PotParams& P = ps->p[ki][b];
        double EF = 0, dF = 0;
        if (P.type == 2) eam_embed64(P, nci, &EF, &dF, A.st);
        A.Fp64[(size_t)b * A.np + i] = dF;
    }
}

// ---- pair and EAM forces, FP64 ------------------------------------------------
// HALF (half lists, verlet-list.cxx:345): the pair-type potentials push the
// pair force onto the neighbour as well (LJs-cut.cxx:57-62, pair.cxx:387-420,
// LJs.cxx:196-222); EAM uses the atom's half alone, as EAM::force does; the
// ghost pass acts on the atom alone (its ghost list is a full one,
// periodic.cxx:77-88). Both sides accumulate with atomics onto the outputs
// prepare cleared, as the reference's += does.
// FORM: the potential of every pair where there is one (POT_LJCUT, POT_EAM;
// Single), 0 = by kind pair. G lanes share an atom (with_lanes64).
template <bool MULTI, int FORM, bool HALF, int G>
__global__ void __launch_bounds__(kBlock64) k_forces64(FArgs A, const PotSet* __restrict__ ps) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = t % G;
    const bool live = t / G < A.n && A.tag[t / G] != 0;
    const int i = live ? t / G : 0;
    double f[3];
    forces64_lanes<MULTI, FORM, HALF, G>(A, ps, live, i, lane, f);
    if (!live || lane) return;
    if (HALF) {
        atomicAdd(&A.fx[i], f[0]);
        atomicAdd(&A.fy[i], f[1]);
        atomicAdd(&A.fz[i], f[2]);
    } else {
        A.fx[i] = f[0];
        A.fy[i] = f[1];
        A.fz[i] = f[2];
    }
}

// ---- EAM density + embedding derivative, FP64 ------------------------------
template <bool MULTI, int G>
__global__ void __launch_bounds__(kBlock64) k_density64(FArgs A, const PotSet* __restrict__ ps) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    density64_lanes<MULTI, G>(A, ps, t / G < A.n, t / G, t % G);
}

// ---- energies and virials, FP64 (LJs-cut.cxx:70-131, EAM.cxx:306-415,
// pair.cxx:228-314, LJs.cxx:103-151); HALF and FORM as for the forces above.
// The virial of a pair is symmetric: six sums.
template <bool MULTI, int FORM, bool HALF, int G>
__global__ void __launch_bounds__(kBlock64) k_virials64(FArgs A, const PotSet* __restrict__ ps) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = t % G;
    const bool live = t / G < A.n && A.tag[t / G] != 0;
    const int i = live ? t / G : 0;
    const int ki = MULTI && live ? (A.kind[i] & 3) : 0;
    double Ep = 0.0;
    double M[6] = {0, 0, 0, 0, 0, 0};  // xx yy zz xy xz yz
    // the kind whose embedding table gives Em: the last ghost's, else the
    // largest listed (both among EAM pairs); -1 and (entry, kind) codes
    int last_main = -1, last_ghost = -1;
    constexpr int kSym[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
    if (live)
        walk64<MULTI, G, !MULTI, true>(A, ps, i, ki, lane, [&](const PotParams& P, int kj, int k, bool ghost) {
            if (!MULTI || P.type != POT_EAM) return;
            if (ghost) last_ghost = 4 * k + kj;
            else last_main = max(last_main, kj);
        }, [&](const PotParams& P, int kj, uint32_t j, const Pair64& p, bool ghost) {
            const int type = FORM ? FORM : P.type;
            double E = 0.0, ff;
            if (type == POT_LJCUT) {
                ff = ljcut_ff64<true>(P, p.r2, E);
            } else if (type == POT_EAM) {
                const double AdF = A.Fp64[(size_t)ki * A.np + j] + A.Fp64[(size_t)kj * A.np + i];
                ff = table_ff64<true, true>(P, p.r2, AdF, E);
            } else if (type == POT_TAB) {
                ff = table_ff64<false, true>(P, p.r2, 0.0, E);
            } else if (type == POT_LJS) {
                ff = ljs_pair64<true>(P, p.r2, E);
            } else {
                return;
            }
            const double h = 0.5 * ff, hx = h * p.dx, hy = h * p.dy;
            Ep += E;
            if (HALF && !ghost && type != POT_EAM) {
                const double m[6] = {hx * p.dx, hy * p.dy, h * p.dz * p.dz, hx * p.dy, hx * p.dz, hy * p.dz};
                for (int q = 0; q < 6; ++q) M[q] += m[q];
                atomicAdd(&A.Ep[j], E);
                for (int k = 0; k < 9; ++k) atomicAdd(&A.V[k][j], m[kSym[k]]);
            } else {
                M[0] = fma(hx, p.dx, M[0]);
                M[1] = fma(hy, p.dy, M[1]);
                M[2] = fma(h * p.dz, p.dz, M[2]);
                M[3] = fma(hx, p.dy, M[3]);
                M[4] = fma(hx, p.dz, M[4]);
                M[5] = fma(hy, p.dz, M[5]);
            }
        });
    Ep = lane_sum<G>(Ep);
    for (int q = 0; q < 6; ++q) M[q] = lane_sum<G>(M[q]);
    if (MULTI) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            last_main = max(last_main, __shfl_xor_sync(0xffffffffu, last_main, o));
            last_ghost = max(last_ghost, __shfl_xor_sync(0xffffffffu, last_ghost, o));
        }
    }
    if (!live || lane) return;
    if (HALF) {
        atomicAdd(&A.Ep[i], Ep);
        for (int k = 0; k < 9; ++k) atomicAdd(&A.V[k][i], M[kSym[k]]);
    } else {
        A.Ep[i] = Ep;
        for (int k = 0; k < 9; ++k) A.V[k][i] = M[kSym[k]];
    }
    if (ps->any_eam) {
        const int last = last_ghost >= 0 ? last_ghost & 3 : last_main;
        const int kb = MULTI ? (last >= 0 ? last : ki) : 0;
        const PotParams& P = ps->p[ki][kb];
        double EF = 0.0, dF = 0.0;
        if (P.type == POT_EAM) {
            eam_embed64(P, A.nc[i], &EF, &dF, A.st);
            A.Em[i] = EF;
        }
    }
}

// Calls f(std::integral_constant<int, G>) with the lanes per atom of n atoms
// (kFewAtoms64).
template <typename F>
static void with_lanes64(size_t n, bool eam, F&& f) {
    if (n < kFewAtoms64) f(std::integral_constant<int, 32>());
    else if (n < some_atoms64(eam)) f(std::integral_constant<int, 16>());
    else if (n < 100000) f(std::integral_constant<int, 4>());
    else f(std::integral_constant<int, 1>());
}

static void launch_density64(const FArgs& A, const PotSet* dps, const PotSet& ps, cudaStream_t st) {
    with_lanes64(A.n, ps.any_eam != 0, [&](auto g) {
        constexpr int G = decltype(g)::value;
        const int nb = (int)(((size_t)A.n * G + kBlock64 - 1) / kBlock64);
        if (ps.multi) k_density64<true, G><<<nb, kBlock64, 0, st>>>(A, dps);
        else k_density64<false, G><<<nb, kBlock64, 0, st>>>(A, dps);
    });
}

static void launch_forces64(const FArgs& A, const PotSet* dps, const PotSet& ps, bool half, cudaStream_t st) {
    const int only = ps.multi ? 0 : ps.any_eam ? POT_EAM : ps.any_lj ? POT_LJCUT : 0;
    with_lanes64(A.n, ps.any_eam != 0, [&](auto g) {
        constexpr int G = decltype(g)::value;
        const int nb = (int)(((size_t)A.n * G + kBlock64 - 1) / kBlock64);
        if (half) {
            if (ps.multi) k_forces64<true, 0, true, G><<<nb, kBlock64, 0, st>>>(A, dps);
            else k_forces64<false, 0, true, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else if (ps.multi) {
            k_forces64<true, 0, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else if (only == POT_EAM) {
            k_forces64<false, POT_EAM, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else if (only == POT_LJCUT) {
            k_forces64<false, POT_LJCUT, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else {
            k_forces64<false, 0, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        }
    });
}

static void launch_virials64(const FArgs& A, const PotSet* dps, const PotSet& ps, bool half, cudaStream_t st) {
    const int only = ps.multi ? 0 : ps.any_eam ? POT_EAM : ps.any_lj ? POT_LJCUT : 0;
    with_lanes64(A.n, ps.any_eam != 0, [&](auto g) {
        constexpr int G = decltype(g)::value;
        const int nb = (int)(((size_t)A.n * G + kBlock64 - 1) / kBlock64);
        if (half) {
            if (ps.multi) k_virials64<true, 0, true, G><<<nb, kBlock64, 0, st>>>(A, dps);
            else k_virials64<false, 0, true, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else if (ps.multi) {
            k_virials64<true, 0, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else if (only == POT_EAM) {
            k_virials64<false, POT_EAM, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else if (only == POT_LJCUT) {
            k_virials64<false, POT_LJCUT, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        } else {
            k_virials64<false, 0, false, G><<<nb, kBlock64, 0, st>>>(A, dps);
        }
    });
}

// ---------------------------------------------------------------------------
// mixed precision (bodies in forces_dev.cuh)
// ---------------------------------------------------------------------------
// Blocks of 256 threads per SM the register budget must allow, measured on
// EAM Cu 1M atoms: the force pass is fastest at 4 (64 registers; 0.229 ms
// against 0.238 ms at 3), the density pass at 4 (0.154 ms against 0.177 ms
// at 3, 0.195 ms at 5, where it spills).
constexpr int kForceMinBlocks = 4;
constexpr int kDensityMinBlocks = 4;
// The Multi force bodies spill at 64 registers; three blocks per SM (up to 85
// registers) are fastest (NiAl B2 1M: 0.497 ms against 0.715 at four), while
// the density's fit (0.313 ms at four, 0.349 at three).
constexpr int kMultiMinBlocks = 3;
// MB = blocks of 256 threads per SM the register budget allows: a system's
// launch shape (mdg_system_set_shape, chosen by the project's autotuner),
// default as above.
template <bool MULTI, bool KICK, int MB>
__global__ void __launch_bounds__(kBlock, MB) k_lj_mixed(FArgs A, const PotSet* __restrict__ ps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.n) lj_mixed_one<MULTI, KICK>(A, ps, i);
}

// KINDS: 0 Single, 2 two kinds, 4 up to four (KindPots).
template <int KINDS, int MB>
__global__ void __launch_bounds__(kBlock, MB) k_density_rec(FArgs A, const PotSet* __restrict__ ps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.n) density_one<RhoGroup<KINDS, true>>(A, ps, i);
}

template <int KINDS, int MB>
__global__ void __launch_bounds__(kBlock, MB) k_density_mixed(FArgs A, const PotSet* __restrict__ ps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.n) density_one<RhoGroup<KINDS, false>>(A, ps, i);
}

template <int KINDS, bool KICK, int MB>
__global__ void __launch_bounds__(kBlock, MB) k_eam_mixed(FArgs A, const PotSet* __restrict__ ps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.n) eam_mixed_one<KINDS, KICK>(A, ps, i);
}

// The blocks-per-SM budget of a pass: the system's shape if set, else the
// measured default for its form.
static int force_blocks(const mdg_system* sys, bool multi) {
    return sys->shape[MDG_SHAPE_FORCE_BLOCKS_PER_SM] ? sys->shape[MDG_SHAPE_FORCE_BLOCKS_PER_SM]
                                                     : (multi ? kMultiMinBlocks : kForceMinBlocks);
}
static int density_blocks(const mdg_system* sys) {
    if (sys->shape[MDG_SHAPE_DENSITY_BLOCKS_PER_SM]) return sys->shape[MDG_SHAPE_DENSITY_BLOCKS_PER_SM];
    return kDensityMinBlocks;
}

template <int KINDS, bool KICK>
static void launch_eam(int mb, const FArgs& A, const PotSet* dps, int nb, cudaStream_t st) {
    if (mb == 3) k_eam_mixed<KINDS, KICK, 3><<<nb, kBlock, 0, st>>>(A, dps);
    else k_eam_mixed<KINDS, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
}

template <bool MULTI, bool KICK>
static void launch_lj(int mb, const FArgs& A, const PotSet* dps, int nb, cudaStream_t st) {
    if (mb == 3) k_lj_mixed<MULTI, KICK, 3><<<nb, kBlock, 0, st>>>(A, dps);
    else k_lj_mixed<MULTI, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
}

template <int KINDS>
static void launch_density(int mb, const FArgs& A, const PotSet* dps, int nb, cudaStream_t st) {
    if (mb == 3) k_density_mixed<KINDS, 3><<<nb, kBlock, 0, st>>>(A, dps);
    else if (mb == 5) k_density_mixed<KINDS, 5><<<nb, kBlock, 0, st>>>(A, dps);
    else k_density_mixed<KINDS, 4><<<nb, kBlock, 0, st>>>(A, dps);
}

template <int KINDS>
static void launch_rec(int mb, const FArgs& A, const PotSet* dps, int nb, cudaStream_t st) {
    if (mb == 3) k_density_rec<KINDS, 3><<<nb, kBlock, 0, st>>>(A, dps);
    else if (mb == 5) k_density_rec<KINDS, 5><<<nb, kBlock, 0, st>>>(A, dps);
    else k_density_rec<KINDS, 4><<<nb, kBlock, 0, st>>>(A, dps);
}

// Calls f(std::integral_constant<int, KINDS>) for a solver's kinds.
template <typename F>
static void with_kinds(const PotSet& ps, F&& f) {
    if (!ps.multi) f(std::integral_constant<int, 0>());
    else if (ps.nkinds <= 2) f(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, 4>());
}

template <bool MULTI, int FORM, bool KICK>
__global__ void __launch_bounds__(kBlock, kForceMinBlocks) k_pair_mixed(FArgs A, const PotSet* __restrict__ ps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.n) pair_mixed_one<MULTI, FORM, KICK>(A, ps, i);
}

// The end of a step's force pass for atom i (k_force_step): the second
// half-kick, and with `next` the next step's start; its rebuild test.
__device__ __forceinline__ bool end_step(const FArgs& A, const IArgs& D, const IArgs& to, int i, bool moved,
                                         bool next, const float f[3]) {
    if (!next) {
        if (moved) store_force<true>(A, i, f[0], f[1], f[2]);
        return false;
    }
    if (moved) return kick_drift_mixed(D, to, A.gx, A.gy, A.gz, i, f[0], f[1], f[2]);
    return drift_mixed_one(D, to, i);  // tag 0: the offsets and the test
}

// ---- eight lanes per atom: systems that do not fill the GPU ------------------
// A block is 256 threads = 32 atoms. The pair loops run with eight lanes per
// atom (lane_sums: the same sums in the same order as one thread's, so the
// same bits); the sums meet in shared memory and the block's first warp does
// the rest, a lane per atom, so that its FP64 instructions carry 32 atoms.
constexpr int kLaneAtoms = kBlock / 8;

template <typename Group>
__device__ __forceinline__ int block_forces(const FArgs& A, const PotSet* __restrict__ ps, float f[3]) {
    __shared__ __align__(kLaneAlign) float sh[kBlock / 32][96];
    __shared__ float sum[3][kLaneAtoms];
    const int a = threadIdx.x >> 3, i = blockIdx.x * kLaneAtoms + a;
    const bool in = i < A.n;
    lane_forces<Group>(A, ps, in, in ? i : 0, sh[threadIdx.x >> 5], f);
    if ((threadIdx.x & 7) == 0)
        for (int k = 0; k < 3; ++k) sum[k][a] = f[k];
    __syncthreads();
    if (threadIdx.x >= kLaneAtoms) return -1;
    for (int k = 0; k < 3; ++k) f[k] = sum[k][threadIdx.x];
    const int me = blockIdx.x * kLaneAtoms + threadIdx.x;
    return me < A.n ? me : -1;
}

// Blocks per SM of the lane kernels: four (64 registers) but for the two-kind
// bodies, which spill there.
constexpr int lane_budget(int kinds) { return kinds == 2 ? 3 : 4; }

template <typename Group, bool KICK, int MB>
__global__ void __launch_bounds__(kBlock, MB) k_lane_forces(FArgs A, const PotSet* __restrict__ ps) {
    float f[3];
    const int i = block_forces<Group>(A, ps, f);
    if (i >= 0 && A.tag[i] != 0) store_force<KICK>(A, i, f[0], f[1], f[2]);
}

template <int KINDS, bool REC>
__global__ void __launch_bounds__(kBlock, lane_budget(KINDS)) k_lane_density(FArgs A, const PotSet* __restrict__ ps) {
    __shared__ __align__(kLaneAlign) float sh[kBlock / 32][32];
    __shared__ float sum[kLaneAtoms];
    const int a = threadIdx.x >> 3, i = blockIdx.x * kLaneAtoms + a, w = i < A.n ? i : 0;
    const bool live = i < A.n && A.tag[w] != 0;
    float rho[1];
    RhoGroup<KINDS, REC> grp(A, ps, w);
    lane_sums<1>(A, live, w, live ? A.ncnt[w] >> 2 : 0, grp, sh[threadIdx.x >> 5], rho);
    if ((threadIdx.x & 7) == 0) sum[a] = rho[0];
    __syncthreads();
    const int me = blockIdx.x * kLaneAtoms + threadIdx.x;
    if (threadIdx.x < kLaneAtoms && me < A.n)
        store_density<(KINDS != 0)>(A, ps, me, A.pos32[me], KINDS ? (A.kind[me] & 3) : 0, sum[threadIdx.x]);
}

// k_force_step with eight lanes per atom.
template <int KINDS>
__global__ void __launch_bounds__(kBlock, lane_budget(KINDS))
    k_lane_force_step(FArgs A, IArgs D, const PotSet* __restrict__ ps, const unsigned long long* __restrict__ left) {
    const bool next = *left > 1ull && A.st->need_rebuild == 0u;
    float f[3];
    const int i = block_forces<EamGroup<KINDS, true>>(A, ps, f);
    if (threadIdx.x >= kLaneAtoms) return;
    const bool need = i >= 0 && end_step(A, D, D, i, A.tag[i] != 0, next, f);
    if (next) flag_need_next(need, A.st);
}

// Whether a system's mixed passes take eight lanes per atom: below 45,000
// atoms with several EAM tables, 30,000 with one, 24,000 without (a pair costs
// less there). One thread per atom leaves the GPU with fewer than nine warps
// per SM at 45,000 atoms; eight lanes cost about twice the instructions where
// it is full. Measured per step, one thread / eight lanes: EAM Cu 4,000 atoms
// 37.9 / 22.0 us, 32,000 39.9 / 41.1, 62,500 46.2 / 64.9; NiAl 31,094
// 92 / 75; LJ argon 4,000 25.6 / 20.6, 32,000 29.2 / 32.4; LJ liquid 62,500
// 37.1 / 48.9.
static bool lanes_mixed(const mdg_system* sys, const PotSet& ps) {
    return !sys->crowded && sys->n < (!ps.any_eam ? 24000u : ps.multi ? 45000u : 30000u);
}
static int lane_blocks(size_t n) { return (int)((n + kLaneAtoms - 1) / kLaneAtoms); }

// ---- Langevin thermostat (thermo_dev.cuh) -------------------------------------
template <bool MIXED>
__global__ void __launch_bounds__(kBlock) k_langevin(ThermoArgs A, const ThermoDev* __restrict__ th) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.n) langevin_one<MIXED>(A, th, i, A.st->therm_calls);
}

__global__ void k_thermo_tick(DevStatus* st) {
    if (threadIdx.x == 0) st->therm_calls += 1u;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static inline int nblk(size_t n, int b = kBlock) { return (int)((n + b - 1) / b); }

FArgs force_args(mdg_system* sys) {
    FArgs A;
    memset(&A, 0, sizeof(A));
    int c = sys->cur;
    A.n = (int)sys->n;
    A.np = (int)sys->np;
    A.rx = sys->f64[RX][c];
    A.ry = sys->f64[RY][c];
    A.rz = sys->f64[RZ][c];
    A.rns = sys->f64[RNS][c];
    A.nbr = sys->nbr;
    A.ncnt = sys->ncnt;
    A.kind = sys->u16[KIND][c];
    A.tag = sys->u16[TAG][c];
    A.bc = sys->bc;
    for (int a = 0; a < 3; ++a) {
        A.L[a] = sys->dom.bmax[a] - sys->dom.bmin[a];
        A.periodic[a] = sys->dom.periodic[a] ? 1 : 0;
        A.uf[a] = (float)(sys->grid.cs[a] / kOffUnits);
    }
    A.fx = sys->f64[FX][c];
    A.fy = sys->f64[FY][c];
    A.fz = sys->f64[FZ][c];
    A.gx = sys->f32[0][c];
    A.gy = sys->f32[1][c];
    A.gz = sys->f32[2][c];
    A.nc = sys->f64[NC][c];
    A.Fp64 = sys->Fp64;
    A.Fp32 = sys->Fp32;
    A.pos32 = sys->pos32;
    A.pos32b = sys->pos32 + sys->np;
    A.cutbits = nullptr;  // set by the passes of a step loop whose force pass moves atoms
    A.Ep = sys->f64[EP][c];
    A.Em = sys->f64[EM][c];
    for (int k = 0; k < 9; ++k) A.V[k] = sys->f64[V0 + k][c];
    A.st = sys->dstat;
    A.m = sys->f64[MASS][c];
    A.vx = sys->f64[VX][c];
    A.vy = sys->f64[VY][c];
    A.vz = sys->f64[VZ][c];
    A.kick_hdt = 0.0f;
    return A;
}

ThermoArgs thermo_args(mdg_system* sys) {
    const int c = sys->cur;
    ThermoArgs T;
    T.n = (int)sys->n;
    T.rx = sys->f64[RX][c];
    T.vx = sys->f64[VX][c];
    T.vy = sys->f64[VY][c];
    T.vz = sys->f64[VZ][c];
    T.m = sys->f64[MASS][c];
    T.orig = sys->u32[ORIG][c];
    T.fx = sys->f64[FX][c];
    T.fy = sys->f64[FY][c];
    T.fz = sys->f64[FZ][c];
    T.gx = sys->f32[0][c];
    T.gy = sys->f32[1][c];
    T.gz = sys->f32[2][c];
    T.st = sys->dstat;
    return T;
}

// Thermostat pass after the force stage (pair.cxx:81), then the call
// counter's increment.
static int launch_thermostat(mdg_system* sys, const ThermoDev* th, int precision) {
    mdg_ctx* ctx = sys->ctx;
    cudaStream_t st = ctx->stream;
    const ThermoArgs T = thermo_args(sys);
    const int nb = spread_blocks(sys->n), nt = spread_threads(sys->n);
    if (precision == MDG_PREC_FP64) k_langevin<false><<<nb, nt, 0, st>>>(T, th);
    else k_langevin<true><<<nb, nt, 0, st>>>(T, th);
    MDG_LAUNCHED(ctx);
    k_thermo_tick<<<1, 32, 0, st>>>(sys->dstat);
    MDG_LAUNCHED(ctx);
    return MDG_OK;
}

template <bool KICK>
static void launch_lane_forces(const FArgs& A, const PotSet* dps, const PotSet& ps, int nb, cudaStream_t st) {
    const bool multi = ps.multi != 0;
    if (ps.any_eam) {
        with_kinds(ps, [&](auto k) {
            constexpr int K = decltype(k)::value;
            k_lane_forces<EamGroup<K, false>, KICK, lane_budget(K)><<<nb, kBlock, 0, st>>>(A, dps);
        });
    } else if (ps.any_tab || ps.any_ljs) {
        if (!multi && ps.any_tab) k_lane_forces<PairGroup<false, 3>, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
        else if (!multi) k_lane_forces<PairGroup<false, 4>, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
        else k_lane_forces<PairGroup<true, 0>, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
    } else {
        if (multi) k_lane_forces<LjGroup<true>, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
        else k_lane_forces<LjGroup<false>, KICK, 4><<<nb, kBlock, 0, st>>>(A, dps);
    }
}

template <bool KICK>
static void launch_forces_mixed(const mdg_system* sys, const FArgs& A, const PotSet* dps, const PotSet& ps, int nb,
                                cudaStream_t st) {
    const bool multi = ps.multi != 0;
    const int mb = force_blocks(sys, multi);
    if (lanes_mixed(sys, ps)) {
        launch_lane_forces<KICK>(A, dps, ps, lane_blocks(sys->n), st);
    } else if (ps.any_eam) {
        with_kinds(ps, [&](auto k) { launch_eam<decltype(k)::value, KICK>(mb, A, dps, nb, st); });
    } else if (ps.any_tab || ps.any_ljs) {
        const int kinds = ps.any_lj + ps.any_tab + ps.any_ljs;
        if (!multi && ps.any_tab) k_pair_mixed<false, 3, KICK><<<nb, kBlock, 0, st>>>(A, dps);
        else if (!multi) k_pair_mixed<false, 4, KICK><<<nb, kBlock, 0, st>>>(A, dps);
        else if (kinds > 1) k_pair_mixed<true, 0, KICK><<<nb, kBlock, 0, st>>>(A, dps);
        else if (ps.any_tab) k_pair_mixed<true, 3, KICK><<<nb, kBlock, 0, st>>>(A, dps);
        else k_pair_mixed<true, 4, KICK><<<nb, kBlock, 0, st>>>(A, dps);
    } else {
        if (multi) launch_lj<true, KICK>(mb, A, dps, nb, st);
        else launch_lj<false, KICK>(mb, A, dps, nb, st);
    }
}

// ---- the force pass that starts the next step -----------------------------
// The step loop's EAM force pass (mixed form, no thermostat) with the step's
// second half-kick. When the next step can start in it — steps remain after
// this one (*left > 1) and no rebuild is due at this step's positions
// (need_rebuild, from the drift that made them) — every atom then also runs
// the next step's first half-kick, drift, offsets refresh and rebuild test
// (kick_drift_mixed; atoms with tag 0 only the last two), the test's result
// into need_next; otherwise the next drift runs as its own pass after the
// rebuild. The decision is the same for every thread. Moving atoms while
// others still read them is safe here because this pass reads its
// neighbours only through the density pass's copies (pos32b, Fp32) and takes
// each pair's cut decision from the density pass (cutbits), where the
// unfused pass would settle pairs near the cutoff on the FP64 positions.
//
// With one table the pass is bound by L1, so what it gains from packed pairs it
// can lose by gathers that come too close together (EAM Cu 1,000,188 atoms 220
// us before, 229 with packed pairs). Blocks of 128 threads, eight an SM, and the
// library's rsqrtf in place of the bare estimate (EamGroup; the same bits) space
// them again, 220 us: 229 with neither, 223 with the blocks, 225 with rsqrtf,
// 227 with unpacked pairs; 442,368 atoms 104 and 103. With several tables: 507
// us (NiAl 1,018,880), 511 with rsqrtf.
constexpr int kForceStepThreads = 128, kForceStepBlocks = 8;
template <int KINDS, int MB, int NT = kBlock>
__global__ void __launch_bounds__(NT, MB)
    k_force_step(FArgs A, IArgs D, const PotSet* __restrict__ ps, const unsigned long long* __restrict__ left) {
    const bool next = *left > 1ull && A.st->need_rebuild == 0u;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool need = false;
    if (i < A.n) {
        float f[3];
        const bool moved = thread_forces<EamGroup<KINDS, true>>(A, ps, i, f);
        need = end_step(A, D, D, i, moved, next, f);
    }
    if (next) flag_need_next(need, A.st);
}

// The LJ force pass of such a step. It reads its neighbours' own offsets (and
// the FP64 positions of pairs near the cutoff), so the moved atoms go to the
// other of two sets of arrays, which the loop's control kernel then takes for
// the current one (DevStatus::flip). The drift as a pass of its own read and
// wrote 190 bytes an atom again: LJ liquid 4,000,000 atoms 956 -> 877 us a
// step, 256,000 86.5 -> 81.0, the rebuilds' share included.
template <bool MULTI, int MB>
__global__ void __launch_bounds__(kBlock, MB)
    k_lj_step(FArgs A, IArgs D, const PosSet other, const PotSet* __restrict__ ps,
              const unsigned long long* __restrict__ left) {
    const bool next = *left > 1ull && A.st->need_rebuild == 0u;
    IArgs to = D;
    if (A.st->flip) {
        A.pos32 = other.pos32;
        A.rx = D.rx = other.rx;
        A.ry = D.ry = other.ry;
        A.rz = D.rz = other.rz;
    } else {
        to.pos32 = other.pos32;
        to.rx = other.rx;
        to.ry = other.ry;
        to.rz = other.rz;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool need = false;
    if (i < A.n) {
        float f[3];
        const bool moved = thread_forces<LjGroup<MULTI>>(A, ps, i, f);
        need = end_step(A, D, to, i, moved, next, f);
    }
    if (next) flag_need_next(need, A.st);
}

// The rest of a mixed step with a thermostat, after its force pass: the
// thermostat, the second half-kick and, as above, the next step's start. (As
// three passes, and one to count the call: EAM Cu 32,000 atoms 57.0 us a step,
// 54.0 as one.)
__global__ void __launch_bounds__(kBlock)
    k_thermo_step(ThermoArgs T, const ThermoDev* __restrict__ th, IArgs D, const unsigned long long* __restrict__ left) {
    const bool next = *left > 1ull && D.st->need_rebuild == 0u;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool need = false;
    if (i < T.n) {
        langevin_one<true>(T, th, i, T.st->therm_calls);
        kick_mixed_one(D, i);
        if (next) need = drift_mixed_one(D, D, i);
    }
    if (next) flag_need_next(need, D.st);
}

int launch_thermo_step(mdg_system* sys, const ThermoDev* th, double dt, const unsigned long long* left) {
    if (sys->n == 0) return MDG_OK;
    k_thermo_step<<<spread_blocks(sys->n), spread_threads(sys->n), 0, sys->ctx->stream>>>(
        thermo_args(sys), th, integrator_args(sys, dt), left);
    MDG_LAUNCHED(sys->ctx);
    return MDG_OK;
}

PosSet other_positions(mdg_system* sys) {
    const int o = sys->cur ^ 1;
    return PosSet{sys->f64[RX][o], sys->f64[RY][o], sys->f64[RZ][o], sys->pos32 + sys->np};
}

// Whether a step loop's LJ pass starts the next step: LJsCut alone, one thread
// per atom, with the GPU to itself.
bool lj_starts_next(const mdg_system* sys, const PotSet& ps) {
    return !sys->crowded && ps.any_lj && !ps.any_eam && !ps.any_tab && !ps.any_ljs && !lanes_mixed(sys, ps);
}

int launch_lj_step(mdg_system* sys, const PotSet* dps, const PotSet& ps, double dt, const unsigned long long* left) {
    if (sys->n == 0) return MDG_OK;
    FArgs A = force_args(sys);
    A.kick_hdt = 0.5f * (float)dt;
    const IArgs D = integrator_args(sys, dt);
    const PosSet other = other_positions(sys);
    const int nb = nblk(sys->n);
    cudaStream_t st = sys->ctx->stream;
    const bool three = force_blocks(sys, ps.multi != 0) == 3;
    if (ps.multi && three) k_lj_step<true, 3><<<nb, kBlock, 0, st>>>(A, D, other, dps, left);
    else if (ps.multi) k_lj_step<true, 4><<<nb, kBlock, 0, st>>>(A, D, other, dps, left);
    else if (three) k_lj_step<false, 3><<<nb, kBlock, 0, st>>>(A, D, other, dps, left);
    else k_lj_step<false, 4><<<nb, kBlock, 0, st>>>(A, D, other, dps, left);
    MDG_LAUNCHED(sys->ctx);
    return MDG_OK;
}

int launch_forces_step(mdg_system* sys, const PotSet* dps, const PotSet& ps, double dt,
                       const unsigned long long* left) {
    if (sys->n == 0) return MDG_OK;
    mdg_ctx* ctx = sys->ctx;
    FArgs A = force_args(sys);
    if (!ps.any_eam || !sys->cutbits || sys->cut_words * 32 < sys->K) {
        set_error("the step-starting force pass needs an EAM solver and the density pass's cut bits");
        return MDG_ERR_STATE;
    }
    A.cutbits = sys->cutbits;
    A.kick_hdt = 0.5f * (float)dt;
    const IArgs D = integrator_args(sys, dt);
    const int nb = nblk(sys->n);
    cudaStream_t st = ctx->stream;
    const bool multi = ps.multi != 0;
    const int mb = multi || sys->shape[MDG_SHAPE_FORCE_BLOCKS_PER_SM] ? force_blocks(sys, multi) : kForceStepBlocks;
    const int nb128 = nblk(sys->n, kForceStepThreads);
    with_kinds(ps, [&](auto k) {
        constexpr int K = decltype(k)::value;
        if (lanes_mixed(sys, ps)) k_lane_force_step<K><<<lane_blocks(sys->n), kBlock, 0, st>>>(A, D, dps, left);
        else if (mb == 3) k_force_step<K, 3><<<nb, kBlock, 0, st>>>(A, D, dps, left);
        else if (mb == kForceStepBlocks)
            k_force_step<K, kForceStepBlocks, kForceStepThreads><<<nb128, kForceStepThreads, 0, st>>>(A, D, dps, left);
        else k_force_step<K, 4><<<nb, kBlock, 0, st>>>(A, D, dps, left);
    });
    MDG_LAUNCHED(ctx);
    return MDG_OK;
}

// The density pass of a step whose force pass moves atoms (k_force_step):
// as the charge stage, recording the band pairs' FP64 decisions.
int launch_density_rec(mdg_system* sys, const PotSet* dps, const PotSet& ps) {
    if (sys->n == 0) return MDG_OK;
    FArgs A = force_args(sys);
    if (!sys->cutbits || sys->cut_words * 32 < sys->K) {
        set_error("the density pass's cut bits are not allocated");
        return MDG_ERR_STATE;
    }
    A.cutbits = sys->cutbits;
    const int nb = nblk(sys->n);
    cudaStream_t st = sys->ctx->stream;
    const int mb = density_blocks(sys);
    with_kinds(ps, [&](auto k) {
        constexpr int K = decltype(k)::value;
        if (lanes_mixed(sys, ps)) k_lane_density<K, true><<<lane_blocks(sys->n), kBlock, 0, st>>>(A, dps);
        else launch_rec<K>(mb, A, dps, nb, st);
    });
    MDG_LAUNCHED(sys->ctx);
    sys->fp_ok = 0;  // nc rewritten (FP32 sums); Fp64 no longer matches it
    return MDG_OK;
}

// The density pass's cut bits of a system (mdg_system::cutbits), sized for
// its list capacity; the force pass that starts the next step reads them.
int ensure_cutbits(mdg_system* sys) {
    const int words = (sys->K + 31) / 32;
    if (sys->cutbits && sys->cut_words >= words) return MDG_OK;
    sys_free(sys, sys->cutbits, (size_t)sys->cut_words * sys->np * sizeof(uint32_t));
    sys->cutbits = nullptr;
    sys->cut_words = 0;
    int rc = sys_malloc(sys, (void**)&sys->cutbits, (size_t)std::max(words, 1) * sys->np * sizeof(uint32_t));
    if (rc) return rc;
    sys->cut_words = std::max(words, 1);
    return MDG_OK;
}

// stage: 0 = charge (density), 1 = forces (then the thermostat, if any).
// kick_dt > 0 (mixed form, force stage, no thermostat): the step's second
// half-kick is applied in the force pass.
int launch_stage(mdg_system* sys, const PotSet* dps, const PotSet& ps, int precision, int stage,
                 const ThermoDev* th, double kick_dt) {
    mdg_ctx* ctx = sys->ctx;
    cudaStream_t st = ctx->stream;
    FArgs A = force_args(sys);
    int nb = nblk(sys->n);
    if (sys->n == 0) return MDG_OK;
    bool multi = ps.multi != 0;
    if (precision == MDG_PREC_FP64) {
        if (stage == 0) {
            launch_density64(A, dps, ps, st);
            sys->fp_ok = 1;
        } else {
            if (ps.any_eam && !sys->fp_ok) {
                if (multi) k_embed64<true><<<nb, kBlock, 0, st>>>(A, dps);
                else k_embed64<false><<<nb, kBlock, 0, st>>>(A, dps);
                MDG_LAUNCHED(ctx);
                sys->fp_ok = 1;
            }
            launch_forces64(A, dps, ps, sys->half != 0, st);
        }
    } else {
        if (stage == 0) {
            with_kinds(ps, [&](auto k) {
                constexpr int K = decltype(k)::value;
                if (lanes_mixed(sys, ps)) k_lane_density<K, false><<<lane_blocks(sys->n), kBlock, 0, st>>>(A, dps);
                else launch_density<K>(density_blocks(sys), A, dps, nb, st);
            });
            sys->fp_ok = 0;  // nc rewritten (FP32 sums); Fp64 no longer matches it
        } else if (kick_dt > 0.0 && !th) {
            A.kick_hdt = 0.5f * (float)kick_dt;
            launch_forces_mixed<true>(sys, A, dps, ps, nb, st);
        } else {
            launch_forces_mixed<false>(sys, A, dps, ps, nb, st);
        }
    }
    MDG_LAUNCHED(ctx);
    if (stage == 1 && th) return launch_thermostat(sys, th, precision);
    return MDG_OK;
}

int launch_virials(mdg_system* sys, const PotSet* dps, const PotSet& ps) {
    mdg_ctx* ctx = sys->ctx;
    if (sys->n == 0) return MDG_OK;
    FArgs A = force_args(sys);
    if (sys->half) {
        // accumulates onto the outputs: cleared first, as prepare leaves them
        int rc = launch_zero_meas(sys);
        if (rc) return rc;
    }
    launch_virials64(A, dps, ps, sys->half != 0, ctx->stream);
    MDG_LAUNCHED(ctx);
    return MDG_OK;
}

// ---------------------------------------------------------------------------
// Potential::value and EAM::embeddingEnergy on arrays (the analysis calls of
// python/mdcraft/solver/potential/_potential.cxx:88-168): the FP64 bodies of
// the force kernels. value: EAM.cxx:141-174 and pair.cxx:81-114 (V(r)/2r
// from the Vpar spline, 0 past the table, no cutoff test), LJs.cxx:61-71;
// LJsCut keeps Base::value (base.cxx:19): 0.
// ---------------------------------------------------------------------------

__global__ void k_pot_values(PotParams P, int n, const double* __restrict__ r2, double* __restrict__ u) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double e = 0.0;
    if (P.type == POT_EAM) eam_ff64(P, r2[i], 0.0, &e);
    else if (P.type == POT_TAB) tab_ff64(P, r2[i], &e);
    else if (P.type == POT_LJS) ljs_ff64(P, r2[i], &e);
    u[i] = e;
}

__global__ void k_pot_embedding(PotParams P, int n, const double* __restrict__ rho, double* __restrict__ F,
                                double* __restrict__ dF, DevStatus* st) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double EF = 0.0, d = 0.0;
    eam_embed64(P, rho[i], &EF, &d, st);
    F[i] = EF;
    dF[i] = d;
}

// ---- Potential::force / virial / density of one atom over an explicit list
// (the per-atom overloads of potential/base.h: LJs-cut.cxx:22-131,
// EAM.cxx:306-354, 465-497, 541-560). One thread walks the list in the
// reference's order with its FP64 arithmetic; recs[0] is the atom and
// slots[k] the record of list entry k. LJsCut with a half list pushes each
// pair's force, energy and virial onto the neighbour too; EAM ignores the
// half flag, as the reference does.
__global__ void k_pot_atom(PotParams P, int what, mdg_atom* recs, const uint32_t* __restrict__ slots, int count,
                           int half, DevStatus* st) {
    if (threadIdx.x != 0 || blockIdx.x != 0 || count == 0) return;
    mdg_atom& a = recs[0];
    const double x = a.r[0], y = a.r[1], z = a.r[2];
    if (P.type == POT_LJCUT) {
        double fx = 0.0, fy = 0.0, fz = 0.0;
        double Vxx = 0.0, Vyy = 0.0, Vzz = 0.0, Vxy = 0.0, Vxz = 0.0, Vyz = 0.0;
        for (int k = 0; k < count; ++k) {
            mdg_atom& nb = recs[slots[k]];
            const double dx = nb.r[0] - x, dy = nb.r[1] - y, dz = nb.r[2] - z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > P.R2cut || r2 < 1e-15) continue;
            const double pref = lj_pref64(P, r2);
            if (what == MDG_ATOM_FORCE) {
                fx += dx * pref;
                fy += dy * pref;
                fz += dz * pref;
                if (half) {
                    nb.f[0] -= dx * pref;
                    nb.f[1] -= dy * pref;
                    nb.f[2] -= dz * pref;
                }
            } else if (what == MDG_ATOM_VIRIAL) {
                const double ff[3] = {pref * dx, pref * dy, pref * dz}, d[3] = {dx, dy, dz};
                Vxx += ff[0] * dx;
                Vyy += ff[1] * dy;
                Vzz += ff[2] * dz;
                Vxy += ff[0] * dy;
                Vxz += ff[0] * dz;
                Vyz += ff[1] * dz;
                const double r2inv = 1.0 / r2;
                const double tmp = P.s6 * (r2inv * r2inv * r2inv);
                const double e = 0.5 * 4 * P.a * tmp * (tmp - 1);
                a.Ep += e;
                if (half) {
                    for (int c = 0; c < 3; ++c)
                        for (int r = 0; r < 3; ++r) nb.V[r + 3 * c] += 0.5 * (ff[r] * d[c]);
                    nb.Ep += e;
                }
            }
        }
        if (what == MDG_ATOM_FORCE) {
            a.f[0] += fx;
            a.f[1] += fy;
            a.f[2] += fz;
        } else if (what == MDG_ATOM_VIRIAL) {
            const double M[9] = {Vxx, Vxy, Vxz, Vxy, Vyy, Vyz, Vxz, Vyz, Vzz};
            for (int q = 0; q < 9; ++q) a.V[q] += 0.5 * M[q];
        }
        return;
    }
    if (P.type != POT_EAM) return;
    if (what == MDG_ATOM_DENSITY) {
        double sd = 0.0;
        for (int k = 0; k < count; ++k) {
            const mdg_atom& nb = recs[slots[k]];
            const double dx = nb.r[0] - x, dy = nb.r[1] - y, dz = nb.r[2] - z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > P.R2cut || r2 < 1e-15) continue;
            sd = sd + eam_rho64(P, sqrt(r2));
        }
        a.nc += sd;
        return;
    }
    // force and virial: F' of every listed neighbour's density and the atom's own
    double EFs = 0.0, dFs = 0.0;
    eam_embed64(P, a.nc, &EFs, &dFs, st);
    double F[3] = {0.0, 0.0, 0.0}, M[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, Ep = 0.0;
    for (int k = 0; k < count; ++k) {
        const mdg_atom& nb = recs[slots[k]];
        double EFj = 0.0, dFj = 0.0;
        eam_embed64(P, nb.nc, &EFj, &dFj, st);
        const double d[3] = {nb.r[0] - x, nb.r[1] - y, nb.r[2] - z};
        const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        if (r2 > P.R2cut || r2 < 1e-15) continue;
        double e = 0.0;
        const double FF = eam_ff64(P, r2, dFj + dFs, &e);
        if (what == MDG_ATOM_FORCE) {
            for (int q = 0; q < 3; ++q) F[q] += FF * d[q];
        } else {
            const double h = 0.5 * FF;
            for (int c = 0; c < 3; ++c)
                for (int r = 0; r < 3; ++r) M[r + 3 * c] += h * d[r] * d[c];
            Ep += e;
        }
    }
    if (what == MDG_ATOM_FORCE) {
        for (int q = 0; q < 3; ++q) a.f[q] += F[q];
    } else {
        a.Em = EFs;
        for (int q = 0; q < 9; ++q) a.V[q] += M[q];
        a.Ep += Ep;
    }
}

int pot_atom(const PotParams& P, int what, mdg_atom* recs_host, size_t nrec, const uint32_t* slots_host,
             size_t count, int half, cudaStream_t st, uint32_t* flags) {
    mdg_atom* d = nullptr;
    uint32_t* ds = nullptr;
    DevStatus* dst = nullptr;
    int rc = MDG_OK;
    cudaError_t e = cudaMalloc(&d, nrec * sizeof(mdg_atom));
    if (e == cudaSuccess) e = cudaMalloc(&ds, std::max<size_t>(count, 1) * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&dst, sizeof(DevStatus));
    if (e == cudaSuccess) e = cudaMemsetAsync(dst, 0, sizeof(DevStatus), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d, recs_host, nrec * sizeof(mdg_atom), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && count)
        e = cudaMemcpyAsync(ds, slots_host, count * sizeof(uint32_t), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        k_pot_atom<<<1, 32, 0, st>>>(P, what, d, ds, (int)count, half, dst);
        e = cudaGetLastError();
    }
    DevStatus hs;
    memset(&hs, 0, sizeof(hs));
    if (e == cudaSuccess) e = cudaMemcpyAsync(recs_host, d, nrec * sizeof(mdg_atom), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hs, dst, sizeof(DevStatus), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = cuda_status(e, "per-atom potential evaluation");
    if (flags) *flags = hs.flags;
    cudaFree(dst);
    cudaFree(ds);
    cudaFree(d);
    return rc;
}

// what = 0: u[k] = value(x[k]); what = 1: F, dF of density x[k]. Host arrays
// in and out through one device scratch block; waits on `st`.
int pot_eval(const PotParams& P, int what, const double* x, size_t n, double* out0, double* out1,
             cudaStream_t st) {
    if (n == 0) return MDG_OK;
    if (n > (size_t)INT32_MAX) {
        set_error("too many values in one call");
        return MDG_ERR_INVALID;
    }
    double* d = nullptr;
    DevStatus* ds = nullptr;
    MDG_CUDA(cudaMalloc(&d, 3 * n * sizeof(double)));
    int rc = MDG_OK;
    cudaError_t e = cudaMalloc(&ds, sizeof(DevStatus));
    if (e == cudaSuccess) e = cudaMemsetAsync(ds, 0, sizeof(DevStatus), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d, x, n * sizeof(double), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        if (what == 0) k_pot_values<<<nblk(n), kBlock, 0, st>>>(P, (int)n, d, d + n);
        else k_pot_embedding<<<nblk(n), kBlock, 0, st>>>(P, (int)n, d, d + n, d + 2 * n, ds);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out0, d + n, n * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && out1)
        e = cudaMemcpyAsync(out1, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = cuda_status(e, "potential evaluation");
    cudaFree(ds);
    cudaFree(d);
    return rc;
}

}  // namespace mdg
