// nlist_dev.cuh — device pieces of the linked-cell rebuild and the Verlet
// list build, shared by the per-stage kernels (nlist.cu) and the fused
// per-system loop (solo.cu) so both compute the same lists bit for bit.
//
// Grid::build / local_index3D / adjacent_cells (mdcraft/neibs/grid.cxx:43-207),
// Domain::fit_in_period (mdcraft/lattice/domain.cxx:41-47) and
// VerletList::build_linked_cells / are_neibs
// (mdcraft/neibs/verlet-list.cxx:306-400).
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "integrate_dev.cuh"
#include "mdg_host.h"
#include "mdg_internal.cuh"

namespace mdg {

// ---- bounds + wrap ----------------------------------------------------------
struct DomainDev {
    double bmin[3], bmax[3], size[3];
    int periodic[3];
    int dim;
};

// One axis of Grid::build (grid.cxx:43-95) from its reduced bounds and the
// largest rns (cell > 0); *small: the axis asks for the small-box build,
// *bad: too many cells.
__host__ __device__ inline void grid_axis(const DomainDev& d, double lo, double hi, double cell, int i,
                                          GridParams& g, bool* small, bool* bad) {
    g.bmin[i] = d.bmin[i];
    g.bmax[i] = d.bmax[i];
    g.size[i] = d.size[i];
    g.periodic[i] = d.periodic[i];
    g.dom_n[i] = 1;
    g.cs[i] = d.size[i];
    *small = *bad = false;
    if (!(cell > 0.0)) return;
    g.num[i] = 1;
    g.gmin[i] = d.bmin[i];
    if (i < d.dim) {
        const double q = floor(d.size[i] / cell);
        const int c = q > 1.0e9 ? 1000000000 : (int)q;
        g.dom_n[i] = c > 1 ? c : 1;
        g.cs[i] = d.size[i] / (double)g.dom_n[i];
        g.offset[i] = (int)floor((lo - d.bmin[i]) / g.cs[i]);
        const int u = (int)floor((hi - d.bmin[i]) / g.cs[i]) + 1;
        g.num[i] = (u < g.dom_n[i] ? u : g.dom_n[i]) - g.offset[i];
        g.gmin[i] = d.bmin[i] + g.cs[i] * g.offset[i];
    }
    g.bricks[i] = (g.num[i] + 3) / 4;
    g.csf[i] = (float)g.cs[i];
    g.Lf[i] = (float)d.size[i];
    g.inv_u[i] = g.cs[i] > 0.0 ? kOffUnits / g.cs[i] : 0.0;
    g.inv_cs[i] = g.cs[i] > 0.0 ? 1.0 / g.cs[i] : 0.0;
    // A periodic axis of 3 cells keeps the fast paths: its cells are at
    // least max rns wide (floor(L / rns) = 3), so every listed pair is
    // nearer than L / 2 and the image of its neighbour cell is the
    // minimum image (no per-pair adjustment, the FP32 prefilter holds).
    // One or two cells per axis (the reference's n = 1, 2 rules), or a
    // local grid short of the periodic box, take the per-atom body,
    // whose prefilter takes a per-pair minimum image.
    *small = d.periodic[i] && i < d.dim && (g.dom_n[i] <= 2 || g.offset[i] != 0 || g.num[i] != g.dom_n[i]);
    *bad = g.num[i] < 1 || g.num[i] > 1023;
}

// The grid's totals once its axes are set (g zeroed before them).
__host__ __device__ inline void grid_totals(const DomainDev& d, double cell, bool small, bool bad, GridParams& g) {
    g.dim = d.dim;
    g.max_rns = cell;
    if (!(cell > 0.0)) {
        g.empty = -1;
        return;
    }
    g.small_box = small ? 1 : 0;
    if (bad) g.empty = -2;
    const long long nc = (long long)g.num[0] * g.num[1] * g.num[2];
    const long long nb = 64LL * g.bricks[0] * g.bricks[1] * g.bricks[2];
    if (nb > (1LL << 30)) g.empty = -2;
    g.ncells = (int)nc;
    g.nbins = (int)nb;
}

// Grid::build from the reduced bounds and the largest rns; shared by the
// device rebuild (whose axes run on three lanes) and the host-side capacity
// sizing, so both get the same parameters bit for bit.
__host__ __device__ inline void grid_from_bounds(const DomainDev& d, const double lo[3], const double hi[3],
                                                 double cell, GridParams& g) {
    memset(&g, 0, sizeof(g));
    bool small = false, bad = false;
    for (int i = 0; i < 3; ++i) {
        bool s, b;
        grid_axis(d, i < d.dim ? lo[i] : 0.0, i < d.dim ? hi[i] : 0.0, cell, i, g, &s, &b);
        small = small || s;
        bad = bad || b;
    }
    grid_totals(d, cell, small, bad, g);
}

// floor(x / cs) with the quotient correctly rounded in FP64, as the
// reference's cell index takes it (grid.cxx). The product with the
// reciprocal 1/cs (itself rounded) lies within 1.5 * 2^-52 (relative) of the
// exact quotient, as does the rounded quotient, so the two have the same
// floor unless an integer lies within that distance of the product. Below
// 2^20 cells that distance is under 3.5e-10: a product within 1.1e-9 of an
// integer, below 2^-10 or beyond 2^20 takes the division instead. The floor
// and the fraction of the product come from its bits (FP64 comparisons and
// conversions run at the FP64 rate, one warp instruction in 16 cycles).
__device__ __forceinline__ int floor_div(double x, double cs, double inv_cs) {
    const long long b = __double_as_longlong(dmul(x, inv_cs));
    const int e = (int)(b >> 52);  // negative products: below 1013
    if (e >= 1013 && e < 1043) {
        const int sh = 1075 - e;   // 33 .. 62
        const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | 0x10000000000000ull;
        const uint32_t frac = (uint32_t)((m << (64 - sh)) >> 32);  // in units of 2^-32
        if (frac >= 5u && frac <= 0xfffffffau) return (int)(m >> sh);
    }
    return (int)floor(__ddiv_rn(x, cs));
}

__device__ __forceinline__ void local_cell(const GridParams& g, double x, double y, double z,
                                           int c[3], bool& clamped) {
    double r[3] = {x, y, z};
    clamped = false;
    for (int a = 0; a < 3; ++a) {
        int v = 0;
        if (a < g.dim) v = floor_div(dsub(r[a], g.bmin[a]), g.cs[a], g.inv_cs[a]) - g.offset[a];
        if (v < 0) { v = 0; clamped = true; }
        if (v >= g.num[a]) { v = g.num[a] - 1; clamped = true; }
        c[a] = v;
    }
}

__device__ inline uint32_t block_excl_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        sh[lane] = s;
    }
    __syncthreads();
    uint32_t base = w > 0 ? sh[w - 1] : 0u;
    uint32_t tot = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    if (total) *total = tot;
    return base + x - v;
}

template <int NF, typename T>
struct GatherSet {
    const T* in[NF];
    T* out[NF];
};

// Positions wrapped into the box on periodic axes (Domain::fit_in_period),
// written back; returns the wrapped position for the bounds.
__device__ __forceinline__ void wrap_one(const DomainDev& d, double* rx, double* ry, double* rz, int i,
                                         double v[3]) {
    double* r[3] = {rx, ry, rz};
    for (int a = 0; a < 3; ++a) {
        double x = r[a][i];
        if (d.periodic[a]) {
            double w = x < d.bmin[a] ? dadd(x, d.size[a]) : x > d.bmax[a] ? dsub(x, d.size[a]) : x;
            if (w != x) r[a][i] = w;
            x = w;
        }
        v[a] = x;
    }
}

// Bounds as integers that order like the doubles: a reduction over them runs
// on the integer pipe (FP64 minima and maxima, 7 values over 5 levels in every
// warp, took 7 to 13 us of a rebuild).
__device__ __forceinline__ long long double_key(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double key_double(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
// No atoms: +max, -max per axis, rns 0 (and a flag word, N = 8).
template <int N>
__device__ __forceinline__ void no_bounds(long long v[N]) {
    for (int k = 0; k < 3; ++k) {
        v[k] = double_key(1.7976931348623157e308);
        v[3 + k] = double_key(-1.7976931348623157e308);
    }
    for (int k = 6; k < N; ++k) v[k] = 0;
}
// An atom's position and rns; NaN counts for nothing, as in fmin and fmax.
__device__ __forceinline__ void add_bounds(long long* v, const double x[3], double rns) {
    const long long inf = 0x7ff0000000000000LL;
    for (int a = 0; a < 3; ++a) {
        const long long b = __double_as_longlong(x[a]);
        if ((b & 0x7fffffffffffffffLL) > inf) continue;
        const long long k = double_key(x[a]);
        v[a] = min(v[a], k);
        v[3 + a] = max(v[3 + a], k);
    }
    const long long q = double_key(rns);
    if (q <= inf) v[6] = max(v[6], q);
}
template <int N>
__device__ __forceinline__ void warp_bounds(long long v[N]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const long long y = __shfl_down_sync(0xffffffffu, v[k], o);
            v[k] = k < 3 ? min(v[k], y) : max(v[k], y);
        }
}

// A packed cell with the atom's clamped flag in its top bit.
constexpr uint32_t kClampedCell = 1u << 31;

// Bin key of atom i, its arrival rank in the bin and its packed cell.
__device__ __forceinline__ void bin_count_one(const GridParams& g, int i, const double* rx, const double* ry,
                                              const double* rz, uint32_t* key, uint32_t* rank, uint32_t* cell,
                                              uint32_t* bin_count, DevStatus* st) {
    int c[3];
    bool cl;
    local_cell(g, rx[i], ry[i], rz[i], c, cl);
    if (cl) {
        atomicOr(&st->flags, FLAG_RANGE);
        atomicOr(&st->build_flags, FLAG_RANGE);
    }
    uint32_t k = (uint32_t)bin_key(g, c[0], c[1], c[2]);
    key[i] = k;
    rank[i] = atomicAdd(&bin_count[k], 1u);
    cell[i] = pack_cell(c[0], c[1], c[2]) | (cl ? kClampedCell : 0u);
}

// Slot of the atom that arrived k-th (src[k] = i) once every bin is ordered
// by caller index: its bin's start plus the number of smaller caller indices
// in the bin (orig_at: caller indices in arrival order).
__device__ __forceinline__ uint32_t sorted_slot(uint32_t k, uint32_t bin, const uint32_t* start,
                                                const uint32_t* orig_at) {
    const uint32_t s = start[bin], e = start[bin + 1], o = orig_at[k];
    uint32_t d = s;
    for (uint32_t m = s; m < e; ++m) d += orig_at[m] < o;
    return d;
}

// Cell centre, cell-relative FP32 offsets and packed cell of the atom in slot
// i, at r with packed cell `cell` (bin_count_one) and caller index o.
__device__ __forceinline__ void cells_one(const GridParams& g, int i, const double r[3], uint32_t cell, uint32_t o,
                                          uint16_t kind, uint32_t* cellp, double* Rx, double* Ry, double* Rz,
                                          int4* pos32, int4* q0, float4* o0, uint32_t* slot_of) {
    const bool cl = (cell & kClampedCell) != 0;
    cell &= ~kClampedCell;
    cellp[i] = cell;
    int c[3];
    unpack_cell(cell, c[0], c[1], c[2]);
    double R[3];
    float of[3];
    int q[3];
    bool outlier = cl;
    for (int a = 0; a < 3; ++a) {
        R[a] = g.gmin[a] + ((double)c[a] + 0.5) * g.cs[a];
        if (a >= g.dim) R[a] = r[a];
        of[a] = (float)(r[a] - R[a]);
        q[a] = off_encode(r[a] - R[a], g.inv_u[a]);
        if (fabsf(of[a]) > 0.75f * g.csf[a] && a < g.dim) outlier = true;
    }
    Rx[i] = R[0];
    Ry[i] = R[1];
    Rz[i] = R[2];
    pos32[i] = make_int4(q[0], q[1], q[2], kind & 3);  // w: the atom's kind (Multi passes)
    q0[i] = make_int4(q[0], q[1], q[2], 0);
    // w: 0 exact offsets; 1 not exact (the FP32 tests send its pairs to FP64);
    // 2 clamped into the grid (also not exact: its list is walked from the
    // unclamped cell, nbuild_atom)
    o0[i] = make_float4(of[0], of[1], of[2], cl ? 2.0f : outlier ? 1.0f : 0.0f);
    slot_of[o] = (uint32_t)i;
}

// Every permuted field of one rebuild: the gathers into the spare buffers
// and the copies back.
struct GatherAll {
    GatherSet<12, double> a, b, a2, b2;
    GatherSet<3, float> fc, fc2;
    GatherSet<2, uint32_t> u, u2;
    GatherSet<2, uint16_t> h, h2;
};

// Every permuted field of atom i into slot d of the spare buffers.
__device__ __forceinline__ void permute_one(const GatherAll& G, uint32_t i, uint32_t d) {
    double x[12];
#pragma unroll
    for (int f = 0; f < 12; ++f) x[f] = G.a.in[f][i];
#pragma unroll
    for (int f = 0; f < 12; ++f) G.a.out[f][d] = x[f];
#pragma unroll
    for (int f = 0; f < 12; ++f) x[f] = G.b.in[f][i];
#pragma unroll
    for (int f = 0; f < 12; ++f) G.b.out[f][d] = x[f];
#pragma unroll
    for (int f = 0; f < 3; ++f) G.fc.out[f][d] = G.fc.in[f][i];
#pragma unroll
    for (int f = 0; f < 2; ++f) G.u.out[f][d] = G.u.in[f][i];
#pragma unroll
    for (int f = 0; f < 2; ++f) G.h.out[f][d] = G.h.in[f][i];
}

// The same by eight threads, `part` 0 .. 7 of them.
__device__ __forceinline__ void permute_part(const GatherAll& G, uint32_t i, uint32_t d, int part) {
    const bool more = part < 4;
    const double a = G.a.in[part][i], b = G.b.in[part][i];
    const double a8 = more ? G.a.in[part + 8][i] : 0.0, b8 = more ? G.b.in[part + 8][i] : 0.0;
    const float f = part < 3 ? G.fc.in[part][i] : 0.f;
    const uint32_t u = part == 3 || part == 4 ? G.u.in[part - 3][i] : 0u;
    const uint16_t h = part == 5 || part == 6 ? G.h.in[part - 5][i] : (uint16_t)0;
    G.a.out[part][d] = a;
    G.b.out[part][d] = b;
    if (more) G.a.out[part + 8][d] = a8;
    if (more) G.b.out[part + 8][d] = b8;
    if (part < 3) G.fc.out[part][d] = f;
    if (part == 3 || part == 4) G.u.out[part - 3][d] = u;
    if (part == 5 || part == 6) G.h.out[part - 5][d] = h;
}

struct CellOut {
    uint32_t* cellp;
    double *Rx, *Ry, *Rz;
    int4 *pos32, *q0;
    float4* o0;
    uint32_t* slot_of;
    float2* trig;
};

// The permuted fields of slot k back into the live buffers, and what follows
// from them.
__device__ __forceinline__ void settle_one(const GridParams& g, const GatherAll& G, int k, uint32_t cell,
                                           const CellOut& C) {
    double x[12];
#pragma unroll
    for (int f = 0; f < 12; ++f) x[f] = G.b2.in[f][k];
#pragma unroll
    for (int f = 0; f < 12; ++f) G.b2.out[f][k] = x[f];
#pragma unroll
    for (int f = 0; f < 3; ++f) G.fc2.out[f][k] = G.fc2.in[f][k];
    const uint32_t orig = G.u2.in[0][k];
    G.u2.out[0][k] = orig;
    G.u2.out[1][k] = G.u2.in[1][k];
    const uint16_t kind = G.h2.in[0][k];
    G.h2.out[0][k] = kind;
    G.h2.out[1][k] = G.h2.in[1][k];
#pragma unroll
    for (int f = 0; f < 12; ++f) x[f] = G.a2.in[f][k];
#pragma unroll
    for (int f = 0; f < 12; ++f) G.a2.out[f][k] = x[f];
    const double r[3] = {x[RX], x[RY], x[RZ]};
    cells_one(g, k, r, cell, orig, kind, C.cellp, C.Rx, C.Ry, C.Rz, C.pos32, C.q0, C.o0, C.slot_of);
    C.trig[k] = trig_of(x[RNS], x[RCUT], g);
}

// The same by eight threads.
__device__ __forceinline__ void settle_part(const GridParams& g, const GatherAll& G, int k, uint32_t cell,
                                            const CellOut& C, int part) {
    const bool more = part < 4, last = part == 7;
    const double a = G.a2.in[part][k], b = G.b2.in[part][k];
    const double a8 = more ? G.a2.in[part + 8][k] : 0.0, b8 = more ? G.b2.in[part + 8][k] : 0.0;
    const float f = part < 3 ? G.fc2.in[part][k] : 0.f;
    const uint32_t u = part == 3 || part == 4 ? G.u2.in[part - 3][k] : 0u;
    const uint16_t h = part == 5 || part == 6 ? G.h2.in[part - 5][k] : (uint16_t)0;
    double r[3] = {0.0, 0.0, 0.0}, rns = 0.0, rcut = 0.0;
    uint32_t orig = 0;
    uint16_t kind = 0;
    if (last) {
        for (int q = 0; q < 3; ++q) r[q] = G.a2.in[RX + q][k];
        rns = G.a2.in[RNS][k];
        rcut = G.a2.in[RCUT][k];
        orig = G.u2.in[0][k];
        kind = G.h2.in[0][k];
    }
    G.a2.out[part][k] = a;
    G.b2.out[part][k] = b;
    if (more) G.a2.out[part + 8][k] = a8;
    if (more) G.b2.out[part + 8][k] = b8;
    if (part < 3) G.fc2.out[part][k] = f;
    if (part == 3 || part == 4) G.u2.out[part - 3][k] = u;
    if (part == 5 || part == 6) G.h2.out[part - 5][k] = h;
    if (!last) return;
    cells_one(g, k, r, cell, orig, kind, C.cellp, C.Rx, C.Ry, C.Rz, C.pos32, C.q0, C.o0, C.slot_of);
    C.trig[k] = trig_of(rns, rcut, g);
}

// Systems (exclusive) whose lists are built by a warp per atom on every grid
// (nbuild_atom_cells).
constexpr int kAtomBuildMost = 8000;

struct NbArgs {
    int n, np, K, half;
    const double *rx, *ry, *rz, *rns, *rcut;
    const uint32_t *orig, *uid, *cellp, *bin_start;
    const float4* o0;
    uint32_t *nbr, *ncnt;
    double *r0x, *r0y, *r0z, *saved_rcut, *saved_rns;
    uint32_t* saved_uid;
    DevStatus* st;
};

// VerletList::are_neibs (verlet-list.cxx:373-400), FP64 without contraction.
__device__ __forceinline__ bool are_neibs_exact(const GridParams& g, double xa, double ya, double za,
                                                double ra, double xb, double yb, double zb, double rb,
                                                const bool edge[3]) {
    double dd = ra < rb ? rb : ra;
    double d2 = dmul(dd, dd);
    double drx = dsub(xa, xb), dry = dsub(ya, yb), drz = dsub(za, zb);
    double xs = g.size[0], ys = g.size[1], zs = g.size[2];
    if (edge[0] && g.periodic[0] && (2 * drx < -xs)) drx = dadd(drx, xs);
    if (edge[0] && g.periodic[0] && (2 * drx > xs)) drx = dsub(drx, xs);
    if (edge[1] && g.periodic[1] && (2 * dry < -ys)) dry = dadd(dry, ys);
    if (edge[1] && g.periodic[1] && (2 * dry > ys)) dry = dsub(dry, ys);
    if (edge[2] && g.periodic[2] && (2 * drz < -zs)) drz = dadd(drz, zs);
    if (edge[2] && g.periodic[2] && (2 * drz > zs)) drz = dsub(drz, zs);
    return sq3_exact(drx, dry, drz) <= d2;
}

// The grid covers every cell of each periodic axis (no local grid short of
// the box).
__host__ __device__ inline bool grid_whole(const GridParams& g) {
    for (int a = 0; a < g.dim; ++a)
        if (g.periodic[a] && (g.offset[a] != 0 || g.num[a] != g.dom_n[a])) return false;
    return true;
}

// Image code of a listed pair (list entry bits above kJBits): per axis the
// cell offset of j's image seen from i's cell (own), from the neighbour
// cell's offset dl, moved by a period on axes of 3 cells or fewer when the
// FP32 displacement (dx, dy, dz: i minus the neighbour cell's image of j)
// says the other image is nearer; bit 6 when the image crossed a periodic
// face (the offset differs from the local cells' difference lc - own).
__device__ __forceinline__ uint32_t pair_image_code(const GridParams& g, const int own[3], const int lc[3],
                                                    const int dl[3], float dx, float dy, float dz,
                                                    DevStatus* st) {
    uint32_t code = 0;
    for (int a = 0; a < 3; ++a) {
        int dlt = dl[a];
        if (g.periodic[a] && a < g.dim && g.dom_n[a] <= 3) {
            float dd = -(a == 0 ? dx : a == 1 ? dy : dz);
            float half = 0.5f * g.Lf[a];
            if (dd > half) dlt -= g.dom_n[a];
            else if (dd < -half) dlt += g.dom_n[a];
        }
        if (dlt < -1 || dlt > 1) {
            atomicOr(&st->flags, FLAG_IMAGE);
            dlt = dlt < -1 ? -1 : 1;
        }
        code |= (uint32_t)(dlt + 1) << (2 * a);
        if (dlt != lc[a] - own[a]) code |= 1u << 6;
    }
    return code;
}

// The nearest image of a displacement d on a periodic axis of length L,
// for |d| < 1.5 L (the offsets of binned atoms are within half a cell of
// their cell centres, so one shift suffices on axes of one or two cells).
__device__ __forceinline__ float min_image_f(float d, float L) {
    const float half = 0.5f * L;
    if (d > half) return d - L;
    if (d < -half) return d + L;
    return d;
}

// The end of atom i's list of cnt entries, by a warp (G = 32) or a thread (1):
// padding to a multiple of four with self entries, the counts and the rebuild
// snapshot.
template <int G>
__device__ __forceinline__ void end_list(const NbArgs& A, uint32_t i, int lane, int cnt) {
    const int padded = (cnt + 3) & ~3;
    if (G == 32) {
        if (cnt + lane < padded && cnt + lane < A.K) A.nbr[nidx(cnt + lane, i, A.np)] = i | kSelfCode;
    } else {
        for (int k = cnt; k < padded && k < A.K; ++k) A.nbr[nidx(k, i, A.np)] = i | kSelfCode;
    }
    if (lane) return;
    A.ncnt[i] = padded < A.K ? padded : A.K;
    if (cnt > A.K) {
        atomicOr(&A.st->flags, FLAG_OVERFLOW);
        atomicOr(&A.st->build_flags, FLAG_OVERFLOW);
    }
    atomicMax(&A.st->max_count, (uint32_t)cnt);
    A.r0x[i] = A.rx[i];
    A.r0y[i] = A.ry[i];
    A.r0z[i] = A.rz[i];
    A.saved_rcut[i] = A.rcut[i];
    A.saved_rns[i] = A.rns[i];
    A.saved_uid[i] = A.uid[i];
}

// The list of atom i, by a warp with its lanes over the candidates (G = 32) or by
// a thread (1): used for grids with a periodic axis of 2 cells or fewer and for
// local grids short of a periodic box (atoms_by_threads says which), and for
// atoms clamped into the grid. Its cell's 27 (or fewer, on small periodic axes)
// neighbour cells in the reference's order, x outer, z inner, each cell's atoms
// in slot order; accepted lanes append in lane order, so both give the same list.
// The FP32 prefilter also holds on periodic axes of one or two cells when the
// grid covers the whole box: every cell there is an edge cell, so the exact test
// takes the minimum image, and the FP32 minimum image of the neighbour cell's
// displacement is the same distance to ~1e-6 of r^2, inside the band that goes to
// FP64. A local grid short of the box keeps the FP64 test for every candidate.
// An atom clamped into the grid (a position on the upper face of a periodic
// axis after the wrap, or outside the grid) is binned in its clamped cell,
// but, as Grid::adjacent_cells (grid.cxx:138-207) takes the cell of the
// position itself, its own walk and edge flags come from the unclamped cell;
// the image codes stay relative to the cell it is binned in.
template <int G>
__device__ __forceinline__ void nbuild_atom(const NbArgs& A, const GridParams& g, uint32_t i, int lane,
                                            bool uniform_rns) {
    // prefilter band: rns^2 (1 -/+ 1e-5), valid when every atom has the same rns
    const float lo2 = (float)(g.max_rns * g.max_rns * (1.0 - 1e-5));
    const float hi2 = (float)(g.max_rns * g.max_rns * (1.0 + 1e-5));
    int cx, cy, cz;
    unpack_cell(A.cellp[i], cx, cy, cz);
    const int own[3] = {cx, cy, cz};
    const double xi = A.rx[i], yi = A.ry[i], zi = A.rz[i], rni = A.rns[i];
    const float4 oi = A.o0[i];
    // the walk's cell (global index) and its offset from the binned cell
    int gc[3] = {cx + g.offset[0], cy + g.offset[1], cz + g.offset[2]};
    int shift[3] = {0, 0, 0};
    if (oi.w == 2.0f) {
        const double r[3] = {xi, yi, zi};
        for (int a = 0; a < g.dim; ++a) {
            const int u = floor_div(dsub(r[a], g.bmin[a]), g.cs[a], g.inv_cs[a]);
            shift[a] = u - gc[a];
            gc[a] = u;
        }
    }
    if (g.dim < 3) gc[2] = 0;
    if (g.dim < 2) gc[1] = 0;
    bool edge[3] = {false, false, false};
    for (int a = 0; a < g.dim; ++a) edge[a] = gc[a] == 0 || gc[a] == g.num[a] - 1;
    bool mi[3] = {false, false, false};
    for (int a = 0; a < g.dim; ++a) mi[a] = g.periodic[a] && g.dom_n[a] <= 2;
    const bool prefilter = uniform_rns && grid_whole(g);
    const uint32_t origi = A.orig[i];
    const bool pfi = prefilter && oi.w == 0.0f;
    int cnt = 0;
    for (int x = -1; x <= 1; ++x) {
        if (g.periodic[0]) {
            if (g.dom_n[0] == 1 && x != 0) continue;
            if (g.dom_n[0] == 2 && x == 1) continue;
        }
        for (int y = -1; y <= 1; ++y) {
            if (g.periodic[1]) {
                if (g.dom_n[1] == 1 && y != 0) continue;
                if (g.dom_n[1] == 2 && y == 1) continue;
            }
            for (int z = -1; z <= 1; ++z) {
                if (g.periodic[2]) {
                    if (g.dom_n[2] == 1 && z != 0) continue;
                    if (g.dom_n[2] == 2 && z == 1) continue;
                }
                int lc[3];
                bool inside = true;
                for (int a = 0; a < 3; ++a) {
                    // the walk's cell is within one cell of the grid, so one period at most
                    int nb = gc[a] + (a == 0 ? x : a == 1 ? y : z);
                    if (g.periodic[a]) nb = nb < 0 ? nb + g.dom_n[a] : nb >= g.dom_n[a] ? nb - g.dom_n[a] : nb;
                    lc[a] = nb - g.offset[a];
                    inside = inside && lc[a] >= 0 && lc[a] < g.num[a];
                }
                if (!inside) continue;
                const int bk = bin_key(g, lc[0], lc[1], lc[2]);
                const uint32_t j0 = A.bin_start[bk], j1 = A.bin_start[bk + 1];
                // image of the neighbour cell relative to the binned cell
                const int dl[3] = {x + shift[0], y + shift[1], z + shift[2]};
                const float sh[3] = {(float)dl[0] * g.csf[0], (float)dl[1] * g.csf[1], (float)dl[2] * g.csf[2]};
                for (uint32_t jb = j0; jb < j1; jb += G) {
                    const uint32_t j = jb + lane;
                    bool acc = j < j1 && j != i && !(A.half && A.orig[j] < origi);
                    float dx = 0.f, dy = 0.f, dz = 0.f;
                    if (acc) {
                        const float4 oj = A.o0[j];
                        dx = oi.x - oj.x - sh[0];
                        dy = oi.y - oj.y - sh[1];
                        dz = oi.z - oj.z - sh[2];
                        const float ex = mi[0] ? min_image_f(dx, g.Lf[0]) : dx;
                        const float ey = mi[1] ? min_image_f(dy, g.Lf[1]) : dy;
                        const float ez = mi[2] ? min_image_f(dz, g.Lf[2]) : dz;
                        const float d2 = ex * ex + ey * ey + ez * ez;
                        if (pfi && oj.w == 0.0f && d2 < lo2) acc = true;
                        else if (pfi && oj.w == 0.0f && d2 > hi2) acc = false;
                        else acc = are_neibs_exact(g, xi, yi, zi, rni, A.rx[j], A.ry[j], A.rz[j], A.rns[j], edge);
                    }
                    const unsigned m = G == 32 ? __ballot_sync(0xffffffffu, acc) : (unsigned)acc;
                    if (acc) {
                        // periodic image code: minimum image of j seen from i
                        const uint32_t code = pair_image_code(g, own, lc, dl, dx, dy, dz, A.st);
                        const int k = cnt + __popc(m & ((1u << lane) - 1u));
                        if (k < A.K) A.nbr[nidx(k, i, A.np)] = j | (code << kJBits);
                    }
                    cnt += __popc(m);
                }
            }
        }
    }
    end_list<G>(A, i, lane, cnt);
}

// Whether the atoms of such a grid take a thread each. A warp's lanes are mostly
// idle in cells of few atoms, but n threads leave the GPU idle where n is small:
// the line rises with the atoms per cell, and lies lower for a local grid short
// of the box, whose tests are all FP64. A rebuild, thread / warp: flat boxes (one
// axis of two cells) with 4 atoms a cell 7,936 155 / 114 us, 31,752 171 / 292,
// 128,016 294 / 970; 24: 16,416 338 / 185, 63,936 364 / 563; 96: 32,448 1,003 /
// 572, 65,664 1,093 / 1,164; 192: 31,104 1,962 / 874. Short grids: 4 a cell 4,000
// 351 / 292, 16,384 368 / 879; 24: 15,552 1,263 / 794, 65,856 2,405 / 3,158; 48:
// 31,104 2,467 / 2,412, 131,712 8,540 / 10,817. A grid's team (TEAM) has fewer
// threads; a step with a rebuild in five: flat argon 30,976 88.5 / 73.8 us, 53,824
// 88.7 / 108; short argon 32,000 191 / 172, 55,296 206 / 263; short copper 16,384
// 146 / 108, 32,000 156 / 177.
template <bool TEAM>
__host__ __device__ inline bool atoms_by_threads(const GridParams& g, long long n) {
    const long long cells = g.ncells;
    if (grid_whole(g)) return 2 * n * cells >= (TEAM ? 3 : 2) * (12000 * cells + 950 * n);
    return 2 * n * cells >= (TEAM ? 5 : 2) * (3000 * cells + 1000 * n);
}
// In one block: a thread as soon as half of them have an atom (LJ argon, 100
// steps: 256 atoms 2.09 / 1.98 ms, 500 3.56 / 4.04, 2,000 45 / 55; EAM Cu 640 6.0 /
// 9.5).
template <int NT>
__device__ __forceinline__ bool block_by_threads(int n) { return 2 * n >= NT; }

// The neighbour cell of lane t < 27, (t / 9 - 1, t / 3 % 3 - 1, t % 3 - 1)
// from the cell at global index gc (local own): its first slot and count (0:
// none, or outside the grid), image code and shift. For grids whose periodic
// axes have 3 cells or more.
__device__ __forceinline__ void neighbour_cell(const GridParams& g, const uint32_t* bin_start, const int gc[3],
                                               const int own[3], int t, uint32_t& j0, uint32_t& count, uint32_t& code,
                                               float4& sh) {
    j0 = count = code = 0;
    sh = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t >= 27) return;
    const int dl[3] = {t / 9 - 1, (t / 3) % 3 - 1, t % 3 - 1};
    int lc[3];
    for (int a = 0; a < 3; ++a) {
        if (g.periodic[a] && ((g.dom_n[a] == 1 && dl[a] != 0) || (g.dom_n[a] == 2 && dl[a] == 1))) return;
        int nb = gc[a] + dl[a];
        if (g.periodic[a]) nb = nb < 0 ? nb + g.dom_n[a] : nb >= g.dom_n[a] ? nb - g.dom_n[a] : nb;
        lc[a] = nb - g.offset[a];
        if (lc[a] < 0 || lc[a] >= g.num[a]) return;
    }
    const int bk = bin_key(g, lc[0], lc[1], lc[2]);
    j0 = bin_start[bk];
    count = bin_start[bk + 1] - j0;
    sh = make_float4((float)dl[0] * g.csf[0], (float)dl[1] * g.csf[1], (float)dl[2] * g.csf[2], 0.f);
    for (int a = 0; a < 3; ++a) {
        code |= (uint32_t)(dl[a] + 1) << (2 * a);
        if (dl[a] != lc[a] - own[a]) code |= 1u << 6;  // the image crossed a periodic face
    }
}

// The list of atom i by a warp on such grids (an atom clamped into the grid
// excepted): 27 lanes fetch the neighbour cells, then the cells in order, 32
// candidates at a time. Some five times the instructions per atom of the
// warp-per-cell build below, but a warp per atom: for systems of so few cells
// that most SMs have none (LJ argon 4,000 atoms has 125: 42 us by cells in
// four parts each, 13 us by atoms).
__device__ __forceinline__ void nbuild_atom_cells(const NbArgs& A, const GridParams& g, uint32_t i, int lane,
                                                  bool uniform_rns) {
    const unsigned full = 0xffffffffu;
    const float lo2 = (float)(g.max_rns * g.max_rns * (1.0 - 1e-5));
    const float hi2 = (float)(g.max_rns * g.max_rns * (1.0 + 1e-5));
    int own[3];
    unpack_cell(A.cellp[i], own[0], own[1], own[2]);
    int gc[3] = {own[0] + g.offset[0], own[1] + g.offset[1], own[2] + g.offset[2]};
    if (g.dim < 3) gc[2] = 0;
    if (g.dim < 2) gc[1] = 0;
    uint32_t j0, count, code;
    float4 sh;
    neighbour_cell(g, A.bin_start, gc, own, lane, j0, count, code, sh);
    const float4 oi = A.o0[i];
    const bool pfi = uniform_rns && oi.w == 0.0f;
    const uint32_t origi = A.half ? A.orig[i] : 0u;
    int cnt = 0;
    for (unsigned left = __ballot_sync(full, count > 0); left; left &= left - 1u) {
        const int c = __ffs(left) - 1;
        const uint32_t c0 = __shfl_sync(full, j0, c), c1 = c0 + __shfl_sync(full, count, c);
        const uint32_t img = __shfl_sync(full, code, c) << kJBits;
        const float sx = __shfl_sync(full, sh.x, c), sy = __shfl_sync(full, sh.y, c), sz = __shfl_sync(full, sh.z, c);
        for (uint32_t jb = c0; jb < c1; jb += 32) {
            const uint32_t j = jb + lane;
            bool acc = j < c1 && j != i && !(A.half && A.orig[j] < origi);
            if (acc) {
                const float4 oj = A.o0[j];
                const float dx = oi.x - (oj.x + sx), dy = oi.y - (oj.y + sy), dz = oi.z - (oj.z + sz);
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                const bool pf = pfi && oj.w == 0.0f;
                if (pf && d2 < lo2) {
                    acc = true;
                } else if (pf && d2 > hi2) {
                    acc = false;
                } else {
                    bool edge[3] = {false, false, false};
                    for (int a = 0; a < g.dim; ++a) edge[a] = gc[a] == 0 || gc[a] == g.num[a] - 1;
                    acc = are_neibs_exact(g, A.rx[i], A.ry[i], A.rz[i], A.rns[i], A.rx[j], A.ry[j], A.rz[j], A.rns[j],
                                          edge);
                }
            }
            const unsigned m = __ballot_sync(full, acc);
            const int k = cnt + __popc(m & ((1u << lane) - 1u));
            if (acc && k < A.K) A.nbr[nidx(k, i, A.np)] = j | img;
            cnt += __popc(m);
        }
    }
    end_list<32>(A, i, lane, cnt);
}

// ---- list build, a warp per cell with lanes over candidates -------------------
// The cell's candidates are the atoms of its neighbour cells in the
// reference's cell order (x outer, z inner), each cell's atoms in slot order.
// Lanes take 32 consecutive candidates (a chunk); the warp walks the cell's
// atoms, one ballot per atom, so a chunk's accept matrix ends as one row per
// atom in shared memory. After CH chunks lane i appends the accepted
// candidates of atom i, in order. Entry order per atom is therefore the order
// of the per-atom loop in nbuild_atom, and the lists are the same, entry for
// entry. Used when no periodic axis has 2 cells or fewer (no minimum-image
// adjustment of the image code, GridParams::small_box); otherwise nbuild_atom
// runs.
//
// The build is bound by instruction issue, so a test is as few instructions
// as it takes, five for 32 pairs: the squared distance from the threshold mid
// as |b|^2 + (|a|^2 - mid) - 2 a.b, three fused operations, two atoms at once
// in packed FP32 pairs, each atom pair read once for two candidates a lane; the
// signs are shifted into a word per candidate, which the warp transposes once
// per chunk to a word per atom (a ballot and a store per atom were four
// instructions more). Appending waits for CH chunks, as the lanes' counts even
// out, and takes two to four lanes per atom where the cell has no more than 16.
// Rebuilds: LJ liquid 4,000,000 atoms 3.54 -> 2.77 ms, NiAl 1,018,880
// 1.16 -> 0.98, EAM Cu 1,000,188 0.87 -> 0.76; with 8 and 24 chunks a turn and
// 32, 28 and 24 warps an SM no pair was faster on all three than 16 and 28.
template <int CH>
struct NbWarpSmem {
    static_assert(CH % 2 == 0, "chunks are tested two at a time");
    float4 csh[27];          // cell shift (x, y, z) of the image
    float4 oa[32];           // pairs of atoms: (-2ax0, -2ax1, -2ay0, -2ay1), (-2az0, -2az1, m0, m1), m = |a|^2 - mid
    uint32_t row[CH][32];    // accept rows of the turn's chunks: bit = candidate, column = atom
    uint32_t cand[CH * 32];  // the turn's list entries (slot | image code)
    uint32_t cj0[27];        // first slot of each non-empty neighbour cell
    uint32_t cpre[28];       // candidate prefix over those cells
    uint32_t ccode[27];      // image code << kJBits
};

// A 32 x 32 matrix of bits, lane l holding row l, transposed over the warp
// (five exchanges of half blocks).
__device__ __forceinline__ unsigned transpose32(unsigned x, int lane) {
    unsigned keep = 0x0000ffffu;
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, k);
        const bool low = (lane & k) == 0;
        const unsigned mine = low ? keep : ~keep;
        x = (x & mine) | (__funnelshift_l(y, y, low ? k : 32 - k) & ~mine);
        keep ^= keep << (k >> 1);
    }
    return x;
}

template <int CH>
__device__ __forceinline__ void nbuild_cell_warp(const NbArgs& A, const GridParams& g, int bin, int lane,
                                                 bool uniform_rns, NbWarpSmem<CH>& S, int part = 0, int parts = 1) {
    const unsigned full = 0xffffffffu;
    const float lo2 = (float)(g.max_rns * g.max_rns * (1.0 - 1e-5));
    const float hi2 = (float)(g.max_rns * g.max_rns * (1.0 + 1e-5));
    const uint32_t s0 = A.bin_start[bin], s1 = A.bin_start[bin + 1];
    // this part's atoms of the cell
    const uint32_t share = (s1 - s0 + parts - 1) / parts, e0 = s0 + share * part, e1 = min(e0 + share, s1);
    if (e0 >= s1) return;
    int cx, cy, cz;
    unpack_cell(A.cellp[s0], cx, cy, cz);
    int gc[3] = {cx + g.offset[0], cy + g.offset[1], cz + g.offset[2]};
    if (g.dim < 3) gc[2] = 0;
    if (g.dim < 2) gc[1] = 0;
    bool edge[3] = {false, false, false};
    for (int a = 0; a < g.dim; ++a) edge[a] = gc[a] == 0 || gc[a] == g.num[a] - 1;

    uint32_t j0, ncand, code;
    float4 sh;
    const int own[3] = {cx, cy, cz};
    neighbour_cell(g, A.bin_start, gc, own, lane, j0, ncand, code, sh);
    const bool use = ncand > 0;
    const unsigned vm = __ballot_sync(full, use);
    const int slot = __popc(vm & ((1u << lane) - 1u));
    const int nc = __popc(vm);
    uint32_t incl = use ? ncand : 0u;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
    }
    if (use) {
        S.cj0[slot] = j0;
        S.cpre[slot] = incl - ncand;
        S.ccode[slot] = code << kJBits;
        S.csh[slot] = sh;
    }
    const uint32_t T = __shfl_sync(full, incl, 31);
    if (lane == 0) S.cpre[nc] = T;
    // the cell itself (lane 13: offset (0, 0, 0)) among the used cells
    const int home = __popc(vm & ((1u << 13) - 1u));
    __syncwarp();

    // The packed test's threshold and its error: the terms are at most
    // |b|^2 < 9.2 cs^2 (offsets within 0.75 cells, one cell apart) and each of
    // its seven roundings adds 2^-24 of the largest partial sum, below 5e-6 cs^2
    // in all; pairs within `half` of the middle go to the exact tests.
    const float csm = fmaxf(g.csf[0], fmaxf(g.csf[1], g.csf[2]));
    const float mid = 0.5f * (lo2 + hi2), half_band = fmaf(6e-6f * csm, csm, 0.5f * (hi2 - lo2));

    // batches of up to 32 atoms, all of nearly the same size
    const uint32_t batches = (e1 - e0 + 31) >> 5, per = (e1 - e0 + batches - 1) / batches;
    for (uint32_t base = e0; base < e1; base += per) {
        const uint32_t ni = e1 - base < per ? e1 - base : per;
        const bool act = (uint32_t)lane < ni;
        const uint32_t me = base + lane;
        float4 oa = make_float4(0.f, 0.f, 0.f, 0.f);
        if (act) {
            oa = A.o0[me];
        }
        const float a2 = fmaf(oa.x, oa.x, fmaf(oa.y, oa.y, oa.z * oa.z));
        // an atom whose offset is not exact (or not a number) takes the batch
        // to the exact tests
        const bool rough = __any_sync(full, oa.w != 0.0f || !(a2 < 1e30f)) || !uniform_rns || A.half;
        {
            // columns past the batch (the second of an odd pair) accept nothing
            const float m = act ? a2 - mid : 3e38f;
            float* q = reinterpret_cast<float*>(&S.oa[lane & ~1]) + (lane & 1);
            q[0] = -2.0f * oa.x;
            q[2] = -2.0f * oa.y;
            q[4] = -2.0f * oa.z;
            q[6] = m;
        }
        // this atom's own candidate index (it is a candidate of its own cell)
        const uint32_t self_t = act ? S.cpre[home] + (me - s0) : 0xffffffffu;
        // appending: `lanes` lanes take an atom's chunks in as many parts
        const int lanes = ni <= 8 ? 4 : ni <= 10 ? 3 : ni <= 16 ? 2 : 1;
        const int ea = lane / lanes, part = lane - ea * lanes;
        const bool appends = (uint32_t)ea < ni;
        const uint32_t mine_e = base + ea;
        __syncwarp();
        int cnt = 0;  // list length of atom mine_e
        int c = 0;    // neighbour cell of this lane's candidate
        // the lane's candidates of the next two chunks, fetched ahead
        uint32_t jn[2] = {0, 0};
        int cn[2] = {0, 0};
        float4 on[2];
        on[0] = on[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        auto fetch = [&](uint32_t t) {
#pragma unroll
            for (int h = 0; h < 2; ++h, t += 32) {
                if (t >= T) return;
                while (S.cpre[c + 1] <= t) ++c;
                cn[h] = c;
                jn[h] = S.cj0[c] + (t - S.cpre[c]);
                on[h] = A.o0[jn[h]];
            }
        };
        fetch(lane);
        for (uint32_t t0 = 0; t0 < T; t0 += CH * 32) {
            const int nch = min((int)((T - t0 + 31) >> 5), CH);
            for (int ch = 0; ch < nch; ch += 2) {
                bool have[2], rest = false;
                uint32_t j[2];
                float px[2], py[2], pz[2], pw[2], b2[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t t = t0 + 32 * (ch + h) + lane;
                    have[h] = t < T;
                    j[h] = jn[h];
                    // the candidate seen from the cell: offset + image shift
                    const float4 sh = S.csh[cn[h]];
                    px[h] = have[h] ? on[h].x + sh.x : 0.f;
                    py[h] = have[h] ? on[h].y + sh.y : 0.f;
                    pz[h] = have[h] ? on[h].z + sh.z : 0.f;
                    pw[h] = on[h].w;
                    S.cand[32 * (ch + h) + lane] = jn[h] | S.ccode[cn[h]];
                    b2[h] = fmaf(px[h], px[h], fmaf(py[h], py[h], pz[h] * pz[h]));
                    rest = rest || (have[h] && (pw[h] != 0.0f || !(b2[h] < 1e30f)));
                }
                fetch(t0 + 32 * ch + 64 + lane);
                bool exact[2];
                exact[0] = exact[1] = rough || __any_sync(full, rest);
                if (!exact[0]) {
                    // a lane tests its two candidates against two atoms at a
                    // time; the signs go to a bit per atom
                    unsigned long long bx[2], by[2], bz[2], bb[2];
                    float near[2];      // least distance from the threshold
                    unsigned col[2];    // accepting atoms
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float q = have[h] ? b2[h] : 3e38f;
                        bx[h] = pack2(px[h], px[h]);
                        by[h] = pack2(py[h], py[h]);
                        bz[h] = pack2(pz[h], pz[h]);
                        bb[h] = pack2(q, q);
                        near[h] = 3e38f;
                        col[h] = 0;
                    }
                    for (int ii = (int)(ni - 1) & ~1; ii >= 0; ii -= 2) {
                        const ulonglong2 u = reinterpret_cast<const ulonglong2*>(S.oa)[ii];
                        const ulonglong2 v = reinterpret_cast<const ulonglong2*>(S.oa)[ii + 1];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float d0, d1;
                            unpack2(fma2(u.x, bx[h], fma2(u.y, by[h], fma2(v.x, bz[h], add2(bb[h], v.y)))), d0, d1);
                            near[h] = fminf(near[h], fminf(fabsf(d0), fabsf(d1)));
                            col[h] = __funnelshift_l(__float_as_uint(d1), col[h], 1);
                            col[h] = __funnelshift_l(__float_as_uint(d0), col[h], 1);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        exact[h] = __any_sync(full, near[h] <= half_band);
                        if (exact[h]) continue;
                        // a bit per atom and lane becomes a bit per lane and
                        // atom; without the atom itself
                        unsigned row = transpose32(col[h], lane);
                        const uint32_t own = self_t - (t0 + 32 * (ch + h));
                        if (own < 32u) row &= ~(1u << own);
                        S.row[ch + h][lane] = row;
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!exact[h]) continue;
                    // pairs within 1e-5 of rns (or of atoms whose offsets are
                    // not exact) are marked in a second row and settled in FP64
                    __syncwarp();
                    unsigned mine = 0, mine_x = 0;
                    const uint32_t origj = A.half && have[h] ? A.orig[j[h]] : 0u;
                    for (uint32_t ii = 0; ii < ni; ++ii) {
                        const float4 oi = A.o0[base + ii];
                        const float dx = oi.x - px[h], dy = oi.y - py[h], dz = oi.z - pz[h];
                        const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        const bool pf = uniform_rns && pw[h] == 0.0f && oi.w == 0.0f;
                        const bool ok = have[h] && j[h] != base + ii && !(A.half && origj < A.orig[base + ii]);
                        const unsigned m = __ballot_sync(full, ok && pf && d2 < lo2);
                        const unsigned mx = __ballot_sync(full, ok && !(pf && (d2 < lo2 || d2 > hi2)));
                        if ((uint32_t)lane == ii) {
                            mine = m;
                            mine_x = mx;
                        }
                    }
                    while (mine_x) {
                        const int b = __ffs(mine_x) - 1;
                        mine_x &= mine_x - 1u;
                        const uint32_t jb = S.cand[32 * (ch + h) + b] & kJMask;
                        if (are_neibs_exact(g, A.rx[me], A.ry[me], A.rz[me], A.rns[me], A.rx[jb], A.ry[jb], A.rz[jb],
                                            A.rns[jb], edge))
                            mine |= 1u << b;
                    }
                    S.row[ch + h][lane] = mine;
                }
            }
            __syncwarp();
            // append the accepted candidates in candidate order
            if (appends) {
                int ch = 0, end = nch, at = cnt;
                if (lanes > 1) {
                    // this part's chunks, and the entries before and after them
                    const int from = nch * part / lanes;
                    end = nch * (part + 1) / lanes;
                    int all = 0;
                    for (int q = 0; q < nch; ++q) {
                        const int k = __popc(S.row[q][ea]);
                        all += k;
                        at += q < from ? k : 0;
                    }
                    cnt += all;
                    ch = from;
                }
                uint32_t* dst = A.nbr + nidx(at, mine_e, A.np);
                unsigned w = 0;
                for (;;) {
                    while (w == 0 && ch < end) w = S.row[ch++][ea];
                    if (w == 0) break;
                    const int b = __ffs(w) - 1;
                    w &= w - 1u;
                    if (at < A.K) *dst = S.cand[32 * (ch - 1) + b];
                    ++at;
                    dst += (at & 3) ? 1 : 4 * (size_t)A.np - 3;
                }
                if (lanes == 1) cnt = at;
            }
            __syncwarp();
        }
        if (appends && part == 0) {
            const uint32_t at = mine_e;
            const int padded = (cnt + 3) & ~3;
            for (int k = cnt; k < padded && k < A.K; ++k) A.nbr[nidx(k, at, A.np)] = at | kSelfCode;
            A.ncnt[at] = padded < A.K ? padded : A.K;
            if (cnt > A.K) {
                atomicOr(&A.st->flags, FLAG_OVERFLOW);
                atomicOr(&A.st->build_flags, FLAG_OVERFLOW);
            }
        }
        if (act) {
            A.r0x[me] = A.rx[me];
            A.r0y[me] = A.ry[me];
            A.r0z[me] = A.rz[me];
            A.saved_rcut[me] = A.rcut[me];
            A.saved_rns[me] = A.rns[me];
            A.saved_uid[me] = A.uid[me];
        }
        // the longest list, one atomic per warp
        const unsigned wmax = __reduce_max_sync(full, appends ? (unsigned)cnt : 0u);
        if (lane == 0) atomicMax(&A.st->max_count, wmax);
        __syncwarp();
    }
}

}  // namespace mdg

struct mdg_system;

namespace mdg {
// Host-side argument builders of a system's rebuild (nlist.cu).
GatherAll gather_sets(const mdg_system* sys);
NbArgs nb_args(const mdg_system* sys);
DomainDev domain_of(const mdg_system* sys);
CellOut cell_out(const mdg_system* sys);
}  // namespace mdg
