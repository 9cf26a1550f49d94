// solo.cu — the whole driver loop of one small system in one kernel.
//
// For small systems (hundreds to tens of thousands of atoms) a step is a few
// microseconds of work, so launching its stages as separate kernels (or graph
// nodes) costs more than the work. Here a team of blocks owns one system and
// runs `steps` iterations of the driver loop of the reference
// (test/python/solver/test-EAM.py:158-200: make_step, then decide() and
// update(-1)) with barriers between the passes:
//   drift + half-skin test -> [EAM density ->] forces -> kick
//   -> if any atom moved half a skin: the rebuild (wrap + bounds, grid,
//      bin count, scan, scatter, permutation of every field, cell offsets,
//      list build) -> next step.
// Every pass calls the same per-atom (or per-bin) device code as the
// per-stage kernels, in the same order, so a system gives the same bits
// here as through the graph of mdg_run. Three teams:
//
//  - one block (the serving loop): a persistent kernel's block takes a whole
//    request from a queue; many systems run at once, a block each, and no
//    block waits on another.
//  - a grid of one block per SM, launched cooperatively (mdg_run and
//    mdg_run_host of a small system): the blocks share the system's atoms and
//    meet at barriers in global memory. Every wait is bounded.
//  - the same with a share of the SMs, for a whole request (the server, while
//    few requests are outstanding).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "forces64_dev.cuh"
#include "forces_dev.cuh"
#include "integrate_dev.cuh"
#include "mdg_host.h"
#include "nlist_dev.cuh"
#include "team_dev.cuh"
#include "team_rules.h"
#include "thermo_dev.cuh"

namespace mdg {

// Completion record of one system's run, in host-mapped pinned memory: the
// block writes it last, `done` after a system-scope fence.
struct SoloOut {
    unsigned long long left;
    DevStatus st;
    volatile uint32_t done;
    volatile uint32_t started;  // a request's team: seq, once its blocks run
    // GPU clock (%globaltimer, ns): the block starts on the request / has
    // written the result records (service time = end - start)
    unsigned long long t_start, t_end;
};

struct alignas(16) SoloArgs {
    IArgs I;
    FArgs F;
    NbArgs N;
    GatherAll G;
    DomainDev D;
    CellOut C;
    const PotSet* ps;
    int n;
    double *rx, *ry, *rz;
    const double* rns;
    uint32_t *key, *rank, *src, *bin_count, *bin_start;
    const uint32_t* orig;
    GridParams* dgrid;
    long long bin_cap;
    long long* part;              // a grid's team: 8 words per block
    DevStatus* st;
    long long steps;              // steps to run
    uint32_t seq;                 // completion value written to out->done
    int np;
    int setup;                    // 1: load the atoms, build the first list, initial forces
    int any_eam;
    const mdg_atom* atoms_in;     // host-mapped input records (setup)
    uint8_t* bc;
    SoloOut* out;                 // host-mapped: steps left, status, completion
    mdg_atom* atoms_out;          // host-mapped: the result records, caller order
};

// Chunks per turn of the list build here: few, as its shared memory is taken
// from the L1 that the force passes gather through.
constexpr int kSoloChunks = 2;
// A grid's team: of few atoms a block, so more chunks (8 against 2 in LJ argon
// 13,500 atoms 16.2 -> 15.6 us a step; 16 take L1 from EAM: Cu 87,808 atoms
// 50.1 -> 53.0).
constexpr int kTeamChunks = 8;

template <int NT>
struct SoloShared {
    long long red[8][NT / 32];
    uint32_t scan[32];
    int differ, said;
};
// The eight-lane passes' exchange (the grid's team only: a request's block
// leaves its shared memory to L1).
template <int NT>
struct LaneShared {
    alignas(kLaneAlign) float part[NT / 32][96];  // lane_sums
    float sum[3][NT];  // of NT atoms at a time
};

// Reduces the bounds (BoundKeys) of the block's threads; `busy` false: the
// whole warp has none. The result is in sh.red[k][0] after a __syncthreads by
// the caller.
template <int NT>
__device__ __forceinline__ void block_bounds8(long long v[8], bool busy, SoloShared<NT>& sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (busy) warp_bounds<8>(v);
    if (lane == 0)
        for (int k = 0; k < 8; ++k) sh.red[k][w] = v[k];
    __syncthreads();
    if (threadIdx.x < 8) {
        const int k = threadIdx.x;
        long long x = sh.red[k][0];
        for (int q = 1; q < NT / 32; ++q) x = k < 3 ? min(x, sh.red[k][q]) : max(x, sh.red[k][q]);
        sh.red[k][0] = x;
    }
}

// The lists of flat and short grids (a function of its own: the rebuild's
// registers are for the other grids).
template <int NT, bool WIDE>
__device__ __noinline__ void small_box_lists(const Team<NT, WIDE>& tm, const NbArgs& N, const GridParams& g, bool uniform) {
    if (WIDE ? atoms_by_threads<true>(g, N.n) : block_by_threads<NT>(N.n)) {
        for (int i = tm.a0 + tm.t; i < tm.a1; i += NT) nbuild_atom<1>(N, g, (uint32_t)i, 0, uniform);
    } else {
        for (int i = tm.gw; i < N.n; i += tm.nw) nbuild_atom<32>(N, g, (uint32_t)i, tm.lane, uniform);
    }
}

// One rebuild by the team (the pipeline of nlist_enqueue). Team-uniform
// result: false when a capacity overflowed (the loop stops and the host grows
// the capacities).
template <int NT, bool WIDE>
__device__ __noinline__ bool solo_rebuild(Team<NT, WIDE>& tm, const SoloArgs& S, GridParams& g, SoloShared<NT>& sh) {
    const int t = tm.t, n = S.n;
    if (tm.gt == 0) {
        S.st->max_count = 0;
        S.st->build_flags = 0;
    }
    // wrap + bounds (min/max are exact, so the order of the reduction is free)
    long long v[8];
    no_bounds<8>(v);
    const double r0 = S.rns[0];
    for (int i = tm.a0 + t; i < tm.a1; i += NT) {
        double x[3];
        wrap_one(S.D, S.rx, S.ry, S.rz, i, x);
        const double q = S.rns[i];
        add_bounds(v, x, q);
        if (q != r0) v[7] = 1;
    }
    for (long long b = tm.gt; b < S.bin_cap; b += tm.gn) S.bin_count[b] = 0;
    block_bounds8<NT>(v, tm.a0 + (t & ~31) < tm.a1, sh);
    __syncthreads();
    if (WIDE) {
        if (t < 8) S.part[tm.rank * 8 + t] = sh.red[t][0];
        tm.sync();
        if (tm.dead) return false;
        no_bounds<8>(v);
        for (int b = t; b < tm.size; b += NT)
            for (int k = 0; k < 8; ++k) {
                const long long y = __ldcg(S.part + b * 8 + k);
                v[k] = k < 3 ? min(v[k], y) : max(v[k], y);
            }
        block_bounds8<NT>(v, (t & ~31) < tm.size, sh);
        __syncthreads();
    }
    // the grid, by every block: three lanes take an axis each
    if (t < 32) {
        const double cell = key_double(sh.red[6][0]);
        if (t == 0) {
            memset(&g, 0, sizeof(g));
            sh.differ = sh.red[7][0] == 1;
        }
        __syncwarp();
        bool small = false, bad = false;
        if (t < 3)
            grid_axis(S.D, t < S.D.dim ? key_double(sh.red[t][0]) : 0.0, t < S.D.dim ? key_double(sh.red[3 + t][0]) : 0.0,
                      cell, t, g, &small, &bad);
        small = __any_sync(0xffffffffu, small);
        bad = __any_sync(0xffffffffu, bad);
        __syncwarp();
        if (t == 0) {
            grid_totals(S.D, cell, small, bad, g);
            if (g.empty == 0 && (long long)g.nbins + 1 > S.bin_cap) {
                g.empty = -3;
                if (tm.rank == 0) {
                    atomicOr(&S.st->flags, FLAG_OVERFLOW);
                    atomicOr(&S.st->build_flags, FLAG_OVERFLOW);
                }
            }
            if (tm.rank == 0) {
                *S.dgrid = g;
                S.st->nonuniform = sh.differ;
            }
        }
    }
    __syncthreads();
    if (g.empty) {
        const bool ok = g.empty != -3;
        tm.sync();
        return ok;
    }
    const int nb = g.nbins;
    // (the bins were cleared before the last barrier)
    for (int i = tm.a0 + t; i < tm.a1; i += NT)
        bin_count_one(g, i, S.rx, S.ry, S.rz, S.key, S.rank, S.N.ncnt, S.bin_count, S.st);
    tm.sync();
    if (tm.dead) return false;
    // exclusive scan, by one block: each thread a contiguous chunk of the bins
    if (tm.rank == 0) {
        const int chunk = (nb + NT - 1) / NT;
        const int b0 = min(t * chunk, nb), b1 = min(b0 + chunk, nb);
        uint32_t sum = 0;
        for (int b = b0; b < b1; ++b) sum += S.bin_count[b];
        uint32_t tot;
        uint32_t off = block_excl_scan(sum, sh.scan, &tot);
        for (int b = b0; b < b1; ++b) {
            uint32_t c = S.bin_count[b];
            S.bin_start[b] = off;
            off += c;
        }
        if (t == 0) S.bin_start[nb] = tot;
    }
    tm.sync();
    if (tm.dead) return false;
    // arrival order (the atoms' cells wait in ncnt, their caller indices in
    // arrival order in cellp), then each bin by caller index
    for (int i = tm.a0 + t; i < tm.a1; i += NT) {
        const uint32_t k = S.bin_start[S.key[i]] + S.rank[i];
        S.src[k] = (uint32_t)i;
        S.C.cellp[k] = S.orig[i];
    }
    tm.sync();
    if (tm.dead) return false;
    // (a wide team's blocks have few atoms: eight threads share an atom's 31
    // fields, whose loads and stores are otherwise one thread's chain)
    const bool eight = WIDE && tm.a1 - tm.a0 <= 2 * (NT / 8);
    for (int base = tm.a0; eight && base < tm.a1; base += NT / 8) {
        const int k = base + (t >> 3), part = t & 7;
        const bool in = k < tm.a1;
        const uint32_t i = in ? S.src[k] : 0u;
        uint32_t d = 0;
        if (in && part == 0) d = sorted_slot((uint32_t)k, S.key[i], S.bin_start, S.C.cellp);
        d = __shfl_sync(0xffffffffu, d, tm.lane & ~7);
        if (!in) continue;
        permute_part(S.G, i, d, part);
        if (part == 7) S.rank[d] = S.N.ncnt[i];
    }
    for (int k = tm.a0 + t; !eight && k < tm.a1; k += NT) {
        const uint32_t i = S.src[k];
        const uint32_t d = sorted_slot((uint32_t)k, S.key[i], S.bin_start, S.C.cellp);
        permute_one(S.G, i, d);
        S.rank[d] = S.N.ncnt[i];
    }
    tm.sync();
    if (tm.dead) return false;
    for (int base = tm.a0; eight && base < tm.a1; base += NT / 8) {
        const int k = base + (t >> 3);
        if (k < tm.a1) settle_part(g, S.G, k, S.rank[k], S.C, t & 7);
    }
    for (int k = tm.a0 + t; !eight && k < tm.a1; k += NT) settle_one(g, S.G, k, S.rank[k], S.C);
    tm.sync();
    if (tm.dead) return false;
    {
        const bool uniform = sh.differ == 0;
        if (!g.small_box && WIDE && n < kAtomBuildMost) {
            for (int i = tm.gw; i < n; i += tm.nw) nbuild_atom_cells(S.N, g, (uint32_t)i, tm.lane, uniform);
        } else if (!g.small_box) {
            // a warp per cell, lanes over candidates (the per-stage list
            // build's body); its per-warp state is the launch's dynamic
            // shared memory
            extern __shared__ __align__(16) unsigned char solo_dyn[];
            using State = NbWarpSmem<WIDE ? kTeamChunks : kSoloChunks>;
            State* nbs = reinterpret_cast<State*>(solo_dyn);
            const int parts = WIDE ? team_parts(tm.nw, n) : 1;
            const long long tasks = team_tasks(nb, parts);
            for (long long b = tm.gw; b < tasks; b += tm.nw)
                nbuild_cell_warp(S.N, g, parts > 1 ? task_bin(b, nb) : (int)b, tm.lane, uniform, nbs[tm.w],
                                 parts > 1 ? task_part(b, nb) : 0, parts);
        } else {
            small_box_lists(tm, S.N, g, uniform);
        }
        tm.sync();
        if (tm.dead) return false;
        // atoms clamped into the grid: their own lists from their unclamped cells
        if (!g.small_box && (__ldcg(&S.st->build_flags) & FLAG_RANGE)) {
            for (int i = tm.gw; i < n; i += tm.nw)
                if (S.N.o0[i].w == 2.0f) nbuild_atom<32>(S.N, g, (uint32_t)i, tm.lane, uniform);
            tm.sync();
        }
    }
    const bool ok = !(__ldcg(&S.st->build_flags) & FLAG_OVERFLOW);
    __syncthreads();
    return ok && !tm.dead;
}

// The input records (mdg_system_upload_atoms' scatter) from host memory.
template <int NT, bool WIDE>
__device__ __noinline__ void solo_read_atoms(const Team<NT, WIDE>& tm, const SoloArgs& S) {
    const GatherAll& G = S.G;
    for (int k = tm.gt; k < S.n; k += tm.gn) {
        const mdg_atom& a = S.atoms_in[k];
        const uint32_t s = S.C.slot_of[k];
        for (int c = 0; c < 3; ++c) {
            G.a2.out[RX + c][s] = a.r[c];
            G.a2.out[VX + c][s] = a.v[c];
            G.a2.out[FX + c][s] = a.f[c];
            G.fc2.out[c][s] = (float)a.f[c];
        }
        G.a2.out[MASS][s] = a.m;
        G.a2.out[RCUT][s] = a.rcut;
        G.a2.out[RNS][s] = a.rns;
        G.b2.out[EP - 12][s] = a.Ep;
        G.b2.out[EM - 12][s] = a.Em;
        G.b2.out[NC - 12][s] = a.nc;
        for (int q = 0; q < 9; ++q) G.b2.out[V0 - 12 + q][s] = a.V[q];
        G.u2.out[1][s] = a.uid;
        G.h2.out[0][s] = a.kind;
        G.h2.out[1][s] = a.tag;
    }
}

// Pair::prepare's output reset (launch_zero) for atom i.
__device__ __forceinline__ void solo_zero_one(const SoloArgs& S, int i) {
    const GatherAll& G = S.G;
    if (G.h.in[1][i] == 0) return;
    G.a2.out[FX][i] = 0.0;
    G.a2.out[FY][i] = 0.0;
    G.a2.out[FZ][i] = 0.0;
    G.b2.out[EP - 12][i] = 0.0;
    for (int k = 0; k < 9; ++k) G.b2.out[V0 - 12 + k][i] = 0.0;
    if (S.any_eam) {
        G.b2.out[EM - 12][i] = 0.0;
        G.b2.out[NC - 12][i] = 0.0;
    }
}

// The force stages, a thread per atom; with KICK the second half-kick rides in
// the force body (the step loop of one block), without it the forces alone
// (the set-up's initial forces).
template <bool EAM, bool KICK, int NT, bool WIDE>
__device__ __forceinline__ void solo_stages(Team<NT, WIDE>& tm, const SoloArgs& S) {
    if (EAM) {
        for (int i = tm.a0 + tm.t; i < tm.a1; i += NT) density_one<RhoGroup<0, false, false>>(S.F, S.ps, i);
        tm.sync();
    }
    for (int i = tm.a0 + tm.t; i < tm.a1; i += NT) {
        float f[3];
        bool live;
        if (EAM) live = thread_forces<EamGroup<0, false, false>>(S.F, S.ps, i, f);
        else live = thread_forces<LjGroup<false, false>>(S.F, S.ps, i, f);
        if (live) store_force<KICK>(S.F, i, f[0], f[1], f[2]);
    }
}

// The set-up of a fresh system, in the order of the host calls it replaces
// (upload, prepare, update(-1), offsets, prepare, stages). False when the
// first list outgrew the capacities sized on the host.
template <bool EAM, int NT, bool WIDE>
__device__ __noinline__ bool solo_setup(Team<NT, WIDE>& tm, const SoloArgs& S, GridParams& g, SoloShared<NT>& sh) {
    const int a0 = tm.a0 + tm.t, a1 = tm.a1;  // this thread's atoms: a0, a0 + NT, ...
    // the fresh system's buffers (what system_alloc clears on a stream)
    for (int k = tm.gt; k < S.np; k += tm.gn) {
        S.G.u2.out[0][k] = (uint32_t)k;  // caller index of slot k
        S.C.slot_of[k] = (uint32_t)k;
        S.N.ncnt[k] = 0;
        S.bc[k] = 0;
        S.C.trig[k] = make_float2(0.0f, 0.0f);
        S.C.Rx[k] = 0.0;
        S.C.Ry[k] = 0.0;
        S.C.Rz[k] = 0.0;
        for (int q = 0; q < kMaxKinds; ++q) S.F.Fp64[(size_t)q * S.np + k] = 0.0;
    }
    if (tm.gt == 0) memset(S.st, 0, sizeof(DevStatus));
    tm.sync();
    solo_read_atoms<NT, WIDE>(tm, S);
    tm.sync();
    for (int i = a0; i < a1; i += NT) drift64_one(S.I, S.I, i, 0, 0);
    __syncthreads();
    if (!solo_rebuild<NT, WIDE>(tm, S, g, sh)) return false;
    for (int i = a0; i < a1; i += NT)
        S.C.pos32[i] = make_int4(off_encode(S.rx[i] - S.C.Rx[i], g.inv_u[0]), off_encode(S.ry[i] - S.C.Ry[i], g.inv_u[1]),
                                 off_encode(S.rz[i] - S.C.Rz[i], g.inv_u[2]), S.F.kind[i] & 3);
    for (int i = a0; i < a1; i += NT) solo_zero_one(S, i);
    __syncthreads();
    for (int i = a0; i < a1; i += NT) drift64_one(S.I, S.I, i, 0, 0);
    tm.sync();
    solo_stages<EAM, false>(tm, S);
    tm.sync();
    return !tm.dead;
}

// The result records (mdg_system_download_atoms' layout) straight into host
// memory; mixed forces are widened to FP64 as the download does.
template <int NT, bool WIDE>
__device__ __noinline__ void solo_write_atoms(const Team<NT, WIDE>& tm, const SoloArgs& S) {
    const GatherAll& G = S.G;
    for (int k = tm.gt; k < S.n; k += tm.gn) {
        const uint32_t s = S.C.slot_of[k];
        mdg_atom a;
        const bool live = G.h.in[1][s] != 0;  // tag
        for (int c = 0; c < 3; ++c) {
            a.r[c] = G.a.in[RX + c][s];
            a.v[c] = G.a.in[VX + c][s];
            a.f[c] = live ? (double)G.fc.in[c][s] : G.a.in[FX + c][s];
        }
        a.m = G.a.in[MASS][s];
        a.rcut = G.a.in[RCUT][s];
        a.rns = G.a.in[RNS][s];
        a.Ep = G.b.in[EP - 12][s];
        a.Em = G.b.in[EM - 12][s];
        a.nc = G.b.in[NC - 12][s];
        for (int q = 0; q < 9; ++q) a.V[q] = G.b.in[V0 - 12 + q][s];
        a.uid = G.u.in[1][s];
        a.kind = G.h.in[0][s];
        a.tag = G.h.in[1][s];
        a.bc = S.bc[s];
        a._pad[0] = a._pad[1] = a._pad[2] = 0;
        S.atoms_out[k] = a;
    }
}

// One request by the whole block: set-up, the loop, the result records and
// the completion record (last, after a system-scope fence).
template <bool EAM, int NT>
__device__ void solo_run(SoloArgs& S, GridParams& g, SoloShared<NT>& sh) {
    const int t = threadIdx.x, n = S.n;
    Team<NT, false> tm(nullptr, nullptr, n, n);
    long long left = S.steps;
    uint32_t rebuilds = 0;
    bool ok = true;
    unsigned long long t_start = 0;
    if (t == 0) t_start = global_ns();
    if (S.setup) ok = solo_setup<EAM>(tm, S, g, sh);
    if (t == 0) {
        S.st->need_rebuild = 0;
        S.st->build_flags = 0;
    }
    while (ok && left > 0) {
        bool need = false;
        for (int i = t; i < n; i += NT) need |= drift_mixed_one(S.I, S.I, i);
        const int any = __syncthreads_or(need);
        solo_stages<EAM, true>(tm, S);
        __syncthreads();
        --left;
        if (any) {
            ++rebuilds;
            ok = solo_rebuild<NT, false>(tm, S, g, sh);
        }
    }
    if (ok && left == 0) solo_write_atoms(tm, S);
    __syncthreads();
    if (t == 0) {
        S.st->need_rebuild = 0;
        S.st->pad[0] = rebuilds;
        S.st->pad[1] = ok ? 0u : 1u;  // 1: a list outgrew its capacities; the run is void
        S.out->left = (unsigned long long)left;
        S.out->st = *S.st;
        S.out->t_start = t_start;
        S.out->t_end = global_ns();
        __threadfence_system();
        S.out->done = S.seq;
    }
    __syncthreads();
}

__device__ __forceinline__ uint32_t ld_acquire_sys(const volatile uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Polls without an entry after which a block exits when no block is running a
// request (about 0.1 ms). While some are, it waits on for idle_limit polls,
// so that the next request finds it. (With idle_limit alone, 100,000 polls,
// a batch's blocks held every SM for 0.23 s after its last result, which any
// other kernel, or a caller that waits for the device, sat through.)
constexpr int kQuietPolls = 64;

// Persistent consumer of the request queue: each block claims the next
// published entry, runs that request, and claims again; a block that finds
// no entry for `idle_limit` polls (about a microsecond apart), or for
// kQuietPolls with no request running, or sees `stop`, exits. Every wait is
// bounded. head[0]: the next entry to claim; head[1]: requests running.
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_solo_persistent(const SoloArgs* desc, SoloQueue* q,
                                                           uint32_t* head, int idle_limit, int gen) {
    __shared__ __align__(16) SoloArgs S;
    __shared__ GridParams g;
    __shared__ SoloShared<NT> sh;
    __shared__ int s_rec;
    // liveness for the host (which set 1 before the launch), so that it tops
    // up the kernel with a further launch when blocks have gone idle and
    // exited while requests wait
    if (threadIdx.x == 0) q->live[gen][blockIdx.x] = 1u;
    for (;;) {
        if (threadIdx.x == 0) {
            int rec = -1, quiet = 0;
            for (int it = 0; it < idle_limit; ++it) {
                const uint32_t tl = ld_acquire_sys(&q->tail);
                const uint32_t h = *(volatile uint32_t*)head;
                if (h < tl) {
                    if (atomicCAS(head, h, h + 1) == h) {
                        atomicAdd(head + 1, 1u);
                        rec = ((volatile int*)q->ring)[h % kSoloRing];
                        break;
                    }
                    continue;
                }
                if (q->stop) break;
                quiet = *(volatile uint32_t*)(head + 1) ? 0 : quiet + 1;
                if (quiet >= kQuietPolls) break;
                __nanosleep(1000);
            }
            s_rec = rec;
        }
        __syncthreads();
        const int rec = s_rec;
        if (rec < 0) break;
        if (threadIdx.x == 0) q->live[gen][blockIdx.x] = 2u;  // 2: running a request
        {
            // the host rewrites a record between the requests of its slot,
            // while this kernel runs: read past L1 (a line kept from the
            // slot's previous record would give this request that one's
            // atom count or buffers)
            const int4* src = reinterpret_cast<const int4*>(desc + rec);
            int4* dst = reinterpret_cast<int4*>(&S);
            for (int k = threadIdx.x; k < (int)(sizeof(SoloArgs) / sizeof(int4)); k += NT) dst[k] = __ldcv(src + k);
        }
        __syncthreads();
        if (S.any_eam) solo_run<true, NT>(S, g, sh);
        else solo_run<false, NT>(S, g, sh);
        if (threadIdx.x == 0) {
            q->live[gen][blockIdx.x] = 1u;  // 1: waiting for the next entry
            atomicSub(head + 1, 1u);
        }
    }
    if (threadIdx.x == 0) {
        __threadfence_system();
        q->live[gen][blockIdx.x] = 0u;
    }
}

// ---- a grid's team: the step loop of mdg_run for small systems ------------------
// A step of a 4,000-atom system is some 5 us of work on the whole GPU, but as
// graph nodes it took 21 us (LJ) to 27 us (EAM): five nodes, each with its
// launch and drain. Here a barrier over the blocks costs about 1.5 us. With
// page-locked host arrays the call's transfers are the kernel's own reads and
// writes over the host link, so a one-step call is one launch.
struct TeamRun {
    const double *hpos, *hvel;      // caller-order positions and velocities to start from (host), or null
    double *opos, *ovel, *oforce;   // caller-order results (host), or null
    const ThermoDev* th;            // thermostat, or null
    ThermoArgs T;
    // the same with the positions' (and LJ offsets') second buffers
    IArgs I1;
    FArgs F1;
    ThermoArgs T1;
    unsigned long long* left_dev;
    unsigned long long* left_host;  // steps left and status at the end (pinned)
    DevStatus* st_host;
    unsigned long long* word;       // the barriers' word
    int per;                        // atoms per block
};

constexpr int kTeamThreads = 768;
static_assert(alignof(LaneShared<kTeamThreads>) >= kLaneAlign, "lane_sums reads its exchange by 16-byte words");

// A step's passes by the team: the forces, the thermostat, the second
// half-kick and, with `next`, the next step's first half-kick and drift;
// whether that leaves a thread's atom due for a rebuild. The drift writes
// positions (and the offsets the LJ pass reads) to the buffers that this
// step's force pass does not read (flips), so blocks that are still in it
// may lag by a barrier; the EAM force pass reads its neighbours only through
// the density pass's copies and takes its cut decisions (k_force_step), so
// the drift stays in place there. One barrier a step, two with EAM.
//
// The mixed passes take eight lanes per atom where a block has fewer than
// kTeamLanesMost atoms, else one thread: its 768 threads hold 96 atoms by
// lanes, and an atom's sum takes a thread about as long as three such rounds.
// Per step, lanes / threads: LJ argon 19,652 atoms (132 a block) 20.0 / 24.1
// us, 32,000 25.3 / 26.2, 48,668 34.2 / 31.7; EAM Cu 32,000 33.7 / 38.3, 48,668
// 44.2 / 41.6.
constexpr int kTeamLanesMost = 272;

template <bool EAM, bool MIXED>
constexpr bool kFlips = !(EAM && MIXED);

template <bool EAM, bool MIXED, int NT, int G>
__device__ __forceinline__ bool team_step(Team<NT, true>& tm, const SoloArgs& S, const TeamRun& R, LaneShared<NT>& sh,
                                          int p, bool next, uint32_t call) {
    const IArgs& I = p ? R.I1 : S.I;
    const IArgs& to = !kFlips<EAM, MIXED> ? I : p ? S.I : R.I1;
    const FArgs& F = p ? R.F1 : S.F;
    const ThermoArgs& T = p ? R.T1 : R.T;
    bool need = false;
    if (!MIXED) {
        // G lanes per atom, NT / G atoms at a time
        const int sub = tm.t / G, lane = tm.t % G;
        if (EAM) {
            for (int base = tm.a0; base < tm.a1; base += NT / G)
                density64_lanes<false, G, false>(F, S.ps, base + sub < tm.a1, base + sub, lane);
            tm.sync();
            if (tm.dead) return false;
        }
        for (int base = tm.a0; base < tm.a1; base += NT / G) {
            const bool live = base + sub < tm.a1 && F.tag[base + sub] != 0;
            const int i = live ? base + sub : tm.a0;
            double f[3];
            forces64_lanes<false, EAM ? POT_EAM : POT_LJCUT, false, G, false>(F, S.ps, live, i, lane, f);
            if (live && lane == 0) {
                F.fx[i] = f[0];
                F.fy[i] = f[1];
                F.fz[i] = f[2];
            }
        }
        __syncthreads();
        for (int i = tm.a0 + tm.t; i < tm.a1; i += NT) {
            if (R.th) langevin_one<false>(T, R.th, i, call);
            kick64_one(I, i);
            if (next) need |= drift64_one(I, to, i, 1, 1);
        }
        return need;
    }
    // the sums of up to NT atoms meet in shared memory, then a thread per atom
    // finishes them (finishing 96 atoms at a time cost a wait for global memory
    // and two barriers each: LJ argon 32,000 atoms 30.0 us a step against 25.3)
    const int sub = tm.t >> 3;
    const bool few = R.per < kTeamLanesMost;
    if (EAM) {
        for (int base = tm.a0; base < tm.a1; base += NT) {
            const int end = min(base + NT, tm.a1);
            if (!few) {
                const int i = base + tm.t;
                float rho[1] = {0.f};
                if (i < end && F.tag[i] != 0) {
                    RhoGroup<0, true, false> grp(F, S.ps, i);
                    group_sums<1>(F, i, F.ncnt[i] >> 2, grp, rho);
                }
                sh.sum[0][tm.t] = rho[0];
            }
            for (int k = 0; few && base + k + 4 * tm.w < end; k += NT / 8) {
                const int i = base + k + sub;
                const bool in = i < end, live = in && F.tag[i] != 0;
                float rho[1];
                RhoGroup<0, true, false> grp(F, S.ps, in ? i : tm.a0);
                lane_sums<1>(F, live, in ? i : tm.a0, live ? F.ncnt[i] >> 2 : 0, grp, sh.part[tm.w], rho);
                if (in && (tm.t & 7) == 0) sh.sum[0][k + sub] = rho[0];
            }
            __syncthreads();
            const int me = base + tm.t;
            if (me < end) store_density<false>(F, S.ps, me, F.pos32[me], 0, sh.sum[0][tm.t]);
            __syncthreads();
        }
        tm.sync();
        if (tm.dead) return false;
    }
    for (int base = tm.a0; base < tm.a1; base += NT) {
        const int end = min(base + NT, tm.a1);
        if (!few) {
            const int i = base + tm.t;
            float f[3] = {0.f, 0.f, 0.f};
            if (i < end) {
                if (EAM) thread_forces<EamGroup<0, true, false>>(F, S.ps, i, f);
                else thread_forces<LjGroup<false, false>>(F, S.ps, i, f);
            }
            for (int q = 0; q < 3; ++q) sh.sum[q][tm.t] = f[q];
        }
        for (int k = 0; few && base + k + 4 * tm.w < end; k += NT / 8) {
            const int i = base + k + sub;
            const bool in = i < end;
            float f[3];
            if (EAM) lane_forces<EamGroup<0, true, false>>(F, S.ps, in, in ? i : tm.a0, sh.part[tm.w], f);
            else lane_forces<LjGroup<false, false>>(F, S.ps, in, in ? i : tm.a0, sh.part[tm.w], f);
            if (in && (tm.t & 7) == 0)
                for (int q = 0; q < 3; ++q) sh.sum[q][k + sub] = f[q];
        }
        __syncthreads();
        const int me = base + tm.t;
        if (me < end) {
            const bool live = F.tag[me] != 0;
            const float fx = sh.sum[0][tm.t], fy = sh.sum[1][tm.t], fz = sh.sum[2][tm.t];
            if (R.th) {
                if (live) store_force<false>(F, me, fx, fy, fz);
                langevin_one<true>(T, R.th, me, call);
                kick_mixed_one(I, me);
                if (next) need |= drift_mixed_one(I, to, me);
            } else if (live && next) {
                need |= kick_drift_mixed(I, to, F.gx, F.gy, F.gz, me, fx, fy, fz);
            } else if (live) {
                store_force<true>(F, me, fx, fy, fz);
            } else if (next) {
                need |= drift_mixed_one(I, to, me);  // tag 0: the offsets and the test alone
            }
        }
        __syncthreads();
    }
    return need;
}

// The offsets of the block's atoms (launch_offsets).
template <int NT>
__device__ __forceinline__ void team_offsets(const Team<NT, true>& tm, const SoloArgs& S) {
    for (int i = tm.a0 + tm.t; i < tm.a1; i += NT)
        S.C.pos32[i] = make_int4(off_encode(S.rx[i] - S.C.Rx[i], S.I.inv_u[0]), off_encode(S.ry[i] - S.C.Ry[i], S.I.inv_u[1]),
                                 off_encode(S.rz[i] - S.C.Rz[i], S.I.inv_u[2]), S.F.kind[i] & 3);
}

// The step loop of a team whose positions are in their first buffers, where
// they are at the end; `ok` false, or a rebuild that outgrew its capacities,
// ends it with steps left.
template <bool EAM, bool MIXED, int NT, int G>
__device__ __forceinline__ void team_steps(Team<NT, true>& tm, const SoloArgs& S, const TeamRun& R, GridParams& g,
                                           SoloShared<NT>& sh, LaneShared<NT>& lanes, bool& ok, long long& left,
                                           uint32_t& rebuilds, uint32_t& call) {
    const int t = tm.t;
    // a step's first half-kick and drift as a pass of its own, in place;
    // whether a rebuild is due after it
    auto drift = [&] {
        bool need = false;
        for (int i = tm.a0 + t; i < tm.a1; i += NT)
            need |= MIXED ? drift_mixed_one(S.I, S.I, i) : drift64_one(S.I, S.I, i, 1, 1);
        return tm.any(need);
    };
    int p = 0;  // the buffers that hold the positions
    bool due = ok && left > 0 && drift();
    while (ok && left > 0 && !tm.dead) {
        const bool next = left > 1 && !due;
        const bool need = team_step<EAM, MIXED, NT, G>(tm, S, R, lanes, p, next, call);
        bool due_next = false;
        if (left > 1 || due) due_next = tm.any(need);
        if (tm.dead) break;
        --left;
        ++call;
        if (next) {
            if (kFlips<EAM, MIXED>) p ^= 1;
            due = due_next;
            continue;
        }
        // the last step, or a rebuild: positions back in their own buffers
        if (p) {
            for (int i = tm.a0 + t; i < tm.a1; i += NT) {
                S.I.rx[i] = R.I1.rx[i];
                S.I.ry[i] = R.I1.ry[i];
                S.I.rz[i] = R.I1.rz[i];
                if (MIXED) S.I.pos32[i] = R.I1.pos32[i];
            }
            p = 0;
        }
        if (due) {
            ++rebuilds;
            ok = solo_rebuild<NT, true>(tm, S, g, sh);
        }
        due = ok && left > 0 && drift();
    }
}

// G: lanes per atom of the FP64 passes.
template <bool EAM, bool MIXED, int G>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_team_run(const __grid_constant__ SoloArgs S, const __grid_constant__ TeamRun R) {
    constexpr int NT = kTeamThreads;
    __shared__ GridParams g;
    __shared__ SoloShared<NT> sh;
    __shared__ LaneShared<NT> lanes;
    Team<NT, true> tm(R.word, &sh.said, S.n, R.per);
    const int t = tm.t;
    if (tm.gt == 0) {
        S.st->build_flags = 0;  // (written by others only after a barrier)
        S.st->pad[0] = 0;
    }
    if (R.hpos) {
        for (int i = tm.a0 + t; i < tm.a1; i += NT) {
            const size_t o = 3 * (size_t)S.orig[i];
            S.I.rx[i] = R.hpos[o];
            S.I.ry[i] = R.hpos[o + 1];
            S.I.rz[i] = R.hpos[o + 2];
            S.I.vx[i] = R.hvel[o];
            S.I.vy[i] = R.hvel[o + 1];
            S.I.vz[i] = R.hvel[o + 2];
        }
        if (!MIXED) team_offsets<NT>(tm, S);  // as a set of the positions does (mixed: below)
    }
    long long left = S.steps;
    uint32_t rebuilds = 0, call = S.st->therm_calls;
    bool ok = true;
    if (MIXED) {
        // the graph's prefix: rcut and boundary flags, a rebuild when an
        // upload moved atoms past the half skin, the offsets
        bool need = false;
        for (int i = tm.a0 + t; i < tm.a1; i += NT) need |= drift64_one(S.I, S.I, i, 0, 1);
        if (tm.any(need)) {
            ++rebuilds;
            ok = solo_rebuild<NT, true>(tm, S, g, sh);
        }
        team_offsets<NT>(tm, S);
    }
    team_steps<EAM, MIXED, NT, G>(tm, S, R, g, sh, lanes, ok, left, rebuilds, call);
    if (left == 0 && R.opos) {
        for (int i = tm.a0 + t; i < tm.a1; i += NT) {
            const size_t o = 3 * (size_t)S.orig[i];
            R.opos[o] = S.rx[i];
            R.opos[o + 1] = S.ry[i];
            R.opos[o + 2] = S.rz[i];
            R.ovel[o] = S.I.vx[i];
            R.ovel[o + 1] = S.I.vy[i];
            R.ovel[o + 2] = S.I.vz[i];
            if (R.oforce) {
                const bool live = !MIXED || S.F.tag[i] == 0;
                R.oforce[o] = live ? S.F.fx[i] : (double)S.F.gx[i];
                R.oforce[o + 1] = live ? S.F.fy[i] : (double)S.F.gy[i];
                R.oforce[o + 2] = live ? S.F.fz[i] : (double)S.F.gz[i];
            }
        }
    }
    // the block that ends last reports, and leaves the barriers' word at zero
    if (tm.gt == 0) {
        S.st->pad[0] = rebuilds;
        if (R.th) S.st->therm_calls = call;
        *R.left_dev = (unsigned long long)left;
    }
    __syncthreads();
    if (t == 0) {
        if (tm.dead) atomicOr(&S.st->pad[1], 1u);
        __threadfence();
        if (atomicAdd(&S.st->team_done, 1u) == gridDim.x - 1) {
            __threadfence();
            S.st->team_done = 0;
            *R.word = 0;
            const volatile uint32_t* from = reinterpret_cast<const volatile uint32_t*>(S.st);
            uint32_t* to = reinterpret_cast<uint32_t*>(R.st_host);
            for (int k = 0; k < (int)(sizeof(DevStatus) / 4); ++k) to[k] = from[k];
            S.st->pad[1] = 0;
            *R.left_host = *(volatile unsigned long long*)R.left_dev;
        }
    }
}

// A served request by a team of its own, while there are fewer requests than
// SMs: what solo_run does, with the result records written by all blocks and
// the completion record by the one that ends last.
template <bool EAM>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_team_request(const __grid_constant__ SoloArgs S, const __grid_constant__ TeamRun R) {
    constexpr int NT = kTeamThreads;
    __shared__ GridParams g;
    __shared__ SoloShared<NT> sh;
    __shared__ LaneShared<NT> lanes;
    Team<NT, true> tm(R.word, &sh.said, S.n, R.per);
    if (tm.gt == 0) {
        S.out->t_start = global_ns();
        S.out->started = S.seq;
    }
    bool ok = solo_setup<EAM>(tm, S, g, sh);
    if (ok && tm.gt == 0) {  // (after a failure other blocks may still read the flags)
        S.st->need_rebuild = 0;
        S.st->build_flags = 0;
    }
    long long left = S.steps;
    uint32_t rebuilds = 0, call = 0;
    team_steps<EAM, true, NT, 8>(tm, S, R, g, sh, lanes, ok, left, rebuilds, call);
    ok = ok && left == 0 && !tm.dead;
    tm.sync();  // every block's atoms are final
    if (ok) solo_write_atoms(tm, S);
    if (tm.gt == 0) {
        S.st->pad[0] = rebuilds;
        *R.left_dev = (unsigned long long)left;
    }
    __threadfence_system();
    __syncthreads();
    if (tm.t == 0) {
        if (tm.dead) atomicOr(&S.st->pad[1], 1u);
        __threadfence();
        if (atomicAdd(&S.st->team_done, 1u) == gridDim.x - 1) {
            __threadfence();
            S.st->team_done = 0;
            *R.word = 0;
            const volatile uint32_t* from = reinterpret_cast<const volatile uint32_t*>(S.st);
            uint32_t* to = reinterpret_cast<uint32_t*>(&S.out->st);
            for (int k = 0; k < (int)(sizeof(DevStatus) / 4); ++k) to[k] = from[k];
            const unsigned long long rest = *(volatile unsigned long long*)R.left_dev;
            S.out->left = rest;
            if (rest != 0) S.out->st.pad[1] = 1;  // void: a list outgrew its capacities
            S.out->t_end = global_ns();
            __threadfence_system();
            S.out->done = S.seq;
        }
    }
}

// Dynamic shared memory of a launch: the list build's state, one per warp.
static size_t team_dyn_bytes() { return (kTeamThreads / 32) * sizeof(NbWarpSmem<kTeamChunks>); }
static size_t solo_dyn_bytes(int threads) { return (size_t)(threads / 32) * sizeof(NbWarpSmem<kSoloChunks>); }

// Mixed systems (exclusive) whose runs go to a grid's team: as many atoms as
// its threads on 152 SMs, below which it beats the graph. Per step, graph /
// team: LJ argon 4,000 atoms 20.3 / 12.2 us, 32,000 33.5 / 25.3, 62,500
// 38.2 / 33.4, 108,000 48.0 / 45.7, 143,748 55.5 / 65.1; EAM Cu 4,000
// 24.2 / 16.0, 32,000 44.8 / 33.7, 62,500 50.5 / 43.4, 108,000 64.3 / 56.1,
// 143,748 79.6 / 91.2. FP64, where 16 or 32 lanes share an atom
// (some_atoms64): argon 500 26.4 / 19.2, 4,000 42.4 / 32.2, 19,652
// 100.9 / 98.7; Cu 500 32.9 / 27.8, 4,000 62.0 / 51.1, 8,788 98.7 / 96.8.
constexpr size_t kTeamMost = 152 * kTeamThreads;

// What both teams need of a system.
static void fill_system(SoloArgs& S, mdg_system* sys, const PotSet* dps, int any_eam, double pot_rcut, int periodic,
                        double dt, long steps) {
    memset(&S, 0, sizeof(S));
    S.I = integrator_args(sys, dt);
    S.I.pot_rcut = pot_rcut;
    S.I.periodic_boundary = periodic;
    S.np = (int)sys->np;
    S.any_eam = any_eam;
    S.F = force_args(sys);
    S.F.kick_hdt = 0.5f * (float)dt;  // the step loop's second half-kick, in the force body
    S.N = nb_args(sys);
    S.G = gather_sets(sys);
    S.D = domain_of(sys);
    S.C = cell_out(sys);
    S.ps = dps;
    S.n = (int)sys->n;
    const int c = sys->cur;
    S.rx = sys->f64[RX][c];
    S.ry = sys->f64[RY][c];
    S.rz = sys->f64[RZ][c];
    S.rns = sys->f64[RNS][c];
    S.key = sys->key;
    S.rank = sys->rank;
    S.src = sys->src;
    S.bin_count = sys->bin_count;
    S.bin_start = sys->bin_start;
    S.orig = sys->u32[ORIG][c];
    S.dgrid = sys->dgrid;
    S.bin_cap = (long long)sys->bin_cap;
    S.st = sys->dstat;
    S.steps = steps;
    S.bc = sys->bc;
}

void solo_fill(void* args, mdg_system* sys, const PotSet* dps, int any_eam, double pot_rcut, int periodic,
               double dt, long steps, const void* atoms_in_dev, void* out_dev, void* atoms_out_dev, uint32_t seq) {
    SoloArgs& S = *reinterpret_cast<SoloArgs*>(args);
    fill_system(S, sys, dps, any_eam, pot_rcut, periodic, dt, steps);
    S.setup = 1;
    S.seq = seq;
    S.atoms_in = reinterpret_cast<const mdg_atom*>(atoms_in_dev);
    S.out = reinterpret_cast<SoloOut*>(out_dev);
    S.atoms_out = reinterpret_cast<mdg_atom*>(atoms_out_dev);
}

// Whether a run of this solver on this system goes to a grid's team: LJsCut
// or EAM, Single, full lists, few enough atoms that the graph's launches are a
// good part of a step, and few enough bins (team_fits).
bool team_eligible(const mdg_solver* s, const mdg_system* sys) {
    if (s->multi || s->nstages < 1 || !s->pot[0][0] || sys->half || sys->pool || sys->ctx->timing) return false;
    const int type = s->pot[0][0]->type;
    if (type != POT_LJCUT && type != POT_EAM) return false;
    if (!sys->cap_ready || sys->n < 1 || !sys->ctx->num_sms) return false;
    if (!team_fits((long long)sys->n, sys->grid.nbins)) return false;
    if (s->precision == MDG_PREC_FP64) return sys->n < some_atoms64(type == POT_EAM);
    return sys->n < kTeamMost;
}

// A cooperative launch; kTeamTooLarge, with nothing enqueued, where the context
// cannot hold the blocks at once.
static int launch_together(const void* fn, int blocks, void** args, size_t dyn, cudaStream_t stream) {
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kTeamThreads), args, dyn, stream);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return kTeamTooLarge;
    }
    return e == cudaSuccess ? MDG_OK : cuda_status(e, "team launch");
}

// Enqueues `steps` steps by a grid's team (any host arrays page-locked); the
// steps left and the status words arrive in hcounter and hstat.
int ensure_cutbits(mdg_system* sys);

static void second_buffers(mdg_system* sys, const SoloArgs& S, TeamRun& R, int eam) {
    // the second buffers: the rebuild's spare position arrays and, for LJ, the
    // offsets' second half (the EAM records)
    R.I1 = S.I;
    R.F1 = S.F;
    R.T1 = R.T;
    R.I1.rx = sys->f64[RX][sys->cur ^ 1];
    R.I1.ry = sys->f64[RY][sys->cur ^ 1];
    R.I1.rz = sys->f64[RZ][sys->cur ^ 1];
    R.F1.rx = R.T1.rx = R.I1.rx;
    R.F1.ry = R.I1.ry;
    R.F1.rz = R.I1.rz;
    if (!eam) R.F1.pos32 = R.I1.pos32 = sys->pos32 + sys->np;
}

int team_launch(mdg_system* sys, const PotSet* dps, const ThermoDev* th, int eam, int mixed, double pot_rcut,
                int periodic, double dt, long steps, const double* hpos, const double* hvel, double* opos,
                double* ovel, double* oforce) {
    mdg_ctx* ctx = sys->ctx;
    SoloArgs S;
    fill_system(S, sys, dps, eam, pot_rcut, periodic, dt, steps);
    TeamRun R;
    memset(&R, 0, sizeof(R));
    R.hpos = hpos;
    R.hvel = hvel;
    R.opos = opos;
    R.ovel = ovel;
    R.oforce = oforce;
    R.th = th;
    R.T = thermo_args(sys);
    if (eam && mixed) {
        int rc = ensure_cutbits(sys);
        if (rc) return rc;
        S.F.cutbits = sys->cutbits;
    }
    second_buffers(sys, S, R, eam);
    R.left_dev = sys->dcounter;
    R.left_host = sys->hcounter;
    R.st_host = sys->hstat;
    // whole warps of eight-lane (mixed) or 32-lane (FP64) atoms, and at least
    // four a block
    const int n = (int)sys->n, least = mixed ? 8 : 4;
    R.per = std::max(least, ((n + ctx->num_sms - 1) / ctx->num_sms + 3) & ~3);
    const int blocks = (n + R.per - 1) / R.per;
    const bool few = sys->n < kFewAtoms64;
    const void* fn = mixed ? (eam ? (const void*)k_team_run<true, true, 8> : (const void*)k_team_run<false, true, 8>)
                     : eam ? (few ? (const void*)k_team_run<true, false, 32> : (const void*)k_team_run<true, false, 16>)
                           : (few ? (const void*)k_team_run<false, false, 32> : (const void*)k_team_run<false, false, 16>);
    if ((size_t)blocks > sys->part_cap) {
        set_error("the list was not sized for the step loop");
        return MDG_ERR_STATE;
    }
    S.part = reinterpret_cast<long long*>(sys->part);
    if (!sys->team_word) {
        int rc = sys_malloc(sys, (void**)&sys->team_word, sizeof(unsigned long long));
        if (rc) return rc;
        MDG_CUDA(cudaMemsetAsync(sys->team_word, 0, sizeof(unsigned long long), ctx->stream));
    }
    R.word = sys->team_word;
    const size_t dyn = team_dyn_bytes();
    MDG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    void* args[2] = {&S, &R};
    int rc = launch_together(fn, blocks, args, dyn, ctx->stream);
    if (rc == MDG_OK) ctx->launches++;
    return rc;
}

// Device scratch of a request's team: the barriers' word, the steps left and 8
// words of bounds per block.
size_t request_team_scratch(int blocks) { return (2 + 8 * (size_t)blocks) * sizeof(unsigned long long); }

// What a system needs before its request's team (allocated on its stream).
int request_team_prepare(mdg_system* sys, int eam) { return eam ? ensure_cutbits(sys) : MDG_OK; }

// The request whose argument record (solo_fill) is `args`, by a team of up to
// `blocks` blocks on `stream`; scratch: request_team_scratch(blocks), word 0
// zero.
int request_team_launch(const void* args, mdg_system* sys, int blocks, unsigned long long* scratch,
                        cudaStream_t stream) {
    SoloArgs S = *reinterpret_cast<const SoloArgs*>(args);
    TeamRun R;
    memset(&R, 0, sizeof(R));
    R.T = thermo_args(sys);
    if (S.any_eam) S.F.cutbits = sys->cutbits;
    second_buffers(sys, S, R, S.any_eam);
    R.word = scratch;
    R.left_dev = scratch + 1;
    S.part = reinterpret_cast<long long*>(scratch + 2);
    R.per = std::max(8, ((S.n + blocks - 1) / blocks + 3) & ~3);
    blocks = (S.n + R.per - 1) / R.per;
    const void* fn = S.any_eam ? (const void*)k_team_request<true> : (const void*)k_team_request<false>;
    const size_t dyn = team_dyn_bytes();
    MDG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    void* argv[2] = {&S, &R};
    return launch_together(fn, blocks, argv, dyn, stream);
}

bool solo_out_started(const void* out_host, uint32_t seq) {
    return reinterpret_cast<const SoloOut*>(out_host)->started == seq;
}

size_t solo_args_bytes() { return sizeof(SoloArgs); }
static_assert(sizeof(SoloArgs) % 16 == 0, "argument records are copied as 16-byte words");
size_t solo_out_bytes() { return sizeof(SoloOut); }

int solo_out_read(const void* out_host, uint32_t* done, unsigned long long* left, DevStatus* st,
                  double* service_s) {
    const SoloOut* o = reinterpret_cast<const SoloOut*>(out_host);
    *done = __atomic_load_n(const_cast<const uint32_t*>(&o->done), __ATOMIC_ACQUIRE);
    if (left) *left = o->left;
    if (st) *st = o->st;
    if (service_s) *service_s = o->t_end > o->t_start ? (double)(o->t_end - o->t_start) * 1e-9 : 0.0;
    return MDG_OK;
}

// The launch's dynamic shared memory exceeds the default 48 KB at 1024
// threads; the attribute is per device, so it is set once per device.
template <int NT>
static cudaError_t solo_prepare_attr() {
    static std::atomic<uint64_t> done{0};  // bit d: set on device d (devices 0..63)
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0ull;
    if (bit && (done.load() & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(k_solo_persistent<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)solo_dyn_bytes(NT));
    if (e == cudaSuccess && bit) done.fetch_or(bit);
    return e;
}

int solo_persistent_launch(cudaStream_t stream, int threads, int blocks, const void* desc_dev, SoloQueue* q_dev,
                           uint32_t* head, int idle_limit, int gen) {
    const SoloArgs* d = reinterpret_cast<const SoloArgs*>(desc_dev);
    if (blocks <= 0) return MDG_OK;
    if (blocks > kSoloMaxBlocks || gen < 0 || gen >= kSoloGens) return MDG_ERR_INVALID;
    const size_t dyn = solo_dyn_bytes(threads);
    if (threads == 640) {
        MDG_CUDA(solo_prepare_attr<640>());
        k_solo_persistent<640><<<blocks, 640, dyn, stream>>>(d, q_dev, head, idle_limit, gen);
    } else if (threads == 768) {
        MDG_CUDA(solo_prepare_attr<768>());
        k_solo_persistent<768><<<blocks, 768, dyn, stream>>>(d, q_dev, head, idle_limit, gen);
    } else if (threads == 896) {
        MDG_CUDA(solo_prepare_attr<896>());
        k_solo_persistent<896><<<blocks, 896, dyn, stream>>>(d, q_dev, head, idle_limit, gen);
    } else if (threads == 256) {
        MDG_CUDA(solo_prepare_attr<256>());
        k_solo_persistent<256><<<blocks, 256, dyn, stream>>>(d, q_dev, head, idle_limit, gen);
    } else if (threads == 1024) {
        MDG_CUDA(solo_prepare_attr<1024>());
        k_solo_persistent<1024><<<blocks, 1024, dyn, stream>>>(d, q_dev, head, idle_limit, gen);
    } else {
        MDG_CUDA(solo_prepare_attr<512>());
        k_solo_persistent<512><<<blocks, 512, dyn, stream>>>(d, q_dev, head, idle_limit, gen);
    }
    MDG_CUDA(cudaGetLastError());
    return MDG_OK;
}

int solo_graph_launch(SoloGraph& G, cudaStream_t stream, int threads, int blocks, const void* desc_dev,
                      SoloQueue* q_dev, uint32_t* head, int idle_limit, int gen) {
    if (blocks <= 0) return MDG_OK;
    if (blocks > kSoloMaxBlocks || gen < 0 || gen >= kSoloGens) return MDG_ERR_INVALID;
    if (!G.exec) {
        // the kernel's shared-memory attribute is set before the capture (it
        // is not a stream operation)
        int per_sm = 0;
        int rc = solo_blocks_per_sm(threads, &per_sm);
        if (rc) return rc;
        MDG_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        rc = solo_persistent_launch(stream, threads, blocks, desc_dev, q_dev, head, idle_limit, gen);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(stream, &g);
        if (rc != MDG_OK || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            return rc != MDG_OK ? rc : cuda_status(e, "persistent kernel capture");
        }
        cudaGraphNode_t node = nullptr;
        size_t nn = 1;
        e = cudaGraphGetNodes(g, &node, &nn);
        if (e == cudaSuccess && nn != 1) {
            cudaGraphDestroy(g);
            set_error("persistent kernel capture: expected one kernel node");
            return MDG_ERR_CUDA;
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&G.exec, g, 0);
        if (e != cudaSuccess) {
            cudaGraphDestroy(g);
            G.exec = nullptr;
            return cuda_status(e, "persistent kernel graph");
        }
        G.graph = g;
        G.node = node;
    } else {
        cudaKernelNodeParams p;
        MDG_CUDA(cudaGraphKernelNodeGetParams(G.node, &p));
        p.gridDim = dim3((unsigned)blocks, 1, 1);
        MDG_CUDA(cudaGraphExecKernelNodeSetParams(G.exec, G.node, &p));
    }
    MDG_CUDA(cudaGraphLaunch(G.exec, stream));
    return MDG_OK;
}

void solo_graph_destroy(SoloGraph& G) {
    if (G.exec) cudaGraphExecDestroy(G.exec);
    if (G.graph) cudaGraphDestroy(G.graph);
    G = SoloGraph();
}

int solo_blocks_per_sm(int threads, int* blocks) {
    cudaError_t e;
    const size_t dyn = solo_dyn_bytes(threads);
    if (threads == 640) {
        MDG_CUDA(solo_prepare_attr<640>());
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_solo_persistent<640>, 640, dyn);
    } else if (threads == 768) {
        MDG_CUDA(solo_prepare_attr<768>());
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_solo_persistent<768>, 768, dyn);
    } else if (threads == 896) {
        MDG_CUDA(solo_prepare_attr<896>());
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_solo_persistent<896>, 896, dyn);
    } else if (threads == 256) {
        MDG_CUDA(solo_prepare_attr<256>());
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_solo_persistent<256>, 256, dyn);
    } else if (threads == 1024) {
        MDG_CUDA(solo_prepare_attr<1024>());
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_solo_persistent<1024>, 1024, dyn);
    } else {
        MDG_CUDA(solo_prepare_attr<512>());
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_solo_persistent<512>, 512, dyn);
    }
    MDG_CUDA(e);
    return MDG_OK;
}

}  // namespace mdg
