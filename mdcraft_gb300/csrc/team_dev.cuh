// team_dev.cuh — the blocks that run one system together (solo.cu) and the
// barrier they meet at.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mdg {

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// How long a team's barrier waits for its blocks before it gives up: ten
// seconds, against rebuild phases of microseconds. The clock is read once in
// kTeamLook polls (each an L2 round trip of some tenths of a microsecond), and
// the polls have a limit of their own.
constexpr unsigned long long kTeamWaitNs = 10000000000ull;
constexpr uint32_t kTeamLook = 4096, kTeamPolls = 1u << 30;

// The blocks that run one system together and this thread's share of it:
// atoms a0 .. a1 of the block, thread gt of gn, warp gw of nw. WIDE: a grid of
// blocks; else one block.
//
// The grid's barrier is one 64-bit word: arrivals in its low half, votes in
// two counters above it, for barriers of even and odd number (a block may
// stand at the next barrier when a slow one reads the word, but never
// further). A block's first thread adds and polls. No field may carry into
// the next one: counts are compared without the field's top bit, and the
// first block takes that bit out once it is set. (A word per block that
// every block reads took 4 to 6 us against 2 here: 143 x 143 polls.) WAIT: the
// barrier's limit in ns.
template <int NT, bool WIDE, unsigned long long WAIT = kTeamWaitNs>
struct Team {
    int t, lane, w, rank, size, a0, a1, gt, gn, gw, nw;
    bool dead = false;  // a barrier gave up; the run is void
    uint32_t epoch = 0;             // barriers passed
    uint32_t cast[2] = {0, 0};      // votes counted so far at even and odd barriers
    unsigned long long* word;       // zero at the kernel's start
    int* said;                      // shared: bit 0 the vote, bit 1 a wait ran out

    __device__ __forceinline__ Team(unsigned long long* wd, int* flag, int n, int per) : word(wd), said(flag) {
        t = threadIdx.x;
        lane = t & 31;
        w = t >> 5;
        rank = WIDE ? (int)blockIdx.x : 0;
        size = WIDE ? (int)gridDim.x : 1;
        a0 = WIDE ? min(rank * per, n) : 0;
        a1 = WIDE ? min(a0 + per, n) : n;
        gt = rank * NT + t;
        gn = size * NT;
        gw = w * size + rank;  // neighbouring tasks on different blocks
        nw = size * (NT / 32);
    }
    // Every block's writes before are visible to every block after; whether
    // any thread of the team has `vote` set.
    __device__ __forceinline__ bool any(bool vote) {
        const int mine = __syncthreads_or(vote);
        if (!WIDE || dead) return mine != 0;
        ++epoch;
        if (t == 0) {
            const int odd = epoch & 1, at = 32 + 16 * odd;
            __threadfence();
            atomicAdd(word, 1ull + ((unsigned long long)(mine ? 1 : 0) << at));
            const uint32_t target = epoch * (uint32_t)size;
            unsigned long long v, since = 0;
            uint32_t polls = 0;
            bool wait;
            do {
                v = *(volatile unsigned long long*)word;
                wait = (((uint32_t)v - target) & 0x7fffffffu) >= 0x40000000u;
                if (wait && ++polls % kTeamLook == 0) {
                    const unsigned long long now = global_ns();
                    if (!since) since = now;
                    if (now - since > WAIT || polls >= kTeamPolls) break;
                }
            } while (wait);
            __threadfence();
            const uint32_t sum = (uint32_t)(v >> at) & 0x7fffu;
            *said = (sum != cast[odd] ? 1 : 0) | (wait ? 2 : 0);
            cast[odd] = sum;
            const unsigned long long top = v & 0x8000800080000000ull;
            if (rank == 0 && top) atomicAdd(word, 0ull - top);
        }
        __syncthreads();
        const int s = *said;
        dead = (s & 2) != 0;
        return (s & 1) != 0;
    }
    __device__ __forceinline__ void sync() {
        if (WIDE) any(false);
        else __syncthreads();
    }
};

}  // namespace mdg
