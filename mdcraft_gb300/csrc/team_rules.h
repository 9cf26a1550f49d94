// team_rules.h — how a grid's team (solo.cu) shares out a rebuild: plain
// arithmetic, the same on the host and in the kernels.
#pragma once

namespace mdg {

// Up to this many warps share a cell of a team's list build.
constexpr int kTeamParts = 4;

// Warps that share a cell where a team has more warps than cells (of some 16
// atoms). LJ argon 13,500 atoms, a rebuild every 15 steps: 17.2 us a step by
// one, 15.6 by four; EAM Cu 32,000: 34.0 by one, 34.4 by two.
constexpr int team_parts(int warps, int n) {
    const long long p = 16LL * warps / (n > 0 ? n : 1);
    return p < 1 ? 1 : p > kTeamParts ? kTeamParts : (int)p;
}

// A list build's tasks, one per bin and part: a grid has up to 2^30 bins, so
// their number takes more than 32 bits.
constexpr long long team_tasks(int bins, int parts) { return (long long)bins * parts; }
constexpr int task_part(long long task, int bins) { return (int)(task / bins); }
constexpr int task_bin(long long task, int bins) { return (int)(task % bins); }

}  // namespace mdg
