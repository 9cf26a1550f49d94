// team_rules.h — how long a grid's team (solo.cu) holds the GPU and how it shares
// out a rebuild: plain arithmetic, the same on the host and in the kernels.
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

// A run's launches are of about this many microseconds: what else wants the GPU
// waits for one of them. A launch costs some 15 us. (At 256 steps a launch they
// were 3 ms for LJ argon of 4,000 atoms and 25 ms for 19,652 in FP64.)
constexpr double kTeamLaunchUs = 4000.0;

// What a step of n atoms with room for K neighbours each may take, in us, before
// one has been timed: somewhat more than the times beside kTeamMost (solo.cu).
constexpr double team_step_us(long long n, int K, bool fp64, bool eam) {
    return 12.0 + (double)n * K * (fp64 ? (eam ? 110e-6 : 50e-6) : 5e-6);
}

// Steps of the next launch, at step_us a step.
constexpr long team_steps(long left, double step_us) {
    const double s = kTeamLaunchUs / step_us;
    const long most = s >= 1e6 ? 1000000 : s >= 1.0 ? (long)s : 1;
    return left < most ? left : most;
}

}  // namespace mdg
