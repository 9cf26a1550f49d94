// team_rules.h — what goes to a grid's team (solo.cu), how long it holds the GPU
// and how it shares out a rebuild: plain arithmetic, the same on the host and in
// the kernels.
#pragma once

namespace mdg {

// Whether a run of n atoms on a grid of so many bins goes to a team (besides
// team_eligible's rule on atoms). A team's rebuild clears and scans every bin,
// the scan by one block while the others wait; the launched rebuild scans more
// than 16,384 bins by many. A cluster in vacuum with atoms in the box's corners,
// a rebuild every 15 steps, us a step by the graph / a team: LJ argon 4,000 atoms
// with 32,768 bins 25.1 / 14.5, 64,000 25.1 / 16.8, 110,592 25.4 / 23.1, 262,144
// 24.8 / 28.8, 884,736 25.4 / 134; 19,652 atoms 31.7 / 28.3, 31.3 / 26.1, 32.1 /
// 34.2, 33.1 / 45.0, 42.2 / 169; 55,296 with 32,768 36.3 / 35.0, 110,592 37.0 /
// 42.3; 97,556 with 32,768 43.6 / 43.6, 110,592 44.5 / 51.3; EAM Cu 78,732 with
// 32,768 60.9 / 53.6, 262,144 61.9 / 65.5.
constexpr bool team_fits(long long n, long long bins) { return bins <= (n < 24000 ? 65536 : 32768); }

// The same for a served request, whose other way is one block that scans the
// bins alone as well: a team unless its blocks would wait at a barrier for a
// good part of a second.
constexpr bool request_team_fits(long long bins) { return bins <= 1LL << 24; }

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
