"""The arithmetic by which a grid's team shares out a rebuild
(mdcraft_gb300/csrc/team_rules.h), compiled and run on the host."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mdcraft_gb300", "csrc")


def _run(tmp_path, body):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include "team_rules.h"\n#include <cstdio>\n#include <initializer_list>\nusing namespace mdg;\n'
                   "#define CHECK(x) do { if (!(x)) { std::printf(\"%s\\n\", #x); return 1; } } while (0)\n"
                   "int main() {\n" + body + "\nreturn 0; }\n")
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_tasks_of_the_largest_grids(tmp_path):
    """Every bin and part once, also where their number exceeds 2^31 (a grid has
    up to 2^30 bins)."""
    _run(tmp_path, """
    for (int bins : {1, 64, 1000, 1 << 20, 600000000, 715827883, 1 << 30})
        for (int parts = 1; parts <= kTeamParts; ++parts) {
            const long long tasks = team_tasks(bins, parts);
            CHECK(tasks / parts == bins && tasks % parts == 0);
            for (int p = 0; p < parts; ++p)
                for (long long b : {0LL, 1LL, bins / 2LL, bins - 1LL}) {
                    if (b >= bins) continue;
                    const long long t = p * (long long)bins + b;
                    CHECK(t < tasks);
                    CHECK(task_part(t, bins) == p && task_bin(t, bins) == (int)b);
                }
            CHECK(task_part(tasks - 1, bins) == parts - 1 && task_bin(tasks - 1, bins) == bins - 1);
        }
    """)


def test_parts(tmp_path):
    """One to four warps a cell, and more only where there are warps to spare."""
    _run(tmp_path, """
    int last = kTeamParts;
    for (int n = 1; n < 200000; ++n) {
        const int p = team_parts(152 * 24, n);
        CHECK(p >= 1 && p <= last);
        last = p;
    }
    CHECK(team_parts(75 * 24, 8000) == 3 && team_parts(152 * 24, 8000) == 4 && team_parts(152 * 24, 58369) == 1);
    """)


def test_steps_of_a_launch(tmp_path):
    """About kTeamLaunchUs of steps, never none, never more than are left; the
    guess before a step was timed grows with the pairs."""
    _run(tmp_path, """
    CHECK(team_steps(1, 1e9) == 1 && team_steps(50, 1e9) == 1 && team_steps(7, 0.0) == 7);
    CHECK(team_steps(1L << 40, 0.0) == 1000000 && team_steps(1L << 40, 1e-12) == 1000000);
    for (double us : {0.5, 12.2, 98.7, 3999.0, 4001.0})
        for (long left : {1L, 10L, 1000000L}) {
            const long k = team_steps(left, us);
            CHECK(k >= 1 && k <= left && (k == 1 || k * us <= kTeamLaunchUs));
            CHECK(k == left || (k + 1) * us > kTeamLaunchUs);
        }
    // FP64 argon of 19,652 atoms takes 98.7 us a step: 256 steps were 25 ms
    CHECK(team_steps(256, team_step_us(19652, 100, true, false)) <= 45);
    CHECK(team_step_us(4000, 100, false, false) < 20.0);
    for (int k = 0; k < 4; ++k)
        CHECK(team_step_us(116000, 400, k & 1, k & 2) > team_step_us(116000, 100, k & 1, k & 2));
    """)


def test_bins_of_a_team(tmp_path):
    """Runs: 65,536 bins below 24,000 atoms, 32,768 from there on; requests: as
    many as the launched scan takes. None where a task would not be an int's."""
    _run(tmp_path, """
    CHECK(team_fits(1, 65536) && !team_fits(1, 65537) && team_fits(23999, 65536));
    CHECK(team_fits(24000, 32768) && !team_fits(24000, 32769) && !team_fits(1, 1 << 30));
    CHECK(request_team_fits(1 << 24) && !request_team_fits((1 << 24) + 1) && !request_team_fits(1 << 30));
    """)
