"""Who has work on a device (mdcraft_gb300/csrc/device_use.h), compiled and run
on the host: a thread counts once however its calls nest, other threads and
requests are seen."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <optional>
#include <thread>
#include "device_use.h"
using namespace mdg;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
    CHECK(DeviceHold::in_flight(0) == 0 && DeviceUse::threads(0) == 0);
    {
        const DeviceUse run(0);
        CHECK(run.alone() && DeviceUse::threads(0) == 1);
        {
            const DeviceUse inner(0);  // an entry point called by another
            CHECK(inner.alone() && run.alone() && DeviceHold::in_flight(0) == 1);
            const DeviceUse other(1);
            CHECK(run.alone() && other.alone());
        }
        CHECK(run.alone());
        bool seen = true, own = true;
        std::thread t([&] {
            const DeviceUse stage(0);
            if (DeviceUse::threads(0) != 2) return;
            own = stage.alone();
            seen = run.alone();
        });
        t.join();
        CHECK(!seen && !own && run.alone());
        std::optional<DeviceHold> request;
        request.emplace(0);
        CHECK(!run.alone() && DeviceUse::threads(0) == 1);
        request.reset();
        CHECK(run.alone());
    }
    CHECK(DeviceHold::in_flight(0) == 0 && DeviceHold::in_flight(1) == 0 && DeviceUse::threads(0) == 0);
    return 0;
}
"""


def test_uses_nest_and_are_seen(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", os.path.join(ROOT, "mdcraft_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
