"""The barrier of a grid's team (mdcraft_gb300/csrc/team_dev.cuh) by itself:
votes over counters that wrap, and a wait that runs out.

A small program is compiled with the header and run as a process of its own.
Nothing in it waits without a limit: the wait that runs out is for a block that
was never launched, five milliseconds long, and ends with the status it sets."""
from __future__ import annotations

import os
import subprocess

import pytest

from mdcraft_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = r"""
#include <cstdio>
#include <cstring>
#include "mdg_host.h"
#include "team_dev.cuh"
using namespace mdg;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
#define OK(x) CHECK((x) == cudaSuccess)
"""

HOST = HEAD + r"""
int main() {
    mdg_system s;
    s.have_list = s.cap_ready = 1;
    s.dirty = 0;
    forget_list(&s);
    CHECK(s.have_list == 0 && s.cap_ready == 0 && s.dirty == 1);
    return 0;
}
"""

DEVICE = HEAD + r"""
constexpr int NT = 64;
__host__ __device__ inline bool votes(unsigned k, unsigned block) {
    const unsigned x = (k * 2654435761u) ^ (block * 40503u);
    return k % 1024 < 600 ? true : (x >> 13) % 16 == 0;
}
// Barriers of votes; bad: outcomes that are not the blocks' votes.
__global__ void k_votes(unsigned long long* word, unsigned first, unsigned rounds, unsigned* bad, unsigned* dead) {
    __shared__ int said;
    Team<NT, true> tm(word, &said, NT * gridDim.x, NT);
    tm.epoch = first;
    for (unsigned k = 0; k < rounds && !tm.dead; ++k) {
        bool expect = false;
        for (unsigned b = 0; b < gridDim.x; ++b) expect |= votes(k, b);
        const bool any = tm.any(tm.t == 5 && votes(k, blockIdx.x));
        if (any != expect && tm.t == 0 && !tm.dead) atomicAdd(bad, 1u);
    }
    if (tm.dead && tm.t == 0) atomicAdd(dead, 1u);
}
// A barrier that waits for one block more than there are.
__global__ void k_alone(unsigned long long* word, unsigned* dead) {
    __shared__ int said;
    Team<NT, true, 5000000ull> tm(word, &said, NT * gridDim.x, NT);
    tm.size += 1;
    tm.any(false);
    tm.any(true);  // no second wait
    if (tm.dead && tm.t == 0) atomicAdd(dead, 1u);
}
int main() {
    unsigned long long* word;
    unsigned *out, h[2];
    OK(cudaMalloc(&word, 8));
    OK(cudaMalloc(&out, 8));
    const int blocks = 24;
    // the arrivals' counter starts at nothing, and just below 2^31 and 2^32
    for (unsigned first : {0u, 2147483648u / blocks - 5u, 4294967295u / blocks - 5u}) {
        unsigned long long w = (unsigned)(first * blocks) & 0x7fffffffu;
        unsigned rounds = 70000;
        OK(cudaMemcpy(word, &w, 8, cudaMemcpyHostToDevice));
        OK(cudaMemset(out, 0, 8));
        unsigned *bad = out, *dead = out + 1;
        void* args[] = {&word, &first, &rounds, &bad, &dead};
        OK(cudaLaunchCooperativeKernel((const void*)k_votes, dim3(blocks), dim3(NT), args, 0, 0));
        OK(cudaDeviceSynchronize());
        OK(cudaMemcpy(h, out, 8, cudaMemcpyDeviceToHost));
        CHECK(h[0] == 0 && h[1] == 0);
    }
    OK(cudaMemset(word, 0, 8));
    OK(cudaMemset(out, 0, 8));
    void* args[] = {&word, &out};
    cudaEvent_t a, b;
    OK(cudaEventCreate(&a));
    OK(cudaEventCreate(&b));
    OK(cudaEventRecord(a));
    OK(cudaLaunchCooperativeKernel((const void*)k_alone, dim3(4), dim3(NT), args, 0, 0));
    OK(cudaEventRecord(b));
    OK(cudaDeviceSynchronize());
    float ms = 0;
    OK(cudaEventElapsedTime(&ms, a, b));
    OK(cudaMemcpy(h, out, 4, cudaMemcpyDeviceToHost));
    std::printf("gave up after %.1f ms\n", ms);
    CHECK(h[0] == 4 && ms > 4.0f && ms < 500.0f);
    return 0;
}
"""


def _program(tmp_path, text):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(text)
    inc = [f"-I{os.path.join(ROOT, d)}" for d in ("mdcraft_gb300/csrc", "include")]
    subprocess.run([B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", *inc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_lost_system_has_no_list(tmp_path):
    """What a run leaves whose team gave up: no list and no capacities, so that
    stages and runs refuse the system (its list lengths may be anything)."""
    _program(tmp_path, HOST)


@pytest.mark.gpu
def test_votes_and_a_wait_that_runs_out(tmp_path):
    _program(tmp_path, DEVICE)
