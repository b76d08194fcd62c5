"""The direction-chain plan is made whole or not at all: an allocation that
fails half way leaves no plan for the next caller to sweep with, and gives back
what it took.  The header's own code, compiled for the host with counting
stand-ins for the device allocations."""
import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include <new>
#include <set>
#include "chain_plan.hpp"
using namespace tycho;

static std::set<uint32_t *> live;
static int make(ChainPlan &c, int fail_at)  // 0 none; 1, 2 positions before / after allocating; 3, 4, 5 offsets
{
    auto take = [](uint32_t *&p) { p = new uint32_t[4]; live.insert(p); };
    auto positions = [&](uint32_t *&p) -> int {
        if (fail_at == 1) return kErrOom;
        take(p);
        return fail_at == 2 ? kErrCuda : kOk;
    };
    auto offsets = [&](uint32_t *&p) -> int {
        if (fail_at == 3) return kErrOom;
        if (fail_at == 4) throw std::bad_alloc();
        take(p);
        return fail_at == 5 ? kErrCuda : kOk;
    };
    auto release = [](uint32_t *p) { if (p) { live.erase(p); delete[] p; } };
    try {
        return c.make(positions, offsets, release);
    } catch (const std::bad_alloc &) {
        return -1;
    }
}

int main()
{
    const int want[6] = {kOk, kErrOom, kErrCuda, kErrOom, -1, kErrCuda};
    for (int f = 1; f <= 5; ++f) {
        ChainPlan c;
        if (make(c, f) != want[f] || c.made() || c.pos || c.off || !live.empty()) return 10 + f;
        // the next request finds no plan and makes one
        if (make(c, 0) != kOk || !c.made() || live.size() != 2) return 20 + f;
        uint32_t *pos = c.pos, *off = c.off;
        if (make(c, 3) != kOk || c.pos != pos || c.off != off) return 30 + f;  // already made
        c.drop([](uint32_t *p) { live.erase(p); delete[] p; });
        if (c.made() || c.pos || c.off || !live.empty()) return 40 + f;
    }
    std::puts("ok");
    return 0;
}
"""


def test_half_made_plan_is_no_plan(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "tycho2_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n"
