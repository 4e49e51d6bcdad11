"""bind_angles sets all of a plan's numbers or, when the host runs out of memory,
none of them: the engine's plan cache binds cached plans in place, and a plan of
half the old and half the new angles would answer later calls.  A small program
around planner.cpp makes each allocation of a call fail in turn."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "quantumsimevo_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "planner.h"
#include "qse_internal.h"

static long left = -1;   // allocations until one fails, -1: none does

void* operator new(std::size_t n)
{
    if (left >= 0 && left-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

namespace qse {
void fail(int status, const std::string& msg) { throw Error(status, msg); }
}
using namespace qse::plan;

// zz: CNOT RZ CNOT triples (fused where the options say so) among single-qubit gates
static std::vector<Gate> circuit(double shift)
{
    std::vector<Gate> g;
    unsigned r = 1;
    auto rnd = [&](unsigned m) {
        r = r * 1664525u + 1013904223u;
        return (r >> 8) % m;
    };
    for (int i = 0; i < 400; ++i) {
        Gate a;
        a.t = rnd(9);
        a.theta = 0.01 * i + shift;
        const int kind = int(rnd(5));
        a.type = kind == 0 ? QSE_GATE_RX : kind == 1 ? QSE_GATE_RY : kind == 2 ? QSE_GATE_RZ : kind == 3 ? QSE_GATE_2X2 : QSE_GATE_CNOT;
        if (kind == 3) {
            a.m[0] = a.m[6] = std::cos(a.theta);
            a.m[3] = a.m[5] = std::sin(a.theta);
        }
        if (kind == 4) {
            a.c = (a.t + 1) % 9;
            Gate z = a;
            z.type = QSE_GATE_RZ;
            g.push_back(a);
            g.push_back(z);
        }
        g.push_back(a);
    }
    return g;
}

static bool same(const Plan& a, const Plan& b)
{
    auto eq = [](const auto& x, const auto& y) {
        return x.size() == y.size() && (x.empty() || std::memcmp(x.data(), y.data(), x.size() * sizeof x[0]) == 0);
    };
    for (size_t i = 0; i < a.passes.size(); ++i)
        if (!eq(a.passes[i].ops, b.passes[i].ops) || !eq(a.passes[i].terms, b.passes[i].terms) ||
            !eq(a.passes[i].mats, b.passes[i].mats))
            return false;
    return a.passes.size() == b.passes.size();
}

int main(int argc, char** argv)
{
    Options opt;
    opt.k = 6;
    opt.rb = 3;
    opt.unit_rot = std::atoi(argv[1]);
    opt.zz_fuse = std::atoi(argv[2]);
    uint32_t perm[64];
    for (uint32_t q = 0; q < 64; ++q) perm[q] = q;
    const std::vector<Gate> before = circuit(0.0), after = circuit(0.5);
    const Plan old = build(before, 9, perm, opt), want = build(after, 9, perm, opt);
    if (same(old, want)) return std::puts("the angles make no difference"), 1;
    for (long n = 0;; ++n) {
        Plan p = old;
        bool threw = false;
        left = n;
        try {
            bind_angles(p, after, opt);
        } catch (const std::bad_alloc&) {
            threw = true;
        }
        left = -1;
        if (!threw) {
            if (!same(p, want)) return std::puts("bound numbers differ from planned ones"), 1;
            break;
        }
        if (!same(p, old)) return std::printf("allocation %ld failed and left a half-bound plan\n", n), 1;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("rebind")
    src = d / "rebind.cpp"
    src.write_text(PROGRAM)
    exe = d / "rebind"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}/include", "-o", str(exe), str(src),
                    os.path.join(CSRC, "planner.cpp")], check=True)
    return str(exe)


@pytest.mark.parametrize("unit_rot", [0, 1])
@pytest.mark.parametrize("zz_fuse", [0, 1])
def test_all_numbers_or_none(program, unit_rot, zz_fuse):
    r = subprocess.run([program, str(unit_rot), str(zz_fuse)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
