"""The cut of a lattice (csrc/step_plan.h) against a search of every chunk length:
the same plan for random sizes, in a bounded number of estimates (a call of the
step on device buffers makes the plan anew, so a tall lattice must not take
longer)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "entropicthreadsafe_b200", "csrc")
SOURCE = r"""
#include "step_plan.h"
#include <chrono>
#include <cmath>
#include <cstdio>
#include <random>
using namespace tslb;
static StepPlan full(int nx, int ny, int nz, bool xper, const PlanCosts& costs, int sms) {
    StepPlan best{BIGW, 1, nz, 0};
    double least = 1e300;
    const long long tx = (xper && nx <= 32) ? 1 : (nx + LXV - 1LL) / LXV;
    for (int w : {BIGW, SMALLW}) {
        const int th = even_rows(ny, w - 2), bps = BIGW / w;
        const long long ty = (ny + th - 1LL) / th, slots = (long long)bps * sms;
        auto plane = [&](long long blocks) { return w == BIGW ? 2.0 : blocks <= sms ? costs.one : costs.two; };
        for (int nc = 1; nc <= nz; ++nc) {
            const int zc = (nz + nc - 1) / nc;
            const long long blocks = tx * ty * ((nz + zc - 1) / zc);
            const double cost = (double)((blocks + slots - 1) / slots) * (zc + 3.0) * plane(blocks) + costs.tail * zc;
            if (cost < least) { least = cost; best = StepPlan{w, th, zc, 0}; }
            if (nc > 1 && blocks > 16 * slots) break;
        }
        const long long parts = std::min(slots / tx, ty * nz);
        if (costs.tail == 0.0 && parts > 0 && ty * nz < (1LL << 31)) {
            const double share = (double)(ty * nz) / parts;
            const double cost = costs.share * (share + 3.0 * (share / nz + 1.0)) * plane(parts * tx);
            if (cost < least) { least = cost; best = StepPlan{w, th, 0, (int)(parts * tx)}; }
        }
    }
    return best;
}
template <class F>
static double time_of(F f) {
    double best = 1e9;
    for (int r = 0; r < 7; ++r) {
        const auto t0 = std::chrono::steady_clock::now();
        volatile int sink = 0;
        for (int i = 0; i < 200; ++i) sink = sink + f(16, 16, 4096 + (i & 1), true, kEvenCosts, 148).zchunk;
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
    }
    return best;
}
int main() {
    std::mt19937 rng(5);
    auto size = [&](int top) { return (int)std::exp(std::uniform_real_distribution<double>(0, std::log((double)top))(rng)); };
    int bad = 0;
    for (int i = 0; i < 20000; ++i) {
        const int top = i % 4 == 0 ? 40 : i % 4 == 1 ? 400 : 5000;
        const int nx = size(top), ny = size(top), nz = size(i % 7 == 0 ? 60000 : top), sms = i % 5 ? 148 : 1 + size(200);
        const bool xper = rng() & 1;
        const PlanCosts all[4] = {kEvenCosts, kEven16Costs, kPhaseCosts, kUnevenCosts}, costs = all[rng() % 4];
        const StepPlan a = step_plan(nx, ny, nz, xper, costs, sms), b = full(nx, ny, nz, xper, costs, sms);
        if (a.warps != b.warps || a.th != b.th || a.zchunk != b.zchunk || a.grid != b.grid) {
            if (bad++ < 5) std::printf("%d x %d x %d %d %.2f %d: %d %d %d %d, full search %d %d %d %d\n", nx, ny, nz, xper, costs.tail, sms,
                                       a.warps, a.th, a.zchunk, a.grid, b.warps, b.th, b.zchunk, b.grid);
        }
    }
    std::printf("different %d\nfaster %.1f\n", bad, time_of(full) / time_of(step_plan));
}
"""


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-o", str(d / "plan"), str(d / "plan.cpp")], check=True)
    return subprocess.run([str(d / "plan")], capture_output=True, text=True, check=True).stdout


def test_same_plan_as_the_full_search(report):
    assert "different 0\n" in report, report


def test_tall_lattices_take_no_longer(report):
    """16 x 16 x 4096: about 35 estimates against 4,700; a factor of 10 leaves room for the machine."""
    assert float(report.split("faster ")[1]) > 10.0, report
