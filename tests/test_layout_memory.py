"""Layouts that find no host memory (CPU): a reason, no exception.

The planners are compiled with an `operator new` that fails once a chosen number of allocations has
succeeded.  For every such number, up to the one with which the layout is built, each planner
must return a reason; the runtime then solves without the layout, and nothing leaves a C entry.
"""
import os
import subprocess

from physik_b200 import _lib as L

SOURCE = r"""
#include "pk_res_plan.h"
#include "pk_slab_plan.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
static std::atomic<long> left{-1};
void* operator new(std::size_t size)
{
    if (left.load() >= 0 && left.fetch_sub(1) <= 0) {
        left = 0;  // and all later ones
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(size ? size : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
    constexpr int n = 5000, band = 6;
    std::vector<int> rs(1, 0), col, lts(n + 1, 0), ltr, ltb;
    for (int r = 0; r < n; ++r) {
        for (int c = r; c < n && c < r + band; ++c) col.push_back(c);
        rs.push_back((int)col.size());
    }
    for (int r = 0; r < n; ++r) {
        for (int c = r > band - 1 ? r - band + 1 : 0; c < r; ++c) {
            ltr.push_back(c);
            ltb.push_back(rs[c] + r - c);
        }
        lts[r + 1] = (int)ltr.size();
    }
    std::vector<double> xyz(3 * n, 0.0);
    for (int r = 0; r < n; ++r) xyz[3 * r] = r;
    const int seg[2] = {0, n};
    for (int kind = 0; kind < 6; ++kind) {
        long refused = 0;
        for (long k = 0;; k += 1 + k / 40) {
            std::string why;
            {
                pk::SlabPlan slab;
                pk::ResPlan res;
                pk::ResLimits limits;
                limits.blocks = 148;
                left = k;
                if (kind < 3)
                    why = pk::build_slab_plan(n, rs.data(), col.data(), lts.data(), ltr.data(), ltb.data(), xyz.data(),
                                              16, slab, kind == 1 ? pk::kSlabSym : pk::kSlabFull, kind == 2);
                else if (kind == 3)
                    why = pk::build_slab_plan_batched(n, rs.data(), col.data(), lts.data(), ltr.data(), ltb.data(),
                                                      xyz.data(), seg, 1, 16, slab, pk::kSlabFull);
                else
                    why = pk::build_res_plan(n, rs.data(), col.data(), lts.data(), ltr.data(), ltb.data(), xyz.data(),
                                             seg, 1, limits, kind == 4 ? 4 : 8, res);
                left = -1;
            }
            if (why.empty()) break;
            ++refused;
        }
        std::printf("%ld\n", refused);
    }
}
"""


def test_a_layout_without_memory_gives_a_reason(tmp_path):
    kernels = os.path.join(L.ROOT, "physik_b200", "csrc", "kernels")
    source, program = tmp_path / "plans.cpp", tmp_path / "plans"
    source.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", kernels, str(source),
                    os.path.join(kernels, "pk_slab_plan.cpp"), os.path.join(kernels, "pk_res_plan.cpp"), "-o",
                    str(program)], check=True)
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, (run.returncode, run.stderr[-500:])
    refused = [int(r) for r in run.stdout.split()]
    assert len(refused) == 6 and min(refused) > 10, refused
