// How large FP32 products are cut for the tensor cores: no two items of one that is
// stored share a tile, the slices cover the reduction with none empty, and what the
// kernel cannot serve is refused.
#include "gemm_split_plan.h"

#include <cstdio>

using namespace vitb200;

static int failures = 0;

static void check(bool ok, const char *what, const FmaGemm &g, const SplitPlan &plan) {
    if (!ok) {
        ++failures;
        printf("%s: [%d,%d] over %d, a_k %d b_k %d add %d: %d slices of %d blocks\n", what,
               g.m, g.n, g.k, g.a_k, g.b_k, g.accumulate, plan.slices,
               plan.blocks_per_slice);
    }
}

int main() {
    alignas(16) static float memory[8];
    const int extents[] = {1, 31, 100, 128, 129, 384, 1000, 4096, 12833, 102400};
    for (int m : extents) {
        for (int n : extents) {
            for (int k : extents) {
                for (int form = 0; form < 8; ++form) {
                    FmaGemm g = {memory, memory, memory, m, n, k, 4, 4, 4,
                                 bool(form & 1), bool(form & 2), bool(form & 4)};
                    const double error = (m + n + k) % 2 ? 1e9 : 0.0;   // none, or all
                    const SplitPlan plan = split_plan(g, 148, error);
                    const bool served = plan.clocks != HUGE_VAL;
                    // An input gradient that adds stays within the error or is refused.
                    check(served == (g.a_k ? !g.accumulate || error > 0.0
                                           : !g.b_k && g.accumulate),
                          "form", g, plan);
                    if (!served) {
                        continue;
                    }
                    check(g.accumulate || plan.slices == 1, "slices that are stored", g, plan);
                    check(plan.slices >= 1 && plan.blocks_per_slice >= 1 &&
                              (plan.slices - 1) * plan.blocks_per_slice < plan.blocks &&
                              plan.slices * plan.blocks_per_slice >= plan.blocks &&
                              plan.blocks * kSplitBlockK >= k,
                          "slices", g, plan);
                    check(plan.chunk == (error == 0.0 && g.accumulate ? 1 : 2),
                          "accumulators", g, plan);
                    // Slices are as long as the error allows.
                    check(error > 0.0 || !g.accumulate ||
                              plan.blocks_per_slice <= (plan.blocks <= 64    ? 16
                                                        : plan.blocks <= 256 ? 32 : 128),
                          "length of slices", g, plan);
                    FmaGemm whole = g;   // a bias belongs to whole sums
                    whole.bias = memory;
                    check(!g.a_k || split_plan(whole, 148, 0.0).slices == 1, "bias", g, plan);
                    g.c = memory + 1;
                    check(split_plan(g, 148, error).clocks == HUGE_VAL, "alignment", g, plan);
                    g.c = memory;
                    g.ldc = 5;
                    check(split_plan(g, 148, error).clocks == HUGE_VAL, "pitch", g, plan);
                }
            }
        }
    }
    printf("%d failures\n", failures);
    return failures != 0;
}
