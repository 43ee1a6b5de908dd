// How a large FP32 product is cut up for the tensor cores (gemm_split.cu), and which
// products are: host arithmetic only, so that it can be checked without a GPU.
#pragma once

#include "kernels.h"

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace vitb200 {

constexpr int kSplitTile = 128, kSplitBlockK = 32;

struct SplitPlan {
    int m_tiles, n_tiles;
    int blocks, blocks_per_slice, slices;   // of the reduction
    double clocks;                          // expected; infinite: not served
};

// Slices of the reduction: of a weight gradient, which adds to C, as many as give every
// SM an item, of four blocks at least.
inline SplitPlan split_plan(const FmaGemm &g, int sms) {
    auto aligned16 = [](const void *pointer) {
        return (reinterpret_cast<uintptr_t>(pointer) & 15) == 0;
    };
    SplitPlan plan = {};
    // (A weight gradient that is stored would have its slices overwrite one another.)
    if ((!g.a_k && (g.b_k || !g.accumulate)) || g.lda % 4 != 0 || g.ldb % 4 != 0 ||
        g.ldc % 4 != 0 || !aligned16(g.a) || !aligned16(g.b) || !aligned16(g.c) ||
        (g.gelu_out && !aligned16(g.gelu_out)) ||
        (g.gelu_input && !aligned16(g.gelu_input)) || (g.bias && !aligned16(g.bias)) ||
        (g.column_partials && g.partial_row_limit < sms)) {
        plan.clocks = HUGE_VAL;
        return plan;
    }
    plan.m_tiles = (g.m + kSplitTile - 1) / kSplitTile;
    plan.n_tiles = (g.n + kSplitTile - 1) / kSplitTile;
    plan.blocks = (g.k + kSplitBlockK - 1) / kSplitBlockK;
    const long long tiles = (long long)plan.m_tiles * plan.n_tiles;
    int slices = 1;
    if (!g.a_k) {
        slices = int(std::max(1LL, std::min<long long>(sms / tiles, plan.blocks / 4)));
    }
    plan.blocks_per_slice = (plan.blocks + slices - 1) / slices;
    plan.slices = (plan.blocks + plan.blocks_per_slice - 1) / plan.blocks_per_slice;
    // The busiest SM walks its blocks in 2000 clocks each; what a tile takes before its
    // first products and after its last makes up the rest.
    const long long rounds = (tiles * plan.slices + sms - 1) / sms;
    plan.clocks = 13000.0 + 2000.0 * double(rounds * plan.blocks_per_slice);
    return plan;
}

}  // namespace vitb200
