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
    int chunk;                              // blocks that a main accumulator lives for
    double clocks;                          // expected; infinite: not served
};

// Errors of sums of positive terms (nothing cancels, and what is cut off adds up), squared
// and in units of 1e-14, as measured in the 2-norm against 64 bits over 300 to 30000 terms
// and 17 widths.  FMAs, in slices of `terms`: a rounding per term, averaged over the
// slices, and one per slice (measured: 0.92 to 1.16 of the root of this).
inline double fma_error(double terms, int slices) {
    return 0.0207 * (terms / slices + slices);
}
// Split: what the tensor core cuts off of accumulators that live for `chunk` blocks, a
// rounding per accumulator and one per slice (0.83 to 1.05).
inline double split_error(int blocks, int slices, int chunk) {
    return chunk == 2 ? std::max(0.70 + 0.01 * slices, 0.42 + 0.0225 * slices) +
                            0.0235 * ((blocks + 1) / 2) / slices
                      : std::max(0.29 + 0.01 * slices, 0.10 + 0.0225 * slices) +
                            0.0164 * blocks / slices;
}

// A product that adds to C is cut into slices: a weight gradient into as many as give
// every SM an item, of four blocks at least, where that stays within `error`, which is
// that of the FMA plan it replaces.  Where it does not, accumulators live for one block
// (half of what is cut off; 3 to 10 % slower); where that does not do either, slices are
// of at most 512 terms (1024 from 2048 on, 4096 from 8192 on): of the cuts within `error`
// the one that is expected to be the fastest.  Where there is none, an input gradient is
// left to the FMAs and a weight gradient takes the cut with the smallest error.
// Measured errors x 1e-7 (FMAs, as many slices as give every SM an item, this):
// [512,2048] over 2048 rows 0.70, 0.86, 0.60, over 4096 0.80, 0.94, 0.65, [512,512] over
// 1600 0.73, 0.82, 0.59, [128,512] over 10000 1.03, 1.13, 1.00.
inline SplitPlan split_plan(const FmaGemm &g, int sms, double error) {
    auto aligned16 = [](const void *pointer) {
        return (reinterpret_cast<uintptr_t>(pointer) & 15) == 0;
    };
    SplitPlan plan = {};
    // (A weight gradient that is stored would have its slices overwrite one another.)
    if (g.k < 1 || (!g.a_k && (g.b_k || !g.accumulate)) || g.lda % 4 != 0 ||
        g.ldb % 4 != 0 || g.ldc % 4 != 0 || !aligned16(g.a) || !aligned16(g.b) || !aligned16(g.c) ||
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
    auto each = [&](int slices) { return (plan.blocks + slices - 1) / slices; };
    const int even =
        int(std::max(1LL, std::min<long long>(sms / tiles, plan.blocks / 4)));
    plan.slices = g.a_k ? 1 : even;
    plan.chunk = 2;
    // (Bias, GELU and column sums belong to whole sums.)
    const bool cut = g.accumulate && !g.bias && !g.gelu_out && !g.gelu_input &&
                     !g.column_partials;
    if (cut && split_error(each(plan.slices), plan.slices, 2) > error) {
        plan.chunk = 1;
    }
    if (cut && split_error(each(plan.slices), plan.slices, plan.chunk) > error) {
        const int least = each(plan.blocks <= 64 ? 16 : plan.blocks <= 256 ? 32 : 128);
        double shortest = 0.0, closest = 0.0;
        int closest_slices = least;
        for (int slices = least; slices <= std::max(2 * least, even); ++slices) {
            const double rounds = double((tiles * slices + sms - 1) / sms);
            const double cost = rounds * (each(slices) + 4);
            const double off = split_error(each(slices), slices, 1);
            if (closest == 0.0 || off < closest) {
                closest = off;
                closest_slices = slices;
            }
            if (off <= error && (shortest == 0.0 || cost < shortest)) {
                shortest = cost;
                plan.slices = slices;
            }
        }
        if (shortest == 0.0) {
            if (g.a_k) {
                plan.clocks = HUGE_VAL;
                return plan;
            }
            plan.slices = closest_slices;
        }
    }
    plan.blocks_per_slice = each(plan.slices);
    plan.slices = (plan.blocks + plan.blocks_per_slice - 1) / plan.blocks_per_slice;
    // The busiest SM walks its blocks in 2000 clocks each; what a tile takes before its
    // first products and after its last makes up the rest.
    const long long rounds = (tiles * plan.slices + sms - 1) / sms;
    plan.clocks = 13000.0 + 2000.0 * double(rounds * plan.blocks_per_slice);
    return plan;
}

}  // namespace vitb200
