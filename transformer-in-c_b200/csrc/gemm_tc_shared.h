// Shared memory of a tensor-core product's CTA (gemm_tc.cu): ring of load stages,
// staging blocks of the epilogue warps, mbarriers.  Host arithmetic only, so that every
// tile, epilogue and switch can be checked without a GPU.
#pragma once

#include <algorithm>

namespace vitb200 {

constexpr int kTileM = 128;
constexpr int kTileN = 128;                 // narrow tiles; the wide variant is 256
constexpr int kBlockK = 32;                 // 128 bytes of FP32 per row
constexpr int kOperandBytes = kTileM * kBlockK * 4;   // 16 KiB
constexpr int kStagingBlock = 32 * 32 * 4;  // what an epilogue warp stages at a time
// Upper bound on the load ring; the launch code picks the depth that fits
// beside the epilogue staging for the chosen number of CTAs per SM.
constexpr int kMaxStages = 8;
constexpr int kSmemLimit = 227 * 1024 - 1024;   // leave room for static shared memory
constexpr int kBarrierBytes = 320;   // 2 x kMaxStages + 4 + 16 mbarriers, TMEM slot

// What the epilogue does with a second matrix.
constexpr int kSecondGelu = 1;       // D = A*B + bias, D2 = gelu(D)
constexpr int kSecondResidual = 2;   // D = A*B + bias, D2 = D + residual
// D = (A*B) * gelu'(H): the backward pass through a GELU folded into the
// product that computes the GELU output's gradient.  H is read through
// map_d2 (one 32 x 32 block per accumulator block, by TMA into the block the
// result is then staged in); there is one output.
constexpr int kGeluSlope = 3;
// The same with eight epilogue warps of one staging block each on the square tile.
constexpr int kGeluSlopeEight = 4;

// The tall tile has a group of four epilogue warps for each of its two
// accumulators, so that both drain at the same time.  So have the GELU's two
// epilogues on the tiles that large products run on, whose warps wait for memory
// between their arithmetic: more of them wait at a time.
constexpr bool tc_two_groups(int tile_m, int tile_n, int second) {
    return tile_m == 2 * kTileM ||
           (tile_n == 256 && (second == kSecondGelu || second == kGeluSlope)) ||
           second == kGeluSlopeEight;
}

constexpr int tc_epilogue_warps(int tile_m, int tile_n, int second) {
    return tc_two_groups(tile_m, tile_n, second) ? 8 : 4;
}

// The least staging that the epilogue writes: a block for each of its warps, two where
// the slope's operand is fetched a block ahead.
constexpr int tc_least_staging(int tile_m, int tile_n, int second) {
    return tc_epilogue_warps(tile_m, tile_n, second) * kStagingBlock *
           (second == kGeluSlope ? 2 : 1);
}

// The environment's tuning switches, 0 where not set.
struct TcForced {
    int stages = 0, staging = 0, ctas = 0;
};

struct TcShared {
    int stages, stage_bytes, staging_bytes, ctas_per_sm;
    int bytes() const { return stages * stage_bytes + staging_bytes + kBarrierBytes; }
};

// spread: a CTA of a narrow tile has its SM to itself.
inline TcShared tc_shared(int tile_m, int tile_n, int second, int k_blocks, bool accumulate,
                          bool spread, const TcForced &forced) {
    const bool slope = second == kGeluSlope || second == kGeluSlopeEight;
    TcShared s;
    s.stage_bytes = (tile_m + tile_n) * kBlockK * 4;
    // Two persistent CTAs per SM, each with a 2-stage load ring and 32 KiB of
    // epilogue staging (97 KiB): they interleave their MMA issue and their
    // epilogues, and measured faster than one CTA with a 4- to 6-stage ring
    // at every size tried (449 against 346 TFLOP/s at [100864,512]x[512,2048]).
    // A single output can give up the second staging buffer of each epilogue
    // warp for a third load stage: more bytes in flight, which is what the
    // short-K, bandwidth-bound products of this model lack.
    s.staging_bytes = 2 * kOperandBytes;
    s.ctas_per_sm = 2;
    s.stages = 2;
    if (second != kSecondResidual && !slope) {
        // (Also the GELU pair: its two outputs share each warp's block.)
        s.stages = 3;
        s.staging_bytes = kOperandBytes;
    }
    if (forced.stages > 0 && forced.stages <= kMaxStages) {
        s.stages = forced.stages;
    }
    if (forced.ctas > 0) {
        s.ctas_per_sm = forced.ctas;
    }
    if (tile_n > kTileN) {
        // One CTA per SM (it owns all of tensor memory): four 48 KiB stages
        // and double-buffered staging, 224 KiB.
        s.ctas_per_sm = 1;
        s.stages = tile_m > kTileM ? 3 : 4;   // 64 KiB stages when the tile is tall
        s.staging_bytes = 2 * kOperandBytes;
    }
    if (forced.staging == 1 && second != kSecondResidual) {
        s.staging_bytes = kOperandBytes;
    } else if (forced.staging == 2 || (forced.stages > 0 && forced.staging == 0)) {
        s.staging_bytes = 2 * kOperandBytes;
    }
    const bool narrowed = tile_n < kTileN;
    if (narrowed && forced.stages == 0) {
        // The ring as deep as the reduction, where a CTA has the SM to itself.
        const int depth = spread && !accumulate ? kMaxStages : 4;
        s.stages = std::max(2, std::min(depth, k_blocks));
    }
    if (slope && tile_n > kTileN) {
        s.staging_bytes = 4 * kOperandBytes;   // two blocks for each of eight warps
        s.stages = 3;
    } else if (slope) {
        s.staging_bytes = 2 * kOperandBytes;
        if (s.stages > 2 && s.ctas_per_sm > 1 && !narrowed) {
            s.stages = 2;
        }
    }
    // A switch may ask for less than the warps write: they get what they write.
    s.staging_bytes = std::max(s.staging_bytes, tc_least_staging(tile_m, tile_n, second));
    // What fits beside the staging blocks, for one or for two CTAs per SM.
    const int room = (narrowed && !spread ? kSmemLimit / 2 : kSmemLimit) -
                     s.staging_bytes - kBarrierBytes;
    s.stages = std::min(s.stages, room / s.stage_bytes);
    return s;
}

}  // namespace vitb200
