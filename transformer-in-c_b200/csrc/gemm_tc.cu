// Tensor-core matrix products for sm_100a: tcgen05.mma (kind::tf32, FP32
// accumulation in tensor memory) fed by TMA.
//
//   D[M,N] (+)= A[M,K] * B[K,N],  all FP32 in global memory, row-major.
//
// Either operand may be stored with the reduction index contiguous ("K-major":
// X in X*W, dY and W in dY*W^T) or with the output index contiguous
// ("MN-major": W in X*W, X and dY in X^T*dY), so the same kernel serves the
// forward product and both gradients of reference src/ops.c:107-165 without a
// transposed copy.  Nothing is converted or re-laid-out in global memory: TMA
// rounds FP32 to TF32 while it fills the shared-memory stages.
//
// Persistent CTAs (two per SM by default: with the short reductions of this
// model, K = 128..512, two shallow pipelines hide the tile-to-tile bubbles
// better than one deep one) walk work items = (128 x 128 output tile, slice
// of the reduction); three warp roles meet only through mbarriers:
//
//   warp 0      TMA producer: per 32-deep reduction block, one 128B-swizzled
//               box (K-major) or a box of 32x32 blocks (MN-major) per operand into
//               a shared-memory ring of 32 KB stages (2 stages by default)
//   warp 1      allocates 256 TMEM columns (two accumulators), issues four
//               K=8 tcgen05.mma per block from one lane, releases stages with
//               tcgen05.commit, and signals a finished accumulator
//   warps 2-5   epilogue, overlapped with the next item's loads and MMAs:
//               each warp tcgen05.ld's its 32 rows, adds the bias, optionally
//               derives a second output (GELU, or + residual), stages 32x32
//               blocks in its own 128B-swizzled buffers and issues its own TMA
//               stores (plain, or FP32 reduce-add for "+=" outputs and for
//               reductions split across CTAs); no block-wide barrier is used
//
// Partial tiles need no special code: TMA zero-fills out-of-range loads and
// clips out-of-range stores.  Every wait on an mbarrier is bounded in time;
// on expiry the kernel records a code in `*status` and all roles fall through
// to the common teardown, which frees the tensor memory.
#include "gemm_tc.h"
#include "gemm_tc_shared.h"
#include "kernels.h"
#include "device_util.cuh"
#include "shared_limit.h"
#include "tcgen05.cuh"

#include <cuda.h>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <unordered_map>

namespace vitb200 {
namespace {

constexpr int kMmaK = 8;                    // tf32 K per instruction
constexpr int kThreads = 192;
constexpr int kThreadsTall = 320;           // with two groups of epilogue warps
template <int TILE_M, int TILE_N, int SECOND>
constexpr bool kTwoGroups = tc_two_groups(TILE_M, TILE_N, SECOND);
template <int TILE_M, int TILE_N, int SECOND>
constexpr int kThreadsOf = kTwoGroups<TILE_M, TILE_N, SECOND> ? kThreadsTall : kThreads;

using namespace tc;

struct TcParams {
    int m, n;                 // output extents
    int k_blocks;             // ceil(reduction / 32)
    int k_blocks_per_split;
    int splits;
    int stages;               // depth of the load ring
    int staging_bytes;        // epilogue staging: 16 or 32 KiB
    int m_tiles, n_tiles;
    int a_mn_major, b_mn_major;
    int a_blocked, b_blocked; // MN-major operand: one copy per tile (see operand_map)
    int reduce_add;           // 1: TMA reduce-add into D, 0: plain store
    const float *bias;        // nullable, length n
    const float *residual;    // [m, n] with residual_pitch, for kSecondResidual
    long long residual_pitch;
    float *column_partials;   // kGeluSlope: [gridDim.x][n] column sums of D, or null
    int *status;              // device-visible word, 0 = ok
};

template <int SECOND>
constexpr bool kIsSlope = SECOND == kGeluSlope || SECOND == kGeluSlopeEight;

// Persistent kernel: each CTA walks work items (output tile x reduction
// slice) item = cta, cta + ctas, ...; the three roles run
// the same sequence and meet only through mbarriers, so the loads and MMAs of
// item i+1 overlap the epilogue of item i (two accumulator buffers in TMEM).
//
// TILE_N = 128: two CTAs per SM share the 512 TMEM columns (2 x 128 each).
// TILE_N = 256: one CTA per SM with all 512 columns; an MMA instruction then
// covers twice the columns for the same A bytes, which is what the
// compute-bound shapes (K >= 256) need from shared memory.  The launch code
// guarantees one CTA per SM for it through the shared-memory request, so the
// two allocations can never wait for each other.
// TILE_M = 256 (with TILE_N = 256): the tile is two 128-row halves, one
// accumulator each (all 512 columns), both multiplied by the same B tile, so
// a CTA fetches (256 + 256) x K operand values for 256 x 256 outputs: a third
// less operand traffic from L2 per multiply-add than the 128 x 256 tile, which
// is what bounds the compute-bound shapes.  The accumulators are not
// double-buffered across tiles then; instead the halves are: the epilogue
// drains half 0 while the last MMAs of half 1 run, and the next tile's MMAs
// start on half 0 while half 1 is still being drained.
// SECOND is the epilogue variant (0 or a kSecond... / kGeluSlope constant): a
// compile-time choice, so that no variant pays for another's registers.
// `cta` of `ctas`: this CTA's place among those that walk the product's items.
template <int TILE_M, int TILE_N, int SECOND>
__device__ __forceinline__ void
walk_product(const CUtensorMap &map_a, const CUtensorMap &map_b, const CUtensorMap &map_d,
             const CUtensorMap &map_d2, const TcParams &p, const int cta, const int ctas) {
    // All shared memory is dynamic, so that it starts at the beginning of the
    // CTA's window and the swizzled tiles get their 1024-byte alignment without
    // padding (two CTAs with three stages each fill the SM to the last KiB):
    //   [stages x 32 KiB operand tiles][epilogue staging][barriers]
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int kHalves = TILE_M / kTileM;   // accumulators per tile
    constexpr int kABytes = TILE_M * kBlockK * 4;
    constexpr int kStageBytes = kABytes + TILE_N * kBlockK * 4;
    constexpr int kTmemColumns = 2 * TILE_N;
    static_assert(TILE_M == kTileM ||
                      (TILE_M == 2 * kTileM && (SECOND == 0 || SECOND == kSecondGelu)),
                  "the tall tile has the plain and the GELU epilogues only");
    const int kStages = p.stages;
    uint8_t *staging = smem + kStages * kStageBytes;
    uint64_t *full_bar = reinterpret_cast<uint64_t *>(staging + p.staging_bytes);
    uint64_t *empty_bar = full_bar + kMaxStages;
    uint64_t *tmem_full_bar = empty_bar + kMaxStages;
    uint64_t *tmem_empty_bar = tmem_full_bar + 2;
    uint32_t &tmem_base_slot = *reinterpret_cast<uint32_t *>(tmem_empty_bar + 2);
    uint64_t *operand_bar = tmem_empty_bar + 3;   // up to two per epilogue warp
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if ((smem_address(smem) & 1023u) != 0) {
        // Never expected; without the alignment the MMA would read garbage.
        grid_dependency_wait();
        if (threadIdx.x == 0) {
            atomicExch(p.status, 6);
        }
        return;
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbarrier_init(&full_bar[s], 1);
            mbarrier_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbarrier_init(&tmem_full_bar[b], 1);
            // One arrival per epilogue warp that reads the accumulator.
            mbarrier_init(&tmem_empty_bar[b],
                          kHalves == 1 && kTwoGroups<TILE_M, TILE_N, SECOND> ? 8 : 4);
        }
        for (int w = 0; w < 16; ++w) {
            mbarrier_init(&operand_bar[w], 1);
        }
        prefetch_tensor_map(&map_a);
        prefetch_tensor_map(&map_b);
        prefetch_tensor_map(&map_d);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile(
            "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::
                "r"(smem_address(&tmem_base_slot)),
            "r"(kTmemColumns)
            : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::
                         : "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    // Barriers and tensor memory are set up; from here on global memory is
    // touched, so the kernel before this one in the stream has to be complete.
    grid_dependency_wait();
    grid_dependency_release();
    if (kIsSlope<SECOND> && p.column_partials) {
        // This CTA's own row of column sums, which its epilogue warps add into.
        for (int c = threadIdx.x; c < p.n; c += blockDim.x) {
            p.column_partials[size_t(cta) * p.n + c] = 0.0f;
        }
        __threadfence();
        __syncthreads();
    }
    const int tiles = p.m_tiles * p.n_tiles;
    const int items = tiles * p.splits;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            // (The next copy waits for what this thread does per block: no divisions,
            // and one branch to the copy of an operand that is stored K-major.)
            int s = 0;             // stage of the ring, across items
            uint32_t phase = 1;    // parity of its last release
            for (int item = cta; item < items && ok; item += ctas) {
                const int tile = item % tiles;
                const int m0 = (tile / p.n_tiles) * TILE_M;
                const int n0 = (tile % p.n_tiles) * TILE_N;
                const int kb_begin = (item / tiles) * p.k_blocks_per_split;
                const int kb_end = min(p.k_blocks, kb_begin + p.k_blocks_per_split);
                for (int kb = kb_begin; kb < kb_end; ++kb) {
                    ok = mbarrier_wait(&empty_bar[s], phase);
                    if (!ok) {
                        atomicExch(p.status, 1);
                        break;
                    }
                    uint8_t *a_tile = smem + s * kStageBytes;
                    uint8_t *b_tile = a_tile + kABytes;
                    const int k0 = kb * kBlockK;
                    mbarrier_expect_tx(&full_bar[s], kStageBytes);
                    if (!p.a_mn_major) {
                        // One box of TILE_M rows (the map's box height).
                        tma_load_2d(a_tile, &map_a, k0, m0, &full_bar[s]);
                    } else if (p.a_blocked) {
                        tma_load_3d(a_tile, &map_a, 0, k0, m0 / 32, &full_bar[s]);
                    } else {
                        for (int j = 0; j < TILE_M / 32; ++j) {
                            tma_load_2d(a_tile + j * 4096, &map_a, m0 + 32 * j, k0,
                                        &full_bar[s]);
                        }
                    }
                    if (!p.b_mn_major) {
                        tma_load_2d(b_tile, &map_b, k0, n0, &full_bar[s]);
                    } else if (p.b_blocked) {
                        tma_load_3d(b_tile, &map_b, 0, k0, n0 / 32, &full_bar[s]);
                    } else {
                        for (int j = 0; j < TILE_N / 32; ++j) {
                            tma_load_2d(b_tile + j * 4096, &map_b, n0 + 32 * j, k0,
                                        &full_bar[s]);
                        }
                    }
                    if (++s == kStages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // kind::tf32, FP32 accumulator, M = 128, N = 128.
            // (The N field is filled in per tile: a last column tile that is
            // only partly inside the matrix gets a narrower instruction.)
            const uint32_t idesc_base = (1u << 4) | (2u << 7) | (2u << 10) |
                                        (uint32_t(p.a_mn_major) << 15) |
                                        (uint32_t(p.b_mn_major) << 16) |
                                        (uint32_t(kTileM >> 4) << 24);
            // K-major: 8-row groups 1024 B apart, K steps of 32 B inside the
            // swizzled row.  MN-major: 32-wide MN atoms one box (4096 B)
            // apart, groups of four 128 B reduction rows 512 B apart, K
            // steps of eight rows.
            const uint32_t a_lead = p.a_mn_major ? 4096 : 16;
            const uint32_t b_lead = p.b_mn_major ? 4096 : 16;
            const uint32_t a_stride = p.a_mn_major ? 512 : 1024;
            const uint32_t b_stride = p.b_mn_major ? 512 : 1024;
            const uint32_t a_step = p.a_mn_major ? 1024 : kMmaK * 4;
            const uint32_t b_step = p.b_mn_major ? 1024 : kMmaK * 4;
            const uint32_t a_layout =
                p.a_mn_major ? kLayoutSwizzle128Base32 : kLayoutSwizzle128;
            const uint32_t b_layout =
                p.b_mn_major ? kLayoutSwizzle128Base32 : kLayoutSwizzle128;
            int s = 0;             // stage of the ring, across items
            uint32_t phase = 0;    // parity of its next arrival
            int local = 0;   // items processed by this CTA
            for (int item = cta; item < items && ok;
                 item += ctas, ++local) {
                const int tile_splits = item / tiles;
                const int n_live = min(TILE_N, p.n - ((item % tiles) % p.n_tiles) * TILE_N);
                const uint32_t idesc =
                    idesc_base | (uint32_t(((n_live + 15) & ~15) >> 3) << 17);
                const int kb_begin = tile_splits * p.k_blocks_per_split;
                const int kb_end = min(p.k_blocks, kb_begin + p.k_blocks_per_split);
                // One accumulator per tile, alternating between tiles; or, for
                // the tall tile, one per 128-row half, both used by every tile.
                const uint32_t buffer_phase =
                    kHalves == 2 ? (local & 1) : ((local >> 1) & 1);
                for (int kb = kb_begin; kb < kb_end; ++kb) {
                    ok = mbarrier_wait(&full_bar[s], phase);
                    if (!ok) {
                        atomicExch(p.status, 2);
                        break;
                    }
                    tcgen05_fence_after();
                    const uint32_t a_base = smem_address(smem + s * kStageBytes);
                    const uint32_t b_base = a_base + kABytes;
#pragma unroll
                    for (int h = 0; h < kHalves; ++h) {
                        const int buffer = kHalves == 2 ? h : (local & 1);
                        if (kb == kb_begin) {
                            // The epilogue must have emptied this accumulator.
                            ok = mbarrier_wait(&tmem_empty_bar[buffer],
                                               buffer_phase ^ 1);
                            if (!ok) {
                                atomicExch(p.status, 4);
                                break;
                            }
                            tcgen05_fence_after();
                        }
                        const uint32_t accumulator = tmem_base + buffer * TILE_N;
#pragma unroll
                        for (int ks = 0; ks < kBlockK / kMmaK; ++ks) {
                            const uint64_t da = operand_descriptor(
                                a_base + h * kOperandBytes + ks * a_step, a_lead,
                                a_stride, a_layout);
                            const uint64_t db = operand_descriptor(
                                b_base + ks * b_step, b_lead, b_stride, b_layout);
                            tcgen05_mma_tf32(accumulator, da, db, idesc,
                                             (kb > kb_begin || ks > 0) ? 1u : 0u);
                        }
                        if (kb == kb_end - 1) {
                            // This half is complete: its rows can leave while
                            // the other half's last products still run.
                            tcgen05_commit(&tmem_full_bar[buffer]);
                        }
                    }
                    if (!ok) {
                        break;
                    }
                    tcgen05_commit(&empty_bar[s]);
                    if (++s == kStages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if constexpr (kIsSlope<SECOND>) {
        // Epilogue of D = (A*B) * gelu'(H).  Each warp walks its 32 x 32 blocks in order
        // (tile after tile, its column chunks of each).  The H values of a block are
        // fetched by the copy engine into the staging block that the result then leaves
        // from: with two staging blocks the ones of block j+1 while block j is
        // multiplied, with one as soon as the result of block j has been read.
        constexpr int kGroups = kTwoGroups<TILE_M, TILE_N, SECOND> ? 2 : 1;
        constexpr int kBlocks = SECOND == kGeluSlopeEight ? 1 : 2;
        constexpr int kChunks = TILE_N / 32 / kGroups;   // of a warp and tile
        const int quarter = warp & 3;
        const int first_chunk = kGroups == 2 ? (warp - 2) / 4 * kChunks : 0;
        uint8_t *my_staging = staging + (warp - 2) * kBlocks * 4096;
        uint64_t *my_bar = operand_bar + (warp - 2) * kBlocks;
        uint32_t phases = 0;   // bit b: parity of the next completion of my_bar[b]
        int issued = 0;        // H blocks requested so far
        int consumed = 0;      // H blocks used so far
        // Requests the H block of (item, chunk) when that block exists.
        auto request = [&](int item, int chunk) {
            const int tile = item % tiles;
            const int m0 = (tile / p.n_tiles) * kTileM + quarter * 32;
            const int col0 = (tile % p.n_tiles) * TILE_N + chunk * 32;
            if (col0 >= p.n || m0 >= p.m) {
                return;
            }
            if (lane == 0) {
                // The block was last read by the store issued for the block
                // before the current one (kBlocks == 1: for the current one).
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                const int b = issued % kBlocks;
                mbarrier_expect_tx(&my_bar[b], 4096);
                tma_load_2d(my_staging + b * 4096, &map_d2, col0, m0, &my_bar[b]);
            }
            ++issued;
        };
        // The block after (item, chunk), possibly the next tile's first.
        auto request_after = [&](int item, int chunk) {
            if (chunk + 1 < first_chunk + kChunks) {
                request(item, chunk + 1);
            } else if (item + ctas < items) {
                request(item + ctas, first_chunk);
            }
        };
        if (cta < items) {
            request(cta, first_chunk);
        }
        int local = 0;
        for (int item = cta; item < items && ok; item += ctas, ++local) {
            const int tile = item % tiles;
            const int m0 = (tile / p.n_tiles) * kTileM + quarter * 32;
            const int n0 = (tile % p.n_tiles) * TILE_N;
            const int buffer = local & 1;
            const uint32_t buffer_phase = (local >> 1) & 1;
            ok = mbarrier_wait(&tmem_full_bar[buffer], buffer_phase);
            ok = __all_sync(0xffffffffu, ok);   // keep the warp in step
            if (!ok) {
                atomicExch(p.status, 3);
                break;
            }
            tcgen05_fence_after();
#pragma unroll 1
            for (int chunk = first_chunk; chunk < first_chunk + kChunks; ++chunk) {
                const int col0 = n0 + chunk * 32;
                const bool chunk_live = col0 < p.n && m0 < p.m;
                uint32_t r[32];
                if (chunk_live) {
                    tcgen05_load_32(tmem_base + (uint32_t(quarter * 32) << 16) +
                                        buffer * TILE_N + chunk * 32,
                                    r);
                }
                if (chunk == first_chunk + kChunks - 1) {
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbarrier_arrive(&tmem_empty_bar[buffer]);
                    }
                }
                if (kBlocks == 2 || !chunk_live) {
                    request_after(item, chunk);
                }
                if (!chunk_live) {
                    continue;   // uniform across the warp
                }
                const int b = consumed % kBlocks;
                ++consumed;
                ok = mbarrier_wait(&my_bar[b], (phases >> b) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    atomicExch(p.status, 7);
                    break;
                }
                phases ^= 1u << b;
                float *block = reinterpret_cast<float *>(my_staging + b * 4096);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    // 128-byte swizzle: 16-byte chunk c of row r lives at
                    // chunk position c ^ (r % 8).
                    const int offset = lane * 32 + 4 * (c ^ (lane & 7));
                    float4 h = *reinterpret_cast<const float4 *>(block + offset);
                    h.x = __uint_as_float(r[4 * c + 0]) * gelu_slope_fast(h.x);
                    h.y = __uint_as_float(r[4 * c + 1]) * gelu_slope_fast(h.y);
                    h.z = __uint_as_float(r[4 * c + 2]) * gelu_slope_fast(h.z);
                    h.w = __uint_as_float(r[4 * c + 3]) * gelu_slope_fast(h.w);
                    *reinterpret_cast<float4 *>(block + offset) = h;
                }
                if (p.column_partials) {
                    // Column sums of the block (rows past the matrix are
                    // zero: their accumulators are), lane = column.
                    __syncwarp();
                    float sum = 0.0f;
#pragma unroll
                    for (int row = 0; row < 32; ++row) {
                        sum += block[row * 32 + 4 * ((lane >> 2) ^ (row & 7)) +
                                     (lane & 3)];
                    }
                    if (col0 + lane < p.n) {
                        atomicAdd(p.column_partials + size_t(cta) * p.n +
                                      col0 + lane,
                                  sum);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(block, &map_d, col0, m0);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                if (kBlocks == 1) {
                    request_after(item, chunk);
                }
            }
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else {
        // Epilogue warps 2..5 own TMEM lane quarters 2, 3, 0, 1, i.e. 32 rows
        // of the tile each.  A warp stages its own 32 x 32 blocks (4 KiB, two
        // buffers per output) and issues its own TMA stores, so the epilogue
        // needs no block-wide barrier at all.
        const int quarter = warp & 3;
        const int outputs = SECOND ? 2 : 1;
        // Per warp: two 4 KiB blocks (one output double-buffered, or one buffer
        // for each of two outputs), or a single block when the load ring was
        // given the space instead.
        // The tall tile: warps 2-5 drain the upper half's accumulator, warps
        // 6-9 the lower half's, each warp through one 4 KiB block.
        // Two groups on one accumulator take half of its columns each.
        constexpr bool kEight = kTwoGroups<TILE_M, TILE_N, SECOND>;
        constexpr int kChunks = TILE_N / 32 / (kEight && kHalves == 1 ? 2 : 1);
        const int half = kHalves == 2 ? (warp - 2) >> 2 : 0;
        const int first_chunk = kEight && kHalves == 1 ? (warp - 2) / 4 * kChunks : 0;
        const int buffers =
            kEight ? 1 : (outputs == 2 ? 1 : p.staging_bytes / (4 * 4096));
        uint8_t *my_staging = kEight
            ? staging + (warp - 2) * 4096
            : staging + quarter * (p.staging_bytes / 4);
        int local = 0;
        int stored = 0;   // blocks handed to TMA so far (selects the buffer)
        for (int item = cta; item < items; item += ctas, ++local) {
            const int tile = item % tiles;
            const int m0 = (tile / p.n_tiles) * TILE_M + half * kTileM + quarter * 32;
            const int n0 = (tile % p.n_tiles) * TILE_N;
            const int buffer = kHalves == 2 ? half : (local & 1);
            const uint32_t buffer_phase =
                kHalves == 2 ? (local & 1) : ((local >> 1) & 1);
            ok = mbarrier_wait(&tmem_full_bar[buffer], buffer_phase);
            ok = __all_sync(0xffffffffu, ok);   // keep the warp in step
            if (!ok) {
                atomicExch(p.status, 3);
                break;
            }
            tcgen05_fence_after();
#pragma unroll 1
            for (int chunk = first_chunk; chunk < first_chunk + kChunks; ++chunk) {
                const int col0 = n0 + chunk * 32;
                const bool chunk_live = col0 < p.n && m0 < p.m;
                // Bias for these 32 columns, requested before the accumulator
                // so the two latencies overlap.
                float4 bias[8];
                if (p.bias && chunk_live) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const int col = col0 + 4 * c;
                        if (col + 3 < p.n) {
                            bias[c] = __ldg(
                                reinterpret_cast<const float4 *>(p.bias + col));
                        } else {
                            bias[c].x = col + 0 < p.n ? __ldg(p.bias + col + 0) : 0.f;
                            bias[c].y = col + 1 < p.n ? __ldg(p.bias + col + 1) : 0.f;
                            bias[c].z = col + 2 < p.n ? __ldg(p.bias + col + 2) : 0.f;
                            bias[c].w = 0.f;
                        }
                    }
                }
                uint32_t r[32];
                if (chunk_live) {
                    tcgen05_load_32(tmem_base + (uint32_t(quarter * 32) << 16) +
                                        buffer * TILE_N + chunk * 32,
                                    r);
                }
                if (chunk == first_chunk + kChunks - 1) {
                    // Everything this warp needs is in registers: hand the
                    // accumulator buffer back to the MMA warp.
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbarrier_arrive(&tmem_empty_bar[buffer]);
                    }
                }
                if (!chunk_live) {
                    continue;   // uniform across the warp
                }
                if (p.bias) {
                    // Folded into the accumulator registers once, so the bias
                    // registers are free again before the stores.
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        r[4 * c + 0] = __float_as_uint(__uint_as_float(r[4 * c + 0]) + bias[c].x);
                        r[4 * c + 1] = __float_as_uint(__uint_as_float(r[4 * c + 1]) + bias[c].y);
                        r[4 * c + 2] = __float_as_uint(__uint_as_float(r[4 * c + 2]) + bias[c].z);
                        r[4 * c + 3] = __float_as_uint(__uint_as_float(r[4 * c + 3]) + bias[c].w);
                    }
                }
                // The buffer about to be rewritten was last read by the store
                // this warp issued two blocks ago.
                if (lane == 0) {
                    if (buffers == 2) {
                        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    } else {
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    }
                }
                __syncwarp();
                const int slot = buffers == 2 ? (stored & 1) : 0;
                ++stored;
                float *first = reinterpret_cast<float *>(my_staging + slot * 4096);
                // With 16 KiB of staging both outputs of a warp go through the
                // same 4 KiB block, one after the other.
                const bool shared_block =
                    outputs == 2 && (kEight || p.staging_bytes == kOperandBytes);
                float *second = shared_block
                    ? first : reinterpret_cast<float *>(my_staging + 4096);
                {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float4 v;
                    v.x = __uint_as_float(r[4 * c + 0]);
                    v.y = __uint_as_float(r[4 * c + 1]);
                    v.z = __uint_as_float(r[4 * c + 2]);
                    v.w = __uint_as_float(r[4 * c + 3]);
                    // 128-byte swizzle: 16-byte chunk c of row r lives at
                    // chunk position c ^ (r % 8).
                    const int offset = lane * 32 + 4 * (c ^ (lane & 7));
                    *reinterpret_cast<float4 *>(first + offset) = v;
                    if (SECOND == kSecondGelu && !shared_block) {
                        v.x = gelu_value_fast(v.x);
                        v.y = gelu_value_fast(v.y);
                        v.z = gelu_value_fast(v.z);
                        v.w = gelu_value_fast(v.w);
                        *reinterpret_cast<float4 *>(second + offset) = v;
                    }
                }
                }
                if (SECOND == kSecondResidual) {
                    // D2 = D + residual.  In the accumulator layout a lane
                    // owns a row, which would read the residual one row per
                    // lane; instead the staged block is walked with eight
                    // lanes per row, so every load covers four full 128-byte
                    // row segments.
                    __syncwarp();
                    const int c = lane & 7;
                    const int col = col0 + 4 * c;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = (lane >> 3) + 4 * i;
                        const int offset = row * 32 + 4 * (c ^ (row & 7));
                        float4 v = *reinterpret_cast<const float4 *>(first + offset);
                        if (m0 + row < p.m) {
                            const float *res = p.residual +
                                size_t(m0 + row) * p.residual_pitch + col;
                            if (col + 3 < p.n) {
                                const float4 x =
                                    __ldcs(reinterpret_cast<const float4 *>(res));
                                v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
                            } else {
                                if (col + 0 < p.n) v.x += res[0];
                                if (col + 1 < p.n) v.y += res[1];
                                if (col + 2 < p.n) v.z += res[2];
                            }
                        }
                        *reinterpret_cast<float4 *>(second + offset) = v;
                    }
                }
                // Make the generic-proxy writes visible to the TMA engine.
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (shared_block && SECOND == kSecondGelu) {
                    // First output out; the second output's values are
                    // computed while the copy engine reads the block, and go
                    // through the same block once it has.
                    if (lane == 0) {
                        tma_store_2d(first, &map_d, col0, m0);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        r[e] = __float_as_uint(gelu_value_fast(__uint_as_float(r[e])));
                    }
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    }
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        float4 v;
                        v.x = __uint_as_float(r[4 * c + 0]);
                        v.y = __uint_as_float(r[4 * c + 1]);
                        v.z = __uint_as_float(r[4 * c + 2]);
                        v.w = __uint_as_float(r[4 * c + 3]);
                        const int offset = lane * 32 + 4 * (c ^ (lane & 7));
                        *reinterpret_cast<float4 *>(second + offset) = v;
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(second, &map_d2, col0, m0);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                } else if (lane == 0) {
                    if (p.reduce_add) {
                        tma_reduce_add_2d(first, &map_d, col0, m0);
                    } else {
                        tma_store_2d(first, &map_d, col0, m0);
                    }
                    if (outputs == 2) {
                        tma_store_2d(second, &map_d2, col0, m0);
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(
                         tmem_base),
                     "r"(kTmemColumns)
                     : "memory");
    }
}

template <int TILE_M, int TILE_N, int SECOND>
__global__ void __launch_bounds__(kThreadsOf<TILE_M, TILE_N, SECOND>)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a,
               const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_d,
               const __grid_constant__ CUtensorMap map_d2, const TcParams p) {
    walk_product<TILE_M, TILE_N, SECOND>(map_a, map_b, map_d, map_d2, p, blockIdx.x,
                                         gridDim.x);
}

// Two independent products side by side: the gradients of one linear layer when
// both are so small that a launch of their own costs more than their work.  The
// first `ctas` CTAs walk the input gradient (with the GELU slope or without), the
// others the weight gradient.
struct TcPairMaps {
    CUtensorMap a, b, d, d2;
};

template <int TILE_N, int SECOND>
__global__ void __launch_bounds__(kThreads)
gemm_tc_pair_kernel(const __grid_constant__ TcPairMaps input,
                    const __grid_constant__ TcPairMaps weight, const TcParams p,
                    const TcParams q, const int ctas) {
    if (int(blockIdx.x) < ctas) {
        walk_product<kTileM, TILE_N, SECOND>(input.a, input.b, input.d, input.d2, p,
                                             blockIdx.x, ctas);
    } else {
        walk_product<kTileM, TILE_N, 0>(weight.a, weight.b, weight.d, weight.d, q,
                                        blockIdx.x - ctas, gridDim.x - ctas);
    }
}

// ---- host side -------------------------------------------------------------

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t,
                                 void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *,
                                 CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static EncodeTiled function = []() -> EncodeTiled {
        void *entry = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry,
                                    cudaEnableDefault, &result) != cudaSuccess ||
            result != cudaDriverEntryPointSuccess) {
            return nullptr;
        }
        return reinterpret_cast<EncodeTiled>(entry);
    }();
    return function;
}

struct MapKey {
    const void *base;
    unsigned long long inner, outer, pitch;
    unsigned box_inner, box_outer, blocks;
    int swizzle;
    bool operator==(const MapKey &o) const {
        return base == o.base && inner == o.inner && outer == o.outer &&
               pitch == o.pitch && box_inner == o.box_inner &&
               box_outer == o.box_outer && blocks == o.blocks &&
               swizzle == o.swizzle;
    }
};

struct MapKeyHash {
    size_t operator()(const MapKey &k) const {
        size_t h = reinterpret_cast<size_t>(k.base);
        h = h * 1000003u ^ k.inner;
        h = h * 1000003u ^ k.outer;
        h = h * 1000003u ^ k.pitch;
        h = h * 1000003u ^ (size_t(k.box_inner) << 16 | k.box_outer);
        h = h * 1000003u ^ (size_t(k.swizzle) << 16 | k.blocks);
        return h;
    }
};

// 2-D FP32 tensor map over a row-major matrix: `inner` contiguous elements per
// row, `outer` rows `pitch` elements apart, with the given 128-byte swizzle
// flavour.  Operand maps use the TFLOAT32 element type, which makes the copy
// engine round the FP32 words to TF32 (nearest) on their way into shared
// memory instead of leaving the truncation to the MMA; the output map is plain
// FP32.  blocks > 0: the row is cut into blocks of box_inner elements (it must be a
// multiple of them) and a copy takes that many blocks of box_outer rows each, one
// after the other, from coordinates (0, row, block) on.  Encoded maps are cached: the
// training step presents the same buffers every iteration.
bool tensor_map(const float *base, unsigned long long inner,
                unsigned long long outer, unsigned long long pitch,
                unsigned box_inner, unsigned box_outer,
                CUtensorMapSwizzle swizzle, bool as_tf32, CUtensorMap *out,
                unsigned blocks = 0) {
    static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
    const MapKey key{base, inner, outer, pitch, box_inner, box_outer, blocks,
                     int(swizzle) * 2 + int(as_tf32)};
    auto found = cache.find(key);
    if (found != cache.end()) {
        *out = found->second;
        return true;
    }
    EncodeTiled encode = encode_tiled();
    if (!encode) {
        return false;
    }
    const cuuint64_t dims[3] = {blocks ? box_inner : inner, outer, inner / box_inner};
    const cuuint64_t strides[2] = {pitch * sizeof(float), box_inner * sizeof(float)};
    const cuuint32_t box[3] = {box_inner, box_outer, blocks};
    const cuuint32_t element_strides[3] = {1, 1, 1};
    const CUresult status = encode(
        out, as_tf32 ? CU_TENSOR_MAP_DATA_TYPE_TFLOAT32
                     : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
        blocks ? 3 : 2, const_cast<float *>(base), dims,
        strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
        swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (status != CUDA_SUCCESS) {
        return false;
    }
    if (cache.size() > 4096) {
        cache.clear();
    }
    cache.emplace(key, *out);
    return true;
}

// MN-major operand: rows = reduction index, inner = output index, in 32 x 32 blocks.  A
// tile is `blocks` of them in one copy where rows are whole blocks; otherwise a copy
// each, whose columns past the row read as zero.  (One thread issues all copies, and
// nine to sixteen for a block of the reduction keep it longer than the products keep
// the tensor core: [65600,384]x[384,1152] 129 -> 109 us, weight gradient [1536,384]
// over 65600 rows 151 -> 128, bias + GELU onto 2048 columns 129 -> 126.)
bool operand_map(const float *base, unsigned long long inner, unsigned long long outer,
                 unsigned long long pitch, unsigned blocks, CUtensorMap *out) {
    return tensor_map(base, inner, outer, pitch, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B,
                      true, out, blocks);
}

int *status_word() {
    static int *word = []() -> int * {
        // (The first product may be one that is being captured, in whose mode an
        // allocation would end the capture.)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        int *memory = nullptr;
        const cudaError_t status = cudaHostAlloc(reinterpret_cast<void **>(&memory),
                                                 sizeof(int), cudaHostAllocMapped);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (status != cudaSuccess) {
            return nullptr;
        }
        *memory = 0;
        return memory;
    }();
    return word;
}

using TcKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap,
                          const CUtensorMap, const TcParams);

// A tile with the kernels built for it, by epilogue.  Boxes of the tensor maps, bytes of
// a stage, ring depth and grid all follow m and n, and a kernel that is handed another
// tile's would write out of range: so kernels are named here, beside their extents,
// and nowhere else.
struct TcTile {
    int m, n;
    // (Null: not built.)
    TcKernel plain, second_gelu, second_residual, gelu_slope, gelu_slope_eight;
    int threads[5];

    TcKernel kernel(int second) const {
        return second == kSecondGelu       ? second_gelu
               : second == kSecondResidual ? second_residual
               : second == kGeluSlope      ? gelu_slope
               : second == kGeluSlopeEight ? gelu_slope_eight
                                           : plain;
    }
};

template <int M, int N>
constexpr TcTile make_tile() {
    TcTile tile = {M, N, gemm_tc_kernel<M, N, 0>, gemm_tc_kernel<M, N, kSecondGelu>,
                   nullptr, nullptr, nullptr,
                   {kThreadsOf<M, N, 0>, kThreadsOf<M, N, kSecondGelu>,
                    kThreadsOf<M, N, kSecondResidual>, kThreadsOf<M, N, kGeluSlope>,
                    kThreadsOf<M, N, kGeluSlopeEight>}};
    if constexpr (M == kTileM) {
        tile.gelu_slope = gemm_tc_kernel<M, N, kGeluSlope>;
    }
    if constexpr (M == kTileM && N == kTileN) {
        tile.second_residual = gemm_tc_kernel<M, N, kSecondResidual>;
        tile.gelu_slope_eight = gemm_tc_kernel<M, N, kGeluSlopeEight>;
    }
    return tile;
}

enum { kNarrow32, kNarrow64, kSquare, kWide, kTall, kTcTileCount };
const TcTile kTcTiles[kTcTileCount] = {
    make_tile<kTileM, 32>(), make_tile<kTileM, 64>(), make_tile<kTileM, kTileN>(),
    make_tile<kTileM, 256>(), make_tile<2 * kTileM, 256>()};

// Lets every kernel use the whole of an SM's shared memory.
bool raise_limits() {
    static SharedMemoryLimit limit;
    const void *kernels[5 * kTcTileCount];
    int count = 0;
    for (const TcTile &tile : kTcTiles) {
        for (TcKernel kernel : {tile.plain, tile.second_gelu, tile.second_residual,
                                tile.gelu_slope, tile.gelu_slope_eight}) {
            if (kernel) {
                kernels[count++] = reinterpret_cast<const void *>(kernel);
            }
        }
    }
    return limit.raise(kernels, count, kSmemLimit);
}

}  // namespace

bool gemm_tc_supported(const TcGemm &g) {
    // TMA needs 16-byte aligned bases and row pitches.  An extent may be
    // smaller than the 32-wide box (the 16-pixel patches of the 28 x 28
    // models): out-of-range elements load as zero and stores are clipped.
    // Tiny extents are left to the FP32 kernel.
    auto aligned = [](const void *p) {
        return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
    };
    return g.m >= 16 && g.n >= 16 && g.k >= 16 && g.lda % 4 == 0 &&
           g.ldb % 4 == 0 && g.ldd % 4 == 0 && aligned(g.a) && aligned(g.b) &&
           aligned(g.d) && (!g.bias || aligned(g.bias)) &&
           (!g.d2 || (aligned(g.d2) && g.ldd2 % 4 == 0 && !g.accumulate)) &&
           (!g.residual || (aligned(g.residual) && g.ld_residual % 4 == 0)) &&
           (!g.gelu_input ||
            (aligned(g.gelu_input) && g.ld_gelu_input % 4 == 0 && !g.accumulate &&
             !g.bias && !g.d2)) &&
           (!g.column_partials || g.gelu_input) &&
           status_word() &&
           encode_tiled();
}

namespace {

// Long reductions onto few output tiles (weight gradients) are cut into slices.
// With a persistent grid the slices should fill the CTA slots evenly: picks the slice
// count that minimises the k-blocks the busiest CTA walks (*walked), charging each item
// about eight k-blocks for its epilogue and reduce-add.
int choose_slices(long long tiles, int k_blocks, long long slots, long long *walked) {
    long long best_cost = -1;
    int slices = 1;
    for (int candidate = 1; candidate <= 512; ++candidate) {
        const int per_slice = (k_blocks + candidate - 1) / candidate;
        if (candidate > 1 && per_slice < 4) {
            break;
        }
        const long long rounds = (tiles * candidate + slots - 1) / slots;
        if (best_cost >= 0 && rounds * (4 + 8) >= best_cost) {
            break;   // more slices take no fewer rounds
        }
        const long long cost = rounds * (per_slice + 8);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            slices = candidate;
        }
    }
    if (walked) {
        *walked = best_cost;
    }
    return slices;
}

// A product ready to be launched.
struct TcLaunch {
    const TcTile *tile;
    int second;
    TcPairMaps maps;
    TcParams p;
    unsigned grid;
    int smem_bytes;
};

// Fills in `out`; false when the product cannot be served.  forced_narrow: one of the
// narrow tiles instead of the choice below, with at most `most_ctas` CTAs (the other
// product of a pair has the rest of the SMs).
bool prepare(const TcGemm &g, int forced_narrow, long long most_ctas, TcLaunch *out) {
    if (!gemm_tc_supported(g) || !raise_limits()) {
        return false;
    }
    // Wide tiles where the product is compute-bound: deep reductions, one
    // output (or the GELU pair), a multiple of 128 columns.
    static const int forced_tile =
        getenv("VITB200_TC_TILE_N") ? atoi(getenv("VITB200_TC_TILE_N")) : 0;
    const bool gelu_pair = g.d2 && !g.residual;
    // (A last tile that is half outside the matrix costs half: its products
    // are issued 128 columns wide.)
    // That pays from 4.5 tiles on, or with a deep reduction (measured at
    // [65600,384]x[384,1152]: +14 %, [65600,1536]x[1536,384]: +6 %,
    // [65600,384]x[384,384]: -3 to -9 %).
    const bool divides = g.n % 256 == 0 ||
                         (g.n % 128 == 0 && g.n >= 256 &&
                          (g.n >= 1024 || (!g.accumulate && g.k >= 1024)));
    bool wide = (!g.d2 || gelu_pair) && g.k >= 256 && divides;
    if (g.gelu_input) {
        // (See the slope's variants below.  Short of 768 terms, not with the SMs' last
        // round of tiles so empty that three quarters of all are not filled:
        // [12800,512] onto 512 columns, 200 tiles for 148 SMs, 1.14 of the square tile.)
        const long long sms = device_sm_count();
        const long long tiles = ((g.m + kTileM - 1LL) / kTileM) * ((g.n + 255) / 256);
        wide = wide && (g.k >= 768 || (g.k >= 512 && 4 * tiles >=
                                                         3 * sms * ((tiles + sms - 1) / sms)));
    }
    if (forced_tile == 128 || (g.d2 && !gelu_pair)) {
        wide = false;
    } else if (forced_tile == 256 && !g.d2 && !g.gelu_input) {
        wide = g.n >= 256;
    }
    // Tall tiles (256 x 256, two accumulator halves) on top of that when there
    // are at least two full row tiles: a third less operand traffic from L2.
    static const int forced_tile_m =
        getenv("VITB200_TC_TILE_M") ? atoi(getenv("VITB200_TC_TILE_M")) : 0;
    // (Not for the shortest reductions, where the double-buffered 128 x 256
    // tile hides its epilogue completely and measured a few percent better.)
    const bool long_enough = g.accumulate || g.k >= 384;
    // A last row tile that is half empty costs a full one: only where that
    // is a small share of the rows.
    const bool fits = g.m % (2 * kTileM) == 0 || g.m % (2 * kTileM) > kTileM ||
                      g.m >= 16 * kTileM;
    bool tall = wide && !g.gelu_input && g.m >= 2 * kTileM && forced_tile_m != 128 &&
                ((long_enough && fits) || forced_tile_m == 256);
    // The GELU pair's epilogue (two stores and a GELU per element) takes
    // longer than the tile's products: the tall tile, whose accumulators are
    // not double-buffered across tiles, leaves it exposed; the 128 x 256 tile
    // hides the next tile's products behind it (measured 3 to 10 % faster at
    // [100864,512]x[512,2048] and [65600,384]x[384,1536]).  Eight epilogue warps on it
    // instead of four: 202 -> 196 us at the latter, 126 -> 124 at [25216,512]x[512,2048].
    static const bool gelu_pair_tall = getenv("VITB200_TC_GELU_TALL") != nullptr;
    if (gelu_pair && tall && !gelu_pair_tall) {
        tall = false;
    }
    if (gelu_pair && !long_enough) {
        // Short reductions: two CTAs per SM on 128 x 128 tiles measured
        // better (0.192 against 0.204 ms at [100864,256]x[256,1024]).
        wide = false;
    }
    // Narrow tiles (128 x 64 or 128 x 32): a product of few tiles is bound by the
    // serial chain of one of them (ring turns, then one 32-column block after
    // the other through the epilogue), not by its operands' traffic, so the
    // columns are cut as long as all tiles are resident at once, two to an SM.
    // Measured without chaining: [1600,128..512] onto 128 columns 9.6 -> 7.6 us
    // (13 tiles before, 52 now), [1600,128]x[128,512] 7.6 -> 5.6 us, with GELU
    // 10.4 -> 7.8; a step of batch 32 762 -> 668 us, of 117 colour images
    // 559 -> 530 us.  With one tile per SM as the limit these were 673 and 542.
    int narrow = forced_narrow;
    if (narrow < 0 && !g.residual && !forced_tile && !forced_tile_m) {
        const long long row_tiles = (g.m + kTileM - 1) / kTileM;
        // (The slices of a split reduction, four blocks each at least.)
        const long long slices =
            g.accumulate ? std::max(1, (g.k + kBlockK - 1) / kBlockK / 4) : 1;
        for (int candidate : {kNarrow32, kNarrow64}) {
            const int width = kTcTiles[candidate].n;
            if (narrow < 0 && row_tiles * ((g.n + width - 1) / width) * slices <=
                                  2 * (long long)device_sm_count()) {
                narrow = candidate;
            }
        }
    }
    // From here on only the tile counts.
    const TcTile &tile =
        kTcTiles[narrow >= 0 ? narrow : (tall ? kTall : (wide ? kWide : kSquare))];
    const int tile_m = tile.m, tile_n = tile.n;
    // The slope: with a short reduction the epilogue outlasts the products, and eight
    // warps on the square tile get through it sooner; with a longer one they are in the
    // way of the products' copies, and from 512 terms on the 128 x 256 tile is the faster.
    // Measured over 12800 to 65600 rows and 384 to 2048 columns, medians (and extremes)
    // of the ratios to four warps on the square tile:
    //          eight warps          128 x 256 tile
    //   128    0.87 (0.79 .. 0.97)  1.27 (1.18 .. 1.59)
    //   256    0.91 (0.81 .. 0.99)  1.21 (1.14 .. 1.42)
    //   320    0.95 (0.85 .. 1.01)  1.17 (1.06 .. 1.31)
    //   384    0.99 (0.87 .. 1.04)  1.14 (1.02 .. 1.24)
    //   448    1.03 (0.92 .. 1.06)  1.08 (0.96 .. 1.19)
    //   512    1.03 (0.96 .. 1.06)  1.01 (0.94 .. 1.15)
    //   576    1.03 (0.98 .. 1.06)  0.94 (0.88 .. 1.11)
    //   768    1.03 (0.96 .. 1.05)  0.85 (0.80 .. 1.03)
    //   1024   1.02 (0.98 .. 1.08)  0.83 (0.78 .. 1.03)
    const bool square = tile_m == kTileM && tile_n == kTileN;
    const int second = g.d2 ? (g.residual ? kSecondResidual : kSecondGelu)
        : !g.gelu_input     ? 0
        : square && g.k <= 320 ? kGeluSlopeEight : kGeluSlope;
    if (!tile.kernel(second)) {
        return false;
    }
    CUtensorMap &map_a = out->maps.a, &map_b = out->maps.b, &map_d = out->maps.d,
                &map_d2 = out->maps.d2;
    // K-major operand: rows = output index, inner = reduction index.
    const CUtensorMapSwizzle chunks16 = CU_TENSOR_MAP_SWIZZLE_128B;
    const bool a_blocked = g.a_mn_major && g.m % 32 == 0;
    const bool b_blocked = g.b_mn_major && g.n % 32 == 0;
    const bool ok_a = g.a_mn_major
        ? operand_map(g.a, g.m, g.k, g.lda, a_blocked ? tile_m / 32 : 0, &map_a)
        : tensor_map(g.a, g.k, g.m, g.lda, 32, tile_m, chunks16, true, &map_a);
    const bool ok_b = g.b_mn_major
        ? operand_map(g.b, g.n, g.k, g.ldb, b_blocked ? tile_n / 32 : 0, &map_b)
        : tensor_map(g.b, g.k, g.n, g.ldb, 32, tile_n, chunks16, true, &map_b);
    const bool ok_d =
        tensor_map(g.d, g.n, g.m, g.ldd, 32, 32, chunks16, false, &map_d);
    map_d2 = map_d;
    const bool ok_d2 = !g.d2 ||
        tensor_map(g.d2, g.n, g.m, g.ldd2, 32, 32, chunks16, false, &map_d2);
    if (!ok_a || !ok_b || !ok_d || !ok_d2) {
        return false;
    }
    if (g.gelu_input &&
        !tensor_map(g.gelu_input, g.n, g.m, g.ld_gelu_input, 32, 32, chunks16,
                    false, &map_d2)) {
        return false;
    }
    TcParams &p = out->p;
    p.m = g.m;
    p.n = g.n;
    p.k_blocks = (g.k + kBlockK - 1) / kBlockK;
    p.n_tiles = (g.n + tile_n - 1) / tile_n;
    const int m_tiles = (g.m + tile_m - 1) / tile_m;
    p.m_tiles = m_tiles;
    const int tiles = m_tiles * p.n_tiles;
    static const TcForced forced = []() {
        auto number = [](const char *name) { return getenv(name) ? atoi(getenv(name)) : 0; };
        TcForced f;
        f.stages = number("VITB200_TC_STAGES");
        f.staging = number("VITB200_TC_STAGING");
        f.ctas = number("VITB200_TC_CTAS");
        return f;
    }();
    const bool spread = tile_n < kTileN && forced_narrow < 0 &&
                        (long long)tiles <= (long long)device_sm_count();
    const TcShared shared =
        tc_shared(tile_m, tile_n, second, p.k_blocks, g.accumulate, spread, forced);
    p.stages = shared.stages;
    p.staging_bytes = shared.staging_bytes;
    if (p.stages < 1) {
        return false;
    }
    // One or two persistent CTAs on every multiprocessor (never more than
    // the per-CTA partial rows provide for).
    const long long slots =
        std::min<long long>({(long long)device_sm_count() * shared.ctas_per_sm,
                             kGemmPartialRows, most_ctas});
    int splits = 1;
    if (g.accumulate) {
        splits = choose_slices(tiles, p.k_blocks, slots, nullptr);
    }
    p.k_blocks_per_split = (p.k_blocks + splits - 1) / splits;
    splits = (p.k_blocks + p.k_blocks_per_split - 1) / p.k_blocks_per_split;
    p.a_mn_major = g.a_mn_major ? 1 : 0;
    p.b_mn_major = g.b_mn_major ? 1 : 0;
    p.a_blocked = a_blocked ? 1 : 0;
    p.b_blocked = b_blocked ? 1 : 0;
    p.reduce_add = g.accumulate ? 1 : 0;
    p.bias = g.bias;
    p.column_partials = g.column_partials;
    p.residual = g.residual;
    p.residual_pitch = g.ld_residual;
    int *device_status = nullptr;
    cudaHostGetDevicePointer(reinterpret_cast<void **>(&device_status),
                             status_word(), 0);
    p.status = device_status;
    p.splits = splits;
    // One persistent CTA per SM (the shared-memory ring fills an SM), fewer
    // when there is less work than SMs.
    const long long items = (long long)tiles * splits;
    out->grid = unsigned(items < slots ? items : slots);
    out->smem_bytes = shared.bytes();
    out->tile = &tile;
    out->second = second;
    return true;
}

}  // namespace

int launch_gemm_tc(const TcGemm &g, cudaStream_t stream, int *partial_rows) {
    TcLaunch launch;
    if (!prepare(g, -1, kGemmPartialRows, &launch)) {
        return -1;
    }
    if (g.column_partials && partial_rows) {
        *partial_rows = int(launch.grid);
    }
    const TcPairMaps &maps = launch.maps;
    launch_chained(launch.tile->kernel(launch.second), launch.grid,
                   launch.tile->threads[launch.second], launch.smem_bytes, stream, maps.a, maps.b, maps.d, maps.d2, launch.p);
    ++g_kernel_launches;
    ++g_tc_products;
    if (launch.tile->n > kTileN) {
        ++g_tc_wide_products;
    }
    return 0;
}

namespace {

// The narrow tile with which the gradients of [m,k] x [k,n] run side by side, or -1:
// all tiles of the input gradient resident at once with a CTA each, and the weight
// gradient on the SMs' other slots done no later than the two would be one after the
// other.  (The gradients of larger products take as long as their work, in one
// launch or two.)
int find_pair_tile(int m, int k, int n) {
    const long long slots = 2LL * device_sm_count();
    const int depth = (n + kBlockK - 1) / kBlockK;
    const int weight_depth = (m + kBlockK - 1) / kBlockK;
    for (int candidate : {kNarrow32, kNarrow64}) {
        const int width = kTcTiles[candidate].n;
        const long long first = (m + kTileM - 1LL) / kTileM * ((k + width - 1) / width);
        const long long second = (k + kTileM - 1LL) / kTileM * ((n + width - 1) / width);
        if (first + second > slots) {
            continue;
        }
        long long beside = 0, alone = 0;
        choose_slices(second, weight_depth, slots - first, &beside);
        choose_slices(second, weight_depth, slots, &alone);
        if (beside <= depth + 8 + alone) {
            return candidate;
        }
    }
    return -1;
}

int pair_tile(int m, int k, int n) {
    // (Asked before the product is held back and again when it is launched.)
    static thread_local int last[4] = {0, 0, 0, -1};
    if (last[0] != m || last[1] != k || last[2] != n) {
        last[0] = m;
        last[1] = k;
        last[2] = n;
        last[3] = find_pair_tile(m, k, n);
    }
    return last[3];
}

}  // namespace

bool gemm_tc_pairs(int m, int k, int n) {
    return pair_tile(m, k, n) >= 0;
}

int launch_gemm_tc_pair(const TcGemm &input, const TcGemm &weight, cudaStream_t stream,
                        int *partial_rows) {
    const int tile = pair_tile(input.m, input.n, input.k);
    if (tile < 0 || input.d2 || weight.d2 || weight.gelu_input || weight.bias) {
        return -1;
    }
    TcLaunch first, second;
    const long long slots = std::min<long long>(2LL * device_sm_count(), kGemmPartialRows);
    if (!prepare(input, tile, slots, &first) ||
        !prepare(weight, tile, slots - first.grid, &second)) {
        return -1;
    }
    const bool slope = first.second == kGeluSlope;
    const auto kernel = tile == kNarrow32
        ? (slope ? gemm_tc_pair_kernel<32, kGeluSlope> : gemm_tc_pair_kernel<32, 0>)
        : (slope ? gemm_tc_pair_kernel<64, kGeluSlope> : gemm_tc_pair_kernel<64, 0>);
    static SharedMemoryLimit limit;
    const void *kernels[4] = {
        reinterpret_cast<const void *>(gemm_tc_pair_kernel<32, 0>),
        reinterpret_cast<const void *>(gemm_tc_pair_kernel<32, kGeluSlope>),
        reinterpret_cast<const void *>(gemm_tc_pair_kernel<64, 0>),
        reinterpret_cast<const void *>(gemm_tc_pair_kernel<64, kGeluSlope>)};
    if (!limit.raise(kernels, 4, kSmemLimit)) {
        return -1;
    }
    if (input.column_partials && partial_rows) {
        *partial_rows = int(first.grid);
    }
    launch_chained(kernel, first.grid + second.grid, kThreads,
                   std::max(first.smem_bytes, second.smem_bytes), stream, first.maps,
                   second.maps, first.p, second.p, int(first.grid));
    ++g_kernel_launches;
    g_tc_products += 2;
    return 0;
}

bool gemm_plain_map(const float *base, unsigned long long inner, unsigned long long outer,
                    unsigned long long pitch, unsigned box_inner, unsigned box_outer,
                    bool swizzled, CUtensorMap *out) {
    return tensor_map(base, inner, outer, pitch, box_inner, box_outer,
                      swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                      false, out);
}

unsigned long long g_tc_products = 0, g_tc_wide_products = 0;

int gemm_tc_status() {
    int *word = status_word();
    return word ? *word : 0;
}

int *tc_status_device_pointer() {
    int *word = status_word();
    int *device = nullptr;
    if (!word || cudaHostGetDevicePointer(reinterpret_cast<void **>(&device),
                                          word, 0) != cudaSuccess) {
        return nullptr;
    }
    return device;
}

}  // namespace vitb200
