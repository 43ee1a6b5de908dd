// Large FP32 products on the tensor cores, at FP32 accuracy.
//
//   C[M,N] (+)= A[M,K] * B[K,N]
//
// in the three storage forms of gemm_fma.cu, whose place it takes where the
// product has enough 128 x 128 tiles (gemm_split_plan.h).
//
// Arithmetic (after Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial
// Intelligence Datatype For Higher-Precision Computations", 2019).  A float is the sum of
// three bfloat16 values (8 + 8 + 8 bits, each the nearest to what the ones before it leave
// over), so a product of two floats is the sum of nine products of bfloat16 values, all of
// them exact in FP32.  The three smallest (2^-24 of the largest and less) are left out, the
// other six are tcgen05.mma kind::f16 instructions into FP32 accumulators: the largest into one
// that lives for 64 terms (four instructions) only, or for 32 (p.chunk), the other five
// into one of their own.  The tensor core's additions truncate, so a long-lived
// accumulator of large terms would drift; instead each is added, rounded to nearest, to
// sums that the epilogue threads keep in registers.  A sum over K then takes K/64
// roundings one after the other where a chain of FMAs takes K.  What this makes of the
// errors, and where FMAs' own are smaller, is in gemm_split_plan.h.  The third part of a
// value holds its bits down to 2^-133, so that values below 2^-110 (8e-34) lose low bits:
// 2-norm error 7.5e-8 with operands down to 2^-108, 1.6e-7 at 2^-112, 3.5e-5 at 2^-120.
// (Products and sums below FP32's normal range keep what FMAs keep of them.)  An
// infinity has no such parts: 32 x 32 values of the result with one among them that is not
// finite are computed again by FMAs, which gives what they give, once the CTA's products
// are done (recompute).
//
// What bounds it: shared memory.  A block of 128 x 128 x 32 is 12 instructions that
// read 8 KiB of operands in 64 clocks each; its 32 KiB of floats are written by the
// copy engine and read by the threads that split them, which write 48 KiB of parts:
// 200 KiB, 1600 clocks at 128 bytes per clock, where the FMA pipes need 4096 (and
// take 6000).  All of these accesses are free of bank conflicts: K-contiguous
// operands arrive in the 128-byte swizzle, others as plain rows, and the parts are
// kept in the K-major layout of 8 x 16-byte core matrices whichever way the operand
// is stored.  (Fetching the floats straight into registers took three times the
// shared-memory cycles in partly used sectors, and threads that fetch, split and
// add up in turn expose the latency of each step.)
//
// Roles: eight warps split operands; eight add up (32 rows x 64 columns of the tile
// each) and write the result while the next tile's blocks are split; one issues the
// copies and, once all eight are done with a block, its products.  They meet at
// mbarriers only: three stages of floats, two of parts, two accumulators of each kind
// in tensor memory.
#include "device_util.cuh"
#include "gemm.h"
#include "gemm_split_plan.h"
#include "gemm_tc.h"
#include "kernels.h"
#include "shared_limit.h"
#include "tcgen05.cuh"

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace vitb200 {
namespace {

using namespace tc;

constexpr int kTile = kSplitTile;
constexpr int kBlockK = kSplitBlockK;
constexpr int kParts = 3;
constexpr int kPartBytes = kTile * kBlockK * 2;             // 8 KiB
constexpr int kOperandBytes = kParts * kPartBytes;
constexpr int kStageBytes = 2 * kOperandBytes;              // parts: 48 KiB
constexpr int kStages = 2;
constexpr int kRawBytes = kTile * kBlockK * 4;              // an operand's floats
constexpr int kRawStageBytes = 2 * kRawBytes;               // 32 KiB
constexpr int kRawStages = 3;
constexpr int kConverters = 8;   // warps
constexpr int kAdders = 8;
constexpr int kIssuer = kConverters + kAdders;              // the last warp
constexpr int kThreads = 32 * (kIssuer + 1);
constexpr int kColumns = kTile / (kAdders / 4);             // of an adding warp: 64
constexpr int kStagingBytes = 32 * 32 * 4;                  // of such a warp
constexpr int kPartsAt = kRawStages * kRawStageBytes;
constexpr int kStagingAt = kPartsAt + kStages * kStageBytes;
constexpr int kBarriersAt = kStagingAt + kAdders * kStagingBytes;
constexpr int kSharedBytes = kBarriersAt + 256;
static_assert(kSharedBytes + 1024 <= 227 * 1024, "fits an SM");
constexpr int kMainColumns = 0, kRestColumns = 2 * kTile;   // in tensor memory

struct SplitParams {
    const float *a, *b;
    const float *bias;         // added per column, or null
    const float *gelu_input;   // C is multiplied by gelu'(this), or null
    int gelu_out;              // second output gelu(C)
    float *partials;           // a row of n column sums of C per CTA, or null
    int m, n, k;
    int m_tiles, n_tiles;
    int blocks, blocks_per_slice, slices;   // of the reduction
    int chunk;                 // blocks that a main accumulator lives for: 1 or 2
    long long lda, ldb, ldc;
    int add;                   // C += instead of C =
    int *status;
};

// An item of work: a tile and a slice of the reduction.
struct Item {
    int m0, n0, begin, end;    // blocks [begin, end)

    __device__ __forceinline__ Item(const SplitParams &p, int index) {
        const int tiles = p.m_tiles * p.n_tiles;
        const int tile = index % tiles;
        m0 = tile / p.n_tiles * kTile;
        n0 = tile % p.n_tiles * kTile;
        begin = index / tiles * p.blocks_per_slice;
        end = min(p.blocks, begin + p.blocks_per_slice);
    }
};

// Where a walk over the CTA's blocks stands: item after item, block after block.
struct Cursor {
    int index;
    Item item;
    int block;

    __device__ __forceinline__ Cursor(const SplitParams &p, int first)
        : index(first), item(p, first), block(item.begin) {}
    __device__ __forceinline__ void step(const SplitParams &p) {
        if (++block == item.end) {
            index += int(gridDim.x);
            item = Item(p, index);
            block = item.begin;
        }
    }
};

// Two floats as packed bfloat16, the first in the low half.
__device__ __forceinline__ uint32_t pack_bf16(float low, float high) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(high), "f"(low));
    return r;
}

// What a converting warp takes of an operand at a time: eight terms ("octet") of 32
// output indices ("rows"), one row per lane.  A block has 16 such units.
//   K-contiguous: lanes 8 rows x 4 octets     otherwise: 32 rows of one octet
template <bool K_CONTIGUOUS>
__device__ __forceinline__ void unit_of_lane(int unit, int &row, int &octet) {
    const int lane = threadIdx.x & 31;
    row = K_CONTIGUOUS ? 8 * unit + (lane & 7) : 32 * (unit & 3) + lane;
    octet = K_CONTIGUOUS ? lane >> 3 : unit >> 2;
}

// The lane's octet from an operand's floats: rows of 32 terms in the 128-byte swizzle
// (16-byte chunk c of row r at c ^ (r % 8)), or 32 terms of 128 rows each.
template <bool K_CONTIGUOUS>
__device__ __forceinline__ void read_octet(const float *raw, int unit, float (&v)[8]) {
    int row, octet;
    unit_of_lane<K_CONTIGUOUS>(unit, row, octet);
    if (K_CONTIGUOUS) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float4 x = *reinterpret_cast<const float4 *>(
                raw + row * kBlockK + 4 * ((2 * octet + q) ^ (row & 7)));
            v[4 * q] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = raw[(8 * octet + e) * kTile + row];
        }
    }
}

// Its three parts to where the tensor core reads them: a part is four columns of core
// matrices (8 terms wide), a column 128 rows of 16 bytes.
template <bool K_CONTIGUOUS>
__device__ __forceinline__ void write_parts(float (&v)[8], int unit, uint32_t operand) {
    int row, octet;
    unit_of_lane<K_CONTIGUOUS>(unit, row, octet);
    const uint32_t address = operand + octet * (kTile * 16) + row * 16;
#pragma unroll
    for (int part = 0; part < kParts; ++part) {
        uint32_t pair[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            pair[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
            if (part + 1 < kParts) {
                v[2 * e] -= __uint_as_float(pair[e] << 16);
                v[2 * e + 1] -= __uint_as_float(pair[e] & 0xffff0000u);
            }
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                         address + part * kPartBytes),
                     "r"(pair[0]), "r"(pair[1]), "r"(pair[2]), "r"(pair[3])
                     : "memory");
    }
}

// D[tmem] (+)= A[smem] * B[smem], bfloat16 operands, FP32 accumulation.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t desc_a,
                                         uint64_t desc_b, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void load_16_columns(uint32_t address, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32"
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15},"
        " [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(address)
        : "memory");
}

// The product of parts `a` and `b` of a stage's operands: 2 x 16 terms, each two
// columns of core matrices, 2 KiB apart, whose groups of eight rows are 128 bytes apart.
__device__ __forceinline__ void multiply_parts(uint32_t accumulator, uint32_t stage, int a,
                                               int b, bool add) {
    // kind::f16, bfloat16 operands, FP32 accumulator, 128 x 128, K-major.
    constexpr uint32_t kInstruction = (1u << 4) | (1u << 7) | (1u << 10) |
                                      (uint32_t(kTile >> 3) << 17) |
                                      (uint32_t(kTile >> 4) << 24);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t step = half * 2 * (kTile * 16);
        mma_bf16(accumulator,
                 operand_descriptor(stage + a * kPartBytes + step, kTile * 16, 128, 0),
                 operand_descriptor(stage + kOperandBytes + b * kPartBytes + step,
                                    kTile * 16, 128, 0),
                 kInstruction, add || half > 0 ? 1u : 0u);
    }
}

// 32 rows (from row0 on) x 32 columns (a lane each, from col on) once more, by FMAs in
// the order of the reduction, a sum of 64 terms at a time, into a block of shared memory:
// for those with an infinity or a NaN among them.  Zeros past the matrix.  The operands
// of eight terms are requested together; rows of which only NaNs are left are done.
template <bool A_K, bool B_K>
__device__ __forceinline__ void recompute(const SplitParams &p, int row0, int col,
                                          int k_begin, int k_end, float *block) {
    constexpr int kRows = 4, kTerms = 8;
    const int lane = threadIdx.x & 31;
    const long long column = min(col + lane, p.n - 1);
    const float *b = p.b + (B_K ? column * p.ldb : column);
    for (int r = 0; r < 32; r += kRows) {
        const float *a[kRows];
        float sum[kRows], part[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const long long row = min(row0 + r + i, p.m - 1);
            a[i] = p.a + (A_K ? row * p.lda : row);
            sum[i] = part[i] = 0.0f;
        }
        for (int k = k_begin; k < k_end; k += kTerms) {
            float x[kRows][kTerms], y[kTerms];
#pragma unroll
            for (int t = 0; t < kTerms; ++t) {
                const long long at = min(k + t, k_end - 1);
                y[t] = __ldg(b + (B_K ? at : at * p.ldb));
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                    x[i][t] = __ldg(a[i] + (A_K ? at : at * p.lda));
                }
            }
#pragma unroll
            for (int t = 0; t < kTerms; ++t) {
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                    part[i] = k + t < k_end ? fmaf(x[i][t], y[t], part[i]) : part[i];
                }
            }
            if (k % 64 == 64 - kTerms || k + kTerms >= k_end) {
                bool numbers = false;
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                    sum[i] += part[i];
                    part[i] = 0.0f;
                    numbers |= sum[i] == sum[i];
                }
                if (!__any_sync(kFullMask, numbers)) {
                    break;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            block[(r + i) * 32 + lane] =
                col + lane < p.n && row0 + r + i < p.m ? sum[i] : 0.0f;
        }
    }
    __syncwarp();
}

// Four floats from column `col` of a row of n, zeros past its end.
__device__ __forceinline__ float4 four_of(const float *row, int col, int n) {
    if (col + 4 <= n) {
        return __ldg(reinterpret_cast<const float4 *>(row + col));
    }
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (col < n) x.x = __ldg(row + col);
    if (col + 1 < n) x.y = __ldg(row + col + 1);
    if (col + 2 < n) x.z = __ldg(row + col + 2);
    return x;
}

// A lane's row of a 32 x 32 block into shared memory, in the 128-byte swizzle.
__device__ __forceinline__ void stage_row(float *block, const float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        *reinterpret_cast<float4 *>(block + lane * 32 + 4 * (c ^ (lane & 7))) =
            make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
}

// Whether all of a warp's sums are finite.
__device__ __forceinline__ bool all_finite(const float (&v)[32]) {
    // Zero times a sum is zero unless the sum is infinite or not a number.
    float probe = 0.0f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        probe = fmaf(v[j], 0.0f, probe);
    }
    return __all_sync(kFullMask, probe == 0.0f);
}

// The copy engine has read the warp's block.
__device__ __forceinline__ void await_block() {
    if ((threadIdx.x & 31) == 0) {
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncwarp();
}

// Everything between a warp's sums (32 rows, one per lane, from row0 on; 32 columns
// from col on) and memory, through the warp's block of shared memory.
__device__ __forceinline__ void finish(const SplitParams &p, const CUtensorMap &map_c,
                                       const CUtensorMap &map_gelu, float *block, int row0,
                                       int col, float (&v)[32]) {
    if (row0 >= p.m || col >= p.n) {
        return;   // uniform across the warp
    }
    const int lane = threadIdx.x & 31, row = row0 + lane;
    await_block();
    if (p.bias) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 x = four_of(p.bias, col + j, p.n);
            v[j] += x.x; v[j + 1] += x.y; v[j + 2] += x.z; v[j + 3] += x.w;
        }
    }
    if (p.gelu_input && row < p.m) {
        const float *h = p.gelu_input + row * p.ldc;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 x = four_of(h, col + j, p.n);
            v[j] *= gelu_slope(x.x);
            v[j + 1] *= gelu_slope(x.y);
            v[j + 2] *= gelu_slope(x.z);
            v[j + 3] *= gelu_slope(x.w);
        }
    }
    auto send = [&](const CUtensorMap &map, bool add) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            if (add) {
                tma_reduce_add_2d(block, &map, col, row0);
            } else {
                tma_store_2d(block, &map, col, row0);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    };
    stage_row(block, v);
    send(map_c, p.add);
    if (p.partials) {
        // Column sums of the block (rows past the matrix are zero), lane = column.
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            sum[r & 3] += block[r * 32 + 4 * ((lane >> 2) ^ (r & 7)) + (lane & 3)];
        }
        if (col + lane < p.n) {
            atomicAdd(p.partials + size_t(blockIdx.x) * p.n + col + lane,
                      (sum[0] + sum[1]) + (sum[2] + sum[3]));
        }
    }
    if (p.gelu_out) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            v[j] = gelu_value(v[j]);
        }
        await_block();
        stage_row(block, v);
        send(map_gelu, false);
    }
}

// The same for 32 x 32 values whose sums were not finite.
template <bool A_K, bool B_K>
__device__ __noinline__ void finish_again(const SplitParams &p, const CUtensorMap &map_c,
                                          const CUtensorMap &map_gelu, float *block,
                                          int row0, int col, int k_begin, int k_end) {
    if (row0 >= p.m || col >= p.n) {
        return;   // uniform across the warp
    }
    await_block();
    recompute<A_K, B_K>(p, row0, col, k_begin, k_end, block);
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        v[j] = block[(threadIdx.x & 31) * 32 + j];
    }
    __syncwarp();
    finish(p, map_c, map_gelu, block, row0, col, v);
}

// The barriers, and what each phase of them stands for.
struct Barriers {
    uint64_t *raw_full;      // floats of a block have arrived
    uint64_t *parts_full;    // ... have been split (and may be overwritten)
    uint64_t *parts_empty;   // its products are done
    uint64_t *main_full, *main_empty;   // an accumulator of large terms
    uint64_t *rest_full, *rest_empty;   // one of small terms (per item)

    __device__ __forceinline__ explicit Barriers(uint8_t *memory) {
        raw_full = reinterpret_cast<uint64_t *>(memory);
        parts_full = raw_full + kRawStages;
        parts_empty = parts_full + kStages;
        main_full = parts_empty + kStages;
        main_empty = main_full + 2;
        rest_full = main_empty + 2;
        rest_empty = rest_full + 2;
    }
};

// A_K / B_K: the operand's rows have K contiguous (otherwise M / N).
template <bool A_K, bool B_K>
__global__ void __launch_bounds__(kThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a,
                  const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_c,
                  const __grid_constant__ CUtensorMap map_gelu,
                  const __grid_constant__ SplitParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_slot;
    const Barriers bars(smem + kBarriersAt);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRawStages; ++s) {
            mbarrier_init(&bars.raw_full[s], 1);
        }
        for (int s = 0; s < kStages; ++s) {
            mbarrier_init(&bars.parts_full[s], kConverters);
            mbarrier_init(&bars.parts_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbarrier_init(&bars.main_full[s], 1);
            mbarrier_init(&bars.main_empty[s], kAdders);
            mbarrier_init(&bars.rest_full[s], 1);
            mbarrier_init(&bars.rest_empty[s], kAdders);
        }
        prefetch_tensor_map(&map_a);
        prefetch_tensor_map(&map_b);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kIssuer) {
        tmem_allocate(&tmem_slot, 4 * kTile);
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = tmem_slot;
    grid_dependency_wait();
    grid_dependency_release();
    if (p.partials) {
        // This CTA's own row of column sums, which its warps add into.
        for (int c = threadIdx.x; c < p.n; c += kThreads) {
            p.partials[size_t(blockIdx.x) * p.n + c] = 0.0f;
        }
        __threadfence();
        __syncthreads();
    }
    const int items = p.m_tiles * p.n_tiles * p.slices;
    bool ok = (smem_address(smem) & 1023u) == 0;   // (what the swizzle relies on)
    if (!ok && threadIdx.x == 0) {
        atomicExch(p.status, 8);
    }

    int total = 0;   // blocks of this CTA
    for (int index = blockIdx.x; index < items; index += gridDim.x) {
        const Item item(p, index);
        total += item.end - item.begin;
    }
    if (warp == kIssuer) {
        if (lane == 0 && ok) {
            Cursor loading(p, blockIdx.x), issuing(p, blockIdx.x);
            int chunks = 0, opened = 0;
            auto load = [&](int g) {
                uint8_t *raw = smem + g % kRawStages * kRawStageBytes;
                uint64_t *full = &bars.raw_full[g % kRawStages];
                const int k0 = loading.block * kBlockK;
                mbarrier_expect_tx(full, kRawStageBytes);
                if (A_K) {
                    tma_load_2d(raw, &map_a, k0, loading.item.m0, full);
                } else {
                    tma_load_2d(raw, &map_a, loading.item.m0, k0, full);
                }
                if (B_K) {
                    tma_load_2d(raw + kRawBytes, &map_b, k0, loading.item.n0, full);
                } else {
                    tma_load_2d(raw + kRawBytes, &map_b, loading.item.n0, k0, full);
                }
                loading.step(p);
            };
            auto multiply = [&](int g) {
                const uint32_t stage = smem_address(smem + kPartsAt + g % kStages * kStageBytes);
                const int position = issuing.block - issuing.item.begin;
                const bool first = position == 0, last = issuing.block + 1 == issuing.item.end;
                const bool chunk_first = (position & (p.chunk - 1)) == 0;
                const int main = chunks & 1, rest = opened & 1;
                bool served = true;
                if (chunk_first) {
                    served = mbarrier_wait(&bars.main_empty[main], ((chunks >> 1) & 1) ^ 1);
                }
                if (first && served) {
                    served = mbarrier_wait(&bars.rest_empty[rest], ((opened >> 1) & 1) ^ 1);
                }
                if (!served) {
                    return false;
                }
                tcgen05_fence_after();
                const uint32_t small = tmem + kRestColumns + rest * kTile;
                multiply_parts(small, stage, 2, 0, !first);
                multiply_parts(small, stage, 0, 2, true);
                multiply_parts(small, stage, 1, 1, true);
                multiply_parts(small, stage, 1, 0, true);
                multiply_parts(small, stage, 0, 1, true);
                multiply_parts(tmem + kMainColumns + main * kTile, stage, 0, 0, !chunk_first);
                tcgen05_commit(&bars.parts_empty[g % kStages]);
                if (last || (position & (p.chunk - 1)) == p.chunk - 1) {
                    tcgen05_commit(&bars.main_full[main]);
                    ++chunks;
                }
                if (last) {
                    tcgen05_commit(&bars.rest_full[rest]);
                    ++opened;
                }
                issuing.step(p);
                return true;
            };
            for (int g = 0; g < kRawStages && g < total; ++g) {
                load(g);
            }
            for (int g = 0; g < total && ok; ++g) {
                ok = mbarrier_wait(&bars.parts_full[g % kStages], (g / kStages) & 1);
                if (ok) {
                    // All have read the block's floats: their stage is free.
                    if (g + kRawStages < total) {
                        load(g + kRawStages);
                    }
                    ok = multiply(g);
                }
            }
            if (!ok) {
                atomicExch(p.status, 11);
            }
        }
    } else if (warp < kConverters) {
        for (int g = 0; g < total && ok; ++g) {
            const int r = g % kRawStages, s = g % kStages;
            ok = __all_sync(kFullMask,
                            mbarrier_wait(&bars.raw_full[r], (g / kRawStages) & 1));
            if (!ok) {
                break;
            }
            const float *raw = reinterpret_cast<const float *>(smem + r * kRawStageBytes);
            float a[2][8], b[2][8];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                read_octet<A_K>(raw, warp + kConverters * i, a[i]);
                read_octet<B_K>(raw + kRawBytes / 4, warp + kConverters * i, b[i]);
            }
            ok = __all_sync(kFullMask,
                            mbarrier_wait(&bars.parts_empty[s], ((g / kStages) & 1) ^ 1));
            if (!ok) {
                break;
            }
            const uint32_t stage = smem_address(smem + kPartsAt + s * kStageBytes);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                write_parts<A_K>(a[i], warp + kConverters * i, stage);
                write_parts<B_K>(b[i], warp + kConverters * i, stage + kOperandBytes);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbarrier_arrive(&bars.parts_full[s]);
            }
        }
        if (!ok && lane == 0) {
            atomicExch(p.status, 9);
        }
    } else {
        const int quarter = warp & 3, group = (warp - kConverters) >> 2;
        float *block = reinterpret_cast<float *>(smem + kStagingAt +
                                                 (warp - kConverters) * kStagingBytes);
        const uint32_t lanes = tmem + (uint32_t(32 * quarter) << 16) + kColumns * group;
        int chunks = 0, opened = 0;
        // Halves of items that are not finite are computed again after the last one
        // (over many rows that takes a while, which the issuer would wait for): a bit
        // each, two per item, those of 16 items in a lane.  (Few products have more than
        // that many items per CTA, and have them after that many.)
        constexpr int kRemembered = 32 * 16;
        uint32_t put_off = 0;
        int ordinal = 0;
        auto again = [&](const Item &item, int half) {
            finish_again<A_K, B_K>(p, map_c, map_gelu, block, item.m0 + 32 * quarter,
                                   item.n0 + kColumns * group + 32 * half,
                                   item.begin * kBlockK, min(p.k, item.end * kBlockK));
        };
        float sums[2][32];
        auto add = [&](uint32_t columns) {
#pragma unroll
            for (int part = 0; part < kColumns; part += 16) {
                uint32_t r[16];
                load_16_columns(lanes + columns + part, r);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    sums[part / 32][part % 32 + j] += __uint_as_float(r[j]);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
        };
        for (int index = blockIdx.x; index < items && ok; index += gridDim.x) {
            const Item item(p, index);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                sums[0][j] = sums[1][j] = 0.0f;
            }
            for (int first = item.begin; first < item.end && ok; first += p.chunk) {
                const int main = chunks & 1;
                ok = __all_sync(kFullMask, mbarrier_wait(&bars.main_full[main],
                                                         (chunks >> 1) & 1));
                if (ok) {
                    tcgen05_fence_after();
                    add(kMainColumns + main * kTile);
                    if (lane == 0) {
                        mbarrier_arrive(&bars.main_empty[main]);
                    }
                    ++chunks;
                }
            }
            const int rest = opened & 1;
            ok = ok && __all_sync(kFullMask, mbarrier_wait(&bars.rest_full[rest],
                                                           (opened >> 1) & 1));
            if (!ok) {
                break;
            }
            tcgen05_fence_after();
            add(kRestColumns + rest * kTile);
            if (lane == 0) {
                mbarrier_arrive(&bars.rest_empty[rest]);
            }
            ++opened;
            uint32_t infinite = 0;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (all_finite(sums[half])) {
                    finish(p, map_c, map_gelu, block, item.m0 + 32 * quarter,
                           item.n0 + kColumns * group + 32 * half, sums[half]);
                } else {
                    infinite |= 1u << half;
                }
            }
            if (lane == ordinal / 16) {
                put_off |= infinite << (2 * (ordinal % 16));
            }
            if (++ordinal < kRemembered && index + int(gridDim.x) < items) {
                continue;
            }
            const int first = index - (ordinal - 1) * int(gridDim.x);
            for (uint32_t left = __ballot_sync(kFullMask, put_off != 0); left;
                 left &= left - 1) {
                const int from = __ffs(left) - 1;
                for (uint32_t bits = __shfl_sync(kFullMask, put_off, from); bits;
                     bits &= bits - 1) {
                    const int bit = __ffs(bits) - 1;
                    again(Item(p, first + (16 * from + bit / 2) * int(gridDim.x)), bit & 1);
                }
            }
            put_off = 0;
            ordinal = 0;
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
        if (!ok && lane == 0) {
            atomicExch(p.status, 10);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == kIssuer) {
        __syncwarp();
        tcgen05_fence_after();
        tmem_free(tmem, 4 * kTile);
    }
}

}  // namespace

// Measured with launches back to back (us; FMA kernel -> this one; 2-norm errors against
// 64 bits of normal values, x 1e-7):
//   [12800,128]x[128,128]   16.4 -> 9.8  (2.0 -> 0.75), its gradients  44 -> 22
//   [12800,128]x[128,512]   46.0 -> 19.3 (2.0 -> 0.75),               100 -> 41
//   [12800,512]x[512,128]   55.5 -> 22.1 (4.0 -> 0.90),                98 -> 39
//   [30000,256]x[256,1024]  337 -> 120   (2.9 -> 0.81),               679 -> 254
//   [4329,96]x[96,384]      13.3 -> 8.7  (1.8 -> 0.69),                31 -> 21
// ([20000,64]x[64,64], 9.9, and [1600,512]x[512,128], 18.6, are left to FMAs by the
// estimate.)  Sums of positive terms 1.5 to 4.3 -> 0.7 to 0.9; what adds to C:
// gemm_split_plan.h.
double gemm_split_clocks(const FmaGemm &g, double error) {
    return split_plan(g, int(device_sm_count()), error).clocks;
}

bool launch_gemm_split(const FmaGemm &g, double error, cudaStream_t stream,
                       int *partial_rows) {
    const SplitPlan plan = split_plan(g, int(device_sm_count()), error);
    if (plan.clocks == HUGE_VAL) {
        return false;
    }
    SplitParams p = {};
    p.a = g.a;
    p.b = g.b;
    p.bias = g.bias;
    p.gelu_out = g.gelu_out ? 1 : 0;
    p.gelu_input = g.gelu_input;
    p.partials = g.column_partials;
    p.m = g.m;
    p.n = g.n;
    p.k = g.k;
    p.lda = g.lda;
    p.ldb = g.ldb;
    p.ldc = g.ldc;
    p.m_tiles = plan.m_tiles;
    p.n_tiles = plan.n_tiles;
    p.blocks = plan.blocks;
    p.blocks_per_slice = plan.blocks_per_slice;
    p.slices = plan.slices;
    p.chunk = plan.chunk;
    p.add = g.accumulate ? 1 : 0;
    const unsigned grid = unsigned(std::min<long long>(
        (long long)p.m_tiles * p.n_tiles * p.slices, device_sm_count()));
    CUtensorMap map_a, map_b, map_c, map_gelu;
    const bool mapped =
        (g.a_k ? gemm_plain_map(g.a, g.k, g.m, g.lda, kBlockK, kTile, true, &map_a)
               : gemm_plain_map(g.a, g.m, g.k, g.lda, kTile, kBlockK, false, &map_a)) &&
        (g.b_k ? gemm_plain_map(g.b, g.k, g.n, g.ldb, kBlockK, kTile, true, &map_b)
               : gemm_plain_map(g.b, g.n, g.k, g.ldb, kTile, kBlockK, false, &map_b)) &&
        gemm_plain_map(g.c, g.n, g.m, g.ldc, 32, 32, true, &map_c) &&
        gemm_plain_map(g.gelu_out ? g.gelu_out : g.c, g.n, g.m, g.ldc, 32, 32, true,
                       &map_gelu);
    p.status = tc_status_device_pointer();
    if (!mapped || !p.status) {
        return false;
    }
    static SharedMemoryLimit limit;
    const void *kernels[3] = {
        reinterpret_cast<const void *>(gemm_split_kernel<true, false>),
        reinterpret_cast<const void *>(gemm_split_kernel<true, true>),
        reinterpret_cast<const void *>(gemm_split_kernel<false, false>)};
    if (!limit.raise(kernels, 3, kSharedBytes)) {
        return false;
    }
    const auto kernel = g.a_k ? (g.b_k ? gemm_split_kernel<true, true>
                                       : gemm_split_kernel<true, false>)
                              : gemm_split_kernel<false, false>;
    if (launch_chained(kernel, grid, kThreads, kSharedBytes, stream, map_a, map_b,
                       map_c, map_gelu, p) !=
        cudaSuccess) {
        return false;
    }
    if (g.column_partials && partial_rows) {
        *partial_rows = int(grid);
    }
    ++g_kernel_launches;
    return true;
}

}  // namespace vitb200
