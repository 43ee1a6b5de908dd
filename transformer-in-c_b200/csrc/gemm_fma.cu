// FP32 FMA matrix products: the FP32 policy (except large ones, gemm_split.cu),
// products too small for the tensor cores and layouts TMA cannot describe.
// C[M,N] (+)= A[M,K] * B[K,N] for the three storage forms of a product and its two
// gradients (reference src/ops.c:123-132 and :153-163):
//   forward        A rows with K contiguous,  B rows with N contiguous
//   input grad     A rows with K contiguous,  B rows with K contiguous
//   weight grad    A rows with M contiguous,  B rows with N contiguous
//
// What bounds it: the FMA pipes for large products (128 FP32 lanes per SM, 74
// TFLOP/s), latency for small ones.  Each thread keeps an RM x RN block of C in
// registers as pairs along N, so that one fma.rn.f32x2 does two of them and the
// issue slots left over hide the shared-memory loads; operand tiles come in
// through a ring of three stages, two blocks ahead.
//
// Tiles of 128 x 128 and 64 x 128 for products that fill the chip with them,
// smaller ones below that (plan_product), and 32 x 32 for the latency-sized
// ones.  The smallest also splits the reduction over a cluster of up to eight
// CTAs, which add their partial tiles through distributed shared memory, so
// that a product of 50 rows over 512 columns of reduction occupies 64 SMs and
// takes one trip to memory instead of a chain of 32 on 2 SMs.  Weight gradients
// (M, N small, K = all rows) split K over blockIdx.z and combine with vector
// reductions in L2.
//
// Measured (B200, against the 64 x 64 kernel with scalar staging this
// replaces): [50,512]x[512,128] 31.5 -> 3.9 us, [50,128]x[128,384] with bias
// 10.5 -> 3.9 us, [12800,128]x[128,512] 61 -> 46 us (36 TFLOP/s), its gradient
// pair 170 -> 97 us, weight gradient 46 TFLOP/s.  Shared-memory bandwidth is what
// keeps the large tiles at two thirds of the FMA rate: with 8 x 8 values per
// thread a step loads 16 floats per lane for 64 multiply-adds, which takes the
// one shared-memory pipe about as long as the four FMA pipes (8 x 16 values per
// thread leave too few warps to cover the latencies: slower).
#include "gemm.h"
#include "gemm_split_plan.h"
#include "kernels.h"
#include "device_util.cuh"
#include "shared_limit.h"

#include <algorithm>
#include <climits>
#include <cstdint>

namespace vitb200 {
namespace {

constexpr int kStages = 3;

struct FmaParams {
    const float *a, *b;
    float *c;
    const float *bias;         // added per column, or null
    float *gelu_out;           // second output gelu(C), or null
    const float *gelu_input;   // C is multiplied by gelu'(this), or null
    float *partials;           // column sums of C, see partial_rows
    int partial_rows;
    int m, n, k;
    int k_per_split;
    long long lda, ldb, ldc;
    int vec_a, vec_b, vec_c;   // 16-byte accesses allowed
    int accumulate;            // C += (one writer per element)
    int reduce;                // C += by reductions (the K slices of a weight gradient)
    int partials_shared;       // several tiles add into one row of partials
};

__device__ __forceinline__ uint32_t shared_address(const void *pointer) {
    return uint32_t(__cvta_generic_to_shared(pointer));
}

// Four consecutive floats, the first `valid` of them real and the rest zero.
__device__ __forceinline__ void copy_chunk(float *to, const float *from,
                                           int valid, bool vec) {
    if (vec) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         shared_address(to)),
                     "l"(from), "r"(valid * 4)
                     : "memory");
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int bytes = e < valid ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                             shared_address(to + e)),
                         "l"(e < valid ? from + e : from), "r"(bytes)
                         : "memory");
        }
    }
}

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}

__device__ __forceinline__ void unpack2(unsigned long long v, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}

__device__ __forceinline__ void fma2(unsigned long long &c, unsigned long long a,
                                     unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// `count` (1, 2 or 4) consecutive elements of row `row` from column `col` on:
// everything that happens between the sum and memory.  Leaves in v what was
// stored (for the column sums).
template <int COUNT>
__device__ __forceinline__ void finish(const FmaParams &p, int row, int col,
                                       float (&v)[COUNT]) {
    if (row >= p.m || col >= p.n) {
#pragma unroll
        for (int e = 0; e < COUNT; ++e) {
            v[e] = 0.0f;
        }
        return;
    }
    float *c = p.c + (long long)row * p.ldc + col;
    const bool full = col + COUNT <= p.n;
    if (p.bias) {
#pragma unroll
        for (int e = 0; e < COUNT; ++e) {
            if (full || col + e < p.n) {
                v[e] += __ldg(p.bias + col + e);
            }
        }
    }
    if (p.gelu_input) {
        const float *h = p.gelu_input + (long long)row * p.ldc + col;
        float x[COUNT];
        if (COUNT == 4 && full && p.vec_c) {
            const float4 four = *reinterpret_cast<const float4 *>(h);
            x[0] = four.x;
            x[COUNT > 1 ? 1 : 0] = four.y;
            x[COUNT > 2 ? 2 : 0] = four.z;
            x[COUNT > 3 ? 3 : 0] = four.w;
        } else {
#pragma unroll
            for (int e = 0; e < COUNT; ++e) {
                x[e] = col + e < p.n ? h[e] : 0.0f;
            }
        }
#pragma unroll
        for (int e = 0; e < COUNT; ++e) {
            v[e] *= gelu_slope(x[e]);
        }
    }
    if (p.reduce) {
        if (COUNT == 4 && full && p.vec_c) {
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(c),
                         "f"(v[0]), "f"(v[COUNT > 1 ? 1 : 0]),
                         "f"(v[COUNT > 2 ? 2 : 0]), "f"(v[COUNT > 3 ? 3 : 0])
                         : "memory");
            return;
        }
#pragma unroll
        for (int e = 0; e < COUNT; ++e) {
            if (col + e < p.n) {
                atomicAdd(c + e, v[e]);
            }
        }
        return;
    }
    if (COUNT == 4 && full && p.vec_c) {
        float4 out = make_float4(v[0], v[COUNT > 1 ? 1 : 0], v[COUNT > 2 ? 2 : 0],
                                 v[COUNT > 3 ? 3 : 0]);
        if (p.accumulate) {
            const float4 old = *reinterpret_cast<const float4 *>(c);
            out.x += old.x; out.y += old.y; out.z += old.z; out.w += old.w;
        }
        *reinterpret_cast<float4 *>(c) = out;
        if (p.gelu_out) {
            out.x = gelu_value(out.x); out.y = gelu_value(out.y);
            out.z = gelu_value(out.z); out.w = gelu_value(out.w);
            *reinterpret_cast<float4 *>(p.gelu_out + (long long)row * p.ldc + col) = out;
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < COUNT; ++e) {
        if (col + e < p.n) {
            const float out = p.accumulate ? c[e] + v[e] : v[e];
            c[e] = out;
            if (p.gelu_out) {
                p.gelu_out[(long long)row * p.ldc + col + e] = gelu_value(out);
            }
        }
    }
}

// One operand's tile, EXTENT output indices (rows of A, columns of B) by KB of
// the reduction, kept as [KB][kPitch] with the output index contiguous, so that
// a thread reads its neighbours with 128-bit loads whatever the storage.
// Operands stored that way already are copied by cp.async; K-contiguous rows
// are fetched into registers two blocks ahead and stored transposed once the
// current block is done (a K-contiguous tile read back along K was measured 1.5
// to 2.5 times slower).
template <int EXTENT, int KB, int THREADS, bool K_CONTIGUOUS>
struct Operand {
    static constexpr int kPitch = EXTENT + (K_CONTIGUOUS ? 4 : 0);
    static constexpr int kFloats = KB * kPitch;
    static constexpr int kChunks = EXTENT * KB / 4;
    static constexpr int kPerThread = (kChunks + THREADS - 1) / THREADS;
    static_assert(kChunks % THREADS == 0 || kPerThread == 1, "whole rounds");

    float4 held[K_CONTIGUOUS ? kPerThread : 1];

    // Starts bringing in the block of the reduction that begins at k0.
    __device__ __forceinline__ void fetch(float *tile, const float *base,
                                          long long pitch, int first, int extent,
                                          int k0, int k_end, bool vec) {
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
            const int chunk = threadIdx.x + i * THREADS;
            if (kChunks < THREADS && chunk >= kChunks) {
                break;
            }
            if (K_CONTIGUOUS) {
                const int r = chunk / (KB / 4), q = chunk % (KB / 4) * 4;
                const int valid = first + r < extent ? min(4, k_end - (k0 + q)) : 0;
                const float *from = base + (long long)(first + r) * pitch + k0 + q;
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (vec && valid == 4) {
                    v = __ldg(reinterpret_cast<const float4 *>(from));
                } else {
                    if (valid > 0) v.x = __ldg(from);
                    if (valid > 1) v.y = __ldg(from + 1);
                    if (valid > 2) v.z = __ldg(from + 2);
                    if (valid > 3) v.w = __ldg(from + 3);
                }
                held[K_CONTIGUOUS ? i : 0] = v;
            } else {
                const int r = chunk / (EXTENT / 4), q = chunk % (EXTENT / 4) * 4;
                const int valid =
                    k0 + r < k_end ? max(0, min(4, extent - (first + q))) : 0;
                copy_chunk(tile + r * kPitch + q,
                           valid ? base + (long long)(k0 + r) * pitch + first + q : base,
                           valid, vec);
            }
        }
    }
    // Puts what fetch() holds where it belongs.
    __device__ __forceinline__ void settle(float *tile) const {
        if (!K_CONTIGUOUS) {
            return;
        }
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
            const int chunk = threadIdx.x + i * THREADS;
            if (kChunks < THREADS && chunk >= kChunks) {
                break;
            }
            const int r = chunk / (KB / 4), q = chunk % (KB / 4) * 4;
            const float4 v = held[K_CONTIGUOUS ? i : 0];
            tile[(q + 0) * kPitch + r] = v.x;
            tile[(q + 1) * kPitch + r] = v.y;
            tile[(q + 2) * kPitch + r] = v.z;
            tile[(q + 3) * kPitch + r] = v.w;
        }
    }
};

// A_K / B_K: the operand's rows have K contiguous (otherwise M / N).
// CLUSTER: blockIdx.z runs over the K slices of one tile, which are the CTAs
// of a cluster and add up through distributed shared memory.
// place: the CTA's tile (x, y) and slice (z) of `slices`.
template <int TM, int TN, int RM, int RN, int KB, bool A_K, bool B_K, bool CLUSTER>
__device__ __forceinline__ void fma_tile(const FmaParams &p, const uint3 place,
                                         const int slices) {
    constexpr int kThreads = TM / RM * (TN / RN);
    constexpr int kLanesX = TN / RN, kLanesY = TM / RM;
    static_assert(kLanesX % 4 == 0 && kLanesY % 8 == 0 && RM % 4 == 0, "warp = 8 x 4 threads");
    using OperandA = Operand<TM, KB, kThreads, A_K>;
    using OperandB = Operand<TN, KB, kThreads, B_K>;
    constexpr int kStage = OperandA::kFloats + OperandB::kFloats;
    constexpr int kGroup = RN < 4 ? RN : 4;   // consecutive columns of a thread
    extern __shared__ __align__(16) float shared[];
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int ty = (warp / (kLanesX / 4)) * 8 + (lane & 7);
    const int tx = (warp % (kLanesX / 4)) * 4 + (lane >> 3);
    const int m0 = int(place.x) * TM;
    const int n0 = int(place.y) * TN;
    const int k_begin = int(place.z) * p.k_per_split;
    const int k_end = min(p.k, k_begin + p.k_per_split);
    const int blocks = k_end > k_begin ? (k_end - k_begin + KB - 1) / KB : 0;

    auto row_of = [&](int i) { return 4 * ty + (i & 3) + (i >> 2) * (4 * kLanesY); };
    auto col_of = [&](int j) {
        return kGroup * tx + j % kGroup + (j / kGroup) * (kGroup * kLanesX);
    };
    OperandA a;
    OperandB b;
    auto fetch = [&](int block) {
        float *stage = shared + (block % kStages) * kStage;
        a.fetch(stage, p.a, p.lda, m0, p.m, k_begin + block * KB, k_end, p.vec_a);
        b.fetch(stage + OperandA::kFloats, p.b, p.ldb, n0, p.n, k_begin + block * KB,
                k_end, p.vec_b);
    };
    auto settle = [&](int block) {
        float *stage = shared + (block % kStages) * kStage;
        a.settle(stage);
        b.settle(stage + OperandA::kFloats);
    };

    unsigned long long acc[RM][RN / 2];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) {
            acc[i][j] = 0ull;
        }
    }
    grid_dependency_wait();
    grid_dependency_release();
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < blocks) {
            fetch(s);
            settle(s);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int block = 0; block < blocks; ++block) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();
        // The stage filled now was read in the previous round.
        const bool more = block + kStages - 1 < blocks;
        if (more) {
            fetch(block + kStages - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *a_tile = shared + (block % kStages) * kStage;
        const float *b_tile = a_tile + OperandA::kFloats;
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            unsigned long long b_pair[RN / 2];
#pragma unroll
            for (int j = 0; j < RN; j += kGroup) {
                const float *from = b_tile + k * OperandB::kPitch + col_of(j);
                if (kGroup == 4) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(from);
                    b_pair[j / 2] = v.x;
                    b_pair[(j / 2 + 1) % (RN / 2)] = v.y;
                } else {
                    b_pair[j / 2] = *reinterpret_cast<const unsigned long long *>(from);
                }
            }
#pragma unroll
            for (int i = 0; i < RM; i += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(
                    a_tile + k * OperandA::kPitch + row_of(i));
                const float a_col[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const unsigned long long twice = pack2(a_col[e], a_col[e]);
#pragma unroll
                    for (int j = 0; j < RN / 2; ++j) {
                        fma2(acc[i + e][j], twice, b_pair[j]);
                    }
                }
            }
        }
        if (more) {
            settle(block + kStages - 1);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    __shared__ float column_sums[TN];
    if (p.partials) {
        for (int c = tid; c < TN; c += kThreads) {
            column_sums[c] = 0.0f;
        }
    }
    int partial_row = place.x;
    if (CLUSTER && slices > 1) {
        // Every CTA of the cluster leaves its partial tile in its own shared
        // memory and finishes an equal share of the rows.
        constexpr int kPitch = TN + 4;
        __syncthreads();   // the stages are free
#pragma unroll
        for (int i = 0; i < RM; ++i) {
#pragma unroll
            for (int j = 0; j < RN / 2; ++j) {
                *reinterpret_cast<unsigned long long *>(
                    shared + row_of(i) * kPitch + col_of(2 * j)) = acc[i][j];
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int rank = place.z;
        const int rows = TM / slices;
        partial_row = place.x * slices + rank;
        for (int e = tid; e < rows * TN; e += kThreads) {
            const int r = rank * rows + e / TN, c = e % TN;
            const uint32_t mine = shared_address(shared + r * kPitch + c);
            float v[1] = {0.0f};
            for (int peer = 0; peer < slices; ++peer) {
                uint32_t theirs;
                float x;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(theirs)
                             : "r"(mine), "r"(peer));
                asm volatile("ld.shared::cluster.f32 %0, [%1];"
                             : "=f"(x)
                             : "r"(theirs)
                             : "memory");
                v[0] += x;
            }
            finish<1>(p, m0 + r, n0 + c, v);
            if (p.partials) {
                atomicAdd(&column_sums[c], v[0]);
            }
        }
        // No CTA leaves while a peer may still read its tile.
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
        float sums[RN];
#pragma unroll
        for (int j = 0; j < RN; ++j) {
            sums[j] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < RM; ++i) {
#pragma unroll
            for (int j = 0; j < RN; j += kGroup) {
                float v[kGroup];
#pragma unroll
                for (int e = 0; e < kGroup; e += 2) {
                    unpack2(acc[i][(j + e) / 2], v[e], v[e + 1]);
                }
                finish<kGroup>(p, m0 + row_of(i), n0 + col_of(j), v);
#pragma unroll
                for (int e = 0; e < kGroup; ++e) {
                    sums[j + e] += v[e];
                }
            }
        }
        if (p.partials) {
#pragma unroll
            for (int j = 0; j < RN; ++j) {
                float s = sums[j];
                s += __shfl_xor_sync(kFullMask, s, 1);
                s += __shfl_xor_sync(kFullMask, s, 2);
                s += __shfl_xor_sync(kFullMask, s, 4);
                if ((lane & 7) == 0) {
                    atomicAdd(&column_sums[col_of(j)], s);
                }
            }
        }
    }
    if (p.partials) {
        __syncthreads();
        float *out = p.partials + (long long)(partial_row % p.partial_rows) * p.n + n0;
        for (int c = tid; c < TN && n0 + c < p.n; c += kThreads) {
            if (p.partials_shared) {
                atomicAdd(out + c, column_sums[c]);
            } else {
                out[c] = column_sums[c];
            }
        }
    }
}

template <int TM, int TN, int RM, int RN, int KB, int CTAS, bool A_K, bool B_K,
          bool CLUSTER>
__global__ void __launch_bounds__(TM / RM * (TN / RN), CTAS)
fma_kernel(const FmaParams p) {
    fma_tile<TM, TN, RM, RN, KB, A_K, B_K, CLUSTER>(p, blockIdx, int(gridDim.z));
}

// The smallest tile, with which latency-sized products run.
constexpr int kSmallRows = 32, kSmallCols = 32, kSmallRm = 4, kSmallRn = 2, kSmallKb = 32;

// The two gradients of a small linear layer side by side, each as a launch of its own
// would compute it.  Tiles of the input gradient first (p, x_tiles x y_tiles of them,
// their slices along z a cluster), then the weight gradient's (q) tiles and slices,
// numbered through.
__global__ void __launch_bounds__(kSmallRows / kSmallRm * (kSmallCols / kSmallRn), 4)
fma_pair_kernel(const FmaParams p, const FmaParams q, const unsigned x_tiles,
                const unsigned y_tiles, const unsigned x_weight, const unsigned y_weight,
                const unsigned weight_slices) {
    const unsigned tiles = x_tiles * y_tiles;
    if (blockIdx.x < tiles) {
        fma_tile<kSmallRows, kSmallCols, kSmallRm, kSmallRn, kSmallKb, true, true, true>(
            p, make_uint3(blockIdx.x % x_tiles, blockIdx.x / x_tiles, blockIdx.z),
            int(gridDim.z));
        return;
    }
    const unsigned index = (blockIdx.x - tiles) * gridDim.z + blockIdx.z;
    const unsigned weight_tiles = x_weight * y_weight;
    if (index >= weight_tiles * weight_slices) {
        grid_dependency_wait();
        return;
    }
    const unsigned tile = index % weight_tiles;
    fma_tile<kSmallRows, kSmallCols, kSmallRm, kSmallRn, kSmallKb, false, false, false>(
        q, make_uint3(tile % x_weight, tile / x_weight, index / weight_tiles), 1);
}

enum class Form { Forward, InputGradient, WeightGradient };

template <int TM, int TN, int RM, int RN, int KB, int CTAS, bool A_K, bool B_K,
          bool CLUSTER>
cudaError_t launch_form(const FmaParams &p, int slices, cudaStream_t stream) {
    constexpr int kThreads = TM / RM * (TN / RN);
    constexpr size_t kRing = size_t(kStages) * sizeof(float) *
                             (Operand<TM, KB, kThreads, A_K>::kFloats +
                              Operand<TN, KB, kThreads, B_K>::kFloats);
    constexpr size_t kPartial = CLUSTER ? size_t(TM) * (TN + 4) * sizeof(float) : 0;
    constexpr size_t kBytes = kRing > kPartial ? kRing : kPartial;
    const auto kernel = fma_kernel<TM, TN, RM, RN, KB, CTAS, A_K, B_K, CLUSTER>;
    if (kBytes > 40 * 1024) {   // (some static shared memory comes on top)
        static SharedMemoryLimit limit;
        if (!limit.raise(reinterpret_cast<const void *>(kernel), int(kBytes))) {
            return cudaErrorInvalidConfiguration;
        }
    }
    const dim3 grid((p.m + TM - 1) / TM, (p.n + TN - 1) / TN, slices);
    return launch_chained_cluster(kernel, grid, kThreads, kBytes,
                                  CLUSTER ? unsigned(slices) : 1u, true, stream, p);
}

// CLUSTER: the slices of the forward product and of the input gradient.  Those
// of a weight gradient are independent.
template <int TM, int TN, int RM, int RN, int KB, int CTAS, bool CLUSTER = false>
cudaError_t launch_tile(const FmaParams &p, Form form, int slices, cudaStream_t stream) {
    switch (form) {
    case Form::Forward:
        return launch_form<TM, TN, RM, RN, KB, CTAS, true, false, CLUSTER>(p, slices,
                                                                          stream);
    case Form::InputGradient:
        return launch_form<TM, TN, RM, RN, KB, CTAS, true, true, CLUSTER>(p, slices,
                                                                         stream);
    default:
        return launch_form<TM, TN, RM, RN, KB, CTAS, false, false, false>(p, slices,
                                                                         stream);
    }
}

// The tiles, with what the choice between them rests on: multiply-adds per
// clock of an SM that is full of them and of a lone CTA, and the fixed part of
// a launch (first trip to memory, epilogue) in clocks.
struct Tile {
    int rows, cols;
    double full, alone, fixed;
};
constexpr Tile kTiles[] = {{128, 128, 85.0, 78.0, 6000.0},
                           {64, 128, 82.0, 73.0, 8000.0},
                           {64, 64, 62.0, 52.0, 3800.0},
                           {64, 32, 50.0, 41.0, 3700.0},
                           {32, 32, 35.0, 28.0, 3500.0}};
constexpr int kTileCount = int(sizeof(kTiles) / sizeof(kTiles[0]));
constexpr int kSmallestTile = kTileCount - 1;

// A way to cut a product: which tile, and how many slices of K.
struct FmaPlan {
    int tile = 0;
    int slices = 1;
    bool cluster = false;   // the slices of a tile meet in a cluster, else in C
    double clocks = 0.0;
};

int slice_length(int k, int slices) {
    return ((k + slices - 1) / slices + 15) / 16 * 16;
}

// Slices that 64 x 64 tiles take to make up two CTAs per SM, of 128 terms at least.
int reference_slices(int m, int n, int k) {
    const long long tiles = ((m + 63LL) / 64) * ((n + 63LL) / 64);
    const long long two = 2LL * device_sm_count();
    const int wanted = int(std::min((two + tiles - 1) / tiles, (k + 127LL) / 128));
    const int each = slice_length(k, std::max(1, wanted));
    return each ? (k + each - 1) / each : 1;
}

// Additions that follow one another in a sum: a slice's terms, then the slices.
long long additions(int k, int slices) {
    return std::min(k, slice_length(k, slices)) + (long long)slices;
}

// Picks the plan with the smallest estimate: the longer of what one CTA takes
// by itself and what an SM takes for all the CTAs it gets, plus the fixed part
// and what combining slices costs.  reduce: C is added to, so that slices may
// meet there (weight gradients); cluster: the smallest tile's slices meet in a
// cluster (forward products and input gradients).  Plans whose sums take more
// than `longest` additions in a row are left out.
FmaPlan plan_product(int m, int n, int k, bool reduce, bool cluster, long long longest) {
    const double sms = double(device_sm_count());
    const int reference = reference_slices(m, n, k);
    FmaPlan best;
    for (int t = 0; t < kTileCount; ++t) {
        const Tile &tile = kTiles[t];
        const double count = double((m + tile.rows - 1) / tile.rows) *
                             double((n + tile.cols - 1) / tile.cols);
        // Slices that meet in C: powers of two, as many as give every SM one to
        // eight CTAs, and the reference; in a cluster 2, 4 or 8.
        const bool in_cluster = cluster && t == kSmallestTile;
        const int choices = in_cluster ? 4 : (reduce ? 17 : 1);
        for (int choice = 0; choice < choices; ++choice) {
            const int slices = choice < 8 ? 1 << choice
                : (choice == 16 ? reference
                                : std::max(1, int((choice - 7) * sms / count)));
            const int per_slice = slice_length(k, slices);
            if (slices > 1 && per_slice < (in_cluster ? 16 : 32)) {
                continue;
            }
            if (additions(k, slices) > longest) {
                continue;
            }
            const double work = double(tile.rows) * tile.cols * per_slice;
            const double per_sm = double((long long)((count * slices + sms - 1) / sms));
            double clocks = std::max(work / tile.alone, per_sm * work / tile.full) +
                            tile.fixed;
            if (slices > 1) {
                clocks += in_cluster ? 2200.0 : double(m) * n * slices / 1500.0;
            }
            if (best.clocks == 0.0 || clocks < best.clocks) {
                best.tile = t;
                best.slices = slices;
                best.cluster = in_cluster;
                best.clocks = clocks;
            }
        }
    }
    return best;
}

// The plan of a product that adds to C.  Its slices bound the rounding error, which
// grows with the square root of the additions in a row: no more of them than the
// reference takes.  (In one chain of 288 the input gradient [4329,288] x [288,96] had an
// error of 3.0e-7, in slices of 96 1.8e-7.)  An input gradient is cut that way only
// where its ordinary plan is longer.
FmaPlan plan_addition(int m, int n, int k, bool input_gradient) {
    const long long longest = additions(k, reference_slices(m, n, k));
    FmaPlan plan = plan_product(m, n, k, !input_gradient, input_gradient, LLONG_MAX);
    if (additions(k, plan.slices) > longest) {
        plan = plan_product(m, n, k, true, input_gradient, longest);
    }
    return plan;
}

bool aligned16(const void *pointer) {
    return (reinterpret_cast<uintptr_t>(pointer) & 15) == 0;
}

}  // namespace

unsigned long long g_fma_products = 0;

namespace {

// A product with its plan, ready to be launched.
struct FmaLaunch {
    FmaParams p;
    Form form;
    int tile, slices;
};

Form form_of(const FmaGemm &g) {
    return g.a_k ? (g.b_k ? Form::InputGradient : Form::Forward) : Form::WeightGradient;
}

// K slices may only add into C.
bool adds_to_c(const FmaGemm &g) {
    return g.accumulate && form_of(g) != Form::Forward;
}

FmaPlan plan_of(const FmaGemm &g) {
    return adds_to_c(g)
        ? plan_addition(g.m, g.n, g.k, form_of(g) == Form::InputGradient)
        : plan_product(g.m, g.n, g.k, false, true, LLONG_MAX);
}

bool prepare(const FmaGemm &g, const FmaPlan &plan, cudaStream_t stream, int *partial_rows,
             FmaLaunch *out) {
    FmaParams &p = out->p;
    p = FmaParams{};
    p.a = g.a;
    p.b = g.b;
    p.c = g.c;
    p.bias = g.bias;
    p.gelu_out = g.gelu_out;
    p.gelu_input = g.gelu_input;
    p.m = g.m;
    p.n = g.n;
    p.k = g.k;
    p.lda = g.lda;
    p.ldb = g.ldb;
    p.ldc = g.ldc;
    p.vec_a = g.lda % 4 == 0 && aligned16(g.a);
    p.vec_b = g.ldb % 4 == 0 && aligned16(g.b);
    p.vec_c = g.ldc % 4 == 0 && aligned16(g.c) &&
              (!g.gelu_out || aligned16(g.gelu_out)) &&
              (!g.gelu_input || aligned16(g.gelu_input));
    p.accumulate = g.accumulate ? 1 : 0;
    const Form form = form_of(g);
    if (form == Form::WeightGradient && (!g.accumulate || g.b_k)) {
        return false;   // no caller has this form
    }
    const bool adds = adds_to_c(g);
    int slices = plan.slices;
    p.k_per_split = slice_length(g.k, slices);
    if (adds && !plan.cluster && slices > 1) {
        slices = (g.k + p.k_per_split - 1) / p.k_per_split;
        p.reduce = slices > 1 ? 1 : 0;
    }
    if (g.column_partials) {
        const int rows =
            (g.m + kTiles[plan.tile].rows - 1) / kTiles[plan.tile].rows * slices;
        p.partials = g.column_partials;
        p.partial_rows = std::min(rows, g.partial_row_limit);
        p.partials_shared = rows > p.partial_rows ? 1 : 0;
        if (p.partials_shared &&
            cudaMemsetAsync(p.partials, 0, size_t(p.partial_rows) * g.n * sizeof(float),
                            stream) != cudaSuccess) {
            return false;
        }
        if (partial_rows) {
            *partial_rows = p.partial_rows;
        }
    }
    out->form = form;
    out->tile = plan.tile;
    out->slices = slices;
    return true;
}

}  // namespace

int launch_gemm_fma(const FmaGemm &g, cudaStream_t stream, int *partial_rows) {
    if (launch_gemm_thin(g, stream)) {
        ++g_fma_products;
        return 0;
    }
    // (Slices in a cluster keep sums of positive terms closer than anything else does.)
    const FmaPlan plan = plan_of(g);
    if (plan.clocks > 15000.0 && !(plan.cluster && plan.slices > 1)) {
        const double error =
            fma_error(std::min(g.k, slice_length(g.k, plan.slices)), plan.slices);
        if (gemm_split_clocks(g, error) < plan.clocks &&
            launch_gemm_split(g, error, stream, partial_rows)) {
            ++g_fma_products;
            return 0;
        }
    }
    FmaLaunch launch;
    if (!prepare(g, plan, stream, partial_rows, &launch)) {
        return -1;
    }
    const FmaParams &p = launch.p;
    const Form form = launch.form;
    const int slices = launch.slices;
    cudaError_t status;
    switch (launch.tile) {
    case 0:
        status = launch_tile<128, 128, 8, 8, 16, 2>(p, form, slices, stream);
        break;
    case 1:
        status = launch_tile<64, 128, 8, 8, 16, 3>(p, form, slices, stream);
        break;
    case 2:
        status = launch_tile<64, 64, 4, 4, 16, 3>(p, form, slices, stream);
        break;
    case 3:
        status = launch_tile<64, 32, 4, 4, 32, 4>(p, form, slices, stream);
        break;
    default:
        status = launch_tile<kSmallRows, kSmallCols, kSmallRm, kSmallRn, kSmallKb, 4, true>(
            p, form, slices, stream);
    }
    if (status != cudaSuccess) {
        return -1;
    }
    ++g_fma_products;
    ++g_kernel_launches;
    return 0;
}

bool gemm_fma_pairs(int m, int k, int n) {
    if (m >= 8192) {
        return false;   // from here on thin products have kernels of their own
    }
    const FmaPlan input = plan_product(m, k, n, false, true, LLONG_MAX);
    const FmaPlan weight = plan_addition(k, n, m, false);
    return input.tile == kSmallestTile && weight.tile == kSmallestTile;
}

int launch_gemm_fma_pair(const FmaGemm &input, const FmaGemm &weight, cudaStream_t stream,
                         int *partial_rows) {
    FmaLaunch first, second;
    if (input.accumulate || !gemm_fma_pairs(input.m, input.n, input.k) ||
        !prepare(input, plan_of(input), stream, partial_rows, &first) ||
        !prepare(weight, plan_of(weight), stream, nullptr, &second) ||
        first.form != Form::InputGradient || second.form != Form::WeightGradient ||
        first.tile != kSmallestTile || second.tile != kSmallestTile) {
        return -1;
    }
    constexpr int kPairThreads = kSmallRows / kSmallRm * (kSmallCols / kSmallRn);
    constexpr size_t kBytes =
        size_t(kStages) * sizeof(float) * 2 *
        Operand<kSmallRows, kSmallKb, kPairThreads, true>::kFloats;
    static_assert(kSmallRows == kSmallCols &&
                      kBytes >= size_t(kSmallRows) * (kSmallCols + 4) * sizeof(float) &&
                      kBytes <= 40 * 1024,
                  "one ring for both forms and for the partial tiles");
    const unsigned x = (first.p.m + kSmallRows - 1) / kSmallRows;
    const unsigned y = (first.p.n + kSmallCols - 1) / kSmallCols;
    const unsigned xw = (second.p.m + kSmallRows - 1) / kSmallRows;
    const unsigned yw = (second.p.n + kSmallCols - 1) / kSmallCols;
    const unsigned depth = unsigned(first.slices);
    const unsigned weight_blocks = (xw * yw * unsigned(second.slices) + depth - 1) / depth;
    const dim3 grid(x * y + weight_blocks, 1, depth);
    if (launch_chained_cluster(fma_pair_kernel, grid, kPairThreads, kBytes, depth, true,
                               stream, first.p, second.p, x, y, xw, yw,
                               unsigned(second.slices)) != cudaSuccess) {
        return -1;
    }
    g_fma_products += 2;
    ++g_kernel_launches;
    return 0;
}

}  // namespace vitb200
