// FP32 products with one extent of at most 16 and a long one: the patch
// projections of small patches (4 to 16 pixels) and their gradients.
//
// They do two to sixteen multiply-adds per float of the one large matrix, so the
// memory rate bounds them, and a tiled product spends its time on staging
// operands instead.  Here the thin operand lives in registers (a float4 column
// group for each of its up to 16 rows) and the large matrix streams past once,
// in 128-bit accesses with several rows in flight:
//
//   forward          Y[m,n] = X[m,k] W[k,n] (+ bias)   k thin: writes Y
//   input gradient   C[m,n] (+)= dY[m,k] W[n,k]^T      n thin: reads dY, a warp
//                    per row, the n dot products reduced while they are
//                    scattered over the lanes
//   weight gradient  C[m,n] += X[k,m]^T dY[k,n]        m thin: reads dY, sums in
//                    registers, one vector reduction per block and column group
//
// Measured against the tiled FMA kernel, 4 features: [100352,4]x[4,256] forward
// 67 -> 18.7 us (104 MB: 16 at the copy rate), input gradient 61 -> 22.8, weight
// gradient 76 -> 21.9; [65536,4]x[4,384] 67 -> 18.3, 59 -> 24.7, 79 -> 20.9.
#include "device_util.cuh"
#include "gemm.h"
#include "kernels.h"

#include <algorithm>
#include <cstdint>

namespace vitb200 {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxGroups = kThreads;       // float4 column groups of the wide extent
// The weight gradient's blocks, one per SM: every block is one more addition in a row
// for each of its sums.  With up to 444 blocks of 256 threads [10007,16]^T [10007,128]
// had an error of 3.2e-7 (2-norm against 64 bits; 2.7e-7 on the tiles the kernel stands
// in for), this way 2.3e-7, and [65536,4]^T [65536,384] 4.0e-7 (6.7e-7), now 2.7e-7.
// The 128 registers leave room for no more threads, so that one block fills the SM and
// no second, half-empty turn of blocks follows: 17.3 -> 13.3 us and 30.3 -> 20.9.
constexpr int kWeightThreads = 512;
// Below this many rows the tiles of the general kernel are as fast.
constexpr int kMinimumRows = 8192;

__device__ __forceinline__ void fma4(float4 &sum, float x, const float4 &w) {
    sum.x = fmaf(x, w.x, sum.x);
    sum.y = fmaf(x, w.y, sum.y);
    sum.z = fmaf(x, w.z, sum.z);
    sum.w = fmaf(x, w.w, sum.w);
}

__device__ __forceinline__ void add(float4 &sum, const float4 &v) {
    sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
}

// The first k of KM values; zeros beyond.
template <int KM>
__device__ __forceinline__ void load_thin(const float *row, int k, bool vector,
                                          float (&x)[KM]) {
    if (vector) {
#pragma unroll
        for (int i = 0; i < KM / 4; ++i) {
            const float4 v = 4 * i < k ? __ldg(reinterpret_cast<const float4 *>(row) + i)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < KM; ++i) {
            x[i] = i < k ? __ldg(row + i) : 0.0f;
        }
    }
}

template <int KM>
__global__ void __launch_bounds__(kThreads)
thin_forward_kernel(const float *__restrict__ a, const float *__restrict__ b,
                    const float *__restrict__ bias, float *__restrict__ c,
                    unsigned m, int k, unsigned groups, size_t lda, size_t ldb,
                    size_t ldc, bool vector) {
    grid_dependency_wait();
    grid_dependency_release();
    constexpr int R = KM <= 4 ? 4 : 2;     // rows in flight
    const unsigned rows = kThreads / groups;
    const unsigned slice = threadIdx.x / groups, group = threadIdx.x % groups;
    if (slice >= rows) {
        return;
    }
    float4 w[KM], shift = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < KM; ++i) {
        w[i] = i < k ? __ldg(reinterpret_cast<const float4 *>(b + i * ldb) + group)
                     : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (bias) {
        shift = make_float4(__ldg(bias + 4 * group), __ldg(bias + 4 * group + 1),
                            __ldg(bias + 4 * group + 2), __ldg(bias + 4 * group + 3));
    }
    const unsigned stride = gridDim.x * rows;
    for (unsigned first = blockIdx.x * rows + slice; first < m; first += stride * R) {
        float x[R][KM];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = first + r * stride;
            load_thin<KM>(a + size_t(min(row, m - 1)) * lda, k, vector, x[r]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = first + r * stride;
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < KM; ++i) {
                fma4(sum, x[r][i], w[i]);
            }
            sum.x += shift.x; sum.y += shift.y; sum.z += shift.z; sum.w += shift.w;
            if (row < m) {
                reinterpret_cast<float4 *>(c + row * ldc)[group] = sum;
            }
        }
    }
}

template <int NM, int NV>
__global__ void __launch_bounds__(kThreads)
thin_input_gradient_kernel(const float *__restrict__ a, const float *__restrict__ b,
                           float *c, unsigned m, int n, unsigned groups, size_t lda,
                           size_t ldb, size_t ldc, bool add) {
    grid_dependency_wait();
    grid_dependency_release();
    constexpr int R = NV * NM <= 8 ? 4 : 2;
    constexpr int kLanes = 32 / NM;        // lanes that share a value at the end
    const unsigned lane = threadIdx.x & 31;
    float4 w[NM][NV];
#pragma unroll
    for (int i = 0; i < NM; ++i) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const unsigned group = 32 * j + lane;
            w[i][j] = i < n && group < groups
                ? __ldg(reinterpret_cast<const float4 *>(b + i * ldb) + group)
                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    const unsigned stride = gridDim.x * (kThreads / 32);
    const unsigned warp = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    for (unsigned first = warp; first < m; first += stride * R) {
        float4 v[R][NV];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const size_t row = min(first + r * stride, m - 1);
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const unsigned group = 32 * j + lane;
                v[r][j] = group < groups
                    ? __ldg(reinterpret_cast<const float4 *>(a + row * lda) + group)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = first + r * stride;
            float sums[NM];
#pragma unroll
            for (int i = 0; i < NM; ++i) {
                sums[i] = 0.0f;
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    sums[i] += (v[r][j].x * w[i][j].x + v[r][j].y * w[i][j].y) +
                               (v[r][j].z * w[i][j].z + v[r][j].w * w[i][j].w);
                }
            }
            // Halve the values a lane is left with until it has one: value
            // lane / kLanes.
            int count = NM / 2;
#pragma unroll
            for (int distance = 16; distance >= kLanes; distance /= 2, count /= 2) {
                const bool upper = (lane & distance) != 0;
#pragma unroll
                for (int i = 0; i < NM / 2; ++i) {
                    if (i < count) {
                        const float low = sums[i], high = sums[i + count];
                        sums[i] = (upper ? high : low) +
                                  __shfl_xor_sync(kFullMask, upper ? low : high, distance);
                    }
                }
            }
#pragma unroll
            for (int distance = kLanes / 2; distance > 0; distance /= 2) {
                sums[0] += __shfl_xor_sync(kFullMask, sums[0], distance);
            }
            const int column = lane / kLanes;
            if (lane % kLanes == 0 && column < n && row < m) {
                float *target = c + row * ldc + column;
                *target = (add ? *target : 0.0f) + sums[0];
            }
        }
    }
}

template <int MM>
__global__ void __launch_bounds__(kWeightThreads, 1)
thin_weight_gradient_kernel(const float *__restrict__ a, const float *__restrict__ b,
                            float *c, int m, unsigned k, unsigned groups, size_t lda,
                            size_t ldb, size_t ldc, bool vector) {
    grid_dependency_wait();
    grid_dependency_release();
    constexpr int R = MM <= 4 ? 8 : (MM <= 8 ? 4 : 2);
    __shared__ float4 fold[kWeightThreads], folded[kWeightThreads];
    const unsigned slices = kWeightThreads / groups;
    const unsigned slice = threadIdx.x / groups, group = threadIdx.x % groups;
    const bool live = slice < slices;
    float4 sums[MM];
#pragma unroll
    for (int i = 0; i < MM; ++i) {
        sums[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const unsigned stride = gridDim.x * slices;
    for (unsigned first = blockIdx.x * slices + slice; live && first < k;
         first += stride * R) {
        float4 v[R];
        float x[R][MM];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned row = first + r * stride;
            load_thin<MM>(a + row * lda, row < k ? m : 0, vector, x[r]);
            v[r] = row < k ? __ldg(reinterpret_cast<const float4 *>(b + row * ldb) + group)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int i = 0; i < MM; ++i) {
                fma4(sums[i], x[r][i], v[r]);
            }
        }
    }
    // The block's slices together, a square root of them at a time, then one
    // reduction into C per column group.
    unsigned lanes = 1;
    while (lanes * lanes < slices) {
        ++lanes;
    }
#pragma unroll
    for (int i = 0; i < MM; ++i) {
        if (i < m) {
            fold[threadIdx.x] = sums[i];
            __syncthreads();
            if (slice < lanes) {
                float4 total = fold[threadIdx.x];
                for (unsigned s = slice + lanes; s < slices; s += lanes) {
                    add(total, fold[s * groups + group]);
                }
                folded[threadIdx.x] = total;
            }
            __syncthreads();
            if (slice == 0) {
                float4 total = folded[group];
                for (unsigned s = 1; s < lanes; ++s) {
                    add(total, folded[s * groups + group]);
                }
                asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::
                                 "l"(c + i * ldc + 4 * group),
                             "f"(total.x), "f"(total.y), "f"(total.z), "f"(total.w)
                             : "memory");
            }
        }
    }
}

bool aligned(const void *pointer) {
    return (reinterpret_cast<uintptr_t>(pointer) & 15) == 0;
}

bool fits(long long ld) {
    return ld % 4 == 0;
}

// A grid of `per_sm` blocks on each multiprocessor, or what the rows need.
unsigned row_blocks(size_t rows, size_t rows_per_block, unsigned per_sm) {
    const size_t wanted = (rows + rows_per_block - 1) / rows_per_block;
    return unsigned(std::min<size_t>(wanted, size_t(device_sm_count()) * per_sm));
}

}  // namespace

bool launch_gemm_thin(const FmaGemm &g, cudaStream_t stream) {
    if (g.gelu_out || g.gelu_input || g.column_partials) {
        return false;
    }
    const size_t lda = g.lda, ldb = g.ldb, ldc = g.ldc;
    cudaError_t status = cudaErrorInvalidValue;
    if (g.a_k && !g.b_k) {
        // Forward: B and C have the wide extent.
        const unsigned groups = g.n / 4;
        if (g.k > 16 || g.m < kMinimumRows || g.n % 4 || !groups ||
            groups > kMaxGroups || g.accumulate || !fits(ldb) || !fits(ldc) ||
            !aligned(g.b) || !aligned(g.c)) {
            return false;
        }
        const bool vector = g.k % 4 == 0 && fits(lda) && aligned(g.a);
        const size_t bytes = 4 * size_t(g.m) * (g.n + g.k);
        const unsigned grid = row_blocks(g.m, 4 * (kThreads / groups), 4);
        auto launch = [&](auto kernel) {
            status = launch_streamed(kernel, grid, kThreads, stream, bytes, g.a, g.b,
                                     g.bias, g.c, unsigned(g.m), g.k, groups, lda,
                                     ldb, ldc, vector);
        };
        if (g.k <= 4) {
            launch(thin_forward_kernel<4>);
        } else if (g.k <= 8) {
            launch(thin_forward_kernel<8>);
        } else if (g.k <= 12) {
            launch(thin_forward_kernel<12>);
        } else {
            launch(thin_forward_kernel<16>);
        }
    } else if (g.a_k && g.b_k) {
        // Input gradient: A and B have the wide extent, the reduction.
        const unsigned groups = g.k / 4;
        const unsigned vectors = (groups + 31) / 32;
        if (g.n > 16 || g.m < kMinimumRows || g.k % 4 || !groups || g.bias ||
            !fits(lda) || !fits(ldb) || !aligned(g.a) || !aligned(g.b)) {
            return false;
        }
        const size_t bytes = 4 * size_t(g.m) * (g.n + g.k);
        const unsigned grid = row_blocks(g.m, 2 * (kThreads / 32), 4);
        auto launch = [&](auto kernel) {
            status = launch_streamed(kernel, grid, kThreads, stream, bytes, g.a, g.b,
                                     g.c, unsigned(g.m), g.n, groups, lda, ldb, ldc,
                                     g.accumulate);
        };
        // (The thin operand takes 4 NM NV registers, at most 64.)
        if (g.n <= 4 && vectors <= 1) {
            launch(thin_input_gradient_kernel<4, 1>);
        } else if (g.n <= 4 && vectors <= 2) {
            launch(thin_input_gradient_kernel<4, 2>);
        } else if (g.n <= 4 && vectors <= 4) {
            launch(thin_input_gradient_kernel<4, 4>);
        } else if (g.n <= 8 && vectors <= 2) {
            launch(thin_input_gradient_kernel<8, 2>);
        } else if (g.n <= 16 && vectors <= 1) {
            launch(thin_input_gradient_kernel<16, 1>);
        } else {
            return false;
        }
    } else if (!g.a_k && !g.b_k) {
        // Weight gradient: B and C have the wide extent, the reduction is long.
        const unsigned groups = g.n / 4;
        if (g.m > 16 || g.k < kMinimumRows || g.n % 4 || !groups ||
            groups > kMaxGroups || !g.accumulate || g.bias || !fits(ldb) ||
            !fits(ldc) || !aligned(g.b) || !aligned(g.c)) {
            return false;
        }
        const bool vector = g.m % 4 == 0 && fits(lda) && aligned(g.a);
        const size_t bytes = 4 * size_t(g.k) * (g.n + g.m);
        const unsigned grid = row_blocks(g.k, 4 * (kWeightThreads / groups), 1);
        auto launch = [&](auto kernel) {
            status = launch_streamed(kernel, grid, kWeightThreads, stream, bytes, g.a, g.b,
                                     g.c, g.m, unsigned(g.k), groups, lda, ldb, ldc,
                                     vector);
        };
        if (g.m <= 4) {
            launch(thin_weight_gradient_kernel<4>);
        } else if (g.m <= 8) {
            launch(thin_weight_gradient_kernel<8>);
        } else if (g.m <= 12) {
            launch(thin_weight_gradient_kernel<12>);
        } else {
            launch(thin_weight_gradient_kernel<16>);
        }
    } else {
        return false;
    }
    if (status != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    ++g_kernel_launches;
    return true;
}

}  // namespace vitb200
