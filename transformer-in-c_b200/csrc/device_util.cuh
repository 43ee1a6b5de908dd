// Small device helpers shared by the kernel files.
#pragma once

#include <cstddef>
#include <cstdlib>
#include <utility>
#include <cuda_runtime.h>

namespace vitb200 {

constexpr unsigned kStreamThreads = 256;
constexpr unsigned kSmCount = 148;         // B200: 2 dies x 74 SMs
constexpr unsigned kStreamBlocksPerSm = 8; // 2048 threads / 256
constexpr unsigned kFullMask = 0xffffffffu;

// Multiprocessors of the current device, asked once (148 on a B200, which is
// also the answer when the query fails).  Persistent grids are sized by it.
inline unsigned device_sm_count() {
    static const unsigned count = []() -> unsigned {
        int device = 0, value = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device) !=
                cudaSuccess ||
            value <= 0) {
            cudaGetLastError();
            return kSmCount;
        }
        return unsigned(value);
    }();
    return count;
}

// Grid for a streaming kernel over `items` work items: enough blocks to cover
// them once, capped at one full wave of resident blocks.
inline unsigned stream_grid(size_t items) {
    const size_t wanted = (items + kStreamThreads - 1) / kStreamThreads;
    const size_t wave = size_t(device_sm_count()) * kStreamBlocksPerSm;
    return static_cast<unsigned>(wanted < 1 ? 1 : (wanted < wave ? wanted : wave));
}

// ---------------------------------------------------------------------------
// Chained launches (programmatic dependent launch).  A kernel launched through
// launch_chained may be scheduled while its predecessor in the stream is still
// running: its blocks become resident as the predecessor's leave, run whatever
// does not touch global memory, and park in grid_dependency_wait() until the
// predecessor has completed and its writes are visible.  That takes the launch
// latency and the block set-up out of the gap between two dependent kernels.
//
// Rules for a kernel launched this way: every thread calls
// grid_dependency_wait() before its first access to global memory and before it
// can return (a grid whose blocks left without waiting would count as complete
// while its predecessors still run, and its successor's wait would pass too
// early).  grid_dependency_release() right after it lets the successor's
// blocks become resident from then on; they park in their own wait.
__device__ __forceinline__ void grid_dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void grid_dependency_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// VITB200_CHAINED_LAUNCHES=0 turns the attribute off (plain stream order).
inline bool chained_launches_enabled() {
    static const bool enabled = []() {
        const char *value = getenv("VITB200_CHAINED_LAUNCHES");
        return !(value && value[0] == '0');
    }();
    return enabled;
}

// cluster_z: CTAs along z that form a cluster (1: none).  chained = false: a
// plain launch.
template <typename... Params, typename... Args>
inline cudaError_t launch_chained_cluster(void (*kernel)(Params...), dim3 grid,
                                          dim3 block, size_t shared_bytes,
                                          unsigned cluster_z, bool chained,
                                          cudaStream_t stream, Args &&...args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = shared_bytes;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed =
        chained && chained_launches_enabled() ? 1 : 0;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = 1;
    attributes[1].val.clusterDim.y = 1;
    attributes[1].val.clusterDim.z = cluster_z;
    config.attrs = attributes;
    config.numAttrs = cluster_z > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid,
                                  dim3 block, size_t shared_bytes,
                                  cudaStream_t stream, Args &&...args) {
    return launch_chained_cluster(kernel, grid, block, shared_bytes, 1, true, stream,
                                  std::forward<Args>(args)...);
}

// Memory-bound kernels: chained up to this many bytes moved.  Beyond, the launch
// latency is nothing beside the kernel, and its blocks, which then move in one by
// one as their predecessor's leave, run slower than blocks dealt out at once: with
// the layer norms of large batches launched the plain way a step takes 1.5 to 2.5 %
// less time (197 tokens 9976 -> 9822 us, 1025 tokens 14116 -> 13939, the wide model
// 12571 -> 12275, prediction of 256 images of 197 tokens 2835 -> 2758), while a
// batch of 32 would lose a quarter without chaining.  Anywhere between 24 and 64 MiB
// measures the same; the evaluation pass of 256 images (26 MB per layer norm)
// stays chained.
constexpr size_t kChainedBytes = size_t(64) << 20;

template <typename... Params, typename... Args>
inline cudaError_t launch_streamed(void (*kernel)(Params...), dim3 grid, dim3 block,
                                   cudaStream_t stream, size_t bytes, Args &&...args) {
    return launch_chained_cluster(kernel, grid, block, 0, 1, bytes < kChainedBytes,
                                  stream, std::forward<Args>(args)...);
}

__device__ __forceinline__ size_t global_thread() {
    return size_t(blockIdx.x) * blockDim.x + threadIdx.x;
}

__device__ __forceinline__ size_t grid_threads() {
    return size_t(gridDim.x) * blockDim.x;
}

// Read-once data: keep it out of L1.
__device__ __forceinline__ float4 ld_stream(const float4 *pointer) {
    return __ldcs(pointer);
}

__device__ __forceinline__ float warp_sum(float value) {
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        value += __shfl_xor_sync(kFullMask, value, offset);
    }
    return value;
}

__device__ __forceinline__ float warp_max(float value) {
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        value = fmaxf(value, __shfl_xor_sync(kFullMask, value, offset));
    }
    return value;
}

// tanh-approximation GELU (reference src/ops.c:944-963); the scale is
// sqrtf(2/pi) rounded to float.
constexpr float kGeluCubic = 0.044715f;
constexpr float kGeluScale = 0.7978845608028654f;

__device__ __forceinline__ float gelu_value(float x) {
    return 0.5f * x * (1.0f + tanhf(kGeluScale * (x + kGeluCubic * x * x * x)));
}

// r = 1 / (1 + exp(2u)) with u = s (x + c x^3), on the fast exponential and
// reciprocal units; tanh(u) = 1 - 2r.
__device__ __forceinline__ float gelu_complement(float x, float x2) {
    constexpr float kScale = 2.0f * 1.4426950408889634f * kGeluScale;
    const float exponent = x * fmaf(kScale * kGeluCubic, x2, kScale);
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(exponent));
    return __fdividef(1.0f, 1.0f + e);
}

// The same function as x (1 - r): absolute error 3.9e-7 at most (5e-8 rms over
// normally distributed values), a fifth of the instructions.  Used where the GELU shares a kernel with a matrix product and
// instruction issue, not memory, is the limit.
__device__ __forceinline__ float gelu_value_fast(float x) {
    return x * (1.0f - gelu_complement(x, x * x));
}

// d/dx of gelu_value (reference src/ops.c:986-992).
__device__ __forceinline__ float gelu_slope(float x) {
    const float t = tanhf(kGeluScale * (x + kGeluCubic * x * x * x));
    return 0.5f * (1.0f + t) +
           0.5f * x * (1.0f - t * t) * kGeluScale *
               (1.0f + 3.0f * kGeluCubic * x * x);
}


// gelu_slope with the same r, for the epilogue of the product that feeds a GELU's
// backward pass (absolute error 2.0e-6 at most, near x = -5; 5e-8 rms over normally
// distributed values):
//   0.5 (1 + t) + 0.5 x (1 - t^2) u' = h + 2 r h x u',  h = 1 - r
// From |x| = 16 on r h is zero and x^2 stays at 256, so that the factor beside it
// is finite for every x whose square is (x u' alone overflows from 1.2e13 on).
__device__ __forceinline__ float gelu_slope_fast(float x) {
    const float x2 = x * x;
    const float r = gelu_complement(x, x2);
    const float h = 1.0f - r;
    const float slope = x * fmaf(6.0f * kGeluScale * kGeluCubic, fminf(x2, 256.0f),
                                 2.0f * kGeluScale);
    return fmaf(h * r, slope, h);
}

}  // namespace vitb200
