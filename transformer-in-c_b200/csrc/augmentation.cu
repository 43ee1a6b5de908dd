// Batch augmentation on the device (reference src/augmentation.c).
//
// The reference walks the batch sample by sample, pixel by pixel, drawing
// from one splitmix64 stream as it goes.  That generator advances its state
// by a constant per draw, so draw number k is mix(state + (k + 1) * step): a
// pure function of the start state.  The order of the draws is fixed except
// for random erasing, which takes four more draws only when its first draw
// says "erase".  A host pass over the batch therefore knows where each sample's
// draws start; after that every sample is independent.  The host keeps only what
// cannot move: the walk along the stream (one mix per sample, for the erasing
// decision) and the rotation's angle, cosine and sine (a second mix), which have to
// come from the same libm as the reference's.
//
// Images whose plane fits shared memory twice (up to 160 x 160) take one kernel,
// a block per image plane:
//   the plane is staged once; bilinear sampling reads and writes shared memory;
//   one lane adds up the plane mean front to back, in the reference's order
//   (a float sum depends on its order: a chain of one addition per pixel, 1.7 us
//   at 28 x 28), while the other warps compute the pixels' Gaussian noise, which
//   is what most of the instructions are for (two 64-bit mixes, a logarithm, a
//   root and a cosine per pixel); a last pass applies contrast, noise, clamp
//   and erasing and stores.
// Larger ones go through global memory between four kernels (parameters, affine,
// plane means, pixels).  Measured at 2048 x 28 x 28 with everything on: the host pass
// takes 18 us of the call's 27 and the kernel 25 us beside the next batch's host pass;
// with all draws on the host that pass took 45 us, the three kernels and the upload of
// its table 58.
//
// Arithmetic that the reference rounds step by step is written with the
// round-to-nearest intrinsics, which the compiler never contracts into fused
// multiply-adds; cos / sin of the rotation are taken on the host with the same
// libm as the reference.  What remains different is logf and cosf inside the
// Box-Muller noise (device libm, an ulp or two), i.e. errors of about 1e-7 of
// the noise amplitude; everything else is bit-identical.
#include "augmentation.h"
#include "kernels.h"
#include "device_util.cuh"
#include "shared_limit.h"

#include <cmath>

namespace vitb200 {
namespace {

constexpr unsigned long long kStep = 0x9E3779B97F4A7C15ull;
constexpr float kPi = 3.14159265358979323846f;

__host__ __device__ inline unsigned long long mix(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// ---- host side: the reference's draws, in its order ------------------------

float unit(uint64_t state) {   // augmentation.c:15-17
    return ((float)(mix(state) >> 40) + 0.5f) / 16777216.0f;
}

bool geometric(const AugmentationSettings &s) {
    return s.max_shift_pixels > 0.0f || s.max_rotation_degrees > 0.0f ||
           s.max_scale_delta > 0.0f;
}

bool intensity(const AugmentationSettings &s) {
    return s.max_brightness_delta > 0.0f || s.max_contrast_delta > 0.0f;
}

// ---- device side -------------------------------------------------------------

__device__ __forceinline__ float clamp_value(float value, float minimum,
                                             float maximum) {
    return value < minimum ? minimum : value > maximum ? maximum : value;
}

// augmentation.c:36-55, every operation rounded on its own.
__device__ __forceinline__ float sample_bilinear(const float *plane, int height,
                                                 int width, float source_y,
                                                 float source_x) {
    const float clamped_y = clamp_value(source_y, 0.0f, float(height - 1));
    const float clamped_x = clamp_value(source_x, 0.0f, float(width - 1));
    const int top = int(clamped_y);
    const int left = int(clamped_x);
    const int bottom = top + 1 < height ? top + 1 : top;
    const int right = left + 1 < width ? left + 1 : left;
    const float wy = __fsub_rn(clamped_y, float(top));
    const float wx = __fsub_rn(clamped_x, float(left));
    const float one_minus_wx = __fsub_rn(1.0f, wx);
    const float upper =
        __fadd_rn(__fmul_rn(plane[top * width + left], one_minus_wx),
                  __fmul_rn(plane[top * width + right], wx));
    const float lower =
        __fadd_rn(__fmul_rn(plane[bottom * width + left], one_minus_wx),
                  __fmul_rn(plane[bottom * width + right], wx));
    return __fadd_rn(__fmul_rn(upper, __fsub_rn(1.0f, wy)),
                     __fmul_rn(lower, wy));
}

// augmentation.c:63-90: the output pixel (y, x) of a plane.
__device__ __forceinline__ float sample_affine(const float *plane,
                                               const AugmentationSample &p, float y,
                                               float x, float center_y,
                                               float center_x, int height,
                                               int width) {
    const float centered_y = __fsub_rn(__fsub_rn(y, center_y), p.shift_y);
    const float centered_x = __fsub_rn(__fsub_rn(x, center_x), p.shift_x);
    const float source_x =
        __fadd_rn(__fadd_rn(__fmul_rn(p.inverse_cosine, centered_x),
                            __fmul_rn(p.inverse_sine, centered_y)),
                  center_x);
    const float source_y =
        __fadd_rn(__fadd_rn(__fmul_rn(-p.inverse_sine, centered_x),
                            __fmul_rn(p.inverse_cosine, centered_y)),
                  center_y);
    return sample_bilinear(plane, height, width, source_y, source_x);
}

// The same for whole batches.  `samples` == nullptr: one transform for all samples.
__global__ void augmentation_affine_kernel(
    const float *__restrict__ source, float *__restrict__ destination,
    const AugmentationSample *__restrict__ samples, AugmentationSample shared,
    size_t batch, int channels, int height, int width) {
    const size_t plane = size_t(height) * width;
    const size_t total = batch * channels * plane;
    const float center_y = __fmul_rn(0.5f, float(height - 1));
    const float center_x = __fmul_rn(0.5f, float(width - 1));
    for (size_t i = global_thread(); i < total; i += grid_threads()) {
        const size_t image_plane = i / plane;   // sample * channels + channel
        const int pixel = int(i % plane);
        const int y = pixel / width, x = pixel % width;
        const AugmentationSample &p =
            samples ? samples[image_plane / channels] : shared;
        destination[i] =
            sample_affine(source + image_plane * plane, p, float(y), float(x), center_y,
                          center_x, height, width);
    }
}

// augmentation.c:118-122: the plane mean, summed front to back.  A float sum
// depends on its order, so the additions stay sequential (lane 0 does them),
// but the loads are the warp's: 32 consecutive pixels at a time, handed to
// lane 0 by shuffles that do not wait for the running sum.
__global__ void augmentation_mean_kernel(const float *__restrict__ images,
                                         float *__restrict__ means,
                                         size_t planes, size_t plane_size) {
    const int lane = threadIdx.x & 31;
    const size_t warp = global_thread() >> 5;
    const size_t warps = grid_threads() >> 5;
    for (size_t p = warp; p < planes; p += warps) {
        const float *plane = images + p * plane_size;
        float sum = 0.0f;
        for (size_t base = 0; base < plane_size; base += 32) {
            const size_t index = base + lane;
            const float mine = index < plane_size ? plane[index] : 0.0f;
            const int live = int(min(size_t(32), plane_size - base));
            for (int l = 0; l < live; ++l) {
                sum = __fadd_rn(sum, __shfl_sync(kFullMask, mine, l));
            }
        }
        if (lane == 0) {
            means[p] = __fdiv_rn(sum, float(plane_size));
        }
    }
}

__device__ __forceinline__ float unit_from_state(unsigned long long state) {
    // (The division by 2^24 as the exact product it is.)
    return __fmul_rn(__fadd_rn(float(unsigned(mix(state) >> 40)), 0.5f), 0x1p-24f);
}

// The sample's parameters from its draws (augmentation.c:92-166), with the
// draws numbered from the sample's start state.
__device__ AugmentationSample sample_parameters(const AugmentationDraws &draws,
                                                const AugmentationSettings &s,
                                                bool geometric, bool intensity,
                                                bool erasing, size_t image_size,
                                                int height, int width) {
    AugmentationSample p = {};
    p.inverse_cosine = 1.0f;
    p.contrast = 1.0f;
    unsigned long long state = draws.state;
    auto symmetric = [&](float magnitude) {
        state += kStep;
        return __fmul_rn(magnitude,
                         __fsub_rn(__fmul_rn(2.0f, unit_from_state(state)), 1.0f));
    };
    if (geometric) {
        p.shift_y = symmetric(s.max_shift_pixels);
        p.shift_x = symmetric(s.max_shift_pixels);
        state += kStep;   // the angle: taken by the host
        const float scale = __fadd_rn(1.0f, symmetric(s.max_scale_delta));
        p.inverse_cosine = __fdiv_rn(draws.cosine, scale);
        p.inverse_sine = __fdiv_rn(draws.sine, scale);
    }
    if (intensity) {
        p.contrast = __fadd_rn(1.0f, symmetric(s.max_contrast_delta));
        p.brightness = symmetric(s.max_brightness_delta);
    }
    if (s.noise_standard_deviation > 0.0f) {
        p.noise_state = state;
        state += 2ull * image_size * kStep;
    }
    if (erasing && draws.erase) {
        state += kStep;   // the decision
        auto index_below = [&](unsigned long long limit) {
            state += kStep;
            return unsigned(mix(state) % limit);
        };
        const unsigned long long max_height = (unsigned long long)fmaxf(
            1.0f, __fmul_rn(s.erasing_max_side_fraction, float(height)));
        const unsigned long long max_width = (unsigned long long)fmaxf(
            1.0f, __fmul_rn(s.erasing_max_side_fraction, float(width)));
        p.erase_height = 1 + index_below(max_height);
        p.erase_width = 1 + index_below(max_width);
        p.erase_top = index_below((unsigned long long)(height - p.erase_height) + 1);
        p.erase_left = index_below((unsigned long long)(width - p.erase_width) + 1);
    }
    return p;
}

// Box-Muller from a pixel's two draws, `first` being the state of the first:
// draws 2k+1 and 2k+2 after the sample's noise start for pixel k of the image
// (augmentation.c:123-140).
__device__ __forceinline__ float noise_normal(unsigned long long first) {
    const float u1 = unit_from_state(first);
    const float u2 = unit_from_state(first + kStep);
    const float radius = __fsqrt_rn(__fmul_rn(-2.0f, logf(u1)));
    return __fmul_rn(radius, cosf(__fmul_rn(2.0f * kPi, u2)));
}

struct AugmentationSteps {
    bool geometric, jitter, noise, clamps, erasing;
};

// augmentation.c:36-229 for one image plane per block.
__global__ void __launch_bounds__(256)
augmentation_plane_kernel(const float *source, float *destination,
                          const AugmentationDraws *__restrict__ draws,
                          const AugmentationSettings settings,
                          const AugmentationSteps steps, int channels, int height,
                          int width) {
    extern __shared__ __align__(16) float planes[];
    __shared__ AugmentationSample shared_sample;
    __shared__ float shared_mean;
    const int plane = height * width;
    const int padded = (plane + 3) & ~3;
    const size_t sample = blockIdx.x / unsigned(channels);
    const int channel = int(blockIdx.x % unsigned(channels));
    const float *from = source + size_t(blockIdx.x) * plane;
    float *to = destination + size_t(blockIdx.x) * plane;
    if (threadIdx.x == 0) {
        // The plan is in page-locked host memory, complete before the launch: the
        // trip over the bus overlaps whatever kernel is still running.
        shared_sample = sample_parameters(draws[sample], settings, steps.geometric,
                                          steps.jitter, steps.erasing,
                                          size_t(plane) * channels, height, width);
    }
    grid_dependency_wait();
    grid_dependency_release();
    const bool vec = plane % 4 == 0 && (reinterpret_cast<uintptr_t>(from) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(to) & 15) == 0;
    float *values = planes, *other = planes + padded;
    if (vec) {
        for (int i = threadIdx.x * 4; i < plane; i += blockDim.x * 4) {
            *reinterpret_cast<float4 *>(values + i) =
                *reinterpret_cast<const float4 *>(from + i);
        }
    } else {
        for (int i = threadIdx.x; i < plane; i += blockDim.x) {
            values[i] = from[i];
        }
    }
    __syncthreads();
    const AugmentationSample p = shared_sample;
    if (steps.geometric) {
        const float center_y = __fmul_rn(0.5f, float(height - 1));
        const float center_x = __fmul_rn(0.5f, float(width - 1));
        // (y, x) of the thread's pixels, stepped instead of divided for.
        const int step_y = int(blockDim.x / unsigned(width));
        const int step_x = int(blockDim.x % unsigned(width));
        int y = int(threadIdx.x / unsigned(width)), x = int(threadIdx.x % unsigned(width));
        for (int i = threadIdx.x; i < plane; i += blockDim.x) {
            other[i] = sample_affine(values, p, float(y), float(x), center_y, center_x,
                                     height, width);
            y += step_y;
            x += step_x;
            if (x >= width) {
                x -= width;
                ++y;
            }
        }
        __syncthreads();
        float *swap = values;
        values = other;
        other = swap;
    }
    const int first_noise_thread = steps.jitter ? 32 : 0;
    if (steps.jitter && threadIdx.x == 0) {
        float sum = 0.0f;
        int i = 0;
#pragma unroll 8
        for (; i + 4 <= plane; i += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(values + i);
            sum = __fadd_rn(sum, v.x);
            sum = __fadd_rn(sum, v.y);
            sum = __fadd_rn(sum, v.z);
            sum = __fadd_rn(sum, v.w);
        }
        for (; i < plane; ++i) {
            sum = __fadd_rn(sum, values[i]);
        }
        shared_mean = __fdiv_rn(sum, float(plane));
    }
    if (steps.noise && int(threadIdx.x) >= first_noise_thread) {
        const int begin = int(threadIdx.x) - first_noise_thread;
        const int stride = int(blockDim.x) - first_noise_thread;
        const unsigned long long k = (unsigned long long)channel * plane + begin;
        unsigned long long state = p.noise_state + (2ull * k + 1ull) * kStep;
        const unsigned long long advance = 2ull * stride * kStep;
        for (int i = begin; i < plane; i += stride) {
            other[i] = noise_normal(state);
            state += advance;
        }
    }
    __syncthreads();
    const float mean = steps.jitter ? shared_mean : 0.0f;
    auto finish = [&](int i) {
        float value = values[i];
        if (steps.jitter) {
            value = __fadd_rn(
                __fadd_rn(mean, __fmul_rn(__fsub_rn(value, mean), p.contrast)),
                p.brightness);
        }
        if (steps.noise) {
            value = __fadd_rn(
                value, __fmul_rn(settings.noise_standard_deviation, other[i]));
        }
        if (steps.clamps) {
            value = clamp_value(value, settings.minimum_value,
                                settings.maximum_value);
        }
        if (steps.erasing && p.erase_height) {
            const unsigned y = unsigned(i) / unsigned(width);
            const unsigned x = unsigned(i) - y * unsigned(width);
            if (y - p.erase_top < p.erase_height && x - p.erase_left < p.erase_width) {
                value = settings.erasing_value;
            }
        }
        return value;
    };
    if (vec) {
        for (int i = threadIdx.x * 4; i < plane; i += blockDim.x * 4) {
            *reinterpret_cast<float4 *>(to + i) =
                make_float4(finish(i), finish(i + 1), finish(i + 2), finish(i + 3));
        }
    } else {
        for (int i = threadIdx.x; i < plane; i += blockDim.x) {
            to[i] = finish(i);
        }
    }
}

// Parameters of all samples, for the kernels of large images.
__global__ void augmentation_parameters_kernel(
    const AugmentationDraws *__restrict__ draws, AugmentationSample *samples,
    const AugmentationSettings settings, const AugmentationSteps steps, size_t batch,
    size_t image_size, int height, int width) {
    for (size_t i = global_thread(); i < batch; i += grid_threads()) {
        samples[i] = sample_parameters(draws[i], settings, steps.geometric,
                                       steps.jitter, steps.erasing, image_size,
                                       height, width);
    }
}

// Everything after the geometric step, per pixel (augmentation.c:123-166 and
// the clamp of :219-223).
__global__ void augmentation_pixel_kernel(
    const float *__restrict__ input, float *__restrict__ destination,
    const AugmentationSample *__restrict__ samples,
    const float *__restrict__ means, AugmentationSettings settings,
    bool jitter, bool noise, bool clamps, bool erasing, size_t batch,
    int channels, int height, int width) {
    const size_t plane = size_t(height) * width;
    const size_t image = plane * channels;
    const size_t total = batch * image;
    for (size_t i = global_thread(); i < total; i += grid_threads()) {
        const size_t sample = i / image;
        const size_t within = i % image;   // the reference's noise loop index
        const AugmentationSample &p = samples[sample];
        float value = input[i];
        if (jitter) {
            const float mean = means[i / plane];
            value = __fadd_rn(
                __fadd_rn(mean, __fmul_rn(__fsub_rn(value, mean), p.contrast)),
                p.brightness);
        }
        if (noise) {
            const float normal =
                noise_normal(p.noise_state + (2ull * within + 1ull) * kStep);
            value = __fadd_rn(
                value, __fmul_rn(settings.noise_standard_deviation, normal));
        }
        if (clamps) {
            value = clamp_value(value, settings.minimum_value,
                                settings.maximum_value);
        }
        if (erasing && p.erase_height) {
            const unsigned pixel = unsigned(within % plane);
            const unsigned y = pixel / unsigned(width);
            const unsigned x = pixel % unsigned(width);
            if (y >= p.erase_top && y < p.erase_top + p.erase_height &&
                x >= p.erase_left && x < p.erase_left + p.erase_width) {
                value = settings.erasing_value;
            }
        }
        destination[i] = value;
    }
}

}  // namespace

namespace {

// Two copies of a plane in shared memory.
constexpr size_t kPlaneBytes = 200 * 1024;

// Whether the kernel of one block per image plane takes the batch: the plane fits
// shared memory twice, the planes a grid.
bool block_per_plane(size_t batch, size_t channels, size_t plane) {
    return 2 * ((plane + 3) & ~size_t(3)) * sizeof(float) <= kPlaneBytes &&
           batch <= 0x7fffffffu / channels;
}

}  // namespace

bool augmentation_enabled(const AugmentationSettings &s) {
    return geometric(s) || intensity(s) || s.noise_standard_deviation > 0.0f ||
           s.erasing_probability > 0.0f;
}

bool augmentation_arguments_valid(const AugmentationSettings *s,
                                  const uint64_t *random_state,
                                  const void *source, const void *destination,
                                  size_t batch, size_t channels, size_t height,
                                  size_t width) {
    return !(!s || !random_state || !source || !destination || batch == 0 ||
             channels == 0 || height == 0 || width == 0 ||
             s->max_shift_pixels < 0.0f || s->max_rotation_degrees < 0.0f ||
             s->max_scale_delta < 0.0f || s->max_scale_delta >= 1.0f ||
             s->max_brightness_delta < 0.0f || s->max_contrast_delta < 0.0f ||
             s->max_contrast_delta >= 1.0f ||
             s->noise_standard_deviation < 0.0f ||
             s->erasing_probability < 0.0f || s->erasing_probability > 1.0f ||
             s->erasing_max_side_fraction < 0.0f ||
             s->erasing_max_side_fraction > 1.0f ||
             (geometric(*s) && source == destination));
}

void augmentation_plan(const AugmentationSettings &s, uint64_t *random_state,
                       size_t batch, size_t channels, size_t height,
                       size_t width, AugmentationDraws *draws) {
    uint64_t state = *random_state;
    const size_t image_size = channels * height * width;
    const bool geometry = geometric(s), erasing = s.erasing_probability > 0.0f;
    // Draws of a sample before the erasing decision (augmentation.c:92-136).
    const uint64_t before = (geometry ? 4 : 0) + (intensity(s) ? 2 : 0) +
        (s.noise_standard_deviation > 0.0f ? 2ull * image_size : 0ull);
    for (size_t sample = 0; sample < batch; ++sample) {
        AugmentationDraws &d = draws[sample];
        float cosine = 1.0f, sine = 0.0f;
        if (geometry) {   // :95-98, :67-68
            const float angle = s.max_rotation_degrees *
                (2.0f * unit(state + 3 * kStep) - 1.0f) * kPi / 180.0f;
            cosine = cosf(angle);
            sine = sinf(angle);
        }
        // :141-166: the decision, and four more draws if it is to erase.
        const bool erase = erasing &&
            !(unit(state + (before + 1) * kStep) >= s.erasing_probability);
        d.state = state;
        d.cosine = cosine;
        d.sine = sine;
        d.erase = erase ? 1u : 0u;
        state += (before + (erasing ? (erase ? 5 : 1) : 0)) * kStep;
    }
    *random_state = state;
}

size_t augmentation_scratch_bytes(size_t batch, size_t channels, size_t height,
                                  size_t width) {
    return block_per_plane(batch, channels, height * width)
        ? 0 : batch * (sizeof(AugmentationSample) + channels * sizeof(float));
}

bool launch_augmentation(const AugmentationSettings &s,
                         const AugmentationDraws *draws, const float *source,
                         float *destination, void *scratch, size_t batch,
                         size_t channels, size_t height, size_t width,
                         cudaStream_t stream) {
    const size_t total = batch * channels * height * width;
    const AugmentationSteps steps = {geometric(s), intensity(s),
                                     s.noise_standard_deviation > 0.0f,
                                     s.minimum_value < s.maximum_value,
                                     s.erasing_probability > 0.0f};
    if (block_per_plane(batch, channels, height * width)) {
        const size_t bytes = 2 * ((height * width + 3) & ~size_t(3)) * sizeof(float);
        if (bytes > 40 * 1024) {
            static SharedMemoryLimit limit;
            if (!limit.raise(reinterpret_cast<const void *>(augmentation_plane_kernel),
                             int(kPlaneBytes))) {
                return false;
            }
        }
        const unsigned threads = height * width <= 1024 ? 128 : 256;
        if (launch_chained(augmentation_plane_kernel, dim3(unsigned(batch * channels)),
                           dim3(threads), bytes, stream, source, destination, draws, s,
                           steps, int(channels), int(height),
                           int(width)) != cudaSuccess) {
            return false;
        }
        ++g_kernel_launches;
        return true;
    }
    AugmentationSample *samples = static_cast<AugmentationSample *>(scratch);
    float *means = reinterpret_cast<float *>(samples + batch);
    augmentation_parameters_kernel<<<stream_grid(batch), kStreamThreads, 0, stream>>>(
        draws, samples, s, steps, batch, channels * height * width, int(height),
        int(width));
    ++g_kernel_launches;
    const float *current = source;
    if (steps.geometric) {
        augmentation_affine_kernel<<<stream_grid(total), kStreamThreads, 0,
                                     stream>>>(
            source, destination, samples, AugmentationSample{}, batch,
            int(channels), int(height), int(width));
        ++g_kernel_launches;
        current = destination;
    }
    if (steps.jitter) {
        augmentation_mean_kernel<<<stream_grid(batch * channels * 32),
                                   kStreamThreads, 0, stream>>>(
            current, means, batch * channels, height * width);
        ++g_kernel_launches;
    }
    if (steps.jitter || steps.noise || steps.clamps || steps.erasing ||
        current != destination) {
        augmentation_pixel_kernel<<<stream_grid(total), kStreamThreads, 0,
                                    stream>>>(
            current, destination, samples, means, s, steps.jitter, steps.noise,
            steps.clamps, steps.erasing, batch, int(channels), int(height),
            int(width));
        ++g_kernel_launches;
    }
    return cudaPeekAtLastError() == cudaSuccess;
}

void launch_augmentation_translate(const float *source, float *destination,
                                   size_t batch, size_t channels, size_t height,
                                   size_t width, float shift_y, float shift_x,
                                   cudaStream_t stream) {
    AugmentationSample all{};
    all.inverse_cosine = cosf(0.0f) / 1.0f;
    all.inverse_sine = sinf(0.0f) / 1.0f;
    all.shift_y = shift_y;
    all.shift_x = shift_x;
    const size_t total = batch * channels * height * width;
    augmentation_affine_kernel<<<stream_grid(total), kStreamThreads, 0, stream>>>(
        source, destination, nullptr, all, batch, int(channels), int(height),
        int(width));
    ++g_kernel_launches;
}

}  // namespace vitb200
