// Batch augmentation on the device: the reference's data_augmentation_apply
// (reference src/augmentation.c:178-229) as a kernel plus a host pass that lays
// the random stream out.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace vitb200 {

// Field for field the reference's DataAugmentation (include/augmentation.h:7-19).
struct AugmentationSettings {
    float max_shift_pixels;
    float max_rotation_degrees;
    float max_scale_delta;
    float max_brightness_delta;
    float max_contrast_delta;
    float noise_standard_deviation;
    float erasing_probability;
    float erasing_max_side_fraction;
    float erasing_value;
    float minimum_value;
    float maximum_value;
};

// Everything the reference draws per sample, and where in the random stream the
// sample's per-pixel noise draws start.
struct AugmentationSample {
    float inverse_cosine, inverse_sine, shift_y, shift_x;
    float contrast, brightness;
    unsigned erase_top, erase_left, erase_height, erase_width;   // height 0: none
    unsigned long long noise_state;   // stream state before the first noise draw
};

// What the host pass leaves for one sample: where its draws start, and what is
// not worth or not possible to draw on the device.
struct AugmentationDraws {
    unsigned long long state;   // stream state before the sample's first draw
    float cosine, sine;         // of the rotation, by the host's libm
    unsigned erase;             // the erasing decision
};

bool augmentation_enabled(const AugmentationSettings &settings);

// The reference's argument checks (src/augmentation.c:182-198).
bool augmentation_arguments_valid(const AugmentationSettings *settings,
                                  const uint64_t *random_state,
                                  const void *source, const void *destination,
                                  size_t batch, size_t channels, size_t height,
                                  size_t width);

// Walks the reference's sequence of draws for `batch` samples starting at
// *random_state, fills draws[0..batch) and leaves *random_state where the
// reference would.
void augmentation_plan(const AugmentationSettings &settings,
                       uint64_t *random_state, size_t batch, size_t channels,
                       size_t height, size_t width, AugmentationDraws *draws);

// Device scratch launch_augmentation needs for images of this size.
size_t augmentation_scratch_bytes(size_t batch, size_t channels, size_t height,
                                  size_t width);

// Applies a plan.  source / destination / scratch are device pointers, draws
// anything the device can read.  source == destination is allowed when no
// geometric transform is configured.  False when a kernel could not be launched; the
// destination's contents are then undefined.
bool launch_augmentation(const AugmentationSettings &settings,
                         const AugmentationDraws *draws, const float *source,
                         float *destination, void *scratch, size_t batch,
                         size_t channels, size_t height, size_t width,
                         cudaStream_t stream);

// data_augmentation_translate (src/augmentation.c:231-245) on device buffers.
void launch_augmentation_translate(const float *source, float *destination,
                                   size_t batch, size_t channels, size_t height,
                                   size_t width, float shift_y, float shift_x,
                                   cudaStream_t stream);

}  // namespace vitb200
