// Column sums of a row-major matrix: out[c] += sum_r in[r*ld + c].
// Used for bias gradients and for the positional / CLS gradients; matrices of many
// columns take column_strips_kernel below.
//
// A block owns a strip of columns (32 threads wide, each thread 1 or 4
// adjacent columns) and a slice of the rows; its 32 row lanes walk the slice
// with fully coalesced 128- or 512-byte row segments, fold through shared
// memory, and one lane per column adds the block's partial with a single
// atomic.  Row slices are sized so the whole grid is about two waves.
#include "kernels.h"
#include "device_util.cuh"

#include <algorithm>

namespace vitb200 {
namespace {

constexpr int kLanesX = 32;
constexpr int kLanesY = 32;

template <int V>
__global__ void __launch_bounds__(kLanesX *kLanesY)
column_sums_kernel(const float *__restrict__ in, float *__restrict__ out,
                   size_t rows, size_t cols, size_t ld, size_t rows_per_block) {
    grid_dependency_wait();
    grid_dependency_release();
    __shared__ float partial[kLanesY][kLanesX * V + 1];
    const size_t col = (size_t(blockIdx.x) * kLanesX + threadIdx.x) * V;
    const size_t row_begin = size_t(blockIdx.y) * rows_per_block;
    const size_t row_end = min(rows, row_begin + rows_per_block);
    float sum[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        sum[j] = 0.0f;
    }
    if (col < cols) {
        for (size_t row = row_begin + threadIdx.y; row < row_end;
             row += kLanesY) {
            const float *p = in + row * ld + col;
            if (V == 4) {
                const float4 v = __ldcs(reinterpret_cast<const float4 *>(p));
                sum[0] += v.x;
                sum[V > 1 ? 1 : 0] += v.y;
                sum[V > 2 ? 2 : 0] += v.z;
                sum[V > 3 ? 3 : 0] += v.w;
            } else {
                sum[0] += __ldcs(p);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
        partial[threadIdx.y][threadIdx.x * V + j] = sum[j];
    }
    __syncthreads();
    // Fold the 32 row lanes: thread (x, y) reduces column slot y*?.. simple
    // tree over y keeps the code independent of V.
    for (int stride = kLanesY / 2; stride > 0; stride >>= 1) {
        if (threadIdx.y < stride) {
#pragma unroll
            for (int j = 0; j < V; ++j) {
                partial[threadIdx.y][threadIdx.x * V + j] +=
                    partial[threadIdx.y + stride][threadIdx.x * V + j];
            }
        }
        __syncthreads();
    }
    if (threadIdx.y == 0 && col < cols) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            atomicAdd(out + col + j, partial[0][threadIdx.x * V + j]);
        }
    }
}

// Many columns, few rows (the positional gradients: a row per image, a column per
// token and feature): eight row lanes with eight loads in flight each, where the
// kernel above has 32 lanes that find two rows each and a fold in five steps.
// Bound by memory: 64 rows of 393600 columns (101 MB, 15 us at the copy rate) take the
// kernel above 72 us, this one 25; 2048 rows of 50432 columns 80 and 72, of 6400
// columns 25 and 18.
//
// The rows are added up as trees (eight loads, then eight lanes), so that a sum's
// error is no larger than there (2-norm against 64 bits, normal values: 0.7e-7 and
// 0.7e-7, 1.6e-7 and 1.0e-7, 1.0e-7 and 1.0e-7 for the three; one row after the other
// gave 1.1e-7, 2.5e-7 and 2.0e-7 in the same time).  The bound on the registers keeps
// the eight loads together: without it 25600 x 4096 takes 96 us instead of 74.
constexpr int kStripLanes = 8;
// From this many columns on, bias gradients as wide as that among them.  At 4096 it
// takes 14 us for 2049 rows (there 20) and 74 for 25600 (91); narrower sums have many
// more rows than columns and stay above.
constexpr size_t kStripColumns = 4096;

// Slices of the rows: what fills two blocks per SM, in whole rounds of them.  (Four
// are resident, but every slice is one more addition in a row for each sum: at four
// 2049 x 4096 had 1.07 of the error above, and is no faster.)
size_t strip_slices(size_t rows, size_t strips) {
    const size_t round = size_t(device_sm_count()) * 2;
    const size_t loads = 8 * kStripLanes;   // rows of a block's round of loads
    const size_t most = std::min<size_t>(
        std::min<size_t>((rows + loads - 1) / loads, 65535),
        std::max<size_t>(4, (round + strips - 1) / strips));
    size_t best = 1;
    double least = 0.0;
    for (size_t slices = 1; slices <= most; ++slices) {
        const double turns = double((strips * slices + round - 1) / round);
        const size_t rows_each = (rows + slices - 1) / slices;
        const double time =
            turns * double((rows_each + loads - 1) / loads) + 0.02 * double(slices);
        if (slices == 1 || time < least) {
            best = slices;
            least = time;
        }
    }
    return best;
}

__device__ __forceinline__ float4 add4(const float4 &a, const float4 &b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

__device__ __forceinline__ float4 tree8(const float4 (&v)[8]) {
    return add4(add4(add4(v[0], v[1]), add4(v[2], v[3])),
                add4(add4(v[4], v[5]), add4(v[6], v[7])));
}

__global__ void __launch_bounds__(kLanesX *kStripLanes, 4)
column_strips_kernel(const float *__restrict__ in, float *__restrict__ out,
                     size_t rows, size_t cols, size_t ld, size_t rows_per_block) {
    grid_dependency_wait();
    grid_dependency_release();
    __shared__ float4 partial[kStripLanes][kLanesX];
    const size_t col = (size_t(blockIdx.x) * kLanesX + threadIdx.x) * 4;
    const size_t row_begin = size_t(blockIdx.y) * rows_per_block;
    const size_t row_end = min(rows, row_begin + rows_per_block);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 sum = zero;
    if (col < cols) {
        for (size_t row = row_begin + threadIdx.y; row < row_end;
             row += 8 * kStripLanes) {
            float4 v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const size_t mine = row + r * kStripLanes;
                v[r] = mine < row_end
                    ? __ldcs(reinterpret_cast<const float4 *>(in + mine * ld + col))
                    : zero;
            }
            sum = add4(sum, tree8(v));
        }
    }
    partial[threadIdx.y][threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.y != 0 || col >= cols || row_begin >= row_end) {
        return;
    }
    float4 lanes[kStripLanes];
#pragma unroll
    for (int y = 0; y < kStripLanes; ++y) {
        lanes[y] = partial[y][threadIdx.x];
    }
    sum = tree8(lanes);
    float *target = out + col;
    if ((reinterpret_cast<size_t>(target) & 15) == 0) {
        asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::
                         "l"(target),
                     "f"(sum.x), "f"(sum.y), "f"(sum.z), "f"(sum.w)
                     : "memory");
    } else {
        atomicAdd(target + 0, sum.x);
        atomicAdd(target + 1, sum.y);
        atomicAdd(target + 2, sum.z);
        atomicAdd(target + 3, sum.w);
    }
}

struct ColumnSumBatch {
    ColumnSumJob job[kColumnSumBatch];
};

// Several small column sums in one launch: block (x, j) sums 128 columns of
// job j (a multiple of four columns wide, a few hundred rows at most), 32
// column lanes of four floats by eight row lanes, folded through shared
// memory.  The result replaces or is added to the destination; a one-row
// source that is a running accumulator is cleared for its next user.
__global__ void __launch_bounds__(256)
column_sums_batch_kernel(const ColumnSumBatch batch) {
    grid_dependency_wait();
    grid_dependency_release();
    __shared__ float4 fold[8][32];
    const ColumnSumJob job = batch.job[blockIdx.y];
    const unsigned lane = threadIdx.x & 31, row_lane = threadIdx.x >> 5;
    const unsigned col = (blockIdx.x * 32 + lane) * 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    if (col < job.cols) {
        for (unsigned row = row_lane; row < job.rows; row += 8) {
            const float4 v = *reinterpret_cast<const float4 *>(
                job.source + size_t(row) * job.cols + col);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
    }
    fold[row_lane][lane] = sum;
    __syncthreads();
    if (row_lane == 0 && col < job.cols) {
#pragma unroll
        for (int other = 1; other < 8; ++other) {
            const float4 v = fold[other][lane];
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        float4 *target = reinterpret_cast<float4 *>(job.destination + col);
        if (job.add) {
            const float4 old = *target;
            sum.x += old.x; sum.y += old.y; sum.z += old.z; sum.w += old.w;
        }
        *target = sum;
        if (job.clear) {
            for (unsigned row = 0; row < job.rows; ++row) {
                *reinterpret_cast<float4 *>(const_cast<float *>(job.source) +
                                            size_t(row) * job.cols + col) =
                    make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
}

}  // namespace

void launch_column_sums_batch(const ColumnSumJob *jobs, int count,
                              cudaStream_t stream) {
    if (count <= 0) {
        return;
    }
    ColumnSumBatch batch = {};
    unsigned widest = 0;
    for (int j = 0; j < count; ++j) {
        batch.job[j] = jobs[j];
        widest = jobs[j].cols > widest ? jobs[j].cols : widest;
    }
    launch_chained(column_sums_batch_kernel, dim3((widest + 127) / 128, count),
                   256, 0, stream, batch);
    ++g_kernel_launches;
}

void launch_column_sums(const float *in, float *out, size_t rows, size_t cols,
                        size_t ld, cudaStream_t stream) {
    if (rows == 0 || cols == 0) {
        return;
    }
    const bool vec = cols % 4 == 0 && ld % 4 == 0;
    if (vec && cols >= kStripColumns) {
        const size_t strips = (cols / 4 + kLanesX - 1) / kLanesX;
        const size_t slices = strip_slices(rows, strips);
        launch_streamed(column_strips_kernel, dim3(unsigned(strips), unsigned(slices)),
                        dim3(kLanesX, kStripLanes), stream, 4 * rows * cols, in, out,
                        rows, cols, ld, (rows + slices - 1) / slices);
        ++g_kernel_launches;
        return;
    }
    const size_t cols_per_block = kLanesX * (vec ? 4 : 1);
    const unsigned grid_x =
        static_cast<unsigned>((cols + cols_per_block - 1) / cols_per_block);
    size_t slices = (2 * kSmCount + grid_x - 1) / grid_x;
    const size_t max_slices = (rows + 4 * kLanesY - 1) / (4 * kLanesY);
    if (slices > max_slices) {
        slices = max_slices;
    }
    if (slices < 1) {
        slices = 1;
    }
    if (slices > 65535) {
        slices = 65535;
    }
    const size_t rows_per_block = (rows + slices - 1) / slices;
    const dim3 grid(grid_x, static_cast<unsigned>(slices));
    const dim3 block(kLanesX, kLanesY);
    if (vec) {
        launch_chained(column_sums_kernel<4>, grid, block, 0, stream, in, out,
                       rows, cols, ld, rows_per_block);
    } else {
        launch_chained(column_sums_kernel<1>, grid, block, 0, stream, in, out,
                       rows, cols, ld, rows_per_block);
    }
    ++g_kernel_launches;
}

}  // namespace vitb200
