// Bidirectional multi-head attention on head-major tensors, with the full
// probability matrix materialised (the host keeps it as a tensor and hands it
// back to the backward pass; reference src/ops.c:1297-1355, :1381-1441): the FP32
// path of sequences that do not fit the whole-group kernels, and of head
// dimensions that have no other.
//
//   forward   row maxima and denominators over one sweep of the keys, then the
//             scores again, P and O = P V
//   backward  D_i = dO_i . O_i
//             query-major kernel: dP = dO V^T, dS = scale P (dP - D), dQ += dS K
//             key-major kernel:   same dS recomputed,  dK += dS^T Q, dV += P^T dO
//
// What bounds it: the FMA pipes (and S^2 floats of P written once and read twice).
// One block per (group, 64 rows), 16 x 16 threads; every product of a 64 x 64 tile
// is taken as 4 x 4 values (or 4 x head_dim / 16) per thread, both operands with the
// contracted index outermost in shared memory, so that 16 multiply-adds cost two
// 128-bit reads.  A thread's four keys of a tile are 16 apart (their operand is
// staged in that order), so that its accesses to rows of P are contiguous across
// lanes.  Measured against 32 x 32 tiles with scalar reads, us forward / backward:
// 153 groups of 442 x 32 608 / 1415 -> 254 / 423, 40 of 1025 x 64 1595 / 3727 -> 671 /
// 1167 (23 TFLOP/s, recomputed scores counted), 6 of 170 x 8 18 / 45 -> 18 / 30.
#include "kernels.h"
#include "gemm.h"
#include "../../include/vitb200.h"
#include "device_util.cuh"
#include "shared_limit.h"

#include <cfloat>
#include <cstdint>
#include <initializer_list>

namespace vitb200 {
namespace {

constexpr int kTile = 64;      // rows per block, and of the other axis per step
constexpr int kSide = 16;      // threads along either axis of a tile
constexpr int kThreads = kSide * kSide;
constexpr int kPitch = kTile + 4;

// Where row r of a tile is kept in an operand whose rows belong to the lanes along x:
// lane x reads positions 4x ... 4x + 3, which are the rows x, x + 16, x + 32, x + 48.
__device__ __forceinline__ int lane_position(int r) {
    return 4 * (r % kSide) + r / kSide;
}

// Four values of row `row` from column d on, zeros past either extent.
__device__ __forceinline__ float4 four_columns(const float *__restrict__ base, int row,
                                               int d, int seq, int head_dim, bool vec) {
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row < seq) {
        const float *from = base + size_t(row) * head_dim + d;
        if (vec && d + 4 <= head_dim) {
            x = __ldg(reinterpret_cast<const float4 *>(from));
        } else {
            if (d < head_dim) x.x = __ldg(from);
            if (d + 1 < head_dim) x.y = __ldg(from + 1);
            if (d + 2 < head_dim) x.z = __ldg(from + 2);
            if (d + 3 < head_dim) x.w = __ldg(from + 3);
        }
    }
    return x;
}

// Rows [row0, row0 + 64) of a [seq, head_dim] matrix with the columns outermost,
// [HD][kPitch]; PERMUTED: rows at their lane positions.
template <int HD, bool PERMUTED>
__device__ __forceinline__ void stage_across(const float *__restrict__ base, float *tile,
                                             int row0, int seq, int head_dim, bool vec) {
    for (int i = threadIdx.x; i < kTile * (HD / 4); i += kThreads) {
        const int r = i % kTile, d = i / kTile * 4;
        const float4 x = four_columns(base, row0 + r, d, seq, head_dim, vec);
        float *to = tile + d * kPitch + (PERMUTED ? lane_position(r) : r);
        to[0] = x.x;
        to[kPitch] = x.y;
        to[2 * kPitch] = x.z;
        to[3 * kPitch] = x.w;
    }
}

// The same rows as they are, [64][HD].
template <int HD>
__device__ __forceinline__ void stage_along(const float *__restrict__ base, float *tile,
                                            int row0, int seq, int head_dim, bool vec) {
    for (int i = threadIdx.x; i < kTile * (HD / 4); i += kThreads) {
        const int r = i / (HD / 4), d = i % (HD / 4) * 4;
        *reinterpret_cast<float4 *>(tile + r * HD + d) =
            four_columns(base, row0 + r, d, seq, head_dim, vec);
    }
}

// values[i][j] = row 4y + i of `rows` . row x + 16j of `lanes` (both [HD][kPitch]).
template <int HD>
__device__ __forceinline__ void tile_product(const float *rows, const float *lanes,
                                             int x, int y, float (&values)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            values[i][j] = 0.0f;
        }
    }
#pragma unroll 8
    for (int d = 0; d < HD; ++d) {
        const float4 r = *reinterpret_cast<const float4 *>(rows + d * kPitch + 4 * y);
        const float4 l = *reinterpret_cast<const float4 *>(lanes + d * kPitch + 4 * x);
        const float row[4] = {r.x, r.y, r.z, r.w}, lane[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                values[i][j] = fmaf(row[i], lane[j], values[i][j]);
            }
        }
    }
}

// Columns of a [64][HD] result that a thread keeps (lanes past HD keep none).
template <int HD>
constexpr int kKept = HD >= kSide ? HD / kSide : 1;

// acc[i][c] += sum over the tile of weights[t][4y + i] * source[t][x * kKept + c].
template <int HD, int PITCH>
__device__ __forceinline__ void tile_update(const float *weights, const float *source,
                                            int x, int y, float (&acc)[4][kKept<HD>]) {
    constexpr int kCount = kKept<HD>;
    if (HD < kSide && x >= HD) {
        return;
    }
#pragma unroll 4
    for (int t = 0; t < kTile; ++t) {
        const float4 w = *reinterpret_cast<const float4 *>(weights + t * PITCH + 4 * y);
        const float weight[4] = {w.x, w.y, w.z, w.w};
        float column[kCount];
        const float *from = source + t * HD + x * kCount;
        if constexpr (kCount % 4 == 0) {
#pragma unroll
            for (int c = 0; c < kCount; c += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(from + c);
                column[c] = f.x;
                column[c + 1] = f.y;
                column[c + 2] = f.z;
                column[c + 3] = f.w;
            }
        } else if constexpr (kCount % 2 == 0) {
#pragma unroll
            for (int c = 0; c < kCount; c += 2) {
                const float2 f = *reinterpret_cast<const float2 *>(from + c);
                column[c] = f.x;
                column[c + 1] = f.y;
            }
        } else {
#pragma unroll
            for (int c = 0; c < kCount; ++c) {
                column[c] = from[c];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int c = 0; c < kCount; ++c) {
                acc[i][c] = fmaf(weight[i], column[c], acc[i][c]);
            }
        }
    }
}

// Row `row` of a [seq, head_dim] result (+)= this thread's columns of it.
template <int HD>
__device__ __forceinline__ void store_columns(float *base, int row, int seq, int head_dim,
                                              int x, const float (&values)[kKept<HD>],
                                              bool add) {
#pragma unroll
    for (int c = 0; c < kKept<HD>; ++c) {
        const int d = x * kKept<HD> + c;
        if (row < seq && d < head_dim) {
            float *target = base + size_t(row) * head_dim + d;
            *target = (add ? *target : 0.0f) + values[c];
        }
    }
}

template <int COUNT>
__device__ __forceinline__ void clear(float (&values)[4][COUNT]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int c = 0; c < COUNT; ++c) {
            values[i][c] = 0.0f;
        }
    }
}

// Floats of the two forms of a staged tile.
template <int HD>
constexpr int kAcross = HD * kPitch;
template <int HD>
constexpr int kAlong = HD * kTile;

template <int HD>
__global__ void __launch_bounds__(kThreads)
attention_forward_kernel(const float *__restrict__ q,
                         const float *__restrict__ k,
                         const float *__restrict__ v, float *__restrict__ p,
                         float *__restrict__ out, int seq, int head_dim,
                         float scale, bool vec) {
    extern __shared__ __align__(16) float shared[];
    float *q_tile = shared;
    float *k_tile = q_tile + kAcross<HD>;
    float *v_tile = k_tile + kAcross<HD>;
    float *p_tile = v_tile + kAlong<HD>;   // [key][row], pitch kPitch

    const size_t group = blockIdx.x;
    const int row0 = blockIdx.y * kTile;
    const int x = threadIdx.x % kSide, y = threadIdx.x / kSide;
    const size_t base = group * seq * head_dim;
    float *gp = p + group * seq * seq;
    stage_across<HD, false>(q + base, q_tile, row0, seq, head_dim, vec);

    // Maxima and denominators of this thread's keys, then of all of a row.
    float maximum[4], denominator[4], scores[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        maximum[i] = -FLT_MAX;
        denominator[i] = 0.0f;
    }
    for (int key0 = 0; key0 < seq; key0 += kTile) {
        __syncthreads();
        stage_across<HD, true>(k + base, k_tile, key0, seq, head_dim, vec);
        __syncthreads();
        tile_product<HD>(q_tile, k_tile, x, y, scores);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float highest = maximum[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                scores[i][j] *= scale;
                if (key0 + x + kSide * j < seq) {
                    highest = fmaxf(highest, scores[i][j]);
                }
            }
            denominator[i] *= expf(maximum[i] - highest);
            maximum[i] = highest;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (key0 + x + kSide * j < seq) {
                    denominator[i] += expf(scores[i][j] - highest);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float highest = maximum[i];
#pragma unroll
        for (int distance = 1; distance < kSide; distance *= 2) {
            highest = fmaxf(highest, __shfl_xor_sync(kFullMask, highest, distance));
        }
        denominator[i] *= expf(maximum[i] - highest);
        maximum[i] = highest;
#pragma unroll
        for (int distance = 1; distance < kSide; distance *= 2) {
            denominator[i] += __shfl_xor_sync(kFullMask, denominator[i], distance);
        }
    }

    float acc[4][kKept<HD>];
    clear(acc);
    for (int key0 = 0; key0 < seq; key0 += kTile) {
        __syncthreads();
        stage_across<HD, true>(k + base, k_tile, key0, seq, head_dim, vec);
        stage_along<HD>(v + base, v_tile, key0, seq, head_dim, vec);
        __syncthreads();
        tile_product<HD>(q_tile, k_tile, x, y, scores);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int key = key0 + x + kSide * j;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = row0 + 4 * y + i;
                float probability = 0.0f;
                if (row < seq && key < seq) {
                    probability =
                        expf(scale * scores[i][j] - maximum[i]) / denominator[i];
                    gp[size_t(row) * seq + key] = probability;
                }
                scores[i][j] = probability;
            }
            *reinterpret_cast<float4 *>(p_tile + (x + kSide * j) * kPitch + 4 * y) =
                make_float4(scores[0][j], scores[1][j], scores[2][j], scores[3][j]);
        }
        __syncthreads();
        tile_update<HD, kPitch>(p_tile, v_tile, x, y, acc);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        store_columns<HD>(out + base, row0 + 4 * y + i, seq, head_dim, x, acc[i], false);
    }
}

// D_i = dO_i . O_i for every attention row; one warp per row.
__global__ void row_dots_kernel(const float *__restrict__ a,
                                const float *__restrict__ b,
                                float *__restrict__ out, size_t rows,
                                int head_dim) {
    const int lane = threadIdx.x & 31;
    const size_t warp = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const size_t warps = (size_t(gridDim.x) * blockDim.x) >> 5;
    for (size_t row = warp; row < rows; row += warps) {
        float sum = 0.0f;
        for (int d = lane; d < head_dim; d += 32) {
            sum += a[row * head_dim + d] * b[row * head_dim + d];
        }
        sum = warp_sum(sum);
        if (lane == 0) {
            out[row] = sum;
        }
    }
}

// The tile's score gradients dS = scale P (dP - D), dP = dO V^T, for rows 4y + i and
// keys x + 16j; P in `probabilities`.
template <int HD>
__device__ __forceinline__ void score_gradients(
    const float *do_tile, const float *v_tile, const float *__restrict__ gp,
    const float *__restrict__ dots, int row0, int key0, int seq, float scale, int x,
    int y, float (&slopes)[4][4], float (&probabilities)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = row0 + 4 * y + i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int key = key0 + x + kSide * j;
            probabilities[i][j] =
                row < seq && key < seq ? __ldg(gp + size_t(row) * seq + key) : 0.0f;
        }
    }
    tile_product<HD>(do_tile, v_tile, x, y, slopes);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = row0 + 4 * y + i;
        const float dot = row < seq ? __ldg(dots + row) : 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool live = row < seq && key0 + x + kSide * j < seq;
            slopes[i][j] =
                live ? scale * probabilities[i][j] * (slopes[i][j] - dot) : 0.0f;
        }
    }
}

template <int HD>
__global__ void __launch_bounds__(kThreads)
attention_backward_query_kernel(const float *__restrict__ k,
                                const float *__restrict__ v,
                                const float *__restrict__ p,
                                const float *__restrict__ dout,
                                const float *__restrict__ row_dots,
                                float *__restrict__ dq, int seq, int head_dim,
                                float scale, bool add_q, bool vec) {
    extern __shared__ __align__(16) float shared[];
    float *do_tile = shared;
    float *v_tile = do_tile + kAcross<HD>;
    float *k_tile = v_tile + kAcross<HD>;
    float *s_tile = k_tile + kAlong<HD>;   // [key][row], pitch kPitch

    const size_t group = blockIdx.x;
    const int row0 = blockIdx.y * kTile;
    const int x = threadIdx.x % kSide, y = threadIdx.x / kSide;
    const size_t base = group * seq * head_dim;
    stage_across<HD, false>(dout + base, do_tile, row0, seq, head_dim, vec);
    float acc[4][kKept<HD>], slopes[4][4], probabilities[4][4];
    clear(acc);
    for (int key0 = 0; key0 < seq; key0 += kTile) {
        __syncthreads();
        stage_across<HD, true>(v + base, v_tile, key0, seq, head_dim, vec);
        stage_along<HD>(k + base, k_tile, key0, seq, head_dim, vec);
        __syncthreads();
        score_gradients<HD>(do_tile, v_tile, p + group * seq * seq,
                            row_dots + group * seq, row0, key0, seq, scale, x, y, slopes,
                            probabilities);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            *reinterpret_cast<float4 *>(s_tile + (x + kSide * j) * kPitch + 4 * y) =
                make_float4(slopes[0][j], slopes[1][j], slopes[2][j], slopes[3][j]);
        }
        __syncthreads();
        tile_update<HD, kPitch>(s_tile, k_tile, x, y, acc);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        store_columns<HD>(dq + base, row0 + 4 * y + i, seq, head_dim, x, acc[i], add_q);
    }
}

template <int HD>
__global__ void __launch_bounds__(kThreads)
attention_backward_key_kernel(const float *__restrict__ q,
                              const float *__restrict__ v,
                              const float *__restrict__ p,
                              const float *__restrict__ dout,
                              const float *__restrict__ row_dots,
                              float *__restrict__ dk, float *__restrict__ dv,
                              int seq, int head_dim, float scale, bool add_k,
                              bool add_v, bool vec) {
    extern __shared__ __align__(16) float shared[];
    float *v_tile = shared;                            // this block's keys
    float *do_across = v_tile + kAcross<HD>;     // current query tile
    float *do_along = do_across + kAcross<HD>;
    float *q_tile = do_along + kAlong<HD>;
    float *p_tile = q_tile + kAlong<HD>;         // [query][key position]
    float *s_tile = p_tile + kTile * kTile;

    const size_t group = blockIdx.x;
    const int key0 = blockIdx.y * kTile;
    const int x = threadIdx.x % kSide, y = threadIdx.x / kSide;
    const size_t base = group * seq * head_dim;
    stage_across<HD, true>(v + base, v_tile, key0, seq, head_dim, vec);
    float acc_k[4][kKept<HD>], acc_v[4][kKept<HD>], slopes[4][4], probabilities[4][4];
    clear(acc_k);
    clear(acc_v);
    for (int query0 = 0; query0 < seq; query0 += kTile) {
        __syncthreads();
        stage_across<HD, false>(dout + base, do_across, query0, seq, head_dim, vec);
        stage_along<HD>(dout + base, do_along, query0, seq, head_dim, vec);
        stage_along<HD>(q + base, q_tile, query0, seq, head_dim, vec);
        __syncthreads();
        score_gradients<HD>(do_across, v_tile, p + group * seq * seq,
                            row_dots + group * seq, query0, key0, seq, scale, x, y,
                            slopes, probabilities);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int at = (4 * y + i) * kTile + 4 * x;
            *reinterpret_cast<float4 *>(p_tile + at) =
                make_float4(probabilities[i][0], probabilities[i][1],
                            probabilities[i][2], probabilities[i][3]);
            *reinterpret_cast<float4 *>(s_tile + at) =
                make_float4(slopes[i][0], slopes[i][1], slopes[i][2], slopes[i][3]);
        }
        __syncthreads();
        tile_update<HD, kTile>(s_tile, q_tile, x, y, acc_k);
        tile_update<HD, kTile>(p_tile, do_along, x, y, acc_v);
    }
    // Positions 4y ... 4y + 3 are the keys y, y + 16, ...
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int key = key0 + y + kSide * i;
        store_columns<HD>(dk + base, key, seq, head_dim, x, acc_k[i], add_k);
        store_columns<HD>(dv + base, key, seq, head_dim, x, acc_v[i], add_v);
    }
}

// 16-byte accesses to rows of head_dim floats.
bool vector_rows(std::initializer_list<const float *> bases, size_t head_dim) {
    for (const float *base : bases) {
        if (reinterpret_cast<uintptr_t>(base) & 15) {
            return false;
        }
    }
    return head_dim % 4 == 0;
}

template <typename Kernel, typename... Args>
void launch(Kernel kernel, size_t groups, size_t seq, size_t floats, cudaStream_t stream,
            SharedMemoryLimit &limit, const Args &...args) {
    const size_t bytes = floats * sizeof(float);
    if (bytes > 48 * 1024) {
        limit.raise(reinterpret_cast<const void *>(kernel), int(bytes));
    }
    const dim3 grid(static_cast<unsigned>(groups),
                    static_cast<unsigned>((seq + kTile - 1) / kTile));
    kernel<<<grid, kThreads, bytes, stream>>>(args...);
    ++g_kernel_launches;
}

template <int HD>
void forward(const float *q, const float *k, const float *v, float *probabilities,
             float *out, size_t groups, size_t seq, size_t head_dim, float scale,
             cudaStream_t stream) {
    static SharedMemoryLimit limit;
    launch(attention_forward_kernel<HD>, groups, seq,
           2 * kAcross<HD> + kAlong<HD> + size_t(kTile) * kPitch, stream,
           limit, q, k, v, probabilities, out, int(seq), int(head_dim), scale,
           vector_rows({q, k, v}, head_dim));
}

template <int HD>
void backward(const float *q, const float *k, const float *v, const float *probabilities,
              const float *dout, const float *row_dots, float *dq, float *dk, float *dv,
              size_t groups, size_t seq, size_t head_dim, float scale, bool add_q,
              bool add_k, bool add_v, cudaStream_t stream) {
    static SharedMemoryLimit query_limit, key_limit;
    const bool vec = vector_rows({q, k, v, dout}, head_dim);
    launch(attention_backward_query_kernel<HD>, groups, seq,
           2 * kAcross<HD> + kAlong<HD> + size_t(kTile) * kPitch, stream,
           query_limit, k, v, probabilities, dout, row_dots, dq, int(seq), int(head_dim),
           scale, add_q, vec);
    launch(attention_backward_key_kernel<HD>, groups, seq,
           2 * kAcross<HD> + 2 * kAlong<HD> + 2 * size_t(kTile) * kTile,
           stream, key_limit, q, v, probabilities, dout, row_dots, dk, dv, int(seq),
           int(head_dim), scale, add_k, add_v, vec);
}

// CALL with the kernels' head dimension: the next of these, zeros beyond head_dim.  (All
// multiples of 16: with 64 and 128 alone, dimensions of 40, 72 and 96 took 1.2, 1.49 and
// 1.25 times what they had taken unpadded, forward.)
#define VITB200_DISPATCH_HD(head_dim, CALL)                                    \
    do {                                                                       \
        if ((head_dim) <= 8) { CALL(8); }                                      \
        else if ((head_dim) <= 16) { CALL(16); }                               \
        else if ((head_dim) <= 32) { CALL(32); }                               \
        else if ((head_dim) <= 48) { CALL(48); }                               \
        else if ((head_dim) <= 64) { CALL(64); }                               \
        else if ((head_dim) <= 80) { CALL(80); }                               \
        else if ((head_dim) <= 96) { CALL(96); }                               \
        else if ((head_dim) <= 112) { CALL(112); }                             \
        else { CALL(128); }                                                    \
    } while (0)

}  // namespace

void launch_attention_forward(const float *q, const float *k, const float *v,
                              float *probabilities, float *out, size_t groups,
                              size_t seq, size_t head_dim, float scale,
                              int precision, cudaStream_t stream) {
    // Short sequences are limited by shared-memory and instruction traffic,
    // not by arithmetic: the FP32 whole-group kernel is as fast there and
    // exact, so tensor cores are used for them only on explicit request.
    const double work = double(groups) * seq * seq * head_dim;
    const bool short_sequence = attention_small_supported(seq, head_dim);
    if (attention_mma_supported(head_dim) &&
        (precision == VITB200_PRECISION_TF32 ||
         (!short_sequence && prefer_tensor_cores(precision, work))) &&
        launch_attention_mma_forward(q, k, v, probabilities, out, groups, seq,
                                     head_dim, scale, stream)) {
        return;
    }
    if (attention_small_supported(seq, head_dim) &&
        launch_attention_small_forward(q, k, v, probabilities, out, groups, seq,
                                       head_dim, scale, true, true, stream)) {
        return;
    }
#define CALL(HD)                                                               \
    forward<HD>(q, k, v, probabilities, out, groups, seq, head_dim, scale, stream)
    VITB200_DISPATCH_HD(head_dim, CALL);
#undef CALL
}

void launch_attention_backward(const float *q, const float *k, const float *v,
                               const float *probabilities, const float *out,
                               const float *dout, float *dq, float *dk,
                               float *dv, float *row_dots, size_t groups,
                               size_t seq, size_t head_dim, float scale,
                               bool add_q, bool add_k, bool add_v,
                               int precision, cudaStream_t stream) {
    const double work = double(groups) * seq * seq * head_dim;
    const bool short_sequence = attention_small_supported(seq, head_dim);
    if (attention_mma_supported(head_dim) &&
        (precision == VITB200_PRECISION_TF32 ||
         (!short_sequence && prefer_tensor_cores(precision, work))) &&
        launch_attention_mma_backward(q, k, v, probabilities, nullptr, out,
                                      dout, dq, dk, dv, row_dots, groups, seq,
                                      head_dim,
                                      scale, add_q, add_k, add_v, stream)) {
        return;
    }
    if (attention_small_supported(seq, head_dim) &&
        launch_attention_small_backward(q, k, v, probabilities, out, dout, dq,
                                        dk, dv, groups, seq, head_dim, scale,
                                        add_q, add_k, add_v, false, stream)) {
        return;
    }
    const size_t rows = groups * seq;
    row_dots_kernel<<<stream_grid(rows * 32), kStreamThreads, 0, stream>>>(
        dout, out, row_dots, rows, int(head_dim));
    ++g_kernel_launches;
#define CALL(HD)                                                               \
    backward<HD>(q, k, v, probabilities, dout, row_dots, dq, dk, dv, groups,   \
                 seq, head_dim, scale, add_q, add_k, add_v, stream)
    VITB200_DISPATCH_HD(head_dim, CALL);
#undef CALL
}

}  // namespace vitb200
