// FP32 attention for short sequences (seq <= 128): one block per (sample, head)
// group with the whole group resident in shared memory, LANES adjacent lanes
// per row.
//
// With 50 tokens and 16-wide heads a group is 9.6 KB of Q/K/V and a 10 KB
// probability matrix, so everything is read from HBM once, the scores never
// leave the SM before they are normalised, and P is written back with fully
// coalesced stores (the host keeps P as a tensor; reference
// src/ops.c:1297-1355).
//
// What bounds these kernels at the sizes that reach them (a batch too small for
// the tensor-core policy, i.e. a few blocks per SM) is the serial chain of one
// row: seq dot products, seq exponentials, seq row updates.  LANES lanes take
// every LANES-th key of a row each and meet in shuffles; the partial rows of the
// updates are summed while they are scattered over the lanes
// (reduce_scatter), so that every lane stores HD / LANES values.  Tile rows are
// padded by four floats, which puts the LANES rows that a warp reads at a time
// into different banks.
//
// Backward (reference src/ops.c:1381-1441):
//   rows     P_ij (rebuilt or loaded), dS_ij = scale P_ij (dO_i.V_j - dO_i.O_i),
//            dQ_i = sum_j dS_ij K_j
//   columns  dV_j = sum_i P_ij dO_i,  dK_j = sum_i dS_ij Q_i
// with P and dS in tiles of their own.  Where these do not fit (64-wide heads), and
// with one lane per row, where more resident blocks are worth more than the
// barriers, dS replaces P after dV is done.
#include "kernels.h"
#include "device_util.cuh"

#include <cfloat>

namespace vitb200 {
namespace {

// Floats between the rows of a shared tile.
template <int HD>
constexpr int kTilePitch = HD + 4;

// Cooperative copy of a [rows, HD] block whose rows are `ld` floats apart into
// a padded shared-memory tile.
template <int HD>
__device__ __forceinline__ void load_rows(const float *__restrict__ source,
                                          float *tile, int rows, int ld) {
    constexpr int kPerRow = HD / 4;
    const int vectors = rows * kPerRow;
    for (int i = threadIdx.x; i < vectors; i += blockDim.x) {
        const int row = i / kPerRow, chunk = i % kPerRow;
        reinterpret_cast<float4 *>(tile + row * kTilePitch<HD>)[chunk] =
            __ldcs(reinterpret_cast<const float4 *>(source + size_t(row) * ld) + chunk);
    }
}

// Offset of a group's first row under a layout (see HeadLayout).
template <int HD>
__device__ __forceinline__ size_t group_offset(size_t group, int seq,
                                               HeadLayout layout) {
    return (group / layout.heads) * size_t(seq) * layout.ld +
           (group % layout.heads) * HD;
}

// Packed FP32 arithmetic: Blackwell issues two FP32 FMAs per instruction on
// register pairs (fma.rn.f32x2), which halves the instruction count of the
// short dot products and row updates below.  Rows live in registers as HD/2
// packed pairs.
typedef unsigned long long pair_t;

__device__ __forceinline__ pair_t pack(float lo, float hi) {
    pair_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}

__device__ __forceinline__ void unpack(pair_t p, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}

__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
    pair_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// row . tile_row; the tile row is read with 128-bit shared-memory loads.
template <int HD>
__device__ __forceinline__ float dot_tile(const pair_t (&row)[HD / 2],
                                          const float *tile_row) {
    const float4 *t = reinterpret_cast<const float4 *>(tile_row);
    pair_t even = pack(0.0f, 0.0f), odd = pack(0.0f, 0.0f);
#pragma unroll
    for (int c = 0; c < HD / 4; ++c) {
        const float4 x = t[c];
        even = fma2(row[2 * c], pack(x.x, x.y), even);
        odd = fma2(row[2 * c + 1], pack(x.z, x.w), odd);
    }
    float a, b, d, e;
    unpack(even, a, b);
    unpack(odd, d, e);
    return (a + b) + (d + e);
}

// row += a * tile_row.
template <int HD>
__device__ __forceinline__ void axpy_tile(pair_t (&row)[HD / 2], float a,
                                          const float *tile_row) {
    const float4 *t = reinterpret_cast<const float4 *>(tile_row);
    const pair_t a2 = pack(a, a);
#pragma unroll
    for (int c = 0; c < HD / 4; ++c) {
        const float4 x = t[c];
        row[2 * c] = fma2(a2, pack(x.x, x.y), row[2 * c]);
        row[2 * c + 1] = fma2(a2, pack(x.z, x.w), row[2 * c + 1]);
    }
}

template <int HD>
__device__ __forceinline__ void clear_row(pair_t (&row)[HD / 2]) {
#pragma unroll
    for (int c = 0; c < HD / 2; ++c) {
        row[c] = pack(0.0f, 0.0f);
    }
}

// Loads a row of HD floats (global or shared) into packed registers.
template <int HD>
__device__ __forceinline__ void load_row_pairs(pair_t (&row)[HD / 2],
                                               const float *source) {
    const float4 *t = reinterpret_cast<const float4 *>(source);
#pragma unroll
    for (int c = 0; c < HD / 4; ++c) {
        const float4 x = t[c];
        row[2 * c] = pack(x.x, x.y);
        row[2 * c + 1] = pack(x.z, x.w);
    }
}

// Sums the rows of LANES adjacent lanes; lane `part` of them is left with the
// HD / LANES sums from column part * HD / LANES on.
template <int HD, int LANES>
__device__ __forceinline__ void reduce_scatter(const pair_t (&row)[HD / 2], int part,
                                               float (&sums)[HD / LANES]) {
    float values[HD];
#pragma unroll
    for (int c = 0; c < HD / 2; ++c) {
        unpack(row[c], values[2 * c], values[2 * c + 1]);
    }
    int count = HD / 2;
#pragma unroll
    for (int distance = LANES / 2; distance > 0; distance /= 2, count /= 2) {
        const bool upper = (part & distance) != 0;
#pragma unroll
        for (int i = 0; i < HD / 2; ++i) {
            if (i < count) {
                const float low = values[i], high = values[i + count];
                const float sent = upper ? low : high;
                values[i] = (upper ? high : low) +
                            __shfl_xor_sync(kFullMask, sent, distance);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < HD / LANES; ++i) {
        sums[i] = values[i];
    }
}

// target (+)= the COUNT values of one lane (reduce_scatter), in accesses as wide
// as they are contiguous; `target` is the row's start.
template <int COUNT>
__device__ __forceinline__ void store_part(float *target, int part,
                                           const float (&values)[COUNT], bool add) {
    target += part * COUNT;
    if constexpr (COUNT >= 4) {
#pragma unroll
        for (int c = 0; c < COUNT / 4; ++c) {
            float4 *t = reinterpret_cast<float4 *>(target) + c;
            float4 v = add ? *t : make_float4(0.f, 0.f, 0.f, 0.f);
            v.x += values[4 * c]; v.y += values[4 * c + 1];
            v.z += values[4 * c + 2]; v.w += values[4 * c + 3];
            *t = v;
        }
    } else if constexpr (COUNT == 2) {
        float2 *t = reinterpret_cast<float2 *>(target);
        float2 v = add ? *t : make_float2(0.f, 0.f);
        v.x += values[0]; v.y += values[1];
        *t = v;
    } else {
        *target = (add ? *target : 0.0f) + values[0];
    }
}

// The sum, or the maximum, over LANES adjacent lanes.
template <int LANES>
__device__ __forceinline__ float lanes_sum(float value) {
#pragma unroll
    for (int distance = LANES / 2; distance > 0; distance /= 2) {
        value += __shfl_xor_sync(kFullMask, value, distance);
    }
    return value;
}

template <int LANES>
__device__ __forceinline__ float lanes_max(float value) {
#pragma unroll
    for (int distance = LANES / 2; distance > 0; distance /= 2) {
        value = fmaxf(value, __shfl_xor_sync(kFullMask, value, distance));
    }
    return value;
}

// Adds one lane's COUNT values, over all rows of the block (the live ones), to the
// column sums of its head; `columns` is in shared memory.
template <int COUNT, int LANES>
__device__ __forceinline__ void add_columns(float *columns, int part,
                                            const float (&values)[COUNT], bool live) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
        float sum = live ? values[i] : 0.0f;
#pragma unroll
        for (int distance = 16; distance >= LANES; distance /= 2) {
            sum += __shfl_xor_sync(kFullMask, sum, distance);
        }
        if ((threadIdx.x & 31) < LANES) {
            atomicAdd(columns + part * COUNT + i, sum);
        }
    }
}

// exp for softmax arguments (<= 0 after subtracting the row maximum):
// ex2.approx on x * log2(e), relative error about 2e-7 in this range.
__device__ __forceinline__ float softmax_exp(float x) {
    return __expf(x);
}

// Copies the group's [seq, seq] probability block between global memory
// (contiguous rows) and the padded shared tile, one row per warp at a time.
template <bool kToGlobal>
__device__ __forceinline__ void move_probabilities(float *global_block,
                                                   float *tile, int seq,
                                                   int pitch) {
    const int lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    for (int r = threadIdx.x >> 5; r < seq; r += warps) {
        for (int c = lane; c < seq; c += 32) {
            if (kToGlobal) {
                global_block[r * seq + c] = tile[r * pitch + c];
            } else {
                tile[r * pitch + c] = __ldcs(global_block + r * seq + c);
            }
        }
    }
}

// This lane's share (keys part, part + LANES, ...) of a row of P: the scores of
// `query` into scores[], then their exponentials.  Returns 1 / the row's sum.
// Nothing is stored when the row is not `live` (lanes past the last row).
template <int HD, int LANES>
__device__ __forceinline__ float softmax_row(const pair_t (&query)[HD / 2],
                                             const float *k_tile, float *scores,
                                             int part, int seq, float scale,
                                             bool live) {
    float maximum = -FLT_MAX;
#pragma unroll 4
    for (int j = part; j < seq; j += LANES) {
        const float dot = scale * dot_tile<HD>(query, k_tile + j * kTilePitch<HD>);
        if (live) {
            scores[j] = dot;
        }
        maximum = fmaxf(maximum, dot);
    }
    maximum = lanes_max<LANES>(maximum);
    float denominator = 0.0f;
#pragma unroll 4
    for (int j = part; j < seq; j += LANES) {
        const float e = softmax_exp(scores[j] - maximum);
        if (live) {
            scores[j] = e;
        }
        denominator += e;
    }
    return 1.0f / lanes_sum<LANES>(denominator);
}

// At most 128 rows x 4 lanes.
constexpr int kMaxThreads = 512;

template <int HD, int LANES>
__global__ void __launch_bounds__(HD == 64 ? kMaxThreads / 2 : kMaxThreads)
attention_small_forward_kernel(
    const float *__restrict__ q, const float *__restrict__ k,
    const float *__restrict__ v, float *__restrict__ p, float *__restrict__ out,
    int seq, float scale, bool write_p, bool write_o, HeadLayout in_layout,
    HeadLayout out_layout) {
    extern __shared__ __align__(16) float shared[];
    constexpr int kPitch = kTilePitch<HD>;
    const int pitch = seq | 1;
    float *k_tile = shared;
    float *v_tile = k_tile + seq * kPitch;
    float *p_tile = v_tile + seq * kPitch;
    const size_t group = blockIdx.x;
    const size_t base = group_offset<HD>(group, seq, in_layout);
    const int part = threadIdx.x % LANES;
    const bool live = threadIdx.x / LANES < seq;
    const int row = min(int(threadIdx.x) / LANES, seq - 1);
    grid_dependency_wait();
    grid_dependency_release();
    load_rows<HD>(k + base, k_tile, seq, in_layout.ld);
    load_rows<HD>(v + base, v_tile, seq, in_layout.ld);
    pair_t query[HD / 2];
    load_row_pairs<HD>(query, q + base + size_t(row) * in_layout.ld);
    __syncthreads();
    float *scores = p_tile + row * pitch;
    const float inverse =
        softmax_row<HD, LANES>(query, k_tile, scores, part, seq, scale, live);
    pair_t result[HD / 2];
    clear_row<HD>(result);
#pragma unroll 4
    for (int j = part; j < seq; j += LANES) {
        const float probability = scores[j] * inverse;
        if (write_p && live) {
            scores[j] = probability;
        }
        axpy_tile<HD>(result, probability, v_tile + j * kPitch);
    }
    float sums[HD / LANES];
    reduce_scatter<HD, LANES>(result, part, sums);
    if (write_o && live) {
        store_part<HD / LANES>(out + group_offset<HD>(group, seq, out_layout) +
                                   size_t(row) * out_layout.ld,
                               part, sums, false);
    }
    if (write_p) {
        __syncthreads();
        move_probabilities<true>(p + group * seq * seq, p_tile, seq, pitch);
    }
}

template <int HD, int LANES>
__global__ void __launch_bounds__(HD == 64 ? kMaxThreads / 2 : kMaxThreads)
attention_small_backward_kernel(
    const float *__restrict__ q, const float *__restrict__ k,
    const float *__restrict__ v, const float *__restrict__ p,
    const float *__restrict__ out, const float *__restrict__ dout,
    float *__restrict__ dq, float *__restrict__ dk, float *__restrict__ dv,
    int seq, float scale, bool add_q, bool add_k, bool add_v, bool recompute,
    HeadLayout in_layout, HeadLayout out_layout, HeadLayout dout_layout,
    HeadLayout grad_layout, float *__restrict__ column_partials) {
    extern __shared__ __align__(16) float shared[];
    constexpr int kPitch = kTilePitch<HD>;
    constexpr bool kTwoTiles = HD < 64 && LANES > 1;   // P and dS side by side,
                                                       // as two_score_tiles()
    const int pitch = seq | 1;
    float *q_tile = shared;
    float *k_tile = q_tile + seq * kPitch;
    float *v_tile = k_tile + seq * kPitch;
    float *do_tile = v_tile + seq * kPitch;
    float *p_tile = do_tile + seq * kPitch;
    float *ds_tile = kTwoTiles ? p_tile + seq * pitch : p_tile;
    // Column sums of this head's dQ, dK and dV, where they are wanted: the QKV bias
    // gradient then reads one row per sample instead of the whole projected gradient
    // in a launch of its own.  (Part of the dynamic allocation, so that fit_shared sees
    // all that a launch takes.)
    float *columns = ds_tile + seq * pitch;
    const size_t group = blockIdx.x;
    const size_t base = group_offset<HD>(group, seq, in_layout);
    const int part = threadIdx.x % LANES;
    const bool live = threadIdx.x / LANES < seq;
    const int row = min(int(threadIdx.x) / LANES, seq - 1);
    for (int c = threadIdx.x; c < 3 * HD; c += blockDim.x) {
        columns[c] = 0.0f;
    }
    grid_dependency_wait();
    grid_dependency_release();
    load_rows<HD>(q + base, q_tile, seq, in_layout.ld);
    load_rows<HD>(k + base, k_tile, seq, in_layout.ld);
    load_rows<HD>(v + base, v_tile, seq, in_layout.ld);
    load_rows<HD>(dout + group_offset<HD>(group, seq, dout_layout), do_tile,
                  seq, dout_layout.ld);
    if (!recompute) {
        move_probabilities<false>(const_cast<float *>(p) + group * seq * seq,
                                  p_tile, seq, pitch);
    }
    const float *out_row = out + group_offset<HD>(group, seq, out_layout) +
                           size_t(row) * out_layout.ld;
    const float *dout_row = dout + group_offset<HD>(group, seq, dout_layout) +
                            size_t(row) * dout_layout.ld;
    float row_dot = 0.0f;
#pragma unroll
    for (int d = 4 * part; d < HD; d += 4 * LANES) {
        const float4 o = __ldcs(reinterpret_cast<const float4 *>(out_row + d));
        const float4 g = __ldcs(reinterpret_cast<const float4 *>(dout_row + d));
        row_dot += (o.x * g.x + o.y * g.y) + (o.z * g.z + o.w * g.w);
    }
    row_dot = lanes_sum<LANES>(row_dot);
    __syncthreads();
    float *probabilities = p_tile + row * pitch;
    if (recompute) {
        // The forward pass did not store P: rebuild this row of it from Q and
        // K with the forward kernel's arithmetic (same order, same rounding).
        pair_t query[HD / 2];
        load_row_pairs<HD>(query, q_tile + row * kPitch);
        const float inverse = softmax_row<HD, LANES>(query, k_tile, probabilities,
                                                     part, seq, scale, live);
        if (live) {
#pragma unroll 4
            for (int j = part; j < seq; j += LANES) {
                probabilities[j] *= inverse;
            }
        }
    }
    const size_t grad_row = group_offset<HD>(group, seq, grad_layout) +
                            size_t(row) * grad_layout.ld;
    float sums[HD / LANES];
    // sum_i weights_i,row source_i, scattered over the row's lanes.
    auto column = [&](const float *weights, const float *source) {
        pair_t acc[HD / 2];
        clear_row<HD>(acc);
#pragma unroll 4
        for (int i = part; i < seq; i += LANES) {
            axpy_tile<HD>(acc, weights[i * pitch + row], source + i * kPitch);
        }
        reduce_scatter<HD, LANES>(acc, part, sums);
    };
    if (!kTwoTiles) {
        // Columns: dV_j = sum_i P_ij dO_i, before dS takes the place of P.
        __syncthreads();
        column(p_tile, do_tile);
        if (live) {
            store_part<HD / LANES>(dv + grad_row, part, sums, add_v);
        }
        if (column_partials) {
            add_columns<HD / LANES, LANES>(columns + 2 * HD, part, sums, live);
        }
        __syncthreads();
    }
    // Rows: score gradients, then dQ_i.  (Every lane meets only its own keys.)
    {
        pair_t g[HD / 2], acc[HD / 2];
        load_row_pairs<HD>(g, do_tile + row * kPitch);
        clear_row<HD>(acc);
        float *slopes = ds_tile + row * pitch;
#pragma unroll 4
        for (int j = part; j < seq; j += LANES) {
            const float dp = dot_tile<HD>(g, v_tile + j * kPitch);
            const float ds = scale * probabilities[j] * (dp - row_dot);
            if (live) {
                slopes[j] = ds;
            }
            axpy_tile<HD>(acc, ds, k_tile + j * kPitch);
        }
        reduce_scatter<HD, LANES>(acc, part, sums);
        if (live) {
            store_part<HD / LANES>(dq + grad_row, part, sums, add_q);
        }
        if (column_partials) {
            add_columns<HD / LANES, LANES>(columns, part, sums, live);
        }
    }
    __syncthreads();
    // Columns: dV_j (unless done), dK_j = sum_i dS_ij Q_i.
    if (kTwoTiles) {
        column(p_tile, do_tile);
        if (live) {
            store_part<HD / LANES>(dv + grad_row, part, sums, add_v);
        }
        if (column_partials) {
            add_columns<HD / LANES, LANES>(columns + 2 * HD, part, sums, live);
        }
    }
    column(ds_tile, q_tile);
    if (live) {
        store_part<HD / LANES>(dk + grad_row, part, sums, add_k);
    }
    if (column_partials) {
        add_columns<HD / LANES, LANES>(columns + HD, part, sums, live);
    }
    if (column_partials) {
        // A row per sample: the columns of the projected gradient it belongs to.
        __syncthreads();
        const size_t heads = size_t(grad_layout.heads);
        float *to = column_partials + group / heads * (3 * heads * HD) +
                    group % heads * HD;
        for (int c = threadIdx.x; c < 3 * HD; c += blockDim.x) {
            to[c / HD * (heads * HD) + c % HD] = columns[c];
        }
    }
}

// Every byte that a launch takes is dynamic (no kernel here has static shared memory):
// up to 48 KiB of it are open to any launch.
template <typename Kernel>
bool fit_shared(Kernel kernel, size_t bytes) {
    if (bytes > 226 * 1024) {
        return false;
    }
    if (bytes > 48 * 1024) {
        return cudaFuncSetAttribute(kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int(bytes)) == cudaSuccess;
    }
    return true;
}

// {0, x} stands for "stored group by group".
HeadLayout resolve_layout(HeadLayout layout, size_t head_dim) {
    return layout.ld ? layout : HeadLayout{int(head_dim), 1};
}

}  // namespace

bool attention_small_supported(size_t seq, size_t head_dim) {
    return seq <= 128 &&
           (head_dim == 8 || head_dim == 16 || head_dim == 32 || head_dim == 64);
}

#define VITB200_DISPATCH(head_dim, lanes, CALL)                                \
    switch (head_dim) {                                                        \
        case 8:                                                                \
            if (lanes == 4) { CALL(8, 4); }                                    \
            else if (lanes == 2) { CALL(8, 2); }                               \
            else { CALL(8, 1); }                                               \
            break;                                                             \
        case 16: if (lanes == 4) { CALL(16, 4); } else { CALL(16, 2); } break; \
        case 32: if (lanes == 4) { CALL(32, 4); } else { CALL(32, 2); } break; \
        default: CALL(64, 2); break;                                           \
    }

namespace {

// Lanes per row.  With a block or less per SM the row's chain is what takes the
// time: four (50 tokens, 16-wide heads, 8 groups: forward 12.2 us with one lane,
// 5.6 with two, 4.6 with four, 4.5 with eight; backward 16.5, 10.5, 9.1, 9.0).
// With more groups the SM's issue slots are, and shuffles and half-used lanes
// cost: two (256 groups: backward 17.5, 12.7, 13.3; 2048 groups: forward 30.9,
// 22.7, 31.3, backward 54.2, 55.3, 73.5).  A row of eight floats is too short
// to be worth even that once the blocks take turns (4096 groups: forward 24.9,
// 28.0, backward 56.1, 63.0; 1024 groups still 9.1, 8.8 and 18.0, 17.8).
int row_lanes(size_t groups, size_t head_dim) {
    const size_t processors = device_sm_count();
    if (head_dim == 64) {
        return 2;   // registers
    }
    if (groups <= processors) {
        return 4;
    }
    return head_dim == 8 && groups > 8 * processors ? 1 : 2;
}

// Whether the backward kernel holds P and dS side by side.
bool two_score_tiles(size_t head_dim, int lanes) {
    return head_dim < 64 && lanes > 1;
}

unsigned block_threads(size_t seq, int lanes) {
    return unsigned((seq * lanes + 31) / 32 * 32);
}

}  // namespace

bool launch_attention_small_forward(const float *q, const float *k,
                                    const float *v, float *probabilities,
                                    float *out, size_t groups, size_t seq,
                                    size_t head_dim, float scale, bool write_p,
                                    bool write_o, cudaStream_t stream,
                                    HeadLayout in_layout,
                                    HeadLayout out_layout) {
    in_layout = resolve_layout(in_layout, head_dim);
    out_layout = resolve_layout(out_layout, head_dim);
    const int lanes = row_lanes(groups, head_dim);
    const size_t bytes =
        (2 * seq * (head_dim + 4) + seq * (seq | 1)) * sizeof(float);
    bool launched = false;
#define CALL(HD, LANES)                                                        \
    if (fit_shared(attention_small_forward_kernel<HD, LANES>, bytes)) {        \
        launched = launch_chained(attention_small_forward_kernel<HD, LANES>,   \
                                  unsigned(groups), block_threads(seq, LANES), \
                                  bytes, stream, q, k, v, probabilities, out,  \
                                  int(seq), scale, write_p, write_o,           \
                                  in_layout, out_layout) == cudaSuccess;       \
    }
    VITB200_DISPATCH(head_dim, lanes, CALL)
#undef CALL
    g_kernel_launches += launched ? 1 : 0;
    return launched;
}

bool launch_attention_small_backward(const float *q, const float *k,
                                     const float *v, const float *probabilities,
                                     const float *out, const float *dout,
                                     float *dq, float *dk, float *dv,
                                     size_t groups, size_t seq, size_t head_dim,
                                     float scale, bool add_q, bool add_k,
                                     bool add_v, bool recompute,
                                     cudaStream_t stream, HeadLayout in_layout,
                                     HeadLayout out_layout,
                                     HeadLayout dout_layout,
                                     HeadLayout grad_layout,
                                     float *column_partials) {
    in_layout = resolve_layout(in_layout, head_dim);
    out_layout = resolve_layout(out_layout, head_dim);
    dout_layout = resolve_layout(dout_layout, head_dim);
    grad_layout = resolve_layout(grad_layout, head_dim);
    const int lanes = row_lanes(groups, head_dim);
    const size_t score_tiles = two_score_tiles(head_dim, lanes) ? 2 : 1;
    const size_t bytes = (4 * seq * (head_dim + 4) + score_tiles * seq * (seq | 1) +
                          3 * head_dim) *
                         sizeof(float);
    bool launched = false;
#define CALL(HD, LANES)                                                        \
    if (fit_shared(attention_small_backward_kernel<HD, LANES>, bytes)) {       \
        launched =                                                             \
            launch_chained(attention_small_backward_kernel<HD, LANES>,         \
                           unsigned(groups), block_threads(seq, LANES), bytes, \
                           stream, q, k, v, probabilities, out, dout, dq, dk,  \
                           dv, int(seq), scale, add_q, add_k, add_v,           \
                           recompute, in_layout, out_layout, dout_layout,      \
                           grad_layout, column_partials) == cudaSuccess;       \
    }
    VITB200_DISPATCH(head_dim, lanes, CALL)
#undef CALL
    g_kernel_launches += launched ? 1 : 0;
    return launched;
}

}  // namespace vitb200
