// Row operators of the decoder graph: embeddings (with and without learned positions), the norms of the F32
// residual stream and of what is added to it, the activations of the feed-forwards, and the F32 projection of
// the F32 profile.
#include <cooperative_groups.h>

#include <type_traits>

#include "linear_f32.cuh"
#include "ops_internal.hpp"

namespace cg = cooperative_groups;

namespace evob {
namespace {

constexpr int kThreads = 256;
constexpr int kCached = 4;  // groups of eight elements a thread keeps between the two sweeps over its row

// One row as groups of eight: thread t owns groups t, t + kThreads, ...  The first kCached of them stay in
// registers between the statistics and the output sweep (rows of up to 8,192 elements read memory once).
template <typename Load, typename Store>
__device__ __forceinline__ void two_sweeps(const int groups, const Load &load, const Store &store,
                                           float *const scratch, const float inverse_width, const float epsilon) {
  float cached[kCached][8];
  float square = 0.0F;
#pragma unroll
  for (int c = 0; c < kCached; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) {
      load(group, cached[c]);
#pragma unroll
      for (int i = 0; i < 8; ++i) square = fmaf(cached[c][i], cached[c][i], square);
    }
  }
  for (int group = threadIdx.x + kCached * kThreads; group < groups; group += kThreads) {
    float v[8];
    load(group, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) square = fmaf(v[i], v[i], square);
  }
  const float total = block_sum<kThreads>(square, scratch);
  const float factor = 1.0F / sqrtf(total * inverse_width + epsilon);
#pragma unroll
  for (int c = 0; c < kCached; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) store(group, cached[c], factor);
  }
  for (int group = threadIdx.x + kCached * kThreads; group < groups; group += kThreads) {
    float v[8];
    load(group, v);
    store(group, v, factor);
  }
}

// kVector: width % 8 == 0 and 16-byte aligned rows.  Otherwise groups of eight with a ragged last one.
template <typename T, bool kVector>
__device__ __forceinline__ void load_group(const T *const row, const int group, const int width, float (&v)[8]) {
  if constexpr (kVector) {
    load_floats<8>(row + 8 * group, v);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 8 * group + i < width ? to_float(row[8 * group + i]) : 0.0F;
  }
}
template <typename T, bool kVector>
__device__ __forceinline__ void store_group(T *const row, const int group, const int width, const float (&v)[8]) {
  if constexpr (kVector) {
    store_floats(row + 8 * group, v);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (8 * group + i < width) row[8 * group + i] = from_float<T>(v[i]);
  }
}

template <bool kVector>
__global__ void __launch_bounds__(kThreads)
embed_positions_kernel(const std::uint32_t *__restrict__ tokens, const bf16 *__restrict__ table,
                       const bf16 *__restrict__ positions, const float *__restrict__ gain, const int width,
                       const std::uint32_t vocabulary, const int position, const int *__restrict__ dynamic_position,
                       const float epsilon, float *__restrict__ output, int *const error_word) {
  wait_for_producers(tokens, table, positions, gain, dynamic_position);
  release_dependents();
  __shared__ float scratch[kThreads / 32];
  const std::size_t row = blockIdx.x;
  const std::uint32_t token = tokens[row];
  float *const out = output + row * width;
  if (token >= vocabulary) {
    for (int i = threadIdx.x; i < width; i += kThreads) out[i] = 0.0F;
    if (threadIdx.x == 0) atomicOr(error_word, 2);
    return;
  }
  const std::size_t at = (dynamic_position != nullptr ? *dynamic_position : position) + row;
  const bf16 *const word = table + static_cast<std::size_t>(token) * width;
  const bf16 *const place = positions + at * width;
  two_sweeps(
      (width + 7) / 8,
      [&](const int group, float (&v)[8]) {
        float p[8];
        load_group<bf16, kVector>(word, group, width, v);
        load_group<bf16, kVector>(place, group, width, p);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += p[i];
      },
      [&](const int group, const float (&v)[8], const float factor) {
        float g[8], y[8];
        load_group<float, kVector>(gain, group, width, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = v[i] * factor * g[i];
        store_group<float, kVector>(out, group, width, y);
      },
      scratch, 1.0F / static_cast<float>(width), epsilon);
}

template <typename T, bool kVector>
__global__ void __launch_bounds__(kThreads)
rms_norm_residual_kernel(const float *__restrict__ input, const float *__restrict__ gain, const int width,
                         const float epsilon, T *__restrict__ output) {
  wait_for_producers(input, gain);
  release_dependents();
  __shared__ float scratch[kThreads / 32];
  const float *const x = input + static_cast<std::size_t>(blockIdx.x) * width;
  T *const out = output + static_cast<std::size_t>(blockIdx.x) * width;
  two_sweeps(
      (width + 7) / 8, [&](const int group, float (&v)[8]) { load_group<float, kVector>(x, group, width, v); },
      [&](const int group, const float (&v)[8], const float factor) {
        float g[8], y[8];
        load_group<float, kVector>(gain, group, width, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = v[i] * factor * g[i];
        store_group<T, kVector>(out, group, width, y);
      },
      scratch, 1.0F / static_cast<float>(width), epsilon);
}

template <typename T, bool kVector>
__global__ void __launch_bounds__(kThreads)
poly_norm_kernel(const T *input, const float *__restrict__ coefficients, const int width, const float epsilon,
                 T *output) {
  wait_for_producers(input, coefficients, output);
  release_dependents();
  __shared__ float scratch[kThreads / 32];
  const T *const z = input + static_cast<std::size_t>(blockIdx.x) * width;
  T *const out = output + static_cast<std::size_t>(blockIdx.x) * width;
  const int groups = (width + 7) / 8;
  constexpr int kKept = kCached;
  float cached[kKept][8];
  float second = 0.0F, fourth = 0.0F, sixth = 0.0F;  // sums of z^2, z^4, z^6
  const auto add = [&](const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = v[i] * v[i];
      second += s;
      fourth = fmaf(s, s, fourth);
      sixth = fmaf(s * s, s, sixth);
    }
  };
#pragma unroll
  for (int c = 0; c < kKept; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) {
      load_group<T, kVector>(z, group, width, cached[c]);
      add(cached[c]);
    }
  }
  for (int group = threadIdx.x + kKept * kThreads; group < groups; group += kThreads) {
    float v[8];
    load_group<T, kVector>(z, group, width, v);
    add(v);
  }
  const float inverse_width = 1.0F / static_cast<float>(width);
  second = block_sum<kThreads>(second, scratch);
  fourth = block_sum<kThreads>(fourth, scratch);
  sixth = block_sum<kThreads>(sixth, scratch);
  const float a = coefficients[0] * rsqrtf(second * inverse_width + epsilon);
  const float b = coefficients[1] * rsqrtf(fourth * inverse_width + epsilon);
  const float c3 = coefficients[2] * rsqrtf(sixth * inverse_width + epsilon);
  const float e = coefficients[3];
  const auto emit = [&](const int group, const float (&v)[8]) {
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = fmaf(fmaf(fmaf(c3, v[i], b), v[i], a), v[i], e);
    store_group<T, kVector>(out, group, width, y);
  };
#pragma unroll
  for (int c = 0; c < kKept; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) emit(group, cached[c]);
  }
  for (int group = threadIdx.x + kKept * kThreads; group < groups; group += kThreads) {
    float v[8];
    load_group<T, kVector>(z, group, width, v);
    emit(group, v);
  }
}

__global__ void __launch_bounds__(kThreads)
distance_bias_kernel(const float *__restrict__ r1, const float *__restrict__ r2, const int distances,
                     float *__restrict__ table) {
  const int head = blockIdx.y;
  for (int d = blockIdx.x * kThreads + threadIdx.x; d < distances; d += gridDim.x * kThreads)
    table[static_cast<std::size_t>(head) * distances + d] = r1[head] * logf(fmaf(r2[head], static_cast<float>(d), 1.0F));
}

template <typename T, bool kVector>
__global__ void __launch_bounds__(kThreads)
embed_rows_kernel(const std::uint32_t *__restrict__ tokens, const bf16 *__restrict__ table, const int width,
                  const std::uint32_t vocabulary, float *__restrict__ stream_rows, T *__restrict__ copy,
                  int *const error_word) {
  wait_for_producers(tokens, table);
  release_dependents();
  const std::size_t row = blockIdx.x;
  const std::uint32_t token = tokens[row];
  const bool known = token < vocabulary;
  if (!known && threadIdx.x == 0) atomicOr(error_word, 2);
  const bf16 *const word = table + static_cast<std::size_t>(known ? token : 0U) * width;
  for (int group = threadIdx.x; group < (width + 7) / 8; group += kThreads) {
    float v[8];
    load_group<bf16, kVector>(word, group, width, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = known ? v[i] : 0.0F;
    store_group<float, kVector>(stream_rows + row * width, group, width, v);
    if (copy != nullptr) store_group<T, kVector>(copy + row * width, group, width, v);
  }
}

struct LayerNormParams {
  const int *slots;
  int parts;
  const float *gain;
  float *residual;
  int width;
  float epsilon;
};

// Mean and variance from the row itself (two sweeps over registers), one read and one write of the residual.  A
// thread keeps kKeep groups of eight elements between the sweeps.
template <typename In, typename Out, bool kVector, int kKeep>
__global__ void __launch_bounds__(kThreads)
layer_norm_kernel(const In *__restrict__ input, Out *__restrict__ output, const LayerNormParams p) {
  wait_for_producers(input);
  release_dependents();
  __shared__ float scratch[kThreads / 32];
  const std::size_t row = blockIdx.x;
  const int groups = (p.width + 7) / 8;
  const float inverse_width = 1.0F / static_cast<float>(p.width);
  const auto load = [&](const int group, float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0F;
    for (int k = 0; k < p.parts; ++k) {
      const std::size_t pair = row * p.parts + k;
      const std::size_t at = p.slots != nullptr ? static_cast<std::size_t>(p.slots[pair]) : pair;
      float w[8];
      load_group<In, kVector>(input + at * p.width, group, p.width, w);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] += w[i];
    }
  };
  const auto live = [&](const int group, const int i) { return kVector || 8 * group + i < p.width; };
  float cached[kKeep][8], old[kKeep][8];
  float sum = 0.0F;
#pragma unroll
  for (int c = 0; c < kKeep; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) {
      load(group, cached[c]);
      if (p.residual != nullptr) load_group<float, kVector>(p.residual + row * p.width, group, p.width, old[c]);
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += cached[c][i];
    }
  }
  for (int group = threadIdx.x + kKeep * kThreads; group < groups; group += kThreads) {
    float v[8];
    load(group, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) sum += v[i];
  }
  const float mean = block_sum<kThreads>(sum, scratch) * inverse_width;
  float square = 0.0F;
  const auto deviate = [&](const int group, const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float d = live(group, i) ? v[i] - mean : 0.0F;
      square = fmaf(d, d, square);
    }
  };
#pragma unroll
  for (int c = 0; c < kKeep; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) deviate(group, cached[c]);
  }
  for (int group = threadIdx.x + kKeep * kThreads; group < groups; group += kThreads) {
    float v[8];
    load(group, v);
    deviate(group, v);
  }
  const float factor = 1.0F / sqrtf(block_sum<kThreads>(square, scratch) * inverse_width + p.epsilon);
  const auto emit = [&](const int group, const float (&v)[8], const float (&before)[8]) {
    float g[8], y[8];
    load_group<float, kVector>(p.gain, group, p.width, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = (v[i] - mean) * factor * g[i];
    if (p.residual != nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] += before[i];
      store_group<float, kVector>(p.residual + row * p.width, group, p.width, y);
    }
    if (output != nullptr) store_group<Out, kVector>(output + row * p.width, group, p.width, y);
  };
#pragma unroll
  for (int c = 0; c < kKeep; ++c) {
    const int group = threadIdx.x + c * kThreads;
    if (group < groups) emit(group, cached[c], old[c]);
  }
  for (int group = threadIdx.x + kKeep * kThreads; group < groups; group += kThreads) {
    float v[8], before[8] = {};
    load(group, v);
    if (p.residual != nullptr) load_group<float, kVector>(p.residual + row * p.width, group, p.width, before);
    emit(group, v, before);
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
convert_kernel(const float *__restrict__ input, T *__restrict__ output, const std::size_t elements) {
  const std::size_t stride = static_cast<std::size_t>(gridDim.x) * kThreads;
  for (std::size_t i = static_cast<std::size_t>(blockIdx.x) * kThreads + threadIdx.x; i < elements; i += stride)
    output[i] = from_float<T>(input[i]);
}

// One row of one 128-column block of the output per iteration.
template <typename T>
__global__ void __launch_bounds__(128)
gated_activation_kernel(const float *__restrict__ input, T *__restrict__ output, const int gate, const float limit,
                        const std::size_t rows, const int inner, const int *__restrict__ tile_count, const int tile_rows) {
  std::size_t live = rows;
  if (tile_count != nullptr) {
    const std::size_t used = static_cast<std::size_t>(*tile_count) * tile_rows;
    live = used < rows ? used : rows;
  }
  const int block = blockIdx.y, column = block * 128 + static_cast<int>(threadIdx.x);
  for (std::size_t row = blockIdx.x; row < live; row += gridDim.x) {
    const float *const pair = input + row * 2 * inner + 256 * block + threadIdx.x;
    output[row * inner + column] = from_float<T>(gated_value(gate, limit, pair[0], pair[128]));
  }
}

// Rows and weights that the tensor cores' kernel does not take (inner sizes that are no multiple of 8 or below 64, operands that
// are not aligned).  A cluster of `splits` CTAs owns one tile of 16 kRows rows x 128 columns and divides K between its CTAs; every thread
// keeps kRows x 8 outputs as packed pairs, the sums over even and over odd K (fma.rn.f32x2, operands straight from
// K-contiguous rows of shared memory).  What bounds it is the F32 pipe; the split gives a few dozen rows (one row tile)
// enough CTAs, and makes the chains of additions short: K / (2 splits) terms in a pair's half, then a sum over the halves
// and the CTAs.
// (90 rows of a 2048-wide model with 8448 inner columns: 25 products in 3.3 ms; one CTA per 64 x 64 tile, which left most
// SMs idle and loaded single values, took 12.8.  Errors against float64 are no larger: 8.7e-7 of the logits, 9.1e-7 before.)
constexpr int kTileColumns = 128, kTileStep = 32, kTileStride = kTileStep + 4;

__device__ __forceinline__ void fma_pair(std::uint64_t &d, const std::uint64_t a, const std::uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_total(const std::uint64_t d) {
  return __uint_as_float(static_cast<std::uint32_t>(d)) + __uint_as_float(static_cast<std::uint32_t>(d >> 32U));
}

template <typename T, int kRows, bool kVector>
__global__ void __launch_bounds__(kThreads, 1)
linear_f32_tile_kernel(const T *__restrict__ input, const F32Params p) {
  constexpr int kTileRows = 16 * kRows, kLines = kTileRows + kTileColumns, kBuffer = kLines * kTileStride;
  extern __shared__ __align__(16) float tiles[];  // two buffers of weight rows and rows; at the end the tile's partial sums
  cg::cluster_group cluster = cg::this_cluster();
  const int splits = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int m0 = blockIdx.y * kTileRows, n0 = blockIdx.x / splits * kTileColumns;
  const bf16 *weight = p.weight;
  if (p.tile_group != nullptr) {
    const int tile = m0 / p.tile_rows;
    if (tile >= *p.tile_count) return;  // (the whole cluster)
    weight += static_cast<std::size_t>(p.tile_group[tile]) * p.out_features * p.in_features;
  }
  const int K = p.in_features, steps = (K + kTileStep - 1) / kTileStep;
  const int step_begin = static_cast<int>(static_cast<long long>(steps) * rank / splits);
  const int step_end = static_cast<int>(static_cast<long long>(steps) * (rank + 1) / splits);

  // a thread stages pieces of eight K values: line tid / 4 + 64 i (weight rows first), values 8 (tid % 4) ...
  constexpr int kRounds = (kLines + 63) / 64;
  float staged[kRounds][8];
  const int line0 = threadIdx.x / 4, k_in = threadIdx.x % 4 * 8;
  const auto fetch = [&](const int step) {
    const int k = step * kTileStep + k_in;
#pragma unroll
    for (int i = 0; i < kRounds; ++i) {
      const int line = line0 + 64 * i;
      const bool is_weight = line < kTileColumns;
      const int at = is_weight ? n0 + line : m0 + line - kTileColumns;
      const bool inside = is_weight ? at < p.out_features : line < kLines && at < p.rows;
      const std::size_t offset = static_cast<std::size_t>(at) * K + k;
      if constexpr (kVector) {
        if (inside && k < K) {
          if (is_weight) load_floats<8>(weight + offset, staged[i]);
          else load_floats<8>(input + offset, staged[i]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) staged[i][j] = 0.0F;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          staged[i][j] = !inside || k + j >= K ? 0.0F : is_weight ? bf2f(weight[offset + j]) : to_float(input[offset + j]);
      }
    }
  };
  const auto publish = [&](float *const buffer) {
#pragma unroll
    for (int i = 0; i < kRounds; ++i)
      if (line0 + 64 * i < kLines) store_floats(buffer + (line0 + 64 * i) * kTileStride + k_in, staged[i]);
  };
  // outputs: rows ty + 16 i, columns tx + 16 j; a warp reads four rows and eight weight rows at a time
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int ty = warp / 2 * 4 + lane / 8, tx = warp % 2 * 8 + lane % 8;
  std::uint64_t acc[kRows][8];
#pragma unroll
  for (int i = 0; i < kRows; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;
  if (step_begin < step_end) {
    fetch(step_begin);
    publish(tiles);
  }
  __syncthreads();
  for (int step = step_begin, at = 0; step < step_end; ++step, at ^= 1) {
    const bool more = step + 1 < step_end;
    if (more) fetch(step + 1);
    const float *const w_lines = tiles + at * kBuffer + tx * kTileStride;
    const float *const x_lines = tiles + at * kBuffer + (kTileColumns + ty) * kTileStride;
#pragma unroll 2
    for (int k = 0; k < kTileStep; k += 4) {
      ulonglong2 x[kRows];
#pragma unroll
      for (int i = 0; i < kRows; ++i) x[i] = *reinterpret_cast<const ulonglong2 *>(x_lines + 16 * i * kTileStride + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(w_lines + 16 * j * kTileStride + k);
#pragma unroll
        for (int i = 0; i < kRows; ++i) fma_pair(acc[i][j], x[i].x, w.x);
#pragma unroll
        for (int i = 0; i < kRows; ++i) fma_pair(acc[i][j], x[i].y, w.y);
      }
    }
    if (more) publish(tiles + (at ^ 1) * kBuffer);
    __syncthreads();
  }
  // every CTA's sums, then a share of the tile's rows per CTA
  constexpr int kSumStride = kTileColumns + 4;
  static_assert(kTileRows * kSumStride <= 2 * kBuffer, "the sums take the buffers' place");
#pragma unroll
  for (int i = 0; i < kRows; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) tiles[(ty + 16 * i) * kSumStride + tx + 16 * j] = pair_total(acc[i][j]);
  cluster.sync();
  for (int item = rank * kThreads + threadIdx.x; item < kTileRows * kTileColumns; item += splits * kThreads) {
    const int r = item / kTileColumns, c = item % kTileColumns;
    if (m0 + r >= p.rows || n0 + c >= p.out_features) continue;
    float sum = 0.0F;
    for (int other = 0; other < splits; ++other) sum += cluster.map_shared_rank(tiles, other)[r * kSumStride + c];
    store_f32_result(p, static_cast<std::size_t>(m0 + r), n0 + c, sum);
  }
  cluster.sync();  // remote shared memory stays alive until every CTA has read it
}

// Few rows: a warp per (row, output).
template <typename T, bool kVector>
__global__ void __launch_bounds__(256)
linear_f32_rows_kernel(const T *__restrict__ input, const F32Params p) {
  const int column = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x % 32;
  if (column >= p.out_features) return;
  const std::size_t row = blockIdx.y;
  const T *const x = input + row / p.row_fanout * p.in_features;
  const std::size_t group = p.row_group != nullptr ? static_cast<std::size_t>(p.row_group[row]) : 0;
  const bf16 *const w = p.weight + (group * p.out_features + column) * p.in_features;
  float sum = 0.0F;
  if constexpr (kVector) {
#pragma unroll 4
    for (int k = 8 * lane; k < p.in_features; k += 256) {
      float a[8], b[8];
      load_floats<8>(x + k, a);
      load_floats<8>(w + k, b);
#pragma unroll
      for (int i = 0; i < 8; ++i) sum = fmaf(a[i], b[i], sum);
    }
  } else {
    for (int k = lane; k < p.in_features; k += 32) sum = fmaf(to_float(x[k]), bf2f(w[k]), sum);
  }
  sum = warp_sum(sum);
  if (lane == 0) store_f32_result(p, row, column, sum);
}

// Two to four rows of many columns: a warp per three columns of all rows, so that the weights come from L2 (or memory) once
// and the rows from L1 once per three columns; a result's sums have the order of the kernel above.  What bounds it is L1 where
// the weights are in L2 (2, 3 and 4 rows of 2048 x 8448: 7.3, 9.4 and 11.4 us; with two columns a warp 8.0, 10.4 and 12.9, with a
// row and a column a warp 14.8, 19.5 and 24.8), and memory where they are not (9.4, 10.8 and 12.7 us, 3.7 to 2.7 TB/s).
constexpr int kFewRowColumns = 3;

template <typename T, int kRows>
__global__ void __launch_bounds__(256)
linear_f32_few_rows_kernel(const T *__restrict__ input, const F32Params p) {
  wait_for_producers(input);
  release_dependents();
  const int column0 = (blockIdx.x * 8 + threadIdx.x / 32) * kFewRowColumns, lane = threadIdx.x % 32;
  if (column0 >= p.out_features) return;
  const bf16 *w[kFewRowColumns];  // (columns beyond the last are computed and dropped)
#pragma unroll
  for (int c = 0; c < kFewRowColumns; ++c)
    w[c] = p.weight + static_cast<std::size_t>(min(column0 + c, p.out_features - 1)) * p.in_features;
  float sum[kRows][kFewRowColumns] = {};
#pragma unroll 4
  for (int k = 8 * lane; k < p.in_features; k += 256) {
    float b[kFewRowColumns][8];
#pragma unroll
    for (int c = 0; c < kFewRowColumns; ++c) load_floats<8>(w[c] + k, b[c]);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      float a[8];
      load_floats<8>(input + static_cast<std::size_t>(r) * p.in_features + k, a);
#pragma unroll
      for (int c = 0; c < kFewRowColumns; ++c)
#pragma unroll
        for (int i = 0; i < 8; ++i) sum[r][c] = fmaf(a[i], b[c][i], sum[r][c]);
    }
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int c = 0; c < kFewRowColumns; ++c) {
      const float total = warp_sum(sum[r][c]);
      if (lane == r * kFewRowColumns + c && column0 + c < p.out_features)
        store_f32_result(p, static_cast<std::size_t>(r), column0 + c, total);
    }
}

bool row_vector_ok(const std::size_t width, const void *a, const void *b, const void *c) {
  return width % 8 == 0 && aligned16(a) && aligned16(b) && aligned16(c);
}

}  // namespace

int embed_positions(const std::uint32_t *tokens, const void *table, const void *positions, const float *gain,
                    const std::size_t rows, const std::size_t width, const std::size_t vocabulary,
                    const std::size_t position, const float epsilon, float *output, cudaStream_t stream,
                    const int *dynamic_position) {
  if (tokens == nullptr || table == nullptr || positions == nullptr || gain == nullptr || output == nullptr ||
      width == 0 || width > 0x7fffff00U || rows > 0x7fffffffU || position > 0x7fffffffU)
    return fail(kInvalidArgument, "embedding arguments are invalid");
  if (rows == 0) return kOk;
  int status = kOk;
  int *const error = device_error_word(&status);
  if (error == nullptr) return status;
  const bool vector = row_vector_ok(width, table, positions, output) && aligned16(gain);
  const auto kernel = vector ? embed_positions_kernel<true> : embed_positions_kernel<false>;
  return launch_dependent("embedding kernel with positions", kernel, dim3(static_cast<unsigned int>(rows)), kThreads, 0, stream,
                          true, 1, tokens, static_cast<const bf16 *>(table), static_cast<const bf16 *>(positions), gain,
                          static_cast<int>(width), static_cast<std::uint32_t>(vocabulary), static_cast<int>(position),
                          dynamic_position, epsilon, output, error);
}

int rms_norm_residual(const float *input, const float *gain, const std::size_t rows, const std::size_t width,
                      const float epsilon, void *output, const Activation type, cudaStream_t stream) {
  if (input == nullptr || gain == nullptr || output == nullptr || width == 0 || width > 0x7fffff00U ||
      rows > 0x7fffffffU)
    return fail(kInvalidArgument, "residual norm arguments are invalid");
  if (rows == 0) return kOk;
  const bool vector = row_vector_ok(width, input, gain, output);
  const unsigned int grid = static_cast<unsigned int>(rows);
  const int w = static_cast<int>(width);
  if (type == Activation::kBf16) {
    const auto kernel = vector ? rms_norm_residual_kernel<bf16, true> : rms_norm_residual_kernel<bf16, false>;
    return launch_dependent("residual norm kernel", kernel, dim3(grid), kThreads, 0, stream, true, 1, input, gain, w, epsilon,
                            static_cast<bf16 *>(output));
  }
  const auto kernel = vector ? rms_norm_residual_kernel<float, true> : rms_norm_residual_kernel<float, false>;
  return launch_dependent("residual norm kernel", kernel, dim3(grid), kThreads, 0, stream, true, 1, input, gain, w, epsilon,
                          static_cast<float *>(output));
}

int poly_norm(const void *input, const float *coefficients, const std::size_t rows, const std::size_t width,
              const float epsilon, void *output, const Activation type, cudaStream_t stream) {
  if (input == nullptr || coefficients == nullptr || output == nullptr || width == 0 || width > 0x7fffff00U ||
      rows > 0x7fffffffU)
    return fail(kInvalidArgument, "polynomial activation arguments are invalid");
  if (rows == 0) return kOk;
  const bool vector = row_vector_ok(width, input, output, nullptr);
  const unsigned int grid = static_cast<unsigned int>(rows);
  const int w = static_cast<int>(width);
  if (type == Activation::kBf16) {
    const auto kernel = vector ? poly_norm_kernel<bf16, true> : poly_norm_kernel<bf16, false>;
    return launch_dependent("polynomial activation kernel", kernel, dim3(grid), kThreads, 0, stream, true, 1,
                            static_cast<const bf16 *>(input), coefficients, w, epsilon, static_cast<bf16 *>(output));
  }
  const auto kernel = vector ? poly_norm_kernel<float, true> : poly_norm_kernel<float, false>;
  return launch_dependent("polynomial activation kernel", kernel, dim3(grid), kThreads, 0, stream, true, 1,
                          static_cast<const float *>(input), coefficients, w, epsilon, static_cast<float *>(output));
}

int distance_bias_table(const float *r1, const float *r2, const std::size_t heads, const std::size_t distances,
                        float *table, cudaStream_t stream) {
  if (r1 == nullptr || r2 == nullptr || table == nullptr || heads == 0 || heads > 65535 || distances == 0 ||
      distances > 0x7fffff00U)
    return fail(kInvalidArgument, "distance bias arguments are invalid");
  const dim3 grid(ceil_div_u(distances, kThreads) > 64 ? 64 : ceil_div_u(distances, kThreads),
                  static_cast<unsigned int>(heads));
  distance_bias_kernel<<<grid, kThreads, 0, stream>>>(r1, r2, static_cast<int>(distances), table);
  return check_launch("distance bias kernel");
}

int embed_rows(const std::uint32_t *tokens, const void *table, const std::size_t rows, const std::size_t width,
               const std::size_t vocabulary, float *stream_rows, void *copy, const Activation type, cudaStream_t stream) {
  if (tokens == nullptr || table == nullptr || stream_rows == nullptr || width == 0 || width > 0x7fffff00U ||
      rows > 0x7fffffffU)
    return fail(kInvalidArgument, "embedding arguments are invalid");
  if (rows == 0) return kOk;
  int status = kOk;
  int *const error = device_error_word(&status);
  if (error == nullptr) return status;
  const bool vector = row_vector_ok(width, table, stream_rows, copy);
  const auto launch = [&](auto tag) {
    using T = decltype(tag);
    const auto kernel = vector ? embed_rows_kernel<T, true> : embed_rows_kernel<T, false>;
    return launch_dependent("embedding kernel of the residual stream", kernel, dim3(static_cast<unsigned int>(rows)), kThreads, 0,
                            stream, true, 1, tokens, static_cast<const bf16 *>(table), static_cast<int>(width),
                            static_cast<std::uint32_t>(vocabulary), stream_rows, static_cast<T *>(copy), error);
  };
  return type == Activation::kBf16 ? launch(bf16{}) : launch(float{});
}

int layer_norm(const LayerNormArgs &a, cudaStream_t stream) {
  if (a.input == nullptr || a.gain == nullptr || (a.residual == nullptr && a.output == nullptr) || a.parts == 0 ||
      a.parts > 0x7fffffffU || a.width == 0 || a.width > 0x7fffff00U || a.rows > 0x7fffffffU)
    return fail(kInvalidArgument, "layer norm arguments are invalid");
  if (a.rows == 0) return kOk;
  const bool vector = row_vector_ok(a.width, a.input, a.gain, a.output) && aligned16(a.residual);
  LayerNormParams p{};
  p.slots = a.slots;
  p.parts = static_cast<int>(a.parts);
  p.gain = a.gain;
  p.residual = a.residual;
  p.width = static_cast<int>(a.width);
  p.epsilon = a.epsilon;
  const auto launch = [&](auto in_tag, auto out_tag) {
    using In = decltype(in_tag);
    using Out = decltype(out_tag);
    const auto kernel = !vector                      ? layer_norm_kernel<In, Out, false, kCached>
                        : a.width <= 8 * kThreads  ? layer_norm_kernel<In, Out, true, 1>
                        : a.width <= 16 * kThreads ? layer_norm_kernel<In, Out, true, 2>
                                                   : layer_norm_kernel<In, Out, true, kCached>;
    return launch_dependent("layer norm kernel", kernel, dim3(static_cast<unsigned int>(a.rows)), kThreads, 0, stream, true, 1,
                            static_cast<const In *>(a.input), static_cast<Out *>(a.output), p);
  };
  if (a.input_type == Activation::kBf16)
    return a.output_type == Activation::kBf16 ? launch(bf16{}, bf16{}) : launch(bf16{}, float{});
  return a.output_type == Activation::kBf16 ? launch(float{}, bf16{}) : launch(float{}, float{});
}

int convert_rows(const float *input, const std::size_t elements, void *output, const Activation type, cudaStream_t stream) {
  if (input == nullptr || output == nullptr) return fail(kInvalidArgument, "conversion arguments are invalid");
  if (elements == 0) return kOk;
  const std::size_t blocks = (elements + kThreads - 1) / kThreads;
  const unsigned int grid = static_cast<unsigned int>(blocks < 8 * kSmCount ? blocks : 8 * kSmCount);
  if (type == Activation::kBf16)
    convert_kernel<<<grid, kThreads, 0, stream>>>(input, static_cast<bf16 *>(output), elements);
  else
    convert_kernel<<<grid, kThreads, 0, stream>>>(input, static_cast<float *>(output), elements);
  return check_launch("conversion kernel");
}

int gated_activation(const float *input, const int gate, const float limit, const std::size_t rows,
                     const std::size_t inner, void *output, const Activation type, const int *tile_count,
                     const std::size_t tile_rows, cudaStream_t stream) {
  if (input == nullptr || output == nullptr || (gate != kGateRelu && gate != kGateClamped) || inner == 0 || inner % 128 != 0 ||
      inner / 128 > 65535 || inner > 0x3fffff00U || tile_rows > 0x7fffffffU)
    return fail(kInvalidArgument, "gated activation arguments are invalid");
  if (rows == 0) return kOk;
  const dim3 grid(static_cast<unsigned int>(rows < 65536 ? rows : 65536), static_cast<unsigned int>(inner / 128));
  if (type == Activation::kBf16)
    gated_activation_kernel<<<grid, 128, 0, stream>>>(input, static_cast<bf16 *>(output), gate, limit, rows,
                                                      static_cast<int>(inner), tile_count, static_cast<int>(tile_rows));
  else
    gated_activation_kernel<<<grid, 128, 0, stream>>>(input, static_cast<float *>(output), gate, limit, rows,
                                                      static_cast<int>(inner), tile_count, static_cast<int>(tile_rows));
  return check_launch("gated activation kernel");
}

int linear_f32(const LinearF32Args &a, cudaStream_t stream) {
  if (a.input == nullptr || a.weight == nullptr || a.output == nullptr || a.in_features == 0 || a.out_features == 0 ||
      a.in_features > 0x7fffff00U || a.out_features > 0x7fffff00U || a.rows > 64 * 65535U || a.row_fanout == 0 ||
      (a.tile_group != nullptr && (a.tile_count == nullptr || a.tile_rows % 64 != 0 || a.row_group != nullptr)) ||
      (a.row_group != nullptr && a.rows > 65535U))
    return fail(kInvalidArgument, "F32 linear arguments are invalid");
  if (a.rows == 0) return kOk;
  // One row: outside a pass's chain of launches the weight stream's ring and its one large CTA per SM have to be set up
  // first, which short rows do not repay (264 x 5000: 8.3 us, 4.5 with a warp per output; 512 x 2048: 5.9 and 4.6; 1024 x
  // 1024: 5.8 and 5.9; 4096 x 4096: 10.6 and 14.3).
  if ((a.weight_stream || a.front.values != nullptr || a.in_features >= 1024) && one_row_linear_f32_applicable(a))
    return one_row_linear_f32(a, stream);
  if (a.front.values != nullptr) return fail(kUnsupported, "operators in front of a projection take one row");
  F32Params p{};
  p.weight = static_cast<const bf16 *>(a.weight);
  p.output = a.output;
  p.rows = static_cast<int>(a.rows);
  p.out_features = static_cast<int>(a.out_features);
  p.in_features = static_cast<int>(a.in_features);
  p.accumulate = a.accumulate ? 1 : 0;
  p.alpha = a.alpha;
  p.softcap = a.softcap;
  p.row_scale = a.row_scale;
  p.bias = a.bias;
  p.row_group = a.row_group;
  p.row_fanout = static_cast<int>(a.row_fanout);
  p.tile_group = a.tile_group;
  p.tile_count = a.tile_count;
  p.tile_rows = static_cast<int>(a.tile_rows);
  const bool vector = a.in_features % 8 == 0 && aligned16(a.input) && aligned16(a.weight);
  // (up to 16 rows that share inputs without a group take a warp per output, the kernel that looks at row_fanout)
  const bool plain = a.row_group == nullptr && a.tile_group == nullptr && a.row_fanout == 1;
  // Three columns a warp need columns for every SM, and more of them the more rows the tensor cores' kernel would take along (weights
  // from memory: 2 rows of 2048 x 2048 7.4 us against 6.8 with a warp per output, of 2048 x 4096 7.9 against 10.6; 3 rows 8.9 against
  // 10.5 on the tensor cores; 4 rows of 2048 x 4096 11.3 against 10.5, of 2048 x 6144 12.3 against 15.8, of 4096 x 11264 37.9 against 39.0).
  const bool few_wide_rows = plain && vector && a.rows >= 2 && a.rows <= 4 && a.out_features >= (a.rows < 4 ? 4096U : 6144U);
  // Every row of a warp per output fetches the weights again, from L2 where they fit.  The tensor cores' kernel fetches them
  // once, but takes 12 us alone to start and to add its shares up: 4 rows of 2048 x 2048 take 14.3 us against 14.3, 12 of 2048 x 512
  // 10.2 against 12.3; 6 of 2048 x 2048 16.4 against 14.3, 16 of 2048 x 8448 96 against 23.
  constexpr std::size_t kFewRowProducts = std::size_t{24} << 20;
  if (!few_wide_rows &&
      (a.tile_group != nullptr || a.rows > 16 || (a.rows > 2 && plain && a.rows * a.in_features * a.out_features > kFewRowProducts)) &&
      tensorcore_linear_f32_applicable(a))
    return tensorcore_linear_f32(a, p, stream);
  // Against the tile kernel on the CUDA cores: 2 rows of 2048 x 8448 take 18 us against 90, 12 rows 72 against 90, 16 rows of
  // 8448 x 2048 90 against 136, of 2048 x 8448 92 against 91; but 16 rows of 4096 x 22528 (185 MB) 520 against 397.
  constexpr std::size_t kL2Weights = std::size_t{96} << 20;
  const bool few_rows = a.row_group != nullptr ||
                        (a.tile_group == nullptr &&
                         (a.rows <= 12 || (a.rows <= 16 && a.in_features * a.out_features * 2 <= kL2Weights)));
  const auto launch = [&](auto tag) {
    using T = decltype(tag);
    const T *const input = static_cast<const T *>(a.input);
    if (few_wide_rows) {
      const auto kernel = a.rows == 2   ? linear_f32_few_rows_kernel<T, 2>
                          : a.rows == 3 ? linear_f32_few_rows_kernel<T, 3>
                                        : linear_f32_few_rows_kernel<T, 4>;
      return launch_dependent("F32 linear kernel (a few wide rows)", kernel, dim3(ceil_div_u(a.out_features, 8 * kFewRowColumns)),
                              256, 0, stream, true, 1, input, p);
    }
    if (few_rows) {
      const auto kernel = vector ? linear_f32_rows_kernel<T, true> : linear_f32_rows_kernel<T, false>;
      return launch_dependent("F32 linear kernel (few rows)", kernel,
                              dim3(ceil_div_u(a.out_features, 8), static_cast<unsigned int>(a.rows)), 256, 0, stream, false, 1,
                              input, p);
    }
    const auto tiled = [&](auto rows_tag) {
      constexpr int kRows = decltype(rows_tag)::value;
      constexpr std::size_t kBytes = 2 * (16 * kRows + kTileColumns) * kTileStride * sizeof(float);
      // two steps or more for every CTA; eight CTAs where K allows, for chains as short as they get
      const std::size_t steps = (a.in_features + kTileStep - 1) / kTileStep;
      const unsigned int splits = steps >= 16 ? 8 : steps >= 8 ? 4 : steps >= 4 ? 2 : 1;
      const auto kernel = vector ? linear_f32_tile_kernel<T, kRows, true> : linear_f32_tile_kernel<T, kRows, false>;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBytes)) != cudaSuccess)
        return fail(kCuda, "cannot raise the shared-memory limit of the F32 linear kernel");
      return launch_dependent("F32 linear kernel", kernel,
                              dim3(ceil_div_u(a.out_features, kTileColumns) * splits, ceil_div_u(a.rows, 16 * kRows)), kThreads,
                              kBytes, stream, false, splits, input, p);
    };
    // the tile height that pads the fewest rows, the larger one of equals; grouped row tiles are made of whole ones
    int best = 4;
    std::size_t padded = ~std::size_t{0};
    for (const int rows16 : {8, 6, 4, 2}) {
      const std::size_t height = 16 * static_cast<std::size_t>(rows16);
      if ((a.tile_group != nullptr && a.tile_rows % height != 0) || (rows16 == 2 && (a.rows > 64 || a.tile_group != nullptr))) continue;
      const std::size_t total = (a.rows + height - 1) / height * height;
      if (total < padded) padded = total, best = rows16;
    }
    switch (best) {
      case 8: return tiled(std::integral_constant<int, 8>{});
      case 6: return tiled(std::integral_constant<int, 6>{});
      case 4: return tiled(std::integral_constant<int, 4>{});
      default: return tiled(std::integral_constant<int, 2>{});
    }
  };
  return a.input_type == Activation::kBf16 ? launch(bf16{}) : launch(float{});
}

int linear_f32(const float *input, const void *weight, const std::size_t rows, const std::size_t in_features,
               const std::size_t out_features, float *output, const bool accumulate, cudaStream_t stream) {
  LinearF32Args a;
  a.input = input;
  a.weight = weight;
  a.rows = rows;
  a.in_features = in_features;
  a.out_features = out_features;
  a.output = output;
  a.accumulate = accumulate;
  return linear_f32(a, stream);
}

}  // namespace evob
