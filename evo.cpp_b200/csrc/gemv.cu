// Small-batch projections (1..8 rows: cached decode and very short prompts).
// At these sizes a projection is a weight stream: every weight byte is read
// once and the arithmetic is negligible, so the tensor-core tile kernel (which
// launches one CTA per 128 x 256 tile and leaves most SMs idle) is replaced by
// kernels in which a CTA owns weight rows, its threads split K in
// 16-byte chunks, and partial sums are folded with shuffles and shared memory.  Same epilogue
// contract as the tile kernel (scale, fused or separately rounded bias,
// residual, gate over row-interleaved up-projections).
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "decoder_types.cuh"
#include "gates.cuh"
#include "ops_internal.hpp"

namespace evob {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxRows = 8;

struct GemvParams {
  const void *x;       // [rows, K] BF16 or E4M3 codes; F32 in one-row streams of F32 activations
  const void *w;       // [N, K] same type
  const bf16 *bias, *residual;
  bf16 *out;
  float *out_f32;           // F32 result instead of out: [out_f32 +] alpha * sum [+ bias_f32]
  const float *bias_f32;
  int accumulate_f32;
  int rows, K, N;      // N = weight rows
  float alpha;
  int bias_mode, gate_mode;
  int dependent_launch;  // launched with programmatic stream serialisation: see the kernel
  bool weight_stream;    // LinearArgs::weight_stream
  float gate_limit, softcap;
  // grouped weights [groups, N, K]: blockIdx.y = output row r, x row r / row_fanout, weight of group row_group[r]
  const int *row_group;
  int row_fanout;
  int row_group_settled;   // LinearArgs::row_group_settled
  const float *row_scale;  // grouped weights only
  const float *front;      // RowFront::values
  float epsilon;
  bool poly_front;
};

template <bool kFp8>
__device__ __forceinline__ void unpack16(const uint4 raw, float (&v)[kFp8 ? 16 : 8]) {
  if constexpr (kFp8) {
    const unsigned int words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const __half2_raw pair = __nv_cvt_fp8x2_to_halfraw2(
            static_cast<__nv_fp8x2_storage_t>((words[i] >> (16 * h)) & 0xffffU), __NV_E4M3);
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&pair));
        v[4 * i + 2 * h] = f.x;
        v[4 * i + 2 * h + 1] = f.y;
      }
    }
  } else {
    Bf16x8 packed;
    packed.raw = raw;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = packed.get(i);
  }
}

__device__ __forceinline__ bf16 gelu_round_small(const float x) {
  const bf16 input = f2bf(x);
  const float value = bf2f(input);
  const bf16 computed = f2bf(value * 0.5F * (1.0F + ::erff(value * 0.70710678118654752440F)));
  switch (__bfloat16_as_ushort(input)) {
    case 0xc049: return __ushort_as_bfloat16(0xbb2d);
    case 0xc081: return __ushort_as_bfloat16(0xb8eb);
    case 0xc089: return __ushort_as_bfloat16(0xb827);
    case 0xc092: return __ushort_as_bfloat16(0xb742);
    case 0xc0a0: return __ushort_as_bfloat16(0xb5c8);
    case 0xc0a8: return __ushort_as_bfloat16(0xb4fc);
    case 0xc0ab: return __ushort_as_bfloat16(0xb4ab);
    default: return computed;
  }
}

// What a result is added to.  A stream reads it beside x, so that the trip to memory does not follow the sums.
struct Addends {
  float first = 0.0F, second = 0.0F;  // F32: the old result and the bias; BF16: the residual and the bias
  __device__ __forceinline__ float old_result() const { return first; }
  __device__ __forceinline__ float bias_f32() const { return second; }
  __device__ __forceinline__ float residual() const { return first; }
  __device__ __forceinline__ float bias() const { return second; }
};
// The same, read where it is used: the kernel of a few rows has no registers to hold it (8 E4M3 rows of 5120 x 1920 18.6 us, 20.5
// with the word that was spilled for it).
struct LateAddends {
  const GemvParams &p;
  std::size_t old_index, residual_index;
  int column;
  __device__ __forceinline__ float old_result() const { return p.out_f32[old_index]; }
  __device__ __forceinline__ float bias_f32() const { return p.bias_f32[column]; }
  __device__ __forceinline__ float residual() const { return bf2f(p.residual[residual_index]); }
  __device__ __forceinline__ float bias() const { return bf2f(p.bias[column]); }
};
__device__ __forceinline__ Addends addends_of(const GemvParams &p, const int r, const std::size_t out_index, const int out_columns,
                                              const int column) {
  Addends a;
  if (p.out_f32 != nullptr) {
    if (p.accumulate_f32 != 0) a.first = p.out_f32[out_index * out_columns + column];
    if (p.bias_f32 != nullptr) a.second = p.bias_f32[column];
  } else if (p.gate_mode == 0) {
    if (p.residual != nullptr) a.first = bf2f(p.residual[static_cast<std::size_t>(r) * out_columns + column]);
    if (p.bias_mode != 0) a.second = bf2f(p.bias[column]);
  }
  return a;
}

// Result `column` of row `out_index` from its sum, or from the sums of a gated pair.
template <class Added, class Total>
__device__ __forceinline__ void finish_column(const GemvParams &p, const std::size_t out_index, const int out_columns,
                                              const int column, const float alpha, const int local, const Added &addends,
                                              const Total &total) {
  if (p.out_f32 != nullptr) {
    float value = total(local) * alpha;
    if (p.bias_f32 != nullptr) value += addends.bias_f32();
    p.out_f32[out_index * out_columns + column] =
        soft_cap(p.accumulate_f32 != 0 ? addends.old_result() + value : value, p.softcap);
    return;
  }
  bf16 *const out_row = p.out + out_index * out_columns;
  if (p.gate_mode >= kGateRelu) {
    float value = total(2 * local) * alpha, up = total(2 * local + 1) * alpha;
    if (p.bias_f32 != nullptr) {
      const int row = (column / 128) * 256 + column % 128;
      value += p.bias_f32[row];
      up += p.bias_f32[row + 128];
    }
    out_row[column] = f2bf(gated_value(p.gate_mode, p.gate_limit, value, up));
  } else if (p.gate_mode != 0) {
    const float first = total(2 * local) * p.alpha, second = rbf(total(2 * local + 1) * p.alpha);
    const float activated = p.gate_mode == 2 ? bf2f(gelu_round_small(first)) : rbf(first);
    out_row[column] = f2bf(activated * second);
  } else {
    float value = total(local) * alpha;
    if (p.bias_mode == 1) value += addends.bias();
    value = rbf(value);
    if (p.bias_mode == 2) value = rbf(value + addends.bias());
    if (p.residual != nullptr) value = rbf(value + addends.residual());
    out_row[column] = f2bf(value);
  }
}

// A CTA owns kColumns weight rows and its eight warps split K between them, so
// the whole weight slab of the CTA (kColumns x K) is requested within the first
// couple of loop iterations - at one row a projection is a latency problem as
// much as a bandwidth one.  Per-warp partial sums are folded with shuffles,
// then across warps through shared memory; the last step applies the same
// epilogue as the tile kernel.  kRows is a compile-time bound on the rows held
// in registers.
constexpr int kWarps = kThreads / 32;

template <bool kFp8, int kRows, int kColumns>
__global__ void __launch_bounds__(kThreads)
gemv_kernel(const GemvParams p) {
  constexpr int kPerChunk = kFp8 ? 16 : 8;   // elements per 16-byte chunk
  __shared__ float partial[kWarps][kColumns][kRows];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const bool gated = p.gate_mode != 0;
  // Output columns handled by this CTA.  When gated, the weight holds blocks
  // of 128 first-projection rows followed by the matching 128 second-projection
  // rows; an output column needs one row of each.
  const int out_columns = gated ? p.N / 2 : p.N;
  const int per_cta = gated ? kColumns / 2 : kColumns;
  const int column0 = blockIdx.x * per_cta;
  int weight_row[kColumns];
#pragma unroll
  for (int c = 0; c < kColumns; ++c) {
    const int column = min(column0 + (gated ? c / 2 : c), out_columns - 1);
    weight_row[c] = gated ? (column / 128) * 256 + column % 128 + (c % 2) * 128 : column;
  }
  float acc[kColumns][kRows];
#pragma unroll
  for (int c = 0; c < kColumns; ++c)
#pragma unroll
    for (int r = 0; r < kRows; ++r) acc[c][r] = 0.0F;
  const int chunks = p.K / kPerChunk;
  const std::size_t row_bytes = static_cast<std::size_t>(p.K) * (kFp8 ? 1 : 2);
  const unsigned char *wb = static_cast<const unsigned char *>(p.w);
  const unsigned char *xb = static_cast<const unsigned char *>(p.x);
  // Programmatic dependent launch (one-row steps inside the captured decode graph): this grid may be
  // started while the kernel that produces x is still running.  The weights do not depend on that
  // kernel, so the CTA first asks L2 for its weight rows, lets the grid after it start as well, and only
  // then waits for the producer to finish and its writes to be visible.  Without such a launch the two
  // instructions do nothing.
  const bool grouped = p.row_group != nullptr;
  if (grouped) {
    // which weights these are is a result of the kernel in front; the one behind may rely on it (row_group_settled)
    const int *row_group = p.row_group;
    wait_for_producers(xb, row_group);
    release_dependents();
    wb += static_cast<std::size_t>(row_group[blockIdx.y]) * p.N * row_bytes;
    xb += static_cast<std::size_t>(blockIdx.y / p.row_fanout) * row_bytes;
  } else if (p.dependent_launch != 0) {
    for (int chunk = threadIdx.x * 8; chunk < chunks; chunk += kThreads * 8) {  // one request per 128-byte line
#pragma unroll
      for (int c = 0; c < kColumns; ++c)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(wb + weight_row[c] * row_bytes + static_cast<std::size_t>(chunk) * 16));
    }
    release_dependents();
    wait_for_producers(xb);
  }
#pragma unroll(kRows == 1 ? 4 : (kRows == 2 ? 2 : 1))
  for (int chunk = threadIdx.x; chunk < chunks; chunk += kThreads) {
    uint4 wraw[kColumns];
#pragma unroll
    for (int c = 0; c < kColumns; ++c)
      wraw[c] = __ldcs(reinterpret_cast<const uint4 *>(wb + weight_row[c] * row_bytes) + chunk);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      if (r < p.rows) {
        float xv[kPerChunk];
        unpack16<kFp8>(reinterpret_cast<const uint4 *>(xb + r * row_bytes)[chunk], xv);
#pragma unroll
        for (int c = 0; c < kColumns; ++c) {
          float wv[kPerChunk];
          unpack16<kFp8>(wraw[c], wv);
#pragma unroll
          for (int i = 0; i < kPerChunk; ++i) acc[c][r] = fmaf(xv[i], wv[i], acc[c][r]);
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kColumns; ++c)
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
#pragma unroll
      for (int offset = 16; offset > 0; offset /= 2)
        acc[c][r] += __shfl_xor_sync(0xffffffffU, acc[c][r], offset);
      if (lane == 0) partial[warp][c][r] = acc[c][r];
    }
  __syncthreads();
  // one thread per (row, output column of the CTA)
  const int item = threadIdx.x;
  if (item >= per_cta * kRows) return;
  const int r = item / per_cta, local = item % per_cta;
  const int column = column0 + local;
  if (r >= p.rows || column >= out_columns) return;
  const std::size_t out_index = grouped ? blockIdx.y : r;
  const float alpha = grouped && p.row_scale != nullptr ? p.alpha * p.row_scale[out_index] : p.alpha;
  const LateAddends addends{p, out_index * out_columns + column, static_cast<std::size_t>(r) * out_columns + column, column};
  finish_column(p, out_index, out_columns, column, alpha, local, addends, [&](const int c) {
    float sum = 0.0F;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += partial[w][c][r];
    return sum;
  });
}

// One row: the projection is a stream of the weights and nothing else, so what counts is that loads are in flight
// all the time, also while kernels in front of this one are still running.  A CTA owns a contiguous share of the
// output columns and each of its eight warps an eighth of K, whose piece of x stays in registers.  A thread
// copies its 16-byte pieces of the weight rows into its own slots of a ring in shared memory
// (cp.async) and reads only what it copied itself: no barrier in the loop, and the ring is filled before the thread
// waits for the producer of x (the weights do not depend on it).  The warps' partial sums of all columns meet in
// shared memory once, at the end.  A CTA is two such teams, and its shared memory keeps a second CTA off the SM: where a
// kernel starts beside others, CTAs that fit twice are packed on half of the SMs (observed: four small CTAs on each of 74),
// and a stream is as slow as its fullest SM.
// Grouped rows (blockIdx.y) take their weights' rows the same way, once they know their group.
// Bound: HBM, and in a step the way from one kernel's end to the next one's first data.  48 decode steps of Gigusun:
// 12.3 ms, 12.8 with two CTAs of one team each that pack; of Kikepel 11.4 and 11.9.  A trip to memory that nothing hides is
// 0.3 us of a kernel: old results and gains read beside x instead of where they are used take Gigusun's steps to 12.07 ms.
constexpr int kTeams = 2, kRingBytes = 48 * 1024;
constexpr int kStreamShared = 116 * 1024;  // more than half of an SM's
constexpr int kTeamShared = kStreamShared / kTeams;
constexpr int kStreamRows = (kTeamShared - kRingBytes) / (kWarps * static_cast<int>(sizeof(float)));  // per team

// What is done to x on the way in.  A norm's statistics are those of the whole row: every CTA takes them itself, which
// costs it a barrier against a launch and a round trip through memory.
enum class Front { kNone, kRms, kPoly };

// kUnit: pieces per thread that are copied and waited for at a time, whole rows (kRowsPerStage of kChunks pieces) or, of
// long rows, single pieces.
template <bool kFp8, class X, Front kFront, int kChunks, int kRowsPerStage, int kUnit>
__global__ void __launch_bounds__(kTeams *kThreads, 1)
gemv_stream_kernel(const GemvParams p) {
  constexpr int kPer = kFp8 ? 16 : 8;  // elements per 16-byte piece
  constexpr int kUnits = kRingBytes / (kUnit * kThreads * 16);
  static_assert(kUnits >= 3 && (kUnit == 1 ? kRowsPerStage == 1 : kUnit == kRowsPerStage * kChunks), "ring");
  extern __shared__ __align__(16) unsigned char stream_smem[];
  const int team = threadIdx.x / kThreads, tid = threadIdx.x % kThreads, warp = tid / 32, lane = tid % 32;
  uint4 *const ring = reinterpret_cast<uint4 *>(stream_smem + team * kTeamShared);     // [kUnits][kUnit][kThreads]
  float *const partial = reinterpret_cast<float *>(ring + kUnits * kUnit * kThreads);  // [rows][kWarps]
  const auto team_barrier = [&] { asm volatile("barrier.cta.sync %0, %1;" ::"r"(team + 1), "n"(kThreads) : "memory"); };
  const bool gated = p.gate_mode != 0, grouped = p.row_group != nullptr;
  const int out_columns = gated ? p.N / 2 : p.N;
  const auto share = [&](const unsigned int index) {
    return static_cast<int>(static_cast<unsigned long long>(out_columns) * index / (kTeams * gridDim.x));
  };
  const unsigned int team_index = kTeams * blockIdx.x + team;
  const int column0 = share(team_index), columns = share(team_index + 1) - column0;
  const int rows = gated ? 2 * columns : columns;  // gated: all first rows, then their partners
  const int groups = (rows + kRowsPerStage - 1) / kRowsPerStage;
  const std::size_t row_bytes = static_cast<std::size_t>(p.K) * (kFp8 ? 1 : 2);
  // the thread's pieces of a row: piece0 + 32 c, the warps' shares side by side
  const int pieces = p.K / kPer, slice = (pieces + kWarps - 1) / kWarps;
  const int piece0 = warp * slice + lane, piece_end = min(pieces, (warp + 1) * slice);
  const unsigned char *weights = static_cast<const unsigned char *>(p.w) + static_cast<std::size_t>(piece0) * 16;
  const auto source_of = [&](const int row) {
    unsigned int weight_row = column0 + row;
    if (gated) {
      const bool second = row >= columns;
      weight_row -= second ? columns : 0;
      weight_row += (weight_row & ~127U) + (second ? 128U : 0U);
    }
    return weights + static_cast<std::size_t>(weight_row) * row_bytes;
  };
  // a step reads its weights once and more of them than L2 holds: they are the first to go, and states, caches, parameters
  // and the kernels' own code stay (48 steps of Gigusun 11.84 -> 11.33 ms, of Kikepel 11.4 -> 10.2, whose chains of small
  // kernels had their code come from memory step after step)
  std::uint64_t once;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
  const auto copy = [&](const int unit, const int piece, const unsigned char *const source, const int c) {
    if (piece0 + 32 * c < piece_end)
      asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(static_cast<std::uint32_t>(
                       __cvta_generic_to_shared(ring + (unit * kUnit + piece) * kThreads + tid))),
                   "l"(source + 512 * c), "l"(once)
                   : "memory");
  };
  int next_row = 0, next_chunk = 0;  // what the next unit holds
  const auto fetch = [&](const int unit) {
    if constexpr (kUnit == 1) {
      if (next_row < rows) copy(unit, 0, source_of(next_row), next_chunk);
      if (++next_chunk == kChunks) next_chunk = 0, ++next_row;
    } else {
#pragma unroll
      for (int r = 0; r < kRowsPerStage; ++r) {
        if (next_row + r < rows) {
          const unsigned char *const source = source_of(next_row + r);
#pragma unroll
          for (int c = 0; c < kChunks; ++c) copy(unit, r * kChunks + c, source, c);
        }
      }
      next_row += kRowsPerStage;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // pieces past the thread's share stay zero, on both sides of the product (single pieces: their slots change, so they
  // are skipped instead)
  if constexpr (kUnit != 1) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (piece0 + 32 * c >= piece_end)
        for (int i = 0; i < kUnits * kRowsPerStage; ++i) ring[(i * kChunks + c) * kThreads + tid] = make_uint4(0U, 0U, 0U, 0U);
  }
  const auto fill = [&] {
#pragma unroll
    for (int unit = 0; unit < kUnits; ++unit) fetch(unit);
  };
  using Source = std::conditional_t<kFront == Front::kRms, float, X>;
  const Source *x = static_cast<const Source *>(p.x);
  if (grouped) {
    // which weights these are is a result of the kernel in front, or of one further back
    const int *row_group = p.row_group;
    if (!p.row_group_settled) wait_for_producers(x, row_group);
    weights += static_cast<std::size_t>(__ldcg(row_group + blockIdx.y)) * p.N * row_bytes;
    fill();
    release_dependents();
    if (p.row_group_settled) wait_for_producers(x);
    x += static_cast<std::size_t>(blockIdx.y / p.row_fanout) * p.K;
  } else {
    fill();
    release_dependents();
    wait_for_producers(x);
  }
  constexpr bool kEarlyAddends = kChunks * kPer <= 64;
  Addends early;
  if (kEarlyAddends && tid < columns) early = addends_of(p, 0, blockIdx.y, out_columns, column0 + tid);
  // what a front multiplies with is on its way beside x as well, where there are registers for it
  constexpr bool kEarlyGain = kFront == Front::kRms && kChunks <= 2;
  float xv[kChunks][kPer], gain[kEarlyGain ? kChunks : 1][8], factors[4];
  if constexpr (kFront == Front::kPoly) {
#pragma unroll
    for (int i = 0; i < 4; ++i) factors[i] = p.front[i];
  }
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    if (piece0 + 32 * c < piece_end) {
      if constexpr (kEarlyGain) load_floats<8>(p.front + static_cast<std::size_t>(piece0 + 32 * c) * 8, gain[c]);
      const Source *const source = x + static_cast<std::size_t>(piece0 + 32 * c) * kPer;
      if constexpr (std::is_same_v<Source, float>) load_floats<8>(source, xv[c]);
      else unpack16<kFp8>(*reinterpret_cast<const uint4 *>(source), xv[c]);
    } else {
#pragma unroll
      for (int i = 0; i < kPer; ++i) xv[c][i] = 0.0F;
    }
  }
  if constexpr (kFront != Front::kNone) {
    __shared__ float team_scratch[kTeams][3][kWarps];
    auto &scratch = team_scratch[team];
    constexpr int kSums = kFront == Front::kPoly ? 3 : 1;
    float sums[3] = {0.0F, 0.0F, 0.0F};  // of squares, fourth and sixth powers
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const float v = xv[c][i], square = v * v;
        if constexpr (kFront == Front::kPoly) {
          sums[0] += square;
          sums[1] = fmaf(square, square, sums[1]);
          sums[2] = fmaf(square * square, square, sums[2]);
        } else {
          sums[0] = fmaf(v, v, sums[0]);
        }
      }
#pragma unroll
    for (int k = 0; k < kSums; ++k) {
      sums[k] = warp_sum(sums[k]);
      if (lane == 0) scratch[k][warp] = sums[k];
    }
    team_barrier();
    const float inverse_width = 1.0F / static_cast<float>(p.K);
#pragma unroll
    for (int k = 0; k < kSums; ++k) {
      sums[k] = 0.0F;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) sums[k] += scratch[k][w];
      sums[k] = sums[k] * inverse_width + p.epsilon;
    }
    const auto rounded = [](const float v) { return to_float(from_float<X>(v)); };
    if constexpr (kFront == Front::kRms) {
      const float factor = 1.0F / sqrtf(sums[0]);
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
        if (piece0 + 32 * c < piece_end) {
          const int at = kEarlyGain ? c : 0;
          if constexpr (!kEarlyGain) load_floats<8>(p.front + static_cast<std::size_t>(piece0 + 32 * c) * 8, gain[0]);
#pragma unroll
          for (int i = 0; i < 8; ++i) xv[c][i] = rounded(xv[c][i] * factor * gain[at][i]);
        }
    } else {
      const float a = factors[0] * rsqrtf(sums[0]), b = factors[1] * rsqrtf(sums[1]), c3 = factors[2] * rsqrtf(sums[2]);
      const float e = factors[3];
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
        if (piece0 + 32 * c < piece_end) {
#pragma unroll
          for (int i = 0; i < kPer; ++i) xv[c][i] = rounded(fmaf(fmaf(fmaf(c3, xv[c][i], b), xv[c][i], a), xv[c][i], e));
        }
    }
  }
  int unit = 0;
  const auto advance = [&] {
    fetch(unit);
    unit = unit + 1 == kUnits ? 0 : unit + 1;
  };
  const auto dot = [&](const int piece, const int c) {
    float wv[kPer], sum = 0.0F;
    unpack16<kFp8>(ring[(unit * kUnit + piece) * kThreads + tid], wv);
#pragma unroll
    for (int i = 0; i < kPer; ++i) sum = fmaf(xv[c][i], wv[i], sum);
    return sum;
  };
  for (int group = 0; group < groups; ++group) {
    float sum[kRowsPerStage];
    if constexpr (kUnit == 1) {
      float part[kChunks];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kUnits - 1) : "memory");
        part[c] = piece0 + 32 * c < piece_end ? dot(0, c) : 0.0F;
        advance();
      }
      sum[0] = part[0];
#pragma unroll
      for (int c = 1; c < kChunks; ++c) sum[0] += part[c];
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(kUnits - 1) : "memory");
#pragma unroll
      for (int r = 0; r < kRowsPerStage; ++r) {
        sum[r] = dot(r * kChunks, 0);
#pragma unroll
        for (int c = 1; c < kChunks; ++c) sum[r] += dot(r * kChunks + c, c);
      }
      advance();
    }
    // halves of the warp keep half of the rows each until one is left per lane
    int row = group * kRowsPerStage, offset = 16;
#pragma unroll
    for (int held = kRowsPerStage; held > 1; held /= 2, offset /= 2) {
      const bool upper = (lane & offset) != 0;
      row += upper ? held / 2 : 0;
#pragma unroll
      for (int r = 0; r < held / 2; ++r) {
        const float keep = upper ? sum[r + held / 2] : sum[r], give = upper ? sum[r] : sum[r + held / 2];
        sum[r] = keep + __shfl_xor_sync(0xffffffffU, give, offset);
      }
    }
#pragma unroll
    for (int step = 16 / kRowsPerStage; step > 0; step /= 2) sum[0] += __shfl_xor_sync(0xffffffffU, sum[0], step);
    if (lane % (32 / kRowsPerStage) == 0 && row < rows) partial[row * kWarps + warp] = sum[0];
  }
  team_barrier();
  const float alpha = p.row_scale != nullptr ? p.alpha * p.row_scale[blockIdx.y] : p.alpha;
  for (int local = tid; local < columns; local += kThreads)
    finish_column(p, blockIdx.y, out_columns, column0 + local, alpha, local,
                  kEarlyAddends && local == tid ? early : addends_of(p, 0, blockIdx.y, out_columns, column0 + local),
                  [&](const int index) {  // (of a gated pair: 2 local, 2 local + 1)
                    const int row = gated ? (index & 1) * columns + index / 2 : index;
                    const float4 a = reinterpret_cast<const float4 *>(partial)[2 * row],
                                 b = reinterpret_cast<const float4 *>(partial)[2 * row + 1];
                    return ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
                  });
}

// CTAs across the columns of each of `rows` output rows: together about one per SM.
int stream_grid(const int out_columns, const int rows) {
  const int wanted = std::max(1, kSmCount / rows);
  return std::min((out_columns + kTeams - 1) / kTeams, wanted);
}
// Sizes that the one-row kernel has registers (K) and partial sums (N) for.
template <bool kFp8>
bool stream_applicable(const GemvParams &p) {
  const int out_columns = p.gate_mode != 0 ? p.N / 2 : p.N, grid = kTeams * stream_grid(out_columns, p.rows);
  return p.K <= (kFp8 ? 6 * 16 : 8 * 8) * kWarps * 32 &&
         ((out_columns - 1) / grid + 1) * (p.gate_mode != 0 ? 2 : 1) <= kStreamRows;
}

// One row, or grouped rows with a weight each.
template <bool kFp8, class X, Front kFront = Front::kNone>
int launch_stream(const GemvParams &p, cudaStream_t stream) {
  constexpr int kPer = kFp8 ? 16 : 8;
  const int pieces = p.K / kPer, chunks = ((pieces + kWarps - 1) / kWarps + 31) / 32;
  const dim3 grid(static_cast<unsigned int>(stream_grid(p.gate_mode != 0 ? p.N / 2 : p.N, p.rows)),
                  static_cast<unsigned int>(p.rows));
  const auto launch = [&](auto chunk_count, auto stage_rows) {
    constexpr int kC = decltype(chunk_count)::value, kR = decltype(stage_rows)::value;
    const auto kernel = gemv_stream_kernel<kFp8, X, kFront, kC, kR, kC >= 4 ? 1 : kC * kR>;
    // (with the largest split for shared memory an SM need not change its split between streams and the kernels with larger
    // tiles: 19 tokens and 3 steps of a 1920-wide model 1.347 -> 1.329 ms, 16 F32 steps of Gigusun 4.30 -> 4.27)
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamShared) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess)
      return fail(kCuda, "cannot raise the shared-memory limit of the one-row projection kernel");
    return launch_dependent("one-row projection kernel", kernel, grid, kTeams * kThreads, kStreamShared, stream, p.dependent_launch != 0,
                            1, p);
  };
  using std::integral_constant;
  switch (chunks) {
    case 1: return launch(integral_constant<int, 1>{}, integral_constant<int, 4>{});
    case 2: return launch(integral_constant<int, 2>{}, integral_constant<int, 2>{});
    case 3: return launch(integral_constant<int, 3>{}, integral_constant<int, 1>{});
    case 4: return launch(integral_constant<int, 4>{}, integral_constant<int, 1>{});
    case 5: return launch(integral_constant<int, 5>{}, integral_constant<int, 1>{});
    case 6: return launch(integral_constant<int, 6>{}, integral_constant<int, 1>{});
    default:
      if constexpr (!kFp8) return launch(integral_constant<int, 8>{}, integral_constant<int, 1>{});
      return fail(kInternal, "one-row projection kernel without registers for this K");
  }
}

// 2..8 rows, single calls, sizes beyond the kernel above: four weight rows per CTA; a gated projection then produces two
// output columns per CTA.
constexpr int kColumnsPerCta = 4;

template <bool kFp8>
int launch_gemv(const GemvParams &p, cudaStream_t stream) {
  if constexpr (!kFp8)
    if (p.front != nullptr)
      return p.poly_front ? launch_stream<false, bf16, Front::kPoly>(p, stream) : launch_stream<false, bf16, Front::kRms>(p, stream);
  // Single calls start behind everything else, with their ring empty: of BF16 weights a CTA per four of them is then as
  // fast or faster (alone: 64 x 64 4.2 us against 5.3, 11264 x 4096 20.5 against 22.2, 8192 x 8192 26.7 against 30.5), of
  // E4M3 up to some thousand columns (8448 x 2048 8.3 and 10.3, 4096 x 4096 8.3 and 8.5; 4096 x 12288 16.5 and 14.3).
  // Grouped rows read a weight each and start with a lookup either way: all but short ones take the stream (4 rows of
  // 2048 x 2816 14.3 and 13.7, 16 rows 45 and 32; 2 rows of 256 x 512 4.4 and 6.1).
  const bool stream_rows = p.weight_stream || (p.row_group != nullptr ? p.K >= 1024 : kFp8 && p.N >= 8192);
  if (stream_rows && (p.rows == 1 || p.row_group != nullptr) && stream_applicable<kFp8>(p))
    return launch_stream<kFp8, std::conditional_t<kFp8, std::uint8_t, bf16>>(p, stream);
  const int out_columns = p.gate_mode != 0 ? p.N / 2 : p.N;
  const int per_cta = p.gate_mode != 0 ? kColumnsPerCta / 2 : kColumnsPerCta;
  const dim3 grid(static_cast<unsigned int>((out_columns + per_cta - 1) / per_cta),
                  p.row_group != nullptr ? static_cast<unsigned int>(p.rows) : 1U);
  GemvParams q = p;
  if (p.row_group != nullptr) q.rows = 1;
  const auto kernel = q.rows == 1   ? gemv_kernel<kFp8, 1, kColumnsPerCta>
                      : q.rows <= 2 ? gemv_kernel<kFp8, 2, kColumnsPerCta>
                      : q.rows <= 4 ? gemv_kernel<kFp8, 4, kColumnsPerCta>
                                    : gemv_kernel<kFp8, 8, kColumnsPerCta>;
  return launch_dependent("small-batch projection kernel", kernel, grid, kThreads, 0, stream, p.dependent_launch != 0, 1, q);
}

}  // namespace

bool small_batch_linear_applicable(const LinearArgs &a) {
  const bool fp8 = a.operand_type == OperandType::kE4m3;
  const std::size_t per_chunk = fp8 ? 16 : 8;
  return a.rows >= 1 && a.rows <= (a.row_group != nullptr ? std::size_t{65535} : static_cast<std::size_t>(kMaxRows)) && !a.force_simt &&
         a.in_features % per_chunk == 0 && a.in_features >= per_chunk &&
         (reinterpret_cast<std::uintptr_t>(a.input) & 15U) == 0 &&
         (reinterpret_cast<std::uintptr_t>(a.weight) & 15U) == 0 &&
         a.out_features <= 0x7fffffffU && a.in_features <= 0x7fffffffU &&
         (a.gate_mode == 0 || a.out_features % 256 == 0);
}

bool row_front_applicable(const RowFront &front, const void *const input, const void *const weight,
                          const std::size_t in_features, const std::size_t out_features) {
  if (in_features % 8 != 0 || in_features == 0 || !aligned16(input) || !aligned16(weight) || (!front.poly && !aligned16(front.values)) || in_features > 0x7fffffffU ||
      out_features > 0x7fffffffU)
    return false;
  GemvParams p{};
  p.rows = 1;
  p.K = static_cast<int>(in_features);
  p.N = static_cast<int>(out_features);
  return stream_applicable<false>(p);
}

bool one_row_linear_f32_applicable(const LinearF32Args &a) {
  if (a.rows != 1 || a.row_group != nullptr || a.tile_group != nullptr || a.in_features % 8 != 0 || !aligned16(a.input) ||
      !aligned16(a.weight) || a.in_features > 0x7fffffffU || a.out_features > 0x7fffffffU)
    return false;
  GemvParams p{};
  p.rows = 1;
  p.K = static_cast<int>(a.in_features);
  p.N = static_cast<int>(a.out_features);
  return stream_applicable<false>(p);
}

int one_row_linear_f32(const LinearF32Args &a, cudaStream_t stream) {
  GemvParams p{};
  p.x = a.input;
  p.w = a.weight;
  p.out_f32 = a.output;
  p.bias_f32 = a.bias;
  p.accumulate_f32 = a.accumulate ? 1 : 0;
  p.rows = 1;
  p.K = static_cast<int>(a.in_features);
  p.N = static_cast<int>(a.out_features);
  p.alpha = a.alpha;
  p.softcap = a.softcap;
  p.row_scale = a.row_scale;
  p.dependent_launch = a.dependent_launch ? 1 : 0;
  p.front = a.front.values;
  p.epsilon = a.front.epsilon;
  if (a.front.values != nullptr)
    return a.front.poly ? launch_stream<false, float, Front::kPoly>(p, stream) : launch_stream<false, float, Front::kRms>(p, stream);
  return a.input_type == Activation::kBf16 ? launch_stream<false, bf16>(p, stream) : launch_stream<false, float>(p, stream);
}

int small_batch_linear(const LinearArgs &a, cudaStream_t stream) {
  GemvParams p{};
  p.x = a.input;
  p.w = a.weight;
  p.bias = static_cast<const bf16 *>(a.bias);
  p.residual = static_cast<const bf16 *>(a.residual);
  p.out = static_cast<bf16 *>(a.output);
  p.out_f32 = a.output_f32;
  p.bias_f32 = a.bias_f32;
  p.accumulate_f32 = a.accumulate_f32 ? 1 : 0;
  p.rows = static_cast<int>(a.rows);
  p.K = static_cast<int>(a.in_features);
  p.N = static_cast<int>(a.out_features);
  p.alpha = a.alpha;
  p.bias_mode = a.bias_mode;
  p.gate_mode = a.gate_mode;
  p.dependent_launch = a.dependent_launch && (a.rows == 1 || a.row_group != nullptr) ? 1 : 0;
  p.weight_stream = a.weight_stream;
  p.gate_limit = a.gate_limit;
  p.softcap = a.softcap;
  p.row_group = a.row_group;
  p.row_fanout = static_cast<int>(a.row_fanout);
  p.row_group_settled = a.row_group_settled && a.dependent_launch ? 1 : 0;
  p.row_scale = a.row_scale;
  p.front = a.front.values;
  p.epsilon = a.front.epsilon;
  p.poly_front = a.front.poly;
  return a.operand_type == OperandType::kE4m3 ? launch_gemv<true>(p, stream)
                                              : launch_gemv<false>(p, stream);
}

}  // namespace evob
