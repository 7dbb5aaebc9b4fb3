// Bit-exact emulation of the Hopper FP8 tensor-core accumulation that
// upstream's "exact" profile pins for the E4M3 Hyena projections
// (src/cuda/ops.cu:277-441, docs/software-fp8.md).  Per output element and
// per group of 32 K values:
//   E     = max(exponent(acc) if acc != 0, max over non-zero products of
//           (e_a + e_b))
//   sum   = trunc(acc / u) + sum_k trunc(a_k b_k / u),  u = 2^(E - 13)
//   acc   = truncate_to_13_fraction_bits(sum u)
// and finally out = bf16(acc * output_scale).
//
// A tensor-core product with an F32 accumulator C adds its 16 products in one alignment: each product's magnitude is cut at
// 2^-25 of the largest exponent among C and the products, and the sum at 2^-23 of its own (measured on the B200 for BF16 and
// F16 operands of mma.sync and tcgen05.mma; every test of this file's results depends on it).  So the emulation's products
// are tensor-core products:
//   * C = 1.5 2^25 u cuts every product at u, for every output its own u;
//   * the sum in C keeps multiples of 4 u only, so every K value takes four of the 16 places, and the sum is 4 times the
//     emulated one and exact;
//   * an E4M3 code's bits in an F16 value's place are the code's value times 2^-8;
//   * the exponent maximum is a product as well: with 2^(6 e) for every operand, a sum over 32 products lies in
//     [2^(6 E), 2^(6 E + 5)], so its F32 exponent divided by 6 is E whatever the accumulator rounds away
//     (e is in [-9, 8], so the exponents stay within F32 and BF16).
// Up to some dozens of rows the products run on mma.sync, here; more rows on tcgen05.mma (qgmma_emulation_tcgen05.cu).
// What bounds it: the unpacking of the weights, of which no step is shared beyond 16 rows, and the latencies of a group's
// chain.  16 rows at 12288 x 4096: 78 us, 8 rows 53 (F32 multiply-adds that truncate, one product in half an instruction and
// its sign in two more: 230).
#include "common.cuh"
#include "ops_internal.hpp"
#include "qgmma_operands.cuh"

namespace evob {
namespace {

using namespace qgmma;

__device__ __forceinline__ void mma_bf16(float (&d)[4], const std::uint32_t (&a)[4], const std::uint32_t b0,
                                         const std::uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_first(float (&d)[4], const std::uint32_t (&a)[4], const std::uint32_t b0,
                                               const std::uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0F));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const std::uint32_t (&a)[4], const std::uint32_t b0,
                                        const std::uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16 weight rows' group as mma.sync's A operands: row g, row g + 8, and for the products the same again.
struct WeightTile {
  std::uint32_t copies[8][4], powers[2][4];
};
__device__ __forceinline__ WeightTile weight_tile_of(const uint2 upper, const uint2 lower) {
  const Operands a = operands_of<true>(upper), b = operands_of<true>(lower);
  WeightTile t;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    t.copies[k][0] = a.copies[k];
    t.copies[k][1] = b.copies[k];
    t.copies[k][2] = a.copies[k];
    t.copies[k][3] = b.copies[k];
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    t.powers[half][0] = a.powers[2 * half];
    t.powers[half][1] = b.powers[2 * half];
    t.powers[half][2] = a.powers[2 * half + 1];
    t.powers[half][3] = b.powers[2 * half + 1];
  }
  return t;
}
// A row's group in shared memory: lane c of a quad reads its eight K values as pairs of copies (two K values per 16-byte
// word, 64 j + 16 c bytes in) and their powers.  Eight lanes of neighbouring rows meet different banks.
struct __align__(16) RowGroup {
  uint4 copies[4][4];
  uint4 powers[4];
};
static_assert(sizeof(RowGroup) % 128 == 64, "neighbouring rows are half of the banks apart");

// One group's step of four accumulators (mma.sync's result layout; 2^-14 of the emulated ones): 16 weight rows and eight
// rows.  Two chains of products halve the wait for each other; they start on either side of zero and meet there.
__device__ __forceinline__ void advance(float (&acc)[4], const WeightTile &w, const RowGroup &x, const int c) {
  float powers[4], sum[4], other[4];
  const uint4 p = x.powers[c];
  mma_bf16_first(powers, w.powers[0], p.x, p.y);
  mma_bf16(powers, w.powers[1], p.z, p.w);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float largest = fmaxf(fabsf(acc[q]), __uint_as_float(sixth_of(__float_as_uint(powers[q]))));
    const float unit = __uint_as_float(__float_as_uint(largest) & 0x7f800000U);
    const float lift = __uint_as_float((__float_as_uint(acc[q]) & 0x80000000U) | 0x44c00000U);  // +-1536: 1.5 2^(12 - 2)
    sum[q] = __fmaf_rz(unit, lift, acc[q]);  // the accumulator's own part, truncated like a product
    other[q] = -(unit * lift);
  }
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const uint4 b = x.copies[k / 2][c];
    mma_f16(sum, w.copies[k], b.x, b.y);
    mma_f16(other, w.copies[k + 1], b.z, b.w);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] = __uint_as_float(__float_as_uint(sum[q] + other[q]) & 0xfffffc00U);  // 13 fraction bits
}

// A CTA owns 16 kWarps output columns (weight rows, unpacked in registers by the one warp that uses them) x 8 kN rows
// (unpacked in shared memory, kDepth groups at a time).
template <int kNTiles, int kWarpCount, int kGroups, int kResident>
struct EmulationShape {
  static constexpr int kN = kNTiles, kWarps = kWarpCount, kDepth = kGroups, kBlocks = kResident;
  static constexpr int kThreads = 32 * kWarps, kRows = 8 * kN, kCols = 16 * kWarps;
  using Stage = RowGroup[kDepth][kRows];
};

template <class Shape>
__global__ void __launch_bounds__(Shape::kThreads, Shape::kBlocks)
qgmma_emulation_kernel(const std::uint8_t *__restrict__ input_codes,
                       const std::uint8_t *__restrict__ weight_codes,
                       bf16 *__restrict__ output, const std::size_t rows,
                       const std::size_t in_features,
                       const std::size_t out_features,
                       const float output_scale) {
  constexpr int kN = Shape::kN, kThreads = Shape::kThreads, kDepth = Shape::kDepth, kRows = Shape::kRows;
  constexpr int kPieces = kRows * 4 * kDepth, kShare = (kPieces + kThreads - 1) / kThreads;
  // (it releases and never waits, so it has to be launched plainly: a dependent launch that completes says nothing about
  // the kernels further back)
  if constexpr (kN == 1) release_dependents();
  using Stage = typename Shape::Stage;
  extern __shared__ __align__(16) unsigned char shared[];
  Stage *const stages = reinterpret_cast<Stage *>(shared);
  const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32, g = lane / 4, c = lane % 4;
  const std::size_t row0 = static_cast<std::size_t>(blockIdx.y) * kRows;
  const std::size_t col0 = static_cast<std::size_t>(blockIdx.x) * Shape::kCols + warp * 16 + g;
  const int groups = static_cast<int>(in_features / kGroup);

  // rows: a thread unpacks eight codes at a time, piece (row, group, eighth)
  uint2 x_codes[kShare];
  const auto fetch_rows = [&](const int group0) {
#pragma unroll
    for (int i = 0; i < kShare; ++i) {
      const int piece = tid + i * kThreads, group = group0 + piece / 4 % kDepth;
      const std::size_t row = row0 + piece / (4 * kDepth);
      x_codes[i] = make_uint2(0U, 0U);
      if ((kPieces % kThreads == 0 || piece < kPieces) && row < rows && group < groups)
        x_codes[i] = __ldg(reinterpret_cast<const uint2 *>(input_codes + row * in_features + group * kGroup + piece % 4 * 8));
    }
  };
  const auto publish_rows = [&](Stage &stage) {
#pragma unroll
    for (int i = 0; i < kShare; ++i) {
      const int piece = tid + i * kThreads;
      if (kPieces % kThreads != 0 && piece >= kPieces) break;
      const Operands o = operands_of<false>(x_codes[i]);
      RowGroup &out = stage[piece / 4 % kDepth][piece / (4 * kDepth)];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        out.copies[j][piece % 4] = make_uint4(o.copies[2 * j], o.copies[2 * j], o.copies[2 * j + 1], o.copies[2 * j + 1]);
      out.powers[piece % 4] = make_uint4(o.powers[0], o.powers[1], o.powers[2], o.powers[3]);
    }
  };
  // weights: a stage's worth of groups in flight
  uint2 w_codes[kDepth][2];
  const std::uint8_t *w_rows[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const std::size_t column = col0 + 8 * h;
    w_rows[h] = weight_codes + (column < out_features ? column : out_features - 1) * in_features + 8 * c;
  }
  const auto fetch_weights = [&](const int d, const int group) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      w_codes[d][h] = __ldg(reinterpret_cast<const uint2 *>(w_rows[h] + min(group, groups - 1) * kGroup));
  };

  float acc[kN][4] = {};
#pragma unroll
  for (int d = 0; d < kDepth; ++d) fetch_weights(d, d);
  fetch_rows(0);
  publish_rows(stages[0]);
  __syncthreads();
  int at = 0;
  for (int group0 = 0; group0 < groups; group0 += kDepth, at ^= 1) {
    const Stage &stage = stages[at];
    const bool more = group0 + kDepth < groups;
    if (more) fetch_rows(group0 + kDepth);
#pragma unroll
    for (int d = 0; d < kDepth; ++d) {  // (a group beyond the last meets rows of zeros and changes nothing)
      const WeightTile w = weight_tile_of(w_codes[d][0], w_codes[d][1]);
      fetch_weights(d, group0 + d + kDepth);
#pragma unroll
      for (int n = 0; n < kN; ++n) advance(acc[n], w, stage[d][8 * n + g], c);
    }
    if (more) publish_rows(stages[at ^ 1]);
    __syncthreads();
  }
#pragma unroll
  for (int n = 0; n < kN; ++n)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const std::size_t column = col0 + q / 2 * 8, row = row0 + 8 * n + 2 * c + q % 2;
      if (row < rows && column < out_features)
        output[row * out_features + column] = f2bf(acc[n][q] * 0x1p14F * output_scale);
    }
}

// One row (cached decode): kLanes neighbouring lanes share one output column and split each 32-product group between them (a
// column's group is one 32-byte sector of codes).  Its products are multiply-adds that round toward zero, of F16 operands into
// F32: positive products are added to 2^23 u, negative ones to -2^23 u, and each addition cuts its product at u.  The row sits
// unpacked in shared memory: magnitudes, powers 2^e, and its sign bits, which the weights' codes take over before they are
// unpacked.  The largest of a group's powers does not need the accumulator: a code's value times the row's power keeps the
// exponent sum.  Maxima and sums go through shuffles side by side; every sum is exact.
constexpr int kRowKernelThreads = 128;
// A row's groups in shared memory: zeros in front of the first (they change nothing) up to whole batches, and two that are
// unpacked ahead.
constexpr int kBatch = 4;
__host__ __device__ constexpr int row_batches(const int groups) { return (groups + kBatch - 1) / kBatch; }
constexpr std::size_t kEightBytes = 2 * sizeof(uint4) + sizeof(uint2);  // per eight K values
constexpr std::size_t row_bytes(const int groups) { return (row_batches(groups) * kBatch + 2) * (kGroup / 8) * kEightBytes; }

// c + the product of a's and b's F16 halves, rounded toward zero.
template <int kHalf>
__device__ __forceinline__ float cut_product(const std::uint32_t a, const std::uint32_t b, const float c) {
  float d;
  asm("fma.rz.f32.f16 %0, %1, %2, %3;"
      : "=f"(d)
      : "h"(static_cast<unsigned short>(kHalf == 0 ? a : a >> 16U)), "h"(static_cast<unsigned short>(kHalf == 0 ? b : b >> 16U)), "f"(c));
  return d;
}
__device__ __forceinline__ std::uint32_t multiplied_halves(const std::uint32_t a, const std::uint32_t b) {
  std::uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ std::uint32_t larger_halves(const std::uint32_t a, const std::uint32_t b) {
  std::uint32_t d;
  asm("max.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ std::uint32_t smaller_halves(const std::uint32_t a, const std::uint32_t b) {
  std::uint32_t d;
  asm("min.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// The larger magnitudes, with some sign.
__device__ __forceinline__ std::uint32_t larger_magnitudes(const std::uint32_t a, const std::uint32_t b) {
  std::uint32_t d;
  asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// Four codes as F16 pairs, 2^-8 of their values.
__device__ __forceinline__ uint2 halves_of(const std::uint32_t codes) {
  const std::uint32_t upper = (codes & 0x80808080U) | ((codes >> 1U) & 0x3f3f3f3fU), lower = (codes << 7U) & 0x80808080U;
  return make_uint2(__byte_perm(lower, upper, 0x5140), __byte_perm(lower, upper, 0x7362));
}

template <int kLanes, int kAhead>
__global__ void __launch_bounds__(kRowKernelThreads)
qgmma_emulation_row_kernel(const std::uint8_t *__restrict__ input_codes,
                            const std::uint8_t *__restrict__ weight_codes,
                            bf16 *__restrict__ output, const std::size_t in_features,
                            const std::size_t out_features, const float output_scale) {
  // (it releases and never waits, so it has to be launched plainly: a dependent launch that completes says nothing about
  // the kernels further back)
  release_dependents();
  constexpr int kCodes = kGroup / kLanes, kWords = kCodes / 4, kEights = kCodes / 8, kGroupEights = kGroup / 8;
  static_assert(kAhead % kBatch == 0 && kAhead > kBatch && kWords % 2 == 0);
  extern __shared__ __align__(16) unsigned char shared[];
  const int groups = static_cast<int>(in_features / kGroup), batches = row_batches(groups);
  const int front = batches * kBatch - groups, eights = (batches * kBatch + 2) * kGroupEights;
  uint4 *const x_magnitude = reinterpret_cast<uint4 *>(shared);            // [eights] 2^5 of the values
  uint4 *const x_power = x_magnitude + eights;                             // [eights] 2^5 of the powers
  uint2 *const x_sign = reinterpret_cast<uint2 *>(x_power + eights);       // [eights] sign bits where the codes have them
  for (int i = threadIdx.x; i < eights; i += kRowKernelThreads) {
    const int at = i - front * kGroupEights;
    const uint2 codes = at >= 0 && at < groups * kGroupEights ? __ldg(reinterpret_cast<const uint2 *>(input_codes) + at) : make_uint2(0U, 0U);
    std::uint32_t magnitude[4], power[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const std::uint32_t word = h == 0 ? codes.x : codes.y;
      const uint2 x = halves_of(word & 0x7f7f7f7fU);
      magnitude[2 * h] = multiplied_halves(x.x, 0x70007000U);  // 2^13: every value but 0 is a normal F16 number then
      magnitude[2 * h + 1] = multiplied_halves(x.y, 0x70007000U);
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) power[h] = magnitude[h] & 0x7c007c00U;
    x_magnitude[i] = make_uint4(magnitude[0], magnitude[1], magnitude[2], magnitude[3]);
    x_power[i] = make_uint4(power[0], power[1], power[2], power[3]);
    x_sign[i] = make_uint2(codes.x & 0x80808080U, codes.y & 0x80808080U);
  }
  __syncthreads();
  const int part_lane = threadIdx.x % kLanes;
  const std::size_t column =
      static_cast<std::size_t>(blockIdx.x) * (kRowKernelThreads / kLanes) + threadIdx.x / kLanes;
  // the lanes of a column are in or out together, and all lanes reach the shuffles below
  const bool active = column < out_features;
  struct alignas(kCodes) Codes {
    std::uint32_t word[kWords];
  };
  const Codes *const weights = reinterpret_cast<const Codes *>(
      weight_codes + (active ? column : 0) * in_features + part_lane * kCodes);
  const auto load = [](const Codes *const from) {
    Codes c;
    if constexpr (kWords == 4) {
      const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(from));
      c.word[0] = v.x, c.word[1] = v.y, c.word[2] = v.z, c.word[3] = v.w;
    } else {
      const uint2 v = __ldcs(reinterpret_cast<const uint2 *>(from));
      c.word[0] = v.x, c.word[1] = v.y;
    }
    return c;
  };
  float acc = 0.0F;  // 2^-3 of the emulated one, as all that follows
  Codes codes[kAhead];
  // a place's group of the row; in front of the first one, whose row's values are zeros, and behind the last one some group
#pragma unroll
  for (int i = 0; i < kAhead; ++i) codes[i] = load(weights + min(max(i - front, 0), groups - 1) * kLanes);
  const auto refill = [&](const int batch, const int slot) {
    const Codes *const from = weights + (min(batch, batches - 1) * kBatch - front) * kLanes;
#pragma unroll
    for (int j = 0; j < kBatch; ++j) codes[slot + j] = load(from + (batches > 1 ? j : max(j, front)) * kLanes);
  };

  // The weights of two groups, by their products' signs, and this lane's part of each group's largest power.
  std::uint32_t positive[2][kCodes / 2], negative[2][kCodes / 2], high[2];
  const auto unpack = [&](const int buffer, const int group, const Codes &raw) {
    std::uint32_t most = 0;
#pragma unroll
    for (int e = 0; e < kEights; ++e) {
      const int at = group * kGroupEights + part_lane * kEights + e;
      const uint4 power = x_power[at];
      const uint2 sign = x_sign[at];
      const uint2 lower = halves_of(raw.word[2 * e] ^ sign.x), upper = halves_of(raw.word[2 * e + 1] ^ sign.y);
      const std::uint32_t pairs[4] = {lower.x, lower.y, upper.x, upper.y}, powers[4] = {power.x, power.y, power.z, power.w};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        positive[buffer][4 * e + h] = larger_halves(pairs[h], 0U);
        negative[buffer][4 * e + h] = smaller_halves(pairs[h], 0U);
        // 2^-3 of a mantissa in [1, 2) times 2^e: exact from 2^-21 to 2^14, subnormals included
        most = larger_magnitudes(most, multiplied_halves(pairs[h], powers[h]));
      }
    }
    high[buffer] = most & 0x7fff7fffU;
  };
  // 2^e of a group's largest product in an F32's exponent, less than any if there is none.
  const auto largest_of = [](const std::uint32_t halves) {
    const float2 both = __half22float2(*reinterpret_cast<const __half2 *>(&halves));
    return __float_as_uint(fmaxf(fmaxf(both.x, both.y), 0x1p-25F));
  };
  unpack(0, 0, codes[0]);
  unpack(1, 1, codes[1]);
  std::uint32_t first = high[0];
#pragma unroll
  for (int step = 1; step < kLanes; step *= 2) first = larger_halves(first, __shfl_xor_sync(0xffffffffU, first, step));
  std::uint32_t largest = largest_of(first);
  for (int base = 0; base < batches; base += kAhead / kBatch) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (i % kBatch == 0) {
        if (base + i / kBatch >= batches) break;
        if (i > 0) refill(base + (kAhead + i) / kBatch - 1, i - kBatch);
      }
      const int group = base * kBatch + i;
      const std::uint32_t top = max(largest, __float_as_uint(acc) & 0x7fffffffU) & 0x7f800000U;
      const float magic = __uint_as_float(top + (10U << 23U));  // 2^23 u
      float plus = magic, minus = -magic;
#pragma unroll
      for (int e = 0; e < kEights; ++e) {
        const uint4 x = x_magnitude[group * kGroupEights + part_lane * kEights + e];
        const std::uint32_t values[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          plus = cut_product<0>(positive[i % 2][4 * e + h], values[h], plus);
          minus = cut_product<0>(negative[i % 2][4 * e + h], values[h], minus);
          plus = cut_product<1>(positive[i % 2][4 * e + h], values[h], plus);
          minus = cut_product<1>(negative[i % 2][4 * e + h], values[h], minus);
        }
      }
      float sum = plus + minus;  // (both below 2^24 u: the difference is exact)
      std::uint32_t next = high[(i + 1) % 2];
#pragma unroll
      for (int step = 1; step < kLanes; step *= 2) {
        const float others = __shfl_xor_sync(0xffffffffU, sum, step);
        const std::uint32_t others_high = __shfl_xor_sync(0xffffffffU, next, step);
        if (step == 1) unpack(i % 2, group + 2, codes[(i + 2) % kAhead]);
        sum += others;
        next = larger_halves(next, others_high);
      }
      largest = largest_of(next);
      // the accumulator's own part is truncated the same way as a product, and the total to 13 fraction bits
      const float lift = copysignf(magic, acc);
      const float own = __fadd_rz(acc, lift) - lift;
      acc = __uint_as_float(__float_as_uint(own + sum) & 0xfffffc00U);
    }
    refill(base + 2 * (kAhead / kBatch) - 1, kAhead - kBatch);
  }
  if (active && part_lane == 0) output[column] = f2bf(acc * 8.0F * output_scale);
}

template <class Kernel>
int allow_shared_memory(Kernel *const kernel, const std::size_t bytes) {
  if (bytes > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(bytes)) != cudaSuccess)
    return fail(kCuda, "cannot raise the emulation kernel shared-memory limit");
  return kOk;
}

template <class Shape>
int launch_tiled(const void *input_codes, const void *weight_codes, const std::size_t rows,
                 const std::size_t in_features, const std::size_t out_features, const float output_scale,
                 void *output, cudaStream_t stream) {
  const dim3 grid(ceil_div_u(out_features, Shape::kCols), ceil_div_u(rows, Shape::kRows));
  if (grid.y > 65535) return fail(kInvalidArgument, "software E4M3 linear has too many rows");
  constexpr std::size_t smem = 2 * sizeof(typename Shape::Stage);
  auto *const kernel = qgmma_emulation_kernel<Shape>;
  const int status = allow_shared_memory(kernel, smem);
  if (status != kOk) return status;
  kernel<<<grid, Shape::kThreads, smem, stream>>>(
      static_cast<const std::uint8_t *>(input_codes), static_cast<const std::uint8_t *>(weight_codes),
      static_cast<bf16 *>(output), rows, in_features, out_features, output_scale);
  return check_launch("software E4M3 QGMMA emulation kernel");
}

}  // namespace

int e4m3_emulated_gemm(const void *input_codes, const void *weight_codes,
                       const std::size_t rows, const std::size_t in_features,
                       const std::size_t out_features,
                       const float output_scale, void *output,
                       cudaStream_t stream) {
  if (input_codes == nullptr || weight_codes == nullptr || output == nullptr ||
      in_features == 0 || out_features == 0 || in_features % kGroup != 0 ||
      !isfinite(output_scale))
    return fail(kInvalidArgument,
                "software E4M3 linear needs K to be a multiple of 32 and "
                "valid buffers");
  if (rows == 0) return kOk;
  if ((reinterpret_cast<std::uintptr_t>(input_codes) & 7U) != 0 ||
      (reinterpret_cast<std::uintptr_t>(weight_codes) & 7U) != 0)
    return fail(kInvalidArgument,
                "software E4M3 linear code buffers must be 8-byte aligned");
  if (rows == 1 && in_features <= 24576 &&
      (reinterpret_cast<std::uintptr_t>(weight_codes) & 15U) == 0) {
    // Two lanes per column share the fixed work of a group between more products, four keep more warps in flight and are
    // the faster ones while three CTAs per SM hold all columns: one row at N x K = 5760 x 1920 takes 18 us with either,
    // at 12288 x 4096 39 with two and 35 with four, at 14336 x 4096 39 and 41, at 24576 x 8192 86 and 112 (the products as
    // pairs of F32 multiply-adds, cut and signed one by one: 25, 48, 55 and 122).  Bound by a group's chain of dependent
    // steps (256 columns x 4096 take 27 us) and then by the unpacking, seven instructions for four codes.
    const bool two_lanes = out_features > 3 * std::size_t{148} * (kRowKernelThreads / 4);
    const unsigned int blocks = ceil_div_u(out_features, kRowKernelThreads / (two_lanes ? 2 : 4));
    auto *const kernel = two_lanes ? qgmma_emulation_row_kernel<2, 16> : qgmma_emulation_row_kernel<4, 16>;
    const std::size_t bytes = row_bytes(static_cast<int>(in_features / kGroup));
    const int status = allow_shared_memory(kernel, bytes);
    if (status != kOk) return status;
    // (not a dependent launch: started beside a projection that still runs, its CTAs crowd on the SMs that are free
    // first, and this kernel is bound by its arithmetic: 85 us against 41 when it was measured)
    kernel<<<blocks, kRowKernelThreads, bytes, stream>>>(
        static_cast<const std::uint8_t *>(input_codes),
        static_cast<const std::uint8_t *>(weight_codes), static_cast<bf16 *>(output),
        in_features, out_features, output_scale);
    return check_launch("software E4M3 QGMMA emulation row kernel");
  }
  const auto tiled = [&](auto shape) {
    return launch_tiled<decltype(shape)>(input_codes, weight_codes, rows, in_features, out_features, output_scale,
                                         output, stream);
  };
  if (rows <= 8) return tiled(EmulationShape<1, 4, 8, 4>{});
  // A group takes about 0.25 us + 1.65 us per 2^20 outputs here (16 rows per warp); with the rows in tiles of 64 on tcgen05.mma
  // 1.4 us while every CTA has an SM of its own and 2.15 us per 296 CTAs beyond (12288 x 4096: 33 rows 135 and 164 us, 64 rows
  // 195 and 164; 5760 x 1920: 128 rows 82 and 90 us, 509 rows 242 and 201).
  const std::size_t flat = (rows + 15) / 16 * 16;
  const std::size_t ctas = (rows + 63) / 64 * ((out_features + 127) / 128), pairs = (ctas + 295) / 296;
  const double here = 0.25 + 1.65e-6 * static_cast<double>(flat) * static_cast<double>(out_features);
  if ((ctas <= 148 ? 1.4 : 2.15 * static_cast<double>(pairs)) < here)
    return e4m3_emulated_gemm_tcgen05(input_codes, weight_codes, rows, in_features, out_features, output_scale, output, stream);
  return tiled(EmulationShape<2, 4, 4, 4>{});
}

}  // namespace evob
