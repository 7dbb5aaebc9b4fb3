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

// An E4M3 magnitude as F32: the code's seven bits are a float's exponent and
// mantissa up to a factor of 2^120, which also normalises subnormal codes
// (src/cuda/ops.cu:310-332; code 0x7f counts as 480).
__device__ __forceinline__ float magnitude_of(const std::uint32_t code_at_bit_20) {
  return __uint_as_float(code_at_bit_20) * 0x1p120F;
}
// The four codes of a word as magnitudes.
__device__ __forceinline__ float4 magnitudes_of(const std::uint32_t codes) {
  return make_float4(magnitude_of((codes & 0x7fU) << 20U), magnitude_of((codes & 0x7f00U) << 12U),
                     magnitude_of((codes & 0x7f0000U) << 4U), magnitude_of((codes >> 4U) & 0x07f00000U));
}
// +1 (0x01) or -1 (0xff) per code of a word.
__device__ __forceinline__ std::uint32_t signs_of(const std::uint32_t codes) {
  return ((codes >> 7U) & 0x01010101U) * 0xfeU + 0x01010101U;
}

// |a0||b0| + m0 and |a1||b1| + m1, both rounded toward zero.
__device__ __forceinline__ std::uint64_t truncated_products(const std::uint64_t a, const std::uint64_t b,
                                                            const std::uint64_t m) {
  std::uint64_t d;
  asm("fma.rz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(m));
  return d;
}
__device__ __forceinline__ std::uint64_t pair_of(const float lo, const float hi) {
  std::uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
// The low halves of both words of a pair.
__device__ __forceinline__ std::uint32_t low_halves(const std::uint64_t pair) {
  return __byte_perm(static_cast<std::uint32_t>(pair), static_cast<std::uint32_t>(pair >> 32U), 0x5410);
}

// One group's step of an accumulator: `sum` is the signed sum of the truncated products in units of u.  The
// accumulator's own part is truncated the same way as a product; all of it is exact in F32 (below 2^24 u).
__device__ __forceinline__ float advanced(const float acc, const int sum, const std::uint32_t largest) {
  const float magic = copysignf(__uint_as_float(largest + (10U << 23U)), acc);
  const float own = __fadd_rz(acc, magic) - magic;
  const float total = __fmaf_rn(static_cast<float>(sum), __uint_as_float(largest - (13U << 23U)), own);
  return __uint_as_float(__float_as_uint(total) & 0xfffffc00U);
}

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

// One row (cached decode): kLanes neighbouring lanes share one output
// column and split each 32-product group between them (a column's group is one
// 32-byte sector of codes).  The group maximum and the aligned integer sum are
// combined across them with shuffles - integer addition is exact, so the
// result is the one accumulator chain of the tiled kernel above, bit for bit.
// The row sits unpacked in shared memory: its magnitudes, signs and, two to a
// word, exponent fields; the maximum of a group's exponent sums does not need
// the accumulator and is taken a group ahead of it.
constexpr int kRowKernelThreads = 128;

template <int kLanes, int kAhead>
__global__ void __launch_bounds__(kRowKernelThreads)
qgmma_emulation_row_kernel(const std::uint8_t *__restrict__ input_codes,
                            const std::uint8_t *__restrict__ weight_codes,
                            bf16 *__restrict__ output, const std::size_t in_features,
                            const std::size_t out_features, const float output_scale) {
  // (it releases and never waits, so it has to be launched plainly: a dependent launch that completes says nothing about
  // the kernels further back)
  release_dependents();
  constexpr int kRows = 1, kCodes = kGroup / kLanes, kWords = kCodes / 4;
  extern __shared__ __align__(16) unsigned char shared[];
  float *const x_magnitude = reinterpret_cast<float *>(shared);                                // [kRows][in_features]
  std::uint32_t *const x_field = reinterpret_cast<std::uint32_t *>(x_magnitude + kRows * in_features);  // [..][/ 2]
  std::uint32_t *const x_sign = x_field + kRows * in_features / 2;                             // [kRows][in_features / 4]
  const auto fields_of = [](const float lo, const float hi) {  // exponent fields at bits 7 and 23
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632) & 0x7f807f80U;
  };
  for (std::size_t i = threadIdx.x; i < kRows * in_features / 4; i += kRowKernelThreads) {
    const std::uint32_t codes = __ldg(reinterpret_cast<const std::uint32_t *>(input_codes) + i);
    const float4 v = magnitudes_of(codes);
    reinterpret_cast<float4 *>(x_magnitude)[i] = v;
    reinterpret_cast<uint2 *>(x_field)[i] = make_uint2(fields_of(v.x, v.y), fields_of(v.z, v.w));
    x_sign[i] = signs_of(codes) ^ 0x01010101U;
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
  const std::size_t groups = in_features / kGroup;
  const auto fetch = [&](const std::size_t group) {
    Codes c;
    const std::size_t at = (group < groups ? group : groups - 1) * kLanes;
    if constexpr (kWords == 4) {
      const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(weights + at));
      c.word[0] = v.x, c.word[1] = v.y, c.word[2] = v.z, c.word[3] = v.w;
    } else {
      const uint2 v = __ldcs(reinterpret_cast<const uint2 *>(weights + at));
      c.word[0] = v.x, c.word[1] = v.y;
    }
    return c;
  };
  float acc[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) acc[r] = 0.0F;
  Codes codes[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) codes[i] = fetch(i);

  float4 w[kWords];  // the current group's weights ...
  std::uint32_t w_sign[kWords];
  std::uint32_t largest[kRows];  // ... and 2^e of its largest product as F32 bits, less than any if there is none
  const auto open = [&](const std::size_t group, const Codes &raw) {
    std::uint32_t w_field[kCodes / 2];
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      w[i] = magnitudes_of(raw.word[i]);
      w_sign[i] = signs_of(raw.word[i]);
      w_field[2 * i] = fields_of(w[i].x, w[i].y);
      w_field[2 * i + 1] = fields_of(w[i].z, w[i].w);
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const uint2 *const f =
          reinterpret_cast<const uint2 *>(x_field + (r * in_features + group * kGroup + part_lane * kCodes) / 2);
      // a zero's field is 0: its sum (at most 135) stays below every real one (fields are 118 to 135)
      std::uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < kWords; ++i) {
        const uint2 v = f[i];
        m = __viaddmax_u16x2(v.x, w_field[2 * i], m);
        m = __viaddmax_u16x2(v.y, w_field[2 * i + 1], m);
      }
      m = max(m >> 16U, m & 0xffffU);  // (e + 254) << 7
#pragma unroll
      for (int step = 1; step < kLanes; step *= 2) m = max(m, __shfl_xor_sync(0xffffffffU, m, step));
      largest[r] = (max(m, 232U << 7U) << 16U) - (127U << 23U);
    }
  };
  open(0, codes[0]);
  for (std::size_t base = 0; base < groups; base += kAhead) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const std::size_t group = base + i;
      if (group >= groups) break;
      codes[i] = fetch(group + kAhead);
      std::uint32_t top[kRows];
      int sum[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        top[r] = max(largest[r], __float_as_uint(acc[r]) & 0x7f800000U);
        const float value = __uint_as_float(top[r] + (10U << 23U));
        const std::uint64_t magic = pair_of(value, value);
        const std::size_t at = r * in_features + group * kGroup + part_lane * kCodes;
        int part[kWords];
#pragma unroll
        for (int i4 = 0; i4 < kWords; ++i4) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(x_magnitude + at + 4 * i4);
          const int sign = static_cast<int>(x_sign[at / 4 + i4] ^ w_sign[i4]);
          part[i4] = __dp2a_lo(
              static_cast<int>(low_halves(truncated_products(x.x, pair_of(w[i4].x, w[i4].y), magic))), sign, 0);
          part[i4] = __dp2a_hi(
              static_cast<int>(low_halves(truncated_products(x.y, pair_of(w[i4].z, w[i4].w), magic))), sign, part[i4]);
        }
        sum[r] = part[0];
#pragma unroll
        for (int i4 = 1; i4 < kWords; ++i4) sum[r] += part[i4];
      }
      if (group + 1 < groups) open(group + 1, codes[(i + 1) % kAhead]);
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
#pragma unroll
        for (int step = 1; step < kLanes; step *= 2) sum[r] += __shfl_xor_sync(0xffffffffU, sum[r], step);
        acc[r] = advanced(acc[r], sum[r], top[r]);
      }
    }
  }
  if (active && part_lane == 0) {
#pragma unroll
    for (int r = 0; r < kRows; ++r)
      output[r * out_features + column] = f2bf(acc[r] * output_scale);
  }
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
  // per K value of a row: magnitude, half a word of exponent field, a sign byte
  const std::size_t row_bytes = rows * in_features * 7;
  if (rows == 1 && row_bytes <= 168 * 1024 &&
      (reinterpret_cast<std::uintptr_t>(weight_codes) & 15U) == 0) {
    // Two lanes per column share the fixed work of a group between more products, four keep more warps in flight:
    // one row at N x K = 24576 x 8192 takes 133 us with two and 166 with four, at 12288 x 4096 66 and 59 us, at
    // 5760 x 1920 38 and 33 us.  From two warps per scheduler on (148 x 256 threads) two lanes are enough.
    const bool two_lanes = out_features * 2 >= std::size_t{148} * 256;
    const unsigned int blocks = ceil_div_u(out_features, kRowKernelThreads / (two_lanes ? 2 : 4));
    auto *const kernel = two_lanes ? qgmma_emulation_row_kernel<2, 8> : qgmma_emulation_row_kernel<4, 16>;
    const int status = allow_shared_memory(kernel, row_bytes);
    if (status != kOk) return status;
    // (not a dependent launch: started beside a projection that still runs, its CTAs crowd on the SMs that are free
    // first, and this kernel is bound by its arithmetic: 85 us against 41)
    kernel<<<blocks, kRowKernelThreads, row_bytes, stream>>>(
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
