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
// No tensor-core product reproduces the per-group alignment, so the products
// are CUDA-core work; the parts around them are arranged to cost little:
//   * a product and its truncation are one FMA: |a||b| + 2^23 u rounded toward
//     zero is 2^23 u + trunc(|a||b| / u) u, because the sum lies in a binade
//     whose ulp is u (|a||b| < 2^(E + 2) = 2^15 u) and |a||b| has 8 significant
//     bits.  The integer is then the low 16 bits of the result.  Two K values
//     share a packed FMA (fma.rz.f32x2);
//   * the integers of two K values are packed into one word and added with
//     their signs by dp2a; the signs are +-1 bytes, four K values per word, and
//     their product is an exclusive or of the operands' words (one of them
//     stored with its bit 0 flipped);
//   * the exponent maximum is a tensor-core product: with 2^(6 e) for every
//     operand, a sum over 32 products lies in [2^(6 E), 2^(6 E + 5)], so its
//     F32 exponent divided by 6 is E whatever the accumulator rounds away
//     (e is in [-9, 8], so the exponents stay within F32 and BF16).
//     mma.sync's result layout is the thread's output tile.
// What bounds it: the ALU (packing, signs, staging) and the half of the FMA pipe
// that dp2a shares with the multiply-adds, busy for 52 and 55 % of the time with 16
// warps per SM, in bursts that meet each other; about 3 instructions per product.  509 rows at 12288 x 4096: 3.5
// ms = 7.4 T products/s; integer shifts per product took 17.1 ms.
#include "common.cuh"
#include "ops_internal.hpp"

namespace evob {
namespace {

constexpr int kGroup = 32;

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

// 2^E as F32 bits.  `powers` is the sum over the group's products of 2^(6 e) times 2^5 (stored with one operand), so
// its exponent field is 132 + 6 E + 0 .. 5.  Without a product this gives E = -22: products' E is at least -18, so an
// accumulator is a multiple of 2^-31 and loses nothing to a unit of 2^-35.
__device__ __forceinline__ std::uint32_t largest_bits(const float powers, const float acc) {
  const std::uint32_t sixth = ((__float_as_uint(powers) >> 15U) * 43691U) >> 26U;  // floor(field / 6)
  return max((sixth << 23U) + (105U << 23U), __float_as_uint(acc) & 0x7f800000U);
}
// One group's step of an accumulator: `sum` is the signed sum of the truncated products in units of u.  The
// accumulator's own part is truncated the same way as a product; all of it is exact in F32 (below 2^24 u).
__device__ __forceinline__ float advanced(const float acc, const int sum, const std::uint32_t largest) {
  const float magic = copysignf(__uint_as_float(largest + (10U << 23U)), acc);
  const float own = __fadd_rz(acc, magic) - magic;
  const float total = __fmaf_rn(static_cast<float>(sum), __uint_as_float(largest - (13U << 23U)), own);
  return __uint_as_float(__float_as_uint(total) & 0xfffffc00U);
}

__device__ __forceinline__ std::uint32_t shared_address(const void *pointer) {
  return static_cast<std::uint32_t>(__cvta_generic_to_shared(pointer));
}
__device__ __forceinline__ void load_matrices(std::uint32_t (&r)[4], const std::uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const std::uint32_t (&a)[4], const std::uint32_t b0,
                                         const std::uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Rows (or columns) of one operand's group in shared memory.  The strides keep the 16-byte accesses of eight
// neighbouring lines on different banks.
template <int kLines>
struct OperandTile {
  float magnitude[kLines][kGroup + 4];
  std::uint32_t sign[kLines][kGroup / 4 + 4];
  std::uint16_t power[kLines][kGroup + 8];  // BF16 2^(6 e) times a scale, 0 for a zero
};

// Two BF16 values 2^(6 e) scale of two magnitudes (0 for a zero).
__device__ __forceinline__ std::uint32_t powers_of(const float lo, const float hi, const std::uint64_t scale) {
  const std::uint64_t p = pair_of(__uint_as_float(__float_as_uint(lo) & 0x7f800000U),
                                  __uint_as_float(__float_as_uint(hi) & 0x7f800000U));
  std::uint64_t square, fourth, result;
  asm("mul.f32x2 %0, %1, %1;" : "=l"(square) : "l"(p));
  asm("mul.f32x2 %0, %1, %2;" : "=l"(fourth) : "l"(square), "l"(scale));
  asm("mul.f32x2 %0, %1, %1;" : "=l"(result) : "l"(square));
  asm("mul.f32x2 %0, %1, %2;" : "=l"(result) : "l"(result), "l"(fourth));
  return __byte_perm(static_cast<std::uint32_t>(result), static_cast<std::uint32_t>(result >> 32U), 0x7632);
}

// Eight codes of line `line`, K positions [k, k + 8) of the group.
template <int kLines>
__device__ __forceinline__ void unpack(OperandTile<kLines> &tile, const int line, const int k, const uint2 codes,
                                       const std::uint32_t sign_flip, const float scale) {
  const float4 lo = magnitudes_of(codes.x), hi = magnitudes_of(codes.y);
  *reinterpret_cast<float4 *>(&tile.magnitude[line][k]) = lo;
  *reinterpret_cast<float4 *>(&tile.magnitude[line][k + 4]) = hi;
  *reinterpret_cast<uint2 *>(&tile.sign[line][k / 4]) =
      make_uint2(signs_of(codes.x) ^ sign_flip, signs_of(codes.y) ^ sign_flip);
  const std::uint64_t scales = pair_of(scale, scale);
  *reinterpret_cast<uint4 *>(&tile.power[line][k]) =
      make_uint4(powers_of(lo.x, lo.y, scales), powers_of(lo.z, lo.w, scales), powers_of(hi.x, hi.y, scales),
                 powers_of(hi.z, hi.w, scales));
}

// A CTA of eight warps owns kTileRows x kTileCols outputs, a warp 16 kM x 8 kN of them in mma.sync's layout.
template <int kTileRows, int kTileCols, int kM, int kN>
struct EmulationShape {
  static constexpr int kRows = kTileRows, kCols = kTileCols, kMTiles = kM, kNTiles = kN;
  static constexpr int kRowWarps = kTileRows / (16 * kM);
  static_assert(kRowWarps * (kTileCols / (8 * kN)) == 8, "eight warps");
  struct Stage {
    OperandTile<kTileRows> a;
    OperandTile<kTileCols> b;
  };
};

constexpr int kEmulationThreads = 256;

template <class Shape>
__global__ void __launch_bounds__(kEmulationThreads)
qgmma_emulation_kernel(const std::uint8_t *__restrict__ input_codes,
                       const std::uint8_t *__restrict__ weight_codes,
                       bf16 *__restrict__ output, const std::size_t rows,
                       const std::size_t in_features,
                       const std::size_t out_features,
                       const float output_scale) {
  constexpr int kM = Shape::kMTiles, kN = Shape::kNTiles;
  using Stage = typename Shape::Stage;
  extern __shared__ __align__(16) unsigned char shared[];
  Stage *const stages = reinterpret_cast<Stage *>(shared);
  const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
  const int warp_row = warp % Shape::kRowWarps * (16 * kM), warp_col = warp / Shape::kRowWarps * (8 * kN);
  const std::size_t row0 = static_cast<std::size_t>(blockIdx.y) * Shape::kRows;
  const std::size_t col0 = static_cast<std::size_t>(blockIdx.x) * Shape::kCols;

  // staging: a thread unpacks eight codes of a line at a time
  constexpr int kALoads = Shape::kRows * 4 / kEmulationThreads, kBLoads = Shape::kCols * 4 / kEmulationThreads;
  constexpr int kAShare = kALoads == 0 ? 1 : kALoads;
  uint2 a_codes[kAShare], b_codes[kBLoads];
  const bool loads_a = kALoads != 0 || tid < Shape::kRows * 4;
  const auto fetch = [&](const std::size_t k0) {
#pragma unroll
    for (int i = 0; i < kAShare; ++i) {
      const std::size_t row = row0 + (tid + i * kEmulationThreads) / 4;
      a_codes[i] = loads_a && row < rows
                       ? __ldg(reinterpret_cast<const uint2 *>(input_codes + row * in_features + k0 + tid % 4 * 8))
                       : make_uint2(0U, 0U);
    }
#pragma unroll
    for (int i = 0; i < kBLoads; ++i) {
      const std::size_t col = col0 + (tid + i * kEmulationThreads) / 4;
      b_codes[i] = col < out_features
                       ? __ldg(reinterpret_cast<const uint2 *>(weight_codes + col * in_features + k0 + tid % 4 * 8))
                       : make_uint2(0U, 0U);
    }
  };
  const auto stage_codes = [&](Stage &stage) {
    if (loads_a) {
#pragma unroll
      for (int i = 0; i < kAShare; ++i) unpack(stage.a, (tid + i * kEmulationThreads) / 4, tid % 4 * 8, a_codes[i], 0U, 1.0F);
    }
#pragma unroll
    for (int i = 0; i < kBLoads; ++i)
      unpack(stage.b, (tid + i * kEmulationThreads) / 4, tid % 4 * 8, b_codes[i], 0x01010101U, 32.0F);
  };

  float acc[kM][kN][4];
#pragma unroll
  for (int m = 0; m < kM; ++m)
#pragma unroll
    for (int n = 0; n < kN; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[m][n][q] = 0.0F;

  fetch(0);
  stage_codes(stages[0]);
  __syncthreads();
  for (std::size_t k0 = 0, at = 0; k0 < in_features; k0 += kGroup, at ^= 1) {
    const Stage &stage = stages[at];
    const bool more = k0 + kGroup < in_features;
    if (more) fetch(k0 + kGroup);

    // E of every output
    float powers[kM][kN][4];
    {
      std::uint32_t b_power[kN][2][2];
#pragma unroll
      for (int n = 0; n < kN; ++n) {
        std::uint32_t r[4];  // the four 8-wide K blocks of eight columns
        load_matrices(r, shared_address(&stage.b.power[warp_col + n * 8 + lane % 8][lane / 8 * 8]));
        b_power[n][0][0] = r[0];
        b_power[n][0][1] = r[1];
        b_power[n][1][0] = r[2];
        b_power[n][1][1] = r[3];
      }
#pragma unroll
      for (int m = 0; m < kM; ++m) {
        std::uint32_t a_power[2][4];
#pragma unroll
        for (int half = 0; half < 2; ++half)
          load_matrices(a_power[half],
                        shared_address(&stage.a.power[warp_row + m * 16 + lane % 16][half * 16 + lane / 16 * 8]));
#pragma unroll
        for (int n = 0; n < kN; ++n) {
#pragma unroll
          for (int q = 0; q < 4; ++q) powers[m][n][q] = 0.0F;
#pragma unroll
          for (int half = 0; half < 2; ++half)
            mma_bf16(powers[m][n], a_power[half], b_power[n][half][0], b_power[n][half][1]);
        }
      }
    }
    std::uint64_t magic[kM][kN][4];
    int sum[kM][kN][4];
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float value = __uint_as_float(largest_bits(powers[m][n][q], acc[m][n][q]) + (10U << 23U));
          magic[m][n][q] = pair_of(value, value);
          sum[m][n][q] = 0;
        }

#pragma unroll  // (two steps at a time: 3 % slower, four 16 %; with all of them the packing mixes with the multiply-adds)
    for (int k = 0; k < kGroup; k += 4) {
      std::uint64_t a_value[kM][2][2], b_value[kN][2][2];
      std::uint32_t a_sign[kM][2], b_sign[kN][2];
#pragma unroll
      for (int m = 0; m < kM; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int line = warp_row + m * 16 + h * 8 + lane / 4;
          const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&stage.a.magnitude[line][k]);
          a_value[m][h][0] = v.x;
          a_value[m][h][1] = v.y;
          a_sign[m][h] = stage.a.sign[line][k / 4];
        }
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int line = warp_col + n * 8 + lane % 4 * 2 + h;
          const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&stage.b.magnitude[line][k]);
          b_value[n][h][0] = v.x;
          b_value[n][h][1] = v.y;
          b_sign[n][h] = stage.b.sign[line][k / 4];
        }
#pragma unroll
      for (int m = 0; m < kM; ++m)
#pragma unroll
        for (int n = 0; n < kN; ++n)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const std::uint64_t t0 = truncated_products(a_value[m][q / 2][0], b_value[n][q % 2][0], magic[m][n][q]);
            const std::uint64_t t1 = truncated_products(a_value[m][q / 2][1], b_value[n][q % 2][1], magic[m][n][q]);
            const int sign = static_cast<int>(a_sign[m][q / 2] ^ b_sign[n][q % 2]);
            sum[m][n][q] = __dp2a_lo(static_cast<int>(low_halves(t0)), sign, sum[m][n][q]);
            sum[m][n][q] = __dp2a_hi(static_cast<int>(low_halves(t1)), sign, sum[m][n][q]);
          }
    }
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          acc[m][n][q] = advanced(acc[m][n][q], sum[m][n][q],
                                  static_cast<std::uint32_t>(magic[m][n][q]) - (10U << 23U));
    if (more) stage_codes(stages[at ^ 1]);
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < kM; ++m)
#pragma unroll
    for (int n = 0; n < kN; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const std::size_t row = row0 + warp_row + m * 16 + q / 2 * 8 + lane / 4;
        const std::size_t column = col0 + warp_col + n * 8 + lane % 4 * 2 + q % 2;
        if (row < rows && column < out_features)
          output[row * out_features + column] = f2bf(acc[m][n][q] * output_scale);
      }
}

// One or two rows (cached decode): kLanes neighbouring lanes share one output
// column and split each 32-product group between them (a column's group is one
// 32-byte sector of codes).  The group maximum and the aligned integer sum are
// combined across them with shuffles - integer addition is exact, so the
// result is the one accumulator chain of the tiled kernel above, bit for bit.
// The rows sit unpacked in shared memory: their magnitudes, signs and, two to a
// word, exponent fields; the maximum of a group's exponent sums does not need
// the accumulator and is taken a group ahead of it.
constexpr int kRowKernelThreads = 128;

template <int kRows, int kLanes, int kAhead>
__global__ void __launch_bounds__(kRowKernelThreads)
qgmma_emulation_rows_kernel(const std::uint8_t *__restrict__ input_codes,
                            const std::uint8_t *__restrict__ weight_codes,
                            bf16 *__restrict__ output, const std::size_t in_features,
                            const std::size_t out_features, const float output_scale) {
  // (it releases and never waits, so it has to be launched plainly: a dependent launch that completes says nothing about
  // the kernels further back)
  release_dependents();
  constexpr int kCodes = kGroup / kLanes, kWords = kCodes / 4;
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
  kernel<<<grid, kEmulationThreads, smem, stream>>>(
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
  if (rows <= 2 && row_bytes <= 168 * 1024 &&
      (reinterpret_cast<std::uintptr_t>(weight_codes) & 15U) == 0) {
    // Two lanes per column share the fixed work of a group between more products, four keep more warps in flight:
    // one row at N x K = 24576 x 8192 takes 133 us with two and 166 with four, at 12288 x 4096 66 and 59 us, at
    // 5760 x 1920 38 and 33 us.  From two warps per scheduler on (148 x 256 threads) two lanes are enough.
    const bool two_lanes = out_features * 2 >= std::size_t{148} * 256;
    const unsigned int blocks = ceil_div_u(out_features, kRowKernelThreads / (two_lanes ? 2 : 4));
    auto *const kernel = rows == 1 ? (two_lanes ? qgmma_emulation_rows_kernel<1, 2, 8> : qgmma_emulation_rows_kernel<1, 4, 16>)
                                   : (two_lanes ? qgmma_emulation_rows_kernel<2, 2, 8> : qgmma_emulation_rows_kernel<2, 4, 16>);
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
  // The largest tile amortises the unpacking and the fixed work of a group best (1,024 rows, 12288 x 4096: 6.8 ms
  // against 7.4 ms with 32 rows), unless it pads more rows or leaves SMs without their two CTAs (61 rows: 0.69
  // against 0.57 ms; 200 rows: 1.98 against 1.79 ms; 16 rows: 0.39 ms with 32 rows per tile, 0.25 ms with 16).
  if (rows <= 16) return tiled(EmulationShape<16, 64, 1, 1>{});
  const std::size_t tiles64 = (rows + 63) / 64, tiles32 = (rows + 31) / 32;
  if (tiles64 * 64 * 100 <= tiles32 * 32 * 106 && tiles64 * ceil_div_u(out_features, 64) >= std::size_t{2} * 148)
    return tiled(EmulationShape<64, 64, 2, 2>{});
  return tiled(EmulationShape<32, 64, 2, 1>{});
}

}  // namespace evob
