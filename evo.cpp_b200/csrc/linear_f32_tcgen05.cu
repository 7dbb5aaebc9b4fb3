// F32 projections of a few rows or more on the tensor cores, with all bits of the operands: an F32 value of at least 2^-110 is
// the exact sum of three BF16 values (its significand's 24 bits in eights, cut toward zero), a BF16 weight is one, and so a
// product is the sum of three exact BF16 products.  Below 2^-110 the bits of a value below 2^-133 are lost, at most 2^-133 |w| of
// a product; multiply-adds keep them.
//
// The weights are the M = 128 operand and stream through shared memory once (TMA, 64 K values a block); the rows are the
// narrow one, split into their planes by eight warps that read them as F32 from L2.  A K block's 192 products per output
// are summed in TMEM, the small planes first, and eight other warps add each block's sums to F32 registers: the tensor
// core cuts its sums toward zero, and 64 terms of the largest plane are as far as that may go.  A cluster divides K and
// adds its CTAs' sums in order.
//
// What bounds it: up to some dozens of rows the weight stream (32 rows of 4096 x 4096: 17 us, 2 TB/s) and the start and end of a
// CTA; at 90 rows the latencies of a block's steps (tensor pipe 33 %, issue slots 37 %, no unit above 45 %); at 1,000 rows L1, which
// takes the rows in as F32 and the planes (71 %), with the tensor pipe at 43 % and issue slots at 51 %.  90 rows of a 2048-wide model with 8448 inner columns: 25 products in 0.48 ms, 3.18
// as multiply-adds on the CUDA cores; 90 rows of 2048 x 8448 20 us behind one another, 1,000 rows 149.
// Errors against float64 (2-norm over normal operands, against multiply-adds in the CUDA cores' tiles): smaller where products
// have both signs, 0.9e-7 against 1.1e-7 at K = 256, 1.05e-7 against 2.1e-7 at 2048, 1.2e-7 against 4.2e-7 at 8448.  Where all
// have one sign the cuts add up: results are 0.85e-7 of themselves too small on average (1.4e-7 where a few values carry a
// sum; multiply-adds below 1e-9), and errors 0.96e-7 against 0.52e-7, 0.99e-7 against 0.67e-7 and 1.00e-7 against 1.02e-7.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "linear_f32.cuh"
#include "ops_internal.hpp"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace evob {
namespace {

using namespace tc;

constexpr int kWeightRows = 128, kBlockK = 64, kMostSplits = 8;
constexpr int kProducerWarp = 0, kMmaWarp = 1, kSplitWarp = 10, kWorkers = 256, kF32Threads = 64 + 2 * kWorkers;

template <int BT, int kPlanes>
struct F32Layout {
  static constexpr int kWBytes = kWeightRows * kBlockK * 2, kPlaneBytes = BT * kBlockK * 2;
  static constexpr int kStageBytes = kWBytes + kPlanes * kPlaneBytes;
  static constexpr int kStages = std::min(216 * 1024 / kStageBytes, 6);
  static constexpr int kBarrierOffset = kStages * kStageBytes;
  static constexpr int kBarrierCount = 3 * kStages + 4;  // weights full[], rows full[], empty[], sums full[2], sums empty[2]
  static constexpr int kTmemPtrOffset = kBarrierOffset + kBarrierCount * 8;
  static constexpr int kAbortOffset = kTmemPtrOffset + 8;
  static constexpr int kColumnOffset = kAbortOffset + 8;  // a byte per weight row of the tile: some weight is infinite
  static constexpr int kTotal = kColumnOffset + kWeightRows + 1024;  // + alignment slack
  static constexpr int kBufferColumns = BT <= 32 ? 32 : BT <= 64 ? 64 : 128;
  static constexpr int kSumStride = kWeightRows + 4;
  static_assert(kStages >= 3 && BT * kSumStride * 4 <= kBarrierOffset, "the sums take the ring's place");
};

// Values that are not finite lie in the largest plane alone, so that their products and sums are those of multiply-adds.  An
// infinite weight is left: planes that are zero meet it and give a NaN where the value gives an infinity.  A column that has
// such a weight makes its results that are not finite again in plain multiply-adds, a warp each; a CTA with any result that is
// not finite looks for these columns once, whatever its rows hold.  (1,024 rows of 2048 x 2816 that fill up eight experts' tiles: 70 us
// where they are finite, 152 where they are NaNs or infinities; 80 and 2700 with every such result made again.)
__device__ __noinline__ bool any_infinite(const bf16 *const w, const int K) {
  std::uint32_t infinite = 0;
#pragma unroll 4
  for (int k = 8 * (threadIdx.x % 32); k < K; k += 256) {
    const uint4 v = *reinterpret_cast<const uint4 *>(w + k);
    const std::uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      infinite |= (words[i] & 0x7fffU) == 0x7f80U || (words[i] & 0x7fff0000U) == 0x7f800000U ? 1U : 0U;
  }
  return __any_sync(0xffffffffU, infinite != 0) != 0;
}
__device__ __forceinline__ std::uint64_t pair_of(const float lo, const float hi) {
  std::uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ std::uint64_t fma_pair(const std::uint64_t a, const std::uint64_t b, const std::uint64_t c) {
  std::uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
template <typename T>
__device__ __noinline__ float plain_product(const T *const x, const bf16 *const w, const int K) {
  float sum = 0.0F;
  for (int k = threadIdx.x % 32; k < K; k += 32) sum = fmaf(to_float(x[k]), bf2f(w[k]), sum);
  return warp_sum(sum);
}

template <typename T, int BT>
__global__ void __launch_bounds__(kF32Threads, 1)
linear_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const T *__restrict__ input, const F32Params p,
                          int *const error_word) {
  constexpr int kPlanes = std::is_same_v<T, float> ? 3 : 1;
  using L = F32Layout<BT, kPlanes>;
  extern __shared__ unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int splits = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int m0 = blockIdx.y * BT, n0 = blockIdx.x / splits * kWeightRows;
  int group = 0;
  if (p.tile_group != nullptr) {
    const int tile = m0 / p.tile_rows;
    if (tile >= *p.tile_count) return;  // (the whole cluster)
    group = p.tile_group[tile];
  }
  const int K = p.in_features, blocks = (K + kBlockK - 1) / kBlockK;
  const int first = static_cast<int>(static_cast<long long>(blocks) * rank / splits);
  const int last = static_cast<int>(static_cast<long long>(blocks) * (rank + 1) / splits);

  unsigned char *const smem = smem_raw + ((1024U - (smem_u32(smem_raw) & 1023U)) & 1023U);
  const std::uint32_t smem_base = smem_u32(smem), bar_base = smem_base + L::kBarrierOffset;
  const auto w_full = [&](const int s) { return bar_base + 8U * s; };
  const auto x_full = [&](const int s) { return bar_base + 8U * (L::kStages + s); };
  const auto empty = [&](const int s) { return bar_base + 8U * (2 * L::kStages + s); };
  const auto sums_full = [&](const int b) { return bar_base + 8U * (3 * L::kStages + b); };
  const auto sums_empty = [&](const int b) { return bar_base + 8U * (3 * L::kStages + 2 + b); };
  volatile std::uint32_t *const tmem_ptr = reinterpret_cast<volatile std::uint32_t *>(smem + L::kTmemPtrOffset);
  volatile int *const abort_flag = reinterpret_cast<volatile int *>(smem + L::kAbortOffset);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::kStages; ++s) {
      mbar_init(w_full(s), 1);
      mbar_init(x_full(s), kWorkers);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(sums_full(b), 1);
      mbar_init(sums_empty(b), kWorkers);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::
                     "r"(smem_u32(const_cast<std::uint32_t *>(tmem_ptr))), "r"(2U * L::kBufferColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const std::uint32_t tmem_base = *tmem_ptr;

  if (warp == kProducerWarp) {
    if (lane == 0) {
      const std::uint64_t once = policy_read_once();
      for (int block = first; block < last; ++block) {
        const int i = block - first, stage = i % L::kStages;
        if (i >= L::kStages && !mbar_wait(empty(stage), (i / L::kStages - 1) & 1, abort_flag)) break;
        mbar_expect_tx(w_full(stage), L::kWBytes);
        const std::uint32_t w_dst = smem_base + stage * L::kStageBytes;
        const int weight_row = group * p.out_features + n0;
        if (gridDim.y == 1) tma_load_2d(w_dst, &map_w, w_full(stage), block * kBlockK, weight_row, once);
        else tma_load_2d(w_dst, &map_w, w_full(stage), block * kBlockK, weight_row);
      }
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      constexpr std::uint32_t idesc = 1U << 4U | 1U << 7U | 1U << 10U | static_cast<std::uint32_t>(BT >> 3) << 17U |
                                      static_cast<std::uint32_t>(kWeightRows >> 4) << 24U;
      for (int block = first; block < last; ++block) {
        const int i = block - first, stage = i % L::kStages, buffer = i % 2;
        if (!mbar_wait(w_full(stage), (i / L::kStages) & 1, abort_flag) ||
            !mbar_wait(x_full(stage), (i / L::kStages) & 1, abort_flag) ||
            (i >= 2 && !mbar_wait(sums_empty(buffer), (i / 2 - 1) & 1, abort_flag)))
          break;
        tc_fence_after();
        const std::uint32_t w_addr = smem_base + stage * L::kStageBytes;
        const std::uint64_t w_desc = smem_descriptor(w_addr);
#pragma unroll
        for (int plane = kPlanes - 1; plane >= 0; --plane) {
          const std::uint64_t x_desc = smem_descriptor(w_addr + L::kWBytes + plane * L::kPlaneBytes);
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)
            tc_mma<false>(tmem_base + buffer * L::kBufferColumns, w_desc + 2U * k, x_desc + 2U * k, idesc,
                          plane == kPlanes - 1 && k == 0 ? 0U : 1U);
        }
        tc_commit(empty(stage));
        tc_commit(sums_full(buffer));
      }
    }
  } else if (warp < kSplitWarp) {
    // a warp adds up half of the rows for the 32 weight rows that it reaches
    constexpr int kHalf = BT / 2;
    const int quarter = warp % 4, half = (warp - 2) / 4;
    const std::uint32_t taddr = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16U) + half * kHalf;
    float sum[kHalf];
#pragma unroll
    for (int t = 0; t < kHalf; ++t) sum[t] = 0.0F;
    bool ok = true;
    for (int block = first; block < last; ++block) {
      const int i = block - first, buffer = i % 2;
      ok = mbar_wait(sums_full(buffer), (i / 2) & 1, abort_flag);
      ok = __all_sync(0xffffffffU, ok) != 0;
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < kHalf; c += 32) {
        std::uint32_t v[2][16];
        tmem_load_16(taddr + buffer * L::kBufferColumns + c, v[0]);
        if (c + 16 < kHalf) tmem_load_16(taddr + buffer * L::kBufferColumns + c + 16, v[1]);
        tmem_load_wait();
#pragma unroll
        for (int j = 0; j < 32 && c + j < kHalf; ++j) sum[c + j] += __uint_as_float(v[j / 16][j % 16]);
      }
      tc_fence_before();
      mbar_arrive(sums_empty(buffer));
    }
    // every product has been made: the sums take the ring's place
    if (ok) {
      float *const sums = reinterpret_cast<float *>(smem) + half * kHalf * L::kSumStride + quarter * 32 + lane;
#pragma unroll
      for (int t = 0; t < kHalf; ++t) sums[t * L::kSumStride] = sum[t];
    }
  } else {
    // pieces of eight K values: row piece / 8, values 8 (piece % 8) of the block; two blocks ahead of the tensor cores' ring
    constexpr int kPieces = BT * 8 / kWorkers;
    const int tid = threadIdx.x - 32 * kSplitWarp, chunk = tid % 8;
    float v[2][kPieces][8];
    const auto fetch = [&](float (&to)[kPieces][8], const int block) {
      const int k = block * kBlockK + 8 * chunk;
#pragma unroll
      for (int j = 0; j < kPieces; ++j) {
        const int row = m0 + tid / 8 + 32 * j;
        if (block < last && row < p.rows && k < K) {
          load_floats<8>(input + static_cast<std::size_t>(row) * K + k, to[j]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) to[j][e] = 0.0F;
        }
      }
    };
    const auto store_plane = [&](const float (&from)[8], const int stage, const int row, const int plane) {
      std::uint32_t words[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        words[e] = __byte_perm(__float_as_uint(from[2 * e]), __float_as_uint(from[2 * e + 1]), 0x7632);
      *reinterpret_cast<uint4 *>(smem + stage * L::kStageBytes + L::kWBytes + plane * L::kPlaneBytes + row * 128 + ((chunk ^ (row & 7)) << 4)) =
          make_uint4(words[0], words[1], words[2], words[3]);
    };
    // what a plane leaves
    const auto take_rest = [](float (&from)[8]) {
      const std::uint64_t minus = pair_of(-1.0F, -1.0F);
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const std::uint64_t top = pair_of(__uint_as_float(__float_as_uint(from[e]) & 0xffff0000U),
                                          __uint_as_float(__float_as_uint(from[e + 1]) & 0xffff0000U));
        const std::uint64_t rest = fma_pair(top, minus, pair_of(from[e], from[e + 1]));
        from[e] = __uint_as_float(static_cast<std::uint32_t>(rest));
        from[e + 1] = __uint_as_float(static_cast<std::uint32_t>(rest >> 32U));
      }
    };
    const auto split = [&](float (&from)[kPieces][8], const int block) {
      const int i = block - first, stage = i % L::kStages;
      if (i >= L::kStages && !mbar_wait(empty(stage), (i / L::kStages - 1) & 1, abort_flag)) return false;
      std::uint64_t probe[kPieces];
#pragma unroll
      for (int j = 0; j < kPieces; ++j) {
        const int row = tid / 8 + 32 * j;
#pragma unroll
        for (int plane = 0; plane < kPlanes; ++plane) {
          store_plane(from[j], stage, row, plane);
          if (plane + 1 < kPlanes) take_rest(from[j]);
        }
        // the last rest of a value that is not finite is a NaN
        probe[j] = 0;
#pragma unroll
        for (int e = 0; e < 8; e += 2) probe[j] = fma_pair(pair_of(from[j][e], from[j][e + 1]), 0ULL, probe[j]);
      }
      if constexpr (kPlanes > 1) {
        std::uint64_t any = probe[0];
#pragma unroll
        for (int j = 1; j < kPieces; ++j) any |= probe[j];
        if ((any & 0x7fffffff7fffffffULL) != 0) {
          fetch(from, block);
#pragma unroll
          for (int j = 0; j < kPieces; ++j) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (isnan(from[j][e])) from[j][e] = __uint_as_float(0x7fff0000U);  // one without its lower half, too
#pragma unroll
            for (int plane = 0; plane < kPlanes; ++plane) {
              store_plane(from[j], stage, tid / 8 + 32 * j, plane);
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (!isfinite(from[j][e])) from[j][e] = 0.0F;
              if (plane + 1 < kPlanes) take_rest(from[j]);
            }
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(x_full(stage));
      return true;
    };
    fetch(v[0], first);
    fetch(v[1], first + 1);
    for (int block = first; block < last; block += 2) {
      if (!split(v[0], block)) break;
      fetch(v[0], block + 2);
      if (block + 1 >= last || !split(v[1], block + 1)) break;
      fetch(v[1], block + 3);
    }
  }
  __syncwarp();
  tc_fence_before();
  cluster.sync();
  if (*abort_flag != 0) {
    const unsigned long long start = global_timer_ns();
    while (global_timer_ns() - start < 200000ULL) __nanosleep(1000);
    if (threadIdx.x == 0) atomicOr(error_word, 1 | 32);  // bit 5: a projection kernel
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2U * L::kBufferColumns)
                 : "memory");
  }
  // a share of the tile's rows per CTA, a warp per row
  float *const sums = reinterpret_cast<float *>(smem);
  constexpr int kWarps = kF32Threads / 32, kColumns = kWeightRows / 32;
  const int rows_end = min(BT, p.rows - m0), first_row = rank * kWarps + warp, row_step = splits * kWarps;
  const auto totals = [&](const int r, float (&total)[kColumns]) {
#pragma unroll
    for (int i = 0; i < kColumns; ++i) total[i] = 0.0F;
#pragma unroll
    for (int other0 = 0; other0 < kMostSplits; other0 += 4) {  // (in order, four CTAs' parts on their way)
      if (other0 >= splits) break;
      float part[4][kColumns] = {};
#pragma unroll
      for (int o = 0; o < 4; ++o)
        if (other0 + o < splits) {
          const float *const from = cluster.map_shared_rank(sums, other0 + o) + r * L::kSumStride + lane;
#pragma unroll
          for (int i = 0; i < kColumns; ++i) part[o][i] = from[32 * i];
        }
#pragma unroll
      for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int i = 0; i < kColumns; ++i) total[i] += part[o][i];
    }
  };
  bool odd = false;  // some result has to be looked at again
  for (int r = first_row; r < rows_end; r += row_step) {
    float total[kColumns];
    totals(r, total);
#pragma unroll
    for (int i = 0; i < kColumns; ++i) {
      const int column = n0 + 32 * i + lane;
      if (column >= p.out_features) continue;
      if (kPlanes == 1 || isfinite(total[i])) store_f32_result(p, static_cast<std::size_t>(m0 + r), column, total[i]);
      else odd = true;
    }
  }
  if (kPlanes > 1 && __syncthreads_or(odd) != 0) {
    unsigned char *const infinite = smem + L::kColumnOffset;
    const bf16 *const weights = p.weight + (static_cast<std::size_t>(group) * p.out_features + n0) * K;
    for (int c = warp; c < min(kWeightRows, p.out_features - n0); c += kWarps) {
      const bool found = any_infinite(weights + static_cast<std::size_t>(c) * K, K);
      if (lane == 0) infinite[c] = found ? 1 : 0;
    }
    __syncthreads();
    for (int r = first_row; r < rows_end; r += row_step) {
      float total[kColumns];
      totals(r, total);
#pragma unroll
      for (int i = 0; i < kColumns; ++i) {
        const int column = n0 + 32 * i + lane;
        const bool left = column < p.out_features && !isfinite(total[i]);
        for (std::uint32_t again = __ballot_sync(0xffffffffU, left && infinite[32 * i + lane] != 0); again != 0; again &= again - 1) {
          const int place = __ffs(static_cast<int>(again)) - 1;
          const float plain = plain_product(input + static_cast<std::size_t>(m0 + r) * K,
                                            weights + static_cast<std::size_t>(32 * i + place) * K, K);
          if (lane == place) total[i] = plain;
        }
        if (left) store_f32_result(p, static_cast<std::size_t>(m0 + r), column, total[i]);
      }
    }
  }
  cluster.sync();  // remote shared memory stays alive until every CTA has read it
}

template <typename T, int BT>
int launch(const LinearF32Args &a, const F32Params &p, cudaStream_t stream) {
  using L = F32Layout<BT, std::is_same_v<T, float> ? 3 : 1>;
  int status = kOk;
  int *const error = error_word(&status, nullptr);
  if (error == nullptr) return status;
  CUtensorMap map;
  // (a tile beyond the last group's rows reads zeros, beyond another's rows of the next group: neither is stored)
  status = make_bf16_tile_map(&map, a.weight, a.out_features * (a.tile_group != nullptr ? a.groups : 1), a.in_features, kWeightRows);
  if (status != kOk) return status;
  const auto kernel = linear_f32_tcgen05_kernel<T, BT>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal) != cudaSuccess)
    return fail(kCuda, "cannot raise the shared-memory limit of the F32 linear kernel");
  const unsigned int tiles = ceil_div_u(a.out_features, kWeightRows), row_tiles = ceil_div_u(a.rows, BT);
  const std::size_t blocks = (a.in_features + kBlockK - 1) / kBlockK;
  // The GPCs of a B200 (148 SMs) take so many clusters of 1 to 8 of these CTAs at once (cudaOccupancyMaxActiveClusters; another part
  // would get the same results in other times).  A CTA's K blocks
  // take about as long as its start and end from four blocks on, so the split with the fewest blocks in all waves is best (4096 x
  // 11264, 90 rows: 94 us undivided in one wave, 98 in halves and 74 in thirds in two, 77 in quarters in three).
  constexpr unsigned int kResident[kMostSplits + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  unsigned int splits = 1;
  std::size_t best = ~std::size_t{0};
  for (unsigned int s = 1; s <= kMostSplits && s <= blocks; ++s) {
    const std::size_t waves = (static_cast<std::size_t>(tiles) * row_tiles + kResident[s] - 1) / kResident[s];
    const std::size_t cost = waves * ((blocks + s - 1) / s + 4);
    if (cost < best) best = cost, splits = s;
  }
  return launch_dependent("F32 linear kernel (tensor cores)", kernel, dim3(tiles * splits, row_tiles), kF32Threads, L::kTotal,
                          stream, false, splits, map, static_cast<const T *>(a.input), p, error);
}

}  // namespace

bool tensorcore_linear_f32_applicable(const LinearF32Args &a) {
  return a.in_features % 8 == 0 && a.in_features >= 64 && a.row_group == nullptr &&
         (reinterpret_cast<std::uintptr_t>(a.input) & 15U) == 0 && (reinterpret_cast<std::uintptr_t>(a.weight) & 15U) == 0 &&
         (a.tile_group == nullptr || (a.groups > 0 && a.groups * a.out_features <= 0x7fffffffU));
}

int tensorcore_linear_f32(const LinearF32Args &a, const F32Params &p, cudaStream_t stream) {
  // the row tile that pads the fewest rows, the larger one of equals; grouped row tiles are made of whole ones
  std::size_t best = 0, padded = ~std::size_t{0};
  for (const std::size_t height : {128, 96, 64, 32}) {
    if ((a.tile_group != nullptr && a.tile_rows % height != 0) || (a.rows + height - 1) / height > 65535) continue;
    const std::size_t total = (a.rows + height - 1) / height * height;
    if (total < padded) padded = total, best = height;
  }
  const auto typed = [&](auto tag) {
    using T = decltype(tag);
    switch (best) {
      case 128: return launch<T, 128>(a, p, stream);
      case 96: return launch<T, 96>(a, p, stream);
      case 64: return launch<T, 64>(a, p, stream);
      default: return launch<T, 32>(a, p, stream);
    }
  };
  return a.input_type == Activation::kBf16 ? typed(bf16{}) : typed(float{});
}

}  // namespace evob
