// What the kernels of F32 projections share: their parameters and the way a product becomes a result.
#pragma once

#include "decoder_types.cuh"
#include "gates.cuh"

namespace evob {

struct F32Params {
  const bf16 *weight;
  float *output;
  int rows, out_features, in_features, accumulate;
  float alpha, softcap;
  const float *row_scale, *bias;
  const int *row_group;
  int row_fanout;
  const int *tile_group, *tile_count;
  int tile_rows;
};

__device__ __forceinline__ void store_f32_result(const F32Params &p, const std::size_t row, const int column,
                                                 const float product) {
  float *const out = p.output + row * p.out_features + column;
  float value = product * (p.row_scale != nullptr ? p.alpha * p.row_scale[row] : p.alpha);
  if (p.accumulate != 0) value += *out;
  if (p.bias != nullptr) value += p.bias[column];
  *out = soft_cap(value, p.softcap);
}

// linear_f32_tcgen05.cu: products of F32 (or BF16) rows on the tensor cores; `groups` weight matrices.
bool tensorcore_linear_f32_applicable(const LinearF32Args &args);
int tensorcore_linear_f32(const LinearF32Args &args, const F32Params &params, cudaStream_t stream);

}  // namespace evob
