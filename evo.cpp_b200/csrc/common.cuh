// Shared device/host helpers for the sm_100a StripedHyena2 hot path.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <string>

namespace evob {

// Status codes shared with the public C ABI (same numeric values as
// evo_status in include/evo/evo.h).
enum : int {
  kOk = 0,
  kInvalidArgument = 2,
  kIo = 3,
  kModelFormat = 4,
  kUnsupported = 5,
  kCuda = 6,
  kInternal = 70,
};

// Thread-local error text for the operator-level C ABI.
void set_error(int code, const std::string &message);
const char *last_error();
int fail(int code, const std::string &message);
int check_launch(const char *what);

using bf16 = __nv_bfloat16;

__host__ __device__ __forceinline__ unsigned int ceil_div_u(
    const std::size_t a, const std::size_t b) {
  return static_cast<unsigned int>((a + b - 1) / b);
}

__device__ __forceinline__ float bf2f(const bf16 v) {
  return __bfloat162float(v);
}
__device__ __forceinline__ bf16 f2bf(const float v) {
  return __float2bfloat16_rn(v);
}
// Round an F32 value to BF16 precision and widen it again.
__device__ __forceinline__ float rbf(const float v) {
  // one instruction: the packed convert puts bf16(v) in the upper half and
  // bf16(+0) in the lower half, which is the F32 bit pattern of the result
  unsigned int bits;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(bits) : "f"(v), "f"(0.0F));
  return __uint_as_float(bits);
}
__device__ __forceinline__ float bits2f_bf16(const unsigned short bits) {
  return __uint_as_float(static_cast<unsigned int>(bits) << 16U);
}

// 8 BF16 values in one 128-bit register quad.
struct alignas(16) Bf16x8 {
  uint4 raw;
  __device__ __forceinline__ float get(const int i) const {
    const unsigned int word = (&raw.x)[i >> 1];
    return __uint_as_float((i & 1) ? (word & 0xffff0000U) : (word << 16U));
  }
};

__device__ __forceinline__ unsigned int pack_bf16x2(const float lo,
                                                    const float hi) {
  const unsigned int l = __bfloat16_as_ushort(__float2bfloat16_rn(lo));
  const unsigned int h = __bfloat16_as_ushort(__float2bfloat16_rn(hi));
  return l | (h << 16U);
}

constexpr int kSmCount = 148;

// Programmatic dependent launch.  A kernel launched by launch_dependent() may start while the kernel in front of it in
// the stream is still running, once that one has called release_dependents() in all its CTAs (or ended).  Before it
// touches memory that other kernels write or read it calls wait_for_producers(), which returns when the kernel in front
// has completed; every such kernel does so in some thread, hence everything further back has completed as well.  The
// pointers passed are opaque to the compiler behind the wait, so that no load through them can move in front of it: a
// kernel passes every __restrict__ pointer that it reads, gains, tables and weights too (a program may have made them with
// the launch in front), and loads nothing with __ldg, which is for memory that nobody writes while the kernel runs.
// Outputs that a kernel only writes are not passed: what goes there has been read behind the wait, and an opaque pointer
// could be the memory of every load behind a store through it (embed_positions() of 8,192 x 4096: 56 us, 68 when opaque;
// rms_norm() of 1,000 x 8192: 8.5 and 13.7, where the pointers had lost their address space, too).
// Kernels other than weight streams release after their wait: a projection that started earlier still would find the SMs
// unevenly taken by the one in front of this kernel, and where its CTAs land is where they stay (a gated 11264 x 2048
// projection took 12.4 us behind early releases, 7.8 with its CTAs spread evenly).  A kernel that releases and never waits
// has to be launched plainly.
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class Pointer>
__device__ __forceinline__ void make_opaque(Pointer &pointer) {
  std::size_t address = __cvta_generic_to_global(pointer);  // still known to be global memory: no load waits for shared stores
  asm volatile("" : "+l"(address)::"memory");
  pointer = static_cast<Pointer>(__cvta_global_to_generic(address));
}
template <class... Pointers>
__device__ __forceinline__ void wait_for_producers(Pointers &...pointers) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (make_opaque(pointers), ...);
}

// With `dependent` false an ordinary launch.  `cluster` CTAs of neighbouring x indices form a cluster.
template <class... Params, class... Args>
int launch_dependent(const char *const what, void (*const kernel)(Params...), const dim3 grid, const unsigned int threads,
                     const std::size_t shared_bytes, cudaStream_t stream, const bool dependent,
                     const unsigned int cluster, const Args &...args) {
  cudaLaunchAttribute attributes[2]{};
  unsigned int count = 0;
  if (cluster > 1) {
    attributes[count].id = cudaLaunchAttributeClusterDimension;
    attributes[count].val.clusterDim.x = cluster;
    attributes[count].val.clusterDim.y = attributes[count].val.clusterDim.z = 1;
    ++count;
  }
  if (dependent) {
    attributes[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[count].val.programmaticStreamSerializationAllowed = 1;
    ++count;
  }
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  config.attrs = attributes;
  config.numAttrs = count;
  const cudaError_t error = cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
  if (error != cudaSuccess)
    return fail(kCuda, std::string("cannot launch the ") + what + ": " + cudaGetErrorString(error));
  return check_launch(what);
}

}  // namespace evob
