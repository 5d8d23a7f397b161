// Shared device helpers for the sm_100a kernels of easyllm_b200.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define ELL_API extern "C" __attribute__((visibility("default")))

namespace ell {

constexpr int kNumSMs = 148;  // B200: 2 dies x 74 SMs

struct __align__(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ bf16x8 pack8(const float* f) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum for blockDim.x <= 1024 (multiple of 32).  `red` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();  // protect `red` from the previous use
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nw ? red[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nw ? red[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// ---- chains of kernels -------------------------------------------------------------------------
// A decode step is some fifty launches of 2 to 30 us, and between two dependent ones the GPU drains and refills.  The kernels
// of that path are therefore launched with programmatic stream serialization: the next kernel's CTAs come in while the last
// ones of this kernel run, set up their barriers, TMEM and tensor maps, and wait where they first touch global memory.
//   * every thread of such a kernel calls chain_wait before its first global access (reads AND writes: the kernel before may
//     still read what this one writes), in every CTA and on every path, so that "kernel N has finished" implies that all
//     kernels before N have;
//   * chain_next lets the next kernel in once all CTAs have called it.  It comes after tcgen05.alloc: a CTA let in earlier
//     could take the TMEM that this one still needs while it waits for this one to finish;
//   * before chain_wait only prefetches into L2 are allowed (of weights).  L2 is coherent, so what an earlier kernel still
//     writes there is not missed.
// Measured, decode steps: 79 launches of a latent-attention model (64 sequences) 751 -> 690 us, 70 of a hybrid (8 sequences)
// 514 -> 479, 48 to 52 of a Llama 480 -> 469 (one sequence) and 1056 -> 1042 (64).
// Without the launch attribute both instructions do nothing.  Every pointer that is `__restrict__`, to constants or not, goes
// through chain_wait: the compiler may take it that a statement which does not get the pointer leaves alone what it points to, and
// move loads, or stores, in front of the wait.
template <typename T>
__device__ __forceinline__ void unknown_pointer(T& p) { asm volatile("" : "+l"(p)::"memory"); }
template <typename... T>
__device__ __forceinline__ void chain_wait(T&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (unknown_pointer(p), ...);
}
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Both, for kernels without TMEM.
template <typename... T>
__device__ __forceinline__ void chain_enter(T&... p) {
  chain_next();
  chain_wait(p...);
}

template <typename T>
struct SameType {
  using type = T;
};
template <typename... P>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  typename SameType<P>::type... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

inline int launch_status() { return (int)cudaGetLastError(); }

}  // namespace ell
