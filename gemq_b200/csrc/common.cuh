// Shared helpers of the gemq_b200 kernels (sm_100a).
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/gemq_b200.h"

namespace gemq {

__host__ __device__ constexpr int cdiv(int a, int b) { return (a + b - 1) / b; }

inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

// A bit width as the kernels read it: tables on the device may hold anything.
__host__ __device__ constexpr int clamp_bits(int b) { return b < 1 ? 1 : (b > 4 ? 4 : b); }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Multiprocessors of the current device, 0 on failure.
inline int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cached[dev] = n;
  }
  return cached[dev];
}

// For rules that also size buffers: without a device those of a whole B200.
inline int sm_count_or_default() {
  const int n = sm_count();
  return n > 0 ? n : 148;
}

// Streaming 128-bit load: weights are read once per step, so they should not
// displace the activation tables or metadata in L1.
__device__ __forceinline__ uint4 ld_stream_v4(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.global.cs.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// Coherent (L2) loads for data another CTA of the same grid has just written.
__device__ __forceinline__ float ld_cg_f32(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// tma.cu
bool tensor_map_2d(CUtensorMap* out, const void* base, int elem_bytes, int inner, long long rows, int box_inner,
                   int box_rows, bool swizzle128);

__device__ __forceinline__ float pow2i(int e) {  // 2^e for e in [-126, 127]
  return __int_as_float((e + 127) << 23);
}

__device__ __forceinline__ float silu_f32(float v) { return v / (1.0f + __expf(-v)); }

// Where the experts of a layer begin: words (w3 lies like w1), and scales and offsets (nullptr: whole matrices one after the other).
struct Offsets {
  const int* words[2];   // of gate and up, of down
  int pitch[2];
  const int* scales[3];
};
inline Offsets expert_offsets(const gemq_moe_layer_t* L) {
  return {{L->w1.wq_strides, L->w2.wq_strides}, {L->ffn, L->hidden}, {L->w1.zs_strides, L->w3.zs_strides, L->w2.zs_strides}};
}
// An expert whose words do not begin at a whole row, or its scales not at a 16-byte boundary: tiled and bulk copies cannot take it.
__device__ __forceinline__ bool off_boundary(const Offsets& off, int e) {
  int o = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i) o |= off.words[i] ? off.words[i][e] % off.pitch[i] : 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) o |= off.scales[i] ? off.scales[i][e] & 7 : 0;
  return o != 0;
}

}  // namespace gemq
