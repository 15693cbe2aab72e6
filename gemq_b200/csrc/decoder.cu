// One decode step of one sequence around the quantised MoE blocks: everything between them.
//
// A step of a layer was about ninety small launches (normalisation, rotary embedding, masks and casts as
// separate tensor operations) of 1.2 to 3 us each around three projections of 12 us: 210 us of a layer's 260.
// Here it is four launches:
//   step_gemv   [x + residual -> RMSNorm ->] one or more unquantised matrices times the vector.  Bound by the
//               weights' bytes: a warp takes a row, all its loads in flight at once; the first row is on its way
//               before the wait for the previous kernel (which must not write it), so the normalisation (which every
//               CTA repeats: 8 KB out of L2) hides behind it
//   step_attn   rotary embedding, cache update and attention over the cached positions; a cluster of eight CTAs
//               per key / value head splits the positions and merges in the first CTA's shared memory
//   step_norm   x + residual -> RMSNorm, as the fp16 vector the MoE block takes
// Roundings are those of the tensor operations: every sum and product of the 16-bit type is rounded to it.
#include "common.cuh"

#include <type_traits>

namespace gemq {
namespace {

template <typename T> struct Num;
template <> struct Num<__half> {
  static __device__ __forceinline__ float f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half r(float v) { return __float2half_rn(v); }
};
template <> struct Num<__nv_bfloat16> {
  static __device__ __forceinline__ float f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 r(float v) { return __float2bfloat16_rn(v); }
};
template <typename T> __device__ __forceinline__ float rnd(float v) { return Num<T>::f(Num<T>::r(v)); }

__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// y = x + T(res) (res: fp16 or T), normalised: the result in `dst` (shared or global), y to `sum_out` if given.
// All threads of the block; returns after a barrier.
template <typename T, int THREADS>
__device__ __forceinline__ void add_norm(const T* __restrict__ x, const void* __restrict__ res, int res_half,
                                         const T* __restrict__ weight, float eps, int K, T* __restrict__ sum_out,
                                         T* __restrict__ dst, float* red) {
  const int tid = threadIdx.x;
  float ss = 0.f;
  for (int i = tid; i < K / 8; i += THREADS) {
    uint4 v = reinterpret_cast<const uint4*>(x)[i];
    T* e = reinterpret_cast<T*>(&v);
    if (res) {
      const uint4 u = reinterpret_cast<const uint4*>(res)[i];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float r = res_half ? rnd<T>(__half2float(reinterpret_cast<const __half*>(&u)[k]))
                                 : Num<T>::f(reinterpret_cast<const T*>(&u)[k]);
        e[k] = Num<T>::r(Num<T>::f(e[k]) + r);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) { const float f = Num<T>::f(e[k]); ss = fmaf(f, f, ss); }
    if (sum_out) reinterpret_cast<uint4*>(sum_out)[i] = v;
    reinterpret_cast<uint4*>(dst)[i] = v;
  }
  if (!weight) { __syncthreads(); return; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) ss += red[i];
  const float inv = rsqrtf(ss / static_cast<float>(K) + eps);
  for (int i = tid; i < K / 8; i += THREADS) {  // a thread's own elements
    uint4 v = reinterpret_cast<const uint4*>(dst)[i];
    const uint4 w = reinterpret_cast<const uint4*>(weight)[i];
    T* e = reinterpret_cast<T*>(&v);
    const T* g = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = Num<T>::r(rnd<T>(Num<T>::f(e[k]) * inv) * Num<T>::f(g[k]));
    reinterpret_cast<uint4*>(dst)[i] = v;
  }
  __syncthreads();
}

constexpr int kGemvThreads = 256;
constexpr int kLoads = 8;  // 16-byte loads of a lane at a time: 2048 columns of a row

struct GemvArgs {
  const void* x;
  const void* res;
  const void* weight;   // RMSNorm, or nullptr
  void* sum_out;        // x + res, or nullptr
  const void* w[3];
  int rows[3];          // of the matrices, in output order
  void* out;
  float eps;
  int res_half, K;
};

template <typename T>
__global__ void __launch_bounds__(kGemvThreads, 2) step_gemv_kernel(const __grid_constant__ GemvArgs P) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float red[kGemvThreads / 32];
  T* xs = reinterpret_cast<T*>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int total = P.rows[0] + P.rows[1] + P.rows[2];
  const int K = P.K, iters = K / 256;
  auto row_ptr = [&](int r) -> const T* {
    int m = 0;
    if (r >= P.rows[0]) { r -= P.rows[0]; m = 1; }
    if (m == 1 && r >= P.rows[1]) { r -= P.rows[1]; m = 2; }
    return static_cast<const T*>(P.w[m]) + static_cast<size_t>(r) * K + 8 * lane;
  };
  // A warp's work is a stream of pieces of kLoads loads, two of them in flight: each piece's registers are filled for
  // the piece after next once they have been used, all at once (filled one by one, every load waits for the ones
  // before it: the output matrix 118 us instead of 45).
  const int step = gridDim.x * (kGemvThreads / 32), pieces = (iters + kLoads - 1) / kLoads;
  const int first = blockIdx.x * (kGemvThreads / 32) + warp;
  uint4 va[kLoads], vb[kLoads];
  struct At { int row, piece; };
  auto next = [&](At& c) {
    if (++c.piece == pieces) { c.piece = 0; c.row += step; }
  };
  auto fill = [&](uint4 (&v)[kLoads], const At& c) {
    if (c.row >= total) return;
    const T* p = row_ptr(c.row) + 256 * kLoads * c.piece;
#pragma unroll
    for (int i = 0; i < kLoads; ++i)
      if (c.piece * kLoads + i < iters)
        asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w) : "l"(p + 256 * i));
  };
  float s = 0.f;
  auto use = [&](const uint4 (&v)[kLoads], const At& c) {
#pragma unroll
    for (int i = 0; i < kLoads; ++i)
      if (c.piece * kLoads + i < iters) {
        const uint4 xv = *reinterpret_cast<const uint4*>(xs + 256 * (c.piece * kLoads + i) + 8 * lane);
        const T *a = reinterpret_cast<const T*>(&v[i]), *b = reinterpret_cast<const T*>(&xv);
#pragma unroll
        for (int k = 0; k < 8; ++k) s = fmaf(Num<T>::f(a[k]), Num<T>::f(b[k]), s);
      }
    if (c.piece == pieces - 1) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) static_cast<T*>(P.out)[c.row] = Num<T>::r(s);
      s = 0.f;
    }
  };
  At cur = {first, 0}, ahead = {first, 0};
  fill(va, ahead);  // the matrices are older than the launch before (in the decoder: than the embedding)
  next(ahead);
  fill(vb, ahead);
  next(ahead);
  pdl_launch();
  pdl_wait();
  add_norm<T, kGemvThreads>(static_cast<const T*>(P.x), P.res, P.res_half, static_cast<const T*>(P.weight), P.eps, K,
                            blockIdx.x == 0 ? static_cast<T*>(P.sum_out) : nullptr, xs, red);
  while (cur.row < total) {
    use(va, cur);
    next(cur);
    fill(va, ahead);
    next(ahead);
    if (cur.row >= total) break;
    use(vb, cur);
    next(cur);
    fill(vb, ahead);
    next(ahead);
  }
}

constexpr int kNormThreads = 512;

template <typename T>
__global__ void __launch_bounds__(kNormThreads) step_norm_kernel(const T* x, const void* res, int res_half, const T* weight, float eps,
                                                                 int K, T* sum_out, __half* out) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float red[kNormThreads / 32];
  T* xs = reinterpret_cast<T*>(smem);
  pdl_launch();
  pdl_wait();
  add_norm<T, kNormThreads>(x, res, res_half, weight, eps, K, sum_out, xs, red);
  for (int i = threadIdx.x; i < K; i += kNormThreads) out[i] = __float2half_rn(Num<T>::f(xs[i]));
}

// ---- attention --------------------------------------------------------------------------------------
constexpr int kAttnCtas = 8;      // cluster per key / value head
constexpr int kAttnThreads = 256;
constexpr int kChunk = 64;        // positions per step of a CTA, four threads each
constexpr int kTopG = 8;          // query heads per key / value head at most

__device__ __forceinline__ uint32_t ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void st_first(float* p, float v) {  // the same place in the first CTA of the cluster
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(b) : "r"(a));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(b), "f"(v) : "memory");
}

struct AttnArgs {
  const void* qkv;         // [(H + 2 Hkv) * HD]
  const float* inv_freq;   // [HD / 2]
  const long long* pos;
  void* keys;              // [Hkv, L, HD]
  void* values;
  void* out;               // [H * HD]
  int H, Hkv, L;
  float scale;
};

template <typename T, int HD, int kMaxG>
__global__ void __launch_bounds__(kAttnThreads) step_attn_kernel(const __grid_constant__ AttnArgs P) {
  __shared__ __align__(16) float q[kMaxG][HD];
  __shared__ __align__(16) T new_k[HD], new_v[HD];
  __shared__ float sin_t[HD / 2], cos_t[HD / 2];
  __shared__ float score[kMaxG][kChunk];
  __shared__ float corr[kMaxG], run_m[kMaxG], run_l[kMaxG];
  __shared__ float part_m[kAttnCtas][kMaxG], part_l[kAttnCtas][kMaxG];
  __shared__ float part_o[kAttnCtas][kMaxG][HD];
  constexpr int TPD = HD / 4;                      // threads that cover HD dimensions, four each
  constexpr int TSETS = kAttnThreads / TPD;        // position subsets of the value product
  const int tid = threadIdx.x, rank = static_cast<int>(ctarank()), h = blockIdx.y;
  const int G = P.H / P.Hkv;
  pdl_launch();
  // remote stores at the end need the peers to have started by then
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  // The position and the cache below it are older than the launch before this one: the first keys and values are
  // on their way, and the angles made, before the wait for the projections.
  const long long at = *P.pos;
  const int pos = static_cast<int>(max(0ll, min(at, static_cast<long long>(P.L - 1))));
  const bool inside = at == pos;  // a position outside the cache: nothing is stored, the result is not a number
  const int chunks = pos / kChunk + 1;
  const T* qkv = static_cast<const T*>(P.qkv);
  T* kc = static_cast<T*>(P.keys) + static_cast<size_t>(h) * P.L * HD;
  T* vc = static_cast<T*>(P.values) + static_cast<size_t>(h) * P.L * HD;
  const int d4 = 4 * (tid % TPD), tset = tid / TPD;
  const int t = tid >> 2, part = tid & 3;  // of the scores: four threads a position, interleaved in pieces of eight
  uint4 kv[HD / 32];
  uint2 vr[kChunk / TSETS];
  auto load_keys = [&](int c) {
    if (c * kChunk + t < pos) {
      const T* kr = kc + static_cast<size_t>(c * kChunk + t) * HD + 8 * part;
#pragma unroll
      for (int j = 0; j < HD / 32; ++j) kv[j] = *reinterpret_cast<const uint4*>(kr + 32 * j);
    }
  };
  auto load_values = [&](int c) {
#pragma unroll
    for (int i = 0; i < kChunk / TSETS; ++i)
      if (c * kChunk + tset + TSETS * i < pos)
        vr[i] = *reinterpret_cast<const uint2*>(vc + static_cast<size_t>(c * kChunk + tset + TSETS * i) * HD + d4);
  };
  load_keys(rank);
  load_values(rank);
  if (tid < HD / 2) sincosf(static_cast<float>(pos) * P.inv_freq[tid], &sin_t[tid], &cos_t[tid]);
  if (tid < G) { run_m[tid] = -INFINITY; run_l[tid] = 0.f; }
  __syncthreads();
  pdl_wait();
  // rotary embedding of the G query heads, and of the new key in the CTA whose piece holds the position
  auto rotate = [&](const T* s, int i, float& a, float& b) {
    const float x1 = Num<T>::f(s[i]), x2 = Num<T>::f(s[i + HD / 2]);
    a = rnd<T>(x1 * cos_t[i] - x2 * sin_t[i]);
    b = rnd<T>(x2 * cos_t[i] + x1 * sin_t[i]);
  };
  for (int i = tid; i < G * (HD / 2); i += kAttnThreads) {
    const int g = i / (HD / 2), d = i - g * (HD / 2);
    rotate(qkv + static_cast<size_t>(h * G + g) * HD, d, q[g][d], q[g][d + HD / 2]);
  }
  if ((chunks - 1) % kAttnCtas == rank) {
    const T* k = qkv + static_cast<size_t>(P.H + h) * HD;
    const T* v = qkv + static_cast<size_t>(P.H + P.Hkv + h) * HD;
    for (int i = tid; i < HD / 2; i += kAttnThreads) {
      float a, b;
      rotate(k, i, a, b);
      new_k[i] = Num<T>::r(a);
      new_k[i + HD / 2] = Num<T>::r(b);
      if (inside) {
        kc[static_cast<size_t>(pos) * HD + i] = Num<T>::r(a);
        kc[static_cast<size_t>(pos) * HD + i + HD / 2] = Num<T>::r(b);
      }
    }
    for (int i = tid; i < HD; i += kAttnThreads) {
      new_v[i] = v[i];
      if (inside) vc[static_cast<size_t>(pos) * HD + i] = v[i];
    }
  }
  float o[kMaxG][4];
#pragma unroll
  for (int g = 0; g < kMaxG; ++g)
#pragma unroll
    for (int k = 0; k < 4; ++k) o[g][k] = 0.f;
  __syncthreads();
#pragma unroll 1
  for (int c = rank; c < chunks; c += kAttnCtas) {
    const int t0 = c * kChunk, n = min(kChunk, pos + 1 - t0);
    if (t0 + t == pos) {
#pragma unroll
      for (int j = 0; j < HD / 32; ++j) kv[j] = *reinterpret_cast<const uint4*>(&new_k[32 * j + 8 * part]);
    }
    float s[kMaxG];
#pragma unroll
    for (int g = 0; g < kMaxG; ++g) s[g] = 0.f;
    if (t < n) {
#pragma unroll
      for (int j = 0; j < HD / 32; ++j) {
        const T* e = reinterpret_cast<const T*>(&kv[j]);
        float kf[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) kf[k] = Num<T>::f(e[k]);
#pragma unroll
        for (int g = 0; g < kMaxG; ++g)
          if (g < G) {
            const float4 a = *reinterpret_cast<const float4*>(&q[g][32 * j + 8 * part]);
            const float4 b = *reinterpret_cast<const float4*>(&q[g][32 * j + 8 * part + 4]);
            s[g] += kf[0] * a.x + kf[1] * a.y + kf[2] * a.z + kf[3] * a.w + kf[4] * b.x + kf[5] * b.y + kf[6] * b.z + kf[7] * b.w;
          }
      }
    }
    load_keys(c + kAttnCtas);  // past the last piece: nothing
#pragma unroll
    for (int g = 0; g < kMaxG; ++g)
      if (g < G) {
        s[g] += __shfl_xor_sync(0xffffffffu, s[g], 1);
        s[g] += __shfl_xor_sync(0xffffffffu, s[g], 2);
        if (part == 0) score[g][t] = t < n ? s[g] * P.scale : -INFINITY;
      }
    __syncthreads();
    if ((tid >> 5) < G) {  // running maximum and sum, a warp a head
      const int g = tid >> 5, l0 = tid & 31;
      const float s0 = score[g][l0], s1 = score[g][l0 + 32];
      float m = fmaxf(s0, s1);
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
      const float old = run_m[g], now = fmaxf(old, m);
      const float p0 = __expf(s0 - now), p1 = __expf(s1 - now);
      float l = p0 + p1;
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
      score[g][l0] = p0;
      score[g][l0 + 32] = p1;
      __syncwarp();
      if (l0 == 0) {
        const float f = __expf(old - now);
        corr[g] = f;
        run_m[g] = now;
        run_l[g] = run_l[g] * f + l;
      }
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < kMaxG; ++g)
      if (g < G) {
        const float f = corr[g];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[g][k] *= f;
      }
#pragma unroll
    for (int i = 0; i < kChunk / TSETS; ++i)
      if (tset + TSETS * i < n) {
        if (t0 + tset + TSETS * i == pos) vr[i] = *reinterpret_cast<const uint2*>(&new_v[d4]);
        const T* e = reinterpret_cast<const T*>(&vr[i]);
        float vf[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) vf[k] = Num<T>::f(e[k]);
#pragma unroll
        for (int g = 0; g < kMaxG; ++g)
          if (g < G) {
            const float p = score[g][tset + TSETS * i];
#pragma unroll
            for (int k = 0; k < 4; ++k) o[g][k] = fmaf(p, vf[k], o[g][k]);
          }
      }
    load_values(c + kAttnCtas);
    __syncthreads();
  }
  // the position subsets of the CTA meet in `q` (done with), then everything in the first CTA
#pragma unroll 1
  for (int s = 0; s < TSETS; ++s) {
    if (tset == s)
#pragma unroll
      for (int g = 0; g < kMaxG; ++g)
        if (g < G) {
          float4* a = reinterpret_cast<float4*>(&q[g][d4]);
          float4 v = s ? *a : make_float4(0.f, 0.f, 0.f, 0.f);
          *a = make_float4(v.x + o[g][0], v.y + o[g][1], v.z + o[g][2], v.w + o[g][3]);
        }
    __syncthreads();
  }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (rank == 0) {
    for (int i = tid; i < G * HD; i += kAttnThreads) part_o[0][i / HD][i % HD] = q[i / HD][i % HD];
    if (tid < G) { part_m[0][tid] = run_m[tid]; part_l[0][tid] = run_l[tid]; }
  } else {
    for (int i = tid; i < G * HD; i += kAttnThreads) st_first(&part_o[rank][i / HD][i % HD], q[i / HD][i % HD]);
    if (tid < G) { st_first(&part_m[rank][tid], run_m[tid]); st_first(&part_l[rank][tid], run_l[tid]); }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank != 0) return;
  for (int i = tid; i < G * HD; i += kAttnThreads) {
    const int g = i / HD, d = i % HD;
    float m = -INFINITY;
#pragma unroll
    for (int r = 0; r < kAttnCtas; ++r) m = fmaxf(m, part_m[r][g]);
    float l = 0.f, a = 0.f;
#pragma unroll
    for (int r = 0; r < kAttnCtas; ++r) {
      const float f = __expf(part_m[r][g] - m);  // 0 for a CTA without positions
      l = fmaf(part_l[r][g], f, l);
      a = fmaf(part_o[r][g][d], f, a);
    }
    static_cast<T*>(P.out)[static_cast<size_t>(h * G) * HD + i] = Num<T>::r(inside ? a / l : __int_as_float(0x7fc00000));
  }
}

cudaLaunchConfig_t config(dim3 grid, int threads, size_t smem, gemq_stream_t st, cudaLaunchAttribute* attr, int cluster) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(st);
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cfg;
}

}  // namespace
}  // namespace gemq

using namespace gemq;

extern "C" int gemq_step_gemv(const void* x, const void* res, int res_is_half, const void* norm_weight, float eps, void* sum_out,
                              const void* w0, int rows0, const void* w1, int rows1, const void* w2, int rows2, void* out, int K,
                              int is_bf16, gemq_stream_t stream) {
  if (!x || !w0 || !out || rows0 <= 0 || rows1 < 0 || rows2 < 0 || (rows1 && !w1) || (rows2 && !w2) || K <= 0) return GEMQ_ERR_BAD_ARG;
  if (K % 256 || K > 16384) return GEMQ_ERR_BAD_SHAPE;
  for (const void* p : {x, res, norm_weight, static_cast<const void*>(sum_out), w0, w1, w2})
    if (p && !aligned16(p)) return GEMQ_ERR_ALIGN;
  GemvArgs P = {x, res, norm_weight, sum_out, {w0, w1, w2}, {rows0, rows1, rows2}, out, eps, res_is_half, K};
  const int sms = sm_count(), total = rows0 + rows1 + rows2;
  if (sms <= 0) return GEMQ_ERR_LAUNCH;
  const int need = cdiv(total, kGemvThreads / 32), grid = need < 2 * sms ? need : 2 * sms;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = config(dim3(grid), kGemvThreads, static_cast<size_t>(K) * 2, stream, attr, 1);
  const cudaError_t e = is_bf16 ? cudaLaunchKernelEx(&cfg, step_gemv_kernel<__nv_bfloat16>, P)
                                : cudaLaunchKernelEx(&cfg, step_gemv_kernel<__half>, P);
  return e == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

extern "C" int gemq_step_norm(const void* x, const void* res, int res_is_half, const void* weight, float eps, void* sum_out,
                              void* out_half, int K, int is_bf16, gemq_stream_t stream) {
  if (!x || !weight || !out_half || K <= 0) return GEMQ_ERR_BAD_ARG;
  if (K % 8 || K > 16384) return GEMQ_ERR_BAD_SHAPE;
  for (const void* p : {x, res, weight, static_cast<const void*>(sum_out)})
    if (p && !aligned16(p)) return GEMQ_ERR_ALIGN;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = config(dim3(1), kNormThreads, static_cast<size_t>(K) * 2, stream, attr, 1);
  cudaError_t e;
  if (is_bf16)
    e = cudaLaunchKernelEx(&cfg, step_norm_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(x), res, res_is_half,
                           static_cast<const __nv_bfloat16*>(weight), eps, K, static_cast<__nv_bfloat16*>(sum_out),
                           static_cast<__half*>(out_half));
  else
    e = cudaLaunchKernelEx(&cfg, step_norm_kernel<__half>, static_cast<const __half*>(x), res, res_is_half,
                           static_cast<const __half*>(weight), eps, K, static_cast<__half*>(sum_out), static_cast<__half*>(out_half));
  return e == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

extern "C" int gemq_step_attention(const void* qkv, const float* inv_freq, const int64_t* pos, void* keys, void* values, void* out,
                                   int heads, int kv_heads, int head_dim, int cache_len, int is_bf16, gemq_stream_t stream) {
  if (!qkv || !inv_freq || !pos || !keys || !values || !out || heads <= 0 || kv_heads <= 0 || cache_len <= 0) return GEMQ_ERR_BAD_ARG;
  if (heads % kv_heads || heads / kv_heads > kTopG || (head_dim != 64 && head_dim != 128) || kv_heads > 65535) return GEMQ_ERR_BAD_SHAPE;
  if (!aligned16(qkv) || !aligned16(keys) || !aligned16(values)) return GEMQ_ERR_ALIGN;
  AttnArgs P = {qkv, inv_freq, reinterpret_cast<const long long*>(pos), keys, values, out, heads, kv_heads, cache_len,
                1.0f / sqrtf(static_cast<float>(head_dim))};
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = config(dim3(kAttnCtas, kv_heads), kAttnThreads, 0, stream, attr, kAttnCtas);
  const int g = heads / kv_heads;
  auto pick = [&](auto t, auto hd) -> void (*)(const AttnArgs) {
    using T = decltype(t);
    constexpr int HD = decltype(hd)::value;
    return g <= 1 ? step_attn_kernel<T, HD, 1> : g <= 2 ? step_attn_kernel<T, HD, 2> : g <= 4 ? step_attn_kernel<T, HD, 4>
                                                                                  : step_attn_kernel<T, HD, 8>;
  };
  auto by_dim = [&](auto t) {
    return head_dim == 128 ? pick(t, std::integral_constant<int, 128>()) : pick(t, std::integral_constant<int, 64>());
  };
  const cudaError_t e = cudaLaunchKernelEx(&cfg, is_bf16 ? by_dim(__nv_bfloat16()) : by_dim(__half()), P);
  return e == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}
