// Router: gate products, softmax, top-k and renormalisation in one launch.
// Results stay on the device (expert ids as int64, like torch.topk returns them).
#include <type_traits>

#include "common.cuh"

namespace gemq {

constexpr int kRouteThreads = 1024;
constexpr int kRouteMaxExperts = 256;
constexpr int kRouteMaxTopK = 16;
constexpr int kRouteMaxParts = 8;

template <typename T> struct Act;
template <> struct Act<__half> {
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
};
template <> struct Act<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};

// mode 0: logits, probabilities, their sum and the quotient are each rounded to the
//         activation dtype (softmax/topk/renorm of a half tensor);
// mode 1: logits rounded to the activation dtype, softmax and renormalisation in fp32;
// mode 2: fp32 throughout.  The returned weights are cast to the activation dtype.
//
// One token per CTA; a warp takes four experts of one segment of the hidden size.
constexpr int kRouteTile = 4;  // experts of a warp task

template <typename T, typename G>
__device__ __forceinline__ void gate8(const uint4& v, float (&f)[8]) {
  const G* e = reinterpret_cast<const G*>(&v);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    f[i] = Act<G>::to_f(e[i]);
    // a gate kept in fp16 is used as the bf16 copy the bf16 model has
    if (sizeof(G) == sizeof(T) && !std::is_same<G, T>::value) f[i] = Act<T>::to_f(Act<T>::from_f(f[i]));
  }
}

// Softmax, top-k and renormalisation of one token's logits (`step` apart in shared memory) by one warp.
// PER: experts per lane (E <= 32 * PER).
template <typename T, int PER>
__device__ __forceinline__ void route_select(const float* row, int step, int E, int A, int mode, int renorm, int lane, size_t token,
                                             long long* __restrict__ idx, T* __restrict__ weights) {
  float p[PER];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    p[i] = e < E ? row[e * step] : -INFINITY;
    mx = fmaxf(mx, p[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    p[i] = (lane + 32 * i) < E ? expf(p[i] - mx) : 0.f;
    sum += p[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  // Probabilities are >= +0: their bit patterns order like integers.  Key 0: beyond E, taken, or not a number.
  unsigned key[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    p[i] = p[i] / sum;
    if (mode == 0) p[i] = Act<T>::to_f(Act<T>::from_f(p[i]));
    key[i] = (lane + 32 * i) < E && p[i] >= 0.f ? __float_as_uint(p[i]) + 1u : 0u;
  }
  // top-k: A rounds of warp arg-max, ties to the lower expert id; lane a keeps the a-th winner
  float my_w = 0.f;
  int my_i = 0;
  for (int a = 0; a < A; ++a) {
    unsigned best = key[0];
#pragma unroll
    for (int i = 1; i < PER; ++i) best = max(best, key[i]);
    const unsigned kmax = __reduce_max_sync(0xffffffffu, best);
    int bi = -1;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const unsigned hit = __ballot_sync(0xffffffffu, key[i] == kmax);
      if (bi < 0 && hit) bi = 32 * i + __ffs(hit) - 1;
    }
    if (lane == a) { my_w = __uint_as_float(kmax - 1u); my_i = bi; }
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i == bi) key[i] = 0u;
  }
  float tot = 0.f;
  for (int a = 0; a < A; ++a) tot += __shfl_sync(0xffffffffu, my_w, a);  // in selection order, like a sum over the top-k tensor
  if (mode == 0) tot = Act<T>::to_f(Act<T>::from_f(tot));
  if (lane < A) {
    const float w = renorm ? my_w / tot : my_w;
    idx[token * A + lane] = my_i;
    weights[token * A + lane] = Act<T>::from_f(w);
  }
}

template <typename T>
__device__ __forceinline__ void route_logit(void* out, int act, size_t at, float s) {
  if (act) static_cast<T*>(out)[at] = Act<T>::from_f(s);
  else static_cast<float*>(out)[at] = s;
}

template <typename T, typename G, int PER>
__global__ void __launch_bounds__(kRouteThreads) route_kernel(const T* __restrict__ x, const G* __restrict__ gate, int D, int E, int A,
                                                              int mode, int renorm, long long* __restrict__ idx,
                                                              T* __restrict__ weights, void* __restrict__ logits_out, int logits_act) {
  __shared__ float part_sum[32 * PER];  // [expert * parts + segment]; a segmented row means E * parts <= 32
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may come from the previous kernel of the stream
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const size_t token = blockIdx.x;
  // An expert row is cut into `parts` segments so that all warps pull on the gate matrix at once.
  int parts = E >= 32 ? 1 : 32 / E;
  parts = parts > kRouteMaxParts ? kRouteMaxParts : parts;
  while (parts > 1 && (D % (parts * 256)) != 0) parts >>= 1;
  const bool vec = (D % 256 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) && ((reinterpret_cast<uintptr_t>(gate) & 15u) == 0);
  if (!vec) parts = 1;
  const int seg = D / parts;
  const int etiles = (E + kRouteTile - 1) / kRouteTile;
  for (int task = warp; task < etiles * parts; task += nw) {
    const int et = task / parts, sg = task - et * parts, e0 = et * kRouteTile;
    float s[kRouteTile] = {};
    if (vec) {
      const G* gp = gate + static_cast<size_t>(sg) * seg + 8 * lane;
      const T* xp = x + token * D + static_cast<size_t>(sg) * seg + 8 * lane;
#pragma unroll 4
      for (int k = 0; k < seg; k += 256) {
        uint4 gq[kRouteTile];
#pragma unroll
        for (int j = 0; j < kRouteTile; ++j)
          gq[j] = *reinterpret_cast<const uint4*>(gp + static_cast<size_t>(min(e0 + j, E - 1)) * D + k);
        const uint4 xq = *reinterpret_cast<const uint4*>(xp + k);
        float gf[kRouteTile][8], xf[8];
#pragma unroll
        for (int j = 0; j < kRouteTile; ++j) gate8<T, G>(gq[j], gf[j]);
        const T* px = reinterpret_cast<const T*>(&xq);
#pragma unroll
        for (int i = 0; i < 8; ++i) xf[i] = Act<T>::to_f(px[i]);
#pragma unroll
        for (int j = 0; j < kRouteTile; ++j) {
          float d = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) d = fmaf(xf[i], gf[j][i], d);
          s[j] += d;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < kRouteTile; ++j) {
        if (e0 + j >= E) break;
        for (int k = lane; k < seg; k += 32) {
          float gv = Act<G>::to_f(gate[static_cast<size_t>(e0 + j) * D + k]);
          if (!std::is_same<G, T>::value) gv = Act<T>::to_f(Act<T>::from_f(gv));
          s[j] = fmaf(Act<T>::to_f(x[token * D + k]), gv, s[j]);
        }
      }
    }
    // Butterfly over the lanes.  The halves of the warp keep half of the values each while there are several:
    // the same pairs are added, in fewer shuffles.
    int first = 0;  // value held in s[0]
    int held = kRouteTile;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      if (held > 1) {
        const bool up = (lane & o) != 0;
        const int half = held / 2;
#pragma unroll
        for (int i = 0; i < kRouteTile / 2; ++i)
          if (i < half) {
            const float give = up ? s[i] : s[i + half], keep = up ? s[i + half] : s[i];
            s[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        if (up) first += half;
        held = half;
      } else {
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
      }
    }
    // lanes that share a value agree on it
    if (e0 + first < E) part_sum[(e0 + first) * parts + sg] = s[0];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    float s = 0.f;
    for (int q = 0; q < parts; ++q) s += part_sum[e * parts + q];
    if (mode != 2) s = Act<T>::to_f(Act<T>::from_f(s));
    part_sum[e * parts] = s;
    if (logits_out) route_logit<T>(logits_out, logits_act, token * E + e, s);
  }
  __syncthreads();
  if (warp == 0) route_select<T, PER>(part_sum, parts, E, A, mode, renorm, lane, token, idx, weights);
}

// Many tokens: 16 of them per CTA against up to 64 experts (NT tiles of eight), the hidden size split over eight
// warps, products on the tensor cores (exact: both operands keep their type; fp32 sums, the warps' added
// in order).  A lane takes eight consecutive elements of its rows at a time, the same for x and gate, so
// both operands come straight from memory in 16-byte loads; which element of k a fragment slot holds does not matter.
// On the CUDA cores the multiply-adds and conversions bound the pass (eight tokens per CTA, packed fp32 or not):
// 29.7 us for 2000 tokens x 64 experts x 2048 and 17.7 for 4096 x 8 x 4096 there, 9.3 and 11.5 here, where the gate
// coming through L2 once per 16 tokens and the start of the launch are what is left.
// A gate kept in fp16 is rounded to bf16 for bf16 tokens, like in the one-token kernel.
constexpr int kRouteRows = 16, kRouteWarps = 8;

// c += a * b.  The 16 products of a sum are added by the tensor core, the sums by rounding additions: a chain of
// accumulating MMAs truncates at every step (relative error of the logits 3e-7 to 7e-7, like this 1e-7).
template <typename T>
__device__ __forceinline__ void route_mma(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  float d[4];
  if constexpr (std::is_same<T, __half>::value)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += d[i];
}

template <typename T, typename G>
__device__ __forceinline__ unsigned gate_pair(unsigned v) {  // two gate elements in the type of the tokens
  if constexpr (std::is_same<G, T>::value) return v;
  const __nv_bfloat162 b = __float22bfloat162_rn(__half22float2(*reinterpret_cast<const __half2*>(&v)));
  return *reinterpret_cast<const unsigned*>(&b);
}

template <typename T, typename G, int NT>
__global__ void __launch_bounds__(32 * kRouteWarps) route_many_kernel(const T* __restrict__ x, const G* __restrict__ gate, int tokens,
                                                                     int D, int E, int A, int mode, int renorm,
                                                                     long long* __restrict__ idx, T* __restrict__ weights,
                                                                     void* __restrict__ logits_out, int logits_act) {
  constexpr int kLd = 8 * NT + 8;  // rows eight banks apart
  __shared__ float sums[kRouteWarps][kRouteRows][kLd];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may come from the previous kernel of the stream
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane >> 2, c = lane & 3;
  const int t0 = blockIdx.x * kRouteRows, nt = min(kRouteRows, tokens - t0);
  const int seg = D / kRouteWarps, k0 = warp * seg + 8 * c;
  const T* x0 = x + static_cast<size_t>(t0 + min(r, nt - 1)) * D + k0;
  const T* x1 = x + static_cast<size_t>(t0 + min(r + 8, nt - 1)) * D + k0;
  const G* gp[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) gp[n] = gate + static_cast<size_t>(min(8 * n + r, E - 1)) * D + k0;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
#pragma unroll NT == 8 ? 2 : 4
  for (int k = 0; k < seg; k += 32) {
    const uint4 a = *reinterpret_cast<const uint4*>(x0 + k), b = *reinterpret_cast<const uint4*>(x1 + k);
    uint4 g[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) g[n] = *reinterpret_cast<const uint4*>(gp[n] + k);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      route_mma<T>(acc[n], a.x, b.x, a.y, b.y, gate_pair<T, G>(g[n].x), gate_pair<T, G>(g[n].y));
      route_mma<T>(acc[n], a.z, b.z, a.w, b.w, gate_pair<T, G>(g[n].z), gate_pair<T, G>(g[n].w));
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    *reinterpret_cast<float2*>(&sums[warp][r][8 * n + 2 * c]) = make_float2(acc[n][0], acc[n][1]);
    *reinterpret_cast<float2*>(&sums[warp][r + 8][8 * n + 2 * c]) = make_float2(acc[n][2], acc[n][3]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nt * E; i += 32 * kRouteWarps) {
    const int t = i / E, e = i - t * E;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kRouteWarps; ++w) s += sums[w][t][e];
    if (mode != 2) s = Act<T>::to_f(Act<T>::from_f(s));
    sums[0][t][e] = s;
    if (logits_out) route_logit<T>(logits_out, logits_act, static_cast<size_t>(t0 + t) * E + e, s);
  }
  __syncthreads();
  for (int t = warp; t < nt; t += kRouteWarps)
    route_select<T, (NT + 3) / 4>(sums[0][t], 1, E, A, mode, renorm, lane, static_cast<size_t>(t0 + t), idx, weights);
}

struct RouteArgs {
  const void* x;
  const void* gate;
  int tokens, D, E, A, mode, renorm;
  long long* idx;
  void* weights;
  void* logits;
  int logits_act;
  cudaStream_t stream;
};

template <typename... P, typename... Q>
static cudaError_t launch_route(void (*kernel)(P...), int grid, int threads, cudaStream_t stream, Q... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename T, typename G, int PER>
static cudaError_t launch_one(const RouteArgs& R) {
  const int parts = R.E >= 32 ? 1 : (32 / R.E < kRouteMaxParts ? 32 / R.E : kRouteMaxParts);
  const int warps = (R.E + kRouteTile - 1) / kRouteTile * parts;
  return launch_route(route_kernel<T, G, PER>, R.tokens, warps * 32 > kRouteThreads ? kRouteThreads : warps * 32, R.stream,
                      static_cast<const T*>(R.x), static_cast<const G*>(R.gate), R.D, R.E, R.A, R.mode, R.renorm, R.idx,
                      static_cast<T*>(R.weights), R.logits, R.logits_act);
}

template <typename T, typename G, int NT>
static cudaError_t launch_many(const RouteArgs& R) {
  return launch_route(route_many_kernel<T, G, NT>, (R.tokens + kRouteRows - 1) / kRouteRows, 32 * kRouteWarps, R.stream,
                      static_cast<const T*>(R.x), static_cast<const G*>(R.gate), R.tokens, R.D, R.E, R.A, R.mode, R.renorm, R.idx,
                      static_cast<T*>(R.weights), R.logits, R.logits_act);
}

template <typename T, typename G>
static cudaError_t launch_route_any(const RouteArgs& R) {
  // The many-token kernel is flat up to 16 tokens per SM (7 to 9 us); one token per CTA is faster while its CTAs are one
  // round: two per SM for 16 warps (64 experts: 301 tokens 11.6 against 8.5 us, 200 tokens 8.3 against 8.4), four below
  // (8 experts: 509 tokens 6.3 against 7.0, 767 tokens 8.3 against 7.2).
  const int round = sm_count_or_default() * (R.E > 32 ? 2 : 4);
  const bool many = R.tokens > round && R.E <= 64 && R.D % (32 * kRouteWarps) == 0 &&
                    ((reinterpret_cast<uintptr_t>(R.x) | reinterpret_cast<uintptr_t>(R.gate)) & 15u) == 0;
  if (many)
    return R.E <= 8 ? launch_many<T, G, 1>(R) : R.E <= 16 ? launch_many<T, G, 2>(R) : R.E <= 32 ? launch_many<T, G, 4>(R)
                                                                                              : launch_many<T, G, 8>(R);
  return R.E <= 32 ? launch_one<T, G, 1>(R) : R.E <= 64 ? launch_one<T, G, 2>(R) : launch_one<T, G, kRouteMaxExperts / 32>(R);
}

// Router with an fp16 gate for bf16 activations, logits in the activation type on request.
int route_tokens(const void* x, const void* gate, bool gate_half, int tokens, int D, int E, int A, int mode, int renorm, bool bf16,
                 int64_t* idx, void* weights, void* logits, bool logits_act, cudaStream_t stream) {
  if (!x || !gate || !idx || !weights || tokens <= 0 || D <= 0 || E <= 0 || A <= 0 || mode < 0 || mode > 2)
    return GEMQ_ERR_BAD_ARG;
  if (E > kRouteMaxExperts || A > kRouteMaxTopK || A > E) return GEMQ_ERR_BAD_SHAPE;
  const RouteArgs R = {x, gate, tokens, D, E, A, mode, renorm, reinterpret_cast<long long*>(idx), weights, logits, logits_act ? 1 : 0,
                       stream};
  const cudaError_t e = !bf16 ? launch_route_any<__half, __half>(R)
                              : (gate_half ? launch_route_any<__nv_bfloat16, __half>(R)
                                           : launch_route_any<__nv_bfloat16, __nv_bfloat16>(R));
  return e == cudaSuccess ? launch_status() : GEMQ_ERR_LAUNCH;
}

}  // namespace gemq

using namespace gemq;

extern "C" int gemq_moe_route(const void* x, const void* gate, int tokens, int D, int E, int A,
                              int mode, int renorm, int x_is_bf16,
                              int64_t* idx, void* weights, float* logits, gemq_stream_t stream) {
  return route_tokens(x, gate, false, tokens, D, E, A, mode, renorm, x_is_bf16 != 0, idx, weights, logits, false,
                      static_cast<cudaStream_t>(stream));
}
