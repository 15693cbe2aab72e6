// Router: gate products, softmax, top-k and renormalisation in one launch.
// Results stay on the device (expert ids as int64, like torch.topk returns them).
#include <type_traits>

#include "common.cuh"

namespace gemq {

constexpr int route_threads(int tt) { return tt == 1 ? 1024 : 512; }  // eight tokens keep 32 sums in registers
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
// A CTA takes TT tokens; a warp takes four experts of one segment of the hidden size for all of them, so
// a gate row is read and converted once per TT tokens (one token per CTA and a gate row per token: 124 us
// for 2000 tokens x 64 experts, all of it re-reading the gate through L2).  Every (token, expert) sum keeps one
// order whatever TT is: a lane adds eight products per 256 elements, lanes are added in a butterfly, the
// segments of a row in order -- the experts a token gets do not depend on the batch it is in.
// PER: experts per lane in the softmax / top-k phase (E <= 32 * PER).
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

template <typename T, typename G, int TT, int PER>
__global__ void __launch_bounds__(route_threads(TT)) route_kernel(const T* __restrict__ x, const G* __restrict__ gate, int tokens,
                                                              int D, int E, int A, int mode, int renorm,
                                                              long long* __restrict__ idx, T* __restrict__ weights,
                                                              void* __restrict__ logits_out, int logits_act) {
  __shared__ float part_sum[TT][32 * PER];  // [token][expert * parts + segment]; a segmented row means E * parts <= 32
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // x may come from the previous kernel of the stream
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const int t0 = blockIdx.x * TT, nt = min(TT, tokens - t0);
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
    float s[TT][kRouteTile];
#pragma unroll
    for (int t = 0; t < TT; ++t)
#pragma unroll
      for (int j = 0; j < kRouteTile; ++j) s[t][j] = 0.f;
    if (vec) {
      const G* gp = gate + static_cast<size_t>(sg) * seg + 8 * lane;
      const T* xp = x + static_cast<size_t>(t0) * D + static_cast<size_t>(sg) * seg + 8 * lane;
#pragma unroll TT == 1 ? 4 : 1
      for (int k = 0; k < seg; k += 256) {
        uint4 gq[kRouteTile], xq[TT];
#pragma unroll
        for (int j = 0; j < kRouteTile; ++j)
          gq[j] = *reinterpret_cast<const uint4*>(gp + static_cast<size_t>(min(e0 + j, E - 1)) * D + k);
#pragma unroll
        for (int t = 0; t < TT; ++t) xq[t] = *reinterpret_cast<const uint4*>(xp + static_cast<size_t>(min(t, nt - 1)) * D + k);
        float gf[kRouteTile][8];
#pragma unroll
        for (int j = 0; j < kRouteTile; ++j) gate8<T, G>(gq[j], gf[j]);
#pragma unroll
        for (int t = 0; t < TT; ++t) {
          const T* px = reinterpret_cast<const T*>(&xq[t]);
          float xf[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) xf[i] = Act<T>::to_f(px[i]);
#pragma unroll
          for (int j = 0; j < kRouteTile; ++j) {
            float d = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) d = fmaf(xf[i], gf[j][i], d);
            s[t][j] += d;
          }
        }
      }
    } else {
      for (int t = 0; t < nt; ++t)
        for (int j = 0; j < kRouteTile && e0 + j < E; ++j) {
          float d = 0.f;
          for (int k = lane; k < seg; k += 32) {
            float gv = Act<G>::to_f(gate[static_cast<size_t>(e0 + j) * D + k]);
            if (!std::is_same<G, T>::value) gv = Act<T>::to_f(Act<T>::from_f(gv));
            d = fmaf(Act<T>::to_f(x[static_cast<size_t>(t0 + t) * D + k]), gv, d);
          }
#pragma unroll
          for (int tt = 0; tt < TT; ++tt)
#pragma unroll
            for (int jj = 0; jj < kRouteTile; ++jj)
              if (tt == t && jj == j) s[tt][jj] = d;
        }
    }
    // Butterfly over the lanes.  With several values per lane the halves of the warp keep half of them each at
    // every step: the same pairs are added, in a fifth of the shuffles.
    constexpr int V = TT * kRouteTile;
    float v[V];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = s[i / kRouteTile][i % kRouteTile];
    int first = 0;  // value held in v[0]
    int held = V;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      constexpr int kAll = V;
      if (held > 1) {
        const bool up = (lane & o) != 0;
        const int half = held / 2;
#pragma unroll
        for (int i = 0; i < kAll / 2; ++i)
          if (i < half) {
            const float give = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        if (up) first += half;
        held = half;
      } else {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      }
    }
    // V <= 32: one value per lane is left; lanes that share a value agree on it
#pragma unroll
    for (int i = 0; i < (V > 32 ? V / 32 : 1); ++i) {
      const int t = (first + i) / kRouteTile, j = (first + i) % kRouteTile;
      if (e0 + j < E) part_sum[t][(e0 + j) * parts + sg] = v[i];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nt * E; i += blockDim.x) {
    const int t = i / E, e = i - t * E;
    float s = 0.f;
    for (int q = 0; q < parts; ++q) s += part_sum[t][e * parts + q];
    if (mode != 2) s = Act<T>::to_f(Act<T>::from_f(s));
    part_sum[t][e * parts] = s;
    if (logits_out) {
      const size_t at = static_cast<size_t>(t0 + t) * E + e;
      if (logits_act) static_cast<T*>(logits_out)[at] = Act<T>::from_f(s);
      else static_cast<float*>(logits_out)[at] = s;
    }
  }
  __syncthreads();
  for (int t = warp; t < nt; t += nw) {
    float p[PER];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      p[i] = e < E ? part_sum[t][e * parts] : -INFINITY;
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
      idx[static_cast<size_t>(t0 + t) * A + lane] = my_i;
      weights[static_cast<size_t>(t0 + t) * A + lane] = Act<T>::from_f(w);
    }
  }
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

template <typename T, typename G, int TT, int PER>
static cudaError_t launch_route(const RouteArgs& R) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((R.tokens + TT - 1) / TT);
  // warps for the tasks of a CTA; its tokens' softmaxes take one each
  const int parts = R.E >= 32 ? 1 : (32 / R.E < kRouteMaxParts ? 32 / R.E : kRouteMaxParts);
  int warps = (R.E + kRouteTile - 1) / kRouteTile * parts;
  warps = warps < TT ? TT : warps;
  cfg.blockDim = dim3(32 * (warps > route_threads(TT) / 32 ? route_threads(TT) / 32 : warps));
  cfg.stream = R.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, route_kernel<T, G, TT, PER>, static_cast<const T*>(R.x), static_cast<const G*>(R.gate), R.tokens,
                            R.D, R.E, R.A, R.mode, R.renorm, R.idx, static_cast<T*>(R.weights), R.logits, R.logits_act);
}

template <typename T, typename G>
static cudaError_t launch_route_any(const RouteArgs& R) {
  // Eight tokens per CTA once that still leaves about a CTA per SM; before, latency counts and a token has its own.
  const bool many = R.tokens >= 8 * 96;
  if (R.E <= 32) return many ? launch_route<T, G, 8, 1>(R) : launch_route<T, G, 1, 1>(R);
  if (R.E <= 64) return many ? launch_route<T, G, 8, 2>(R) : launch_route<T, G, 1, 2>(R);
  return launch_route<T, G, 1, kRouteMaxExperts / 32>(R);
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
