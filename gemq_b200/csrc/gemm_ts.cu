// Launchers of the tcgen05 GEMM (gemm_ts.cuh) and the dense quantised GEMM entry points.
#include "gemm_ts.cuh"

namespace gemq {
namespace ts {

template <int OUT, bool BF16>
static int launch(const Params& P, int tiles_bound, cudaStream_t stream) {
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GEMQ_ERR_LAUNCH;
  const size_t smem = sizeof(Smem) + 1024;
  if (!done[dev]) {
    if (cudaFuncSetAttribute(gemm_ts_kernel<OUT, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
        cudaSuccess)
      return GEMQ_ERR_LAUNCH;
    done[dev] = true;
  }
  const int sms = sm_count();
  if (sms < 2 || tiles_bound <= 0) return GEMQ_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (tiles_bound < sms / 2 ? tiles_bound : sms / 2));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, gemm_ts_kernel<OUT, BF16>, P) == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

bool activation_maps(CUtensorMap (&maps)[4], const void* x, int K, long long rows) {
  for (int i = 0; i < 4; ++i)
    if (!tensor_map_blocks(&maps[i], x, K, rows, 32 * (i + 1))) return false;
  return true;
}

int launch_up(const Params& P, int tiles_bound, cudaStream_t stream) { return launch<kOutUp, false>(P, tiles_bound, stream); }
int launch_down(const Params& P, int tiles_bound, cudaStream_t stream) { return launch<kOutDown, false>(P, tiles_bound, stream); }

}  // namespace ts
}  // namespace gemq

using namespace gemq;
using namespace gemq::ts;

extern "C" int gemq_linear_gemm(const void* x, const int64_t* expert, const int32_t* wq, const void* scales, const void* zeros,
                                const int32_t* nbits, const int32_t* wq_strides, const int32_t* zs_strides, int fixed_bits,
                                const void* bias, void* y, int M, int N, int K, int group_size, int x_is_bf16, int32_t* err,
                                gemq_stream_t stream) {
  if (!x || !wq || !scales || !zeros || !y || !err || M <= 0 || N <= 0 || K <= 0 || group_size <= 0) return GEMQ_ERR_BAD_ARG;
  if (!nbits && (fixed_bits < 1 || fixed_bits > 4)) return GEMQ_ERR_BAD_ARG;
  if (N % 32 || K % kBK || group_size % kBK || K % group_size) return GEMQ_ERR_BAD_SHAPE;
  if (!aligned16(x) || !aligned16(y)) return GEMQ_ERR_ALIGN;
  Params P = {};
  if (!activation_maps(P.b_map[0], x, K, M)) return GEMQ_ERR_LAUNCH;
  Family& F = P.fam[0];
  F.scales[0] = static_cast<const __half*>(scales);
  F.zeros[0] = static_cast<const __half*>(zeros);
  F.wq[0] = reinterpret_cast<const uint32_t*>(wq);
  F.nbits = nbits; F.wq_strides = wq_strides; F.zs_strides[0] = zs_strides;
  F.bits = fixed_bits;
  F.N = N; F.K = K; F.G = group_size;
  F.out = y;
  P.expert = reinterpret_cast<const long long*>(expert);
  P.rows = M;
  P.bias = bias;
  P.err = err;
  // Fewer tokens per tile (which then costs its de-quantisation; that does not shrink with the tokens) as
  // long as there are CTA pairs to take the tiles.
  const int pairs = sm_count() / 2;
  F.col_tiles = cdiv(N, 2 * kCols);
  P.tile_rows = kTokens;
  while (P.tile_rows > 32 && F.col_tiles * cdiv(M, P.tile_rows / 2) <= pairs) P.tile_rows /= 2;
  const int tiles = F.col_tiles * cdiv(M, P.tile_rows);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = x_is_bf16 ? launch<kOutLinear, true>(P, tiles, st) : launch<kOutLinear, false>(P, tiles, st);
  return rc ? rc : launch_status();
}

extern "C" int gemq_dequant_gemm_tc(const void* x, const int64_t* expert, const int32_t* wq, const void* scales,
                                    const void* zeros, const int32_t* nbits, const int32_t* wq_strides,
                                    const int32_t* zs_strides, int fixed_bits, void* y, int M, int N, int K,
                                    int group_size, int x_is_bf16, int32_t* err, gemq_stream_t stream) {
  return gemq_linear_gemm(x, expert, wq, scales, zeros, nbits, wq_strides, zs_strides, fixed_bits, nullptr, y, M, N, K, group_size,
                          x_is_bf16, err, stream);
}
