// Launchers of the tcgen05 GEMM (gemm_ts.cuh) and the dense quantised GEMM entry points.
#include "gemm_ts.cuh"

namespace gemq {
namespace ts {

template <int OUT, bool BF16>
static int launch(const Params& P, int tiles_bound, cudaStream_t stream) {
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GEMQ_ERR_LAUNCH;
  const size_t smem = sizeof(Smem);
  static_assert(sizeof(Smem) <= 227 * 1024, "shared memory of a CTA");
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

bool word_maps(CUtensorMap (&maps)[4], const void* wq, const void* scales, const void* zeros, int N, long long rows, int G, int bits,
               int columns) {
  if (!aligned16(wq) || !aligned16(scales) || !aligned16(zeros) || rows <= 0 || G % kStageK) return false;
  for (int b = 1; b <= 4; ++b)
    if ((!bits || b == bits) && !tensor_map_2d(&maps[b - 1], wq, 4, N, rows, columns, stage_rows(b), false)) return false;
  return true;
}

int launch_up(const Params& P, int tiles_bound, cudaStream_t stream) { return launch<kOutUp, false>(P, tiles_bound, stream); }
int launch_down(const Params& P, int tiles_bound, cudaStream_t stream) { return launch<kOutDown, false>(P, tiles_bound, stream); }

// A tile's time is its k-blocks': the de-quantisation of 256 columns (by bit width, whatever the tokens), or the MMAs of
// many tokens.  Few tokens and few columns leave most of the 74 pairs without a tile, so the tokens go to smaller tiles
// (more of them, each with its own de-quantisation) or k is split (fp32 parts through memory and a second launch),
// whichever is estimated to end first.  4096 x 4096, 2 bits, 32 rows: 19.4 us unsplit, on 16 pairs, 10.8 as taken; 14336 x 1024:
// 56.4, on 4, and 11.2.  linear_plan's constants are a fit (4 % rms) to 623 times of 64 to 1000 rows, 11 shapes of 512 to 14336 wide, 1
// to 4 bits, one call behind the other on weights out of L2: 5.3 us for the start and the end; a block of 64 k its de-quantisation or its
// MMAs; the epilogue of a tile by its rows; parts of k 1.3 us and their sums' way through memory.  (Fewer rows are outside the fit.)  Of 401
// calls of other shapes whose tiles or parts they changed, against the constants of linear_line_us on the GEMM before this one: 12 % less
// time, 349 faster and 12 slower by more than 3 % (148 rows of 14336 x 1024, 3 bits, 16 parts instead of 14: 15.0 -> 16.8 us).
struct GemmTimes {
  float start, block[4], block_row;  // us; of 64 k by bit width, and by row of the tile
  float epilogue_row;                // of a tile
  float parts, part_value;           // parts of k: their launch, a value of a part
  float smaller, more;               // what smaller tiles, more parts have to come down to
};
static LinearPlan fastest(const GemmTimes& t, int M, int N, int K, int bits, bool may_split) {
  const int pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1, KB = K / kBK, ct = cdiv(N, 2 * kCols);
  LinearPlan best = {kTokens, 1, (KB + 1) & ~1, 1e30f};
  for (int tr = kTokens; tr >= 32; tr /= 2) {
    const long long tiles = static_cast<long long>(ct) * cdiv(M, tr);
    const float rows = static_cast<float>(M < tr ? M : tr);
    const float mma = 0.37f * rows / kTokens, dequant = t.block[bits >= 1 && bits <= 4 ? bits - 1 : 1] + t.block_row * rows;
    for (int sp = 1; sp == 1 || (may_split && sp <= 16 && tiles * sp <= pairs && KB / sp >= 8); ++sp) {
      const int kb = (cdiv(KB, sp) + 1) & ~1;
      if (sp > 1 && cdiv(KB, kb) != sp) continue;
      const float rounds = static_cast<float>((tiles * sp + pairs - 1) / pairs);
      float us = t.start + rounds * (static_cast<float>(kb) * (mma > dequant ? mma : dequant) + t.epilogue_row * rows);
      if (sp > 1) us += t.parts + t.part_value * static_cast<float>(sp) * static_cast<float>(M) * static_cast<float>(N);
      if (us < (tr < best.tile_rows ? t.smaller : t.more) * best.us) best = {tr, sp, kb, us};  // more tiles, more copies of both operands
    }
  }
  return best;
}
LinearPlan linear_plan(int M, int N, int K, int bits, bool may_split) {
  return fastest({5.3f, {0.22f, 0.225f, 0.32f, 0.24f}, 0.0002f, 0.0056f, 1.3f, 1e-6f, 0.94f, 0.99f}, M, N, K, bits, may_split);
}
float linear_line_us(int M, int N, int K, int bits) {
  return fastest({3.f, {0.20f, 0.20f, 0.39f, 0.25f}, 0.f, 0.f, 2.5f, 2e-6f, 0.97f, 0.97f}, M, N, K, bits, true).us;
}

// The parts of k, in order, rounded and biased like the one launch does.  A thread takes four columns.
template <typename T>
__global__ void __launch_bounds__(256) linear_sum_kernel(const float* __restrict__ partial, const T* __restrict__ bias, T* __restrict__ y,
                                                         int splits, long long total, int N) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const long long i = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (i >= total) return;
  float4 v = *reinterpret_cast<const float4*>(partial + i);
#pragma unroll 4
  for (int s = 1; s < splits; ++s) {
    const float4 u = *reinterpret_cast<const float4*>(partial + s * total + i);
    v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
  }
  const float f[4] = {v.x, v.y, v.z, v.w};
  T o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    o[k] = as_act<T>(f[k]);
    if (bias) o[k] = as_act<T>(as_float<T>(o[k]) + as_float<T>(bias[i % N + k]));
  }
  *reinterpret_cast<uint2*>(y + i) = *reinterpret_cast<const uint2*>(o);
}

template <typename T>
static int launch_sum(const Params& P, void* y, cudaStream_t st) {
  const long long total = static_cast<long long>(P.rows) * P.fam[0].N;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((total / 4 + 255) / 256));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, linear_sum_kernel<T>, static_cast<const float*>(P.partial), static_cast<const T*>(P.bias),
                            static_cast<T*>(y), P.splits, total, P.fam[0].N) == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

}  // namespace ts
}  // namespace gemq

using namespace gemq;
using namespace gemq::ts;

extern "C" size_t gemq_linear_gemm_scratch_bytes(int M, int N, int K, int nbits) {
  if (M <= 0 || N <= 0 || K <= 0 || N % 32 || K % kBK) return 0;
  const LinearPlan L = linear_plan(M, N, K, nbits, true);
  return L.splits > 1 ? static_cast<size_t>(L.splits) * M * N * sizeof(float) : 0;
}

extern "C" int gemq_linear_gemm(const void* x, const int64_t* expert, const int32_t* wq, const void* scales, const void* zeros,
                                const int32_t* nbits, const int32_t* wq_strides, const int32_t* zs_strides, int fixed_bits,
                                const void* bias, void* y, int M, int N, int K, int group_size, int x_is_bf16, int32_t* err,
                                void* scratch, size_t scratch_bytes, gemq_stream_t stream) {
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
  P.staged = !expert && !nbits && !wq_strides && !zs_strides &&
             word_maps(P.w_map[0][0], wq, scales, zeros, N, fixed_bits == 3 ? cdiv(K, 10) : K * fixed_bits / 32, group_size, fixed_bits, kCols);
  P.rows = M;
  P.bias = bias;
  P.err = err;
  F.col_tiles = cdiv(N, 2 * kCols);
  const size_t need = scratch && aligned16(scratch) && !nbits ? gemq_linear_gemm_scratch_bytes(M, N, K, fixed_bits) : 0;
  const LinearPlan L = linear_plan(M, N, K, nbits ? 2 : fixed_bits, need > 0 && scratch_bytes >= need);
  P.tile_rows = L.tile_rows;
  P.splits = L.splits;
  P.split_kb = L.split_kb;
  P.partial = static_cast<float*>(scratch);
  const int tiles = F.col_tiles * cdiv(M, P.tile_rows) * P.splits;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc;
  if (P.splits > 1) {
    rc = x_is_bf16 ? launch<kOutPartial, true>(P, tiles, st) : launch<kOutPartial, false>(P, tiles, st);
    if (!rc) rc = x_is_bf16 ? launch_sum<__nv_bfloat16>(P, y, st) : launch_sum<__half>(P, y, st);
  } else {
    rc = x_is_bf16 ? launch<kOutLinear, true>(P, tiles, st) : launch<kOutLinear, false>(P, tiles, st);
  }
  return rc ? rc : launch_status();
}

extern "C" int gemq_dequant_gemm_tc(const void* x, const int64_t* expert, const int32_t* wq, const void* scales,
                                    const void* zeros, const int32_t* nbits, const int32_t* wq_strides,
                                    const int32_t* zs_strides, int fixed_bits, void* y, int M, int N, int K,
                                    int group_size, int x_is_bf16, int32_t* err, gemq_stream_t stream) {
  return gemq_linear_gemm(x, expert, wq, scales, zeros, nbits, wq_strides, zs_strides, fixed_bits, nullptr, y, M, N, K, group_size,
                          x_is_bf16, err, nullptr, 0, stream);
}
