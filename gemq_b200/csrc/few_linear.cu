// Dense quantised linear for a few rows in one launch (few_rows.cuh has the arithmetic).
//
// A CTA computes 64 columns; its four consumer warps split the reduction length, and a cluster of up to
// eight CTAs splits it further while the column tiles alone do not fill the chip.  Every consumer warp
// builds the table of its own part of the activation (a scale per row and group, so no exchange is needed) while
// the first weights travel; the partial sums meet in shared memory and, across the cluster, in rank 0's
// shared memory, and are added in a fixed order.  A table built by a launch of its own cost 3 us and a
// dependent launch per call, as much as the product itself.
#include "few_table.cuh"
#include "gemm_ts.cuh"

namespace gemq {
namespace few {

struct alignas(64) LinearParams {
  CUtensorMap wmap;      // strips of 32 columns, box of two
  const __half* sc;
  const __half* zr;
  const void* x;
  const void* bias;
  void* y;
  int* err;
  int ldx, vec;          // row pitch; 1: every row of x is 16-byte aligned
  int rows, tile_rows;   // all rows; rows of a tile (grid.z)
  int N, K, bits;
  int splits;            // cluster size
  int ring, tab_bytes;   // ring stages; table bytes of a warp
};

constexpr int kLinStage = kWStage + kMetaStage;

struct LinearShared {
  unsigned long long full[kMaxRing], empty[kMaxRing];
  int lo[kCons], hi[kCons];  // stages of each consumer warp
  alignas(16) unsigned char zero[16];
};

template <typename T, int B, int NB>
__device__ __forceinline__ void consume_linear(State<NB>& A, LinearShared& S, const LinearParams& P, unsigned char* ring,
                                               unsigned char* tab, const T* x, int rows, int iters, int warp, int lane) {
  const int lo = S.lo[warp], hi = S.hi[warp];
  const Rows R = {P.K, P.ldx, P.vec};
  if (B == 3) build_b3<T>(R, tab, x, rows, lo, hi, lane);
  else build_pow2<T, B == 3 ? 2 : B>(R, tab, x, rows, lo, hi, lane);
  __syncwarp();
  const uint32_t zero = smem_u32(S.zero), tab32 = smem_u32(tab), ring32 = smem_u32(ring), none = lds32(zero);
  int slot = 0;
  uint32_t par = 0;
#pragma unroll 1
  for (int it = 0; it < iters; ++it) {
    const uint32_t st = ring32 + slot * kLinStage;
    mbar_sleep_wait(&S.full[slot], par, P.err, kErrFewFull);
    const int sg = lo + it;
    if (sg < hi)
      stage_any<B, NB, kStrip>(A, st + warp * 2 * kStrip, tab32 + it * table_stage_bytes(B, rows), zero, st + kWStage + warp * 1024,
                               rows, sg, P.K / kGroup, lane);
    release_stage<NB>(A, &S.empty[slot], none, lane);
    if (++slot == P.ring) { slot = 0; par ^= 1u; }
  }
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void st_cluster_f4(uint32_t addr, uint32_t rank, const float4& v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

template <typename T, int NB>
__global__ void __launch_bounds__(kThreads, NB == 1 ? 3 : 2) few_linear_kernel(const __grid_constant__ LinearParams P) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ LinearShared S;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part = static_cast<int>(blockIdx.x % P.splits), n0 = 64 * static_cast<int>(blockIdx.x / P.splits);
  if (tid == 0) {
    for (int s = 0; s < kMaxRing; ++s) {
      mbar_init(&S.full[s], 1 + 32);  // the transaction count and the producer's cp.async lanes
      mbar_init(&S.empty[s], kCons);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid >= 32 && tid < 32 + kCons) {
    int lo, hi;
    stage_range(P.bits, P.K, part * kCons + tid - 32, P.splits * kCons, lo, hi);
    S.lo[tid - 32] = lo;
    S.hi[tid - 32] = hi;
  }
  if (tid >= 64 && tid < 68) reinterpret_cast<uint32_t*>(S.zero)[tid - 64] = 0u;
  pdl_launch();
  __syncthreads();
  // remote stores at the end need the peers to have started by then
  if (P.splits > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  int iters = 0;
#pragma unroll
  for (int q = 0; q < kCons; ++q) iters = max(iters, S.hi[q] - S.lo[q]);
  const int row0 = blockIdx.z * P.tile_rows;
  const int rows = min(P.tile_rows, P.rows - row0);
  float* red = reinterpret_cast<float*>(ring);  // the warps' sums, over the drained ring

  if (warp == kCons) {
    // ---- producer ------------------------------------------------------------------------------
    const int gshift = P.bits == 3 ? 1 : (P.bits == 4 ? 0 : (P.bits == 2 ? 1 : 2));  // log2 of the groups per stage
    const int ngroups = P.K / kGroup;
    const int piece = lane & 3, mst = (lane >> 2) & 1, kind = (lane >> 3) & 1;
    const int col = n0 + 32 * mst + 8 * piece;
    const __half* mbase = (kind ? P.zr : P.sc) + col;
    const uint32_t mdst = kWStage + kind * 128 + mst * 64 + piece * 16;
    const bool box = lane < kCons;
    const int my_lo = S.lo[lane & 3], my_hi = S.hi[lane & 3];
    // The matrix may be a result of the launch before (a layer packed and called at once): up to the wait its first
    // stages come into L2 only, where such a result goes, too.
    for (int it = 0; it < min(iters, P.ring); ++it)
      if (box && my_lo + it < my_hi) tma_prefetch_strips(&P.wmap, (my_lo + it) * kStageRows, n0 >> 5);
    if ((lane & 7) == 0 && col < P.N)
      for (int i = lane >> 4; i < (kCons << gshift); i += 2) {
        const int cw = i >> gshift, gi = i & ((1 << gshift) - 1), sg = S.lo[cw];
        const int grp = P.bits == 3 ? 5 * (sg >> 2) + (sg & 3) + gi : (sg << gshift) + gi;
        if (sg < S.hi[cw] && grp < ngroups) prefetch_l2(mbase + static_cast<size_t>(grp) * P.N);
      }
    pdl_wait();
    int slot = 0;
    uint32_t par = 1;
    for (int it = 0; it < iters; ++it) {
      mbar_sleep_wait(&S.empty[slot], par, P.err, kErrFewEmpty);
      unsigned char* st = ring + slot * kLinStage;
      const bool on = box && my_lo + it < my_hi;
      const unsigned boxes = __popc(__ballot_sync(0xffffffffu, on));
      if (lane == 0) mbar_arrive_expect_tx(&S.full[slot], boxes * 2 * kStrip);
      __syncwarp();
      if (on) tma_load_strips(st + lane * 2 * kStrip, &P.wmap, (my_lo + it) * kStageRows, n0 >> 5, &S.full[slot]);
      // scales | offsets: a lane copies 16 bytes of one group; (warp, group) units go two at a time
      const uint32_t dst = smem_u32(st) + mdst;
#pragma unroll 2
      for (int i = lane >> 4; i < (kCons << gshift); i += 2) {
        const int cw = i >> gshift, gi = i & ((1 << gshift) - 1);
        const int sg = S.lo[cw] + it;
        const int grp = P.bits == 3 ? 5 * (sg >> 2) + (sg & 3) + gi : (sg << gshift) + gi;
        if (sg < S.hi[cw] && grp < ngroups && col < P.N)
          cp_async16(dst + cw * 1024 + gi * 256, mbase + static_cast<size_t>(grp) * P.N);
      }
      cp_async_arrive(&S.full[slot]);
      if (++slot == P.ring) { slot = 0; par ^= 1u; }
    }
  } else {
    pdl_wait();  // x
    State<NB> A;
    clear(A);
    const T* x = static_cast<const T*>(P.x) + static_cast<size_t>(row0) * P.ldx;
    unsigned char* tab = ring + P.ring * kLinStage + warp * P.tab_bytes;
    if (P.bits == 1) consume_linear<T, 1, NB>(A, S, P, ring, tab, x, rows, iters, warp, lane);
    else if (P.bits == 2) consume_linear<T, 2, NB>(A, S, P, ring, tab, x, rows, iters, warp, lane);
    else if (P.bits == 3) consume_linear<T, 3, NB>(A, S, P, ring, tab, x, rows, iters, warp, lane);
    else consume_linear<T, 4, NB>(A, S, P, ring, tab, x, rows, iters, warp, lane);
    // the sums go over the ring: every consumer has to be done with it
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kCons) : "memory");
    const int g = lane >> 2, c = lane & 3;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int t = 8 * nb + 2 * c + o;
#pragma unroll
        for (int st = 0; st < 2; ++st)
          *reinterpret_cast<float4*>(red + (warp * kTileRows + t) * 64 + 32 * st + 4 * g) =
              result4<NB>(A, st, nb, o);
      }
  }
  // ---- add the warps' and the cluster's parts of k, in order ----------------------------------------
  __syncthreads();
  if (P.splits > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  float* mine = reinterpret_cast<float*>(ring + P.ring * kLinStage + kCons * P.tab_bytes);  // [splits][tile_rows][64] in rank 0
  const uint32_t rank = P.splits > 1 ? cluster_rank() : 0u;
  for (int i = tid; i < rows * 16; i += kThreads) {
    const int t = i >> 4, n4 = (i & 15) * 4;
    float4 v = *reinterpret_cast<const float4*>(red + t * 64 + n4);
#pragma unroll
    for (int q = 1; q < kCons; ++q) {
      const float4 u = *reinterpret_cast<const float4*>(red + (q * kTileRows + t) * 64 + n4);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    float* dst = mine + (rank * P.tile_rows + t) * 64 + n4;
    if (rank == 0) *reinterpret_cast<float4*>(dst) = v;
    else st_cluster_f4(smem_u32(dst), 0u, v);
  }
  if (P.splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (rank != 0) return;
  // a thread adds what it stored itself when there is no cluster: same loop, same indices
  for (int i = tid; i < rows * 16; i += kThreads) {
    const int t = i >> 4, n4 = (i & 15) * 4, n = n0 + n4;
    if (n >= P.N) continue;
    float4 v = *reinterpret_cast<const float4*>(mine + t * 64 + n4);
    for (int q = 1; q < P.splits; ++q) {
      const float4 u = *reinterpret_cast<const float4*>(mine + (q * P.tile_rows + t) * 64 + n4);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    const float f[4] = {v.x, v.y, v.z, v.w};
    T o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      o[k] = from_f<T>(f[k]);
      if (P.bias) o[k] = from_f<T>(to_f<T>(o[k]) + to_f<T>(static_cast<const T*>(P.bias)[n + k]));
    }
    *reinterpret_cast<uint2*>(static_cast<T*>(P.y) + static_cast<size_t>(row0 + t) * P.N + n) = *reinterpret_cast<const uint2*>(o);
  }
}

template <typename T, int NB>
static int launch_linear(const LinearParams& P, dim3 grid, size_t smem, cudaStream_t st) {
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GEMQ_ERR_LAUNCH;
  if (!done[dev]) {
    if (cudaFuncSetAttribute(few_linear_kernel<T, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDyn) != cudaSuccess)
      return GEMQ_ERR_LAUNCH;
    done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = P.splits;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = P.splits > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, few_linear_kernel<T, NB>, P) == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

}  // namespace few
}  // namespace gemq

using namespace gemq;
using namespace gemq::few;

// A warp's part of k is whole stages.  The cluster grows while the CTAs run at once (three per SM) and every warp
// keeps a stage, and as long as the warps' tables do not fit twice per SM.  448 CTAs on 444 places: 12.4 us
// instead of 9.3 (4 rows, 2816 x 14336, 2 bits).
static bool linear_split(int rows, int N, int K, int nbits, int* tile_rows, int* splits_out, int* tab_bytes, size_t* smem) {
  const int cols = cdiv(N, 64), units = n_stages(K, nbits), sms = sm_count();
  if (sms <= 0) return false;
  for (int tr = rows < kTileRows ? rows : kTileRows; tr > 0; tr = tr > 1 ? (tr + 1) / 2 : 0) {
    const int tiles = cdiv(rows, tr);
    int splits = 1;
    while (splits < 8 && cols * tiles * splits * 2 <= 3 * sms && units >= kCons * splits * 2) splits *= 2;
    for (;; splits *= 2) {
      *tab_bytes = (cdiv(units, kCons * splits) * table_stage_bytes(nbits, tr) + 127) / 128 * 128;
      *smem = 1024 + static_cast<size_t>(kMaxRing) * kLinStage + static_cast<size_t>(kCons) * *tab_bytes +
              static_cast<size_t>(splits) * tr * 64 * sizeof(float);
      if (*smem <= kMaxDyn / 2 || splits == 8 || units < kCons * splits * 2) break;
    }
    *tile_rows = tr;
    *splits_out = splits;
    if (*smem <= kMaxDyn) return true;
  }
  return false;
}

// Estimates in us of what the two kernels were measured to take (1 to 64 rows of 14 shapes, 512 to 14336 wide).  The
// GEMM: linear_line_us; the few-row kernel: rounds of the chip, each with a start and a table of the k of a warp.  The 3-bit table
// costs up to 2.5 times the others'.  Of 352 pairs (11 shapes, 1 to 4 bits, 4 to 64 rows, back to back) 52 take the one that is slower
// by more than 5 %: mostly 1- and 2-bit matrices, whose GEMM is estimated too low (8 rows of 4096 x 4096, 1 bit:
// few-row kernel 7.4 us, GEMM 10.2; the worst, 4 rows of 14336 x 14336, 1 bit: 36.6 and 61.1).
// The line does not follow the constants that linear_plan has since: the kernels round differently (weights to the activation type
// in the GEMM, not at all here), and drawn by those it is no better.  Of 518 calls that would come here 267 gain more than
// 3 % and 179 lose as much (128 rows of 4096 x 576, 4 bits: GEMM 9.4 us, few-row kernel 17.1); 3 rows of 14336 x 2816, 3 bits, bf16, would
// go to the GEMM and from an error of 1.65e-3 to 2.38e-3.
extern "C" int gemq_linear_takes_gemm(int rows, int N, int K, int nbits) {
  int tr, splits, tab;
  size_t smem;
  const int sms = sm_count();
  if (rows <= 0 || N <= 0 || K <= 0 || nbits < 1 || nbits > 4 || sms <= 0) return rows >= 32;
  if (!linear_split(rows, N, K, nbits, &tr, &splits, &tab, &smem)) return 1;
  const float gemm = ts::linear_line_us(rows, N, K, nbits);
  const int per_sm = tr > 8 || 3 * (smem + 2048) > kMaxDyn ? (2 * (smem + 2048) > kMaxDyn ? 1 : 2) : 3;
  const int rounds = cdiv(cdiv(N, 64) * splits * cdiv(rows, tr), per_sm * sms);
  const float warp_k = static_cast<float>(K) / static_cast<float>(kCons * splits);
  const float few = rounds * (rounds > 2 ? 1.5f : 1.f) * (tr > 8 ? 3.f + 0.024f * warp_k : 3.f + warp_k * (0.003f + 0.0011f * tr)) *
                    (nbits == 3 ? 1.2f + 0.17f * (tr > 8 ? 8 : tr) : 1.f);
  return gemm < few;
}

extern "C" int gemq_linear_rows(const void* x, int ldx, int x_is_bf16, const int32_t* wq, const void* scales, const void* zeros,
                                const void* bias, void* y, int rows, int N, int K, int nbits, int group_size, int32_t* err,
                                gemq_stream_t stream) {
  if (!x || !wq || !scales || !zeros || !y || !err || rows <= 0 || N <= 0 || K <= 0 || nbits < 1 || nbits > 4)
    return GEMQ_ERR_BAD_ARG;
  if (group_size != kGroup || K % kGroup || N % 32 || K > 32768) return GEMQ_ERR_BAD_SHAPE;
  if (!aligned16(wq) || !aligned16(scales) || !aligned16(zeros) || !aligned16(y)) return GEMQ_ERR_ALIGN;
  LinearParams P = {};
  if (!tensor_map_strips(&P.wmap, wq, N, packed_rows(K, nbits), 2)) return GEMQ_ERR_LAUNCH;
  P.sc = static_cast<const __half*>(scales);
  P.zr = static_cast<const __half*>(zeros);
  P.x = x; P.bias = bias; P.y = y; P.err = err;
  P.ldx = ldx;
  P.vec = aligned16(x) && (ldx % 8 == 0 || rows == 1);
  P.rows = rows; P.N = N; P.K = K; P.bits = nbits;
  size_t smem;
  if (!linear_split(rows, N, K, nbits, &P.tile_rows, &P.splits, &P.tab_bytes, &smem)) return GEMQ_ERR_BAD_SHAPE;
  P.ring = kMaxRing;
  const int tiles = cdiv(rows, P.tile_rows);
  if (tiles > 65535) return GEMQ_ERR_BAD_SHAPE;
  const dim3 grid(cdiv(N, 64) * P.splits, 1, tiles);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (P.tile_rows > 8)
    return x_is_bf16 ? launch_linear<__nv_bfloat16, 2>(P, grid, smem, st) : launch_linear<__half, 2>(P, grid, smem, st);
  return x_is_bf16 ? launch_linear<__nv_bfloat16, 1>(P, grid, smem, st) : launch_linear<__half, 1>(P, grid, smem, st);
}
