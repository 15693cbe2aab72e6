// Decode batches of a MoE layer: every selected expert is read once for its handful of rows
// (few_rows.cuh has the arithmetic; the large grouped GEMM takes over where the rows per expert make the
// tensor cores the better place).
//
//   plan     one CTA: rows grouped by expert in tiles of at most 16, the longest first
//   table    one CTA per row: the activation as tensor-core fragments of the expert's bit width.  Done once
//            per call: every CTA of the products would otherwise convert all rows for a few columns
//   up       128 gate and the same 128 up columns per CTA over the whole reduction length; the epilogue
//            forms h = silu(x1) * x3 and writes it as fragments of the down projection: its 128 columns
//            are one quantisation group there, so scale and sum need no exchange between CTAs
//   down     256 columns per CTA, k split over CTAs into fp32 partial rows
//   combine  adds the splits in order, then the token's experts with their weights
// All launches overlap their prologues with the kernel before (programmatic dependent launch).
#include "few_rows.cuh"

namespace gemq {
namespace few {

enum { kUp = 0, kDown = 1 };
constexpr int kErrBadExpertId = 21, kErrOffBoundary = 22;

// Tile of an expert: {expert (-1: the shared expert), first sorted row, rows, 0}.
struct Plan {
  int4* tiles;
  int* n_tiles;
  int* src;        // sorted row -> token
  int* inv;        // (token, slot) -> sorted row, -1: expert id out of range
  __half* row_w;   // sorted row -> routing weight
};

struct alignas(64) MoeParams {
  CUtensorMap wmap[4];       // [2 * family + matrix], family 1 = shared expert
  const __half* sc[4];
  const __half* zr[4];
  const int* nbits;          // of the matrices of this launch, routed experts
  const int* wqs;
  const int* zss[2];
  int sbits;
  int N[2], K[2];
  const int4* tiles;
  const int* n_tiles;
  const unsigned char* table;
  size_t tile_stride;
  unsigned char* next;       // up: the table of the down projection
  size_t next_stride;
  const int* next_nbits;
  int next_sbits;
  float* partial;            // down: [splits][partial_rows][N]
  int partial_rows, splits;
  int stage_bytes, ring;
  int* err;
};

struct MoeShared {
  unsigned long long full[kMaxRing], empty[kMaxRing];
  alignas(16) unsigned char zero[16];
};

// Strip distance of a warp's two strips: the gate columns' boxes come first, then the up columns'.
template <int MODE> constexpr int kStripStep = MODE == kUp ? kCons * kStrip : kStrip;

template <int MODE, int NB, int B>
__device__ __forceinline__ void consume_moe(State<NB>& A, MoeShared& S, const MoeParams& P, uint32_t ring, int lo, int hi, int rows,
                                            int ngroups, int warp, int lane) {
  const uint32_t zero = smem_u32(S.zero), none = lds32(zero);
  int slot = 0;
  uint32_t par = 0;
#pragma unroll 1
  for (int sg = lo; sg < hi; ++sg) {
    const uint32_t st = ring + slot * P.stage_bytes;
    mbar_sleep_wait(&S.full[slot], par, P.err, kErrFewFull);
    stage_any<B, NB, kStripStep<MODE>>(A, st + (MODE == kUp ? 1 : 2) * warp * kStrip, st + kWStage + kMetaStage, zero,
                                       st + kWStage + warp * 1024, rows, sg, ngroups, lane);
    release_stage<NB>(A, &S.empty[slot], none, lane);
    if (++slot == P.ring) { slot = 0; par ^= 1u; }
  }
}

template <int MODE, int NB>
__device__ __forceinline__ void run_tile(MoeShared& S, const MoeParams& P, unsigned char* ring, int bits, int lo, int hi, int rows,
                                         int row0, int N, int ngroups, int n0, unsigned char* next, int next_bits, int warp,
                                         int lane) {
  State<NB> A;
  clear(A);
  if (bits == 1) consume_moe<MODE, NB, 1>(A, S, P, smem_u32(ring), lo, hi, rows, ngroups, warp, lane);
  else if (bits == 2) consume_moe<MODE, NB, 2>(A, S, P, smem_u32(ring), lo, hi, rows, ngroups, warp, lane);
  else if (bits == 3) consume_moe<MODE, NB, 3>(A, S, P, smem_u32(ring), lo, hi, rows, ngroups, warp, lane);
  else consume_moe<MODE, NB, 4>(A, S, P, smem_u32(ring), lo, hi, rows, ngroups, warp, lane);
  const int g = lane >> 2, c = lane & 3;
  if (MODE == kUp) {
    // h of the tile over the drained ring, then half a warp per row turns it into fragments
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kCons) : "memory");
    __half* hb = reinterpret_cast<__half*>(ring);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int t = 8 * nb + 2 * c + o;
        const float4 a = result4<NB>(A, 0, nb, o), b = result4<NB>(A, 1, nb, o);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
        __half h[4];
        // silu(x1) * x3 on fp16 tensors: x1, x3, silu(x1) and the product are rounded
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __float2half_rn(round_h(silu_f32(round_h(av[i]))) * round_h(bv[i]));
        if (t < rows) *reinterpret_cast<uint2*>(hb + t * kGroup + 32 * warp + 4 * g) = *reinterpret_cast<const uint2*>(h);
      }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kCons) : "memory");
    for (int t0 = 2 * warp; t0 < rows; t0 += 2 * kCons) {
      const int t = min(t0 + (lane >> 4), rows - 1);  // an odd row count: both halves write the last row alike
      group_to_table<__half>(hb + t * kGroup, next_bits, n0 / kGroup, next, rows, t, lane);
    }
  } else {
    float* dst = P.partial + (static_cast<size_t>(blockIdx.x % P.splits) * P.partial_rows + row0) * N;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int t = 8 * nb + 2 * c + o;
#pragma unroll
        for (int st = 0; st < 2; ++st) {
          const int n = n0 + 64 * warp + 32 * st + 4 * g;
          if (t < rows && n < N) *reinterpret_cast<float4*>(dst + static_cast<size_t>(t) * N + n) = result4<NB>(A, st, nb, o);
        }
      }
  }
}

// MAXNB = 1: tiles of at most eight rows; 2: at most sixteen.
template <int MODE, int MAXNB>
__global__ void __launch_bounds__(kThreads, 3) few_moe_kernel(const __grid_constant__ MoeParams P) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // barriers in the first kilobyte, then the ring (1024-byte aligned like the array): three CTAs share an SM's
  // 228 KB to the last kilobyte
  MoeShared& S = *reinterpret_cast<MoeShared*>(smem_raw);
  unsigned char* ring = smem_raw + 1024;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Tiles and weights are read ahead of the wait, the table after it: the first stages travel under the tail of the launch
  // before (16 DeepSeek-V2-Lite tokens 87.4 -> 82.5 us).  What makes this sound is the table launch: each of its CTAs waits
  // before it lets up start, so the plan, and what came before the call, is complete before a CTA of up runs, and those of down start
  // after some of up's.  (That the producer warps release ahead of their wait does not matter then; released by the other warps
  // alone, after theirs: 83.1 -> 83.9 us.)  The plan of the call before may lie at the same place, and this kernel has not
  // waited yet: it is read from L2.
  const int tile = blockIdx.y;
  const int n_tiles = __ldcg(P.n_tiles);
  const int4 d = __ldcg(P.tiles + tile);  // the list is as long as the grid
  if (tid == 0) {
    for (int s = 0; s < kMaxRing; ++s) {
      mbar_init(&S.full[s], 1 + 32);
      mbar_init(&S.empty[s], kCons);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid >= 64 && tid < 68) reinterpret_cast<uint32_t*>(S.zero)[tid - 64] = 0u;
  if (tile >= n_tiles) {
    if (tile == 0) pdl_wait();  // a grid without a tile does not end before the launch ahead of it, either
    return;
  }
  const int fam = d.x < 0 ? 1 : 0, row0 = d.y, rows = d.z;
  const int N = P.N[fam], K = P.K[fam], ngroups = K / kGroup;
  constexpr int kCols = MODE == kUp ? 32 * kCons : 64 * kCons;
  const int part = static_cast<int>(blockIdx.x % P.splits), n0 = kCols * static_cast<int>(blockIdx.x / P.splits);
  if (n0 >= N) return;  // the launch covers the wider of the two families
  int bits = fam ? P.sbits : P.nbits[d.x];
  bits = clamp_bits(bits);
  int lo, hi;
  stage_range(bits, K, part, P.splits, lo, hi);
  __syncthreads();
  if (warp != kCons) pdl_wait();  // the producer: behind its first loads
  pdl_launch();

  if (warp == kCons) {
    // ---- producer --------------------------------------------------------------------------------
    const int wrow = fam ? 0 : static_cast<int>(static_cast<unsigned>(P.wqs[d.x]) / static_cast<unsigned>(N));
    const int gshift = bits == 3 ? 1 : (bits == 4 ? 0 : (bits == 2 ? 1 : 2));  // log2 of the groups per stage
    const int tb = table_stage_bytes(bits, rows);
    const unsigned char* table = P.table + tile * P.tile_stride;
    // scales | offsets: a lane copies 16 bytes of one group; (warp, group) units go two at a time
    const int piece = lane & 3, mst = (lane >> 2) & 1, kind = (lane >> 3) & 1;
    const int m = 2 * fam + (MODE == kUp ? mst : 0);
    size_t zoff = 0;
    if (!fam) {
      const int* zs = P.zss[MODE == kUp ? mst : 0];
      zoff = zs ? static_cast<size_t>(zs[d.x]) : static_cast<size_t>(d.x) * ngroups * N;
    }
    const int col = n0 + (MODE == kUp ? 0 : 32 * mst) + 8 * piece;
    const __half* mbase = (kind ? P.zr[m] : P.sc[m]) + zoff + col;
    const uint32_t mdst = kWStage + kind * 128 + mst * 64 + piece * 16;
    constexpr int kColStep = MODE == kUp ? 32 : 64;
    int slot = 0;
    uint32_t par = 1;
    const int ahead = min(lo + P.ring, hi);  // stages that are on their way before the wait
    auto load_table = [&](int sg, int at) {
      bulk_load(ring + at * P.stage_bytes + kWStage + kMetaStage, table + static_cast<size_t>(sg) * tb, tb, &S.full[at]);
    };
    for (int sg = lo; sg < hi; ++sg) {
      if (sg >= ahead) mbar_sleep_wait(&S.empty[slot], par, P.err, kErrFewEmpty);
      unsigned char* st = ring + slot * P.stage_bytes;
      if (lane == 0) {
        mbar_arrive_expect_tx(&S.full[slot], kWStage + tb);
        tma_load_strips(st, &P.wmap[2 * fam], wrow + sg * kStageRows, n0 >> 5, &S.full[slot]);
        if (MODE == kUp)
          tma_load_strips(st + kCons * kStrip, &P.wmap[2 * fam + 1], wrow + sg * kStageRows, n0 >> 5, &S.full[slot]);
        if (sg >= ahead) load_table(sg, slot);
      }
      __syncwarp();
      const uint32_t dst = smem_u32(st) + mdst;
#pragma unroll 2
      for (int i = lane >> 4; i < (kCons << gshift); i += 2) {
        const int cw = i >> gshift, gi = i & ((1 << gshift) - 1);
        const int grp = bits == 3 ? 5 * (sg >> 2) + (sg & 3) + gi : (sg << gshift) + gi;
        if (grp < ngroups && col + kColStep * cw < N)
          cp_async16(dst + cw * 1024 + gi * 256, mbase + static_cast<size_t>(grp) * N + kColStep * cw);
      }
      cp_async_arrive(&S.full[slot]);
      if (sg + 1 == ahead) {
        pdl_wait();
        if (lane == 0)
          for (int i = lo; i < ahead; ++i) load_table(i, i - lo);
      }
      if (++slot == P.ring) { slot = 0; par ^= 1u; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  unsigned char* next = MODE == kUp ? P.next + tile * P.next_stride : nullptr;
  int nbits2 = 0;
  if (MODE == kUp) {
    nbits2 = fam ? P.next_sbits : P.next_nbits[d.x];
    nbits2 = clamp_bits(nbits2);
  }
  if (MAXNB == 1 || rows <= 8)
    run_tile<MODE, 1>(S, P, ring, bits, lo, hi, rows, row0, N, ngroups, n0, next, nbits2, warp, lane);
  else
    run_tile<MODE, MAXNB>(S, P, ring, bits, lo, hi, rows, row0, N, ngroups, n0, next, nbits2, warp, lane);
}

// ---- activation table of the up projection: one CTA per (tile, row) ------------------------------
struct TableParams {
  const void* x;
  int K;
  const int4* tiles;
  const int* n_tiles;
  const int* src;
  const int* nbits;
  int sbits;
  unsigned char* table;
  size_t tile_stride;
};

constexpr int kTabThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kTabThreads) few_table_kernel(const __grid_constant__ TableParams P) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  T* xs = reinterpret_cast<T*>(smem_raw);
  const int tile = blockIdx.y, t = blockIdx.x, tid = threadIdx.x;
  pdl_wait();
  pdl_launch();  // after the wait, in every CTA: the products read the plan and the weights ahead of theirs
  if (tile >= *P.n_tiles) return;
  const int4 d = P.tiles[tile];
  if (t >= d.z) return;
  int bits = d.x < 0 ? P.sbits : P.nbits[d.x];
  bits = clamp_bits(bits);
  const T* src = static_cast<const T*>(P.x) + static_cast<size_t>(P.src[d.y + t]) * P.K;
  for (int i = tid; i < P.K / 8; i += kTabThreads) reinterpret_cast<uint4*>(xs)[i] = reinterpret_cast<const uint4*>(src)[i];
  __syncthreads();
  unsigned char* tab = P.table + tile * P.tile_stride;
  const int ngroups = P.K / kGroup;
  for (int g0 = 2 * (tid >> 5); g0 < ngroups; g0 += kTabThreads / 16) {
    const int grp = min(g0 + ((tid >> 4) & 1), ngroups - 1);
    group_to_table<T>(xs + grp * kGroup, bits, grp, tab, d.z, t, tid & 31);
  }
}

// ---- permutation of the batch: one CTA -----------------------------------------------------------
constexpr int kPlanThreads = 512;

// Experts that begin off a whole row of words or a 16-byte boundary of scales cannot be copied by these launches: their rows are
// left out like those of an id out of range, and reported.  (The GEMM, which larger batches take, loads them.)
// Sorted rows: the experts whose tiles take longest first (the CTAs start in this order); the shared
// expert's tokens come behind the routed rows, its tiles lead the tile list.
template <typename T>
__global__ void __launch_bounds__(kPlanThreads) few_plan_kernel(Plan pl, const long long* __restrict__ idx, const T* __restrict__ w,
                                                                const int* __restrict__ nbits, Offsets off, int R, int A, int E,
                                                                int tokens, int tile_rows, int shared, int* err) {
  __shared__ int count[256], start[256], n_tile[256], key[256];
  const int tid = threadIdx.x;
  for (int e = tid; e < E; e += kPlanThreads) { count[e] = 0; key[e] = off_boundary(off, e) ? -1 : clamp_bits(nbits[e]); }
  pdl_launch();
  pdl_wait();
  if (tid == 0) *err = 0;
  __syncthreads();
  // A thread's first kHeld pairs stay in registers, loads in flight together; longer lists go through pl.inv.
  constexpr int kHeld = 2;
  int ex[kHeld], at[kHeld];
  T wt[kHeld];
  long long id[kHeld];
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    const int i = tid + u * kPlanThreads;
    id[u] = i < R ? idx[i] : 0;
    if (i < R) wt[u] = w[i];
  }
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    ex[u] = -1;
    if (tid + u * kPlanThreads < R) {
      if (id[u] < 0 || id[u] >= E) atomicExch(err, kErrBadExpertId);
      else if (key[static_cast<int>(id[u])] < 0) atomicExch(err, kErrOffBoundary);
      else {
        ex[u] = static_cast<int>(id[u]);
        at[u] = atomicAdd(&count[ex[u]], 1);
      }
    }
  }
  for (int i = tid + kHeld * kPlanThreads; i < R; i += kPlanThreads) {
    const long long e = idx[i];
    const int bad = e < 0 || e >= E ? kErrBadExpertId : (key[static_cast<int>(e)] < 0 ? kErrOffBoundary : 0);
    if (bad) atomicExch(err, bad);
    pl.inv[i] = bad ? -1 : atomicAdd(&count[static_cast<int>(e)], 1);
  }
  __syncthreads();
  // longest first: two blocks of eight rows take twice the MMAs of one, more bits more copying
  for (int e = tid; e < E; e += kPlanThreads) {
    key[e] += count[e] > 8 ? 8 : 0;
    n_tile[e] = cdiv(count[e], tile_rows);
  }
  __syncthreads();
  const int sh_tiles = shared ? cdiv(tokens, tile_rows) : 0;
  for (int e = tid; e < E; e += kPlanThreads) {
    int row = 0, tile = sh_tiles, total = sh_tiles;
    const int mine = key[e];
#pragma unroll 4
    for (int o = 0; o < E; ++o) {
      const int n = count[o], nt = n_tile[o], k = key[o];
      total += nt;
      if (k > mine || (k == mine && o < e)) { row += n; tile += nt; }
    }
    start[e] = row;
    for (int r = 0; r < count[e]; r += tile_rows) pl.tiles[tile++] = make_int4(e, row + r, min(tile_rows, count[e] - r), 0);
    if (e == 0) *pl.n_tiles = total;
  }
  for (int i = tid; i < sh_tiles; i += kPlanThreads)
    pl.tiles[i] = make_int4(-1, R + i * tile_rows, min(tile_rows, tokens - i * tile_rows), 0);
  if (shared)
    for (int i = tid; i < tokens; i += kPlanThreads) pl.src[R + i] = i;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    const int i = tid + u * kPlanThreads;
    if (i >= R) continue;
    const int pos = ex[u] < 0 ? -1 : start[ex[u]] + at[u];
    if (pos >= 0) {
      pl.src[pos] = i / A;
      pl.row_w[pos] = __float2half_rn(to_f<T>(wt[u]));
    }
    pl.inv[i] = pos;
  }
  for (int i = tid + kHeld * kPlanThreads; i < R; i += kPlanThreads) {
    const int p = pl.inv[i];
    if (p < 0) continue;
    const int pos = start[static_cast<int>(idx[i])] + p;
    pl.src[pos] = i / A;
    pl.row_w[pos] = __float2half_rn(to_f<T>(w[i]));
    pl.inv[i] = pos;
  }
}

// out[t]: the k splits of a row are added in order, rounded and weighted like the rows of the large
// grouped GEMM; the token's experts are added in increasing id, each sum rounded to the activation
// type (index_add_ in the loop of gemq/inference/moe_block.py:191-195), then the shared expert.
template <typename T>
__global__ void __launch_bounds__(128) few_combine_kernel(const int* __restrict__ inv, const long long* __restrict__ idx,
                                                          const __half* __restrict__ row_w, const float* __restrict__ partial,
                                                          int partial_rows, int splits, int shared_row0, T* __restrict__ out, int A,
                                                          int D) {
  __shared__ int rows[kMaxSlots + 1];
  __shared__ float wts[kMaxSlots + 1];
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.y;
  if (threadIdx.x < A) {  // rank of the slot by (expert id, slot)
    const int a = threadIdx.x;
    const long long e = idx[static_cast<size_t>(t) * A + a];
    int rank = 0;
    for (int b = 0; b < A; ++b) {
      const long long o = idx[static_cast<size_t>(t) * A + b];
      rank += (o < e || (o == e && b < a)) ? 1 : 0;
    }
    const int r = inv[static_cast<size_t>(t) * A + a];
    rows[rank] = r;
    wts[rank] = r >= 0 ? __half2float(row_w[r]) : 0.f;
  }
  if (threadIdx.x == 0) {
    rows[A] = shared_row0 >= 0 ? shared_row0 + t : -1;
    wts[A] = 1.f;
  }
  __syncthreads();
  const int n = 4 * (blockIdx.x * 128 + threadIdx.x);
  if (n >= D) return;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int a = 0; a <= A; ++a) {
    const int r = rows[a];
    if (r < 0) continue;
    const float* p = partial + static_cast<size_t>(r) * D + n;
    float4 v = *reinterpret_cast<const float4*>(p);
#pragma unroll 4
    for (int s = 1; s < splits; ++s) {
      const float4 u = *reinterpret_cast<const float4*>(p + static_cast<size_t>(s) * partial_rows * D);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float y = round_h(round_h(f[k]) * wts[a]);
      acc[k] = to_f<T>(from_f<T>(acc[k] + to_f<T>(from_f<T>(y))));
    }
  }
  T o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) o[k] = from_f<T>(acc[k]);
  *reinterpret_cast<uint2*>(out + static_cast<size_t>(t) * D + n) = *reinterpret_cast<const uint2*>(o);
}

// ---- host -------------------------------------------------------------------------------------------
struct Layout {
  Plan plan;
  unsigned char* tabx;
  unsigned char* tabh;
  float* partial;
  size_t stride_x, stride_h;
  int tile_rows, max_tiles, rows, splits;
};

// Tiles of eight rows leave registers and shared memory for a third CTA per SM; sixteen pay off once most
// experts have more than eight rows.
static int tile_rows_of(const gemq_moe_layer_t* L, int tokens) {
  return static_cast<long long>(tokens) * L->top_k <= 5ll * L->n_experts ? 8 : 16;
}

// k splits of the down projection: enough CTAs for about six per SM.
static int down_splits(const gemq_moe_layer_t* L, int tokens, int tile_rows) {
  const int R = tokens * L->top_k, E = L->n_experts;
  const int tiles = (R < E ? R : E) + (L->shared_ffn ? cdiv(tokens, tile_rows) : 0);
  const int kmax = L->ffn > L->shared_ffn ? L->ffn : L->shared_ffn;
  const int want = 6 * sm_count_or_default() / (cdiv(L->hidden, 64 * kCons) * tiles);
  const int most = kmax / 512;  // a part keeps at least 512 of the reduction
  int s = want < 1 ? 1 : want;
  s = s > most ? most : s;
  return s < 1 ? 1 : (s > 16 ? 16 : s);
}

size_t moe_few_rows_layout(const gemq_moe_layer_t* L, int tokens, Layout* Y, char* base) {
  const int E = L->n_experts, SF = L->shared_ffn;
  const size_t R = static_cast<size_t>(tokens) * L->top_k;
  const int tr = tile_rows_of(L, tokens);
  const size_t routed = R / tr + (R < static_cast<size_t>(E) ? R : static_cast<size_t>(E));
  const size_t tiles = routed + (SF ? cdiv(tokens, tr) : 0);
  const size_t rows = R + (SF ? tokens : 0);
  const int kmax = L->ffn > SF ? L->ffn : SF;
  const size_t sx = (table_tile_bytes(L->hidden, tr) + 255) / 256 * 256, sh = (table_tile_bytes(kmax, tr) + 255) / 256 * 256;
  const int splits = down_splits(L, tokens, tr);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 255) / 256 * 256;
    return base ? base + o : nullptr;
  };
  char* tl = take(sizeof(int4) * tiles);
  char* nt = take(sizeof(int));
  char* src = take(sizeof(int) * rows);
  char* inv = take(sizeof(int) * R);
  char* rw = take(sizeof(__half) * R);
  char* tx = take(sx * tiles);
  char* th = take(sh * tiles);
  char* pt = take(sizeof(float) * splits * rows * L->hidden);
  if (Y) {
    Y->plan.tiles = reinterpret_cast<int4*>(tl);
    Y->plan.n_tiles = reinterpret_cast<int*>(nt);
    Y->plan.src = reinterpret_cast<int*>(src);
    Y->plan.inv = reinterpret_cast<int*>(inv);
    Y->plan.row_w = reinterpret_cast<__half*>(rw);
    Y->tabx = reinterpret_cast<unsigned char*>(tx);
    Y->tabh = reinterpret_cast<unsigned char*>(th);
    Y->partial = reinterpret_cast<float*>(pt);
    Y->stride_x = sx; Y->stride_h = sh;
    Y->tile_rows = tr; Y->max_tiles = static_cast<int>(tiles); Y->rows = static_cast<int>(rows); Y->splits = splits;
  }
  return off;
}

template <typename... P, typename... A>
static bool launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}

static bool init_attrs() {
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (done[dev]) return true;
  auto allow = [](const void* k, int bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
  };
  if (!allow(reinterpret_cast<const void*>(few_moe_kernel<kUp, 1>), kMaxDyn) ||
      !allow(reinterpret_cast<const void*>(few_moe_kernel<kUp, 2>), kMaxDyn) ||
      !allow(reinterpret_cast<const void*>(few_moe_kernel<kDown, 1>), kMaxDyn) ||
      !allow(reinterpret_cast<const void*>(few_moe_kernel<kDown, 2>), kMaxDyn) ||
      !allow(reinterpret_cast<const void*>(few_table_kernel<__half>), 64 * 1024) ||
      !allow(reinterpret_cast<const void*>(few_table_kernel<__nv_bfloat16>), 64 * 1024))
    return false;
  done[dev] = true;
  return true;
}

// Layers and batches this path takes: group 128, extents in whole groups, and on average at most kFewAverage rows per
// expert.  Above, the GEMM takes over, whose cost hardly grows with the rows.  It would be the faster from 16 to 20 rows on, but
// it rounds every weight to fp16 (and bf16 activations, which end at 65504 there), where these launches take the codes, scales and
// offsets as they are: a faster call is no reason to move the line down.  us of a layer, here and by the GEMM:
//   64 experts of 2048 x 1408    16 rows 174 173   18 rows 184 175   24 rows 218 177
//   32 of them                   16 rows 108 112   18 rows 113 112   24 rows 136 114
//   16 of 2048 x 3456            16 rows  97 103   18 rows 106 105   24 rows 117 105
//   8 of 4096 x 7168             14 rows 129 143   16 rows 146 143   24 rows 165 145
//   8 of 4096 x 14336            18 rows 269 295   20 rows 272 295   24 rows 320 295
constexpr int kFewAverage = 24;
bool moe_few_rows_ok(const gemq_moe_layer_t* L, int tokens) {
  const int D = L->hidden, F = L->ffn, SF = L->shared_ffn;
  if (L->group_size != kGroup || D % kGroup || F % kGroup || SF % kGroup || D > 32768) return false;
  if (SF && (L->s1.group_size != kGroup || L->s3.group_size != kGroup || L->s2.group_size != kGroup)) return false;
  if (L->top_k > kMaxSlots || L->n_experts > 256) return false;
  const void* ptrs[] = {L->w1.wq, L->w1.scales, L->w1.zeros, L->w3.wq, L->w3.scales, L->w3.zeros, L->w2.wq, L->w2.scales,
                        L->w2.zeros};
  for (const void* p : ptrs)
    if (!aligned16(p)) return false;
  const void* shared[] = {L->s1.wq, L->s1.scales, L->s1.zeros, L->s3.wq, L->s3.scales, L->s3.zeros, L->s2.wq, L->s2.scales,
                          L->s2.zeros};
  if (SF)
    for (const void* p : shared)
      if (!aligned16(p)) return false;
  if (L->w1.wq_rows <= 0 || L->w3.wq_rows <= 0 || L->w2.wq_rows <= 0) return false;
  const long long R = static_cast<long long>(tokens) * L->top_k;
  return R <= static_cast<long long>(kFewAverage) * L->n_experts && tokens <= 4096;
}

size_t moe_few_rows_bytes(const gemq_moe_layer_t* L, int tokens) { return moe_few_rows_layout(L, tokens, nullptr, nullptr); }

int moe_few_rows(const gemq_moe_layer_t* L, const void* x, void* out, const long long* idx, const void* w, int tokens, bool bf16,
                 char* scratch, int* err, cudaStream_t st) {
  if (!init_attrs()) return GEMQ_ERR_LAUNCH;
  const int D = L->hidden, F = L->ffn, SF = L->shared_ffn, A = L->top_k, E = L->n_experts, R = tokens * A;
  Layout Y;
  moe_few_rows_layout(L, tokens, &Y, scratch);
  bool ok;
  if (bf16)
    ok = launch(few_plan_kernel<__nv_bfloat16>, dim3(1), kPlanThreads, 0, st, Y.plan, idx, static_cast<const __nv_bfloat16*>(w),
                static_cast<const int*>(L->w1.nbits), expert_offsets(L), R, A, E, tokens, Y.tile_rows, SF > 0 ? 1 : 0, err);
  else
    ok = launch(few_plan_kernel<__half>, dim3(1), kPlanThreads, 0, st, Y.plan, idx, static_cast<const __half*>(w),
                static_cast<const int*>(L->w1.nbits), expert_offsets(L), R, A, E, tokens, Y.tile_rows, SF > 0 ? 1 : 0, err);
  if (!ok) return GEMQ_ERR_LAUNCH;

  TableParams T = {};
  T.x = x; T.K = D;
  T.tiles = Y.plan.tiles; T.n_tiles = Y.plan.n_tiles; T.src = Y.plan.src;
  T.nbits = L->w1.nbits; T.sbits = L->s1.nbits;
  T.table = Y.tabx; T.tile_stride = Y.stride_x;
  const dim3 tgrid(Y.tile_rows, Y.max_tiles);
  ok = bf16 ? launch(few_table_kernel<__nv_bfloat16>, tgrid, kTabThreads, static_cast<size_t>(D) * 2, st, T)
            : launch(few_table_kernel<__half>, tgrid, kTabThreads, static_cast<size_t>(D) * 2, st, T);
  if (!ok) return GEMQ_ERR_LAUNCH;

  const int nb = Y.tile_rows / 8;
  int tab = 0;
  for (int b = 1; b <= 4; ++b) tab = table_stage_bytes(b, Y.tile_rows) > tab ? table_stage_bytes(b, Y.tile_rows) : tab;
  const int stage = (kWStage + kMetaStage + tab + 1023) / 1024 * 1024;
  const int ring = 2;  // three CTAs per SM
  const size_t smem = 1024 + static_cast<size_t>(ring) * stage;

  MoeParams U = {};
  const gemq_stacked_t* up[2] = {&L->w1, &L->w3};
  const gemq_single_t* sup[2] = {&L->s1, &L->s3};
  for (int m = 0; m < 2; ++m) {
    if (!tensor_map_strips(&U.wmap[m], up[m]->wq, F, up[m]->wq_rows, kCons)) return GEMQ_ERR_LAUNCH;
    U.sc[m] = static_cast<const __half*>(up[m]->scales);
    U.zr[m] = static_cast<const __half*>(up[m]->zeros);
    U.zss[m] = up[m]->zs_strides;
    if (SF) {
      if (!tensor_map_strips(&U.wmap[2 + m], sup[m]->wq, SF, packed_rows(D, L->s1.nbits), kCons)) return GEMQ_ERR_LAUNCH;
      U.sc[2 + m] = static_cast<const __half*>(sup[m]->scales);
      U.zr[2 + m] = static_cast<const __half*>(sup[m]->zeros);
    }
  }
  U.nbits = L->w1.nbits; U.wqs = L->w1.wq_strides; U.sbits = L->s1.nbits;
  U.N[0] = F; U.N[1] = SF; U.K[0] = U.K[1] = D;
  U.tiles = Y.plan.tiles; U.n_tiles = Y.plan.n_tiles;
  U.table = Y.tabx; U.tile_stride = Y.stride_x;
  U.next = Y.tabh; U.next_stride = Y.stride_h; U.next_nbits = L->w2.nbits; U.next_sbits = L->s2.nbits;
  U.splits = 1; U.stage_bytes = stage; U.ring = ring; U.err = err;
  const dim3 ugrid(cdiv(F > SF ? F : SF, 32 * kCons), Y.max_tiles);
  ok = nb == 1 ? launch(few_moe_kernel<kUp, 1>, ugrid, kThreads, smem, st, U)
               : launch(few_moe_kernel<kUp, 2>, ugrid, kThreads, smem, st, U);
  if (!ok) return GEMQ_ERR_LAUNCH;

  MoeParams Q = {};
  if (!tensor_map_strips(&Q.wmap[0], L->w2.wq, D, L->w2.wq_rows, 2 * kCons)) return GEMQ_ERR_LAUNCH;
  Q.sc[0] = static_cast<const __half*>(L->w2.scales);
  Q.zr[0] = static_cast<const __half*>(L->w2.zeros);
  Q.zss[0] = L->w2.zs_strides;
  if (SF) {
    if (!tensor_map_strips(&Q.wmap[2], L->s2.wq, D, packed_rows(SF, L->s2.nbits), 2 * kCons)) return GEMQ_ERR_LAUNCH;
    Q.sc[2] = static_cast<const __half*>(L->s2.scales);
    Q.zr[2] = static_cast<const __half*>(L->s2.zeros);
  }
  Q.nbits = L->w2.nbits; Q.wqs = L->w2.wq_strides; Q.sbits = L->s2.nbits;
  Q.N[0] = Q.N[1] = D; Q.K[0] = F; Q.K[1] = SF;
  Q.tiles = Y.plan.tiles; Q.n_tiles = Y.plan.n_tiles;
  Q.table = Y.tabh; Q.tile_stride = Y.stride_h;
  Q.partial = Y.partial; Q.partial_rows = Y.rows;
  Q.splits = Y.splits; Q.stage_bytes = stage; Q.ring = ring; Q.err = err;
  const dim3 dgrid(cdiv(D, 64 * kCons) * Y.splits, Y.max_tiles);
  ok = nb == 1 ? launch(few_moe_kernel<kDown, 1>, dgrid, kThreads, smem, st, Q)
               : launch(few_moe_kernel<kDown, 2>, dgrid, kThreads, smem, st, Q);
  if (!ok) return GEMQ_ERR_LAUNCH;

  const dim3 cgrid(cdiv(D, 512), tokens);
  const int* inv = Y.plan.inv;
  const __half* rw = Y.plan.row_w;
  const float* pt = Y.partial;
  ok = bf16 ? launch(few_combine_kernel<__nv_bfloat16>, cgrid, 128, 0, st, inv, idx, rw, pt, Y.rows, Y.splits, SF > 0 ? R : -1,
                     static_cast<__nv_bfloat16*>(out), A, D)
            : launch(few_combine_kernel<__half>, cgrid, 128, 0, st, inv, idx, rw, pt, Y.rows, Y.splits, SF > 0 ? R : -1,
                     static_cast<__half*>(out), A, D);
  return ok ? launch_status() : GEMQ_ERR_LAUNCH;
}

}  // namespace few
}  // namespace gemq
