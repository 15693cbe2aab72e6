// n-token forward of a quantised MoE layer (gemq/inference/moe_block.py:165-198, :448-486):
//
//   route -> plan (rows grouped by expert, tiles of up to 256) -> gather (rows in fp16, in the order of the
//   expert's packed words) -> gate/up GEMM with the SiLU product -> down GEMM with the routing weight ->
//   combine (the token's experts in increasing id, then the shared expert)
//
// The shared expert's tokens are further rows of the same launches.  Batches with few rows per
// expert take few_moe.cu instead.  Nothing of the routing reaches the host.
#include "gemm_ts.cuh"

namespace gemq {

// route.cu
int route_tokens(const void* x, const void* gate, bool gate_half, int tokens, int D, int E, int A, int mode, int renorm, bool bf16,
                 int64_t* idx, void* weights, void* logits, bool logits_act, cudaStream_t stream);

namespace few {  // few_moe.cu
bool moe_few_rows_ok(const gemq_moe_layer_t* L, int tokens);
size_t moe_few_rows_bytes(const gemq_moe_layer_t* L, int tokens);
int moe_few_rows(const gemq_moe_layer_t* L, const void* x, void* out, const long long* idx, const void* w, int tokens, bool bf16,
                 char* scratch, int* err, cudaStream_t st);
}  // namespace few

namespace {

constexpr int kTile = ts::kTokens;
constexpr int kUpCols = ts::kCols;        // h columns of a gate/up tile (of a CTA pair)
constexpr int kDownCols = 2 * ts::kCols;
// Expert ids outside [0, E) (only possible with caller-supplied routing) are left out of the
// permutation and reported through the error word; they contribute nothing to the output.
constexpr int kErrBadExpert = 21;

struct Plan {
  int4* tiles;     // {expert (-1: shared), first row, rows, 1: matrices off whole rows}: the shared expert's tiles first
  int* n_tiles;
  int* start;      // expert -> its first sorted row
  int* at;         // (token, slot) -> place among its expert's rows, -1: expert id out of range
  int* inv;        // (token, slot) -> sorted row, -1: expert id out of range (from the gather on)
  __half* row_w;   // sorted row -> routing weight (from the gather on)
};

constexpr int kPlanThreads = 1024;

// One CTA; it reads the expert ids once, four trips of loads in flight, and leaves everything per row to the gather
// (with that here, 12000 rows took 28 us).  Lanes with the same expert claim their rows together: one shared-memory
// atomic per warp and expert.
__global__ void __launch_bounds__(kPlanThreads) prefill_plan_kernel(Plan pl, const long long* __restrict__ idx,
                                                                    const int* __restrict__ nbits, Offsets off, int R, int E, int tokens,
                                                                    bool shared, int* err) {
  __shared__ int odd[256], count[256], start[256], first_tile[256], cost[256], order[256];
  const int tid = threadIdx.x, lane = tid & 31;
  int width = 0;
  for (int e = tid; e < E; e += kPlanThreads) {
    count[e] = 0;
    width = nbits[e];
    odd[e] = off_boundary(off, e) ? 1 : 0;
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid == 0) *err = 0;
  __syncthreads();
  constexpr int kAhead = 4;
#pragma unroll 1
  for (int p0 = tid; p0 < R + tid; p0 += kAhead * kPlanThreads) {
    long long id[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) id[u] = p0 + u * kPlanThreads < R ? idx[p0 + u * kPlanThreads] : 0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int p = p0 + u * kPlanThreads;
      int e = -1;
      if (p < R) {
        if (id[u] >= 0 && id[u] < E) e = static_cast<int>(id[u]);
        else atomicExch(err, kErrBadExpert);
      }
      const unsigned peers = __match_any_sync(0xffffffffu, e);
      int at = 0;
      if (e >= 0 && lane == __ffs(peers) - 1) at = atomicAdd(&count[e], __popc(peers));
      at = __shfl_sync(0xffffffffu, at, __ffs(peers) - 1);
      if (p < R) pl.at[p] = e >= 0 ? at + __popc(peers & ((1u << lane) - 1u)) : -1;
    }
  }
  __syncthreads();
  // Experts with the longest tiles first: cycles of 128 k by the tile's MMAs, or by the de-quantisation, as they were when the producers
  // waited for their words.  Since the words have a ring of their own they are 590 to 770 at 1, 2 and 4 bits, 850 to 1030 at 3 and
  // 880 to 1025 for 225 to 256 rows of any width, so 3-bit tiles of few rows stand too far ahead; not fitted anew.  (By bit width alone
  // the pairs' shares differed by a quarter where 400 tokens meet 32 experts unevenly.)  E <= 256: one expert a thread.
  if (tid < E) {
    const int n = count[tid], nt = (n + kTile - 1) / kTile, rows = nt ? (n + nt - 1) / nt : 0;
    const int mma = 4 * rows + 76, words = width == 3 ? 1700 : (width == 4 ? 1050 : (width == 2 ? 900 : 850));
    cost[tid] = n ? (mma > words ? mma : words) : 0;
  }
  __syncthreads();
  if (tid < E) {
    int r = 0;
    const int mine = cost[tid];
#pragma unroll 8
    for (int o = 0; o < E; ++o) r += cost[o] > mine || (cost[o] == mine && o < tid) ? 1 : 0;
    order[r] = tid;
  }
  __syncthreads();
  const int sh_tiles = shared ? (tokens + kTile - 1) / kTile : 0;
  if (tid < 32) {  // scan of rows and tiles over the experts
    int row = 0, tile = sh_tiles;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane < E ? order[e0 + lane] : -1;
      const int n = e >= 0 ? count[e] : 0, nt = (n + kTile - 1) / kTile;
      int sr = n, stl = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, sr, o), b = __shfl_up_sync(0xffffffffu, stl, o);
        if (lane >= o) { sr += a; stl += b; }
      }
      if (e >= 0) {
        start[e] = row + sr - n;
        pl.start[e] = start[e];
        first_tile[e] = tile + stl - nt;
      }
      row += __shfl_sync(0xffffffffu, sr, 31);
      tile += __shfl_sync(0xffffffffu, stl, 31);
    }
    if (lane == 0) *pl.n_tiles = tile;
  }
  __syncthreads();
  // an expert's tiles are of even size, in whole blocks of 16 rows
  for (int e = tid >> 5; e < E; e += kPlanThreads / 32) {
    const int n = count[e], nt = (n + kTile - 1) / kTile, blocks = (n + 15) / 16;
    for (int t = lane; t < nt; t += 32) {
      const int lo = 16 * (blocks * t / nt), hi = min(n, 16 * (blocks * (t + 1) / nt));
      pl.tiles[first_tile[e] + t] = make_int4(e, start[e] + lo, hi - lo, odd[e]);
    }
  }
  for (int i = tid; i < sh_tiles; i += kPlanThreads)
    pl.tiles[i] = make_int4(-1, R + i * kTile, min(kTile, tokens - i * kTile), 0);
}

// The sorted rows of a token's experts, and its row of the shared expert, <- its activation in fp16 (bf16 activations
// are converted here), k in the order in which a packed word's codes become MMA operands: code q next to code
// q + eps / 2; 3-bit words keep the natural order.  A thread handles 32 k of a token for all of them.
template <typename T>
__global__ void __launch_bounds__(128) prefill_gather_kernel(Plan pl, const T* __restrict__ x, const long long* __restrict__ idx,
                                                             const T* __restrict__ w, const int* __restrict__ nbits,
                                                             __half* __restrict__ xs, int tokens, int A, int D, int shared_bits) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int per_row = D / 32;
  const int i = blockIdx.x * 128 + threadIdx.x;
  const int tok = i / per_row, c = i - tok * per_row;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tok >= tokens) return;
  const uint4* s = reinterpret_cast<const uint4*>(x + static_cast<size_t>(tok) * D + 32 * c);
  __half h[32];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 v = s[j];
    const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k) h[8 * j + k] = __float2half_rn(ts::as_float<T>(e[k]));
  }
  auto put = [&](int row, auto EPS) {
    constexpr int E = decltype(EPS)::value;
    __half o[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int q = k / E, j = k % E;
      o[q * E + 2 * (j % (E / 2)) + j / (E / 2)] = h[k];
    }
    __half* d = xs + static_cast<size_t>(row) * D + 32 * c;
    const uint32_t* v = reinterpret_cast<const uint32_t*>(o);
#pragma unroll
    for (int j = 0; j < 2; ++j)  // whole 32-byte sectors
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(d + 16 * j), "r"(v[8 * j]), "r"(v[8 * j + 1]),
                   "r"(v[8 * j + 2]), "r"(v[8 * j + 3]), "r"(v[8 * j + 4]), "r"(v[8 * j + 5]), "r"(v[8 * j + 6]), "r"(v[8 * j + 7])
                   : "memory");
  };
  const int R = tokens * A;
  int rows[kMaxSlots], bits[kMaxSlots];
#pragma unroll
  for (int a = 0; a < kMaxSlots; ++a) {  // all of a token's loads in flight
    rows[a] = -1;
    if (a < A) {
      const int at = pl.at[tok * A + a];
      const int e = at < 0 ? 0 : static_cast<int>(idx[tok * A + a]);
      if (at >= 0) rows[a] = pl.start[e] + at;
      bits[a] = clamp_bits(nbits[e]);
    }
  }
#pragma unroll
  for (int a = 0; a < kMaxSlots; ++a) {
    if (a >= A) break;
    if (c == 0) pl.inv[tok * A + a] = rows[a];
    if (rows[a] < 0) continue;
    if (c == 0) pl.row_w[rows[a]] = __float2half_rn(ts::as_float<T>(w[tok * A + a]));
    if (bits[a] == 1) put(rows[a], std::integral_constant<int, 32>{});
    else if (bits[a] == 2) put(rows[a], std::integral_constant<int, 16>{});
    else if (bits[a] == 4) put(rows[a], std::integral_constant<int, 8>{});
    else put(rows[a], std::integral_constant<int, 2>{});
  }
  if (shared_bits == 1) put(R + tok, std::integral_constant<int, 32>{});
  else if (shared_bits == 2) put(R + tok, std::integral_constant<int, 16>{});
  else if (shared_bits == 4) put(R + tok, std::integral_constant<int, 8>{});
  else if (shared_bits) put(R + tok, std::integral_constant<int, 2>{});
}

// out[t] = contributions of the token's experts added in increasing expert id, each addition
// rounded to the activation dtype (index_add_ in the loop of moe_block.py:191-195), then the
// shared-expert output (moe_block.py:483).  A thread takes eight columns: one 16-byte load per expert row,
// all of them in flight before the first addition.
template <typename T>
__global__ void __launch_bounds__(128) prefill_combine_kernel(const int* __restrict__ inv, const long long* __restrict__ idx,
                                                              const __half* __restrict__ ys, int shared_row0, T* __restrict__ out,
                                                              int A, int D) {
  __shared__ int rows[kMaxSlots + 1];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int t = blockIdx.x;
  if (threadIdx.x < A) {  // rank of the slot by (expert id, slot)
    const int a = threadIdx.x;
    const long long e = idx[static_cast<size_t>(t) * A + a];
    int rank = 0;
    for (int b = 0; b < A; ++b) {
      const long long o = idx[static_cast<size_t>(t) * A + b];
      rank += (o < e || (o == e && b < a)) ? 1 : 0;
    }
    rows[rank] = inv[static_cast<size_t>(t) * A + a];
  }
  if (threadIdx.x == 0) rows[A] = shared_row0 >= 0 ? shared_row0 + t : -1;
  __syncthreads();
  for (int i = threadIdx.x; i < D / 8; i += blockDim.x) {
    uint4 v[kMaxSlots + 1];
#pragma unroll
    for (int a = 0; a <= kMaxSlots; ++a)
      if (a <= A && rows[a] >= 0) v[a] = reinterpret_cast<const uint4*>(ys + static_cast<size_t>(rows[a]) * D)[i];
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
#pragma unroll
    for (int a = 0; a <= kMaxSlots; ++a)
      if (a <= A && rows[a] >= 0) {
        const __half* h = reinterpret_cast<const __half*>(&v[a]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float c = ts::as_float<T>(ts::as_act<T>(__half2float(h[k])));
          acc[k] = ts::as_float<T>(ts::as_act<T>(acc[k] + c));
        }
      }
    uint4 o;
    T* q = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = ts::as_act<T>(acc[k]);
    reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * D)[i] = o;
  }
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

struct Scratch {
  Plan plan;
  int* err;
  __half* xs;   // [R + T, D]
  __half* h;    // [R, F]
  __half* hs;   // [T, SF]
  __half* ys;   // [R + T, D]
  char* few;    // scratch of the few-row path (shares the bytes behind the error word)
  int max_tiles;
};

// The gather stores 32 bytes at a time, callers align their scratch to 16: the pieces start at the next multiple of 32.
constexpr size_t kAlign = 32, kSlack = kAlign - 16;

size_t layout(const gemq_moe_layer_t* L, int tokens, Scratch* S, char* base) {
  if (base) base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(base) + kAlign - 1) / kAlign * kAlign);
  const size_t R = static_cast<size_t>(tokens) * L->top_k, SF = L->shared_ffn;
  const size_t rows = R + (SF ? tokens : 0);
  const size_t tiles = R / kTile + (R < static_cast<size_t>(L->n_experts) ? R : L->n_experts) + (SF ? cdiv(tokens, kTile) : 0);
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off += up256(bytes); return base ? base + o : nullptr; };
  char* er = take(2 * sizeof(int));
  const size_t few_at = off;
  char* tl = take(sizeof(int4) * tiles);
  char* starts = take(sizeof(int) * L->n_experts);
  char* at = take(sizeof(int) * R);
  char* inv = take(sizeof(int) * R);
  char* rw = take(sizeof(__half) * R);
  char* xs = take(2 * rows * L->hidden);
  char* h = take(2 * R * L->ffn);
  char* hs = take(2 * static_cast<size_t>(tokens) * SF);
  char* ys = take(2 * rows * L->hidden);
  if (S) {
    S->err = reinterpret_cast<int*>(er);
    S->plan.n_tiles = S->err + 1;
    S->plan.tiles = reinterpret_cast<int4*>(tl);
    S->plan.start = reinterpret_cast<int*>(starts);
    S->plan.at = reinterpret_cast<int*>(at);
    S->plan.inv = reinterpret_cast<int*>(inv);
    S->plan.row_w = reinterpret_cast<__half*>(rw);
    S->xs = reinterpret_cast<__half*>(xs);
    S->h = reinterpret_cast<__half*>(h);
    S->hs = reinterpret_cast<__half*>(hs);
    S->ys = reinterpret_cast<__half*>(ys);
    S->few = base ? base + few_at : nullptr;
    S->max_tiles = static_cast<int>(tiles);
  }
  if (few::moe_few_rows_ok(L, tokens)) {
    const size_t n = few_at + few::moe_few_rows_bytes(L, tokens);
    off = n > off ? n : off;
  }
  return off + kSlack;
}

void fill(ts::Family& F, int m, const gemq_stacked_t& W) {
  F.wq[m] = reinterpret_cast<const uint32_t*>(W.wq);
  F.scales[m] = static_cast<const __half*>(W.scales);
  F.zeros[m] = static_cast<const __half*>(W.zeros);
  F.zs_strides[m] = W.zs_strides;
}
void fill(ts::Family& F, int m, const gemq_single_t& W) {
  F.wq[m] = reinterpret_cast<const uint32_t*>(W.wq);
  F.scales[m] = static_cast<const __half*>(W.scales);
  F.zeros[m] = static_cast<const __half*>(W.zeros);
}

template <typename... P, typename... A>
bool launch_pdl(void (*kernel)(P...), dim3 grid, int threads, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}

int rows_of(int K, int bits) { return bits == 3 ? cdiv(K, 10) : K * bits / 32; }

bool shape_ok(int N, int K, int G) { return N % 128 == 0 && K % ts::kBK == 0 && G % ts::kBK == 0 && K % G == 0; }

template <typename T>
int run(const gemq_moe_layer_t* L, const Scratch& S, const void* x, void* out, const long long* idx, const void* w, int tokens,
        cudaStream_t st) {
  const int D = L->hidden, F = L->ffn, A = L->top_k, E = L->n_experts, SF = L->shared_ffn, R = tokens * A;
  const int sh_tiles = SF ? cdiv(tokens, kTile) : 0;
  const int* nbits = static_cast<const int*>(L->w1.nbits);
  const Offsets off = expert_offsets(L);
  bool ok = launch_pdl(prefill_plan_kernel, dim3(1), kPlanThreads, st, S.plan, idx, nbits, off, R, E, tokens, SF > 0, S.err);
  const size_t items = static_cast<size_t>(tokens) * (D / 32);
  ok = ok && launch_pdl(prefill_gather_kernel<T>, dim3(static_cast<unsigned>((items + 127) / 128)), 128, st, S.plan,
                        static_cast<const T*>(x), idx, static_cast<const T*>(w), nbits, S.xs, tokens, A, D,
                        SF ? clamp_bits(L->s1.nbits) : 0);
  if (!ok) return GEMQ_ERR_LAUNCH;

  ts::Params U = {};
  if (!ts::activation_maps(U.b_map[0], S.xs, D, R)) return GEMQ_ERR_LAUNCH;
  fill(U.fam[0], 0, L->w1);
  fill(U.fam[0], 1, L->w3);
  U.fam[0].nbits = L->w1.nbits; U.fam[0].wq_strides = L->w1.wq_strides; U.fam[0].out_nbits = L->w2.nbits;
  U.fam[0].N = F; U.fam[0].K = D; U.fam[0].G = L->group_size; U.fam[0].col_tiles = cdiv(F, kUpCols); U.fam[0].out = S.h;
  U.tiles = S.plan.tiles; U.n_tiles = S.plan.n_tiles; U.shared_tiles = sh_tiles; U.err = S.err;
  if (SF) {
    if (!ts::activation_maps(U.b_map[1], S.xs + static_cast<size_t>(R) * D, D, tokens))
      return GEMQ_ERR_LAUNCH;
    fill(U.fam[1], 0, L->s1);
    fill(U.fam[1], 1, L->s3);
    U.fam[1].bits = L->s1.nbits; U.fam[1].out_bits = L->s2.nbits;
    U.fam[1].N = SF; U.fam[1].K = D; U.fam[1].G = L->s1.group_size; U.fam[1].col_tiles = cdiv(SF, kUpCols);
    U.fam[1].out = S.hs; U.fam[1].row0 = R;
  }
  const gemq_stacked_t* const up[2] = {&L->w1, &L->w3};
  const gemq_single_t* const sup[2] = {&L->s1, &L->s3};
  const int sb = clamp_bits(L->s1.nbits), sb2 = clamp_bits(L->s2.nbits);  // as the tiles look the maps up
  U.staged = 1;
  for (int m = 0; m < 2 && U.staged; ++m)
    U.staged = ts::word_maps(U.w_map[0][m], up[m]->wq, up[m]->scales, up[m]->zeros, F, up[m]->wq_rows, L->group_size, 0, kUpCols / 2) &&
               (!SF || ts::word_maps(U.w_map[1][m], sup[m]->wq, sup[m]->scales, sup[m]->zeros, SF, rows_of(D, sb), L->s1.group_size,
                                     sb, kUpCols / 2));
  const int routed_tiles = S.max_tiles - sh_tiles;
  if (int rc = ts::launch_up(U, routed_tiles * cdiv(F, kUpCols) + sh_tiles * cdiv(SF, kUpCols), st)) return rc;

  const int ct = cdiv(D, kDownCols);
  ts::Params Q = {};
  if (!ts::activation_maps(Q.b_map[0], S.h, F, R)) return GEMQ_ERR_LAUNCH;
  fill(Q.fam[0], 0, L->w2);
  Q.fam[0].nbits = L->w2.nbits; Q.fam[0].wq_strides = L->w2.wq_strides;
  Q.fam[0].N = D; Q.fam[0].K = F; Q.fam[0].G = L->group_size; Q.fam[0].col_tiles = ct; Q.fam[0].out = S.ys;
  Q.tiles = S.plan.tiles; Q.n_tiles = S.plan.n_tiles; Q.shared_tiles = sh_tiles; Q.row_w = S.plan.row_w; Q.err = S.err;
  if (SF) {
    if (!ts::activation_maps(Q.b_map[1], S.hs, SF, tokens)) return GEMQ_ERR_LAUNCH;
    fill(Q.fam[1], 0, L->s2);
    Q.fam[1].bits = L->s2.nbits;
    Q.fam[1].N = D; Q.fam[1].K = SF; Q.fam[1].G = L->s2.group_size; Q.fam[1].col_tiles = ct;
    Q.fam[1].out = S.ys + static_cast<size_t>(R) * D; Q.fam[1].row0 = R;
  }
  Q.staged = ts::word_maps(Q.w_map[0][0], L->w2.wq, L->w2.scales, L->w2.zeros, D, L->w2.wq_rows, L->group_size, 0, ts::kCols) &&
             (!SF || ts::word_maps(Q.w_map[1][0], L->s2.wq, L->s2.scales, L->s2.zeros, D, rows_of(SF, sb2), L->s2.group_size, sb2,
                                   ts::kCols));
  if (int rc = ts::launch_down(Q, S.max_tiles * ct, st)) return rc;
  ok = launch_pdl(prefill_combine_kernel<T>, dim3(tokens), 128, st, static_cast<const int*>(S.plan.inv), idx,
                  static_cast<const __half*>(S.ys), SF ? R : -1, static_cast<T*>(out), A, D);
  return ok ? launch_status() : GEMQ_ERR_LAUNCH;
}

}  // namespace
}  // namespace gemq

using namespace gemq;

extern "C" size_t gemq_moe_prefill_scratch_bytes(const gemq_moe_layer_t* L, int tokens) {
  if (!L || tokens <= 0 || L->top_k <= 0 || L->n_experts <= 0) return 0;
  return layout(L, tokens, nullptr, nullptr);
}

extern "C" int gemq_moe_prefill(const gemq_moe_layer_t* L, const void* x, void* out, int64_t* idx, void* w,
                                void* logits, int tokens, int do_route, int route_mode, int x_is_bf16,
                                void* scratch, size_t scratch_bytes, gemq_stream_t stream) {
  if (!L || !x || !out || !idx || !w || !scratch || tokens <= 0) return GEMQ_ERR_BAD_ARG;
  const int D = L->hidden, F = L->ffn, A = L->top_k, E = L->n_experts, SF = L->shared_ffn, G = L->group_size;
  if (A > kMaxSlots || E > 256) return GEMQ_ERR_BAD_SHAPE;
  if (!shape_ok(F, D, G) || !shape_ok(D, F, G)) return GEMQ_ERR_BAD_SHAPE;
  if (SF && (!shape_ok(SF, D, L->s1.group_size) || !shape_ok(D, SF, L->s2.group_size))) return GEMQ_ERR_BAD_SHAPE;
  if (!aligned16(scratch) || !aligned16(x) || !aligned16(out)) return GEMQ_ERR_ALIGN;
  Scratch S;
  if (layout(L, tokens, &S, static_cast<char*>(scratch)) > scratch_bytes) return GEMQ_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool bf = x_is_bf16 != 0;
  if (do_route) {
    const int rc = route_tokens(x, L->gate, true, tokens, D, E, A, route_mode, L->renorm, bf, idx, w, logits, do_route == 2, st);
    if (rc) return rc;
  }
  const long long* ids = reinterpret_cast<const long long*>(idx);
  if (few::moe_few_rows_ok(L, tokens)) return few::moe_few_rows(L, x, out, ids, w, tokens, bf, S.few, S.err, st);
  return bf ? run<__nv_bfloat16>(L, S, x, out, ids, w, tokens, st) : run<__half>(L, S, x, out, ids, w, tokens, st);
}

// Error word of the last gemq_moe_prefill on this scratch (0 = no wait expired); device pointer.
extern "C" const int32_t* gemq_moe_prefill_error_word(const gemq_moe_layer_t* L, int tokens, void* scratch) {
  if (!L || !scratch || tokens <= 0) return nullptr;
  Scratch S;
  layout(L, tokens, &S, static_cast<char*>(scratch));
  return S.err;
}
