// One token of a MoE layer in two launches behind the router (gemq/inference/moe_block.py:200-235, :488-531), on the
// few-row core (few_rows.cuh).
//
//   up     a CTA takes 32 gate and the same 32 up columns of one slot over the whole reduction length, split over its
//          four consumer warps: h = silu(x1) * x3 needs no other CTA
//   down   a CTA takes 64 columns of one slot and a part of its h; the parts and the slots of a column tile are one
//          cluster, whose first CTA adds them and applies the routing weights
//
// What bounds it.  In a layer of small experts the starts: three launches of 2 us, the expert ids, then the table
// (1.6 us up, 3.5 down) with the first weights travelling next to it.  One persistent kernel for both phases
// (decode_fused.cu) needs every CTA's sums to meet in global memory between them: arrival counters, fences and flags,
// 10 us from the last weight of the first phase to the first product of the second, and 7 us of routing and planning
// ahead in every CTA.  Here the tiles are complete in one CTA or one cluster: DeepSeek-V2-Lite's layer 45 -> 30 us,
// 8 experts of 2048 x 3456 27 -> 19.  In a layer of large experts the products (475 cycles per 64 columns and group on
// a sub-partition, 3 bits twice that) on CTAs that start and end separately: two of 4096 x 14336 take 62 us here and
// 54 there, two of 4096 x 7168 40 and 41; moe_one_ok draws the line between.
//
// h stays fp32.  Its table has two rows, fp16 values and what they lack: MMA columns that one token leaves idle.
#include "few_table.cuh"

namespace gemq {
namespace few {

constexpr int kOneMaxE = 256;
constexpr int kErrOneExpert = 7, kErrOneWait = 33;

struct alignas(64) OneParams {
  CUtensorMap wmap[4];        // up: gate, up, shared gate, shared up (one strip a box); down: experts, shared (two strips)
  const __half* sc[4];
  const __half* zr[4];
  const int* nbits;           // of the launch's matrices, per expert
  const int* wqs;
  const int* zss[2];          // nullptr: expert * groups * N
  int sbits;
  const long long* idx;       // [A]
  const __half* w;            // [A]
  const void* x;              // up: fp16 [K]; down: fp32, slot after slot
  float* h;                   // up
  __half* out;                // down
  int* counters;              // error and wait limit words
  int A, S, E;
  int N[2], K[2];             // routed, shared
  int splits, ring, tab_bytes;
};

struct OneShared {
  unsigned long long full[kMaxRing], empty[kMaxRing];
  alignas(16) unsigned char zero[16];
  int lim;
  int nbits[kOneMaxE], wqs[kOneMaxE], zs[2][kOneMaxE];
};

// Waits `lim` polls, reports when they run out, and then goes on waiting (bounded, too): copies are in flight.
__device__ __forceinline__ void one_wait(unsigned long long* bar, uint32_t parity, int lim, int* err) {
  if (lim > 0) {
    for (int i = 0; i < lim; ++i) {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
      if (ok) return;
    }
    atomicExch(err, kErrOneWait);
  }
  mbar_sleep_wait(bar, parity, err, kErrOneWait);
}

// fp32 activations as two fp16 rows, 1/2/4-bit.  A piece's eight values arrive raw where the piece of the first row
// (the first four) and of the second row (the others) will stand.
template <int B>
__device__ __forceinline__ void build_pair(unsigned char* tab, const float* x, int K, int lo, int hi, int lane) {
  using F = Fmt<B>;
  constexpr int EPS = F::kEps, QW = EPS / 8;
  const int goff = stage_pieces(B) * 64 * 2, tb = table_stage_bytes(B, 2);
  const int wr = (lane >> 2) & 3, c = lane & 3, h = lane >> 4;
  const int slot = B == 1 ? wr : (B == 2 ? wr >> 1 : 0);
  const int kl = (lo * kStageRows + 8 * (wr >> 1) + F::row(c, wr & 1)) * EPS;
  unsigned char* mine = tab + wr * QW * 2 * 64 + c * 16;
  const int ns = hi - lo;
#pragma unroll 1
  for (int sg = h; sg < ns; sg += 2) {
    const int k0 = kl + sg * kStageRows * EPS;
    const float* src = x + (k0 < K ? k0 : 0);
#pragma unroll
    for (int j = 0; j < 2 * QW; ++j)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(mine + sg * tb + j * 64)), "l"(src + 4 * j),
                   "r"(k0 < K ? 16 : 0)
                   : "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll 1
  for (int s0 = 0; s0 < ns; s0 += 2) {
    const bool on = s0 + h < ns;
    unsigned char* st = tab + (on ? s0 + h : s0) * tb;
    unsigned char* dst = st + wr * QW * 2 * 64 + c * 16;
    float xv[EPS];
    float mx = 0.f, sm = 0.f;
#pragma unroll
    for (int j = 0; j < 2 * QW; ++j) {
      const float4 v = *reinterpret_cast<const float4*>(dst + j * 64);
      xv[4 * j] = v.x; xv[4 * j + 1] = v.y; xv[4 * j + 2] = v.z; xv[4 * j + 3] = v.w;
    }
#pragma unroll
    for (int k = 0; k < EPS; ++k) { mx = fmaxf(mx, fabsf(xv[k])); sm += xv[k]; }
#pragma unroll
    for (int o = 1; o < 4 * B; o <<= 1) {
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      sm += __shfl_xor_sync(0xffffffffu, sm, o);
    }
    if (on) {
      const int ce = group_exponent(mx);
      const float f = pow2i(ce);
      if ((lane & (4 * B - 1)) == 0) {
        const float2 fs = group_pair(ce, sm);
        *reinterpret_cast<float4*>(st + goff + slot * 16) = make_float4(fs.x, fs.y, fs.x, 0.f);
      }
      // the pieces carry 2^-pos of their codes: the second row is what the first one's fp16 lacks
      float lov[EPS];
#pragma unroll
      for (int k = 0; k < EPS; ++k) {
        xv[k] *= f;
        const float hi16 = round_h(xv[k]);
        lov[k] = xv[k] - hi16;
        xv[k] = hi16;
      }
      word_pieces<B>(xv, 1.f, dst, 64 * 2);
      word_pieces<B>(lov, 1.f, dst + 64, 64 * 2);
    }
  }
}

// The same for 3 bits.
__device__ __forceinline__ void build_pair_b3(unsigned char* tab, const float* x, int K, int lo, int hi, int lane) {
  const int goff = stage_pieces(3) * 64 * 2, tb = table_stage_bytes(3, 2);
  const int ngroups = K / kGroup;
  const int g0 = 5 * (lo >> 2) + (lo & 3), ng = hi > lo ? min(ngroups, 5 * ((hi - 1) >> 2) + ((hi - 1) & 3) + 2) - g0 : 0;
  constexpr int kAhead = 4;
#pragma unroll 1
  for (int i0 = 0; i0 < ng; i0 += kAhead) {  // a warp a group
    float4 v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      v[u] = i0 + u < ng ? __ldcg(reinterpret_cast<const float4*>(x + static_cast<size_t>(g0 + i0 + u) * kGroup) + lane)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      float mx = fmaxf(fmaxf(fabsf(v[u].x), fabsf(v[u].y)), fmaxf(fabsf(v[u].z), fabsf(v[u].w)));
      float sm = (v[u].x + v[u].y) + (v[u].z + v[u].w);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sm += __shfl_xor_sync(0xffffffffu, sm, o);
      }
      if (lane == 0 && i0 + u < ng) {
        const int grp = g0 + i0 + u, i5 = grp % 5;
        int sg, slot;
        group_place(3, grp, sg, slot);
        const float2 fs = group_pair(group_exponent(mx), sm);
        const float4 q = make_float4(fs.x, fs.y, fs.x, 0.f);
        if (sg >= lo && sg < hi) *reinterpret_cast<float4*>(tab + (sg - lo) * tb + goff + slot * 16) = q;
        if (i5 >= 1 && i5 <= 3 && sg > lo) *reinterpret_cast<float4*>(tab + (sg - 1 - lo) * tb + goff + 16) = q;
      }
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < (hi - lo) * 12; i += 32) {
    const int sg = i / 12, r = i - 12 * sg, pass = r >> 2, c = r & 3;
    const PassB3 p = pass_of_b3(lo + sg, pass, c);
    const bool on = p.grp < ngroups;  // past the last group: zeros
    float v[20], l[20];
#pragma unroll
    for (int j = 0; j < 20; j += 4) {
      const float4 q = on && p.k0 + j < K ? __ldcg(reinterpret_cast<const float4*>(x + p.k0 + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[j] = q.x; v[j + 1] = q.y; v[j + 2] = q.z; v[j + 3] = q.w;
    }
    const float un = *reinterpret_cast<const float*>(tab + sg * tb + goff + p.slot * 16);  // 2^(24 - ce)
    const float f = on ? pow2i(24 - (static_cast<int>(__float_as_uint(un) >> 23) - 127)) : 0.f;
#pragma unroll
    for (int j = 0; j < 20; ++j) {
      const float s = v[j] * f;  // of the neighbouring group maybe, beyond fp16: masked below, but not as a NaN
      const float hi16 = round_h(fminf(fmaxf(s, -65504.f), 65504.f));
      l[j] = fminf(fmaxf(s - hi16, -65504.f), 65504.f);
      v[j] = hi16;
    }
    unsigned char* dst = tab + sg * tb + 3 * pass * 2 * 64 + c * 16;
    put_pass_b3(v, 1.f, p, dst, 64 * 2);
    put_pass_b3(l, 1.f, p, dst + 64, 64 * 2);
  }
}

template <int MODE, int B>
__device__ __forceinline__ void consume_one(State<1>& A, OneShared& S, const OneParams& P, unsigned char* ring, unsigned char* tab,
                                            const void* x, int K, int lo, int hi, int iters, int lim, int warp, int lane) {
  constexpr int kRows = MODE == 0 ? 1 : 2;
  if (MODE == 0) {
    const Rows R = {K, K, 1};
    if (B == 3) build_b3<__half>(R, tab, static_cast<const __half*>(x), 1, lo, hi, lane);
    else build_pow2<__half, B == 3 ? 2 : B>(R, tab, static_cast<const __half*>(x), 1, lo, hi, lane);
  } else {
    if (B == 3) build_pair_b3(tab, static_cast<const float*>(x), K, lo, hi, lane);
    else build_pair<B == 3 ? 2 : B>(tab, static_cast<const float*>(x), K, lo, hi, lane);
  }
  __syncwarp();
  const uint32_t zero = smem_u32(S.zero), tab32 = smem_u32(tab), ring32 = smem_u32(ring), none = lds32(zero);
  int slot = 0;
  uint32_t par = 0;
#pragma unroll 1
  for (int it = 0; it < iters; ++it) {
    const uint32_t st = ring32 + slot * (kWStage + kMetaStage);
    one_wait(&S.full[slot], par, lim, P.counters + kErrWord);
    if (lo + it < hi)
      stage_any<B, 1, kStrip>(A, st + warp * 2 * kStrip, tab32 + it * table_stage_bytes(B, kRows), zero, st + kWStage + warp * 1024,
                              kRows, lo + it, K / kGroup, lane);
    release_stage<1>(A, &S.empty[slot], none, lane);
    if (++slot == P.ring) { slot = 0; par ^= 1u; }
  }
}

// MODE 0: up, 1: down.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 3) few_one_kernel(const __grid_constant__ OneParams P) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ OneShared S;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int members = MODE == 0 ? 1 : P.S * P.splits;  // of the cluster
  const int rank = MODE == 0 ? 0 : static_cast<int>(blockIdx.x % members);
  const int per_slot = P.N[0] / 32, tile = static_cast<int>(blockIdx.x) / members;
  const int s = MODE == 0 ? min(tile / per_slot, P.A) : rank / P.splits;  // slot; up: the shared expert's tiles come last
  const int part = MODE == 0 ? 0 : rank % P.splits;
  const int n0 = MODE == 0 ? 32 * (tile - s * per_slot) : 64 * tile;
  const int fam = s >= P.A ? 1 : 0;
  const int N = P.N[fam], K = P.K[fam], ngroups = K / kGroup;
  // what does not depend on the kernel before: barriers, the experts' bit widths and offsets
  if (tid == 0) {
    for (int i = 0; i < kMaxRing; ++i) {
      mbar_init(&S.full[i], 1 + 32);
      mbar_init(&S.empty[i], kCons);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid >= 64 && tid < 68) reinterpret_cast<uint32_t*>(S.zero)[tid - 64] = 0u;
  for (int e = tid; e < P.E; e += kThreads) {
    S.nbits[e] = P.nbits[e];
    S.wqs[e] = P.wqs[e];
#pragma unroll
    for (int m = 0; m < 2; ++m) S.zs[m][e] = P.zss[m] ? P.zss[m][e] : 0;
  }
  pdl_launch();
  if (MODE == 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // peers have started by the wait below
  pdl_wait();
  if (tid == 0) S.lim = P.counters[kLimitWord];
  int e = 0;
  if (!fam) {
    const long long id = P.idx[s];
    e = id < 0 ? 0 : (id >= P.E ? P.E - 1 : static_cast<int>(id));
    if (id != e && tid == 0) atomicExch(P.counters + kErrWord, kErrOneExpert);
  }
  __syncthreads();
  int bits = fam ? P.sbits : S.nbits[e];
  bits = bits < 1 ? 1 : (bits > 4 ? 4 : bits);
  const int lim = S.lim;
  const int parts = P.splits * kCons;
  int iters = 0;
#pragma unroll
  for (int q = 0; q < kCons; ++q) {
    int lo, hi;
    stage_range(bits, K, part * kCons + q, parts, lo, hi);
    iters = max(iters, hi - lo);
  }
  int my_lo, my_hi;  // of the consumer warp; producer: of warp lane & 3
  stage_range(bits, K, part * kCons + (warp == kCons ? lane & 3 : warp), parts, my_lo, my_hi);
  float* red = reinterpret_cast<float*>(ring);

  if (warp == kCons) {
    const int wrow = fam ? 0 : static_cast<int>(static_cast<unsigned>(S.wqs[e]) / static_cast<unsigned>(N));
    const int gshift = bits == 3 ? 1 : (bits == 4 ? 0 : (bits == 2 ? 1 : 2));  // log2 of the groups per stage
    const int piece = lane & 3, mst = (lane >> 2) & 1, kind = (lane >> 3) & 1;
    const int m = MODE == 0 ? mst : 0;
    const size_t zoff = fam ? 0 : (P.zss[m] ? static_cast<size_t>(S.zs[m][e]) : static_cast<size_t>(e) * ngroups * N);
    const int col = n0 + (MODE == 0 ? 0 : 32 * mst) + 8 * piece;
    const int mat = MODE == 0 ? 2 * fam + m : fam;
    const __half* mbase = (kind ? P.zr[mat] : P.sc[mat]) + zoff + col;
    const uint32_t mdst = kWStage + kind * 128 + mst * 64 + piece * 16;
    int slot = 0;
    uint32_t par = 1;
    for (int it = 0; it < iters; ++it) {
      one_wait(&S.empty[slot], par, 0, P.counters + kErrWord);
      unsigned char* st = ring + slot * (kWStage + kMetaStage);
      const bool on = lane < kCons && my_lo + it < my_hi;
      const unsigned boxes = __popc(__ballot_sync(0xffffffffu, on));
      if (lane == 0) mbar_arrive_expect_tx(&S.full[slot], boxes * 2 * kStrip);
      __syncwarp();
      if (on) {
        const int row = wrow + (my_lo + it) * kStageRows;
        if (MODE == 0) {
          tma_load_strips(st + lane * 2 * kStrip, &P.wmap[2 * fam], row, n0 >> 5, &S.full[slot]);
          tma_load_strips(st + lane * 2 * kStrip + kStrip, &P.wmap[2 * fam + 1], row, n0 >> 5, &S.full[slot]);
        } else {
          tma_load_strips(st + lane * 2 * kStrip, &P.wmap[fam], row, n0 >> 5, &S.full[slot]);
        }
      }
      const uint32_t dst = smem_u32(st) + mdst;
#pragma unroll 2
      for (int i = lane >> 4; i < (kCons << gshift); i += 2) {
        const int cw = i >> gshift, gi = i & ((1 << gshift) - 1);
        const int sg = __shfl_sync(0xffffffffu, my_lo, cw) + it;
        const int end = __shfl_sync(0xffffffffu, my_hi, cw);
        const int grp = bits == 3 ? 5 * (sg >> 2) + (sg & 3) + gi : (sg << gshift) + gi;
        if (sg < end && grp < ngroups && col < N) cp_async16(dst + cw * 1024 + gi * 256, mbase + static_cast<size_t>(grp) * N);
      }
      cp_async_arrive(&S.full[slot]);
      if (++slot == P.ring) { slot = 0; par ^= 1u; }
    }
  } else {
    State<1> A;
    clear(A);
    const void* x = MODE == 0 ? P.x : static_cast<const void*>(static_cast<const float*>(P.x) + static_cast<size_t>(s) * P.K[0]);
    unsigned char* tab = ring + P.ring * (kWStage + kMetaStage) + warp * P.tab_bytes;
    if (bits == 1) consume_one<MODE, 1>(A, S, P, ring, tab, x, K, my_lo, my_hi, iters, lim, warp, lane);
    else if (bits == 2) consume_one<MODE, 2>(A, S, P, ring, tab, x, K, my_lo, my_hi, iters, lim, warp, lane);
    else if (bits == 3) consume_one<MODE, 3>(A, S, P, ring, tab, x, K, my_lo, my_hi, iters, lim, warp, lane);
    else consume_one<MODE, 4>(A, S, P, ring, tab, x, K, my_lo, my_hi, iters, lim, warp, lane);
    // the sums go over the ring: every consumer has to be done with it
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kCons) : "memory");
    if ((lane & 3) == 0) {  // MMA columns 0 and 1
      const int g = lane >> 2;
#pragma unroll
      for (int st = 0; st < 2; ++st) {
        float4 v = result4<1>(A, st, 0, 0);
        if (MODE == 1) {
          const float4 u = result4<1>(A, st, 0, 1);
          v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        *reinterpret_cast<float4*>(red + warp * 64 + 32 * st + 4 * g) = v;
      }
    }
  }
  __syncthreads();
  if (MODE == 0) {
    if (tid < 32 && n0 + tid < N) {
      float a = red[tid], b = red[32 + tid];
#pragma unroll
      for (int q = 1; q < kCons; ++q) { a += red[64 * q + tid]; b += red[64 * q + 32 + tid]; }
      P.h[static_cast<size_t>(s) * P.N[0] + n0 + tid] = silu_f32(round_h(a)) * round_h(b);
    }
    return;
  }
  // the cluster's first CTA: parts of a slot in order, slots in order
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  float* mine = reinterpret_cast<float*>(ring + P.ring * (kWStage + kMetaStage) + kCons * P.tab_bytes);  // [members][64]
  if (tid < 64) {
    float v = red[tid];
#pragma unroll
    for (int q = 1; q < kCons; ++q) v += red[64 * q + tid];
    float* dst = mine + rank * 64 + tid;
    if (rank == 0) {
      *dst = v;
    } else {
      uint32_t a;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(dst)));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank != 0 || tid >= 64 || n0 + tid >= N) return;
  float acc = 0.f, res = 0.f;
  for (int q = 0; q < P.S; ++q) {
    float v = mine[q * P.splits * 64 + tid];
    for (int r = 1; r < P.splits; ++r) v += mine[(q * P.splits + r) * 64 + tid];
    v = round_h(v);
    if (q < P.A) {
      acc = fmaf(__half2float(P.w[q]), v, acc);
      if (q == P.A - 1) res = round_h(acc);
    } else {
      res = round_h(res + v);
    }
  }
  P.out[n0 + tid] = __float2half_rn(res);
}

// Table bytes of a warp at any bit width.
static int one_table_bytes(int K, int parts, int rows) {
  int most = 0;
  for (int b = 1; b <= 4; ++b) {
    const int n = cdiv(n_stages(K, b), parts) * table_stage_bytes(b, rows);
    most = n > most ? n : most;
  }
  return (most + 127) / 128 * 128;
}

static size_t one_smem(int tab_bytes, int cluster, int ring) {
  return 1024 + static_cast<size_t>(kCons) * tab_bytes + static_cast<size_t>(cluster) * 64 * 4 + ring * static_cast<size_t>(kWStage + kMetaStage);
}

// Dynamic shared memory of a launch: 227 KB less the static part.
constexpr size_t kOneDyn = kMaxDyn - 8192;

// Ring stages: a third one where it costs no CTA of the three an SM can hold; 0: not even two fit.
static int one_ring(int tab_bytes, int cluster) {
  auto per_sm = [&](int ring) { return 227 * 1024 / (one_smem(tab_bytes, cluster, ring) + sizeof(OneShared) + 1024); };
  const bool third = per_sm(kMaxRing) >= 3 || per_sm(kMaxRing) == per_sm(2);
  if (third && one_smem(tab_bytes, cluster, kMaxRing) <= kOneDyn) return kMaxRing;
  return one_smem(tab_bytes, cluster, 2) <= kOneDyn ? 2 : 0;
}

// Shape of the two launches of a layer; `ok`: both fit.
struct OnePlan {
  int tab[2], ring[2];  // up, down
  int splits;           // of the down launch: parts of a slot
  bool ok;
};
static OnePlan one_plan(const gemq_moe_layer_t* L) {
  OnePlan p = {};
  const int D = L->hidden, F = L->ffn, SF = L->shared_ffn, S = L->top_k + (SF > 0 ? 1 : 0);
  const int most = F > SF ? F : SF, shorter = SF && SF < F ? SF : F, tiles = cdiv(D, 64), sms = sm_count();
  // as many parts as run at once (their tables decide how many CTAs an SM holds), a group a warp at least
  for (p.splits = 8 / S; p.splits > 1; --p.splits) {
    const size_t smem = one_smem(one_table_bytes(most, kCons * p.splits, 2), S * p.splits, 2) + sizeof(OneShared) + 1024;
    const int per_sm = static_cast<int>(227 * 1024 / smem);
    if (shorter >= kGroup * kCons * p.splits && tiles * S * p.splits <= (per_sm > 3 ? 3 : per_sm) * sms) break;
  }
  p.tab[0] = one_table_bytes(D, kCons, 1);
  p.tab[1] = one_table_bytes(most, kCons * p.splits, 2);
  p.ring[0] = one_ring(p.tab[0], 1);
  p.ring[1] = one_ring(p.tab[1], S * p.splits);
  p.ok = sms > 0 && p.ring[0] && p.ring[1];
  return p;
}

template <int MODE>
static int launch_one(const OneParams& P, dim3 grid, int cluster, cudaStream_t st) {
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return GEMQ_ERR_LAUNCH;
  if (!done[dev]) {
    if (cudaFuncSetAttribute(few_one_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneDyn) != cudaSuccess)
      return GEMQ_ERR_LAUNCH;
    done[dev] = true;
  }
  const size_t smem = one_smem(P.tab_bytes, cluster, P.ring);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, few_one_kernel<MODE>, P) == cudaSuccess ? GEMQ_OK : GEMQ_ERR_LAUNCH;
}

}  // namespace few

using namespace few;

// Layers this path takes: extents in whole groups, eight slots at most (the cluster), tables that leave room for a ring
// in either launch, and fewer weights than where the persistent kernel is the faster.
bool moe_one_ok(const gemq_moe_layer_t* L) {
  const int D = L->hidden, F = L->ffn, SF = L->shared_ffn, A = L->top_k, S = A + (SF > 0 ? 1 : 0);
  if (L->group_size != kGroup || D % kGroup || F % kGroup || SF % kGroup || S > 8 || L->n_experts > kOneMaxE) return false;
  if (D > 16384 || F > 32768 || SF > 32768) return false;
  if (3ll * D * (static_cast<long long>(A) * F + SF) > (256ll << 20)) return false;
  if (SF && (L->s1.group_size != kGroup || L->s3.group_size != kGroup || L->s2.group_size != kGroup)) return false;
  const void* ptrs[] = {L->w1.wq, L->w1.scales, L->w1.zeros, L->w3.wq, L->w3.scales, L->w3.zeros, L->w2.wq, L->w2.scales, L->w2.zeros};
  for (const void* p : ptrs)
    if (!p || !aligned16(p)) return false;
  const void* shared[] = {L->s1.wq, L->s1.scales, L->s1.zeros, L->s3.wq, L->s3.scales, L->s3.zeros, L->s2.wq, L->s2.scales, L->s2.zeros};
  if (SF)
    for (const void* p : shared)
      if (!p || !aligned16(p)) return false;
  return L->w1.wq_rows > 0 && L->w3.wq_rows > 0 && L->w2.wq_rows > 0 && one_plan(L).ok;
}

// One token; idx / w hold its routing (written by the launch before or older), h [S slots] fp32 scratch.
int moe_one(const gemq_moe_layer_t* L, const __half* x, __half* out, const int64_t* idx, const __half* w, int* counters, float* h,
            cudaStream_t st) {
  const int D = L->hidden, F = L->ffn, SF = L->shared_ffn, A = L->top_k, S = A + (SF > 0 ? 1 : 0);
  const OnePlan plan = one_plan(L);
  if (!plan.ok) return GEMQ_ERR_BAD_SHAPE;
  OneParams U = {};
  U.idx = reinterpret_cast<const long long*>(idx);
  U.w = w; U.counters = counters; U.h = h;
  U.A = A; U.S = S; U.E = L->n_experts;
  U.splits = 1;
  OneParams Q = U;
  bool ok = tensor_map_strips(&U.wmap[0], L->w1.wq, F, L->w1.wq_rows, 1) && tensor_map_strips(&U.wmap[1], L->w3.wq, F, L->w3.wq_rows, 1) &&
            tensor_map_strips(&Q.wmap[0], L->w2.wq, D, L->w2.wq_rows, 2);
  auto half = [](const void* p) { return static_cast<const __half*>(p); };
  U.sc[0] = half(L->w1.scales); U.zr[0] = half(L->w1.zeros);
  U.sc[1] = half(L->w3.scales); U.zr[1] = half(L->w3.zeros);
  Q.sc[0] = half(L->w2.scales); Q.zr[0] = half(L->w2.zeros);
  U.nbits = L->w1.nbits; U.wqs = L->w1.wq_strides; U.zss[0] = L->w1.zs_strides; U.zss[1] = L->w3.zs_strides;
  Q.nbits = L->w2.nbits; Q.wqs = L->w2.wq_strides; Q.zss[0] = L->w2.zs_strides;
  if (SF) {
    ok = ok && tensor_map_strips(&U.wmap[2], L->s1.wq, SF, packed_rows(D, L->s1.nbits), 1) &&
         tensor_map_strips(&U.wmap[3], L->s3.wq, SF, packed_rows(D, L->s1.nbits), 1) &&
         tensor_map_strips(&Q.wmap[1], L->s2.wq, D, packed_rows(SF, L->s1.nbits), 2);
    U.sc[2] = half(L->s1.scales); U.zr[2] = half(L->s1.zeros);
    U.sc[3] = half(L->s3.scales); U.zr[3] = half(L->s3.zeros);
    Q.sc[1] = half(L->s2.scales); Q.zr[1] = half(L->s2.zeros);
    U.sbits = Q.sbits = L->s1.nbits;
  }
  if (!ok) return GEMQ_ERR_LAUNCH;
  U.x = x;
  U.K[0] = U.K[1] = D;
  U.N[0] = F; U.N[1] = SF;
  U.tab_bytes = plan.tab[0];
  U.ring = plan.ring[0];
  if (const int rc = launch_one<0>(U, dim3(A * (F / 32) + SF / 32), 1, st)) return rc;
  Q.x = h;
  Q.out = out;
  Q.K[0] = F; Q.K[1] = SF;
  Q.N[0] = Q.N[1] = D;
  Q.splits = plan.splits;
  Q.tab_bytes = plan.tab[1];
  Q.ring = plan.ring[1];
  return launch_one<1>(Q, dim3(cdiv(D, 64) * S * plan.splits), S * plan.splits, st);
}

}  // namespace gemq
