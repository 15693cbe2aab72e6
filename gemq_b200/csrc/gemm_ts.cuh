// De-quantising GEMM on the 5th-generation tensor cores with the weights as the TMEM operand.
//
//   D[128 weight columns, tokens] += W^T[128 columns, k] (tensor memory) * X^T[k, tokens] (shared memory)
//
// What bounds it.  With activations as the row operand both operands stood in shared memory, which
// moved 1280 cycles' worth of bytes per 1024 cycles of MMAs (both operands written once, the weight tile
// read once per 128 rows), and a CTA spent 390 instructions on 64 weights: 0.6 of the tensor peak.  Here
// the producers put the de-quantised weights straight from their registers into tensor memory (tcgen05.st;
// thread = weight column = TMEM lane) and shared memory only carries the activations.  The weights are
// de-quantised exactly as the reference does, fp16(fma(q, s, z)): three instructions per two weights when
// the activations come in the order in which the codes lie in a word (no byte permutes; the kernels
// that write the activations of the MoE layers store them so), four in natural order.
//
// Two CTAs of a cluster (one per SM, persistent) work on a tile of 256 weight columns and up to 256 tokens as one
// cta_group::2 MMA: each holds 128 columns of the weights and of the fp32 result in its tensor memory and
// half of the tokens in its shared memory.  (One CTA alone on 128 columns x 256 tokens reads 64 bytes a cycle of
// activations out of shared memory and has to bring in as many: 128 bytes a cycle, all shared memory can do;
// 660 instead of 512 cycles per k-block.)  Tiles of the gate/up pass hold 64 gate and the same 64 up
// columns per CTA, 16 + 16 per warp, so that a shuffle brings them together.
//   16 producer warps  four groups that take 64-wide k-blocks in turn: packed words from shared memory (or loaded a
//                      block of the group ahead), de-quantise 64 k x 32 columns per warp, store them to the A ring;
//                      they never stop between tiles
//   1 TMA warp         per stage an activation box (32 to 128 tokens x 128 k, 128B swizzle)
//   2 word warps       packed words; scales, offsets and the next tile's description.  They run ahead of the stages in rings of
//                      their own (words asked for when the MMAs release their stage: 1100 of a block's 1950 cycles a wait;
//                      1000 rows of 4096 x 4096, 4 bits 35.3 -> 32.5 us, 509 Mixtral tokens 455 -> 408, 2000 DeepSeek-V2-Lite
//                      tokens 391 -> 343, the epilogue's part in these named there)
//   1 MMA warp         (first CTA) issues tcgen05.mma and the commits that free the ring stages
//   4 epilogue warps   round the accumulators to 16 bits into shared memory, which frees them for the next
//                      tile, then finish and store whole rows while it is computed.  Tiles of up to 128 tokens
//                      use the two halves of the accumulator columns in turn.  (With the producers doing
//                      this between tiles, a tile of 128 tokens and 64 k-blocks took 28 us, 9 of them here.)
// Every wait is bounded.
#pragma once

#include <type_traits>

#include "gemv.cuh"
#include "ptx.cuh"

namespace gemq {

// tma.cu
bool tensor_map_blocks(CUtensorMap* out, const void* base, int K, long long rows, int box_rows);

namespace ts {

constexpr int kBK = 64;            // k-block of a producer warp
constexpr int kStageK = 128;       // two of them per ring stage: a stage's waits, fences and branches cost the TMA and
                                   // the MMA warp about 300 cycles each, 64 k of a half-filled tile only 256 of MMAs
constexpr int kCols = 128;         // weight columns of a CTA = TMEM lanes
constexpr int kTokens = 256;       // most tokens of a tile
constexpr int kRowBytes = kBK * 2;
constexpr int kStages = 4;
constexpr int kProducers = 16;
constexpr int kGroups = kProducers / 4;
constexpr int kTmaWarp = kProducers, kMmaWarp = kProducers + 1, kWordWarp = kProducers + 2, kEpiWarp = kProducers + 4;
constexpr int kThreads = 32 * (kEpiWarp + 4);
constexpr int kOutPitch = kCols * 2;  // bytes of a staged row of results, its 16-byte pieces swizzled by the row
constexpr int kStageBytes = kTokens / 2 * 2 * kRowBytes;  // half of the tokens
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemA = 256;   // A ring behind the accumulators: 64 columns per stage

enum { kErrFull = 11, kErrEmpty = 13, kErrAcc = 14, kErrDrained = 15, kErrTile = 16 };
enum { kOutUp = 0,      // silu(gate) * up, fp16, stored in the order of the down projection's words
       kOutDown = 1,    // times the row's routing weight, fp16
       kOutLinear = 2,  // activation type
       kOutPartial = 3  // linear, a part of k: fp32 sums, added by linear_sum_kernel
};

// One matrix family of a launch: routed experts, or the shared expert.
struct Family {
  const uint32_t* wq[2];
  const __half* scales[2];
  const __half* zeros[2];
  const int* nbits;          // [E] or nullptr -> bits
  const int* wq_strides;     // [E] or nullptr
  const int* zs_strides[2];  // [E] or nullptr -> e * (K / G) * N
  const int* out_nbits;      // up: bit widths of the matrices that read h, or nullptr -> out_bits
  int bits, out_bits;
  int N, K, G;               // row pitch of the packed words, reduction length, group size
  int col_tiles;             // tiles (of a CTA pair) along N
  void* out;                 // row 0 of the family's output rows
  int row0;                  // first sorted row of the family: its output row 0
};

struct alignas(64) Params {
  // packed words per family, matrix and bit width (linear: [0][0][0]): boxes of a CTA's columns x the rows of 128 k
  CUtensorMap w_map[2][2][4];
  // activations per family as (64 k, rows, K / 64): boxes of 32, 64, 96, 128 rows x 128 k, 128B swizzle
  CUtensorMap b_map[2][4];
  Family fam[2];
  const int4* tiles;       // {expert (-1: shared), first row, rows, 1: offsets not staged}, shared tiles first; nullptr: linear
  const int* n_tiles;
  int shared_tiles;
  const long long* expert; // linear: expert id read on the device, or nullptr -> 0
  int rows, tile_rows;     // linear: rows, tokens per tile
  int splits, split_kb;    // linear: parts of k, k-blocks of a part (even)
  float* partial;          // [splits][rows][N]
  const __half* row_w;     // down: routing weight per sorted row
  const void* bias;        // linear
  int* err;
  int staged;              // the words come through shared memory
};

// Packed words, scales and offsets of 128 k have a ring of their own: a place is asked for again as soon as the producers are
// done with its words, not when the MMAs release the stage: about three stages before the next ones are wanted.
constexpr int kWordBytes = 16 * kCols * 4;  // 4 bits
// Packed rows of 128 k; 3-bit rows from the one in which the first code lies.
__host__ __device__ constexpr int stage_rows(int bits) { return bits == 3 ? 14 : 4 * bits; }

// A tile of the launch, as one CTA of the pair sees it.
struct alignas(16) Tile {
  int fam, expert, row0, rows, col0;
  int kb0, kbn, part;      // its k-blocks, its part of k
  int bits, out_bits;      // of its matrices, of the matrix that reads h
  int odd;                 // its matrices do not begin at whole rows and 16-byte boundaries
  int woff, wrow;          // where its packed words begin: words, rows
  long long zoff[2];       // ... its scales and offsets
  // tokens of the MMA (32, 64, ..), of which each CTA brings half
  __device__ __forceinline__ int n() const { return (rows + 31) & ~31; }
  // first accumulator column of the CTA's tile number j
  __device__ __forceinline__ int acc(uint32_t j) const { return rows <= kTokens / 2 ? static_cast<int>(j & 1) * (kTokens / 2) : 0; }
};
constexpr int kTileSlots = 8;

struct Smem {
  alignas(1024) unsigned char b[kStages][kStageBytes];
  alignas(16) unsigned char out[kTokens * kOutPitch];  // accumulators rounded to 16 bits
  alignas(128) unsigned char packed[kStages][kWordBytes];
  alignas(16) unsigned char scales[kStages][kCols * 4];  // of the stage's group: [matrix][scales, offsets][columns]
  alignas(8) unsigned long long full[kStages], empty[kStages], words[kStages], freed[kStages];
  unsigned long long acc_full[2], drained[2];  // by the tile's parity
  unsigned long long tile_full[kTileSlots], tile_free[kTileSlots];
  Tile tiles[kTileSlots];
  uint32_t tmem_base;
};

__device__ __forceinline__ bool elect_one() {
  uint32_t on;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(on));
  return on != 0;
}

// ---- tcgen05 forms used here --------------------------------------------------------------------
// D[tmem] (+)= A[tmem] * B[smem] over the CTA pair; issued by one thread of the first CTA.
__device__ __forceinline__ void umma_ts_f16(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 32 lanes x 32 columns from registers: thread i writes lane (base + i).
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- the CTA pair --------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The first CTA's copy of a barrier, as a cluster address.
__device__ __forceinline__ uint32_t first_cta(const unsigned long long* bar) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(bar)));
  return a;
}
// What is handed over lies in tensor memory and is complete (tcgen05.wait) before this: a release at cluster
// scope would also wait for the packed words in flight, 1500 cycles per k-block.
__device__ __forceinline__ void arrive_at(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Arrive at the barrier of both CTAs once the pair's MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(static_cast<unsigned short>(3))
               : "memory");
}
// Box of rows x two 64-wide k-blocks into this CTA's shared memory; its bytes count on a barrier of the first CTA (cluster address).
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* map, int row, int block, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(row), "r"(block), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- de-quantisation -----------------------------------------------------------------------------
template <bool BF16>
__device__ __forceinline__ uint32_t act2(__half2 v) {
  if (BF16) {
    const float2 f = __half22float2(v);
    const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&b);
  }
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ __half2 h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }

// W^T[k, n] = fp16(fma(fp16(q), s, z)) (gemq/triton_kernels/utils.py:206-210), two weights at a time: the
// masked word holds one code in each half, `pos` bits up; under the exponent of 2^(10 - pos) the code counts in
// units of one, the half reads 2^(10 - pos) + q and one exact subtraction leaves q.  The exponents are kept in
// registers, so that masking and setting the exponent is one instruction (as literals they are two): five
// positions at most, the word is shifted for the others.
template <int B>
struct Exps {
  static constexpr int kPos = B == 1 ? 5 : 10 / B;
  uint32_t e[kPos];
  __device__ __forceinline__ Exps() {
#pragma unroll
    for (int j = 0; j < kPos; ++j) {
      e[j] = (0x6400u - (static_cast<uint32_t>(B * j) << 10)) * 0x00010001u;
      asm volatile("" : "+r"(e[j]));  // not a literal for the compiler
    }
  }
  // code j of the two halves of w
  template <int J>
  __device__ __forceinline__ __half2 weights(uint32_t w, __half2 s2, __half2 z2) const {
    constexpr uint32_t MASK = (((1u << B) - 1u) * 0x00010001u) << (B * J);
    uint32_t v;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(w), "n"(MASK), "r"(e[J]));  // (w & MASK) | exponent
    return __hfma2(__hsub2(h2(v), __float2half2_rn(static_cast<float>(1 << (10 - B * J)))), s2, z2);
  }
};

// Codes Q and Q + eps / 2 of a packed word.
template <int B, int Q>
__device__ __forceinline__ __half2 word_pair(const Exps<B>& X, uint32_t w, __half2 s2, __half2 z2) {
  constexpr int NPOS = Exps<B>::kPos, JJ = Q % NPOS, SH = (Q / NPOS) * NPOS * B;
  return X.template weights<JJ>(w >> SH, s2, z2);
}

// 32 of a column's codes (B words) as 16 TMEM words.  NAT: neighbouring k share a word; else codes q and q + eps / 2 of a
// packed word do (the activations are stored in that order).
template <int B, bool BF16, bool NAT, int I, int Q>
__device__ __forceinline__ void dequant_word(const Exps<B>& X, uint32_t (&o)[16], uint32_t w, __half2 s2, __half2 z2) {
  constexpr int PAIRS = 16 / B;
  if constexpr (Q < PAIRS) {
    const __half2 a = word_pair<B, Q>(X, w, s2, z2);
    if constexpr (!NAT) {
      o[I * PAIRS + Q] = act2<BF16>(a);
      dequant_word<B, BF16, NAT, I, Q + 1>(X, o, w, s2, z2);
    } else {
      const __half2 b = word_pair<B, Q + 1>(X, w, s2, z2);
      o[I * PAIRS + Q / 2] = act2<BF16>(h2(__byte_perm(u32(a), u32(b), 0x5410)));
      o[I * PAIRS + PAIRS / 2 + Q / 2] = act2<BF16>(h2(__byte_perm(u32(a), u32(b), 0x7632)));
      dequant_word<B, BF16, NAT, I, Q + 2>(X, o, w, s2, z2);
    }
  }
}
template <int B, bool BF16, bool NAT, int I>
__device__ __forceinline__ void dequant_words(const Exps<B>& X, uint32_t (&o)[16], const uint32_t* w, __half2 s2, __half2 z2) {
  if constexpr (I < B) {
    dequant_word<B, BF16, NAT, I, 0>(X, o, w[I], s2, z2);
    dequant_words<B, BF16, NAT, I + 1>(X, o, w, s2, z2);
  }
}

// 3-bit: a 64-code window starts at an even code of its first word and spans eight words; always natural
// order.  All 40 pairs are formed, the window is the 32 from pair (k0 mod 10) / 2 on.
template <bool BF16>
__device__ __forceinline__ void dequant_b3(const Exps<3>& X, uint32_t (&pr)[40], const uint32_t* w, __half2 s2, __half2 z2) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t m = (w[i] & 0x00007fffu) | ((w[i] << 1) & 0x7fff0000u);  // codes 0..4 | 5..9
    const uint32_t mh = m >> 9;
    const uint32_t v0 = u32(X.weights<0>(m, s2, z2)), v1 = u32(X.weights<1>(m, s2, z2)), v2 = u32(X.weights<2>(m, s2, z2));
    const uint32_t v3 = u32(X.weights<0>(mh, s2, z2)), v4 = u32(X.weights<1>(mh, s2, z2));
    pr[5 * i + 0] = act2<BF16>(h2(__byte_perm(v0, v1, 0x5410)));  // codes 0, 1
    pr[5 * i + 1] = act2<BF16>(h2(__byte_perm(v2, v3, 0x5410)));  // 2, 3
    pr[5 * i + 2] = act2<BF16>(h2(__byte_perm(v4, v0, 0x7610)));  // 4, 5
    pr[5 * i + 3] = act2<BF16>(h2(__byte_perm(v1, v2, 0x7632)));  // 6, 7
    pr[5 * i + 4] = act2<BF16>(h2(__byte_perm(v3, v4, 0x7632)));  // 8, 9
  }
}

// The tiles of a launch, read from the list and the experts' tables by the second word warp of a CTA for all roles.  Each step uses
// what the one before it has loaded: three reads from L2 in a row, 1500 to 2500 cycles where every role did them for itself
// when it got to the tile, in which no MMA ran.
template <int COLS, bool LINEAR>  // COLS: columns of a CTA along N (gate/up: 64)
struct TileReader {
  const Params& P;
  const int rank;
  int n_tiles;
  Tile t;
  int4 d;                            // step 0
  int bits, out_bits, woff, zoff[2];  // step 1
  __device__ __forceinline__ TileReader(const Params& p, int r) : P(p), rank(r) { n_tiles = LINEAR ? 0 : *P.n_tiles; }
  __device__ __forceinline__ void find(int idx) {
    t = Tile{};
    if (LINEAR) {
      t.kbn = P.fam[0].K / kBK;
      if (P.splits > 1) {
        t.part = idx % P.splits;
        idx /= P.splits;
        t.kb0 = t.part * P.split_kb;
        t.kbn = min(P.split_kb, t.kbn - t.kb0);
      }
      const int ct = P.fam[0].col_tiles, mt = idx / ct;
      t.col0 = (2 * (idx - mt * ct) + rank) * COLS;
      d = make_int4(P.expert ? static_cast<int>(*P.expert) : 0, mt * P.tile_rows, min(P.tile_rows, P.rows - mt * P.tile_rows), 0);
    } else {
      const int sh = P.shared_tiles * P.fam[1].col_tiles;
      t.fam = idx < sh ? 1 : 0;
      const int i = t.fam ? idx : idx - sh, ct = P.fam[t.fam].col_tiles, mt = (t.fam ? 0 : P.shared_tiles) + i / ct;
      t.kbn = P.fam[t.fam].K / kBK;
      t.col0 = (2 * (i % ct) + rank) * COLS;
      d = make_int4(0, 0, 0, 0);
      if (mt < n_tiles) d = P.tiles[mt];
    }
  }
  __device__ __forceinline__ void look_up() {
    t.expert = d.x;
    t.row0 = d.y;
    t.rows = max(d.z, 0);
    t.odd = d.w;
    const Family& F = P.fam[t.fam];
    const int e = t.expert;
    bits = F.bits;
    out_bits = F.out_bits;
    woff = zoff[0] = zoff[1] = 0;
    if (t.rows > 0 && e >= 0) {
      if (F.nbits) bits = F.nbits[e];
      if (F.out_nbits) out_bits = F.out_nbits[e];
      if (F.wq_strides) woff = F.wq_strides[e];
#pragma unroll
      for (int m = 0; m < 2; ++m)
        if (F.zs_strides[m]) zoff[m] = F.zs_strides[m][e];
    }
  }
  __device__ __forceinline__ void finish() {
    const Family& F = P.fam[t.fam];
    t.bits = clamp_bits(bits);  // indexes the maps of packed words
    t.out_bits = clamp_bits(out_bits);
    t.woff = woff;
    t.wrow = woff ? static_cast<int>(static_cast<unsigned>(woff) / static_cast<unsigned>(F.N)) : 0;
#pragma unroll
    for (int m = 0; m < 2; ++m)
      t.zoff[m] = t.expert < 0 ? 0 : (F.zs_strides[m] || t.expert == 0 ? zoff[m] : static_cast<long long>(t.expert) * (F.K / F.G) * F.N);
  }
  // Of a linear whose words are staged: no expert, no tables, nothing to read.
  __device__ __forceinline__ void finish_plain() {
    t.row0 = d.y;
    t.rows = max(d.z, 0);
    t.bits = clamp_bits(P.fam[0].bits);
  }
  // step 0, 1, 2 of the CTA's tile j, number idx of the launch; step 2 hands it over
  __device__ __forceinline__ void step(Smem& S, int n, int idx, uint32_t j, int* err) {
    if (n == 0) find(idx);
    if (n == 1) look_up();
    if (n == 2) {
      finish();
      const uint32_t s = j % kTileSlots;
      mbar_look_wait(&S.tile_free[s], ((j / kTileSlots) & 1) ^ 1, err, kErrTile);
      if ((threadIdx.x & 31) == 0) {
        S.tiles[s] = t;
        mbar_arrive(&S.tile_full[s]);
      }
      __syncwarp();
    }
  }
};

__device__ __forceinline__ bool staged(const Params& P, const Tile& t) { return P.staged && !t.odd; }

// The launch's tiles in the CTA's order, as its tile warp leaves them; nullptr: no more.
__device__ __forceinline__ const Tile* next_tile(Smem& S, uint32_t j, int* err) {
  const uint32_t s = j % kTileSlots;
  if (!mbar_look_wait(&S.tile_full[s], (j / kTileSlots) & 1, err, kErrTile)) return nullptr;
  return S.tiles[s].rows > 0 ? &S.tiles[s] : nullptr;
}
__device__ __forceinline__ void done_tile(Smem& S, uint32_t j) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(&S.tile_free[j % kTileSlots]);
}

// What the two word warps bring into a CTA's stages of a tile: the first one the packed words as tiled copies, the second one
// the scales and offsets, 16 bytes a lane.  (Scales and offsets as bulk copies cost the issuing lane 250 to 300 cycles each,
// and a group's number by division as many: 950 cycles a stage.)
template <bool UP>
struct TileWords {
  static constexpr int kColumns = UP ? kCols / 2 : kCols;
  const CUtensorMap* map;
  const __half* sc;  // where the lane copies from
  int bits, row0, col;
  bool on;           // its columns exist
  size_t N;
  int at, per;       // stages since the group's first, of a group
  __device__ __forceinline__ void init(const Params& P, const Tile& t, int lane) {
    const Family& F = P.fam[t.fam];
    bits = t.bits;
    N = F.N;
    per = F.G / kStageK;
    col = t.col0;
    row0 = t.wrow;
    map = &P.w_map[t.fam][0][bits - 1];
    const bool second = UP && lane >= 16, offsets = UP ? (lane >> 3) & 1 : lane >= 16;
    const int c = 8 * (lane & (UP ? 7 : 15)), sb0 = t.kb0 / 2;
    on = col + c < F.N;
    at = sb0 % per;
    const size_t off = static_cast<size_t>(t.zoff[second ? 1 : 0]) + col + c + static_cast<size_t>(sb0 / per) * N;
    sc = (offsets ? (second ? F.zeros[1] : F.zeros[0]) : (second ? F.scales[1] : F.scales[0])) + off;
  }
  __device__ __forceinline__ void load_words(unsigned char* dst, unsigned long long* bar, int kb) const {
    const int k0 = kb * kBK, row = row0 + (bits == 3 ? k0 / 10 : k0 * bits / 32), bytes = stage_rows(bits) * kColumns * 4;
    mbar_arrive_expect_tx(bar, UP ? 2 * bytes : bytes);
    tma_load_2d(dst, map, col, row, bar);
    if (UP) tma_load_2d(dst + bytes, map + 4, col, row, bar);  // the second matrix's maps come behind the four of the first
  }
  __device__ __forceinline__ void load_scales(uint32_t dst) {  // stages in order
    if (on) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(sc) : "memory");
    if (++at == per) { at = 0; sc += N; }
  }
};

// ---- producer ------------------------------------------------------------------------------------
// All k-blocks of a tile; `base` = k-blocks this CTA has handled before the tile (even).  An odd number of
// blocks is followed by one of zeros: the activations of its stage end in zeros, too.
// (Out of line: inlined, the 80 registers of 24 warps spill in the k loop.  What it reads of the tile comes by value: through a
// pointer a linear's tile, which every role works out, lies in local memory: 10 rows of 512 x 576 6.1 us instead of 5.7, 1000 of
// 4096 x 4096 27.3 instead of 27.0.)
// STAGED: packed words, scales and offsets lie in the ring.
template <bool UP, bool BF16, bool NAT, int B, bool STAGED>
__device__ __noinline__ void produce(Smem& S, const Params& P, int fam, int col0, int kb0, int kbn, int first_word, long long first_scale,
                                     uint32_t base, uint32_t tmem) {
  constexpr int NW = B == 3 ? 8 : 2 * B;  // words of a 64-code window
  const Family& F = P.fam[NAT ? 0 : fam];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mi = UP ? lane >> 4 : 0;
  // columns past the end repeat the last one; their results are not stored
  const int col = UP ? col0 + 16 * (warp & 3) + (lane & 15) : min(col0 + 32 * (warp & 3) + lane, F.N - 1);
  const size_t N = F.N;
  const size_t woff = static_cast<size_t>(first_word), zoff = static_cast<size_t>(first_scale);
  const uint32_t* wp = (mi ? F.wq[1] : F.wq[0]) + woff + col;
  const __half* sp = (mi ? F.scales[1] : F.scales[0]) + zoff + col;
  const __half* zp = (mi ? F.zeros[1] : F.zeros[0]) + zoff + col;
  // Parameters used in the loop live in registers: through the reference every use is a load.
  const int G = F.G, K = F.K;
  int* const err = P.err;
  const int gshift = (G & (G - 1)) == 0 ? __ffs(G) - 1 : -1;
  int kb = static_cast<int>(((warp >> 2) + kGroups - base % kGroups) % kGroups);  // first k-block of this warp's group
  const int real = kb0 + kbn, kb1 = kb0 + ((kbn + 1) & ~1);
  base -= kb0;  // base + kb counts the blocks this CTA has handled
  kb += kb0;
  if (kb >= kb1) return;
  struct Set { uint32_t w[NW]; __half s, z; };
  Set ring[STAGED ? 1 : 2];
  const Exps<B> X;
  if (B != 3) wp += static_cast<size_t>(kb) * (2 * B) * N;
  auto fetch = [&](Set& R, int k) {  // blocks in order
    if (k >= real) {
#pragma unroll
      for (int i = 0; i < NW; ++i) R.w[i] = 0u;
      R.s = R.z = __float2half_rn(0.f);
      return;
    }
    const int k0 = k * kBK;
    const int g = gshift >= 0 ? k0 >> gshift : k0 / G;
    if (B == 3) {  // the last window of a matrix may end before its eighth word
      const int first = k0 / 10, left = (K + 9) / 10 - first;
      const uint32_t* q = wp + static_cast<size_t>(first) * N;
#pragma unroll
      for (int i = 0; i < NW; ++i) R.w[i] = q[static_cast<size_t>(min(i, left - 1)) * N];
    } else {
      const uint32_t* q = wp;
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        R.w[i] = *q;
        q += N;
      }
      wp += static_cast<size_t>(kGroups * 2 * B) * N;
    }
    R.s = sp[static_cast<size_t>(g) * N];
    R.z = zp[static_cast<size_t>(g) * N];
  };
  const uint32_t c = (base + kb) >> 1;  // groups 0 and 1 fill a stage, 2 and 3 the next
  uint32_t s = c % kStages, par = ((c / kStages) & 1) ^ 1;
  const uint32_t full0 = first_cta(&S.full[0]);
  const uint32_t dst0 = tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + kTmemA + ((base + kb) & 1) * 32;
  // STAGED
  constexpr uint32_t kPitch = UP ? kCols * 2 : kCols * 4;
  const int in_row = UP ? 16 * (warp & 3) + (lane & 15) : 32 * (warp & 3) + lane;
  const uint32_t words0 = smem_u32(S.packed[0]) + mi * stage_rows(B) * kPitch + 4 * in_row;
  const uint32_t scales0 = smem_u32(S.scales[0]) + mi * 256 + 2 * in_row;
  // The barriers of the words flip in every use of a stage, staged or not: a use and the one before it are the same warps'.
  auto words_ready = [&]() { mbar_look_wait(&S.words[s], par ^ 1u, err, kErrFull); };
  auto words_free = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&S.freed[s]);
  };
  auto stage_free = [&]() {
    if (!STAGED) {
      words_ready();
      words_free();
    }
    mbar_look_wait(&S.empty[s], par, err, kErrEmpty);
  };
  auto take = [&](Set& R) {  // whole stages: no block of zeros
    words_ready();
    const int row = B == 3 ? kb * kBK / 10 - (kb & ~1) * kBK / 10 : (kb & 1) * 2 * B;
    const uint32_t w = words0 + s * kWordBytes + row * kPitch, sc = scales0 + s * (kCols * 4);
#pragma unroll
    for (int i = 0; i < NW; ++i) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(R.w[i]) : "r"(w + i * kPitch) : "memory");
    unsigned short a, b;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(a) : "r"(sc) : "memory");
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(b) : "r"(sc + kPitch / 2) : "memory");
    R.s = __ushort_as_half(a);
    R.z = __ushort_as_half(b);
  };
  auto put = [&](const Set& cur) {
    const __half2 s2 = __half2half2(cur.s), z2 = __half2half2(cur.z);
    const uint32_t dst = dst0 + s * 64;
    if constexpr (B == 3) {
      uint32_t pr[40];
      dequant_b3<BF16>(X, pr, cur.w, s2, z2);
      stage_free();
      tc_fence_after_sync();
      switch ((kb * kBK % 10) >> 1) {  // uniform
        case 0: tmem_st32(dst, pr); break;
        case 1: tmem_st32(dst, pr + 1); break;
        case 2: tmem_st32(dst, pr + 2); break;
        case 3: tmem_st32(dst, pr + 3); break;
        default: tmem_st32(dst, pr + 4); break;
      }
    } else {
      // in two halves: 16 result registers instead of 32
      uint32_t o[16];
      dequant_words<B, BF16, NAT, 0>(X, o, cur.w, s2, z2);
      stage_free();
      tc_fence_after_sync();
      tmem_st16(dst, o);
      dequant_words<B, BF16, NAT, 0>(X, o, cur.w + B, s2, z2);
      tmem_st16(dst + 16, o);
    }
    // Behind the stores, which hold what came of the words: an arrival does not wait for the shared-memory reads ahead of it, and TMA
    // writes past them (reads that waited behind the epilogue's: the next words were there before 4 to 32 lanes had read the last row).
    if (STAGED) words_free();
    tmem_wait_st();
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) arrive_at(full0 + s * 8);
    s += kGroups / 2;
    if (s >= kStages) { s -= kStages; par ^= 1u; }
  };
  if constexpr (STAGED) {
#pragma unroll 1
    for (; kb < kb1; kb += kGroups) {
      take(ring[0]);
      put(ring[0]);
    }
  } else {
    fetch(ring[0], kb);
#pragma unroll 1
    for (;;) {
      if constexpr (B == 3) {  // one copy of the long body, the sets are moved
        if (kb + kGroups < kb1) fetch(ring[1], kb + kGroups);
        put(ring[0]);
        kb += kGroups;
        if (kb >= kb1) return;
        ring[0] = ring[1];
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (kb + kGroups < kb1) fetch(ring[u ^ 1], kb + kGroups);
          put(ring[u]);
          kb += kGroups;
          if (kb >= kb1) return;
        }
      }
    }
  }
}

template <bool UP, bool BF16, bool NAT, bool STAGED>
__device__ __forceinline__ void produce_bits(Smem& S, const Params& P, const Tile& T, uint32_t base, uint32_t tmem) {
  const int bits = T.bits;
  const long long zoff = T.zoff[UP ? (threadIdx.x >> 4) & 1 : 0];  // of the lane's matrix
  if (bits == 1) produce<UP, BF16, NAT, 1, STAGED>(S, P, T.fam, T.col0, T.kb0, T.kbn, T.woff, zoff, base, tmem);
  else if (bits == 2) produce<UP, BF16, NAT, 2, STAGED>(S, P, T.fam, T.col0, T.kb0, T.kbn, T.woff, zoff, base, tmem);
  else if (bits == 3) produce<UP, BF16, NAT, 3, STAGED>(S, P, T.fam, T.col0, T.kb0, T.kbn, T.woff, zoff, base, tmem);
  else produce<UP, BF16, NAT, 4, STAGED>(S, P, T.fam, T.col0, T.kb0, T.kbn, T.woff, zoff, base, tmem);
}
template <bool UP, bool BF16, bool NAT>
__device__ __forceinline__ void produce_any(Smem& S, const Params& P, const Tile& T, uint32_t base, uint32_t tmem) {
  if (staged(P, T)) produce_bits<UP, BF16, NAT, true>(S, P, T, base, tmem);
  else produce_bits<UP, BF16, NAT, false>(S, P, T, base, tmem);
}

// ---- epilogue --------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float as_float(T v);
template <> __device__ __forceinline__ float as_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float as_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T as_act(float v);
template <> __device__ __forceinline__ __half as_act<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 as_act<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Waits for the tensor-memory loads into r: what uses r stays behind it (the loads alone define the registers for the compiler).
template <int N>
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i])::"memory");
}
// 32 lanes x 16 columns into registers.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  tmem_wait_ld(r);
}

// 16 tokens of 16 lanes: two mma fragments (a thread has two neighbouring tokens of lanes l / 4 and l / 4 + 8) of 8 tokens each.
__device__ __forceinline__ void tmem_ld_fragments(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
template <typename T>
__device__ __forceinline__ uint32_t pack_act(uint32_t lo, uint32_t hi) {
  const T v[2] = {as_act<T>(__uint_as_float(lo)), as_act<T>(__uint_as_float(hi))};
  return *reinterpret_cast<const uint32_t*>(v);
}

// The accumulators of a warp's 32 weight columns, rounded, to rows of tokens in shared memory.  What the MMAs of the next
// tile wait for, so few instructions: fragments whose 8 x 8 blocks stmatrix transposes, per 16 tokens two loads, eight
// conversions, two stores (a column's values one by one took 16 stores of two bytes), the loads of 32 tokens in flight.
template <typename T>
__device__ __forceinline__ void drain(Smem& S, uint32_t at, int rows, int lq, int lane) {
  uint32_t dst = smem_u32(S.out) + (8 * (lane >> 4) + (lane & 7)) * kOutPitch;
  const uint32_t piece = 4 * lq + ((lane >> 3) & 1), at16[2] = {16 * (piece ^ (lane & 7)), 16 * ((piece + 2) ^ (lane & 7))};
#pragma unroll 1
  for (int c = 0; c < rows; c += 32, dst += 32 * kOutPitch) {  // the MMAs' tokens are whole blocks of 32
    uint32_t d[32];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      tmem_ld_fragments(at + c + 16 * u, d + 16 * u);
      tmem_ld_fragments(at + (16u << 16) + c + 16 * u, d + 16 * u + 8);
    }
    tmem_wait_ld(d);
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t* v = d + 16 * u + 8 * h;
        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(dst + 16 * u * kOutPitch + at16[h]),
                     "r"(pack_act<T>(v[0], v[1])), "r"(pack_act<T>(v[2], v[3])), "r"(pack_act<T>(v[4], v[5])),
                     "r"(pack_act<T>(v[6], v[7]))
                     : "memory");
      }
  }
}

// A part of k: the fp32 sums of a column, a warp's 32 columns next to each other.
__device__ __forceinline__ void drain_partial(const Params& P, const Tile& t, uint32_t at, int col) {
  const size_t pitch = P.fam[0].N;
  float* dst = P.partial + (static_cast<size_t>(t.part) * P.rows + t.row0) * pitch + col;
  const int rows = t.rows;
  const bool on = col < P.fam[0].N;
#pragma unroll 1
  for (int c = 0; c < rows; c += 16) {
    uint32_t d[16];
    tmem_ld16(at + c, d);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (on && c + i < rows) dst[static_cast<size_t>(c + i) * pitch] = __uint_as_float(d[i]);
  }
}

// 32 neighbouring h in the order of the words of a matrix with EPS codes per word.
template <int EPS>
__device__ __forceinline__ void word_order(const __half (&h)[32], uint32_t (&o)[16]) {
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int w = k / (EPS / 2), j = k % (EPS / 2);
    const __half2 v = __halves2half2(h[w * EPS + j], h[w * EPS + j + EPS / 2]);
    o[k] = *reinterpret_cast<const uint32_t*>(&v);
  }
}

// The quotient by reciprocal, good to two units of fp32's last place.  Over all finite fp16 v, after the rounding to fp16, 1 of 63488 is
// not the rounded fp64 value (3 with the division), the mean error is the same (3.74731e-5), infinities and NaN come out alike.
// The epilogue of a gate/up tile is 16 K of these per CTA: with an IEEE division and every product in fp32, its four warps took
// longer than the MMAs of a tile of 2048 k (waits of 9 to 15 thousand cycles for the accumulators against 14 thousand of MMAs).
__device__ __forceinline__ float silu_quick(float v) { return __fdividef(v, 1.0f + __expf(-v)); }

// h = F.silu(x1) * x3 on fp16 tensors, each step rounded: a thread takes 32 columns of a token (x1 and x3 of
// 16 columns each in two warps' worth of staged columns).
__device__ __forceinline__ void finish_up(const Smem& S, const Params& P, const Tile& t, int tid) {
  const Family& F = P.fam[t.fam];
  const int bits = t.out_bits;
  const size_t pitch = F.N;
  __half* const out = static_cast<__half*>(F.out) + static_cast<size_t>(t.row0 - F.row0) * pitch + t.col0;
  const int rows = t.rows;
#pragma unroll 1
  for (int i = tid; i < 2 * rows; i += 128) {
    const int grp = i >= rows ? 1 : 0, row = i - grp * rows;
    const unsigned char* src = S.out + row * kOutPitch;
    alignas(4) __half h[32];
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // eight columns each
      const int piece = 8 * grp + 4 * (q >> 1) + (q & 1);
      const uint4 g = *reinterpret_cast<const uint4*>(src + 16 * (piece ^ (row & 7)));
      const uint4 u = *reinterpret_cast<const uint4*>(src + 16 * ((piece + 2) ^ (row & 7)));
      const __half2 *gh = reinterpret_cast<const __half2*>(&g), *uh = reinterpret_cast<const __half2*>(&u);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 v = __half22float2(gh[k]);
        *reinterpret_cast<__half2*>(h + 8 * q + 2 * k) = __hmul2(__floats2half2_rn(silu_quick(v.x), silu_quick(v.y)), uh[k]);
      }
    }
    uint32_t o[16];
    if (bits == 1) word_order<32>(h, o);
    else if (bits == 2) word_order<16>(h, o);
    else if (bits == 3) word_order<2>(h, o);  // 3-bit matrices read their rows in natural order
    else word_order<8>(h, o);
    uint4* dst = reinterpret_cast<uint4*>(out + row * pitch + 32 * grp);
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
  }
}

// Eight columns of a row per thread: times the routing weight, or plus the bias.
template <int OUT, typename T>
__device__ __forceinline__ void finish_rows(const Smem& S, const Params& P, const Tile& t, int tid) {
  const Family& F = P.fam[t.fam];
  const size_t pitch = F.N;
  const int q = tid & 15, col = t.col0 + 8 * q;
  if (col >= F.N) return;  // N is a multiple of 32
  T* const out = static_cast<T*>(F.out) + static_cast<size_t>(t.row0 - F.row0) * pitch + col;
  const __half* const rw = OUT == kOutDown && t.fam == 0 ? P.row_w + t.row0 : nullptr;
  const bool has_bias = OUT == kOutLinear && P.bias != nullptr;
  uint4 bias = make_uint4(0u, 0u, 0u, 0u);
  if (has_bias) {
#pragma unroll
    for (int k = 0; k < 8; ++k) reinterpret_cast<T*>(&bias)[k] = static_cast<const T*>(P.bias)[col + k];
  }
  const int rows = t.rows;
#pragma unroll 2
  for (int row = tid >> 4; row < rows; row += 8) {
    uint4 v = *reinterpret_cast<const uint4*>(S.out + row * kOutPitch + 16 * (q ^ (row & 7)));
    T* e = reinterpret_cast<T*>(&v);
    if constexpr (OUT == kOutDown) {
      if (rw) {
        const __half2 f = __half2half2(rw[row]);
#pragma unroll
        for (int k = 0; k < 4; ++k) reinterpret_cast<__half2*>(&v)[k] = __hmul2(reinterpret_cast<__half2*>(&v)[k], f);
      }
    } else if (has_bias) {
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = as_act<T>(as_float<T>(e[k]) + as_float<T>(reinterpret_cast<const T*>(&bias)[k]));
    }
    *reinterpret_cast<uint4*>(out + row * pitch) = v;
  }
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(map)) : "memory");
}

template <int OUT, bool BF16>
__global__ void __launch_bounds__(kThreads, 1) gemm_ts_kernel(const __grid_constant__ Params P) {
  constexpr bool UP = OUT == kOutUp, LINEAR = OUT == kOutLinear || OUT == kOutPartial;
  constexpr int COLS = UP ? kCols / 2 : kCols;
  using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);  // no other shared memory: aligned like the array
  const int warp = threadIdx.x >> 5;
  const int rank = static_cast<int>(pair_rank());
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&S.full[s], 17);  // in the first CTA: two groups' warps of either CTA, the activation boxes
      mbar_init(&S.empty[s], 1);
      mbar_init(&S.words[s], 33);  // the words, the lanes that copy scales
      mbar_init(&S.freed[s], 8);   // two groups' warps
    }
    for (int j = 0; j < 2; ++j) {
      mbar_init(&S.acc_full[j], 1);
      mbar_init(&S.drained[j], 8);  // in the first CTA: the epilogue warps of both
    }
    for (int j = 0; !LINEAR && j < kTileSlots; ++j) {
      mbar_init(&S.tile_full[j], 1);
      mbar_init(&S.tile_free[j], kThreads / 32 - (rank == 0 ? 0 : 1));  // every warp; the second CTA's MMA warp has no work
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc_pair(&S.tmem_base, kTmemCols);
  // The maps are launch parameters: their first use finds them in the cache.  (A linear has one of each, and its tile at once: there
  // this gains nothing and takes 0.1 us of a short call.)
  const int lane = static_cast<int>(threadIdx.x & 31);
  if (!LINEAR && warp == kTmaWarp && lane < 4) prefetch_map(&P.b_map[0][lane]);
  if (!LINEAR && warp == kWordWarp && P.staged && lane < (UP ? 8 : 4)) prefetch_map(&P.w_map[0][lane >> 2][lane & 3]);
  tc_fence_before_sync();
  __syncthreads();
  pair_sync();
  tc_fence_after_sync();
  const uint32_t tmem = S.tmem_base;
  // Only now: a CTA of the next kernel must not take this SM's tensor memory first.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // Everything may be a result of the launch before, a linear's packed words, too (a layer packed and called at once): no
  // early look at them.  It would gain where linears follow one another with nothing in between (4096 x 1024, 2 bits,
  // 64 rows: 7.9 instead of 9.9 us; 1000 rows of 4096 x 4096, 4 bits: 30.5 instead of 31.6), behind any other kernel nothing.
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // Tiles go to the pairs back and forth: the list is sorted by falling time, so who got a long one in a round gets
  // a short one in the next.
  const int step = static_cast<int>(gridDim.x >> 1), first = static_cast<int>(blockIdx.x >> 1);
  auto tile_of = [&](int i) { return i * step + ((i & 1) ? step - 1 - first : first); };
  // The CTA's tile j.  A linear's needs no look at memory: every role works it out (through the slots, 1010 rows of 512 x 576
  // took 8.7 us instead of 7.9; with the steps that read the tables, 10 rows of 256 x 640 5.5 instead of 5.2).
  auto tile_at = [&](uint32_t j, Tile& own) -> const Tile* {
    if (!LINEAR) return next_tile(S, j, P.err);
    TileReader<COLS, LINEAR> reader(P, rank);
    reader.find(tile_of(j));
    if (P.staged) {
      reader.finish_plain();
    } else {
      reader.look_up();
      reader.finish();
    }
    own = reader.t;
    return own.rows > 0 ? &own : nullptr;
  };
  auto tile_done = [&](uint32_t j) {
    if (!LINEAR) done_tile(S, j);
  };
  Tile own;
  int* const err = P.err;
  if (warp < kProducers) {
    uint32_t base = 0;
#pragma unroll 1
    for (uint32_t j = 0; const Tile* t = tile_at(j, own); ++j) {
      produce_any<UP, BF16, LINEAR>(S, P, *t, base, tmem);
      base += (t->kbn + 1) & ~1;
      tile_done(j);
    }
  } else if (warp == kTmaWarp) {
    uint32_t c = 0;
    const uint32_t full0 = first_cta(&S.full[0]);
    for (uint32_t j = 0; const Tile* at = tile_at(j, own); ++j) {
      const Tile t = *at;
      tile_done(j);
      const Family& F = P.fam[t.fam];
      const int SB = (t.kbn + 1) / 2, half = t.n() / 2;
      const int box = (half + 31) / 32;  // in 32 rows: an odd number of 16-row blocks brings the next 16 rows, too
      const uint32_t bytes = 2 * 32 * box * kRowBytes;
      const int row = t.row0 - F.row0 + rank * half;
      const CUtensorMap* const map = &P.b_map[t.fam][box - 1];
      for (int sb = 0; sb < SB; ++sb, ++c) {
        const uint32_t s = c % kStages;
        mbar_look_wait(&S.empty[s], ((c / kStages) & 1) ^ 1, err, kErrEmpty);
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(&S.full[s], 2 * bytes);
          tma_load_pair(S.b[s], map, row, t.kb0 + 2 * sb, full0 + s * 8);
        }
        __syncwarp();
      }
    }
  } else if (warp >= kWordWarp && warp < kEpiWarp) {
    const int which = warp - kWordWarp;
    constexpr uint32_t kTilesAhead = 1;
    TileReader<COLS, LINEAR> reader(P, rank);
    if (which && !LINEAR)
      for (uint32_t j = 0; j < kTilesAhead; ++j)
        for (int n = 0; n < 3; ++n) reader.step(S, n, tile_of(j), j, err);
    uint32_t c = 0;
    for (uint32_t j = 0; const Tile* next = tile_at(j, own); ++j) {
      const Tile t = *next;
      tile_done(j);
      int step = which && !LINEAR ? 0 : 3;
      const int SB = (t.kbn + 1) / 2;
      const bool on = staged(P, t);  // the barrier's phases follow the stages, staged or not
      TileWords<UP> words;
      if (on) words.init(P, t, lane);
      for (int sb = 0; sb < SB; ++sb, ++c) {
        const uint32_t s = c % kStages;
        const int kb = t.kb0 + 2 * sb;
        mbar_look_wait(&S.freed[s], ((c / kStages) & 1) ^ 1, err, kErrEmpty);
        if (which) {
          if (on) {
            words.load_scales(smem_u32(S.scales[s]) + 16 * lane);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&S.words[s])) : "memory");
          } else {
            mbar_arrive(&S.words[s]);
          }
        }
        if (!which && elect_one()) {
          if (on) words.load_words(S.packed[s], &S.words[s], kb);
          else mbar_arrive(&S.words[s]);
        }
        __syncwarp();
        if (step < 3) reader.step(S, step++, tile_of(j + kTilesAhead), j + kTilesAhead, err);
      }
      for (; step < 3; ++step) reader.step(S, step, tile_of(j + kTilesAhead), j + kTilesAhead, err);
    }
  } else if (warp == kMmaWarp && rank == 0) {
    // The whole warp runs the loop and one elected lane issues: descriptors and addresses stay in uniform
    // registers.  (In a one-lane branch every tcgen05.mma cost 85 cycles to issue.)
    uint32_t s = 0, par = 0, j = 0;
    const Tile* next;
    bool small = true;  // the tile before fits one half of the accumulators
    const uint64_t desc0 = umma_desc_k_sw128(smem_u32(S.b[0]));
    for (; (next = tile_at(j, own)) != nullptr; ++j) {
      const Tile t = *next;
      tile_done(j);
      const int SB = (t.kbn + 1) / 2;
      const uint32_t idesc = umma_idesc_f16(BF16 ? 1 : 0, 2 * kCols, t.n());
      const uint32_t second = ((t.n() / 2 + 31) / 32 * 32 * kRowBytes) >> 4;  // distance of a stage's second k-block
      // The accumulators of the tile two back are out; with a tile over 128 tokens also those of the last.
      mbar_look_wait(&S.drained[j & 1], ((j >> 1) & 1) ^ 1, err, kErrDrained);
      const bool now_small = t.rows <= kTokens / 2;
      if (j > 0 && !(small && now_small)) mbar_look_wait(&S.drained[(j - 1) & 1], ((j - 1) >> 1) & 1, err, kErrDrained);
      small = now_small;
      const uint32_t acc = tmem + t.acc(j);
      for (int sb = 0; sb < SB; ++sb) {
        mbar_look_wait(&S.full[s], par, err, kErrFull);
        tc_fence_after_sync();
        const uint64_t bd = desc0 + s * (kStageBytes >> 4);
        const uint32_t a = tmem + kTmemA + s * 64;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kStageK / 16; ++k)
            umma_ts_f16(acc, a + k * 8, bd + (k & 3) * 2 + (k < 4 ? 0u : second), idesc, k != 0 || sb != 0);
          umma_commit_pair(&S.empty[s]);
          if (sb == SB - 1) umma_commit_pair(&S.acc_full[j & 1]);
        }
        __syncwarp();
        if (++s == kStages) { s = 0; par ^= 1u; }
      }
    }
  }
  if (warp >= kEpiWarp) {
    const int lq = warp & 3, tid = static_cast<int>(threadIdx.x) - 32 * kEpiWarp;
#pragma unroll 1
    for (uint32_t j = 0; const Tile* next = tile_at(j, own); ++j) {
      const Tile t = *next;
      tile_done(j);
      mbar_look_wait(&S.acc_full[j & 1], (j >> 1) & 1, err, kErrAcc);
      tc_fence_after_sync();
      const uint32_t at = tmem + (static_cast<uint32_t>(32 * lq) << 16) + t.acc(j);
      const int column = 32 * lq + static_cast<int>(threadIdx.x & 31);
      if (OUT == kOutPartial) drain_partial(P, t, at, t.col0 + column);
      else drain<T>(S, at, t.rows, lq, lane);
      tc_fence_before_sync();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) arrive_at(first_cta(&S.drained[j & 1]));  // a later tile's MMAs may overwrite them
      if (OUT == kOutPartial) continue;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (UP) finish_up(S, P, t, tid);
      else finish_rows<OUT, T>(S, P, t, tid);
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
  }
  __syncthreads();
  pair_sync();  // nobody touches the other's barriers or tensor memory from here on
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem, kTmemCols);
  }
}

// gemm_ts.cu: tokens of a tile and parts of k of a linear, and the time they are estimated to take
struct LinearPlan {
  int tile_rows, splits, split_kb;
  float us;
};
LinearPlan linear_plan(int M, int N, int K, int bits, bool may_split);
// What the line between the few-row kernel and the GEMM is drawn by (few_linear.cu): constants of their own.
float linear_line_us(int M, int N, int K, int bits);

// gemm_ts.cu; tiles_bound: most tiles the launch can have
int launch_up(const Params& P, int tiles_bound, cudaStream_t stream);
int launch_down(const Params& P, int tiles_bound, cudaStream_t stream);
bool activation_maps(CUtensorMap (&maps)[4], const void* x, int K, long long rows);
// Maps of a matrix's packed words (rows of N; all widths, or one) and whether words, scales and offsets can be staged: tiled copies
// and copies of 16 bytes a lane want 16-byte boundaries, a stage one group.
bool word_maps(CUtensorMap (&maps)[4], const void* wq, const void* scales, const void* zeros, int N, long long rows, int G, int bits,
               int columns);

}  // namespace ts
}  // namespace gemq
