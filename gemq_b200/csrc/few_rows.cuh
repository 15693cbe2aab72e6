// Products of a few activation rows (at most 16 per tile) with packed matrices: the streaming core
// shared by the dense linears (few_linear.cu) and the decode batches of the MoE layers (few_moe.cu).
//
// What bounds it.  Each weight is used for at most 16 rows, so the matrices have to stream at the
// memory rate and the arithmetic per weight has to stay small.  The codes are not de-quantised: an
// fp16 whose exponent field is zero is the subnormal m * 2^-24, so `word & mask` IS a pair of fp16
// operands holding two codes (times 2^pos for codes that sit `pos` bits up), and it goes straight
// into mma.sync.m16n8k16 as the A operand (16 weight columns x 16 k).  The B operand is the
// activation of eight rows, scaled per row and group by a power of two and per k by 2^-pos: exact.
// Products are summed per quantisation group in fp32; a closed group is added with its scale, the offsets
// times the groups' activation sums come in as one tf32 MMA per stage.  Per 8192 weights (64 columns, one
// group) and eight rows: 144 to 160 ANDs and shifts -- the ALU pipe takes two cycles for each -- 32 MMAs of
// eight cycles, and about 50 instructions to close the group on the otherwise idle FMA pipe.
//
// A CTA is four consumer warps of 64 columns each and one producer warp that keeps a ring of stages
// filled.  A stage is 16 packed rows: TMA boxes of 32-column strips (128B swizzle: conflict-free
// 16-byte reads), scales and offsets as cp.async, all completing on one mbarrier.  Rings in registers
// do not work: a warp has six scoreboards, so eight loads in flight serialise (3.0 against 6.2 TB/s in
// a copy-only probe).
//
// The B operands ("table") lie in shared memory in fragment order, 64 bytes per row and two k-steps;
// MMA columns past the last row read a block of zeros.
#pragma once

#include "gemv.cuh"
#include "ptx.cuh"

namespace gemq {
namespace few {

constexpr int kCons = 4;
constexpr int kThreads = 32 * (kCons + 1);
constexpr int kMaxRing = 3;
constexpr int kStageRows = 16;               // packed rows per pipeline stage
constexpr int kTileRows = 16;                // activation rows of a tile: one or two blocks of eight MMA columns
constexpr int kStrip = 2048;                 // 16 packed rows x 32 columns
constexpr int kWStage = kCons * 2 * kStrip;
constexpr int kMetaStage = kCons * 4 * 256;  // per warp and group: 64 scales, 64 offsets
constexpr int kMaxDyn = 225 * 1024;          // dynamic shared memory: 227 KB less the static part

enum { kErrFewFull = 31, kErrFewEmpty = 32 };

__host__ __device__ constexpr int packed_rows(int K, int bits) { return bits == 3 ? (K + 9) / 10 : K * bits / 32; }
__host__ __device__ constexpr int n_stages(int K, int bits) { return cdiv(packed_rows(K, bits), kStageRows); }
// Table pieces of a stage: 16 bytes per row and lane column = the B registers of two k-steps.
// 3-bit: three passes of five k-steps, padded to six.
__host__ __device__ constexpr int stage_pieces(int bits) { return bits == 3 ? 9 : 16 / bits; }
// Group slots of a stage.  3-bit: the two groups that a stage (160 k) meets; the one that ends in it is the first.
__host__ __device__ constexpr int stage_slots(int bits) { return bits == 3 ? 2 : 4 / bits; }
// Bytes of a stage of the table: pieces [piece][row][lane column], then per group slot and row (row count
// rounded up to even) what undoes the row's scaling of the group, and the sum of its activations.
__host__ __device__ constexpr int table_stage_bytes(int bits, int rows) {
  return stage_pieces(bits) * 64 * rows + stage_slots(bits) * 16 * ((rows + 1) / 2);
}
// Bytes that hold a tile of `rows` rows at any bit width.
__host__ __device__ constexpr size_t table_tile_bytes(int K, int rows) {
  size_t most = 0;
  for (int b = 1; b <= 4; ++b) {
    const size_t n = static_cast<size_t>(n_stages(K, b)) * table_stage_bytes(b, rows);
    most = n > most ? n : most;
  }
  return most;
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The first k-step of a group: no accumulators to clear.
__device__ __forceinline__ void mma16816_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// d += z * (hi + lo) over four k slots; fp16 offsets are exact in tf32, the two halves carry 22 bits of a group sum
__device__ __forceinline__ void mma_offsets(float (&d)[4], float z0, float z1, uint32_t hi, uint32_t lo) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%4,%5}, {%6,%7}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(__float_as_uint(z0)), "r"(__float_as_uint(z1)), "r"(hi), "r"(lo));
}

// Shared-memory reads by 32-bit address: pointers would be carried as 64 bits.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
// Two fp32 lanes per instruction.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void mul_add2(float& o0, float& o1, float a0, float a1, unsigned long long f, unsigned long long sc) {
  unsigned long long t = pack2(a0, a1), o = pack2(o0, o1);
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(t) : "l"(f));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(o) : "l"(t), "l"(sc));
  asm("mov.b64 {%0,%1}, %2;" : "=f"(o0), "=f"(o1) : "l"(o));
}

// Operand q of a packed word: two codes in place, `pos` bits up in their half.
template <int B>
struct Fmt {
  static constexpr int kEps = B == 3 ? 10 : 32 / B;
  static constexpr int kPos = 10 / B;       // operands that fit the ten mantissa bits without a shift
  static constexpr uint32_t kMask = ((1u << B) - 1u) * 0x00010001u;
  // 3-bit words are spread first: codes 0..4 to the lower half, 5..9 to the upper one
  __device__ static __forceinline__ uint32_t spread(uint32_t w) {
    return B == 3 ? ((w & 0x00007fffu) | ((w << 1) & 0x7fff0000u)) : w;
  }
  // codes q and q + kEps / 2
  __device__ static __forceinline__ uint32_t operand(uint32_t w, int q) {
    return (w >> ((q / kPos) * kPos * B)) & (kMask << (B * (q % kPos)));
  }
  __host__ __device__ static constexpr int pos(int q) { return B * (q % kPos); }
  // packed row (of eight) that lane column c reads as its word r = 0, 1.  1-bit groups are four rows long.
  __host__ __device__ static constexpr int row(int c, int r) { return B == 1 ? c + 4 * r : 2 * c + r; }
};

template <int NB>
struct State {
  float acc[2][2][NB][4];   // open group: [strip][column pair][row block][C fragment]
  float out[2][2][NB][4];   // closed groups: scale * sum(code * x) + offset * sum(x)
};

template <int NB>
__device__ __forceinline__ void clear(State<NB>& S) {
#pragma unroll
  for (int st = 0; st < 2; ++st)
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int e = 0; e < 4; ++e) S.acc[st][s][nb][e] = S.out[st][s][nb][e] = 0.f;
}

__device__ __forceinline__ void half4(uint32_t p, float (&f)[4]) {
  const uint2 r = lds64(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

// Close a group: out += scale * acc.  `meta` = its scales and offsets of the warp's 64 columns, `ft` = its
// (unscale, sum) pairs.  CLEAR: leave the accumulators at zero.
template <int NB, bool CLEAR>
__device__ __forceinline__ void fold(State<NB>& S, uint32_t meta, uint32_t ft, int rows, int lane) {
  const int g = lane >> 2, c = lane & 3;
  unsigned long long f[NB];  // of rows 8 nb + 2 c and the next; rows past the last repeat a valid one, nobody reads them
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const uint4 t = lds128(ft + 16 * min(4 * nb + c, (rows - 1) >> 1));
    f[nb] = pack2(__uint_as_float(t.x), __uint_as_float(t.z));
  }
#pragma unroll
  for (int st = 0; st < 2; ++st) {
    float sc[4];
    half4(meta + 64 * st + 8 * g, sc);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned long long s2 = pack2(sc[k], sc[k]);
      const int s = k >> 1, e = 2 * (k & 1);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        mul_add2(S.out[st][s][nb][e], S.out[st][s][nb][e + 1], S.acc[st][s][nb][e], S.acc[st][s][nb][e + 1], f[nb], s2);
        if (CLEAR) S.acc[st][s][nb][e] = S.acc[st][s][nb][e + 1] = 0.f;
      }
    }
  }
}

// Offset term of a stage: out += offset * sum(x), its groups in the k slots of one MMA per column pair.
// `on`: the lane column's group slot exists.
template <int NB>
__device__ __forceinline__ void add_offsets(State<NB>& S, uint32_t meta, uint32_t ft, int rows, bool on, int lane) {
  const int g = lane >> 2, c = lane & 3, re = (rows + 1) & ~1;
  uint32_t hi[NB], lo[NB];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    hi[nb] = lo[nb] = 0u;
    if (on) {
      const uint32_t v = lds32(ft + (c * re + min(g + 8 * nb, rows - 1)) * 8 + 4);
      hi[nb] = v & 0xffffe000u;
      lo[nb] = __float_as_uint(__uint_as_float(v) - __uint_as_float(hi[nb]));
    }
  }
#pragma unroll
  for (int st = 0; st < 2; ++st) {
    float zr[4] = {0.f, 0.f, 0.f, 0.f};
    if (on) half4(meta + c * 256 + 128 + 64 * st + 8 * g, zr);
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) mma_offsets(S.out[st][s][nb], zr[2 * s], zr[2 * s + 1], hi[nb], lo[nb]);
  }
}

// Where a lane finds its B operands: MMA column g of block nb is row g + 8 nb; columns past the last
// row stay on the zero block.
template <int NB>
struct TablePtr {
  uint32_t p[NB];
  uint32_t step[NB];  // bytes from a piece to the next
};
template <int NB>
__device__ __forceinline__ TablePtr<NB> table_ptr(uint32_t T, uint32_t zero, int rows, int lane) {
  TablePtr<NB> t;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int r = (lane >> 2) + 8 * nb;
    t.p[nb] = r < rows ? T + r * 64 + (lane & 3) * 16 : zero;
    t.step[nb] = r < rows ? rows * 64 : 0;
  }
  return t;
}

// Word r of the lane in block j (eight packed rows), both strips (STEP bytes apart).
template <int B, int STEP>
__device__ __forceinline__ void load_words(uint4 (&w)[2], uint32_t W, int j, int r, int g, int c) {
  const int row = Fmt<B>::row(c, r);
#pragma unroll
  for (int st = 0; st < 2; ++st)
    w[st] = lds128(W + st * STEP + (8 * j + row) * 128 + ((g ^ row) << 4));
}

// A stage (16 packed rows) of a 1/2/4-bit matrix: 4 / B groups, each eight k-steps of 16.
template <int B, int NB, int STEP>
__device__ __forceinline__ void stage_pow2(State<NB>& S, uint32_t W, uint32_t T, uint32_t zero, uint32_t meta, int rows, int groups,
                                           int lane) {
  using F = Fmt<B>;
  const int g = lane >> 2, c = lane & 3;
  constexpr int QW = F::kEps / 8;  // pieces per packed word
  TablePtr<NB> t = table_ptr<NB>(T, zero, rows, lane);
  // one group per trip: two blocks of rows leave no registers for more in flight
#pragma unroll 1
  for (int gi = 0; gi < groups; ++gi) {
#pragma unroll
    for (int wl = 0; wl < B; ++wl) {
      uint4 w[2];
      // the group's words: 1-bit row gi (block gi / 2), 2-bit block gi, 4-bit both blocks
      load_words<B, STEP>(w, W, B == 1 ? gi >> 1 : (B == 2 ? gi : wl >> 1), B == 1 ? gi & 1 : wl & 1, g, c);
#pragma unroll
      for (int q = 0; q < QW; ++q) {
        uint4 b[NB];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          b[nb] = lds128(t.p[nb]);
          t.p[nb] += t.step[nb];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = 2 * (2 * q + h);
#pragma unroll
          for (int st = 0; st < 2; ++st) {
            const uint32_t wv[4] = {w[st].x, w[st].y, w[st].z, w[st].w};
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const uint32_t a0 = F::operand(wv[2 * s], m), a1 = F::operand(wv[2 * s + 1], m);
              const uint32_t a2 = F::operand(wv[2 * s], m + 1), a3 = F::operand(wv[2 * s + 1], m + 1);
#pragma unroll
              for (int nb = 0; nb < NB; ++nb) {
                if (wl == 0 && m == 0) mma16816_first(S.acc[st][s][nb], a0, a1, a2, a3, b[nb].x, b[nb].y);
                else mma16816(S.acc[st][s][nb], a0, a1, a2, a3, h ? b[nb].z : b[nb].x, h ? b[nb].w : b[nb].y);
              }
            }
          }
        }
      }
    }
    fold<NB, false>(S, meta + gi * 256, T + stage_pieces(B) * 64 * rows + gi * 16 * ((rows + 1) >> 1), rows, lane);
  }
  add_offsets<NB>(S, meta, T + stage_pieces(B) * 64 * rows, rows, c < groups, lane);
}

// Five k-steps over an 8-row block of 3-bit words; `t` moves on by the pass's three pieces.
template <int NB, int STEP>
__device__ __forceinline__ void pass_b3(State<NB>& S, uint32_t W, TablePtr<NB>& t, int j, int lane) {
  using F = Fmt<3>;
  const int g = lane >> 2, c = lane & 3;
  uint4 wa[2], wb[2];
  load_words<3, STEP>(wa, W, j, 0, g, c);
  load_words<3, STEP>(wb, W, j, 1, g, c);
  uint32_t v[2][2][4];
#pragma unroll
  for (int st = 0; st < 2; ++st) {
    v[st][0][0] = F::spread(wa[st].x); v[st][0][1] = F::spread(wa[st].y);
    v[st][0][2] = F::spread(wa[st].z); v[st][0][3] = F::spread(wa[st].w);
    v[st][1][0] = F::spread(wb[st].x); v[st][1][1] = F::spread(wb[st].y);
    v[st][1][2] = F::spread(wb[st].z); v[st][1][3] = F::spread(wb[st].w);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    uint4 b[NB];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      b[nb] = lds128(t.p[nb]);
      t.p[nb] += t.step[nb];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = 2 * q + h;
      if (m < 5) {
        const int s0 = 2 * m, s1 = 2 * m + 1;  // operand slots: five of the first word, five of the second
#pragma unroll
        for (int st = 0; st < 2; ++st)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const uint32_t a0 = F::operand(v[st][s0 / 5][2 * s], s0 % 5), a1 = F::operand(v[st][s0 / 5][2 * s + 1], s0 % 5);
            const uint32_t a2 = F::operand(v[st][s1 / 5][2 * s], s1 % 5), a3 = F::operand(v[st][s1 / 5][2 * s + 1], s1 % 5);
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
              mma16816(S.acc[st][s][nb], a0, a1, a2, a3, h ? b[nb].z : b[nb].x, h ? b[nb].w : b[nb].y);
          }
      }
    }
  }
}

// A stage of a 3-bit matrix.  64 packed rows = 640 k = five groups = four stages; a group ends inside
// blocks 1, 3, 4, 6 of the run and at its end.  A block with two groups takes two passes whose table
// entries hold only the one or the other.  Both groups of a stage are folded in it, so that a reduction can be
// split at any stage: 4096 k are 26 of them, but only 7 runs.  `s4` = stage of the run, `left` = groups from the
// run's first on.
template <int NB, int STEP>
__device__ __forceinline__ void stage_b3(State<NB>& S, uint32_t W, uint32_t T, uint32_t zero, uint32_t meta, int rows, int s4, int left,
                                         int lane) {
  const uint32_t ft = T + stage_pieces(3) * 64 * rows;
  const bool late = s4 >= 2;  // the group ends in the stage's first block, not in its second
  TablePtr<NB> t = table_ptr<NB>(T, zero, rows, lane);
#pragma unroll 1
  for (int p = 0; p < 3; ++p) {
    pass_b3<NB, STEP>(S, W, t, late ? p >> 1 : (p + 1) >> 1, lane);
    const bool first = p == (late ? 0 : 1);
    if (first || (p == 2 && s4 + 1 < left))
      fold<NB, true>(S, meta + (first ? 0 : 256), ft + (first ? 0 : 16 * ((rows + 1) >> 1)), rows, lane);
  }
  const int c = lane & 3;
  add_offsets<NB>(S, meta, ft, rows, c == 0 || (c == 1 && s4 == 3 && left > 4), lane);
}

template <int B, int NB, int STEP>
__device__ __forceinline__ void stage_any(State<NB>& S, uint32_t W, uint32_t T, uint32_t zero, uint32_t meta, int rows, int sg, int ngroups,
                                          int lane) {
  if (B == 3) stage_b3<NB, STEP>(S, W, T, zero, meta, rows, sg & 3, ngroups - 5 * (sg >> 2), lane);
  else stage_pow2<B == 3 ? 2 : B, NB, STEP>(S, W, T, zero, meta, rows, min(4 / B, ngroups - (4 / B) * sg), lane);
}

// Gives a stage back behind the sums that came of everything read from it.  The refill is written past the order of a warp's
// shared-memory accesses (TMA): with the arrival right behind the reads, and 22 other warps in bank conflicts, 22 % of the words
// that a probe read were the next refill's; with an arrival whose address takes in what was read, none of 1.5e9.  (Refills by
// stores or cp.async: none either way.)  `none` is a zero that the compiler does not know.  One fragment per strip and row block will
// do, they share their loads.  Costs nothing (all of them: 1 % of 32 Mixtral rows).
template <int NB>
__device__ __forceinline__ void release_stage(const State<NB>& S, unsigned long long* empty, uint32_t none, int lane) {
  uint32_t used = 0u;
#pragma unroll
  for (int st = 0; st < 2; ++st)
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) used |= __float_as_uint(S.out[st][0][nb][0]);
  const uint32_t bar = smem_u32(empty) + (used & none);
  __syncwarp();
  if (lane == 0) mbar_arrive_at(bar);
}

// Columns 4g .. 4g + 3 of strip st for row 8 nb + 2 c + o.
template <int NB>
__device__ __forceinline__ float4 result4(const State<NB>& S, int st, int nb, int o) {
  return make_float4(S.out[st][0][nb][o], S.out[st][0][nb][2 + o], S.out[st][1][nb][o], S.out[st][1][nb][2 + o]);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(unsigned long long* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Box of a strip map (tma.cu): (column 0 of 32, packed row, strip); strips and rows past the end are zero-filled.
__device__ __forceinline__ void tma_load_strips(void* dst, const CUtensorMap* map, int row, int strip, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(row), "r"(strip), "r"(smem_u32(bar))
      : "memory");
}
// The same box into L2.
__device__ __forceinline__ void tma_prefetch_strips(const CUtensorMap* map, int row, int strip) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<unsigned long long>(map)),
               "r"(0), "r"(row), "r"(strip)
               : "memory");
}
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Part p of n of a matrix's stages.
__device__ __forceinline__ void stage_range(int bits, int K, int p, int n, int& lo, int& hi) {
  const int st = n_stages(K, bits);
  lo = st * p / n;
  hi = st * (p + 1) / n;
}

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ float round_h(float v) { return __half2float(__float2half_rn(v)); }

// Exponent that puts the largest |x| of a group into [2^14, 2^15): no bit of x is lost down to 2^-20 of it.
__device__ __forceinline__ int group_exponent(float mx) {
  const int ce = 14 - (static_cast<int>((__float_as_uint(mx) >> 23) & 0xffu) - 127);
  return ce < -100 ? -100 : (ce > 100 ? 100 : ce);
}
// (unscale, sum) of a group and the factor its activations are written with.
__device__ __forceinline__ float2 group_pair(int ce, float sum) { return make_float2(pow2i(24 - ce), sum); }

// The pieces of one packed word of a 1/2/4-bit matrix: x = its activations, f = the group's factor.
template <int B>
__device__ __forceinline__ void word_pieces(const float (&x)[32 / B], float f, unsigned char* dst, int step) {
  using F = Fmt<B>;
  constexpr int EPS = F::kEps;
#pragma unroll
  for (int q = 0; q < EPS / 8; ++q) {
    __half2 h[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float s = f * pow2i(-F::pos(4 * q + p));
      h[p] = __floats2half2_rn(x[4 * q + p] * s, x[4 * q + p + EPS / 2] * s);
    }
    *reinterpret_cast<uint4*>(dst + q * step) = *reinterpret_cast<const uint4*>(h);
  }
}

// 3-bit: the three pieces that pass `pass` (0..2) of stage sg has for lane column c.  They hold the lane's twenty
// activations k0 .. k0 + 19 (two packed words); the ones outside the pass's group are masked out, two per operand.
struct PassB3 {
  int k0, grp, slot;
  uint32_t mask[10];
};
__device__ __forceinline__ PassB3 pass_of_b3(int sg, int pass, int c) {
  const int s4 = sg & 3;
  // pass -> block of the stage, and which of its two groups (0: it has one, 1: the first, 2: the second)
  const int blk = 2 * sg + (s4 < 2 ? (pass > 0) : (pass == 2));
  const int part = s4 < 2 ? pass : (pass == 2 ? 0 : pass + 1);
  const int end = 5 * (sg >> 2) + s4;  // the group that ends in this stage
  PassB3 p;
  p.slot = part == 0 ? (s4 < 2 ? 0 : 1) : part - 1;
  p.grp = end + p.slot;
  p.k0 = 80 * blk + 20 * c;
  const int first = max(p.grp * kGroup - p.k0, 0), last = min(max((p.grp + 1) * kGroup - p.k0, 0), 20);
  const uint32_t on = first < 20 ? (1u << last) - (1u << first) : 0u;
#pragma unroll
  for (int s = 0; s < 10; ++s) {
    const int j = 10 * (s / 5) + s % 5;
    p.mask[s] = ((on >> j) & 1u ? 0x0000ffffu : 0u) | ((on >> (j + 5)) & 1u ? 0xffff0000u : 0u);
  }
  return p;
}
// x = the twenty activations, f = the group's factor, step = bytes from a piece to the next.
__device__ __forceinline__ void put_pass_b3(const float (&x)[20], float f, const PassB3& p, unsigned char* dst, int step) {
  uint32_t h[12];
#pragma unroll
  for (int s = 0; s < 10; ++s) {
    const int j = 10 * (s / 5) + s % 5;
    const float m = f * pow2i(-Fmt<3>::pos(s % 5));
    const __half2 v = __floats2half2_rn(x[j] * m, x[j + 5] * m);
    h[s] = *reinterpret_cast<const uint32_t*>(&v) & p.mask[s];
  }
  h[10] = h[11] = 0u;
#pragma unroll
  for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * step) = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
}

// Stage and slot of a group; 3-bit: the ones in which it ends.  What undoes its scaling also goes to slot 1 of the
// stage before, where groups 1 to 3 of a run begin.
__device__ __forceinline__ void group_place(int bits, int grp, int& sg, int& slot) {
  if (bits == 3) { sg = 4 * (grp / 5) + min(grp % 5, 3); slot = grp % 5 == 4 ? 1 : 0; }
  else { const int n = 4 / bits; sg = grp / n; slot = grp - sg * n; }
}

// Half a warp writes one group of one row to the table: `v` = its 128 activations in shared memory, t = the
// row's place in its tile.  All pieces of the group are written: the ones of its words, for 3-bit the ones of
// its passes.
template <typename T>
__device__ __forceinline__ void group_to_table(const T* v, int bits, int grp, unsigned char* tab, int rows, int t, int lane) {
  const int l16 = lane & 15;
  float mx = 0.f, sm = 0.f;
  {
    const uint4 r = *reinterpret_cast<const uint4*>(v + 8 * l16);
    const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float f = to_f<T>(e[k]);
      mx = fmaxf(mx, fabsf(f));
      sm += f;
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    sm += __shfl_xor_sync(0xffffffffu, sm, o);
  }
  const int ce = group_exponent(mx);
  const float f = pow2i(ce);
  int sg, slot;
  group_place(bits, grp, sg, slot);
  const int tb = table_stage_bytes(bits, rows), re = (rows + 1) & ~1;
  if (l16 == 0)
    *reinterpret_cast<float2*>(tab + sg * tb + stage_pieces(bits) * 64 * rows + (slot * re + t) * 8) = group_pair(ce, sm);
  if (bits == 3) {
    const int i5 = grp % 5, run = grp / 5;
    if (l16 == 0 && i5 >= 1 && i5 <= 3)
      *reinterpret_cast<float2*>(tab + (sg - 1) * tb + stage_pieces(3) * 64 * rows + (re + t) * 8) = group_pair(ce, sm);
    // the group's passes, counted from the run's first: 0, 1 | 2, 3, 4 | 5, 6 | 7, 8, 9 | 10, 11
    const int first = i5 == 0 ? 0 : (i5 == 1 ? 2 : (i5 == 2 ? 5 : (i5 == 3 ? 7 : 10)));
    const int count = (i5 == 1 || i5 == 3) ? 3 : 2;
    if (l16 < 4 * count) {
      const int ps = first + (l16 >> 2), c = l16 & 3, s3 = 4 * run + ps / 3, pass = ps % 3;
      const PassB3 p = pass_of_b3(s3, pass, c);
      float x[20];
#pragma unroll
      for (int j = 0; j < 20; ++j) {
        const int k = p.k0 + j - grp * kGroup;
        x[j] = k >= 0 && k < kGroup ? to_f<T>(v[k]) : 0.f;
      }
      put_pass_b3(x, f, p, tab + s3 * tb + (3 * pass * rows + t) * 64 + c * 16, 64 * rows);
    }
    return;
  }
  // 16 pieces: lane -> packed word of the group (eps activations), piece of the word
  const int eps = 32 / bits, qw = 4 / bits;
  const int w = l16 / qw, q = l16 - w * qw;
  const int c = bits == 1 ? w : (w & 7) >> 1;
  const int wr = bits == 1 ? slot : (bits == 2 ? 2 * slot + (w & 1) : 2 * (w >> 3) + (w & 1));
  const int npos = bits == 1 ? 10 : (bits == 2 ? 5 : 2);
  __half2 h[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int pr = 4 * q + p;
    const float sc = f * pow2i(-bits * (pr >= npos ? pr - npos : pr));  // at most two shifts per word
    h[p] = __floats2half2_rn(to_f<T>(v[w * eps + pr]) * sc, to_f<T>(v[w * eps + pr + (eps >> 1)]) * sc);
  }
  *reinterpret_cast<uint4*>(tab + sg * tb + ((wr * qw + q) * rows + t) * 64 + c * 16) = *reinterpret_cast<const uint4*>(h);
}

}  // namespace few

// tma.cu: packed words [rows, N] as strips of 32 columns, box 16 rows x `strips` strips, 128B swizzle.
bool tensor_map_strips(CUtensorMap* out, const void* base, int N, long long rows, int strips);

}  // namespace gemq
