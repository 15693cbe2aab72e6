// The activation table of a few rows, built by the warp that uses it (few_rows.cuh has its layout).
#pragma once

#include "few_rows.cuh"

namespace gemq {
namespace few {

struct Rows {
  int K, ldx;
  int vec;  // 1: every row is 16-byte aligned
};

// Eight neighbouring activations; k is a multiple of eight.
template <typename T>
__device__ __forceinline__ uint4 load8(const T* p, bool vec) {
  uint4 v;
  if (vec) v = *reinterpret_cast<const uint4*>(p);
  else {
    T* e = reinterpret_cast<T*>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = p[k];
  }
  return v;
}

// The raw activations of `items` (stage, row) pairs become pieces in place.
template <typename T, int B, int kAhead>
__device__ __forceinline__ void convert_pow2(unsigned char* tab, int rows, int items, int lane) {
  using F = Fmt<B>;
  constexpr int EPS = F::kEps, QW = EPS / 8;
  const int goff = stage_pieces(B) * 64 * rows, tb = table_stage_bytes(B, rows), re = (rows + 1) & ~1;
  const int wr = (lane >> 2) & 3, c = lane & 3, h = lane >> 4;
  const int slot = B == 1 ? wr : (B == 2 ? wr >> 1 : 0);  // the group of the lane's word
  auto advance = [&](int& sg, int& t) {
    for (t += 2; t >= rows; t -= rows) ++sg;
  };
  int sg = 0, t = h;
  if (t >= rows) { t = 0; sg = 1; }
#pragma unroll 1
  for (int i0 = h; i0 < items + h; i0 += 2 * kAhead) {
    uint4 raw[kAhead][QW];
    unsigned char* st[kAhead];
    int row[kAhead];
    float mx[kAhead], sm[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const bool on = i0 + 2 * u < items;
      st[u] = tab + (on ? sg : 0) * tb;
      row[u] = on ? t : 0;
#pragma unroll
      for (int j = 0; j < QW; ++j)
        raw[u][j] = *reinterpret_cast<const uint4*>(st[u] + ((wr * QW + j) * rows + row[u]) * 64 + c * 16);
      advance(sg, t);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      mx[u] = sm[u] = 0.f;
#pragma unroll
      for (int j = 0; j < QW; ++j) {
        const T* e = reinterpret_cast<const T*>(&raw[u][j]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float f = to_f<T>(e[k]);
          mx[u] = fmaxf(mx[u], fabsf(f));
          sm[u] += f;
        }
      }
    }
#pragma unroll
    for (int o = 1; o < 4 * B; o <<= 1)
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], o));
        sm[u] += __shfl_xor_sync(0xffffffffu, sm[u], o);
      }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (i0 + 2 * u < items) {
        const int ce = group_exponent(mx[u]);
        if ((lane & (4 * B - 1)) == 0) *reinterpret_cast<float2*>(st[u] + goff + (slot * re + row[u]) * 8) = group_pair(ce, sm[u]);
        float xv[EPS];
#pragma unroll
        for (int j = 0; j < QW; ++j) {
          const T* e = reinterpret_cast<const T*>(&raw[u][j]);
#pragma unroll
          for (int k = 0; k < 8; ++k) xv[8 * j + k] = to_f<T>(e[k]);
        }
        word_pieces<B>(xv, pow2i(ce), st[u] + (wr * QW * rows + row[u]) * 64 + c * 16, 64 * rows);
      }
  }
}

// One warp: table of the k range of stages [lo, hi) for `rows` rows, 1/2/4-bit.  A lane takes one packed
// word's activations (32 / B neighbours), a half-warp a stage, 4 * B lanes a group.  The activations are
// first copied raw to where their pieces will stand (same size, same lane), all copies in flight at once,
// and rewritten in place: the loops stay short, which counts in a kernel this small -- its instructions
// come from a cold cache.
template <typename T, int B>
__device__ __forceinline__ void build_pow2(const Rows& P, unsigned char* tab, const T* x, int rows, int lo, int hi, int lane) {
  using F = Fmt<B>;
  constexpr int EPS = F::kEps, QW = EPS / 8;
  const int tb = table_stage_bytes(B, rows);
  const bool vec = P.vec != 0;
  const int wr = (lane >> 2) & 3, c = lane & 3, h = lane >> 4;
  const int items = (hi - lo) * rows;  // (stage, row), half a warp each
  const int kl = (lo * kStageRows + 8 * (wr >> 1) + F::row(c, wr & 1)) * EPS;  // first activation of the word in stage lo
  unsigned char* mine = tab + wr * QW * rows * 64 + c * 16;
  auto advance = [&](int& sg, int& t) {  // two items on
    for (t += 2; t >= rows; t -= rows) ++sg;
  };
  {
    int sg = 0, t = h;
    if (t >= rows) { t = 0; sg = 1; }
#pragma unroll 2
    for (int i = h; i < items; i += 2) {
      const int k0 = kl + sg * kStageRows * EPS;
      const T* src = x + static_cast<size_t>(t) * P.ldx + (k0 < P.K ? k0 : 0);
      unsigned char* dst = mine + sg * tb + t * 64;
#pragma unroll
      for (int j = 0; j < QW; ++j) {
        if (vec) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + j * 64 * rows)), "l"(src + 8 * j),
                       "r"(k0 < P.K ? 16 : 0)
                       : "memory");
        } else {
          *reinterpret_cast<uint4*>(dst + j * 64 * rows) = k0 < P.K ? load8(src + 8 * j, false) : make_uint4(0u, 0u, 0u, 0u);
        }
      }
      advance(sg, t);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // One row: an item at a time.  More: two items of a half-warp side by side, the shuffles of a group's maximum and sum
  // are a chain.  Not more: the instructions come from a cold cache, the largest stall of a kernel this small (8 rows,
  // 4096 x 4096, 2 bits: 6.2, 6.1, 6.3 us with one, two, four; 4 rows: 5.7, 5.8, 6.4).
  if (rows == 1 || B == 1) convert_pow2<T, B, 1>(tab, rows, items, lane);
  else convert_pow2<T, B, 2>(tab, rows, items, lane);
}

// 3-bit: groups are not word aligned.  Group statistics first (half a warp per group and row), then the pieces,
// a lane's two words at a time.
template <typename T>
__device__ __forceinline__ void build_b3(const Rows& P, unsigned char* tab, const T* x, int rows, int lo, int hi, int lane) {
  const int goff = stage_pieces(3) * 64 * rows, tb = table_stage_bytes(3, rows), re = (rows + 1) & ~1;
  const bool vec = P.vec != 0;
  // the groups that its stages meet
  const int g0 = 5 * (lo >> 2) + (lo & 3), ng = hi > lo ? min(P.K / kGroup, 5 * ((hi - 1) >> 2) + ((hi - 1) & 3) + 2) - g0 : 0;
  const int h = lane >> 4, l16 = lane & 15;
  // four loads in flight: one after the other they cost a trip to L2 each, 40 us for 16 rows of 4096
  constexpr int kAhead = 4;
#pragma unroll 1
  for (int i0 = h; i0 < rows * ng + h; i0 += 2 * kAhead) {
    uint4 v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + 2 * u, t = i / ng;
      v[u] = i < rows * ng ? load8(x + static_cast<size_t>(t) * P.ldx + (g0 + i - t * ng) * kGroup + 8 * l16, vec)
                           : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + 2 * u, t = i / ng;
      const T* e = reinterpret_cast<const T*>(&v[u]);
      float mx = 0.f, sm = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float f = to_f<T>(e[k]);
        mx = fmaxf(mx, fabsf(f));
        sm += f;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sm += __shfl_xor_sync(0xffffffffu, sm, o);
      }
      if (l16 == 0 && i < rows * ng) {
        const int grp = g0 + i - t * ng, i5 = grp % 5;
        int sg, slot;
        group_place(3, grp, sg, slot);
        const float2 fs = group_pair(group_exponent(mx), sm);
        if (sg >= lo && sg < hi) *reinterpret_cast<float2*>(tab + (sg - lo) * tb + goff + (slot * re + t) * 8) = fs;
        if (i5 >= 1 && i5 <= 3 && sg > lo) *reinterpret_cast<float2*>(tab + (sg - 1 - lo) * tb + goff + (re + t) * 8) = fs;
      }
    }
  }
  __syncwarp();
  const int halves = (hi - lo) * 12 <= 16 ? 2 : 1;  // one stage: half the lanes take the odd rows
#pragma unroll 1
  for (int i = lane & (32 / halves - 1); i < (hi - lo) * 12; i += 32 / halves) {
    const int sg = i / 12, r = i - 12 * sg, pass = r >> 2, c = r & 3;
    const PassB3 p = pass_of_b3(lo + sg, pass, c);
    const bool on = p.grp < P.K / kGroup;  // past the last group: zeros
    const unsigned char* un = tab + sg * tb + goff + p.slot * re * 8;
    unsigned char* dst = tab + sg * tb + 3 * pass * rows * 64 + c * 16;
#pragma unroll 2
    for (int t = halves == 2 ? lane >> 4 : 0; t < rows; t += halves) {
      const T* xr = x + static_cast<size_t>(t) * P.ldx + p.k0;  // out of L1 now
      float v[20];
#pragma unroll
      for (int j = 0; j < 20; j += 4) {
        uint2 q = make_uint2(0u, 0u);
        T* e = reinterpret_cast<T*>(&q);
        if (on && p.k0 + j < P.K) {
          if (vec) q = *reinterpret_cast<const uint2*>(xr + j);
          else {
#pragma unroll
            for (int k = 0; k < 4; ++k) e[k] = xr[j + k];
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) v[j + k] = to_f<T>(e[k]);
      }
      // un = 2^(24 - ce)
      const float f = on ? pow2i(24 - (static_cast<int>(__float_as_uint(*reinterpret_cast<const float*>(un + t * 8)) >> 23) - 127)) : 0.f;
      put_pass_b3(v, f, p, dst + t * 64, 64 * rows);
    }
  }
}

}  // namespace few
}  // namespace gemq
