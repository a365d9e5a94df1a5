// The piece of a neighbour table that a block of a pooling kernel works on, in shared memory.
#pragma once
#include "ssc_common.cuh"

namespace ssc {

struct PoolShape {
  int rows, grid;       // rows per block (0: the table of a single row does not fit), blocks
  size_t smem;
};

// 32 rows per block: enough items for 256 threads from 32 channels up, and a warp reads 128 bytes of a table line;
// fewer where that many table columns would not fit into 48 KB; a single row may take all an SM has (56 k offsets).
static inline PoolShape pool_shape(long long n, int K) {
  const size_t per_row = ((size_t)K + (K + 31) / 32) * sizeof(int32_t);
  int rows = 32;
  while (rows > 1 && rows * per_row > 48 * 1024) rows >>= 1;
  if (rows * per_row > 227 * 1024) rows = 0;
  return {rows, rows ? (int)((n + rows - 1) / rows) : 0, rows * per_row};
}

struct PoolTile {
  const int32_t *entry;    // [K][R]
  const uint32_t *mask;    // [ceil(K / 32)][R]: offsets present
  int first, rows, stride;
};

// Called by all 256 threads of the block.
static __device__ __forceinline__ PoolTile pool_tile(const int32_t *__restrict__ nbr, int K, int row_stride, int n_live, int R, int32_t *smem) {
  const int words = (K + 31) / 32;
  int32_t *entry = smem;
  uint32_t *mask = (uint32_t *)(smem + K * R);
  const int first = (int)blockIdx.x * R;
  const int rows = n_live - first < R ? (n_live - first > 0 ? n_live - first : 0) : R;
  for (int i = threadIdx.x; i < words * R; i += 256) mask[i] = 0u;
  __syncthreads();
  const int shift = __ffs(R) - 1;                  // R is a power of two
#pragma unroll 4
  for (int i = threadIdx.x; i < K * R; i += 256) {
    const int k = i >> shift, r = i & (R - 1);
    if (r >= rows) continue;
    const int32_t v = __ldg(nbr + (size_t)k * row_stride + first + r);
    if (v >= 0) {
      entry[i] = v;
      atomicOr(mask + (k >> 5) * R + r, 1u << (k & 31));
    }
  }
  __syncthreads();
  return {entry, mask, first, rows, R};
}

// use(entry, v) for the present offsets of row r of the tile, in ascending order, v filled by load(entry, v); the rows of
// G offsets are asked for before the first of them is used.
template <int G, typename V, typename L, typename U>
static __device__ __forceinline__ void pool_visit(const PoolTile &t, int r, int K, L load, U use) {
  for (int w = 0; w * 32 < K; ++w) {
    uint32_t m = t.mask[w * t.stride + r];
    while (G == 1 && m != 0u) {
      const int at = t.entry[(w * 32 + __ffs((int)m) - 1) * t.stride + r];
      m &= m - 1u;
      V v;
      load(at, v);
      use(at, v);
    }
    while (m != 0u) {
      int at[G];
      V v[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        at[j] = m != 0u ? t.entry[(w * 32 + __ffs((int)m) - 1) * t.stride + r] : -1;
        m &= m - 1u;
      }
#pragma unroll
      for (int j = 0; j < G; ++j)
        if (at[j] >= 0) load(at[j], v[j]);
#pragma unroll
      for (int j = 0; j < G; ++j)
        if (at[j] >= 0) use(at[j], v[j]);
    }
  }
}

// A thread of a pool works on four channels.  PIECE of them move per request: all four where rows are 16-byte aligned
// (c a multiple of 4), two where c is even, else one; the last thread of a row has `valid` of them.  A thread per channel
// where rows are not aligned took 92 us for 169 k rows of 30 channels and 27 offsets, pairs take 50.
struct Channels { float v[4]; };

static inline int pool_piece(int c, uintptr_t pointers) {
  return c % 4 == 0 && pointers % 16 == 0 ? 4 : c % 2 == 0 && pointers % 8 == 0 ? 2 : 1;
}

template <int PIECE>
static __device__ __forceinline__ void load_rows(const float *__restrict__ p, int valid, Channels &x) {
  if (PIECE == 4) {
    const float4 f = __ldg((const float4 *)p);
    x.v[0] = f.x; x.v[1] = f.y; x.v[2] = f.z; x.v[3] = f.w;
  } else if (PIECE == 2) {
    const float2 f = __ldg((const float2 *)p), g = valid > 2 ? __ldg((const float2 *)p + 1) : make_float2(0.f, 0.f);
    x.v[0] = f.x; x.v[1] = f.y; x.v[2] = g.x; x.v[3] = g.y;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) x.v[q] = q < valid ? __ldg(p + q) : 0.f;
  }
}

template <int PIECE>
static __device__ __forceinline__ void store_rows(float *__restrict__ p, int valid, const Channels &x) {
  if (PIECE == 4) {
    *(float4 *)p = make_float4(x.v[0], x.v[1], x.v[2], x.v[3]);
  } else if (PIECE == 2) {
    *(float2 *)p = make_float2(x.v[0], x.v[1]);
    if (valid > 2) *((float2 *)p + 1) = make_float2(x.v[2], x.v[3]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < valid) p[q] = x.v[q];
  }
}

// acc += x / d for a count d (whole_count) with r = 1 / d rounded to nearest: correctly rounded, as x / d is.  Two
// corrections by the exact remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000", 1990: a quotient within an ulp, corrected by r times its remainder, is the correctly rounded
// one); sizes whose remainder might not be representable, infinities and NaNs are divided.  Half of the values
// behind a ReLU are zeros, on which a division costs more: three average pools took 182 us with it, 105 us without.
static __device__ __forceinline__ void add_quotients(Channels &acc, const Channels &x, float d, float r) {
  bool fast = true;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float a = fabsf(x.v[q]);
    fast = fast && (a == 0.f || (a > 8.0779357e-28f && a < 1.2676506e30f));      // 2^-90, 2^100
  }
  if (fast) {
    const f32x2 rr = pair_of(r, r), dd = pair_of(-d, -d);        // (two channels per instruction: 138 k rows of 27 offsets 42.5 -> 40.6 us)
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
      const f32x2 xx = pair_of(x.v[q], x.v[q + 1]);
      f32x2 y = mul_pair(xx, rr);
      y = fma_pair(fma_pair(dd, y, xx), rr, y);
      const float2 sum = halves(add_pair(pair_of(acc.v[q], acc.v[q + 1]), fma_pair(fma_pair(dd, y, xx), rr, y)));
      acc.v[q] = sum.x;
      acc.v[q + 1] = sum.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) acc.v[q] += x.v[q] / d;
  }
}

// What add_quotients takes.  Counts are the caller's: all others are divided by (0 gives an infinity).
static __device__ __forceinline__ bool whole_count(int32_t d) { return (uint32_t)(d - 1) < (1u << 20); }

}  // namespace ssc
