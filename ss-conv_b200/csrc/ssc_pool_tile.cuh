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

// f(entry) for the present offsets of row r of the tile, in ascending order.
template <typename F>
static __device__ __forceinline__ void pool_visit(const PoolTile &t, int r, int K, F f) {
  for (int w = 0; w * 32 < K; ++w) {
    uint32_t m = t.mask[w * t.stride + r];
    while (m != 0u) {
      const int k = w * 32 + __ffs((int)m) - 1;
      m &= m - 1u;
      f(t.entry[k * t.stride + r]);
    }
  }
}

// x / d for a count d (a whole number of 1 .. 2^20) with r = 1 / d rounded to nearest: correctly rounded, as x / d is.
// Two corrections by the exact remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000", 1990: a quotient within an ulp, corrected by r times its remainder, is the correctly rounded
// one); sizes whose remainder might not be representable, infinities and NaNs are divided.  Half of the values
// behind a ReLU are zeros, on which a division costs more: three average pools took 182 us with it, 105 us without.
static __device__ __forceinline__ float divide_by_count(float x, float d, float r) {
  const float a = fabsf(x);
  if (!(a == 0.f || (a > 8.0779357e-28f && a < 1.2676506e30f))) return x / d;      // 2^-90, 2^100
  float q = x * r;
  q = fmaf(fmaf(-d, q, x), r, q);
  return fmaf(fmaf(-d, q, x), r, q);
}

}  // namespace ssc
