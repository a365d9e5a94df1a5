// Voxelization (Point2Voxel), point<-voxel interpolation (Voxel2Point) helpers.  HBM-bound.
#include "ssc_common.cuh"
#include "ssc_scan.cuh"

namespace ssc {

// ------------------------------------------------------------ voxel2point_map / voxelize
__global__ void v2p_map_kernel(const int32_t *__restrict__ inverse, const int32_t *__restrict__ ids, int32_t *maps,
                               int n_point, int n_voxel, int max_active, int mode) {
  after_previous();
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_point) return;
  int v = inverse[p];
  if ((unsigned)v >= (unsigned)n_voxel) return;
  int id = ids[p];
  int32_t *row = maps + (size_t)v * (max_active + 1);
  if (mode == 1) {
    atomicMin(row + 1, id);
    row[0] = 1;
  } else if (mode == 2) {
    atomicMax(row + 1, id);
    row[0] = 1;
  } else {
    int slot = atomicAdd(row, 1);
    if (slot < max_active) row[slot + 1] = id;
  }
}

// Modes 3/4: order every row's ids ascending so that later sums are reproducible.
__global__ void v2p_sort_rows_kernel(int32_t *maps, int n_voxel, int max_active) {
  after_previous();
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_voxel) return;
  int32_t *row = maps + (size_t)v * (max_active + 1);
  int n = row[0];
  if (n > max_active) n = max_active;
  for (int i = 2; i <= n; ++i) {
    int key = row[i], j = i - 1;
    while (j >= 1 && row[j] > key) {
      row[j + 1] = row[j];
      --j;
    }
    row[j + 1] = key;
  }
}

__global__ void voxelize_fwd_kernel(const float *__restrict__ feats, float *__restrict__ out,
                                    const int32_t *__restrict__ maps, int average, int n_voxel, int max_active, int c) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n_voxel * c) return;
  int v = (int)(t / c), ch = (int)(t - (long long)v * c);
  const int32_t *row = maps + (size_t)v * (max_active + 1);
  int n = row[0];
  float mult = (average && n > 0) ? __fdiv_rn(1.f, (float)n) : 1.f;
  float acc = 0.f;
  for (int i = 1; i <= n; ++i) acc = __fadd_rn(acc, __fmul_rn(mult, __ldg(feats + (size_t)row[i] * c + ch)));
  out[t] = acc;
}

// ----------------------------------------------------------------- fused Point2Voxel core
struct P2VScratch {
  uint32_t *bitmap, *word_prefix, *block_sums;
  uint32_t *count;   // [n_point + 1] per-voxel point count, then exclusive start offsets
  uint32_t *cursor;  // [n_point] arrival rank of every point in its voxel (modes 3/4) or selected point per voxel (modes 1/2)
  int32_t *order;    // [n_point] point ids grouped by voxel
  uint32_t *block_sums2;
  int32_t *misc;
  long long n_words;
  size_t total;
};

static P2VScratch carve_p2v(void *base, int n_point, int batch, const int grid[3]) {
  P2VScratch s;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    void *p = base ? (char *)base + off : nullptr;
    off += align_up(bytes, 256);
    return p;
  };
  long long cells = (long long)batch * grid[0] * grid[1] * grid[2];
  s.n_words = (cells + 31) / 32;
  s.bitmap = (uint32_t *)take((size_t)s.n_words * 4);
  s.word_prefix = (uint32_t *)take((size_t)s.n_words * 4);
  s.block_sums = (uint32_t *)take(((size_t)((s.n_words + 1023) / 1024) + 2) * 4);
  s.count = (uint32_t *)take(((size_t)n_point + 2) * 4);
  s.cursor = (uint32_t *)take(((size_t)n_point + 2) * 4);
  s.order = (int32_t *)take(((size_t)n_point + 2) * 4);
  s.block_sums2 = (uint32_t *)take(((size_t)((n_point + 1023) / 1024) + 2) * 4);
  s.misc = (int32_t *)take(256);
  s.total = off;
  return s;
}

struct VoxelGrid {
  int grid[3];
  float unit[3];
  float half[3];
};

// Cell of a point: int((p + half) / unit), fp32 arithmetic, truncation toward zero, exactly
// the element-wise torch expression it replaces.  Returns false when the cell lies outside
// the grid (such a point is dropped).
__device__ __forceinline__ bool point_cell(const float *p, int b, int batch, const VoxelGrid &g, uint32_t &flat) {
  int c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c[d] = (int)__fdiv_rn(__fadd_rn(p[d], g.half[d]), g.unit[d]);
    if ((unsigned)c[d] >= (unsigned)g.grid[d]) return false;
  }
  if ((unsigned)b >= (unsigned)batch) return false;
  flat = (uint32_t)(((b * g.grid[0] + c[0]) * g.grid[1] + c[1]) * g.grid[2] + c[2]);
  return true;
}

__global__ void p2v_mark_kernel(const float *__restrict__ points, const int32_t *__restrict__ batch_ids, int n,
                                int batch, VoxelGrid g, uint32_t *bitmap, int32_t *status) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float p[3] = {points[i * 3 + 0], points[i * 3 + 1], points[i * 3 + 2]};
  uint32_t flat;
  if (!point_cell(p, batch_ids[i], batch, g, flat)) {
    atomicOr(status, 1);
    return;
  }
  atomicOr(bitmap + (flat >> 5), 1u << (flat & 31));
}

__device__ __forceinline__ bool point_inside(const float *__restrict__ p, const VoxelGrid &g) {
  bool out = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int c = (int)__fdiv_rn(__fadd_rn(p[d], g.half[d]), g.unit[d]);
    out = out || fabsf(p[d]) > g.half[d] || (unsigned)c >= (unsigned)g.grid[d];
  }
  return !out;
}

// What the host needs to know about a point batch before voxelizing it, in one pass:
// stats[0] points outside the grid (|p| > half extent or cell index out of range),
// stats[1] positions where the batch id decreases, stats[2] positions where it changes,
// stats[3] the last batch id.
__global__ void p2v_stats_kernel(const float *__restrict__ points, const int32_t *__restrict__ batch_ids, int n,
                                 VoxelGrid g, int32_t *stats) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool out = false, down = false, change = false;
  if (i < n) {
    out = !point_inside(points + i * 3, g);
    if (i > 0) {
      const int a = batch_ids[i - 1], b = batch_ids[i];
      down = b < a;
      change = b != a;
    }
    if (i == n - 1) stats[3] = batch_ids[i];
  }
  const int n_out = __syncthreads_count(out), n_down = __syncthreads_count(down), n_change = __syncthreads_count(change);
  if (threadIdx.x == 0) {
    if (n_out) atomicAdd(stats + 0, n_out);
    if (n_down) atomicAdd(stats + 1, n_down);
    if (n_change) atomicAdd(stats + 2, n_change);
  }
}

// Dropping the points outside the grid from a batch whose ids ascend without gaps from 0: a sample that loses all
// its points keeps a single one, at the origin and with zero features, where its first point stood.
__global__ void __launch_bounds__(256)
p2v_kept_kernel(const float *__restrict__ points, const int32_t *__restrict__ batch_ids, int n, VoxelGrid g, int n_sample,
                int32_t *__restrict__ kept) {
  after_previous();
  const int i = blockIdx.x * 256 + threadIdx.x;
  int b = -1;
  if (i < n && point_inside(points + (size_t)i * 3, g)) b = __ldg(batch_ids + i);
  const unsigned same = __match_any_sync(0xffffffffu, b);
  if ((unsigned)b < (unsigned)n_sample && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(kept + b, __popc(same));
}
// A bit per point: it stays, itself or as its sample's stand-in.  flag [n_sample]: 1 for samples with points left.
__global__ void __launch_bounds__(256)
p2v_stays_kernel(const float *__restrict__ points, const int32_t *__restrict__ batch_ids, int n, VoxelGrid g, int n_sample,
                 const int32_t *__restrict__ kept, uint32_t *__restrict__ bitmap, float *__restrict__ flag, int32_t *__restrict__ n_empty) {
  after_previous();
  const int i = blockIdx.x * 256 + threadIdx.x;
  bool stays = false, empty = false;
  if (i < n) {
    const int b = __ldg(batch_ids + i);
    empty = (i == 0 || __ldg(batch_ids + i - 1) != b) && (unsigned)b < (unsigned)n_sample && __ldg(kept + b) == 0;
    stays = empty || point_inside(points + (size_t)i * 3, g);
  }
  const unsigned word = __ballot_sync(0xffffffffu, stays), lost = __ballot_sync(0xffffffffu, empty);
  if ((threadIdx.x & 31) == 0 && i < n) bitmap[i >> 5] = word;
  if ((threadIdx.x & 31) == 0 && lost) atomicAdd(n_empty, __popc(lost));
  if (i < n_sample) flag[i] = __ldg(kept + i) > 0 ? 1.f : 0.f;
}
// VEC channels per thread; HBM-bound.
template <int VEC>
__global__ void __launch_bounds__(256)
p2v_gather_kernel(const float *__restrict__ points, const int32_t *__restrict__ batch_ids, const float *__restrict__ feats, int n, int c,
                  VoxelGrid g, const uint32_t *__restrict__ bitmap, const uint32_t *__restrict__ prefix,
                  float *__restrict__ new_points, int32_t *__restrict__ new_ids, float *__restrict__ new_feats) {
  after_previous();
  const uint32_t groups = (uint32_t)(c / VEC);
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
  if (t >= (long long)n * groups) return;
  const int i = t < 0x7fffffffll ? (int)((uint32_t)t / groups) : (int)(t / groups);
  const int q = (int)(t - (long long)i * groups);
  const uint32_t bits = __ldg(bitmap + (i >> 5));
  if (!((bits >> (i & 31)) & 1u)) return;
  const size_t to = __ldg(prefix + (i >> 5)) + (uint32_t)__popc(bits & ((1u << (i & 31)) - 1u));
  const float *p = points + (size_t)i * 3;
  const bool real = point_inside(p, g);
  if (VEC == 4) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (real) v = __ldg((const float4 *)(feats + (size_t)i * c) + q);
    ((float4 *)(new_feats + to * c))[q] = v;
  } else {
    new_feats[to * c + q] = real ? __ldg(feats + (size_t)i * c + q) : 0.f;
  }
  if (q == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) new_points[to * 3 + d] = real ? p[d] : 0.f;
    new_ids[to] = __ldg(batch_ids + i);
  }
}

__global__ void p2v_inverse_kernel(const float *__restrict__ points, const int32_t *__restrict__ batch_ids, int n,
                                   int batch, VoxelGrid g, const uint32_t *__restrict__ bitmap,
                                   const uint32_t *__restrict__ word_prefix, int mode, int32_t *inverse,
                                   uint32_t *count, uint32_t *select) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float p[3] = {points[i * 3 + 0], points[i * 3 + 1], points[i * 3 + 2]};
  uint32_t flat;
  if (!point_cell(p, batch_ids[i], batch, g, flat)) {
    inverse[i] = -1;
    return;
  }
  uint32_t w = flat >> 5, bit = flat & 31;
  int v = (int)(word_prefix[w] + __popc(bitmap[w] & ((1u << bit) - 1u)));
  inverse[i] = v;
  if (mode == 1) atomicMin(select + v, (uint32_t)i);
  else if (mode == 2) atomicMax(select + v, (uint32_t)i);
  else select[i] = atomicAdd(count + v, 1u);   // modes 3 / 4: arrival rank of the point in its voxel (select is per point then)
}

// order[start of the point's voxel + its arrival rank] = point: the rank was taken when the points were
// counted, so this pass needs no atomics (the lists are put into point order by the pass after it).
__global__ void p2v_scatter_kernel(const int32_t *__restrict__ inverse, int n, const uint32_t *__restrict__ start,
                                   const uint32_t *__restrict__ rank, int32_t *order) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int v = inverse[i];
  if (v < 0) return;
  order[__ldg(start + v) + __ldg(rank + i)] = i;
}

__global__ void p2v_sort_segments_kernel(const uint32_t *__restrict__ start, int n_voxel, int32_t *order) {
  after_previous();
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_voxel) return;
  int a = (int)start[v], b = (int)start[v + 1];
  for (int i = a + 1; i < b; ++i) {
    int key = order[i], j = i - 1;
    while (j >= a && order[j] > key) {
      order[j + 1] = order[j];
      --j;
    }
    order[j + 1] = key;
  }
}

__global__ void p2v_reduce_kernel(const float *__restrict__ feats, int c, const uint32_t *__restrict__ start,
                                  const int32_t *__restrict__ order, int n_voxel, int average, float *__restrict__ out) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n_voxel * c) return;
  int v = (int)(t / c), ch = (int)(t - (long long)v * c);
  int a = (int)start[v], b = (int)start[v + 1];
  int n = b - a;
  float mult = (average && n > 0) ? __fdiv_rn(1.f, (float)n) : 1.f;
  float acc = 0.f;
  for (int i = a; i < b; ++i) acc = __fadd_rn(acc, __fmul_rn(mult, __ldg(feats + (size_t)order[i] * c + ch)));
  out[t] = acc;
}

// The same sums with one thread per voxel and the channels (at most 8: xyz, colour, a few scalars)
// in registers: the point list is read once per voxel instead of once per channel, no 64-bit
// division.  Per (voxel, channel) the additions happen in the same order as above: same bits.
template <int CMAX>
__global__ void __launch_bounds__(256)
p2v_reduce_small_kernel(const float *__restrict__ feats, int c, const uint32_t *__restrict__ start,
                        const int32_t *__restrict__ order, int n_voxel, int average, float *__restrict__ out) {
  after_previous();
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_voxel) return;
  const int a = (int)start[v], b = (int)start[v + 1];
  const int n = b - a;
  const float mult = (average && n > 0) ? __fdiv_rn(1.f, (float)n) : 1.f;
  float acc[CMAX];
#pragma unroll
  for (int ch = 0; ch < CMAX; ++ch) acc[ch] = 0.f;
  for (int i = a; i < b; ++i) {
    const float *fp = feats + (size_t)__ldg(order + i) * c;
#pragma unroll
    for (int ch = 0; ch < CMAX; ++ch)
      if (ch < c) acc[ch] = __fadd_rn(acc[ch], __fmul_rn(mult, __ldg(fp + ch)));
  }
  float *op = out + (size_t)v * c;
#pragma unroll
  for (int ch = 0; ch < CMAX; ++ch)
    if (ch < c) op[ch] = acc[ch];
}

__global__ void p2v_select_kernel(const float *__restrict__ feats, int c, const uint32_t *__restrict__ select,
                                  int n_voxel, int n_point, float *__restrict__ out) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n_voxel * c) return;
  int v = (int)(t / c), ch = (int)(t - (long long)v * c);
  uint32_t p = select[v];
  out[t] = p < (uint32_t)n_point ? __ldg(feats + (size_t)p * c + ch) : 0.f;
}

static void fill_grid(VoxelGrid &g, const int grid[3], const float unit[3]) {
  for (int d = 0; d < 3; ++d) {
    g.grid[d] = grid[d];
    g.unit[d] = unit[d];
    float total = (float)grid[d] * unit[d];
    g.half[d] = 0.5f * total;
  }
}

// ----------------------------------------------------------------------- three_nn
// Known points in tiles of 1024 (ranges: batch ids of a tile) and chunks of 32 (chunks: batch ids and x coordinates of a
// chunk; points in grid order, as the voxelizer and the rulebook give them, have a slab of few x).
constexpr int NN_CHUNK = 32, NN_TILE = 32 * NN_CHUNK;

// A tile's ranges of batch ids and x.  shares: how many of its chunks, of 1024, a point of it lies in by their ranges of
// batch ids and x, on average of 32 points: a few tens in grid order, 1024 where nothing can be passed over.
constexpr int NN_SHARES = 1024;

__global__ void __launch_bounds__(NN_TILE)
nn_ranges_kernel(const float4 *__restrict__ known, int m, float2 *__restrict__ ranges, float4 *__restrict__ chunks, float4 *__restrict__ tiles,
                 int32_t *__restrict__ shares) {
  after_previous();
  __shared__ float4 chunk_s[32];
  __shared__ int in_s[32];
  const int lane = threadIdx.x & 31, c = threadIdx.x >> 5, k = blockIdx.x * NN_TILE + (int)threadIdx.x;
  const float4 p = k < m ? __ldg(known + k) : make_float4(NAN, NAN, NAN, NAN);
  auto widen = [](float4 r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      r.x = fminf(r.x, __shfl_xor_sync(0xffffffffu, r.x, o));
      r.y = fmaxf(r.y, __shfl_xor_sync(0xffffffffu, r.y, o));
      r.z = fminf(r.z, __shfl_xor_sync(0xffffffffu, r.z, o));
      r.w = fmaxf(r.w, __shfl_xor_sync(0xffffffffu, r.w, o));
    }
    return r;
  };
  // (fminf and fmaxf pass over a coordinate that is not a number: such a point is nobody's neighbour)
  const float4 r = widen(make_float4(fminf(INFINITY, p.x), fmaxf(-INFINITY, p.x), fminf(INFINITY, p.y), fmaxf(-INFINITY, p.y)));
  if (lane == 0) {
    chunk_s[c] = r;
    if (chunks != nullptr) chunks[blockIdx.x * (NN_TILE / NN_CHUNK) + c] = r;
  }
  __syncthreads();
  const float4 other = chunk_s[lane];
  const int middle = min(max(m - (k - lane), 1), NN_CHUNK) / 2;           // of the chunk's points
  const float sample = __shfl_sync(0xffffffffu, p.x, middle), x = __shfl_sync(0xffffffffu, p.y, middle);
  const unsigned in = __ballot_sync(0xffffffffu, other.x <= sample && sample <= other.y && other.z <= x && x <= other.w);
  if (lane == 0) in_s[c] = __popc(in);
  __syncthreads();
  if (c == 0) {
    const int all = __reduce_add_sync(0xffffffffu, in_s[lane]), have = min((m - (int)blockIdx.x * NN_TILE + NN_CHUNK - 1) / NN_CHUNK, 32);
    const float4 t = widen(other);
    if (lane == 0) {
      ranges[blockIdx.x] = make_float2(t.x, t.y);
      if (chunks != nullptr) {
        tiles[blockIdx.x] = t;
        shares[blockIdx.x] = have > 0 ? NN_SHARES * all / (have * have) : 0;
      }
    }
  }
}

// The contraction nvcc applies to the reference's dx*dx + dy*dy + dz*dz
// (interpolate_cuda_kernel.cu:39), checked bit for bit against the reference's own kernel.
__device__ __forceinline__ float nn_dist2(const float4 &u, const float4 &k) {
  const float dx = __fsub_rn(u.y, k.y), dy = __fsub_rn(u.z, k.z), dz = __fsub_rn(u.w, k.w);
  return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

// Where most points have to be looked at: SPLIT threads per query; known points stream through shared memory in
// tiles of 1024, tiles whose batch-id range cannot match any query of the block are skipped.  Thread s of a query
// looks at every SPLIT-th point of a tile; the three best of them are merged by (distance, index), which is
// the result of the exhaustive reference loop (ascending k, strict <): the smallest index wins ties.
template <int SPLIT>
__device__ __forceinline__ void nn_by_tiles(int first, int n, int m, const float4 *__restrict__ unknown, const float4 *__restrict__ known,
                                            const float2 *__restrict__ ranges, float *__restrict__ dist2, int32_t *__restrict__ idx) {
  __shared__ float4 tile[NN_TILE];
  __shared__ float qmin_s[8], qmax_s[8];
  const int q = first + (int)threadIdx.x / SPLIT, part = threadIdx.x % SPLIT;
  float4 u = q < n ? unknown[q] : make_float4(NAN, 0.f, 0.f, 0.f);
  float lo = q < n ? u.x : INFINITY, hi = q < n ? u.x : -INFINITY;
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_down_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_down_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    qmin_s[threadIdx.x >> 5] = lo;
    qmax_s[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  float qmin = qmin_s[0], qmax = qmax_s[0];
  for (int w = 1; w < 8; ++w) {
    qmin = fminf(qmin, qmin_s[w]);
    qmax = fmaxf(qmax, qmax_s[w]);
  }
  float best[3] = {INFINITY, INFINITY, INFINITY};
  int at[3] = {0, 0, 0};
  // (d, i) into the ordered triple; equal distances stay behind
  auto take = [&](float d, int i) {
    if (d < best[0]) {
      best[2] = best[1]; at[2] = at[1];
      best[1] = best[0]; at[1] = at[0];
      best[0] = d; at[0] = i;
    } else if (d < best[1]) {
      best[2] = best[1]; at[2] = at[1];
      best[1] = d; at[1] = i;
    } else if (d < best[2]) {
      best[2] = d; at[2] = i;
    }
  };
  const int n_tiles = (m + NN_TILE - 1) / NN_TILE;
  for (int t = 0; t < n_tiles; ++t) {
    const float2 r = ranges[t];
    if (r.y < qmin || r.x > qmax) continue;  // block-uniform
    __syncthreads();
    const int base = t * NN_TILE;
    for (int i = threadIdx.x; i < NN_TILE; i += 256) tile[i] = base + i < m ? known[base + i] : make_float4(NAN, 0.f, 0.f, 0.f);
    __syncthreads();
    const int cnt = min(NN_TILE, m - base);
    if (q < n && !(r.y < u.x || r.x > u.x)) {
#pragma unroll 4
      for (int i = part; i < cnt; i += SPLIT) {
        const float4 k = tile[i];
        const float d = nn_dist2(u, k);
        if (k.x == u.x && d < best[2]) take(d, base + i);
      }
    }
  }
  // merge the partners' triples (a slot that was never filled is infinite and loses to everything)
#pragma unroll
  for (int o = 1; o < SPLIT; o <<= 1) {
    float od[3];
    int oi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      od[k] = __shfl_xor_sync(0xffffffffu, best[k], o);
      oi[k] = __shfl_xor_sync(0xffffffffu, at[k], o);
    }
    float md[3];
    int mi[3], a = 0, c = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float da = a == 0 ? best[0] : a == 1 ? best[1] : best[2], dc = c == 0 ? od[0] : c == 1 ? od[1] : od[2];
      const int ia = a == 0 ? at[0] : a == 1 ? at[1] : at[2], ic = c == 0 ? oi[0] : c == 1 ? oi[1] : oi[2];
      const bool mine = da < dc || (da == dc && ia <= ic);
      md[k] = mine ? da : dc;
      mi[k] = mine ? ia : ic;
      a += mine ? 1 : 0;
      c += mine ? 0 : 1;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) { best[k] = md[k]; at[k] = mi[k]; }
  }
  if (q < n && part == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dist2[q * 3 + k] = best[k];
      idx[q * 3 + k] = best[k] == INFINITY ? 0 : at[k];
    }
  }
}

// The tiles that can hold points of a sample: all within [first, end), multiples of 32.  share: how many of 1024 of their
// chunks a point lies in, on average of those among the first 32 that hold any.
struct NnSpan {
  float sample;
  int first, end, share;
};
__device__ __forceinline__ NnSpan nn_span(float sample, int n_tiles, const float4 *__restrict__ tiles, const int32_t *__restrict__ shares) {
  const int lane = threadIdx.x & 31;
  NnSpan s = {sample, 0, 0, 0};
  for (int t0 = 0; t0 < n_tiles; t0 += 32) {
    const bool there = t0 + lane < n_tiles;
    const float4 r = there ? __ldg(tiles + t0 + lane) : make_float4(INFINITY, -INFINITY, 0.f, 0.f);
    const int share = there ? __ldg(shares + t0 + lane) : 0;
    const bool mine = r.x <= sample && sample <= r.y;
    const int have = __popc(__ballot_sync(0xffffffffu, mine));
    if (have == 0) continue;
    if (s.end == 0) {
      s.first = t0;
      s.share = __reduce_add_sync(0xffffffffu, mine ? share : 0) / have;
    }
    s.end = t0 + 32;
  }
  return s;
}

// Where ranges of x are narrow: a warp per query.  Its lanes look at the ranges of 32 tiles at a time, then at the 32 chunks of a
// tile that can hold points of the query's sample: first at the points of the chunks nearest in x, then of those whose distance in
// x alone does not exceed the third best so far.  That distance, rounded like the points' own, is never more than theirs:
// every rounding involved is monotonic.  Of several tiles the nearest in x comes first: in order, each of those before it
// would hold the best so far and be looked at whole (4096 queries among 40 k points in order: 1170 us, 586 by tiles, 102 like this).
// Each lane keeps its three best by (distance, index); the three best of the warp by that order are the result of the
// exhaustive reference loop.
constexpr int NN_QUERIES = 4;                     // of a warp, one after the other
__device__ __forceinline__ void nn_by_warps(int q0, float4 next, NnSpan span, int n, int m, const float4 *__restrict__ unknown, const float4 *__restrict__ known,
                                            const float4 *__restrict__ chunks, const float4 *__restrict__ tiles, const int32_t *__restrict__ shares,
                                            float *__restrict__ dist2, int32_t *__restrict__ idx) {
  const int lane = threadIdx.x & 31, n_tiles = (m + NN_TILE - 1) / NN_TILE, n_chunks = (m + NN_CHUNK - 1) / NN_CHUNK;
  for (int q = q0; q < min(q0 + NN_QUERIES, n); ++q) {
    const float4 u = next;
    next = __ldg(unknown + min(q + 1, n - 1));    // (on its way while this one is looked for)
    if (u.x != span.sample) span = nn_span(u.x, n_tiles, tiles, shares);
    float d0 = INFINITY, d1 = INFINITY, d2 = INFINITY, limit = INFINITY;       // limit: no less than the warp's third best
    int i0 = 0, i1 = 0, i2 = 0;
    auto before = [](float d, int i, float e, int j) { return d < e || (d == e && i < j); };
    auto take = [&](const float4 &k, int i) {
      const float d = nn_dist2(u, k);
      if (k.x == u.x && d <= limit && d < INFINITY && before(d, i, d2, i2)) {
        if (before(d, i, d1, i1)) {
          d2 = d1; i2 = i1;
          if (before(d, i, d0, i0)) { d1 = d0; i1 = i0; d0 = d; i0 = i; }
          else { d1 = d; i1 = i; }
        } else {
          d2 = d; i2 = i;
        }
      }
    };
    const float4 none = make_float4(NAN, 0.f, 0.f, 0.f);
    auto look_at = [&](int c0, unsigned left) {
      for (; (left & (left - 1u)) != 0u;) {
        const int a = (c0 + __ffs((int)left) - 1) * NN_CHUNK + lane;
        left &= left - 1u;
        const int b = (c0 + __ffs((int)left) - 1) * NN_CHUNK + lane;
        left &= left - 1u;
        const float4 ka = a < m ? __ldg(known + a) : none, kb = b < m ? __ldg(known + b) : none;
        take(ka, a);
        take(kb, b);
      }
      if (left != 0u) {
        const int a = (c0 + __ffs((int)left) - 1) * NN_CHUNK + lane;
        take(a < m ? __ldg(known + a) : none, a);
      }
    };
    // (distances are not negative: their order is that of their bits)
    auto third_best = [&]() {
      uint32_t a = __float_as_uint(d0), b = __float_as_uint(d1), c = __float_as_uint(d2), least = 0u;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        least = __reduce_min_sync(0xffffffffu, a);
        const int holder = __ffs((int)__ballot_sync(0xffffffffu, a == least)) - 1;
        if (lane == holder) { a = b; b = c; c = 0x7f800000u; }
      }
      return __uint_as_float(least);
    };
    // the square of the distance in x to the nearest point with lo <= x <= hi
    auto least_of = [&](float lo, float hi) {
      const float off = fmaxf(0.f, fmaxf(__fsub_rn(lo, u.y), __fsub_rn(u.y, hi)));
      return __fmul_rn(off, off);
    };
    bool stale = false;                           // points were taken since `limit` was found
    auto look_in = [&](int tile) {
      const int c0 = tile * (NN_TILE / NN_CHUNK);
      const float4 c = c0 + lane < n_chunks ? __ldg(chunks + c0 + lane) : make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
      const bool may = c.x <= u.x && u.x <= c.y;
      const float least = may ? least_of(c.z, c.w) : INFINITY;
      const uint32_t nearest = __reduce_min_sync(0xffffffffu, __float_as_uint(least));
      const bool near = may && __float_as_uint(least) == nearest;
      look_at(c0, __ballot_sync(0xffffffffu, near));
      limit = third_best();
      const unsigned rest = __ballot_sync(0xffffffffu, may && !near && least <= limit);
      look_at(c0, rest);
      stale = rest != 0u;
    };
    int home = -1, n_mine = 0;
    float nearest = INFINITY;
    for (int t0 = span.first; t0 < span.end; t0 += 32) {
      const float4 r = t0 + lane < n_tiles ? __ldg(tiles + t0 + lane) : make_float4(INFINITY, -INFINITY, 0.f, 0.f);
      const bool mine = r.x <= u.x && u.x <= r.y;
      const unsigned have = __ballot_sync(0xffffffffu, mine);
      if (have == 0u) continue;
      n_mine += __popc(have);
      const float least = mine ? least_of(r.z, r.w) : INFINITY;
      const float here = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(least)));
      if (home >= 0 && !(here < nearest)) continue;
      nearest = here;
      home = t0 + __ffs((int)__ballot_sync(0xffffffffu, mine && least == here)) - 1;
    }
    if (home >= 0) look_in(home);
    for (int t0 = span.first; n_mine > 1 && t0 < span.end; t0 += 32) {
      const float4 r = t0 + lane < n_tiles ? __ldg(tiles + t0 + lane) : make_float4(INFINITY, -INFINITY, 0.f, 0.f);
      const bool mine = r.x <= u.x && u.x <= r.y && t0 + lane != home;
      const float least = mine ? least_of(r.z, r.w) : INFINITY;
      for (unsigned left = __ballot_sync(0xffffffffu, mine && least <= limit); left != 0u; left &= left - 1u) {
        const int t = __ffs((int)left) - 1;
        if (stale) limit = third_best();
        stale = false;
        if (__shfl_sync(0xffffffffu, least, t) <= limit) look_in(t0 + t);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint32_t least = __reduce_min_sync(0xffffffffu, __float_as_uint(d0));
      const bool best = __float_as_uint(d0) == least;
      const uint32_t at = __reduce_min_sync(0xffffffffu, best ? (uint32_t)i0 : 0xffffffffu);
      if (lane == 0) {
        dist2[q * 3 + k] = __uint_as_float(least);
        idx[q * 3 + k] = least == 0x7f800000u ? 0 : (int32_t)at;
      }
      if (best && (uint32_t)i0 == at) { d0 = d1; i0 = i1; d1 = d2; i1 = i2; d2 = INFINITY; i2 = 0; }
    }
  }
}

// A group's queries all go the way that suits the first one's sample: by warps where a point of its tiles lies in up to three eighths of
// their chunks, by tiles where more of them would have to be looked at anyhow, at twice the instructions per point.  (64 samples of
// 4096 queries and 1024 points, us: in grid order 147 by warps, 269 by tiles; in any order 484 and 251.  By warps at a half already:
// 24 samples of 1000 each in any order 78, like this 55.)
constexpr int NN_MOST = 3 * NN_SHARES / 8;
// Up to 256 points are no matter of chunks (100 k queries among 20: 10.7 us by tiles at once, 15.4 with ranges and a second kernel).
constexpr int NN_FEW = 8 * NN_CHUNK;
template <int GROUP>
__device__ __forceinline__ NnSpan nn_group(int first, int m, const float4 *__restrict__ unknown, const float4 *__restrict__ tiles, const int32_t *__restrict__ shares) {
  return nn_span(__ldg(&unknown[first / GROUP * GROUP].x), (m + NN_TILE - 1) / NN_TILE, tiles, shares);
}

// Few queries: 32 to a block, whichever way they go.
__global__ void __launch_bounds__(256)
three_nn_kernel(int n, int m, const float4 *__restrict__ unknown, const float4 *__restrict__ known, const float2 *__restrict__ ranges,
                const float4 *__restrict__ chunks, const float4 *__restrict__ tiles, const int32_t *__restrict__ shares, float *__restrict__ dist2,
                int32_t *__restrict__ idx) {
  after_previous();
  const int first = (int)blockIdx.x * 32, q0 = first + ((int)threadIdx.x >> 5) * NN_QUERIES;
  const float4 own = __ldg(unknown + min(q0, n - 1));
  NnSpan span = {0.f, 0, 0, NN_SHARES};
  if (chunks != nullptr) span = nn_group<32>(first, m, unknown, tiles, shares);
  if (span.share <= NN_MOST) nn_by_warps(q0, own, span, n, m, unknown, known, chunks, tiles, shares, dist2, idx);
  else nn_by_tiles<8>(first, n, m, unknown, known, ranges, dist2, idx);
}

// Many: each way has its own kernel, which passes over the other's groups of 64.
__global__ void __launch_bounds__(256)
three_nn_warps_kernel(int n, int m, const float4 *__restrict__ unknown, const float4 *__restrict__ known, const float4 *__restrict__ chunks,
                      const float4 *__restrict__ tiles, const int32_t *__restrict__ shares, float *__restrict__ dist2, int32_t *__restrict__ idx) {
  after_previous();
  const int first = (int)blockIdx.x * 32, q0 = first + ((int)threadIdx.x >> 5) * NN_QUERIES;
  const float4 own = __ldg(unknown + min(q0, n - 1));
  const NnSpan span = nn_group<64>(first, m, unknown, tiles, shares);
  if (span.share <= NN_MOST) nn_by_warps(q0, own, span, n, m, unknown, known, chunks, tiles, shares, dist2, idx);
}
__global__ void __launch_bounds__(256)
three_nn_tiles_kernel(int n, int m, const float4 *__restrict__ unknown, const float4 *__restrict__ known, const float2 *__restrict__ ranges,
                      const float4 *__restrict__ tiles, const int32_t *__restrict__ shares, float *__restrict__ dist2, int32_t *__restrict__ idx) {
  after_previous();
  const int first = (int)blockIdx.x * 64;
  if (tiles != nullptr && nn_group<64>(first, m, unknown, tiles, shares).share <= NN_MOST) return;
  nn_by_tiles<4>(first, n, m, unknown, known, ranges, dist2, idx);
}

// Rows (batch id, x, y, z) as three_nn takes them, and the interpolation weights from its squared distances:
// element for element the torch expressions of Voxel2Point, a dozen launches of a few microseconds otherwise.
__global__ void __launch_bounds__(256)
voxel_centres_kernel(const int4 *__restrict__ indices, int n, float3 unit, float3 half_extent, float3 half_unit, float4 *__restrict__ out) {
  after_previous();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int4 v = __ldg(indices + i);
  out[i] = make_float4((float)v.x, __fadd_rn(__fsub_rn(__fmul_rn((float)v.y, unit.x), half_extent.x), half_unit.x),
                       __fadd_rn(__fsub_rn(__fmul_rn((float)v.z, unit.y), half_extent.y), half_unit.y),
                       __fadd_rn(__fsub_rn(__fmul_rn((float)v.w, unit.z), half_extent.z), half_unit.z));
}
__global__ void __launch_bounds__(256)
point_rows_kernel(const float *__restrict__ points, const int32_t *__restrict__ ids, int n, float4 *__restrict__ out) {
  after_previous();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) out[i] = make_float4((float)__ldg(ids + i), __ldg(points + (size_t)i * 3), __ldg(points + (size_t)i * 3 + 1), __ldg(points + (size_t)i * 3 + 2));
}
__global__ void __launch_bounds__(256)
nn_weights_kernel(const float *__restrict__ dist2, int n, float *__restrict__ weight) {
  after_previous();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  float r[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) r[k] = __fdiv_rn(1.f, __fadd_rn(__fsqrt_rn(__ldg(dist2 + (size_t)i * 3 + k)), 1e-8f));
  const float s = __fadd_rn(__fadd_rn(r[0], r[2]), r[1]);      // (the order of torch.sum)
#pragma unroll
  for (int k = 0; k < 3; ++k) weight[(size_t)i * 3 + k] = __fdiv_rn(r[k], s);
}

__global__ void three_interpolate_kernel(int c, int n, const float *__restrict__ points,
                                         const int32_t *__restrict__ idx, const float *__restrict__ weight,
                                         float *__restrict__ out) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n * c) return;
  int p = (int)(t / c), ch = (int)(t - (long long)p * c);
  float w0 = weight[p * 3 + 0], w1 = weight[p * 3 + 1], w2 = weight[p * 3 + 2];
  int i0 = idx[p * 3 + 0], i1 = idx[p * 3 + 1], i2 = idx[p * 3 + 2];
  // w0*p0 + w1*p1 + w2*p2 as nvcc contracts it in the reference (interpolate_cuda_kernel.cu:100),
  // checked bit for bit against the reference's own kernel
  float b = __fmul_rn(w1, __ldg(points + (size_t)i1 * c + ch));
  float a = __fmaf_rn(w0, __ldg(points + (size_t)i0 * c + ch), b);
  out[t] = __fmaf_rn(w2, __ldg(points + (size_t)i2 * c + ch), a);
}

// Four channels per thread (16-byte gathers and stores, 32-bit index arithmetic) for channel
// counts that are multiples of four; the same arithmetic per element.
__global__ void __launch_bounds__(256)
three_interpolate_vec4_kernel(uint32_t groups, uint32_t total, const float4 *__restrict__ points,
                              const int32_t *__restrict__ idx, const float *__restrict__ weight, float4 *__restrict__ out) {
  after_previous();
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const uint32_t p = t / groups, g = t - p * groups;
  const float w0 = __ldg(weight + p * 3 + 0), w1 = __ldg(weight + p * 3 + 1), w2 = __ldg(weight + p * 3 + 2);
  const int i0 = __ldg(idx + p * 3 + 0), i1 = __ldg(idx + p * 3 + 1), i2 = __ldg(idx + p * 3 + 2);
  const float4 p0 = __ldg(points + (size_t)i0 * groups + g);
  const float4 p1 = __ldg(points + (size_t)i1 * groups + g);
  const float4 p2 = __ldg(points + (size_t)i2 * groups + g);
  float4 r;
  r.x = __fmaf_rn(w2, p2.x, __fmaf_rn(w0, p0.x, __fmul_rn(w1, p1.x)));
  r.y = __fmaf_rn(w2, p2.y, __fmaf_rn(w0, p0.y, __fmul_rn(w1, p1.y)));
  r.z = __fmaf_rn(w2, p2.z, __fmaf_rn(w0, p0.z, __fmul_rn(w1, p1.z)));
  r.w = __fmaf_rn(w2, p2.w, __fmaf_rn(w0, p0.w, __fmul_rn(w1, p1.w)));
  out[t] = r;
}

}  // namespace ssc

using namespace ssc;

extern "C" int ssc_voxel2point_map(const int32_t *inverse, const int32_t *ids, int32_t *maps, int n_point,
                                   int n_voxel, int max_active, int mode, void *stream) {
  SSC_REQUIRE(mode >= 1 && mode <= 4, "voxel2point_map: mode %d not in 1..4", mode);
  SSC_REQUIRE(n_point >= 0 && n_voxel >= 0 && max_active >= 1, "voxel2point_map: bad sizes");
  if (n_point == 0 || n_voxel == 0) return SSC_OK;
  SSC_REQUIRE(inverse && ids && maps, "voxel2point_map: null pointer");
  cudaStream_t st = as_stream(stream);
  { launch_ready(v2p_map_kernel, dim3(ceil_div(n_point, 256)), dim3(256), 0, st, inverse, ids, maps, n_point, n_voxel, max_active, mode); note_launches(1); }
  if (mode >= 3) { launch_ready(v2p_sort_rows_kernel, dim3(ceil_div(n_voxel, 128)), dim3(128), 0, st, maps, n_voxel, max_active); note_launches(1); }
  SSC_CHECK_LAUNCH("voxel2point_map");
  return SSC_OK;
}

extern "C" int ssc_voxelize_fwd(const float *feats, float *out, const int32_t *maps, int mode, int n_voxel,
                                int max_active, int c, void *stream) {
  SSC_REQUIRE(n_voxel >= 0 && max_active >= 1 && c >= 1, "voxelize_fwd: bad sizes");
  if (n_voxel == 0) return SSC_OK;
  SSC_REQUIRE(feats && out && maps, "voxelize_fwd: null pointer");
  long long threads = (long long)n_voxel * c;
  { launch_ready(voxelize_fwd_kernel, dim3(ceil_div(threads, 256)), dim3(256), 0, as_stream(stream), feats, out, maps, mode == 4, n_voxel,
                                                                            max_active, c); note_launches(1); }
  SSC_CHECK_LAUNCH("voxelize_fwd");
  return SSC_OK;
}

extern "C" size_t ssc_p2v_scratch_bytes(int n_point, int batch, const int grid[3]) {
  if (n_point < 0 || batch < 1 || !grid) return 0;
  return carve_p2v(nullptr, n_point, batch, grid).total;
}

// Feature steering: every point is moved into the frame of its sample, new_p = (p - t_b) . R_b
// (/ (s_b + 1e-8)), and every irrep block of its feature row is multiplied from the right by the
// sample's representation matrix D^l_b.  One thread per (point, output channel or coordinate).
// Real Wigner-D matrices of the samples' rotations: D^l(R) = Y_l(R v) pinv(Y_l(v)) over fixed directions v (the
// projection the host tables were made for), in double precision.  Real spherical harmonics at a unit
// vector (x, y, z): sqrt(2) N P~_l^m(z) Re / Im (x + i y)^m with P~ the Legendre functions without their
// sin^m factor (standard recurrences in l; no trigonometry).  A block per sample: a thread per direction puts the
// harmonics of the rotated direction into shared memory, then a thread per matrix element adds them up.
// dirs / pinv: per order l, 6 (2 l + 1) + 8 directions [S, 3] and the pseudo-inverse [S, 2 l + 1], one order after
// the other.  axes != 0: the rotation is described in the frame whose polar axis is y (R -> S R S^T).
// T: the rotations as the caller has them, fp32 or double (rounded to fp32 first they cost 4e-8 per entry and order).
template <typename T>
__global__ void __launch_bounds__(128)
steer_matrices_kernel(const T *__restrict__ rot, int orders, const double *__restrict__ dirs,
                      const double *__restrict__ pinv, int axes, int stride, float *__restrict__ dmats) {
  after_previous();
  extern __shared__ double ys[];                 // per order [S][2 l + 1], as pinv
  const int b = blockIdx.x;
  double R[3][3], Q[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) R[i][j] = (double)rot[(size_t)b * 9 + i * 3 + j];
  const double det = R[0][0] * (R[1][1] * R[2][2] - R[1][2] * R[2][1]) - R[0][1] * (R[1][0] * R[2][2] - R[1][2] * R[2][0]) +
                     R[0][2] * (R[1][0] * R[2][1] - R[1][1] * R[2][0]);
  const double sign = det > 0.0 ? 1.0 : (det < 0.0 ? -1.0 : 0.0);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) Q[i][j] = sign * (axes ? R[(i + 2) % 3][(j + 2) % 3] : R[i][j]);
  int d0 = 0, p0 = 0;
  for (int l = 0; l < orders; ++l) {
    const int d = 2 * l + 1, s_cnt = 6 * d + 8;
    for (int s = (int)threadIdx.x - (d0 / 3) % (int)blockDim.x; s < s_cnt; s += blockDim.x) {   // orders side by side over the threads
      if (s < 0) continue;
      const double vx = dirs[d0 + s * 3], vy = dirs[d0 + s * 3 + 1], vz = dirs[d0 + s * 3 + 2];
      double x = Q[0][0] * vx + Q[0][1] * vy + Q[0][2] * vz, y = Q[1][0] * vx + Q[1][1] * vy + Q[1][2] * vz;
      double z = Q[2][0] * vx + Q[2][1] * vy + Q[2][2] * vz;
      z = z > 1.0 ? 1.0 : (z < -1.0 ? -1.0 : z);
      const double xy = sqrt(x * x + y * y), want = sqrt(1.0 - z * z);   // the azimuth of (x, y) at the polar angle of z
      if (xy > 0.0) {
        x *= want / xy;
        y *= want / xy;
      } else {
        x = want;
        y = 0.0;
      }
      double re = 1.0, im = 0.0, pmm = 1.0, fact = (2.0 * l + 1.0) / 12.566370614359172954;   // fact: N^2 of order m
      for (int m = 0; m <= l; ++m) {
        if (m > 0) {
          const double t = re * x - im * y;
          im = re * y + im * x;
          re = t;
          pmm *= 2.0 * m - 1.0;
          fact /= (double)(l + m) * (double)(l - m + 1);
        }
        double p_prev = 0.0, p = pmm;
        for (int ll = m + 1; ll <= l; ++ll) {
          const double t = ((2.0 * ll - 1.0) * z * p - (ll + m - 1.0) * p_prev) / (double)(ll - m);
          p_prev = p;
          p = t;
        }
        const double n = sqrt(fact) * (m > 0 ? 1.4142135623730950488 : 1.0) * p;
        ys[p0 + s * d + l + m] = n * re;
        if (m > 0) ys[p0 + s * d + l - m] = n * im;
      }
    }
    d0 += 3 * s_cnt;
    p0 += s_cnt * d;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < stride; e += blockDim.x) {
    int l = 0, off = 0;
    p0 = 0;
    while (e >= off + (2 * l + 1) * (2 * l + 1)) {
      off += (2 * l + 1) * (2 * l + 1);
      p0 += (6 * (2 * l + 1) + 8) * (2 * l + 1);
      ++l;
    }
    const int d = 2 * l + 1, row = (e - off) / d, col = (e - off) - row * d, s_cnt = 6 * d + 8;
    double acc = 0.0;
#pragma unroll 8
    for (int s = 0; s < s_cnt; ++s) acc = fma(ys[p0 + s * d + row], pinv[p0 + s * d + col], acc);
    dmats[(size_t)b * stride + e] = (float)acc;
  }
}

__global__ void steer_kernel(const float *__restrict__ points, const float *__restrict__ feats,
                             const int32_t *__restrict__ ids, const float *__restrict__ rot, const float *__restrict__ trans,
                             const float *__restrict__ scale, const float *__restrict__ dmats, int d_stride,
                             const int32_t *__restrict__ chan, int n, int c, int n_sample, float *__restrict__ new_points,
                             float *__restrict__ new_feats) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int width = c + 3;
  if (t >= (long long)n * width) return;
  const int p = (int)(t / width), k = (int)(t - (long long)p * width);
  const int b = ids[p];
  if ((unsigned)b >= (unsigned)n_sample) {  // foreign batch id: leave a defined value
    if (k < c) new_feats[(size_t)p * c + k] = 0.f;
    else new_points[(size_t)p * 3 + (k - c)] = 0.f;
    return;
  }
  if (k >= c) {
    const int j = k - c;
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) acc += (points[(size_t)p * 3 + i] - trans[b * 3 + i]) * rot[b * 9 + i * 3 + j];
    if (scale) acc = acc / (scale[b] + 1e-8f);
    new_points[(size_t)p * 3 + j] = acc;
    return;
  }
  const int start = chan[k * 3 + 0], d = chan[k * 3 + 1], off = chan[k * 3 + 2];
  const int j = k - start;
  const float *D = dmats + (size_t)b * d_stride + off;
  float acc = 0.f;
  for (int i = 0; i < d; ++i) acc += feats[(size_t)p * c + start + i] * D[i * d + j];
  new_feats[(size_t)p * c + k] = acc;
}

template <typename T>
static int steer_matrices(const T *rot, int batch, int orders, const double *dirs, const double *pinv, int axes, float *dmats, void *stream) {
  SSC_REQUIRE(batch >= 0 && orders >= 1 && orders <= SSC_STEER_MAX_ORDERS, "steer_matrices: bad sizes");
  if (batch == 0) return SSC_OK;
  SSC_REQUIRE(rot && dirs && pinv && dmats, "steer_matrices: null pointer");
  int stride = 0, harmonics = 0;
  for (int l = 0; l < orders; ++l) {
    stride += (2 * l + 1) * (2 * l + 1);
    harmonics += (6 * (2 * l + 1) + 8) * (2 * l + 1);
  }
  const size_t smem = (size_t)harmonics * sizeof(double);       // 5 KB for orders 0..3, below 48 KB up to order 8
  if (smem > 48 * 1024) {
    cudaError_t e = allow_smem((const void *)steer_matrices_kernel<T>, smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "steer_matrices: smem attribute: %s", cudaGetErrorString(e));
  }
  { launch_ready(steer_matrices_kernel<T>, dim3(batch), dim3(128), smem, as_stream(stream), rot, orders, dirs, pinv, axes, stride, dmats); note_launches(1); }
  SSC_CHECK_LAUNCH("steer_matrices");
  return SSC_OK;
}

extern "C" int ssc_steer_matrices(const float *rot, int batch, int orders, const double *dirs, const double *pinv, int axes,
                                  float *dmats, void *stream) {
  return steer_matrices(rot, batch, orders, dirs, pinv, axes, dmats, stream);
}

extern "C" int ssc_steer_matrices64(const double *rot, int batch, int orders, const double *dirs, const double *pinv, int axes,
                                    float *dmats, void *stream) {
  return steer_matrices(rot, batch, orders, dirs, pinv, axes, dmats, stream);
}

extern "C" int ssc_steer_fwd(const float *points, const float *feats, const int32_t *ids, const float *rot,
                             const float *trans, const float *scale, const float *dmats, int d_stride,
                             const int32_t *chan, int n, int c, int n_sample, float *new_points, float *new_feats,
                             void *stream) {
  SSC_REQUIRE(n >= 0 && c >= 1 && n_sample >= 1 && d_stride >= 1, "steer_fwd: bad sizes");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(points && feats && ids && rot && trans && dmats && chan && new_points && new_feats, "steer_fwd: null pointer");
  long long total = (long long)n * (c + 3);
  { launch_ready(steer_kernel, dim3(ceil_div(total, 256)), dim3(256), 0, as_stream(stream), points, feats, ids, rot, trans, scale, dmats, d_stride,
                                                                    chan, n, c, n_sample, new_points, new_feats); note_launches(1); }
  SSC_CHECK_LAUNCH("steer_fwd");
  return SSC_OK;
}

extern "C" int ssc_p2v_stats(const float *points, const int32_t *batch_ids, int n_point, const int grid[3],
                             const float unit[3], int32_t *stats_dev, void *stream) {
  SSC_REQUIRE(n_point >= 0 && grid && unit && stats_dev, "p2v_stats: bad arguments");
  cudaStream_t st = as_stream(stream);
  cudaMemsetAsync(stats_dev, 0, 4 * sizeof(int32_t), st);
  if (n_point == 0) return SSC_OK;
  SSC_REQUIRE(points && batch_ids, "p2v_stats: null pointer");
  VoxelGrid g;
  fill_grid(g, grid, unit);
  { launch_ready(p2v_stats_kernel, dim3(ceil_div(n_point, 256)), dim3(256), 0, st, points, batch_ids, n_point, g, stats_dev); note_launches(1); }
  SSC_CHECK_LAUNCH("p2v_stats");
  return SSC_OK;
}

extern "C" size_t ssc_p2v_keep_scratch_bytes(int n_point, int n_sample) {
  const size_t words = (size_t)(n_point > 0 ? n_point : 1) / 32 + 1;
  return align_up((size_t)n_sample * 4, 256) + 2 * align_up(words * 4, 256) + align_up((words / 1024 + 3) * 4, 256);
}

extern "C" int ssc_p2v_keep(const float *points, const int32_t *batch_ids, const float *feats, int n_point, int c, int n_sample,
                            const int grid[3], const float unit[3], float *new_points, int32_t *new_ids, float *new_feats,
                            float *flag, int32_t *counts_dev, void *scratch, size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(n_point >= 1 && c >= 1 && n_sample >= 1 && n_sample <= n_point && grid && unit, "p2v_keep: bad sizes");
  SSC_REQUIRE(points && batch_ids && feats && new_points && new_ids && new_feats && flag && counts_dev, "p2v_keep: null pointer");
  if (!scratch || scratch_bytes < ssc_p2v_keep_scratch_bytes(n_point, n_sample)) return fail(SSC_ERR_SCRATCH, "p2v_keep: scratch too small");
  cudaStream_t st = as_stream(stream);
  VoxelGrid g;
  fill_grid(g, grid, unit);
  const size_t words = (size_t)(n_point + 31) / 32, room = align_up(((size_t)n_point / 32 + 1) * 4, 256);
  int32_t *kept = (int32_t *)scratch;
  uint32_t *bitmap = (uint32_t *)((char *)scratch + align_up((size_t)n_sample * 4, 256)), *prefix = (uint32_t *)((char *)bitmap + room);
  uint32_t *sums = (uint32_t *)((char *)prefix + room);
  cudaMemsetAsync(kept, 0, (size_t)n_sample * 4, st);
  cudaMemsetAsync(counts_dev, 0, 8, st);
  const int blocks = ceil_div(n_point, 256);
  launch_ready(p2v_kept_kernel, dim3(blocks), dim3(256), 0, st, points, batch_ids, n_point, g, n_sample, kept);
  launch_ready(p2v_stays_kernel, dim3(blocks), dim3(256), 0, st, points, batch_ids, n_point, g, n_sample, kept, bitmap, flag, counts_dev + 1);
  note_launches(2);
  if (int e = exclusive_scan_u32<true>(bitmap, (long long)words, prefix, sums, counts_dev, nullptr, st)) return e;
  if (c % 4 == 0 && (((uintptr_t)feats | (uintptr_t)new_feats) & 15u) == 0)
    launch_ready(p2v_gather_kernel<4>, dim3(ceil_div((long long)n_point * (c / 4), 256)), dim3(256), 0, st, points, batch_ids, feats, n_point, c, g, bitmap, prefix, new_points, new_ids, new_feats);
  else
    launch_ready(p2v_gather_kernel<1>, dim3(ceil_div((long long)n_point * c, 256)), dim3(256), 0, st, points, batch_ids, feats, n_point, c, g, bitmap, prefix, new_points, new_ids, new_feats);
  note_launches(1);
  SSC_CHECK_LAUNCH("p2v_keep");
  return SSC_OK;
}

extern "C" int ssc_voxel_centres(const int32_t *indices, int n, const float unit[3], const float extent[3], float *rows, void *stream) {
  SSC_REQUIRE(n >= 0 && unit && extent, "voxel_centres: bad arguments");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(indices && rows, "voxel_centres: null pointer");
  launch_ready(voxel_centres_kernel, dim3(ceil_div(n, 256)), dim3(256), 0, as_stream(stream), (const int4 *)indices, n, make_float3(unit[0], unit[1], unit[2]),
                                                                        make_float3(0.5f * extent[0], 0.5f * extent[1], 0.5f * extent[2]),
                                                                        make_float3(0.5f * unit[0], 0.5f * unit[1], 0.5f * unit[2]), (float4 *)rows);
  note_launches(1);
  SSC_CHECK_LAUNCH("voxel_centres");
  return SSC_OK;
}

extern "C" int ssc_point_rows(const float *points, const int32_t *ids, int n, float *rows, void *stream) {
  SSC_REQUIRE(n >= 0, "point_rows: bad size");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(points && ids && rows, "point_rows: null pointer");
  launch_ready(point_rows_kernel, dim3(ceil_div(n, 256)), dim3(256), 0, as_stream(stream), points, ids, n, (float4 *)rows);
  note_launches(1);
  SSC_CHECK_LAUNCH("point_rows");
  return SSC_OK;
}

extern "C" int ssc_nn_weights(const float *dist2, int n, float *weight, void *stream) {
  SSC_REQUIRE(n >= 0, "nn_weights: bad size");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(dist2 && weight, "nn_weights: null pointer");
  launch_ready(nn_weights_kernel, dim3(ceil_div(n, 256)), dim3(256), 0, as_stream(stream), dist2, n, weight);
  note_launches(1);
  SSC_CHECK_LAUNCH("nn_weights");
  return SSC_OK;
}

extern "C" int ssc_p2v_count(const float *points, const int32_t *batch_ids, int n_point, int batch, const int grid[3],
                             const float unit[3], int32_t *n_voxel_dev, int32_t *status, void *scratch,
                             size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(n_point >= 0 && batch >= 1 && grid && unit && n_voxel_dev, "p2v_count: bad arguments");
  long long cells = (long long)batch * grid[0] * grid[1] * grid[2];
  SSC_REQUIRE(cells > 0 && cells < 2147483647ll, "p2v_count: batch*volume does not fit the int32 flat index");
  P2VScratch s = carve_p2v(scratch, n_point, batch, grid);
  if (!scratch || scratch_bytes < s.total) return fail(SSC_ERR_SCRATCH, "p2v_count: scratch %zu < %zu bytes", scratch_bytes, s.total);
  cudaStream_t st = as_stream(stream);
  VoxelGrid g;
  fill_grid(g, grid, unit);
  cudaMemsetAsync(s.bitmap, 0, (size_t)s.n_words * 4, st);
  cudaMemsetAsync(s.misc, 0, 256, st);
  if (n_point > 0) { launch_ready(p2v_mark_kernel, dim3(ceil_div(n_point, 256)), dim3(256), 0, st, points, batch_ids, n_point, batch, g, s.bitmap, status ? status : s.misc + 1); note_launches(1); }
  SSC_CHECK_LAUNCH("p2v_mark");
  if (int e = exclusive_scan_u32<true>(s.bitmap, s.n_words, s.word_prefix, s.block_sums, s.misc, n_voxel_dev, st)) return e;
  SSC_CHECK_LAUNCH("p2v_count");
  return SSC_OK;
}

extern "C" int ssc_p2v_fill(const float *points, const int32_t *batch_ids, const float *feats, int n_point, int c,
                            int batch, const int grid[3], const float unit[3], int mode, int n_voxel,
                            int32_t *voxel_indices, int32_t *inverse, float *voxel_feats, void *scratch,
                            size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(mode >= 1 && mode <= 4, "p2v_fill: mode %d not in 1..4", mode);
  SSC_REQUIRE(n_point >= 0 && n_voxel >= 0 && n_voxel <= n_point && c >= 1 && grid && unit, "p2v_fill: bad arguments");
  if (n_voxel == 0) return SSC_OK;
  SSC_REQUIRE(points && batch_ids && feats && voxel_indices && inverse && voxel_feats, "p2v_fill: null pointer");
  P2VScratch s = carve_p2v(scratch, n_point, batch, grid);
  if (!scratch || scratch_bytes < s.total) return fail(SSC_ERR_SCRATCH, "p2v_fill: scratch %zu < %zu bytes", scratch_bytes, s.total);
  cudaStream_t st = as_stream(stream);
  VoxelGrid g;
  fill_grid(g, grid, unit);
  if (int e = bitmap_decode(s.bitmap, s.word_prefix, s.n_words, grid, n_voxel, voxel_indices, st)) return e;
  if (mode >= 3) cudaMemsetAsync(s.count, 0, ((size_t)n_voxel + 1) * 4, st);
  else cudaMemsetAsync(s.cursor, mode == 1 ? 0xFF : 0x00, (size_t)n_voxel * 4, st);
  { launch_ready(p2v_inverse_kernel, dim3(ceil_div(n_point, 256)), dim3(256), 0, st, points, batch_ids, n_point, batch, g, s.bitmap, s.word_prefix,
                                                            mode, inverse, s.count, s.cursor); note_launches(1); }
  SSC_CHECK_LAUNCH("p2v_inverse");
  long long threads = (long long)n_voxel * c;
  if (mode >= 3) {
    // counts -> exclusive start offsets (in place), cursor = copy
    if (int e = exclusive_scan_u32<false>(s.count, (long long)n_voxel + 1, s.count, s.block_sums2, nullptr, nullptr, st)) return e;
    { launch_ready(p2v_scatter_kernel, dim3(ceil_div(n_point, 256)), dim3(256), 0, st, inverse, n_point, s.count, s.cursor, s.order); note_launches(1); }
    { launch_ready(p2v_sort_segments_kernel, dim3(ceil_div(n_voxel, 128)), dim3(128), 0, st, s.count, n_voxel, s.order); note_launches(1); }
    if (c <= 4) {
      { launch_ready(p2v_reduce_small_kernel<4>, dim3(ceil_div(n_voxel, 256)), dim3(256), 0, st, feats, c, s.count, s.order, n_voxel, mode == 4, voxel_feats); note_launches(1); }
    } else if (c <= 8) {
      { launch_ready(p2v_reduce_small_kernel<8>, dim3(ceil_div(n_voxel, 256)), dim3(256), 0, st, feats, c, s.count, s.order, n_voxel, mode == 4, voxel_feats); note_launches(1); }
    } else {
      { launch_ready(p2v_reduce_kernel, dim3(ceil_div(threads, 256)), dim3(256), 0, st, feats, c, s.count, s.order, n_voxel, mode == 4, voxel_feats); note_launches(1); }
    }
  } else {
    { launch_ready(p2v_select_kernel, dim3(ceil_div(threads, 256)), dim3(256), 0, st, feats, c, s.cursor, n_voxel, n_point, voxel_feats); note_launches(1); }
  }
  SSC_CHECK_LAUNCH("p2v_fill");
  return SSC_OK;
}

// [tiles x chunks of a tile] chunk ranges, [tiles] ranges of batch ids and x, [tiles] of batch ids, [tiles] shares; 16 bytes to align them
static size_t nn_tiles(int m) { return (size_t)ceil_div(m > 0 ? m : 1, NN_TILE); }

extern "C" size_t ssc_three_nn_scratch_bytes(int m) {
  return nn_tiles(m) * ((NN_TILE / NN_CHUNK + 1) * sizeof(float4) + sizeof(float2) + sizeof(int32_t)) + 16;
}

extern "C" int ssc_three_nn(int n, int m, const float *unknown, const float *known, float *dist2, int32_t *idx,
                            void *scratch, size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(n >= 0 && m >= 0, "three_nn: bad sizes");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(unknown && dist2 && idx && (m == 0 || known), "three_nn: null pointer");
  cudaStream_t st = as_stream(stream);
  // a buffer for the tiles' ranges alone will do: every point of a tile is looked at then
  if (!scratch || scratch_bytes < nn_tiles(m) * sizeof(float2))
    return fail(SSC_ERR_SCRATCH, "three_nn: scratch %zu < %zu bytes", scratch_bytes, nn_tiles(m) * sizeof(float2));
  float4 *chunks = nullptr, *tiles = nullptr;
  float2 *ranges = (float2 *)scratch;
  int32_t *shares = nullptr;
  if (m > NN_FEW && scratch_bytes >= ssc_three_nn_scratch_bytes(m)) {
    chunks = (float4 *)(((uintptr_t)scratch + 15) & ~(uintptr_t)15);
    tiles = chunks + nn_tiles(m) * (NN_TILE / NN_CHUNK);
    ranges = (float2 *)(tiles + nn_tiles(m));
    shares = (int32_t *)(ranges + nn_tiles(m));
  }
  { launch_ready(nn_ranges_kernel, dim3((int)nn_tiles(m)), dim3(NN_TILE), 0, st, (const float4 *)known, m, ranges, chunks, tiles, shares); note_launches(1); }
  // 32 queries to a block fill the SMs up to 256 queries per SM; beyond, by tiles, a tile's way to shared memory and the merging pay
  // for 64 only (64 k queries in any order 131 us in one kernel, 123 in two; in grid order 77 and 79.  20 k: 309 and 357).
  if (n < sm_count() * 256) {
    { launch_ready(three_nn_kernel, dim3(ceil_div(n, 32)), dim3(256), 0, st, n, m, (const float4 *)unknown, (const float4 *)known, ranges, chunks, tiles, shares, dist2, idx); note_launches(1); }
  } else {
    { launch_ready(three_nn_tiles_kernel, dim3(ceil_div(n, 64)), dim3(256), 0, st, n, m, (const float4 *)unknown, (const float4 *)known, ranges, tiles, shares, dist2, idx); note_launches(1); }
    if (chunks != nullptr)
      { launch_ready(three_nn_warps_kernel, dim3(ceil_div(n, 32)), dim3(256), 0, st, n, m, (const float4 *)unknown, (const float4 *)known, chunks, tiles, shares, dist2, idx); note_launches(1); }
  }
  SSC_CHECK_LAUNCH("three_nn");
  return SSC_OK;
}

extern "C" int ssc_three_interpolate_fwd(int c, int m, int n, const float *points, const int32_t *idx,
                                         const float *weight, float *out, void *stream) {
  SSC_REQUIRE(c >= 1 && n >= 0 && m >= 0, "three_interpolate: bad sizes");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(points && idx && weight && out, "three_interpolate: null pointer");
  long long threads = (long long)n * c;
  if ((c & 3) == 0 && threads / 4 < (1ll << 31) && (((uintptr_t)points | (uintptr_t)out) & 15u) == 0) {
    const uint32_t groups = (uint32_t)(c >> 2), total = (uint32_t)(threads >> 2);
    { launch_ready(three_interpolate_vec4_kernel, dim3(ceil_div(total, 256)), dim3(256), 0, as_stream(stream), groups, total, (const float4 *)points, idx, weight, (float4 *)out); note_launches(1); }
    SSC_CHECK_LAUNCH("three_interpolate");
    return SSC_OK;
  }
  { launch_ready(three_interpolate_kernel, dim3(ceil_div(threads, 256)), dim3(256), 0, as_stream(stream), c, n, points, idx, weight, out); note_launches(1); }
  SSC_CHECK_LAUNCH("three_interpolate");
  return SSC_OK;
}
