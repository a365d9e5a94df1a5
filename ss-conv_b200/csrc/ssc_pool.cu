// Sparse max / avg pooling over the output-major neighbour table (one launch, each output
// row written once) and per-sample global pooling.  All HBM-bound.
#include <cuda_fp16.h>

#include "ssc_common.cuh"
#include "ssc_pool_tile.cuh"
#include "ssc_scan.cuh"

namespace ssc {

// Rows of fp32, fp16 or bf16 (IN = 0, 1, 2) channels.
template <int IN, int PIECE>
__device__ __forceinline__ void load_channels(const void *__restrict__ rows, size_t at, int valid, Channels &x) {
  if (IN == 0) {
    load_rows<PIECE>((const float *)rows + at, valid, x);
    return;
  }
  const uint16_t *p = (const uint16_t *)rows + at;
  uint16_t h[4];
  if (PIECE == 4) {
    const uint2 w = __ldg((const uint2 *)p);
    h[0] = (uint16_t)w.x; h[1] = (uint16_t)(w.x >> 16); h[2] = (uint16_t)w.y; h[3] = (uint16_t)(w.y >> 16);
  } else if (PIECE == 2) {
    const uint32_t w = __ldg((const uint32_t *)p), u = valid > 2 ? __ldg((const uint32_t *)p + 1) : 0u;
    h[0] = (uint16_t)w; h[1] = (uint16_t)(w >> 16); h[2] = (uint16_t)u; h[3] = (uint16_t)(u >> 16);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) h[q] = q < valid ? __ldg(p + q) : (uint16_t)0;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) x.v[q] = IN == 2 ? __uint_as_float((uint32_t)h[q] << 16) : __half2float(__ushort_as_half(h[q]));
}

// MODE 0 = max (output starts at 0), 1 = avg (sum of x / divisor in ascending offset order).
template <int MODE>
__device__ __forceinline__ void pool_add(Channels &acc, const Channels &x, float div, float inv) {
  if (MODE == 1) {
    add_quotients(acc, x, div, inv);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) acc.v[q] = x.v[q] > acc.v[q] ? x.v[q] : acc.v[q];
  }
}

// A block takes R output rows.  Most table entries are absent (a strided 3^3 pool over surface voxels: 1.5 to 11 of 27
// per row), and what bounded one thread per (row, 4 channels) walking the table was that walk, done once
// per channel group: 74 us for 27 offsets of 140 k rows of 76 channels.  Here the block brings its piece of the table into shared memory
// once, with a presence mask per row, and the threads then visit only
// what is there, two rows in flight (169 k rows with 11 of 27 present, 76 channels: max 94 us, with one row 100, with four 104).
template <int MODE, int IN, int PIECE>
__global__ void __launch_bounds__(256)
pool_fwd_kernel(const void *__restrict__ features, int c, const int32_t *__restrict__ nbr, int K,
                int n_out, const int32_t *__restrict__ summaryrf, float *__restrict__ out,
                const int32_t *__restrict__ n_out_dev, int R) {
  after_previous();
  extern __shared__ int32_t pool_smem[];
  const PoolTile tile = pool_tile(nbr, K, n_out, live_rows(n_out, n_out_dev), R, pool_smem);   // n_out: row stride of nbr
  const uint32_t cg = (uint32_t)(c + 3) / 4, items = (uint32_t)tile.rows * cg;
  for (uint32_t t = threadIdx.x; t < items; t += 256) {
    const int r = (int)(t / cg), c0 = (int)(t - (uint32_t)r * cg) * 4, valid = c - c0;
    const int o = tile.first + r;
    Channels acc = {{0.f, 0.f, 0.f, 0.f}};
    const float div = MODE == 1 ? (summaryrf ? (float)__ldg(summaryrf + o) : (float)K) : 1.f, inv = __frcp_rn(div);
    pool_visit<2, Channels>(tile, r, K,
        [&](int src, Channels &x) { load_channels<IN, PIECE>(features, (size_t)src * c + c0, valid, x); },
        [&](int, const Channels &x) { pool_add<MODE>(acc, x, div, inv); });
    store_rows<PIECE>(out + (size_t)o * c + c0, valid, acc);
  }
}

// The same for kernels of up to eight offsets (pools of 2^3 windows, most of whose entries are present): one
// thread per (row, 4 channels), all entries loaded at once and G rows at a time; G = 4, or 1 for fewer
// than four offsets, where threads in flight count for more (544 k rows, one offset, 76 channels: 71 us
// for 102; 119 k rows, eight offsets: avg 58 us for 78, offset by offset).
template <int MODE, int IN, int PIECE, int G>
__global__ void __launch_bounds__(256)
pool_fwd_few_kernel(const void *__restrict__ features, int c, const int32_t *__restrict__ nbr, int K, int n_out,
                    const int32_t *__restrict__ summaryrf, float *__restrict__ out, const int32_t *__restrict__ n_out_dev) {
  after_previous();
  const uint32_t cg = (uint32_t)(c + 3) / 4;
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
  if (t >= (long long)live_rows(n_out, n_out_dev) * cg) return;
  const int o = t < 0x7fffffffll ? (int)((uint32_t)t / cg) : (int)(t / cg);
  const int c0 = (int)(t - (long long)o * cg) * 4, valid = c - c0;
  const float div = MODE == 1 ? (summaryrf ? (float)__ldg(summaryrf + o) : (float)K) : 1.f, inv = __frcp_rn(div);
  Channels acc = {{0.f, 0.f, 0.f, 0.f}};
  if (G == 1) {
    for (int k = 0; k < K; ++k) {
      const int src = __ldg(nbr + (size_t)k * n_out + o);
      if (src < 0) continue;
      Channels x;
      load_channels<IN, PIECE>(features, (size_t)src * c + c0, valid, x);
      pool_add<MODE>(acc, x, div, inv);
    }
  } else {
    int src[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) src[k] = k < K ? __ldg(nbr + (size_t)k * n_out + o) : -1;
#pragma unroll
    for (int k0 = 0; k0 < 8; k0 += G) {
      Channels x[G];
#pragma unroll
      for (int k = 0; k < G; ++k)
        if (src[k0 + k] >= 0) load_channels<IN, PIECE>(features, (size_t)src[k0 + k] * c + c0, valid, x[k]);
#pragma unroll
      for (int k = 0; k < G; ++k)
        if (src[k0 + k] >= 0) pool_add<MODE>(acc, x[k], div, inv);
    }
  }
  store_rows<PIECE>(out + (size_t)o * c + c0, valid, acc);
}

// The rows of an average pool whose counts the kernels above do not take (whole_count), once more by plain division: a warp
// looks at the counts of 32 rows, nearly all of which have nothing to do.  Looked for in the kernels themselves, even
// once per row, they cost 3 to 10 % of every average pool (83 k rows of 8 offsets and 76 channels 43.9 -> 45.6 us, with a
// row's test in front of its loop 47.5; 134 k rows of 27 92.2 -> 95.1 and 101.3); this runs only where a caller
// brings counts.
template <int IN>
__global__ void __launch_bounds__(256)
pool_divided_rows_kernel(const void *__restrict__ features, int c, const int32_t *__restrict__ nbr, int K, int n_out,
                         const int32_t *__restrict__ summaryrf, float *__restrict__ out, const int32_t *__restrict__ n_out_dev) {
  after_previous();
  const int lane = threadIdx.x & 31, row0 = (int)(blockIdx.x * 256 + (threadIdx.x & ~31u)), n_rows = live_rows(n_out, n_out_dev);
  const int count = lane < n_rows - row0 ? __ldg(summaryrf + row0 + lane) : 1;
  for (unsigned left = __ballot_sync(0xffffffffu, !whole_count(count)); left != 0u; left &= left - 1u) {
    const int r = __ffs((int)left) - 1, o = row0 + r;
    const float div = (float)__shfl_sync(0xffffffffu, count, r);
    for (int ch = lane; ch < c; ch += 32) {
      float acc = 0.f;
      for (int k = 0; k < K; ++k) {
        const int src = __ldg(nbr + (size_t)k * n_out + o);
        if (src < 0) continue;
        Channels x;
        load_channels<IN, 1>(features, (size_t)src * c + ch, 1, x);
        acc += x.v[0] / div;
      }
      out[(size_t)o * c + ch] = acc;
    }
    __syncwarp();
  }
}

__global__ void summary_rf_kernel(const int32_t *__restrict__ nbr, int K, int n_out, int32_t *__restrict__ rf) {
  after_previous();
  int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_out) return;
  int cnt = 0;
  for (int kappa = 0; kappa < K; ++kappa) cnt += nbr[(size_t)kappa * n_out + o] >= 0;
  rf[o] = cnt;
}

// grid (samples, channel groups of 32), block (32, 8): the 8 row groups stride over the
// sample's rows, partial results are combined in shared memory.
template <bool MAX>
__global__ void global_pool_kernel(const float *__restrict__ feats, const int32_t *__restrict__ offsets, int c,
                                   float *__restrict__ out, int32_t *__restrict__ maxidx) {
  after_previous();
  __shared__ float sv[8][33];
  __shared__ int si[8][33];
  int s = blockIdx.x;
  int ch = blockIdx.y * 32 + threadIdx.x;
  int start = offsets[s], end = offsets[s + 1];
  float acc = MAX ? -INFINITY : 0.f;
  int arg = -1;
  if (ch < c) {
    for (int r = start + threadIdx.y; r < end; r += 8) {
      float v = __ldg(feats + (size_t)r * c + ch);
      if (MAX) {
        if (v > acc) { acc = v; arg = r; }
      } else {
        acc += v;
      }
    }
  }
  sv[threadIdx.y][threadIdx.x] = acc;
  si[threadIdx.y][threadIdx.x] = arg;
  __syncthreads();
  if (threadIdx.y == 0 && ch < c) {
    for (int g = 1; g < 8; ++g) {
      float v = sv[g][threadIdx.x];
      int a = si[g][threadIdx.x];
      if (MAX) {
        if (a >= 0 && (v > acc || (v == acc && (arg < 0 || a < arg)))) { acc = v; arg = a; }
      } else {
        acc += v;
      }
    }
    if (MAX) {
      out[(size_t)s * c + ch] = acc;
      if (maxidx) maxidx[(size_t)s * c + ch] = arg;
    } else {
      out[(size_t)s * c + ch] = acc / (float)(end - start);
    }
  }
}

// offsets[b+1] = number of rows with batch id <= b: histogram, then an in-place scan by one warp.  Rows of a
// sample follow one another nearly always: the lanes of a warp with the same id send one atomic (one per
// row queued up at a single address: 38 us for 138 k rows).
__global__ void batch_count_kernel(const int4 *__restrict__ indices, int n, int batch, int32_t *offsets,
                                   const int32_t *__restrict__ n_dev) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int b = -1;
  if (i < live_rows(n, n_dev)) b = __ldg((const int32_t *)(indices + i));
  const unsigned same = __match_any_sync(0xffffffffu, b);
  if ((unsigned)b < (unsigned)batch && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(offsets + b + 1, __popc(same));
}

__global__ void batch_scan_kernel(int32_t *offsets, int batch) {
  after_previous();
  int lane = threadIdx.x;
  int running = 0;
  for (int base = 1; base <= batch; base += 32) {
    int i = base + lane;
    int v = i <= batch ? offsets[i] : 0;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (i <= batch) offsets[i] = running + incl;
    running += __shfl_sync(0xffffffffu, incl, 31);
  }
}

// The three steps for few rows, in one block: what bounds them there is the launches.
constexpr int kOffsetsRows = 16384, kOffsetsBatch = 4096;
__global__ void __launch_bounds__(1024)
batch_offsets_small_kernel(const int4 *__restrict__ indices, int n, int batch, int32_t *__restrict__ offsets,
                           const int32_t *__restrict__ n_dev) {
  after_previous();
  __shared__ int hist[kOffsetsBatch];
  __shared__ uint32_t sums[33];
  for (int i = threadIdx.x; i < batch; i += 1024) hist[i] = 0;
  __syncthreads();
  const int live = live_rows(n, n_dev);
  for (int r0 = 0; r0 < live; r0 += 1024) {
    const int r = r0 + (int)threadIdx.x;
    const int b = r < live ? __ldg(&indices[r].x) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, b);
    if ((unsigned)b < (unsigned)batch && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(hist + b, __popc(same));
  }
  __syncthreads();
  uint32_t running = 0;
  for (int b0 = 0; b0 < batch; b0 += 1024) {
    const int b = b0 + (int)threadIdx.x;
    const uint32_t v = b < batch ? (uint32_t)hist[b] : 0u;
    uint32_t total;
    const uint32_t before = block_exclusive_scan(v, sums, &total);
    if (b < batch) offsets[b + 1] = (int32_t)(running + before + v);
    running += total;
  }
  if (threadIdx.x == 0) offsets[0] = 0;
}

}  // namespace ssc

using namespace ssc;

template <int MODE, int IN, int PIECE>
static int launch_pool_as(const void *features, int c, const int32_t *nbr, int K, int n_out, const int32_t *rf,
                          float *out, const int32_t *n_out_dev, void *stream, const char *name) {
  cudaStream_t st = as_stream(stream);
  if (K <= 8) {
    const int blocks = ceil_div((long long)n_out * ((c + 3) / 4), 256);
    if (K >= 4) launch_ready(pool_fwd_few_kernel<MODE, IN, PIECE, 4>, dim3(blocks), dim3(256), 0, st, features, c, nbr, K, n_out, rf, out, n_out_dev);
    else launch_ready(pool_fwd_few_kernel<MODE, IN, PIECE, 1>, dim3(blocks), dim3(256), 0, st, features, c, nbr, K, n_out, rf, out, n_out_dev);
  } else {
    const PoolShape p = pool_shape(n_out, K);
    SSC_REQUIRE(p.rows > 0, "%s: kernel of %d offsets is too large", name, K);
    if (p.smem > 48 * 1024) {
      cudaError_t e = allow_smem((const void *)pool_fwd_kernel<MODE, IN, PIECE>, p.smem);
      if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "%s: smem attribute: %s", name, cudaGetErrorString(e));
    }
    launch_ready(pool_fwd_kernel<MODE, IN, PIECE>, dim3(p.grid), dim3(256), p.smem, st, features, c, nbr, K, n_out, rf, out, n_out_dev, p.rows);
  }
  note_launches(1);
  if (MODE == 1 && rf != nullptr) {
    launch_ready(pool_divided_rows_kernel<IN>, dim3(ceil_div(n_out, 256)), dim3(256), 0, st, features, c, nbr, K, n_out, rf, out, n_out_dev);
    note_launches(1);
  }
  SSC_CHECK_LAUNCH(name);
  return SSC_OK;
}

template <int MODE, int IN>
static int launch_pool(const void *features, int c, const int32_t *nbr, int K, int n_out, const int32_t *rf,
                       float *out, const int32_t *n_out_dev, void *stream, const char *name) {
  SSC_REQUIRE(c > 0 && K > 0 && n_out >= 0, "%s: bad sizes", name);
  if (n_out == 0) return SSC_OK;
  SSC_REQUIRE(features && nbr && out, "%s: null pointer", name);
  const int piece = pool_piece(c, (uintptr_t)features | (uintptr_t)out);
  auto launch = piece == 4 ? launch_pool_as<MODE, IN, 4> : piece == 2 ? launch_pool_as<MODE, IN, 2> : launch_pool_as<MODE, IN, 1>;
  return launch(features, c, nbr, K, n_out, rf, out, n_out_dev, stream, name);
}

extern "C" int ssc_maxpool_fwd(const float *features, int c, const int32_t *nbr, int K, int n_out, float *out,
                               const int32_t *n_out_dev, void *stream) {
  return launch_pool<0, 0>(features, c, nbr, K, n_out, nullptr, out, n_out_dev, stream, "maxpool_fwd");
}

extern "C" int ssc_avgpool_fwd(const float *features, int c, const int32_t *nbr, int K, int n_out,
                               const int32_t *summaryrf, float *out, const int32_t *n_out_dev, void *stream) {
  return launch_pool<1, 0>(features, c, nbr, K, n_out, summaryrf, out, n_out_dev, stream, "avgpool_fwd");
}

extern "C" int ssc_pool_fwd16(const void *features, int precision, int average, int c, const int32_t *nbr, int K, int n_out,
                              const int32_t *summaryrf, float *out, const int32_t *n_out_dev, void *stream) {
  SSC_REQUIRE(precision == SSC_PREC_F16 || precision == SSC_PREC_BF16, "pool_fwd16: precision must be SSC_PREC_F16 or SSC_PREC_BF16");
  if (precision == SSC_PREC_BF16)
    return average ? launch_pool<1, 2>(features, c, nbr, K, n_out, summaryrf, out, n_out_dev, stream, "pool_fwd16")
                   : launch_pool<0, 2>(features, c, nbr, K, n_out, nullptr, out, n_out_dev, stream, "pool_fwd16");
  return average ? launch_pool<1, 1>(features, c, nbr, K, n_out, summaryrf, out, n_out_dev, stream, "pool_fwd16")
                 : launch_pool<0, 1>(features, c, nbr, K, n_out, nullptr, out, n_out_dev, stream, "pool_fwd16");
}

extern "C" int ssc_summary_rf(const int32_t *nbr, int K, int n_out, int32_t *rf, void *stream) {
  SSC_REQUIRE(K > 0 && n_out >= 0, "summary_rf: bad sizes");
  if (n_out == 0) return SSC_OK;
  SSC_REQUIRE(nbr && rf, "summary_rf: null pointer");
  { launch_ready(summary_rf_kernel, dim3(ceil_div(n_out, 256)), dim3(256), 0, as_stream(stream), nbr, K, n_out, rf); note_launches(1); }
  SSC_CHECK_LAUNCH("summary_rf");
  return SSC_OK;
}

extern "C" int ssc_global_avgpool_fwd(const float *feats, const int32_t *offsets, int n_samples, int c, float *out,
                                      void *stream) {
  SSC_REQUIRE(n_samples >= 0 && c > 0, "global_avgpool: bad sizes");
  if (n_samples == 0) return SSC_OK;
  SSC_REQUIRE(offsets && out, "global_avgpool: null pointer");
  dim3 grid(n_samples, ceil_div(c, 32)), block(32, 8);
  { launch_ready(global_pool_kernel<false>, dim3(grid), dim3(block), 0, as_stream(stream), feats, offsets, c, out, nullptr); note_launches(1); }
  SSC_CHECK_LAUNCH("global_avgpool");
  return SSC_OK;
}

extern "C" int ssc_global_maxpool_fwd(const float *feats, const int32_t *offsets, int n_samples, int c, float *out,
                                      int32_t *maxidx, void *stream) {
  SSC_REQUIRE(n_samples >= 0 && c > 0, "global_maxpool: bad sizes");
  if (n_samples == 0) return SSC_OK;
  SSC_REQUIRE(offsets && out, "global_maxpool: null pointer");
  dim3 grid(n_samples, ceil_div(c, 32)), block(32, 8);
  { launch_ready(global_pool_kernel<true>, dim3(grid), dim3(block), 0, as_stream(stream), feats, offsets, c, out, maxidx); note_launches(1); }
  SSC_CHECK_LAUNCH("global_maxpool");
  return SSC_OK;
}

extern "C" int ssc_batch_offsets(const int32_t *indices, int n, int batch, int32_t *offsets, const int32_t *n_dev,
                                 void *stream) {
  SSC_REQUIRE(n >= 0 && batch >= 1 && offsets, "batch_offsets: bad arguments");
  cudaStream_t st = as_stream(stream);
  if (n <= kOffsetsRows && batch <= kOffsetsBatch) {
    launch_ready(batch_offsets_small_kernel, dim3(1), dim3(1024), 0, st, (const int4 *)indices, n, batch, offsets, n_dev);
    note_launches(1);
    SSC_CHECK_LAUNCH("batch_offsets");
    return SSC_OK;
  }
  cudaMemsetAsync(offsets, 0, (size_t)(batch + 1) * 4, st);
  if (n > 0) { launch_ready(batch_count_kernel, dim3(ceil_div(n, 256)), dim3(256), 0, st, (const int4 *)indices, n, batch, offsets, n_dev); note_launches(1); }
  { launch_ready(batch_scan_kernel, dim3(1), dim3(32), 0, st, offsets, batch); note_launches(1); }
  SSC_CHECK_LAUNCH("batch_offsets");
  return SSC_OK;
}
