// Steerable kernel materialisation and the exact-fp32 (CUDA core) output-stationary
// gather-GEMM kernel.  The tensor-core (tcgen05) variant lives in ssc_conv_tc.cu.
#include "ssc_conv_internal.cuh"

namespace ssc {

// filters[kappa][cin][cout] = sum_b w[u,v,b] * basis[b,a,c,kappa]; one thread per element,
// cout fastest so the (large) filter tensor is written coalesced; the basis blob is small
// and stays in L1/L2.
__global__ void materialize_kernel(const float *__restrict__ weight, const float *__restrict__ basis,
                                   const int32_t *__restrict__ block_table, int n_blocks_in,
                                   const int32_t *__restrict__ out_field, const int32_t *__restrict__ in_field,
                                   int c_out, int c_in, int K, float *__restrict__ filters) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)K * c_in * c_out;
  if (t >= total) return;
  int co = (int)(t % c_out);
  long long r = t / c_out;
  int ci = (int)(r % c_in);
  int kappa = (int)(r / c_in);
  int i = out_field[co * 3 + 0], u = out_field[co * 3 + 1], a = out_field[co * 3 + 2];
  int j = in_field[ci * 3 + 0], v = in_field[ci * 3 + 1], c = in_field[ci * 3 + 2];
  const int32_t *blk = block_table + (size_t)(i * n_blocks_in + j) * 6;
  int boff = blk[0];
  float acc = 0.f;
  if (boff >= 0) {
    int woff = blk[1], nb = blk[2], m_in = blk[3], d_out = blk[4], d_in = blk[5];
    const float *w = weight + woff + (size_t)(u * m_in + v) * nb;
    const float *bp = basis + boff + (size_t)(a * d_in + c) * K + kappa;
    size_t bstride = (size_t)d_out * d_in * K;
    for (int b = 0; b < nb; ++b) acc = fmaf(w[b], bp[b * bstride], acc);
  }
  filters[t] = acc;
}

// Adjoint: d_w[u,v,b] = sum over a, c, kappa of d_filters[kappa][cin][cout] * basis[b,a,c,kappa].  One block per
// (output field copy, input field copy): its d_filters entries (at most 49 K for orders up to 3) go to
// shared memory in the basis' own order, read in runs along cout, then every basis element is one
// coalesced dot product; eight warps share the basis elements.  One launch of a few microseconds per layer:
// as one small library contraction per pair of orders it was 20 launches and 1 ms of host time.
constexpr int kMatBwdThreads = 256;
__global__ void __launch_bounds__(kMatBwdThreads)
materialize_bwd_kernel(const float *__restrict__ g, const float *__restrict__ basis, const int32_t *__restrict__ block_table,
                       int n_blocks_in, const int32_t *__restrict__ out_field, const int32_t *__restrict__ in_field,
                       const int32_t *__restrict__ out_start, const int32_t *__restrict__ in_start, int c_out, int c_in, int K,
                       int staged, float *__restrict__ d_weight) {
  after_previous();
  extern __shared__ float gs[];
  const int co0 = out_start[blockIdx.y], ci0 = in_start[blockIdx.x];
  const int i = out_field[co0 * 3], u = out_field[co0 * 3 + 1], j = in_field[ci0 * 3], v = in_field[ci0 * 3 + 1];
  const int32_t *blk = block_table + (size_t)(i * n_blocks_in + j) * 6;
  const int boff = blk[0];
  if (boff < 0) return;
  const int nb = blk[2], m_in = blk[3], d_out = blk[4], d_in = blk[5], total = d_out * d_in * K;
  if (staged) {
#pragma unroll 4
    for (int t = threadIdx.x; t < total; t += kMatBwdThreads) {      // a fastest: runs of d_out floats
      const int a = t % d_out, r = t / d_out, kappa = r % K, c = r / K;
      gs[(a * d_in + c) * K + kappa] = __ldg(g + ((size_t)kappa * c_in + ci0 + c) * c_out + co0 + a);
    }
    __syncthreads();
  }
  float *dw = d_weight + blk[1] + (size_t)(u * m_in + v) * nb;
  for (int b = threadIdx.x >> 5; b < nb; b += kMatBwdThreads / 32) {
    const float *bp = basis + boff + (size_t)b * total;
    float s = 0.f;
    if (staged) {
#pragma unroll 8
      for (int t = threadIdx.x & 31; t < total; t += 32) s = fmaf(gs[t], __ldg(bp + t), s);
    } else {
      for (int t = threadIdx.x & 31; t < total; t += 32) {
        const int kappa = t % K, r = t / K, c = r % d_in, a = r / d_in;
        s = fmaf(__ldg(g + ((size_t)kappa * c_in + ci0 + c) * c_out + co0 + a), __ldg(bp + t), s);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) dw[b] = s;
  }
}

// ---------------------------------------------------------------------------------------
// Exact fp32 path: tile of 64 output rows x 64 output channels per block, 256 threads with a
// 4x4 register tile each, reduction over (kernel offset, input channel) in chunks of 16.
// Offsets with no neighbour inside the tile are skipped.
constexpr int BM = 64, BN = 64, BK = 16;

__global__ void __launch_bounds__(256)
conv_fwd_fp32_kernel(const float *__restrict__ features, int c_in, const float *__restrict__ filters, int K,
                     int c_out, const int32_t *__restrict__ nbr, int n_out, int rev, float *__restrict__ out,
                     const int32_t *__restrict__ n_out_dev) {
  after_previous();
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  __shared__ int rows[BM];
  int tid = threadIdx.x;
  int tx = tid & 15, ty = tid >> 4;
  int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int n_rows = live_rows(n_out, n_out_dev);
  if (m0 >= n_rows) return;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int kappa = 0; kappa < K; ++kappa) {
    int r = -1;
    if (tid < BM && m0 + tid < n_rows) r = nbr[(size_t)(rev ? K - 1 - kappa : kappa) * n_out + m0 + tid];
    __syncthreads();  // previous iteration finished reading rows/As/Bs
    if (tid < BM) rows[tid] = r;
    if (!__syncthreads_or(r >= 0)) continue;
    const float *wk = filters + (size_t)kappa * c_in * c_out;
    for (int kc = 0; kc < c_in; kc += BK) {
      {  // A tile: 64 rows x 16 channels, 4 consecutive channels per thread
        int m = tid >> 2, k4 = (tid & 3) * 4;
        int row = rows[m];
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (row >= 0) {
          const float *src = features + (size_t)row * c_in + kc + k4;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (kc + k4 + q < c_in) v[q] = __ldg(src + q);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) As[k4 + q][m] = v[q];
      }
      {  // B tile: 16 input channels x 64 output channels
        int k = tid >> 4, n4 = (tid & 15) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (kc + k < c_in) {
          const float *src = wk + (size_t)(kc + k) * c_out + n0 + n4;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (n0 + n4 + q < c_out) v[q] = __ldg(src + q);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) Bs[k][n4 + q] = v[q];
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        float a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx * 4 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int m = m0 + ty * 4 + i;
    if (m >= n_rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int n = n0 + tx * 4 + j;
      if (n < c_out) out[(size_t)m * c_out + n] = acc[i][j];
    }
  }
}

// The same sums for up to four input channels (a first layer on point features), in the same order: per output
// element fused multiply-adds over ascending offsets and channels, present neighbours only.  Two forms; fp32_by_lanes chooses.
//
// By lanes: a lane has an output row and CB of its channels, two to a register pair; the filters stand in shared memory, where all
// lanes read the same word at a time.  Table entries and input rows of nine offsets are in flight together.  Bound by what
// shared memory hands out, 16 bytes a lane for four multiply-adds: a warp runs through every offset that one of its 32 rows has.
// (215 k rows of 3 -> 36 channels, 6 neighbours a row: 58 us, by warps 94.  Two rows to a lane and zeros for absent
// neighbours: 92; three offsets in flight: 76; blocks of four warps, each with its copy of the filters: 71.)
constexpr int SM_WARPS = 8, SM_AHEAD = 9;
template <int CB>
__global__ void __launch_bounds__(SM_WARPS * 32)
conv_fwd_fp32_lanes_kernel(const float *__restrict__ features, int c_in, const float *__restrict__ filters, int K,
                           int c_out, const int32_t *__restrict__ nbr, int n_out, int rev, float *__restrict__ out,
                           const int32_t *__restrict__ n_out_dev) {
  after_previous();
  extern __shared__ __align__(16) float ws[];   // [K][c_in][CB]
  const int n_rows = live_rows(n_out, n_out_dev);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n0 = blockIdx.y * CB;
  if ((int)blockIdx.x * SM_WARPS * 32 >= n_rows) return;
  for (int i = threadIdx.x; i < K * c_in * CB; i += SM_WARPS * 32) {
    const int ch = i % CB, kc = i / CB;
    ws[i] = n0 + ch < c_out ? __ldg(filters + (size_t)kc * c_out + n0 + ch) : 0.f;
  }
  __syncthreads();
  const bool vec = (c_out & 3) == 0 && ((uintptr_t)out & 15u) == 0;
  for (int m0 = ((int)blockIdx.x * SM_WARPS + warp) * 32; m0 < n_rows; m0 += (int)gridDim.x * SM_WARPS * 32) {
    const int row = m0 + lane;
    f32x2 acc[CB / 2];
#pragma unroll
    for (int j = 0; j < CB / 2; ++j) acc[j] = 0ull;
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += SM_AHEAD) {
      int idx[SM_AHEAD];
      float x[SM_AHEAD][4];
#pragma unroll
      for (int i = 0; i < SM_AHEAD; ++i) {
        const int k = k0 + i;
        idx[i] = (k < K && row < n_rows) ? __ldg(nbr + (size_t)(rev ? K - 1 - k : k) * n_out + row) : -1;
      }
#pragma unroll
      for (int i = 0; i < SM_AHEAD; ++i) {
        const float *fp = features + (size_t)(idx[i] >= 0 ? idx[i] : 0) * c_in;
        if (c_in == 4) {
          const float4 f = idx[i] >= 0 ? __ldg((const float4 *)fp) : make_float4(0.f, 0.f, 0.f, 0.f);
          x[i][0] = f.x; x[i][1] = f.y; x[i][2] = f.z; x[i][3] = f.w;
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) x[i][c] = (c < c_in && idx[i] >= 0) ? __ldg(fp + c) : 0.f;
        }
      }
#pragma unroll
      for (int i = 0; i < SM_AHEAD; ++i) {
        if (idx[i] < 0) continue;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c >= c_in) break;
          const f32x2 xx = pair_of(x[i][c], x[i][c]);
          const ulonglong2 *w = (const ulonglong2 *)(ws + ((size_t)(k0 + i) * c_in + c) * CB);
#pragma unroll
          for (int j = 0; j < CB / 2; j += 2) {
            const ulonglong2 v = w[j / 2];
            acc[j] = fma_pair(xx, v.x, acc[j]);
            acc[j + 1] = fma_pair(xx, v.y, acc[j + 1]);
          }
        }
      }
    }
    if (row >= n_rows) continue;
    float *to = out + (size_t)row * c_out + n0;
#pragma unroll
    for (int j = 0; j < CB / 2; j += 2) {
      const int ch = n0 + 2 * j;
      const float2 a = halves(acc[j]), b = halves(acc[j + 1]);
      if (vec) {
        if (ch < c_out) *(float4 *)(to + 2 * j) = make_float4(a.x, a.y, b.x, b.y);
      } else {
        if (ch < c_out) to[2 * j] = a.x;
        if (ch + 1 < c_out) to[2 * j + 1] = a.y;
        if (ch + 2 < c_out) to[2 * j + 2] = b.x;
        if (ch + 3 < c_out) to[2 * j + 3] = b.y;
      }
    }
  }
}

// Channels of a lane, in how many passes over the rows.
struct LaneShape { int channels, passes; };
static LaneShape lane_shape(int c_out) {
  const int passes = ceil_div(c_out, 48);
  return {max((ceil_div(c_out, passes) + 7) & ~7, 16), passes};
}
static size_t lane_smem(int K, int c_in, int c_out) { return (size_t)K * c_in * lane_shape(c_out).channels * sizeof(float); }

// By lanes from as many rows as fill the SMs with work enough for a row; a form by warps has four times the blocks, and pays per
// neighbour where the other pays per offset, but as much for few channels as for 32.  `work`: multiply-adds of a row and offset by
// lanes, 40 more for a pass.  In us by warps / by lanes, 27 offsets, at 3, 6 and 12 neighbours a row:
//   1 -> 16 (work 16)    300 rows 7.8/6.9, 9.7/6.8, 12/7.2
//   3 -> 36 (120)        10 k 10/14, 12/15, 15/15; 20 k 12/14, 15/15, 19/15; 30 k 17/14, 21/15, 26/15; 100 k 37/30, 48/33, 58/34
//   4 -> 48 (192)        30 k 17/19, 21/19, 27/20; 60 k 25/30, 32/31, 40/32; 215 k 72/81, 95/84, 120/88
//   3 -> 64 (232)        60 k 25/35, 31/38, 39/41; 1 M 316/407, 418/438, 526/484   (27 neighbours: 843/615)
//   3 -> 92 (328)        60 k 30/47, 39/50, 48/54; 1 M 394/546, 515/577, 648/624   (27 neighbours: 1023/763)
// Tables that have fewer than three neighbours a row for their sizes alone (a layer that spreads few rows) are for warps from work 150
// on (4 -> 48, 100 k rows, 1.5 neighbours: 28/39).  Filters beyond 100 KB leave no two blocks on an SM: by warps, through L1.
static bool fp32_by_lanes(int n_in, int c_in, int K, int c_out, int n_out) {
  const LaneShape s = lane_shape(c_out);
  const long long work = (long long)c_in * s.channels * s.passes + 40 * (s.passes - 1);
  const bool sparse = (long long)K * n_in < 3LL * n_out;
  return lane_smem(K, c_in, c_out) <= 100 * 1024 && work <= (sparse ? 150 : 200) && n_out >= 350 * (work - 48);
}

template <int CB>
static int launch_fp32_lanes(const float *features, int c_in, const float *filters, int K, int c_out, const int32_t *nbr, int n_out,
                             int rev, float *out, const int32_t *n_out_dev, cudaStream_t st) {
  const size_t smem = (size_t)K * c_in * CB * sizeof(float);
  const int blocks = ceil_div(n_out, SM_WARPS * 32), most = sm_count() * 2;
  const dim3 grid(blocks < most ? blocks : most, ceil_div(c_out, CB));
  auto kernel = conv_fwd_fp32_lanes_kernel<CB>;
  if (smem > 48 * 1024) {
    cudaError_t e = allow_smem((const void *)kernel, smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd(fp32): smem attribute: %s", cudaGetErrorString(e));
  }
  { launch_ready(kernel, grid, dim3(SM_WARPS * 32), smem, st, features, c_in, filters, K, c_out, nbr, n_out, rev, out, n_out_dev); note_launches(1); }
  SSC_CHECK_LAUNCH("conv_fwd_fp32");
  return SSC_OK;
}

// By warps: a warp takes eight output rows at a time; lanes hold NJ output channels each (lane, lane + 32, ...), the
// filters stand in shared memory.  All 28 x 8 table entries of a pass, then all present input rows, are
// loaded at once, a lane per (offset, row); they reach the other lanes by shuffles.  Bound by instruction
// issue (about 200 per row of 6 neighbours and 64 channels).  The tiled kernel above pads the
// channels to 16 and multiplies absent rows: 399 us for 215 k rows of 3 -> 48 channels.
// (Four lanes to a row with their own channels, rows handed round by shuffles: 1.1 to 1.6 times as long, every lane reads its filters.)
constexpr int SM_GROUP = 8;
template <int NJ, bool STAGED>
__global__ void __launch_bounds__(SM_WARPS * 32)
conv_fwd_fp32_warps_kernel(const float *__restrict__ features, int c_in, const float *__restrict__ filters, int K,
                           int c_out, const int32_t *__restrict__ nbr, int n_out, int rev, float *__restrict__ out,
                           const int32_t *__restrict__ n_out_dev) {
  after_previous();
  extern __shared__ float ws[];               // [K][c_in][NJ * 32]
  const int n_rows = live_rows(n_out, n_out_dev);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n0 = blockIdx.y * NJ * 32;
  if (STAGED) {
    for (int i = threadIdx.x; i < K * c_in * NJ * 32; i += SM_WARPS * 32) {
      const int ch = i % (NJ * 32), kc = i / (NJ * 32);
      ws[i] = n0 + ch < c_out ? __ldg(filters + (size_t)kc * c_out + n0 + ch) : 0.f;
    }
    __syncthreads();
  }
  for (int m0 = ((int)blockIdx.x * SM_WARPS + warp) * SM_GROUP; m0 < n_rows; m0 += (int)gridDim.x * SM_WARPS * SM_GROUP) {
    float acc[SM_GROUP][NJ];
#pragma unroll
    for (int r = 0; r < SM_GROUP; ++r)
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[r][j] = 0.f;
    const int my_row = m0 + (lane & 7);
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += 28) {
      int idx[7];
      float x[7][4];
#pragma unroll
      for (int t = 0; t < 7; ++t) {            // entry (offset k0 + 4 t + lane / 8, row lane % 8)
        const int k = k0 + 4 * t + (lane >> 3);
        idx[t] = (k < K && my_row < n_rows) ? __ldg(nbr + (size_t)(rev ? K - 1 - k : k) * n_out + my_row) : -1;
      }
#pragma unroll
      for (int t = 0; t < 7; ++t) {
        const float *fp = features + (size_t)(idx[t] >= 0 ? idx[t] : 0) * c_in;
        if (c_in == 4) {
          const float4 f = idx[t] >= 0 ? __ldg((const float4 *)fp) : make_float4(0.f, 0.f, 0.f, 0.f);
          x[t][0] = f.x; x[t][1] = f.y; x[t][2] = f.z; x[t][3] = f.w;
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) x[t][c] = (c < c_in && idx[t] >= 0) ? __ldg(fp + c) : 0.f;
        }
      }
#pragma unroll
      for (int t = 0; t < 7; ++t) {
        const unsigned have = __ballot_sync(0xffffffffu, idx[t] >= 0);
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          const unsigned m = (have >> (8 * q)) & 255u;
          if (m == 0u) continue;
          const int k = k0 + 4 * t + q;
          float w[4][NJ];
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              if (STAGED) w[c][j] = c < c_in ? ws[((size_t)k * c_in + c) * (NJ * 32) + j * 32 + lane] : 0.f;
              else w[c][j] = (c < c_in && n0 + j * 32 + lane < c_out) ? __ldg(filters + ((size_t)k * c_in + c) * c_out + n0 + j * 32 + lane) : 0.f;
            }
#pragma unroll
          for (int r = 0; r < SM_GROUP; ++r) {
            if (!((m >> r) & 1u)) continue;    // the same for the whole warp
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float xv = __shfl_sync(0xffffffffu, x[t][c], 8 * q + r);
              if (c < c_in) {
#pragma unroll
                for (int j = 0; j < NJ; ++j) acc[r][j] = fmaf(xv, w[c][j], acc[r][j]);
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < SM_GROUP; ++r) {
      if (m0 + r >= n_rows) break;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int ch = n0 + j * 32 + lane;
        if (ch < c_out) out[(size_t)(m0 + r) * c_out + ch] = acc[r][j];
      }
    }
  }
}

template <int NJ>
static int launch_fp32_warps(const float *features, int c_in, const float *filters, int K, int c_out, const int32_t *nbr, int n_out,
                             int rev, float *out, const int32_t *n_out_dev, cudaStream_t st) {
  const size_t smem = (size_t)K * c_in * NJ * 32 * sizeof(float);
  const bool staged = smem <= 100 * 1024;     // two blocks per SM at least; larger filter sets are read through L1
  const int blocks = ceil_div(n_out, SM_WARPS * SM_GROUP), most = sm_count() * 3;
  const dim3 grid(blocks < most ? blocks : most, ceil_div(c_out, NJ * 32));
  auto kernel = staged ? conv_fwd_fp32_warps_kernel<NJ, true> : conv_fwd_fp32_warps_kernel<NJ, false>;
  if (staged && smem > 48 * 1024) {
    cudaError_t e = allow_smem((const void *)kernel, smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd(fp32): smem attribute: %s", cudaGetErrorString(e));
  }
  { launch_ready(kernel, grid, dim3(SM_WARPS * 32), staged ? smem : 0, st, features, c_in, filters, K, c_out, nbr, n_out, rev, out, n_out_dev); note_launches(1); }
  SSC_CHECK_LAUNCH("conv_fwd_fp32");
  return SSC_OK;
}

}  // namespace ssc

using namespace ssc;

extern "C" int ssc_materialize(const float *weight, const float *basis, const int32_t *block_table,
                               int n_blocks_in, const int32_t *out_field, const int32_t *in_field, int c_out,
                               int c_in, int K, float *filters, void *stream) {
  SSC_REQUIRE(c_out > 0 && c_in > 0 && K > 0 && n_blocks_in > 0, "materialize: bad sizes");
  SSC_REQUIRE(weight && basis && block_table && out_field && in_field && filters, "materialize: null pointer");
  long long total = (long long)K * c_in * c_out;
  { launch_ready(materialize_kernel, dim3(ceil_div(total, 256)), dim3(256), 0, as_stream(stream), weight, basis, block_table, n_blocks_in,
                                                                         out_field, in_field, c_out, c_in, K, filters); note_launches(1); }
  SSC_CHECK_LAUNCH("materialize");
  return SSC_OK;
}

extern "C" int ssc_materialize_bwd(const float *d_filters, const float *basis, const int32_t *block_table, int n_blocks_in,
                                   const int32_t *out_field, const int32_t *in_field, const int32_t *out_start, int n_out,
                                   const int32_t *in_start, int n_in, int max_pair, int c_out, int c_in, int K,
                                   float *d_weight, void *stream) {
  SSC_REQUIRE(c_out > 0 && c_in > 0 && K > 0 && n_blocks_in > 0 && n_out > 0 && n_in > 0 && n_out <= 65535 && max_pair > 0, "materialize_bwd: bad sizes");
  SSC_REQUIRE(d_filters && basis && block_table && out_field && in_field && out_start && in_start && d_weight, "materialize_bwd: null pointer");
  // a field pair that does not fit shared memory (very high orders with large kernels) is read in place
  const size_t need = (size_t)K * max_pair * sizeof(float);
  const int staged = need <= 200 * 1024 ? 1 : 0;
  if (staged && need > 48 * 1024) {
    cudaError_t e = allow_smem((const void *)materialize_bwd_kernel, need);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "materialize_bwd: smem attribute: %s", cudaGetErrorString(e));
  }
  { launch_ready(materialize_bwd_kernel, dim3(n_in, n_out), dim3(kMatBwdThreads), staged ? need : 0, as_stream(stream), 
        d_filters, basis, block_table, n_blocks_in, out_field, in_field, out_start, in_start, c_out, c_in, K, staged, d_weight); note_launches(1); }
  SSC_CHECK_LAUNCH("materialize_bwd");
  return SSC_OK;
}

extern "C" size_t ssc_conv_scratch_bytes(int n_in, int c_in, int c_out, int precision) {
  if (n_in < 0 || c_in < 1 || c_out < 1) return 0;
  (void)c_out;
  if (precision == SSC_PREC_F16 || precision == SSC_PREC_BF16) return conv_f16_scratch_bytes(n_in, c_in);
  if (precision != SSC_PREC_TF32) return 0;
  return conv_tf32_scratch_bytes(n_in, c_in);
}

extern "C" int ssc_conv_stage(const float *features, int n_in, int c_in, int precision, void *scratch, size_t scratch_bytes,
                              void *stream) {
  SSC_REQUIRE(c_in > 0 && n_in >= 0 && (n_in == 0 || features) && scratch, "conv_stage: bad arguments");
  SSC_REQUIRE(precision == SSC_PREC_TF32 || precision == SSC_PREC_F16 || precision == SSC_PREC_BF16, "conv_stage: precision %d has no staged image", precision);
  SSC_REQUIRE(scratch_bytes + 16 >= ssc_conv_scratch_bytes(n_in, c_in, 1, precision) && ((uintptr_t)scratch & 15u) == 0,
              "conv_stage: scratch too small or not 16-byte aligned");
  return precision == SSC_PREC_TF32 ? stage_features(features, n_in, c_in, scratch, as_stream(stream))
                                    : stage_features_16(features, n_in, c_in, precision == SSC_PREC_BF16, scratch, as_stream(stream));
}

extern "C" int ssc_conv_fwd_ordered(const float *features, int n_in, int c_in, const void *filters, int K, int c_out,
                                    const int32_t *nbr, int n_out, int precision, float *out, int32_t *status,
                                    void *scratch, size_t scratch_bytes, const int32_t *n_out_dev,
                                    const int32_t *row_order, void *stream) {
  SSC_REQUIRE(c_in > 0 && c_out > 0 && K > 0 && n_in >= 0 && n_out >= 0, "conv_fwd: bad sizes");
  const bool prestaged = (precision & SSC_CONV_PRESTAGED) != 0;
  const int table_form = precision & (SSC_CONV_TABLE_IN_ORDER | SSC_CONV_TABLE_REVERSED);
  precision &= ~(SSC_CONV_PRESTAGED | SSC_CONV_TABLE_IN_ORDER | SSC_CONV_TABLE_REVERSED);
  if (n_out == 0) return SSC_OK;
  SSC_REQUIRE(filters && nbr && out && (n_in == 0 || features || prestaged), "conv_fwd: null pointer");
  SSC_REQUIRE(!(table_form & SSC_CONV_TABLE_IN_ORDER) || (row_order && precision != SSC_PREC_FP32),
              "conv_fwd: SSC_CONV_TABLE_IN_ORDER needs a row order and a tensor-core precision");
  cudaStream_t st = as_stream(stream);
  if (precision == SSC_PREC_FP32) {
    if (c_in <= 4 && (c_in != 4 || ((uintptr_t)features & 15u) == 0)) {
      const int rev = table_form != 0;
      const float *w = (const float *)filters;
      if (fp32_by_lanes(n_in, c_in, K, c_out, n_out)) {
        switch (lane_shape(c_out).channels) {
          case 16: return launch_fp32_lanes<16>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
          case 24: return launch_fp32_lanes<24>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
          case 32: return launch_fp32_lanes<32>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
          case 40: return launch_fp32_lanes<40>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
          default: return launch_fp32_lanes<48>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
        }
      }
      if (c_out <= 32) return launch_fp32_warps<1>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
      if (c_out <= 64) return launch_fp32_warps<2>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
      return launch_fp32_warps<3>(features, c_in, w, K, c_out, nbr, n_out, rev, out, n_out_dev, st);
    }
    dim3 grid(ceil_div(n_out, BM), ceil_div(c_out, BN));
    { launch_ready(conv_fwd_fp32_kernel, dim3(grid), dim3(256), 0, st, features, c_in, (const float *)filters, K, c_out, nbr, n_out, table_form != 0, out, n_out_dev); note_launches(1); }
    SSC_CHECK_LAUNCH("conv_fwd_fp32");
    return SSC_OK;
  }
  if (precision == SSC_PREC_TF32) return conv_fwd_tf32(features, n_in, c_in, filters, K, c_out, nbr, n_out, out, status, scratch, scratch_bytes, n_out_dev, row_order, prestaged, table_form, GateEpilogue{}, st);
  if (precision == SSC_PREC_F16 || precision == SSC_PREC_BF16)
    return conv_fwd_16(features, n_in, c_in, precision == SSC_PREC_BF16, filters, K, c_out, nbr, n_out, out, status, scratch, scratch_bytes, n_out_dev, row_order, prestaged, table_form, GateEpilogue{}, st);
  return fail(SSC_ERR_INVALID, "conv_fwd: unknown precision %d", precision);
}

extern "C" int ssc_conv_gate_covered(int c_in, int c_out, int c_keep, int precision, int n_out) {
  return conv_gate_covered(c_in, c_out, c_keep, precision, n_out) ? 1 : 0;
}

extern "C" int ssc_conv_fwd_gated(const float *features, int n_in, int c_in, const void *filters, int K, int c_out,
                                  const int32_t *nbr, int n_out, int precision, const float *scale, const float *shift,
                                  const int32_t *gate_of_channel, int c_keep, int scalar_act, int gate_act, int out_precision,
                                  void *out, int32_t *status, void *scratch, size_t scratch_bytes, const int32_t *n_out_dev,
                                  const int32_t *row_order, void *stream) {
  SSC_REQUIRE(c_in > 0 && c_out > 0 && K > 0 && n_in >= 0 && n_out >= 0, "conv_fwd_gated: bad sizes");
  const bool prestaged = (precision & SSC_CONV_PRESTAGED) != 0;
  precision &= ~SSC_CONV_PRESTAGED;
  SSC_REQUIRE(conv_gate_covered(c_in, c_out, c_keep, precision, n_out), "conv_fwd_gated: %d -> %d (%d kept) channels at precision %d are not covered", c_in, c_out, c_keep, precision);
  SSC_REQUIRE(out_precision == SSC_PREC_FP32 || ((out_precision == SSC_PREC_F16 || out_precision == SSC_PREC_BF16) && c_keep % 8 == 0),
              "conv_fwd_gated: rows of %d channels cannot be stored at precision %d", c_keep, out_precision);
  if (n_out == 0) return SSC_OK;
  SSC_REQUIRE(filters && nbr && out && scratch && gate_of_channel && (scale == nullptr) == (shift == nullptr) && (n_in == 0 || features || prestaged),
              "conv_fwd_gated: null pointer");
  const GateEpilogue gate = {scale, shift, gate_of_channel, c_keep, scalar_act, gate_act,
                             out_precision == SSC_PREC_F16 ? 1 : out_precision == SSC_PREC_BF16 ? 2 : 0};
  if (precision == SSC_PREC_TF32)
    return conv_fwd_tf32(features, n_in, c_in, filters, K, c_out, nbr, n_out, (float *)out, status, scratch, scratch_bytes, n_out_dev, row_order, prestaged, 0, gate, as_stream(stream));
  return conv_fwd_16(features, n_in, c_in, precision == SSC_PREC_BF16, filters, K, c_out, nbr, n_out, (float *)out, status, scratch, scratch_bytes, n_out_dev, row_order, prestaged, 0, gate, as_stream(stream));
}

extern "C" int ssc_conv_fwd(const float *features, int n_in, int c_in, const void *filters, int K, int c_out,
                            const int32_t *nbr, int n_out, int precision, float *out, int32_t *status,
                            void *scratch, size_t scratch_bytes, const int32_t *n_out_dev, void *stream) {
  return ssc_conv_fwd_ordered(features, n_in, c_in, filters, K, c_out, nbr, n_out, precision, out, status, scratch,
                              scratch_bytes, n_out_dev, nullptr, stream);
}
