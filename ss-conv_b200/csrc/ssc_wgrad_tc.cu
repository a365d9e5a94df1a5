// Filter gradient of the sparse convolution.
//
//   dW[kappa][ci][co] = sum over output rows o with a neighbour i = nbr[kappa][o]:  x[i][ci] * dy[o][co]
//
// The (output row, input row) pairs of every kernel offset are first compacted into lists (a
// bitmap of the neighbour table, a popcount scan, a scatter: ascending output row inside an
// offset, so the lists - and the sums below - are repeatable); rows without a neighbour, more
// than half of the table of a strided convolution, then cost nothing.
//
// The lists differ in length by orders of magnitude (the centre of a submanifold layer holds every
// row, a corner a few of them), so the work is cut by pairs, not by offsets: the chunks of 32 pairs of
// all offsets stand in one row and every CTA takes an equal share of it.  Where a share crosses into
// another offset the sums so far are written out as a partial tile and start again; the partial of
// (share b, offset kappa) has place b + kappa, which no other pair takes because both only grow
// along the row.  wgrad_reduce_kernel adds the partials of an offset in ascending order of shares:
// bitwise repeatable.  (One CTA range per offset: 237 us on 61 k surface voxels, 64 -> 76 channels, of
// which the centre offset alone kept ten CTAs busy.)
//
// conv_wgrad_tc_kernel (TF32 operands, tcgen05): a CTA accumulates D[co][ci] (M = 128 rows = output channels
// of one block of 128, N = input channels) in tensor memory; K = pairs, 32 per chunk.  Both operands have
// to be K-major, i.e. transposed with respect to how the rows lie in memory, so the producer warps
// transpose on the way into shared memory: lane = pair of the chunk; for every channel the 32 lanes
// store 32 consecutive K elements of that channel's operand row (one conflict-free 128-byte store, in the
// 128-byte-swizzled layout), rounded to TF32; lanes past the end of a list store zeros.  Operand rows of
// channels past c_out / c_in are zeroed once and never touched again.
//   warps 0-7: producers, two per ring slot (dy rows and x rows), indices one chunk ahead
//   warp 8: tensor-memory allocation and the MMA-issuing thread
//   warps 9-12: write finished partials (two accumulator buffers where tensor memory allows, so that
//   the next offset's sums run meanwhile)
// conv_wgrad_small_kernel (exact fp32, up to 16 input channels): a warp is a share, lanes = output channels.
// Every wait is bounded (status bit 16 on expiry).
#include "ssc_conv_internal.cuh"
#include "ssc_scan.cuh"
#include "ssc_tc_ptx.cuh"

namespace ssc {

constexpr int WT_M = 128;          // output channels per CTA
constexpr int WT_K = 32;           // output rows per chunk
constexpr int WT_STAGES = 4;
constexpr int WT_A_BYTES = WT_M * 128;
constexpr int WT_PRODUCERS = 2 * WT_STAGES;
constexpr int WT_MMA_WARP = WT_PRODUCERS;
constexpr int WT_THREADS = (WT_PRODUCERS + 1 + 4) * 32;

// One warp per 32 output rows of one kernel offset: which of them have a neighbour.
__global__ void pair_bitmap_kernel(const int32_t *__restrict__ nbr, int K, int n_out, int words_per_row,
                                   uint32_t *__restrict__ bitmap) {
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (gw >= (long long)K * words_per_row) return;
  const int kappa = (int)(gw / words_per_row), r = (int)(gw % words_per_row) * 32 + (int)(threadIdx.x & 31);
  const bool have = r < n_out && __ldg(nbr + (size_t)kappa * n_out + r) >= 0;
  const unsigned m = __ballot_sync(0xffffffffu, have);
  if ((threadIdx.x & 31) == 0) bitmap[gw] = m;
}
// prefix[w] = number of pairs before word w (over all offsets): the lists of the offsets follow one
// another in pair_out / pair_in, starts[kappa] is where the list of offset kappa begins.
__global__ void pair_scatter_kernel(const int32_t *__restrict__ nbr, int K, int n_out, int words_per_row,
                                    const uint32_t *__restrict__ bitmap, const uint32_t *__restrict__ prefix,
                                    int32_t *__restrict__ pair_out, int32_t *__restrict__ pair_in, int32_t *__restrict__ starts) {
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (gw >= (long long)K * words_per_row) return;
  const int lane = threadIdx.x & 31;
  const int kappa = (int)(gw / words_per_row), w = (int)(gw % words_per_row), r = w * 32 + lane;
  const uint32_t m = bitmap[gw], base = prefix[gw];
  if (w == 0 && lane == 0) starts[kappa] = (int32_t)base;
  if ((m >> lane) & 1u) {
    const uint32_t pos = base + (uint32_t)__popc(m & ((1u << lane) - 1u));
    pair_out[pos] = r;
    pair_in[pos] = __ldg(nbr + (size_t)kappa * n_out + r);
  }
}

__device__ __forceinline__ uint32_t wt_off(int row, int k) {  // byte offset of element (row, k) of a K-major SW128 tile
  return (uint32_t)(row >> 3) * 1024u + (uint32_t)(row & 7) * 128u + ((((uint32_t)k >> 2) ^ (uint32_t)(row & 7)) << 4) +
         ((uint32_t)k & 3u) * 4u;
}

// ---------------------------------------------------------------- shares of the row of chunks
// first[kappa] = chunks before offset kappa, for all K + 1 values, in shared memory (blockDim.x >= 32).
__device__ __forceinline__ void chunk_prefix(const int32_t *__restrict__ starts, int K, int *first) {
  if (threadIdx.x < 32) {
    int run = 0;
    for (int k0 = 0; k0 < K; k0 += 32) {
      const int k = k0 + (int)threadIdx.x;
      int v = k < K ? (starts[k + 1] - starts[k] + WT_K - 1) / WT_K : 0, incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += u;
      }
      if (k < K) first[k] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) first[K] = run;
  }
  __syncthreads();
}
__device__ __forceinline__ int share_begin(int b, int total, int shares) { return (int)((long long)b * total / shares); }
// the share that chunk q belongs to
__device__ __forceinline__ int share_of(int q, int total, int shares) {
  int b = (int)((long long)q * shares / total);
  while (b + 1 < shares && share_begin(b + 1, total, shares) <= q) ++b;
  while (b > 0 && share_begin(b, total, shares) > q) --b;
  return b;
}

__global__ void __launch_bounds__(WT_THREADS)
conv_wgrad_tc_kernel(const float *__restrict__ features, int c_in, const float *__restrict__ out_grad, int c_out,
                     const int32_t *__restrict__ pair_out, const int32_t *__restrict__ pair_in,
                     const int32_t *__restrict__ starts, int K, int n_pad, uint32_t buf_cols, int n_buf,
                     float *__restrict__ partial, int32_t *status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int first[257];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int b_bytes = n_pad * 128;
  const int stage_bytes = WT_A_BYTES + b_bytes;
  uint8_t *ctrl = smem + (size_t)WT_STAGES * stage_bytes;
  uint64_t *full_bars = (uint64_t *)ctrl;                  // [WT_STAGES]
  uint64_t *empty_bars = full_bars + WT_STAGES;            // [WT_STAGES]
  uint64_t *accf_bars = empty_bars + WT_STAGES;            // [2] a partial is complete
  uint64_t *acce_bars = accf_bars + 2;                     // [2] and has been read out
  uint64_t *done_bar = acce_bars + 2;
  uint32_t *tmem_slot = (uint32_t *)(done_bar + 1);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int co0 = blockIdx.y * WT_M;
  if (tid == 0) {
    for (int s = 0; s < WT_STAGES; ++s) {
      mbar_init(smem_u32(full_bars + s), 64);
      mbar_init(smem_u32(empty_bars + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(accf_bars + b), 1);
      mbar_init(smem_u32(acce_bars + b), 4);
    }
    mbar_init(smem_u32(done_bar), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WT_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(buf_cols * (uint32_t)n_buf)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // operand rows of channels that do not exist stay zero for the whole kernel
  for (int i = tid; i < WT_STAGES * stage_bytes / 16; i += WT_THREADS) ((uint4 *)smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_async_smem();
  chunk_prefix(starts, K, first);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t smem_base = smem_u32(smem);
  const int m_cnt = min(WT_M, c_out - co0);   // output channels of this CTA
  const int total = first[K];
  const int q_begin = share_begin((int)blockIdx.x, total, (int)gridDim.x), q_end = share_begin((int)blockIdx.x + 1, total, (int)gridDim.x);
  int kappa0 = 0;                             // the offset the share begins in
  while (kappa0 + 1 < K && first[kappa0 + 1] <= q_begin) ++kappa0;

  if (warp < WT_PRODUCERS) {
    // ====================================== producers ========================================
    // Chunk q uses ring slot (q - q_begin) % WT_STAGES; warps 2s and 2s + 1 serve slot s: the first brings
    // the dy rows (operand A), the second the x rows (operand B).
    const int slot = warp >> 1, part = warp & 1;
    uint32_t par = 0;
    uint8_t *tile = smem + (size_t)slot * stage_bytes + (part ? WT_A_BYTES : 0);
    const bool vec = ((c_in | c_out) & 3) == 0 && (((uintptr_t)features | (uintptr_t)out_grad) & 15u) == 0;
    const int32_t *list = part ? pair_in : pair_out;
    const float *rows = part ? features : out_grad + co0;
    const int width = part ? c_in : c_out, n_ch = part ? c_in : m_cnt;
    int kappa = kappa0;
    auto row_of = [&](int q) -> int {          // this lane's row of chunk q, or -1
      if (q >= q_end) return -1;
      while (first[kappa + 1] <= q) ++kappa;
      const int j = __ldg(starts + kappa) + (q - first[kappa]) * WT_K + lane;
      return j < __ldg(starts + kappa + 1) ? __ldg(list + j) : -1;
    };
    int next = row_of(q_begin + slot);
    for (int q = q_begin + slot; q < q_end; q += WT_STAGES) {
      const int row = next;
      next = row_of(q + WT_STAGES);
      const bool valid = row >= 0;
      const float *g = rows + (size_t)(valid ? row : 0) * width;
      bool waited = q < q_begin + WT_STAGES, ok = true;
      if (vec) {
        // 32 channels at a time: eight independent 16-byte loads in flight, then 32 transposed stores
        for (int c0 = 0; c0 < n_ch && ok; c0 += 32) {
          float4 v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            v[k] = (valid && c0 + k * 4 < n_ch) ? __ldg((const float4 *)(g + c0 + k * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
          if (!waited) {      // the slot is needed only now, with the first loads on their way
            ok = mbar_wait_warp(smem_u32(empty_bars + slot), par ^ 1u, abort_flag);
            tc_fence_after();
            waited = true;
            if (!ok) break;
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int c = c0 + k * 4;
            if (c < n_ch) {
              *(uint32_t *)(tile + wt_off(c + 0, lane)) = to_tf32(v[k].x);
              *(uint32_t *)(tile + wt_off(c + 1, lane)) = to_tf32(v[k].y);
              *(uint32_t *)(tile + wt_off(c + 2, lane)) = to_tf32(v[k].z);
              *(uint32_t *)(tile + wt_off(c + 3, lane)) = to_tf32(v[k].w);
            }
          }
        }
      } else {
        if (!waited) {
          ok = mbar_wait_warp(smem_u32(empty_bars + slot), par ^ 1u, abort_flag);
          tc_fence_after();
        }
        for (int c0 = 0; c0 < n_ch && ok; c0 += 8) {
          float v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = (valid && c0 + k < n_ch) ? __ldg(g + c0 + k) : 0.f;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (c0 + k < n_ch) *(uint32_t *)(tile + wt_off(c0 + k, lane)) = to_tf32(v[k]);
        }
      }
      if (!ok) break;
      fence_async_smem();
      mbar_arrive(smem_u32(full_bars + slot));
      par ^= 1u;
    }
  } else if (warp == WT_MMA_WARP) {
    // ====================================== MMA issuer =======================================
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n_pad >> 3) << 17) | ((uint32_t)(WT_M >> 4) << 24);
      int kappa = kappa0, seg = 0;
      bool alive = true;
      uint32_t s = 0, par = 0;
      for (int q = q_begin; q < q_end && alive;) {
        while (first[kappa + 1] <= q) ++kappa;
        const int stop = min(q_end, first[kappa + 1]), buf = seg % n_buf, use = seg / n_buf;
        if (use > 0) {
          if (!mbar_wait(smem_u32(acce_bars + buf), (uint32_t)(use - 1) & 1u, abort_flag)) break;
          tc_fence_after();
        }
        const uint32_t d = tmem_base + (uint32_t)buf * buf_cols;
        for (const int q0 = q; q < stop; ++q) {
          if (!mbar_wait(smem_u32(full_bars + s), par, abort_flag)) { alive = false; break; }
          tc_fence_after();
          const uint32_t a_lo = desc_lo(smem_base + s * (uint32_t)stage_bytes);
          const uint32_t b_lo = desc_lo(smem_base + s * (uint32_t)stage_bytes + WT_A_BYTES);
          mma_tf32_ss(d, a_lo, b_lo, idesc, q > q0 ? 1u : 0u);
          mma_tf32_ss(d, a_lo + 2u, b_lo + 2u, idesc, 1u);
          mma_tf32_ss(d, a_lo + 4u, b_lo + 4u, idesc, 1u);
          mma_tf32_ss(d, a_lo + 6u, b_lo + 6u, idesc, 1u);
          mma_commit(smem_u32(empty_bars + s));
          if (++s == WT_STAGES) { s = 0; par ^= 1u; }
        }
        if (alive) mma_commit(smem_u32(accf_bars + buf));
        ++seg;
      }
      // everything issued above (on any path) retires before the tensor memory is handed back
      mma_commit(smem_u32(done_bar));
      mbar_wait_drain(smem_u32(done_bar), 0u);
    }
  } else {
    // ====================================== epilogue ===========================================
    const int quarter = warp & 3;
    const int co = co0 + quarter * 32 + lane;
    int kappa = kappa0, seg = 0;
    for (int q = q_begin; q < q_end; ++seg) {
      while (first[kappa + 1] <= q) ++kappa;
      q = min(q_end, first[kappa + 1]);
      const int buf = seg % n_buf;
      if (!mbar_wait_warp_backoff(smem_u32(accf_bars + buf), (uint32_t)(seg / n_buf) & 1u, abort_flag, 64)) break;
      tc_fence_after();
      float *dst = partial + ((size_t)blockIdx.x + kappa) * (size_t)c_in * c_out;
      for (int c0 = 0; c0 < n_pad; c0 += 16) {
        uint32_t v[16];
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * buf_cols + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (co < c_out) {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (c0 + k < c_in) dst[(size_t)(c0 + k) * c_out + co] = __uint_as_float(v[k]);  // lanes = consecutive co: coalesced
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(acce_bars + buf));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag && status) atomicOr(status, 16);
  if (warp == WT_MMA_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(buf_cols * (uint32_t)n_buf) : "memory");
  }
}

// Exact fp32, up to 16 input channels (a first layer): a warp is a share; a lane holds the sums of one output
// channel (blockIdx.y = 32 of them) with all CMAX input channels in registers.  Per pair one coalesced load
// of dy and CMAX broadcast loads of x; eight pairs in flight.
template <int CMAX>
__global__ void __launch_bounds__(128)
conv_wgrad_small_kernel(const float *__restrict__ features, int c_in, const float *__restrict__ out_grad, int c_out,
                        const int32_t *__restrict__ pair_out, const int32_t *__restrict__ pair_in,
                        const int32_t *__restrict__ starts, int K, float *__restrict__ partial) {
  __shared__ int first[257];
  chunk_prefix(starts, K, first);
  const int lane = threadIdx.x & 31, co = blockIdx.y * 32 + lane;
  const int share = blockIdx.x * 4 + (threadIdx.x >> 5), shares = gridDim.x * 4;
  const int total = first[K], q_end = share_begin(share + 1, total, shares);
  int kappa = 0;
  for (int q = share_begin(share, total, shares); q < q_end;) {
    while (first[kappa + 1] <= q) ++kappa;
    const int stop = min(q_end, first[kappa + 1]), list0 = starts[kappa], n_pairs = starts[kappa + 1] - list0;
    float acc[CMAX];
#pragma unroll
    for (int c = 0; c < CMAX; ++c) acc[c] = 0.f;
    for (; q < stop; ++q) {
      const int j0 = (q - first[kappa]) * WT_K, j = j0 + lane;
      const int ro = j < n_pairs ? __ldg(pair_out + list0 + j) : 0, ri = j < n_pairs ? __ldg(pair_in + list0 + j) : 0;
      const int cnt = min(WT_K, n_pairs - j0);
#pragma unroll 8
      for (int k = 0; k < cnt; ++k) {
        const int o = __shfl_sync(0xffffffffu, ro, k), i = __shfl_sync(0xffffffffu, ri, k);
        const float g = co < c_out ? __ldg(out_grad + (size_t)o * c_out + co) : 0.f;
        const float *xp = features + (size_t)i * c_in;
#pragma unroll
        for (int c = 0; c < CMAX; ++c) acc[c] = fmaf(c < c_in ? __ldg(xp + c) : 0.f, g, acc[c]);
      }
    }
    if (co < c_out) {
      float *dst = partial + ((size_t)share + kappa) * (size_t)c_in * c_out + co;
#pragma unroll
      for (int c = 0; c < CMAX; ++c)
        if (c < c_in) dst[(size_t)c * c_out] = acc[c];
    }
  }
}

// d_filters[kappa] = sum of the offset's partials in ascending order of shares.  grid (elements / 256, K).
__global__ void __launch_bounds__(256)
wgrad_reduce_shares_kernel(const float *__restrict__ partial, const int32_t *__restrict__ starts, int K, int shares, int elems,
                           float *__restrict__ out) {
  __shared__ int first[257];
  chunk_prefix(starts, K, first);
  const int kappa = blockIdx.y, e = blockIdx.x * 256 + threadIdx.x, total = first[K];
  if (e >= elems) return;
  float s = 0.f;
  if (first[kappa + 1] > first[kappa]) {
    const int lo = share_of(first[kappa], total, shares), hi = share_of(first[kappa + 1] - 1, total, shares);
    const float *p = partial + ((size_t)lo + kappa) * elems + e;
#pragma unroll 8
    for (int b = lo; b <= hi; ++b, p += elems) s += share_begin(b + 1, total, shares) > share_begin(b, total, shares) ? __ldg(p) : 0.f;
  }
  out[(size_t)kappa * elems + e] = s;
}

size_t pair_lists_bytes(int K, int n_out) {
  const size_t wpr = (size_t)ceil_div(n_out > 0 ? n_out : 1, 32), words = (size_t)K * wpr;
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  return 2 * al(words * 4) + al((words / 1024 + 2) * 4) + 2 * al((size_t)K * n_out * 4) + al((size_t)(K + 1) * 4);
}

namespace {
struct ListPlan {
  uint32_t *bitmap, *prefix, *block_sums;
  int32_t *pair_out, *pair_in, *starts;
  int wpr;
  long long words;
};
ListPlan plan_lists(void *lists, int K, int n_out) {
  ListPlan p;
  p.wpr = ceil_div(n_out > 0 ? n_out : 1, 32);
  p.words = (long long)K * p.wpr;
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  uint8_t *sp = (uint8_t *)lists;
  p.bitmap = (uint32_t *)sp;
  sp += al((size_t)p.words * 4);
  p.prefix = (uint32_t *)sp;
  sp += al((size_t)p.words * 4);
  p.block_sums = (uint32_t *)sp;
  sp += al(((size_t)p.words / 1024 + 2) * 4);
  p.pair_out = (int32_t *)sp;
  sp += al((size_t)K * n_out * 4);
  p.pair_in = (int32_t *)sp;
  sp += al((size_t)K * n_out * 4);
  p.starts = (int32_t *)sp;
  return p;
}
}  // namespace

PairLists pair_lists_view(void *lists, int K, int n_out) {
  const ListPlan p = plan_lists(lists, K, n_out);
  return PairLists{p.pair_out, p.pair_in, p.starts};
}

// bitmap of the table, popcount scan, scatter: three small launches
int pair_lists_build(const int32_t *nbr, int K, int n_out, void *lists, PairLists *out, cudaStream_t st) {
  const ListPlan p = plan_lists(lists, K, n_out);
  { pair_bitmap_kernel<<<ceil_div(p.words * 32, 256), 256, 0, st>>>(nbr, K, n_out, p.wpr, p.bitmap); note_launches(1); }
  SSC_CHECK_LAUNCH("pair_bitmap");
  int rc = exclusive_scan_u32<true>(p.bitmap, p.words, p.prefix, p.block_sums, p.starts + K, nullptr, st);
  if (rc != 0) return rc;
  { pair_scatter_kernel<<<ceil_div(p.words * 32, 256), 256, 0, st>>>(nbr, K, n_out, p.wpr, p.bitmap, p.prefix, p.pair_out, p.pair_in, p.starts); note_launches(1); }
  SSC_CHECK_LAUNCH("pair_scatter");
  if (out) *out = PairLists{p.pair_out, p.pair_in, p.starts};
  return SSC_OK;
}

// Shapes and shares of the two list kernels.
struct WgradPlan {
  bool tc, small;
  int n_pad, n_buf, co_blocks, shares;
  uint32_t buf_cols;
  size_t smem;
};
static WgradPlan wgrad_plan(int K, int c_in, int c_out, int n_out, bool tf32) {
  WgradPlan p;
  memset(&p, 0, sizeof(p));
  // never more shares than the table could hold chunks
  const long long most = (long long)K * ceil_div(n_out > 0 ? n_out : 1, WT_K);
  if (tf32) {
    p.n_pad = (c_in + 15) & ~15;
    p.smem = (size_t)WT_STAGES * (WT_A_BYTES + p.n_pad * 128) + 1024 + 256;
    if (p.n_pad > 256 || p.smem > 227 * 1024) return p;
    p.tc = true;
    p.buf_cols = 32;
    while ((int)p.buf_cols < p.n_pad) p.buf_cols <<= 1;
    // two CTAs per SM (tensor memory: 512 columns) where their rings fit; two accumulator buffers each where the columns allow
    const int ctas = p.smem <= 112 * 1024 ? 2 : 1;
    p.n_buf = (int)p.buf_cols * 2 * ctas <= 512 ? 2 : 1;
    p.co_blocks = ceil_div(c_out, WT_M);
    p.shares = ctas * sm_count() / p.co_blocks;
  } else {
    if (c_in > 16) return p;
    p.small = true;
    p.co_blocks = ceil_div(c_out, 32);
    p.shares = 16 * sm_count();          // warps: four blocks of four per SM
  }
  if (p.shares > most) p.shares = (int)most;
  if (p.shares < 1) p.shares = 1;
  if (p.small) p.shares = ceil_div(p.shares, 4) * 4;
  return p;
}

size_t conv_wgrad_lists_partial_bytes(int K, int c_in, int c_out, int n_out, bool tf32) {
  const WgradPlan p = wgrad_plan(K, c_in, c_out, n_out, tf32);
  return (p.tc || p.small) ? (size_t)(p.shares + K) * c_in * c_out * sizeof(float) : 0;
}

// returns -1 when the shape is not covered (the caller then uses the CUDA-core kernel over the table)
int conv_wgrad_lists(const float *features, int c_in, const float *out_grad, int c_out, const PairLists &pl, int K, int n_out,
                     bool tf32, float *partial, float *d_filters, int32_t *status, cudaStream_t st) {
  const WgradPlan p = wgrad_plan(K, c_in, c_out, n_out, tf32);
  if (p.tc) {
    cudaError_t e = cudaFuncSetAttribute(conv_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_wgrad(tf32): smem attribute: %s", cudaGetErrorString(e));
    { conv_wgrad_tc_kernel<<<dim3(p.shares, p.co_blocks), WT_THREADS, p.smem, st>>>(features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in,
                                                                                  pl.starts, K, p.n_pad, p.buf_cols, p.n_buf, partial, status); note_launches(1); }
    SSC_CHECK_LAUNCH("conv_wgrad_tc");
  } else if (p.small) {
    const dim3 grid(p.shares / 4, p.co_blocks);
    if (c_in <= 4) { conv_wgrad_small_kernel<4><<<grid, 128, 0, st>>>(features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in, pl.starts, K, partial); note_launches(1); }
    else if (c_in <= 8) { conv_wgrad_small_kernel<8><<<grid, 128, 0, st>>>(features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in, pl.starts, K, partial); note_launches(1); }
    else { conv_wgrad_small_kernel<16><<<grid, 128, 0, st>>>(features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in, pl.starts, K, partial); note_launches(1); }
    SSC_CHECK_LAUNCH("conv_wgrad_small");
  } else {
    return -1;
  }
  const int elems = c_in * c_out;
  { wgrad_reduce_shares_kernel<<<dim3(ceil_div(elems, 256), K), 256, 0, st>>>(partial, pl.starts, K, p.shares, elems, d_filters); note_launches(1); }
  SSC_CHECK_LAUNCH("conv_wgrad_reduce");
  return SSC_OK;
}

}  // namespace ssc
