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
// conv_wgrad_tc_kernel (TF32 operands, tcgen05): a CTA accumulates D[co][ci] (or D[ci][co], see wgrad_plan; M = 128 rows = output channels
// of one block of 128, N = input channels) in tensor memory; K = pairs, 32 per chunk.  The rows go to
// shared memory as they lie in global memory (channels contiguous) and the tensor core takes both
// operands MN-major: 32 channels of a pair are one 128-byte line, pairs follow one another, the 32-byte
// pieces of line k are exchanged by XOR with k & 3 (swizzle mode "128 bytes with 32-byte atoms", the one
// the 32-bit formats have for this order).  Eight lanes fetch a line with 16-byte cp.async, so a gather
// costs one L1 line per 128 bytes; transposed on the way in (lane = pair, one 16-byte piece of 32 rows
// per instruction) it was bound by that at 32 lines per instruction.  Rows that are not rounded to
// TF32 yet are rounded in place once they have landed.  Pairs past the end of a list are zero rows;
// channels past c_out / c_in are whatever the buffer holds: they only reach rows and columns of D
// that nobody reads.
//   warps 0 .. 2 stages - 1: producers, two to a ring slot (gradients, inputs), pair indices one round ahead
//   the next warp: tensor-memory allocation and the MMA-issuing thread
//   four more: write finished partials (two accumulator buffers where tensor memory allows, so that
//   the next offset's sums run meanwhile)
// conv_wgrad_small_kernel (exact fp32, up to 16 input channels): a warp is a share, lanes = output channels.
// Every wait is bounded (status bit 16 on expiry).
#include "ssc_conv_internal.cuh"
#include "ssc_scan.cuh"
#include "ssc_tc_ptx.cuh"

namespace ssc {

constexpr int WT_M = 128;          // output channels per CTA
constexpr int WT_K = 32;           // pairs per chunk
constexpr int WT_MAX_STAGES = 8;   // of a CTA by itself on its SM; two of 15 warps with 64 registers a thread fit one: 5 each
constexpr int wt_stages(int ctas) { return ctas == 2 ? 5 : WT_MAX_STAGES; }
constexpr int WT_BLOCK = WT_K * 128;   // 32 channels of a chunk's pairs

// Which output rows have a neighbour: a warp makes four words (128 rows) of one kernel offset (blockIdx.y), four
// loads in flight per lane.  HBM-bound: the table is read once.
__global__ void __launch_bounds__(256)
pair_bitmap_kernel(const int32_t *__restrict__ nbr, int n_out, int words_per_row, uint32_t *__restrict__ bitmap) {
  after_previous();
  const int w0 = ((int)blockIdx.x * 8 + (int)(threadIdx.x >> 5)) * 4, lane = threadIdx.x & 31;
  if (w0 >= words_per_row) return;
  const int32_t *row = nbr + (size_t)blockIdx.y * n_out;
  int v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = (w0 + i) * 32 + lane;
    v[i] = r < n_out ? __ldg(row + r) : -1;
  }
  uint32_t mine = 0u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const unsigned m = __ballot_sync(0xffffffffu, v[i] >= 0);
    if (lane == i) mine = m;
  }
  if (lane < 4 && w0 + lane < words_per_row) bitmap[(size_t)blockIdx.y * words_per_row + w0 + lane] = mine;
}
// prefix[w] = number of pairs before word w (over all offsets): the lists of the offsets follow one
// another in pair_out / pair_in, starts[kappa] is where the list of offset kappa begins.  A warp takes 32
// words: every lane lists the set bits of its word in shared memory, then the warp copies the list out, loads in flight
// and stores side by side (a lane that writes its own word's pairs one after the other: 52 to 83 us for the
// 22 M entries of a 5^3 layer of 177 k rows; a warp per word 96 us).
__global__ void __launch_bounds__(256)
pair_scatter_kernel(const int32_t *__restrict__ nbr, int n_out, int words_per_row,
                    const uint32_t *__restrict__ bitmap, const uint32_t *__restrict__ prefix,
                    int32_t *__restrict__ pair_out, int32_t *__restrict__ pair_in, int32_t *__restrict__ starts) {
  after_previous();
  __shared__ uint16_t list_s[8][1024];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kappa = blockIdx.y;
  const int w0 = ((int)blockIdx.x * 8 + warp) * 32, w = w0 + lane;
  if (w0 >= words_per_row) return;
  uint16_t *list = list_s[warp];
  const bool in = w < words_per_row;
  uint32_t m = in ? __ldg(bitmap + (size_t)kappa * words_per_row + w) : 0u;
  const uint32_t pos = __ldg(prefix + (size_t)kappa * words_per_row + (in ? w : w0));
  const uint32_t base = __shfl_sync(0xffffffffu, pos, 0);
  if (w == 0) starts[kappa] = (int32_t)pos;
  const int total = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(m));
  for (uint32_t at = pos - base; m != 0u; m &= m - 1u) list[at++] = (uint16_t)(lane * 32 + __ffs((int)m) - 1);
  __syncwarp();
  const int32_t *row = nbr + (size_t)kappa * n_out + w0 * 32;
#pragma unroll 4
  for (int e = lane; e < total; e += 32) {
    const int r = list[e];
    pair_out[base + e] = w0 * 32 + r;
    pair_in[base + e] = __ldg(row + r);
  }
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

struct WtParams {
  const float *x, *dy;         // [n][x_words], [n][y_words]
  int c_in, c_out;
  int x_words, y_words;        // row strides
  int x_round, y_round;        // 1: rows still to be rounded to TF32
  int n_pad, a_bytes, stage_bytes, stages, n_buf;
  int in_rows;                 // 1: D[ci][co], input channels are the rows of a product; 0: D[co][ci]
  uint32_t buf_cols;
  int32_t *alarm;              // mapped host word that tells of an expired wait (may be NULL)
};

// smem descriptor halves of an MN-major operand: 32-channel blocks WT_BLOCK bytes apart (leading offset), four
// pairs 512 bytes (stride offset), swizzle mode 1 (128 bytes, 32-byte atoms), descriptor version 1
constexpr uint32_t kMnDescHi = (uint32_t)(512 >> 4) | (1u << 14) | (1u << 29);
__device__ __forceinline__ uint32_t mn_desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | ((uint32_t)(WT_BLOCK >> 4) << 16); }
__device__ __forceinline__ void mma_tf32_mn(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %3, {%6, %6, %6, %6}, p;\n\t}"
      :
      : "r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kMnDescHi), "r"(0u)
      : "memory");
}

// Eight pairs' pieces of one 32-channel block, OFF bytes into the rows and BLK into the operand (constants: with running addresses half
// of the fetch was additions).
template <int OFF, int BLK>
__device__ __forceinline__ void copy_block(uint32_t dst, const float *const (&g)[WT_K / 4], const uint32_t (&bytes)[WT_K / 4], bool on) {
#pragma unroll
  for (int i = 0; i < WT_K / 4; ++i)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t"
        "@p cp.async.cg.shared.global [%0+%4], [%1+%5], 16, %2;\n\t}" ::"r"(dst + (uint32_t)i * 512u), "l"(g[i]), "r"(bytes[i]), "r"((uint32_t)on), "n"(BLK), "n"(OFF)
        : "memory");
}

template <int CTAS>
__global__ void __launch_bounds__((2 * wt_stages(CTAS) + 5) * 32, CTAS)
conv_wgrad_tc_kernel(WtParams p, const int32_t *__restrict__ pair_out, const int32_t *__restrict__ pair_in,
                     const int32_t *__restrict__ starts, int K, float *__restrict__ partial, int32_t *status) {
  after_previous();
  extern __shared__ uint8_t smem_raw[];
  __shared__ int first[257];
  __shared__ uint64_t full_bars[WT_MAX_STAGES], empty_bars[WT_MAX_STAGES], accf_bars[2], acce_bars[2], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

  const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
  const int S = p.stages, mma_warp = 2 * S;
  const bool in_rows = p.in_rows != 0;
  const int co0 = (int)blockIdx.y * (in_rows ? p.n_pad : WT_M);
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(full_bars + s), 64);      // the lanes of the slot's two warps
      mbar_init(smem_u32(empty_bars + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(accf_bars + b), 1);
      mbar_init(smem_u32(acce_bars + b), 4);
    }
    mbar_init(smem_u32(&done_bar), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(p.buf_cols * (uint32_t)p.n_buf)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  chunk_prefix(starts, K, first);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  const uint32_t smem_base = smem_u32(smem);
  const int co_cnt = min(in_rows ? p.n_pad : WT_M, p.c_out - co0);   // output channels of this CTA
  const int total = first[K];
  const int q_begin = share_begin((int)blockIdx.x, total, (int)gridDim.x), q_end = share_begin((int)blockIdx.x + 1, total, (int)gridDim.x);
  int kappa0 = 0;                               // the offset the share begins in
  while (kappa0 + 1 < K && first[kappa0 + 1] <= q_begin) ++kappa0;

  if (warp < mma_warp) {
    // ====================================== producers ========================================
    // Two warps to a slot, one for the gradients' rows and one for the inputs'.  (A warp for both: 1500 of a slot's 3800 cycles went into its
    // copies and 900 into rounding; 93 k rows of 64 -> 76 channels 101 -> 89 us, with rows rounded before 64: then the rows' way from L2
    // is the bound, 8 TB/s.)
    uint32_t par = 0;
    int kappa = kappa0;
    const int own = warp >> 1;                  // slot
    const bool second = (warp & 1) != 0, is_x = second != in_rows;    // which operand, whose rows
    const int32_t *list = is_x ? pair_in : pair_out;
    int next_row = -1;                          // this lane's row of the next chunk
    auto load_row = [&](int q) {
      next_row = -1;
      if (q >= q_end) return;
      while (first[kappa + 1] <= q) ++kappa;
      const int j = __ldg(starts + kappa) + (q - first[kappa]) * WT_K + lane;
      if (j < __ldg(starts + kappa + 1)) next_row = __ldg(list + j);
    };
    const int sub = lane & 7, grp = lane >> 3;  // 16-byte piece of a line, pair of a group of four
    // lines 0 .. 31 of every 32-channel block; piece `sub` of line k lies at 32-byte atom (sub >> 1) ^ (k & 3)
    const uint32_t piece = (uint32_t)grp * 128u + ((((uint32_t)sub >> 1) ^ (uint32_t)grp) << 5) + ((uint32_t)sub & 1u) * 16u;
    const float *rows = is_x ? p.x : p.dy + co0;
    const int words = is_x ? p.x_words : p.y_words, n_ch = is_x ? p.c_in : co_cnt, rounds = is_x ? p.x_round : p.y_round;
    const bool vec = (words & 3) == 0 && ((uintptr_t)rows & 15u) == 0;
    auto fetch = [&](int my_row, uint32_t tile) {
      const float *g[WT_K / 4];
      uint32_t bytes[WT_K / 4];
#pragma unroll
      for (int i = 0; i < WT_K / 4; ++i) {
        const int row = __shfl_sync(0xffffffffu, my_row, i * 4 + grp);
        g[i] = rows + (unsigned long long)(uint32_t)(row >= 0 ? row : 0) * (uint32_t)words + sub * 4;
        bytes[i] = row >= 0 ? 16u : 0u;
      }
      uint32_t dst = tile + piece;
      int left = n_ch - sub * 4;                // channels from this lane's first piece on
      if (vec) {
        for (int c0 = 0; c0 < n_ch; c0 += 128, left -= 128, dst += 4 * WT_BLOCK) {
          copy_block<0, 0>(dst, g, bytes, left > 0);
          if (c0 + 32 < n_ch) copy_block<128, WT_BLOCK>(dst, g, bytes, left > 32);
          if (c0 + 64 < n_ch) copy_block<256, 2 * WT_BLOCK>(dst, g, bytes, left > 64);
          if (c0 + 96 < n_ch) copy_block<384, 3 * WT_BLOCK>(dst, g, bytes, left > 96);
          if (c0 + 128 < n_ch) {
#pragma unroll
            for (int i = 0; i < WT_K / 4; ++i) g[i] += 128;
          }
        }
      } else {
        for (; left > 0; left -= 32, dst += WT_BLOCK) {
          for (int i = 0; i < WT_K / 4; ++i)
            for (int e = 0; e < 4; ++e)
              if (e < left) cp_async4(dst + (uint32_t)i * 512u + 4u * e, g[i] + e, bytes[i] >> 2);
#pragma unroll
          for (int i = 0; i < WT_K / 4; ++i) g[i] += 32;
        }
      }
    };
    auto round_tile = [&](int n_ch, uint8_t *tile) {   // this lane's pieces, in place
      uint8_t *at = tile + piece;
      for (int left = n_ch - sub * 4; left > 0; left -= 32, at += WT_BLOCK) {
        uint4 v[WT_K / 4];
#pragma unroll
        for (int i = 0; i < WT_K / 4; ++i) v[i] = *(const uint4 *)(at + i * 512);
#pragma unroll
        for (int i = 0; i < WT_K / 4; ++i) {
          v[i].x = to_tf32(__uint_as_float(v[i].x));
          v[i].y = to_tf32(__uint_as_float(v[i].y));
          v[i].z = to_tf32(__uint_as_float(v[i].z));
          v[i].w = to_tf32(__uint_as_float(v[i].w));
          *(uint4 *)(at + i * 512) = v[i];
        }
      }
    };
    const uint32_t operand = second ? (uint32_t)p.a_bytes : 0u;
    uint8_t *slot = smem + (size_t)own * p.stage_bytes + operand;
    const uint32_t slot_addr = smem_base + (uint32_t)own * (uint32_t)p.stage_bytes + operand;
    load_row(q_begin + own);
    for (int q = q_begin + own; q < q_end; q += S) {
      const int row = next_row;
      load_row(q + S);
      if (q >= q_begin + S) {
        if (!mbar_wait_straight(smem_u32(empty_bars + own), par ^ 1u, abort_flag)) break;
        tc_fence_after();
      }
      fetch(row, slot_addr);
      cp_async_commit();
      cp_async_wait(0);
      if (rounds) round_tile(n_ch, slot);
      fence_async_smem();
      mbar_arrive(smem_u32(full_bars + own));
      par ^= 1u;
    }
  } else if (warp == mma_warp) {
    // ====================================== MMA issuer: the whole warp, one elected lane issues =====
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(p.n_pad >> 3) << 17) | ((uint32_t)(WT_M >> 4) << 24);
    int kappa = kappa0, seg = 0;
    bool alive = true;
    uint32_t s = 0, par = 0;
    for (int q = q_begin; q < q_end && alive;) {
      while (first[kappa + 1] <= q) ++kappa;
      const int stop = min(q_end, first[kappa + 1]), buf = seg % p.n_buf, use = seg / p.n_buf;
      if (use > 0) {
        if (!mbar_wait_uniform(smem_u32(acce_bars + buf), (uint32_t)(use - 1) & 1u, abort_flag)) break;
        tc_fence_after();
      }
      const uint32_t d = tmem_base + (uint32_t)buf * p.buf_cols;
      for (const int q0 = q; q < stop; ++q) {
        if (!mbar_wait_uniform(smem_u32(full_bars + s), par, abort_flag)) { alive = false; break; }
        tc_fence_after();
        const uint32_t a_lo = mn_desc_lo(smem_base + s * (uint32_t)p.stage_bytes);
        const uint32_t b_lo = mn_desc_lo(smem_base + s * (uint32_t)p.stage_bytes + (uint32_t)p.a_bytes);
        if (elect_one()) {
          mma_tf32_mn(d, a_lo, b_lo, idesc, q > q0 ? 1u : 0u);      // eight pairs per instruction: 1024 bytes apart
          mma_tf32_mn(d, a_lo + 64u, b_lo + 64u, idesc, 1u);
          mma_tf32_mn(d, a_lo + 128u, b_lo + 128u, idesc, 1u);
          mma_tf32_mn(d, a_lo + 192u, b_lo + 192u, idesc, 1u);
          mma_commit(smem_u32(empty_bars + s));
        }
        if (++s == (uint32_t)S) { s = 0; par ^= 1u; }
      }
      if (alive && elect_one()) mma_commit(smem_u32(accf_bars + buf));
      ++seg;
    }
    // everything issued above (on any path) retires before the tensor memory is handed back
    if (elect_one()) mma_commit(smem_u32(&done_bar));
    mbar_wait_drain(smem_u32(&done_bar), 0u);
  } else {
    // ====================================== epilogue ===========================================
    const int quarter = warp & 3;
    const int co = co0 + quarter * 32 + lane, ci = quarter * 32 + lane;
    const bool vec = (p.c_out & 3) == 0 && ((uintptr_t)partial & 15u) == 0;
    int kappa = kappa0, seg = 0;
    for (int q = q_begin; q < q_end; ++seg) {
      while (first[kappa + 1] <= q) ++kappa;
      q = min(q_end, first[kappa + 1]);
      const int buf = seg % p.n_buf;
      if (!mbar_wait_warp_backoff(smem_u32(accf_bars + buf), (uint32_t)(seg / p.n_buf) & 1u, abort_flag, 64)) break;
      tc_fence_after();
      float *dst = partial + ((size_t)blockIdx.x + kappa) * (size_t)p.c_in * p.c_out;
      for (int c0 = 0; c0 < p.n_pad; c0 += 16) {
        uint32_t v[16];
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * p.buf_cols + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (in_rows) {
          if (ci < p.c_in) {
            float *to = dst + (size_t)ci * p.c_out + co0 + c0;
#pragma unroll
            for (int k = 0; k < 16; k += 4) {
              if (vec && c0 + k < co_cnt) *(uint4 *)(to + k) = make_uint4(v[k], v[k + 1], v[k + 2], v[k + 3]);
              for (int i = k; !vec && i < k + 4; ++i)
                if (c0 + i < co_cnt) to[i] = __uint_as_float(v[i]);
            }
          }
        } else if (co < p.c_out) {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (c0 + k < p.c_in) dst[(size_t)(c0 + k) * p.c_out + co] = __uint_as_float(v[k]);  // lanes = consecutive co: coalesced
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(acce_bars + buf));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag) report_expired(status, p.alarm);
  if (warp == mma_warp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.buf_cols * (uint32_t)p.n_buf) : "memory");
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
  after_previous();
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

// d_filters[kappa] = sum of the offset's partials, in a fixed order.  grid (x, K), block 32 groups of VEC elements x 8
// slices: slice s adds every eighth share (the centre offset has most of them), the slices are added one after
// the other.  A block goes on to further elements: where its shares lie costs it more than adding them up
// (with 32 elements per block 16 us for 27 x 64 x 76, nine tenths of it that).
template <int VEC>
__global__ void __launch_bounds__(256)
wgrad_reduce_shares_kernel(const float *__restrict__ partial, const int32_t *__restrict__ starts, int K, int shares, int elems,
                           float *__restrict__ out) {
  after_previous();
  __shared__ int first[257];
  __shared__ float sm[8][32 * VEC + 1];
  chunk_prefix(starts, K, first);
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int kappa = blockIdx.y, total = first[K];
  const bool any = first[kappa + 1] > first[kappa], gaps = total < shares;      // gaps: shares without a chunk wrote nothing
  const int lo = any ? share_of(first[kappa], total, shares) : 0, hi = any ? share_of(first[kappa + 1] - 1, total, shares) : -1;
  for (int e0 = (int)blockIdx.x * 32 * VEC; e0 < elems; e0 += (int)gridDim.x * 32 * VEC) {
    const int e = e0 + lane * VEC;
    float s[VEC];
#pragma unroll
    for (int q = 0; q < VEC; ++q) s[q] = 0.f;
    if (e < elems) {
      const float *p = partial + ((size_t)lo + slice + kappa) * elems + e;
#pragma unroll 4
      for (int b = lo + slice; b <= hi; b += 8, p += (size_t)8 * elems) {
        if (gaps && share_begin(b + 1, total, shares) <= share_begin(b, total, shares)) continue;
        if (VEC == 4) {
          const float4 v = __ldg((const float4 *)p);
          s[0] += v.x; s[1 % VEC] += v.y; s[2 % VEC] += v.z; s[3 % VEC] += v.w;
        } else {
          s[0] += __ldg(p);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < VEC; ++q) sm[slice][lane * VEC + q] = s[q];
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * VEC && e0 + i < elems; i += 256) {
      float r = sm[0][i];
#pragma unroll
      for (int k = 1; k < 8; ++k) r += sm[k][i];
      out[(size_t)kappa * elems + e0 + i] = r;
    }
    __syncthreads();
  }
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
  { launch_ready(pair_bitmap_kernel, dim3(ceil_div(p.wpr, 32), K), dim3(256), 0, st, nbr, n_out, p.wpr, p.bitmap); note_launches(1); }
  SSC_CHECK_LAUNCH("pair_bitmap");
  int rc = exclusive_scan_u32<true>(p.bitmap, p.words, p.prefix, p.block_sums, p.starts + K, nullptr, st);
  if (rc != 0) return rc;
  { launch_ready(pair_scatter_kernel, dim3(ceil_div(p.wpr, 256), K), dim3(256), 0, st, nbr, n_out, p.wpr, p.bitmap, p.prefix, p.pair_out, p.pair_in, p.starts); note_launches(1); }
  SSC_CHECK_LAUNCH("pair_scatter");
  if (out) *out = PairLists{p.pair_out, p.pair_in, p.starts};
  return SSC_OK;
}

// Shapes and shares of the two list kernels.
struct WgradPlan {
  bool tc, small, in_rows;
  int n_pad, n_buf, co_blocks, shares, ctas, stages, a_bytes, stage_bytes;
  uint32_t buf_cols;
  size_t smem;
};
static WgradPlan wgrad_plan(int K, int c_in, int c_out, int n_out, bool tf32) {
  WgradPlan p;
  memset(&p, 0, sizeof(p));
  if (K > 256) return p;               // (chunk_prefix keeps the offsets in shared memory)
  // never more shares than the table could hold chunks
  const long long most = (long long)K * ceil_div(n_out > 0 ? n_out : 1, WT_K);
  if (tf32) {
    // Blocks of 128 output channels bring the input rows in once each.  Where there are several and the input channels fit the rows of a
    // product, they are those, and up to 256 output channels its columns (93 k rows of 64 -> 152 169 -> 101 us, 30 k of 128 -> 152 64 -> 40, of 128 -> 304 90 -> 68).
    // One block has twice the shares of two, so twice the partial sums are written and added up, by a lane per input channel: few
    // pairs do not pay for it, the fewer the wider the block (27 offsets; output, input channels as rows, us at 1.5 and 9 neighbours: 128 -> 152
    // 4000 rows 21.0, 27.2 and 23.5, 26.8, 8000 22.1, 34.2 and 24.2, 30.6; 128 -> 256 8000 25.9, 38.3 and 32.1, 39.1, 16 k 28.2, 53.4 and 32.6, 49.0, 40 k
    // 36.0, 102 and 38.4, 81; 128 -> 224, where those stores are dearest, 16 k 26.7, 51.8 and 35.3, 52.0, 40 k 34.1, 101 and 41.6, 83).
    // The shares end elsewhere then, and the sums are cut there: against 64 bits, operands that are TF32 already, 93 k rows of 64 -> 152
    // 2.4e-5 with the output channels as rows of a product and 1.3e-5 with the input channels.
    p.in_rows = c_out > WT_M && c_in <= WT_M && n_out >= (ceil_div(c_out, ceil_div(c_out, 256)) > 176 ? 16384 : 4096);
    if (p.in_rows) {
      p.co_blocks = ceil_div(c_out, 256);
      p.n_pad = (ceil_div(c_out, p.co_blocks) + 15) & ~15;
    } else {
      p.co_blocks = ceil_div(c_out, WT_M);
      p.n_pad = (c_in + 15) & ~15;
    }
    if (p.n_pad > 256) return p;
    p.tc = true;
    p.buf_cols = 32;
    while ((int)p.buf_cols < p.n_pad) p.buf_cols <<= 1;
    // The 128 rows of an MMA are always read: channels that do not exist come from whatever lies behind the
    // operand's real blocks (the slack behind the last slot keeps that inside the buffer).
    const int m_side = p.in_rows ? c_in : c_out;
    p.a_bytes = ceil_div(m_side < WT_M ? m_side : WT_M, 32) * WT_BLOCK;
    p.stage_bytes = p.a_bytes + ceil_div(p.n_pad, 32) * WT_BLOCK;
    // two CTAs per SM (tensor memory: 512 columns) where four slots fit each; two accumulator buffers where the columns allow
    const size_t slack = 1024 + (size_t)4 * WT_BLOCK, fixed = 2048;
    const int ctas = 4 * (size_t)p.stage_bytes + slack + fixed <= 113 * 1024 ? 2 : 1;
    p.stages = (int)(((ctas == 2 ? 113 : 226) * 1024 - slack - fixed) / p.stage_bytes);
    if (p.stages > wt_stages(ctas)) p.stages = wt_stages(ctas);
    p.ctas = ctas;
    if (p.stages < 2) { p.tc = false; return p; }
    p.smem = (size_t)p.stages * p.stage_bytes + slack;
    p.n_buf = (int)p.buf_cols * 2 * ctas <= 512 ? 2 : 1;
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

// staged: bit 0 / 1: features / out_grad are TF32 images (ssc_conv_stage: rows padded to a multiple of four floats).
// Returns -1 when the shape is not covered (conv_wgrad_lists_partial_bytes is 0: the caller then uses the CUDA-core kernel
// over the table).
int conv_wgrad_lists(const float *features, int c_in, const float *out_grad, int c_out, const PairLists &pl, int K, int n_out,
                     bool tf32, int staged, float *partial, float *d_filters, int32_t *status, cudaStream_t st) {
  const WgradPlan p = wgrad_plan(K, c_in, c_out, n_out, tf32);
  if (p.tc) {
    auto kernel = p.ctas == 2 ? conv_wgrad_tc_kernel<2> : conv_wgrad_tc_kernel<1>;
    cudaError_t e = allow_smem((const void *)kernel, p.smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_wgrad(tf32): smem attribute: %s", cudaGetErrorString(e));
    const WtParams w = {features, out_grad, c_in, c_out, (staged & 1) ? (c_in + 3) & ~3 : c_in, (staged & 2) ? (c_out + 3) & ~3 : c_out,
                        (staged & 1) ? 0 : 1, (staged & 2) ? 0 : 1, p.n_pad, p.a_bytes, p.stage_bytes, p.stages, p.n_buf, p.in_rows ? 1 : 0, p.buf_cols, alarm_word()};
    { launch_ready(kernel, dim3(p.shares, p.co_blocks), dim3((2 * p.stages + 5) * 32), p.smem, st, w, pl.pair_out, pl.pair_in, pl.starts, K, partial, status); note_launches(1); }
    SSC_CHECK_LAUNCH("conv_wgrad_tc");
  } else if (p.small) {
    const dim3 grid(p.shares / 4, p.co_blocks);
    if (c_in <= 4) { launch_ready(conv_wgrad_small_kernel<4>, dim3(grid), dim3(128), 0, st, features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in, pl.starts, K, partial); note_launches(1); }
    else if (c_in <= 8) { launch_ready(conv_wgrad_small_kernel<8>, dim3(grid), dim3(128), 0, st, features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in, pl.starts, K, partial); note_launches(1); }
    else { launch_ready(conv_wgrad_small_kernel<16>, dim3(grid), dim3(128), 0, st, features, c_in, out_grad, c_out, pl.pair_out, pl.pair_in, pl.starts, K, partial); note_launches(1); }
    SSC_CHECK_LAUNCH("conv_wgrad_small");
  } else {
    return -1;
  }
  const int elems = c_in * c_out;
  const bool vec = (elems & 3) == 0 && ((uintptr_t)partial & 15u) == 0;
  const int tiles = ceil_div(elems, vec ? 128 : 32), most = ceil_div(8 * sm_count(), K);      // one wave of blocks
  const dim3 grid(tiles < most ? tiles : most, K);
  if (vec) launch_ready(wgrad_reduce_shares_kernel<4>, dim3(grid), dim3(256), 0, st, partial, pl.starts, K, p.shares, elems, d_filters);
  else launch_ready(wgrad_reduce_shares_kernel<1>, dim3(grid), dim3(256), 0, st, partial, pl.starts, K, p.shares, elems, d_filters);
  note_launches(1);
  SSC_CHECK_LAUNCH("conv_wgrad_reduce");
  return SSC_OK;
}

}  // namespace ssc
