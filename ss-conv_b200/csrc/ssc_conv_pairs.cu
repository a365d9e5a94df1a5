// Pair-list gather-GEMM-scatter on the 5th-generation tensor cores (tcgen05, sm_100a): the forward
// convolution for layers whose neighbour table is sparsely filled (wide submanifold layers: a
// 5^3 kernel at 10 % occupancy has 12 of its 125 offsets present per output row, so an
// output-stationary tile would spend 90 % of every MMA on absent rows).
//
//   for every kernel offset kappa, for every 128 pairs (i, o) of its compacted pair list:
//       D[128, Cout] = X[i, :] * W[kappa]          (dense M tile, all rows live)
//       out[o, :]   += D                           (one output row occurs once per offset)
//
// which is what the reference does with a gather, a cuBLAS GEMM and a scatter-add per offset
// (SS_Conv_lib/src/conv/indice_conv.h:290-338), here as ONE persistent launch:
//
//   * The work is cut into strips.  A strip belongs to one kernel offset (times one range of
//     output channels when the filter matrix of an offset does not fit shared memory whole) and is
//     every c-th 128-pair tile of that offset's list.  A CTA keeps the filter matrix of its strip
//     RESIDENT in shared memory (one bulk copy per 32/64-channel slab, once per strip), so the
//     only operand traffic per tile is the gathered rows.  All strips walk their lists from the
//     first row to the last at the same pace, so at any time the CTAs of the grid read and update
//     the same window of rows: the gathers and the reductions hit L2.
//   * warps 0 .. 3: producers.  They fill every ring slot together, 32 pairs each, four lanes to a row:
//     16-byte cp.async copies of the row's 128-byte slab from the staged operand image (TF32-rounded
//     fp32, fp16 or bf16) into the K-major 128-byte-swizzled operand layout.  Nobody waits for
//     copies: their completion arrives on the slot's "full" mbarrier by itself, and the issuing warp
//     orders the rows for the tensor core.  (A warp per slot that waited for its own copies let
//     a slot turn round in 5000 cycles: 1240 us for 2.2 M pairs of 256 -> 256 channels.)
//   * warp 4: the filter matrix of each strip, tensor-memory allocation and the MMA-issuing thread: tcgen05.mma M=128, N<=256,
//     accumulating over the slabs of a tile in one of TWO accumulator buffers, tcgen05.commit to
//     the slot's "empty" barrier and, after the last slab, to the buffer's "accumulator full"
//     barrier.
//   * warps 5 .. 12: epilogue, two per quarter of the tensor-memory lanes (they take the
//     32-column blocks in turn).  tcgen05.ld (lane = pair), a transposition through shared memory,
//     16 rows at a time, so that eight neighbouring lanes hold the 128 contiguous bytes of one
//     output row, then red.global.add.v4.f32: the reductions reach L2 as whole 128-byte lines (a warp has every other block).
//     The epilogue of tile t runs under the MMAs of tile t+1.
//
// The output must be zero before the launch (the host wrapper clears it).  The sums of an output
// row arrive in no fixed order, so results are reproducible only up to fp32 rounding of a sum of
// about K/2 terms; the output-stationary kernel (ssc_conv_tc.cu) is the bitwise-repeatable one.
// Every wait is bounded; on expiry status bit 16 is set, tensor memory is freed, the kernel returns.
#include "ssc_conv_internal.cuh"
#include "ssc_tc_ptx.cuh"

namespace ssc {

constexpr int PL_M = 128;                 // pairs per tile
constexpr int PL_A_BYTES = PL_M * 128;    // one gathered slab
constexpr int PL_MAX_STAGES = 6;
constexpr int PL_EPI_WARPS = 8;
constexpr int PL_PRODUCERS = 4;           // producer warps
constexpr int PL_STG_ROW = 128;           // bytes per row of the epilogue's transpose block (pieces swizzled by the row)
constexpr int PL_STG_BYTES = PL_EPI_WARPS * 16 * PL_STG_ROW;
constexpr int PL_CTRL_BYTES = 1024;
constexpr int PL_MAX_CTAS = 320;

struct PlParams {
  int k_slabs;      // 128-byte slabs per operand row
  int slab_words;   // 4-byte words of a staged row that are real data (the rest of the last slab is zero-filled)
  int row_words;    // row stride of the staged image in 4-byte words
  int n_pad;        // rows of one slab of the packed filter image
  int n_split;      // ranges of output channels (each a strip of its own)
  int n_cta;        // output channels per CTA = n_pad / n_split: multiple of 16, <= 256
  int acc_cols;     // tensor-memory columns of one accumulator buffer (power of two >= n_cta, >= 32)
  int stages;       // ring slots
  int w_bytes;      // k_slabs * n_cta * 128: the resident filter matrix
  int threads;
  int ctas_per_sm;
  uint32_t idesc;
  int32_t *alarm;   // mapped host word that tells of an expired wait (may be NULL)
  int pair;         // 1: two CTAs to a strip, half of the filter matrix in each; n_cta is the whole width then, a tile 256 pairs
  int f16;          // kind::f16 (fp16 / bf16 operands) instead of kind::tf32
};

// Strip table of one (pair lists, grid) combination.
//   strips[s] = {virtual offset kv = kappa * n_split + half, first tile, tile stride, number of tiles}
//   owner[s]  = the CTA that runs strip s (a CTA runs its strips in ascending s)
//   hdr       = {number of strips, K, n_split, n_ctas, rows of a tile}: the table is kept with the pair lists and only
//               built when the header does not match (another grid or channel split)
// L = the grid's fair share of all tiles.  An offset with T <= L tiles is one strip; up to 1.5 L it
// is a main strip of L tiles plus a tail; beyond that it is cut into round(T / L) interleaved strips
// (tiles r, r + c, ...: the centre offset of a submanifold layer).  Strips then go to the CTAs
// greedily, main strips first, each to the CTA with the least work so far: every CTA starts with a
// strip that walks its offset's list from the first row (all CTAs sweep the rows together, which keeps
// gathers and reductions in L2) and the tails fill the CTAs whose offsets were short.
// What bounds it is the greedy assignment, one strip after the other: with the CTAs' loads in shared memory each
// strip cost a scan of all of them, 140 us for the 330 strips of a 5^3 layer; with a load per thread of the
// block and two barriers per strip 30 us.  One warp now holds ten loads per lane in registers (the lowest
// CTA wins ties); the first strip of every CTA needs no decision (all loads are zero, so they go in order).
__device__ __forceinline__ void deal_strips(const int32_t *__restrict__ starts, int K, int n_split, int tile, int n_ctas,
                                            int32_t *__restrict__ hdr, int4 *__restrict__ strips, int32_t *__restrict__ owner) {
  __shared__ int tiles[256], first[257], tiles_of[PL_MAX_CTAS];
  __shared__ int L_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (hdr[0] > 0 && hdr[1] == K && hdr[2] == n_split && hdr[3] == n_ctas && hdr[4] == tile) return;   // built before for this grid
  int T = 0;
  if (tid < K) {
    const int n = starts[tid + 1] - starts[tid];
    T = n > 0 ? (n + tile - 1) / tile : 0;
  }
  if (tid < 256) tiles[tid] = T;
  __syncthreads();
  if (tid < 32) {
    long long tot = 0;
    for (int k = tid; k < K; k += 32) tot += tiles[k];
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    const long long L = (tot * n_split + n_ctas - 1) / n_ctas;
    if (tid == 0) L_s = L < 1 ? 1 : (int)L;
  }
  __syncthreads();
  const int L = L_s;
  int mains = 0, tail = 0;
  if (T > 0) {
    if (T > L + L / 2) mains = (T + L / 2) / L;
    else { mains = 1; tail = T > L ? 1 : 0; }
  }
  if (tid < 256) tiles[tid] = (mains + tail) * n_split;
  __syncthreads();
  if (tid < 32) {
    int run = 0;
    for (int k0 = 0; k0 < 256; k0 += 32) {
      int v = k0 + lane < K ? tiles[k0 + lane] : 0, incl = v;
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      first[k0 + lane] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) first[256] = run;
  }
  __syncthreads();
  const int n_strips = first[256];
  if (tid < K && T > 0) {
    int s = first[tid];
    for (int h = 0; h < n_split; ++h) {
      const int kv = tid * n_split + h;
      if (mains > 1) {
        for (int r = 0; r < mains; ++r) { strips[s] = make_int4(kv, r, mains, (T - r + mains - 1) / mains); owner[s++] = -1; }
      } else {
        strips[s] = make_int4(kv, 0, 1, T < L ? T : L);
        owner[s++] = -1;
        if (tail) { strips[s] = make_int4(kv, L, 1, T - L); owner[s++] = -2; }
      }
    }
  }
  __syncthreads();
  // main strips (-1) first, then tails (-2), each to the CTA with the least work so far.  Work and CTA in one word:
  // a load is at most the number of tiles of a table, which stays below 2^22 for 2^31 / 128 / K pairs.
  __shared__ int n_main_s;
  if (tid < 32) {              // the main strips among the first n_ctas strips of that kind
    int seen = 0;
    for (int s0 = 0; s0 < n_strips && seen < n_ctas; s0 += 32) {
      const int s = s0 + lane;
      const bool is = s < n_strips && owner[s] == -1;
      const unsigned b = __ballot_sync(0xffffffffu, is);
      const int at = seen + __popc(b & ((1u << lane) - 1u));
      if (is && at < n_ctas) {
        owner[s] = at;
        tiles_of[at] = strips[s].w;
      }
      seen += __popc(b);
    }
    if (lane == 0) n_main_s = seen < n_ctas ? seen : n_ctas;
  }
  __syncthreads();
  if (warp == 0) {
    constexpr int PER = PL_MAX_CTAS / 32;
    unsigned key[PER];                              // of CTA 32 j + lane
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int cta = j * 32 + lane;
      key[j] = cta < n_ctas ? ((cta < n_main_s ? (unsigned)tiles_of[cta] : 0u) << 9) | (unsigned)cta : 0xffffffffu;
    }
    for (int pass = -1; pass >= -2; --pass) {
      for (int s0 = 0; s0 < n_strips; s0 += 32) {
        const int s = s0 + lane, kind = s < n_strips ? owner[s] : 0, work = s < n_strips ? strips[s].w : 0;
        int to = kind;
        for (unsigned left = __ballot_sync(0xffffffffu, kind == pass); left != 0u; left &= left - 1u) {
          const int i = __ffs((int)left) - 1;
          unsigned m = key[0];
#pragma unroll
          for (int j = 1; j < PER; ++j) m = min(m, key[j]);
          m = __reduce_min_sync(0xffffffffu, m);
          const unsigned add = (unsigned)__shfl_sync(0xffffffffu, work, i) << 9;
#pragma unroll
          for (int j = 0; j < PER; ++j) key[j] += key[j] == m ? add : 0u;
          if (lane == i) to = (int)(m & 511u);
        }
        if (kind == pass) owner[s] = to;
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    hdr[1] = K;
    hdr[2] = n_split;
    hdr[3] = n_ctas;
    hdr[4] = tile;
    __threadfence();
    hdr[0] = n_strips;
  }
}

// What the persistent kernel needs beforehand, in one launch: the strip table (block 0: 16 us of one block's
// serial work), the operand image of the rows (n_stage pieces of 16 bytes, as ssc_conv_stage.cu writes it; 0 where it is there
// already) and a cleared output.  The last two are bound by memory, and the strips come in their shadow (and bound the launch
// where rows are few).  One piece at a time: four loads before the first store, as ssc_conv_stage.cu has them, were not tried here.
// (42 k rows 192 -> 192 bf16: 9 + 7 + 16 us one after the other, 22 like this; the whole layer 246 -> 232.)
template <bool F16>
__global__ void __launch_bounds__(PL_MAX_CTAS)
pl_prepare_kernel(const int32_t *__restrict__ starts, int K, int n_split, int tile, int n_ctas, int32_t *__restrict__ hdr, int4 *__restrict__ strips,
                  int32_t *__restrict__ owner, const float4 *__restrict__ rows, long long n_stage, int bf16, uint4 *__restrict__ staged,
                  float4 *__restrict__ out, long long n_clear) {
  after_previous();
  if (blockIdx.x == 0) {
    deal_strips(starts, K, n_split, tile, n_ctas, hdr, strips, owner);
    return;
  }
  const long long first = (long long)(blockIdx.x - 1) * PL_MAX_CTAS + threadIdx.x, step = (long long)(gridDim.x - 1) * PL_MAX_CTAS;
  for (long long i = first; i < n_stage; i += step) {
    if (F16) staged[i] = stage_piece_16(__ldg(rows + 2 * i), __ldg(rows + 2 * i + 1), bf16 != 0);
    else staged[i] = stage_piece(__ldg(rows + i));
  }
  for (long long i = first; i < n_clear; i += step) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// A lane's piece of two rows (none of a negative one), OFF bytes into its part of the slot.
template <int OFF>
__device__ __forceinline__ void copy_two_rows(int a, int b, uint32_t dst0, uint32_t dst1, const char *base, uint32_t stride, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 s, t;\n\tsetp.ge.s32 p, %0, 0;\n\tsetp.ge.s32 q, %1, 0;\n\t"
      "mad.wide.u32 s, %0, %5, %4;\n\tmad.wide.u32 t, %1, %5, %4;\n\t"
      "@p cp.async.cg.shared.global [%2+%7], [s], 16, %6;\n\t"
      "@q cp.async.cg.shared.global [%3+%7], [t], 16, %6;\n\t}" ::"r"(a), "r"(b), "r"(dst0), "r"(dst1), "l"(base), "r"(stride), "r"(bytes), "n"(OFF)
      : "memory");
}

template <bool PAIR>
__device__ __forceinline__ void pl_commit(uint32_t bar) {
  if (PAIR) mma_commit_pair(bar);
  else mma_commit(bar);
}

// Two CTAs to a strip (a cluster): its tiles have 256 pairs, 128 each, multiplied as one (cta_group::2), and each CTA holds half of the
// filter matrix, so that a matrix that does not fit one CTA needs no second gather of its rows.  CTA 0 issues for both; what it
// has to know of the other (rows landed, filters landed, accumulators read out) comes as asynchronous stores of
// 16 bytes that count on its barriers.
template <bool F16, bool PAIR>
__device__ __forceinline__ void
conv_fwd_pairs_body(const float *__restrict__ staged, const uint4 *__restrict__ packed, int c_out,
                    const int32_t *__restrict__ pair_out, const int32_t *__restrict__ pair_in,
                    const int32_t *__restrict__ starts, const int4 *__restrict__ strips,
                    const int32_t *__restrict__ owner, const int32_t *__restrict__ n_strips_dev,
                    float *__restrict__ out, int32_t *status, const PlParams &p) {
  const int unit = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, rank = PAIR ? (int)blockIdx.x & 1 : 0;
  constexpr int TILE = PAIR ? 2 * PL_M : PL_M;
  const int tile_row0 = rank * PL_M;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  uint8_t *w_smem = smem;                                       // resident filters, [k_slabs][n_cta][128 B]
  uint8_t *a_smem = smem + p.w_bytes;                           // [stages][16 KB]
  uint8_t *stg = a_smem + (size_t)p.stages * PL_A_BYTES;        // epilogue transpose blocks
  uint8_t *ctrl = stg + PL_STG_BYTES;
  uint64_t *full_bars = (uint64_t *)ctrl;                       // [stages] gathered slab landed
  uint64_t *empty_bars = full_bars + PL_MAX_STAGES;             // [stages] its MMAs retired
  uint64_t *accf_bars = empty_bars + PL_MAX_STAGES;             // [2] accumulator buffer complete
  uint64_t *acce_bars = accf_bars + 2;                          // [2] accumulator buffer read out
  uint64_t *wfull_bar = acce_bars + 2;                          // filters of the strip landed
  uint64_t *wfree_bar = wfull_bar + 1;                          // every MMA of the strip retired
  uint64_t *final_bar = wfree_bar + 1;
  uint32_t *tmem_slot = (uint32_t *)(final_bar + 1);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const uint32_t news = smem_u32(ctrl + 512);                   // where the other CTA's stores go

  const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
  const int S = p.stages;
  constexpr int mma_warp = PL_PRODUCERS;
  const int n_strips = *n_strips_dev;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(full_bars + s), PL_PRODUCERS * 32 + (PAIR && rank == 0 ? 1 : 0));    // arrivals by copies, the other CTA's news
      mbar_init(smem_u32(empty_bars + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(accf_bars + b), 1);
      mbar_init(smem_u32(acce_bars + b), PL_EPI_WARPS);
    }
    mbar_init(smem_u32(wfull_bar), 1);
    mbar_init(smem_u32(wfree_bar), 1);
    mbar_init(smem_u32(final_bar), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == mma_warp) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)(2 * p.acc_cols)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)(2 * p.acc_cols)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();                               // the other CTA's barriers stand
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t a_base = smem_u32(a_smem), w_base = smem_u32(w_smem);

  // Every role walks the same strips and keeps the same counters: ring slot and its parity, tcount = tiles so far
  // (buffer tcount % 2), scount = strips so far.
  if (warp < PL_PRODUCERS) {
    // ==================================== producers =============================================
    // Lane l copies the 16-byte piece l & 7 of rows 4 * pass + l / 8 of its warp's 32, eight passes: a row's 128 bytes are
    // one request (with four lanes to a row they are two, and the way out of the SM, which the reductions
    // share, was what bound the kernel).  The input rows of the next tile are on their way meanwhile.
    const int piece = lane & 7, row4 = lane >> 3;
    const uint32_t warp_rows = a_base + (uint32_t)warp * 4096u;
    const uint32_t first0 = warp_rows + (uint32_t)row4 * 128u + (uint32_t)((piece ^ row4) << 4);
    const uint32_t first1 = warp_rows + (uint32_t)(row4 + 4) * 128u + (uint32_t)((piece ^ row4 ^ 4) << 4);
    const uint32_t full0 = smem_u32(full_bars), empty0 = smem_u32(empty_bars), row_bytes = (uint32_t)p.row_words * 4u;
    const char *lane_rows = (const char *)staged + piece * 16;
    const int k_slabs = p.k_slabs, slab_words = p.slab_words;
    int slot = 0;
    uint32_t par = 1;                                     // (a fresh barrier counts as passed with parity 1)
    bool alive = true;
    for (int si = 0; si < n_strips && alive; ++si) {
      if (__ldg(owner + si) != unit) continue;
      const int4 sd = __ldg(strips + si);
      const int kappa = sd.x / p.n_split;
      const int list0 = __ldg(starts + kappa), n_pairs = __ldg(starts + kappa + 1) - list0;
      const int n_tiles = sd.w;
      auto row_of = [&](int ti) {                         // input row of this lane's pair
        const int j = (sd.y + ti * sd.z) * TILE + tile_row0 + warp * 32 + lane;
        return ti < n_tiles && j < n_pairs ? __ldg(pair_in + list0 + j) : -1;
      };
      int src = row_of(0);
      for (int ti = 0; ti < n_tiles && alive; ++ti) {
        const int next = row_of(ti + 1);
        int from[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) from[i] = __shfl_sync(0xffffffffu, src, i * 4 + row4);
#pragma unroll 1
        for (int slab = 0; slab < k_slabs && alive; ++slab) {
          // pieces past the last channel are zero-filled (and read nothing)
          const uint32_t bytes = slab * 32 + piece * 4 < slab_words ? 16u : 0u, stride = bytes ? row_bytes : 0u;
          const char *base = bytes ? lane_rows + slab * 128 : (const char *)staged;
          const uint32_t full = full0 + (uint32_t)slot * 8u, slot_off = (uint32_t)slot * (uint32_t)PL_A_BYTES;
          alive = mbar_wait_straight(empty0 + (uint32_t)slot * 8u, par, abort_flag);
          if (PAIR && rank == 0 && warp == 0 && elect_one()) mbar_expect_tx(full, 16u);
          const uint32_t dst0 = first0 + slot_off, dst1 = first1 + slot_off;
          copy_two_rows<0>(from[0], from[1], dst0, dst1, base, stride, bytes);
          copy_two_rows<1024>(from[2], from[3], dst0, dst1, base, stride, bytes);
          copy_two_rows<2048>(from[4], from[5], dst0, dst1, base, stride, bytes);
          copy_two_rows<3072>(from[6], from[7], dst0, dst1, base, stride, bytes);
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full) : "memory");
          if (++slot == S) { slot = 0; par ^= 1u; }
        }
        src = next;
      }
    }
    cp_async_wait_all();
  } else if (warp == mma_warp) {
    // ==================================== MMA issuer: the whole warp, one elected lane issues ====
    int tcount = 0, scount = 0, w_issued = 0;
    uint32_t slot = 0, slot_par = 0;
    bool alive = true;
    const uint32_t news0 = PAIR ? peer_address(news, 0u) : 0u, full0_there = PAIR ? peer_address(smem_u32(full_bars), 0u) : 0u;
    for (int si = 0; si < n_strips && alive; ++si) {
      if (__ldg(owner + si) != unit) continue;
      const int4 sd = __ldg(strips + si);
      const int n_tiles = sd.w, kappa = sd.x / p.n_split, half = sd.x - kappa * p.n_split;
      // the strip's filter matrix: one bulk copy per slab, after the MMAs of the last strip retired
      if (scount > 0 && !mbar_wait_uniform(smem_u32(wfree_bar), (uint32_t)(scount - 1) & 1u, abort_flag)) break;
      const uint32_t own_rows = (uint32_t)(PAIR ? p.n_cta >> 1 : p.n_cta), slab_bytes = own_rows * 128u;    // filter rows in this CTA
      if (elect_one()) {
        const uint32_t bar = smem_u32(wfull_bar);
        mbar_expect_tx(bar, (uint32_t)p.w_bytes + (PAIR && rank == 0 ? 16u : 0u));
        for (int s = 0; s < p.k_slabs; ++s)
          bulk_g2s(w_base + (uint32_t)s * slab_bytes,
                   packed + ((size_t)kappa * p.k_slabs + s) * (size_t)(p.n_pad * 8) + (size_t)(PAIR ? rank : half) * (size_t)(own_rows * 8), slab_bytes, bar);
      }
      ++w_issued;
      if (!(PAIR ? mbar_wait_straight_cluster(smem_u32(wfull_bar), (uint32_t)scount & 1u, abort_flag) : mbar_wait_straight(smem_u32(wfull_bar), (uint32_t)scount & 1u, abort_flag))) break;
      tc_fence_after();
      if (PAIR && rank == 1) {                            // only tells the other CTA
        if (elect_one()) st_async_v4(news0, make_uint4(0u, 0u, 0u, 0u), peer_address(smem_u32(wfull_bar), 0u));
        for (int n = n_tiles * p.k_slabs; n > 0 && alive; --n) {
          alive = mbar_wait_straight(smem_u32(full_bars + slot), slot_par, abort_flag);
          fence_async_smem();
          if (alive && elect_one()) st_async_v4(news0, make_uint4(0u, 0u, 0u, 0u), full0_there + slot * 8u);
          if (++slot == (uint32_t)S) { slot = 0; slot_par ^= 1u; }
        }
        ++scount;
        continue;
      }
      for (int ti = 0; ti < n_tiles && alive; ++ti, ++tcount) {
        const int buf = tcount & 1;
        if (tcount >= 2) {
          const uint32_t bar = smem_u32(acce_bars + buf), passed = (uint32_t)((tcount >> 1) - 1) & 1u;
          if (!(PAIR ? mbar_wait_straight_cluster(bar, passed, abort_flag) : mbar_wait_straight(bar, passed, abort_flag))) { alive = false; break; }
          tc_fence_after();
        }
        const uint32_t d = tmem_base + (uint32_t)(buf * p.acc_cols);
        for (int s = 0; s < p.k_slabs; ++s) {
          if (!(PAIR ? mbar_wait_straight_cluster(smem_u32(full_bars + slot), slot_par, abort_flag) : mbar_wait_uniform(smem_u32(full_bars + slot), slot_par, abort_flag))) { alive = false; break; }
          fence_async_smem();                             // the rows other threads' copies left, for the tensor core
          tc_fence_after();
          const uint32_t a_lo = desc_lo(a_base + slot * PL_A_BYTES);
          const uint32_t b_lo = desc_lo(w_base + (uint32_t)s * slab_bytes);
          if (elect_one()) {
#pragma unroll
            for (uint32_t kk = 0; kk < 4; ++kk) {
              if (PAIR) mma_pair<F16>(d, a_lo + 2u * kk, b_lo + 2u * kk, p.idesc, (s | (int)kk) != 0 ? 1u : 0u);
              else if (F16) mma_f16_ss(d, a_lo + 2u * kk, b_lo + 2u * kk, p.idesc, (s | (int)kk) != 0 ? 1u : 0u);
              else mma_tf32_ss(d, a_lo + 2u * kk, b_lo + 2u * kk, p.idesc, (s | (int)kk) != 0 ? 1u : 0u);
            }
            pl_commit<PAIR>(smem_u32(empty_bars + slot));
          }
          if (++slot == (uint32_t)S) { slot = 0; slot_par ^= 1u; }
        }
        if (alive && elect_one()) pl_commit<PAIR>(smem_u32(accf_bars + buf));
      }
      if (alive && elect_one()) pl_commit<PAIR>(smem_u32(wfree_bar));
      ++scount;
    }
    // everything issued above (on any path) retires before the CTA hands its tensor memory back
    if (rank == 0 && elect_one()) pl_commit<PAIR>(smem_u32(final_bar));
    mbar_wait_drain(smem_u32(final_bar), 0u);
    // a wait gave up while a filter copy may still be in flight: let it land before the CTA exits
    if (*abort_flag && w_issued > 0) mbar_wait_drain(smem_u32(wfull_bar), (uint32_t)(w_issued - 1) & 1u);
  } else {
    // ==================================== epilogue ==============================================
    // Two warps per quarter of the tensor-memory lanes; they take the 32-column blocks of the
    // accumulator in turn.  Their chain of instructions bounds the kernel (8300 of a tile's 9100 cycles for 256 channels, whether the
    // reductions are issued or not), so a tile's addresses are worked out once and four loads from shared memory are in flight: 679 -> 644 us,
    // bf16 192 -> 192 136 -> 128.  (Twelve warps gain nothing more, sixteen leave less room for the ring: 736 us.)
    const uint32_t news0 = PAIR ? peer_address(news, 0u) : 0u;
    const int ew = warp - mma_warp - 1;                    // 0 .. 7
    const int quarter = warp & 3;                          // the 32 tensor-memory lanes this warp may read
    const int part = ew >> 2;                              // blocks part, part + 2, ... (eight warps)
    uint8_t *blk = stg + (size_t)ew * 16 * PL_STG_ROW;
    const bool vec_ok = (c_out & 3) == 0 && ((uintptr_t)out & 15u) == 0;
    const int sub = lane & 7, grp = lane >> 3;             // 16-byte piece of a row, row of a pass
    int tcount = 0;
    bool alive = true;
    for (int si = 0; si < n_strips && alive; ++si) {
      if (__ldg(owner + si) != unit) continue;
      const int4 sd = __ldg(strips + si);
      const int kappa = sd.x / p.n_split, half = sd.x - kappa * p.n_split;
      const int list0 = __ldg(starts + kappa), n_pairs = __ldg(starts + kappa + 1) - list0;
      const int n_tiles = sd.w;
      const int col0 = half * p.n_cta;
      const int cols = min(p.n_cta, c_out - col0);
      const int n_blocks = cols > 0 ? (cols + 31) >> 5 : 0;       // 32-column blocks with real columns
      // output row of this lane's pair, fetched one tile ahead
      auto out_row_of = [&](int ti) {
        const int j = (sd.y + ti * sd.z) * TILE + tile_row0 + quarter * 32 + lane;
        return (ti < n_tiles && j < n_pairs) ? __ldg(pair_out + list0 + j) : -1;
      };
      int next_out = out_row_of(0);
      for (int ti = 0; ti < n_tiles; ++ti, ++tcount) {
        const int buf = tcount & 1;
        const int my_out = next_out;
        next_out = out_row_of(ti + 1);
        if (!mbar_wait_warp(smem_u32(accf_bars + buf), (uint32_t)(tcount >> 1) & 1u, abort_flag)) { alive = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * p.acc_cols);
        // this lane's places: row 16 h + 4 i + grp, 16-byte piece `sub` of the strip's columns
        float *place[8];
        uint32_t there = 0u;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int orow = __shfl_sync(0xffffffffu, my_out, 4 * r + grp);
          place[r] = out + (size_t)(orow >= 0 ? orow : 0) * c_out + col0 + sub * 4;
          if (orow >= 0) there |= 1u << r;
        }
        // A 32 x 32 block at a time.  The 32 columns of 16 lanes' rows go to shared memory, then four rows per pass come back with
        // eight neighbouring lanes holding the 128 contiguous bytes of one output row: the
        // reductions reach L2 as whole 128-byte lines (the L2 slices take ~20 % more bytes per
        // second in that shape than in 64-byte pieces).
        for (int b = part; b < n_blocks; b += PL_EPI_WARPS / 4) {
          uint32_t v[32];
          tmem_ld16(v, taddr + (uint32_t)(b * 32));
          if (b * 32 + 16 < p.n_cta) tmem_ld16(v + 16, taddr + (uint32_t)(b * 32 + 16));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const bool in = b * 32 + sub * 4 < cols;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if ((lane >> 4) == h) {
#pragma unroll
              for (int q = 0; q < 8; ++q)
                *(uint4 *)(blk + (lane & 15) * PL_STG_ROW + ((q ^ (lane & 7)) << 4)) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
            __syncwarp();
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = *(const float4 *)(blk + (4 * i + grp) * PL_STG_ROW + ((sub ^ ((4 * i + grp) & 7)) << 4));
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (!in || !((there >> (4 * h + i)) & 1u)) continue;
              float *dst = place[4 * h + i] + b * 32;
              if (vec_ok) {
                red_add_v4(dst, x[i]);
              } else {
                const int cc = col0 + b * 32 + sub * 4;
                atomicAdd(dst, x[i].x);
                if (cc + 1 < c_out) atomicAdd(dst + 1, x[i].y);
                if (cc + 2 < c_out) atomicAdd(dst + 2, x[i].z);
                if (cc + 3 < c_out) atomicAdd(dst + 3, x[i].w);
              }
            }
          }
        }
        // this warp has read its share of the buffer: the MMA thread may overwrite it
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR && rank == 1) st_async_v4(news0, make_uint4(0u, 0u, 0u, 0u), peer_address(smem_u32(acce_bars + buf), 0u));
          else if (PAIR && ew == 0) mbar_expect_tx(smem_u32(acce_bars + buf), PL_EPI_WARPS * 16u);     // (an arrival too)
          else mbar_arrive(smem_u32(acce_bars + buf));
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag) report_expired(status, p.alarm);
  if (PAIR) {                                              // neither leaves while the other may still signal it
    cluster_sync();
    if (warp == mma_warp) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * p.acc_cols)) : "memory");
    cluster_sync();
  } else if (warp == mma_warp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * p.acc_cols)) : "memory");
  }
}

#define PL_ARGS const float *__restrict__ staged, const uint4 *__restrict__ packed, int c_out, const int32_t *__restrict__ pair_out, const int32_t *__restrict__ pair_in, \
      const int32_t *__restrict__ starts, const int4 *__restrict__ strips, const int32_t *__restrict__ owner, const int32_t *__restrict__ n_strips, \
      float *__restrict__ out, int32_t *status, const __grid_constant__ PlParams p
template <bool F16>
__global__ void __launch_bounds__((PL_PRODUCERS + 1 + PL_EPI_WARPS) * 32, 1) conv_fwd_pairs_kernel(PL_ARGS) {
  after_previous();
  conv_fwd_pairs_body<F16, false>(staged, packed, c_out, pair_out, pair_in, starts, strips, owner, n_strips, out, status, p);
}
template <bool F16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((PL_PRODUCERS + 1 + PL_EPI_WARPS) * 32, 1) conv_fwd_pairs_by_two_kernel(PL_ARGS) {
  after_previous();
  conv_fwd_pairs_body<F16, true>(staged, packed, c_out, pair_out, pair_in, starts, strips, owner, n_strips, out, status, p);
}
#undef PL_ARGS

static size_t pl_smem_bytes(const PlParams &p) {
  return (size_t)p.w_bytes + (size_t)p.stages * PL_A_BYTES + PL_STG_BYTES + PL_CTRL_BYTES + 1024 /*alignment slack*/;
}

// Shapes the kernel covers: the filter matrix of one offset (or one range of its output channels)
// resident in shared memory next to at least three ring slots.
static bool pl_params(int c_in, int c_out, int precision, PlParams &p, bool by_two = true) {
  p.pair = 0;
  const bool is16 = precision == SSC_PREC_F16 || precision == SSC_PREC_BF16;
  if (!is16 && tf32_offsets_per_row(c_in) > 1) return false;   // those filters are packed several offsets per row
  const int words = is16 ? f16_row_words(c_in) : c_in;
  int tile_n, n_tiles;
  if (!tc_operand_layout(words, c_out, &p.k_slabs, &p.n_pad, &tile_n, &n_tiles)) return false;
  p.f16 = is16 ? 1 : 0;
  p.slab_words = is16 ? words : c_in;
  p.row_words = is16 ? words : ((c_in + 3) & ~3);
  const size_t budget = 227 * 1024 - PL_STG_BYTES - PL_CTRL_BYTES - 1024;
  p.n_split = 0;
  for (int ns = 1; ns <= 8; ++ns) {
    if (p.n_pad % (16 * ns) != 0) continue;
    const int n_cta = p.n_pad / ns;
    if (n_cta > 256) continue;
    const size_t w = (size_t)p.k_slabs * n_cta * 128;
    if (w + 3 * (size_t)PL_A_BYTES > budget) continue;
    p.n_split = ns;
    p.n_cta = n_cta;
    p.w_bytes = (int)w;
    break;
  }
  if (p.n_split == 0 || p.n_cta < 16) return false;
  // A matrix that one CTA cannot hold whole goes to two (with ranges of its channels every row is gathered once per range): 177 k rows
  // of 256 -> 256 TF32 866 -> 679 us, 50 k rows of 208 -> 224 330 -> 239.  One that fits stays: 41 k rows of 192 -> 192 bf16 178 and 182.
  if (by_two && p.n_split > 1 && p.n_pad <= 256 && (size_t)p.k_slabs * (p.n_pad / 2) * 128 + 3 * (size_t)PL_A_BYTES <= budget) {
    p.pair = 1;
    p.n_split = 1;
    p.n_cta = p.n_pad;
    p.w_bytes = p.k_slabs * (p.n_pad / 2) * 128;
  }
  p.acc_cols = 32;
  while (p.acc_cols < p.n_cta) p.acc_cols <<= 1;
  p.ctas_per_sm = 1;      // 13 warps with ~120 registers each: one persistent CTA per SM
  const size_t b = budget;
  p.stages = (int)((b - p.w_bytes) / PL_A_BYTES);
  if (p.stages > PL_MAX_STAGES) p.stages = PL_MAX_STAGES;
  if (p.stages < 3) return false;
  p.threads = (PL_PRODUCERS + 1 + PL_EPI_WARPS) * 32;
  const uint32_t fmt = is16 ? (precision == SSC_PREC_BF16 ? 1u : 0u) : 2u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.n_cta >> 3) << 17) | ((uint32_t)((p.pair ? 2 * PL_M : PL_M) >> 4) << 24);
  return true;
}

bool conv_pairs_supported(int c_in, int c_out, int precision) {
  PlParams p;
  return pl_params(c_in, c_out, precision, p);
}

static size_t max_strips(int K) { return (size_t)PL_MAX_CTAS + 16 * (size_t)K + 16; }   // mains + tails of K * n_split (<= 8) virtual offsets

size_t conv_pairs_strip_bytes(int K) { return 256 + max_strips(K) * (sizeof(int4) + sizeof(int32_t)); }

// `staged`: the operand image of the feature rows (ssc_conv_stage); `strip_mem`: conv_pairs_strip_bytes(K) bytes.
// rows: the features to be staged, null where `staged` holds their image.
int conv_fwd_pairs(const float *rows, int n_in, void *staged, int c_in, const void *packed, int K, int c_out, int precision,
                   const PairLists &pl, int n_out, float *out, int32_t *status, void *strip_mem, cudaStream_t st) {
  PlParams p;
  // Lists of few pairs, most of them shorter than a CTA's 128, leave the second CTA of a tile idle, and with channels that are added one by one
  // the adding, which it does not share.  27 offsets, 2 and 9 neighbours a row, ranges of channels and two CTAs, us: 200 rows of
  // 256 -> 256 15.0, 15.0 and 15.5, 15.8; 600 15.1, 20.1 and 16.1, 17.0; 2000 20.2, 26.6 and 17.4, 23.8; of 200 -> 250 200 rows 17.4, 20.7 and 17.7, 23.6;
  // 2000 28.4, 48.0 and 31.6, 50.6; 5000 40.0, 109.9 and 36.7, 90.7.  (125 offsets: 35.5 and 29.0 for 200 rows.)
  const bool by_two = K >= 64 || n_out >= ((c_out & 3) == 0 ? 1024 : 4096);
  if (K > 256 || !pl_params(c_in, c_out, precision, p, by_two))
    return fail(SSC_ERR_INVALID, "conv_fwd_pairs: shape (c_in %d, c_out %d, kernel volume %d) not covered by the pair-list kernel", c_in, c_out, K);
  p.alarm = alarm_word();
  int n_ctas = sm_count() * p.ctas_per_sm;
  if (n_ctas > PL_MAX_CTAS) n_ctas = PL_MAX_CTAS;
  if (p.pair) n_ctas &= ~1;
  int32_t *hdr = (int32_t *)strip_mem;
  int4 *strips = (int4 *)((uint8_t *)strip_mem + 256);
  int32_t *owner = (int32_t *)(strips + max_strips(K));
  // the image in 16-byte pieces where rows and image have no padding (else by the general kernel), the output likewise
  const bool bf16 = precision == SSC_PREC_BF16;
  const int per_piece = p.f16 ? 8 : 4;
  long long n_stage = 0, n_clear = 0;
  cudaError_t e;
  if (rows != nullptr && n_in > 0) {
    if (c_in % per_piece == 0 && (((uintptr_t)rows | (uintptr_t)staged) & 15u) == 0) {
      n_stage = (long long)n_in * c_in / per_piece;
    } else {
      const int rc = p.f16 ? stage_features_16(rows, n_in, c_in, bf16, staged, st) : stage_features(rows, n_in, c_in, staged, st);
      if (rc != SSC_OK) return rc;
    }
  }
  if (((uintptr_t)out & 15u) == 0 && ((long long)n_out * c_out & 3) == 0) {
    n_clear = (long long)n_out * c_out / 4;
  } else {
    e = cudaMemsetAsync(out, 0, (size_t)n_out * c_out * sizeof(float), st);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd_pairs: clearing the output: %s", cudaGetErrorString(e));
  }
  const int want = ceil_div(n_stage > n_clear ? n_stage : n_clear, PL_MAX_CTAS * 2), most = sm_count() * 6;
  const int blocks = 1 + (want < most ? want : most);
  auto prepare = p.f16 ? pl_prepare_kernel<true> : pl_prepare_kernel<false>;
  { launch_ready(prepare, dim3(blocks), dim3(PL_MAX_CTAS), 0, st, pl.starts, K, p.n_split, p.pair ? 2 * PL_M : PL_M, p.pair ? n_ctas / 2 : n_ctas, hdr, strips, owner, (const float4 *)rows, n_stage, bf16 ? 1 : 0, (uint4 *)staged, (float4 *)out, n_clear); note_launches(1); }
  SSC_CHECK_LAUNCH("pl_prepare");
  const size_t smem = pl_smem_bytes(p);
  auto kernel = p.pair ? (p.f16 ? conv_fwd_pairs_by_two_kernel<true> : conv_fwd_pairs_by_two_kernel<false>)
                       : (p.f16 ? conv_fwd_pairs_kernel<true> : conv_fwd_pairs_kernel<false>);
  e = allow_smem((const void *)kernel, smem);
  if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd_pairs: smem attribute: %s", cudaGetErrorString(e));
  { launch_ready(kernel, dim3(n_ctas), dim3(p.threads), smem, st, (const float *)staged, (const uint4 *)packed, c_out, pl.pair_out, pl.pair_in, pl.starts,
                                          strips, owner, hdr, out, status, p); note_launches(1); }
  SSC_CHECK_LAUNCH("conv_fwd_pairs");
  return SSC_OK;
}

}  // namespace ssc

using namespace ssc;

extern "C" size_t ssc_conv_pairs_list_bytes(int K, int n_out) {
  if (K < 1 || K > 256 || n_out < 0) return 0;
  return align_up(pair_lists_bytes(K, n_out), 256) + conv_pairs_strip_bytes(K);
}

extern "C" int ssc_conv_pairs_supported(int c_in, int c_out, int precision) {
  return (c_in >= 1 && c_out >= 1 && conv_pairs_supported(c_in, c_out, precision)) ? 1 : 0;
}

extern "C" int ssc_conv_pairs_build(const int32_t *nbr, int K, int n_out, void *lists, size_t list_bytes, void *stream) {
  SSC_REQUIRE(K >= 1 && K <= 256 && n_out >= 1 && nbr && lists, "conv_pairs_build: bad arguments");
  SSC_REQUIRE(list_bytes >= ssc_conv_pairs_list_bytes(K, n_out) && ((uintptr_t)lists & 255u) == 0,
              "conv_pairs_build: list buffer too small or not 256-byte aligned");
  // the strip table kept behind the lists belongs to the old lists: forget it
  void *strip_mem = (uint8_t *)lists + align_up(pair_lists_bytes(K, n_out), 256);
  cudaError_t e = cudaMemsetAsync(strip_mem, 0, 256, as_stream(stream));
  if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_pairs_build: %s", cudaGetErrorString(e));
  return pair_lists_build(nbr, K, n_out, lists, nullptr, as_stream(stream));
}

extern "C" int ssc_conv_fwd_pairs(const float *features, int n_in, int c_in, const void *packed, int K, int c_out,
                                  void *lists, size_t list_bytes, int n_out, int precision, float *out, int32_t *status,
                                  void *scratch, size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(c_in > 0 && c_out > 0 && K > 0 && K <= 256 && n_in >= 0 && n_out >= 0, "conv_fwd_pairs: bad sizes");
  const bool prestaged = (precision & SSC_CONV_PRESTAGED) != 0;
  precision &= ~SSC_CONV_PRESTAGED;
  if (n_out == 0) return SSC_OK;
  SSC_REQUIRE(packed && lists && out && scratch && (n_in == 0 || features || prestaged), "conv_fwd_pairs: null pointer");
  SSC_REQUIRE(precision == SSC_PREC_TF32 || precision == SSC_PREC_F16 || precision == SSC_PREC_BF16,
              "conv_fwd_pairs: precision %d has no tensor-core form", precision);
  SSC_REQUIRE(list_bytes >= ssc_conv_pairs_list_bytes(K, n_out) && ((uintptr_t)lists & 255u) == 0,
              "conv_fwd_pairs: list buffer too small or not 256-byte aligned");
  SSC_REQUIRE(scratch_bytes + 16 >= ssc_conv_scratch_bytes(n_in, c_in, c_out, precision) && ((uintptr_t)scratch & 15u) == 0,
              "conv_fwd_pairs: staging buffer too small or not 16-byte aligned");
  cudaStream_t st = as_stream(stream);
  const PairLists pl = pair_lists_view(lists, K, n_out);
  void *strip_mem = (uint8_t *)lists + align_up(pair_lists_bytes(K, n_out), 256);
  return conv_fwd_pairs(prestaged ? nullptr : features, n_in, scratch, c_in, packed, K, c_out, precision, pl, n_out, out, status, strip_mem, st);
}
