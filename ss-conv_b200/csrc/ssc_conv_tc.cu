// Output-stationary gather-GEMM on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// One CTA owns 128 output rows (consecutive ones, or those of a row order) and runs a warp-specialised pipeline over the
// steps (kernel offset) x (128-byte slab of the input's channels); the operand ring has up to eight slots:
//   * producer warps fetch the rows' neighbours into the slot, in the K-major 128-byte-swizzled operand layout;
//     the pre-packed filter slab (already rounded, already in operand layout) comes with one bulk
//     asynchronous copy, and both arrive on the slot's "full" mbarrier.
//   * one MMA warp waits for it, issues tcgen05.mma (M=128, N<=256), accumulating in tensor memory (fp32),
//     rows without a neighbour switched off by the output-lane mask, and commits the group to the slot's
//     "empty" mbarrier, which frees the slot.
// There is no CTA-wide barrier inside the loop.  Accumulators stay in tensor memory across all offsets; the
// producer warps then read them with tcgen05.ld and write each output row exactly once (no scatter
// atomics, one stated order of the sums).
// Two kernels share this plan.  conv_fwd_rows_kernel is the one the layers run: rows staged once (rounded to TF32, or
// fp16 / bf16), four warps to a slot.  conv_fwd_tf32_kernel takes what it does not cover: layers of up to 16
// input channels, several offsets per operand row (GROUPED), and fp32 rows without a staging buffer, rounded
// in shared memory (callers that bring no scratch); a producer warp per slot there.
//
// Every wait on an mbarrier is bounded: on expiry the thread records an error in `status`
// through a shared flag, every other wait then gives up too, and the kernel frees its tensor
// memory and returns.
#include "ssc_conv_epilogue.cuh"
#include <type_traits>

namespace ssc {

constexpr int TC_M = 128;
constexpr int TC_SLAB = 32;            // tf32 elements per 128-byte operand row
constexpr int TC_MAX_STAGES = 8;       // producer warps = ring slots
constexpr int TC_EPI_WARPS = 4;        // warps 0..3 also run the epilogue (one TMEM lane quarter each)
constexpr int TC_A_BYTES = TC_M * 128;
constexpr int TC_CTRL_BYTES = 1024;

struct TcParams {
  int k_slabs;    // ceil(c_in / 32)
  int n_pad;      // padded output channels (n_tiles * tile_n)
  int n_tiles;    // MMA instructions along N per k-step
  int tile_n;     // N of one MMA, multiple of 16, <= 256
  int tmem_cols;  // power of two >= max(32, n_pad)
  int stages;     // operand ring depth = number of producer warps (>= 4)
  int threads;    // (max(n_prod, 4) + 1) * 32
  int ctas;       // CTAs that share an SM
  int n_prod;     // producer warps: a multiple of the slots (several warps share a slot's rows)
  int b_bytes;    // n_pad * 128
  int sps;        // 32-channel slabs per ring slot (a step covers sps slabs of one kernel offset)
  int k_groups;   // ceil(k_slabs / sps) = steps per kernel offset
  int nt_cta;     // N tiles handled by one CTA: n_tiles, or 1 when the N tiles are spread over gridDim.y
  int n_cta;      // nt_cta * tile_n: accumulator columns / filter-slab rows per CTA
  int fmt16;      // 16-bit operands: 0 = fp16, 1 = bf16 (operand format field of the instruction descriptor)
  int last_kk;    // MMA k-steps (32 bytes of K each) that hold real channels in the LAST slab: 1..4
  int opk;        // kernel offsets per 128-byte operand row: 1, or 32 / c_pad for TF32 layers with c_pad = 4, 8, 16
                  // channels (a first layer with 3 input channels packs 8 offsets into one step)
  int rev;        // 1: the table's row of kernel offset kappa is K - 1 - kappa (the transpose of a centred submanifold table)
  int32_t *alarm; // mapped host word that tells of an expired wait (may be NULL)
  int pair;       // 1: two CTAs with 128 rows each share the filter slabs (half a slab in each) and the products
  int nbr_by_pos; // 1: the table's columns are already in the order of `order` (column j <-> output row order[j])
};

// Shared-memory plan: [stages x (A 16 KB + B)] [control 1 KB].
static bool tc_params(int c_in, int c_out, TcParams &p, bool split_n = false, int max_ctas = 4, int opk = 1, bool pair = false) {
  p.pair = pair;
  p.k_slabs = (c_in + TC_SLAB - 1) / TC_SLAB;
  p.last_kk = (c_in - (p.k_slabs - 1) * TC_SLAB + 7) / 8;     // c_in counts 4-byte words of an operand row
  p.opk = opk;
  p.nbr_by_pos = 0;
  p.rev = 0;
  p.alarm = nullptr;
  if (opk > 1) {     // grouped offsets: one full slab per group of offsets
    p.k_slabs = 1;
    p.last_kk = 4;
  }
  int n16 = (c_out + 15) / 16 * 16;
  p.n_tiles = (n16 + 255) / 256;
  p.tile_n = ((n16 + p.n_tiles - 1) / p.n_tiles + 15) / 16 * 16;
  p.n_pad = p.n_tiles * p.tile_n;
  if (p.n_pad > 512) return false;
  // A layer with few row tiles and more than one N tile gets one CTA per (row tile, N tile): more
  // CTAs in flight, each with a smaller accumulator and filter slab (the rows are gathered twice).
  p.nt_cta = (split_n && p.n_tiles > 1) ? 1 : p.n_tiles;
  p.n_cta = p.nt_cta * p.tile_n;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.n_cta) p.tmem_cols <<= 1;
  p.b_bytes = p.n_cta * 128;
  // One 32-channel slab per step: two slabs per step halve the per-step bookkeeping but also the
  // resident CTAs, and measured slower (0.21 vs 0.18 ms on the 64 -> 76 channel layer).
  p.sps = 1;
  p.fmt16 = 0;
  p.k_groups = (p.k_slabs + p.sps - 1) / p.sps;
  int stage = p.sps * (TC_A_BYTES + (pair ? p.b_bytes / 2 : p.b_bytes));
  // behind the slots: control block, alignment slack
  int fixed = TC_CTRL_BYTES + 1024;
  // Resident CTAs hide each other's per-step latencies, so take as many per SM as tensor
  // memory (512 columns) and shared memory (two ring slots each at least) allow, up to four and to as many as the launch has for an
  // SM: what is left of the shared memory goes into ring slots (a deeper pipeline is what few CTAs have against the latency of a step).
  int ctas = 512 / p.tmem_cols;
  if (ctas > 4) ctas = 4;
  if (ctas > max_ctas) ctas = max_ctas;
  while (ctas > 1 && ((227 * 1024) / ctas - 1024 - fixed) / stage < 2) --ctas;
  p.stages = ((227 * 1024) / ctas - 1024 - fixed) / stage;
  if (p.stages > TC_MAX_STAGES) p.stages = TC_MAX_STAGES;
  p.ctas = ctas;
  if (p.stages < 2) return false;
  // producer warps: one per slot with four or more slots, else the slots' rows are split over four warps
  p.n_prod = p.stages < TC_EPI_WARPS ? (TC_EPI_WARPS / p.stages) * p.stages : p.stages;
  p.threads = ((p.n_prod > TC_EPI_WARPS ? p.n_prod : TC_EPI_WARPS) + 1) * 32;
  return true;
}

// Geometry of the packed filter image, for the other kernels that consume it.
bool tc_operand_layout(int c_in, int c_out, int *k_slabs, int *n_pad, int *tile_n, int *n_tiles) {
  TcParams p;
  if (!tc_params(c_in, c_out, p)) return false;
  *k_slabs = p.k_slabs;
  *n_pad = p.n_pad;
  *tile_n = p.tile_n;
  *n_tiles = p.n_tiles;
  return true;
}

// Filter packing: filters [K, c_in, c_out] fp32 -> [K][k_slabs][n_pad rows][32 tf32] in the
// swizzled operand layout (row = output channel, 16-byte chunk index XOR (row & 7)).
__global__ void pack_filters_tf32_kernel(const float *__restrict__ filters, int K, int c_in, int c_out, TcParams p,
                                         uint4 *__restrict__ packed) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)K * p.k_slabs * p.n_pad * 8;
  if (t >= total) return;
  int chunk = (int)(t & 7);
  long long r = t >> 3;
  int n = (int)(r % p.n_pad);
  r /= p.n_pad;
  int slab = (int)(r % p.k_slabs);
  int kappa = (int)(r / p.k_slabs);
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int ci = slab * TC_SLAB + chunk * 4 + q;
    float f = (ci < c_in && n < c_out) ? filters[((size_t)kappa * c_in + ci) * c_out + n] : 0.f;
    v[q] = to_tf32(f);
  }
  size_t block = ((size_t)kappa * p.k_slabs + slab) * (size_t)(p.n_pad * 8);
  size_t off = (size_t)(n >> 3) * 64 + (size_t)(n & 7) * 8 + (size_t)(chunk ^ (n & 7));
  packed[block + off] = make_uint4(v[0], v[1], v[2], v[3]);
}

// The grouped form for few input channels (c_pad = 4, 8, 16; opk = 32 / c_pad offsets per operand row):
// [ceil(K / opk)][n_pad rows][32 tf32], word (o' * c_pad + c) of a row = W[g * opk + o', c, n].
__global__ void pack_filters_tf32_grouped_kernel(const float *__restrict__ filters, int K, int c_in, int c_out, int c_pad,
                                                 int opk, int n_groups, int n_pad, uint4 *__restrict__ packed) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)n_groups * n_pad * 8;
  if (t >= total) return;
  const int chunk = (int)(t & 7);
  long long r = t >> 3;
  const int n = (int)(r % n_pad), g = (int)(r / n_pad);
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int w = chunk * 4 + q, o = w / c_pad, ci = w - o * c_pad, kappa = g * opk + o;
    const float f = (o < opk && kappa < K && ci < c_in && n < c_out) ? filters[((size_t)kappa * c_in + ci) * c_out + n] : 0.f;
    v[q] = to_tf32(f);
  }
  const size_t block = (size_t)g * (size_t)(n_pad * 8);
  const size_t off = (size_t)(n >> 3) * 64 + (size_t)(n & 7) * 8 + (size_t)(chunk ^ (n & 7));
  packed[block + off] = make_uint4(v[0], v[1], v[2], v[3]);
}

// Warps 0 .. n_prod-1 are producers (warp w <-> ring slot w; with fewer than four slots the
// spare warps only help in the prologue and epilogue), the last warp issues the MMAs.
// GROUPED: staged rows of few channels, several kernel offsets per operand row; else fp32 rows as they are, rounded
// in shared memory.
template <bool GROUPED>
__global__ void __launch_bounds__((TC_MAX_STAGES + 1) * 32)
conv_fwd_tf32_kernel(const float *__restrict__ features, int c_in, const uint4 *__restrict__ packed, int K,
                     int c_out, const int32_t *__restrict__ nbr, int n_out, float *__restrict__ out,
                     int32_t *status, TcParams p, const int32_t *__restrict__ n_out_dev,
                     const int32_t *__restrict__ order) {
  after_previous();
  // `order` (may be NULL): the rows of tile t are order[128 t .. 128 t + 127] instead of the same
  // consecutive numbers; rows that use the same kernel offsets, put next to each other, make a
  // tile skip the offsets none of them uses.
  // n_out is the row stride of nbr and the launch bound; the exact row count may still be on the
  // device (a rulebook sized optimistically): CTAs past it have nothing to do.
  const int n_rows = live_rows(n_out, n_out_dev);
  if ((int)blockIdx.x * TC_M >= n_rows) return;
  extern __shared__ uint8_t smem_raw[];
  // operand stages need 1024-byte alignment for the 128-byte swizzle
  uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  const int stage_bytes = p.sps * (TC_A_BYTES + p.b_bytes);   // [sps x gathered slab][sps x filter slab]
  uint8_t *ctrl = smem + (size_t)p.stages * stage_bytes;
  uint64_t *empty_bars = (uint64_t *)ctrl;                 // [stages] slot free (its MMAs retired)
  uint64_t *fulla_bars = (uint64_t *)(ctrl + 64);          // [stages] gathered rows ready
  uint64_t *done_bar = (uint64_t *)(ctrl + 192);           // all MMAs of the tile retired
  uint32_t *tmem_slot = (uint32_t *)(ctrl + 200);
  volatile int *abort_flag = (volatile int *)(ctrl + 204);
  int *n_act_s = (int *)(ctrl + 208);
  uint8_t *act_flag = ctrl + 256;                          // [256]
  uint8_t *act_list = ctrl + 512;                          // [256]
  uint32_t *slot_masks = (uint32_t *)(ctrl + 768);         // [stages][4] rows of the step WITHOUT a neighbour

  const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
  const int n_warps = blockDim.x >> 5;
  const int mma_warp = n_warps - 1;
  const int m0 = blockIdx.x * TC_M;
  const int nt0 = (int)blockIdx.y * p.nt_cta;   // first N tile of this CTA
  const int S = p.stages;
  // table row of a kernel offset
  auto table = [&](int kap) { return nbr + (size_t)(p.rev ? K - 1 - kap : kap) * n_out; };

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(empty_bars + s), 1);
      // one barrier per slot for both operands: every producer lane arrives for its gathered rows,
      // and the lane that starts the filter copy arrives once more with the copy's byte count
      // (the issuing thread then pays one barrier round trip per step, not two)
      mbar_init(smem_u32(fulla_bars + s), 32u * (uint32_t)(p.n_prod / S) + 1u);
    }
    mbar_init(smem_u32(done_bar), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)p.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else if (!GROUPED) {   // (grouped offsets: every group is a step, absent neighbours are zero-filled pieces)
    // which kernel offsets touch this tile: four offsets per pass so that 16 loads are in
    // flight per lane before the first ballot
    int scan_rows[4];  // this lane's four rows of the tile (-1 past the end)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = m0 + q * 32 + lane;
      scan_rows[q] = r < n_rows ? ((order && !p.nbr_by_pos) ? __ldg(order + r) : r) : -1;
    }
    for (int k0 = warp * 4; k0 < K; k0 += mma_warp * 4) {
      int v[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = scan_rows[q];
          v[i][q] = (k0 + i < K && r >= 0) ? __ldg(table(k0 + i) + r) : -1;
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        bool any = (v[i][0] >= 0) | (v[i][1] >= 0) | (v[i][2] >= 0) | (v[i][3] >= 0);
        unsigned b = __ballot_sync(0xffffffffu, any);
        if (lane == 0 && k0 + i < K) act_flag[k0 + i] = b != 0;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp < TC_EPI_WARPS) {
    // Clear the accumulators.  Every MMA below accumulates, and rows without a neighbour at a
    // step are switched off through the MMA's disable-output-lane mask, so the gathered operand
    // never has to hold zero rows (stale rows of an earlier step are simply not written back).
    for (int c0 = 0; c0 < p.n_cta; c0 += 16) {
      const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
          "r"(0u)
          : "memory");
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    int n = 0;
    if (GROUPED) {   // steps are groups of opk offsets, all of them
      for (int g = 0; g * p.opk < K; ++g) act_list[n++] = (uint8_t)g;
    } else {
      for (int kappa = 0; kappa < K; ++kappa)
        if (act_flag[kappa]) act_list[n++] = (uint8_t)kappa;
    }
    *n_act_s = n;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const int n_act = *n_act_s;
  const int n_iter = n_act * p.k_groups;
  const uint32_t smem_base = smem_u32(smem);

  const int n_prod = p.n_prod;  // producer warps (2 slots -> 4 warps)
  if (warp < n_prod) {
    // ====================== producer warp ====================================================
    // With S >= 4 ring slots, warp w owns slot w and prepares all 128 rows of the steps
    // w, w+S, ...; with fewer slots several warps share a slot and split its rows.
    const int slot = warp % S;
    const int share = n_prod / S;              // warps per slot
    const int part = warp / S;                 // which share of the rows this warp prepares
    const int q_per = 4 / share;               // 32-row groups per warp (share is 1, 2 or 4)
    const int q0 = part * q_per;
    const bool vec_ok = (c_in & 3) == 0;
    const uint32_t slot_addr = smem_base + (uint32_t)slot * (uint32_t)stage_bytes;
    uint8_t *slot_ptr = smem + (size_t)slot * stage_bytes;
    (void)slot_ptr;
    const uint32_t sw = (uint32_t)(lane & 7);
    // row q*32+lane of the slot: 8-row group (q*4 + lane/8), row-in-group lane%8
    uint32_t row_off[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) row_off[q] = (uint32_t)(q * 4 + (lane >> 3)) * 1024u + sw * 128u;
    uint32_t par = 0;          // parity of the slot's current use
    int src[4], nxt[4];
    int my_rows[4];            // this lane's four rows of the tile (-1 past the end)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = m0 + q * 32 + lane;
      my_rows[q] = r < n_rows ? ((order && !p.nbr_by_pos) ? __ldg(order + r) : r) : -1;
    }
    auto load_rows = [&](int j, int *dst) {
      const int kap = act_list[j / p.k_groups];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        dst[q] = (q >= q0 && q < q0 + q_per && my_rows[q] >= 0) ? __ldg(table(kap) + my_rows[q]) : -1;
    };
    if (GROUPED) {
      // Grouped offsets (TF32, staged rows of c_in = 4, 8 or 16 floats): the 128-byte operand row of a
      // step holds the rows' neighbours at opk consecutive offsets side by side; a missing neighbour is
      // a zero-filled piece, so no row is ever switched off.  The filter slab of the group is packed to match.
      const int cpc = c_in >> 2;                   // 16-byte chunks per offset
      // (the loops over the 32-row groups are kept rolled: this path runs four steps per CTA, and as
      //  straight-line code it spent most of its time waiting for instruction fetches)
      for (int j = slot; j < n_iter; j += S) {
        const int group = act_list[j];
        if (j >= S) {
          if (!mbar_wait_warp(smem_u32(empty_bars + slot), par ^ 1u, abort_flag)) break;
          tc_fence_after();
        }
        if (part == 0 && lane == 0) {
          const uint4 *bsrc = packed + (size_t)group * (size_t)(p.n_pad * 8) + (size_t)nt0 * (size_t)(p.tile_n * 8);
          const uint32_t bar = smem_u32(fulla_bars + slot), nbytes = (uint32_t)p.b_bytes;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(nbytes) : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           slot_addr + (uint32_t)TC_A_BYTES),
                       "l"(bsrc), "r"(nbytes), "r"(bar)
                       : "memory");
        }
#pragma unroll 1
        for (int q = q0; q < q0 + q_per; ++q) {
          const int row = m0 + q * 32 + lane;
          const int my_row = row < n_rows ? ((order && !p.nbr_by_pos) ? __ldg(order + row) : row) : -1;
          int idx[8];
#pragma unroll
          for (int o = 0; o < 8; ++o) {
            const int kap = group * p.opk + o;
            idx[o] = (o < p.opk && kap < K && my_row >= 0) ? __ldg(table(kap) + my_row) : -1;
          }
          if (lane == 0) slot_masks[slot * 4 + q] = 0u;          // every row takes part
          const uint32_t a_row = slot_addr + (uint32_t)(q * 4 + (lane >> 3)) * 1024u + sw * 128u;
#pragma unroll
          for (int o = 0; o < 8; ++o) {
            if (o >= p.opk) break;
            const int src_row = idx[o];
            const float *fp = features + (size_t)(src_row >= 0 ? src_row : 0) * c_in;
#pragma unroll 1
            for (int cc = 0; cc < cpc; ++cc) {
              const uint32_t chunk = (uint32_t)(o * cpc + cc);
              cp_async16_cg(a_row + ((chunk ^ sw) << 4), fp + cc * 4, src_row >= 0 ? 16u : 0u);
            }
          }
        }
        cp_async_commit();
        cp_async_wait(0);
        fence_async_smem();
        mbar_arrive(smem_u32(fulla_bars + slot));
        par ^= 1u;
      }
    } else {
    if (slot < n_iter) load_rows(slot, nxt);
    for (int j = slot; j < n_iter; j += S) {
      const int act = j / p.k_groups, slab0 = (j - act * p.k_groups) * p.sps;
      const int n_sub = min(p.sps, p.k_slabs - slab0);   // slabs of this step
      const int kappa = act_list[act];
#pragma unroll
      for (int q = 0; q < 4; ++q) src[q] = nxt[q];
      if (j + S < n_iter) load_rows(j + S, nxt);  // neighbour rows of this warp's next step
      unsigned have[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) have[q] = __ballot_sync(0xffffffffu, src[q] >= 0);
      if (j >= S) {
        if (!mbar_wait_warp(smem_u32(empty_bars + slot), par ^ 1u, abort_flag)) break;
        tc_fence_after();
      }
      if (part == 0 && lane == 0) {  // the pre-packed filter slab of this step: one bulk copy
        const uint4 *bsrc = packed + ((size_t)kappa * p.k_slabs + slab0) * (size_t)(p.n_pad * 8) +
                            (size_t)nt0 * (size_t)(p.tile_n * 8);
        const uint32_t bar = smem_u32(fulla_bars + slot), nbytes = (uint32_t)(n_sub * p.b_bytes);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(nbytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         slot_addr + (uint32_t)(p.sps * TC_A_BYTES)),
                     "l"(bsrc), "r"(nbytes), "r"(bar)
                     : "memory");
      }
      uint32_t present = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q)    // rows of this step that the MMA must leave alone
        if (lane == 0 && q >= q0 && q < q0 + q_per) slot_masks[slot * 4 + q] = ~have[q];
      for (int ss = 0; ss < n_sub; ++ss) {
      const int ch0 = (slab0 + ss) * TC_SLAB;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (src[q] >= 0 && ch0 < c_in) {
          const float *fp = features + (size_t)src[q] * c_in + ch0;
          const uint32_t a_row = slot_addr + (uint32_t)(ss * TC_A_BYTES) + row_off[q];
          if (vec_ok) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {  // chunks past the last channel are zero-filled
              bool ok = ch0 + c * 4 < c_in;
              cp_async16(a_row + ((c ^ sw) << 4), ok ? (const void *)(fp + c * 4) : (const void *)features, ok ? 16u : 0u);
            }
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                bool ok = ch0 + c * 4 + e < c_in;
                cp_async4(a_row + ((c ^ sw) << 4) + 4u * e, ok ? (const void *)(fp + c * 4 + e) : (const void *)features,
                          ok ? 4u : 0u);
              }
          }
          present |= 1u << q;
        }
      }
      }
      cp_async_commit();
      cp_async_wait(0);
      // copies landed: round the gathered rows to TF32 in place
      for (int ss = 0; ss < n_sub; ++ss)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (present & (1u << q)) {
          uint8_t *row = slot_ptr + (size_t)ss * TC_A_BYTES + row_off[q];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint4 *ptr = (uint4 *)(row + ((c ^ sw) << 4));
            uint4 v = *ptr;
            v.x = to_tf32(__uint_as_float(v.x));
            v.y = to_tf32(__uint_as_float(v.y));
            v.z = to_tf32(__uint_as_float(v.z));
            v.w = to_tf32(__uint_as_float(v.w));
            *ptr = v;
          }
        }
      }
      if (present) fence_async_smem();  // make this lane's rows visible to the tensor core
      mbar_arrive(smem_u32(fulla_bars + slot));
      par ^= 1u;
    }
    }   // one offset per step
  } else if (warp == mma_warp) {
    // ================================ MMA issuer: the whole warp, one elected lane issues ========
    // slot index, parity and descriptor halves are running values; fp32 accumulator, TF32 operands
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(p.tile_n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
    const uint32_t a_lo0 = desc_lo(smem_base), slot_step = (uint32_t)stage_bytes >> 4, n_step = (uint32_t)(p.tile_n * 128) >> 4;
    const uint32_t fulla0 = smem_u32(fulla_bars), empty0 = smem_u32(empty_bars);
    uint32_t s = 0, par = 0, a_lo = a_lo0;
    int grp = 0;  // which slab group of its kernel offset the current step is
    for (int it = 0; it < n_iter; ++it) {
      if (!mbar_wait_uniform(fulla0 + s * 8u, par, abort_flag)) break;
      tc_fence_after();
      const uint4 off = *(const uint4 *)(slot_masks + s * 4u);  // rows to leave untouched
      const int n_sub = min(p.sps, p.k_slabs - grp * p.sps);
      for (int ss = 0; ss < n_sub; ++ss) {
        const uint32_t an = a_lo + (uint32_t)ss * (TC_A_BYTES >> 4);
        // k-steps of this slab that hold real channels (the rest of the last slab is zero on both
        // sides: a 3-channel first layer needs one MMA per step, not four)
        const int n_kk = grp * p.sps + ss == p.k_slabs - 1 ? p.last_kk : 4;
        for (int nt = 0; nt < p.nt_cta; ++nt) {
          const uint32_t dn = tmem_base + (uint32_t)(nt * p.tile_n);
          const uint32_t bn = a_lo + (uint32_t)(p.sps * TC_A_BYTES >> 4) + (uint32_t)ss * ((uint32_t)p.b_bytes >> 4) + (uint32_t)nt * n_step;
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              if (kk >= n_kk) break;
              mma_tf32_ss_masked(dn, an + 2u * (uint32_t)kk, bn + 2u * (uint32_t)kk, idesc, off);
            }
          }
        }
      }
      if (++grp == p.k_groups) grp = 0;
      if (elect_one()) mma_commit(empty0 + s * 8u);
      a_lo += slot_step;
      if (++s == (uint32_t)S) { s = 0; par ^= 1u; a_lo = a_lo0; }
    }
    if (elect_one()) mma_commit(smem_u32(done_bar));  // arrives once everything issued above has retired
  }

  // ================================ epilogue: TMEM -> registers -> global ====================
  if (warp < TC_EPI_WARPS) {
    __syncwarp();
    bool ok = !*abort_flag;
    ok = __all_sync(0xffffffffu, ok);
    if (ok && n_iter > 0) ok = mbar_wait_warp(smem_u32(done_bar), 0u, abort_flag);
    ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld below is warp-collective
    tc_fence_after();
    const int m_tile = m0 + warp * 32 + lane;
    const int m = m_tile < n_rows ? (order ? __ldg(order + m_tile) : m_tile) : n_rows;
    const int col0 = nt0 * p.tile_n;   // first output channel of this CTA
    for (int c0 = 0; c0 < p.n_cta && col0 + c0 < c_out; c0 += 16) {
      uint32_t r[16];
      if (ok && n_iter > 0) {
        uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int q = 0; q < 16; ++q) r[q] = 0u;
      }
      if (m < n_rows) {
        float *op = out + (size_t)m * c_out + col0 + c0;
        if ((c_out & 3) == 0) {
#pragma unroll
          for (int q = 0; q < 16; q += 4)
            if (col0 + c0 + q < c_out)
              *(float4 *)(op + q) = make_float4(__uint_as_float(r[q]), __uint_as_float(r[q + 1]),
                                                __uint_as_float(r[q + 2]), __uint_as_float(r[q + 3]));
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q)
            if (col0 + c0 + q < c_out) op[q] = __uint_as_float(r[q]);
        }
      }
    }
  }
  // a wait gave up: the instructions already issued still arrive on done_bar (committed above on
  // every path); let them retire before the accumulators are handed back
  if (warp == mma_warp && lane == 0 && *abort_flag && n_iter > 0) mbar_wait_drain(smem_u32(done_bar), 0u);
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag) report_expired(status, p.alarm);
  if (warp == mma_warp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------
// (one lane) a word for the issuing warp and the arrival that releases it.
__device__ __forceinline__ void store_and_arrive(bool on, uint32_t at, uint32_t word, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t"
      "@p st.shared.u32 [%1], %2;\n\t"
      "@p mbarrier.arrive.shared::cta.b64 _, [%3];\n\t}" ::"r"((uint32_t)on), "r"(at), "r"(word), "r"(bar)
      : "memory");
}

// The issuing warp of the kernel below: its state and its loop.  Its own chain of instructions is what it takes a step for, so
// the loop is straight: unrolled over N tiles, no way out of it from the middle, whole slabs with four products and
// no test between them, and only tables with a row order are asked whether a step has any row (in others nearly all have).  In
// isolation a step takes 225 cycles like this and took 450 with a loop of N tiles, a vote on the masks, a test before every
// product and a way out after the wait.  Two steps to a turn take 167, but the kernel's first launch after others then waits
// 3.5 us longer for instructions and later ones gain nothing.  (1.1 M rows 64 -> 76: 712 -> 690 us, 82 k rows 128 -> 152 bf16
// 67.3 -> 64.5, 47 k rows 256 -> 304 bf16 119 -> 111, 16 k rows 59.8 -> 55.7.)
struct RowsIssuer {
  uint32_t idesc, a_lo0, a_lo, s, par, full0, empty0, d0, b_bytes;
  const uint32_t *masks;      // [slots][4], with a pair of CTAs [slots][8]
  volatile int *abort_flag;
};
template <bool PAIR>
__device__ __forceinline__ void rows_commit(uint32_t bar) {
  if (PAIR) mma_commit_pair(bar);
  else mma_commit(bar);
}
template <bool F16, bool PAIR>
__device__ __forceinline__ void rows_mma(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint4 off, uint4 off2) {
  if (PAIR) mma_pair_masked<F16>(d, a_lo, b_lo, idesc, off, off2);
  else if (F16) mma_f16_ss_masked(d, a_lo, b_lo, idesc, off);
  else mma_tf32_ss_masked(d, a_lo, b_lo, idesc, off);
}
template <bool F16, int NT, bool SCAN, bool WHOLE, bool PAIR>
__device__ __forceinline__ bool rows_issue_step(RowsIssuer &w, const TcParams &p) {
  const bool alive = PAIR ? mbar_wait_straight_cluster(w.full0 + w.s * 8u, w.par, w.abort_flag) : mbar_wait_straight(w.full0 + w.s * 8u, w.par, w.abort_flag);
  fence_async_smem();                             // the rows other threads' copies left, for the tensor core
  tc_fence_after();
  const uint4 off = *(const uint4 *)(w.masks + w.s * (PAIR ? 8u : 4u));
  uint4 off2 = off;
  if (PAIR) off2 = *(const uint4 *)(w.masks + w.s * 8u + 4u);
  bool any = true;
  if (SCAN) any = __any_sync(0xffffffffu, (off.x & off.y & off.z & off.w) != 0xffffffffu);
  if (any) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const uint32_t dn = w.d0 + (uint32_t)(nt * p.tile_n), bn = w.a_lo + (uint32_t)(TC_A_BYTES >> 4) + (uint32_t)nt * ((uint32_t)(p.tile_n * (PAIR ? 64 : 128)) >> 4);
      if (WHOLE) {
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) rows_mma<F16, PAIR>(dn, w.a_lo + 2u * (uint32_t)kk, bn + 2u * (uint32_t)kk, w.idesc, off, off2);
        }
      } else {
#pragma unroll 1
        for (int kk = 0; kk < p.last_kk; ++kk)
          if (elect_one()) rows_mma<F16, PAIR>(dn, w.a_lo + 2u * (uint32_t)kk, bn + 2u * (uint32_t)kk, w.idesc, off, off2);
      }
    }
  }
  if (elect_one()) rows_commit<PAIR>(w.empty0 + w.s * 8u);
  w.a_lo += (uint32_t)(TC_A_BYTES + w.b_bytes) >> 4;
  if (++w.s == (uint32_t)p.stages) { w.s = 0; w.par ^= 1u; w.a_lo = w.a_lo0; }
  return alive;
}
template <bool F16, int NT, bool SCAN, bool PAIR>
__device__ __forceinline__ void rows_issue_all(RowsIssuer &w, const TcParams &p, int n_act) {
  const int whole = p.last_kk == 4 ? p.k_slabs : p.k_slabs - 1;   // slabs with four k-steps of real channels (the rest is zero on both sides)
  bool alive = true;
  if (whole == p.k_slabs) {
    const int n = n_act * whole;
#pragma unroll 1
    for (int i = 0; i < n && alive; ++i) alive = rows_issue_step<F16, NT, SCAN, true, PAIR>(w, p);
  } else {
#pragma unroll 1
    for (int a = 0; a < n_act && alive; ++a) {
#pragma unroll 1
      for (int i = 0; i < whole; ++i) alive &= rows_issue_step<F16, NT, SCAN, true, PAIR>(w, p);
      alive &= rows_issue_step<F16, NT, SCAN, false, PAIR>(w, p);
    }
  }
}

// The kernel for staged operands (TF32-rounded fp32 rows, or fp16 / bf16 rows: F16), one kernel offset and one
// 128-byte slab per step.  GROUPS of four warps produce, a lane per output row of the tile (and run the epilogue); two
// groups fill every other slot each.  The last warp issues the MMAs.
//
// What bounds it is the way of an operand slot: free -> rows gathered -> multiplied -> free, against the slots that
// fit an SM (eight of 26 KB for 64 -> 76 channels).  With a warp per slot that built its row lists, waited
// for its own copies and arrived, that way was 3700 cycles, of which about 2300 were the warp's own
// 250 dependent instructions.  Hence here:
//   * the four warps fill every slot together, 32 rows each, four lanes to a row, and work out the source rows
//     once per kernel offset for all its slabs;
//   * nobody waits for copies: the copies' completion arrives on the slot's barrier by itself
//     (cp.async.mbarrier.arrive.noinc), the warps go on to the next free slot, and the issuing warp orders
//     the landed rows for the tensor core (fence.proxy.async behind the barrier);
//   * table entries are loaded two offsets ahead, and whole slabs of a row are copied at constants from one address.
// Sums are accumulated in the order of the steps (ascending offset, ascending slab), whatever the tile's
// other rows need.
//
// GATED: batch norm and gated activation on the way out.  As a pass of its own (ssc_bn_gate_fwd) they read and write
// every row once more: 164 us of the 12 layers of a backbone, 320 us of 24 with bf16 rows.  A row's gate
// scalars are evaluated first, a lane per row, into shared memory; the arithmetic is that pass's, so are the bits.
//
// PAIR: two CTAs of a cluster, 128 rows each, as one product of 256 rows (cta_group::2).  Every tile brings in the whole filter image, and
// that is most of what its steps move (10 of 14 KB for 64 -> 76 channels, 20 of 26 for 152); of a pair each holds half of a slab.
// CTA 0 issues for both.  A slot of CTA 1 is full on a barrier there; its last warp passes that on, with the row masks, by one
// asynchronous store that counts on CTA 0's barrier (a store and a released arrival one after the other: 2100 cycles a step).
template <bool F16, bool GATED, int GROUPS, bool PAIR>
__device__ __forceinline__ void
conv_fwd_rows(const float *__restrict__ features, int row_words, const uint4 *__restrict__ packed, int K, int c_out,
              const int32_t *__restrict__ nbr, int n_out, float *__restrict__ out, int32_t *status, const TcParams &p,
              const int32_t *__restrict__ n_out_dev, const int32_t *__restrict__ order, const GateEpilogue &gate) {
  // Every CTA walks the filters in the same order at the same time, so each slab that is not in L2 stalls all of them.  Before
  // it waits for the kernel before this one, each thread asks for one line of 128 bytes; of a grid too small to cover the
  // image only the first slabs are asked for.  Nothing is read yet: L2 is where a filter that is still being packed is
  // written.  Strided layer with a pool 207 -> 202 us, voxel codec 206 -> 203, plain-12 network 1064 -> 1055.
  const int line = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (line < K * p.k_slabs * p.n_pad) asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)packed + (size_t)line * 128));
  after_previous();
  const int n_rows = live_rows(n_out, n_out_dev);
  if ((int)(PAIR ? blockIdx.x & ~1u : blockIdx.x) * TC_M >= n_rows) return;
  const int rank = PAIR ? (int)blockIdx.x & 1 : 0;                   // in the pair: 0 issues for both
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t empty_bars[TC_MAX_STAGES], full_bars[TC_MAX_STAGES], done_bar;
  __shared__ __align__(16) uint32_t slot_masks[TC_MAX_STAGES * (PAIR ? 8 : 4)];   // rows of the slot's step WITHOUT a neighbour
  __shared__ uint32_t act_bits[8];
  __shared__ uint8_t act_list[256];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word, n_act_s;
  volatile int *abort_flag = &abort_word;
  // operand slots need 1024-byte alignment for the 128-byte swizzle
  uint8_t *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  const int b_bytes = PAIR ? p.b_bytes >> 1 : p.b_bytes;             // (a pair's filter slab lies half in each)
  const int stage_bytes = TC_A_BYTES + b_bytes;
  const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
  constexpr int groups = GROUPS, mma_warp = groups * 4;              // producer groups of four warps
  const int quarter = warp & 3;                                      // the 32 rows of the tile a producer warp works on
  const int m0 = blockIdx.x * TC_M, nt0 = (int)blockIdx.y * p.nt_cta, S = p.stages;
  auto table = [&](int kap) { return nbr + (size_t)(p.rev ? K - 1 - kap : kap) * n_out; };

  // Rows in a row order were put together by the offsets they use, so that a tile can leave out the others: the
  // table is scanned for them first.  In any other order nearly every offset has a row among 128, the
  // scan (8 us when all CTAs of the first wave do it at once) finds nothing, and a step without a
  // row costs its filter copy but no multiplication.
  const bool scan = !PAIR && order != nullptr;
  const int m_tile = m0 + quarter * 32 + lane;    // (producers) this lane's row of the tile
  int my_row = -1;                                // its column of the table
  if (warp == mma_warp) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)p.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)p.tmem_cols) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  } else {
    if (tid < 8) act_bits[tid] = 0u;
    if (tid == 32) {
      for (int s = 0; s < S; ++s) {
        mbar_init(smem_u32(empty_bars + s), 1);
        // 128 arrivals by copies, one per warp for the row mask, one for the filter copy's byte count, which in the
        // issuing CTA of a pair has 16 bytes more, of the store that tells of all these in the other
        mbar_init(smem_u32(full_bars + s), 128 + 4 + 1);
      }
      mbar_init(smem_u32(&done_bar), 1);
      *abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (m_tile < n_rows) my_row = (order && !p.nbr_by_pos) ? __ldg(order + m_tile) : m_tile;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  if (warp < 4) {
    // Clear the accumulators: every MMA accumulates, rows without a neighbour at a step are switched off
    // through the MMA's disable-output-lane mask, so the gathered operand never holds zero rows.
#pragma unroll 1
    for (int c0 = 0; c0 < p.n_cta; c0 += 16) {
      const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
          "r"(0u)
          : "memory");
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  if (scan) {
    if (warp < mma_warp) {
#pragma unroll 1
      for (int k0 = 9 * (warp >> 2); k0 < K; k0 += 9 * groups) {     // nine loads in flight per lane
        int v[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = (k0 + i < K && my_row >= 0) ? __ldg(table(k0 + i) + my_row) : -1;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const unsigned b = __ballot_sync(0xffffffffu, v[i] >= 0);
          if (lane == 0 && b) atomicOr(&act_bits[(k0 + i) >> 5], 1u << ((k0 + i) & 31));
        }
      }
    }
    __syncthreads();
    if (warp == mma_warp) {
      int n = 0;
      for (int w = 0; w * 32 < K; ++w) {
        const uint32_t bits = act_bits[w];
        if ((bits >> lane) & 1u) act_list[n + __popc(bits & ((1u << lane) - 1u))] = (uint8_t)(w * 32 + lane);
        n += __popc(bits);
      }
      if (lane == 0) n_act_s = n;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();                       // the other CTA's barriers stand and its accumulators are clear
  tc_fence_after();
  const int n_act = scan ? n_act_s : K, n_iter = n_act * p.k_slabs;
  const uint32_t smem_base = smem_u32(smem);

  if (warp < mma_warp) {
    // ====================== producers =========================================================
    // Four lanes per row, eight rows per pass: lane l copies the 16-byte pieces l & 3 and (l & 3) + 4 of the row
    // 8 * pass + l / 4 of its warp's 32 rows, where that row has a neighbour.  Step `it` is slab it % k_slabs of the
    // it / k_slabs-th offset; of two groups each takes every other step.  A group that comes to a slot may find its
    // "empty" barrier at most one phase behind the one it waits for (the wait tells phases apart by their parity
    // only): its step before, it - 2, was let through when step it - 2 - S had been multiplied, and a phase behind
    // means step it - 2 S, which came no later as long as there are two slots.
    const int sub = lane & 3, row8 = lane >> 2, group = warp >> 2;
    const uint32_t warp_rows = smem_base + (uint32_t)quarter * 4096u + (uint32_t)row8 * 128u;   // row of the warp's first 8-row group
    const uint32_t first0 = warp_rows + (((uint32_t)sub ^ (uint32_t)row8) << 4);                // (its second piece: bit 6 the other way)
    const uint32_t full0 = smem_u32(full_bars), empty0 = smem_u32(empty_bars), masks0 = smem_u32(slot_masks + quarter);
    constexpr uint32_t mask_step = PAIR ? 32u : 16u;
    const uint32_t b_to = smem_base + (uint32_t)TC_A_BYTES, row_bytes = (uint32_t)row_words * 4u;
    const char *lane_rows = (const char *)features + sub * 16;
    const char *b_from = (const char *)packed + (size_t)nt0 * (size_t)(p.tile_n * 128);
    const bool in_rows = my_row >= 0, lead = lane == 0;
    const int32_t *my_entries = nbr + (p.rev ? (size_t)(K - 1) * n_out : 0) + max(my_row, 0);
    const int k_slabs = p.k_slabs, offset_step = p.rev ? -n_out : n_out, last = n_act - 1;
    const int a_step = GROUPS == 2 && k_slabs == 1 ? 2 : 1;           // a group's offsets
    const int whole = row_words / TC_SLAB;                            // slabs that a row fills
    // A table entry is loaded into the register it is used from, two offsets ahead (handed on from one to another it would be
    // waited for at once: with two groups 600 of a step's 1100 cycles).
    int a = a_step == 2 ? group : 0, asked = a;
    const long long entry_step = (long long)offset_step * a_step;
    const int32_t *ent = my_entries + (long long)min(a, max(last, 0)) * offset_step;
    auto next_entry = [&]() {                     // (past the last offset: that one again, not used)
      if (scan) ent = my_entries + (long long)act_list[min(asked, last)] * offset_step;
      const int v = __ldg(ent);
      asked += a_step;
      if (!scan && asked <= last) ent += entry_step;
      return v;
    };
    uint32_t slot = (uint32_t)group, par = 1u;    // (two slots at least); parity the slot's "empty" barrier has to have passed (a fresh one: has)
    bool alive = true;
    uint32_t lost = 0u;                           // rows of the warp without a neighbour
    int from[4];
    const char *at[4];
    auto turn = [&](auto piece, int kappa, int slab) {
      alive = mbar_wait_straight(empty0 + slot * 8u, par, abort_flag);
      const uint32_t full = full0 + slot * 8u, slot_off = slot * (uint32_t)stage_bytes, dst0 = first0 + slot_off, dst1 = dst0 ^ 64u;
      if (quarter == 0 && elect_one()) {          // the pre-packed filter slab of this step
        mbar_expect_tx(full, (uint32_t)b_bytes + (PAIR && rank == 0 ? 16u : 0u));   // (and the other CTA's masks)
        const char *from_slab = b_from + (size_t)(uint32_t)(kappa * k_slabs + slab) * (uint32_t)(p.n_pad * 128);
        if (PAIR) {                               // this CTA's half of every N tile
          const uint32_t half = (uint32_t)p.tile_n * 64u;
          for (int nt = 0; nt < p.nt_cta; ++nt) bulk_g2s(b_to + slot_off + (uint32_t)nt * half, from_slab + (uint32_t)(2 * nt + rank) * half, half, full);
        } else {
          bulk_g2s(b_to + slot_off, from_slab, (uint32_t)b_bytes, full);
        }
      }
      if constexpr (decltype(piece)::value >= 0) {
        copy_rows<decltype(piece)::value>(from, at, dst0, dst1);
      } else {                                    // the last slab of a row that does not fill it
        const char *base = lane_rows + slab * 128;
        const int words = row_words - slab * TC_SLAB - sub * 4;       // from this lane's first piece to the row's end
        const uint32_t bytes0 = words > 0 ? 16u : 0u, bytes1 = words > 16 ? 16u : 0u;
        const char *base0 = bytes0 ? base : (const char *)features, *base1 = bytes1 ? base + 64 : (const char *)features;
        const uint32_t stride0 = bytes0 ? row_bytes : 0u, stride1 = bytes1 ? row_bytes : 0u;
        copy_row_ends<0>(from[0], dst0, dst1, base0, stride0, bytes0, base1, stride1, bytes1);
        copy_row_ends<1024>(from[1], dst0, dst1, base0, stride0, bytes0, base1, stride1, bytes1);
        copy_row_ends<2048>(from[2], dst0, dst1, base0, stride0, bytes0, base1, stride1, bytes1);
        copy_row_ends<3072>(from[3], dst0, dst1, base0, stride0, bytes0, base1, stride1, bytes1);
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full) : "memory");
      store_and_arrive(lead, masks0 + slot * mask_step, lost, full);
      slot += GROUPS;
      if (slot >= (uint32_t)S) { slot -= (uint32_t)S; par ^= 1u; }
    };
    auto offset = [&](int &e) {                   // the group's slabs of the next of its offsets
      const int src = in_rows ? e : -1;
      lost = ~__ballot_sync(0xffffffffu, src >= 0);
#pragma unroll
      for (int i = 0; i < 4; ++i) from[i] = __shfl_sync(0xffffffffu, src, i * 8 + row8);
      e = next_entry();
      const int kappa = scan ? (int)act_list[a] : a;
#pragma unroll 1
      for (int slab = GROUPS == 1 || a_step == 2 ? 0 : (group ^ (a & k_slabs)) & 1; slab < whole; slab += 2) {
        const char *base = lane_rows + slab * 128;
#pragma unroll
        for (int i = 0; i < 4; ++i) at[i] = base + (unsigned long long)(uint32_t)from[i] * row_bytes;
        turn(std::integral_constant<int, 0>{}, kappa, slab);
        if (GROUPS == 1 && slab + 1 < whole) turn(std::integral_constant<int, 128>{}, kappa, slab + 1);
      }
      // (of two groups the one whose turn it is)
      if (whole < k_slabs && (GROUPS == 1 || a_step == 2 || ((group ^ (a & k_slabs) ^ whole) & 1) == 0)) turn(std::integral_constant<int, -1>{}, kappa, whole);
      a += a_step;
    };
    if (a < n_act) {
      int e0 = next_entry(), e1 = next_entry();
#pragma unroll 1
      while (a < n_act && alive) {
        offset(e0);
        if (a < n_act && alive) offset(e1);
      }
    }
    cp_async_wait_all();
  } else if (PAIR && rank == 1) {
    // ================================ the other CTA of a pair: tells the issuing one of its full slots =====
    const uint32_t full0 = smem_u32(full_bars);
    const uint32_t there = peer_address(full0, 0u), masks_there = peer_address(smem_u32(slot_masks), 0u) + 16u;
    uint32_t s = 0, par = 0;
    bool alive = true;
#pragma unroll 1
    for (int it = 0; it < n_iter && alive; ++it) {
      alive = mbar_wait_straight(full0 + s * 8u, par, abort_flag);
      fence_async_smem();
      const uint4 off = *(const uint4 *)(slot_masks + s * 8u);
      if (alive && elect_one()) st_async_v4(masks_there + s * 32u, off, there + s * 8u);
      if (++s == (uint32_t)S) { s = 0; par ^= 1u; }
    }
  } else {
    // ================================ MMA issuer: the whole warp, one elected lane issues ========
    // fp32 accumulator; operand formats: kind::tf32 2 = TF32; kind::f16 0 = fp16, 1 = bf16
    RowsIssuer w;
    const uint32_t fmt = F16 ? (uint32_t)p.fmt16 : 2u;
    w.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.tile_n >> 3) << 17) | ((uint32_t)((PAIR ? 2 * TC_M : TC_M) >> 4) << 24);
    w.b_bytes = (uint32_t)b_bytes;
    w.a_lo = w.a_lo0 = desc_lo(smem_base);
    w.s = w.par = 0;
    w.full0 = smem_u32(full_bars); w.empty0 = smem_u32(empty_bars);
    w.masks = slot_masks; w.d0 = tmem_base; w.abort_flag = abort_flag;
    if (PAIR) {
      if (p.nt_cta == 1) rows_issue_all<F16, 1, false, true>(w, p, n_act);
      else rows_issue_all<F16, 2, false, true>(w, p, n_act);
    } else if (p.nt_cta == 1) {
      if (scan) rows_issue_all<F16, 1, true, false>(w, p, n_act);
      else rows_issue_all<F16, 1, false, false>(w, p, n_act);
    } else {
      if (scan) rows_issue_all<F16, 2, true, false>(w, p, n_act);
      else rows_issue_all<F16, 2, false, false>(w, p, n_act);
    }
    if (elect_one()) rows_commit<PAIR>(smem_u32(&done_bar));   // arrives once everything issued above has retired
  }

  // ================================ epilogue: TMEM -> shared memory -> global ====================
  // The producer warps again: 32 rows each, with two groups every other 32 columns.
  if (warp < mma_warp) {
    const int group = warp >> 2;
    __syncwarp();
    float4 consts[2];                             // (GATED) scale, shift, gate of the channels this thread hands round
    if (GATED) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tid + 128 * i < c_out) consts[i] = gate_channel(gate, tid + 128 * i);
    }
    bool ok = __all_sync(0xffffffffu, !*abort_flag);
    if (ok && n_iter > 0) ok = mbar_wait_warp(smem_u32(&done_bar), 0u, abort_flag);
    ok = __all_sync(0xffffffffu, ok) && n_iter > 0;   // tcgen05.ld below is warp-collective
    tc_fence_after();
    const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16);
    auto load16 = [&](uint32_t *q, int c0) {
      if (ok && c0 < p.n_cta) {
        tmem_ld16(q, acc + (uint32_t)c0);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) q[i] = 0u;
      }
    };
    const int col0 = nt0 * p.tile_n;              // first output channel of this CTA
    // 32 columns of the warp's 32 rows at a time go through the warp's 4 KB of the slots (free now), so that eight
    // lanes write the 128 contiguous bytes of a row
    float *blk = (float *)(smem + (size_t)warp * 4096u);
    const int c_row = GATED ? gate.c_keep : c_out;          // channels of a stored row
    const bool vec = (c_row & 3) == 0 && ((uintptr_t)out & 15u) == 0;
    const int m = m_tile < n_rows ? (order ? __ldg(order + m_tile) : m_tile) : -1;   // this lane's row of `out`
    if (GATED) {                                  // one CTA has all channels
      float4 *chan = (float4 *)(smem + (size_t)groups * 4u * 4096u);   // [c_out]
      // act(gate g) of row r of the quarter at g * 33 + r, and a last line of ones
      const int n_gates = c_out - c_row;
      const bool whole = vec && order == nullptr && m0 + TC_M <= n_rows;
      float *gates = (float *)(chan + c_out) + quarter * 33 * (n_gates + 1);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tid + 128 * i < c_out && group == 0) chan[tid + 128 * i] = consts[i];
      for (int ch = tid + 256; ch < c_out && group == 0; ch += 128) chan[ch] = gate_channel(gate, ch);
      asm volatile("bar.sync 1, %0;" ::"r"(groups * 128) : "memory");
      if (group == 0) gates[n_gates * 33 + lane] = 1.f;
      gate_scalars(load16, gate, chan, gates, c_out, lane, (c_row & ~15) + 16 * group, 16 * groups);
      asm volatile("bar.sync 1, %0;" ::"r"(groups * 128) : "memory");
      store_gated(load16, gate, chan, gates, blk, out, c_out, m0 + quarter * 32, m, whole, vec, lane, 32 * group, 32 * groups);
    } else {
      store_plain(load16, blk, out, m, col0, p.n_cta, c_row, vec, lane, 32 * group, 32 * groups);
    }
  }
  // a wait gave up: what was issued still arrives on done_bar (committed on every path) and filter copies land
  // within microseconds; both before the accumulators and the shared memory are handed back
  if (*abort_flag) {
    if (warp == mma_warp && lane == 0 && n_iter > 0) mbar_wait_drain(smem_u32(&done_bar), 0u);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag) report_expired(status, p.alarm);
  if (PAIR) {                                     // neither leaves while the other may still signal it
    cluster_sync();
    if (warp == mma_warp) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
    cluster_sync();
  } else if (warp == mma_warp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
  }
}

template <bool F16, bool GATED, int GROUPS>
__global__ void __launch_bounds__(GROUPS * 128 + 32, GROUPS == 1 ? 4 : 2)
conv_fwd_rows_kernel(const float *__restrict__ features, int row_words, const uint4 *__restrict__ packed, int K, int c_out,
                     const int32_t *__restrict__ nbr, int n_out, float *__restrict__ out, int32_t *status, const __grid_constant__ TcParams p,
                     const int32_t *__restrict__ n_out_dev, const int32_t *__restrict__ order, const __grid_constant__ GateEpilogue gate) {
  conv_fwd_rows<F16, GATED, GROUPS, false>(features, row_words, packed, K, c_out, nbr, n_out, out, status, p, n_out_dev, order, gate);
}
template <bool F16, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(2 * 128 + 32, 2)
conv_fwd_pair_rows_kernel(const float *__restrict__ features, int row_words, const uint4 *__restrict__ packed, int K, int c_out,
                          const int32_t *__restrict__ nbr, int n_out, float *__restrict__ out, int32_t *status, const __grid_constant__ TcParams p,
                          const int32_t *__restrict__ n_out_dev, const int32_t *__restrict__ order, const __grid_constant__ GateEpilogue gate) {
  conv_fwd_rows<F16, GATED, 2, true>(features, row_words, packed, K, c_out, nbr, n_out, out, status, p, n_out_dev, order, gate);
}

static size_t tc_smem_bytes(const TcParams &p) {
  return (size_t)p.stages * p.sps * (TC_A_BYTES + (p.pair ? p.b_bytes / 2 : p.b_bytes)) + 1024 /*alignment slack*/ + TC_CTRL_BYTES;
}

// 16-bit operands: filters [K, c_in, c_out] fp32 -> [K][k_slabs][n_pad rows][64 fp16 or bf16], same
// swizzle (a 16-byte chunk holds 8 input channels).
template <bool BF16>
__global__ void pack_filters_16_kernel(const float *__restrict__ filters, int K, int c_in, int c_out, TcParams p,
                                        uint4 *__restrict__ packed) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)K * p.k_slabs * p.n_pad * 8;
  if (t >= total) return;
  int chunk = (int)(t & 7);
  long long r = t >> 3;
  int n = (int)(r % p.n_pad);
  r /= p.n_pad;
  int slab = (int)(r % p.k_slabs);
  int kappa = (int)(r / p.k_slabs);
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float f[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int ci = slab * 64 + chunk * 8 + q * 2 + h;
      f[h] = (ci < c_in && n < c_out) ? filters[((size_t)kappa * c_in + ci) * c_out + n] : 0.f;
    }
    v[q] = BF16 ? pack_bf16x2(f[0], f[1]) : pack_f16x2(f[0], f[1]);
  }
  size_t block = ((size_t)kappa * p.k_slabs + slab) * (size_t)(p.n_pad * 8);
  size_t off = (size_t)(n >> 3) * 64 + (size_t)(n & 7) * 8 + (size_t)(chunk ^ (n & 7));
  packed[block + off] = make_uint4(v[0], v[1], v[2], v[3]);
}

// The plan of a launch over n_out rows: few row tiles spread the N tiles over CTAs too, and no more CTAs are put on an SM than
// the launch has for it, so that they share its memory for deeper rings (256 tiles of 64 -> 76 bf16 channels, two on an SM instead of
// four: 20.2 -> 15.7 us).  Row tiles that fit the SMs by themselves but not with their N tiles
// spread stay whole: a few SMs with two CTAs would make all wait for rings of half the depth (79 row tiles
// of 256 -> 304 bf16 channels: 62 us spread).  Rows of one slab take four CTAs on an SM where the launch has three: their rings turn
// over quickly, and a fourth place takes the tiles of a row order that are left (45 k rows, 3 and 4 CTAs: 16 -> 22 in order 32.2 and 30.8 us,
// 32 -> 38 in order 32.3 and 30.9, 8 -> 22 21.1 and 19.4, 20 -> 38 28.2 and 28.5; of three slabs, 76 -> 64 in order, 39.1 and 44.7).
// Pairs: from 128 columns a CTA and four slabs an offset on, up to two tiles an SM.  There the filter slab, which every
// tile brings in whole, is most of what a step moves (TF32 128 -> 152, 238 tiles: 59.1 -> 52.3 us; 256 -> 304 bf16, 125 tiles: 54.4 -> 52.6).  The second CTA's
// news reaches the issuing one some 300 cycles late, so short loops lose (256 tiles of 128 -> 152 bf16: 30.8 -> 31.9), rings of two slots
// more so (64 -> 76, 1.1 M rows: 690 -> 770), and with many tiles on an SM another one fills the time (637 tiles of 128 -> 152 bf16: 63 -> 65).
// Of eight TF32 and four 16-bit widths at 19 sizes one lost, where its second wave begins a few tiles earlier than single CTAs' (187 tiles of
// 256 -> 304: 163 -> 174; 174 tiles 160 -> 151, 200 tiles 176 and 176).
static bool rows_params(int words, int c_out, int n_out, TcParams &p, int opk = 1, bool pairs = false) {
  const int grid = n_out > 0 ? ceil_div(n_out, TC_M) : 1, sms = sm_count();
  auto plan = [&](bool pair) {
    const int ctas = ceil_div(grid, sms);
    if (!tc_params(words, c_out, p, false, ctas == 3 && words <= TC_SLAB ? 4 : ctas, opk, pair)) return false;
    if (p.n_tiles == 1 || grid >= 2 * sms || (grid <= sms && grid * p.n_tiles > sms)) return true;
    return tc_params(words, c_out, p, true, ceil_div(grid * p.n_tiles, sms), opk, pair);
  };
  if (!plan(false)) return false;
  if (pairs && grid > 1 && grid <= 2 * sms && p.n_cta >= 128 && p.k_slabs >= 4) return plan(true);
  return true;
}

// Producer groups.  Three or four CTAs on an SM have producers enough between them, and a second group in each would leave
// its threads 56 registers, which costs more instructions than it brings; one or two CTAs need both (64 -> 76
// channels, four CTAs: 95 us with two groups, 88 with one; 128 -> 152 bf16 channels, two CTAs: 77 and 83).
static int rows_groups(const TcParams &p) { return p.ctas > 2 && !p.pair ? 1 : 2; }     // (pairs have two CTAs on an SM at most)

using RowsKernel = void (*)(const float *, int, const uint4 *, int, int, const int32_t *, int, float *, int32_t *, TcParams, const int32_t *,
                            const int32_t *, GateEpilogue);
template <bool F16>
static RowsKernel rows_kernel(const TcParams &p, bool gated) {
  if (p.pair) return gated ? conv_fwd_pair_rows_kernel<F16, true> : conv_fwd_pair_rows_kernel<F16, false>;
  if (rows_groups(p) == 1) return gated ? conv_fwd_rows_kernel<F16, true, 1> : conv_fwd_rows_kernel<F16, false, 1>;
  return gated ? conv_fwd_rows_kernel<F16, true, 2> : conv_fwd_rows_kernel<F16, false, 2>;
}
static int rows_threads(const TcParams &p) { return rows_groups(p) * 128 + 32; }

// What the gated epilogue needs: 4 KB per producer warp, the channel constants and the gates of 128 rows, in the
// operand slots that are free by then.
static bool gate_fits(const TcParams &p, int c_out, int c_keep) {
  const size_t warps = (size_t)rows_groups(p) * 4;
  return p.nt_cta == p.n_tiles &&
         warps * 4096 + (size_t)c_out * 16 + (size_t)4 * 33 * 4 * (c_out - c_keep + 1) <= (size_t)p.stages * (TC_A_BYTES + (p.pair ? p.b_bytes / 2 : p.b_bytes));
}

bool conv_gate_covered(int c_in, int c_out, int c_keep, int precision, int n_out) {
  if (c_in < 1 || c_keep < 1 || c_keep > c_out) return false;
  const bool tf32 = precision == SSC_PREC_TF32;
  if (!tf32 && precision != SSC_PREC_F16 && precision != SSC_PREC_BF16) return false;
  if (tf32 && tf32_offsets_per_row(c_in) > 1) return false;
  TcParams p;
  return rows_params(tf32 ? c_in : f16_row_words(c_in), c_out, n_out, p) && gate_fits(p, c_out, c_keep);
}

int conv_fwd_16(const float *features, int n_in, int c_in, bool bf16, const void *packed, int K, int c_out,
                const int32_t *nbr, int n_out, float *out, int32_t *status, void *scratch, size_t scratch_bytes,
                const int32_t *n_out_dev, const int32_t *order, bool prestaged, int table_form, const GateEpilogue &gate, cudaStream_t st) {
  if (K > 256) return fail(SSC_ERR_INVALID, "conv_fwd(16-bit): kernel volume %d > 256", K);
  const int words = f16_row_words(c_in);
  if (scratch == nullptr || scratch_bytes + 16 < conv_f16_scratch_bytes(n_in, c_in) || ((uintptr_t)scratch & 15u) != 0)
    return fail(SSC_ERR_INVALID, "conv_fwd(16-bit): needs the staging buffer of ssc_conv_scratch_bytes (16-byte aligned)");
  int grid = ceil_div(n_out, TC_M);
  TcParams p;
  const bool gated = gate.gate_of_channel != nullptr;
  bool planned = rows_params(words, c_out, n_out, p, 1, order == nullptr);
  if (planned && gated && p.pair && !gate_fits(p, c_out, gate.c_keep)) planned = rows_params(words, c_out, n_out, p);
  if (!planned) return fail(SSC_ERR_INVALID, "conv_fwd(16-bit): c_out %d / kernel volume %d not supported", c_out, K);
  p.fmt16 = bf16 ? 1 : 0;
  p.nbr_by_pos = ((table_form & SSC_CONV_TABLE_IN_ORDER) && order) ? 1 : 0;
  p.rev = (table_form & SSC_CONV_TABLE_REVERSED) ? 1 : 0;
  p.alarm = alarm_word();
  if (!prestaged) {
    int rc = stage_features_16(features, n_in, c_in, bf16, scratch, st);
    if (rc != SSC_OK) return rc;
  }
  const size_t smem = tc_smem_bytes(p);
  if (gated && !gate_fits(p, c_out, gate.c_keep)) return fail(SSC_ERR_INVALID, "conv_fwd(16-bit): the gated epilogue does not cover %d -> %d channels", c_out, gate.c_keep);
  const RowsKernel kernel = rows_kernel<true>(p, gated);
  cudaError_t e = allow_smem((const void *)kernel, smem);
  if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd(16-bit): smem attribute: %s", cudaGetErrorString(e));
  const dim3 grid2(p.pair ? (grid + 1) & ~1 : grid, p.n_tiles / p.nt_cta);
  e = launch_ready(kernel, grid2, dim3(rows_threads(p)), smem, st, (const float *)scratch, words, (const uint4 *)packed, K, c_out, nbr, n_out, out, status, p, n_out_dev, order, gate);
  note_launches(1);
  SSC_CHECK_LAUNCH("conv_fwd_16");
  return SSC_OK;
}

int conv_fwd_tf32(const float *features, int n_in, int c_in, const void *packed, int K, int c_out,
                  const int32_t *nbr, int n_out, float *out, int32_t *status, void *scratch, size_t scratch_bytes,
                  const int32_t *n_out_dev, const int32_t *order, bool prestaged, int table_form, const GateEpilogue &gate, cudaStream_t st) {
  TcParams p;
  if (K > 256) return fail(SSC_ERR_INVALID, "conv_fwd(tf32): kernel volume %d > 256", K);
  int grid = ceil_div(n_out, TC_M);
  const int opk = tf32_offsets_per_row(c_in);
  const bool gated = gate.gate_of_channel != nullptr;
  // (a pair runs on staged rows only, and those come with a scratch buffer)
  const bool fits = scratch != nullptr && scratch_bytes + 16 >= conv_tf32_scratch_bytes(n_in, c_in) && ((uintptr_t)scratch & 15u) == 0;
  bool planned = rows_params(c_in, c_out, n_out, p, opk, order == nullptr && fits && opk == 1);
  if (planned && gated && p.pair && !gate_fits(p, c_out, gate.c_keep)) planned = rows_params(c_in, c_out, n_out, p, opk);
  if (!planned) return fail(SSC_ERR_INVALID, "conv_fwd(tf32): c_out %d / kernel volume %d not supported", c_out, K);
  p.nbr_by_pos = ((table_form & SSC_CONV_TABLE_IN_ORDER) && order) ? 1 : 0;
  p.rev = (table_form & SSC_CONV_TABLE_REVERSED) ? 1 : 0;
  p.alarm = alarm_word();
  size_t smem = tc_smem_bytes(p);
  // With a staging buffer the feature rows are rounded to TF32 once, up front, instead of after
  // every gather (a row is gathered about K/2 times).
  const int c_pad = (c_in + 3) & ~3;  // row stride of the staged image (zero-padded channels)
  if (prestaged && !fits) return fail(SSC_ERR_INVALID, "conv_fwd(tf32): SSC_CONV_PRESTAGED without the staged image in scratch");
  // layers with few input channels have their filters packed for several offsets per operand row,
  // which the kernel can only feed from the staged (padded) rows
  if (opk > 1 && !fits) return fail(SSC_ERR_SCRATCH, "conv_fwd(tf32): a layer with %d input channels needs the staging buffer (ssc_conv_scratch_bytes)", c_in);
  // whoever brings a staging buffer gets the kernel that runs on staged rows: also a layer of a few tiles, whose
  // CTAs are alone on their SMs (512 rows of 120 -> 240 channels: 104 us unstaged)
  const bool staged = fits;
  if (staged && !prestaged) {
    int rc = stage_features(features, n_in, c_in, scratch, st);
    if (rc != SSC_OK) return rc;
  }
  const dim3 grid2(p.pair ? (grid + 1) & ~1 : grid, p.n_tiles / p.nt_cta);
  const bool rows = staged && opk == 1;
  if (gated && !(rows && gate_fits(p, c_out, gate.c_keep)))
    return fail(SSC_ERR_INVALID, "conv_fwd(tf32): the gated epilogue does not cover %d -> %d channels without a staging buffer", c_out, gate.c_keep);
  if (rows) {
    const RowsKernel kernel = rows_kernel<false>(p, gated);
    cudaError_t e = allow_smem((const void *)kernel, smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd(tf32): smem attribute: %s", cudaGetErrorString(e));
    e = launch_ready(kernel, grid2, dim3(rows_threads(p)), smem, st, (const float *)scratch, c_pad, (const uint4 *)packed, K, c_out, nbr, n_out, out, status, p, n_out_dev, order, gate);
  } else {
    auto kernel = opk > 1 ? conv_fwd_tf32_kernel<true> : conv_fwd_tf32_kernel<false>;
    cudaError_t e = allow_smem((const void *)kernel, smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "conv_fwd(tf32): smem attribute: %s", cudaGetErrorString(e));
    launch_ready(kernel, grid2, dim3(p.threads), smem, st, staged ? (const float *)scratch : features, staged ? c_pad : c_in, (const uint4 *)packed, K, c_out, nbr, n_out, out, status, p, n_out_dev, order);
  }
  note_launches(1);
  SSC_CHECK_LAUNCH("conv_fwd_tf32");
  return SSC_OK;
}

}  // namespace ssc

using namespace ssc;

static bool is16(int precision) { return precision == SSC_PREC_F16 || precision == SSC_PREC_BF16; }

extern "C" size_t ssc_conv_packed_bytes(int K, int c_in, int c_out, int precision) {
  if ((precision != SSC_PREC_TF32 && !is16(precision)) || K < 1 || c_in < 1 || c_out < 1) return 0;
  TcParams p;
  if (!tc_params(is16(precision) ? f16_row_words(c_in) : c_in, c_out, p)) return 0;
  if (!is16(precision) && tf32_offsets_per_row(c_in) > 1)
    return (size_t)ceil_div(K, tf32_offsets_per_row(c_in)) * p.n_pad * 128;
  return (size_t)K * p.k_slabs * p.n_pad * 128;
}

extern "C" int ssc_conv_pack_filters(const float *filters, int K, int c_in, int c_out, int precision, void *packed,
                                     void *stream) {
  SSC_REQUIRE(precision == SSC_PREC_TF32 || is16(precision), "conv_pack_filters: only SSC_PREC_TF32, SSC_PREC_F16 and SSC_PREC_BF16 have a packed form");
  SSC_REQUIRE(filters && packed && K >= 1 && c_in >= 1 && c_out >= 1, "conv_pack_filters: bad arguments");
  TcParams p;
  SSC_REQUIRE(tc_params(is16(precision) ? f16_row_words(c_in) : c_in, c_out, p), "conv_pack_filters: c_out %d not supported (max 512)", c_out);
  if (precision == SSC_PREC_TF32 && tf32_offsets_per_row(c_in) > 1) {
    const int opk = tf32_offsets_per_row(c_in), n_groups = ceil_div(K, opk);
    const long long total_g = (long long)n_groups * p.n_pad * 8;
    { launch_ready(pack_filters_tf32_grouped_kernel, dim3(ceil_div(total_g, 256)), dim3(256), 0, as_stream(stream), filters, K, c_in, c_out, (c_in + 3) & ~3, opk,
                                                                                         n_groups, p.n_pad, (uint4 *)packed); note_launches(1); }
    SSC_CHECK_LAUNCH("pack_filters");
    return SSC_OK;
  }
  long long total = (long long)K * p.k_slabs * p.n_pad * 8;
  const int blocks = ceil_div(total, 256);
  if (precision == SSC_PREC_F16) { launch_ready(pack_filters_16_kernel<false>, dim3(blocks), dim3(256), 0, as_stream(stream), filters, K, c_in, c_out, p, (uint4 *)packed); note_launches(1); }
  else if (precision == SSC_PREC_BF16) { launch_ready(pack_filters_16_kernel<true>, dim3(blocks), dim3(256), 0, as_stream(stream), filters, K, c_in, c_out, p, (uint4 *)packed); note_launches(1); }
  else { launch_ready(pack_filters_tf32_kernel, dim3(blocks), dim3(256), 0, as_stream(stream), filters, K, c_in, c_out, p, (uint4 *)packed); note_launches(1); }
  SSC_CHECK_LAUNCH("pack_filters");
  return SSC_OK;
}
