// Declarations shared by the convolution sources (ssc_conv*.cu, ssc_wgrad_tc.cu).
#pragma once
#include "ssc_common.cuh"

namespace ssc {

// staged operand images (ssc_conv_stage.cu)
size_t conv_tf32_scratch_bytes(int n_in, int c_in);
size_t conv_f16_scratch_bytes(int n_in, int c_in);
int stage_features(const float *features, int n_in, int c_in, void *staged, cudaStream_t st);
int stage_features_16(const float *features, int n_in, int c_in, bool bf16, void *staged, cudaStream_t st);

// Width of a 16-bit (fp16 / bf16) operand row in 4-byte units; rows are padded to 16 bytes.  The
// kernels gather such a row like an fp32 image of that many channels.
inline int f16_row_words(int c_in) { return ((c_in + 7) & ~7) / 2; }

// TF32 layers with few input channels: kernel offsets that share one 128-byte operand row (rows of
// the staged image are c_pad = 4, 8 or 16 floats): 8, 4, 2; else 1.  Decides the packed filter layout.
inline int tf32_offsets_per_row(int c_in) {
  const int c_pad = (c_in + 3) & ~3;
  return (c_pad == 4 || c_pad == 8 || c_pad == 16) ? 32 / c_pad : 1;
}

// geometry of the packed filter image [K][k_slabs][n_pad][128 bytes] (ssc_conv_tc.cu)
bool tc_operand_layout(int c_in_words, int c_out, int *k_slabs, int *n_pad, int *tile_n, int *n_tiles);

// A per-channel affine map (an eval-mode batch norm folded up; scale NULL: none) and the gated activation, applied to
// the rows of a convolution before they are stored: channels [0, c_keep) are kept, the rest are the gate
// scalars (ssc_bn_gate_fwd with c_gate_base = c_keep and no biases).
struct GateEpilogue {
  const float *scale, *shift;
  const int32_t *gate_of_channel;   // NULL: the convolution's own rows are stored
  int c_keep, scalar_act, gate_act;
  int out16;                        // 0: fp32 rows, 1: fp16, 2: bf16
};
bool conv_gate_covered(int c_in, int c_out, int c_keep, int precision, int n_out);

// output-stationary tensor-core kernels (ssc_conv_tc.cu); table_form: SSC_CONV_TABLE_IN_ORDER | SSC_CONV_TABLE_REVERSED
int conv_fwd_tf32(const float *features, int n_in, int c_in, const void *packed, int K, int c_out,
                  const int32_t *nbr, int n_out, float *out, int32_t *status, void *scratch, size_t scratch_bytes,
                  const int32_t *n_out_dev, const int32_t *order, bool prestaged, int table_form, const GateEpilogue &gate, cudaStream_t st);
int conv_fwd_16(const float *features, int n_in, int c_in, bool bf16, const void *packed, int K, int c_out,
                const int32_t *nbr, int n_out, float *out, int32_t *status, void *scratch, size_t scratch_bytes,
                const int32_t *n_out_dev, const int32_t *order, bool prestaged, int table_form, const GateEpilogue &gate, cudaStream_t st);

// compacted per-offset pair lists of a neighbour table (ssc_wgrad_tc.cu): the lists of the kernel
// offsets follow one another in pair_out / pair_in (ascending output row inside an offset),
// starts[kappa] .. starts[kappa + 1] is the range of offset kappa, starts[K] the number of pairs.
struct PairLists {
  int32_t *pair_out;
  int32_t *pair_in;
  int32_t *starts;   // [K + 1]
};
size_t pair_lists_bytes(int K, int n_out);
int pair_lists_build(const int32_t *nbr, int K, int n_out, void *lists, PairLists *out, cudaStream_t st);
PairLists pair_lists_view(void *lists, int K, int n_out);

// filter gradient over pair lists (ssc_wgrad_tc.cu): bytes of its partial tiles, 0 where the shape is not covered
size_t conv_wgrad_lists_partial_bytes(int K, int c_in, int c_out, int n_out, bool tf32);
int conv_wgrad_lists(const float *features, int c_in, const float *out_grad, int c_out, const PairLists &pl, int K, int n_out,
                     bool tf32, int staged, float *partial, float *d_filters, int32_t *status, cudaStream_t st);

}  // namespace ssc
