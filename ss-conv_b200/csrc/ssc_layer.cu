// A layer that runs ahead of its output count, in one call: what bounds a small layer is the host that queues its
// kernels, so the rulebook and the kernel on it are queued here without going back to the caller in between,
// and all intermediates share one workspace.
#include "ssc_conv_internal.cuh"

namespace ssc {

struct LayerSpace {
  size_t table, staged, rows, total;   // byte offsets behind the rulebook's scratch
  size_t rulebook_bytes;
};

static bool gate_fused(const ssc_layer &a) {
  return a.op == 0 && a.gate_of_channel != nullptr && a.precision != SSC_PREC_FP32 &&
         conv_gate_covered(a.c_in, a.c_out, a.c_keep, a.precision, a.n_out);
}

static LayerSpace layer_space(const ssc_layer &a) {
  LayerSpace s;
  const int K = a.ksize[0] * a.ksize[1] * a.ksize[2];
  s.rulebook_bytes = ssc_rulebook_scratch_bytes(a.n_in, a.batch, a.in_shape, a.out_shape, K);
  size_t off = align_up(s.rulebook_bytes, 256);
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += align_up(bytes, 256);
    return at;
  };
  s.table = take((size_t)K * a.n_out * sizeof(int32_t));
  s.staged = take(a.op == 0 && a.stored == 0 ? ssc_conv_scratch_bytes(a.n_in, a.c_in, a.c_out, a.precision) : 0);
  s.rows = take(a.op == 0 && a.gate_of_channel != nullptr && !gate_fused(a) ? (size_t)a.n_out * a.c_out * sizeof(float) : 0);
  s.total = off;
  return s;
}

}  // namespace ssc

using namespace ssc;

extern "C" size_t ssc_layer_struct_bytes(void) { return sizeof(ssc_layer); }

extern "C" size_t ssc_layer_ahead_bytes(const ssc_layer *layer) { return layer ? layer_space(*layer).total : 0; }

extern "C" int ssc_layer_ahead(const ssc_layer *layer) {
  SSC_REQUIRE(layer, "layer_ahead: null pointer");
  const ssc_layer &a = *layer;
  SSC_REQUIRE(a.op >= 0 && a.op <= 2 && a.n_in > 0 && a.n_out > 0 && a.c_in > 0 && a.n_out_dev && a.features && a.out && a.workspace, "layer_ahead: bad arguments");
  SSC_REQUIRE(a.stored == 0 || a.op != 0 || a.precision == a.stored, "layer_ahead: rows stored at precision %d cannot be convolved at %d", a.stored, a.precision);
  const LayerSpace s = layer_space(a);
  if (a.workspace_bytes < s.total) return fail(SSC_ERR_SCRATCH, "layer_ahead: workspace %zu < %zu bytes", a.workspace_bytes, s.total);
  char *ws = (char *)a.workspace;
  int32_t *nbr = (int32_t *)(ws + s.table);
  const int K = a.ksize[0] * a.ksize[1] * a.ksize[2];
  int rc = ssc_rulebook_conv_ahead(a.indices, a.n_in, a.batch, a.in_shape, a.out_shape, a.ksize, a.stride, a.padding, a.dilation, a.transpose,
                                   a.n_out, a.out_indices, nbr, a.n_out_dev, a.status, ws, s.rulebook_bytes, a.n_in_dev, a.place, a.stream);
  if (rc != SSC_OK) return rc;
  if (a.op != 0) {
    if (a.stored != 0) return ssc_pool_fwd16(a.features, a.stored, a.op == 2, a.c_in, nbr, K, a.n_out, nullptr, (float *)a.out, a.n_out_dev, a.stream);
    return a.op == 1 ? ssc_maxpool_fwd((const float *)a.features, a.c_in, nbr, K, a.n_out, (float *)a.out, a.n_out_dev, a.stream)
                     : ssc_avgpool_fwd((const float *)a.features, a.c_in, nbr, K, a.n_out, nullptr, (float *)a.out, a.n_out_dev, a.stream);
  }
  // rows stored in 16 bits are their own staged image
  const float *rows = a.stored ? nullptr : (const float *)a.features;
  void *image = a.stored ? (void *)a.features : (void *)(ws + s.staged);
  const size_t image_bytes = a.stored ? (size_t)a.n_in * a.c_in * 2 : s.rows - s.staged;
  const int precision = a.precision | (a.stored ? SSC_CONV_PRESTAGED : 0);
  if (gate_fused(a))
    return ssc_conv_fwd_gated(rows, a.n_in, a.c_in, a.filters, K, a.c_out, nbr, a.n_out, precision, a.scale, a.shift, a.gate_of_channel,
                              a.c_keep, a.scalar_act, a.gate_act, a.out_precision, a.out, a.status, image, image_bytes, a.n_out_dev, nullptr, a.stream);
  float *conv = a.gate_of_channel ? (float *)(ws + s.rows) : (float *)a.out;
  rc = ssc_conv_fwd(rows, a.n_in, a.c_in, a.filters, K, a.c_out, nbr, a.n_out, precision, conv, a.status,
                    a.precision == SSC_PREC_FP32 ? nullptr : image, a.precision == SSC_PREC_FP32 ? 0 : image_bytes, a.n_out_dev, a.stream);
  if (rc != SSC_OK || a.gate_of_channel == nullptr) return rc;
  if (a.out_precision != SSC_PREC_FP32)
    return ssc_bn_gate_fwd16(conv, a.n_out, a.c_out, a.scale, a.shift, a.gate_of_channel, a.c_keep, a.c_keep, a.scalar_act, a.gate_act,
                             nullptr, nullptr, a.out_precision, a.out, a.stream);
  return ssc_bn_gate_fwd(conv, a.n_out, a.c_out, a.scale, a.shift, a.gate_of_channel, a.c_keep, a.c_keep, a.scalar_act, a.gate_act,
                         nullptr, nullptr, (float *)a.out, a.stream);
}
