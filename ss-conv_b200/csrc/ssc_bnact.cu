// Irrep-wise BatchNorm (eval: folded per-channel affine; train: statistics) and the gated
// activation, as single elementwise passes.  HBM-bound.
#include "ssc_act.cuh"
#include "ssc_common.cuh"
#include "ssc_tc_ptx.cuh"

namespace ssc {

__global__ void bn_fold_kernel(const float *running_mean, const float *running_var, const float *weight,
                               const float *bias, const int32_t *field_of_channel, const int32_t *scalar_of_channel,
                               int c, float eps, float *scale, float *shift) {
  after_previous();
  int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= c) return;
  int f = field_of_channel[ch], s = scalar_of_channel[ch];
  float sc = 1.0f / sqrtf(running_var[f] + eps);
  if (weight) sc *= weight[f];
  float sh = 0.f;
  if (s >= 0) {
    sh = -running_mean[s] * sc;
    if (bias) sh += bias[s];
  }
  scale[ch] = sc;
  shift[ch] = sh;
}

// One thread per output element (any channel counts / alignment).
__global__ void bn_gate_kernel(const float *__restrict__ x, long long total, int c_in_total,
                               const float *__restrict__ scale, const float *__restrict__ shift,
                               const int32_t *__restrict__ gate_of_channel, int c_out, int c_gate_base,
                               int scalar_act, int gate_act, const float *__restrict__ scalar_bias,
                               const float *__restrict__ gate_bias, float *__restrict__ out) {
  after_previous();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  long long row = t / c_out;
  int ch = (int)(t - row * c_out);
  const float *xr = x + row * c_in_total;
  float v = xr[ch];
  if (scale) v = fmaf(v, scale[ch], shift[ch]);
  if (gate_of_channel) {
    int g = gate_of_channel[ch];
    if (g == -1) {
      if (scalar_bias) v += scalar_bias[ch];
      v = apply_act(v, scalar_act);
    } else if (g >= 0) {
      float gv = xr[c_gate_base + g];
      if (scale) gv = fmaf(gv, scale[c_gate_base + g], shift[c_gate_base + g]);
      if (gate_bias) gv += gate_bias[g];
      v *= apply_act(gv, gate_act);
    }
  }
  out[t] = v;
}

// Four consecutive output channels per thread (16-byte loads and stores, 32-bit index arithmetic):
// channel counts that are multiples of four, 16-byte aligned rows.  Same arithmetic per element
// as the scalar kernel.  groups = c_out / 4; total = rows * groups < 2^31.
__global__ void __launch_bounds__(256)
bn_gate_vec4_kernel(const float *__restrict__ x, uint32_t total, uint32_t groups, int c_in_total,
                    const float *__restrict__ scale, const float *__restrict__ shift,
                    const int32_t *__restrict__ gate_of_channel, int c_gate_base, int scalar_act, int gate_act,
                    const float *__restrict__ scalar_bias, const float *__restrict__ gate_bias, float *__restrict__ out) {
  after_previous();
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const uint32_t row = t / groups, g4 = t - row * groups;
  const int ch0 = (int)g4 * 4;
  const float *xr = x + (size_t)row * c_in_total;
  const float4 xv = __ldg((const float4 *)(xr + ch0));
  float v[4] = {xv.x, xv.y, xv.z, xv.w};
  if (scale) {
    const float4 sc = __ldg((const float4 *)(scale + ch0)), sh = __ldg((const float4 *)(shift + ch0));
    v[0] = fmaf(v[0], sc.x, sh.x);
    v[1] = fmaf(v[1], sc.y, sh.y);
    v[2] = fmaf(v[2], sc.z, sh.z);
    v[3] = fmaf(v[3], sc.w, sh.w);
  }
  if (gate_of_channel) {
    const int4 gi = __ldg((const int4 *)(gate_of_channel + ch0));
    const int g[4] = {gi.x, gi.y, gi.z, gi.w};
    int last_g = -2;
    float last_a = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (g[q] == -1) {
        if (scalar_bias) v[q] += scalar_bias[ch0 + q];
        v[q] = apply_act(v[q], scalar_act);
      } else if (g[q] >= 0) {
        if (g[q] != last_g) {   // the channels of a field share their gate
          float gv = __ldg(xr + c_gate_base + g[q]);
          if (scale) gv = fmaf(gv, scale[c_gate_base + g[q]], shift[c_gate_base + g[q]]);
          if (gate_bias) gv += gate_bias[g[q]];
          last_a = apply_act(gv, gate_act);
          last_g = g[q];
        }
        v[q] *= last_a;
      }
    }
  }
  *(float4 *)(out + (size_t)t * 4) = make_float4(v[0], v[1], v[2], v[3]);
}

// The same with a 16-bit result (OUT = 1 fp16, 2 bf16): the features leave the layer in the operand
// precision of the next convolution, which then gathers them as they are (no staging pass).
// Four consecutive output channels per thread:
// channel counts that are multiples of four, 16-byte aligned rows.  Same arithmetic per element
// as the scalar kernel.  groups = c_out / 4; total = rows * groups < 2^31.
template <int OUT>
__global__ void __launch_bounds__(256)
bn_gate_vec4_out16_kernel(const float *__restrict__ x, uint32_t total, uint32_t groups, int c_in_total,
                    const float *__restrict__ scale, const float *__restrict__ shift,
                    const int32_t *__restrict__ gate_of_channel, int c_gate_base, int scalar_act, int gate_act,
                    const float *__restrict__ scalar_bias, const float *__restrict__ gate_bias, uint2 *__restrict__ out) {
  after_previous();
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const uint32_t row = t / groups, g4 = t - row * groups;
  const int ch0 = (int)g4 * 4;
  const float *xr = x + (size_t)row * c_in_total;
  const float4 xv = __ldg((const float4 *)(xr + ch0));
  float v[4] = {xv.x, xv.y, xv.z, xv.w};
  if (scale) {
    const float4 sc = __ldg((const float4 *)(scale + ch0)), sh = __ldg((const float4 *)(shift + ch0));
    v[0] = fmaf(v[0], sc.x, sh.x);
    v[1] = fmaf(v[1], sc.y, sh.y);
    v[2] = fmaf(v[2], sc.z, sh.z);
    v[3] = fmaf(v[3], sc.w, sh.w);
  }
  if (gate_of_channel) {
    const int4 gi = __ldg((const int4 *)(gate_of_channel + ch0));
    const int g[4] = {gi.x, gi.y, gi.z, gi.w};
    int last_g = -2;
    float last_a = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (g[q] == -1) {
        if (scalar_bias) v[q] += scalar_bias[ch0 + q];
        v[q] = apply_act(v[q], scalar_act);
      } else if (g[q] >= 0) {
        if (g[q] != last_g) {   // the channels of a field share their gate
          float gv = __ldg(xr + c_gate_base + g[q]);
          if (scale) gv = fmaf(gv, scale[c_gate_base + g[q]], shift[c_gate_base + g[q]]);
          if (gate_bias) gv += gate_bias[g[q]];
          last_a = apply_act(gv, gate_act);
          last_g = g[q];
        }
        v[q] *= last_a;
      }
    }
  }
  out[t] = OUT == 2 ? make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]))
                    : make_uint2(pack_f16x2(v[0], v[1]), pack_f16x2(v[2], v[3]));
}

// The gated pass with every gate evaluated ONCE per row: a block owns R = 256 / groups whole rows,
// first fills gate_s[r][g] = act(BN(x[row, c_gate_base + g]) + bias) for its rows (one value per
// thread), then every thread finishes four consecutive channels of one row and takes its gates
// from shared memory.  The per-element arithmetic is that of the kernels above (same bits); what
// changes is the instruction count: a thread of the kernels above evaluates up to four
// sigmoids (expf + IEEE division each, every path taken by some lane of the warp), which made
// the pass instruction-bound at half the memory rate.  OUT = 0 fp32, 1 fp16, 2 bf16 result.
template <int OUT, int VEC>
__global__ void __launch_bounds__(256)
bn_gate_rows_kernel(const float *__restrict__ x, uint32_t n_rows, uint32_t groups, int c_in_total,
                    const float *__restrict__ scale, const float *__restrict__ shift,
                    const int32_t *__restrict__ gate_of_channel, int c_gate_base, int n_gates, int scalar_act,
                    int gate_act, const float *__restrict__ scalar_bias, const float *__restrict__ gate_bias,
                    void *__restrict__ out) {
  after_previous();
  extern __shared__ float gate_s[];                    // [R][n_gates]
  // block = (groups, R): threadIdx.x is the group of VEC channels, threadIdx.y the row of the block
  // (no integer division anywhere in the kernel).  VEC = 4 / 2 / 1 for channel counts that are
  // multiples of four / even / odd (rows 16- / 8- / 4-byte aligned).
  const uint32_t R = blockDim.y, r = threadIdx.y, gq = threadIdx.x, row = blockIdx.x * R + r;
  const bool active = row < n_rows;
  const int ch0 = (int)gq * VEC;
  // this thread's channels: the load goes out before the gate phase, so that both phases'
  // memory latencies overlap
  float v[VEC];
#pragma unroll
  for (int q = 0; q < VEC; ++q) v[q] = 0.f;
  if (active) {
    const float *xp = x + (size_t)row * c_in_total + ch0;
    if (VEC == 4) {
      const float4 t = __ldg((const float4 *)xp);
      v[0] = t.x; v[1 % VEC] = t.y; v[2 % VEC] = t.z; v[3 % VEC] = t.w;
    } else if (VEC == 2) {
      const float2 t = __ldg((const float2 *)xp);
      v[0] = t.x; v[1 % VEC] = t.y;
    } else {
      v[0] = __ldg(xp);
    }
    float *my_gates_w = gate_s + r * (uint32_t)n_gates;
    for (uint32_t g = gq; g < (uint32_t)n_gates; g += groups) {
      float gv = __ldg(x + (size_t)row * c_in_total + c_gate_base + g);
      if (scale) gv = fmaf(gv, scale[c_gate_base + g], shift[c_gate_base + g]);
      if (gate_bias) gv += gate_bias[g];
      my_gates_w[g] = apply_act(gv, gate_act);
    }
  }
  __syncthreads();
  if (!active) return;
  const float *my_gates = gate_s + r * (uint32_t)n_gates;
  float sc[VEC], sh[VEC];
  int gi[VEC];
  if (VEC == 4) {   // 16-byte aligned tables (checked by the caller)
    const int4 t = __ldg((const int4 *)(gate_of_channel + ch0));
    gi[0] = t.x; gi[1 % VEC] = t.y; gi[2 % VEC] = t.z; gi[3 % VEC] = t.w;
    if (scale) {
      const float4 a = __ldg((const float4 *)(scale + ch0)), b = __ldg((const float4 *)(shift + ch0));
      sc[0] = a.x; sc[1 % VEC] = a.y; sc[2 % VEC] = a.z; sc[3 % VEC] = a.w;
      sh[0] = b.x; sh[1 % VEC] = b.y; sh[2 % VEC] = b.z; sh[3 % VEC] = b.w;
    }
  } else {
#pragma unroll
    for (int q = 0; q < VEC; ++q) {
      gi[q] = __ldg(gate_of_channel + ch0 + q);
      if (scale) { sc[q] = __ldg(scale + ch0 + q); sh[q] = __ldg(shift + ch0 + q); }
    }
  }
#pragma unroll
  for (int q = 0; q < VEC; ++q) {
    if (scale) v[q] = fmaf(v[q], sc[q], sh[q]);
    const int g = gi[q];
    if (g == -1) {
      if (scalar_bias) v[q] += scalar_bias[ch0 + q];
      v[q] = apply_act(v[q], scalar_act);
    } else if (g >= 0) {
      v[q] *= my_gates[g];
    }
  }
  const size_t t = (size_t)row * groups + gq;
  if (OUT == 0) {
    if (VEC == 4) ((float4 *)out)[t] = make_float4(v[0], v[1 % VEC], v[2 % VEC], v[3 % VEC]);
    else if (VEC == 2) ((float2 *)out)[t] = make_float2(v[0], v[1 % VEC]);
    else ((float *)out)[t] = v[0];
  } else if (OUT == 2) {
    ((uint2 *)out)[t] = make_uint2(pack_bf16x2(v[0], v[1 % VEC]), pack_bf16x2(v[2 % VEC], v[3 % VEC]));
  } else {
    ((uint2 *)out)[t] = make_uint2(pack_f16x2(v[0], v[1 % VEC]), pack_f16x2(v[2 % VEC], v[3 % VEC]));
  }
}

// Launch of the row-block kernel when it applies (gated pass, at most 256 channel groups per row).
template <int OUT, int VEC>
static bool launch_bn_gate_rows(const float *x, int n, uint32_t groups, int c_in_total, const float *scale, const float *shift,
                                const int32_t *gate_of_channel, int c_gate_base, int scalar_act, int gate_act,
                                const float *scalar_bias, const float *gate_bias, void *out, cudaStream_t st) {
  const int n_gates = c_in_total - c_gate_base;
  if (gate_of_channel == nullptr || n_gates < 1 || groups < 1 || groups > 256) return false;
  const uint32_t R = 256u / groups;
  const size_t smem = (size_t)R * n_gates * sizeof(float);
  if (smem > 48 * 1024) return false;
  { launch_ready(bn_gate_rows_kernel<OUT, VEC>, dim3(ceil_div(n, (int)R)), dim3(groups, R), smem, st, x, (uint32_t)n, groups, c_in_total, scale, shift,
                                                                          gate_of_channel, c_gate_base, n_gates, scalar_act, gate_act,
                                                                          scalar_bias, gate_bias, out); note_launches(1); }
  return true;
}

// ---------------------------------------------------------------- batch statistics, training mode
// Column sums over the rows in an order that depends on the row count alone: rows L, L + chains, L + 2 chains ...
// form chain L of a channel (chains = 8 per row block, at most 512), added one after the other; the
// eight chains of a row block are added in order, then the row blocks, then the channels of a field.
// Batch statistics therefore repeat bit for bit, whatever grid or load width computes them.
// A thread walks one chain of VEC channels with AHEAD loads in flight, the last of a chain too: chains are few (20 k threads
// for 38 channels), so what bounds it is how many rows are on their way.  Whole batches of rows without a test between
// the loads, then the rest.  (ssc_bn_train: 121 k rows of 38 / 76 / 150 channels 16.9 / 19.9 / 22.4 us; with sixteen ahead and a rest one by one
// 25.1 / 39.6 / 27.5; with 32 or 64 ahead and a test before every load 25.4 / 27.3 / 46.4.  32 instead of 24: 16.8 / 19.3 / 23.2.)
// MODE 0: sum of x; 1: sum of (x - mean_ch)^2.  part [chains][c].
static int bn_row_blocks(int n) {
  const int rb = ceil_div(n, 8 * 64);
  return rb > 64 ? 64 : (rb < 1 ? 1 : rb);
}
template <int MODE, int VEC>
__global__ void __launch_bounds__(256)
bn_colsum_kernel(const float *__restrict__ x, int n, int c, int chains, int lanes, const float *__restrict__ chan_mean,
                 float *__restrict__ part) {
  after_previous();
  const int groups = c / VEC;
  const int lane = threadIdx.x / (blockDim.x / lanes), chain = blockIdx.x * lanes + lane;
  if (lane >= lanes || chain >= chains) return;
  for (int g = threadIdx.x % (blockDim.x / lanes); g < groups; g += blockDim.x / lanes) {
    const float *p = x + (size_t)chain * c + (size_t)g * VEC;
    const size_t step = (size_t)chains * c;
    constexpr int AHEAD = 24;
    float s[VEC], mu[VEC];
#pragma unroll
    for (int q = 0; q < VEC; ++q) {
      s[q] = 0.f;
      mu[q] = MODE != 0 ? chan_mean[g * VEC + q] : 0.f;
    }
    float v[AHEAD][VEC];
    auto load = [&](int i) {
      if (VEC == 4) {
        const float4 f = __ldg((const float4 *)(p + i * step));
        v[i][0] = f.x; v[i][1 % VEC] = f.y; v[i][2 % VEC] = f.z; v[i][3 % VEC] = f.w;
      } else {
        v[i][0] = __ldg(p + i * step);
      }
    };
    auto add = [&](int i) {
#pragma unroll
      for (int q = 0; q < VEC; ++q) {
        const float d = v[i][q] - mu[q];
        s[q] = MODE == 0 ? s[q] + d : fmaf(d, d, s[q]);
      }
    };
    int left = (n - chain + chains - 1) / chains;          // rows of the chain (chain < n, or none)
#pragma unroll 1
    for (; left >= AHEAD; left -= AHEAD, p += AHEAD * step) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) load(i);
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) add(i);
    }
#pragma unroll
    for (int i = 0; i < AHEAD - 1; ++i)
      if (i < left) load(i);
#pragma unroll
    for (int i = 0; i < AHEAD - 1; ++i)
      if (i < left) add(i);
#pragma unroll
    for (int q = 0; q < VEC; ++q) part[(size_t)chain * c + g * VEC + q] = s[q];
  }
}

// Sum of the chains of `count` consecutive channels from ch0, by one block, in the order stated above: the
// row blocks' sums of eight chains in parallel, then one thread adds them up.  Result in every thread.
constexpr int kFinishThreads = 512;        // (128: two rounds of loads for a field of four channels; ssc_bn_train of 72 k rows of 152: 18.0 us for 17.6)
constexpr int kFinishTile = 16 * 64;       // (channel, row block) sums in shared memory at a time
__device__ __forceinline__ float chain_total(const float *__restrict__ part, int row_blocks, int c, int ch0, int count) {
  __shared__ float sm[kFinishTile];
  __shared__ float result;
  float s = 0.f;
  for (int k0 = 0; k0 < count; k0 += 16) {
    const int m = min(16, count - k0) * row_blocks;
    for (int i = threadIdx.x; i < m; i += kFinishThreads) {
      const int k = i / row_blocks, rb = i - k * row_blocks;
      const float *p = part + (size_t)rb * 8 * c + ch0 + k0 + k;
      float v[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = __ldg(p + (size_t)t * c);
#pragma unroll
      for (int t = 1; t < 8; ++t) v[0] += v[t];
      sm[i] = v[0];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 16
      for (int i = 0; i < m; ++i) s += sm[i];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) result = s;
  __syncthreads();
  s = result;
  __syncthreads();
  return s;
}

// Block per channel: batch mean of the scalar channels (0 for the others), running mean updated with the
// arithmetic of running.mul_(1 - m).add_(m * mean).
__global__ void __launch_bounds__(kFinishThreads)
bn_finish_mean_kernel(const float *__restrict__ part, int row_blocks, int n, int c, const int32_t *__restrict__ scalar_of_channel,
                      float momentum, float keep, float *running_mean, float *mean, float *chan_mean) {
  after_previous();
  const int ch = blockIdx.x, s = scalar_of_channel[ch];
  if (s < 0) {
    if (threadIdx.x == 0) chan_mean[ch] = 0.f;
    return;
  }
  const float mu = chain_total(part, row_blocks, c, ch, 1) / (float)n;
  if (threadIdx.x == 0) {
    chan_mean[ch] = mu;
    mean[s] = mu;
    if (running_mean) running_mean[s] = __fadd_rn(__fmul_rn(running_mean[s], keep), __fmul_rn(momentum, mu));
  }
}

// First channel and number of channels of a field (the channels of a field are consecutive).
__device__ __forceinline__ int2 field_channels(const int32_t *__restrict__ field_of_channel, int c, int f) {
  __shared__ int first, count;
  if (threadIdx.x == 0) { first = c; count = 0; }
  __syncthreads();
  for (int ch = threadIdx.x; ch < c; ch += blockDim.x)
    if (field_of_channel[ch] == f) { atomicMin(&first, ch); atomicAdd(&count, 1); }
  __syncthreads();
  return make_int2(first, count);
}

// Block per field: mean squared norm, running value, and (scale != NULL) the per-channel affine of the pass.
__global__ void __launch_bounds__(kFinishThreads)
bn_finish_var_kernel(const float *__restrict__ part, int row_blocks, int n, int c, const int32_t *__restrict__ field_of_channel,
                     const int32_t *__restrict__ scalar_of_channel, const float *__restrict__ chan_mean,
                     const float *__restrict__ weight, const float *__restrict__ bias, float eps, float momentum, float keep,
                     float *running_var, float *var, float *scale, float *shift) {
  after_previous();
  const int f = blockIdx.x;
  const int2 fc = field_channels(field_of_channel, c, f);
  const float v = chain_total(part, row_blocks, c, fc.x, fc.y) / (float)n;
  if (threadIdx.x == 0) {
    var[f] = v;
    if (running_var) running_var[f] = __fadd_rn(__fmul_rn(running_var[f], keep), __fmul_rn(momentum, v));
  }
  if (scale)
    for (int k = threadIdx.x; k < fc.y; k += kFinishThreads) {
      const int ch = fc.x + k, sc_i = scalar_of_channel[ch];
      float sc = 1.0f / sqrtf(v + eps), sh = 0.f;
      if (weight) sc *= weight[f];
      if (sc_i >= 0) {
        // the roundings of bn_fold_kernel, so that a fold of the same statistics gives the same bits
        sh = __fmul_rn(-chan_mean[ch], sc);
        if (bias) sh = __fadd_rn(sh, bias[sc_i]);
      }
      scale[ch] = sc;
      shift[ch] = sh;
    }
}

// ------------------------------------------- backward of batch norm and gated activation, one pair of passes
// Forward of a row: y = x * scale + shift (batch norm), then out[ch] = y[ch] (copy), act(y[ch]) (scalars) or
// y[ch] * act(y[gate of ch]).  Backward, with g = gradient of y from the gradient of out:
//   copy: g = go;  scalar: g = go * act'(y);  gated: g = go * act(y_gate);
//   gate scalar j: g = act'(y_gate) * sum over its field of go[ch] * y[ch],
// and through y = (x - mu) * r * w (+ b), r = (v + eps)^-1/2, v = mean of the squared field norm:
//   A_f = sum over rows and components of g * (x - mu),  G_s = sum over rows of g:
//   d_w[f] = r A_f,  d_b[s] = G_s,  gx = ks g - ka (x - mu) - kg  with
//   ks = r w, ka = w r^3 A / N, kg = r w G / N (ka = kg = 0 with running statistics).
// y and g are recomputed from x and go in both passes (PASS 0 adds up A and G, PASS 1 writes gx), so neither
// is ever stored: 2 reads of x and go and one write of gx per backward, instead of four tensors more.
// A block takes R whole rows at a time into shared memory, every warp the rows w, w + 8, ... on its own: it copies them
// (the next tile's are on their way while it works on this one), evaluates their gates and turns go into g.
// PASS 0: block = one chain of rows (the order of the sums is that of the batch statistics above); the
// warps meet and a thread adds up its channels' rows.  PASS 1: R consecutive rows, and the warp writes gx.
// Without a gate table g = go (batch norm alone); without ks gx = g (activation alone).  Issue-bound, hence: the
// per-channel constants stand in shared memory as two 16-byte words, a sigmoid is evaluated once for value and
// slope, a lane works on two rows of its gate at a time (with constants read from global memory per
// element a row of 76 channels took 400 warp instructions: 33 + 38 us for 61 k rows).
struct BnGateBwd {
  const float *x, *go;
  int n, c, c_out, n_gates, rows, chains;      // rows = R
  const float *scale, *shift, *mu;             // per channel (may be NULL: identity / zero)
  const int32_t *gate_of_channel, *field_start, *field_len;
  int s_act, g_act;
};

constexpr int kBwdMaxAcc = 4;                  // channels of a thread in PASS 0

// Slope of the activation at v, `value` there given (the sigmoid's slope follows from it).
__device__ __forceinline__ float act_grad(float v, float value, int kind) {
  if (kind == 1) return v > 0.f ? 1.f : 0.f;
  if (kind == 2) return value * (1.f - value);
  return 1.f;
}
__host__ __device__ constexpr size_t align4(size_t floats) { return (floats + 3) & ~(size_t)3; }

template <int VEC>
__device__ __forceinline__ void copy_floats(float *dst, const float *src) {      // VEC floats, asynchronously
  const uint32_t to = smem_u32(dst);
  if (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
  else if (VEC == 2) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(src) : "memory");
}

template <int PASS, int VEC>
__global__ void __launch_bounds__(256)
bn_gate_bwd_kernel(BnGateBwd p, const float *__restrict__ ks, const float *__restrict__ ka, const float *__restrict__ kg,
                   float *__restrict__ gx, float *__restrict__ part_a, float *__restrict__ part_g) {
  after_previous();
  extern __shared__ __align__(16) float sm[];
  const int R = p.rows, c = p.c, c_out = p.c_out, n_gates = p.n_gates;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t buffer = (size_t)R * (c + c_out);                   // x rows, then go rows
  float *as = sm + 2 * buffer, *gg = as + (size_t)R * n_gates;
  // the block's rows are PASS 0 blockIdx.x, + chains, ..., PASS 1 R consecutive ones of every gridDim.x tiles: `row` of
  // its tile's first and `left` how many follow
  const int row_step = PASS == 0 ? p.chains : 1;
  const int tile_step = PASS == 0 ? R * p.chains : R * (int)gridDim.x;
  auto load = [&](int row, int rows, int buf) {
    float *xs = sm + buf * buffer, *gs = xs + (size_t)R * c;
    for (int r = warp; r < rows; r += 8) {
      const size_t at = (size_t)(row + r * row_step);
      for (int i = lane * VEC; i < c; i += 32 * VEC) copy_floats<VEC>(xs + r * c + i, p.x + at * c + i);
      for (int i = lane * VEC; i < c_out; i += 32 * VEC) copy_floats<VEC>(gs + r * c_out + i, p.go + at * c_out + i);
    }
    cp_async_commit();
  };
  // gates over the lanes: several rows at a time where a row has few
  const bool few = n_gates > 0 && n_gates <= 32;
  const int per = few ? 32 / n_gates : 1, lane_row = few ? lane / n_gates : 0, lane_gate = few ? lane % n_gates : lane;
  const bool affine = p.scale != nullptr;
  // constants of a channel: (scale, shift, mean, gate: -3 itself a gate scalar, -2 copy, -1 scalar), (ks, ka, kg)
  float4 *chan = (float4 *)(sm + align4(2 * buffer + 2 * (size_t)R * n_gates)), *coef = chan + c;
  for (int ch = tid; ch < c; ch += 256) {
    const int gate = p.gate_of_channel ? (ch < c_out ? __ldg(p.gate_of_channel + ch) : -3) : -2;
    chan[ch] = make_float4(affine ? __ldg(p.scale + ch) : 1.f, affine ? __ldg(p.shift + ch) : 0.f, p.mu ? __ldg(p.mu + ch) : 0.f, __int_as_float(gate));
    if (PASS == 1) coef[ch] = ks ? make_float4(__ldg(ks + ch), __ldg(ka + ch), __ldg(kg + ch), 0.f) : make_float4(1.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  float sum_a[kBwdMaxAcc], sum_g[kBwdMaxAcc];
#pragma unroll
  for (int i = 0; i < kBwdMaxAcc; ++i) sum_a[i] = sum_g[i] = 0.f;
  const int ch_block = PASS == 0 ? (int)blockIdx.y * 256 * kBwdMaxAcc : 0;

  const int first = PASS == 0 ? (int)blockIdx.x : (int)blockIdx.x * R;
  int left = PASS == 0 ? (p.n - first + p.chains - 1) / p.chains : 0;      // PASS 0: rows of the chain still to come
  auto rows_at = [&](int row, int in_chain) { return max(0, min(R, PASS == 0 ? in_chain : p.n - row)); };
  int buf = 0, rows = rows_at(first, left);
  load(first, rows, 0);
  for (int r0 = first; rows > 0; r0 += tile_step, buf ^= 1) {
    const int next = r0 > p.n - tile_step ? 0 : rows_at(r0 + tile_step, left - R);   // (r0 + tile_step stays below n)
    load(r0 + tile_step, next, buf ^ 1);                           // (nothing behind the last tile)
    cp_async_wait(1);
    __syncwarp();
    float *xs = sm + buf * buffer, *gs = xs + (size_t)R * c;
    if (lane_row < per) {
      for (int j = lane_gate; j < n_gates; j += 32) {
        const float4 kc = chan[c_out + j];
        const int s0 = __ldg(p.field_start + j), len = __ldg(p.field_len + j);
        for (int r = warp + 8 * lane_row; r < rows; r += 16 * per) {
          const int r2 = r + 8 * per < rows ? r + 8 * per : r;
          const float *xa = xs + r * c, *xb = xs + r2 * c, *ga = gs + r * c_out + s0, *gb = gs + r2 * c_out + s0;
          float va = xa[c_out + j], vb = xb[c_out + j], acc_a = 0.f, acc_b = 0.f;
          if (affine) {
            va = fmaf(va, kc.x, kc.y);
            vb = fmaf(vb, kc.x, kc.y);
          }
          for (int q = 0; q < len; ++q) {
            const float2 k = *(const float2 *)(chan + s0 + q);
            float ya = xa[s0 + q], yb = xb[s0 + q];
            if (affine) {
              ya = fmaf(ya, k.x, k.y);
              yb = fmaf(yb, k.x, k.y);
            }
            acc_a = fmaf(ga[q], ya, acc_a);
            acc_b = fmaf(gb[q], yb, acc_b);
          }
          const float fa = apply_act(va, p.g_act), fb = apply_act(vb, p.g_act);
          as[r * n_gates + j] = fa;
          gg[r * n_gates + j] = acc_a * act_grad(va, fa, p.g_act);
          if (r2 != r) {
            as[r2 * n_gates + j] = fb;
            gg[r2 * n_gates + j] = acc_b * act_grad(vb, fb, p.g_act);
          }
        }
      }
    }
    __syncwarp();
    // go of a channel into g; gates' values and the gate scalars' gradients stand in shared memory
    for (int ch0 = 0; ch0 < (PASS == 0 ? c_out : c); ch0 += 32) {
      const int ch = ch0 + lane;
      const bool in = ch < (PASS == 0 ? c_out : c);
      const float4 kc = chan[in ? ch : 0];
      const int gate = in ? __float_as_int(kc.w) : -2;
      const bool scalars = __any_sync(0xffffffffu, gate == -1);
      // where g comes from and what it is multiplied by (nothing: gate < 0)
      const float *from = gate == -3 ? gg + (ch - c_out) : gs + ch, *by = as + (gate >= 0 ? gate : 0);
      const int step = gate == -3 ? n_gates : c_out;
      if (!in || (PASS == 0 && gate < -1)) continue;
      const float4 kd = PASS == 1 ? coef[ch] : make_float4(0.f, 0.f, 0.f, 0.f);
      float *to = PASS == 1 ? gx + (size_t)(r0 + warp) * c + ch : gs + warp * c_out + ch;
#pragma unroll 4
      for (int r = warp; r < rows; r += 8) {
        const float x = PASS == 1 || scalars ? xs[r * c + ch] : 0.f;
        float g = from[r * step];
        if (gate >= 0) g *= by[r * n_gates];
        if (scalars && gate == -1) {
          const float y = affine ? fmaf(x, kc.x, kc.y) : x;
          g *= act_grad(y, p.s_act == 2 ? apply_act(y, 2) : 0.f, p.s_act);
        }
        *to = PASS == 0 ? g : ks ? kd.x * g - kd.y * (x - kc.z) - kd.z : g;
        to += PASS == 1 ? 8 * (size_t)c : 8 * (size_t)c_out;
      }
    }
    if (PASS == 0) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < kBwdMaxAcc; ++i) {
        const int ch = ch_block + tid + i * 256;
        if (ch < c) {
          const float mu = chan[ch].z;
          const float *gp = ch < c_out ? gs + ch : gg + (ch - c_out), *xp = xs + ch;
          const int gstep = ch < c_out ? c_out : n_gates;
          float s = sum_g[i], a = sum_a[i];
#pragma unroll 8
          for (int r = 0; r < rows; ++r) {
            const float g = gp[r * gstep];
            s += g;
            a = fmaf(g, xp[r * c] - mu, a);
          }
          sum_g[i] = s;
          sum_a[i] = a;
        }
      }
      __syncthreads();
    } else {
      __syncwarp();
    }
    left -= R;
    rows = next;
  }
  cp_async_wait_all();
  if (PASS == 0) {
#pragma unroll
    for (int i = 0; i < kBwdMaxAcc; ++i) {
      const int ch = ch_block + tid + i * 256;
      if (ch < c) {
        part_a[(size_t)blockIdx.x * c + ch] = sum_a[i];
        part_g[(size_t)blockIdx.x * c + ch] = sum_g[i];
      }
    }
  }
}

// The two passes for rows of up to 256 kept channels in fours, which is what the layers have: a lane has four channels (QL: or
// eight) of a row, L lanes a row, 32 / L rows a warp at a time, straight from and to global memory, other warps' rows on their way.
// Through shared memory go only (go, y), for the gates' sums, and the gates' values; a gate scalar belongs to one lane (or two do to one
// lane), which keeps its sums like those of its kept channels.  PASS 0 adds up rows in registers: the warps' rows in ascending order, then a warp's
// rows, then a block's warps in order; a block is one chain of the totals.  That is another order than the form above has, at the same
// distance from 64 bits (gradient of the weight, relative, mean of twelve: 162 k rows of 32 + 6 2.0e-7 both, 20 k of 16 + 4 1.2e-7 and 1.3e-7, 700 of 32 + 8
// 1.0e-7 and 0.9e-7).  The form above hands every element through shared memory
// and adds up a channel per thread, 32 rows at a time, while the other threads wait: 162 k rows of 32 + 6 channels 47 + 33 us, here
// 19 + 16; 93 k rows of 64 + 12 30 + 25, here 18 + 16 (the bytes of the two passes take 8 and 12).  A gate's sum takes fields of up
// to seven channels at once: as a loop it was half of the kernel.  Wider rows, others than fours and some of many rows (launch_bwd) stay above.
template <int VEC>
__device__ __forceinline__ void row_quad(const float *at, float (&v)[4]) {
  if (VEC == 4) {
    const float4 q = __ldg((const float4 *)at);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else if (VEC == 2) {
    const float2 a = __ldg((const float2 *)at), b = __ldg((const float2 *)at + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __ldg(at + i);
  }
}
template <int PASS, int VEC, int GVEC, int QL>
__global__ void __launch_bounds__(256, QL == 1 ? 4 : 2)
bn_gate_bwd_lanes_kernel(BnGateBwd p, int L, const float *__restrict__ ks, const float *__restrict__ ka, const float *__restrict__ kg,
                         float *__restrict__ gx, float *__restrict__ part_a, float *__restrict__ part_g) {
  after_previous();
  extern __shared__ __align__(16) float sm[];
  constexpr int GL = QL;                       // gate scalars of a lane
  const int c = p.c, c_out = p.c_out, n_gates = p.n_gates, n = p.n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int at = lane & (L - 1), slot = lane / L, per = 32 / L;
  const bool affine = p.scale != nullptr;
  float2 *pairs = (float2 *)sm + (size_t)(warp * per + slot) * c_out;                    // (go, y) of the lane's row
  float *acts = sm + (size_t)16 * per * c_out + (size_t)(warp * per + slot) * (n_gates + 1);   // its gates' values, and a one
  // constants of the lane's channels
  float sc[QL][4], sh[QL][4], mu[QL][4], cs[QL][4], ca[QL][4], cg[QL][4];
  const float *act[QL][4];                     // what a channel's gradient is multiplied by
  uint32_t scalars = 0u;                       // bit 4 q + i
  bool mine[QL];
#pragma unroll
  for (int q = 0; q < QL; ++q) {
    mine[q] = (at + q * L) * 4 < c_out;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ch = mine[q] ? (at + q * L) * 4 + i : 0;
      sc[q][i] = affine ? __ldg(p.scale + ch) : 1.f;
      sh[q][i] = affine ? __ldg(p.shift + ch) : 0.f;
      mu[q][i] = p.mu ? __ldg(p.mu + ch) : 0.f;
      const int gate = p.gate_of_channel ? __ldg(p.gate_of_channel + ch) : -2;
      act[q][i] = acts + (gate >= 0 ? gate : n_gates);
      if (gate == -1 && p.s_act != 0) scalars |= 1u << (4 * q + i);
      if (PASS == 1 && ks) { cs[q][i] = __ldg(ks + ch); ca[q][i] = __ldg(ka + ch); cg[q][i] = __ldg(kg + ch); }
    }
  }
  float gsc[GL], gsh[GL], gmu[GL], gcs[GL], gca[GL], gcg[GL];
  const float2 *field[GL];
  int glen[GL];
  bool has[GL];
#pragma unroll
  for (int k = 0; k < GL; ++k) {
    const int j = at + k * L, ch = c_out + j;
    has[k] = j < n_gates;
    gsc[k] = has[k] && affine ? __ldg(p.scale + ch) : 1.f;
    gsh[k] = has[k] && affine ? __ldg(p.shift + ch) : 0.f;
    gmu[k] = has[k] && p.mu ? __ldg(p.mu + ch) : 0.f;
    field[k] = pairs + (has[k] ? __ldg(p.field_start + j) : 0);
    glen[k] = has[k] ? __ldg(p.field_len + j) : 0;
    if (PASS == 1 && ks && has[k]) { gcs[k] = __ldg(ks + ch); gca[k] = __ldg(ka + ch); gcg[k] = __ldg(kg + ch); }
  }
  if (at == 0) acts[n_gates] = 1.f;
  float sum_a[QL][4], sum_g[QL][4], gsum_a[GL], gsum_g[GL];
#pragma unroll
  for (int q = 0; q < QL; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) sum_a[q][i] = sum_g[q][i] = 0.f;
#pragma unroll
  for (int k = 0; k < GL; ++k) gsum_a[k] = gsum_g[k] = 0.f;
  __syncwarp();

  const int step = (int)gridDim.x * 8 * per;
  int row = ((int)blockIdx.x * 8 + warp) * per + slot;
  for (int left = n - (row - slot); left > 0; left -= step, row += step) {     // rows from the warp's first on
    const bool in = slot < left;
    float x[QL][4], go[QL][4], xg[GL], gate_g[GL];
    const float *xr = p.x + (size_t)row * c, *gr = p.go + (size_t)row * c_out;
#pragma unroll
    for (int q = 0; q < QL; ++q) {
#pragma unroll
      for (int i = 0; i < 4; ++i) x[q][i] = go[q][i] = 0.f;
      if (in && mine[q]) {
        row_quad<VEC>(xr + (at + q * L) * 4, x[q]);
        row_quad<GVEC>(gr + (at + q * L) * 4, go[q]);
      }
    }
#pragma unroll
    for (int k = 0; k < GL; ++k) xg[k] = in && has[k] ? __ldg(xr + c_out + at + k * L) : 0.f;
    if (n_gates > 0) {
#pragma unroll
      for (int q = 0; q < QL; ++q)
        if (mine[q]) {
          float y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = affine ? fmaf(x[q][i], sc[q][i], sh[q][i]) : x[q][i];
          float4 *to = (float4 *)(pairs + (at + q * L) * 4);
          to[0] = make_float4(go[q][0], y[0], go[q][1], y[1]);
          to[1] = make_float4(go[q][2], y[2], go[q][3], y[3]);
        }
      __syncwarp();
      float v[GL], f[GL];
#pragma unroll
      for (int k = 0; k < GL; ++k) {
        float2 t[7];                           // (fields of up to order three at once)
#pragma unroll
        for (int i = 0; i < 7; ++i) t[i] = i < glen[k] ? field[k][i] : make_float2(0.f, 0.f);
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < 7; ++i)
          if (i < glen[k]) acc = fmaf(t[i].x, t[i].y, acc);
        for (int i = 7; i < glen[k]; ++i) {
          const float2 u = field[k][i];
          acc = fmaf(u.x, u.y, acc);
        }
        gate_g[k] = acc;
        v[k] = affine ? fmaf(xg[k], gsc[k], gsh[k]) : xg[k];
        f[k] = v[k];
      }
      if (p.g_act == 2) {
        apply_sigmoids<GL>(f);
      } else {
#pragma unroll
        for (int k = 0; k < GL; ++k) f[k] = apply_act(v[k], p.g_act);
      }
#pragma unroll
      for (int k = 0; k < GL; ++k) {
        gate_g[k] *= act_grad(v[k], f[k], p.g_act);
        if (has[k]) acts[at + k * L] = f[k];
      }
      __syncwarp();
    }
#pragma unroll
    for (int q = 0; q < QL; ++q) {
      float g[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = n_gates > 0 ? go[q][i] * *act[q][i] : go[q][i];
      if ((scalars >> (4 * q)) & 15u) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if ((scalars >> (4 * q + i)) & 1u) {
            const float y = affine ? fmaf(x[q][i], sc[q][i], sh[q][i]) : x[q][i];
            g[i] *= act_grad(y, p.s_act == 2 ? apply_act(y, 2) : 0.f, p.s_act);
          }
      }
      if (!in || !mine[q]) continue;
      if (PASS == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sum_g[q][i] += g[i];
          sum_a[q][i] = fmaf(g[i], x[q][i] - mu[q][i], sum_a[q][i]);
        }
      } else {
        float o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = ks ? cs[q][i] * g[i] - ca[q][i] * (x[q][i] - mu[q][i]) - cg[q][i] : g[i];
        float *to = gx + (size_t)row * c + (at + q * L) * 4;
        if (VEC == 4) {
          *(float4 *)to = make_float4(o[0], o[1], o[2], o[3]);
        } else if (VEC == 2) {
          *(float2 *)to = make_float2(o[0], o[1]);
          *((float2 *)to + 1) = make_float2(o[2], o[3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) to[i] = o[i];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < GL; ++k)
      if (in && has[k]) {
        const float d = xg[k] - gmu[k];
        if (PASS == 0) {
          gsum_g[k] += gate_g[k];
          gsum_a[k] = fmaf(gate_g[k], d, gsum_a[k]);
        } else {
          gx[(size_t)row * c + c_out + at + k * L] = ks ? gcs[k] * gate_g[k] - gca[k] * d - gcg[k] : gate_g[k];
        }
      }
  }
  if (PASS == 0) {
    auto rows_of_warp = [&](float v) {
      for (int o = L; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      return v;
    };
    __syncthreads();
    float *ra = sm + (size_t)warp * 2 * c, *rg = ra + c;
#pragma unroll
    for (int q = 0; q < QL; ++q)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float a = rows_of_warp(sum_a[q][i]), g = rows_of_warp(sum_g[q][i]);
        if (slot == 0 && mine[q]) { ra[(at + q * L) * 4 + i] = a; rg[(at + q * L) * 4 + i] = g; }
      }
#pragma unroll
    for (int k = 0; k < GL; ++k) {
      const float a = rows_of_warp(gsum_a[k]), g = rows_of_warp(gsum_g[k]);
      if (slot == 0 && has[k]) { ra[c_out + at + k * L] = a; rg[c_out + at + k * L] = g; }
    }
    __syncthreads();
    for (int ch = threadIdx.x; ch < c; ch += 256) {
      float a = sm[ch], g = sm[c + ch];
#pragma unroll
      for (int w = 1; w < 8; ++w) { a += sm[(size_t)w * 2 * c + ch]; g += sm[(size_t)w * 2 * c + c + ch]; }
      part_a[(size_t)blockIdx.x * c + ch] = a;
      part_g[(size_t)blockIdx.x * c + ch] = g;
    }
  }
}

// The same for rows of which not even one fits shared memory twice with its constants (more than about 4800
// channels): a thread per channel, everything read where it lies.  Same sums in the same order.
template <int PASS>
__global__ void __launch_bounds__(256)
bn_gate_bwd_wide_kernel(BnGateBwd p, const float *__restrict__ ks, const float *__restrict__ ka, const float *__restrict__ kg,
                        float *__restrict__ gx, float *__restrict__ part_a, float *__restrict__ part_g) {
  after_previous();
  const int ch = (int)(blockIdx.y * 256 + threadIdx.x);
  if (ch >= p.c) return;
  auto normed = [&](const float *xr, int k) { return p.scale ? fmaf(__ldg(xr + k), __ldg(p.scale + k), __ldg(p.shift + k)) : __ldg(xr + k); };
  const int gate = p.gate_of_channel ? (ch < p.c_out ? __ldg(p.gate_of_channel + ch) : -3) : -2;
  const float mu = p.mu ? __ldg(p.mu + ch) : 0.f;
  float sum_a = 0.f, sum_g = 0.f;
  const int step = PASS == 0 ? p.chains : (int)gridDim.x;
  for (long long r = blockIdx.x; r < p.n; r += step) {
    const float *xr = p.x + (size_t)r * p.c, *gr = p.go + (size_t)r * p.c_out;
    float g;
    if (gate == -3) {
      const int s0 = __ldg(p.field_start + ch - p.c_out), len = __ldg(p.field_len + ch - p.c_out);
      float acc = 0.f;
      for (int q = 0; q < len; ++q) acc = fmaf(__ldg(gr + s0 + q), normed(xr, s0 + q), acc);
      const float v = normed(xr, ch);
      g = acc * act_grad(v, apply_act(v, p.g_act), p.g_act);
    } else {
      g = __ldg(gr + ch);
      if (gate >= 0) {
        g *= apply_act(normed(xr, p.c_out + gate), p.g_act);
      } else if (gate == -1) {
        const float y = normed(xr, ch);
        g *= act_grad(y, p.s_act == 2 ? apply_act(y, 2) : 0.f, p.s_act);
      }
    }
    const float d = __ldg(xr + ch) - mu;
    if (PASS == 0) {
      sum_g += g;
      sum_a = fmaf(g, d, sum_a);
    } else {
      gx[(size_t)r * p.c + ch] = ks ? __ldg(ks + ch) * g - __ldg(ka + ch) * d - __ldg(kg + ch) : g;
    }
  }
  if (PASS == 0) {
    part_a[(size_t)blockIdx.x * p.c + ch] = sum_a;
    part_g[(size_t)blockIdx.x * p.c + ch] = sum_g;
  }
}

// Block per field: A and G from the chains, the field's coefficients and parameter gradients.
__global__ void __launch_bounds__(kFinishThreads)
bn_bwd_finish_kernel(const float *__restrict__ part_a, const float *__restrict__ part_g, int row_blocks, int n, int c,
                     const int32_t *__restrict__ field_of_channel, const int32_t *__restrict__ scalar_of_channel,
                     const float *__restrict__ var, const float *__restrict__ weight, float eps, int training,
                     float *__restrict__ ks, float *__restrict__ ka, float *__restrict__ kg, float *__restrict__ d_weight,
                     float *__restrict__ d_bias) {
  after_previous();
  const int f = blockIdx.x;
  const int2 fc = field_channels(field_of_channel, c, f);
  const float A = chain_total(part_a, row_blocks, c, fc.x, fc.y);
  const int s = fc.y == 1 ? scalar_of_channel[fc.x] : -1;
  const float G = s >= 0 ? chain_total(part_g, row_blocks, c, fc.x, 1) : 0.f;
  const float r = 1.0f / sqrtf(var[f] + eps), w = weight ? weight[f] : 1.f;
  for (int k = threadIdx.x; k < fc.y; k += kFinishThreads) {
    const int ch = fc.x + k;
    ks[ch] = r * w;
    ka[ch] = training ? w * r * r * r * A / (float)n : 0.f;
    kg[ch] = (training && s >= 0) ? r * w * G / (float)n : 0.f;
  }
  if (threadIdx.x == 0) {
    if (d_weight) d_weight[f] = A / sqrtf(var[f] + eps);
    if (s >= 0 && d_bias) d_bias[s] = G;
  }
}

// chan_mean[ch] = mean of a scalar channel (0 for l>0 channels).
__global__ void bn_chan_mean_kernel(const float *mean, const int32_t *scalar_of_channel, int c, float *chan_mean) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c) return;
  const int s = scalar_of_channel[i];
  chan_mean[i] = s >= 0 ? mean[s] : 0.f;
}

}  // namespace ssc

using namespace ssc;

extern "C" int ssc_bn_fold(const float *running_mean, const float *running_var, const float *weight,
                           const float *bias, const int32_t *field_of_channel, const int32_t *scalar_of_channel,
                           int c, float eps, float *scale, float *shift, void *stream) {
  SSC_REQUIRE(c >= 1 && running_var && field_of_channel && scalar_of_channel && scale && shift, "bn_fold: bad arguments");
  { launch_ready(bn_fold_kernel, dim3(ceil_div(c, 128)), dim3(128), 0, as_stream(stream), running_mean, running_var, weight, bias,
                                                                 field_of_channel, scalar_of_channel, c, eps, scale, shift); note_launches(1); }
  SSC_CHECK_LAUNCH("bn_fold");
  return SSC_OK;
}

extern "C" int ssc_bn_gate_fwd(const float *x, int n, int c_in_total, const float *scale, const float *shift,
                               const int32_t *gate_of_channel, int c_out, int c_gate_base, int scalar_act,
                               int gate_act, const float *scalar_bias, const float *gate_bias, float *out,
                               void *stream) {
  SSC_REQUIRE(n >= 0 && c_in_total >= 1 && c_out >= 1 && c_out <= c_in_total, "bn_gate_fwd: bad sizes");
  SSC_REQUIRE((scale == nullptr) == (shift == nullptr), "bn_gate_fwd: scale and shift go together");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(x && out, "bn_gate_fwd: null pointer");
  long long total = (long long)n * c_out;
  const bool vec = (c_out & 3) == 0 && (c_in_total & 3) == 0 && (c_gate_base & 3) == 0 && total / 4 < (1ll << 31) &&
                   (((uintptr_t)x | (uintptr_t)out | (uintptr_t)scale | (uintptr_t)shift | (uintptr_t)gate_of_channel) & 15u) == 0;
  if (vec) {
    const uint32_t groups = (uint32_t)(c_out >> 2), total4 = (uint32_t)(total >> 2);
    if (launch_bn_gate_rows<0, 4>(x, n, groups, c_in_total, scale, shift, gate_of_channel, c_gate_base, scalar_act, gate_act,
                                  scalar_bias, gate_bias, out, as_stream(stream))) {
      SSC_CHECK_LAUNCH("bn_gate_fwd");
      return SSC_OK;
    }
    { launch_ready(bn_gate_vec4_kernel, dim3(ceil_div(total4, 256)), dim3(256), 0, as_stream(stream), x, total4, groups, c_in_total, scale, shift,
                                                                            gate_of_channel, c_gate_base, scalar_act, gate_act,
                                                                            scalar_bias, gate_bias, out); note_launches(1); }
    SSC_CHECK_LAUNCH("bn_gate_fwd");
    return SSC_OK;
  }
  // channel counts that are not multiples of four: two channels per thread when everything is even,
  // else one (the row-block kernel still evaluates every gate once per row)
  const bool even = (c_out & 1) == 0 && (c_in_total & 1) == 0 && (((uintptr_t)x | (uintptr_t)out) & 7u) == 0;
  if (even ? launch_bn_gate_rows<0, 2>(x, n, (uint32_t)(c_out >> 1), c_in_total, scale, shift, gate_of_channel, c_gate_base,
                                       scalar_act, gate_act, scalar_bias, gate_bias, out, as_stream(stream))
           : launch_bn_gate_rows<0, 1>(x, n, (uint32_t)c_out, c_in_total, scale, shift, gate_of_channel, c_gate_base,
                                       scalar_act, gate_act, scalar_bias, gate_bias, out, as_stream(stream))) {
    SSC_CHECK_LAUNCH("bn_gate_fwd");
    return SSC_OK;
  }
  { launch_ready(bn_gate_kernel, dim3(ceil_div(total, 256)), dim3(256), 0, as_stream(stream), x, total, c_in_total, scale, shift, gate_of_channel,
                                                                     c_out, c_gate_base, scalar_act, gate_act,
                                                                     scalar_bias, gate_bias, out); note_launches(1); }
  SSC_CHECK_LAUNCH("bn_gate_fwd");
  return SSC_OK;
}

extern "C" int ssc_bn_gate_fwd16(const float *x, int n, int c_in_total, const float *scale, const float *shift,
                                 const int32_t *gate_of_channel, int c_out, int c_gate_base, int scalar_act,
                                 int gate_act, const float *scalar_bias, const float *gate_bias, int precision,
                                 void *out16, void *stream) {
  SSC_REQUIRE(n >= 0 && c_in_total >= 1 && c_out >= 1 && c_out <= c_in_total, "bn_gate_fwd16: bad sizes");
  SSC_REQUIRE(precision == SSC_PREC_F16 || precision == SSC_PREC_BF16, "bn_gate_fwd16: precision must be SSC_PREC_F16 or SSC_PREC_BF16");
  SSC_REQUIRE((scale == nullptr) == (shift == nullptr), "bn_gate_fwd16: scale and shift go together");
  SSC_REQUIRE((c_out & 7) == 0 && (c_in_total & 3) == 0 && (c_gate_base & 3) == 0,
              "bn_gate_fwd16: needs c_out a multiple of 8 (16-byte rows) and c_in_total, c_gate_base multiples of 4");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(x && out16, "bn_gate_fwd16: null pointer");
  SSC_REQUIRE((((uintptr_t)x | (uintptr_t)out16 | (uintptr_t)scale | (uintptr_t)shift | (uintptr_t)gate_of_channel) & 15u) == 0,
              "bn_gate_fwd16: pointers must be 16-byte aligned");
  const long long total = (long long)n * c_out;
  SSC_REQUIRE(total / 4 < (1ll << 31), "bn_gate_fwd16: tensor too large");
  const uint32_t groups = (uint32_t)(c_out >> 2), total4 = (uint32_t)(total >> 2);
  if (precision == SSC_PREC_BF16
          ? launch_bn_gate_rows<2, 4>(x, n, groups, c_in_total, scale, shift, gate_of_channel, c_gate_base, scalar_act, gate_act,
                                   scalar_bias, gate_bias, out16, as_stream(stream))
          : launch_bn_gate_rows<1, 4>(x, n, groups, c_in_total, scale, shift, gate_of_channel, c_gate_base, scalar_act, gate_act,
                                   scalar_bias, gate_bias, out16, as_stream(stream))) {
    SSC_CHECK_LAUNCH("bn_gate_fwd16");
    return SSC_OK;
  }
  if (precision == SSC_PREC_BF16) {
    { launch_ready(bn_gate_vec4_out16_kernel<2>, dim3(ceil_div(total4, 256)), dim3(256), 0, as_stream(stream), x, total4, groups, c_in_total, scale, shift, gate_of_channel, c_gate_base, scalar_act, gate_act, scalar_bias, gate_bias, (uint2 *)out16); note_launches(1); }
  } else {
    { launch_ready(bn_gate_vec4_out16_kernel<1>, dim3(ceil_div(total4, 256)), dim3(256), 0, as_stream(stream), x, total4, groups, c_in_total, scale, shift, gate_of_channel, c_gate_base, scalar_act, gate_act, scalar_bias, gate_bias, (uint2 *)out16); note_launches(1); }
  }
  SSC_CHECK_LAUNCH("bn_gate_fwd16");
  return SSC_OK;
}

extern "C" size_t ssc_bn_scratch_bytes(int n, int c) {
  if (n < 0 || c < 1) return 0;
  // two planes of chain sums [8 row blocks, c], per-channel mean and three coefficient rows
  return ((size_t)2 * 8 * bn_row_blocks(n) * c + (size_t)4 * c + 64) * sizeof(float);
}

static int launch_colsum(int mode, const float *x, int n, int c, const float *chan_mean, float *part, cudaStream_t st) {
  const bool vec = (c & 3) == 0 && ((uintptr_t)x & 15u) == 0;
  const int groups = vec ? c / 4 : c, chains = 8 * bn_row_blocks(n);
  // two blocks per SM where there are that many chains
  int lanes = chains / (2 * 148);
  if (lanes > 256 / groups) lanes = 256 / groups;
  if (lanes < 1) lanes = 1;
  const int threads = lanes * (groups < 256 ? groups : 256), blocks = ceil_div(chains, lanes);
  if (vec) {
    if (mode == 0) launch_ready(bn_colsum_kernel<0, 4>, dim3(blocks), dim3(threads), 0, st, x, n, c, chains, lanes, chan_mean, part);
    else launch_ready(bn_colsum_kernel<1, 4>, dim3(blocks), dim3(threads), 0, st, x, n, c, chains, lanes, chan_mean, part);
  } else {
    if (mode == 0) launch_ready(bn_colsum_kernel<0, 1>, dim3(blocks), dim3(threads), 0, st, x, n, c, chains, lanes, chan_mean, part);
    else launch_ready(bn_colsum_kernel<1, 1>, dim3(blocks), dim3(threads), 0, st, x, n, c, chains, lanes, chan_mean, part);
  }
  note_launches(1);
  SSC_CHECK_LAUNCH("bn_colsum");
  return SSC_OK;
}

extern "C" int ssc_bn_train(const float *x, int n, int c, const int32_t *field_of_channel, const int32_t *scalar_of_channel,
                            int n_field, int n_scalar, const float *weight, const float *bias, float eps, double momentum,
                            float *running_mean, float *running_var, float *mean, float *var, float *chan_mean,
                            float *scale, float *shift, void *scratch, size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(n >= 1 && c >= 1 && n_field >= 1 && n_scalar >= 0, "bn_train: bad sizes");
  SSC_REQUIRE(x && field_of_channel && scalar_of_channel && mean && var && chan_mean, "bn_train: null pointer");
  SSC_REQUIRE((scale == nullptr) == (shift == nullptr), "bn_train: scale and shift go together");
  SSC_REQUIRE(scratch && scratch_bytes >= ssc_bn_scratch_bytes(n, c), "bn_train: scratch too small (ssc_bn_scratch_bytes)");
  cudaStream_t st = as_stream(stream);
  float *part = (float *)scratch;
  const int rb = bn_row_blocks(n);
  const float m = (float)momentum, keep = (float)(1.0 - momentum);
  if (int e = launch_colsum(0, x, n, c, nullptr, part, st)) return e;
  { launch_ready(bn_finish_mean_kernel, dim3(c), dim3(kFinishThreads), 0, st, part, rb, n, c, scalar_of_channel, m, keep, running_mean, mean, chan_mean); note_launches(1); }
  if (int e = launch_colsum(1, x, n, c, chan_mean, part, st)) return e;
  { launch_ready(bn_finish_var_kernel, dim3(n_field), dim3(kFinishThreads), 0, st, part, rb, n, c, field_of_channel, scalar_of_channel, chan_mean, weight, bias,
                                                           eps, m, keep, running_var, var, scale, shift); note_launches(1); }
  SSC_CHECK_LAUNCH("bn_train");
  return SSC_OK;
}

// var must have room for n_field + c floats (the tail holds the per-channel means); scratch holds the
// partial sums: ssc_bn_scratch_bytes(n, c).
extern "C" int ssc_bn_stats(const float *x, int n, int c, const int32_t *field_of_channel,
                            const int32_t *scalar_of_channel, int n_field, int n_scalar, float *mean, float *var,
                            void *scratch, size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(var, "bn_stats: null pointer");
  return ssc_bn_train(x, n, c, field_of_channel, scalar_of_channel, n_field, n_scalar, nullptr, nullptr, 0.f, 0.0, nullptr, nullptr,
                      mean, var, var + n_field, nullptr, nullptr, scratch, scratch_bytes, stream);
}

// Rows per tile of the backward kernels: a multiple of eight (a row per warp), as many as 44 KB of shared memory hold
// twice (five blocks per SM); fewer where eight rows do not fit.
static int bwd_tile_rows(int c, int c_out, int n_gates, int most, size_t *smem) {
  const size_t per_row = (size_t)(2 * (c + c_out) + 2 * n_gates) * sizeof(float), fixed = (size_t)c * 32 + 16;
  int rows = most;
  while (rows > 8 && rows * per_row + fixed > 44 * 1024) rows -= 8;
  while (rows > 1 && rows * per_row + fixed > 200 * 1024) --rows;
  *smem = rows * per_row + fixed;
  return rows;
}

template <int PASS, int VEC>
static int launch_bwd_vec(const BnGateBwd &p, size_t smem, const float *ks, const float *ka, const float *kg, float *gx, float *part_a, float *part_g, cudaStream_t st) {
  if (smem > 48 * 1024) {
    cudaError_t e = allow_smem((const void *)bn_gate_bwd_kernel<PASS, VEC>, smem);
    if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "bn_gate_bwd: smem attribute: %s", cudaGetErrorString(e));
  }
  int blocks = PASS == 0 ? p.chains : ceil_div(p.n, p.rows);
  if (PASS == 1 && blocks > 5 * 148) blocks = 5 * 148;
  launch_ready(bn_gate_bwd_kernel<PASS, VEC>, dim3(blocks, PASS == 0 ? ceil_div(p.c, 256 * kBwdMaxAcc) : 1), dim3(256), smem, st, p, ks, ka, kg, gx, part_a, part_g);
  note_launches(1);
  SSC_CHECK_LAUNCH("bn_gate_bwd");
  return SSC_OK;
}

template <int PASS, int QL>
static void launch_bwd_lanes(const BnGateBwd &p, int lanes, const float *ks, const float *ka, const float *kg, float *gx, float *part_a, float *part_g, cudaStream_t st) {
  const int per = 32 / lanes;
  size_t smem = ((size_t)16 * per * p.c_out + (size_t)8 * per * (p.n_gates + 1)) * sizeof(float);
  if (PASS == 0 && smem < (size_t)16 * p.c * sizeof(float)) smem = (size_t)16 * p.c * sizeof(float);
  int blocks = p.chains;
  if (PASS == 1) {
    blocks = ceil_div(p.n, 8 * per);
    const int most = (QL == 1 ? 4 : 2) * sm_count();
    if (blocks > most) blocks = most;
  }
  // (the order of the sums does not depend on where rows and gradients lie: only how they are loaded does)
  const uintptr_t at = (uintptr_t)p.x | (uintptr_t)gx;
  auto kernel = bn_gate_bwd_lanes_kernel<PASS, 1, 1, QL>;
  if (((uintptr_t)p.go & 15u) == 0)
    kernel = (p.c & 3) == 0 && (at & 15u) == 0  ? bn_gate_bwd_lanes_kernel<PASS, 4, 4, QL>
             : (p.c & 1) == 0 && (at & 7u) == 0 ? bn_gate_bwd_lanes_kernel<PASS, 2, 4, QL>
                                                : bn_gate_bwd_lanes_kernel<PASS, 1, 4, QL>;
  launch_ready(kernel, dim3(blocks), dim3(256), smem, st, p, lanes, ks, ka, kg, gx, part_a, part_g);
  note_launches(1);
}

template <int PASS>
static int launch_bwd(BnGateBwd p, const float *ks, const float *ka, const float *kg, float *gx, float *part_a, float *part_g, cudaStream_t st) {
  size_t smem;
  p.chains = 8 * bn_row_blocks(p.n);
  int lanes = 1;
  while (lanes < 32 && lanes * 4 < p.c_out) lanes <<= 1;
  // Of many rows of which two fifths of the lanes have no channels the other form is the faster one where its copies are of 16 bytes and
  // little else is to do: 132 to 152 normed channels without gates (144: 60 k rows 63.6 and 61.4 us here, 100 k
  // 97.9 and 105.6, 600 k 518 and 565), the gate's gradient alone of 68 and 72 (72 + 16: 100 k rows 36.3 and 38.4, 600 k 205 and 222).
  const bool idle = p.n > 65536 && p.c_out * 5 < lanes * (p.c_out <= 128 ? 12 : 24) && (p.c & 3) == 0;
  const bool wide = p.c_out > 128 ? p.n_gates == 0 : PASS == 1 && ks == nullptr && p.c_out > 64;
  if ((p.c_out & 3) == 0 && p.c_out <= 256 && p.n_gates <= 2 * lanes && !(idle && wide)) {
    if (p.c_out <= 128 && p.n_gates <= lanes) launch_bwd_lanes<PASS, 1>(p, lanes, ks, ka, kg, gx, part_a, part_g, st);
    else launch_bwd_lanes<PASS, 2>(p, lanes, ks, ka, kg, gx, part_a, part_g, st);
    SSC_CHECK_LAUNCH("bn_gate_bwd");
    return SSC_OK;
  }
  p.rows = bwd_tile_rows(p.c, p.c_out, p.n_gates, PASS == 0 ? 32 : 64, &smem);
  if (smem > 227 * 1024) {
    const int blocks = PASS == 0 ? p.chains : (p.n < 4 * 148 ? p.n : 4 * 148);
    launch_ready(bn_gate_bwd_wide_kernel<PASS>, dim3(blocks, ceil_div(p.c, 256)), dim3(256), 0, st, p, ks, ka, kg, gx, part_a, part_g);
    note_launches(1);
    SSC_CHECK_LAUNCH("bn_gate_bwd");
    return SSC_OK;
  }
  const int odd = p.c | p.c_out;
  const uintptr_t at = (uintptr_t)p.x | (uintptr_t)p.go;
  if ((odd & 3) == 0 && (at & 15u) == 0) return launch_bwd_vec<PASS, 4>(p, smem, ks, ka, kg, gx, part_a, part_g, st);
  if ((odd & 1) == 0 && (at & 7u) == 0) return launch_bwd_vec<PASS, 2>(p, smem, ks, ka, kg, gx, part_a, part_g, st);
  return launch_bwd_vec<PASS, 1>(p, smem, ks, ka, kg, gx, part_a, part_g, st);
}

extern "C" int ssc_bn_gate_bwd(const float *x, const float *gout, int n, int c, int c_out, const int32_t *field_of_channel,
                               const int32_t *scalar_of_channel, int n_field, const float *scale, const float *shift,
                               const float *chan_mean, const float *var, const float *weight, float eps, int training,
                               const int32_t *gate_of_channel, const int32_t *field_start, const int32_t *field_len,
                               int scalar_act, int gate_act, float *gx, float *d_weight, float *d_bias, void *scratch,
                               size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(n >= 1 && c >= 1 && c_out >= 1 && c_out <= c && n_field >= 1, "bn_gate_bwd: bad sizes");
  SSC_REQUIRE(x && gout && field_of_channel && scalar_of_channel && chan_mean && var && gx, "bn_gate_bwd: null pointer");
  SSC_REQUIRE(gate_of_channel ? (scale && shift && (c == c_out || (field_start && field_len))) : c == c_out, "bn_gate_bwd: gate tables do not fit the channels");
  SSC_REQUIRE(scratch && scratch_bytes >= ssc_bn_scratch_bytes(n, c), "bn_gate_bwd: scratch too small (ssc_bn_scratch_bytes)");
  cudaStream_t st = as_stream(stream);
  const int rb = bn_row_blocks(n);
  float *part_a = (float *)scratch, *part_g = part_a + (size_t)8 * rb * c;
  float *ks = part_g + (size_t)8 * rb * c, *ka = ks + c, *kg = ka + c;
  BnGateBwd p = {x, gout, n, c, c_out, gate_of_channel ? c - c_out : 0, 0, 0, scale, shift, chan_mean, gate_of_channel, field_start, field_len,
                 scalar_act, gate_act};
  if (int e = launch_bwd<0>(p, nullptr, nullptr, nullptr, nullptr, part_a, part_g, st)) return e;
  { launch_ready(bn_bwd_finish_kernel, dim3(n_field), dim3(kFinishThreads), 0, st, part_a, part_g, rb, n, c, field_of_channel, scalar_of_channel, var, weight, eps,
                                                           training, ks, ka, kg, d_weight, d_bias); note_launches(1); }
  SSC_CHECK_LAUNCH("bn_bwd_finish");
  return launch_bwd<1>(p, ks, ka, kg, gx, nullptr, nullptr, st);
}

extern "C" int ssc_bn_bwd(const float *x, const float *gy, int n, int c, const int32_t *field_of_channel,
                          const int32_t *scalar_of_channel, int n_field, int n_scalar, const float *mean,
                          const float *var, const float *weight, float eps, int training, float *gx,
                          float *d_weight, float *d_bias, void *scratch, size_t scratch_bytes, void *stream) {
  SSC_REQUIRE(n >= 1 && c >= 1 && n_field >= 1 && n_scalar >= 0, "bn_bwd: bad sizes");
  SSC_REQUIRE(n_scalar == 0 || mean, "bn_bwd: null pointer");
  SSC_REQUIRE(scalar_of_channel && scratch && scratch_bytes >= ssc_bn_scratch_bytes(n, c), "bn_bwd: scratch too small (ssc_bn_scratch_bytes)");
  float *chan_mean = (float *)scratch + (size_t)2 * 8 * bn_row_blocks(n) * c + (size_t)3 * c;
  { launch_ready(bn_chan_mean_kernel, dim3(ceil_div(c, 128)), dim3(128), 0, as_stream(stream), mean, scalar_of_channel, c, chan_mean); note_launches(1); }
  SSC_CHECK_LAUNCH("bn_chan_mean");
  return ssc_bn_gate_bwd(x, gy, n, c, c, field_of_channel, scalar_of_channel, n_field, nullptr, nullptr, chan_mean, var, weight, eps, training,
                         nullptr, nullptr, nullptr, 0, 0, gx, d_weight, d_bias, scratch, scratch_bytes, stream);
}

extern "C" int ssc_gate_bwd(const float *x, const float *gy, int n, int c_total, int c_out,
                            const int32_t *gate_of_channel, const int32_t *field_start, const int32_t *field_len,
                            int scalar_act, int gate_act, float *gx, void *stream) {
  SSC_REQUIRE(n >= 0 && c_total >= 1 && c_out >= 1 && c_out <= c_total, "gate_bwd: bad sizes");
  if (n == 0) return SSC_OK;
  SSC_REQUIRE(x && gy && gx && gate_of_channel && (c_total == c_out || (field_start && field_len)), "gate_bwd: null pointer");
  BnGateBwd p = {x, gy, n, c_total, c_out, c_total - c_out, 0, 0, nullptr, nullptr, nullptr, gate_of_channel, field_start, field_len,
                 scalar_act, gate_act};
  return launch_bwd<1>(p, nullptr, nullptr, nullptr, gx, nullptr, nullptr, as_stream(stream));
}
