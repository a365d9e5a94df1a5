// The way out of the output-stationary convolution kernels: accumulators of a tile's 128 rows (tensor memory, a
// lane per row) to rows in global memory, optionally through a folded batch norm and the gated activation.
// Four warps have 32 rows each (a quarter of the tile).  `load(q, c0)` asks for sixteen columns of the warp's rows from
// column c0; the wait for them is here.  32 columns at a time go through the warp's 4 KB of shared memory (`blk`), so
// that eight lanes write the 128 contiguous bytes of a row.
#pragma once
#include "ssc_act.cuh"
#include "ssc_conv_internal.cuh"
#include "ssc_tc_ptx.cuh"

namespace ssc {

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Scale, shift and gate (of kept channels; -2: of none) of channel ch.
__device__ __forceinline__ float4 gate_channel(const GateEpilogue &gate, int ch) {
  const bool bn = gate.scale != nullptr;
  return make_float4(bn ? __ldg(gate.scale + ch) : 0.f, bn ? __ldg(gate.shift + ch) : 0.f,
                     __int_as_float(ch < gate.c_keep ? __ldg(gate.gate_of_channel + ch) : -2), 0.f);
}

// act(gate g) of row `lane` to gates[g * 33 + lane], from the sixteen columns at first, first + step, ...
// Eight side by side (one after the other they are all latency), and only eights that hold a gate: sixteen at a time
// evaluated ten sigmoids for nothing at 32 -> 38 channels (121 k rows: 48.0 -> 46.3 us).
template <class Load>
__device__ __forceinline__ void gate_scalars(Load load, const GateEpilogue &gate, const float4 *chan, float *gates, int c_out, int lane, int first, int step) {
  for (int c0 = first; c0 < c_out; c0 += step) {
    uint32_t q[16];
    load(q, c0);
    tmem_wait_ld();
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      if (c0 + h + 8 <= gate.c_keep || c0 + h >= c_out) continue;
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 k = chan[c0 + h + i < c_out ? c0 + h + i : 0];
        v[i] = __uint_as_float(q[h + i]);
        if (gate.scale) v[i] = fmaf(v[i], k.x, k.y);
      }
      if (gate.gate_act == 2) {
        apply_sigmoids<8>(v);
      } else if (gate.gate_act == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = apply_act(v[i], 1);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + h + i >= gate.c_keep && c0 + h + i < c_out) gates[(c0 + h + i - gate.c_keep) * 33 + lane] = v[i];
    }
  }
}

// 32 words of row `lane` each as pieces of a 32 x 32 block: piece q of a row at place q ^ (lane & 7), so that both
// directions touch every bank once per phase.
__device__ __forceinline__ void block_from_columns(float *blk, const uint32_t *r, int lane) {
#pragma unroll
  for (int q = 0; q < 8; ++q) *(uint4 *)(blk + lane * 32 + ((q ^ (lane & 7)) << 2)) = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
}

// Finished rows, 32 columns at first, first + step, ...  gates: of this quarter, and a last line of ones.  row0: the quarter's
// first row; whole: the tile is full, in its own order and its rows are stored as vectors; else m: this lane's row of `out`, -1 for none.
// The columns that hold scalars, nearly always the first 32, go the same way as the others with a relu on top: by the general way, one
// pair of rows after the other, they took 4600 cycles of a tile's way out and now take 1000.
template <class Load>
__device__ __forceinline__ void store_gated(Load load, const GateEpilogue &gate, const float4 *chan, const float *gates, float *blk, float *out, int c_out, int row0, int m,
                                            bool whole, bool vec, int lane, int first, int step) {
  const int c_row = gate.c_keep, n_gates = c_out - c_row;
  const bool affine = gate.scale != nullptr;
  for (int c0 = first; c0 < c_row; c0 += step) {
    uint32_t r[32];
    load(r, c0);
    load(r + 16, c0 + 16);
    tmem_wait_ld();
    __syncwarp();
    block_from_columns(blk, r, lane);
    __syncwarp();
    const int q = lane & 7, row4 = lane >> 3, col = c0 + 4 * q;
    float sc[4], sh[4];
    const float *gp[4];
    bool scalar[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 k = chan[col + j < c_out ? col + j : 0];
      const int g = __float_as_int(k.z);
      sc[j] = k.x;
      sh[j] = k.y;
      scalar[j] = g == -1;
      gp[j] = gates + (g >= 0 ? g : n_gates) * 33 + row4;
    }
    const bool scalars = gate.scalar_act != 0 && __any_sync(0xffffffffu, scalar[0] || scalar[1] || scalar[2] || scalar[3]);
    // rows 4 i + row4 of the warp's 32: the swizzle of even and odd i, the rest are constants
    const float *even = blk + row4 * 32 + ((q ^ row4) << 2), *odd = blk + row4 * 32 + ((q ^ row4 ^ 4) << 2);
    auto finished = [&](int i, int act) {         // act: 0 no scalar among the columns, 1 relu, 2 whatever it is
      const float4 x = *(const float4 *)((i & 1 ? odd : even) + i * 128);
      float v[4] = {x.x, x.y, x.z, x.w};
      if (affine) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = fmaf(v[j], sc[j], sh[j]);
      }
      if (act == 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = scalar[j] && !(v[j] > 0.f) ? 0.f : v[j];
      } else if (act == 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (scalar[j]) v[j] = apply_act(v[j], gate.scalar_act);
      }
      return make_float4(v[0] * gp[0][4 * i], v[1] * gp[1][4 * i], v[2] * gp[2][4 * i], v[3] * gp[3][4 * i]);
    };
    auto packed = [&](float4 v) {
      return gate.out16 == 2 ? make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w)) : make_uint2(pack_f16x2(v.x, v.y), pack_f16x2(v.z, v.w));
    };
    if (whole && (!scalars || gate.scalar_act == 1)) {   // most tiles
      if (col >= c_row) continue;
      const size_t at = (size_t)(row0 + row4) * c_row + col;
      if (gate.out16 == 0) {
        float *to = out + at;
        if (!scalars) {
#pragma unroll
          for (int i = 0; i < 8; ++i, to += 4 * c_row) *(float4 *)to = finished(i, 0);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i, to += 4 * c_row) *(float4 *)to = finished(i, 1);
        }
      } else {
        uint16_t *to = (uint16_t *)out + at;
        if (!scalars) {
#pragma unroll
          for (int i = 0; i < 8; ++i, to += 4 * c_row) *(uint2 *)to = packed(finished(i, 0));
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i, to += 4 * c_row) *(uint2 *)to = packed(finished(i, 1));
        }
      }
    } else {
#pragma unroll 2
      for (int i = 0; i < 8; ++i) {
        const int to = __shfl_sync(0xffffffffu, m, 4 * i + row4);
        if (to < 0 || col >= c_row) continue;
        const float4 v = finished(i, scalars ? 2 : 0);
        const size_t at = (size_t)to * c_row + col;
        if (gate.out16 != 0) {                    // c_row is a multiple of eight
          *(uint2 *)((uint16_t *)out + at) = packed(v);
        } else if (vec) {
          *(float4 *)(out + at) = v;
        } else {
          const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col + j < c_row) out[at + j] = e[j];
        }
      }
    }
  }
}

// The rows as they are: of the tile's n_cols columns, 32 at first, first + step, ... as channels col0 + ... of rows of c_row.
// m: this lane's row of `out`, -1 for none.
template <class Load>
__device__ __forceinline__ void store_plain(Load load, float *blk, float *out, int m, int col0, int n_cols, int c_row, bool vec, int lane, int first, int step) {
  for (int c0 = first; c0 < n_cols && col0 + c0 < c_row; c0 += step) {
    uint32_t r[32];
    load(r, c0);
    load(r + 16, c0 + 16);
    tmem_wait_ld();
    if (vec) {
      __syncwarp();
      block_from_columns(blk, r, lane);
      __syncwarp();
      const int q = lane & 7, col = col0 + c0 + 4 * q;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = 4 * i + (lane >> 3);
        const int to = __shfl_sync(0xffffffffu, m, row);
        if (to >= 0 && col < c_row && c0 + 4 * q < n_cols)
          *(uint4 *)(out + (size_t)to * c_row + col) = *(const uint4 *)(blk + row * 32 + ((q ^ (row & 7)) << 2));
      }
    } else if (m >= 0) {
      float *op = out + (size_t)m * c_row + col0 + c0;
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (col0 + c0 + q < c_row && c0 + q < n_cols) op[q] = __uint_as_float(r[q]);
    }
  }
}

}  // namespace ssc
