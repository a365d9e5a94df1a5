// Shared host/device helpers for the ssconv_b200 library (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../../include/ssconv_b200.h"

namespace ssc {

// Per-thread error message behind ssc_last_error().
char *error_buffer();
int fail(int code, const char *fmt, ...);

// Kernel-launch bookkeeping behind ssc_kernel_launches().
void note_launches(int n);

// Lets a kernel have `bytes` of dynamic shared memory on the current device, for this launch and all others.
cudaError_t allow_smem(const void *kernel, size_t bytes);

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

#define SSC_CHECK_LAUNCH(name)                                                     \
  do {                                                                             \
    cudaError_t e__ = cudaGetLastError();                                          \
    if (e__ != cudaSuccess)                                                        \
      return ssc::fail(SSC_ERR_CUDA, "%s: %s", name, cudaGetErrorString(e__));     \
  } while (0)

#define SSC_REQUIRE(cond, ...)                                                     \
  do {                                                                             \
    if (!(cond)) return ssc::fail(SSC_ERR_INVALID, __VA_ARGS__);                   \
  } while (0)

// Number of valid rows of a launch whose row count may still be on the device: `cap` is the
// host-side bound (and the row stride of the tables), `n_dev` (may be null) the exact count.
__device__ __forceinline__ int live_rows(int cap, const int32_t *n_dev) {
  if (n_dev == nullptr) return cap;
  const int v = *n_dev;
  return v < 0 ? 0 : (v < cap ? v : cap);
}

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }
inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// 3-D geometry of one rulebook request, passed by value to kernels.
struct Geometry {
  int in_shape[3];
  int out_shape[3];
  int ksize[3];
  int stride[3];
  int padding[3];
  int dilation[3];
  int K;
  int transpose;
};

// ----------------------------------------------------------------------------------
// Coordinate hash: open addressing over 4-slot buckets (one 32-byte sector per probe).
// A slot packs (key << 32 | row); the all-ones word marks an empty slot.
// ----------------------------------------------------------------------------------
constexpr unsigned long long kEmptySlot = 0xFFFFFFFFFFFFFFFFull;
constexpr int kBucketSlots = 4;

__host__ __device__ inline uint32_t hash_mix(uint32_t k) {
  k ^= k >> 16;
  k *= 0x85ebca6bu;
  k ^= k >> 13;
  k *= 0xc2b2ae35u;
  k ^= k >> 16;
  return k;
}

inline uint32_t hash_buckets_for(int n) {
  // load factor <= 0.5 over 4-slot buckets, power of two, at least 64 buckets
  uint32_t want = (uint32_t)((2ll * (n > 0 ? n : 1) + kBucketSlots - 1) / kBucketSlots);
  uint32_t b = 64;
  while (b < want) b <<= 1;
  return b;
}

int bitmap_decode(const uint32_t *bitmap, const uint32_t *word_prefix, long long n_words, const int shape[3],
                  int n_out, int32_t *out_indices, cudaStream_t st);

// SMs of the current device (ssc_conv_stage.cu).
int sm_count();

// The process's alarm (ssc_alarm_open), null while nobody has opened it.
int32_t *alarm_word();

// A count for the host (ssc_count_open): status word and count, then the number the host watches for.
struct CountPost {
  int32_t *host;        // null: nobody asked
  int32_t seq;
};
CountPost next_post(void *place);
void launch_post(const CountPost &post, const int32_t *n_dev, const int32_t *status, cudaStream_t st);

#ifdef __CUDACC__
// Two floats in a register pair; operations on both halves at once, each correctly rounded.
typedef unsigned long long f32x2;
static __device__ __forceinline__ f32x2 pair_of(float lo, float hi) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
static __device__ __forceinline__ float2 halves(f32x2 v) {
  float2 h;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(h.x), "=f"(h.y) : "l"(v));
  return h;
}
static __device__ __forceinline__ f32x2 fma_pair(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
static __device__ __forceinline__ f32x2 mul_pair(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
static __device__ __forceinline__ f32x2 add_pair(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// (one thread) a bounded wait ran out and the output is incomplete: status bit 16, then the alarm, which the host sees
// without reading anything back.
static __device__ __forceinline__ void report_expired(int32_t *status, int32_t *alarm) {
  if (status != nullptr) atomicOr(status, 16);
  if (alarm != nullptr) {
    __threadfence_system();
    *(volatile int32_t *)alarm = 16;
  }
}

static __device__ __forceinline__ void post_count(const CountPost &post, int32_t count, const int32_t *status) {
  volatile int32_t *dst = post.host;
  dst[1] = status != nullptr ? *(const volatile int32_t *)status : 0;
  dst[2] = count;
  __threadfence_system();
  dst[0] = post.seq;
}
#endif

// A launch that is made ready while the kernel before it in the stream still runs, for kernels that begin with
// after_previous(): behind it everything before in the stream is complete and visible, so the order is that of any
// other launch.  What is saved is the gap of one to two microseconds between the end of one kernel and the first
// instruction of the next (the arguments, the first fetch of the code), which at these calls is a tenth of the time: a
// chain of small kernels is most of them (plain-12 network, eval 1220 -> 1142 us, strided layer with a pool 220 -> 204, voxel
// codec 230 -> 214).  Blocks are placed once all blocks of the kernel before have ended.  No kernel lets them in earlier
// (griddepcontrol.launch_dependents): they took the room that was free first, two to an SM here and none there, and waited
// in it, and the instruction itself is dear where a block does little (us without it, with it, and of an ordinary launch:
// gradients of 10 k rows of 250 normed channels 35.4, 46.5, 36.2; max pool over 27 offsets, 20 k rows of 76 15.7, 20.8, 16.0;
// filter gradient of 300 rows 32 -> 38 12.6, 16.3, 14.2; transpose of a table of 27 offsets, 700 k rows 29.6, 54.8, 29.6).
template <class T>
struct AsIs { using type = T; };      // (keeps a parameter out of the deduction: arguments convert to the kernel's types as in a call)
template <class... P>
inline cudaError_t launch_ready(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, typename AsIs<P>::type... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace ssc
