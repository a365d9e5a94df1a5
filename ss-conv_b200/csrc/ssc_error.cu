// Error reporting, identification and the read-back of device words.
#include <stdarg.h>
#include <deque>
#include <map>
#include <mutex>
#include <utility>
#include <vector>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "ssc_common.cuh"

namespace ssc {
unsigned long long launches();
char *error_buffer() {
  static thread_local char buf[512] = {0};
  return buf;
}
int fail(int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(error_buffer(), 512, fmt, ap);
  va_end(ap);
  return code;
}
static unsigned long long g_launches = 0;
void note_launches(int n) { __atomic_fetch_add(&g_launches, (unsigned long long)n, __ATOMIC_RELAXED); }
unsigned long long launches() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

// The limit is the kernel's, not the launch's, and calls of other sizes set it too: set by every call to what that call
// needs, one thread could take it away from another between its setting and its launch ("invalid argument", or "too many
// resources requested": four threads on one network, once in some thousand passes).  So it only ever grows.
cudaError_t allow_smem(const void *kernel, size_t bytes) {
  static std::mutex lock;
  static std::map<std::pair<int, const void *>, size_t> allowed;
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  std::lock_guard<std::mutex> hold(lock);
  size_t &have = allowed[{dev, kernel}];
  if (bytes <= have) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) have = bytes;
  else (void)cudaGetLastError();
  return e;
}

// Kernels that give up set this word too, besides their status word: row counts are posted to the host before the
// convolution behind them has run, so nothing that is read back tells of it in time.  Mapped host memory, kept
// for the life of the process (recorded graphs hold its address).
static int32_t *g_alarm = nullptr;
int32_t *alarm_word() { return __atomic_load_n(&g_alarm, __ATOMIC_ACQUIRE); }

// Read-back of a few device words.  What bounds it is latency: through a device-to-host copy and a stream
// synchronisation one word costs 20 - 25 us after the last kernel (staging of the pageable
// destination, copy engine start, completion interrupt path); a one-warp kernel that stores the
// words and then a sequence number into mapped host memory, watched by the host, costs 8 - 10 us.
constexpr int kReadMax = 31;
struct ReadList {
  const int32_t *word[kReadMax];
};
__global__ void read_words_kernel(ReadList list, int n, volatile int32_t *dst, int32_t seq) {
  const int lane = threadIdx.x;
  if (lane < n) dst[1 + lane] = *(const volatile int32_t *)list.word[lane];
  __threadfence_system();
  __syncwarp();
  if (lane == 0) dst[0] = seq;
}

namespace {
// One 128-byte mapped buffer per read in progress: taken from and given back to a list, so there are
// never more of them than threads that have read at the same time.
struct ReadSlot {
  int32_t *host;
  int32_t seq;
};
std::mutex g_slots_lock;
std::vector<ReadSlot> g_slots;

bool take_slot(ReadSlot &s) {
  {
    std::lock_guard<std::mutex> hold(g_slots_lock);
    if (!g_slots.empty()) {
      s = g_slots.back();
      g_slots.pop_back();
      return true;
    }
  }
  void *p = nullptr;
  if (cudaHostAlloc(&p, 128, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) return false;
  memset(p, 0, 128);
  s.host = (int32_t *)p;
  s.seq = 0;
  return true;
}
void give_slot(const ReadSlot &s) {
  std::lock_guard<std::mutex> hold(g_slots_lock);
  g_slots.push_back(s);
}

int read_some(const int32_t *const *words, int n, int32_t *out, cudaStream_t st) {
  ReadSlot s;
  if (!take_slot(s)) return fail(SSC_ERR_CUDA, "read_words: no mapped host memory: %s", cudaGetErrorString(cudaGetLastError()));
  ReadList list;
  for (int i = 0; i < n; ++i) list.word[i] = words[i];
  s.seq = s.seq == 0x7fffffff ? 1 : s.seq + 1;
  { read_words_kernel<<<1, 32, 0, st>>>(list, n, s.host, s.seq); note_launches(1); }
  cudaError_t e = cudaGetLastError();
  for (unsigned spin = 1; e == cudaSuccess && __atomic_load_n(s.host, __ATOMIC_ACQUIRE) != s.seq; ++spin) {
#if defined(__x86_64__)
    _mm_pause();
#endif
    if ((spin & 0x3ffu) == 0) {     // the stream's own state now and then: a launch that failed never writes
      e = cudaStreamQuery(st);
      if (e == cudaErrorNotReady) {
        (void)cudaGetLastError();
        e = cudaSuccess;
      } else if (e == cudaSuccess && __atomic_load_n(s.host, __ATOMIC_ACQUIRE) != s.seq) {
        e = cudaErrorUnknown;       // the stream is done and the number has not arrived
      }
    }
  }
  if (e != cudaSuccess) return fail(SSC_ERR_CUDA, "read_words: %s", cudaGetErrorString(e));   // the buffer stays out of the list
  for (int i = 0; i < n; ++i) out[i] = s.host[1 + i];
  give_slot(s);
  return SSC_OK;
}

// Places for posted counts.  A place that was given back may still be written by a kernel that nobody waited for: it is
// taken again only when its last number has arrived, the longest given back first.
struct CountPlace {
  int32_t *host;      // [number, status, count]
  int32_t seq;        // number of the last post
};
std::mutex g_places_lock;
std::deque<CountPlace *> g_places;
constexpr int kPlacesPerPage = 64;

bool arrived(const CountPlace *p) { return __atomic_load_n(p->host, __ATOMIC_ACQUIRE) == p->seq; }

__global__ void post_count_kernel(const int32_t *n_dev, const int32_t *status, CountPost post) {
  post_count(post, *n_dev, status);
}
}  // namespace

CountPost next_post(void *place) {
  CountPlace *p = (CountPlace *)place;
  if (p == nullptr) return {nullptr, 0};
  p->seq = p->seq == 0x7fffffff ? 1 : p->seq + 1;
  return {p->host, p->seq};
}

void launch_post(const CountPost &post, const int32_t *n_dev, const int32_t *status, cudaStream_t st) {
  if (post.host == nullptr) return;
  post_count_kernel<<<1, 1, 0, st>>>(n_dev, status, post);
  note_launches(1);
}
}  // namespace ssc

extern "C" void *ssc_count_open(void) {
  using namespace ssc;
  std::lock_guard<std::mutex> hold(g_places_lock);
  for (size_t tries = g_places.size() < 4 ? g_places.size() : 4; tries > 0; --tries) {
    CountPlace *p = g_places.front();
    g_places.pop_front();
    if (arrived(p)) return p;
    g_places.push_back(p);
  }
  char *page = nullptr;
  if (cudaHostAlloc((void **)&page, kPlacesPerPage * 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  memset(page, 0, kPlacesPerPage * 64);
  for (int i = 0; i < kPlacesPerPage; ++i) g_places.push_front(new CountPlace{(int32_t *)(page + 64 * i), 0});
  CountPlace *p = g_places.front();
  g_places.pop_front();
  return p;
}

extern "C" int ssc_count_wait(void *place, int *out, void *stream) {
  using namespace ssc;
  SSC_REQUIRE(place && out, "count_wait: null pointer");
  const CountPlace *p = (const CountPlace *)place;
  out[0] = out[1] = out[2] = 0;
  for (unsigned spin = 1; !arrived(p); ++spin) {
#if defined(__x86_64__)
    _mm_pause();
#endif
    if ((spin & 0x3ffu) != 0) continue;
    const cudaError_t e = cudaStreamQuery(as_stream(stream));
    if (e == cudaErrorNotReady) {
      (void)cudaGetLastError();
    } else if (e != cudaSuccess) {
      return fail(SSC_ERR_CUDA, "count_wait: %s", cudaGetErrorString(e));
    } else if (!arrived(p)) {
      return SSC_OK;
    }
  }
  out[0] = p->host[2];
  out[1] = p->host[1];
  out[2] = 1;
  return SSC_OK;
}

extern "C" int ssc_count_post(const int32_t *n_dev, const int32_t *status, void *place, void *stream) {
  SSC_REQUIRE(n_dev && place, "count_post: null pointer");
  ssc::launch_post(ssc::next_post(place), n_dev, status, ssc::as_stream(stream));
  SSC_CHECK_LAUNCH("count_post");
  return SSC_OK;
}

extern "C" int ssc_count_close(void *place) {
  SSC_REQUIRE(place, "count_close: null pointer");
  std::lock_guard<std::mutex> hold(ssc::g_places_lock);
  ssc::g_places.push_back((ssc::CountPlace *)place);
  return SSC_OK;
}

extern "C" int ssc_read_words(const int32_t *const *words, int n, int32_t *out, void *stream) {
  SSC_REQUIRE(n >= 0 && (n == 0 || (words && out)), "read_words: bad arguments");
  for (int i = 0; i < n; i += ssc::kReadMax) {
    const int m = n - i < ssc::kReadMax ? n - i : ssc::kReadMax;
    for (int k = 0; k < m; ++k) SSC_REQUIRE(words[i + k], "read_words: null pointer");
    if (int e = ssc::read_some(words + i, m, out + i, ssc::as_stream(stream))) return e;
  }
  return SSC_OK;
}

extern "C" int32_t *ssc_alarm_open(void) {
  using namespace ssc;
  std::lock_guard<std::mutex> hold(g_places_lock);
  if (alarm_word() == nullptr) {
    void *p = nullptr;
    if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    memset(p, 0, 64);
    __atomic_store_n(&g_alarm, (int32_t *)p, __ATOMIC_RELEASE);
  }
  return alarm_word();
}

extern "C" int ssc_version(void) { return 100; }
extern "C" const char *ssc_last_error(void) { return ssc::error_buffer(); }
extern "C" int ssc_has_tcgen05(void) { return 1; }
extern "C" unsigned long long ssc_kernel_launches(void) { return ssc::launches(); }
