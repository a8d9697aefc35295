// Library-wide plumbing of the C ABI: version, per-thread error text, device facts.
#include <atomic>
#include <mutex>

#include "common.cuh"

namespace anima {

namespace {
thread_local char g_error[512] = "";
std::atomic<int64_t> g_launches{0};
}

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

int sm_count() {
  static int cached[64];
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

}  // namespace anima

extern "C" int anima_abi_version(void) { return ANIMA_ABI_VERSION; }
extern "C" const char* anima_last_error(void) { return anima::g_error; }

extern "C" int64_t anima_kernel_launches(void) { return anima::g_launches.load(std::memory_order_relaxed); }
