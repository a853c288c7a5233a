// Library-wide state: the last error message and a version word for the bindings.
#include "common.cuh"

#include <pthread.h>
#include <stdlib.h>

namespace ms {
static thread_local char g_error[512] = "";
char* error_buffer() { return g_error; }

static int g_dependent_launch = -1;
bool dependent_launch_enabled() {
  if (g_dependent_launch < 0) {
    const char* value = getenv("MINISERVE_B200_DEPENDENT_LAUNCH");
    g_dependent_launch = (value != nullptr && value[0] == '0') ? 0 : 1;
  }
  return g_dependent_launch == 1;
}

// (kernel, device) and the bytes it may have, by open addressing; nothing in it throws.  Beyond its size the driver is asked each time.
struct Allowed { const void* kernel; int device; size_t bytes; };
constexpr int kAllowed = 512;
static Allowed g_allowed[kAllowed];
static pthread_mutex_t g_allowed_lock = PTHREAD_MUTEX_INITIALIZER;

cudaError_t allow_shared_bytes(const void* kernel, size_t bytes) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  pthread_mutex_lock(&g_allowed_lock);
  Allowed* entry = nullptr;
  const size_t at = reinterpret_cast<size_t>(kernel) / 16 + (size_t)device;
  for (int i = 0; i < kAllowed && entry == nullptr; ++i) {
    Allowed* here = &g_allowed[(at + i) % kAllowed];
    if (here->kernel == nullptr || (here->kernel == kernel && here->device == device)) entry = here;
  }
  if (entry == nullptr || entry->kernel == nullptr || entry->bytes < bytes) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && entry != nullptr) *entry = Allowed{kernel, device, bytes};
  }
  pthread_mutex_unlock(&g_allowed_lock);
  return e;
}
}  // namespace ms

MS_EXPORT const char* ms_last_error() { return ms::error_buffer(); }

// Bumped whenever an exported signature changes; the bindings refuse a library that
// reports another number.
MS_EXPORT int ms_abi_version() { return 15; }

// 1: kernels are launched as programmatic dependents (default); 0: plain stream order.
MS_EXPORT void ms_set_dependent_launch(int enabled) { ms::g_dependent_launch = enabled ? 1 : 0; }
