// Library-wide pieces of the C ABI: error text, version, device properties, status words.
#include "common.cuh"

#include <atomic>
#include <mutex>

namespace b200 {

char* last_error_buffer() {
  static thread_local char buf[512] = {0};
  return buf;
}

const DeviceInfo& device_info() {
  static DeviceInfo info[64];
  static bool have[64] = {false};
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!have[dev]) {
    DeviceInfo d;
    d.sm_count = 148;
    d.max_smem_optin = 48 * 1024;
    d.l2_bytes = 0;
    cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&d.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&d.l2_bytes, cudaDevAttrL2CacheSize, dev);
    info[dev] = d;
    have[dev] = true;
  }
  return info[dev];
}

cudaError_t set_function_attribute_once(const void* kernel, cudaFuncAttribute attr, int value) {
  struct Entry { const void* kernel; int attr, device; };
  static Entry done[512];
  static int used = 0;
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < used; ++i)
    if (done[i].kernel == kernel && done[i].attr == (int)attr && done[i].device == dev) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, attr, value);
  // a full table only means that the same value is set again
  if (e == cudaSuccess && used < 512) done[used++] = Entry{kernel, (int)attr, dev};
  return e;
}

cudaError_t allow_dynamic_smem(const void* kernel, size_t bytes) {
  struct Entry { const void* kernel; int device; size_t limit; };
  static Entry done[256];
  static int used = 0;
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < used; ++i)
    if (done[i].kernel == kernel && done[i].device == dev) return bytes <= done[i].limit ? cudaSuccess : cudaErrorInvalidValue;
  cudaFuncAttributes attr;
  e = cudaFuncGetAttributes(&attr, kernel);
  if (e != cudaSuccess) return e;
  const size_t optin = (size_t)device_info().max_smem_optin;
  const size_t limit = optin > attr.sharedSizeBytes ? optin - attr.sharedSizeBytes : 0;
  if (bytes > limit) return cudaErrorInvalidValue;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
  if (e == cudaSuccess && used < 256) done[used++] = Entry{kernel, dev, limit};
  return e;
}

static std::mutex& launch_order(cudaStream_t st) {
  static std::mutex mutexes[64];
  uintptr_t key = reinterpret_cast<uintptr_t>(st);
  if (st == nullptr || st == cudaStreamLegacy) {  // one stream per device under two names
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    key = (uintptr_t)dev << 4;
  }
  return mutexes[((key >> 4) * 0x9e3779b97f4a7c15ull) >> 58];
}

LaunchesTogether::LaunchesTogether(cudaStream_t st) : held_(&launch_order(st)) { static_cast<std::mutex*>(held_)->lock(); }
LaunchesTogether::~LaunchesTogether() { static_cast<std::mutex*>(held_)->unlock(); }

int cached_occupancy(const void* fn, int threads, size_t smem) {
  struct Entry { const void* fn; int threads, device; size_t smem; int blocks; };
  static Entry cache[256];
  static int used = 0;
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < used; ++i)
    if (cache[i].fn == fn && cache[i].threads == threads && cache[i].smem == smem && cache[i].device == dev)
      return cache[i].blocks;
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    blocks = 1;
  }
  if (blocks < 1) blocks = 1;
  if (used < 256) cache[used++] = Entry{fn, threads, dev, smem, blocks};
  return blocks;
}

static std::atomic<long long> g_launches{0};
static thread_local const char* t_path_tag = nullptr;
static thread_local char t_last_kernel[160] = {0};

void set_path_tag(const char* tag) { t_path_tag = tag; }

void note_launch(const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (t_path_tag)
    snprintf(t_last_kernel, sizeof(t_last_kernel), "%s [%s]", what, t_path_tag);
  else
    snprintf(t_last_kernel, sizeof(t_last_kernel), "%s", what);
  t_path_tag = nullptr;
}

}  // namespace b200

// Number of kernels this library has launched in this process so far.
extern "C" int64_t b200_launch_count(void) { return b200::g_launches.load(std::memory_order_relaxed); }

// Name of the kernel this thread launched last, with the variant the launcher chose in brackets
// (e.g. "b200_row_reduce [vector, warp per row]"); "" before the first launch. A diagnostic: sweep
// reports use it to tell tuned paths from the element-wise ones.
extern "C" const char* b200_last_kernel(void) { return b200::t_last_kernel; }

extern "C" const char* b200_last_error(void) { return b200::last_error_buffer(); }

extern "C" int b200_version(void) { return 1; }

extern "C" int b200_sm_count(void) { return b200::device_info().sm_count; }

extern "C" int b200_l2_bytes(void) { return b200::device_info().l2_bytes; }

// Reads the status words of a scratch buffer used by the norm backward (BwdWords in norm_bwd.cuh).
// Synchronises the stream: a diagnostic call, never part of a timed or captured region.
extern "C" int b200_check_status(const void* scratch, void* stream) {
  if (!scratch) return b200::fail(B200_ERR_INVALID, "b200_check_status: null scratch");
  unsigned int words[4] = {0, 0, 0, 0};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(words, scratch, sizeof(words), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return b200::fail((int)e, "b200_check_status: %s", cudaGetErrorString(e));
  if (words[1] != 0)
    return b200::fail(B200_ERR_DEVICE_WAIT,
                      "a bounded wait ran out in a norm backward: its column sums were not formed (arrivals=%u)", words[0]);
  return B200_OK;
}
