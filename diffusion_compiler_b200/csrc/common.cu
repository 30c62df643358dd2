// Host-side helpers shared by the difb200 entry points: error text, CUDA status mapping,
// the per-device status words that kernels with bounded waits report through.
#include "common.cuh"

#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <unordered_map>
#include <utility>

namespace difb200 {

namespace {
thread_local std::string g_last_error;
std::mutex g_mutex;
std::unordered_map<int, DeviceStatus *> g_status_words;
std::unordered_map<int, int> g_sm_counts;
std::mutex g_once_mutex;
std::map<std::pair<const void *, int>, int> g_once_values;
} // namespace

namespace {
std::atomic<unsigned long long> g_wait_limit_ns{1500ull * 1000ull * 1000ull};
std::atomic<uint32_t> g_withhold_kb{0xffffffffu};
std::atomic<unsigned long long> g_withheld_maximum_ns{0};
} // namespace

unsigned long long wait_limit_ns() { return g_wait_limit_ns.load(); }
void set_wait_limit_ns(unsigned long long ns) { g_wait_limit_ns.store(ns ? ns : 1500ull * 1000ull * 1000ull); }
void withhold_next_gemm_load(uint32_t k_block) { g_withhold_kb.store(k_block); }
bool gemm_load_is_withheld() { return g_withhold_kb.load() != 0xffffffffu; }
void withhold_next_row_maximum(unsigned long long limit_ns) { g_withheld_maximum_ns.store(limit_ns); }
unsigned long long take_withheld_row_maximum() { return g_withheld_maximum_ns.exchange(0); }
uint32_t take_withheld_gemm_load() { return g_withhold_kb.exchange(0xffffffffu); }

int per_device_once(const void *key, int device, int (*init)(void *arg, int *value), void *arg, int *value) {
  std::lock_guard<std::mutex> lock(g_once_mutex);
  const auto it = g_once_values.find({key, device});
  if (it != g_once_values.end()) {
    if (value)
      *value = it->second;
    return kOk;
  }
  int v = 0;
  if (int rc = init(arg, &v))
    return rc;
  g_once_values[{key, device}] = v;
  if (value)
    *value = v;
  return kOk;
}

int current_device_once(const void *key, int (*init)(void *arg, int *value), void *arg, int *value) {
  int device = 0;
  if (int rc = check_cuda(cudaGetDevice(&device), "cudaGetDevice"))
    return rc;
  return per_device_once(key, device, init, arg, value);
}

int resident_blocks(const void *kernel, int threads, size_t dynamic_smem, int *blocks) {
  struct Key {
    const void *kernel;
    int device, threads;
    size_t smem;
    bool operator<(const Key &o) const {
      return std::tie(kernel, device, threads, smem) < std::tie(o.kernel, o.device, o.threads, o.smem);
    }
  };
  static std::map<Key, int> known;
  static std::map<std::pair<const void *, int>, size_t> opted_in; // the limit is per function: it only grows
  Key key{kernel, 0, threads, dynamic_smem};
  if (int rc = check_cuda(cudaGetDevice(&key.device), "cudaGetDevice"))
    return rc;
  std::lock_guard<std::mutex> lock(g_once_mutex);
  const auto it = known.find(key);
  if (it != known.end()) {
    *blocks = it->second;
    return kOk;
  }
  size_t &limit = opted_in[{kernel, key.device}];
  if (dynamic_smem > 48 * 1024 && dynamic_smem > limit) {
    if (int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dynamic_smem),
                            "cudaFuncSetAttribute(dynamic shared memory)"))
      return rc;
    limit = dynamic_smem;
  }
  int n = 0;
  if (int rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, dynamic_smem), "occupancy"))
    return rc;
  known[key] = *blocks = n < 1 ? 1 : n;
  return kOk;
}

void set_last_error(const std::string &text) { g_last_error = text; }
const std::string &last_error() { return g_last_error; }

int fail(int status, const std::string &text) {
  g_last_error = text;
  return status;
}

int check_cuda(cudaError_t code, const char *what) {
  if (code == cudaSuccess)
    return kOk;
  std::string text = std::string(what) + ": " + cudaGetErrorName(code) + " (" +
                     cudaGetErrorString(code) + ")";
  return fail(code == cudaErrorMemoryAllocation ? kOutOfMemory : kExecutionError, text);
}

namespace {
std::atomic<unsigned long long> g_launches{0};
}
int launched(cudaError_t code, const char *what) {
  if (code == cudaSuccess)
    g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_cuda(code, what);
}
unsigned long long launch_count() { return g_launches.load(); }

int sm_count() {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess)
    return 148;
  std::lock_guard<std::mutex> lock(g_mutex);
  auto it = g_sm_counts.find(device);
  if (it != g_sm_counts.end())
    return it->second;
  int count = 148;
  cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device);
  g_sm_counts[device] = count;
  return count;
}

int StreamScratch::allocate(size_t bytes, const char *what) {
  static std::unordered_map<int, cudaMemPool_t> pools;
  int device = 0;
  if (int rc = check_cuda(cudaGetDevice(&device), what))
    return rc;
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    const auto it = pools.find(device);
    if (it != pools.end()) {
      pool = it->second;
    } else {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device;
      if (int rc = check_cuda(cudaMemPoolCreate(&pool, &props), what))
        return rc;
      unsigned long long kept = 4ull << 20; // the statistics of half a million rows
      if (int rc = check_cuda(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept), what)) {
        cudaMemPoolDestroy(pool);
        return rc;
      }
      pools[device] = pool;
    }
  }
  return check_cuda(cudaMallocFromPoolAsync(&data_, bytes, pool, stream_), what);
}

StreamScratch::~StreamScratch() {
  if (data_)
    cudaFreeAsync(data_, stream_);
}

namespace {
// Zero from the start, and there with the device's copy of this code: a call that first needs the words allocates nothing, waits for
// nothing, and may stand beside a stream capture (of its own stream or of another thread).
__device__ DeviceStatus g_status_storage;
} // namespace

DeviceStatus *device_status_words() {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess)
    return nullptr;
  std::lock_guard<std::mutex> lock(g_mutex);
  auto it = g_status_words.find(device);
  if (it != g_status_words.end())
    return it->second;
  void *words = nullptr;
  if (cudaGetSymbolAddress(&words, g_status_storage) != cudaSuccess) {
    cudaGetLastError(); // the caller reports it; a later launch must not
    return nullptr;
  }
  return g_status_words[device] = static_cast<DeviceStatus *>(words);
}

int poll_device_status(const char *what) {
  DeviceStatus *words = device_status_words();
  if (!words)
    return fail(kInternalError, "device status words are unavailable");
  DeviceStatus host{};
  if (int rc = check_cuda(cudaMemcpy(&host, words, sizeof(host), cudaMemcpyDeviceToHost), what))
    return rc;
  if (host.flag == 0)
    return kOk;
  cudaMemset(words, 0, sizeof(DeviceStatus));
  return fail(kExecutionError, std::string(what) + ": a bounded device-side wait ran out (kernel " +
                                   std::to_string(host.kernel) + ", role " + std::to_string(host.role) +
                                   ", detail " + std::to_string(host.detail) + ")");
}

} // namespace difb200
