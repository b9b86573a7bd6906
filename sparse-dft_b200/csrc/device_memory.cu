// Stream-ordered device memory from one library pool per device, and the
// kernels' shared-memory limits.
#include <cstdint>
#include <map>
#include <mutex>
#include <shared_mutex>
#include <tuple>
#include <utility>

#include "common.cuh"

namespace sdft_b200 {

namespace {

constexpr int kMaxDevices = 64;
std::once_flag pool_once[kMaxDevices];
cudaMemPool_t pools[kMaxDevices] = {};

cudaMemPool_t current_pool() {
  int device = 0;
  SDFT_CUDA(cudaGetDevice(&device));
  if (device < 0 || device >= kMaxDevices) throw CudaError("device ordinal outside the library's pool table");
  std::call_once(pool_once[device], [device] {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    SDFT_CUDA(cudaMemPoolCreate(&pool, &props));
    // Freed blocks stay in the pool (no release at synchronisation points),
    // so a released buffer's memory serves the next allocation on any stream
    // of this device without mapping new memory.
    std::uint64_t keep = UINT64_MAX;
    SDFT_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    pools[device] = pool;
  });
  return pools[device];
}

}  // namespace

void* stream_alloc(std::size_t bytes, cudaStream_t stream) {
  void* ptr = nullptr;
  SDFT_CUDA(cudaMallocFromPoolAsync(&ptr, std::max<std::size_t>(bytes, 1), current_pool(), stream));
  return ptr;
}

void stream_free(void* ptr, cudaStream_t stream) {
  if (ptr) cudaFreeAsync(ptr, stream);
}

void trim_pool() {
  SDFT_CUDA(cudaMemPoolTrimTo(current_pool(), 0));
}

// The attribute and occupancy calls take a lock of the driver that every launch in
// the process waits for: with the shared-memory attribute set at each launch, four
// solves on four threads queued behind one another (four 8-atom k-points 102 ms; 62
// ms with that call made once per kernel and device). A single thread's launches cost the same either way.
std::size_t dynamic_smem_limit(const void* kernel) {
  static std::shared_mutex mutex;
  static std::map<std::pair<int, const void*>, std::size_t> limits;
  int device = 0;
  SDFT_CUDA(cudaGetDevice(&device));
  const std::pair<int, const void*> key{device, kernel};
  {
    std::shared_lock<std::shared_mutex> lock(mutex);
    const auto found = limits.find(key);
    if (found != limits.end()) return found->second;
  }
  cudaFuncAttributes attributes;
  SDFT_CUDA(cudaFuncGetAttributes(&attributes, kernel));
  const std::size_t limit = kMaxDynamicSmem - std::min(kMaxDynamicSmem, attributes.sharedSizeBytes);
  SDFT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit)));
  std::unique_lock<std::shared_mutex> lock(mutex);
  limits[key] = limit;
  return limit;
}

long long resident_blocks(const void* kernel, int threads, std::size_t smem) {
  static std::shared_mutex mutex;
  static std::map<std::tuple<int, const void*, int, std::size_t>, long long> counts;
  int device = 0;
  SDFT_CUDA(cudaGetDevice(&device));
  const std::tuple<int, const void*, int, std::size_t> key{device, kernel, threads, smem};
  {
    std::shared_lock<std::shared_mutex> lock(mutex);
    const auto found = counts.find(key);
    if (found != counts.end()) return found->second;
  }
  int per_sm = 0, sms = 0;
  SDFT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  SDFT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const long long count = static_cast<long long>(std::max(per_sm, 1)) * sms;
  std::unique_lock<std::shared_mutex> lock(mutex);
  counts[key] = count;
  return count;
}

}  // namespace sdft_b200
