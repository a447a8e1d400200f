// gb_common.cu -- host side of the shared infrastructure: the library's
// stream-ordered scratch pool and cached device properties.
#include <mutex>
#include <new>

#include "gb_common.cuh"

namespace gb {

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mutex;
cudaMemPool_t g_pools[kMaxDevices] = {};
int g_sm_count[kMaxDevices] = {};

cudaError_t pool_for_current_device(cudaMemPool_t* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool;
    e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    // Keep freed blocks cached in the pool instead of returning them to the
    // driver at every synchronisation: scratch is small and reused per call.
    uint64_t threshold = ~0ull;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold);
    if (e != cudaSuccess) return e;
    g_pools[dev] = pool;
  }
  *out = g_pools[dev];
  return cudaSuccess;
}
}  // namespace

cudaError_t scratch_alloc(void** ptr, size_t bytes, cudaStream_t stream) {
  cudaMemPool_t pool;
  cudaError_t e = pool_for_current_device(&pool);
  if (e != cudaSuccess) return e;
  if (bytes == 0) bytes = 256;
  return cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
}

cudaError_t scratch_free(void* ptr, cudaStream_t stream) {
  if (!ptr) return cudaSuccess;
  return cudaFreeAsync(ptr, stream);
}

Readback::Buffer* Readback::free_[kMaxDevices] = {};

cudaError_t Readback::take() {
  cudaError_t e = cudaGetDevice(&device_);
  if (e != cudaSuccess) return e;
  if (device_ < 0 || device_ >= kMaxDevices) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    buffer_ = free_[device_];
    if (buffer_) free_[device_] = buffer_->next;
  }
  if (buffer_) return cudaSuccess;
  Buffer* b = new (std::nothrow) Buffer;
  if (!b) return cudaErrorMemoryAllocation;
  e = cudaHostAlloc((void**)&b->words, sizeof(unsigned long long) * kWords, cudaHostAllocDefault);
  if (e == cudaSuccess) {
    e = cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming);
    if (e != cudaSuccess) cudaFreeHost(b->words);
  }
  if (e == cudaSuccess) buffer_ = b;
  else delete b;
  return e;
}

cudaError_t Readback::queue(const void* src, int n, cudaStream_t stream) {
  if (n < 0 || n > kWords - count_) return cudaErrorInvalidValue;
  cudaError_t e = buffer_ ? cudaSuccess : take();
  if (e != cudaSuccess) return e;
  pending_ = true;
  e = cudaMemcpyAsync(buffer_->words + count_, src, sizeof(unsigned long long) * n,
                      cudaMemcpyDeviceToHost, stream);
  count_ += n;
  if (e != cudaSuccess) buffer_ = nullptr;  // (not used again: see the destructor)
  return e;
}

cudaError_t Readback::mark(cudaStream_t stream) {
  const cudaError_t e = cudaEventRecord(buffer_->done, stream);
  if (e != cudaSuccess) buffer_ = nullptr;
  return e;
}

cudaError_t Readback::wait() {
  const cudaError_t e = cudaEventSynchronize(buffer_->done);
  if (e == cudaSuccess) pending_ = false;
  return e;
}

cudaError_t Readback::wait_stream(cudaStream_t stream) {
  const cudaError_t e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess) pending_ = false;
  return e;
}

Readback::~Readback() {
  // (a buffer that may still be written is not used again: the copy became part
  // of a graph, or the device has failed)
  if (!buffer_ || pending_) return;
  std::lock_guard<std::mutex> lock(g_mutex);
  buffer_->next = free_[device_];
  free_[device_] = buffer_;
}

int device_sm_count() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 1;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_sm_count[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 1;
    g_sm_count[dev] = n;
  }
  return g_sm_count[dev];
}

cudaError_t scan_tiles_alloc(ScanTiles* st, void** base, long long ntiles, cudaStream_t stream) {
  size_t bytes = (size_t)(ntiles + 1) * sizeof(unsigned long long);
  cudaError_t e = scratch_alloc(base, bytes, stream);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(*base, 0, bytes, stream);
  if (e != cudaSuccess) return e;
  st->ticket = reinterpret_cast<unsigned long long*>(*base);
  st->status = st->ticket + 1;
  return cudaSuccess;
}

}  // namespace gb

// dst[i] (host) = *src[i] (int64 device words), n <= 16, once `stream` has got
// there: one wait for all of them.
GB_EXPORT int awkward_gb300_read_words(int64_t* dst, const int64_t* const* src, int64_t n,
                                       void* stream) {
  if (n < 0 || n > gb::Readback::kWords) return (int)cudaErrorInvalidValue;
  cudaStream_t s = (cudaStream_t)stream;
  gb::Readback r;
  cudaError_t e = cudaSuccess;
  for (int64_t i = 0; i < n && e == cudaSuccess; i++) e = r.queue(src[i], 1, s);
  cudaError_t w = n > 0 ? r.wait_stream(s) : cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = w;
  for (int64_t i = 0; i < n && e == cudaSuccess; i++) dst[i] = (int64_t)r.words()[i];
  return (int)e;
}

// Library identification for the host-side loader.
GB_EXPORT const char* awkward_gb300_version() { return "awkward_gb300 0.1 (sm_103a)"; }
