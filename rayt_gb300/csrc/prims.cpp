// C ABI of the stand-alone feedback primitives (GPUSort, GPUScan and the
// feedback extractor's GetUnique).  Scratch memory is per-device buffers the
// library grows on demand and keeps; calls are serialised by one mutex, so
// concurrent host threads do not share it mid-operation.
#include <algorithm>
#include <mutex>
#include "internal.h"

namespace rayt {
namespace {
// Memory and bookkeeping of one device.  The look-back words have a buffer of
// their own: they are recognised by their tag, so no other data may ever lie
// where a later call looks for them.
struct Device {
  void* scratch = nullptr;
  size_t scratch_bytes = 0;
  unsigned long long* status = nullptr;  // look-back words
  size_t status_bytes = 0;
  void* area = nullptr;       // the allocation-free entry point's look-back words
  size_t area_bytes = 0;
  uint32_t epoch = 0;         // of the last call since the tables were cleared
  int* host = nullptr;        // mapped pinned: [0] error flag, [1..2] result, [3] number of the last call done
  int* host_dev = nullptr;
  int* ctas = nullptr;        // device: CTAs of the call's last kernel that have ended
  unsigned int calls = 0;     // number of the last call
};
Device g_devices[64];
constexpr uint32_t kEpochLimit = (1u << 27) - 1;

int current_device(Device** d) {
  int dev = 0;
  RAYT_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(RAYT_E_ARG, "device ordinal out of range");
  *d = &g_devices[dev];
  return RAYT_OK;
}

// Clears the look-back tables on s.
int clear_tables(Device& d, cudaStream_t s) {
  if (d.status) RAYT_CUDA_TRY(cudaMemsetAsync(d.status, 0, d.status_bytes, s));
  if (d.area) RAYT_CUDA_TRY(cudaMemsetAsync(d.area, 0, d.area_bytes, s));
  d.epoch = 0;
  return RAYT_OK;
}

template <typename T>
int grow(T** p, size_t* have, size_t bytes) {
  if (*have >= bytes) return RAYT_OK;
  if (*p) {
    RAYT_CUDA_TRY(cudaDeviceSynchronize());
    cudaFree(*p);
    *p = nullptr;
    *have = 0;
  }
  if (cudaMalloc((void**)p, bytes) != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return fail(RAYT_E_OOM, "scratch allocation failed");
  }
  *have = bytes;
  return RAYT_OK;
}

// The current device's memory for a call, and the call's epoch.
int begin(size_t scratch_bytes, size_t status_bytes, cudaStream_t s, Device** out, uint32_t* epoch) {
  int rc = current_device(out);
  if (rc != RAYT_OK) return rc;
  Device& d = **out;
  if (!d.host) {
    RAYT_CUDA_TRY(cudaHostAlloc(&d.host, 4 * sizeof(int), cudaHostAllocMapped));
    for (int k = 0; k < 4; ++k) d.host[k] = 0;
    RAYT_CUDA_TRY(cudaHostGetDevicePointer((void**)&d.host_dev, d.host, 0));
  }
  if (!d.ctas) {
    if (cudaMalloc(&d.ctas, sizeof(int)) != cudaSuccess) return fail(RAYT_E_OOM, "scratch allocation failed");
    RAYT_CUDA_TRY(cudaMemsetAsync(d.ctas, 0, sizeof(int), s));
  }
  if ((rc = grow(&d.scratch, &d.scratch_bytes, scratch_bytes)) != RAYT_OK) return rc;
  if (d.status_bytes < status_bytes) {
    if ((rc = grow(&d.status, &d.status_bytes, status_bytes)) != RAYT_OK) return rc;
    // look-back words are epoch-tagged, never cleared: start from zeros,
    // ordered before the call's kernels on the caller's stream
    RAYT_CUDA_TRY(cudaMemsetAsync(d.status, 0, d.status_bytes, s));
  }
  return lookback_epoch_step(s, epoch);
}

int check_error(Device& d) {
  volatile int* flag = d.host;
  if (!*flag) return RAYT_OK;
  *flag = 0;
  return fail(RAYT_E_TIMEOUT, "a bounded device wait gave up (look-back did not complete)");
}

// The flag that the last kernel of the device work to be launched sets.
DoneFlag next_done(Device& d) {
  return DoneFlag{d.ctas, reinterpret_cast<unsigned int*>(d.host_dev) + 3, ++d.calls};
}

// Waits for that, or until early(result), and reads the error flag.
int finish(Device& d, cudaStream_t s, bool (*early)(const int*) = nullptr) {
  const int rc = wait_word(reinterpret_cast<const unsigned int*>(d.host) + 3, d.calls, s, early, d.host + 1);
  return rc != RAYT_OK ? rc : check_error(d);
}
}  // namespace

std::mutex& prims_mutex() {
  static std::mutex mu;
  return mu;
}

void register_lookback_area(void* p, size_t bytes) {
  Device* d = nullptr;
  if (current_device(&d) != RAYT_OK) return;
  d->area = p;
  d->area_bytes = bytes;
}

int lookback_epoch_step(cudaStream_t s, uint32_t* epoch) {
  Device* d = nullptr;
  int rc = current_device(&d);
  if (rc != RAYT_OK) return rc;
  // the next epoch would reuse a tag that old look-back words may still carry:
  // zero every table (a zero word is never "published") and restart
  if (d->epoch >= kEpochLimit && (rc = clear_tables(*d, s)) != RAYT_OK) return rc;
  *epoch = ++d->epoch;
  return RAYT_OK;
}
}  // namespace rayt

using rayt::fail;

extern "C" {

int rayt_sort_i32(int32_t* data, int n, void* stream) {
  if (n < 0 || (n > 0 && !data)) return fail(RAYT_E_ARG, "rayt_sort_i32: bad arguments");
  if (n >= (1 << 30)) return fail(RAYT_E_LIMIT, "rayt_sort_i32: n must be below 2^30");
  if (n <= 1) return RAYT_OK;
  std::lock_guard<std::mutex> lock(rayt::prims_mutex());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rayt::Device* d = nullptr;
  uint32_t epoch = 0;
  int rc = rayt::begin(rayt::sort_scratch_bytes(n), rayt::sort_status_bytes(n), s, &d, &epoch);
  if (rc != RAYT_OK) return rc;
  int *err = d->host_dev, *again = d->host_dev + 1;
  d->host[1] = 0;
  RAYT_CUDA_TRY(
      rayt::sort_i32_device(data, n, d->scratch, d->status, epoch, again, err, rayt::next_done(*d), s));
  if ((rc = rayt::finish(*d, s)) != RAYT_OK) return rc;
  if (!rayt::sort_needs_passes(d->host + 1)) return RAYT_OK;
  RAYT_CUDA_TRY(rayt::sort_passes_device(data, n, d->scratch, d->status, epoch, err, rayt::next_done(*d), s));
  return rayt::finish(*d, s);
}

int rayt_scan_i32(int32_t* data, int n, void* stream) {
  if (n < 0 || (n > 0 && !data)) return fail(RAYT_E_ARG, "rayt_scan_i32: bad arguments");
  if (n >= (1 << 30)) return fail(RAYT_E_LIMIT, "rayt_scan_i32: n must be below 2^30");
  if (n == 0) return RAYT_OK;
  std::lock_guard<std::mutex> lock(rayt::prims_mutex());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rayt::Device* d = nullptr;
  uint32_t epoch = 0;
  const int rc = rayt::begin(0, rayt::scan_status_bytes(n), s, &d, &epoch);
  if (rc != RAYT_OK) return rc;
  RAYT_CUDA_TRY(rayt::scan_i32_device(data, n, d->status, epoch, d->host_dev, rayt::next_done(*d), s));
  return rayt::finish(*d, s);
}

int rayt_testing_set_lookback_epoch(uint32_t calls) {
  if (calls >= (1u << 27)) return fail(RAYT_E_ARG, "rayt_testing_set_lookback_epoch: epoch out of range");
  std::lock_guard<std::mutex> lock(rayt::prims_mutex());
  rayt::Device* d = nullptr;
  const int rc = rayt::current_device(&d);
  if (rc != RAYT_OK) return rc;
  RAYT_CUDA_TRY(cudaDeviceSynchronize());
  d->epoch = calls;
  return RAYT_OK;
}

int rayt_selftest_bounded_wait(double limit_s, void* stream) {
  if (!(limit_s > 0) || limit_s > 10) return fail(RAYT_E_ARG, "rayt_selftest_bounded_wait: limit out of range (0, 10] s");
  std::lock_guard<std::mutex> lock(rayt::prims_mutex());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rayt::Device* d = nullptr;
  uint32_t epoch = 0;
  int rc = rayt::begin(0, 0, s, &d, &epoch);
  if (rc != RAYT_OK) return rc;
  RAYT_CUDA_TRY(rayt::bounded_wait_probe(limit_s, d->host_dev, s));  // synchronises the stream
  rc = rayt::check_error(*d);
  if (rc == RAYT_E_TIMEOUT) return RAYT_OK;  // the wait gave up as it must
  return rc != RAYT_OK ? rc : fail(RAYT_E_STATE, "bounded wait did not give up");
}

int rayt_feedback_unique(const int32_t* words, int n, int nib, int32_t* unique, int* unique_count, void* stream) {
  if (n < 0 || !unique_count || (n > 0 && (!words || !unique)) || nib < 0)
    return fail(RAYT_E_ARG, "rayt_feedback_unique: bad arguments");
  if (n >= (1 << 30)) return fail(RAYT_E_LIMIT, "rayt_feedback_unique: n must be below 2^30");
  if (n == 0) {
    *unique_count = 0;
    return RAYT_OK;
  }
  std::lock_guard<std::mutex> lock(rayt::prims_mutex());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rayt::Device* d = nullptr;
  uint32_t epoch = 0;
  int rc = rayt::begin(rayt::feedback_scratch_bytes(n), rayt::feedback_status_bytes(n), s, &d, &epoch);
  if (rc != RAYT_OK) return rc;
  int *err = d->host_dev, *result = d->host_dev + 1;
  d->host[1] = d->host[2] = 0;
  RAYT_CUDA_TRY(rayt::feedback_unique_device(words, n, nib, unique, d->scratch, d->status, epoch, result, err, rayt::next_done(*d), s));
  if ((rc = rayt::finish(*d, s, rayt::feedback_unique_needs_radix)) != RAYT_OK) return rc;
  if (rayt::feedback_unique_needs_radix(d->host + 1)) {
    const cudaError_t e =
        rayt::feedback_unique_radix_device(n, unique, d->scratch, d->status, epoch, result, err, rayt::next_done(*d), s);
    if (e != cudaSuccess) cudaStreamSynchronize(s);  // the kernels before may still be using the scratch memory
    RAYT_CUDA_TRY(e);
    if ((rc = rayt::finish(*d, s)) != RAYT_OK) return rc;
  }
  *unique_count = d->host[1];
  return RAYT_OK;
}

}  // extern "C"
