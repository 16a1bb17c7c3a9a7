// Host runtime of libmultifloats_cuda: error latch, device checks, staging
// buffers for the drop-in (host-pointer) symbols, workspace allocation.
#include <cuda.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

#include "common.cuh"

namespace mfcuda {

static thread_local int t_last_error = MFCUDA_OK;
void set_last_error(int code) { t_last_error = code; }
int last_error() { return t_last_error; }

static constexpr int kMaxDevices = 64;

int require_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return MFCUDA_ERR_NO_DEVICE;
  }
  if (dev < 0 || dev >= kMaxDevices) return MFCUDA_ERR_NO_DEVICE;
  static std::atomic<int> major_cache[kMaxDevices];
  int major = major_cache[dev].load(std::memory_order_relaxed);
  if (major == 0) {
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) {
      (void)cudaGetLastError();
      return MFCUDA_ERR_NO_DEVICE;
    }
    major_cache[dev].store(major, std::memory_order_relaxed);
  }
  // The kernels are built for sm_100a only.
  return major == 10 ? MFCUDA_OK : MFCUDA_ERR_NO_DEVICE;
}

int sm_count() {
  int dev = 0;
  cudaGetDevice(&dev);
  static std::atomic<int> cache[kMaxDevices];
  int v = (dev >= 0 && dev < kMaxDevices) ? cache[dev].load() : 0;
  if (v == 0) {
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (v <= 0) v = 148;
    if (dev >= 0 && dev < kMaxDevices) cache[dev].store(v);
  }
  return v;
}

bool injected_alloc_failure() {
  static std::atomic<long> counter{0};
  static long target = [] {
    const char *s = std::getenv("MFCUDA_FAIL_ALLOC");
    return s ? std::atol(s) : 0L;
  }();
  if (target <= 0) return false;
  return counter.fetch_add(1) + 1 == target;
}

static std::atomic<uint64_t> g_wait_limit_ns{0};  // 0: the default
static constexpr uint64_t kDefaultWaitNs = 2000000000ull;
uint64_t wait_limit_ns() {
  const uint64_t v = g_wait_limit_ns.load(std::memory_order_relaxed);
  return v ? v : kDefaultWaitNs;
}

namespace {
struct DeviceStaging {
  std::mutex mu;
  cudaStream_t stream = nullptr, copy = nullptr;
  cudaEvent_t ev[kStagingEvents] = {};
  bool have_ev = false;
  void *buf[4] = {nullptr, nullptr, nullptr, nullptr};
  size_t cap[4] = {0, 0, 0, 0};
};
DeviceStaging g_staging[kMaxDevices];
}  // namespace

int staging_acquire(Staging &st, const size_t bytes[4]) {
  int dev = 0;
  MF_TRY_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return MFCUDA_ERR_NO_DEVICE;
  DeviceStaging &ds = g_staging[dev];
  st.lock = std::unique_lock<std::mutex>(ds.mu);
  if (!ds.stream) MF_TRY_CUDA(cudaStreamCreateWithFlags(&ds.stream, cudaStreamNonBlocking));
  if (!ds.copy) MF_TRY_CUDA(cudaStreamCreateWithFlags(&ds.copy, cudaStreamNonBlocking));
  if (!ds.have_ev) {
    for (int i = 0; i < kStagingEvents; ++i)
      MF_TRY_CUDA(cudaEventCreateWithFlags(&ds.ev[i], cudaEventDisableTiming));
    ds.have_ev = true;
  }
  st.stream = ds.stream;
  st.copy = ds.copy;
  for (int i = 0; i < kStagingEvents; ++i) st.ev[i] = ds.ev[i];
  for (int i = 0; i < 4; ++i) {
    if (bytes[i] > ds.cap[i]) {
      if (ds.buf[i]) {
        MF_TRY_CUDA(cudaStreamSynchronize(ds.stream));
        MF_TRY_CUDA(cudaFree(ds.buf[i]));
        ds.buf[i] = nullptr;
        ds.cap[i] = 0;
      }
      if (injected_alloc_failure()) return MFCUDA_ERR_ALLOC;
      size_t want = bytes[i] < 256 ? 256 : bytes[i];
      MF_TRY_CUDA(device_malloc(&ds.buf[i], want));
      ds.cap[i] = want;
    }
    st.buf[i] = ds.buf[i];
  }
  return MFCUDA_OK;
}

// Workspace pool.  The device's default pool gives its free memory back to the
// system whenever the stream is synchronised, and a call that waits for its
// result (or a caller that waits between calls) then pays for mapping the
// workspace again: 1.6 GB at 4096^3, 20 ms on a 2.2 ms product.  The library
// therefore allocates from a pool of its own that keeps up to kWorkspaceKeep
// bytes of free memory; what is above that goes back at the next
// synchronisation.  A request of this process that needs the free memory gets it
// (tried with larger workspaces, cudaMalloc, cuMemCreate and the default pool);
// for other processes mfcuda_release_workspace gives it back.  Allocation stays
// stream-ordered, so any number of threads
// and streams may use the pool.  A pool belongs to the context it was made
// under (contexts are told apart by their id, which is never reused), so one
// that died with a device reset is never touched again.
namespace {
constexpr uint64_t kWorkspaceKeep = 4ull << 30;
constexpr int kMaxPools = 64;
struct WorkspacePool {
  unsigned long long ctx = 0;
  cudaMemPool_t pool = nullptr;
};
std::mutex g_pool_mu;
WorkspacePool g_pools[kMaxPools];
int g_npools = 0;

using CtxGetId = CUresult (*)(CUcontext, unsigned long long *);
CtxGetId ctx_get_id() {
  static const CtxGetId fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<CtxGetId>(p);
  }();
  return fn;
}

// Making or trimming a pool touches no stream, but a stream capture in its global
// or thread-local mode refuses such calls and is lost by them.  In the relaxed
// mode, which is this thread's alone, it allows them.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { exchange(); }
  ~RelaxedCapture() { exchange(); }
  void exchange() {
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) (void)cudaGetLastError();
  }
};

// The current context's pool, made on first use (which may be inside a stream
// capture); nullptr where there is none (the device's default pool serves then).
cudaMemPool_t workspace_pool(bool create) {
  unsigned long long id = 0;
  const CtxGetId fn = ctx_get_id();
  if (!fn || fn(nullptr, &id) != CUDA_SUCCESS) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  for (int i = 0; i < g_npools; ++i)
    if (g_pools[i].ctx == id) return g_pools[i].pool;
  if (!create || g_npools == kMaxPools) return nullptr;
  RelaxedCapture relaxed;
  int dev = 0;
  cudaMemPool_t pool = nullptr;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  uint64_t keep = kWorkspaceKeep;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  props.location.id = dev;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    (void)cudaGetLastError();
    (void)cudaMemPoolDestroy(pool);
    return nullptr;
  }
  g_pools[g_npools].ctx = id;
  g_pools[g_npools].pool = pool;
  ++g_npools;
  return pool;
}
}  // namespace

static int ws_release_free() {
  if (cudaMemPool_t pool = workspace_pool(false)) {
    RelaxedCapture relaxed;
    MF_TRY_CUDA(cudaMemPoolTrimTo(pool, 0));
  }
  return MFCUDA_OK;
}

cudaError_t device_malloc(void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {  // free workspace memory may be what is missing
    (void)cudaGetLastError();
    (void)ws_release_free();
    e = cudaMalloc(p, bytes);
  }
  return e;
}

int ws_alloc(void **p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  if (bytes == 0) return MFCUDA_OK;
  if (injected_alloc_failure()) return MFCUDA_ERR_ALLOC;
  if (cudaMemPool_t pool = workspace_pool(true)) {
    if (cudaMallocFromPoolAsync(p, bytes, pool, s) == cudaSuccess) return MFCUDA_OK;
    (void)cudaGetLastError();
    *p = nullptr;
  }
  MF_TRY_CUDA(cudaMallocAsync(p, bytes, s));
  return MFCUDA_OK;
}
void ws_free(void *p, cudaStream_t s) {
  if (p) (void)cudaFreeAsync(p, s);
}

}  // namespace mfcuda

extern "C" {

MULTIFLOATS_CUDA_API int mfcuda_last_error(void) { return mfcuda::last_error(); }

MULTIFLOATS_CUDA_API const char *mfcuda_error_string(int code) {
  switch (code) {
    case MFCUDA_OK: return "success";
    case MFCUDA_ERR_INVALID_ARG: return "invalid argument";
    case MFCUDA_ERR_CUDA: return "CUDA runtime error";
    case MFCUDA_ERR_ALLOC: return "allocation failed";
    case MFCUDA_ERR_NO_DEVICE: return "no sm_100 device";
    case MFCUDA_ERR_TIMEOUT: return "device-side wait timed out";
    case MFCUDA_ERR_WORKSPACE: return "workspace too small";
    case MFCUDA_ERR_UNSUPPORTED: return "unsupported shape or parameter";
    default: return "unknown error";
  }
}

MULTIFLOATS_CUDA_API const char *mfcuda_version(void) { return "0.1.0"; }

MULTIFLOATS_CUDA_API int mfcuda_release_workspace(void) {
  MF_TRY(mfcuda::require_device());
  return mfcuda::ws_release_free();
}

MULTIFLOATS_CUDA_API uint64_t mfcuda_set_wait_limit_ns(uint64_t ns) {
  return mfcuda::g_wait_limit_ns.exchange(ns);
}

}  // extern "C"
