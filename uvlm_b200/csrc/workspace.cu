// workspace.cu -- device memory of the context-free calls.
//
// Each of them needs a dozen arrays for the length of the call.  cudaMalloc and
// cudaFree of those cost 0.5 to 1 ms per call (each maps or unmaps memory and
// every cudaFree waits for the device), many times the work of a small call:
// InducedVelocity of 9 points over a 4 x 8 sheet took 730 us, 24 us of it on
// the device.  The arrays therefore come from one CUDA memory pool per device,
// stream-ordered on the legacy default stream that all these calls use: an array
// freed by one call is handed to the next one, of any thread, in the order of
// that stream.  The pool is the library's own (the device's default pool, which
// the host program may use, is not touched).  It keeps at most
// kKeptWorkspaceBytes between calls: a call that ends with more reserved waits
// for the stream and trims the pool (a release threshold alone takes effect at
// the program's next synchronisation, whenever that is; 2.0 GB stayed after 3
// million points), and uvlm_release_workspace gives all of it back.  A thread that
// works in a driver context of its own takes its arrays from that context instead.
#include <cuda.h>

#include <mutex>

#include "../../include/uvlm_b200.h"
#include "device_once.h"
#include "workspace.cuh"

namespace uvlm {
namespace {

// The 4096 x 4096 dense solve (134 MB of matrix, 67 MB of FP32 factors) fits.
constexpr unsigned long long kKeptWorkspaceBytes = 256ull << 20;

// The driver's context calls (NULL where there is no driver).
struct Driver {
  CUresult (*get_current)(CUcontext*) = nullptr;
  CUresult (*set_current)(CUcontext) = nullptr;
  CUresult (*get_id)(CUcontext, unsigned long long*) = nullptr;
  CUresult (*device_get)(CUdevice*, int) = nullptr;
  CUresult (*primary_state)(CUdevice, unsigned*, int*) = nullptr;
  CUresult (*primary_retain)(CUcontext*, CUdevice) = nullptr;
  CUresult (*primary_release)(CUdevice) = nullptr;
  Driver() {
    find("cuCtxGetCurrent", get_current);
    find("cuCtxSetCurrent", set_current);
    find("cuCtxGetId", get_id);
    find("cuDeviceGet", device_get);
    find("cuDevicePrimaryCtxGetState", primary_state);
    find("cuDevicePrimaryCtxRetain", primary_retain);
    find("cuDevicePrimaryCtxRelease", primary_release);
  }
  template <class F>
  static void find(const char* name, F& f) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      f = reinterpret_cast<F>(fn);
    else
      cudaGetLastError();
  }
};
const Driver& driver() {
  static const Driver d;
  return d;
}

std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};
unsigned long long g_pool_ctx[kMaxDevices] = {};  // context the pool belongs to

Error pool_of(int dev, cudaMemPool_t* out) {
  if (dev < 0 || dev >= kMaxDevices) return fail(kErrUnsupported, "device ordinal out of range");
  const unsigned long long ctx = current_context_id();
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool[dev] || g_pool_ctx[dev] != ctx) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    UVLM_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
    unsigned long long keep = kKeptWorkspaceBytes;
    const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return fail(kErrCuda, std::string("cudaMemPoolSetAttribute: ") + cudaGetErrorString(e));
    }
    g_pool[dev] = pool;
    g_pool_ctx[dev] = ctx;
  }
  *out = g_pool[dev];
  return ok();
}

}  // namespace

unsigned long long current_context_id() {
  const Driver& d = driver();
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (d.get_current && d.get_id && d.get_current(&ctx) == CUDA_SUCCESS && ctx) d.get_id(ctx, &id);
  return id;
}

bool workspace_in_primary_context() {
  const Driver& d = driver();
  int dev = 0;
  if (!d.get_current || !d.device_get || !d.primary_state || !d.primary_retain || !d.primary_release ||
      cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  CUcontext now = nullptr, primary = nullptr;
  if (d.get_current(&now) != CUDA_SUCCESS) now = nullptr;
  if (!now) return cudaSetDevice(dev) == cudaSuccess;
  // the state first: retaining would bring up a context that the program does without
  unsigned flags = 0;
  int active = 0;
  CUdevice device = 0;
  if (d.device_get(&device, dev) != CUDA_SUCCESS || d.primary_state(device, &flags, &active) != CUDA_SUCCESS ||
      !active || d.primary_retain(&primary, device) != CUDA_SUCCESS)
    return false;
  d.primary_release(device);
  return primary == now;
}

Error workspace_alloc(void** p, size_t bytes, bool pooled) {
  *p = nullptr;
  if (!pooled) {
    UVLM_CUDA_TRY(cudaMalloc(p, bytes));
    return ok();
  }
  int dev = 0;
  UVLM_CUDA_TRY(cudaGetDevice(&dev));
  cudaMemPool_t pool = nullptr;
  UVLM_TRY(pool_of(dev, &pool));
  cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, nullptr);
  if (e == cudaErrorMemoryAllocation) {
    // what the pool keeps may be what is missing
    cudaGetLastError();
    cudaStreamSynchronize(nullptr);
    cudaMemPoolTrimTo(pool, 0);
    e = cudaMallocFromPoolAsync(p, bytes, pool, nullptr);
  }
  if (e != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return fail(kErrCuda, std::string("device memory: ") + cudaGetErrorString(e));
  }
  return ok();
}

void workspace_free(void* p, bool pooled) {
  if (!p) return;
  if (pooled)
    cudaFreeAsync(p, nullptr);
  else
    cudaFree(p);
}

void workspace_settle() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    pool = g_pool[dev];
  }
  unsigned long long reserved = 0;
  if (!pool) return;
  if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  // of several calls at once, the last to end sees what all of them reserved
  if (reserved > kKeptWorkspaceBytes && cudaStreamSynchronize(nullptr) == cudaSuccess)
    cudaMemPoolTrimTo(pool, kKeptWorkspaceBytes);
}

}  // namespace uvlm

extern "C" int uvlm_release_workspace(int32_t device) {
  using namespace uvlm;
  auto run = [&]() -> Error {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
      cudaGetLastError();
      return fail(kErrCuda, "no CUDA device");
    }
    if (device < 0 || device >= ndev || device >= kMaxDevices) return fail(kErrInvalid, "no such device");
    // in the device's primary context; the caller's own is current again afterwards
    const Driver& d = driver();
    int before = 0;
    CUcontext ctx = nullptr;
    UVLM_CUDA_TRY(cudaGetDevice(&before));
    if (d.get_current) d.get_current(&ctx);
    {
      std::lock_guard<std::mutex> lk(g_pool_mu);
      if (!g_pool[device]) return ok();  // nothing was ever kept
    }
    UVLM_CUDA_TRY(cudaSetDevice(device));
    cudaMemPool_t pool = nullptr;
    Error e = pool_of(device, &pool);
    if (!e.code && (cudaStreamSynchronize(nullptr) != cudaSuccess || cudaMemPoolTrimTo(pool, 0) != cudaSuccess))
      e = fail(kErrCuda, "the workspace could not be released");
    if (ctx && d.set_current)
      d.set_current(ctx);
    else
      cudaSetDevice(before);
    return e;
  };
  const Error e = run();
  if (e.code) set_global_error(e.msg);
  return e.code;
}
