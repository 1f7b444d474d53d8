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
// million points), and uvlm_release_workspace gives all of it back.
#include <cuda.h>

#include <mutex>

#include "../../include/uvlm_b200.h"
#include "device_once.h"
#include "workspace.cuh"

namespace uvlm {
namespace {

// The 4096 x 4096 dense solve (134 MB of matrix, 67 MB of FP32 factors) fits.
constexpr unsigned long long kKeptWorkspaceBytes = 256ull << 20;

std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};
unsigned long long g_pool_ctx[kMaxDevices] = {};  // context the pool belongs to

Error pool_of(int dev, cudaMemPool_t* out) {
  if (dev < 0 || dev >= kMaxDevices) return fail(kErrUnsupported, "device ordinal out of range");
  UVLM_CUDA_TRY(cudaSetDevice(dev));  // makes the primary context current, also after a reset
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
  using GetCurrent = CUresult (*)(CUcontext*);
  using GetId = CUresult (*)(CUcontext, unsigned long long*);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(fn);
    if (cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(fn);
  });
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_current && get_id && get_current(&ctx) == CUDA_SUCCESS && ctx) get_id(ctx, &id);
  return id;
}

Error workspace_alloc(void** p, size_t bytes) {
  *p = nullptr;
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

void workspace_free(void* p) {
  if (p) cudaFreeAsync(p, nullptr);
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
    int ndev = 0, before = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
      cudaGetLastError();
      return fail(kErrCuda, "no CUDA device");
    }
    if (device < 0 || device >= ndev || device >= kMaxDevices) return fail(kErrInvalid, "no such device");
    cudaMemPool_t pool = nullptr;
    UVLM_CUDA_TRY(cudaGetDevice(&before));
    Error e = pool_of(device, &pool);
    if (!e.code && (cudaStreamSynchronize(nullptr) != cudaSuccess || cudaMemPoolTrimTo(pool, 0) != cudaSuccess))
      e = fail(kErrCuda, "the workspace could not be released");
    cudaSetDevice(before);
    return e;
  };
  const Error e = run();
  if (e.code) set_global_error(e.msg);
  return e.code;
}
