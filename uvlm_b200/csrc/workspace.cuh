// workspace.cuh -- device memory for the length of a context-free call.
#pragma once

#include <vector>

#include "common.cuh"

namespace uvlm {

// Whether the calling thread works in its device's primary context (made current
// if there is none), where the pool lives.  A program may have a context of its
// own current instead: its calls stay in it and allocate there.
bool workspace_in_primary_context();
// pooled: from the pool, stream-ordered on the legacy default stream of the
// current device; else from the current context.
Error workspace_alloc(void** p, size_t bytes, bool pooled);
void workspace_free(void* p, bool pooled);
// After a call's last workspace_free: gives back what is kept beyond the bound.
void workspace_settle();
// Unique id of the context current on this thread (0 if the driver entry
// points are unavailable).  A cudaDeviceReset destroys the primary context and
// what belongs to it; the next primary context has another id.
unsigned long long current_context_id();

// Device buffers of one call, freed at scope exit.  Small ones share slabs.
struct Scratch {
  const bool pooled = workspace_in_primary_context();
  std::vector<void*> p;
  char* slab = nullptr;
  size_t left = 0;
  Scratch() = default;
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  ~Scratch() {
    for (void* q : p) workspace_free(q, pooled);
    if (pooled && !p.empty()) workspace_settle();
  }
  Error bytes(void** out, size_t count) {
    constexpr size_t kSlab = 1u << 20;
    *out = nullptr;
    if (count == 0) return ok();
    const size_t need = (count + 255) & ~(size_t)255;
    if (need < count) return fail(kErrCapacity, "buffer size out of range");
    if (need <= kSlab / 2) {
      if (need > left) {
        void* s = nullptr;
        UVLM_TRY(workspace_alloc(&s, kSlab, pooled));
        p.push_back(s);
        slab = static_cast<char*>(s);
        left = kSlab;
      }
      *out = slab;
      slab += need;
      left -= need;
      return ok();
    }
    UVLM_TRY(workspace_alloc(out, need, pooled));
    p.push_back(*out);
    return ok();
  }
  template <class T>
  Error get(T** out, size_t count) {
    return bytes(reinterpret_cast<void**>(out), sizeof(T) * count);
  }
  template <class T>
  Error up(T** out, const T* host, size_t count) {
    UVLM_TRY(get(out, count));
    if (count) UVLM_CUDA_TRY(cudaMemcpy(*out, host, sizeof(T) * count, cudaMemcpyHostToDevice));
    return ok();
  }
};

}  // namespace uvlm
