// refapi_util.cuh -- helpers shared by the context-free C-ABI entry points
// (refapi.cu, legacy.cu): the
// FP64/FP32 N-body of sheets and of AoS rings at arbitrary targets and a
// fixed-order block sum.
#pragma once

#include <algorithm>
#include "../../include/uvlm_b200.h"
#include "common.cuh"
#include "nbody.cuh"
#include "workspace.cuh"

using namespace uvlm;

namespace {

int report(const Error& e) {
  if (e.code) set_global_error(e.msg);
  return e.code;
}

int sms() {
  int d = 0, v = 148;
  cudaGetDevice(&d);
  cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d);
  return v;
}

constexpr int kSumThreads = 256;

__device__ inline d3 block_sum3(d3 v, double* sh) {
  for (int off = 16; off; off >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, off);
    v.y += __shfl_down_sync(0xffffffffu, v.y, off);
    v.z += __shfl_down_sync(0xffffffffu, v.z, off);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sh[3 * wid] = v.x;
    sh[3 * wid + 1] = v.y;
    sh[3 * wid + 2] = v.z;
  }
  __syncthreads();
  d3 r = mk(0, 0, 0);
  for (int w = 0; w < kSumThreads / 32; ++w) r = add(r, mk(sh[3 * w], sh[3 * w + 1], sh[3 * w + 2]));
  return r;
}

inline int gfor(long long n) { return (int)std::min<long long>(std::max<long long>((n + 255) / 256, 1), 65535); }

// Records of the sheets and room for the partial sums: 64 splits of few target
// tiles; from 64 tiles on fewer splits fill the device.
Error sources_at(const SheetView* views, int nv, NBodyPrec prec, long long nt, NBodyWork* w, SourceBlock* blocks,
                 Scratch& S) {
  long long recs = 0;
  for (int i = 0; i < nv; ++i) recs += (long long)views[i].num * views[i].node_rows * (views[i].cols + 1);
  w->records_cap = std::max<long long>(recs, 1) * (long long)(prec == kNBodyFP32 ? sizeof(RecF) : sizeof(RecD));
  UVLM_TRY(S.get(reinterpret_cast<char**>(&w->records), (size_t)w->records_cap));
  w->partial_cap = 3 * std::max<long long>(nt, 1) * (nt > 64 * 256 ? 24 : kMaxSplits);
  UVLM_TRY(S.get(&w->partial, (size_t)w->partial_cap));
  return nbody_build_sources(views, nv, prec, w, blocks, 0);
}

// Velocities of the sheets at SoA targets in the order given.
Error velocity_soa(const SheetView* views, int nv, NBodyPrec prec, const double* tx, const double* ty,
                   const double* tz, long long nt, double* vx, double* vy, double* vz, Scratch& S) {
  NBodyWork w;
  SourceBlock blocks[4];
  UVLM_TRY(sources_at(views, nv, prec, nt, &w, blocks, S));
  const int variant = prec == kNBodyFP32 ? kDefaultVariantF32 : kDefaultVariantF64;
  return nbody_eval(blocks, nv, prec, tx, ty, tz, nt, vx, vy, vz, &w, variant, sms(), 0);
}

// Velocities of the sheets at arbitrary AoS targets.
Error velocity_at(const SheetView* views, int nv, NBodyPrec prec, const double* d_targets, long long nt,
                  double* d_out, Scratch& S) {
  NBodyWork w;
  SourceBlock blocks[4];
  double* soa;
  char* order;
  UVLM_TRY(S.get(&soa, 3 * nt));
  UVLM_TRY(S.get(&order, nbody_order_bytes(nt)));
  UVLM_TRY(sources_at(views, nv, prec, nt, &w, blocks, S));
  return nbody_eval_points(blocks, nv, prec, d_targets, nt, d_out, &w, soa, order, sms(), 0);
}

// out = base + (velocity induced by AoS rings at AoS targets + add3) scale, all
// on the device, FP64 (base and add3 may be NULL).
Error rings_at(const double* d_rings, const double* d_gamma, long long n_rings, bool chordwise_only,
               const double* d_targets, long long nt, const double* add3, const double* base, double scale,
               double* d_out, Scratch& S) {
  double* partial = nullptr;
  const int n_sms = sms();
  UVLM_TRY(S.get(&partial, rings_partial_size(n_rings, nt, n_sms)));
  return rings_eval(d_rings, d_gamma, n_rings, chordwise_only, d_targets, nt, add3, base, scale, partial, d_out, n_sms,
                    0);
}

}  // namespace
