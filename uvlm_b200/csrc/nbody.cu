// nbody.cu -- strip-tiled Biot-Savart N-body (FP32 hi/lo and FP64 forms).
#include <algorithm>
#include <climits>
#include <type_traits>

#include <cooperative_groups.h>

#include "device_once.h"
#include "nbody.cuh"

namespace uvlm {
namespace {

template <class Rec>
__global__ void build_records_kernel(SheetView v, Rec* out) {
  const long long total = (long long)v.num * v.node_rows * (v.cols + 1);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < total;
       k += (long long)gridDim.x * blockDim.x)
    out[k] = build_record<Rec>(v, k);
}

// cp.async 16-byte staging of one strip into shared memory ([r][j] records)
template <class Rec>
__device__ inline void stage_strip(Rec* sm, const Rec* rec, const StripInfo& si) {
  constexpr int kChunks = sizeof(Rec) / 16;
  const int total = si.nr * si.n_cols * kChunks;
  for (int q = threadIdx.x; q < total; q += blockDim.x) {
    const int part = q % kChunks;
    const int rj = q / kChunks;
    const int r = rj / si.n_cols, j = rj % si.n_cols;
    const char* src = reinterpret_cast<const char*>(rec + si.first + (long long)r * si.row_stride + j) + 16 * part;
    char* dst = reinterpret_cast<char*>(sm + rj) + 16 * part;
    const unsigned sdst = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sdst), "l"(src));
  }
  asm volatile("cp.async.commit_group;");
}

// Full-tile staging: always (H + 1) x (kStripCols + 1) records; entries past
// the strip's rows or columns are all-zero records (zero strengths, zero
// segment vectors), whose segments have d = 0 and are cut exactly like a
// degenerate segment, so they add +0 to every target.
template <class Rec, int H>
__device__ inline void stage_strip_padded(Rec* sm, const Rec* rec, const StripInfo& si) {
  constexpr int kChunks = sizeof(Rec) / 16;
  constexpr int kCols = kStripCols + 1;
  constexpr int total = (H + 1) * kCols * kChunks;
  for (int q = threadIdx.x; q < total; q += blockDim.x) {
    const int part = q % kChunks;
    const int rj = q / kChunks;
    const int r = rj / kCols, j = rj % kCols;
    char* dst = reinterpret_cast<char*>(sm + rj) + 16 * part;
    if (r < si.nr && j < si.n_cols) {
      const char* src = reinterpret_cast<const char*>(rec + si.first + (long long)r * si.row_stride + j) + 16 * part;
      const unsigned sdst = (unsigned)__cvta_generic_to_shared(dst);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sdst), "l"(src));
    } else {
      *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  asm volatile("cp.async.commit_group;");
}

template <class T>
struct Tgt {
  T hx, hy, hz;  // FP32: hi part; FP64: the position
  T lx, ly, lz;  // FP32: lo part; FP64: unused
};

template <class T>
struct NodeV {
  T rx, ry, rz;  // x - p
  T n;           // |x - p| (0 when x == p; such pairs are cut by |d|^2)
};

__device__ __forceinline__ float nb_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float nb_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// FP64 1/sqrt(x) and 1/x from the hardware's approximations (PTX rsqrt.approx
// / rcp.approx .ftz.f64, relative error about 2^-20) by one step of a
// third-order (Householder) iteration each, the series of the exact correction
// cut after its second term: with e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^(-1/2) =
// y (1 + e/2 + 3 e^2/8 + O(e^3)); with e = 1 - x y, 1/x = y (1 + e + e^2 +
// O(e^3)).  Measured over 4 million arguments of all exponents against 80-bit
// arithmetic: 1/sqrt(x) below 0.993 ulp, 0.331 rms; 1/x below 0.507, 0.289 rms.
// Five and three FP64 operations, without the
// special cases of the library functions: the arguments are squared distances
// and denominators that the callers' cuts keep away from 0 (what a zero gives
// is dropped by a select), and what an infinite one gives (a NaN) is dropped too.
__device__ __forceinline__ double nb_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// sqrt(x) by the same step from s = x y: with e = 1 - s y, sqrt(x) = s (1 + e/2 +
// 3 e^2/8 + O(e^3)).  The rounding of s enters halved, so a length is closer than
// x times the rounded 1/sqrt(x) (rms 0.32 and 0.48 ulp, below 0.76 and 1.74), in
// one operation less.
__device__ __forceinline__ double nb_sqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double s = x * y, e = fma(-s, y, 1.0);
  return fma(s * e, fma(0.375, e, 0.5), s);
}
__device__ __forceinline__ double nb_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

template <class T, class Rec>
__device__ __forceinline__ NodeV<T> node_from(const Rec& r, const Tgt<T>& t) {
  NodeV<T> n;
  if constexpr (sizeof(T) == 4) {
    n.rx = (t.hx - r.hi.x) + (t.lx - r.lo.x);
    n.ry = (t.hy - r.hi.y) + (t.ly - r.lo.y);
    n.rz = (t.hz - r.hi.z) + (t.lz - r.lo.z);
    const float q = n.rx * n.rx + n.ry * n.ry + n.rz * n.rz;
    n.n = q >= (float)kCutR2 ? q * nb_rsqrt(q) : 0.f;  // |x - p| < 1e-10: marked 0 for the node cut
  } else {
    n.rx = t.hx - r.a.x;
    n.ry = t.hy - r.a.y;
    n.rz = t.hz - r.a.z;
    const double q = n.rx * n.rx + n.ry * n.ry + n.rz * n.rz;
    n.n = q >= kCutR2 ? nb_sqrt(q) : 0.0;
  }
  return n;
}

template <class T>
struct SegV {
  T x, y, z;
};

template <class T, class Rec>
__device__ __forceinline__ void rec_fields(const Rec& r, T& gS, T& gH, SegV<T>& s0, SegV<T>& h0) {
  if constexpr (sizeof(T) == 4) {
    gS = r.hi.w;
    gH = r.lo.w;
    s0 = SegV<T>{r.sv.x, r.sv.y, r.sv.z};
    h0 = SegV<T>{r.sv.w, r.hv.x, r.hv.y};
  } else {
    gS = r.a.w;
    gH = r.b.x;
    s0 = SegV<T>{r.b.y, r.b.z, r.b.w};
    h0 = SegV<T>{r.c.x, r.c.y, r.c.z};
  }
}

// Segment start=A -> end=B at x (src/vortex.cpp:24-38): r1 = x - A,
// r2 = x - B, r0 = B - A, d = r1 x r2 = r0 x r1 and the reference's factor
// F = r0.(r1/|r1| - r2/|r2|) / |d|^2.  F is evaluated in forms that are
// algebraically equal to it but free of cancellation:
//   r1.r2 >= 0 (x beyond an end):  F = (|r1| + |r2|) / (|r1||r2| (|r1||r2| + r1.r2))
//   r1.r2 <  0 (x alongside):      F = (|r1| + |r2|) (|r1||r2| - r1.r2) / (|r1||r2| |d|^2)
// (the second from |r1|^2|r2|^2 - (r1.r2)^2 = |d|^2).  The reference form
// subtracts two nearly equal unit vectors when x is near the extension of the
// segment, which is where every wake node sees its lattice neighbours; in FP32
// that costs up to O(1) relative error there (1e-7 .. 1e-4 with these forms).
// Cut, as the reference does, when |d|^2 < 1e-10 or |x - A| < 1e-10 or
// |x - B| < 1e-10 (node_from marks such nodes with n = 0).  The node test is
// not implied by the |d|^2 test in FP32: for a stretched wake segment
// (|r0| ~ 10) whose end node is the target itself, the once-rounded r0 and
// x - A differ by an ulp and leave |d|^2 just above 1e-10.
template <class T>
__device__ __forceinline__ void seg(const SegV<T>& r0, const NodeV<T>& a, const NodeV<T>& b, T g, T& vx, T& vy,
                                    T& vz) {
  const T dx = r0.y * a.rz - r0.z * a.ry;
  const T dy = r0.z * a.rx - r0.x * a.rz;
  const T dz = r0.x * a.ry - r0.y * a.rx;
  const T d2 = dx * dx + dy * dy + dz * dz;
  const T dot12 = a.rx * b.rx + a.ry * b.ry + a.rz * b.rz;
  const T nn = a.n * b.n;
  const bool beyond = dot12 >= (T)0;
  const T num = (a.n + b.n) * (beyond ? (T)1 : nn - dot12);
  const T den = nn * (beyond ? nn + dot12 : d2);
  T k = g * num * nb_rcp(den);
  bool keep = d2 >= (T)kCutD2 && nn > (T)0;
  // an infinite denominator (|r| above about 1e77): the velocity underflows,
  // and nb_rcp has no answer
  if constexpr (sizeof(T) == 8) keep = keep && __double2hiint(den) != 0x7ff00000;
  k = keep ? k : (T)0;
  vx += k * dx;
  vy += k * dy;
  vz += k * dz;
}

// Walk one staged strip for TPT targets: per node column, the H+1 node
// quantities, then the H chordwise segments of the column and the H spanwise
// segments that end in it.
template <class T, class Rec, int H, int TPT>
__device__ __forceinline__ void walk_strip(const Rec* sm, const StripInfo& si, const Tgt<T> (&tg)[TPT],
                                           T (&acc)[TPT][3]) {
  NodeV<T> prev[TPT][H];
  SegV<T> ps0[H];
  T pgS[H];
  const int nr = si.nr, n_rows = si.n_rows, n_cols = si.n_cols;
  for (int j = 0; j < n_cols; ++j) {
    NodeV<T> cur[TPT][H + 1];
    T gS[H], gH[H];
    SegV<T> s0[H], h0[H];
#pragma unroll
    for (int r = 0; r <= H; ++r) {
      if (r < nr) {
        const Rec rec = sm[r * n_cols + j];
        if (r < H) rec_fields<T, Rec>(rec, gS[r], gH[r], s0[r], h0[r]);
#pragma unroll
        for (int q = 0; q < TPT; ++q) cur[q][r] = node_from<T, Rec>(rec, tg[q]);
      }
    }
    const bool col_h = (j < n_cols - 1) || si.last_h;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      if (r < n_rows && r + 1 < nr && col_h) {
#pragma unroll
        for (int q = 0; q < TPT; ++q) seg<T>(h0[r], cur[q][r], cur[q][r + 1], gH[r], acc[q][0], acc[q][1], acc[q][2]);
      }
    }
    if (j > 0) {
#pragma unroll
      for (int r = 0; r < H; ++r) {
        if (r < n_rows) {
#pragma unroll
          for (int q = 0; q < TPT; ++q) seg<T>(ps0[r], prev[q][r], cur[q][r], pgS[r], acc[q][0], acc[q][1], acc[q][2]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < H; ++r) {
      if (r < n_rows) {
        pgS[r] = gS[r];
        ps0[r] = s0[r];
#pragma unroll
        for (int q = 0; q < TPT; ++q) prev[q][r] = cur[q][r];
      }
    }
  }
}

// One node column of a full strip (H owned node rows plus the row below,
// kStripCols + 1 columns, record stride kStripCols + 1 in shared memory): the
// node quantities of the column, its H chordwise segments (DO_H) and the H
// spanwise segments that end in it (!FIRST).  The column's quantities become
// `prev` for the next column; with the column loop unrolled by two the
// compiler renames instead of copying.
template <class T, class Rec, int H, int TPT, bool FIRST, bool DO_H>
__device__ __forceinline__ void full_column(const Rec* col, const Tgt<T> (&tg)[TPT], NodeV<T> (&prev)[TPT][H],
                                            SegV<T> (&ps0)[H], T (&pgS)[H], T (&acc)[TPT][3]) {
  NodeV<T> cur[TPT][H + 1];
  T gS[H], gH[H];
  SegV<T> s0[H], h0[H];
#pragma unroll
  for (int r = 0; r <= H; ++r) {
    const Rec rec = col[r * (kStripCols + 1)];
    if (r < H) rec_fields<T, Rec>(rec, gS[r], gH[r], s0[r], h0[r]);
#pragma unroll
    for (int q = 0; q < TPT; ++q) cur[q][r] = node_from<T, Rec>(rec, tg[q]);
  }
  if (DO_H) {
#pragma unroll
    for (int r = 0; r < H; ++r)
#pragma unroll
      for (int q = 0; q < TPT; ++q) seg<T>(h0[r], cur[q][r], cur[q][r + 1], gH[r], acc[q][0], acc[q][1], acc[q][2]);
  }
  if (!FIRST) {
#pragma unroll
    for (int r = 0; r < H; ++r)
#pragma unroll
      for (int q = 0; q < TPT; ++q) seg<T>(ps0[r], prev[q][r], cur[q][r], pgS[r], acc[q][0], acc[q][1], acc[q][2]);
  }
#pragma unroll
  for (int r = 0; r < H; ++r) {
    pgS[r] = gS[r];
    ps0[r] = s0[r];
#pragma unroll
    for (int q = 0; q < TPT; ++q) prev[q][r] = cur[q][r];
  }
}

// A full strip: compile-time bounds, no per-column predicates.  The last
// column owns its chordwise segments only at the sheet's last column.
template <class T, class Rec, int H, int TPT>
__device__ __forceinline__ void walk_full_strip(const Rec* sm, bool last_h, const Tgt<T> (&tg)[TPT],
                                                T (&acc)[TPT][3]) {
  NodeV<T> prev[TPT][H];
  SegV<T> ps0[H];
  T pgS[H];
  full_column<T, Rec, H, TPT, true, true>(sm, tg, prev, ps0, pgS, acc);
#pragma unroll 2
  for (int j = 1; j < kStripCols; ++j) full_column<T, Rec, H, TPT, false, true>(sm + j, tg, prev, ps0, pgS, acc);
  if (last_h)
    full_column<T, Rec, H, TPT, false, true>(sm + kStripCols, tg, prev, ps0, pgS, acc);
  else
    full_column<T, Rec, H, TPT, false, false>(sm + kStripCols, tg, prev, ps0, pgS, acc);
}

// ------------------------------------------------ packed FP32x2 walker
// The same arithmetic for the thread's two targets at once: lane .x is
// target 0, lane .y target 1, and every add/mul/fma is one sm_100 FP32x2
// instruction (__fadd2_rn / __fmul2_rn / __ffma2_rn) instead of two.  The
// reciprocal square roots, reciprocals and the per-lane selects stay scalar.
__device__ __forceinline__ float2 bc2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

struct Node2 {
  float2 rx, ry, rz, n;
};

__device__ __forceinline__ float node_len(float q) { return q >= (float)kCutR2 ? q * nb_rsqrt(q) : 0.f; }

__device__ __forceinline__ Node2 node_from2(const RecF& r, const Tgt<float> (&tg)[2]) {
  const float2 thx = make_float2(tg[0].hx, tg[1].hx), thy = make_float2(tg[0].hy, tg[1].hy),
               thz = make_float2(tg[0].hz, tg[1].hz);
  const float2 tlx = make_float2(tg[0].lx, tg[1].lx), tly = make_float2(tg[0].ly, tg[1].ly),
               tlz = make_float2(tg[0].lz, tg[1].lz);
  Node2 n;
  n.rx = add2(add2(thx, bc2(-r.hi.x)), add2(tlx, bc2(-r.lo.x)));
  n.ry = add2(add2(thy, bc2(-r.hi.y)), add2(tly, bc2(-r.lo.y)));
  n.rz = add2(add2(thz, bc2(-r.hi.z)), add2(tlz, bc2(-r.lo.z)));
  const float2 q = fma2(n.rz, n.rz, fma2(n.ry, n.ry, mul2(n.rx, n.rx)));
  n.n = make_float2(node_len(q.x), node_len(q.y));
  return n;
}

// seg() for both lanes (same forms, same cut-offs).
__device__ __forceinline__ void seg2(const SegV<float>& r0, const Node2& a, const Node2& b, float g, float2& vx,
                                     float2& vy, float2& vz) {
  const float2 dx = fma2(bc2(r0.y), a.rz, mul2(bc2(-r0.z), a.ry));
  const float2 dy = fma2(bc2(r0.z), a.rx, mul2(bc2(-r0.x), a.rz));
  const float2 dz = fma2(bc2(r0.x), a.ry, mul2(bc2(-r0.y), a.rx));
  const float2 d2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
  const float2 dot12 = fma2(a.rz, b.rz, fma2(a.ry, b.ry, mul2(a.rx, b.rx)));
  const float2 nn = mul2(a.n, b.n);
  const float2 sn = add2(a.n, b.n);
  const float2 tp = add2(nn, dot12);
  const float2 tm = fma2(dot12, bc2(-1.f), nn);
  const bool bx = dot12.x >= 0.f, by = dot12.y >= 0.f;
  const float2 num = mul2(sn, make_float2(bx ? 1.f : tm.x, by ? 1.f : tm.y));
  const float2 den = mul2(nn, make_float2(bx ? tp.x : d2.x, by ? tp.y : d2.y));
  float2 k = mul2(mul2(bc2(g), num), make_float2(nb_rcp(den.x), nb_rcp(den.y)));
  k.x = (d2.x >= (float)kCutD2 && nn.x > 0.f) ? k.x : 0.f;
  k.y = (d2.y >= (float)kCutD2 && nn.y > 0.f) ? k.y : 0.f;
  vx = fma2(k, dx, vx);
  vy = fma2(k, dy, vy);
  vz = fma2(k, dz, vz);
}

template <int H, bool FIRST, bool DO_H>
__device__ __forceinline__ void full_column2(const RecF* col, const Tgt<float> (&tg)[2], Node2 (&prev)[H],
                                             SegV<float> (&ps0)[H], float (&pgS)[H], float2 (&acc)[3]) {
  Node2 cur[H + 1];
  float gS[H], gH[H];
  SegV<float> s0[H], h0[H];
#pragma unroll
  for (int r = 0; r <= H; ++r) {
    const RecF rec = col[r * (kStripCols + 1)];
    if (r < H) rec_fields<float, RecF>(rec, gS[r], gH[r], s0[r], h0[r]);
    cur[r] = node_from2(rec, tg);
  }
  if (DO_H) {
#pragma unroll
    for (int r = 0; r < H; ++r) seg2(h0[r], cur[r], cur[r + 1], gH[r], acc[0], acc[1], acc[2]);
  }
  if (!FIRST) {
#pragma unroll
    for (int r = 0; r < H; ++r) seg2(ps0[r], prev[r], cur[r], pgS[r], acc[0], acc[1], acc[2]);
  }
#pragma unroll
  for (int r = 0; r < H; ++r) {
    pgS[r] = gS[r];
    ps0[r] = s0[r];
    prev[r] = cur[r];
  }
}

// A strip of n_cols node columns, rows padded with zero records.  (Padding the
// columns of narrow strips as well, or walking them unpacked, took up to twice
// the time: FP32, 60,000 points, 20 x 20 rings, 122 -> 96 us.)
template <int H>
__device__ __forceinline__ void walk_cols2(const RecF* sm, int n_cols, bool last_h, const Tgt<float> (&tg)[2],
                                           float (&acc)[2][3]) {
  Node2 prev[H];
  SegV<float> ps0[H];
  float pgS[H];
  float2 a2[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  // a strip has at least two node columns
  full_column2<H, true, true>(sm, tg, prev, ps0, pgS, a2);
#pragma unroll 2
  for (int j = 1; j < n_cols - 1; ++j) full_column2<H, false, true>(sm + j, tg, prev, ps0, pgS, a2);
  if (last_h)
    full_column2<H, false, true>(sm + n_cols - 1, tg, prev, ps0, pgS, a2);
  else
    full_column2<H, false, false>(sm + n_cols - 1, tg, prev, ps0, pgS, a2);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    acc[0][c] += a2[c].x;
    acc[1][c] += a2[c].y;
  }
}

// ------------------------------------------------ FP64 near field
// Near pairs in FP64 (the FP64 form's, and the mixed form's where the context
// asks for it): the near-field arithmetic seg<double> on FP64 records for one
// target, n_cols node columns of H owned rows from `base` (nr rows present; rows
// past them read as zero records), accumulated in FP64.
template <int H>
__device__ __forceinline__ void walk_near64(const RecD* base, int stride, int nr, int n_cols, bool last_h,
                                            const Tgt<double>& tg, double (&acc)[3]) {
  // before the first column stand nodes marked as cut (see walk_near2)
  NodeV<double> prev[H];
  SegV<double> ps0[H];
  double pgS[H];
#pragma unroll
  for (int r = 0; r < H; ++r) {
    prev[r] = NodeV<double>{0.0, 0.0, 0.0, 0.0};
    ps0[r] = SegV<double>{0.0, 0.0, 0.0};
    pgS[r] = 0.0;
  }
#pragma unroll 1
  for (int j = 0; j < n_cols; ++j) {
    const double own = j < n_cols - 1 || last_h ? 1.0 : 0.0;
    NodeV<double> cur[H + 1];
    double gS[H], gH[H];
    SegV<double> s0[H], h0[H];
#pragma unroll
    for (int r = 0; r <= H; ++r) {
      RecD rec;
      if (r < nr) {
        rec = base[(long long)r * stride + j];
      } else {
        rec.a = make_double4(0, 0, 0, 0);
        rec.b = rec.a;
        rec.c = rec.a;
      }
      if (r < H) rec_fields<double, RecD>(rec, gS[r], gH[r], s0[r], h0[r]);
      cur[r] = node_from<double, RecD>(rec, tg);
    }
#pragma unroll
    for (int r = 0; r < H; ++r) {
      seg<double>(h0[r], cur[r], cur[r + 1], own * gH[r], acc[0], acc[1], acc[2]);
      seg<double>(ps0[r], prev[r], cur[r], pgS[r], acc[0], acc[1], acc[2]);
      pgS[r] = gS[r];
      ps0[r] = s0[r];
      prev[r] = cur[r];
    }
  }
}

// Targets tile0 + threadIdx.x + q BLOCK (clamped to the last one) of the
// SoA arrays, as hi/lo FP32 pairs or FP64.
template <class T, int TPT, int BLOCK>
__device__ __forceinline__ void load_targets(const double* __restrict__ tx, const double* __restrict__ ty,
                                             const double* __restrict__ tz, long long base, long long tile0,
                                             long long n_targets, Tgt<T> (&tg)[TPT]) {
#pragma unroll
  for (int q = 0; q < TPT; ++q) {
    long long t = tile0 + threadIdx.x + (long long)q * BLOCK;
    if (t >= n_targets) t = n_targets - 1;  // padded lanes recompute the last target
    const double x = tx[base + t], y = ty[base + t], z = tz[base + t];
    if constexpr (sizeof(T) == 4) {
      tg[q].hx = (float)x; tg[q].hy = (float)y; tg[q].hz = (float)z;
      tg[q].lx = (float)(x - (double)tg[q].hx);
      tg[q].ly = (float)(y - (double)tg[q].hy);
      tg[q].lz = (float)(z - (double)tg[q].hz);
    } else {
      tg[q].hx = x; tg[q].hy = y; tg[q].hz = z;
      tg[q].lx = tg[q].ly = tg[q].lz = 0;
    }
  }
}

}  // namespace
}  // namespace uvlm

#include "nbody_parts.cuh"

namespace uvlm {
namespace {

// Strips [s_begin, s_end) of B for the thread's targets, double-buffered
// through shared memory; FP32 partial sums per strip, FP64 across strips.
// PK: 0 generic walkers, 1 packed FP32x2 walker.
template <class T, class Rec, int H, int TPT, int BLOCK, bool PAD, int PK>
__device__ __forceinline__ void eval_strips(const Blocks& B, long long s_begin, long long s_end,
                                            const Rec* __restrict__ rec, Rec* buf0, Rec* buf1,
                                            const Tgt<T> (&tg)[TPT], double (&accd)[TPT][3], long long s_stride) {
  if (s_begin >= s_end) return;
  StripInfo si = decode_strip<H>(B, s_begin);
  if constexpr (PAD)
    stage_strip_padded<Rec, H>(buf0, rec, si);
  else
    stage_strip<Rec>(buf0, rec, si);
  long long it = 0;
  for (long long s = s_begin; s < s_end; s += s_stride, ++it) {
    Rec* cur = (it & 1) ? buf1 : buf0;
    Rec* nxt = (it & 1) ? buf0 : buf1;
    StripInfo sn;
    const bool has_next = s + s_stride < s_end;
    if (has_next) {
      sn = decode_strip<H>(B, s + s_stride);
      if constexpr (PAD)
        stage_strip_padded<Rec, H>(nxt, rec, sn);
      else
        stage_strip<Rec>(nxt, rec, sn);
      asm volatile("cp.async.wait_group 1;");
    } else {
      asm volatile("cp.async.wait_group 0;");
    }
    __syncthreads();
    T acc[TPT][3];
#pragma unroll
    for (int q = 0; q < TPT; ++q) acc[q][0] = acc[q][1] = acc[q][2] = (T)0;
    if constexpr (PAD && PK == 1 && sizeof(T) == 4 && TPT == 2) {
      walk_cols2<H>(cur, si.n_cols, si.last_h, tg, acc);
    } else if constexpr (PAD)
      walk_full_strip<T, Rec, H, TPT>(cur, si.last_h, tg, acc);
    else
      walk_strip<T, Rec, H, TPT>(cur, si, tg, acc);
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
      accd[q][0] += (double)acc[q][0];
      accd[q][1] += (double)acc[q][1];
      accd[q][2] += (double)acc[q][2];
    }
    __syncthreads();  // everyone done with `cur` before it is refilled
    if (has_next) si = sn;
  }
}

template <class T, class Rec, int H, int TPT, int BLOCK, int MINB, bool PAD, int PK>
__global__ void __launch_bounds__(BLOCK, MINB) nbody_kernel(Blocks B, long long n_strips,
                                                       const double* __restrict__ tx, const double* __restrict__ ty,
                                                       const double* __restrict__ tz, long long n_targets,
                                                       const Rec* __restrict__ rec, double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Rec* buf0 = reinterpret_cast<Rec*>(smem_raw);
  Rec* buf1 = buf0 + (H + 1) * (kStripCols + 1);

  const long long tile0 = (long long)blockIdx.x * BLOCK * TPT;
  Tgt<T> tg[TPT];
  double accd[TPT][3];
  load_targets<T, TPT, BLOCK>(tx, ty, tz, 0, tile0, n_targets, tg);
#pragma unroll
  for (int q = 0; q < TPT; ++q) accd[q][0] = accd[q][1] = accd[q][2] = 0.0;
  // interleaved source strips, as in nbody_parts_kernel
  eval_strips<T, Rec, H, TPT, BLOCK, PAD, PK>(B, (long long)blockIdx.y, n_strips, rec, buf0, buf1, tg, accd,
                                              (long long)gridDim.y);
  store_partial<TPT, BLOCK>(partial + (long long)blockIdx.y * 3 * n_targets, tile0, n_targets, accd);
}

// ------------------------------------------------------ batched evaluation
// Plans of all problems: strips, tiles, splits and the exclusive prefixes of
// items, partial sums and targets.  One CTA; a blockwide scan in chunks.
template <int H, int TPC>
__global__ void __launch_bounds__(256) batch_plan_kernel(const NBodyBatchInput* __restrict__ in, int n,
                                                         NBodyBatchPlan* __restrict__ plan, long long partial_cap,
                                                         bool coarse, long long* totals, int* status) {
  __shared__ long long sh[3][256];
  __shared__ long long carry[3];
  if (threadIdx.x < 3) carry[threadIdx.x] = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 256) {
    const int c = base + threadIdx.x;
    long long v[3] = {0, 0, 0};
    NBodyBatchPlan p{};
    if (c < n) {
      const NBodyBatchInput& x = in[c];
      p.n_strips = fill_parts(p.B, x.blocks, x.n_blocks, H, kMaxParts);
      p.tgt_off = x.tgt_off;
      p.n_tgt = x.n_tgt;
      p.tiles = (p.n_tgt + TPC - 1) / TPC;
      p.splits = batch_splits(p.n_strips, x.blocks, x.n_blocks, coarse);
      v[0] = p.tiles * p.splits;
      v[1] = p.splits * 3 * p.n_tgt;
      v[2] = p.n_tgt;
    }
    for (int k = 0; k < 3; ++k) sh[k][threadIdx.x] = v[k];
    __syncthreads();
    // Hillis-Steele inclusive scan of the three counters
    for (int off = 1; off < 256; off <<= 1) {
      long long t[3];
      for (int k = 0; k < 3; ++k) t[k] = threadIdx.x >= off ? sh[k][threadIdx.x - off] : 0;
      __syncthreads();
      for (int k = 0; k < 3; ++k) sh[k][threadIdx.x] += t[k];
      __syncthreads();
    }
    if (c < n) {
      p.item_off = carry[0] + sh[0][threadIdx.x] - v[0];
      p.part_off = carry[1] + sh[1][threadIdx.x] - v[1];
      p.tgt_prefix = carry[2] + sh[2][threadIdx.x] - v[2];
      plan[c] = p;
    }
    __syncthreads();
    if (threadIdx.x < 3) carry[threadIdx.x] += sh[threadIdx.x][255];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const bool fits = carry[1] <= partial_cap;
    // an over-full plan evaluates and reduces nothing (the status reports it)
    totals[0] = fits ? carry[0] : 0;
    totals[1] = carry[1];
    totals[2] = fits ? carry[2] : 0;
    if (!fits) status[0] = 1;
  }
}

// Last problem whose prefix (member at `Off`) is <= w.
template <class F>
__device__ inline int plan_search(const NBodyBatchPlan* plan, int n, long long w, F key) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (key(plan[mid]) <= w)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

template <class T, class Rec, int h, int TPT, int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) batch_nbody_kernel(const NBodyBatchPlan* __restrict__ plan, int n,
                                                             const long long* __restrict__ totals,
                                                             const double* __restrict__ tx,
                                                             const double* __restrict__ ty,
                                                             const double* __restrict__ tz,
                                                             const Rec* __restrict__ rec,
                                                             double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<PartsSmem<T, Rec, h, BLOCK>*>(smem_raw);
  const long long items = totals[0];
  for (long long w = blockIdx.x; w < items; w += gridDim.x) {
    const int c = plan_search(plan, n, w, [](const NBodyBatchPlan& p) { return p.item_off; });
    const NBodyBatchPlan& P = plan[c];
    const long long local = w - P.item_off;
    const long long tile = local / P.splits, split = local % P.splits;
    const long long tile0 = tile * BLOCK * TPT;
    Tgt<T> tg[TPT];
    double accd[TPT][3];
    load_targets<T, TPT, BLOCK>(tx, ty, tz, P.tgt_off, tile0, P.n_tgt, tg);
#pragma unroll
    for (int q = 0; q < TPT; ++q) accd[q][0] = accd[q][1] = accd[q][2] = 0.0;
    // interleaved source strips (split s: strips s, s + splits, ...), as in
    // nbody_parts_kernel: a tile's near strips spread over its items
    eval_parts<T, Rec, h, TPT, BLOCK, false>(P.B, P.n_strips, (int)P.splits, (int)split, (int)split + 1, rec, nullptr,
                                             sm, tg, accd);
    store_partial<TPT, BLOCK>(partial + P.part_off + split * 3 * P.n_tgt, tile0, P.n_tgt, accd);
  }
}

__global__ void batch_reduce_kernel(const NBodyBatchPlan* __restrict__ plan, int n,
                                    const long long* __restrict__ totals, const double* __restrict__ partial,
                                    double* vx, double* vy, double* vz) {
  const long long total = totals[2];
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const int c = plan_search(plan, n, g, [](const NBodyBatchPlan& p) { return p.tgt_prefix; });
    const NBodyBatchPlan& P = plan[c];
    const long long t = g - P.tgt_prefix;
    double x = 0, y = 0, z = 0;
    for (long long s = 0; s < P.splits; ++s) {
      const double* p = partial + P.part_off + s * 3 * P.n_tgt;
      x += p[t];
      y += p[P.n_tgt + t];
      z += p[2 * P.n_tgt + t];
    }
    vx[P.tgt_off + t] = x;
    vy[P.tgt_off + t] = y;
    vz[P.tgt_off + t] = z;
  }
}

// Batched tiles: rows per lane, targets per thread, CTAs per SM.
constexpr int kBatchBlock = 128;
constexpr int kBatchTptF = 2, kBatchTptD = 1, kBatchHD = 2, kBatchMinB = 3;

__global__ void reduce_partials_kernel(const double* __restrict__ partial, int splits, long long n, double* vx,
                                       double* vy, double* vz, double* aos, const int* __restrict__ perm) {
  const long long n3 = 3 * n;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n3;
       q += (long long)gridDim.x * blockDim.x) {
    double v = 0;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) v += partial[s * n3 + q];
    const int c = (q >= n) + (q >= 2 * n);
    const long long t = q - c * n;
    if (aos)
      aos[3 * (perm ? (long long)perm[t] : t) + c] = v;
    else
      (c == 0 ? vx : c == 1 ? vy : vz)[t] = v;
  }
}

// ------------------------------------------------------------- variants
struct Variant {
  const char* name;
  int prec;  // NBodyPrec
  int H, TPT, BLOCK, MINB;
  int packed;  // 1: FP32x2 near walker (FP32, TPT = 2); 2: the far-field walkers over sheet parts
};

// Tile shapes: H owned node rows per strip (packed = 2: rows per lane of a
// part, two lanes in FP32), TPT targets per thread, BLOCK threads, MINB
// resident CTAs per SM requested from the register allocator.
constexpr Variant kVariants[] = {
    {"fp64_h4_t1_b128", kNBodyFP64, 4, 1, 128, 1, 0},
    {"fp64_h2_t1_b256", kNBodyFP64, 2, 1, 256, 1, 0},
    {"fp32_h4_t1_b256", kNBodyFP32, 4, 1, 256, 2, 0},
    {"fp32_h4_t2_b128", kNBodyFP32, 4, 2, 128, 3, 0},
    {"fp32_h2_t2_b128", kNBodyFP32, 2, 2, 128, 3, 0},
    {"fp32_h4_t1_b128_m4", kNBodyFP32, 4, 1, 128, 4, 0},
    {"fp32_h3_t2_b128_m4", kNBodyFP32, 3, 2, 128, 4, 0},
    {"fp32_h2_t1_b256_m3", kNBodyFP32, 2, 1, 256, 3, 0},
    {"fp64_h2_t2_b128", kNBodyFP64, 2, 2, 128, 1, 0},
    {"fp64_h2_t1_b128_m3", kNBodyFP64, 2, 1, 128, 3, 0},
    {"fp64_h2_t1_b256_m2", kNBodyFP64, 2, 1, 256, 2, 0},
    {"fp32_h3_t2_b128", kNBodyFP32, 3, 2, 128, 3, 0},
    {"fp32_h4_t2_b128_x2", kNBodyFP32, 4, 2, 128, 3, 1},
    {"fp32_h3_t2_b128_x2", kNBodyFP32, 3, 2, 128, 3, 1},
    {"fp32_h2_t2_b128_x2", kNBodyFP32, 2, 2, 128, 3, 1},
    {"fp32_h4_t2_b128_x2f", kNBodyFP32, 4, 2, 128, 2, 2},
    {"fp32_h3_t2_b128_x2f", kNBodyFP32, 3, 2, 128, 3, 2},
    {"fp32_h2_t2_b128_x2f", kNBodyFP32, 2, 2, 128, 3, 2},
    {"fp64_h2_t1_b128_m3f", kNBodyFP64, 2, 1, 128, 3, 2},
    {"fp64_h3_t1_b128_m2f", kNBodyFP64, 3, 1, 128, 2, 2},
    {"fp64_h2_t2_b128_f", kNBodyFP64, 2, 2, 128, 1, 2},
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

// Full-tile (padded) walking pays when the sheets fill most of the padded
// columns: a sheet of C rings per row uses C + chunks of the chunks x
// (kStripCols + 1) staged node columns.
bool use_padded(const Blocks& B) {
  for (int i = 0; i < B.n; ++i) {
    const long long real = B.b[i].cols + B.chunks[i];
    const long long staged = (long long)B.chunks[i] * (kStripCols + 1);
    if (4 * real < 3 * staged) return false;
  }
  return true;
}

// The splits of each target tile's n_strips source strips over CTAs, of which
// `resident` run at a time and which start in the order of their splits.  Each
// split takes half of an even share of the classes that are left, so that the
// CTAs that start last are short and the launch ends evenly although near and
// far strips cost up to three times as much as one another (guided
// self-scheduling).  Equal splits lose up to a whole wave: at 52k targets and
// 134 strips, 8 % between two neighbouring split counts and 30 % where all
// CTAs just fit at once.
SplitTable make_splits(long long tiles, long long n_strips, long long resident, long long most) {
  SplitTable t{};
  most = std::max(1LL, std::min(most, (long long)kMaxSplits));
  // as many classes as leave no more splits than the partial sums have room for
  for (int classes = (int)std::min<long long>(n_strips, kMaxSplits); classes >= 1; --classes) {
    t.n = 0;
    t.classes = classes;
    for (int at = 0; at < classes && t.n < most;) {
      const int left = classes - at;
      const int share = (int)((double)left * (double)tiles / (2.0 * (double)resident));
      at += std::max(1, std::min(share, left));
      t.begin[++t.n] = (unsigned char)at;
    }
    if (t.begin[t.n] == classes) break;
  }
  return t;
}

// Equal splits (the tiles that walk no parts): the number that ends first, a
// whole number of waves of `resident` CTAs at a time, each taking its strips
// plus about a third of one.  cost (where set): the time in strips.
long long choose_splits(long long tiles, long long n_strips, long long resident, long long most,
                        double* cost_out = nullptr) {
  most = std::max(1LL, std::min(most, std::min(n_strips, (long long)kMaxSplits)));
  long long best = 1;
  double best_cost = 1e300;
  for (long long s = 1; s <= most; ++s) {
    const long long waves = (tiles * s + resident - 1) / resident;
    const double cost = (double)waves * ((double)n_strips / (double)s + 0.35) + 0.5 * (double)((n_strips + s - 1) / s);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  if (cost_out) *cost_out = best_cost;
  return best;
}

// The shared-memory limit of a kernel is a per-device attribute: set it once
// on every device this process launches on.
Error set_smem_once(PerDeviceOnce& once, const void* kern, size_t smem) {
  int dev = 0;
  UVLM_CUDA_TRY(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  if (!once_on_device(once, dev, [&] {
        attr_err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return attr_err == cudaSuccess;
      }))
    return fail(kErrCuda, std::string("nbody: the shared-memory attribute could not be set on this device") +
                              (attr_err != cudaSuccess ? std::string(": ") + cudaGetErrorString(attr_err) : ""));
  return ok();
}

Error reduce_partials(const NBodyWork* work, long long splits, long long n_targets, double* vx, double* vy, double* vz,
                      int num_sms, cudaStream_t st) {
  const int rb = 256;
  const int rg = (int)std::min<long long>((3 * n_targets + rb - 1) / rb, (long long)num_sms * 8);
  reduce_partials_kernel<<<rg, rb, 0, st>>>(work->partial, (int)splits, n_targets, vx, vy, vz, work->aos, work->perm);
  UVLM_LAUNCH_CHECK();
  return ok();
}

// Most source splits the caller's scratch allows (0: not even one).
long long most_splits(const NBodyWork* work, long long n_targets) {
  const long long fit = work->partial_cap / (3 * n_targets);
  return work->max_splits > 0 ? std::min(fit, work->max_splits) : fit;
}

template <class T, class Rec, int H, int TPT, int BLOCK, int MINB, int PK = 0>
Error launch_variant(const SourceBlock* blocks, int n_blocks, const double* tx, const double* ty, const double* tz,
                     long long n_targets, const Rec* rec, NBodyWork* work, double* vx, double* vy, double* vz,
                     int num_sms, cudaStream_t st) {
  Blocks B{};
  const long long n_strips = fill_blocks(B, blocks, n_blocks, H);
  // the packed walker takes strips of any width, the generic one padded strips only where most are full
  const bool pad = PK == 1 || use_padded(B);
  auto kern = nbody_kernel<T, Rec, H, TPT, BLOCK, MINB, true, PK>;
  if constexpr (PK != 1)
    if (!pad) kern = nbody_kernel<T, Rec, H, TPT, BLOCK, MINB, false, PK>;
  const size_t smem = 2 * sizeof(Rec) * (H + 1) * (kStripCols + 1);
  static PerDeviceOnce attr_once[2];
  UVLM_TRY(set_smem_once(attr_once[pad ? 1 : 0], (const void*)kern, smem));
  int occ = 0;
  UVLM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BLOCK, smem));
  if (occ < 1) occ = 1;
  const long long tiles = (n_targets + (long long)BLOCK * TPT - 1) / ((long long)BLOCK * TPT);
  const long long most = most_splits(work, n_targets);
  if (most < 1) return fail(kErrCapacity, "nbody partial buffer too small");
  const long long splits = choose_splits(tiles, n_strips, (long long)num_sms * occ, most);
  kern<<<dim3((unsigned)tiles, (unsigned)splits), BLOCK, smem, st>>>(B, n_strips, tx, ty, tz, n_targets, rec,
                                                                     work->partial);
  UVLM_LAUNCH_CHECK();
  return reduce_partials(work, splits, n_targets, vx, vy, vz, num_sms, st);
}

// The far-field walkers (nbody_parts.cuh), h node rows per lane.
template <class T, class Rec, int h, int TPT, int BLOCK, int MINB>
Error launch_parts(const SourceBlock* blocks, int n_blocks, const double* tx, const double* ty, const double* tz,
                   long long n_targets, const Rec* rec, NBodyWork* work, double* vx, double* vy, double* vz,
                   int num_sms, cudaStream_t st) {
  // the mixed form's near pairs in FP64
  constexpr bool kCanNear64 = sizeof(T) == 4;
  const RecD* rec64 = (kCanNear64 && work->near64) ? reinterpret_cast<const RecD*>(work->records64) : nullptr;
  if (kCanNear64 && work->near64 && !rec64) return fail(kErrInvalid, "FP64 near field without FP64 records");
  auto kern = nbody_parts_kernel<T, Rec, h, TPT, BLOCK, MINB, false>;
  if constexpr (kCanNear64)
    if (rec64) kern = nbody_parts_kernel<T, Rec, h, TPT, BLOCK, MINB, true>;
  constexpr size_t smem = sizeof(PartsSmem<T, Rec, h, BLOCK>);
  static PerDeviceOnce attr_once[2];
  UVLM_TRY(set_smem_once(attr_once[rec64 ? 1 : 0], (const void*)kern, smem));
  int occ = 0;
  UVLM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BLOCK, smem));
  if (occ < 1) occ = 1;
  const long long tiles = (n_targets + (long long)BLOCK * TPT - 1) / ((long long)BLOCK * TPT);
  const long long resident = (long long)num_sms * occ;
  const long long most = most_splits(work, n_targets);
  if (most < 1) return fail(kErrCapacity, "nbody partial buffer too small");
  // one part per strip where whole strips would be too few to even out
  PartBlocks B{};
  long long n_strips = fill_parts(B, blocks, n_blocks, h * LaneOf<T>::kLanes, kMaxParts);
  if (tiles * n_strips < 4 * resident) n_strips = fill_parts(B, blocks, n_blocks, h * LaneOf<T>::kLanes, 1);
  const SplitTable split = make_splits(tiles, n_strips, resident, most);
  kern<<<dim3((unsigned)tiles, (unsigned)split.n), BLOCK, smem, st>>>(B, n_strips, tx, ty, tz, n_targets, rec,
                                                                      work->partial, rec64, split);
  UVLM_LAUNCH_CHECK();
  return reduce_partials(work, split.n, n_targets, vx, vy, vz, num_sms, st);
}

}  // namespace

int nbody_num_variants() { return kNumVariants; }
int nbody_variant_prec(int v) { return (v >= 0 && v < kNumVariants) ? kVariants[v].prec : -1; }
bool nbody_variant_far(int v) { return v >= 0 && v < kNumVariants && kVariants[v].packed == 2; }
bool nbody_variant_near64(int v) {
  return v >= 0 && v < kNumVariants && kVariants[v].prec == kNBodyFP32 && kVariants[v].packed == 2 &&
         kVariants[v].TPT == 2;
}
const char* nbody_variant_name(int v) { return (v >= 0 && v < kNumVariants) ? kVariants[v].name : "?"; }

long long nbody_unique_segments(const SourceBlock* blocks, int n_blocks) {
  long long s = 0;
  for (int i = 0; i < n_blocks; ++i) {
    const long long R = blocks[i].node_rows - 1, C = blocks[i].cols;
    if (R < 0) continue;
    s += (long long)blocks[i].num * ((R + 1) * C + R * (C + 1));
  }
  return s;
}

Error nbody_build_sources(const SheetView* views, int n_views, NBodyPrec prec, NBodyWork* work,
                          SourceBlock* blocks, cudaStream_t st) {
  long long off = 0;
  const size_t rsz = prec == kNBodyFP32 ? sizeof(RecF) : sizeof(RecD);
  for (int i = 0; i < n_views; ++i) {
    const SheetView& v = views[i];
    const long long cnt = (long long)v.num * v.node_rows * (v.cols + 1);
    blocks[i] = SourceBlock{off, v.num, v.node_rows, v.cols};
    if ((off + cnt) * (long long)rsz > work->records_cap) return fail(kErrCapacity, "nbody record buffer too small");
    if (cnt > 0) {
      const int bs = 256;
      const int gs = (int)std::min<long long>((cnt + bs - 1) / bs, 4096);
      if (prec == kNBodyFP32)
        build_records_kernel<RecF><<<gs, bs, 0, st>>>(v, reinterpret_cast<RecF*>(work->records) + off);
      else
        build_records_kernel<RecD><<<gs, bs, 0, st>>>(v, reinterpret_cast<RecD*>(work->records) + off);
      UVLM_LAUNCH_CHECK();
      if (prec == kNBodyFP32 && work->near64) {
        // FP64 records of the same nodes for the FP64 near field
        if ((off + cnt) * (long long)sizeof(RecD) > work->records64_cap)
          return fail(kErrCapacity, "nbody FP64 record buffer too small");
        build_records_kernel<RecD><<<gs, bs, 0, st>>>(v, reinterpret_cast<RecD*>(work->records64) + off);
        UVLM_LAUNCH_CHECK();
      }
    }
    off += cnt;
  }
  return ok();
}

Error nbody_eval(const SourceBlock* blocks, int n_blocks, NBodyPrec prec, const double* tx, const double* ty,
                 const double* tz, long long n_targets, double* vx, double* vy, double* vz, NBodyWork* work,
                 int variant, int num_sms, cudaStream_t st) {
  if (n_targets <= 0) return ok();
  if (variant < 0 || variant >= kNumVariants || kVariants[variant].prec != prec)
    return fail(kErrInvalid, "nbody variant does not match precision");
  Blocks none{};
  if (fill_blocks(none, blocks, n_blocks, 1) == 0) {  // no segments
    UVLM_CUDA_TRY(cudaMemsetAsync(vx, 0, sizeof(double) * n_targets, st));
    UVLM_CUDA_TRY(cudaMemsetAsync(vy, 0, sizeof(double) * n_targets, st));
    UVLM_CUDA_TRY(cudaMemsetAsync(vz, 0, sizeof(double) * n_targets, st));
    return ok();
  }
  const RecF* rf = reinterpret_cast<const RecF*>(work->records);
  const RecD* rd = reinterpret_cast<const RecD*>(work->records);
  switch (variant) {
    case 0: return launch_variant<double, RecD, 4, 1, 128, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 1: return launch_variant<double, RecD, 2, 1, 256, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 2: return launch_variant<float, RecF, 4, 1, 256, 2>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 3: return launch_variant<float, RecF, 4, 2, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 4: return launch_variant<float, RecF, 2, 2, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 5: return launch_variant<float, RecF, 4, 1, 128, 4>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 6: return launch_variant<float, RecF, 3, 2, 128, 4>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 7: return launch_variant<float, RecF, 2, 1, 256, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 8: return launch_variant<double, RecD, 2, 2, 128, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 9: return launch_variant<double, RecD, 2, 1, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 10: return launch_variant<double, RecD, 2, 1, 256, 2>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 11: return launch_variant<float, RecF, 3, 2, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 12: return launch_variant<float, RecF, 4, 2, 128, 3, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 13: return launch_variant<float, RecF, 3, 2, 128, 3, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 14: return launch_variant<float, RecF, 2, 2, 128, 3, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 15: return launch_parts<float, RecF, 4, 2, 128, 2>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 16: return launch_parts<float, RecF, 3, 2, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 17: return launch_parts<float, RecF, 2, 2, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rf, work, vx, vy, vz, num_sms, st);
    case 18: return launch_parts<double, RecD, 2, 1, 128, 3>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 19: return launch_parts<double, RecD, 3, 1, 128, 2>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    case 20: return launch_parts<double, RecD, 2, 2, 128, 1>(blocks, n_blocks, tx, ty, tz, n_targets, rd, work, vx, vy, vz, num_sms, st);
    default: return fail(kErrInvalid, "bad nbody variant");
  }

}

}  // namespace uvlm

namespace uvlm {

// FP32 batch tiles the batch autotuner chooses from: the far-field walkers
// with h node rows per lane.
constexpr int kBatchTileH[kNumBatchTilesF] = {3, 2, 4};

const char* nbody_batch_tile_name(NBodyPrec prec, int tile) {
  static const char* names[kNumBatchTilesF] = {"fp32_h3_t2_b128_x2f", "fp32_h2_t2_b128_x2f", "fp32_h4_t2_b128_x2f"};
  if (prec != kNBodyFP32) return "fp64_h2_t1_b128";
  return (tile >= 0 && tile < kNumBatchTilesF) ? names[tile] : "?";
}

long long nbody_batch_partial_doubles(NBodyPrec prec, const NBodyBatchInput* in, int n, bool coarse) {
  // the bound of every tile the batch may run (the fewest rows per strip
  // make the most strips, hence the most source splits)
  long long worst = 0;
  const int tiles = prec == kNBodyFP32 ? kNumBatchTilesF : 1;
  for (int t = 0; t < tiles; ++t) {
    const int H = prec == kNBodyFP32 ? LaneOf<float>::kLanes * kBatchTileH[t] : kBatchHD;
    long long total = 0;
    for (int c = 0; c < n; ++c) {
      PartBlocks B{};
      const long long strips = fill_parts(B, in[c].blocks, in[c].n_blocks, H, kMaxParts);
      const long long splits = batch_splits(strips, in[c].blocks, in[c].n_blocks, coarse);
      total += splits * 3 * in[c].n_tgt;
    }
    worst = std::max(worst, total);
  }
  return worst;
}

namespace {
template <class T, class Rec, int h, int TPT>
int batch_grid_of(int num_sms) {
  const void* k = (const void*)batch_nbody_kernel<T, Rec, h, TPT, kBatchBlock, kBatchMinB>;
  constexpr size_t smem = sizeof(PartsSmem<T, Rec, h, kBatchBlock>);
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kBatchBlock, smem) != cudaSuccess || occ < 1) occ = 1;
  return num_sms * occ;
}

template <class T, class Rec, int h, int TPT>
Error batch_eval(const NBodyBatchInput* d_in, int n, const double* tx, const double* ty, const double* tz,
                 const void* records, double* partial, long long partial_cap, NBodyBatchPlan* d_plan,
                 long long* d_totals, int* status, bool coarse, int grid, cudaStream_t st) {
  batch_plan_kernel<h * LaneOf<T>::kLanes, kBatchBlock * TPT><<<1, 256, 0, st>>>(d_in, n, d_plan, partial_cap, coarse,
                                                                                 d_totals, status);
  UVLM_LAUNCH_CHECK();
  batch_nbody_kernel<T, Rec, h, TPT, kBatchBlock, kBatchMinB>
      <<<grid, kBatchBlock, sizeof(PartsSmem<T, Rec, h, kBatchBlock>), st>>>(
          d_plan, n, d_totals, tx, ty, tz, reinterpret_cast<const Rec*>(records), partial);
  UVLM_LAUNCH_CHECK();
  return ok();
}
}  // namespace

NBodyBatchGrids nbody_batch_grids(NBodyPrec prec, int num_sms) {
  NBodyBatchGrids g;
  if (prec == kNBodyFP32) {
    g.tiles[0] = batch_grid_of<float, RecF, kBatchTileH[0], kBatchTptF>(num_sms);
    g.tiles[1] = batch_grid_of<float, RecF, kBatchTileH[1], kBatchTptF>(num_sms);
    g.tiles[2] = batch_grid_of<float, RecF, kBatchTileH[2], kBatchTptF>(num_sms);
  } else {
    g.fp64 = batch_grid_of<double, RecD, kBatchHD, kBatchTptD>(num_sms);
  }
  return g;
}

Error nbody_batch_eval(NBodyPrec prec, const NBodyBatchInput* d_in, int n, const double* tx, const double* ty,
                       const double* tz, double* vx, double* vy, double* vz, const void* records, double* partial,
                       long long partial_cap, NBodyBatchPlan* d_plan, long long* d_totals, int* status,
                       const NBodyBatchGrids& grids, cudaStream_t st) {
  if (n <= 0) return ok();
  auto run = [&](auto eval, int grid) -> Error {
    UVLM_TRY(eval(d_in, n, tx, ty, tz, records, partial, partial_cap, d_plan, d_totals, status, grids.coarse, grid,
                  st));
    batch_reduce_kernel<<<grid, 256, 0, st>>>(d_plan, n, d_totals, partial, vx, vy, vz);
    UVLM_LAUNCH_CHECK();
    return ok();
  };
  if (prec != kNBodyFP32) return run(batch_eval<double, RecD, kBatchHD, kBatchTptD>, grids.fp64);
  // the FP32 tile the batch's autotuner chose
  switch (grids.tile) {
    case 1: return run(batch_eval<float, RecF, kBatchTileH[1], kBatchTptF>, grids.tiles[1]);
    case 2: return run(batch_eval<float, RecF, kBatchTileH[2], kBatchTptF>, grids.tiles[2]);
    default: return run(batch_eval<float, RecF, kBatchTileH[0], kBatchTptF>, grids.tiles[0]);
  }
}

namespace {
__global__ void arithmetic_kernel(NBodyArith f, const double* __restrict__ x, long long n, double* __restrict__ out) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    out[k] = f == kNBodyRcp ? nb_rcp(x[k]) : f == kNBodySqrt ? nb_sqrt(x[k]) : nb_rsqrt(x[k]);
}
}  // namespace

Error nbody_arithmetic(NBodyArith f, const double* x, long long n, double* out, cudaStream_t st) {
  if (n <= 0) return ok();
  arithmetic_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(f, x, n, out);
  UVLM_LAUNCH_CHECK();
  return ok();
}

// ------------------------------------------------------ arbitrary points
// The far walkers decide per warp, so their speed depends on how close together
// the targets of a warp lie; points that a program hands over in any order are
// first put in the order of a space-filling curve.  Twelve bits: each halves the
// longest edge of the cells (an elongated wake gets most of them along its
// length), the bits of a point's cell in that order are its key, and a stable
// counting sort in two passes of six bits orders the keys, so that the order,
// and with it every rounding, is the same in every run.
//
// One cluster of 8 CTAs does all of it in one launch: histograms per warp, their
// sums over the CTAs through distributed shared memory.  Every warp owns a
// contiguous range of the points and ranks 32 of them at a time.
// FP64, 9001 shuffled points around 3 x 61 x 47 rings: 554 -> 409 us with the
// ordering (about 12 us); FP32, 32768 points, 400 x 128 rings: 4369 -> 2570.
constexpr int kOrderCtas = 8, kOrderThreads = 1024, kOrderWarps = kOrderThreads / 32;
constexpr int kOrderBits = 12, kOrderDigit = 6, kOrderBins = 1 << kOrderDigit;

namespace {
struct OrderSmem {
  int hist[kOrderWarps][kOrderBins];  // counts per warp, then each warp's next position
  int total[kOrderBins];              // counts of this CTA
  int wsum[2];
  int lo[3], hi[3];                   // bounding box as ordered integers
  float scale[3], org[3];
  int bits[3];
  unsigned dims;                      // two bits per key bit: the dimension it halves
};

__device__ __forceinline__ int ordered_int(float x) {
  const int b = __float_as_int(x);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float ordered_float(int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); }

// Lanes whose point has this lane's digit (points past the end: digit -1).
__device__ __forceinline__ void order_count(OrderSmem& sm, int warp, int digit) {
  const unsigned same = __match_any_sync(0xffffffffu, digit);
  if (digit >= 0 && (int)(threadIdx.x & 31) == __ffs(same) - 1) sm.hist[warp][digit] += __popc(same);
  __syncwarp();
}
__device__ __forceinline__ int order_place(OrderSmem& sm, int warp, int digit) {
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xffffffffu, digit);
  const int at = digit >= 0 ? sm.hist[warp][digit] + __popc(same & ((1u << lane) - 1)) : 0;
  __syncwarp();
  if (digit >= 0 && lane == __ffs(same) - 1) sm.hist[warp][digit] += __popc(same);
  __syncwarp();
  return at;
}

// Turns the warps' counts into their first positions.  Every thread of the
// cluster calls it; the counts of this CTA are complete for the calling warp only.
__device__ __forceinline__ void order_scan(cooperative_groups::cluster_group& cl, OrderSmem& sm) {
  const int tid = threadIdx.x, rank = (int)cl.block_rank();
  __syncthreads();
  if (tid < kOrderBins) {
    int s = 0;
    for (int w = 0; w < kOrderWarps; ++w) {
      const int c = sm.hist[w][tid];
      sm.hist[w][tid] = s;
      s += c;
    }
    sm.total[tid] = s;
  }
  cl.sync();
  int first = 0;
  if (tid < kOrderBins) {
    int all = 0;
#pragma unroll
    for (int c = 0; c < kOrderCtas; ++c) {
      const int v = *cl.map_shared_rank(&sm.total[tid], c);
      all += v;
      first += c < rank ? v : 0;
    }
    int scan = all;  // inclusive over the bins of the warp
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, scan, off);
      if ((tid & 31) >= off) scan += v;
    }
    if ((tid & 31) == 31) sm.wsum[tid >> 5] = scan;
    first += scan - all;
  }
  __syncthreads();
  if (tid < kOrderBins) {
    if (tid >= 32) first += sm.wsum[0];
    for (int w = 0; w < kOrderWarps; ++w) sm.hist[w][tid] += first;
  }
  __syncthreads();
}

__global__ void __cluster_dims__(kOrderCtas, 1, 1) __launch_bounds__(kOrderThreads)
    order_points_kernel(const double* __restrict__ x, int n, unsigned short* keys, int* first_order, int* perm,
                        double* __restrict__ tx, double* __restrict__ ty, double* __restrict__ tz) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ OrderSmem sm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_warp = (int)(((long long)n + 32 * kOrderCtas * kOrderWarps - 1) / (32 * kOrderCtas * kOrderWarps)) * 32;
  const long long begin = (long long)per_warp * ((int)cl.block_rank() * kOrderWarps + warp);
  const int i0 = (int)min((long long)n, begin), i1 = (int)min((long long)n, begin + per_warp);
  constexpr int kBatch = 4;  // rows of 32 points whose loads are issued together

  // ---- bounding box of the finite points
  if (tid < 3) {
    sm.lo[tid] = INT_MAX;
    sm.hi[tid] = INT_MIN;
  }
  for (int q = tid; q < kOrderWarps * kOrderBins; q += kOrderThreads) (&sm.hist[0][0])[q] = 0;
  __syncthreads();
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
#pragma unroll 4
  for (int i = i0 + lane; i < i1; i += 32) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float f = (float)x[3LL * i + d];
      if (fabsf(f) < 1e30f) {
        lo[d] = min(lo[d], ordered_int(f));
        hi[d] = max(hi[d], ordered_int(f));
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
    hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
    if (lane == 0) {
      atomicMin(&sm.lo[d], lo[d]);
      atomicMax(&sm.hi[d], hi[d]);
    }
  }
  cl.sync();
  if (warp == 0) {
    float edge[3], org[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int l = lane < kOrderCtas ? *cl.map_shared_rank(&sm.lo[d], lane) : INT_MAX;
      const int h = lane < kOrderCtas ? *cl.map_shared_rank(&sm.hi[d], lane) : INT_MIN;
      const int L = __reduce_min_sync(0xffffffffu, l), H = __reduce_max_sync(0xffffffffu, h);
      org[d] = L <= H ? ordered_float(L) : 0.f;
      edge[d] = L <= H ? ordered_float(H) - org[d] : 0.f;
    }
    if (lane == 0) {
      const float whole[3] = {edge[0], edge[1], edge[2]};
      int bits[3] = {0, 0, 0};
      unsigned dims = 0;
      for (int b = 0; b < kOrderBits; ++b) {
        const int d = edge[0] >= edge[1] && edge[0] >= edge[2] ? 0 : (edge[1] >= edge[2] ? 1 : 2);
        edge[d] *= 0.5f;
        bits[d] += 1;
        dims |= (unsigned)d << (2 * b);
      }
      sm.dims = dims;
      for (int d = 0; d < 3; ++d) {
        sm.bits[d] = bits[d];
        sm.org[d] = org[d];
        sm.scale[d] = whole[d] > 0.f ? (float)(1 << bits[d]) / whole[d] : 0.f;
      }
    }
  }
  __syncthreads();
  const unsigned dims = sm.dims;
  auto key_of = [&](const double (&p)[3]) {
    int q[3], left[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      left[d] = sm.bits[d];
      q[d] = min(max((int)(((float)p[d] - sm.org[d]) * sm.scale[d]), 0), (1 << left[d]) - 1);
    }
    int key = 0;
#pragma unroll
    for (int b = 0; b < kOrderBits; ++b) {
      const int d = dims >> (2 * b) & 3;
      const int l = --(d == 0 ? left[0] : d == 1 ? left[1] : left[2]);
      key = key << 1 | ((d == 0 ? q[0] : d == 1 ? q[1] : q[2]) >> l & 1);
    }
    return key;
  };

  // ---- pass 1: the keys' low digits, in the given order
  for (int r = i0; r < i1; r += 32 * kBatch) {
    double p[kBatch][3];
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
#pragma unroll
      for (int d = 0; d < 3; ++d) p[b][d] = r + 32 * b + lane < i1 ? x[3LL * (r + 32 * b + lane) + d] : 0.0;
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      if (r + 32 * b >= i1) break;
      const bool in = r + 32 * b + lane < i1;
      const int key = key_of(p[b]);
      if (in) keys[r + 32 * b + lane] = (unsigned short)key;
      order_count(sm, warp, in ? key & (kOrderBins - 1) : -1);
    }
  }
  order_scan(cl, sm);
  unsigned short* keys2 = keys + n;
  for (int r = i0; r < i1; r += 32 * kBatch) {
    int key[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) key[b] = r + 32 * b + lane < i1 ? keys[r + 32 * b + lane] : -1;
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      if (r + 32 * b >= i1) break;
      const int at = order_place(sm, warp, key[b] >= 0 ? key[b] & (kOrderBins - 1) : -1);
      if (key[b] >= 0) {
        keys2[at] = (unsigned short)key[b];
        first_order[at] = r + 32 * b + lane;
      }
    }
  }
  cl.sync();  // the first order is complete, and the positions are no longer read

  // ---- pass 2: the high digits, in the first order
  for (int q = tid; q < kOrderWarps * kOrderBins; q += kOrderThreads) (&sm.hist[0][0])[q] = 0;
  __syncthreads();
  for (int r = i0; r < i1; r += 32 * kBatch) {
    int key[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) key[b] = r + 32 * b + lane < i1 ? (int)__ldcg(keys2 + r + 32 * b + lane) : -1;
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      if (r + 32 * b >= i1) break;
      order_count(sm, warp, key[b] >= 0 ? key[b] >> kOrderDigit : -1);
    }
  }
  order_scan(cl, sm);
  for (int r = i0; r < i1; r += 32 * kBatch) {
    int key[kBatch], id[kBatch];
    double p[kBatch][3];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      const int i = r + 32 * b + lane;
      key[b] = i < i1 ? (int)__ldcg(keys2 + i) : -1;
      id[b] = i < i1 ? __ldcg(first_order + i) : 0;
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
#pragma unroll
      for (int d = 0; d < 3; ++d) p[b][d] = x[3LL * id[b] + d];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      if (r + 32 * b >= i1) break;
      const int at = order_place(sm, warp, key[b] >= 0 ? key[b] >> kOrderDigit : -1);
      if (key[b] >= 0) {
        perm[at] = id[b];
        tx[at] = p[b][0];
        ty[at] = p[b][1];
        tz[at] = p[b][2];
      }
    }
  }
  cl.sync();  // no CTA leaves while its counts may be read
}

__global__ void split_points_kernel(const double* __restrict__ a, long long n, double* __restrict__ x,
                                    double* __restrict__ y, double* __restrict__ z) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < 3 * n;
       q += (long long)gridDim.x * blockDim.x) {
    const long long t = q / 3;
    const int c = (int)(q - 3 * t);
    (c == 0 ? x : c == 1 ? y : z)[t] = a[q];
  }
}
}  // namespace

size_t nbody_order_bytes(long long n_targets) { return (size_t)n_targets * 12 + 16; }

// The rule, from shuffled points in and around sheets of 22 to 50,000 segments.
// In order, by the far walkers: FP64 from 2^24 pairs and 1000 segments per target
// on (60 x 60 rings and 3000 points, 106 us in order; 20 x 20 and 60,000, 243 in
// order, 224 by the near walker), FP32 from 2^27 pairs and 2000 segments on
// (3 x 61 x 47 rings and 9001 points, 325 us as given, 227 in order).  Below,
// points in any order leave the far walkers little and cost them their set-up
// and divergence, and the near walkers take every pair: FP64 8 x 36 rings and
// 200,000 points 678 us far, 516 near; but below 2^21 pairs the far walkers'
// narrower strips fill more of the device (8 x 36 and 180 points: 27 us, 37).
constexpr int kNearVariantF64 = 9;  // fp64_h2_t1_b128_m3

// FP32 near tile: the rows per strip whose strips end first, 3 where 2 gain less
// than 3 % (4 would sum more segments in FP32).  A strip costs about its padded
// rows and the row below: 7 node rows take 352 us in three strips of 3, 298 in
// four of 2 (200,000 points, 64 columns); few points want the most strips (400
// points, 50 x 50 rings: 31 and 36 us with 2 and 3 rows).
int nbody_near_variant_f32(const SourceBlock* blocks, int n_blocks, long long n_targets, int num_sms) {
  constexpr int kVariant[2] = {14, 13};  // fp32_h2_t2_b128_x2, fp32_h3_t2_b128_x2
  const long long tiles = (n_targets + 255) / 256;
  double cost[2];
  for (int i = 0; i < 2; ++i) {
    Blocks B{};
    choose_splits(tiles, fill_blocks(B, blocks, n_blocks, i + 2), 3LL * num_sms, kMaxSplits, &cost[i]);
    cost[i] *= i + 3;
  }
  return kVariant[cost[0] < 0.97 * cost[1] ? 0 : 1];
}

Error nbody_eval_points(const SourceBlock* blocks, int n_blocks, NBodyPrec prec, const double* targets,
                        long long n_targets, double* out, NBodyWork* work, double* soa, void* order, int num_sms,
                        cudaStream_t st) {
  if (n_targets <= 0) return ok();
  const long long segs = nbody_unique_segments(blocks, n_blocks);
  if (segs == 0) {
    UVLM_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * 3 * n_targets, st));
    return ok();
  }
  double *tx = soa, *ty = soa + n_targets, *tz = soa + 2 * n_targets;
  const bool f32 = prec == kNBodyFP32;
  const bool sort = n_targets < (1 << 30) && segs >= (f32 ? 2000 : 1000) &&
                    segs >= (1LL << (f32 ? 27 : 24)) / n_targets;
  NBodyWork w = *work;
  w.aos = out;
  w.perm = nullptr;
  if (sort) {
    int* first = reinterpret_cast<int*>(order);
    int* perm = first + n_targets;
    unsigned short* keys = reinterpret_cast<unsigned short*>(perm + n_targets);
    order_points_kernel<<<kOrderCtas, kOrderThreads, 0, st>>>(targets, (int)n_targets, keys, first, perm, tx, ty, tz);
    w.perm = perm;
  } else {
    const int blocks_n = (int)std::min<long long>((3 * n_targets + 255) / 256, (long long)num_sms * 8);
    split_points_kernel<<<blocks_n, 256, 0, st>>>(targets, n_targets, tx, ty, tz);
  }
  UVLM_LAUNCH_CHECK();
  int variant = f32 ? kDefaultVariantF32 : kDefaultVariantF64;
  if (!sort && f32) variant = nbody_near_variant_f32(blocks, n_blocks, n_targets, num_sms);
  if (!sort && !f32 && segs >= (1LL << 21) / n_targets) variant = kNearVariantF64;
  return nbody_eval(blocks, n_blocks, prec, tx, ty, tz, n_targets, nullptr, nullptr, nullptr, &w, variant, num_sms,
                    st);
}

// ------------------------------------------------------------- AoS rings
// Rings that share nothing with each other (the legacy loop's containers): a
// thread keeps one target and walks rings from shared memory, four node
// quantities and four segments each.  Bound: the FP64 pipe, about 165
// operations per ring and target against 13 16-byte shared-memory reads; the
// ring range is split so that about eight CTAs per SM have work (pieces of at
// least kRingTile rings) and the pieces' sums are added in order.  As 1 x 1
// sheets through the strip walkers there was a far-field test for every four
// nodes: a wake advection call with 1088 rings and 3840 targets took 267 us
// (with records, layouts and partial sums in kernels of their own), now 162.
// A ring's segments are summed on their own: they nearly cancel, and added to
// the sum one by one, each rounds at the sum's magnitude.  Opposite segments run
// the same way, so that two rings of a lattice evaluate the segment that they
// share alike and its errors cancel with it.  Error against 80-bit arithmetic, 30
// / 250 rings: 6.0e-16 / 1.0e-15 without either, 3.3e-16 / 6.1e-16 now.
namespace {
constexpr int kRingThreads = 128, kRingTile = 32;

struct alignas(16) RingRec {
  double p[12];   // nodes
  double r0[12];  // segments n0 -> n1, n1 -> n2, n3 -> n2, n0 -> n3
  double g, pad;  // circulation of the walk n0 -> n1 -> n2 -> n3, over 4 pi
};

template <bool CHORDWISE>
__global__ void __launch_bounds__(kRingThreads, 4)
    rings_kernel(const double* __restrict__ rings, const double* __restrict__ gamma, long long n_rings,
                 long long per_split, const double* __restrict__ targets, long long nt, double* __restrict__ partial) {
  __shared__ RingRec sm[kRingTile];
  const long long t = blockIdx.x * (long long)kRingThreads + threadIdx.x;
  const double* x = targets + 3 * (t < nt ? t : nt - 1);
  const double tx = x[0], ty = x[1], tz = x[2];
  const long long begin = blockIdx.y * per_split, end = min(n_rings, begin + per_split);
  double vx = 0, vy = 0, vz = 0;
  for (long long k0 = begin; k0 < end; k0 += kRingTile) {
    const int cnt = (int)min((long long)kRingTile, end - k0);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt * 12; q += kRingThreads) {
      const int r = q / 12, c = q - 12 * r;
      const double* src = rings + 12 * (k0 + r);
      const double a = src[c], b = src[c < 9 ? c + 3 : c - 9];
      sm[r].p[c] = a;
      sm[r].r0[c] = c < 6 ? b - a : a - b;
    }
    if (threadIdx.x < cnt) sm[threadIdx.x].g = -gamma[k0 + threadIdx.x] * (1.0 / (4.0 * kPi));
    __syncthreads();
#pragma unroll 1
    for (int r = 0; r < cnt; ++r) {
      const RingRec& rec = sm[r];
      NodeV<double> n[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        n[k].rx = tx - rec.p[3 * k];
        n[k].ry = ty - rec.p[3 * k + 1];
        n[k].rz = tz - rec.p[3 * k + 2];
        const double q = n[k].rx * n[k].rx + n[k].ry * n[k].ry + n[k].rz * n[k].rz;
        n[k].n = q >= kCutR2 ? nb_sqrt(q) : 0.0;
      }
      const double g = rec.g;
      double rx = 0, ry = 0, rz = 0;
#pragma unroll
      for (int k = 0; k < 4; k += CHORDWISE ? 2 : 1) {
        const int a = k == 2 ? 3 : k == 3 ? 0 : k, b = k == 2 ? 2 : k == 3 ? 3 : k + 1;
        seg<double>(SegV<double>{rec.r0[3 * k], rec.r0[3 * k + 1], rec.r0[3 * k + 2]}, n[a], n[b], k < 2 ? g : -g, rx,
                    ry, rz);
      }
      vx += rx;
      vy += ry;
      vz += rz;
    }
  }
  if (t < nt) {
    double* o = partial + 3 * ((long long)blockIdx.y * nt + t);
    o[0] = vx;
    o[1] = vy;
    o[2] = vz;
  }
}

__global__ void rings_sum_kernel(const double* __restrict__ partial, int splits, long long n3,
                                 const double* __restrict__ add3, const double* base, double scale, double* out) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n3;
       q += (long long)gridDim.x * blockDim.x) {
    double v = 0;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) v += partial[s * n3 + q];
    if (add3) v += add3[q % 3];
    out[q] = base ? base[q] + v * scale : v * scale;
  }
}

// Splits of the ring range: about eight CTAs per SM, pieces of at least one tile.
int rings_splits(long long n_rings, long long n_targets, int num_sms) {
  const long long tiles = ceil_div(n_targets, kRingThreads);
  const long long want = std::max<long long>((8LL * num_sms + tiles - 1) / tiles, 1);
  return (int)std::min<long long>(want, std::max<long long>(ceil_div(n_rings, kRingTile), n_rings > 0));
}

}  // namespace

long long rings_partial_size(long long n_rings, long long n_targets, int num_sms) {
  return 3 * n_targets * rings_splits(n_rings, n_targets, num_sms);
}

Error rings_eval(const double* rings, const double* gamma, long long n_rings, bool chordwise_only,
                 const double* targets, long long n_targets, const double* add3, const double* base, double scale,
                 double* partial, double* out, int num_sms, cudaStream_t st) {
  if (n_targets <= 0) return ok();
  int splits = 0;
  if (n_rings > 0) {
    splits = rings_splits(n_rings, n_targets, num_sms);
    const long long per = (n_rings + splits - 1) / splits;
    const dim3 grid(ceil_div(n_targets, kRingThreads), splits);
    if (chordwise_only)
      rings_kernel<true><<<grid, kRingThreads, 0, st>>>(rings, gamma, n_rings, per, targets, n_targets, partial);
    else
      rings_kernel<false><<<grid, kRingThreads, 0, st>>>(rings, gamma, n_rings, per, targets, n_targets, partial);
    UVLM_LAUNCH_CHECK();
  }
  const int blocks = (int)std::min<long long>((3 * n_targets + 255) / 256, 65535);
  rings_sum_kernel<<<blocks, 256, 0, st>>>(partial, splits, 3 * n_targets, add3, base, scale, out);
  UVLM_LAUNCH_CHECK();
  return ok();
}

}  // namespace uvlm
