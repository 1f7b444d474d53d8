// nbody_parts.cuh -- the far-field N-body walkers over sheet parts.
//
// A source sheet is cut into PARTS of H owned node rows (plus the row below)
// x at most kPartCols segment columns, and a strip is a run of consecutive
// parts that together fill at most kStripSlots node columns: two 32-column
// parts of a wide sheet, or several row groups of a narrow one, so that a
// strip's fixed cost (two block barriers, the far-field set-up) is spread over
// about the same number of segments whatever the sheet's width.
//
// Let a part's nodes all lie within rho of one of them, O, and its segments be
// no longer than l.  Where |x - O| >= rho + l + 1e-3 for a target x, no node is
// cut (|r| >= l + 1e-3), every r1.r2 > 0, and the segment factor of
// src/vortex.cpp:24-38 has one form without cancellation:
//   2 g (|r1| + |r2|) / (|r1||r2| ((|r1| + |r2|)^2 - |r0|^2))
//     = 2 g (1/|r1| + 1/|r2|) / ((|r1| + |r2|)^2 - |r0|^2) = 2 g k.
// With 1/|r| and |r| of every node at hand that is four operations and one
// reciprocal per segment.  The velocity is the sum of 2 g k (r0 x r) with r
// taken at either end of the segment, so the chordwise segment that starts in
// a node and the spanwise segment that ends in it share one cross product:
//   v += (kH (2 gH h0) + kS (2 gS s0)) x r,
// six operations per segment (weighted vectors from shared memory) where a
// cross product and an accumulation of its own for each would take nine.
//
// The reference drops a segment when |r1 x r2|^2 < 1e-10.  Evaluating that
// test for every pair costs as much again as the sum above (the cross product
// of each segment on its own, its square, a compare and a select), so the
// walker decides once per part, segment kind (chordwise, spanwise) and warp
// whether any of its pairs can be cut at all.  With a unit vector u, P the
// projection across u, a <= |r0.u| and e >= |r0 - (r0.u) u| over the part's
// segments of that kind,
//   |r0 x (x - A)| >= a (|P(x - O)| - |P(A - O)|) - e |x - A|,
// and where that exceeds 1.1e-5 for all of the warp's targets nothing is cut
// and the test is left out; elsewhere the walker makes it pair by pair.
//
// FP64 takes this walker from there on.  FP32 does with positions relative to O
// (one subtraction per component) where |x - O| >= 2 rho + 1e-3, so that their
// rounding stays below 1.5 ulp(|r|): the FAR targets; in between, the MIDDLE
// ones, it takes the positions' hi and lo parts (three operations per
// component).  A part that is closer is tested again in blocks of 8 columns,
// and only the blocks that are closer still are left to the near walkers.  With
// the near field in FP64, the pairs of every part that is not far are FP64.
//
// Bound: the FMA pipe (65 % busy in FP32) with the reciprocal unit at 54 %; 12
// warps per SM.  Advection stage of an RK2 step, 52k targets x
// 111k segments, against a pairwise cut-off test and a cross product per
// segment: FP32 10.66 -> 8.69 ms, FP64 (8 x 128 wing, 103k segments) 38.2 ->
// 20.6 ms; at a 50-row wake FP32 0.40 -> 0.40 ms, FP64 0.90 -> 0.59 ms.
//
// FP32: the two lanes of the sm_100 FP32x2 instructions hold two SOURCE rows
// of the part (rows r and r + h), so records are read from shared memory as
// ready-made pairs and only the targets, kept in registers for the whole
// kernel, are duplicated.  FP64: one row per lane, the same code.
#pragma once

#include "nbody.cuh"

namespace uvlm {
namespace {

// ------------------------------------------------------------ lane types
// The walkers' value type: two FP32 source rows (FP32x2 instructions) or one
// FP64 row.  Both are 8 bytes, so shared memory holds them in 16-byte slots
// of two.
template <class T>
struct LaneOf;
template <>
struct LaneOf<float> {
  using V = float2;
  static constexpr int kLanes = 2;
};
template <>
struct LaneOf<double> {
  using V = double;
  static constexpr int kLanes = 1;
};

__device__ __forceinline__ float2 v_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 v_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 v_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 v_neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 v_dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 v_rsq(float2 a) { return make_float2(nb_rsqrt(a.x), nb_rsqrt(a.y)); }
__device__ __forceinline__ float2 v_rcp(float2 a) { return make_float2(nb_rcp(a.x), nb_rcp(a.y)); }
// k where e >= 0, else 0; whether any lane of e is negative
__device__ __forceinline__ float2 v_keep(float2 k, float2 e) {
  return make_float2(e.x >= 0.f ? k.x : 0.f, e.y >= 0.f ? k.y : 0.f);
}
__device__ __forceinline__ bool v_negative(float2 e) {
  return (int)(__float_as_uint(e.x) | __float_as_uint(e.y)) < 0;
}
__device__ __forceinline__ float v_first(float2 a) { return a.x; }
__device__ __forceinline__ float v_second(float2 a) { return a.y; }
__device__ __forceinline__ double v_first(double a) { return a; }
__device__ __forceinline__ double v_second(double a) { return a; }
__device__ __forceinline__ double v_sum(float2 a) { return (double)a.x + (double)a.y; }

__device__ __forceinline__ double v_add(double a, double b) { return a + b; }
__device__ __forceinline__ double v_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double v_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double v_neg(double a) { return -a; }
__device__ __forceinline__ double v_dup(double a) { return a; }
__device__ __forceinline__ double v_rsq(double a) { return nb_rsqrt(a); }
__device__ __forceinline__ double v_rcp(double a) { return nb_rcp(a); }
__device__ __forceinline__ double v_keep(double k, double e) { return e >= 0.0 ? k : 0.0; }
__device__ __forceinline__ bool v_negative(double e) { return __double2hiint(e) < 0; }
__device__ __forceinline__ double v_sum(double a) { return a; }

// A 16-byte shared-memory slot of two values.
template <class V>
struct alignas(16) Slot {
  V a, b;
};
__device__ __forceinline__ Slot<float2> ld_slot(const Slot<float2>* p) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  return Slot<float2>{make_float2(f.x, f.y), make_float2(f.z, f.w)};
}
__device__ __forceinline__ Slot<double> ld_slot(const Slot<double>* p) {
  const double2 f = *reinterpret_cast<const double2*>(p);
  return Slot<double>{f.x, f.y};
}

// Slots of one node column in shared memory: for each of the h rows of a lane
//   0, 1  -(position) (relative to O in FP32, absolute in FP64)
//   2, 3  2 gH h0 and -|h0|^2 of the chordwise segment that starts in the node
//   4, 5  2 gS s0 and -|s0|^2 of the spanwise segment that ends in it
//   6     -(2 gH)^2 and -(2 gS)^2 times the reference's cut-off 1e-10
// and slots 0, 1 of the row below; in FP32 then, for the rows 0 .. h, three
// slots each with the hi and lo parts of -(position).  The vectors' components are rotated
// (a cyclic permutation, which keeps cross products) so that the part's normal
// lies mostly along the last one.
constexpr int kRowSlots = 7;
constexpr int kHiLoSlots = 3;
template <class T, int h>
constexpr int kHiLoAt = kRowSlots * h + 2;
template <class T, int h>
constexpr int kColSlots = kHiLoAt<T, h> + (sizeof(T) == 4 ? kHiLoSlots * (h + 1) : 0);

// Part data the whole block reads after the set-up.
template <class T>
struct PartMeta {
  T o[6];      // O: hi and lo parts (FP32), the position (FP64)
  float u[6];  // unit vectors of the chordwise and the spanwise kind
  int rot;     // component i of the walkers is component (i + rot) % 3
};

// v's components from `rot` on.
template <class V>
__device__ __forceinline__ void rotate3(V (&v)[3], int rot) {
  if (rot == 0) return;
  const V a = v[0], b = v[1], c = v[2];
  v[0] = rot == 1 ? b : c;
  v[1] = rot == 1 ? c : a;
  v[2] = rot == 1 ? a : b;
}
// Per warp that set a part up: rho^2, max |P|^2 across uH and across uS, max
// |2 g|, max e^2 and min a of both kinds, max |r0|^2.
struct alignas(16) PartRed {
  float v[12];
};

template <class T, class Rec, int h, int BLOCK>
struct alignas(16) PartsSmem {
  static constexpr int H = h * LaneOf<T>::kLanes;
  // record buffers: a second one for the next strip where it does not cost a
  // CTA per SM (three of them then, which the registers allow as well)
  static constexpr int kBufs = sizeof(T) == 8 || h <= 2 ? 2 : 1;
  Rec raw[kBufs][(H + 1) * kStripSlots];
  Slot<typename LaneOf<T>::V> loc[kColSlots<T, h> * kStripSlots];
  PartRed red[kMaxParts][BLOCK / 32];
  PartMeta<T> meta[kMaxParts];
  PartInfo info[2][kMaxParts];
  int count[2], width1[2];
};

__device__ __forceinline__ float nb_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void rec_vectors(const RecF& r, float (&s0)[3], float (&h0)[3], float& gS, float& gH) {
  s0[0] = r.sv.x, s0[1] = r.sv.y, s0[2] = r.sv.z;
  h0[0] = r.sv.w, h0[1] = r.hv.x, h0[2] = r.hv.y;
  gS = r.hi.w;
  gH = r.lo.w;
}
__device__ __forceinline__ void rec_vectors(const RecD& r, double (&s0)[3], double (&h0)[3], double& gS, double& gH) {
  s0[0] = r.b.y, s0[1] = r.b.z, s0[2] = r.b.w;
  h0[0] = r.c.x, h0[1] = r.c.y, h0[2] = r.c.z;
  gS = r.a.w;
  gH = r.b.x;
}
// The walker's position of a node (FP32: p - O; FP64: p) and p - O in FP32.
__device__ __forceinline__ void rec_local(const RecF& r, const float (&o)[6], float (&p)[3], float (&l)[3]) {
  l[0] = p[0] = (r.hi.x - o[0]) + (r.lo.x - o[3]);
  l[1] = p[1] = (r.hi.y - o[1]) + (r.lo.y - o[4]);
  l[2] = p[2] = (r.hi.z - o[2]) + (r.lo.z - o[5]);
}
__device__ __forceinline__ void rec_local(const RecD& r, const double (&o)[6], double (&p)[3], float (&l)[3]) {
  p[0] = r.a.x, p[1] = r.a.y, p[2] = r.a.z;
  l[0] = (float)(p[0] - o[0]);
  l[1] = (float)(p[1] - o[1]);
  l[2] = (float)(p[2] - o[2]);
}
__device__ __forceinline__ void rec_origin(const RecF& r, float (&o)[6]) {
  o[0] = r.hi.x, o[1] = r.hi.y, o[2] = r.hi.z, o[3] = r.lo.x, o[4] = r.lo.y, o[5] = r.lo.z;
}
__device__ __forceinline__ void rec_origin(const RecD& r, double (&o)[6]) {
  o[0] = r.a.x, o[1] = r.a.y, o[2] = r.a.z, o[3] = o[4] = o[5] = 0.0;
}
// The walker's coordinates of a target (FP32: x - O; FP64: x) and x - O in FP32.
__device__ __forceinline__ void local_target(const Tgt<float>& t, const float (&o)[6], float (&w)[3], float (&l)[3]) {
  l[0] = w[0] = (t.hx - o[0]) + (t.lx - o[3]);
  l[1] = w[1] = (t.hy - o[1]) + (t.ly - o[4]);
  l[2] = w[2] = (t.hz - o[2]) + (t.lz - o[5]);
}
__device__ __forceinline__ void local_target(const Tgt<double>& t, const double (&o)[6], double (&w)[3],
                                             float (&l)[3]) {
  w[0] = t.hx, w[1] = t.hy, w[2] = t.hz;
  l[0] = (float)(t.hx - o[0]);
  l[1] = (float)(t.hy - o[1]);
  l[2] = (float)(t.hz - o[2]);
}

__device__ __forceinline__ float dot3(const float (&a)[3], const float (&b)[3]) {
  return fmaf(a[2], b[2], fmaf(a[1], b[1], a[0] * b[0]));
}
// |a - au u|^2, the part of a across the unit (or zero) vector u, au = a.u
__device__ __forceinline__ float across2(const float (&a)[3], const float (&u)[3], float au) {
  const float x = fmaf(-au, u[0], a[0]), y = fmaf(-au, u[1], a[1]), z = fmaf(-au, u[2], a[2]);
  return fmaf(z, z, fmaf(y, y, x * x));
}
__device__ __forceinline__ void unit3(float (&u)[3]) {
  const float q = dot3(u, u);
  const float i = q > 0.f ? nb_rsqrt(q) : 0.f;
  u[0] *= i;
  u[1] *= i;
  u[2] *= i;
}

// Warps that share the set-up of a part.
template <int BLOCK>
__device__ __forceinline__ int warps_per_part(int count) {
  constexpr int NW = BLOCK / 32;
  return count == 1 ? NW : (count == 2 ? NW / 2 : 1);
}

// Maxima and minima of non-negative values, taken on their bit patterns: the
// order is the same and a NaN, which is larger than any number there, stays
// visible (every test below then fails, and the part is left to the near
// walker).
__device__ __forceinline__ void keep_max(unsigned& m, float x) { m = max(m, __float_as_uint(x)); }
__device__ __forceinline__ void keep_min(unsigned& m, float x) { m = min(m, __float_as_uint(x)); }

// Set-up of the staged strip: the walkers' slots of every part and the bounds
// of its far and cut-off tests.
template <class T, class Rec, int h, int BLOCK>
__device__ __forceinline__ void parts_prepare(PartsSmem<T, Rec, h, BLOCK>& sm, int cur) {
  constexpr int kBufs = PartsSmem<T, Rec, h, BLOCK>::kBufs;
  using V = typename LaneOf<T>::V;
  constexpr int L = LaneOf<T>::kLanes, H = h * L;
  const int count = sm.count[cur], w1 = sm.width1[cur];
  const int wpp = warps_per_part<BLOCK>(count);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = warp % wpp;
#pragma unroll 1
  for (int p = warp / wpp; p < count; p += (BLOCK / 32) / wpp) {
    const int nr = sm.info[cur][p].nr, nc = sm.info[cur][p].nc;
    const bool last_h = sm.info[cur][p].last_h != 0;
    const Rec* raw = sm.raw[cur % kBufs] + (H + 1) * w1 * p;
    Slot<V>* loc = sm.loc + kColSlots<T, h> * w1 * p;
    T o[6];
    float uH[3], uS[3];
    {
      const Rec& ro = raw[((nr - 1) >> 1) * w1 + ((nc - 1) >> 1)];
      T s0[3], h0[3], gS, gH;
      rec_origin(ro, o);
      rec_vectors(ro, s0, h0, gS, gH);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        uH[d] = (float)h0[d];
        uS[d] = (float)s0[d];
      }
      unit3(uH);
      unit3(uS);
    }
    // the component with most of the normal uH x uS becomes the last one
    const float nx = fabsf(uH[1] * uS[2] - uH[2] * uS[1]), ny = fabsf(uH[2] * uS[0] - uH[0] * uS[2]),
                nz = fabsf(uH[0] * uS[1] - uH[1] * uS[0]);
    const int rot = nz >= nx && nz >= ny ? 0 : (nx >= ny ? 1 : 2);
    unsigned rho2 = 0, pH2 = 0, pS2 = 0, gm = 0, eH2 = 0, eS2 = 0, l2 = 0;
    unsigned aH = __float_as_uint(1e30f), aS = aH;
    for (int e = sub * 32 + lane; e < (h + 1) * nc; e += wpp * 32) {
      const int r = e / nc, j = e - r * nc;
      T f[L][kRowSlots * 2], hl[L][kHiLoSlots * 2];
#pragma unroll
      for (int l = 0; l < L; ++l) {
        const int R = r + l * h;
#pragma unroll
        for (int i = 0; i < kRowSlots * 2; ++i) f[l][i] = (T)0;
        if constexpr (sizeof(T) == 4) {
          T hi[3] = {o[0], o[1], o[2]}, lo[3] = {o[3], o[4], o[5]};
          if (R < nr) {
            const Rec& rec = raw[R * w1 + j];
            hi[0] = rec.hi.x, hi[1] = rec.hi.y, hi[2] = rec.hi.z;
            lo[0] = rec.lo.x, lo[1] = rec.lo.y, lo[2] = rec.lo.z;
          }
          rotate3(hi, rot);
          rotate3(lo, rot);
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            hl[l][d] = -hi[d];
            hl[l][3 + d] = -lo[d];
          }
        }
        // rows past the sheet sit at O, a finite distance away, with zero strengths
        T pos[3] = {(T)0, (T)0, (T)0}, bH[3] = {(T)0, (T)0, (T)0}, bS[3] = {(T)0, (T)0, (T)0};
        if constexpr (sizeof(T) == 8) pos[0] = o[0], pos[1] = o[1], pos[2] = o[2];
        if (R < nr) {
          const Rec rec = raw[R * w1 + j];
          float lp[3];
          rec_local(rec, o, pos, lp);
          keep_max(rho2, dot3(lp, lp));
          keep_max(pH2, across2(lp, uH, dot3(lp, uH)));
          keep_max(pS2, across2(lp, uS, dot3(lp, uS)));
          if (r < h) {
            T s0[3], h0[3], gS, gH;
            rec_vectors(rec, s0, h0, gS, gH);
            const T g = (j < nc - 1 || last_h) ? gH + gH : (T)0;
            if (g != (T)0) {
              const float v[3] = {(float)h0[0], (float)h0[1], (float)h0[2]};
              const float a = dot3(v, uH);
              keep_min(aH, fabsf(a));
              keep_max(eH2, across2(v, uH, a));
              keep_max(gm, fabsf((float)g));
            }
            bH[0] = g * h0[0], bH[1] = g * h0[1], bH[2] = g * h0[2];
            f[l][7] = -(h0[0] * h0[0] + h0[1] * h0[1] + h0[2] * h0[2]);
            keep_max(l2, (float)-f[l][7]);
            f[l][12] = -(g * g * (T)kCutD2);
            if (j > 0) {
              T gHl;
              rec_vectors(raw[R * w1 + j - 1], s0, h0, gS, gHl);
              const T gs = gS + gS;
              if (gs != (T)0) {
                const float v[3] = {(float)s0[0], (float)s0[1], (float)s0[2]};
                const float a = dot3(v, uS);
                keep_min(aS, fabsf(a));
                keep_max(eS2, across2(v, uS, a));
                keep_max(gm, fabsf((float)gs));
              }
              bS[0] = gs * s0[0], bS[1] = gs * s0[1], bS[2] = gs * s0[2];
              f[l][11] = -(s0[0] * s0[0] + s0[1] * s0[1] + s0[2] * s0[2]);
              keep_max(l2, (float)-f[l][11]);
              f[l][13] = -(gs * gs * (T)kCutD2);
            }
          }
        }
        rotate3(pos, rot);
        rotate3(bH, rot);
        rotate3(bS, rot);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          f[l][d] = -pos[d];
          f[l][4 + d] = bH[d];
          f[l][8 + d] = bS[d];
        }
      }
      Slot<V>* out = loc + kColSlots<T, h> * j + kRowSlots * r;
#pragma unroll
      for (int i = 0; i < kRowSlots; ++i) {
        if (i < 2 || r < h) {
          if constexpr (L == 2)
            *reinterpret_cast<float4*>(out + i) =
                make_float4(f[0][2 * i], f[L - 1][2 * i], f[0][2 * i + 1], f[L - 1][2 * i + 1]);
          else
            *reinterpret_cast<double2*>(out + i) = make_double2(f[0][2 * i], f[0][2 * i + 1]);
        }
      }
      if constexpr (L == 2) {
        out = loc + kColSlots<T, h> * j + kHiLoAt<T, h> + kHiLoSlots * r;
#pragma unroll
        for (int i = 0; i < kHiLoSlots; ++i)
          *reinterpret_cast<float4*>(out + i) =
              make_float4(hl[0][2 * i], hl[L - 1][2 * i], hl[0][2 * i + 1], hl[L - 1][2 * i + 1]);
      }
    }
    rho2 = __reduce_max_sync(0xffffffffu, rho2);
    pH2 = __reduce_max_sync(0xffffffffu, pH2);
    pS2 = __reduce_max_sync(0xffffffffu, pS2);
    gm = __reduce_max_sync(0xffffffffu, gm);
    eH2 = __reduce_max_sync(0xffffffffu, eH2);
    eS2 = __reduce_max_sync(0xffffffffu, eS2);
    aH = __reduce_min_sync(0xffffffffu, aH);
    aS = __reduce_min_sync(0xffffffffu, aS);
    l2 = __reduce_max_sync(0xffffffffu, l2);
    if (lane == 0) {
      uint4* d = reinterpret_cast<uint4*>(sm.red[p][sub].v);
      d[0] = make_uint4(rho2, pH2, pS2, gm);
      d[1] = make_uint4(eH2, eS2, aH, aS);
      d[2] = make_uint4(l2, 0u, 0u, 0u);
      if (sub == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) sm.meta[p].o[q] = o[q];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          sm.meta[p].u[q] = uH[q];
          sm.meta[p].u[3 + q] = uS[q];
        }
        sm.meta[p].rot = rot;
      }
    }
  }
}

constexpr float kPartsReach2 = 1e30f;  // square of the distance from which on the near walkers take every pair

// The tests of one part for this warp's targets; ts receives the walker's
// target coordinates.  Bit 0: far; bit 1: chordwise pairs may be cut; bit 2:
// spanwise pairs may be cut; bit 3: at least middle; bit 4: strengths that the
// pairwise cut-off test can square.  Warp-uniform.  longest: the part's longest
// segment.  The FP32 roundings of
// the projections stay below 1e-6 (|x - O| + rho), which the test gives away.
// Left to the near walkers, which have no such limits: a part of strengths whose
// squares would leave the FP32 range (|2 g| < 1e-13 everywhere, or above 1e15),
// and pairs at or above a distance of 1e15, whose squares and their products do
// (a part's radius and longest segment are then below that too).
template <class T, class Rec, int h, int BLOCK, int TPT>
__device__ __forceinline__ unsigned parts_test(const PartsSmem<T, Rec, h, BLOCK>& sm, int p, int wpp,
                                               const Tgt<T> (&tg)[TPT], typename LaneOf<T>::V (&ts)[TPT][3],
                                               float& longest) {
  uint4 x = *reinterpret_cast<const uint4*>(&sm.red[p][0].v[0]);
  uint4 y = *reinterpret_cast<const uint4*>(&sm.red[p][0].v[4]);
  for (int s = 1; s < wpp; ++s) {
    const uint4 a = *reinterpret_cast<const uint4*>(&sm.red[p][s].v[0]);
    const uint4 b = *reinterpret_cast<const uint4*>(&sm.red[p][s].v[4]);
    x = make_uint4(max(x.x, a.x), max(x.y, a.y), max(x.z, a.z), max(x.w, a.w));
    y = make_uint4(max(y.x, b.x), max(y.y, b.y), min(y.z, b.z), min(y.w, b.w));
  }
  unsigned l2 = __float_as_uint(sm.red[p][0].v[8]);
  for (int s = 1; s < wpp; ++s) l2 = max(l2, __float_as_uint(sm.red[p][s].v[8]));
  T o[6];
#pragma unroll
  for (int d = 0; d < 6; ++d) o[d] = sm.meta[p].o[d];
  const float uH[3] = {sm.meta[p].u[0], sm.meta[p].u[1], sm.meta[p].u[2]};
  const float uS[3] = {sm.meta[p].u[3], sm.meta[p].u[4], sm.meta[p].u[5]};
  const float rho = nb_sqrt(__uint_as_float(x.x)), pH = nb_sqrt(__uint_as_float(x.y)),
              pS = nb_sqrt(__uint_as_float(x.z)), gm = __uint_as_float(x.w);
  const float eH = 1.001f * nb_sqrt(__uint_as_float(y.x)), eS = 1.001f * nb_sqrt(__uint_as_float(y.y));
  const float aH = 0.999f * __uint_as_float(y.z), aS = 0.999f * __uint_as_float(y.w);
  const float lim2 = 1.000002f * (rho + nb_sqrt(__uint_as_float(l2))) + 1e-3f;
  const float lim = sizeof(T) == 8 ? lim2 : 2.000001f * rho + 1e-3f;
  const bool strong = gm == 0.f || (gm >= 1e-13f && gm <= 1e15f);
  bool far = strong, mid = strong, freeH = true, freeS = true;
#pragma unroll
  for (int q = 0; q < TPT; ++q) {
    T w[3];
    float l[3];
    local_target(tg[q], o, w, l);
    rotate3(w, sm.meta[p].rot);
#pragma unroll
    for (int d = 0; d < 3; ++d) ts[q][d] = v_dup(w[d]);
    const float t2 = dot3(l, l);
    far = far && t2 >= lim * lim && t2 < kPartsReach2;
    mid = mid && t2 >= lim2 * lim2 && t2 < kPartsReach2;
    const float reach = nb_sqrt(t2) + rho;
    const float tH = nb_sqrt(across2(l, uH, dot3(l, uH))), tS = nb_sqrt(across2(l, uS, dot3(l, uS)));
    freeH = freeH && aH * (tH - pH - 1e-6f * reach) - eH * reach > 1.1e-5f;
    freeS = freeS && aS * (tS - pS - 1e-6f * reach) - eS * reach > 1.1e-5f;
  }
  const unsigned bits = (far ? 1u : 0u) | (freeH ? 2u : 0u) | (freeS ? 4u : 0u) | (mid ? 8u : 0u) | (strong ? 16u : 0u);
  longest = nb_sqrt(__uint_as_float(l2));
  return __reduce_and_sync(0xffffffffu, bits) ^ 6u;
}

// v += w x r
template <class V>
__device__ __forceinline__ void add_cross(const V (&w)[3], const V (&r)[3], V (&v)[3]) {
  v[0] = v_fma(v_neg(w[2]), r[1], v_fma(w[1], r[2], v[0]));
  v[1] = v_fma(v_neg(w[0]), r[2], v_fma(w[2], r[0], v[1]));
  v[2] = v_fma(v_neg(w[1]), r[0], v_fma(w[0], r[1], v[2]));
}

// The pairwise cut-off of segments b at r for all of the thread's targets:
// k = 0 where |b x r|^2 < thr (nthr = -thr).  The last component alone, which
// is the largest for targets spread out in the plane of a sheet, usually shows
// that no lane of the warp is below; the other two are formed when it does not.
template <class V, int TPT>
__device__ __forceinline__ void cut_pairs(const V (&b)[3], const V (&r)[TPT][3], V nthr, V (&k)[TPT]) {
  V e[TPT];
  bool small = false;
#pragma unroll
  for (int q = 0; q < TPT; ++q) {
    const V dz = v_fma(v_neg(b[1]), r[q][0], v_mul(b[0], r[q][1]));
    e[q] = v_fma(dz, dz, nthr);
    small = small || v_negative(e[q]);
  }
  if (__any_sync(0xffffffffu, small)) {
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
      const V dx = v_fma(v_neg(b[2]), r[q][1], v_mul(b[1], r[q][2]));
      const V dy = v_fma(v_neg(b[0]), r[q][2], v_mul(b[2], r[q][0]));
      k[q] = v_keep(k[q], v_fma(dy, dy, v_fma(dx, dx, e[q])));
    }
  }
}

// 1 / d for the thread's targets.
template <class V, int TPT>
__device__ __forceinline__ void v_rcps(V (&d)[TPT]) {
#pragma unroll
  for (int q = 0; q < TPT; ++q) d[q] = v_rcp(d[q]);
}

// One node column of a far part: the nodes of its rows, the chordwise segments
// between them and the spanwise segments that end in them (a part's first
// column has zero vectors there).  pn and pv hold |r| and 1/|r| of the previous
// column's nodes and receive this column's.
// TH, TS: the chordwise / spanwise segments need the pairwise cut-off test.
// MID (FP32): positions from their hi and lo parts (tl: the targets' lo parts).
// BLOCKS: own_s and own_h are 0 where the spanwise segments belong to the block
// of columns before or the chordwise ones to the block after, else 1.
template <class T, int h, int TPT, bool TH, bool TS, bool MID, bool BLOCKS>
__device__ __forceinline__ void far_col(const Slot<typename LaneOf<T>::V>* col,
                                        const typename LaneOf<T>::V (&ts)[TPT][3],
                                        const typename LaneOf<T>::V (&tl)[TPT][3],
                                        typename LaneOf<T>::V (&pn)[TPT][h], typename LaneOf<T>::V (&pv)[TPT][h],
                                        typename LaneOf<T>::V (&acc)[TPT][3], T own_s, T own_h) {
  using V = typename LaneOf<T>::V;
  V un[TPT], uv[TPT], ur[TPT][3], kS[TPT], C[3];
#pragma unroll
  for (int r = 0; r <= h; ++r) {
    const Slot<V>* s = col + kRowSlots * r;
    V n[TPT], v[TPT], x[TPT][3];
    if constexpr (MID) {
      const Slot<V>* m = col + kHiLoAt<T, h> + kHiLoSlots * r;
      const Slot<V> m0 = ld_slot(m), m1 = ld_slot(m + 1), m2 = ld_slot(m + 2);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        x[q][0] = v_add(v_add(ts[q][0], m0.a), v_add(tl[q][0], m1.b));
        x[q][1] = v_add(v_add(ts[q][1], m0.b), v_add(tl[q][1], m2.a));
        x[q][2] = v_add(v_add(ts[q][2], m1.a), v_add(tl[q][2], m2.b));
      }
    } else {
      const Slot<V> a0 = ld_slot(s), a1 = ld_slot(s + 1);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        x[q][0] = v_add(ts[q][0], a0.a);
        x[q][1] = v_add(ts[q][1], a0.b);
        x[q][2] = v_add(ts[q][2], a1.a);
      }
    }
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
      const V q2 = v_fma(x[q][2], x[q][2], v_fma(x[q][1], x[q][1], v_mul(x[q][0], x[q][0])));
      v[q] = v_rsq(q2);
      n[q] = v_mul(q2, v[q]);
    }
    if (r > 0) {
      // the chordwise segment of the row above, and that row's sum
      const Slot<V> b0 = ld_slot(s - kRowSlots + 2), b1 = ld_slot(s - kRowSlots + 3);
      const V B[3] = {b0.a, b0.b, b1.a};
      V kH[TPT];
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        const V sn = v_add(un[q], n[q]);
        kH[q] = v_fma(sn, sn, b1.b);
      }
      v_rcps<V, TPT>(kH);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        kH[q] = v_mul(v_add(uv[q], v[q]), kH[q]);
        if (BLOCKS) kH[q] = v_mul(kH[q], v_dup(own_h));
      }
      if (TH) cut_pairs<V, TPT>(B, ur, ld_slot(s - kRowSlots + 6).a, kH);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        V w[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) w[c] = v_fma(kH[q], B[c], v_mul(kS[q], C[c]));
        add_cross<V>(w, ur[q], acc[q]);
      }
    }
    if (r < h) {
      const Slot<V> c0 = ld_slot(s + 4), c1 = ld_slot(s + 5);
      C[0] = c0.a, C[1] = c0.b, C[2] = c1.a;
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        const V sn = v_add(pn[q][r], n[q]);
        kS[q] = v_fma(sn, sn, c1.b);
      }
      v_rcps<V, TPT>(kS);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        kS[q] = v_mul(v_add(pv[q][r], v[q]), kS[q]);
        if (BLOCKS) kS[q] = v_mul(kS[q], v_dup(own_s));
      }
      if (TS) cut_pairs<V, TPT>(C, x, ld_slot(s + 6).b, kS);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        pn[q][r] = un[q] = n[q];
        pv[q][r] = uv[q] = v[q];
#pragma unroll
        for (int c = 0; c < 3; ++c) ur[q][c] = x[q][c];
      }
    }
  }
}

// Columns [0, nc) at loc: a part, or (BLOCKS) some of its blocks, without the
// chordwise segments of the last column where they are the next block's.  The
// nodes before the first column sit at a made-up distance of 1, which nothing
// depends on.
template <class T, int h, int TPT, bool TH, bool TS, bool MID = false, bool BLOCKS = false>
__device__ __forceinline__ void far_part(const Slot<typename LaneOf<T>::V>* loc, int nc,
                                         const typename LaneOf<T>::V (&ts)[TPT][3],
                                         const typename LaneOf<T>::V (&tl)[TPT][3],
                                         typename LaneOf<T>::V (&acc)[TPT][3], bool end = true) {
  using V = typename LaneOf<T>::V;
  V pn[TPT][h], pv[TPT][h];
#pragma unroll
  for (int q = 0; q < TPT; ++q)
#pragma unroll
    for (int r = 0; r < h; ++r) pn[q][r] = pv[q][r] = v_dup((T)1);
#pragma unroll 1
  for (int j = 0; j < nc; ++j, loc += kColSlots<T, h>)
    far_col<T, h, TPT, TH, TS, MID, BLOCKS>(loc, ts, tl, pn, pv, acc, j > 0 ? (T)1 : (T)0,
                                            j < nc - 1 || end ? (T)1 : (T)0);
}

// Whether all of the warp's targets are at least middle for the columns
// [0, nc) at loc alone (a block of a part that is near as a whole): the radius
// about the block's middle node from the slots' positions, whose FP32 rounding
// the factor 1.00001 covers, then the test against it.  l: the part's longest
// segment; ts: the walker's target coordinates.  Warp-uniform.
template <class T, int h, int TPT>
__device__ __forceinline__ bool block_mid(const Slot<typename LaneOf<T>::V>* loc, int nc, float l,
                                          const typename LaneOf<T>::V (&ts)[TPT][3]) {
  const Slot<typename LaneOf<T>::V>* oc = loc + kColSlots<T, h> * (nc >> 1) + kRowSlots * (h >> 1);
  const auto o0 = ld_slot(oc), o1 = ld_slot(oc + 1);
  const T o[3] = {v_first(o0.a), v_first(o0.b), v_first(o1.a)};  // minus the position
  unsigned rho2 = 0;
  for (int e = threadIdx.x & 31; e < (h + 1) * nc; e += 32) {
    const int r = e / nc, j = e - r * nc;
    const auto p0 = ld_slot(loc + kColSlots<T, h> * j + kRowSlots * r);
    const auto p1 = ld_slot(loc + kColSlots<T, h> * j + kRowSlots * r + 1);
    const float a[3] = {(float)(v_first(p0.a) - o[0]), (float)(v_first(p0.b) - o[1]), (float)(v_first(p1.a) - o[2])};
    const float b[3] = {(float)(v_second(p0.a) - o[0]), (float)(v_second(p0.b) - o[1]),
                        (float)(v_second(p1.a) - o[2])};
    keep_max(rho2, dot3(a, a));
    keep_max(rho2, dot3(b, b));
  }
  const float lim = 1.00001f * (nb_sqrt(__uint_as_float(__reduce_max_sync(0xffffffffu, rho2))) + l) + 1e-3f;
  bool mid = true;
#pragma unroll
  for (int q = 0; q < TPT; ++q) {
    const float t[3] = {(float)(v_first(ts[q][0]) + o[0]), (float)(v_first(ts[q][1]) + o[1]),
                        (float)(v_first(ts[q][2]) + o[2])};
    const float t2 = dot3(t, t);
    mid = mid && t2 >= lim * lim && t2 < kPartsReach2;
  }
  return __all_sync(0xffffffffu, mid);
}
constexpr int kBlockCols = 8;  // segment columns of a block of a near part

// Near parts: the record walkers of nbody.cu on the staged records, HN node rows
// at a time; rows past the sheet read as zero records.  One body serves every
// column (a part's walkers together have to stay in the instruction cache: four
// bodies here, for the first, the inner and the two kinds of last column, made
// near parts 1.3 times slower): before the first column stand nodes marked as
// cut, and the last one's chordwise strengths are zero where it does not own
// them.  The body is there twice, so that a column's nodes become the previous
// ones without copies: four wings of 16 x 64 at 300 wake rows, advection of a
// step 27.8 -> 26.1 ms (26.8 before the parts), 32 x 128 at 400 rows 8.98 -> 8.69;
// three times: 26.3 and 8.88; 4 rows at a time instead: 27.3 and 8.77.
template <int HN>
__device__ __forceinline__ void walk_near2(const RecF* base, int stride, int nr, int nc, bool last_h,
                                           const Tgt<float> (&tg)[2], float2 (&acc)[3]) {
  Node2 prev[HN];
  SegV<float> ps0[HN];
  float pgS[HN];
#pragma unroll
  for (int r = 0; r < HN; ++r) {
    prev[r].rx = prev[r].ry = prev[r].rz = prev[r].n = make_float2(0.f, 0.f);
    ps0[r] = SegV<float>{0.f, 0.f, 0.f};
    pgS[r] = 0.f;
  }
#pragma unroll 2
  for (int j = 0; j < nc; ++j) {
    const RecF* col = base + j;
    const float own = j < nc - 1 || last_h ? 1.f : 0.f;
    Node2 cur[HN + 1];
    float gS[HN], gH[HN];
    SegV<float> s0[HN], h0[HN];
#pragma unroll
    for (int r = 0; r <= HN; ++r) {
      RecF rec;
      if (r < nr) {
        rec = col[r * stride];
      } else {
        rec.hi = make_float4(0.f, 0.f, 0.f, 0.f);
        rec.lo = rec.sv = rec.hv = rec.hi;
      }
      if (r < HN) rec_fields<float, RecF>(rec, gS[r], gH[r], s0[r], h0[r]);
      cur[r] = node_from2(rec, tg);
    }
#pragma unroll
    for (int r = 0; r < HN; ++r) {
      seg2(h0[r], cur[r], cur[r + 1], own * gH[r], acc[0], acc[1], acc[2]);
      seg2(ps0[r], prev[r], cur[r], pgS[r], acc[0], acc[1], acc[2]);
      pgS[r] = gS[r];
      ps0[r] = s0[r];
      prev[r] = cur[r];
    }
  }
}

// Near columns [0, nc) of a part (base: the record of its first node there)
// for the thread's targets, accumulated in FP64 after every HN rows.
template <int HN, int H>
__device__ __forceinline__ void near_fp32(const RecF* base, int stride, int nr, int nc, bool last_h,
                                          const Tgt<float> (&tg)[2], double (&accd)[2][3]) {
#pragma unroll 1
  for (int r0 = 0; r0 < H && r0 < nr; r0 += HN) {
    float2 a[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    walk_near2<HN>(base + (long long)r0 * stride, stride, nr - r0, nc, last_h, tg, a);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      accd[0][c] += (double)a[c].x;
      accd[1][c] += (double)a[c].y;
    }
  }
}

template <int HN, int H, class T, int TPT>
__device__ __forceinline__ void near_fp64(const RecD* base, int stride, int nr, int nc, bool last_h,
                                          const Tgt<T> (&tg)[TPT], double (&accd)[TPT][3]) {
#pragma unroll 1
  for (int q = 0; q < TPT; ++q) {
    Tgt<double> td;
    td.hx = (double)tg[q].hx + (double)tg[q].lx;
    td.hy = (double)tg[q].hy + (double)tg[q].ly;
    td.hz = (double)tg[q].hz + (double)tg[q].lz;
    td.lx = td.ly = td.lz = 0.0;
    double a[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int r0 = 0; r0 < H && r0 < nr; r0 += HN)
      walk_near64<HN>(base + (long long)r0 * stride, stride, nr - r0, nc, last_h, td, a);
#pragma unroll
    for (int c = 0; c < 3; ++c) accd[q][c] += a[c];
  }
}

// cp.async staging of the records of a strip.
template <class T, class Rec, int h, int BLOCK>
__device__ __forceinline__ void parts_stage(PartsSmem<T, Rec, h, BLOCK>& sm, int buf, const Rec* __restrict__ rec) {
  constexpr int H = h * LaneOf<T>::kLanes, kChunks = sizeof(Rec) / 16;
  const int count = sm.count[buf], w1 = sm.width1[buf];
  const int total = count * (H + 1) * w1 * kChunks;
  for (int q = threadIdx.x; q < total; q += BLOCK) {
    const int slot = q / kChunks, piece = q - slot * kChunks;
    const int pr = slot / w1, j = slot - pr * w1;
    const int p = pr / (H + 1), r = pr - p * (H + 1);
    const PartInfo& pi = sm.info[buf][p];
    if (r < pi.nr && j < pi.nc) {
      const char* src = reinterpret_cast<const char*>(rec + pi.first + (long long)r * pi.stride + j) + 16 * piece;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(
          reinterpret_cast<char*>(sm.raw[buf % PartsSmem<T, Rec, h, BLOCK>::kBufs] + slot) + 16 * piece);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// The strips s < n with s mod stride in [begin, end), for the thread's
// targets.  Per strip: its records are brought into shared memory, the block
// sets the walkers' slots up, the next strip's records are requested, and every
// warp walks the parts.  An FP32 sum holds the segments of one row group of a
// sheet in one lane (h rows, at most 64 columns), whatever the number of parts
// in a strip, and goes to FP64 then: over the whole strip of a narrow sheet (up
// to 8 row groups) its rounding grew with the square root of their number and
// more (2100 x 8 rings seen from far away, rms error in ulps of a mean term: h2
// 4528, h3 5300, h4 7616 against 798, 1092, 1410 now).
template <class T, class Rec, int h, int TPT, int BLOCK, bool NEAR64>
__device__ __forceinline__ void eval_parts(const PartBlocks& B, long long n, int stride, int begin, int end,
                                           const Rec* __restrict__ rec, const RecD* __restrict__ rec64,
                                           PartsSmem<T, Rec, h, BLOCK>& sm, const Tgt<T> (&tg)[TPT],
                                           double (&accd)[TPT][3]) {
  using V = typename LaneOf<T>::V;
  constexpr int H = h * LaneOf<T>::kLanes;
  constexpr int kBufs = PartsSmem<T, Rec, h, BLOCK>::kBufs;
  constexpr int HN = H % 2 ? H : 2;  // rows of the near walkers
  static_assert(H % HN == 0, "near rows must tile the part");
  auto decode = [&](long long s, int buf) {
    if (threadIdx.x < kMaxParts) {
      PartInfo pi;
      int w1;
      const int count = decode_part<H>(B, s, (int)threadIdx.x, pi, w1);
      if ((int)threadIdx.x < count) sm.info[buf][threadIdx.x] = pi;
      if (threadIdx.x == 0) {
        sm.count[buf] = count;
        sm.width1[buf] = w1;
      }
    }
  };
  if (begin >= end || begin >= n) return;
  __syncthreads();  // a previous item's walkers are done with the shared memory
  decode(begin, 0);
  if constexpr (kBufs == 2) {
    __syncthreads();
    parts_stage(sm, 0, rec);
  }
  int cur = 0, cls = begin;
  bool more = true;
#pragma unroll 1
  for (long long s = begin; more; cur ^= 1) {
    if constexpr (kBufs == 1) {
      __syncthreads();  // the strip is decoded; the last strip's walkers are done
      parts_stage(sm, cur, rec);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the strip's records are there; the last strip's walkers are done
    s += stride;
    if (s >= n) s = ++cls;
    more = cls < end && s < n;
    if (more) decode(s, cur ^ 1);
    parts_prepare(sm, cur);
    __syncthreads();  // slots and bounds are there
    if constexpr (kBufs == 2)
      if (more) parts_stage(sm, cur ^ 1, rec);
    V acc[TPT][3];
    int rot = 0;  // the rotation acc is in
#pragma unroll
    for (int q = 0; q < TPT; ++q)
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[q][c] = V();
    auto turn = [&](int to) {
      const int by = (to - rot + 3) % 3;
      if (by) {
#pragma unroll
        for (int q = 0; q < TPT; ++q) {
          V a[3] = {acc[q][0], acc[q][1], acc[q][2]};
          rotate3(a, by);
          for (int c = 0; c < 3; ++c) acc[q][c] = a[c];
        }
        rot = to;
      }
    };
    const int count = sm.count[cur], w1 = sm.width1[cur];
    const int wpp = warps_per_part<BLOCK>(count);
#pragma unroll 1
    for (int p = 0; p < count; ++p) {
      V ts[TPT][3];
      float longest;
      const unsigned bits = parts_test<T, Rec, h, BLOCK, TPT>(sm, p, wpp, tg, ts, longest);
      const unsigned kind = bits & 7u;
      const Slot<V>* loc = sm.loc + kColSlots<T, h> * w1 * p;
      const int nc = sm.info[cur][p].nc;
      const int rot_p = sm.meta[p].rot;
      if (kind == 1u) {
        turn(rot_p);
        far_part<T, h, TPT, false, false>(loc, nc, ts, ts, acc);
      } else if (kind == 3u) {
        turn(rot_p);
        far_part<T, h, TPT, true, false>(loc, nc, ts, ts, acc);
      } else if (kind & 1u) {
        turn(rot_p);
        far_part<T, h, TPT, true, true>(loc, nc, ts, ts, acc);
      } else {
        const int nr = sm.info[cur][p].nr;
        const bool last_h = sm.info[cur][p].last_h != 0;
        const Rec* raw = sm.raw[cur % kBufs] + (H + 1) * w1 * p;
        if constexpr (NEAR64) {
          near_fp64<HN, H>(rec64 + sm.info[cur][p].first, sm.info[cur][p].stride, nr, nc, last_h, tg, accd);
        } else {
          // the part as a whole (middle targets) or its blocks
          V th[TPT][3], tl[TPT][3];
          if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int q = 0; q < TPT; ++q) {
              T a[3] = {tg[q].hx, tg[q].hy, tg[q].hz}, b[3] = {tg[q].lx, tg[q].ly, tg[q].lz};
              rotate3(a, rot_p);
              rotate3(b, rot_p);
#pragma unroll
              for (int c = 0; c < 3; ++c) {
                th[q][c] = v_dup(a[c]);
                tl[q][c] = v_dup(b[c]);
              }
            }
          }
          const int blocks = (nc - 1 + kBlockCols - 1) / kBlockCols;
          unsigned mids = 0xffu;  // bit b: block b is middle
          if (!(bits & 8u)) {
            mids = 0;
            if (bits & 16u)
#pragma unroll 1
              for (int b = 0; b < blocks; ++b)
                if (block_mid<T, h, TPT>(loc + kColSlots<T, h> * kBlockCols * b, min(kBlockCols, nc - 1 - kBlockCols * b) + 1,
                                         longest, ts))
                  mids |= 1u << b;
          }
#pragma unroll 1
          for (int b = 0; b < blocks;) {  // runs of blocks of one kind
            const bool is_mid = (mids >> b & 1u) != 0;
            const int j0 = kBlockCols * b;
            do ++b;
            while (b < blocks && ((mids >> b & 1u) != 0) == is_mid);
            const int n = min(kBlockCols * b, nc - 1) - j0 + 1;
            const bool end = j0 + n == nc;
            const Slot<V>* lj = loc + kColSlots<T, h> * j0;
            if (is_mid) {
              turn(rot_p);
              if constexpr (sizeof(T) == 4)
                far_part<T, h, TPT, true, true, true, true>(lj, n, th, tl, acc, end);
              else
                far_part<T, h, TPT, true, true, false, true>(lj, n, ts, ts, acc, end);
            } else if constexpr (sizeof(T) == 4) {
              near_fp32<HN, H>(raw + j0, w1, nr, n, end && last_h, tg, accd);
            } else {
              near_fp64<HN, H>(raw + j0, w1, nr, n, end && last_h, tg, accd);
            }
          }
        }
      }
      if (p == count - 1 || (sizeof(T) == 4 && sm.info[cur][p].last_h)) {
        turn(0);
#pragma unroll
        for (int q = 0; q < TPT; ++q)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            accd[q][c] += v_sum(acc[q][c]);
            acc[q][c] = V();
          }
      }
    }
  }
}

// Partial sums [3][n_targets] of one split.
template <int TPT, int BLOCK>
__device__ __forceinline__ void store_partial(double* __restrict__ px, long long tile0, long long n_targets,
                                              const double (&accd)[TPT][3]) {
#pragma unroll
  for (int q = 0; q < TPT; ++q) {
    const long long t = tile0 + threadIdx.x + (long long)q * BLOCK;
    if (t < n_targets) {
      px[t] = accd[q][0];
      px[n_targets + t] = accd[q][1];
      px[2 * n_targets + t] = accd[q][2];
    }
  }
}

template <class T, class Rec, int h, int TPT, int BLOCK, int MINB, bool NEAR64>
__global__ void __launch_bounds__(BLOCK, MINB)
    nbody_parts_kernel(PartBlocks B, long long n_strips, const double* __restrict__ tx, const double* __restrict__ ty,
                       const double* __restrict__ tz, long long n_targets, const Rec* __restrict__ rec,
                       double* __restrict__ partial, const RecD* __restrict__ rec64, SplitTable split) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<PartsSmem<T, Rec, h, BLOCK>*>(smem_raw);
  const long long tile0 = (long long)blockIdx.x * BLOCK * TPT;
  Tgt<T> tg[TPT];
  double accd[TPT][3];
  load_targets<T, TPT, BLOCK>(tx, ty, tz, 0, tile0, n_targets, tg);
#pragma unroll
  for (int q = 0; q < TPT; ++q) accd[q][0] = accd[q][1] = accd[q][2] = 0.0;
  eval_parts<T, Rec, h, TPT, BLOCK, NEAR64>(B, n_strips, split.classes, split.begin[blockIdx.y],
                                            split.begin[blockIdx.y + 1], rec, rec64, sm, tg, accd);
  store_partial<TPT, BLOCK>(partial + (long long)blockIdx.y * 3 * n_targets, tile0, n_targets, accd);
}

}  // namespace
}  // namespace uvlm
