// march.cuh -- device functions of the volume march (sm_103a).  (On the times in
// the comments see internal.h.)
//
// Restates the reference's per-pixel path (deviceCode.cpp:94-107 ray
// generation, 41-57 slab test, 245-254 firstSampleT, 256-298 integrateBrick,
// 354-416 output stage).  This file is compiled with -fmad=false: every fused
// multiply-add is an explicit fmaf, so the results are bit-identical to the
// CPU restatement, which fixes the same evaluation order.
//
// Sampling: voxel-unit coordinate u = o + t*d - voxelRange.lower; the value
// tap is the trilinear interpolation at u, the six gradient taps sit at
// u +- 1/2 (the reference's tc +- 0.5/N, deviceCode.cpp:278-284).  u - 1/2 and
// u + 1/2 differ by exactly 1, so all seven taps read one 20-voxel cross
// around the cell and share their fractional weights.  With the zy-quad brick
// layout (each element holds a voxel's 2x2 (y, z) neighbourhood) the cross is
// five 16-byte and two 8-byte loads per sample (56 texel fetches in the
// reference).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "internal.h"
#include "steps.h"

namespace aloha {

__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_primary() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ float lerpf(float a, float b, float w) { return fmaf(w, b - a, a); }

__device__ __forceinline__ uint32_t pcg_hash(uint32_t v) {
  uint32_t state = v * 747796405u + 2891336453u;
  uint32_t word = ((state >> ((state >> 28u) + 4u)) ^ state) * 277803737u;
  return (word >> 22u) ^ word;
}

// Per-brick ray offset ils_t0 (deviceCode.cpp:386) from (pixel, accumID, draw).
__device__ __forceinline__ float jitter(int mode, float value, uint32_t pixel, uint32_t accum_id, uint32_t draw) {
  if (mode == ALOHA_JITTER_CONST) return value;
  if (mode == ALOHA_JITTER_HASH) {
    uint32_t h = pcg_hash(pixel ^ pcg_hash(accum_id ^ pcg_hash(draw)));
    return (float)(h >> 8) * (1.0f / 16777216.0f);
  }
  return 0.0f;
}

struct Ray {
  float o[3], d[3];
};

// generateRay (deviceCode.cpp:94-107).
__device__ __forceinline__ Ray generate_ray(const DevView& v, int x, int y) {
  Ray r;
  const float su = (float)x + 0.5f, sv = (float)y + 0.5f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    r.o[a] = v.org[a];
    r.d[a] = fmaf(sv, v.dir_dv[a], fmaf(su, v.dir_du[a], v.dir_00[a]));
  }
  const float len2 = fmaf(r.d[2], r.d[2], fmaf(r.d[1], r.d[1], r.d[0] * r.d[0]));
  const float inv = 1.0f / sqrtf(len2);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    r.d[a] = r.d[a] * inv;
    if (fabsf(r.d[a]) < 1e-5f) r.d[a] = 1e-5f;
  }
  return r;
}

// Slab test (deviceCode.cpp:41-57) against a brick's space range.
__device__ __forceinline__ bool slab(const Ray& r, const float lo[3], const float hi[3], float tmin, float tmax,
                                     float& t0, float& t1) {
  float nr[3], fr[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float l = (lo[a] - r.o[a]) / r.d[a];
    const float h = (hi[a] - r.o[a]) / r.d[a];
    nr[a] = fminf(l, h);
    fr[a] = fmaxf(l, h);
  }
  t0 = fmaxf(tmin, fmaxf(fmaxf(nr[0], nr[1]), nr[2]));
  t1 = fminf(tmax, fminf(fminf(fr[0], fr[1]), fr[2]));
  return t0 < t1;
}

// Seven-tap stencil at voxel coordinate (ux, uy, uz) of a padded brick.
// Evaluation order (shared with the CPU restatement): taps displaced along an
// axis interpolate bilinearly across that axis first (x: y then z; y: x then
// z; z: x then y), then lerp along it; the value tap lerps the x-tap columns
// along x.  lerp(a, b, w) = fmaf(w, b - a, a).
struct StencilOut {
  float value, gx, gy, gz;
};

// One axis of the stencil's coordinates at voxel coordinate u: the weight of
// the centre (g = u - floor u) and of the displaced taps (f = m - floor m,
// m = u - 1/2), whether floor m = floor u - 1 (h), and the clamped indices
// i = floor m and c = floor u.  floor u comes from one round-down conversion
// to an integer k; for |u| < 2^22 (every coordinate of a sample inside a
// brick) k and k - 1 are exact floats and m = RN(u - 1/2) lies in
// [k - 1/2, k + 1/2], so floor m = k - (m < k): the same bits as floorf.  For
// a degenerate coordinate beyond that the indices still clamp into the apron,
// where every tap along the axis reads the same edge value, so the (finite)
// weights cannot change the result.
struct AxisCoord {
  int i, c;
  float f, g;
  bool h;
};

__device__ __forceinline__ AxisCoord axis_coord(float u, int n) {
  const float m = u - 0.5f;
  const int k = __float2int_rd(u);
  const float fc = (float)k;
  AxisCoord a;
  a.h = m < fc;
  a.f = m - (a.h ? fc - 1.0f : fc);
  a.g = u - fc;
  a.c = min(max(k, -kApron), n);
  a.i = min(max(a.c - (a.h ? 1 : 0), -kApron), n - 1);
  return a;
}

// The same coordinates from two float floors per axis (floor u, floor m),
// each converted to an index.  One more conversion per axis, but the weights
// do not wait for an integer-to-float conversion: the render's march, bound
// by the latency of its dependent chain, measured faster this way, the
// backward (which also scatters) the other way.
__device__ __forceinline__ AxisCoord axis_coord_floors(float u, int n) {
  const float m = u - 0.5f;
  const float fm = floorf(m), fc = floorf(u);
  AxisCoord a;
  a.h = fc != fm;
  a.f = m - fm;
  a.g = u - fc;
  a.c = min(max((int)fc, -kApron), n);
  a.i = min(max((int)fm, -kApron), n - 1);
  return a;
}

// Coordinates of a sample inside its brick (InnerCoords launches: |u| < 2^22,
// see internal.h): floor u from one round-down addition of 1.5 * 2^23, whose
// low mantissa bits then hold floor u as an integer.  The same bits as the
// floors above (the sum is exact up to the rounding down, and r - 1.5 * 2^23
// is exact), without the quarter-rate conversions and without clamps.
constexpr float kFloorMagic = 12582912.0f;            // 1.5 * 2^23
constexpr uint32_t kFloorMagicBits = 0x4b400000u;

struct InnerAxis {
  uint32_t bits;  // floor u + kFloorMagicBits
  float f, g;
  bool h;
};

__device__ __forceinline__ InnerAxis inner_axis(float u) {
  const float m = u - 0.5f;
  const float r = __fadd_rd(u, kFloorMagic);
  const float fc = r - kFloorMagic;
  const float d = m - fc;  // exact: in [-1/2, 1/2)
  InnerAxis a;
  a.bits = __float_as_uint(r);
  a.h = d < 0.0f;
  a.f = a.h ? d + 1.0f : d;
  a.g = u - fc;
  return a;
}

__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long x, y, r;
  memcpy(&x, &a, 8);
  memcpy(&y, &b, 8);
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  float2 o;
  memcpy(&o, &r, 8);
  return o;
}
// lerpf on both halves (packed fp32x2 instructions round each half like the
// scalar ones).
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 w) { return __ffma2_rn(w, sub2(b, a), a); }

// The stencil's arithmetic from its seven loads (shared by the direct loads
// of stencil() and the staged loads of StagedLoads, so both give the same
// bits).  c0, c1: the quads at x = cx, cx+1 of row (cy, cz); cx_: the quad of
// the third column (x = cx - 1 if hx, else cx + 2); y0, y1: (z, z+1) pairs at
// x = cx, cx+1 of the third row; z0, z1: (y, y+1) pairs at x = cx, cx+1 of the
// third slice.  The core is indexed by floor u, so the value tap and the
// shared x lerps need no selection; h only says on which side of the core the
// third column, row and slice lie.  The quads' halves are (z, z+1) pairs, so
// lerps along y (columns) and x (shared rows) run two at a time.
__device__ __forceinline__ StencilOut stencil_quads(const float4 c0, const float4 c1, const float4 cx_,
                                                    const float2 y0, const float2 y1, const float2 z0,
                                                    const float2 z1, float fx, float fy, float fz, float gx, float gy,
                                                    float gz, bool hx, bool hy, bool hz) {
  const float2 gx2 = make_float2(gx, gx), gy2 = make_float2(gy, gy);
  // x taps: columns X = bilinear (y by gy, then z by gz) at x = cx, cx+1 and
  // the third column.
  auto column = [&](const float4 q) {
    const float2 l = lerp2(make_float2(q.x, q.y), make_float2(q.z, q.w), gy2);
    return lerpf(l.x, l.y, gz);
  };
  const float Xc0 = column(c0), Xc1 = column(c1), Xe = column(cx_);
  StencilOut s;
  s.value = lerpf(Xc0, Xc1, gx);
  const float X0 = hx ? Xe : Xc0, X1 = hx ? Xc0 : Xc1, X2 = hx ? Xc1 : Xe;
  s.gx = lerpf(X1, X2, fx) - lerpf(X0, X1, fx);

  // x lerps shared by the y and z taps: L0 = (z, z+1) at cy, L1 at cy+1
  const float2 L0 = lerp2(make_float2(c0.x, c0.y), make_float2(c1.x, c1.y), gx2);
  const float2 L1 = lerp2(make_float2(c0.z, c0.w), make_float2(c1.z, c1.w), gx2);

  // y taps: rows bilinear (x by gx, then z by gz).
  const float Yc0 = lerpf(L0.x, L0.y, gz);
  const float Yc1 = lerpf(L1.x, L1.y, gz);
  const float2 ly = lerp2(y0, y1, gx2);
  const float Ye = lerpf(ly.x, ly.y, gz);
  const float Y0 = hy ? Ye : Yc0, Y1 = hy ? Yc0 : Yc1, Y2 = hy ? Yc1 : Ye;
  s.gy = lerpf(Y1, Y2, fy) - lerpf(Y0, Y1, fy);

  // z taps: slices bilinear (x by gx, then y by gy).
  const float2 Zc = lerp2(L0, L1, gy2);
  const float Ze = lerpf(lerpf(z0.x, z1.x, gx), lerpf(z0.y, z1.y, gx), gy);
  const float Z0 = hz ? Ze : Zc.x, Z1 = hz ? Zc.x : Zc.y, Z2 = hz ? Zc.y : Ze;
  s.gz = lerpf(Z1, Z2, fz) - lerpf(Z0, Z1, fz);
  return s;
}

// Element offset of voxel (0, 0, 0) for indices that still carry
// kFloorMagicBits (32-bit wrap-around arithmetic).
__device__ __forceinline__ uint32_t inner_origin(int sy, int sz) {
  return 0u - kFloorMagicBits * (1u + (uint32_t)sy + (uint32_t)sz);
}

// INNER: the brick's samples all lie inside it (InnerCoords), no index needs
// a clamp.  Else ROUND_DOWN picks axis_coord (one conversion per axis) over
// axis_coord_floors.  All give the same bits.  The march around it is bound by
// the L1 data pipe in batches (83 % of its cycles; 60 % of issue slots) and by
// latency, issue and the pipe together in a single frame (512^3: 56 % of issue
// slots, 60 % of the pipe), so instructions count: unclamped, packed and indexed
// by floor u it executes 10 % fewer and half the conversions, and loads the same
// 96 bytes.  512^3 frame 857 -> 815 us, 64^3 frame 104 -> 97,
// 1024^3 frame of 64 ranks 4.86 -> 4.57 ms, uneven batch 10.0 -> 9.7 ms.
template <bool INNER, bool ROUND_DOWN = false>
__device__ __forceinline__ StencilOut stencil(const float4* __restrict__ base, int sy, int sz, int nx, int ny,
                                              int nz, float ux, float uy, float uz) {
  int at, dx, dy, dz;  // core element; element offsets of the third column, row and slice
  float fx, fy, fz, gx, gy, gz;
  bool hx, hy, hz;
  if constexpr (INNER) {
    const InnerAxis X = inner_axis(ux), Y = inner_axis(uy), Z = inner_axis(uz);
    fx = X.f, fy = Y.f, fz = Z.f, gx = X.g, gy = Y.g, gz = Z.g;
    hx = X.h, hy = Y.h, hz = Z.h;
    at = (int)(Z.bits * (uint32_t)sz + inner_origin(sy, sz) + Y.bits * (uint32_t)sy + X.bits);
    dx = hx ? -1 : 2;
    dy = (hy ? -1 : 2) * sy;
    dz = (hz ? -1 : 2) * sz;
  } else {
    // Indices, clamped into the apron.  Every index the oracle clamps to the
    // edge maps to an apron voxel holding that edge value, so these clamps only
    // keep pathological coordinates in bounds and never change a value.
    const AxisCoord X = ROUND_DOWN ? axis_coord(ux, nx) : axis_coord_floors(ux, nx);
    const AxisCoord Y = ROUND_DOWN ? axis_coord(uy, ny) : axis_coord_floors(uy, ny);
    const AxisCoord Z = ROUND_DOWN ? axis_coord(uz, nz) : axis_coord_floors(uz, nz);
    fx = X.f, fy = Y.f, fz = Z.f, gx = X.g, gy = Y.g, gz = Z.g;
    hx = X.h, hy = Y.h, hz = Z.h;
    at = Z.c * sz + Y.c * sy + X.c;
    dx = (hx ? X.i : X.i + 2) - X.c;
    dy = ((hy ? Y.i : Y.i + 2) - Y.c) * sy;
    dz = ((hz ? Z.i : Z.i + 2) - Z.c) * sz;
  }
  const float4* p = base + at;
  const float4* px = base + (at + dx);
  const float2* py = reinterpret_cast<const float2*>(base + (at + dy));  // (z, z+1): the quads' first halves
  const float4* pz = base + (at + dz);                                   // (y, y+1) at z: components 0 and 2
  const float4 c0 = __ldg(p), c1 = __ldg(p + 1), ce = __ldg(px);
  const float2 y0 = __ldg(py), y1 = __ldg(py + 2);
  const float4 z0 = __ldg(pz), z1 = __ldg(pz + 1);
  return stencil_quads(c0, c1, ce, y0, y1, make_float2(z0.x, z0.z), make_float2(z1.x, z1.z), fx, fy, fz, gx, gy, gz,
                       hx, hy, hz);
}

// ---- Where the stencil's rows come from -----------------------------------
// DirectLoads: read-only loads from the brick when the sample is evaluated.
// StagedLoads: the rows of the next sample along the ray are copied into this
// thread's own shared-memory slots with cp.async while the current sample is
// evaluated (double buffering), so the gather's latency overlaps the
// arithmetic without holding registers.  Each thread stages only for itself,
// so no warp or CTA synchronisation is involved; a staged sample is used only
// when the march reaches exactly its t within the same brick march (t is
// strictly increasing there), else it is dropped.  The values are the same
// as the direct loads', so frames are bit-identical.
struct DirectLoads {
  static constexpr bool kStaged = false;
  static constexpr bool kInner = true;  // unclamped coordinates where they are proven (InnerCoords)
  static constexpr int kSteps = 1;      // march steps per loop trip
  __device__ __forceinline__ void begin_brick() {}
  __device__ __forceinline__ void finish() {}
};

// Direct loads with the march loop written out STEPS steps per trip (a
// step-unrolled march: the same steps in the same order, the same bits).
template <int STEPS>
struct UnrolledDirectLoads : DirectLoads {
  static constexpr bool kInner = false;
  static constexpr int kSteps = STEPS;
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(a), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Shared memory of the staged loads: [2 slots][7 rows][kRenderThreads] float4
// (each thread's rows strided by the CTA size, so a warp's row reads are
// contiguous): the seven zy-quads of stencil(), in its order.
constexpr int kStageRows = 7;
constexpr size_t kStageBytes = (size_t)2 * kStageRows * kRenderThreads * sizeof(float4);

struct StagedLoads {
  static constexpr bool kStaged = true;
  static constexpr bool kInner = false;
  static constexpr int kSteps = 1;
  float4* col;     // this thread's column: row e of slot k at col[(k * kStageRows + e) * kRenderThreads]
  float t_staged;  // t of the sample in slot `cur` (NaN: none)
  int cur;
  bool inflight;   // copies may be outstanding
  __device__ __forceinline__ void init(float4* stage_smem) {
    col = stage_smem + threadIdx.x;
    t_staged = __int_as_float(0x7fffffff);
    cur = 0;
    inflight = false;
  }
  __device__ __forceinline__ void begin_brick() { t_staged = __int_as_float(0x7fffffff); }
  // Outstanding copies must land before the CTA's shared memory is released.
  __device__ __forceinline__ void finish() {
    if (inflight) cp_async_wait_all();
    inflight = false;
  }
  __device__ __forceinline__ float4* row(int slot, int e) const { return col + (slot * kStageRows + e) * kRenderThreads; }

  // Starts the copies of the stencil rows at (ux, uy, uz) into `slot`: the
  // addresses of stencil(), clamped into the apron.
  __device__ __forceinline__ void issue(int slot, const float4* __restrict__ base, int sy, int sz, int nx, int ny,
                                        int nz, float ux, float uy, float uz) const {
    const AxisCoord X = axis_coord_floors(ux, nx), Y = axis_coord_floors(uy, ny), Z = axis_coord_floors(uz, nz);
    const int xe = X.h ? X.i : X.i + 2, ye = Y.h ? Y.i : Y.i + 2, ze = Z.h ? Z.i : Z.i + 2;
    const float4* p0 = base + (Z.c * sz + Y.c * sy + X.c);
    const float4* p1 = base + (Z.c * sz + ye * sy + X.c);
    const float4* p2 = base + (ze * sz + Y.c * sy + X.c);
    cp_async16(row(slot, 0), p0);
    cp_async16(row(slot, 1), p0 + 1);
    cp_async16(row(slot, 2), p0 + (xe - X.c));
    cp_async16(row(slot, 3), p1);
    cp_async16(row(slot, 4), p1 + 1);
    cp_async16(row(slot, 5), p2);
    cp_async16(row(slot, 6), p2 + 1);
    cp_async_commit();
  }

  // The sample at t (voxel coordinate u): its rows from the slot it was
  // staged in (or loaded now), after starting the copies of the next sample
  // t + dt when that one lies before t1.
  __device__ __forceinline__ StencilOut sample(const float4* __restrict__ base, int sy, int sz, int nx, int ny, int nz,
                                               float ux, float uy, float uz, float t, float t1, float dt,
                                               const float o[3], const float d[3], float lox, float loy, float loz) {
    if (!(t_staged == t)) {
      if (inflight) cp_async_wait_all();  // a dropped copy may still be landing in `cur`
      issue(cur, base, sy, sz, nx, ny, nz, ux, uy, uz);
    }
    const float tn = t + dt;  // the march's next t, by the same addition
    const bool next = tn < t1;
    if (next) {
      issue(cur ^ 1, base, sy, sz, nx, ny, nz, fmaf(tn, d[0], o[0]) - lox, fmaf(tn, d[1], o[1]) - loy,
            fmaf(tn, d[2], o[2]) - loz);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    const AxisCoord X = axis_coord_floors(ux, nx), Y = axis_coord_floors(uy, ny), Z = axis_coord_floors(uz, nz);
    const float4 e0 = *row(cur, 3), e1 = *row(cur, 4), f0 = *row(cur, 5), f1 = *row(cur, 6);
    const StencilOut s = stencil_quads(*row(cur, 0), *row(cur, 1), *row(cur, 2), make_float2(e0.x, e0.y),
                                       make_float2(e1.x, e1.y), make_float2(f0.x, f0.z), make_float2(f1.x, f1.z), X.f,
                                       Y.f, Z.f, X.g, Y.g, Z.g, X.h, Y.h, Z.h);
    t_staged = next ? tn : __int_as_float(0x7fffffff);
    inflight = next;
    cur ^= 1;
    return s;
  }
};

// tex1D on the transfer function (linear, normalized coords, border 0;
// waikikiRenderer.cpp:990-1008).  tf_s holds the n entries at [2, n+2) with
// two zero entries on each side.
template <bool INNER = false>
__device__ __forceinline__ float4 tf_lookup(const float4* __restrict__ tf_s, int n, float nf, float v) {
  const float xb = v * nf - 0.5f;
  float fl;
  int i;
  if constexpr (INNER) {  // |v| n < 2^21
    const float r = __fadd_rd(xb, kFloorMagic);
    fl = r - kFloorMagic;
    i = (int)(__float_as_uint(r) - kFloorMagicBits);
  } else {
    fl = floorf(xb);
    i = (int)fl;
  }
  const float w = xb - fl;
  i = min(max(i, -2), n);
  const float4 e0 = tf_s[i + 2];
  const float4 e1 = tf_s[i + 3];
  const float2 w2 = make_float2(w, w);
  const float2 lo = lerp2(make_float2(e0.x, e0.y), make_float2(e1.x, e1.y), w2);
  const float2 hi = lerp2(make_float2(e0.z, e0.w), make_float2(e1.z, e1.w), w2);
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// Gradient shading .1 + .9 |N.d|, N = g / |g + 1e-4| (deviceCode.cpp:285,294),
// evaluated as (g.d) / |g + 1e-4|.
__device__ __forceinline__ float shade_factor(const StencilOut& s, const Ray& r) {
  const float ex = s.gx + 1e-4f, ey = s.gy + 1e-4f, ez = s.gz + 1e-4f;
  const float len = sqrtf(fmaf(ez, ez, fmaf(ey, ey, ex * ex)));
  const float gd = fmaf(s.gz, r.d[2], fmaf(s.gy, r.d[1], s.gx * r.d[0]));
  return fmaf(0.9f, fabsf(gd / len), 0.1f);
}

// Front-to-back compositing of one sample (deviceCode.cpp:292-296).
__device__ __forceinline__ void composite_step(float4& color, const float4 c, float shade) {
  const float oma = 1.0f - color.w;
  const float s1 = oma * c.w;
  color.x = fmaf(s1 * c.x, shade, color.x);
  color.y = fmaf(s1 * c.y, shade, color.y);
  color.z = fmaf(s1 * c.z, shade, color.z);
  color.w = fmaf(oma, c.w, color.w);
}

// A macrocell at voxel coordinate u: its code, and the ray parameter (at most
// t1) up to which every sample stays in the box of cells of its kind around it
// (its reach), shrunk by eps.
struct Cell {
  int x, y, z, code;
  __device__ __forceinline__ bool empty() const { return code < kCellFull; }
};
__device__ __forceinline__ Cell cell_at(const uint8_t* __restrict__ cells, int mnx, int mny, int nx, int ny, int nz,
                                        float ux, float uy, float uz) {
  Cell c;
  c.x = min(max(__float2int_rd(ux), 0), nx - 1) >> kMacroShift;
  c.y = min(max(__float2int_rd(uy), 0), ny - 1) >> kMacroShift;
  c.z = min(max(__float2int_rd(uz), 0), nz - 1) >> kMacroShift;
  c.code = __ldg(cells + (c.z * mny + c.y) * mnx + c.x);
  return c;
}
__device__ __forceinline__ float cell_exit(const Cell& c, const float d[3], float offx, float offy, float offz,
                                           float idx, float idy, float idz, float eps, float t1) {
  const int reach = c.code & (kCellFull - 1);
  auto face = [&](int m, float dir) {
    return dir > 0.f ? (float)((m + reach) << kMacroShift) - eps : (float)((m + 1 - reach) << kMacroShift) + eps;
  };
  return fminf(fminf(fminf((face(c.x, d[0]) - offx) * idx, (face(c.y, d[1]) - offy) * idy),
                     (face(c.z, d[2]) - offz) * idz), t1);
}

// A march hook sees every sample, full or skipped, before it is taken: its
// t, the samples already taken in the brick and the colour so far.  The
// render passes NoHook; the differentiable forward stores checkpoints.  An
// active hook keeps `left`, the samples it lets pass before it needs to see
// one again, so runs of skipped samples only stop where it does, and is told
// of full samples through `full_segment`.
struct NoHook {
  static constexpr bool kActive = false;
  __device__ __forceinline__ void operator()(float, uint32_t, const float4&) {}
};

// integrateBrick (deviceCode.cpp:256-298) over [t0, t1); returns the number
// of samples taken.
//
// The lanes of a warp reach empty space at different samples, and the warp
// pays for a lookup and a jump whenever one of them does.  So the march
// alternates: lookups and jumps, at most kMarchJumps of them, then kMarchRun
// samples that need none; the lanes meet at both.
// With a lookup before every sample that leaves a box, a 64^3 frame at 512^2
// executed 313 instructions per warp and sample, which at 16 to 20 warps per SM
// its longest rays wait for one after the other.  512^3 frame / 64^3 frame /
// 24-view batch: 752 us / 90.7 us / 7.66 ms with boxes, 689 / 75 / 7.47 with 2
// jumps and 6 samples (4 CTAs per SM for the frames); 1 and 6: 707 / 78 / 7.83;
// 3 and 6: 697 / 76 / 7.35; 2 and 5: 692 / 75 / 7.45; 2 and 8: 688 / 76 / 7.52;
// as many jumps as it takes and 4: 935 / 90 / 7.97.
constexpr int kMarchJumps = 2, kMarchRun = 6;
template <bool INNER, class Hook, class Loads = DirectLoads>
__device__ __forceinline__ uint32_t march_brick(const DevBrick& b, const float4* __restrict__ tf_s, int n_tf,
                                                const Ray& r, float t0, float t1, float ils, float dt, float et,
                                                bool tame, float4& color, Hook& hook, Loads& loads) {
  const float4* __restrict__ base = b.base;
  const int sy = b.sy, sz = b.sz, nx = b.n[0], ny = b.n[1], nz = b.n[2];
  const float lox = b.lo[0], loy = b.lo[1], loz = b.lo[2];
  const float nf = (float)n_tf;
  const uint32_t cap = march_cap(t0, t1, dt);
  const uint8_t* __restrict__ cells = b.cells;
  const int mnx = (nx + kMacro - 1) >> kMacroShift, mny = (ny + kMacro - 1) >> kMacroShift;
  // Brick-local ray origin, inverse direction and the rounding margin (voxel
  // units) that makes the macrocell exit bound below conservative: u = o + t d
  // - lo is computed with a few ulps of the largest magnitude involved.
  const float offx = r.o[0] - lox, offy = r.o[1] - loy, offz = r.o[2] - loz;
  const float idx_ = 1.0f / r.d[0], idy = 1.0f / r.d[1], idz = 1.0f / r.d[2];
  const float mag = fmaxf(fmaxf(fabsf(r.o[0]) + fabsf(lox), fabsf(r.o[1]) + fabsf(loy)),
                          fabsf(r.o[2]) + fabsf(loz)) + fabsf(t1);
  const float eps = 2e-6f * mag + 1e-4f;
  uint32_t n = 0;
  float t = first_sample_t(t0, dt, ils);
  const bool exact = exact_steps(t, t1, dt);
  const float inv_dt = 1.0f / dt;
  const int run = INNER || tame ? kMarchRun : 1;
  loads.begin_brick();
  while (t < t1 && color.w < et && n < cap) {
    // Up to kMarchJumps steps over empty boxes, until the ray is at a sample in
    // a full macrocell.  A sample in an empty one has alpha exactly 0 and leaves
    // the colour unchanged, so only t and the sample count advance (the same t
    // += dt sequence as full samples) up to the box's end.  The first is always
    // taken.  The rest of the run is one jump (one more per power of two it
    // crosses, and one per checkpoint the hook needs).
    int jumps = 0;
    for (; jumps < kMarchJumps && t < t1 && n < cap; ++jumps) {
      const Cell cell = cell_at(cells, mnx, mny, nx, ny, nz, fmaf(t, r.d[0], r.o[0]) - lox,
                                fmaf(t, r.d[1], r.o[1]) - loy, fmaf(t, r.d[2], r.o[2]) - loz);
      if (!cell.empty()) break;
      const float tb = cell_exit(cell, r.d, offx, offy, offz, idx_, idy, idz, eps, t1);
      hook(t, n, color);
      ++n;
      t = t + dt;
      if constexpr (!Hook::kActive) {
        if (exact)
          run_steps(t, n, tb, cap, dt, inv_dt, 0xffffffffu);
        else
          run_steps_any(t, n, tb, cap, dt, 0xffffffffu);
      } else if (exact) {
        for (;;) {
          hook.left -= run_steps(t, n, tb, cap, dt, inv_dt, hook.left);
          if (!(t < tb && n < cap)) break;
          hook(t, n, color);  // a checkpoint falls due here (hook.left == 0)
          ++n;
          t = t + dt;
        }
      } else {
        // step by step: a second jump form in here cost the training forward
        // of the exact steps 4 % (16 views of 128^3 at 256^2)
        while (t < tb && n < cap) {
          uint32_t k = hook.left;
          while (k > 0 && t < tb && n < cap) {
            ++n;
            t = t + dt;
            --k;
          }
          hook.left = k;
          if (k == 0 && t < tb && n < cap) {
            hook(t, n, color);
            ++n;
            t = t + dt;
          }
        }
      }
    }
    if (jumps == kMarchJumps) continue;
    // Up to kMarchRun samples without another lookup (one in an empty macrocell
    // leaves the colour unchanged as well), or one if the scene is not tame.
    int k = 0;
    auto step = [&]() {
      if (!(k < run && t < t1 && color.w < et && n < cap)) return false;
      const float ux = fmaf(t, r.d[0], r.o[0]) - lox;
      const float uy = fmaf(t, r.d[1], r.o[1]) - loy;
      const float uz = fmaf(t, r.d[2], r.o[2]) - loz;
      hook(t, n, color);
      if constexpr (Hook::kActive) hook.full_segment = true;
      ++n;
      ++k;
      StencilOut s;
      if constexpr (Loads::kStaged)
        s = loads.sample(base, sy, sz, nx, ny, nz, ux, uy, uz, t, t1, dt, r.o, r.d, lox, loy, loz);
      else
        s = stencil<INNER>(base, sy, sz, nx, ny, nz, ux, uy, uz);
      const float shade = shade_factor(s, r);
      const float4 c = tf_lookup<INNER>(tf_s, n_tf, nf, s.value);
      composite_step(color, c, shade);
      t = t + dt;
      return true;
    };
    if constexpr (Loads::kSteps > 1) {
      for (bool go = true; go;) {
#pragma unroll
        for (int i = 0; i < Loads::kSteps; ++i) go = go && step();
      }
    } else {
#pragma unroll 1
      while (step()) {
      }
    }
  }
  return n;
}

template <bool INNER, class Hook>
__device__ __forceinline__ uint32_t march_brick(const DevBrick& b, const float4* __restrict__ tf_s, int n_tf,
                                                const Ray& r, float t0, float t1, float ils, float dt, float et,
                                                bool tame, float4& color, Hook& hook) {
  DirectLoads direct;
  return march_brick<INNER>(b, tf_s, n_tf, r, t0, t1, ils, dt, et, tame, color, hook, direct);
}

// ---- Sample-parallel lane groups ------------------------------------------
// G lanes of a warp march one ray together: all hold the serial march's state
// (t, n, colour, t_cell) identically.  One group iteration replaces up to G
// iterations of march_brick:
//  1. at the base sample (t, n) the loop test and the macrocell test run as
//     in the serial loop; an empty macrocell starts the same skip run, taken
//     identically by every lane;
//  2. lane j takes sample j of the group, at the t the serial loop reaches by
//     j more rounded additions of dt, if it lies before t1 and under the
//     iteration cap; past t_cell it looks up its own macrocell and drops the
//     sample if that one is empty (the serial loop would skip it; a full
//     sample of alpha 0 leaves the colour unchanged either way);
//  3. every lane evaluates its sample (stencil, shading, lookup) at once;
//  4. the samples are composited in lane order from shuffled values, in every
//     lane: before sample j the serial loop's head test (t_j < t1, colour
//     alpha < ET, n < cap) decides whether it and the later ones are taken;
//     each taken sample adds 1 to n and dt to t.
// The colour, n and t leave the iteration as the serial loop would leave them
// after the same samples, bit for bit.  A ray's samples take about G times
// fewer dependent steps, at the cost of the shuffles and of the samples
// evaluated past the ray's end.
struct LaneGroup {
  int lane;       // index in the group, 0..G-1
  unsigned mask;  // the group's lanes in the warp
  int base;       // first lane of the group in the warp
};

template <int G>
__device__ __forceinline__ uint32_t march_brick_group(const DevBrick& b, const float4* __restrict__ tf_s, int n_tf,
                                                      const Ray& r, float t0, float t1, float ils, float dt, float et,
                                                      float4& color, const LaneGroup& g) {
  const float4* __restrict__ base = b.base;
  const int sy = b.sy, sz = b.sz, nx = b.n[0], ny = b.n[1], nz = b.n[2];
  const float lox = b.lo[0], loy = b.lo[1], loz = b.lo[2];
  const float nf = (float)n_tf;
  const uint32_t cap = march_cap(t0, t1, dt);
  const uint8_t* __restrict__ cells = b.cells;
  const int mnx = (nx + kMacro - 1) >> kMacroShift, mny = (ny + kMacro - 1) >> kMacroShift;
  const float offx = r.o[0] - lox, offy = r.o[1] - loy, offz = r.o[2] - loz;
  const float idx_ = 1.0f / r.d[0], idy = 1.0f / r.d[1], idz = 1.0f / r.d[2];
  const float mag = fmaxf(fmaxf(fabsf(r.o[0]) + fabsf(lox), fabsf(r.o[1]) + fabsf(loy)),
                          fabsf(r.o[2]) + fabsf(loz)) + fabsf(t1);
  const float eps = 2e-6f * mag + 1e-4f;
  uint32_t n = 0;
  float t = first_sample_t(t0, dt, ils);
  const bool exact = exact_steps(t, t1, dt);
  const float inv_dt = 1.0f / dt;
  float t_cell = t0;
  while (t < t1 && color.w < et && n < cap) {
    if (!(t < t_cell)) {
      const float ux = fmaf(t, r.d[0], r.o[0]) - lox;
      const float uy = fmaf(t, r.d[1], r.o[1]) - loy;
      const float uz = fmaf(t, r.d[2], r.o[2]) - loz;
      const Cell cell = cell_at(cells, mnx, mny, nx, ny, nz, ux, uy, uz);
      const float tb = cell_exit(cell, r.d, offx, offy, offz, idx_, idy, idz, eps, t1);
      if (cell.empty()) {
        ++n;
        t = t + dt;
        if (exact)
          run_steps(t, n, tb, cap, dt, inv_dt, 0xffffffffu);
        else
          run_steps_any(t, n, tb, cap, dt, 0xffffffffu);
        continue;
      }
      t_cell = tb;
    }
    // this lane's sample: the serial loop's t after g.lane more steps
    float tk = t;
    for (int j = 0; j < g.lane; ++j) tk = tk + dt;
    const bool in_range = tk < t1 && n + (uint32_t)g.lane < cap;
    bool full = in_range;
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
    float shade = 0.f;
    if (in_range) {
      const float vx = fmaf(tk, r.d[0], r.o[0]) - lox;
      const float vy = fmaf(tk, r.d[1], r.o[1]) - loy;
      const float vz = fmaf(tk, r.d[2], r.o[2]) - loz;
      if (!(tk < t_cell)) full = !cell_at(cells, mnx, mny, nx, ny, nz, vx, vy, vz).empty();
      if (full) {
        const StencilOut s = stencil<false>(base, sy, sz, nx, ny, nz, vx, vy, vz);
        shade = shade_factor(s, r);
        c = tf_lookup(tf_s, n_tf, nf, s.value);
      }
    }
    const unsigned in_mask = __ballot_sync(g.mask, in_range) >> g.base;
    const unsigned full_mask = __ballot_sync(g.mask, full) >> g.base;
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const float cx = __shfl_sync(g.mask, c.x, j, G), cy = __shfl_sync(g.mask, c.y, j, G);
      const float cz = __shfl_sync(g.mask, c.z, j, G), cw = __shfl_sync(g.mask, c.w, j, G);
      const float sh = __shfl_sync(g.mask, shade, j, G);
      if (!((in_mask >> j) & 1u) || !(color.w < et)) break;
      if ((full_mask >> j) & 1u) composite_step(color, make_float4(cx, cy, cz, cw), sh);
      ++n;
      t = t + dt;
    }
  }
  return n;
}

// Two lanes per ray: march_brick with the ray's state (t, n, colour) in both
// lanes and its samples two at a time, the first lane taking the sample at t,
// the second the one after it; both composite the two in order from exchanged
// values, so the state leaves a step as march_brick leaves it after the same
// samples, bit for bit.  A ray's chain of dependent steps is half as long and a
// warp waits for the longest of 16 rays, not of 32; the lookups, jumps and the
// composite are done twice, so all chunks of a full GPU are slower this way
// (512^3 at 1024^2 678 -> 711 us, 24-view batch 7.5 -> 9.4 ms) and those of a
// GPU with idle warps faster (512^3 at 512^2 576 -> 371 us, 256^3 235 -> 185).
// kPairRun 6 / 8 / 12: 256^3 at 512^2 with an upload 430 / 425 / 432 us.
constexpr int kPairRun = 8;
template <bool INNER>
__device__ __forceinline__ uint32_t march_brick_pair(const DevBrick& b, const float4* __restrict__ tf_s, int n_tf,
                                                     const Ray& r, float t0, float t1, float ils, float dt, float et,
                                                     bool tame, float4& color, const LaneGroup& g) {
  const float4* __restrict__ base = b.base;
  const int sy = b.sy, sz = b.sz, nx = b.n[0], ny = b.n[1], nz = b.n[2];
  const float lox = b.lo[0], loy = b.lo[1], loz = b.lo[2];
  const float nf = (float)n_tf;
  const uint32_t cap = march_cap(t0, t1, dt);
  const uint8_t* __restrict__ cells = b.cells;
  const int mnx = (nx + kMacro - 1) >> kMacroShift, mny = (ny + kMacro - 1) >> kMacroShift;
  const float offx = r.o[0] - lox, offy = r.o[1] - loy, offz = r.o[2] - loz;
  const float idx_ = 1.0f / r.d[0], idy = 1.0f / r.d[1], idz = 1.0f / r.d[2];
  const float mag = fmaxf(fmaxf(fabsf(r.o[0]) + fabsf(lox), fabsf(r.o[1]) + fabsf(loy)),
                          fabsf(r.o[2]) + fabsf(loz)) + fabsf(t1);
  const float eps = 2e-6f * mag + 1e-4f;
  const bool first = g.lane == 0;
  uint32_t n = 0;
  float t = first_sample_t(t0, dt, ils);
  const bool exact = exact_steps(t, t1, dt);
  const float inv_dt = 1.0f / dt;
  const int run = INNER || tame ? kPairRun : 1;  // 1: of the first lane's samples alone
  while (t < t1 && color.w < et && n < cap) {
    int jumps = 0;  // as in march_brick, by both lanes
    for (; jumps < kMarchJumps && t < t1 && n < cap; ++jumps) {
      const Cell cell = cell_at(cells, mnx, mny, nx, ny, nz, fmaf(t, r.d[0], r.o[0]) - lox,
                                fmaf(t, r.d[1], r.o[1]) - loy, fmaf(t, r.d[2], r.o[2]) - loz);
      if (!cell.empty()) break;
      const float tb = cell_exit(cell, r.d, offx, offy, offz, idx_, idy, idz, eps, t1);
      ++n;
      t = t + dt;
      if (exact)
        run_steps(t, n, tb, cap, dt, inv_dt, 0xffffffffu);
      else
        run_steps_any(t, n, tb, cap, dt, 0xffffffffu);
    }
    if (jumps == kMarchJumps) continue;
#pragma unroll 1
    for (int k = 0; k < run && t < t1 && color.w < et && n < cap; k += 2) {
      // past the ray's end the second lane takes the first one's sample again
      // (its coordinates are known to be the brick's) and drops it
      const float t2 = t + dt;
      const bool two = t2 < t1 && n + 1 < cap && (INNER || run > 1);
      const float tk = !first && two ? t2 : t;
      const StencilOut s =
          stencil<INNER>(base, sy, sz, nx, ny, nz, fmaf(tk, r.d[0], r.o[0]) - lox, fmaf(tk, r.d[1], r.o[1]) - loy,
                         fmaf(tk, r.d[2], r.o[2]) - loz);
      const float shade = shade_factor(s, r);
      const float4 c = tf_lookup<INNER>(tf_s, n_tf, nf, s.value);
      const float os = __shfl_xor_sync(g.mask, shade, 1);
      const float ox = __shfl_xor_sync(g.mask, c.x, 1), oy = __shfl_xor_sync(g.mask, c.y, 1);
      const float oz = __shfl_xor_sync(g.mask, c.z, 1), ow = __shfl_xor_sync(g.mask, c.w, 1);
      composite_step(color, make_float4(first ? c.x : ox, first ? c.y : oy, first ? c.z : oz, first ? c.w : ow),
                     first ? shade : os);
      ++n;
      t = t2;
      if (two && color.w < et) {
        composite_step(color, make_float4(first ? ox : c.x, first ? oy : c.y, first ? oz : c.z, first ? ow : c.w),
                       first ? os : shade);
        ++n;
        t = t + dt;
      }
    }
  }
  return n;
}

__device__ __forceinline__ float saturatef_(float x) { return fminf(fmaxf(x, 0.0f), 1.0f); }

// temperature_to_rgb (deviceCode.cpp:300-314).
__device__ __forceinline__ void heat_color(float t, float out[3]) {
  const float K = 4.0f / 6.0f;
  const float h = K - K * t;
  const float v = 0.5f + 0.5f * t;
  const float s = saturatef_(h) * 6.0f;
  out[0] = v * saturatef_(fabsf(s - 3.0f) - 1.0f);
  out[1] = v * saturatef_(2.0f - fabsf(s - 2.0f));
  out[2] = v * saturatef_(2.0f - fabsf(s - 4.0f));
}

__device__ __forceinline__ uint32_t quantize8(float x) {
  const float c = fminf(fmaxf(x, 0.0f), 1.0f);
  return (uint32_t)(c * 255.0f + 0.5f);
}

__device__ __forceinline__ uint32_t pack_rgba(float4 c) {
  return quantize8(c.x) | (quantize8(c.y) << 8) | (quantize8(c.z) << 16) | (quantize8(c.w) << 24);
}

__device__ __forceinline__ bool scene_inner(const FrameArgs& a) { return __ldg(a.scene_flags) & kSceneInner; }

// Loads the transfer function into shared memory with two zero entries on
// each side (border addressing).
__device__ __forceinline__ void load_tf(float4* tf_s, const float4* __restrict__ tf, int n) {
  for (int i = threadIdx.x; i < n + 4; i += blockDim.x) {
    const int k = i - 2;
    tf_s[i] = (k >= 0 && k < n) ? __ldg(tf + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// One virtual rank's march for one pixel (deviceCode.cpp:378-399): the
// rank's bricks [j0, j1) of the view schedule front to back, spp draws, early
// termination on the rank's own alpha.  ONE: spp is known to be 1; ROLLED: one
// copy of the march for all passes.  Returns the spp sum of the colours;
// z = nearest brick entry / max depth, ns = samples taken.
template <bool INNER, class Loads = DirectLoads, int G = 1, bool ONE = false, bool ROLLED = false>
__device__ __forceinline__ float4 march_rank(const FrameArgs& a, const DevView& v, const float4* tf_s, const Ray& ray,
                                             const int* __restrict__ rbricks, int j0, int j1, int pixel, float& z,
                                             uint32_t& ns, Loads& loads, const LaneGroup& g = LaneGroup{0, 0u, 0}) {
  uint32_t draw = 0;
  // one pass of the rank's bricks (one sample per pixel of spp)
  auto pass = [&]() -> float4 {
    float4 color = make_float4(0.f, 0.f, 0.f, 0.f);
    float tmin = 0.0f;
    for (int j = j0; j < j1; ++j) {
      const DevBrick b = a.bricks[__ldg(rbricks + j)];
      float t0, t1;
      if (!slab(ray, b.space_lo, b.space_hi, tmin, 1e10f, t0, t1)) continue;
      const float ils = jitter(a.jitter_mode, a.jitter_value, (uint32_t)pixel, (uint32_t)a.accum_id, draw++);
      const float tnear = (t0 > tmin ? t0 : 0.0f) + tmin;
      z = fminf(z, tnear / v.max_depth);
      NoHook none;
      const bool tame = INNER || (__ldg(a.scene_flags) & kSceneTame);
      if constexpr (G == 2) {
        ns += march_brick_pair<INNER>(b, tf_s, a.n_tf, ray, t0, t1, ils, a.dt, a.et_alpha, tame, color, g);
      } else if constexpr (G > 1) {
        ns += march_brick_group<G>(b, tf_s, a.n_tf, ray, t0, t1, ils, a.dt, a.et_alpha, color, g);
      } else {
        ns += march_brick<INNER>(b, tf_s, a.n_tf, ray, t0, t1, ils, a.dt, a.et_alpha, tame, color, none, loads);
      }
      tmin = t1 + 1e-20f;
      if (!(color.w < a.et_alpha)) break;
    }
    return color;
  };
  // The sum over passes starts from the first pass's colour: 0 + c = c, as a
  // march colour is never -0 (it starts at +0 and every update is an fmaf
  // onto it, and an exact zero sum rounds to +0).  With one pass no sum is
  // then live across the march.
  if constexpr (ONE) return pass();
  if constexpr (ROLLED) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int s = 0; s < a.spp; ++s) {
      const float4 color = pass();
      sum.x = sum.x + color.x;
      sum.y = sum.y + color.y;
      sum.z = sum.z + color.z;
      sum.w = sum.w + color.w;
    }
    return sum;
  }
  float4 acc = pass();
  for (int s = 1; s < a.spp; ++s) {
    const float4 color = pass();
    acc.x = acc.x + color.x;
    acc.y = acc.y + color.y;
    acc.z = acc.z + color.z;
    acc.w = acc.w + color.w;
  }
  return acc;
}

// renderFrame's per-rank output stage (deviceCode.cpp:400-416): heat map,
// accumulation buffer, 1/(accumID+1) scale, crosshair, 1/spp.  Writes the
// rank's image and depth into the given [n_ranks][H*W] planes when they are
// not null; returns the rank image.
__device__ __forceinline__ float4 rank_output(const FrameArgs& a, int W, int H, int r, int x, int y, int pixel,
                                              size_t npx, float4 acc, uint32_t ns, float z, float4* img_planes,
                                              float* depth_planes) {
  if (a.heat_map) {
    float hc[3];
    heat_color((float)ns * (a.heat_map_scale / (float)a.spp), hc);
    acc.x = fmaf(0.5f, acc.x, hc[0]);
    acc.y = fmaf(0.5f, acc.y, hc[1]);
    acc.z = fmaf(0.5f, acc.z, hc[2]);
    acc.w = fmaf(0.5f, acc.w, 0.5f);
  }
  if (a.accum) {
    float4* ap = a.accum + ((size_t)r * npx + pixel);
    if (a.accum_id > 0) {
      const float4 old = *ap;
      acc.x = acc.x + old.x;
      acc.y = acc.y + old.y;
      acc.z = acc.z + old.z;
      acc.w = acc.w + old.w;
    }
    if (a.accumulate) *ap = acc;
  }
  const float scale = 1.0f / (float)(a.accum_id + 1);
  acc.x = acc.x * scale;
  acc.y = acc.y * scale;
  acc.z = acc.z * scale;
  acc.w = acc.w * scale;
  if (a.crosshair && (x == W / 2 || y == H / 2)) {
    acc.x = 1.0f - acc.x;
    acc.y = 1.0f - acc.y;
    acc.z = 1.0f - acc.z;
    acc.w = 1.0f - acc.w;
  }
  const float inv_spp = 1.0f / (float)a.spp;
  const float4 img = make_float4(acc.x * inv_spp, acc.y * inv_spp, acc.z * inv_spp, acc.w * inv_spp);
  if (img_planes) img_planes[(size_t)r * npx + pixel] = img;
  if (depth_planes) depth_planes[(size_t)r * npx + pixel] = z;
  return img;
}

// True when renderFrame's output stage leaves a rank image equal to the
// march's colour: one sample per pixel, no accumulation, heat map or
// crosshair (then img = acc * (1 / 1) * (1 / 1) = acc exactly); plain_output
// also wants no rank planes.
__device__ __forceinline__ bool plain_output_stage(const FrameArgs& a) {
  return a.spp == 1 && a.accum_id == 0 && !a.heat_map && !a.crosshair && !(a.accum && a.accumulate);
}
__device__ __forceinline__ bool plain_output(const FrameArgs& a) {
  return plain_output_stage(a) && !a.rank_images && !a.rank_depth;
}

// Front-to-back ordered "over" of rank images (IceT BLEND with
// ORDERED_COMPOSITE, waikikiRenderer.cpp:910-917,1042-1079): in fp32, or on
// images quantised to 8 bits per channel like IceT's RGBA_UBYTE buffers.
// One float4 holds the state of either mode (the ubyte channels as the bits
// of its components; all-zero bits are 0.0f and 0u), so the blend keeps four
// registers live across the march, not eight.
struct OverBlend {
  float4 comp = make_float4(0.f, 0.f, 0.f, 0.f);
  __device__ __forceinline__ void add(int mode, float4 img) {
    if (mode == ALOHA_COMPOSITE_UBYTE) {
      const uint32_t q0 = quantize8(img.x), q1 = quantize8(img.y), q2 = quantize8(img.z), q3 = quantize8(img.w);
      const uint32_t c0 = __float_as_uint(comp.x), c1 = __float_as_uint(comp.y), c2 = __float_as_uint(comp.z),
                     c3 = __float_as_uint(comp.w);
      const uint32_t f = 255u - c3;
      comp.x = __uint_as_float(min(255u, c0 + (q0 * f + 127u) / 255u));
      comp.y = __uint_as_float(min(255u, c1 + (q1 * f + 127u) / 255u));
      comp.z = __uint_as_float(min(255u, c2 + (q2 * f + 127u) / 255u));
      comp.w = __uint_as_float(min(255u, c3 + (q3 * f + 127u) / 255u));
    } else {
      const float oma = 1.0f - comp.w;
      comp.x = fmaf(oma, img.x, comp.x);
      comp.y = fmaf(oma, img.y, comp.y);
      comp.z = fmaf(oma, img.z, comp.z);
      comp.w = fmaf(oma, img.w, comp.w);
    }
  }
  __device__ __forceinline__ uint32_t pack(int mode) const {
    return mode == ALOHA_COMPOSITE_UBYTE ? (__float_as_uint(comp.x) | (__float_as_uint(comp.y) << 8) |
                                            (__float_as_uint(comp.z) << 16) | (__float_as_uint(comp.w) << 24))
                                         : pack_rgba(comp);
  }
};

// Island membership of a pixel (16x16 tiles dealt round-robin).
__device__ __forceinline__ bool pixel_in_island(const FrameArgs& a, int W, int x, int y) {
  if (a.num_islands <= 1) return true;
  const int tiles_x = (W + 15) / 16;
  return (((x >> 4) + tiles_x * (y >> 4)) % a.num_islands) == a.island_id;
}

// One pixel of one view: every virtual rank marches its bricks and runs
// renderFrame's output stage; the rank images are blended front to back.
// Returns the number of samples.
// With G > 1 the G lanes of `g` render the pixel together (a lane group);
// only the group's first lane runs the output stage and writes.  Groups of
// more than two have no accumulation buffer and no rank planes (the caller
// ensures it).
// ONE: one copy of the march for plain InnerCoords frames of one pass and one for
// everything else, for kernels that hold several marches and are short of
// instruction cache rather than registers (2 spp frame with two lanes per ray
// 335 -> 299 us, 512^3 at 1024^2 678 -> 673; the 72-register instances spill
// more with it, 7.47 -> 7.67 ms for a 24-view batch).
template <bool INNER, class Loads = DirectLoads, int G = 1, bool ONE = false>
__device__ __forceinline__ uint32_t render_pixel(const FrameArgs& a, const DevView& v, const float4* tf_s, int x,
                                                 int y, uint32_t* fb_out, size_t fb_index, Loads& loads,
                                                 const LaneGroup& g = LaneGroup{0, 0u, 0}) {
  const int W = v.width, H = v.height;
  const int pixel = x + W * y;
  const size_t npx = (size_t)W * H;
  const int R = v.n_ranks;
  const int* __restrict__ order = a.sched + v.sched;
  const int* __restrict__ rstart = order + R;
  const int* __restrict__ rbricks = rstart + R + 1;
  const bool in_island = pixel_in_island(a, W, x, y);
  const Ray ray = generate_ray(v, x, y);
  OverBlend blend;
  uint32_t total = 0;
  if ((INNER || !ONE) && plain_output(a)) {
    // the output stage is the identity (acc * 1 * 1): nothing it needs stays
    // live across the march
    for (int k = 0; k < R; ++k) {
      const int r = __ldg(order + k);
      float z = 1.0f;
      uint32_t ns = 0;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in_island)
        acc = march_rank<INNER, Loads, G, ONE>(a, v, tf_s, ray, rbricks, __ldg(rstart + r), __ldg(rstart + r + 1),
                                               pixel, z, ns, loads, g);
      blend.add(a.composite_mode, acc);
      total += ns;
    }
  } else {
    for (int k = 0; k < R; ++k) {
      const int r = __ldg(order + k);
      float z = 1.0f;
      uint32_t ns = 0;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in_island)
        acc = march_rank<INNER, Loads, G, false, ONE>(a, v, tf_s, ray, rbricks, __ldg(rstart + r),
                                                      __ldg(rstart + r + 1), pixel, z, ns, loads, g);
      if (G == 1 || g.lane == 0)
        blend.add(a.composite_mode, rank_output(a, W, H, r, x, y, pixel, npx, acc, ns, z, a.rank_images, a.rank_depth));
      total += ns;
    }
  }
  if (fb_out && (G == 1 || g.lane == 0)) fb_out[fb_index] = blend.pack(a.composite_mode);
  return total;
}

// Pixel of a lane in its warp's 8x4 tile: each quarter warp, the unit in which
// 16-byte loads are served, takes a 2x4 block, whose rays read fewer distinct
// quads than a row of eight does.
__device__ __forceinline__ int tile_x(int lane) { return (lane & 1) | ((lane >> 2) & 6); }
__device__ __forceinline__ int tile_y(int lane) { return (lane >> 1) & 3; }

// The same for pixel p of a 4x4 tile whose rays have two lanes each.
__device__ __forceinline__ int pair_x(int p) { return (p & 1) | ((p >> 1) & 2); }
__device__ __forceinline__ int pair_y(int p) { return ((p >> 1) & 1) | ((p >> 2) & 2); }

// Work slot k of a view -> chunk (cx, cy) in centre-out square rings; false
// for slots outside the chunk grid.  Ring r >= 1 holds slots
// [(2r-1)^2, (2r+1)^2), walked up the right edge, left along the top, down
// the left edge and right along the bottom.
__device__ __forceinline__ bool ring_chunk(int k, int cxn, int cyn, int& cx, int& cy) {
  int x = 0, y = 0;
  if (k > 0) {
    int r = (int)((sqrtf((float)k) + 1.0f) * 0.5f);
    while ((2 * r + 1) * (2 * r + 1) <= k) ++r;
    while (r > 1 && (2 * r - 1) * (2 * r - 1) > k) --r;
    const int j = k - (2 * r - 1) * (2 * r - 1);
    const int side = j / (2 * r), off = j % (2 * r);
    if (side == 0) {
      x = r;
      y = -r + 1 + off;
    } else if (side == 1) {
      x = r - 1 - off;
      y = r;
    } else if (side == 2) {
      x = -r;
      y = r - 1 - off;
    } else {
      x = -r + 1 + off;
      y = -r;
    }
  }
  cx = x + (cxn - 1) / 2;
  cy = y + (cyn - 1) / 2;
  return cx >= 0 && cx < cxn && cy >= 0 && cy < cyn;
}

// Warp-aggregated add of per-thread sample counts into a 64-bit counter.
__device__ __forceinline__ void count_samples(unsigned long long* counter, uint32_t n) {
  if (!counter) return;
  const unsigned s = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(counter, (unsigned long long)s);
}

}  // namespace aloha
