// adjoint.cu -- differentiable form of the march (no reference counterpart).
//
// Forward (training): every pixel marches the single virtual rank's bricks
// front to back exactly as render_pixel does (same arithmetic, so the image
// is bit-identical to a render with one rank) and stores the march state
// every K samples: colour, t, the brick walk position, tmin, the jitter draw
// index and the samples already taken in the brick.  It also appends one work
// item per K-sample segment.
//
// Backward: one thread per segment.  With front-to-back compositing the
// colour adjoint g_rgb = dL/dC_rgb is the same for every sample, and the
// adjoint of alpha after sample i has the closed form
//     gA_{i+1} = (g_a (1 - a_N) - g_rgb . (rgb_N - rgb_{i+1})) / (1 - a_{i+1})
// (a_N, rgb_N: the final state).  So every segment is independent: a thread
// replays its K samples from the checkpoint and scatters
//     dL/dalpha_i = (1-a_i)(s_i g.c_i + gA_{i+1}),  dL/dc_i = g (1-a_i) alpha_i s_i,
//     dL/ds_i = (1-a_i) alpha_i g.c_i
// through the transfer-function lookup (shared-memory accumulation, one flush
// per CTA), the shading and the seven-tap stencil (20 voxel weights, atomic
// adds into the density gradient on the caller's grid).  Early termination is
// held fixed, as usual for a discontinuity.
//
// One launch serves one view or many: the forward marches the chunks of all
// its views position-major (every view's first chunk, then every view's
// second, ...), and the backward replays the segments of all its views, each
// item finding its view in a prefix of the views' segment counts.  A launch
// of one view passes it in the kernel parameters instead (backward_kernel's
// MULTI = false), which keeps its pointers out of the replay's registers.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>

#include "adjoint.h"
#include "march.cuh"

namespace aloha {

namespace {

struct Walk {
  int j;          // position in the rank's brick list
  float tmin;     // ray tmin at the start of this brick
  uint32_t draw;  // next jitter draw index
};

// Schedule of the single virtual rank: [rank_order 1][rank_start 2][bricks].
__device__ __forceinline__ const int* rank_bricks(const TrainArgs& a, const DevView& v) { return a.sched + v.sched + 3; }

// Samples of one pixel along the single rank's bricks, starting at walk
// state `w` (and, when `resume`, inside brick w.j at t_resume with nb0
// samples already taken there).  Calls `visit` before compositing each
// sample; stops after max_samples.  The walk, jitter draws and sample
// arithmetic are those of render_pixel / march_brick.
//
// With SKIP, samples in empty macrocells (transfer-function alpha exactly 0,
// see march_brick) are counted and stepped over without a `visit` (in one
// jump when the steps are exact).  Only the density gradient may skip them: a
// zero-alpha sample still carries a gradient for the alpha entries.
//
// With CAN_STOP the walk also ends, before the next sample, once *stop is set
// (by the visitor).
template <bool INNER, bool SKIP, bool CAN_STOP = false, class Visit>
__device__ __forceinline__ uint32_t walk_samples(const TrainArgs& a, const DevView& v, const float4* tf_s,
                                                 const Ray& ray, uint32_t pixel, Walk w, float t_resume,
                                                 uint32_t nb0, bool resume, float4& color, uint32_t max_samples,
                                                 Visit visit, const bool* stop = nullptr) {
  const int* __restrict__ rb = rank_bricks(a, v);
  const int j1 = __ldg(a.sched + v.sched + 2);
  const float nf = (float)a.n_tf;
  const float dt = a.dt;
  uint32_t n = 0;
  for (; w.j < j1; ++w.j) {
    const DevBrick b = a.bricks[__ldg(rb + w.j)];
    float t0, t1;
    if (!slab(ray, b.space_lo, b.space_hi, w.tmin, 1e10f, t0, t1)) continue;
    float t;
    uint32_t nb = 0;
    if (resume) {
      t = t_resume;
      nb = nb0;
      resume = false;
    } else {
      const float ils = jitter(a.jitter_mode, a.jitter_value, pixel, (uint32_t)a.accum_id, w.draw++);
      t = first_sample_t(t0, dt, ils);
    }
    const uint32_t cap = march_cap(t0, t1, dt);
    const bool exact = SKIP && exact_steps(t, t1, dt);
    const int mnx = (b.n[0] + kMacro - 1) >> kMacroShift, mny = (b.n[1] + kMacro - 1) >> kMacroShift;
    const float mag = fmaxf(fmaxf(fabsf(ray.o[0]) + fabsf(b.lo[0]), fabsf(ray.o[1]) + fabsf(b.lo[1])),
                            fabsf(ray.o[2]) + fabsf(b.lo[2])) + fabsf(t1);
    const float eps = 2e-6f * mag + 1e-4f;
    float inv_d[3];  // 1 / direction, once per brick (the lookups below reuse it)
    float inv_dt = 0.0f;
    if (SKIP) {
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) inv_d[ax] = 1.0f / ray.d[ax];
      inv_dt = 1.0f / dt;
    }
    // Samples before t_cell lie in a box of full macrocells and need no lookup.
    // (The render's alternation of jumps and short runs was slower here: 2.57
    // against 2.50 ms for the 256^3 density step.)
    float t_cell = t0;
    while (t < t1 && color.w < a.et_alpha && nb < cap) {
      if (n == max_samples) return n;
      if (CAN_STOP && *stop) return n;
      const float ux = fmaf(t, ray.d[0], ray.o[0]) - b.lo[0];
      const float uy = fmaf(t, ray.d[1], ray.o[1]) - b.lo[1];
      const float uz = fmaf(t, ray.d[2], ray.o[2]) - b.lo[2];
      if (SKIP && !(t < t_cell)) {
        const Cell cell = cell_at(b.cells, mnx, mny, b.n[0], b.n[1], b.n[2], ux, uy, uz);
        const float tb = cell_exit(cell, ray.d, ray.o[0] - b.lo[0], ray.o[1] - b.lo[1], ray.o[2] - b.lo[2], inv_d[0],
                                   inv_d[1], inv_d[2], eps, t1);
        if (!cell.empty()) {
          t_cell = tb;
        } else {
          ++n;
          ++nb;
          t = t + dt;
          n += exact ? run_steps(t, nb, tb, cap, dt, inv_dt, max_samples - n)
                     : run_steps_any(t, nb, tb, cap, dt, max_samples - n);
          continue;
        }
      }
      const StencilOut s = stencil<INNER, true>(b.base, b.sy, b.sz, b.n[0], b.n[1], b.n[2], ux, uy, uz);
      const float shade = shade_factor(s, ray);
      const float4 c = tf_lookup<INNER>(tf_s, a.n_tf, nf, s.value);
      visit(b, t, w, nb, ux, uy, uz, s, shade, c, color);
      composite_step(color, c, shade);
      ++n;
      ++nb;
      t = t + dt;
    }
    w.tmin = t1 + 1e-20f;
    if (!(color.w < a.et_alpha)) break;
  }
  return n;
}

// Stores the march state before every K-th sample (evaluated or skipped):
// colour, t, the brick walk position, tmin, the jitter draw index and the
// samples already taken in the brick.  The brick loop sets j, tmin, draw.
struct CheckpointHook {
  static constexpr bool kActive = true;
  Checkpoint* ck;
  uint32_t K, cap;
  int* overflow;
  uint32_t left = 0, m = 0;  // samples to the next checkpoint, checkpoints so far
  // Whether the open segment holds a full sample, and the closed segments that
  // do (bit m; segments beyond the 64th always count as holding one).
  bool full_segment = false;
  uint32_t full_lo = 0, full_hi = 0;
  __device__ __forceinline__ void close_segment() {
    if (full_segment) {
      const uint32_t i = m - 1;
      if (i < 32)
        full_lo |= 1u << i;
      else if (i < 64)
        full_hi |= 1u << (i - 32);
    }
    full_segment = false;
  }
  int j = 0;
  float tmin = 0.0f;
  uint32_t draw = 0;
  __device__ __forceinline__ void operator()(float t, uint32_t nb, const float4& col) {
    if (left == 0) {
      left = K;
      close_segment();
      if (m < cap) {
        Checkpoint c;
        c.r = col.x;
        c.g = col.y;
        c.b = col.z;
        c.a = col.w;
        c.t = t;
        c.tmin = tmin;
        c.jd = (uint32_t)j | (draw << 16);
        c.nb = nb;
        ck[m] = c;
      } else {
        atomicOr(overflow, 1);
      }
      ++m;
    }
    --left;
  }
};

// Training forward of one warp's 8 x 4 pixels at (x, y): the single rank's
// march (march_rank's brick walk with one draw, through march_brick, so the
// colour is the render's bit for bit), checkpoints, final colour, and the
// warp-aggregated append of (pixel, segment) items.  Returns the lane's
// sample count.
template <bool INNER>
__device__ __forceinline__ uint32_t train_subtile(const TrainArgs& a, const TrainView& tv, const DevView& v,
                                                  const float4* tf_s, int x, int y, int lane) {
  const bool active = x < v.width && y < v.height;
  uint32_t n = 0, nseg = 0;
  uint32_t pixel = 0;
  uint32_t full_lo = 0, full_hi = 0;
  if (active) {
    pixel = (uint32_t)x + (uint32_t)v.width * (uint32_t)y;
    const Ray ray = generate_ray(v, x, y);
    float4 color = make_float4(0.f, 0.f, 0.f, 0.f);
    CheckpointHook hook{tv.ckpt + (size_t)pixel * tv.ckpt_cap, a.k, tv.ckpt_cap, tv.overflow};
    const int* __restrict__ rb = rank_bricks(a, v);
    const int j1 = __ldg(a.sched + v.sched + 2);
    for (int j = 0; j < j1; ++j) {
      const DevBrick b = a.bricks[__ldg(rb + j)];
      float t0, t1;
      if (!slab(ray, b.space_lo, b.space_hi, hook.tmin, 1e10f, t0, t1)) continue;
      const float ils = jitter(a.jitter_mode, a.jitter_value, pixel, (uint32_t)a.accum_id, hook.draw++);
      hook.j = j;
      n += march_brick<INNER>(b, tf_s, a.n_tf, ray, t0, t1, ils, a.dt, a.et_alpha, a.tame, color, hook);
      hook.tmin = t1 + 1e-20f;
      if (!(color.w < a.et_alpha)) break;
    }
    tv.final_rgba[pixel] = color;
    if (tv.out_rgba) tv.out_rgba[pixel] = color;
    nseg = min((n + a.k - 1) / a.k, tv.ckpt_cap);
    hook.close_segment();
    full_lo = nseg < 32 ? hook.full_lo & ((1u << nseg) - 1u) : hook.full_lo;  // (nseg is short of the
    full_hi = nseg < 64 ? hook.full_hi & (nseg < 32 ? 0u : (1u << (nseg - 32)) - 1u)  // segments only on overflow)
                        : hook.full_hi;
  }
  // Warp-aggregated append of (pixel, segment) items, ordered by segment then
  // lane so that a backward warp replays neighbouring rays together.  Segments
  // that lie in empty macrocells altogether go to the list's back: their
  // samples have alpha 0, so they add nothing to the density or colour
  // gradients and leave the colour unchanged (backward_empty_kernel).
  const unsigned all = 0xffffffffu;
  const unsigned beyond = nseg > 64 ? nseg - 64 : 0;
  const unsigned nfull = __popc(full_lo) + __popc(full_hi) + beyond, nempty = nseg - nfull;
  // samples of the all-empty segments: K each, fewer in the ray's last one
  unsigned empty_samples = nempty * a.k;
  if (nseg > 0 && nseg <= 64 && !(((nseg <= 32 ? full_lo >> (nseg - 1) : full_hi >> (nseg - 33))) & 1u))
    empty_samples -= nseg * a.k - n;
  const unsigned total_full = __reduce_add_sync(all, nfull), total_empty = __reduce_add_sync(all, nempty);
  const unsigned total_samples = __reduce_add_sync(all, empty_samples);
  const unsigned maxseg = __reduce_max_sync(all, nseg);
  unsigned base = 0, ebase = 0;
  if (lane == 0) {
    if (total_full) base = atomicAdd(tv.work_count, total_full);
    if (total_empty) {
      ebase = atomicAdd(tv.work_count + 1, total_empty);
      atomicAdd(reinterpret_cast<unsigned long long*>(tv.work_count + 2), (unsigned long long)total_samples);
    }
  }
  base = __shfl_sync(all, base, 0);
  ebase = tv.work_cap - 1u - __shfl_sync(all, ebase, 0);
  const unsigned below = (1u << lane) - 1u;
  for (unsigned m = 0; m < maxseg; ++m) {
    const bool full = m >= 64 || ((m < 32 ? full_lo >> m : full_hi >> (m - 32)) & 1u);
    const unsigned in = __ballot_sync(all, m < nseg), f = __ballot_sync(all, full) & in, e = in & ~f;
    if (m < nseg) {
      const unsigned slot = full ? base + __popc(f & below) : ebase - __popc(e & below);
      if (slot < tv.work_cap) tv.work[slot] = make_uint2(pixel, m);
    }
    base += __popc(f);
    ebase -= __popc(e);
  }
  return n;
}

// Item `item` of a forward launch -> (view slot, chunk position): the run
// holding it (binary search over the few runs), then position-major within
// the run.
__device__ __forceinline__ void forward_item(const TrainArgs& a, unsigned item, int& slot, int& pos) {
  int lo = 0, hi = a.n_runs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&a.runs[mid].item0) <= item)
      lo = mid;
    else
      hi = mid - 1;
  }
  const int p0 = __ldg(&a.runs[lo].p0), active = __ldg(&a.runs[lo].active);
  const unsigned off = item - __ldg(&a.runs[lo].item0);
  pos = p0 + (int)(off / (unsigned)active);
  slot = __ldg(a.run_views + off % (unsigned)active);
}

// Persistent training forward over the launch's views: warps pull items
// (a view's 8 x 4 chunk, in its cost order when it has one, else
// centre-out, as the render does) from the launch's counter.
template <bool INNER>
__global__ void __launch_bounds__(128, kTrainForwardBlocks) forward_train_kernel(TrainArgs a, unsigned items) {
  extern __shared__ float4 tf_s[];
  load_tf(tf_s, a.tf, a.n_tf);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint32_t n = 0;
  for (;;) {
    unsigned item = 0;
    if (lane == 0) item = atomicAdd(a.grab, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= items) break;
    int slot, pos;
    forward_item(a, item, slot, pos);
    const TrainView& tv = a.tv[slot];
    const DevView v = a.views[tv.view];
    const int cxn = (v.width + 7) / 8, cyn = (v.height + 3) / 4;
    int ccx, ccy;
    if (tv.chunk_order) {
      const int id = __ldg(tv.chunk_order + pos);
      ccx = id % cxn;
      ccy = id / cxn;
    } else if (!ring_chunk(pos, cxn, cyn, ccx, ccy)) {
      continue;
    }
    n += train_subtile<INNER>(a, tv, v, tf_s, ccx * 8 + tile_x(lane), ccy * 4 + tile_y(lane), lane);
  }
  count_samples(a.counter, n);
}

__device__ __forceinline__ void red_add(float* p, float v) {
  if (v != 0.f) atomicAdd(p, v);
}

// Adds weights of brick voxels (x..x+2, y, z) (y, z already clamped to the
// brick) into the quad gradient: one float4 atomic when the three voxels are
// inside the brick, else one scalar atomic per clamped voxel.
__device__ __forceinline__ void scatter3(const TrainArgs& a, const DevBrick& b, const int4 org, int x, int y, int z,
                                         float w0, float w1, float w2) {
  if (w0 == 0.f && w1 == 0.f && w2 == 0.f) return;
  float4* row = a.dgrid4 + ((size_t)(z + org.z) * a.grid_dims[1] + (size_t)(y + org.y)) * a.grid_dims[0] + org.x;
  if (x >= 0 && x + 2 < b.n[0]) {
    atomicAdd(row + x, make_float4(w0, w1, w2, 0.f));
  } else {
    const int hi = b.n[0] - 1;
    red_add(&row[min(max(x, 0), hi)].x, w0);
    red_add(&row[min(max(x + 1, 0), hi)].x, w1);
    red_add(&row[min(max(x + 2, 0), hi)].x, w2);
  }
}

// The same for voxels (x, x+1): one float2 atomic on the quad's first half.
__device__ __forceinline__ void scatter2(const TrainArgs& a, const DevBrick& b, const int4 org, int x, int y, int z,
                                         float w0, float w1) {
  if (w0 == 0.f && w1 == 0.f) return;
  float4* row = a.dgrid4 + ((size_t)(z + org.z) * a.grid_dims[1] + (size_t)(y + org.y)) * a.grid_dims[0] + org.x;
  if (x >= 0 && x + 1 < b.n[0]) {
    atomicAdd(reinterpret_cast<float2*>(row + x), make_float2(w0, w1));
  } else {
    const int hi = b.n[0] - 1;
    red_add(&row[min(max(x, 0), hi)].x, w0);
    red_add(&row[min(max(x + 1, 0), hi)].x, w1);
  }
}

// Density-gradient scatter of one sample: the 20 voxels of the stencil with
// their combined weights (value tap and the six gradient taps), as 4 row
// quads and 4 row pairs.  Indices are clamped to the brick (the derivative of
// clamp addressing) and mapped to the caller's grid, so ghost and apron copies
// accumulate into the voxel they copy.
__device__ __forceinline__ void stencil_backward(const DevBrick& b, const TrainArgs& a, int brick, float ux,
                                                 float uy, float uz, float dv, float dgx, float dgy, float dgz) {
  // the forward stencil's coordinates (same indices and weights)
  const AxisCoord X = axis_coord(ux, b.n[0]), Y = axis_coord(uy, b.n[1]), Z = axis_coord(uz, b.n[2]);
  const float fx = X.f, fy = Y.f, fz = Z.f, gx = X.g, gy = Y.g, gz = Z.g;
  const bool hx = X.h, hy = Y.h, hz = Z.h;
  const int ix = X.i, iy = Y.i, iz = Z.i, cx = X.c, cy = Y.c, cz = Z.c;
  const int4 org = a.brick_grid_origin[brick];
  const int ny1 = b.n[1] - 1, nz1 = b.n[2] - 1;
  const float wx[2] = {1.f - gx, gx}, wy[2] = {1.f - gy, gy}, wz[2] = {1.f - gz, gz};
  const float wxg[3] = {-(1.f - fx), (1.f - fx) - fx, fx};
  const float wyg[3] = {-(1.f - fy), (1.f - fy) - fy, fy};
  const float wzg[3] = {-(1.f - fz), (1.f - fz) - fz, fz};
  const float wv[3] = {hx ? 0.f : wx[0], hx ? wx[0] : wx[1], hx ? wx[1] : 0.f};
  const int myc = hy ? 1 : 0, mzc = hz ? 1 : 0;
#pragma unroll
  for (int l = 0; l < 2; ++l)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float wyz = wy[j] * wz[l];
      const float side = fmaf(dgy * wyg[myc + j], wz[l], dgz * wzg[mzc + l] * wy[j]);
      float w[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) w[k] = fmaf(wyz, fmaf(dgx, wxg[k], dv * wv[k]), wv[k] * side);
      scatter3(a, b, org, ix, min(max(cy + j, 0), ny1), min(max(cz + l, 0), nz1), w[0], w[1], w[2]);
    }
  const int ye = min(max(hy ? iy : iy + 2, 0), ny1), ze = min(max(hz ? iz : iz + 2, 0), nz1);
  const float wye = dgy * wyg[hy ? 0 : 2], wze = dgz * wzg[hz ? 0 : 2];
#pragma unroll
  for (int l = 0; l < 2; ++l)
    scatter2(a, b, org, cx, ye, min(max(cz + l, 0), nz1), wye * wx[0] * wz[l], wye * wx[1] * wz[l]);
#pragma unroll
  for (int j = 0; j < 2; ++j)
    scatter2(a, b, org, cx, min(max(cy + j, 0), ny1), ze, wze * wx[0] * wy[j], wze * wx[1] * wy[j]);
}

// out[v] += q[v].x + q[v-1].y + q[v-2].z along x (each voxel written by one
// thread), leaving every quad it read zero again: a quad is rewritten only if
// it was nonzero, so a backward that touched part of the grid pays for that
// part only, and the next backward finds the buffer clear without a memset.
// CTAs take grid rows (y, z) and walk each in chunks of blockDim.x quads
// staged in shared memory behind the previous chunk's last two, so no quad
// is cleared before its three readers have it.
__global__ void fold_quads_kernel(float4* __restrict__ q, float* __restrict__ out, int dx, int rows) {
  extern __shared__ float4 sq[];  // [2 + blockDim.x]: q[x0-2], q[x0-1], then the chunk
  const int bd = (int)blockDim.x, i = (int)threadIdx.x;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    float4* __restrict__ qr = q + (size_t)r * dx;
    float* __restrict__ orow = out + (size_t)r * dx;
    if (i < 2) sq[i] = zero;
    for (int x0 = 0; x0 < dx; x0 += bd) {
      const int x = x0 + i;
      const float4 v = x < dx ? qr[x] : zero;
      sq[2 + i] = v;
      __syncthreads();
      if (x < dx) {
        float s = v.x;
        if (x >= 1) s += sq[1 + i].y;
        if (x >= 2) s += sq[i].z;
        if (s != 0.f) orow[x] += s;
        if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f) qr[x] = zero;
      }
      __syncthreads();
      if (i < 2) sq[i] = sq[bd + i];
      __syncthreads();
    }
  }
}

// Adds a pending transfer-function gradient (four channels of entry e) to this
// lane's copy in shared memory.
__device__ __forceinline__ void add_tf_entry(float* dtf_s, int copies, int n, int e, const float* pend) {
  if (e < 0 || e >= n) return;
  float* p = dtf_s + e * 4 * copies;
#pragma unroll
  for (int ch = 0; ch < 4; ++ch)
    if (pend[ch] != 0.f) atomicAdd(p + ch * copies, pend[ch]);
}

// Adds the pending gradient of entries i and i + 1.
__device__ __forceinline__ void flush_tf(float* dtf_s, int copies, int n, int i, const float pend[8]) {
  add_tf_entry(dtf_s, copies, n, i, pend);
  add_tf_entry(dtf_s, copies, n, i + 1, pend + 4);
}

// Near-opaque samples.  The closed form for the adjoint of the accumulated
// alpha after sample i,
//     gA = (g_a (1 - a_N) - g_rgb . (rgb_N - rgb_{i+1})) / (1 - a_{i+1}),
// divides two vanishing quantities once a sample leaves almost no
// transmittance, and gives 0 for a sample of alpha exactly 1 (1 - a = 0),
// where the true value is g_a R_a - g_rgb . R_rgb with R the composite of the
// rest of the ray normalised to the transmittance after the sample:
//     R_a = prod_j (1 - alpha_j),  R_rgb = sum_j prod_{l<j} (1 - alpha_l) alpha_j s_j c_j.
// The replay records such a sample as an event (the closed form stands in
// for it meanwhile); after the segment, suffix_composite marches on from the
// sample after it and the event's alpha adjoint is corrected by the
// difference.  A ray has at most three events: each one cuts the
// transmittance by more than 256 from above kVisible.
constexpr float kOpaqueStep = 1.0f / 256.0f;  // alpha above 1 - 1/256
constexpr float kVisible = 1e-5f;             // ... and the sample not hidden already
constexpr int kMaxEvents = 3;

struct OpaqueEvent {
  Walk w;          // walk position of the sample (next jitter draw)
  float t_next;    // t and brick sample count of the sample after it
  uint32_t nb_next;
  float4 after;    // colour after the sample
  float oma;       // transmittance before it
  float gA;        // the closed form's value
  float value;     // interpolated value (transfer-function lookup)
  float ux, uy, uz;
  int brick;
};

// R after an event: the forward's following samples replayed from
// (w, t_next, nb_next) with the colour after the event (so that early
// termination ends the ray where the forward ended it), until R's
// transmittance is below 2^-24 (the rest cannot move the result) or the ray
// ends.  Skipped samples (alpha 0) leave R unchanged, so empty space is
// stepped over.  Returns (R_rgb, R_a).
template <bool INNER>
__device__ __forceinline__ float4 suffix_composite(const TrainArgs& a, const DevView& v, const float4* tf_s,
                                                   const Ray& ray, uint32_t pixel, const OpaqueEvent& e) {
  float r0 = 0.f, r1 = 0.f, r2 = 0.f, tp = 1.0f;
  bool stop = false;
  float4 col = e.after;
  walk_samples<INNER, true, true>(
      a, v, tf_s, ray, pixel, e.w, e.t_next, e.nb_next, true, col, 0xffffffffu,
      [&](const DevBrick&, float, const Walk&, uint32_t, float, float, float, const StencilOut&, float shade,
          const float4& c, const float4&) {
        const float k = tp * c.w * shade;
        r0 = fmaf(k, c.x, r0);
        r1 = fmaf(k, c.y, r1);
        r2 = fmaf(k, c.z, r2);
        tp = tp * (1.0f - c.w);
        if (tp < 5.96e-8f) stop = true;
      },
      &stop);
  return make_float4(r0, r1, r2, tp);
}

// Copies of the transfer-function gradient in a replaying CTA's shared memory,
// interleaved (a lane's copy has banks of its own): adding to a float there is a
// loop until no other lane interferes.  As many as fit kTfCopyBytes, which at 5
// CTAs per SM leaves the L1 its share.  With one copy / 2 / 4 / 8, ms: one 512^3
// view's transfer-function step 5.64 / 5.46 / 5.35 / 5.34, 16 views of 128^3, both
// gradients, 2.39 / 2.31 / 2.27 / 2.27, 2 views of 512^3 13.4 / 13.2 / 13.05 / 13.2;
// moving a sum along with the lookup index (backward_item) then 5.25, 2.27, 12.9.
// Bytes, 512 entries, 512^3 backward: 23 KB (1 copy) 5.04, 36 (2) 4.96, 64 (4) 5.09.
constexpr int kTfCopies = 4;
constexpr size_t kTfCopyBytes = 36 * 1024;
constexpr int kBackwardEmptyBlocks = 6;   // CTAs per SM of the all-empty segments' kernel
constexpr unsigned kBackwardGrab = 256;  // most items a backward warp takes per grab (8 rows of 32)

// One backward item: the replay of segment (pixel, ck) of view v and its
// adjoint, added to dtf_s (shared, WITH_TF) and the x-quad density gradient
// (WITH_DENSITY).  Returns the samples replayed.
template <bool INNER, bool WITH_TF, bool WITH_DENSITY>
__device__ __forceinline__ uint32_t backward_item(const TrainArgs& a, const DevView& v, const int* __restrict__ rb,
                                                  const float4* tf_s, float* dtf_s, float nf, uint32_t pixel,
                                                  const Checkpoint& ck, const float4 F, const float4 g) {
  const int x = (int)(pixel % (uint32_t)v.width), y = (int)(pixel / (uint32_t)v.width);
  const Ray ray = generate_ray(v, x, y);
  const float gfin = g.w * (1.0f - F.w);
  float4 color = make_float4(ck.r, ck.g, ck.b, ck.a);
  const Walk w0{(int)(ck.jd & 0xffffu), ck.tmin, ck.jd >> 16};
  // transfer-function gradient of consecutive samples with the same lookup
  // index is summed in registers and added to shared memory once per index
  int pend_i = INT_MIN;
  float pend[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  OpaqueEvent events[kMaxEvents];
  int n_events = 0;
  const uint32_t n = walk_samples<INNER, !WITH_TF>(
      a, v, tf_s, ray, pixel, w0, ck.t, ck.nb, true, color, a.k,
      [&](const DevBrick& b, float t, const Walk& wcur, uint32_t nb, float ux, float uy, float uz,
          const StencilOut& s, float shade, const float4& c, const float4& col) {
        // Backward-only arithmetic below is free to contract and to use
        // approximate reciprocals (the gradient tolerance is relative); the
        // replay that feeds it is the exact forward.
        float4 nxt = col;  // state after this sample
        composite_step(nxt, c, shade);
        const float oma = 1.0f - col.w;
        const float tn1 = 1.0f - nxt.w;
        // dL/d(accumulated alpha after this sample), closed form
        const float gA =
            __fdividef(gfin - fmaf(g.x, F.x - nxt.x, fmaf(g.y, F.y - nxt.y, g.z * (F.z - nxt.z))),
                       fmaxf(tn1, 1e-6f));
        if (tn1 < kOpaqueStep * oma && oma > kVisible && n_events < kMaxEvents) {
          OpaqueEvent& e = events[n_events++];
          e.w = wcur;
          e.t_next = t + a.dt;
          e.nb_next = nb + 1;
          e.after = nxt;
          e.oma = oma;
          e.gA = gA;
          e.value = s.value;
          e.ux = ux;
          e.uy = uy;
          e.uz = uz;
          e.brick = __ldg(rb + wcur.j);
        }
        const float gc = fmaf(g.x, c.x, fmaf(g.y, c.y, g.z * c.z));
        const float dA = oma * fmaf(shade, gc, gA);  // dL/d(alpha of this sample)
        // transfer function lookup backward (the lookup of tf_lookup)
        const float xb = s.value * nf - 0.5f;
        const int i0 = __float2int_rd(xb);
        const float wt = xb - (float)i0;
        const int ic = min(max(i0, -2), a.n_tf);
        const float4 e0 = tf_s[ic + 2], e1 = tf_s[ic + 3];
        if (WITH_TF && i0 != pend_i) {
          // moved by one entry: one sum is complete, the other moves along
          const bool up = i0 == pend_i + 1, down = i0 == pend_i - 1;
          if (!down) add_tf_entry(dtf_s, a.tf_copies, a.n_tf, pend_i, pend);
          if (!up) add_tf_entry(dtf_s, a.tf_copies, a.n_tf, pend_i + 1, pend + 4);
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            const float lo = pend[ch];
            pend[ch] = up ? pend[4 + ch] : 0.f;
            pend[4 + ch] = down ? lo : 0.f;
          }
          pend_i = i0;
        }
        if (e0.w == 0.f && e1.w == 0.f) {
          // Alpha is exactly 0 at this sample: only the two alpha entries of
          // the lookup receive gradient; the colour entries, the shading and
          // the density gradients all carry a factor alpha or d(alpha)/dv = 0.
          if (WITH_TF) {
            pend[3] = fmaf(1.f - wt, dA, pend[3]);
            pend[7] = fmaf(wt, dA, pend[7]);
          }
          return;
        }
        const float kc = oma * c.w * shade;
        const float dch[4] = {g.x * kc, g.y * kc, g.z * kc, dA};
        if (WITH_TF) {
  #pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            pend[ch] = fmaf(1.f - wt, dch[ch], pend[ch]);
            pend[4 + ch] = fmaf(wt, dch[ch], pend[4 + ch]);
          }
        }
        if (!WITH_DENSITY) return;
        const float ds = oma * c.w * gc;
        const float de[4] = {e1.x - e0.x, e1.y - e0.y, e1.z - e0.z, e1.w - e0.w};
        float dv = 0.f;
  #pragma unroll
        for (int ch = 0; ch < 4; ++ch) dv = fmaf(dch[ch], de[ch], dv);
        dv *= nf;
        // shading backward: s = .1 + .9 |q|, q = (g.d)/|g + 1e-4|
        const float ex = s.gx + 1e-4f, ey = s.gy + 1e-4f, ez = s.gz + 1e-4f;
        const float len2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
        const float inv = rsqrtf(len2);
        const float gd = fmaf(s.gx, ray.d[0], fmaf(s.gy, ray.d[1], s.gz * ray.d[2]));
        const float kk = ds * 0.9f * (gd > 0.f ? 1.f : (gd < 0.f ? -1.f : 0.f));
        const float c3 = gd * inv * inv * inv;
        const float ki = kk * inv, kc3 = kk * c3;
        stencil_backward(b, a, __ldg(rb + wcur.j), ux, uy, uz, dv, fmaf(ki, ray.d[0], -kc3 * ex),
                         fmaf(ki, ray.d[1], -kc3 * ey), fmaf(ki, ray.d[2], -kc3 * ez));
      });
  if (WITH_TF) flush_tf(dtf_s, a.tf_copies, a.n_tf, pend_i, pend);
  // near-opaque samples: correct the alpha adjoint by the true one
  for (int k = 0; k < n_events; ++k) {
    const OpaqueEvent& e = events[k];
    const float4 R = suffix_composite<INNER>(a, v, tf_s, ray, pixel, e);
    const float gtrue = fmaf(g.w, R.w, -fmaf(g.x, R.x, fmaf(g.y, R.y, g.z * R.z)));
    const float dd = e.oma * (gtrue - e.gA);  // change of dL/d(alpha of the sample)
    if (dd == 0.f) continue;
    const float xb = e.value * nf - 0.5f;
    const int i0 = __float2int_rd(xb);
    const float wt = xb - (float)i0;
    if (WITH_TF) {
      if (i0 >= 0 && i0 < a.n_tf) atomicAdd(dtf_s + (i0 * 4 + 3) * a.tf_copies, (1.f - wt) * dd);
      if (i0 + 1 >= 0 && i0 + 1 < a.n_tf) atomicAdd(dtf_s + ((i0 + 1) * 4 + 3) * a.tf_copies, wt * dd);
    }
    if (WITH_DENSITY) {
      const int ic = min(max(i0, -2), a.n_tf);
      const float dv = nf * dd * (tf_s[ic + 3].w - tf_s[ic + 2].w);
      if (dv != 0.f) {
        const DevBrick b = a.bricks[e.brick];
        stencil_backward(b, a, e.brick, e.ux, e.uy, e.uz, dv, 0.f, 0.f, 0.f);
      }
    }
  }
  return n;
}

// WITH_TF: the transfer-function gradient; WITH_DENSITY: the density
// gradient (at least one of them).  Without the transfer-function gradient
// the replay skips empty macrocells like the forward: a sample there has
// transfer-function alpha 0 at both lookup entries, so its density and
// shading gradients vanish and only the alpha entries would receive any.
// Without the density gradient the shading and stencil adjoints are skipped.
// MULTI: the launch's items belong to several views (item_base, tv), each
// item looks its view up; else to the one view passed in the parameters
// (a.one), whose pointers then stay in the constant bank, as the replay's
// register budget wants.
template <bool INNER, bool WITH_TF, bool WITH_DENSITY, bool MULTI>
__global__ void __launch_bounds__(128, 5) backward_kernel(TrainArgs a) {
  extern __shared__ float4 smem[];
  float4* tf_s = smem;                                         // n_tf + 4 entries
  float* dtf_all = reinterpret_cast<float*>(smem + a.n_tf + 4);  // n_tf * 4 * tf_copies (WITH_TF)
  float* dtf_s = WITH_TF ? dtf_all + (threadIdx.x & (a.tf_copies - 1)) : nullptr;
  load_tf(tf_s, a.tf, a.n_tf);
  if (WITH_TF)
    for (int i = threadIdx.x; i < a.n_tf * 4 * a.tf_copies; i += blockDim.x) dtf_all[i] = 0.f;
  __syncthreads();
  const unsigned count = MULTI ? __ldg(a.item_base + a.n_views) : a.one_items;
  const float nf = (float)a.n_tf;
  uint32_t nsamp = 0;
  DevView v1{};
  const int* rb1 = nullptr;
  if constexpr (!MULTI) {
    v1 = a.views[a.one.view];
    rb1 = rank_bricks(a, v1);
  }
  // Warps take kBackwardGrab consecutive items at a time.  The forward lays
  // out each of its 8x4 tiles as rows of 32 (segment m of every lane, then
  // m + 1, ...), so a warp replays consecutive segments of the same rays and
  // finds the bricks warm in L1 from the previous segment.
  // The grab shrinks (to one row) when there are too few items to give every
  // warp several grabs.
  const unsigned lane = threadIdx.x & 31u;
  const unsigned warps = gridDim.x * (blockDim.x / 32u);
  const unsigned take = max(32u, min(kBackwardGrab, (count / (warps * 8u)) & ~31u));
  for (;;) {
    unsigned grab = 0;
    if (lane == 0) grab = atomicAdd(a.grab, take);
    grab = __shfl_sync(0xffffffffu, grab, 0);
    if (grab >= count) break;
    const unsigned end = min(grab + take, count);
    for (unsigned item = grab + lane; item < end; item += 32u) {
      if constexpr (MULTI) {
        int slot = 0;  // item_base[slot] <= item < item_base[slot + 1]
        for (int hi = a.n_views - 1; slot < hi;) {
          const int mid = (slot + hi + 1) >> 1;
          if (__ldg(a.item_base + mid) <= item)
            slot = mid;
          else
            hi = mid - 1;
        }
        const TrainView& tv = a.tv[slot];
        const DevView v = a.views[tv.view];
        const uint2 wk = tv.work[item - __ldg(a.item_base + slot)];
        const Checkpoint ck = tv.ckpt[(size_t)wk.x * tv.ckpt_cap + wk.y];
        nsamp += backward_item<INNER, WITH_TF, WITH_DENSITY>(a, v, rank_bricks(a, v), tf_s, dtf_s, nf, wk.x, ck,
                                                      tv.final_rgba[wk.x], tv.dl_drgba[wk.x]);
      } else {
        const uint2 wk = a.one.work[item];
        const Checkpoint ck = a.one.ckpt[(size_t)wk.x * a.one.ckpt_cap + wk.y];
        nsamp += backward_item<INNER, WITH_TF, WITH_DENSITY>(a, v1, rb1, tf_s, dtf_s, nf, wk.x, ck, a.one.final_rgba[wk.x],
                                                      a.one.dl_drgba[wk.x]);
      }
    }
  }
  count_samples(a.counter, nsamp);
  if (WITH_TF) {
    __syncthreads();
    for (int i = threadIdx.x; i < a.n_tf * 4; i += blockDim.x) {
      float v = 0.f;
      for (int c = 0; c < a.tf_copies; ++c) v += dtf_all[i * a.tf_copies + c];
      red_add(a.dtf + i, v);
    }
  } else if (a.counter && blockIdx.x == 0) {
    // the samples of all-empty segments, which nothing replays
    for (int i = threadIdx.x; i < a.n_views; i += blockDim.x)
      atomicAdd(a.counter, *reinterpret_cast<const unsigned long long*>((MULTI ? a.tv[i] : a.one).work_count + 2));
  }
}

// All-empty segments (every sample in an empty macrocell, so of alpha exactly
// 0): the gradient of the transfer function's alpha entries,
//     dL/d(alpha of the sample) = (1 - a)(s g.c + gA),
// with the colour of the segment's checkpoint for all its samples.  No sample
// waits for the one before it and nothing here has to round as the forward
// does: no composite, an approximate reciprocal square root in the shading, two
// pending sums instead of eight.  Bound by the L1 data pipe (83 % busy), mostly
// with the stencil's 96 bytes per sample: so two lanes take a segment's samples
// in turn, and a quarter warp, the unit of 16-byte loads, covers 2x2 rays by two
// samples, whose quads collide in fewer banks than those of 2x4 rays (counting
// the quads that share a 16-byte bank group: 41 instead of 55 cycles for a warp's
// seven loads at 0.83 voxels per pixel).  The two lanes want the same bins, and adding to a
// float in shared memory is a loop until no other lane interferes, so the bins
// are kept in COPIES, interleaved so that a lane's copy has banks of its own.
// Per pass of a 512^3 1024^2 transfer-function step, ms: one lane and one copy
// 5.95, two lanes 6.51, two lanes and 2 / 4 / 8 / 16 / 32 copies 5.95 / 5.78 /
// 5.67 / 5.62 / 6.09, one lane and 2 / 16 copies 5.83 / 5.89; at 5 / 7 / 8 CTAs
// per SM 1.7 / 1.8 / 7.4 % slower.  One 512^3 view's transfer-function backward
// with every segment replayed: 5.82 ms; 1.20 ms for the replayed ones and 3.08
// here.  The density-only replay of 6 views of 256^3, which only loses the empty
// rows between its lanes, went from 2.2 to 1.3 ms with the split.
template <bool INNER, bool MULTI, int COPIES>
__global__ void __launch_bounds__(128, kBackwardEmptyBlocks) backward_empty_kernel(TrainArgs a) {
  extern __shared__ float4 smem[];
  float4* tf_s = smem;                                         // n_tf + 4 entries
  float* dalpha_s = reinterpret_cast<float*>(smem + a.n_tf + 4);  // n_tf + 4: alpha entries, two unused on each side
  load_tf(tf_s, a.tf, a.n_tf);
  for (int i = threadIdx.x; i < (a.n_tf + 4) * COPIES; i += blockDim.x) dalpha_s[i] = 0.f;
  float* const bins = dalpha_s + threadIdx.x % COPIES;
  __syncthreads();
  const unsigned count = MULTI ? __ldg(a.empty_base + a.n_views) : a.one_empty;
  const float nf = (float)a.n_tf, dt = a.dt;
  uint32_t nsamp = 0;
  const unsigned lane = threadIdx.x & 31u;
  const bool second = lane & 1u;  // two lanes per item: the samples at even and odd places
  const unsigned warps = gridDim.x * (blockDim.x / 32u);
  const unsigned take = max(32u, min(kBackwardGrab, (count / (warps * 8u)) & ~31u));
  for (;;) {
    unsigned grab = 0;
    if (lane == 0) grab = atomicAdd(a.grab + 1, take);
    grab = __shfl_sync(0xffffffffu, grab, 0);
    if (grab >= count) break;
    const unsigned end = min(grab + take, count);
    for (unsigned item = grab + (lane >> 1); item < end; item += 16u) {
      int slot = 0;
      unsigned first = 0;
      if constexpr (MULTI) {
        for (int hi = a.n_views - 1; slot < hi;) {  // empty_base[slot] <= item < empty_base[slot + 1]
          const int mid = (slot + hi + 1) >> 1;
          if (__ldg(a.empty_base + mid) <= item)
            slot = mid;
          else
            hi = mid - 1;
        }
        first = __ldg(a.empty_base + slot);
      }
      const TrainView& tv = MULTI ? a.tv[slot] : a.one;
      const DevView& v = a.views[tv.view];
      const uint2 wk = tv.work[tv.work_cap - 1u - (item - first)];
      const Checkpoint ck = tv.ckpt[(size_t)wk.x * tv.ckpt_cap + wk.y];
      const float4 F = tv.final_rgba[wk.x], g = tv.dl_drgba[wk.x];
      const int* __restrict__ rb = rank_bricks(a, v);
      const int j1 = __ldg(a.sched + v.sched + 2);
      const Ray ray = generate_ray(v, (int)(wk.x % (uint32_t)v.width), (int)(wk.x / (uint32_t)v.width));
      const float oma = 1.0f - ck.a;
      const float gA = __fdividef(g.w * (1.0f - F.w) -
                                      fmaf(g.x, F.x - ck.r, fmaf(g.y, F.y - ck.g, g.z * (F.z - ck.b))),
                                  fmaxf(oma, 1e-6f));
      int j = (int)(ck.jd & 0xffffu);
      uint32_t draw = ck.jd >> 16, n = 0, nb = ck.nb;
      float tmin = ck.tmin, t = ck.t;
      int pend_i = -2;
      float pend0 = 0.f, pend1 = 0.f;
      float gc0 = 0.f, gcd = 0.f;  // g.c at the pending index's entry, and the step to the next one (alpha 0 entries)
      for (bool resume = true; j < j1 && n < a.k; ++j) {
        const DevBrick& b = a.bricks[__ldg(rb + j)];
        float t0, t1;
        if (!slab(ray, b.space_lo, b.space_hi, tmin, 1e10f, t0, t1)) continue;
        if (!resume) {
          t = first_sample_t(t0, dt, jitter(a.jitter_mode, a.jitter_value, wk.x, (uint32_t)a.accum_id, draw++));
          nb = 0;
        }
        resume = false;
        const uint32_t cap = march_cap(t0, t1, dt);
        const float4* __restrict__ base = b.base;
        const int sy = b.sy, sz = b.sz, nx = b.n[0], ny = b.n[1], nz = b.n[2];
        const float lox = b.lo[0], loy = b.lo[1], loz = b.lo[2];
        while (t < t1 && nb < cap && n < a.k) {
          // two samples at a time; without a second one its lane adds nothing
          const float t2 = t + dt;
          const bool two = t2 < t1 && nb + 1 < cap && n + 1 < a.k;
          const float tk = second && two ? t2 : t;
          const StencilOut s =
              stencil<INNER, true>(base, sy, sz, nx, ny, nz, fmaf(tk, ray.d[0], ray.o[0]) - lox,
                                   fmaf(tk, ray.d[1], ray.o[1]) - loy, fmaf(tk, ray.d[2], ray.o[2]) - loz);
          const float ex = s.gx + 1e-4f, ey = s.gy + 1e-4f, ez = s.gz + 1e-4f;
          const float inv = rsqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
          const float gd = fmaf(s.gx, ray.d[0], fmaf(s.gy, ray.d[1], s.gz * ray.d[2]));
          const float shade = fmaf(0.9f, fabsf(gd * inv), 0.1f);
          const float xb = s.value * nf - 0.5f;
          const int i0 = __float2int_rd(xb);
          const float wt = xb - (float)i0;
          const int ic = min(max(i0, -2), a.n_tf);
          // the lookup index mostly moves by one: then one sum is complete and
          // the other moves along
          const int step = ic - pend_i;
          if (step != 0) {
            const bool down = step == -1;
            atomicAdd(bins + (pend_i + (down ? 3 : 2)) * COPIES, down ? pend1 : pend0);
            if (step != 1 && !down) atomicAdd(bins + (pend_i + 3) * COPIES, pend1);
            const float next0 = step == 1 ? pend1 : 0.f;
            pend1 = down ? pend0 : 0.f;
            pend0 = next0;
            pend_i = ic;
            const float4 e0 = tf_s[ic + 2], e1 = tf_s[ic + 3];
            gc0 = fmaf(g.x, e0.x, fmaf(g.y, e0.y, g.z * e0.z));
            gcd = fmaf(g.x, e1.x, fmaf(g.y, e1.y, g.z * e1.z)) - gc0;
          }
          const float dA = second && !two ? 0.f : oma * fmaf(shade, fmaf(wt, gcd, gc0), gA);
          pend0 = fmaf(1.f - wt, dA, pend0);
          pend1 = fmaf(wt, dA, pend1);
          n += two ? 2 : 1;
          nb += two ? 2 : 1;
          t = two ? t2 + dt : t2;
        }
        tmin = t1 + 1e-20f;
      }
      atomicAdd(bins + (pend_i + 2) * COPIES, pend0);
      atomicAdd(bins + (pend_i + 3) * COPIES, pend1);
      nsamp += second ? 0u : n;
    }
  }
  count_samples(a.counter, nsamp);
  __syncthreads();
  for (int i = threadIdx.x; i < a.n_tf; i += blockDim.x) {
    float v = 0.f;
    for (int c = 0; c < COPIES; ++c) v += dalpha_s[(i + 2) * COPIES + c];
    red_add(a.dtf + 4 * i + 3, v);
  }
}

size_t backward_smem(int n_tf, int tf_copies) {
  return (size_t)(n_tf + 4) * sizeof(float4) + (size_t)n_tf * 4 * sizeof(float) * tf_copies;
}

int backward_tf_copies(int n_tf) {
  for (int copies = kTfCopies; copies > 1; copies /= 2)
    if (backward_smem(n_tf, copies) <= kTfCopyBytes) return copies;
  return 1;
}

}  // namespace

cudaError_t launch_forward_train(const TrainArgs& a, unsigned items, int max_grid, bool inner, cudaStream_t s) {
  int grid = (int)std::min<unsigned>((items + 3) / 4, (unsigned)max_grid);
  if (grid < 1) grid = 1;
  const size_t smem = (size_t)(a.n_tf + 4) * sizeof(float4);
  if (inner)
    forward_train_kernel<true><<<grid, 128, smem, s>>>(a, items);
  else
    forward_train_kernel<false><<<grid, 128, smem, s>>>(a, items);
  return cudaGetLastError();
}

int forward_train_blocks_per_sm(int n_tf) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, forward_train_kernel<true>, 128,
                                                    (size_t)(n_tf + 4) * sizeof(float4)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

using BackwardKernel = void (*)(TrainArgs);
template <bool INNER>
static BackwardKernel backward(bool with_tf, bool with_density, bool multi) {
  if (multi)
    return !with_tf ? backward_kernel<INNER, false, true, true>
                    : (with_density ? backward_kernel<INNER, true, true, true> : backward_kernel<INNER, true, false, true>);
  return !with_tf ? backward_kernel<INNER, false, true, false>
                  : (with_density ? backward_kernel<INNER, true, true, false> : backward_kernel<INNER, true, false, false>);
}

cudaError_t launch_backward(const TrainArgs& args, int grid, bool inner, cudaStream_t s) {
  TrainArgs a = args;
  const bool with_tf = a.dtf != nullptr, with_density = a.dgrid4 != nullptr;
  a.tf_copies = with_tf ? backward_tf_copies(a.n_tf) : 0;
  if (!with_tf && !with_density) return cudaErrorInvalidValue;
  const size_t smem = backward_smem(a.n_tf, a.tf_copies);
  const bool multi = a.n_views > 1;
  const BackwardKernel k = inner ? backward<true>(with_tf, with_density, multi) : backward<false>(with_tf, with_density, multi);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k<<<grid, 128, smem, s>>>(a);
  return cudaGetLastError();
}

template <int COPIES>
static BackwardKernel backward_empty(bool inner, bool multi) {
  if (inner) return multi ? backward_empty_kernel<true, true, COPIES> : backward_empty_kernel<true, false, COPIES>;
  return multi ? backward_empty_kernel<false, true, COPIES> : backward_empty_kernel<false, false, COPIES>;
}

cudaError_t launch_backward_empty(const TrainArgs& a, int sms, bool inner, cudaStream_t s) {
  // As many copies of the bins as leave most of an SM's memory to the L1 (six
  // CTAs), at least two where they fit.  A 1024^2 backward of 512^3, us, by
  // entries, one thread per segment and one copy first: 16: 4807 / 4451 (16
  // copies), 256: 5267 / 4881 (16), 512: 5611 / 5237 (4), 1024: 5811 / 5789 (2;
  // 9260 with 4), 2044: 10476 / 7476 (2).
  auto bytes = [&](int copies) { return (size_t)(a.n_tf + 4) * (sizeof(float4) + copies * sizeof(float)); };
  const int copies = bytes(16) <= 23 * 1024 ? 16 : (bytes(4) <= 23 * 1024 ? 4 : (bytes(2) <= 48 * 1024 ? 2 : 1));
  const bool multi = a.n_views > 1;
  const BackwardKernel k = copies == 16  ? backward_empty<16>(inner, multi)
                           : copies == 4 ? backward_empty<4>(inner, multi)
                           : copies == 2 ? backward_empty<2>(inner, multi)
                                         : backward_empty<1>(inner, multi);
  k<<<sms * kBackwardEmptyBlocks, 128, bytes(copies), s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fold_quads(float4* quads, float* out, const int dims[3], cudaStream_t s) {
  const long long rows = (long long)dims[1] * dims[2];
  if (rows <= 0 || rows > 0x7fffffffll || dims[0] <= 0) return cudaErrorInvalidValue;
  const int threads = dims[0] >= 256 ? 256 : 128;
  const int grid = (int)(rows < 152 * 32 ? rows : 152 * 32);
  fold_quads_kernel<<<grid, threads, (threads + 2) * sizeof(float4), s>>>(quads, out, dims[0], (int)rows);
  return cudaGetLastError();
}

int backward_blocks_per_sm(int n_tf) {
  // the instance with the transfer-function gradient needs more shared memory
  const size_t smem = backward_smem(n_tf, backward_tf_copies(n_tf));
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(backward_kernel<true, true, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, backward_kernel<true, true, true, true>, 128, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace aloha
