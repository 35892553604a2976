// render.cu -- forward kernels: fused per-view render, persistent batched
// render, ordered-over composite, brick padding.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "internal.h"
#include "march.cuh"

namespace aloha {

// Half `half` (4x4 pixels) of an 8x4 chunk, two lanes per ray (march_brick_pair).
// INNER: the view and scene are InnerCoords.  Returns the samples, counted in
// the rays' first lanes.
template <bool INNER, class Loads>
__device__ __forceinline__ uint32_t render_half_chunk(const BatchArgs& b, const DevView& v, const float4* tf_s, int ccx,
                                                      int ccy, int half, int lane, uint32_t* fb, Loads& loads) {
  const int p = lane >> 1, x = ccx * 8 + 4 * half + pair_x(p), y = ccy * 4 + pair_y(p);
  if (x >= v.width || y >= v.height) return 0;  // both lanes of the ray
  const LaneGroup g{lane & 1, 3u << (lane & 30), lane & 30};
  const size_t at = (size_t)x + (size_t)v.width * y;
  uint32_t ns;
  if (INNER || (b.f.inner && v.inner && scene_inner(b.f)))
    ns = render_pixel<true, Loads, 2, true>(b.f, v, tf_s, x, y, fb, at, loads, g);
  else
    ns = render_pixel<false, Loads, 2, true>(b.f, v, tf_s, x, y, fb, at, loads, g);
  return g.lane == 0 ? ns : 0;
}

// Persistent render: every warp pulls CW x CH pixel chunks of the launch's
// items (views) from one atomic counter -- a single view in cost order when
// b.chunk_order is set (schedule.cu), else centre-out per view -- and renders
// each chunk as 8 x 4-pixel sub-tiles, so the 32 rays of a warp start within
// a few voxels of each other.  Warps are independent (no barrier after the
// transfer function is staged): a warp with long rays never holds finished
// warps of its CTA, and views end without a per-launch tail.  Nothing waits
// on other warps or CTAs.
// MINB CTAs of 128 threads per SM: a single view ends with its slowest
// chunks, which run faster with more registers per thread (5 CTAs, 96
// registers, or 4 when there are few chunks); a batch of views is
// throughput-bound and runs faster with more resident warps (7 CTAs, 72
// registers).
// STAGE selects the stencil loads: 0 direct, 1 the next sample's rows staged
// in shared memory with cp.async (StagedLoads; shared memory after the
// transfer function), kStageUnroll2 (batches) direct with the march loop
// written out two steps per trip.  LG == 2 (single view in cost order, 8x4
// chunks): the first *pair_chunks positions of an InnerCoords scene are two
// items each, the chunk's 4x4 halves with two lanes per ray.  LG == kRingPairs:
// the same for all positions of the ring order of any scene.  LG > 2 (single view in
// cost order, 8x4 chunks, frame buffer only): work positions [0, LG * group_chunks) are the costliest
// group_chunks chunks, each as LG items of 32 / LG pixels rendered by lane
// groups of LG lanes per ray; the remaining positions are the other chunks of
// the cost order, rendered as usual.
template <int CW, int CH, int MINB, int STAGE, int LG = 1>
__global__ void __launch_bounds__(kRenderThreads, MINB) render_warps_kernel(BatchArgs b) {
  extern __shared__ float4 tf_s[];
  load_tf(tf_s, b.f.tf, b.f.n_tf);
  __syncthreads();
  using Loads = typename std::conditional<
      STAGE == 1, StagedLoads,
      typename std::conditional<STAGE == kStageUnroll2, UnrolledDirectLoads<2>, DirectLoads>::type>::type;
  constexpr bool kOne = MINB < kBatchRenderBlocks;  // render_pixel's ONE
  Loads loads;
  if constexpr (STAGE == 1) loads.init(tf_s + (b.f.n_tf + 4));
  // pairs are for InnerCoords scenes alone here (fewer copies of the march)
  const bool may_pair =
      LG == 2 && b.pair_chunks && b.f.inner && b.f.views[b.single_view].inner && scene_inner(b.f);
  wait_for_primary();  // the chunk order and the cleared counters
  const int lane = threadIdx.x & 31;
  const int pairs = LG == kRingPairs ? b.total_tiles : (may_pair ? __ldcg(b.pair_chunks) : 0);
  uint32_t n = 0;
  for (;;) {
    int chunk = 0;
    if (lane == 0) chunk = (int)atomicAdd(b.work_counter, 1u);
    chunk = __shfl_sync(0xffffffffu, chunk, 0);
    if (chunk >= b.total_tiles + pairs) break;
    int item = 0, first = 0;
    if (b.tile_prefix) {
      // item = last index with tile_prefix[item] <= chunk
      int lo = 0, hi = b.n_items - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(b.tile_prefix + mid) <= chunk)
          lo = mid;
        else
          hi = mid - 1;
      }
      item = lo;
      first = __ldg(b.tile_prefix + item);
    }
    const DevView v = b.f.views[b.view_ids ? __ldg(b.view_ids + item) : b.single_view];
    uint32_t* fb = b.fbs ? b.fbs[item] : b.f.fb;
    int ccx, ccy;
    const int cxn = (v.width + CW - 1) / CW;
    if constexpr (LG == 2) {
      if (chunk < 2 * pairs) {
        const int id = __ldg(b.chunk_order + (chunk >> 1));
        n += render_half_chunk<true>(b, v, tf_s, id % cxn, id / cxn, chunk & 1, lane, fb, loads);
        continue;
      }
      chunk -= pairs;
    }
    if constexpr (LG == kRingPairs) {
      if (ring_chunk(chunk >> 1, cxn, (v.height + CH - 1) / CH, ccx, ccy))
        n += render_half_chunk<false>(b, v, tf_s, ccx, ccy, chunk & 1, lane, fb, loads);
      continue;
    }
    if constexpr (LG > 2) {
      if (chunk < b.group_chunks * LG) {
        const int id = __ldg(b.chunk_order + chunk / LG), part = chunk % LG;
        const int gl = lane % LG, p = part * (32 / LG) + lane / LG;
        const int x = (id % cxn) * 8 + (p & 7), y = (id / cxn) * 4 + (p >> 3);
        const LaneGroup g{gl, ((1u << LG) - 1u) << (lane - gl), lane - gl};
        // the group's lanes share x and y, so they take this branch together
        if (x < v.width && y < v.height) {
          const uint32_t ns =
              render_pixel<false, Loads, LG>(b.f, v, tf_s, x, y, fb, (size_t)x + (size_t)v.width * y, loads, g);
          if (gl == 0) n += ns;
        }
        continue;
      }
      chunk -= b.group_chunks * (LG - 1);  // position in the cost order of the remaining chunks
    }
    if (b.chunk_order) {
      const int id = __ldg(b.chunk_order + chunk);
      ccx = id % cxn;
      ccy = id / cxn;
    } else if (!ring_chunk(chunk - first, cxn, (v.height + CH - 1) / CH, ccx, ccy)) {
      continue;
    }
    const int x0 = ccx * CW, y0 = ccy * CH;
    // The march with unclamped coordinates (InnerCoords) or the clamped one,
    // decided per chunk from device memory, so that a recorded launch follows
    // later scenes and cameras.  Both are inlined: decided per sample, the
    // branch cost what it saved; the clamped march as an out-of-line call made
    // the 72-register instances spill around it (uneven batch 10.8 ms, against
    // 9.7 ms this way and 9.6 ms without a clamped form).
    const bool inner = Loads::kInner && b.f.inner && v.inner && scene_inner(b.f);
#pragma unroll 1
    for (int sub = 0; sub < (CW / 8) * (CH / 4); ++sub) {
      const int x = x0 + (sub % (CW / 8)) * 8 + tile_x(lane);
      const int y = y0 + (sub / (CW / 8)) * 4 + tile_y(lane);
      if (x < v.width && y < v.height) {
        if (inner)
          n += render_pixel<Loads::kInner, Loads, 1, kOne>(b.f, v, tf_s, x, y, fb, (size_t)x + (size_t)v.width * y,
                                                           loads);
        else
          n += render_pixel<false, Loads, 1, kOne>(b.f, v, tf_s, x, y, fb, (size_t)x + (size_t)v.width * y, loads);
      }
    }
  }
  loads.finish();
  count_samples(b.f.counter, n);
}

// ---- Rank-split render of one view -------------------------------------
// A work item is one 8x4-pixel chunk for one virtual rank, so the bricks along
// a pixel's ray are marched by different warps at the same time.  The ranks
// of a pixel never interact before the composite (each has its own
// accumulator and early termination, like the reference's one process per
// rank), so this is render_pixel's arithmetic in another schedule.
//
// split_mask_kernel marks, per chunk slot, the ranks whose screen rectangle
// covers the chunk (bit k = k-th rank in visibility order); no pixel ray of
// an unmarked rank can enter its bricks, so its image is the output stage of
// an empty march.  The scan kernels and split_emit_kernel list the work items
// in position order (the cost order when s.chunk_order is set, else the
// centre-out ring): one per marked rank, or one compositing-only
// item for a chunk no rank covers.  render_split_kernel marches each item's rank into its
// image plane; the warp that completes a chunk's last marked rank (a ticket
// per chunk, taken after a fence) blends the chunk front to back, evaluating
// the unmarked ranks' images in place, and resets the ticket for the next
// launch.  No warp waits on another.

// Chunk of work position p: the p-th of the cost order when there is one,
// else ring slot p (false off the chunk grid).
__device__ __forceinline__ bool split_chunk(const SplitArgs& s, int p, int cxn, int cyn, int& cx, int& cy) {
  if (s.chunk_order) {
    const int id = __ldg(s.chunk_order + p);
    cx = id % cxn;
    cy = id / cxn;
    return true;
  }
  return ring_chunk(p, cxn, cyn, cx, cy);
}

__device__ __forceinline__ bool rect_covers(const int* __restrict__ q, int cx, int cy) {
  return cx >= __ldg(q) && cy >= __ldg(q + 1) && cx <= __ldg(q + 2) && cy <= __ldg(q + 3);
}

// Per slot: the mask of covering ranks and the number of items it lists
// (one per covering rank, one for a covered-by-none chunk, 0 off the grid).
__global__ void split_mask_kernel(SplitArgs s) {
  const DevView& v = s.f.views[s.view];
  const int W = v.width, H = v.height, R = v.n_ranks;
  const int* __restrict__ order = s.f.sched + v.sched;
  const int* __restrict__ rects = s.f.sched + v.rects;
  const int cxn = (W + 7) / 8, cyn = (H + 3) / 4;
  for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < s.n_slots; slot += gridDim.x * blockDim.x) {
    int cx, cy;
    unsigned long long m = 0ull;
    uint32_t items = 0;
    if (split_chunk(s, slot, cxn, cyn, cx, cy)) {
      for (int k = 0; k < R; ++k)
        if (rect_covers(rects + 4 * __ldg(order + k), cx, cy)) m |= 1ull << k;
      items = m ? (uint32_t)__popcll(m) : 1u;
    }
    s.masks[slot] = m;
    s.offsets[slot] = items;
  }
}

// Exclusive scan of the per-slot item counts in place, and the item total,
// in two levels: per-block sums of kScanTile slots, a one-CTA scan of the
// block sums, then each block scans its tile and adds its base.
constexpr int kScanBlock = 256, kScanPer = 4, kScanTile = kScanBlock * kScanPer;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sum, uint32_t& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = lane < nw ? warp_sum[lane] : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += o;
    }
    if (lane < nw) warp_sum[lane] = w;
  }
  __syncthreads();
  total = warp_sum[nw - 1];
  return incl - v + (wid > 0 ? warp_sum[wid - 1] : 0u);
}

__global__ void __launch_bounds__(kScanBlock) split_block_sums_kernel(SplitArgs s, uint32_t* sums) {
  __shared__ uint32_t warp_sum[kScanBlock / 32];
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanPer;
  uint32_t v = 0;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i)
    if (base + i < s.n_slots) v += s.offsets[base + i];
  uint32_t total;
  block_exclusive_scan(v, warp_sum, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One CTA: exclusive scan of the block sums (contiguous ranges per thread).
__global__ void __launch_bounds__(1024) split_sums_scan_kernel(SplitArgs s, uint32_t* sums, int n) {
  __shared__ uint32_t warp_sum[1024 / 32];
  const int per = (n + 1023) / 1024;
  const int lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
  uint32_t v = 0;
  for (int i = lo; i < hi; ++i) v += sums[i];
  uint32_t total;
  uint32_t at = block_exclusive_scan(v, warp_sum, total);
  for (int i = lo; i < hi; ++i) {
    const uint32_t c = sums[i];
    sums[i] = at;
    at += c;
  }
  if (threadIdx.x == 0) *s.n_items = total;
}

__global__ void __launch_bounds__(kScanBlock) split_tile_scan_kernel(SplitArgs s, const uint32_t* sums) {
  __shared__ uint32_t warp_sum[kScanBlock / 32];
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanPer;
  uint32_t c[kScanPer], v = 0;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    c[i] = base + i < s.n_slots ? s.offsets[base + i] : 0u;
    v += c[i];
  }
  uint32_t total;
  uint32_t at = block_exclusive_scan(v, warp_sum, total) + sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kScanPer; ++i)
    if (base + i < s.n_slots) {
      s.offsets[base + i] = at;
      at += c[i];
    }
}

// Writes each slot's items at its offset: slot << 7 | rank position, or the
// compositing-only item of a chunk no rank covers.
__global__ void split_emit_kernel(SplitArgs s) {
  const DevView& v = s.f.views[s.view];
  const int cxn = (v.width + 7) / 8, cyn = (v.height + 3) / 4;
  for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < s.n_slots; slot += gridDim.x * blockDim.x) {
    int cx, cy;
    if (!split_chunk(s, slot, cxn, cyn, cx, cy)) continue;
    uint32_t at = s.offsets[slot];
    unsigned long long m = s.masks[slot];
    const uint32_t base = (uint32_t)slot << 7;
    if (!m) {
      s.items[at] = base | kSplitBackground;
      continue;
    }
    while (m) {
      const int k = __ffsll((long long)m) - 1;
      m &= m - 1ull;
      s.items[at++] = base | (uint32_t)k;
    }
  }
}

template <int MINB>
__global__ void __launch_bounds__(kRenderThreads, MINB) render_split_kernel(SplitArgs s) {
  extern __shared__ float4 tf_s[];
  load_tf(tf_s, s.f.tf, s.f.n_tf);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int W = s.f.views[s.view].width, H = s.f.views[s.view].height, R = s.f.views[s.view].n_ranks;
  const size_t npx = (size_t)W * H;
  const int* __restrict__ order = s.f.sched + s.f.views[s.view].sched;
  const int* __restrict__ rstart = order + R;
  const int* __restrict__ rbricks = rstart + R + 1;
  const int cxn = (W + 7) / 8, cyn = (H + 3) / 4;
  const uint32_t n_items = *s.n_items;
  float4* __restrict__ planes = s.f.rank_images;
  const bool inner = s.f.inner && s.f.views[s.view].inner && scene_inner(s.f);
  uint32_t n = 0;
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(s.work_counter, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= n_items) break;
    const uint32_t code = __ldg(s.items + item);
    const int slot = (int)(code >> 7), k = (int)(code & 127u);
    int cx, cy;
    split_chunk(s, slot, cxn, cyn, cx, cy);
    const int x = cx * 8 + tile_x(lane), y = cy * 4 + tile_y(lane);
    const bool valid = x < W && y < H;
    const int pixel = x + W * y;
    const unsigned long long mask = __ldg(s.masks + slot);
    if (k != kSplitBackground) {
      if (valid) {
        const DevView v = s.f.views[s.view];
        const int r = __ldg(order + k);
        float z = 1.0f;
        uint32_t ns = 0;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        DirectLoads direct;
        const bool in_island = pixel_in_island(s.f, W, x, y);
        if (plain_output_stage(s.f)) {
          // the output stage is the identity: only the plane store is left,
          // so nothing else it needs stays live across the march
          if (in_island && inner)
            acc = march_rank<true>(s.f, v, tf_s, generate_ray(v, x, y), rbricks, __ldg(rstart + r), __ldg(rstart + r + 1),
                                   pixel, z, ns, direct);
          else if (in_island)
            acc = march_rank<false>(s.f, v, tf_s, generate_ray(v, x, y), rbricks, __ldg(rstart + r), __ldg(rstart + r + 1),
                             pixel, z, ns, direct);
          planes[(size_t)r * npx + pixel] = acc;
        } else {
          if (in_island)
            acc = march_rank<false>(s.f, v, tf_s, generate_ray(v, x, y), rbricks, __ldg(rstart + r), __ldg(rstart + r + 1),
                             pixel, z, ns, direct);
          rank_output(s.f, W, H, r, x, y, pixel, npx, acc, ns, z, planes, nullptr);
        }
        n += ns;
      }
      __threadfence();
      __syncwarp();
      unsigned ticket = 0;
      if (lane == 0) ticket = atomicAdd(s.chunk_done + slot, 1u);
      ticket = __shfl_sync(0xffffffffu, ticket, 0);
      if (ticket != (unsigned)(__popcll(mask) - 1)) continue;
      __threadfence();
    }
    if (valid) {
      OverBlend blend;
      for (int kk = 0; kk < R; ++kk) {
        const int r = __ldg(order + kk);
        const float4 img = (mask >> kk) & 1ull
                               ? __ldcg(planes + (size_t)r * npx + pixel)
                               : rank_output(s.f, W, H, r, x, y, pixel, npx, make_float4(0.f, 0.f, 0.f, 0.f), 0u,
                                             1.0f, nullptr, nullptr);
        blend.add(s.f.composite_mode, img);
      }
      s.f.fb[pixel] = blend.pack(s.f.composite_mode);
    }
    if (lane == 0 && k != kSplitBackground) s.chunk_done[slot] = 0u;
  }
  count_samples(s.f.counter, n);
}

// The order of a composite: from device memory, or from the launch parameters.
struct MemoryOrder {
  const int* r;
  __device__ __forceinline__ int operator[](int k) const { return __ldg(r + k); }
};
struct ParamOrder {
  uint16_t r[kParamRanks];
  __device__ __forceinline__ int operator[](int k) const { return r[k]; }
};

// Ordered "over" of per-rank float images (IceT BLEND with ORDERED_COMPOSITE,
// waikikiRenderer.cpp:910-917,1042-1079), front to back.
template <class Order>
__global__ void composite_f32_kernel(const float4* __restrict__ imgs, const __grid_constant__ Order order, int n_ranks,
                                     int npx, int mode, uint32_t* __restrict__ fb) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npx; p += gridDim.x * blockDim.x) {
    OverBlend blend;
#pragma unroll 4
    for (int k = 0; k < n_ranks; ++k) blend.add(mode, __ldg(imgs + (size_t)order[k] * npx + p));
    fb[p] = blend.pack(mode);
  }
}

// 8-bit ordered over of external RGBA8 rank images.
template <class Order>
__global__ void composite_u8_kernel(const uint32_t* __restrict__ imgs, const __grid_constant__ Order order,
                                    int n_ranks, int npx, uint32_t* __restrict__ fb) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npx; p += gridDim.x * blockDim.x) {
    uint32_t c8[4] = {0u, 0u, 0u, 0u};
#pragma unroll 4
    for (int k = 0; k < n_ranks; ++k) {
      const uint32_t q = __ldg(imgs + (size_t)order[k] * npx + p);
      const uint32_t f = 255u - c8[3];
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) c8[ch] = min(255u, c8[ch] + (((q >> (8 * ch)) & 255u) * f + 127u) / 255u);
    }
    fb[p] = c8[0] | (c8[1] << 8) | (c8[2] << 16) | (c8[3] << 24);
  }
}

// Fills a brick's padded array: element (x,y,z) holds V(x,y,z), V(x,y,z+1),
// V(x,y+1,z), V(x,y+1,z+1) with every index clamped to the brick (the apron and
// the quads' far rows and slices repeat edge values); flags non-finite voxels
// and values too large for InnerCoords or a tame scene (in page-locked host memory); and takes each macrocell's value range:
// a sample whose value-tap cell is c (c = clamp(floor(u), 0, n-1)) reads voxels
// c and c+1 (clamped), so macrocell m covers voxels [m*kMacro, m*kMacro +
// kMacro] per axis.  A CTA takes kMacro rows of kMacro slices, each thread one
// column: it loads the (kMacro + 1)^2 voxels of the column once, coalesced
// along x, and has both the quads of its rows and the column's minimum and
// maximum in registers; the columns meet in shared memory.
constexpr int kFillThreads = 128, kFillColumns = kFillThreads - kMacro;
__global__ void __launch_bounds__(kFillThreads) fill_brick_kernel(const float* __restrict__ src, int nx, int ny,
                                                                  int nz, float4* __restrict__ dst, int px, int sz,
                                                                  int blocks_y, float2* __restrict__ ranges,
                                                                  int* flags) {
  constexpr int N = kMacro + 1;
  __shared__ float lo_s[kFillThreads], hi_s[kFillThreads];
  const int my = (int)(blockIdx.x % (unsigned)blocks_y) - 1, mz = (int)(blockIdx.x / (unsigned)blocks_y) - 1;
  const int y0 = my * kMacro, z0 = mz * kMacro;
  const int mnx = (nx + kMacro - 1) >> kMacroShift, mny = (ny + kMacro - 1) >> kMacroShift;
  const bool in_cells = my >= 0 && my < mny && mz >= 0 && mz * kMacro < nz;
  const int t = (int)threadIdx.x;
  bool bad = false, wide = false, huge = false;
  for (int x0 = -kMacro; x0 < px - kApron; x0 += kFillColumns) {
    const int x = x0 + t, xc = min(max(x, 0), nx - 1);
    float v[N][N];  // [z][y]
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int j = 0; j < N; ++j)
        v[k][j] = __ldg(src + ((size_t)min(max(z0 + k, 0), nz - 1) * ny + min(max(y0 + j, 0), ny - 1)) * nx + xc);
    float lo = v[0][0], hi = lo;
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int j = 0; j < N; ++j) {
        lo = fminf(lo, v[k][j]);
        hi = fmaxf(hi, v[k][j]);
        bad |= !isfinite(v[k][j]);
      }
    wide |= hi > kInnerValue || lo < -kInnerValue;
    huge |= hi > kTame || lo < -kTame;
    if (t < kFillColumns && x >= -kApron && x < px - kApron) {
#pragma unroll
      for (int k = 0; k < kMacro; ++k)
#pragma unroll
        for (int j = 0; j < kMacro; ++j) {
          const int y = y0 + j + kApron, z = z0 + k + kApron;
          if (y >= 0 && y < ny + 2 * kApron && z >= 0 && z < nz + 2 * kApron)
            dst[(size_t)z * sz + (size_t)y * px + (x + kApron)] =
                make_float4(v[k][j], v[k + 1][j], v[k][j + 1], v[k + 1][j + 1]);
        }
    }
    if (in_cells) {
      __syncthreads();  // the previous chunk's readers
      lo_s[t] = lo;
      hi_s[t] = hi;
      __syncthreads();
      const int mx = (x0 >> kMacroShift) + t;
      if (t < kFillColumns / kMacro && mx >= 0 && mx < mnx) {
        lo = lo_s[t * kMacro];
        hi = hi_s[t * kMacro];
#pragma unroll
        for (int i = 1; i < N; ++i) {
          lo = fminf(lo, lo_s[t * kMacro + i]);
          hi = fmaxf(hi, hi_s[t * kMacro + i]);
        }
        ranges[((size_t)mz * mny + my) * mnx + mx] = make_float2(lo, hi);
      }
    }
  }
  // One thread per CTA brings what it found to the host's word, and only bits that
  // are not there yet: a volume of scanner units is wide throughout (256^3: 162 us
  // with an atomic of every thread over the host link, 87 this way, 83 for values
  // in range).
  const int found = (bad ? kVoxelNonfinite : 0) | (wide ? kVoxelWide : 0) | (huge ? kVoxelHuge : 0);
  if (__syncthreads_or(found)) {
    __shared__ int found_s[kFillThreads / 32];
    const int of_warp = (int)__reduce_or_sync(0xffffffffu, (unsigned)found);
    if ((t & 31) == 0) found_s[t >> 5] = of_warp;
    __syncthreads();
    if (t == 0) {
      int all = 0;
      for (int w = 0; w < kFillThreads / 32; ++w) all |= found_s[w];
      if (all & ~*static_cast<volatile int*>(flags)) atomicOr_system(flags, all);
    }
  }
}

// Macrocell codes.  A macrocell is empty when every transfer-function entry
// its lookups can touch has alpha 0: indices floor(v*n - 1/2) and +1 for v in
// [lo, hi], with one index of margin on each side for rounding of the
// interpolated value.  The reach is found along x first (here, from the kinds of
// the neighbours as bits), then over y, then over z (reach.h).  A table change
// waits for all three passes.  The 17.6 million cells of 1024^3 in 64 bricks take
// 80 + 63 + 61 us (512^3: 14 + 11 + 11): the first waits for its ranges, 141 MB,
// four loads in flight per thread; the others are bound by instructions, some 50
// per cell.  With a loop over each cell's neighbours in every pass and a grid for
// the largest brick of each, 152 + 170 + 170 (23 + 24 + 24).
constexpr int kCodeThreads = 256, kKindLoads = 4, kKindCells = kKindLoads * kCodeThreads - 2 * (kMaxReach - 1);
__global__ void __launch_bounds__(kCodeThreads) macrocell_kinds_kernel(const DevBrick* __restrict__ bricks,
                                                                       const uint8_t* cells,
                                                                       const float2* __restrict__ ranges,
                                                                       const int* __restrict__ prefix, int n,
                                                                       uint8_t* __restrict__ out) {
  constexpr int W = kMaxReach - 1;
  __shared__ uint32_t full_bits[kKindLoads * kCodeThreads / 32 + 1];
  const DevBrick& b = bricks[blockIdx.y];
  const size_t first = (size_t)(b.cells - cells);
  const int mnx = (b.n[0] + kMacro - 1) >> kMacroShift;
  const int count = mnx * ((b.n[1] + kMacro - 1) >> kMacroShift) * ((b.n[2] + kMacro - 1) >> kMacroShift);
  const float nf = (float)n;
  const int t = (int)threadIdx.x;
  if (t == 0) full_bits[kKindLoads * kCodeThreads / 32] = 0u;
  // kKindCells cells per CTA and trip, and W more on either side
  for (int i0 = blockIdx.x * kKindCells; i0 < count; i0 += gridDim.x * kKindCells) {
    float2 r[kKindLoads];
    bool full[kKindLoads];
#pragma unroll
    for (int q = 0; q < kKindLoads; ++q) {
      const int i = i0 - W + q * kCodeThreads + t;
      r[q] = i >= 0 && i < count ? __ldcs(ranges + first + i) : make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int q = 0; q < kKindLoads; ++q) {
      const float xl = fminf(fmaxf(r[q].x * nf - 0.5f, -8.0f), nf + 8.0f);
      const float xh = fminf(fmaxf(r[q].y * nf - 0.5f, -8.0f), nf + 8.0f);
      const int lo = max((int)floorf(xl) - 1, 0);
      const int hi = min((int)floorf(xh) + 2, n - 1);
      full[q] = lo <= hi && __ldg(prefix + hi + 1) != __ldg(prefix + lo);
    }
    __syncthreads();  // the previous cells' readers
#pragma unroll
    for (int q = 0; q < kKindLoads; ++q) {
      const uint32_t bits = __ballot_sync(0xffffffffu, full[q]);
      if ((t & 31) == 0) full_bits[(q * kCodeThreads + t) >> 5] = bits;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kKindLoads; ++q) {
      const int at = q * kCodeThreads + t - W, i = i0 + at;
      if (at >= 0 && at < kKindCells && i < count) {
        const uint32_t window = __funnelshift_r(full_bits[at >> 5], full_bits[(at >> 5) + 1], at & 31);
        out[first + i] = (uint8_t)((full[q] ? kCellFull : 0) | row_reach(window, i % mnx, mnx));
      }
    }
  }
}

// The pass along y (AXIS 1) or z: a thread takes kReachCells cells in a row along
// the axis, whose neighbours' codes it loads once, coalesced along x.
constexpr int kReachCells = 8;
template <int AXIS>
__global__ void __launch_bounds__(kCodeThreads) macrocell_reach_kernel(const DevBrick* __restrict__ bricks,
                                                                       const uint8_t* cells,
                                                                       const uint8_t* __restrict__ in,
                                                                       uint8_t* __restrict__ out) {
  constexpr int W = kMaxReach - 1, N = kReachCells + 2 * W;
  const DevBrick& b = bricks[blockIdx.y];
  const size_t first = (size_t)(b.cells - cells);
  const int mnx = (b.n[0] + kMacro - 1) >> kMacroShift, mny = (b.n[1] + kMacro - 1) >> kMacroShift,
            mnz = (b.n[2] + kMacro - 1) >> kMacroShift;
  const int len = AXIS == 1 ? mny : mnz, stride = AXIS == 1 ? mnx : mnx * mny;
  const int runs = (len + kReachCells - 1) / kReachCells;
  const int items = mnx * runs * (AXIS == 1 ? mnz : mny);
  for (int i = blockIdx.x * kCodeThreads + threadIdx.x; i < items; i += gridDim.x * kCodeThreads) {
    const int x = i % mnx, rest = i / mnx;
    const int p0 = kReachCells * (AXIS == 1 ? rest % runs : rest / mny);
    const size_t row = first + x + (AXIS == 1 ? (rest / runs) * mnx * mny : (rest % mny) * mnx);
    const int8_t* at = reinterpret_cast<const int8_t*>(in) + row;
    int s[N];
#pragma unroll
    for (int k = 0; k < N; ++k) s[k] = __ldg(at + min(max(p0 + k - W, 0), len - 1) * stride);
#pragma unroll
    for (int k = 0; k < kReachCells; ++k)
      if (p0 + k < len) out[row + (p0 + k) * stride] = (uint8_t)axis_code(s + W + k);
  }
}

static size_t tf_smem(int n_tf) { return (size_t)(n_tf + 4) * sizeof(float4); }
static size_t render_smem(int n_tf, int stage) {
  return tf_smem(n_tf) + (stage == ALOHA_STAGING_NEXT_SAMPLE ? kStageBytes : 0);
}

cudaError_t launch_macrocell_codes(const DevBrick* bricks, int n_bricks, int most_cells, size_t all_cells, const float2* ranges,
                                   const int* prefix, int n_tf, uint8_t* cells, uint8_t* tmp, cudaStream_t s) {
  for (int b0 = 0; b0 < n_bricks; b0 += 65535) {  // a grid's y extent
    // the largest brick's share of the CTAs that fill the GPU, and no more than it
    // has work for: CTAs that find none cost as much as the passes do
    const int share = (int)((152ll * 8 * most_cells + (long long)all_cells - 1) / (long long)all_cells);
    auto grid = [&](int per_cta) {
      return dim3(min((most_cells + per_cta - 1) / per_cta, share), min(n_bricks - b0, 65535));
    };
    macrocell_kinds_kernel<<<grid(kKindCells), kCodeThreads, 0, s>>>(bricks + b0, cells, ranges, prefix, n_tf, cells);
    const dim3 runs = grid(kCodeThreads * kReachCells);
    macrocell_reach_kernel<1><<<runs, kCodeThreads, 0, s>>>(bricks + b0, cells, cells, tmp);
    macrocell_reach_kernel<2><<<runs, kCodeThreads, 0, s>>>(bricks + b0, cells, tmp, cells);
  }
  return cudaGetLastError();
}

namespace {

// The kernel instance for a chunk shape, launch mode and staging, or null.
using RenderKernel = void (*)(BatchArgs);
template <int MINB, int STAGE>
RenderKernel render_kernel_for(int chunk_w, int chunk_h) {
  if (chunk_w == 8 && chunk_h == 4) return render_warps_kernel<8, 4, MINB, STAGE>;
  if (chunk_w == 8 && chunk_h == 8) return render_warps_kernel<8, 8, MINB, STAGE>;
  if (chunk_w == 16 && chunk_h == 8) return render_warps_kernel<16, 8, MINB, STAGE>;
  if (chunk_w == 32 && chunk_h == 4) return render_warps_kernel<32, 4, MINB, STAGE>;
  return nullptr;
}

RenderKernel render_kernel(int chunk_w, int chunk_h, bool batch, int stage, bool lane_groups, bool few, bool ring_pairs) {
  if (lane_groups)
    return (!batch && stage == ALOHA_STAGING_NONE && chunk_w == 8 && chunk_h == 4)
               ? render_warps_kernel<8, 4, kSingleRenderBlocks, 0, kLaneGroup>
               : nullptr;
  if (stage == ALOHA_STAGING_NEXT_SAMPLE)
    return batch ? render_kernel_for<kBatchRenderBlocks, 1>(chunk_w, chunk_h)
                 : render_kernel_for<kSingleRenderBlocks, 1>(chunk_w, chunk_h);
  if (stage == kStageUnroll2) return batch ? render_kernel_for<kBatchRenderBlocks, kStageUnroll2>(chunk_w, chunk_h)
                                           : nullptr;
  if (stage != ALOHA_STAGING_NONE) return nullptr;
  if (few && !batch && chunk_w == 8 && chunk_h == 4)
    return ring_pairs ? render_warps_kernel<8, 4, kFewChunkRenderBlocks, 0, kRingPairs>
                      : render_warps_kernel<8, 4, kFewChunkRenderBlocks, 0, 2>;
  return batch ? render_kernel_for<kBatchRenderBlocks, 0>(chunk_w, chunk_h)
               : render_kernel_for<kSingleRenderBlocks, 0>(chunk_w, chunk_h);
}

}  // namespace

cudaError_t launch_render_warps(const BatchArgs& b, int chunk_w, int chunk_h, int grid, bool batch, cudaStream_t s,
                                int stage, bool lane_groups, bool few, bool beside) {
  if (lane_groups && (!b.chunk_order || b.f.rank_images || b.f.rank_depth || b.f.accum)) return cudaErrorInvalidValue;
  const RenderKernel k = render_kernel(chunk_w, chunk_h, batch, stage, lane_groups, few, few && b.ring_pairs);
  if (!k) return cudaErrorInvalidValue;
  return launch_beside(k, grid, kRenderThreads, render_smem(b.f.n_tf, stage), s, beside, b);
}

int render_blocks_per_sm(int chunk_w, int chunk_h, int n_tf, bool batch, int stage, bool lane_groups, bool few) {
  const RenderKernel k = render_kernel(chunk_w, chunk_h, batch, stage, lane_groups, few, false);
  int n = 0;
  if (!k || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kRenderThreads, render_smem(n_tf, stage)) !=
                cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// Many ranks make short (chunk, rank) items, so the launch is throughput-bound
// and runs best with more resident warps (64 ranks of 1024^3 at 2048^2:
// 5.58 ms at 5 CTAs/SM, 5.26 ms at 7); with few ranks the longest items
// bound the frame and 5 CTAs/SM is best (8 ranks: 0.89 vs 0.96 ms).
using SplitKernel = void (*)(SplitArgs);
static SplitKernel split_kernel(bool many_ranks) {
  return many_ranks ? render_split_kernel<kManyRankSplitBlocks> : render_split_kernel<kSingleRenderBlocks>;
}

cudaError_t launch_render_split(const SplitArgs& a, int grid, bool many_ranks, cudaStream_t s) {
  int mg = (a.n_slots + 255) / 256;
  mg = mg < 1 ? 1 : (mg > 152 * 8 ? 152 * 8 : mg);
  split_mask_kernel<<<mg, 256, 0, s>>>(a);
  const int tiles = (a.n_slots + kScanTile - 1) / kScanTile;
  split_block_sums_kernel<<<tiles, kScanBlock, 0, s>>>(a, a.block_sums);
  split_sums_scan_kernel<<<1, 1024, 0, s>>>(a, a.block_sums, tiles);
  split_tile_scan_kernel<<<tiles, kScanBlock, 0, s>>>(a, a.block_sums);
  split_emit_kernel<<<mg, 256, 0, s>>>(a);
  cudaError_t e = cudaMemsetAsync(a.work_counter, 0, sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  split_kernel(many_ranks)<<<grid, kRenderThreads, tf_smem(a.f.n_tf), s>>>(a);
  return cudaGetLastError();
}

int render_split_blocks_per_sm(int n_tf, bool many_ranks) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, split_kernel(many_ranks), kRenderThreads, tf_smem(n_tf)) !=
      cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

static int composite_grid(int npx) {
  int g = (npx + 255) / 256;
  return g < 1 ? 1 : (g > 152 * 16 ? 152 * 16 : g);
}

static bool param_order(const int* host_order, int n_ranks, ParamOrder& o) {
  if (!host_order || n_ranks > kParamRanks) return false;
  for (int k = 0; k < n_ranks; ++k) o.r[k] = (uint16_t)host_order[k];
  return true;
}

cudaError_t launch_composite_f32(const float4* imgs, const int* order, const int* host_order, int n_ranks, int npx,
                                 int mode, uint32_t* fb, cudaStream_t s) {
  ParamOrder o;
  if (order)
    composite_f32_kernel<<<composite_grid(npx), 256, 0, s>>>(imgs, MemoryOrder{order}, n_ranks, npx, mode, fb);
  else if (param_order(host_order, n_ranks, o))
    composite_f32_kernel<<<composite_grid(npx), 256, 0, s>>>(imgs, o, n_ranks, npx, mode, fb);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_composite_u8(const uint32_t* imgs, const int* order, const int* host_order, int n_ranks, int npx,
                                uint32_t* fb, cudaStream_t s) {
  ParamOrder o;
  if (order)
    composite_u8_kernel<<<composite_grid(npx), 256, 0, s>>>(imgs, MemoryOrder{order}, n_ranks, npx, fb);
  else if (param_order(host_order, n_ranks, o))
    composite_u8_kernel<<<composite_grid(npx), 256, 0, s>>>(imgs, o, n_ranks, npx, fb);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_fill_brick(const DevBrick& b, const float* src, float4* dst, float2* ranges, int* flags,
                              cudaStream_t s) {
  // blocks of kMacro rows and slices from -kMacro to the last apron row
  const int blocks_y = (b.n[1] + kApron - 1) / kMacro + 2, blocks_z = (b.n[2] + kApron - 1) / kMacro + 2;
  fill_brick_kernel<<<blocks_y * blocks_z, kFillThreads, 0, s>>>(src, b.n[0], b.n[1], b.n[2], dst, b.sy, b.sz, blocks_y,
                                                               ranges, flags);
  return cudaGetLastError();
}

}  // namespace aloha
