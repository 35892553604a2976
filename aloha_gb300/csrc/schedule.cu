// schedule.cu -- cost-ordered chunks for single-view renders (both work
// divisions) and the differentiable forward.
//
// A frame ends with its slowest chunk (an 8x4 tile whose rays march far
// through translucent space), so the order in which warps take chunks sets
// the length of its tail: started last, a long chunk runs on an almost idle
// GPU.  Longest-first ordering needs the cost before the frame.  A coarse
// probe gives a good enough estimate: four rays of the chunk (a 2x2 sample),
// each through the bricks of every rank whose screen rectangle covers it,
// counting strides of 16 samples in non-empty macrocells (no voxel loads, no
// early termination); the chunk's cost is the largest of the four, as a warp
// runs as long as its longest ray.  The chunks are then sorted stably by cost
// class (a quarter octave each), most expensive first; ring order within a
// class keeps neighbouring chunks together.  The order only changes when a
// pixel is rendered, never how, so frames are bit-identical to ring order.
//
// Kernels: probe (4 threads per ring slot; each CTA also adds its class
// counts into its sort block's histogram column), and a stable scatter, which
// scans the histogram table (class-major) itself or, for large frames, finds it
// scanned by a one-CTA kernel, and zeroes it.
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"
#include "march.cuh"

namespace aloha {

namespace {

constexpr uint8_t kNoChunk = 0xff;
constexpr float kProbeStride = 16.0f;  // samples per probe step
constexpr int kProbeMaxSteps = 8192;   // per brick (the probe only estimates)
constexpr int kSortThreads = 1024;     // slots per sort block (histogram column, scatter CTA)
constexpr int kProbeThreads = 256;     // 4 per slot: 64 slots per probe CTA
constexpr int kScanThreads = 1024;

// Non-empty probe steps of one ray through every rank's bricks.  Bound by the
// chain of dependent table reads of the longest ray, so it reads one code per
// box of equal cells, not one per stride; with the launches beside each other
// (launch_chunk_order) a 701x395 frame of 181x113x237 voxels at 2 spp and dt 0.3
// took 383 -> 353 us, 512^3 at 1024^2 688 -> 679.
__device__ uint32_t probe_ray(const ChunkOrderArgs& a, const DevView& v, const int* __restrict__ order,
                              const int* __restrict__ rstart, const int* __restrict__ rbricks, int x, int y) {
  const Ray ray = generate_ray(v, x, y);
  const float stride = kProbeStride * a.f.dt;
  const float idx = __fdividef(1.0f, ray.d[0]), idy = __fdividef(1.0f, ray.d[1]), idz = __fdividef(1.0f, ray.d[2]);
  // ranks whose screen rectangle (in 8x4 chunks) misses the pixel cannot be hit
  const int* __restrict__ rects = a.f.sched + v.rects;
  const int qx = x >> 3, qy = y >> 2;
  uint32_t c = 0;
  for (int k = 0; k < v.n_ranks; ++k) {
    const int r = __ldg(order + k);
    const int* q = rects + 4 * r;
    if (qx < __ldg(q) || qy < __ldg(q + 1) || qx > __ldg(q + 2) || qy > __ldg(q + 3)) continue;
    float tmin = 0.0f;
    for (int j = __ldg(rstart + r); j < __ldg(rstart + r + 1); ++j) {
      const DevBrick b = a.f.bricks[__ldg(rbricks + j)];
      float t0, t1;
      if (!slab(ray, b.space_lo, b.space_hi, tmin, 1e10f, t0, t1)) continue;
      tmin = t1 + 1e-20f;
      const float span = (t1 - t0) / stride;
      const int steps = span < (float)kProbeMaxSteps ? (int)span + 1 : kProbeMaxSteps;
      const int mnx = (b.n[0] + kMacro - 1) >> kMacroShift, mny = (b.n[1] + kMacro - 1) >> kMacroShift;
      const float offx = ray.o[0] - b.lo[0], offy = ray.o[1] - b.lo[1], offz = ray.o[2] - b.lo[2];
      const float inv = __fdividef(1.0f, stride);
      // one lookup per box of cells of one kind, not per stride
      for (int i = 0; i < steps;) {
        const float t = fmaf((float)i, stride, t0);
        const Cell cell = cell_at(b.cells, mnx, mny, b.n[0], b.n[1], b.n[2], fmaf(t, ray.d[0], offx),
                                  fmaf(t, ray.d[1], offy), fmaf(t, ray.d[2], offz));
        const float end = cell_exit(cell, ray.d, offx, offy, offz, idx, idy, idz, 0.0f, t1);
        const int k = min(max(__float2int_ru((end - t) * inv), 1), steps - i);
        if (!cell.empty()) c += (uint32_t)k;
        i += k;
      }
    }
  }
  return c;
}

// Cost class: 0 for the most expensive, one class per quarter octave.
__device__ __forceinline__ uint8_t cost_class(uint32_t c) {
  const int q = (int)(4.0f * log2f((float)c + 1.0f));
  return (uint8_t)(kOrderClasses - 1 - min(q, kOrderClasses - 1));
}

// Four threads per ring slot (lanes 4s..4s+3 of a warp): each probes one ray
// of the chunk's 2x2 sample; the slot's class comes from the largest.  A CTA
// covers kProbeThreads / 4 slots and adds its class counts into the histogram
// column of the sort block (kSortThreads slots) it belongs to.
__global__ void probe_chunks_kernel(ChunkOrderArgs a) {
  launch_dependents();
  __shared__ uint32_t h[kOrderClasses];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (a.zero_work) *a.zero_work = 0u;
    if (a.zero_samples) *a.zero_samples = 0ull;
  }
  for (int i = threadIdx.x; i < kOrderClasses; i += kProbeThreads) h[i] = 0;
  __syncthreads();
  const DevView& v = a.f.views[a.view];
  const int W = v.width, H = v.height, R = v.n_ranks;
  const int* __restrict__ order = a.f.sched + v.sched;
  const int cxn = (W + a.cw - 1) / a.cw, cyn = (H + a.ch - 1) / a.ch;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = gid >> 2, q = gid & 3;
  uint32_t c = 0;
  bool valid = false;
  int cx = 0, cy = 0;
  if (slot < a.n_slots && ring_chunk(slot, cxn, cyn, cx, cy)) {
    valid = true;
    const int x = min(cx * a.cw + ((q & 1) ? (3 * a.cw) / 4 : a.cw / 4), W - 1);
    const int y = min(cy * a.ch + ((q & 2) ? (3 * a.ch) / 4 : a.ch / 4), H - 1);
    c = probe_ray(a, v, order, order + R, order + 2 * R + 1, x, y);
  }
  c = max(c, __shfl_xor_sync(0xffffffffu, c, 1));
  c = max(c, __shfl_xor_sync(0xffffffffu, c, 2));
  if (q == 0 && slot < a.n_slots) {
    const uint8_t k = valid ? cost_class(c) : kNoChunk;
    a.key[slot] = k;
    a.cid[slot] = cx + cxn * cy;
    if (valid) atomicAdd(&h[k], 1u);
  }
  __syncthreads();
  const int blocks = (a.n_slots + kSortThreads - 1) / kSortThreads;
  const int block = (int)(((long long)blockIdx.x * (kProbeThreads / 4)) / kSortThreads);
  for (int i = threadIdx.x; i < kOrderClasses; i += kProbeThreads)
    if (h[i]) atomicAdd(a.hist + i * blocks + block, h[i]);
}

// Exclusive scan of the histogram table in place (one CTA; each thread scans
// a contiguous range).
__global__ void __launch_bounds__(kScanThreads) class_scan_kernel(ChunkOrderArgs a, int n) {
  if (threadIdx.x == 0) *a.pairs = 0;  // large frames fill the GPU
  __shared__ uint32_t warp_sum[kScanThreads / 32];
  const int per = (n + kScanThreads - 1) / kScanThreads;
  const int lo = min(n, (int)threadIdx.x * per), hi = min(n, lo + per);
  uint32_t count = 0;
  for (int i = lo; i < hi; ++i) count += a.hist[i];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = count;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = warp_sum[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += o;
    }
    warp_sum[lane] = w;
  }
  __syncthreads();
  uint32_t at = incl - count + (wid > 0 ? warp_sum[wid - 1] : 0u);
  for (int i = lo; i < hi; ++i) {
    const uint32_t c = a.hist[i];
    a.hist[i] = at;
    at += c;
  }
}

// How many chunks at the head of the order two lanes per ray render sooner
// than one: all that the probe found samples in, or none.  `waves` is the
// frame's work against what the resident warps do while the costliest chunk
// runs: the fewer, the more warps only wait for that chunk, which two lanes per
// ray shorten, the more so the longer its rays (each lane also repeats a ray's
// set-up).  One / two lanes, us, over (waves, strides of the costliest chunk):
//   wins:   (.23, 18) 148 / 115   (.34, 37) 352 / 298   (.36, 53) 579 / 371
//           (.38, 26) 199 / 157   (.43, 15) 111 / 99    (.45, 31) 239 / 209   (.50, 53) 561 / 394
//   losses: (.47, 7) 224 / 252    (.49, 18) 261 / 287   (.51, 7) 68 / 74      (.74, 31) 249 / 254
// The line below runs between these eleven, narrowly: it leaves (.43, 15) .004 and
// (.49, 18) .013, where either way costs some 10 %, and a frame near it changes whole.
// One warp: classes 2 lane and 2 lane + 1 hold t0 and t1 chunks.
__device__ __forceinline__ void pair_rule(const ChunkOrderArgs& a, int lane, uint32_t t0, uint32_t t1) {
  const float c0 = exp2f(0.25f * (float)(kOrderClasses - 1 - 2 * lane)) - 1.0f;
  const float c1 = exp2f(0.25f * (float)(kOrderClasses - 2 - 2 * lane)) - 1.0f;
  float sum = fmaf((float)t0, c0, (float)t1 * c1), most = t0 ? c0 : (t1 ? c1 : 0.f);
  int active = (int)t0 + (lane == 31 ? 0 : (int)t1);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, d);
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
    active += __shfl_xor_sync(0xffffffffu, active, d);
  }
  const float waves = 0.22f + most * (1.0f / 70.0f);
  if (lane == 0) *a.pairs = sum < waves * most * (float)a.warps ? active : 0;
}

// Stable scatter: a slot's position is its class's base for this CTA plus the
// slots of the same class before it in the CTA (earlier warps, then earlier
// lanes of its warp).  SCAN: the CTA finds its classes' bases itself, from the
// counts of all sort blocks, and the last CTA to have read them zeroes the
// table for the next launch; else the table holds the bases (class_scan_kernel)
// and each CTA zeroes its own column.
template <bool SCAN>
__global__ void __launch_bounds__(kSortThreads) class_scatter_kernel(ChunkOrderArgs a) {
  constexpr int kWarps = kSortThreads / 32;
  __shared__ uint32_t wc[kWarps][kOrderClasses];
  __shared__ uint32_t class_base[kOrderClasses], class_total[kOrderClasses];
  __shared__ bool last;
  launch_dependents();
  for (int i = threadIdx.x; i < kWarps * kOrderClasses; i += kSortThreads) (&wc[0][0])[i] = 0;
  wait_for_primary();
  const int blocks = (int)gridDim.x;
  if (SCAN) {
    constexpr int kPer = kSortThreads / kOrderClasses;  // threads per class, part of a warp
    const int k = threadIdx.x / kPer, part = threadIdx.x % kPer;
    uint32_t total = 0, before = 0;
    for (int i = part; i < blocks; i += kPer) {
      const uint32_t c = __ldcg(a.hist + k * blocks + i);
      total += c;
      if (i < (int)blockIdx.x) before += c;
    }
#pragma unroll
    for (int d = kPer / 2; d > 0; d >>= 1) {
      total += __shfl_xor_sync(0xffffffffu, total, d);
      before += __shfl_xor_sync(0xffffffffu, before, d);
    }
    if (part == 0) {
      class_total[k] = total;
      class_base[k] = before;
    }
  } else {
    for (int i = threadIdx.x; i < kOrderClasses; i += kSortThreads) class_base[i] = a.hist[i * blocks + blockIdx.x];
  }
  __syncthreads();
  if (SCAN) {
    if (threadIdx.x == 0) last = atomicAdd(a.readers, 1u) == (unsigned)blocks - 1u;
    if (threadIdx.x < 32) {  // exclusive scan of the classes' totals, two per lane
      const int lane = threadIdx.x;
      const uint32_t t0 = class_total[2 * lane], t1 = class_total[2 * lane + 1];
      uint32_t incl = t0 + t1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
      }
      if (blockIdx.x == 0) pair_rule(a, lane, t0, t1);
      class_base[2 * lane] += incl - t0 - t1;
      class_base[2 * lane + 1] += incl - t1;
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int slot = blockIdx.x * kSortThreads + threadIdx.x;
  const uint8_t k = slot < a.n_slots ? a.key[slot] : kNoChunk;
  const unsigned peers = __match_any_sync(0xffffffffu, (unsigned)k);
  const unsigned rank = __popc(peers & ((1u << lane) - 1u));
  if (k != kNoChunk && lane == __ffs(peers) - 1) wc[w][k] = __popc(peers);
  __syncthreads();
  if (k != kNoChunk) {
    uint32_t pos = class_base[k] + rank;
    for (int e = 0; e < w; ++e) pos += wc[e][k];
    if (pos < (uint32_t)a.n_chunks) a.order[pos] = a.cid[slot];
  }
  if (SCAN) {
    if (last) {
      for (int i = threadIdx.x; i < kOrderClasses * blocks; i += kSortThreads) a.hist[i] = 0u;
      if (threadIdx.x == 0) *a.readers = 0u;
    }
  } else {
    // the block's histogram column is consumed: zero it for the next launch
    __syncthreads();
    for (int i = threadIdx.x; i < kOrderClasses; i += kSortThreads) a.hist[i * blocks + blockIdx.x] = 0u;
  }
}

}  // namespace

int chunk_order_blocks(int n_slots) { return (n_slots + kSortThreads - 1) / kSortThreads; }

// The histogram (a.hist, kOrderClasses x chunk_order_blocks(n_slots)) and
// a.readers must be zero when this is called; the scatter leaves them zero
// again.  Up to kScanBlocks sort blocks the scatter scans the table itself: one
// launch less, but every CTA reads the whole table, so the work grows with the
// square of the blocks.  Against the scan kernel, frames of a 64^3 volume:
// 512^2 (17 blocks) 62.2 -> 58.5 us, 2048^2 (258) 467 -> 458, 4096^2 (1027)
// 1777 -> 1760, 5120^2 (1603) 2767 -> 2747, 6144^2 (2308) 3956 -> 3968, 8192^2
// (4101) 6976 -> 7143, 16000^2 (15633) 26510 -> 30400.  The two cross near 2000
// blocks; the line lies below that, where either is within 1 %.  The scatter, and the render
// after it, start beside the kernel before them and wait for it when they need
// its results (programmatic dependent launch).
cudaError_t launch_chunk_order(const ChunkOrderArgs& a, cudaStream_t s) {
  static_assert(kSortThreads % (kProbeThreads / 4) == 0, "probe CTAs must tile sort blocks");
  static_assert(kOrderClasses == 64 && 32 % (kSortThreads / kOrderClasses) == 0, "scan layout");
  constexpr int kScanBlocks = 1100;
  const int probe_grid = (int)(((long long)a.n_slots * 4 + kProbeThreads - 1) / kProbeThreads);
  probe_chunks_kernel<<<probe_grid, kProbeThreads, 0, s>>>(a);
  const int blocks = chunk_order_blocks(a.n_slots);
  cudaError_t e;
  if (blocks <= kScanBlocks) {
    e = launch_beside(class_scatter_kernel<true>, blocks, kSortThreads, 0, s, true, a);
  } else {
    class_scan_kernel<<<1, kScanThreads, 0, s>>>(a, kOrderClasses * blocks);
    e = launch_beside(class_scatter_kernel<false>, blocks, kSortThreads, 0, s, true, a);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {  // counts may stay behind: clear them for the next launch
    cudaMemsetAsync(a.hist, 0, (size_t)kOrderClasses * blocks * sizeof(uint32_t), s);
    cudaMemsetAsync(a.readers, 0, sizeof(uint32_t), s);
  }
  return e;
}

}  // namespace aloha
