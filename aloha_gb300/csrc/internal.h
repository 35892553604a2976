// internal.h -- structures shared by the host side and the kernels.
//
// Times in the comments of these files weigh a choice against its alternatives:
// all of one comment were taken in turn on one machine, with the code around the
// choice as it was then, so later changes moved them together.  What whole calls
// take now, on one GB300 (us): a 64^3 frame of 512^2 73; 181x113x237 in 5 bricks,
// 701x395, 2 spp, dt 0.3, 343; 512^3 in 8 ranks at 1024^2 into page-locked memory
// 645; 1024^3 in 64 ranks at 2048^2 3615; 24 uneven views of 512^3 7282; 8 rank
// images of 256^3 at 800x600 and their composite 264; 16 views of 128^3 at 256^2
// with both gradients 2372; 512^3 at 1024^2 with the transfer function's 5003; 6
// views of 256^3 at 512^2 with the density's 2304; 2 of 512^3 at 1024^2 with both
// 13163.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/aloha.h"
#include "reach.h"

namespace aloha {

// Padded brick storage: every brick is stored with an apron of kApron voxels
// on each side, filled with the clamped edge values (cudaAddressModeClamp of
// waikikiRenderer.cpp:753-755), so the march loop needs no per-tap clamps.
// Each stored element is a zy-quad: the float4 (V(x,y,z), V(x,y,z+1),
// V(x,y+1,z), V(x,y+1,z+1)) (indices clamped), so one 16-byte load fetches a
// voxel's 2x2 (y, z) neighbourhood, its halves are (z, z+1) pairs that packed
// fp32x2 instructions interpolate together, and the stencil's core comes from three
// neighbouring elements of one row (x-quads, V(x..x+3), took the same bytes
// from four rows and hit L1 less often).  Quads cut the loads per sample from
// 20 to 7 at four times the HBM footprint.
constexpr int kApron = 2;
// Pitches of the padded array, in quads.  A warp's 16-byte loads are served a
// quarter warp at a time, and quads of different 128-byte lines collide when
// they lie at the same offset (of eight) in their line.  Neighbouring rays
// read neighbouring voxels, along any axis, so the pitches are chosen for
// steps along y and z to land on other offsets: rows of 2 or 6 (mod 8) quads,
// slices of 4 (mod 8).  With rows of nx + 4 and slices of their product, a
// brick of 128, 256 or 512 voxels had slices of 0 (mod 8), so all rays of a
// pixel row that ran along z collided.  Together with the 2x4 quarter warps
// of tile_x / tile_y: uneven 24-view batch 10.46 -> 10.01 ms, 512^3
// transfer-function step 6.35 -> 6.16 ms, odd volume's frame 681 -> 626 us.
// A brick that fits kMaxBrickQuads without this padding only (1024 x 1440 x
// 1440), and a scene that fits the device's memory without it only, take plain
// pitches: rows of an even number of
// quads, slices of their product.
struct BrickPitch {
  int row;
  long long slice;
  long long quads(int nz) const { return slice * (nz + 2 * kApron); }
};
constexpr long long kMaxBrickQuads = (1ll << 31) - 1;  // element offsets are ints
inline BrickPitch plain_pitch(int nx, int ny) {
  const int row = (nx + 2 * kApron + 1) & ~1;
  return {row, (long long)row * (ny + 2 * kApron)};
}
inline BrickPitch spread_pitch(int nx, int ny) {
  const int px = nx + 2 * kApron, row = px + ((2 - px) & 3);
  const long long slice = (long long)row * (ny + 2 * kApron);
  return {row, slice + ((4 - slice) & 7)};
}
constexpr int kMaxViews = 4096;
constexpr int kMaxTF = 2048;  // (n + 4) float4 entries stay under 48 KB of shared memory

// Empty-space macrocells: kMacro^3 voxels; a sample whose value-tap cell lies
// in an empty macrocell has transfer-function alpha exactly 0.  Each has a
// code byte: its kind (kCellFull: not empty) and the Chebyshev distance, at
// most kMaxReach, to the nearest cell of the other kind in its brick, so that
// the box of cells closer than that is all of one kind: a ray steps over, or
// marches without another lookup, to the box's end.  Small cells leave fewer
// samples to evaluate (of the 512^3 blob field's samples 11.4 % lie outside
// empty cells of 8^3, 10.0 % of 4^3 and 8.4 % have an alpha at all; of a 64^3
// one's 45, 30 and 16 %); the reach makes up for their number.  512^3 frame /
// 24-view batch / 1024^3 frame: 821 us / 9.68 ms / 4.57 ms with plain 8^3 cells;
// 4^3 cells of reach 1, 894 / 11.3 / 5.48; of reach 3, 767 / 8.03 / 3.93; of
// reach 8, 756 / 7.66 / 3.77; 8^3 cells of reach 5, 763 / 8.23 / 3.90.
constexpr int kMacroShift = 2;
constexpr int kMacro = 1 << kMacroShift;

// InnerCoords.  When a sample's voxel coordinates provably lie in [-1/4, n +
// 1/4] along every axis of its brick, the stencil's indices need no clamps (the
// apron holds every voxel they reach) and floors can be taken with an addition
// instead of a conversion (|u| < 2^22).  That is so when
//  - the brick's space range lies inside its voxel range, within kInnerSpace of
//    the origin, and its values within +-kInnerValue (times at most kMaxTF
//    entries: below 2^21 for the lookup's floor): DevBrick::inner;
//  - the eye lies within kInnerEye of the origin and every pixel has a proper
//    direction: DevView::inner;
//  - the step is at most kInnerStep and a constant jitter at most kInnerJitter
//    steps: FrameArgs::inner.
//  - the scene is tame (below): kSceneInner.
// Ray parameters then stay below 2^17, and their rounding, the lattice's and
// the position's add up to less than 1/16 voxel.  Anything else takes the
// clamped form, which gives the same bits.
constexpr float kInnerSpace = 16384.0f, kInnerEye = 32768.0f, kInnerValue = 1024.0f, kInnerStep = 1024.0f,
                kInnerJitter = 16.0f;

// A scene is tame (kSceneTame) when its voxels and its transfer function's
// entries lie within +-kTame: then every sample's lookup is finite and, but for a
// gradient of exactly -1e-4 along all three axes (whose shade divides by 0), so
// is its shade, and a sample of alpha 0 leaves the colour unchanged even if it is
// evaluated.
constexpr float kTame = 1e18f;
constexpr int kSceneInner = 1, kSceneTame = 2;  // FrameArgs::scene_flags

// One brick as the kernels see it (80 bytes).
struct DevBrick {
  const float4* base;    // quad of voxel (0,0,0) of the voxel range inside the padded array
  const uint8_t* cells;  // [mz][my][mx] macrocell codes
  int sy, sz;            // padded row and slice pitch, in quads
  int n[3];              // voxel range size
  float lo[3];           // voxelRange.lower (voxel-unit origin of the brick)
  float space_lo[3], space_hi[3];
  int inner;             // InnerCoords (the host's; kernels read FrameArgs::scene_flags)
};

// Per-view state read by the kernels.
struct DevView {
  float org[3], dir_00[3], dir_du[3], dir_dv[3];
  int width, height;
  float max_depth;
  int n_ranks;
  int sched;          // offset of the view's schedule in the schedule buffer:
                      // [rank_order n_ranks][rank_start n_ranks+1][rank_bricks n_bricks]
  int pixel_offset;   // offset of the view's first pixel in batched outputs
  int rects;          // offset of the ranks' screen rectangles in the schedule buffer:
                      // per rank [cx0, cy0, cx1, cy1] in 8x4 chunks, inclusive
  int inner;          // InnerCoords
};

// Everything one render launch needs, passed by value.
struct FrameArgs {
  const DevBrick* bricks;
  const DevView* views;
  const int* sched;
  const float4* tf;
  int n_tf;
  float dt, et_alpha;
  int jitter_mode;
  float jitter_value;
  int crosshair, spp, accum_id, accumulate, heat_map;
  float heat_map_scale;
  int composite_mode, island_id, num_islands;
  int inner;                    // InnerCoords
  const int* scene_flags;       // kSceneInner: every brick is InnerCoords; kSceneTame
  // outputs
  uint32_t* fb;                 // [H*W] (single view) RGBA8
  float4* rank_images;          // [n_ranks][H*W] or null
  float* rank_depth;            // [n_ranks][H*W] or null
  float4* accum;                // [n_ranks][H*W] or null
  unsigned long long* counter;  // total samples (atomic) or null
};

// One persistent render launch over a list of (view, output) items: warps
// pull pixel chunks from an atomic work counter.  A single view leaves
// view_ids, fbs and tile_prefix null and uses single_view and f.fb.
struct BatchArgs {
  FrameArgs f;
  const int* view_ids;       // [n_items] view of each batch item
  uint32_t* const* fbs;      // [n_items] output frame buffers (device)
  const int* tile_prefix;    // [n_items+1] prefix sum of chunks per item
  int n_items;
  int single_view;
  int total_tiles;           // chunks in the launch
  unsigned int* work_counter;
  const int* chunk_order;    // single view: chunk ids in the order to render them, or null (ring order)
  const int* pair_chunks;    // the instance of few chunks, single view in cost order (or null): so many first
                             // positions are rendered with two lanes per ray, as two items each
  bool ring_pairs;           // ... in ring order: every position is
  int group_chunks;          // single view in cost order: the first group_chunks chunks of chunk_order are
                             // rendered by lane groups (kLaneGroup lanes per ray), as kLaneGroup items each
};

// Lanes per ray of the lane-group render (march_brick_group).
constexpr int kLaneGroup = 4;

// Cost-ordered chunks of one view (schedule.cu): a coarse probe per chunk
// estimates its cost, and the chunks are sorted stably by cost class, most
// expensive first, so the frame does not end on a long chunk started last.
constexpr int kOrderClasses = 64;  // cost classes, a quarter octave apart
struct ChunkOrderArgs {
  FrameArgs f;
  int view;
  int cw, ch;        // chunk shape
  int n_slots;       // ring slots of the chunk grid (the probe's input order)
  uint8_t* key;      // [n_slots] cost class per slot (0xff off the grid)
  int* cid;          // [n_slots] chunk id per slot
  uint32_t* hist;    // [kOrderClasses][chunk_order_blocks(n_slots)] counts; zero between launches
  int warps;         // resident warps of the render
  int* pairs;        // set: chunks at the head of the order that two lanes per ray render sooner
  uint32_t* readers; // scatter CTAs that have read hist; zero between launches
  int* order;        // [chunks] chunk ids, most expensive first
  int n_chunks;      // chunks of the grid (entries of `order`)
  // counters of the render launch that follows, zeroed by the probe (or null)
  unsigned int* zero_work;
  unsigned long long* zero_samples;
};
int chunk_order_blocks(int n_slots);

// Programmatic dependent launch: `beside` lets the kernel start before the
// stream's previous kernel has finished (once all its CTAs have called
// launch_dependents or ended); it waits for that kernel's results with
// wait_for_primary (at once when launched in the ordinary way).
template <class... Args>
cudaError_t launch_beside(void (*kernel)(Args...), int grid, int threads, size_t smem, cudaStream_t s, bool beside,
                          Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = beside ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
cudaError_t launch_chunk_order(const ChunkOrderArgs& a, cudaStream_t s);

// Rank-split render of one view into f.fb: work items are (8x4 chunk, rank)
// pairs for the ranks whose screen rectangle covers the chunk; f.rank_images
// is the scratch plane set [n_ranks][H*W] of the marched ranks.  At most
// kSplitMaxRanks ranks (one mask bit each).
constexpr int kSplitMaxRanks = 64;
constexpr uint32_t kSplitBackground = 127u;  // item code of a chunk no rank covers
struct SplitArgs {
  FrameArgs f;
  int view;
  int n_slots;                     // work positions: ring slots of 8x4 chunks, or chunks when ordered (< 2^25)
  const int* chunk_order;          // chunk ids by position (cost order), or null (ring order)
  unsigned long long* masks;       // [n_slots] covering ranks per slot
  uint32_t* offsets;               // [n_slots] first item of each slot
  uint32_t* block_sums;            // [ceil(n_slots / 1024)] scan scratch
  uint32_t* items;                 // [n_slots * max(1, n_ranks)] slot << 7 | rank position
  uint32_t* n_items;               // items listed (written by the plan kernel)
  unsigned int* chunk_done;        // [n_slots] tickets, zero between launches
  unsigned int* work_counter;
};

// Chunk shapes (pixels a warp takes per work-counter grab, rendered as 8x4
// sub-tiles): 8x4, 8x8, 16x8 or 32x4.
inline bool known_chunk(int w, int h) {
  return (w == 8 && h == 4) || (w == 8 && h == 8) || (w == 16 && h == 8) || (w == 32 && h == 4);
}
// Chunks are handed out centre-out, in square rings around the image centre
// (the longest rays usually cross the middle, so they start first and the
// frame's tail is short).  Work slots cover the smallest odd square of rings
// that contains the chunk grid; slots outside the grid are skipped.
__host__ __device__ inline int ring_radius(int cxn, int cyn) {
  const int cx = (cxn - 1) / 2, cy = (cyn - 1) / 2;
  int r = cx > cxn - 1 - cx ? cx : cxn - 1 - cx;
  const int ry = cy > cyn - 1 - cy ? cy : cyn - 1 - cy;
  return r > ry ? r : ry;
}
__host__ __device__ inline int ring_slots(int width, int height, int cw, int ch) {
  const int r = ring_radius((width + cw - 1) / cw, (height + ch - 1) / ch);
  return (2 * r + 1) * (2 * r + 1);
}
constexpr int kRenderThreads = 128;
// Ordered composite; the order is in device memory, or, up to kParamRanks
// ranks, in host memory and passed with the launch.
constexpr int kParamRanks = 1024;
cudaError_t launch_composite_f32(const float4* imgs, const int* order, const int* host_order, int n_ranks, int npx,
                                 int mode, uint32_t* fb, cudaStream_t s);
cudaError_t launch_composite_u8(const uint32_t* imgs, const int* order, const int* host_order, int n_ranks, int npx,
                                uint32_t* fb, cudaStream_t s);
// Fills a brick's padded array from its voxels (x fastest) and the value range
// of each macrocell.  Sets flag bits: kVoxelNonfinite, kVoxelWide (a value
// beyond +-kInnerValue), kVoxelHuge (beyond +-kTame).
constexpr int kVoxelNonfinite = 1, kVoxelWide = 2, kVoxelHuge = 4;
cudaError_t launch_fill_brick(const DevBrick& b, const float* src, float4* dst_alloc, float2* ranges, int* flags,
                              cudaStream_t s);
// Persistent render launch; `batch` selects the instance tuned for batches.
constexpr int kSingleRenderBlocks = 5, kBatchRenderBlocks = 7;  // CTAs per SM
// A single view of few 8x4 chunks per resident warp ends on its longest rays,
// which run faster with fewer, less spilling neighbours (4 / 5 CTAs per SM, us,
// one lane per ray:
// 64^3 at 512^2 81 / 89, 256^3 at 1024x768 257 / 263, 512^3 at 512^2 599 / 633);
// with many, throughput counts (64^3 at 1024^2 155 / 146, 256^3 at 1280x1024 354
// / 331, 512^3 at 1920x1080 650 / 630; 512^3 at 1024^2, 10.8 chunks per warp of
// the 5-CTA instance, 602 / 605).
// Without a cost order, frames of at most kPairRingChunks chunks are rendered
// with two lanes per ray throughout (one / two, us: 64^3 at 256^2 69 / 53, at
// 480^2, 7200 chunks, 69 / 69; 512^3 at 64^2 420 / 281, at 480^2 487 / 336; a
// GPU's warps are 2432 at a time).
constexpr int kFewChunkRenderBlocks = 4, kFewChunksPerWarp = 9, kPairRingChunks = 8192;
constexpr int kRingPairs = -2;  // the kernel's LG for ring_pairs
// CTAs per SM of the differentiable form's forward (checkpointed march).  Six
// 512^2 views of 256^3: 785 us at 5, 820 at 6, 875 at 7; one 1024^2 view of
// 512^3: 900 at 5, 914 at 4.
constexpr int kTrainForwardBlocks = 5;
// `stage`: ALOHA_STAGING_NONE or _NEXT_SAMPLE (the stencil loads), or, for
// batches, kStageUnroll2: direct loads with the march loop written out two
// steps per trip.
constexpr int kStageUnroll2 = 2;
// `lane_groups`: the instance that renders the first a.group_chunks chunks of
// the cost order with lane groups (single view, 8x4 chunks, direct loads).
// `few`: the 8x4 instance for few chunks per warp (single view, direct loads).
// `beside`: the launch before it in the stream is launch_chunk_order's.
cudaError_t launch_render_warps(const BatchArgs& a, int chunk_w, int chunk_h, int grid, bool batch, cudaStream_t s,
                                int stage = ALOHA_STAGING_NONE, bool lane_groups = false, bool few = false, bool beside = false);
// The macrocell codes of all bricks from their value ranges; prefix[k] = number
// of transfer-function entries below k with non-zero alpha.  Cells of brick b
// start at bricks[b].cells - cells in each array; tmp is scratch of their size.
cudaError_t launch_macrocell_codes(const DevBrick* bricks, int n_bricks, int most_cells, size_t all_cells, const float2* ranges,
                                   const int* prefix, int n_tf, uint8_t* cells, uint8_t* tmp, cudaStream_t s);
inline int macrocells(const DevBrick& b) {
  return ((b.n[0] + kMacro - 1) >> kMacroShift) * ((b.n[1] + kMacro - 1) >> kMacroShift) *
         ((b.n[2] + kMacro - 1) >> kMacroShift);
}
// CTAs of the render kernel that fit on one SM for a chunk shape (0 if the shape is unknown).
int render_blocks_per_sm(int chunk_w, int chunk_h, int n_tf, bool batch, int stage = ALOHA_STAGING_NONE,
                         bool lane_groups = false, bool few = false);
// `many_ranks` selects the instance tuned for many short (chunk, rank) items.
constexpr int kManyRankSplitBlocks = 7;  // CTAs per SM
cudaError_t launch_render_split(const SplitArgs& a, int grid, bool many_ranks, cudaStream_t s);
int render_split_blocks_per_sm(int n_tf, bool many_ranks);

}  // namespace aloha
