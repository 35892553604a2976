// A host stand-in for the CUDA runtime calls of api.cpp, for tests of what the
// host side puts in which order.  "Device" memory is reserved host memory, so a
// check can look at it.  Work is put off as the runtime may put it off:
//  - a copy from pageable memory has left the source when the call returns, but
//    reaches the device only when its stream is waited for;
//  - a kernel has run only when its stream is waited for.
// Streams are non-blocking: none waits for another.
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <utility>
#include <vector>

#include "adjoint.h"
#include "internal.h"

namespace fake {

struct Block {
  size_t bytes;
  cudaMemoryType type;
};
inline std::map<char*, Block> blocks;
inline std::map<cudaStream_t, std::vector<std::function<void()>>> pending;
inline size_t device_bytes = size_t(280) << 30, device_used = 0;
inline int waits = 0;                         // waits of the host for a stream or the device
inline std::vector<aloha::BatchArgs> renders;  // launches of the pixel render
inline std::vector<int> rendered_flags;       // *scene_flags as each of them would read it
inline cudaStream_t capturing = reinterpret_cast<cudaStream_t>(-1);  // its work is recorded, not run
inline int dirty_counts = 0;                  // chunk orders whose counters were not zero when they ran
inline int fill_flags = 0;                    // what the next uploads find (kVoxel*)

inline const Block* find(const void* p) {
  auto it = blocks.upper_bound((char*)p);
  if (it == blocks.begin()) return nullptr;
  --it;
  return (char*)p < it->first + it->second.bytes ? &it->second : nullptr;
}
inline cudaError_t reserve(void** p, size_t bytes, cudaMemoryType type) {
  void* m = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
  blocks[(char*)m] = {bytes, type};
  *p = m;
  return cudaSuccess;
}
inline void finish(cudaStream_t s) {
  if (s == capturing) return;
  auto work = std::move(pending[s]);
  pending[s].clear();
  for (auto& w : work) w();
}
inline void wait(cudaStream_t s) {
  ++waits;
  finish(s);
}
inline void wait_all() {
  ++waits;
  for (auto& p : pending) finish(p.first);
}
inline void copy(void* dst, const void* src, size_t n, cudaStream_t s) {
  const Block *to = find(dst), *from = find(src);
  if (to && !from) {  // pageable to device: staged now, lands later
    std::vector<char> stage((const char*)src, (const char*)src + n);
    pending[s].push_back([dst, stage] { std::memcpy(dst, stage.data(), stage.size()); });
  } else {
    pending[s].push_back([=] { std::memcpy(dst, src, n); });
  }
}

}  // namespace fake

extern "C" {

cudaError_t cudaMalloc(void** p, size_t n) {
  if (fake::device_used + n > fake::device_bytes) return cudaErrorMemoryAllocation;
  fake::device_used += n;
  return fake::reserve(p, n, cudaMemoryTypeDevice);
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  const fake::Block b = fake::blocks.at((char*)p);
  fake::device_used -= b.bytes;
  fake::blocks.erase((char*)p);
  munmap(p, b.bytes);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return fake::reserve(p, n, cudaMemoryTypeHost); }
cudaError_t cudaFreeHost(void* p) {
  const size_t n = fake::blocks.at((char*)p).bytes;
  fake::blocks.erase((char*)p);
  munmap(p, n);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* p, unsigned) {
  *d = p;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_b, size_t* total) {
  *free_b = fake::device_bytes - fake::device_used;
  *total = fake::device_bytes;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  const fake::Block* b = fake::find(p);
  *a = cudaPointerAttributes{};
  a->type = b ? b->type : cudaMemoryTypeUnregistered;
  a->devicePointer = b ? (void*)p : nullptr;
  return cudaSuccess;
}
// On the default stream: waits for what is there, then copies; only a copy to
// the host, or one on the device side, has landed when it returns.
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
  fake::finish(nullptr);
  fake::copy(dst, src, n, nullptr);
  if (kind != cudaMemcpyHostToDevice) fake::wait(nullptr);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
  fake::copy(dst, src, n, s);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  fake::pending[s].push_back([=] { std::memset(p, v, n); });
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  fake::wait(s);
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  fake::wait_all();
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
  *st = s == fake::capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  *p = cudaDeviceProp{};
  p->major = 10;
  p->minor = 3;
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }

}  // extern "C"

namespace aloha {

int chunk_order_blocks(int n_slots) { return (n_slots + 1023) / 1024; }
// Writes all that the kernels write, and leaves the counters zero as they do.
cudaError_t launch_chunk_order(const ChunkOrderArgs& a, cudaStream_t s) {
  fake::pending[s].push_back([a] {
    bool zero = *a.readers == 0u;
    for (int i = 0; i < kOrderClasses * chunk_order_blocks(a.n_slots); ++i) zero = zero && a.hist[i] == 0u;
    fake::dirty_counts += !zero;
    std::memset(a.key, 0xab, a.n_slots);
    std::memset(a.cid, 0xab, 4 * (size_t)a.n_slots);
    std::memset(a.order, 0xab, 4 * (size_t)a.n_chunks);
    *a.pairs = 3;
  });
  return cudaSuccess;
}
cudaError_t launch_composite_f32(const float4*, const int*, const int*, int, int npx, int, uint32_t* fb,
                                 cudaStream_t s) {
  fake::pending[s].push_back([=] { std::memset(fb, 0x5a, (size_t)npx * 4); });
  return cudaSuccess;
}
cudaError_t launch_composite_u8(const uint32_t*, const int*, const int*, int, int npx, uint32_t* fb, cudaStream_t s) {
  return launch_composite_f32(nullptr, nullptr, nullptr, 0, npx, 0, fb, s);
}
cudaError_t launch_fill_brick(const DevBrick&, const float*, float4*, float2*, int* flags, cudaStream_t s) {
  const int found = fake::fill_flags;
  fake::pending[s].push_back([=] { *flags |= found; });
  return cudaSuccess;
}
cudaError_t launch_render_warps(const BatchArgs& a, int, int, int, bool, cudaStream_t s, int, bool, bool, bool) {
  fake::finish(s);  // the launch runs at once; other streams' work may still be on its way
  fake::renders.push_back(a);
  fake::rendered_flags.push_back(*a.f.scene_flags);
  return cudaSuccess;
}
cudaError_t launch_macrocell_codes(const DevBrick*, int, int, size_t, const float2*, const int*, int, uint8_t*, uint8_t*,
                                   cudaStream_t) {
  return cudaSuccess;
}
int render_blocks_per_sm(int, int, int, bool, int, bool, bool) { return 5; }
cudaError_t launch_render_split(const SplitArgs&, int, bool, cudaStream_t) { return cudaSuccess; }
int render_split_blocks_per_sm(int, bool) { return 5; }
cudaError_t launch_forward_train(const TrainArgs&, unsigned, int, bool, cudaStream_t) { return cudaSuccess; }
int forward_train_blocks_per_sm(int) { return 5; }
cudaError_t launch_backward(const TrainArgs&, int, bool, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_backward_empty(const TrainArgs&, int, bool, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_fold_quads(float4*, float*, const int[3], cudaStream_t) { return cudaSuccess; }
int backward_blocks_per_sm(int) { return 5; }

}  // namespace aloha
