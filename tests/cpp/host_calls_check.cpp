// Checks of what the host side of the C ABI (api.cpp) leaves done when a call
// returns, on a stand-in for the CUDA runtime.  Arguments: the checks to run.
// Prints one line per failure; status 1 if there was any.
#include <cmath>
#include <random>
#include <string>

#include "aloha.h"
#include "fake_cuda.h"

namespace {

int failures = 0;
#define CHECK(cond)                                                        \
  do {                                                                     \
    if (!(cond)) {                                                         \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #cond);               \
      ++failures;                                                          \
    }                                                                      \
  } while (0)

const cudaStream_t kSide = reinterpret_cast<cudaStream_t>(0x1000);

aloha_brick_desc brick(int nx, int ny, int nz, float grow = 0.0f) {
  aloha_brick_desc d{};
  const int n[3] = {nx, ny, nz};
  for (int a = 0; a < 3; ++a) {
    d.voxel_hi[a] = d.cell_hi[a] = n[a];
    d.space_lo[a] = -grow;
    d.space_hi[a] = (float)n[a] + grow;
  }
  return d;
}

void* device(size_t bytes) {
  void* p = nullptr;
  cudaMalloc(&p, bytes);
  return p;
}

// A context with a camera, a size and a table, ready to render.
aloha_ctx* context(const aloha_brick_desc& d, const float* voxels) {
  aloha_ctx* c = nullptr;
  CHECK(aloha_create(0, &c) == ALOHA_OK);
  const float tf[8] = {0, 0, 0, 0, 1, 1, 1, 1};
  CHECK(aloha_set_bricks(c, &d, &voxels, 1) == ALOHA_OK);
  CHECK(aloha_set_transfer_function(c, tf, 2) == ALOHA_OK);
  const float org[3] = {4, 4, -20}, d00[3] = {-0.4f, -0.4f, 1}, du[3] = {0.1f, 0, 0}, dv[3] = {0, 0.1f, 0};
  CHECK(aloha_set_camera(c, 0, org, d00, du, dv) == ALOHA_OK);
  CHECK(aloha_resize(c, 0, 8, 8) == ALOHA_OK);
  return c;
}

// The flags that let kernels drop their clamps and lookups are the scene's when
// a render is launched on any stream, also one that does not wait for the default stream.
void scene_flag() {
  const float* voxels = static_cast<const float*>(device(8 * 8 * 8 * 4));
  uint32_t* fb = static_cast<uint32_t*>(device(8 * 8 * 4));
  const aloha_brick_desc inside = brick(8, 8, 8), beyond = brick(8, 8, 8, 1.0f);
  aloha_ctx* c = context(inside, voxels);
  auto flags = [&] {
    CHECK(aloha_render(c, 0, fb, kSide) == ALOHA_OK);
    return fake::rendered_flags.back();
  };
  const int kAll = aloha::kSceneInner | aloha::kSceneTame;
  CHECK(flags() == kAll);
  CHECK(aloha_set_bricks(c, &beyond, &voxels, 1) == ALOHA_OK);
  CHECK(flags() == aloha::kSceneTame);
  CHECK(aloha_set_bricks(c, &inside, &voxels, 1) == ALOHA_OK);
  CHECK(flags() == kAll);
  fake::fill_flags = aloha::kVoxelWide;
  CHECK(aloha_update_brick(c, 0, voxels) == ALOHA_OK);
  CHECK(flags() == aloha::kSceneTame);
  fake::fill_flags = aloha::kVoxelWide | aloha::kVoxelHuge;
  CHECK(aloha_update_brick(c, 0, voxels) == ALOHA_OK);
  CHECK(flags() == 0);
  fake::fill_flags = 0;
  CHECK(aloha_update_brick(c, 0, voxels) == ALOHA_OK);
  CHECK(flags() == kAll);
  float tf[8] = {0, 0, 0, 0, 1, 2e18f, 1, 1};
  CHECK(aloha_set_transfer_function(c, tf, 2) == ALOHA_OK);
  CHECK(flags() == 0);
  tf[5] = 1e18f;
  CHECK(aloha_set_transfer_function(c, tf, 2) == ALOHA_OK);
  CHECK(flags() == kAll);
  // bricks that are refused half-way: a recorded launch may still be replayed
  fake::fill_flags = aloha::kVoxelNonfinite;
  const int* flag = fake::renders.back().f.scene_flags;
  CHECK(aloha_set_bricks(c, &beyond, &voxels, 1) == ALOHA_ERR_INVALID_ARGUMENT);
  CHECK((*flag & aloha::kSceneInner) == 0);
  fake::fill_flags = 0;
  aloha_destroy(c);
}

// The table is on the device when the call returns.
void table() {
  const float* voxels = static_cast<const float*>(device(8 * 8 * 8 * 4));
  uint32_t* fb = static_cast<uint32_t*>(device(8 * 8 * 4));
  aloha_ctx* c = context(brick(8, 8, 8), voxels);
  CHECK(aloha_render(c, 0, fb, kSide) == ALOHA_OK);
  const float4* tf = fake::renders.back().f.tf;
  for (int k = 0; k < 3; ++k) {
    const float rgba[8] = {0.25f * k, 0, 0, 0, 1, 1, 0.5f * k, 1};
    CHECK(aloha_set_transfer_function(c, rgba, 2) == ALOHA_OK);
    CHECK(std::memcmp(tf, rgba, sizeof rgba) == 0);
    const int want[3] = {0, 0, 1};  // entries of non-zero alpha before each
    CHECK(std::memcmp(tf + 2, want, sizeof want) == 0);
  }
  aloha_destroy(c);
}

// The composite waits for its stream unless images and frame buffer are plain
// device memory.
void composite() {
  const int w = 16, h = 8, n = 3, order[n] = {2, 0, 1};
  const size_t in_bytes = (size_t)n * w * h * 16, out_bytes = (size_t)w * h * 4;
  void *dev_in = device(in_bytes), *dev_out = device(out_bytes), *man_in = nullptr, *man_out = nullptr;
  fake::reserve(&man_in, in_bytes, cudaMemoryTypeManaged);
  fake::reserve(&man_out, out_bytes, cudaMemoryTypeManaged);
  std::vector<char> host_in(in_bytes), host_out(out_bytes);
  for (bool u8 : {false, true})
    for (void* in : {dev_in, man_in, (void*)host_in.data()})
      for (void* out : {dev_out, man_out, (void*)host_out.data()}) {
        std::memset(out, 0, out_bytes);
        const int waits = fake::waits;
        const int rc = u8 ? aloha_composite_over_rgba8((uint32_t*)in, order, n, w, h, (uint32_t*)out, kSide)
                          : aloha_composite_over((float*)in, order, n, w, h, ALOHA_COMPOSITE_FP32, (uint32_t*)out, kSide);
        CHECK(rc == ALOHA_OK);
        if (in != dev_in || out != dev_out)
          CHECK(*(uint32_t*)out == 0x5a5a5a5au);
        else
          CHECK(fake::waits == waits);
        fake::wait_all();
      }
}

// Bricks up to 2^31 quads of plain pitches, and scenes up to the device's
// memory of them, are taken.
void large() {
  const float* voxels = static_cast<const float*>(device(4096));
  aloha_ctx* c = nullptr;
  CHECK(aloha_create(0, &c) == ALOHA_OK);
  auto set = [&](int nx, int ny, int nz) {
    const aloha_brick_desc d = brick(nx, ny, nz);
    return aloha_set_bricks(c, &d, &voxels, 1);
  };
  const int sizes[][3] = {{1024, 1440, 1440}, {512, 2036, 2036}, {256, 2860, 2860}, {1, 1, 1}, {128, 128, 128}};
  for (const auto& n : sizes) {
    CHECK(set(n[0], n[1], n[2]) == ALOHA_OK);
    aloha_stats st;
    CHECK(aloha_get_stats(c, &st) == ALOHA_OK);
    const long long plain = aloha::plain_pitch(n[0], n[1]).quads(n[2]);
    CHECK(plain <= aloha::kMaxBrickQuads && st.brick_bytes >= (size_t)plain * 16);
  }
  CHECK(set(1025, 1440, 1440) == ALOHA_ERR_INVALID_ARGUMENT);
  CHECK(set(1024, 1443, 1440) == ALOHA_ERR_INVALID_ARGUMENT);
  aloha_destroy(c);
  // memory for plain pitches only: 124^3 is 128^3 quads, padded 130 x 128 + 4
  CHECK(aloha_create(0, &c) == ALOHA_OK);
  const size_t plain = (size_t)128 * 128 * 128 * 16, padded = (size_t)(130 * 128 + 4) * 128 * 16, cells = 31 * 31 * 31;
  CHECK((size_t)aloha::spread_pitch(124, 124).quads(124) * 16 == padded);
  const size_t all = fake::device_bytes;
  fake::device_bytes = fake::device_used + plain + 10 * cells + 65536;
  CHECK(set(124, 124, 124) == ALOHA_OK);
  fake::device_bytes = fake::device_used - 65536;
  CHECK(set(128, 124, 124) == ALOHA_ERR_OUT_OF_MEMORY);
  fake::device_bytes = all;
  CHECK(set(124, 124, 124) == ALOHA_OK);
  aloha_stats st;
  CHECK(aloha_get_stats(c, &st) == ALOHA_OK && st.brick_bytes >= padded);
  aloha_destroy(c);
}

// A view whose rays may take unclamped coordinates has an eye within the limit
// and a proper direction at every pixel; ordinary cameras are such views.
void views() {
  const float* voxels = static_cast<const float*>(device(8 * 8 * 8 * 4));
  uint32_t* fb = static_cast<uint32_t*>(device(64 * 64 * 4));
  aloha_ctx* c = context(brick(8, 8, 8), voxels);
  std::mt19937_64 rng(11u);
  std::uniform_real_distribution<float> u(-1.0f, 1.0f);
  int inner = 0, degenerate = 0;
  for (int k = 0; k < 4000; ++k) {
    float org[3], d00[3], du[3], dv[3];
    const float scale = ldexpf(1.0f, (int)(rng() % 60) - 40);  // eyes and pixels of all sizes
    for (int a = 0; a < 3; ++a) {
      org[a] = u(rng) * (k % 4 ? 30000.0f : 60000.0f);
      d00[a] = u(rng) * scale;
      du[a] = u(rng) * 0.02f * scale;
      dv[a] = u(rng) * 0.02f * scale;
    }
    const int w = 1 + (int)(rng() % 64), h = 1 + (int)(rng() % 64), form = k % 8;
    const int px = (int)(rng() % w), py = (int)(rng() % h);
    const float along = u(rng);
    for (int a = 0; a < 3; ++a) {
      if (form == 1) dv[a] = du[a] * 2.0f;                           // one line of directions
      if (form == 3 && (k & 8)) dv[a] = du[a] * 3.0f;
      if (form == 2) du[a] = dv[a] = 0.0f;                           // one direction
      if (form == 3) d00[a] = -(px + 0.5f) * du[a] - (py + 0.5f) * dv[a];  // none at a pixel
      if (form == 4) dv[a] = k & 8 ? nextafterf(du[a], 1e30f) : du[a] * 3.0f;  // almost one line
      if (form == 5) d00[a] = du[a] * along + dv[a];                  // the eye in the image's plane
    }
    degenerate += form >= 1 && form <= 5;
    CHECK(aloha_set_camera(c, 0, org, d00, du, dv) == ALOHA_OK && aloha_resize(c, 0, w, h) == ALOHA_OK);
    CHECK(aloha_render(c, 0, fb, kSide) == ALOHA_OK);
    fake::wait_all();
    const aloha::DevView& v = fake::renders.back().f.views[0];
    if (!v.inner) continue;
    ++inner;
    CHECK(form != 1 && form != 2 && form != 3 && form != 5);
    bool proper = true;
    for (int a = 0; a < 3; ++a) proper = proper && std::fabs(org[a]) <= aloha::kInnerEye;
    for (int y = 0; y < h; ++y)
      for (int x = 0; x < w; ++x) {  // generate_ray
        float d[3], len2 = 0.0f, unit2 = 0.0f;
        for (int a = 0; a < 3; ++a) d[a] = fmaf(y + 0.5f, dv[a], fmaf(x + 0.5f, du[a], d00[a]));
        len2 = fmaf(d[2], d[2], fmaf(d[1], d[1], d[0] * d[0]));
        const float inv = 1.0f / sqrtf(len2);
        for (int a = 0; a < 3; ++a) unit2 += d[a] * inv * (d[a] * inv);
        proper = proper && std::fabs(unit2 - 1.0f) < 1e-5f;
      }
    CHECK(proper);
  }
  CHECK(inner > 500 && degenerate > 2000);
  fake::renders.clear();
  aloha_destroy(c);
}

// The chunk order's counters are zero whenever its kernels run: after other frame
// sizes, after a recorded frame that was never replayed, and when one is replayed
// after frames of other sizes.
void chunk_counters() {
  const float* voxels = static_cast<const float*>(device(8 * 8 * 8 * 4));
  uint32_t* fb = static_cast<uint32_t*>(device(4096 * 4096 * 4));
  aloha_ctx* c = context(brick(8, 8, 8), voxels);
  CHECK(aloha_set_chunk_order(c, ALOHA_CHUNKS_PROBED) == ALOHA_OK);
  const cudaStream_t recorded = reinterpret_cast<cudaStream_t>(0x2000);
  auto frame = [&](int w, int h, cudaStream_t s) {
    CHECK(aloha_resize(c, 0, w, h) == ALOHA_OK && aloha_render(c, 0, fb, s) == ALOHA_OK);
    fake::wait_all();
  };
  frame(1024, 1024, kSide);
  frame(100, 60, kSide);
  frame(1024, 1024, kSide);
  frame(3000, 2000, kSide);
  frame(640, 480, kSide);
  CHECK(aloha_resize(c, 0, 800, 600) == ALOHA_OK);
  int n = 0, order[1];
  CHECK(aloha_get_composite_order(c, 0, order, 1, &n) == ALOHA_OK);  // the view's state is on the device
  fake::capturing = recorded;
  CHECK(aloha_render(c, 0, fb, recorded) == ALOHA_OK);
  const auto graph = fake::pending[recorded];
  fake::pending[recorded].clear();
  fake::capturing = reinterpret_cast<cudaStream_t>(-1);
  frame(800, 600, kSide);
  auto replay = [&] {
    for (const auto& work : graph) work();
  };
  replay();
  for (int w : {160, 2048, 700}) {
    frame(w, w, kSide);
    replay();
    frame(w, w, kSide);
  }
  CHECK(fake::dirty_counts == 0);
  aloha_destroy(c);
}

}  // namespace

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    const std::string a = argv[i];
    if (a == "scene_flag") scene_flag();
    else if (a == "table") table();
    else if (a == "composite") composite();
    else if (a == "large") large();
    else if (a == "views") views();
    else if (a == "chunk_counters") chunk_counters();
    else ++failures;
  }
  std::printf("failures %d\n", failures);
  return failures == 0 ? 0 : 1;
}
