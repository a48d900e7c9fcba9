// kf_pyramid.cu - bilateral filter, 2x2 downsample and vertex/normal maps of
// the depth pyramid (depth_processing.hpp:54-284, depth_processing.cu:70-122).
//
// The bilateral filter (level 0), then one fused kernel per level that writes
// the vertex map, the normal map and, for every pixel of the next level, its
// 2x2 downsample.  A CTA projects its pixels and a border of one from the depth
// image into shared memory, where the normals find their four neighbours: one
// level stays in one launch, and the border's vertices are the same float
// expression as the CTA's that owns them.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "kf_internal.h"

namespace kf {
namespace {

struct DepthParams {
  float depth_scale, min_depth, max_depth;
  float max_normal_depth_jump, max_downsample_depth_jump;
  int radius;
  float spatial_scale, range_scale;
};

DepthParams depth_params(const kf_depth_options& o) {
  DepthParams p;
  p.depth_scale = o.depth_scale;
  p.min_depth = o.min_depth;
  p.max_depth = o.max_depth;
  p.max_normal_depth_jump = o.max_normal_depth_jump;
  p.max_downsample_depth_jump = o.max_downsample_depth_jump;
  p.radius = o.bilateral_radius;
  // gaussian_exponent_scale (depth_processing.hpp:118-121)
  p.spatial_scale = -0.5f / (o.bilateral_spatial_sigma * o.bilateral_spatial_sigma);
  p.range_scale = -0.5f / (o.bilateral_depth_sigma * o.bilateral_depth_sigma);
  return p;
}

constexpr int kTileX = 32;
constexpr int kTileY = 8;

// The bilateral weight of a float exponent in [-104, 0]: exp evaluated in
// double and rounded once to float, the correctly rounded value (the CPU
// oracle computes the same).  Table-driven as in Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic" (1989): x = (32 m + j) ln2 / 32 + r, exp(x) = 2^m 2^(j/32) e^r
// with e^r from its Taylor series to r^5 (|r| <= ln2 / 64, error below
// 2^-48).  A result within 2^-45 of a float rounding boundary, and one that
// rounds to a subnormal float, takes the library's exp instead.
constexpr int kExpTable = 32;
__device__ __forceinline__ float gaussian(float arg, const double* s_exp2) {
  const double x = static_cast<double>(arg);
  const double shifted = __fma_rn(x, 46.16624130844683, 6755399441055744.0);  // 32 / ln2, 1.5 * 2^52
  const int k = __double2loint(shifted);
  const double kd = shifted - 6755399441055744.0;
  // ln2 / 32 in two parts, the first of 26 bits: kd (13 bits) times it is exact
  double r = __fma_rn(kd, -0.02166084898635745, x);
  r = __fma_rn(kd, -4.06140840434059e-10, r);
  double e = __fma_rn(r, 1.0 / 120.0, 1.0 / 24.0);
  e = __fma_rn(r, e, 1.0 / 6.0);
  e = __fma_rn(r, e, 0.5);
  e = __fma_rn(r, e, 1.0);
  e = __fma_rn(r, e, 1.0);
  e *= s_exp2[k & (kExpTable - 1)];
  const unsigned low = static_cast<unsigned>(__double2loint(e));
  const double y = __hiloint2double(__double2hiint(e) + ((k >> 5) << 20), static_cast<int>(low));
  // the 29 bits below a float's last: half way is 2^28
  if (((low - 0x10000000u + 0x80u) & 0x1FFFFFFFu) < 0x100u || !(arg >= -87.0f)) return static_cast<float>(exp(x));
  return static_cast<float>(y);
}

// BilateralFilter::operator() (depth_processing.hpp:71-115).  A CTA stages its
// pixels and their border of `radius` as metres (NaN where the depth is not
// usable) and raw values, so each depth is divided and range-tested once
// instead of once per window it is in.  Bound by its double arithmetic:
// 640x480 at radius 2, 24.7 us against 29.6 us with exp and a division per
// sample.
template <bool Tile>
__global__ void __launch_bounds__(kTileX* kTileY)
    bilateral_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int width,
                     int height, DepthParams p) {
  extern __shared__ float s_tile[];
  __shared__ double s_exp2[kExpTable];
  const int span_x = kTileX + 2 * p.radius, span_y = kTileY + 2 * p.radius;
  float* s_metres = s_tile;
  float* s_raw = s_tile + span_x * span_y;
  const int tid = threadIdx.y * kTileX + threadIdx.x;
  const int left = static_cast<int>(blockIdx.x) * kTileX - p.radius;
  const int top = static_cast<int>(blockIdx.y) * kTileY - p.radius;
  auto pixel = [&](int x, int y, float& m, float& value) {
    m = kNaN;
    value = 0.0f;
    if (x >= 0 && y >= 0 && x < width && y < height) {
      const uint16_t raw = __ldg(in + y * width + x);
      value = static_cast<float>(raw);
      if (!depth_in_range(raw, p.depth_scale, p.min_depth, p.max_depth, m)) m = kNaN;
    }
  };
  if constexpr (Tile) {
    for (int i = tid; i < span_x * span_y; i += kTileX * kTileY) {
      pixel(left + i % span_x, top + i / span_x, s_metres[i], s_raw[i]);
    }
  }
  if (tid < kExpTable) s_exp2[tid] = exp2(static_cast<double>(tid) * (1.0 / kExpTable));
  __syncthreads();
  const int col = blockIdx.x * kTileX + threadIdx.x;
  const int row = blockIdx.y * kTileY + threadIdx.y;
  if (col >= width || row >= height) return;
  auto staged = [&](int dx, int dy, float& m, float& value) {
    if constexpr (Tile) {
      const int i = (static_cast<int>(threadIdx.y) + p.radius + dy) * span_x + static_cast<int>(threadIdx.x) + p.radius + dx;
      m = s_metres[i];
      value = s_raw[i];
    } else {
      pixel(col + dx, row + dy, m, value);
    }
  };
  float center, unused;
  staged(0, 0, center, unused);
  uint16_t result = 0;
  if (center == center) {
    float weighted_sum = 0.0f;
    float weight_sum = 0.0f;
    // the reference's window, clipped to the image
    const int x0 = max(-p.radius, -col), x1 = min(p.radius, width - 1 - col);
    const int y0 = max(-p.radius, -row), y1 = min(p.radius, height - 1 - row);
    for (int dy = y0; dy <= y1; ++dy) {
      for (int dx = x0; dx <= x1; ++dx) {
        float sample, raw;
        staged(dx, dy, sample, raw);
        if (sample != sample) continue;
        const float d2 = static_cast<float>((dx * dx) + (dy * dy));
        const float dd = sample - center;
        const float arg = (d2 * p.spatial_scale) + (dd * dd * p.range_scale);
        if (arg < -104.0f) continue;  // rounds to zero: adds nothing
        const float weight = gaussian(arg, s_exp2);
        weighted_sum += weight * raw;
        weight_sum += weight;
      }
    }
    if (weight_sum > 0.0f) {
      result = static_cast<uint16_t>(lroundf(weighted_sum / weight_sum));
    }
  }
  out[row * width + col] = result;
}

// The same filter at radius 2, the default.  A pair of pixels has one weight,
// whichever of the two is the window's centre (the depth difference enters
// squared), so the CTA computes each pair once, for the twelve neighbours
// after a pixel in row order, and a pixel reads the other twelve from the
// pixels before it: 15 exponentials per pixel with the tile's border instead
// of 25.  640x480: 19.49 us against 24.7 us.
constexpr int kPairRows = 16;              // pixel rows of a CTA's tile
constexpr int kPairSpanX = kTileX + 4;     // with the border
constexpr int kPairSpanY = kPairRows + 4;
constexpr int kPairs = 12;
constexpr int kPairFrom = (kPairRows + 2) * kPairSpanX;  // pixels whose later neighbours matter
__host__ __device__ constexpr int pair_dy(int f) { return f < 2 ? 0 : (f < 7 ? 1 : 2); }
__host__ __device__ constexpr int pair_dx(int f) { return f < 2 ? f + 1 : (f < 7 ? f - 4 : f - 9); }
__global__ void __launch_bounds__(256)
    bilateral_pairs_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, int width, int height,
                           DepthParams p) {
  __shared__ float s_metres[kPairSpanY * kPairSpanX], s_raw[kPairSpanY * kPairSpanX];
  __shared__ float s_weight[kPairs][kPairFrom];
  __shared__ double s_exp2[kExpTable];
  const int tid = threadIdx.x;
  const int left = static_cast<int>(blockIdx.x) * kTileX - 2, top = static_cast<int>(blockIdx.y) * kPairRows - 2;
  for (int i = tid; i < kPairSpanY * kPairSpanX; i += 256) {
    const int x = left + i % kPairSpanX, y = top + i / kPairSpanX;
    float m = kNaN, value = 0.0f;
    if (x >= 0 && y >= 0 && x < width && y < height) {
      const uint16_t raw = __ldg(in + y * width + x);
      value = static_cast<float>(raw);
      if (!depth_in_range(raw, p.depth_scale, p.min_depth, p.max_depth, m)) m = kNaN;
    }
    s_metres[i] = m;
    s_raw[i] = value;
  }
  if (tid < kExpTable) s_exp2[tid] = exp2(static_cast<double>(tid) * (1.0 / kExpTable));
  __syncthreads();
  for (int i = tid; i < kPairFrom; i += 256) {
    const int x = i % kPairSpanX;
    const float here = s_metres[i];
#pragma unroll
    for (int f = 0; f < kPairs; ++f) {
      const int tx = x + pair_dx(f);
      float weight = 0.0f;  // of an unusable neighbour, and of one past the border (never read)
      if (tx >= 0 && tx < kPairSpanX) {
        const float dd = s_metres[i + pair_dy(f) * kPairSpanX + pair_dx(f)] - here;
        const float d2 = static_cast<float>(pair_dx(f) * pair_dx(f) + pair_dy(f) * pair_dy(f));
        const float arg = (d2 * p.spatial_scale) + (dd * dd * p.range_scale);
        if (arg >= -104.0f) weight = gaussian(arg, s_exp2);  // below: rounds to zero
      }
      s_weight[f][i] = weight;
    }
  }
  __syncthreads();
  const int col = left + 2 + tid % kTileX;
  for (int ty = tid / kTileX; ty < kPairRows; ty += 256 / kTileX) {
    const int row = top + 2 + ty;
    if (col >= width || row >= height) continue;
    const int at = (ty + 2) * kPairSpanX + tid % kTileX + 2;
    uint16_t result = 0;
    if (s_metres[at] == s_metres[at]) {
      float weighted_sum = 0.0f, weight_sum = 0.0f;
      // the window in row order; a zero weight adds nothing, as skipping does
#pragma unroll
      for (int f = kPairs - 1; f >= 0; --f) {
        const int from = at - pair_dy(f) * kPairSpanX - pair_dx(f);
        const float weight = s_weight[f][from];
        weighted_sum += weight * s_raw[from];
        weight_sum += weight;
      }
      weighted_sum += s_raw[at];  // the centre's weight is exactly 1
      weight_sum += 1.0f;
#pragma unroll
      for (int f = 0; f < kPairs; ++f) {
        const float weight = s_weight[f][at];
        weighted_sum += weight * s_raw[at + pair_dy(f) * kPairSpanX + pair_dx(f)];
        weight_sum += weight;
      }
      if (weight_sum > 0.0f) result = static_cast<uint16_t>(lroundf(weighted_sum / weight_sum));
    }
    out[row * width + col] = result;
  }
}

// VertexProjection::operator() (depth_processing.hpp:215-226), identity pose.
__device__ __forceinline__ f3 vertex_at(const uint16_t* __restrict__ depth, int width, int x, int y,
                                        const Intr& k, const DepthParams& p) {
  float d;
  if (!depth_in_range(__ldg(depth + y * width + x), p.depth_scale, p.min_depth, p.max_depth, d)) {
    return nan3();
  }
  return back_project(k, static_cast<float>(x), static_cast<float>(y), d);
}

// One level: vertex + NormalEstimation (depth_processing.hpp:251-279) +
// BlockDownsample into the next level (depth_processing.hpp:153-187).  The
// CTA's vertices and a border of one pixel are projected once, into shared
// memory, instead of five times per pixel (640x480: 9.0 -> 6.7 us).
__global__ void __launch_bounds__(kTileX* kTileY)
    level_kernel(const uint16_t* __restrict__ depth, int width, int height, Intr k, DepthParams p,
                 float* __restrict__ vertices, float* __restrict__ normals,
                 uint16_t* __restrict__ next) {
  constexpr int kSpanX = kTileX + 2, kSpanY = kTileY + 2;
  __shared__ float s_x[kSpanX * kSpanY], s_y[kSpanX * kSpanY], s_z[kSpanX * kSpanY];
  const int tid = threadIdx.y * kTileX + threadIdx.x;
  const int left = static_cast<int>(blockIdx.x) * kTileX - 1, top = static_cast<int>(blockIdx.y) * kTileY - 1;
  for (int i = tid; i < kSpanX * kSpanY; i += kTileX * kTileY) {
    const int x = left + i % kSpanX, y = top + i / kSpanX;
    f3 v = nan3();
    if (x >= 0 && y >= 0 && x < width && y < height) v = vertex_at(depth, width, x, y, k, p);
    s_x[i] = v.x;
    s_y[i] = v.y;
    s_z[i] = v.z;
  }
  __syncthreads();
  const int col = blockIdx.x * kTileX + threadIdx.x;
  const int row = blockIdx.y * kTileY + threadIdx.y;
  if (col >= width || row >= height) return;
  const int at = (threadIdx.y + 1) * kSpanX + threadIdx.x + 1;
  auto vertex = [&](int i) { return make(s_x[i], s_y[i], s_z[i]); };
  const f3 c = vertex(at);
  const size_t pix = static_cast<size_t>(row) * width + col;
  store3(vertices + pix * 3, c);

  f3 n = nan3();
  if (col != 0 && row != 0 && col + 1 < width && row + 1 < height) {
    const f3 l = vertex(at - 1);
    const f3 r = vertex(at + 1);
    const f3 t = vertex(at - kSpanX);
    const f3 b = vertex(at + kSpanX);
    if (finite3((((c + l) + r) + t) + b) &&
        !(fabsf(r.z - l.z) > p.max_normal_depth_jump || fabsf(b.z - t.z) > p.max_normal_depth_jump)) {
      const f3 nn = cross(b - t, r - l);
      const float length = norm(nn);
      if (length > 0.0f) n = nn / length;
    }
  }
  store3(normals + pix * 3, n);

  if (next != nullptr) {
    const int nw = width / 2, nh = height / 2;
    if (col < nw && row < nh) {
      uint32_t sum = 0, count = 0;
      uint16_t lo = 0xFFFF, hi = 0;
#pragma unroll
      for (int dy = 0; dy < 2; ++dy) {
#pragma unroll
        for (int dx = 0; dx < 2; ++dx) {
          const uint16_t s = __ldg(depth + (row * 2 + dy) * width + (col * 2 + dx));
          if (s == 0) continue;
          sum += s;
          ++count;
          lo = s < lo ? s : lo;
          hi = hi < s ? s : hi;
        }
      }
      uint16_t result = 0;
      if (count != 0) {
        const float max_m = static_cast<float>(hi) / p.depth_scale;
        const float min_m = static_cast<float>(lo) / p.depth_scale;
        if (!(max_m - min_m > p.max_downsample_depth_jump)) {
          result = static_cast<uint16_t>((sum + (count / 2u)) / count);
        }
      }
      next[row * nw + col] = result;
    }
  }
}

kf_intrinsics scaled(kf_intrinsics k, uint32_t level) {
  // CameraIntrinsics::scaled (rgbd.hpp:66-70)
  const float s = 1.0f / static_cast<float>(1u << level);
  return kf_intrinsics{k.fx * s, k.fy * s, k.cx * s, k.cy * s};
}

void validate(const kf_depth_options& o) {
  // DepthProcessingOptions::validated (depth_processing.cpp:74-94)
  require(o.levels > 0u, "Depth pyramid must have at least one level");
  require(o.levels <= 4u, "Depth pyramid supports at most 4 levels");
  require(o.depth_scale > 0.0f, "Depth scale must be positive");
  require(o.min_depth >= 0.0f && o.max_depth > o.min_depth, "Depth range is invalid");
  require(o.max_normal_depth_jump >= 0.0f, "Normal depth jump threshold must be non-negative");
  require(o.max_downsample_depth_jump >= 0.0f, "Downsample depth jump threshold must be non-negative");
  require(o.bilateral_radius >= 0, "Bilateral filter radius must be non-negative");
  require(o.bilateral_spatial_sigma > 0.0f, "Bilateral spatial sigma must be positive");
  require(o.bilateral_depth_sigma > 0.0f, "Bilateral depth sigma must be positive");
}

}  // namespace

uint32_t Pyramid::prepare(uint32_t w, uint32_t h, kf_intrinsics k) {
  require(w > 0 && h > 0, "Depth image must be non-empty");
  if (raw.count != static_cast<size_t>(w) * h) {
    generation = next_generation();
    raw.resize(static_cast<size_t>(w) * h);
  }
  width = w;
  height = h;
  intrinsics = k;
  if (levels.size() < options.levels) levels.resize(options.levels);
  uint32_t lw = w, lh = h, count = 0;
  for (uint32_t level = 0; level < options.levels; ++level) {
    if (lw == 0 || lh == 0) break;
    PyramidLevelBuffers& b = levels[level];
    const size_t n = static_cast<size_t>(lw) * lh;
    if (b.depth.count != n || b.vertices.count != n * 3 || b.normals.count != n * 3) {
      generation = next_generation();
      b.depth.resize(n);
      b.vertices.resize(n * 3);
      b.normals.resize(n * 3);
    }
    b.width = lw;
    b.height = lh;
    b.intrinsics = scaled(k, level);
    ++count;
    lw /= 2;
    lh /= 2;
  }
  level_count = count;
  return count;
}

void Pyramid::launch(cudaStream_t s) const {
  DepthParams p = depth_params(options);
  // no window reaches past the image: any non-negative radius is accepted, and
  // the filter's sizes and indices stay those of the image
  p.radius = std::min(p.radius, static_cast<int>(std::max(width, height)) - 1);
  for (uint32_t level = 0; level < level_count; ++level) {
    const PyramidLevelBuffers& b = levels[level];
    const dim3 block(kTileX, kTileY);
    const dim3 grid(ceil_div(b.width, kTileX), ceil_div(b.height, kTileY));
    if (level == 0) {
      if (!options.bilateral_filter || options.bilateral_radius == 0) {
        check(cudaMemcpyAsync(b.depth.ptr, raw.ptr, raw.bytes(), cudaMemcpyDeviceToDevice, s),
              "pyramid level-0 copy");
      } else {
        // a window too large for the staging (48 KB) reads its pixels directly
        const size_t tile = 2 * sizeof(float) * (kTileX + 2 * static_cast<size_t>(p.radius)) *
                            (kTileY + 2 * static_cast<size_t>(p.radius));
        // pairs: scales and metres all finite, so that a pair's weight is the
        // same number from both ends and the centre's is exactly 1
        if (options.bilateral_radius == 2 && std::isfinite(p.spatial_scale) && std::isfinite(p.range_scale) &&
            std::isfinite(65535.0f / p.depth_scale)) {
          bilateral_pairs_kernel<<<dim3(ceil_div(b.width, kTileX), ceil_div(b.height, kPairRows)), 256, 0, s>>>(
              raw.ptr, b.depth.ptr, static_cast<int>(b.width), static_cast<int>(b.height), p);
        } else if (tile <= 47u * 1024u) {
          bilateral_kernel<true><<<grid, block, tile, s>>>(raw.ptr, b.depth.ptr, static_cast<int>(b.width),
                                                           static_cast<int>(b.height), p);
        } else {
          bilateral_kernel<false><<<grid, block, 0, s>>>(raw.ptr, b.depth.ptr, static_cast<int>(b.width),
                                                         static_cast<int>(b.height), p);
        }
        check(cudaGetLastError(), "bilateral_kernel launch");
      }
    }
    uint16_t* next = level + 1 < level_count ? levels[level + 1].depth.ptr : nullptr;
    level_kernel<<<grid, block, 0, s>>>(b.depth.ptr, static_cast<int>(b.width),
                                        static_cast<int>(b.height), intr_from(b.intrinsics), p,
                                        b.vertices.ptr, b.normals.ptr, next);
    check(cudaGetLastError(), "level_kernel launch");
  }
}

}  // namespace kf

using namespace kf;

extern "C" {

void kf_default_depth_options(kf_depth_options* o) {
  // DepthProcessingOptions defaults (depth_processing.hpp:24-41, rgbd.hpp:15-17)
  o->levels = 3;
  o->depth_scale = 5000.0f;
  o->min_depth = 0.4f;
  o->max_depth = 8.0f;
  o->max_normal_depth_jump = 0.1f;
  o->max_downsample_depth_jump = 0.1f;
  o->bilateral_filter = 1;
  o->bilateral_radius = 2;
  o->bilateral_spatial_sigma = 2.0f;
  o->bilateral_depth_sigma = 0.08f;
}

kf_status kf_pyramid_create(const kf_depth_options* options, kf_pyramid** out) {
  return guarded([&] {
    require(options != nullptr && out != nullptr, "kf_pyramid_create: null argument");
    validate(*options);
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
      throw CudaError("no CUDA device available");
    }
    auto* p = new kf_pyramid();
    p->impl.options = *options;
    *out = p;
  });
}

kf_status kf_pyramid_destroy(kf_pyramid* pyramid) {
  return guarded([&] { delete pyramid; });
}

kf_status kf_pyramid_build(kf_pyramid* pyramid, const uint16_t* depth, uint32_t width, uint32_t height,
                           kf_intrinsics intrinsics, int32_t memory, uint32_t* level_count) {
  return guarded([&] {
    require(pyramid != nullptr && depth != nullptr, "kf_pyramid_build: null argument");
    Pyramid& p = pyramid->impl;
    const uint32_t count = p.prepare(width, height, intrinsics);
    const cudaMemcpyKind kind = memory == KF_MEMORY_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    check(cudaMemcpyAsync(p.raw.ptr, depth, p.raw.bytes(), kind, 0), "pyramid depth upload");
    p.launch(0);
    check(cudaStreamSynchronize(0), "pyramid build");
    if (level_count) *level_count = count;
  });
}

kf_status kf_pyramid_level(const kf_pyramid* pyramid, uint32_t index, kf_level_view* out) {
  return guarded([&] {
    require(pyramid != nullptr && out != nullptr, "kf_pyramid_level: null argument");
    const Pyramid& p = pyramid->impl;
    require(index < p.level_count, "kf_pyramid_level: level index out of range");
    const PyramidLevelBuffers& b = p.levels[index];
    out->depth = b.depth.ptr;
    out->vertices = b.vertices.ptr;
    out->normals = b.normals.ptr;
    out->width = b.width;
    out->height = b.height;
    out->intrinsics = b.intrinsics;
  });
}

kf_status kf_pyramid_raw_depth(const kf_pyramid* pyramid, const uint16_t** depth) {
  return guarded([&] {
    require(pyramid != nullptr && depth != nullptr, "kf_pyramid_raw_depth: null argument");
    const Pyramid& p = pyramid->impl;
    require(p.level_count > 0, "kf_pyramid_raw_depth: no frame built yet");
    *depth = p.raw.ptr;
  });
}

kf_status kf_pyramid_download_level(const kf_pyramid* pyramid, uint32_t index, uint16_t* depth,
                                    float* vertices, float* normals) {
  return guarded([&] {
    require(pyramid != nullptr, "kf_pyramid_download_level: null pyramid");
    const Pyramid& p = pyramid->impl;
    require(index < p.level_count, "kf_pyramid_download_level: level index out of range");
    const PyramidLevelBuffers& b = p.levels[index];
    if (depth) check(cudaMemcpy(depth, b.depth.ptr, b.depth.bytes(), cudaMemcpyDeviceToHost), "download depth");
    if (vertices)
      check(cudaMemcpy(vertices, b.vertices.ptr, b.vertices.bytes(), cudaMemcpyDeviceToHost), "download vertices");
    if (normals)
      check(cudaMemcpy(normals, b.normals.ptr, b.normals.bytes(), cudaMemcpyDeviceToHost), "download normals");
  });
}

}  // extern "C"
