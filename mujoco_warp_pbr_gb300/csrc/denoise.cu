// Edge-avoiding a-trous denoiser of the path-traced tier (Dammertz et al. 2010;
// mujoco_warp_pbr/_src/denoise.py:101-248): `denoise_iterations` passes of a 5 x 5 B3-spline filter
// with holes (steps 1, 2, 4, ...) over the demodulated radiance, weighted by normal, depth, albedo
// and luminance differences, the luminance tolerance following the per-pixel noise estimate
// (sample variance, 3 x 3 Gaussian-smoothed, propagated through the passes as in SVGF).
//
// GB300 layout: the path tracer already wrote the demodulated radiance + variance (one float4 per
// pixel) into denoise_buffers[0] and the filter's guide as one 16-byte record per pixel (normal and
// albedo as half floats, depth). Passes of steps up to 4 (launch_pass) stage a 16 x 16 tile and its 2-step border in
// shared memory once, unpacked and with the luminance, 48 bytes a pixel: a tap is three 128-bit loads at
// constant offsets, without conversions, bounds (pixels outside the image have a zero normal, so zero
// weight) or addresses. Bound by the taps' arithmetic (some 55 instructions; 86 where every tap loads and
// unpacks, the form of the wider steps, whose border does not fit). 1024 worlds of 128 x 128, steps 1, 2
// and 4 with the finish: 1.00, 1.02 and 1.16 ms (1.57, 1.57 and 2.00 with every tap from global memory). The last pass remodulates, tone maps and writes the display
// RGB (and the HDR) directly: no separate demodulate / finish passes over the image.
#include <algorithm>

#include "abi_internal.h"
#include "denoise_common.cuh"
#include "shading.cuh"

namespace mjpbr {
namespace {

constexpr int kTile = 16;

struct Images {
  int32_t ncam;
  int32_t width[MJPBR_MAX_RENDER], height[MJPBR_MAX_RENDER], adr[MJPBR_MAX_RENDER];
  int32_t tiles_x[MJPBR_MAX_RENDER];
  int32_t tile_base[MJPBR_MAX_RENDER + 1];
};

struct Filter {
  int32_t step;  // 0: no filtering (finish only)
  float sigma_color, sigma_normal, sigma_depth, sigma_albedo;
};

MJ_DEV float b3(int i) { return i == 2 ? 0.375f : ((i == 1 || i == 3) ? 0.25f : 0.0625f); }

// The finish of a pixel (address adr in the output rows, world w): remodulation, tone map, outputs.
MJ_DEV void finish_pixel(const MjpbrScene& s, int32_t w, int64_t adr, float4 out, V3 albedo) {
  const float* e = s.aov_emission + adr * 3;
  const V3 exposed = remodulate(out, V3{e[0], e[1], e[2]}, albedo);
  if (s.settings.render_hdr) {
    const V3 hdr = exposed / bf(s.exposure, w, 1, 0);
    s.hdr_data[adr * 3] = hdr.x;
    s.hdr_data[adr * 3 + 1] = hdr.y;
    s.hdr_data[adr * 3 + 2] = hdr.z;
  }
  s.rgb_data[adr] = encode_display(display_transform(exposed, s.settings.tone_mapper));
}

// 3 x 3 Gaussian of the variance: the per-pixel estimate from few samples is itself noisy.
MJ_DEV float smooth_variance(const float4* in, int32_t px, int32_t py, int32_t W, int32_t H) {
  float variance = 0.0f, variance_weight = 0.0f;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int32_t y = min(max(py + j - 1, 0), H - 1);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int32_t x = min(max(px + i - 1, 0), W - 1);
      const float g = (i == 1 ? 0.5f : 0.25f) * (j == 1 ? 0.5f : 0.25f);
      variance += g * __ldg(in + y * W + x).w;
      variance_weight += g;
    }
  }
  return variance / variance_weight;
}

// What the taps of a pixel share, and their sums.
struct Taps {
  V3 normal, albedo;
  float depth, l0, inv_sigma_l, inv_sigma_a, inv_sigma_z, sigma_normal;
  V3 total;
  float total_variance, weight_sum;
  MJ_DEV void begin(const Guide& g0, float4 c, float variance, const Filter& f) {
    normal = g0.normal;
    albedo = g0.albedo;
    depth = g0.depth;
    inv_sigma_l = 1.0f / (f.sigma_color * sqrtf(fmaxf(variance, 0.0f)) + 1.0e-6f);
    l0 = luminance(V3{c.x, c.y, c.z});
    inv_sigma_a = 1.0f / f.sigma_albedo;
    // depth differences are relative and grow with the filter footprint
    inv_sigma_z = 1.0f / fmaxf(f.sigma_depth * g0.depth * (float)f.step, 1.0e-6f);
    sigma_normal = f.sigma_normal;
    total = v3(0.0f);
    total_variance = weight_sum = 0.0f;
  }
  // background neighbours (zero normal) get zero weight
  MJ_DEV void add(float kernel, V3 c, float variance, float lum, V3 n, V3 a, float z) {
    const float wn = fast_pow(fmaxf(dot(normal, n), 0.0f), sigma_normal);
    const float distance = fabsf(z - depth) * inv_sigma_z + fabsf(lum - l0) * inv_sigma_l + length(a - albedo) * inv_sigma_a;
    const float weight = kernel * wn * __expf(-distance);
    total += c * weight;
    total_variance += weight * weight * variance;
    weight_sum += weight;
  }
  // the centre pixel always contributes, so weight_sum > 0
  MJ_DEV float4 result() const {
    const V3 c = total / weight_sum;
    return make_float4(c.x, c.y, c.z, total_variance / (weight_sum * weight_sum));
  }
};

// The pass of step kStep, tiles staged in shared memory (three float4 per pixel of the tile and its border).
template <int kStep, bool kFinish>
__global__ void __launch_bounds__(kTile* kTile) atrous_tile_kernel(const __grid_constant__ MjpbrScene s, const __grid_constant__ Images im,
                                                                   Filter f, const float4* __restrict__ src, float4* __restrict__ dst) {
  constexpr int kEdge = kTile + 4 * kStep, kPixels = kEdge * kEdge;
  extern __shared__ float4 staged[];  // [3][kPixels]: colour, luminance; normal, depth; albedo, variance
  const int32_t t = blockIdx.x;
  int32_t cam = 0;
  while (cam + 1 < im.ncam && t >= im.tile_base[cam + 1]) ++cam;
  const int32_t lt = t - im.tile_base[cam];
  const int32_t W = im.width[cam], H = im.height[cam];
  const int32_t x0 = (lt % im.tiles_x[cam]) * kTile, y0 = (lt / im.tiles_x[cam]) * kTile;
  const int32_t tx = threadIdx.x % kTile, ty = threadIdx.x / kTile;
  const int32_t px = x0 + tx, py = y0 + ty;
  for (int32_t w = blockIdx.y; w < s.nworld; w += gridDim.y) {
    const int64_t base = (int64_t)w * s.rgb_stride + im.adr[cam];
    const uint4* guide = reinterpret_cast<const uint4*>(s.aov_guide) + base;
    const float4* in = src + base;
    __syncthreads();  // the last world's tile has been read
    for (int32_t i = threadIdx.x; i < kPixels; i += kTile * kTile) {
      const int32_t y = y0 - 2 * kStep + i / kEdge, x = x0 - 2 * kStep + i % kEdge;
      float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      Guide g;
      g.normal = g.albedo = v3(0.0f);
      g.depth = 0.0f;
      if (x >= 0 && x < W && y >= 0 && y < H) {
        c = __ldg(in + y * W + x);
        g = unpack_guide(__ldg(guide + y * W + x));
      }
      staged[i] = make_float4(c.x, c.y, c.z, luminance(V3{c.x, c.y, c.z}));
      staged[kPixels + i] = make_float4(g.normal.x, g.normal.y, g.normal.z, g.depth);
      staged[2 * kPixels + i] = make_float4(g.albedo.x, g.albedo.y, g.albedo.z, c.w);
    }
    __syncthreads();
    if (px >= W || py >= H) continue;
    const float4* mine = staged + ty * kEdge + tx;  // the tap (0, 0)
    constexpr int kCentre = 2 * kStep * kEdge + 2 * kStep;
    const float4 c0 = mine[kCentre], n0 = mine[kPixels + kCentre], a0 = mine[2 * kPixels + kCentre];
    const Guide g0{V3{n0.x, n0.y, n0.z}, V3{a0.x, a0.y, a0.z}, n0.w};
    float4 out = make_float4(c0.x, c0.y, c0.z, a0.w);
    if (length_sq(g0.normal) != 0.0f) {
      Taps taps;
      taps.begin(g0, out, smooth_variance(in, px, py, W, H), f);
#pragma unroll
      for (int j = 0; j < 5; ++j) {
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const int at = j * kStep * kEdge + i * kStep;
          const float4 c = mine[at], n = mine[kPixels + at], a = mine[2 * kPixels + at];
          taps.add(b3(i) * b3(j), V3{c.x, c.y, c.z}, a.w, c.w, V3{n.x, n.y, n.z}, V3{a.x, a.y, a.z}, n.w);
        }
      }
      out = taps.result();
    }
    if (kFinish) {
      finish_pixel(s, w, base + py * W + px, out, g0.albedo);
    } else {
      dst[base + py * W + px] = out;
    }
  }
}

// Any step, every tap from global memory; step 0 is the finish alone.
template <bool kFinish>
__global__ void __launch_bounds__(kTile* kTile) atrous_kernel(const __grid_constant__ MjpbrScene s,
                                                              const __grid_constant__ Images im, Filter f,
                                                              const float4* __restrict__ src, float4* __restrict__ dst) {
  const int32_t t = blockIdx.x;
  int32_t cam = 0;
  while (cam + 1 < im.ncam && t >= im.tile_base[cam + 1]) ++cam;
  const int32_t lt = t - im.tile_base[cam];
  const int32_t W = im.width[cam], H = im.height[cam];
  const int32_t px = (lt % im.tiles_x[cam]) * kTile + (int32_t)(threadIdx.x % kTile);
  const int32_t py = (lt / im.tiles_x[cam]) * kTile + (int32_t)(threadIdx.x / kTile);
  if (px >= W || py >= H) return;
  for (int32_t w = blockIdx.y; w < s.nworld; w += gridDim.y) {
    const int64_t base = (int64_t)w * s.rgb_stride + im.adr[cam];
    const uint4* guide = reinterpret_cast<const uint4*>(s.aov_guide) + base;
    const float4* in = src + base;
    const int32_t idx = py * W + px;
    const Guide g0 = unpack_guide(__ldg(guide + idx));
    float4 out = __ldg(in + idx);
    if (f.step > 0 && length_sq(g0.normal) != 0.0f) {
      Taps taps;
      taps.begin(g0, out, smooth_variance(in, px, py, W, H), f);
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const int32_t y = py + (j - 2) * f.step;
        if (y < 0 || y >= H) continue;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const int32_t x = px + (i - 2) * f.step;
          if (x < 0 || x >= W) continue;
          const int32_t q = y * W + x;
          const float4 sq = __ldg(in + q);
          const Guide gq = unpack_guide(__ldg(guide + q));
          const V3 c{sq.x, sq.y, sq.z};
          taps.add(b3(i) * b3(j), c, sq.w, luminance(c), gq.normal, gq.albedo, gq.depth);
        }
      }
      out = taps.result();
    }
    if (kFinish) {
      finish_pixel(s, w, base + idx, out, g0.albedo);
    } else {
      dst[base + idx] = out;
    }
  }
}

template <int kStep, bool kFinish>
int launch_tile(const MjpbrScene& s, const Images& im, const Filter& f, const float4* src, float4* dst, dim3 grid, cudaStream_t stream) {
  const size_t smem = (size_t)3 * (kTile + 4 * kStep) * (kTile + 4 * kStep) * sizeof(float4);
  if (int rc = ensure_smem(reinterpret_cast<const void*>(atrous_tile_kernel<kStep, kFinish>), smem, "denoise")) return rc;
  atrous_tile_kernel<kStep, kFinish><<<grid, kTile * kTile, smem, stream>>>(s, im, f, src, dst);
  return check_launch("atrous_tile_kernel");
}

// Passes by tile up to step 4, and at 8 if it is the last: a tile and its border are then 110 KB, two CTAs an SM,
// and a plain pass takes 853 us where the taps from global memory take 740; with the finish 898 and 916 (512
// worlds of 128 x 128). Negative sigmas, whose weights grow with the distance, never by tile: a pixel outside
// the image would count 0 x infinity there.
template <bool kFinish>
int launch_pass(const MjpbrScene& s, const Images& im, const Filter& f, const float4* src, float4* dst, dim3 grid, cudaStream_t stream) {
  const bool decays = f.sigma_color >= 0.0f && f.sigma_albedo >= 0.0f;
  switch (decays ? f.step : 0) {
    case 1: return launch_tile<1, kFinish>(s, im, f, src, dst, grid, stream);
    case 2: return launch_tile<2, kFinish>(s, im, f, src, dst, grid, stream);
    case 4: return launch_tile<4, kFinish>(s, im, f, src, dst, grid, stream);
    case 8:
      if constexpr (kFinish) return launch_tile<8, true>(s, im, f, src, dst, grid, stream);
      [[fallthrough]];
    default:
      atrous_kernel<kFinish><<<grid, kTile * kTile, 0, stream>>>(s, im, f, src, dst);
      return check_launch("atrous_kernel");
  }
}

}  // namespace

int denoise_launch(const MjpbrScene& s, cudaStream_t stream) {
  if (!s.aov_guide || !s.aov_emission || !s.denoise_buffers[0] || !s.denoise_buffers[1] || !s.rgb_data) {
    return set_error(MJPBR_ERR_ARG, "the denoiser needs aov_guide, aov_emission, denoise_buffers and rgb_data");
  }
  if (s.settings.render_hdr && !s.hdr_data) return set_error(MJPBR_ERR_ARG, "render_hdr needs hdr_data");
  if (s.denoise_iterations < 0 || s.denoise_iterations > 16) {
    return set_error(MJPBR_ERR_ARG, "denoise_iterations %d outside [0, 16]", s.denoise_iterations);
  }
  Images im{};
  im.ncam = 0;
  im.tile_base[0] = 0;
  for (int32_t c = 0; c < s.nrender; ++c) {
    if (!s.render_rgb[c] || s.rgb_adr[c] < 0) continue;
    const int32_t k = im.ncam++;
    im.width[k] = s.cam_res[c][0];
    im.height[k] = s.cam_res[c][1];
    im.adr[k] = s.rgb_adr[c];
    im.tiles_x[k] = (im.width[k] + kTile - 1) / kTile;
    im.tile_base[k + 1] = im.tile_base[k] + im.tiles_x[k] * ((im.height[k] + kTile - 1) / kTile);
  }
  const int32_t tiles = im.tile_base[im.ncam];
  if (tiles == 0 || s.nworld == 0) return MJPBR_OK;
  Filter f{0, s.settings.denoise_sigma_color, s.settings.denoise_sigma_normal, s.settings.denoise_sigma_depth,
           s.settings.denoise_sigma_albedo};
  const dim3 grid(tiles, std::min(s.nworld, 65535));
  float4* buf[2] = {reinterpret_cast<float4*>(s.denoise_buffers[0]), reinterpret_cast<float4*>(s.denoise_buffers[1])};
  const int32_t passes = s.denoise_iterations;
  for (int32_t i = 0; i < passes - 1; ++i) {
    f.step = 1 << i;
    if (int rc = launch_pass<false>(s, im, f, buf[i & 1], buf[(i + 1) & 1], grid, stream)) return rc;
  }
  f.step = passes > 0 ? 1 << (passes - 1) : 0;
  return launch_pass<true>(s, im, f, buf[passes > 0 ? (passes - 1) & 1 : 0], nullptr, grid, stream);
}

}  // namespace mjpbr
