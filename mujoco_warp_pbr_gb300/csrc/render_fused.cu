// Real-time tier of scenes without meshes and with few geoms (fused_supported): one kernel, one
// thread per camera sample, from the camera ray to the shaded sample.
//
// Such scenes are traced by the warp-wide scan (scan.cuh), in which a warp's lanes stay together, so
// splitting a sample's work over kernels (render_wave.cu) buys no convergence any more, while the
// records between its stages cost 230 bytes of HBM traffic per sample and six launches. Here a sample's
// record stays on the SM: each segment (the camera ray, then its mirror ray) is traced, its surface
// evaluated and parked in shared memory, every light's shadow rays traced into counts in shared
// memory, and then the surface shaded with the counts, by the wavefront's own functions in its order
// (the images are bit-identical). Parking keeps the shading state out of the registers while rays are
// traced.
//
// Bound by instruction issue and fetch: the phases' code together is several times the instruction
// cache, so a CTA's warps take each phase together (500 x 84 x 84 worlds: 1.42 ms without the barriers,
// 1.24 with), the more of them the better (1.10 -> 0.87 with CTAs of 512 threads for 256), and a bulb's
// rays test only the boxes around its centre's ray (500 x 84 x 84: 942 us a frame with one test for all of a
// light's rays, 930 so). 2048 worlds with cameras of 64, 128 and 256 pixels: 23.2 ms (28.5 with CTAs of 256); the
// staged kernels with the same scan take 40.
#include <algorithm>
#include <type_traits>

#include "abi_internal.h"
// one call in each kernel
#define MJPBR_SURFACE_CALL __forceinline__
#include "rt_shade.cuh"
#include "scan.cuh"

namespace mjpbr {
namespace {

constexpr int kTile = 16;            // pixel tiles of 16 x 16, addressed in Z order within the tile
constexpr int32_t kMaxLights = 16;   // shadow counts in shared memory, 1 KB per light
// CTAs of 512 threads, two an SM, when there are kWideCtas of them per SM and they take no more lanes
// than CTAs of 256, three an SM: phases taken by twice the warps are fetched half as often, but the
// work comes in larger pieces. us a frame, 512 / 256 threads: worlds of 64 x 64 with 100 worlds (5 CTAs an
// SM) 105 / 121, 64 worlds 78 / 80, 32 worlds 51 / 48, one 35 / 30; of 256 x 256 with 8 worlds 105 / 112, 4
// worlds (3.4 CTAs an SM) 63 / 59; 2000 of 16 x 16, half of whose lanes would idle, 293 / 253.
constexpr int kWide = 512, kNarrow = 256;
constexpr int64_t kWideCtas = 4;
constexpr size_t kFusedSmem = 100 * 1024;

// CTAs of each camera: its pixels, tile by tile, kThreads / samples per CTA.
struct FusedMap {
  int32_t w0;
  int32_t tiles_x[MJPBR_MAX_RENDER];
  int32_t cta_base[MJPBR_MAX_RENDER + 1];
};

// A surface parked in shared memory: word k of a thread at base[k * kThreads] (conflict-free).
constexpr int32_t kSurfaceWords = 14;
template <int kThreads>
MJ_DEV void park_surface(float* base, const Surface& sf, V3 normal) {
  const float v[kSurfaceWords] = {sf.base_color.x, sf.base_color.y, sf.base_color.z, sf.metallic, sf.roughness, sf.reflectance, sf.occlusion,
                                  sf.emissive.x, sf.emissive.y, sf.emissive.z, sf.alpha, normal.x, normal.y, normal.z};
#pragma unroll
  for (int k = 0; k < kSurfaceWords; ++k) base[k * kThreads] = v[k];
}
template <int kThreads>
MJ_DEV Surface take_surface(const float* base, V3* normal) {
  float v[kSurfaceWords];
#pragma unroll
  for (int k = 0; k < kSurfaceWords; ++k) v[k] = base[k * kThreads];
  Surface sf;
  sf.base_color = V3{v[0], v[1], v[2]};
  sf.metallic = v[3];
  sf.roughness = v[4];
  sf.reflectance = v[5];
  sf.occlusion = v[6];
  sf.emissive = V3{v[7], v[8], v[9]};
  sf.alpha = v[10];
  *normal = V3{v[11], v[12], v[13]};
  return sf;
}

// Shadow visibility from the counts of the thread's shadow rays, one word per light.
template <int kThreads>
struct CountedVis {
  const int32_t* counts;
  MJ_DEV float visibility(RtCtx& c, const Light& light, V3, V3, V3, float, uint32_t, int32_t, int32_t, int32_t li) {
    const MjpbrSettings& st = c.s->settings;
    return visible_fraction(light, st.shadow_samples, counts[li * kThreads], st.shadow_light_fraction);
  }
};

template <bool kTex, int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads == kWide ? 2 : 3) rt_fused_kernel(const __grid_constant__ MjpbrScene s, uint32_t seed,
                                                                                       const __grid_constant__ FusedMap fm) {
  using Shade = RtShade<kTex, CountedVis<kThreads>>;
  extern __shared__ __align__(16) float smem[];
  const int32_t w = fm.w0 + blockIdx.y;
  const MjpbrSettings& st = s.settings;
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  stage_world_block(s, w, smem, kThreads);
  const float* blk = smem;
  float* shared = smem + s.world_block_floats;
  const Stack stack = shared_stack(shared, kThreads, stack_entries(st.stack_depth));
  shared += kThreads * stack_entries(st.stack_depth) * 2;
  float* parked = shared + threadIdx.x;
  shared += kThreads * kSurfaceWords;
  int32_t* counts = reinterpret_cast<int32_t*>(shared) + threadIdx.x;
  shared += kThreads * s.nlight;
  float* sums = shared;  // samples_per_axis > 1: display and HDR of every thread's sample
  __shared__ __align__(16) float boxes[kSlotBoxFloats];
  if (threadIdx.x == 0) boxes[kSlotBoxFloats - 4] = 0.0f;
  __syncthreads();
  stage_boxes(blk, L, boxes, kThreads);
  __syncthreads();
  const SlotBoxes slots = staged_boxes(boxes);
  int32_t cam = 0;
  while (cam + 1 < s.nrender && (int32_t)blockIdx.x >= fm.cta_base[cam + 1]) ++cam;
  const bool rgb = s.render_rgb[cam] != 0;
  const int32_t n = rgb ? st.samples_per_axis : 1, nn = n * n;
  const int32_t ppc = kThreads / nn;
  const int32_t lp = threadIdx.x / nn, smp = threadIdx.x - lp * nn;
  const int32_t pos = (blockIdx.x - fm.cta_base[cam]) * ppc + lp;
  const int32_t tile = pos / (kTile * kTile), q = pos % (kTile * kTile);
  Pixel p;
  p.cam = cam;
  p.width = s.cam_res[cam][0];
  p.height = s.cam_res[cam][1];
  p.rec = blk + L.cam_off + cam * kCamFloats;
  p.px = (tile % fm.tiles_x[cam]) * kTile + z_x(q);
  p.py = (tile / fm.tiles_x[cam]) * kTile + z_y(q);
  p.pixelid = p.py * p.width + p.px;
  const bool active = lp < ppc && p.px < p.width && p.py < p.height;
  const bool cull = st.cull_backfaces != 0;
  RtCtx c;
  init_ctx(c, s, blk, L, w, kTex);
  int32_t err = 0;
  const M3 R = cam_mat(p.rec);
  const float inv_n = 1.0f / (float)n;
  V3 so = v3(0.0f), sd = v3(0.0f);
  float max_dist = 0.0f, depth_z = 0.0f, spread = 0.0f, cone = 0.0f;
  if (active) {
    V3 dcam, ocam;
    primary_ray(s, p, n, smp % n, smp / n, &dcam, &ocam, &max_dist, &depth_z);
    so = V3{p.rec[0], p.rec[1], p.rec[2]} + mul(R, ocam);
    sd = mul(R, dcam);
    if (rgb) {
      float pixel_spread, pixel_width;
      pixel_cone(s, p, &pixel_spread, &pixel_width);
      spread = pixel_spread * inv_n;
      cone = pixel_width * inv_n;
    }
  }
  const uint32_t pseed = seed + (uint32_t)w * (uint32_t)s.total_rays + (uint32_t)(s.ray_adr[cam] + p.pixelid);
  const int32_t ns = max(st.shadow_samples, 1);
  V3 radiance = v3(0.0f), albedo = v3(0.0f), gnormal = v3(0.0f);
  float weight = 1.0f;
  // the camera ray's segment, then its mirror ray's. The CTA's warps take each phase together: the
  // code of all phases is several times the instruction cache, that of one fits
  bool live = active;
#pragma unroll 1
  for (int32_t seg = 0; seg < 2; ++seg) {
    int32_t slot = -1;
    V3 point, normal;
    if (live) {
      const Hit hit = scan_trace<false>(slots, s, stack, blk, L, Ray{so, sd}, max_dist, cull, &err);
      if (seg == 0 && smp == 0) write_geometry(s, w, p, hit, depth_z);
      live = rgb;
      slot = hit.slot;
      if (live && hit.geom == -1) {
        radiance += Shade::background(c, sd, spread) * weight;
        live = false;
      }
      if (live) {
        point = so + sd * hit.dist;
        cone = cone + spread * hit.dist;
        const Surface sf = eval_surface<false, kTex>(s, blk, L, w, hit, hit.slot, point, sd, cone, &normal);
        park_surface<kThreads>(parked, sf, normal);
        if (seg == 0) {
          albedo = sf.base_color;
          gnormal = normal;
        }
      }
    }
    if (!__syncthreads_or(live)) break;
    if (live) {
      const V3 origin = point + normal * kRayOffset;
#pragma unroll 1
      for (int32_t li = 0; li < L.nlight; ++li) {
        const Light light = load_light(blk + L.light_off + li * kLightFloats);
        V3 l;
        float dist;
        if (!light.active || !shadow_setup(st, light, point, normal, &l, &dist)) continue;
        const int32_t rays = shadow_ray_count(light, ns);
        // a bulb's rays test only the boxes around the ray to its centre: positions along it in fractions of the
        // way, so that a ray to a point of the disc is at most the bulb's radius off, and the rounding of
        // both box tests, some ulp of the coordinates, further
        uint32_t around = slots.valid;
        if (rays > 1) {
          const V3 to = light.pos - origin;
          const float rounding = 1.0e-6f * (vmax3(vabs(origin)) + vmax3(vabs(to)) + fabsf(light.bulbradius));
          around = slots.mask_around(origin, to, 1.0f + kRayTolRel, fabsf(light.bulbradius) * 1.001f + 1.0e-5f + rounding);
        }
        int32_t visible = 0;
        if (around == 0) {
          visible = rays;
        } else {
#pragma unroll 1
          for (int32_t k = 0; k < rays; ++k) {
            Ray r;
            float len;
            r.o = origin;
            shadow_ray(light, ns, origin, l, dist, pseed, 2 * smp + seg, L.nlight, li, k, &r.d, &len);
            uint32_t meshes;
            const uint32_t mask = SlotBoxes{slots.box, around}.mask(make_inv(r), len * (1.0f + kRayTolRel) + kRayTolAbs);
            if (!scan_any<false>(mask, blk, L, r, len, cull, &meshes)) ++visible;
          }
        }
        counts[li * kThreads] = visible;
      }
    }
    __syncthreads();
    if (live) {
      const Surface sf = take_surface<kThreads>(parked, &normal);
      CountedVis<kThreads> vis{counts};
      const V3 head_dir = -V3{R.m[2], R.m[5], R.m[8]};
      const V3 shaded = Shade::shade_surface(c, vis, sf, point, normal, -sd, head_dir, pseed, 2 * smp + seg);
      if (seg == 1) {
        radiance += shaded * weight;
      } else {
        const float mirror = st.has_reflection ? mirror_reflectance(c, slot) : 0.0f;
        radiance += shaded * ((1.0f - mirror) * 1.0f);
        live = mirror > 0.0f;
        if (live) {
          weight = mirror * 1.0f;
          max_dist = kMaxVal;
          V3 mo, md;
          mirror_ray(point, normal, sd, &mo, &md);
          so = mo;
          sd = md;
        }
      }
    }
    if (!st.has_reflection) break;
  }
  if (active) {
    if (rgb) {
      const int64_t adr = (int64_t)w * s.rgb_stride + s.rgb_adr[cam] + p.pixelid;
      if (smp == 0) write_guides(s, adr, albedo, gnormal);
      const V3 display = display_transform(radiance * c.exposure, st.tone_mapper);
      if (nn == 1) {
        write_image(s, adr, v3(0.0f) + display, v3(0.0f) + radiance);  // 0 + x as the sums below
      } else {
        float* v = sums + threadIdx.x;
        v[0] = display.x, v[kThreads] = display.y, v[2 * kThreads] = display.z;
        v[3 * kThreads] = radiance.x, v[4 * kThreads] = radiance.y, v[5 * kThreads] = radiance.z;
      }
    }
  }
  if (err && s.error_word) atomicOr(s.error_word, err);
  if (nn == 1) return;
  __syncthreads();
  if (!active || smp != 0) return;
  V3 display = v3(0.0f), hdr = v3(0.0f);
  for (int32_t k = 0; k < nn; ++k) {  // the samples in sample order
    const float* v = sums + threadIdx.x + k;
    display += V3{v[0], v[kThreads], v[2 * kThreads]};
    hdr += V3{v[3 * kThreads], v[4 * kThreads], v[5 * kThreads]};
  }
  const int64_t adr = (int64_t)w * s.rgb_stride + s.rgb_adr[cam] + p.pixelid;
  const float inv_nn = inv_n * inv_n;
  write_image(s, adr, display * inv_nn, hdr * inv_nn);
}

size_t fused_smem(const MjpbrScene& s, int32_t threads) {
  const size_t nn = (size_t)s.settings.samples_per_axis * s.settings.samples_per_axis;
  const size_t words = (size_t)stack_entries(s.settings.stack_depth) * 2 + kSurfaceWords + std::max(s.nlight, 0) + (nn > 1 ? 6 : 0);
  return (size_t)s.world_block_floats * sizeof(float) + words * threads * sizeof(float);
}

FusedMap fused_map(const MjpbrScene& s, int32_t threads) {
  FusedMap fm;
  fm.w0 = 0;
  fm.cta_base[0] = 0;
  for (int32_t c = 0; c < s.nrender; ++c) {
    const int32_t W = s.cam_res[c][0], H = s.cam_res[c][1];
    const int32_t n = s.render_rgb[c] ? s.settings.samples_per_axis : 1;
    const int32_t ppc = threads / (n * n);
    const bool any = s.render_rgb[c] || s.render_depth[c] || s.render_seg[c];
    fm.tiles_x[c] = (W + kTile - 1) / kTile;
    const int64_t tiles = (int64_t)fm.tiles_x[c] * ((H + kTile - 1) / kTile);
    fm.cta_base[c + 1] = fm.cta_base[c] + (any ? (int32_t)((tiles * kTile * kTile + ppc - 1) / ppc) : 0);
  }
  return fm;
}

template <bool kTex, int kThreads>
int launch_fused(const MjpbrScene& s, uint32_t seed, FusedMap fm, cudaStream_t stream) {
  const size_t smem = fused_smem(s, kThreads);
  if (int rc = ensure_smem(reinterpret_cast<const void*>(rt_fused_kernel<kTex, kThreads>), smem, "fused render")) return rc;
  for (int32_t w0 = 0; w0 < s.nworld; w0 += kMaxGridWorlds) {
    fm.w0 = w0;
    const dim3 grid(fm.cta_base[s.nrender], std::min(kMaxGridWorlds, s.nworld - w0));
    rt_fused_kernel<kTex, kThreads><<<grid, kThreads, smem, stream>>>(s, seed, fm);
    if (int rc = check_launch("rt_fused_kernel")) return rc;
  }
  return MJPBR_OK;
}

}  // namespace

bool fused_supported(const MjpbrScene& s) {
  const bool mesh = s.nmesh + s.nhfield > 0 && s.blas_root != nullptr;
  return !mesh && !s.settings.has_transparency && s.nbvh_geom <= kScanGeoms && s.nlight <= kMaxLights && s.settings.samples_per_axis <= 16 &&
         fused_smem(s, kNarrow) <= kFusedSmem;
}

int render_fused_launch(const MjpbrScene& s, uint32_t seed, cudaStream_t stream) {
  const bool tex = s.settings.textures || s.settings.has_env || s.settings.env_background;
  const FusedMap wide = fused_map(s, kWide);
  if (wide.cta_base[s.nrender] == 0) return MJPBR_OK;
  const FusedMap narrow = fused_map(s, kNarrow);
  const int64_t nwide = wide.cta_base[s.nrender], nnarrow = narrow.cta_base[s.nrender];
  if (fused_smem(s, kWide) <= kFusedSmem && nwide * s.nworld >= kWideCtas * device_sm_count() && nwide * kWide <= nnarrow * kNarrow * 9 / 8) {
    return tex ? launch_fused<true, kWide>(s, seed, wide, stream) : launch_fused<false, kWide>(s, seed, wide, stream);
  }
  return tex ? launch_fused<true, kNarrow>(s, seed, narrow, stream) : launch_fused<false, kNarrow>(s, seed, narrow, stream);
}

}  // namespace mjpbr

#ifdef MJPBR_COUNT_OPS
namespace mjpbr {
// Counting build: this unit's copy of the counter array pointer (see opcount.cuh).
int fused_count_set(void* counts) { return cudaMemcpyToSymbol(g_op_counts, &counts, sizeof(counts)) == cudaSuccess ? 0 : 1; }
}  // namespace mjpbr
#endif
