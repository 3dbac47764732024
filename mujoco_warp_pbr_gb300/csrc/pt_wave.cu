// Path-traced tier as a staged wavefront (the schedule MJPBR_SCHEDULE_WAVEFRONT of the path tier):
// the bounce loop of mujoco_warp_pbr/_src/pathtrace.py:200-421 over every path of a chunk of
// worlds at once, one kernel per stage and compacted path queues between the bounces:
//
//   geometry depth / segmentation of cameras without RGB (one ray per pixel)
//   per bounce, over the queue of live paths:
//     extend   closest hit of every path (scenes of few geoms by the warp-wide scan, scan.cuh; meshes and
//              larger scenes with lanes refilled from the queue: refill.cuh), hits and misses queued apart;
//              depth / segmentation from sample 0's first hit; the first bounce's extend starts
//              the paths itself, one per (pixel, sample) of the RGB cameras (pt_bounce.cuh
//              start_sample), and writes each path record once, after its hit
//     shade    the bounce after the hit (PtCore's phases, taken by a CTA's warps together): emission, mirror lobe, next-event
//              estimation recorded per path (each light's unshadowed contribution, the environment
//              sample's term) with each shadow ray appended to the shadow queue as it is recorded
//              (one atomic per group of converged lanes), the BSDF sample and Russian roulette;
//              the paths that continue are appended to the next queue (one atomic per CTA)
//     shadow   any hit of every queued shadow ray (persistent, lanes refilled)
//   (the recorded terms of the unoccluded rays are added to the path's radiance, in light order,
//   by the next bounce's extend stage, or by the resolve stage for a path that ended: the
//   persistent kernel's exact additions in its order)
//   resolve  one thread per pixel: its samples summed in sample order, tone map / denoiser inputs
//
// Each stage runs one kind of work on a full set of lanes and has its own register budget; the
// image is the persistent kernel's, bit for bit (the random numbers are counter-based per sample
// and bounce, so the order in which paths run does not matter).
//
// Scratch (MjpbrScene.wave_scratch), per path of a chunk: the path record (80 B every bounce moves,
// 48 B of first-surface features), its hit (32 B), its next-event record (16 B + 16 B per slot: each
// light, the headlight, the environment), one visibility byte per slot, two queue entries and up to
// one shadow entry (32 B) per slot.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "abi_internal.h"
#include <cooperative_groups.h>

// The shade stage is the only kernel here that calls these, each from few places: inline, so that lights,
// hits and surfaces pass through registers.
#define MJPBR_PT_INLINE
#define MJPBR_LIGHT_QUERY __forceinline__
#ifndef MJPBR_SURFACE_CALL
#define MJPBR_SURFACE_CALL __forceinline__
#endif
#include "pt_bounce.cuh"
#include "refill.cuh"
#include "scan.cuh"

namespace mjpbr {
namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;
// Resident CTAs per SM the shade stage's register allocation targets.
#ifndef MJPBR_PTW_SHADE_CTAS
#define MJPBR_PTW_SHADE_CTAS 3
#endif
#ifndef MJPBR_PTW_TEX_CTAS
#define MJPBR_PTW_TEX_CTAS 3
#endif

// Resident CTAs per SM of the scanned trace stages (scan.cuh): they wait for path records and world blocks
// more than they need registers. 1024 x 128 x 128 paths at three, four and five: extend 3.08, 2.67, 2.64 ms;
// two 256 x 256 cameras of 128 worlds 2.60, 2.30, 2.25 and, the first extend, 2.11, 2.03, 2.09.
constexpr int kScanCtas = 4;

// A path between stages: 80 bytes every bounce reads and writes, and the first surface's denoiser
// features (48 bytes), written by the bounces of a camera ray. Each 16-byte field is an array of its own
// over the paths of the chunk, so that a warp's lanes, on neighbouring paths, move whole lines.
enum PathField : int32_t {
  kPathOrigin,      // origin, max_dist
  kPathDir,         // direction, pdf_prev
  kPathBeta,        // throughput, dcam_z
  kPathRadiance,    // radiance, first-hit depth (sample 0)
  kPathMeta,        // (int bits) depth, passes, sample, flags (1 camera ray, 2 delta)
  kPathFeature0,    // first surface: albedo xyz, normal x
  kPathFeature1,    // normal yz, emission xy
  kPathFeature2,    // emission z, base colour xyz
  kPathFields
};

// A path's hit: two such fields (distance, ref, face, u; v, normal), ref -1 a miss, else
// slot | (mesh + 1) << 16.
constexpr int32_t kHitFields = 2;

// A shadow ray: two fields over the queue (origin, ray length; direction, target (int bits)), the
// target slot * path_cap + path.
constexpr int32_t kShadowFields = 2;

// Next-event state of a path's slot, a byte: what its term does to the radiance. kNeeActive is set in the
// last slot (the environment's) while the path has terms to be added.
constexpr uint8_t kNeeSkip = 0;      // inactive light: nothing added
constexpr uint8_t kNeeZero = 1;      // the light does not reach the point: zero added
constexpr uint8_t kNeeAdd = 2;       // unshadowed contribution: added
constexpr uint8_t kNeePending = 3;   // added if its shadow ray is unoccluded: zero added
constexpr uint8_t kNeeVisible = 4;   // kNeePending whose ray was unoccluded: added
constexpr uint8_t kNeeActive = 0x80;

struct PtWaveMap {
  int32_t w0, nw;          // worlds of this chunk
  int32_t nsample;         // samples per pixel
  int32_t pixels;          // RGB pixels per world
  int32_t npath;           // paths of this chunk: nw * pixels * nsample
  int32_t nslot;           // next-event slots: nlight, the headlight, the environment
  int32_t pix_base[MJPBR_MAX_RENDER];  // first RGB pixel of each camera within a world (-1: no RGB)
  int32_t geo_base[MJPBR_MAX_RENDER + 1];  // pixels of the cameras without RGB (prefix sums)
  float4* path;            // (kPathFields, path_cap)
  float4* hit;             // (kHitFields, path_cap)
  float4* nee;             // (1 + nslot, path_cap): the bounce's throughput, then each slot's term
  uint8_t* state;          // (nslot, path_cap)
  int32_t* live;           // paths to extend
  int32_t* reached;        // extended paths: those that hit from the front, those that missed from the end (path_cap)
  float4* shadow;          // (kShadowFields, shadow_cap)
  // [0], [1] length of `live` in even and odd bounces, [2] shadow entries, [3] hits and [8] misses in
  // `reached`; 64-bit fetch counters of extend [4..5] and shadow [6..7]. Zero before the first bounce; then each
  // stage clears what the stages before it are done with and the ones after it count again.
  int32_t* counters;
  int64_t path_cap, shadow_cap;
};

MJ_DEV Stack wave_stack(const MjpbrScene& s, float* base) {
  return shared_stack(base, kThreads, stack_entries(s.settings.stack_depth));
}

// World, camera, pixel id and sample of a chunk-local path index (paths: world-major, then RGB
// pixels in camera order, then samples).
MJ_DEV void path_pixel(const MjpbrScene& s, const PtWaveMap& wm, int32_t path, int32_t* w, Pixel* p, int32_t* sample) {
  const int32_t pix_all = path / wm.nsample;
  *sample = path - pix_all * wm.nsample;
  const int32_t wl = pix_all / wm.pixels;
  const int32_t pix = pix_all - wl * wm.pixels;
  int32_t cam = 0;
  for (int32_t k = 0; k < s.nrender; ++k) {
    if (wm.pix_base[k] >= 0 && wm.pix_base[k] <= pix) cam = k;
  }
  *w = wm.w0 + wl;
  p->cam = cam;
  p->width = s.cam_res[cam][0];
  p->height = s.cam_res[cam][1];
  p->pixelid = pix - wm.pix_base[cam];
  p->px = p->pixelid % p->width;
  p->py = p->pixelid / p->width;
}

MJ_DEV const float* world_block(const MjpbrScene& s, int32_t w) { return s.world_blocks + (int64_t)w * s.world_block_floats; }

MJ_DEV uint32_t pixel_seed_of(const MjpbrScene& s, uint32_t seed, int32_t w, const Pixel& p) {
  return seed + (uint32_t)w * (uint32_t)s.total_rays + (uint32_t)(s.ray_adr[p.cam] + p.pixelid);
}

MJ_DEV float4& path_field(const PtWaveMap& wm, PathField f, int32_t path) { return wm.path[f * wm.path_cap + path]; }

MJ_DEV void store_path_radiance(const PtWaveMap& wm, int32_t path, const PathState& ps, float first_depth) {
  path_field(wm, kPathRadiance, path) = make_float4(ps.radiance.x, ps.radiance.y, ps.radiance.z, first_depth);
}

// What the next bounce needs besides the radiance.
MJ_DEV void store_path_live(const PtWaveMap& wm, int32_t path, const PathState& ps) {
  path_field(wm, kPathOrigin, path) = make_float4(ps.o.x, ps.o.y, ps.o.z, ps.max_dist);
  path_field(wm, kPathDir, path) = make_float4(ps.d.x, ps.d.y, ps.d.z, ps.pdf_prev);
  path_field(wm, kPathBeta, path) = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, ps.dcam_z);
  path_field(wm, kPathMeta, path) = make_float4(__int_as_float(ps.depth), __int_as_float(ps.passes), __int_as_float(ps.sample),
                                                __int_as_float((ps.camera_ray ? 1 : 0) | (ps.delta ? 2 : 0)));
}

MJ_DEV void store_path_features(const PtWaveMap& wm, int32_t path, const PathState& ps) {
  path_field(wm, kPathFeature0, path) = make_float4(ps.albedo.x, ps.albedo.y, ps.albedo.z, ps.normal.x);
  path_field(wm, kPathFeature1, path) = make_float4(ps.normal.y, ps.normal.z, ps.emission.x, ps.emission.y);
  path_field(wm, kPathFeature2, path) = make_float4(ps.emission.z, ps.base_color.x, ps.base_color.y, ps.base_color.z);
}

// The state of a path before a bounce. Its features are start_sample's until the bounce that ends its
// camera ray sets them, so none are loaded.
MJ_DEV PathState load_path(const PtWaveMap& wm, int32_t path, float* first_depth) {
  PathState ps;
  const float4 o = path_field(wm, kPathOrigin, path), d = path_field(wm, kPathDir, path), beta = path_field(wm, kPathBeta, path);
  const float4 rad = path_field(wm, kPathRadiance, path), meta = path_field(wm, kPathMeta, path);
  ps.o = V3{o.x, o.y, o.z};
  ps.max_dist = o.w;
  ps.d = V3{d.x, d.y, d.z};
  ps.pdf_prev = d.w;
  ps.beta = V3{beta.x, beta.y, beta.z};
  ps.dcam_z = beta.w;
  ps.radiance = V3{rad.x, rad.y, rad.z};
  *first_depth = rad.w;
  ps.depth = __float_as_int(meta.x);
  ps.passes = __float_as_int(meta.y);
  ps.sample = __float_as_int(meta.z);
  const int32_t flags = __float_as_int(meta.w);
  ps.camera_ray = (flags & 1) != 0;
  ps.delta = (flags & 2) != 0;
  start_features(ps);
  return ps;
}

MJ_DEV void store_hit(const PtWaveMap& wm, int32_t path, const Hit& h) {
  const int32_t ref = h.geom == -1 ? -1 : (h.slot | ((h.mesh + 1) << 16));
  wm.hit[path] = make_float4(h.dist, __int_as_float(ref), __int_as_float(h.face), h.u);
  wm.hit[wm.path_cap + path] = make_float4(h.v, h.normal.x, h.normal.y, h.normal.z);
}

MJ_DEV Hit load_hit(const PtWaveMap& wm, int32_t path, const float* blk, const BlockLayout& L) {
  const float4 a = wm.hit[path];
  const int32_t ref = __float_as_int(a.y);
  Hit h;
  h.dist = a.x;
  if (ref == -1) {
    h.geom = h.slot = h.mesh = h.face = -1;
    h.u = h.v = 0.0f;
    h.normal = v3(0.0f);
    return h;
  }
  const float4 b = wm.hit[wm.path_cap + path];
  h.slot = ref & 0xffff;
  h.mesh = (ref >> 16) - 1;
  h.geom = __float_as_int(blk[L.geom_off + h.slot * kGeomFloats + 16]);
  h.face = __float_as_int(a.z);
  h.u = a.w;
  h.v = b.x;
  h.normal = V3{b.y, b.z, b.w};
  return h;
}

// Appends one entry per thread with `want` as one contiguous run per CTA (one atomic per CTA;
// warps in order, lanes in order). Every thread of the CTA must make the call; `scan` holds
// kThreads / 32 + 1 ints of shared memory. Returns the thread's position or -1.
MJ_DEV int64_t cta_append(bool want, int32_t* counter, int64_t cap, int32_t* scan, int32_t* err) {
  const unsigned full = 0xffffffffu;
  const unsigned m = __ballot_sync(full, want);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = kThreads / 32;
  if (lane == 0) scan[warp] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t total = 0;
    for (int k = 0; k < kWarps; ++k) {
      const int32_t c = scan[k];
      scan[k] = total;
      total += c;
    }
    scan[kWarps] = total > 0 ? atomicAdd(counter, total) : 0;
  }
  __syncthreads();
  const int64_t base = (int64_t)scan[kWarps] + scan[warp];
  __syncthreads();
  if (!want) return -1;
  const int64_t pos = base + __popc(m & ((1u << lane) - 1u));
  if (pos >= cap) {
    *err |= kErrWorkQueue;
    return -1;
  }
  return pos;
}

// Next-event estimation of the wavefront: each slot's term is recorded in the path's record and
// its shadow ray appended to the shadow queue at once (one atomic per group of converged lanes);
// the shadow stage traces the rays and the next extend (or resolve) adds the terms.
struct RecordedNee {
  int32_t path;
  V3 origin;
  const PtWaveMap* wm;
  int32_t* err;
  MJ_DEV uint8_t& state(int32_t slot) const { return wm->state[slot * wm->path_cap + path]; }
  MJ_DEV void begin(const PathState&, V3 o) {
    origin = o;
    for (int32_t k = 0; k < wm->nslot - 1; ++k) state(k) = kNeeSkip;
  }
  MJ_DEV void shadow_ray(int32_t slot, V3 dir, float len) {
    cg::coalesced_group g = cg::coalesced_threads();
    int32_t base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(wm->counters + 2, (int32_t)g.size());
    const int64_t pos = (int64_t)g.shfl(base, 0) + g.thread_rank();
    if (pos >= wm->shadow_cap) {
      *err |= kErrWorkQueue;
      return;
    }
    wm->shadow[pos] = make_float4(origin.x, origin.y, origin.z, len);
    wm->shadow[wm->shadow_cap + pos] = make_float4(dir.x, dir.y, dir.z, __int_as_float((int32_t)(slot * wm->path_cap + path)));
  }
  MJ_DEV void none(int32_t slot) { state(slot) = kNeeZero; }
  template <class F>
  MJ_DEV void light(RtCtx&, int32_t slot, bool shadowed, V3, V3 dir, float max_t, F contribution) {
    const V3 c = contribution();
    wm->nee[(1 + slot) * wm->path_cap + path] = make_float4(c.x, c.y, c.z, 0.0f);
    state(slot) = shadowed ? kNeePending : kNeeAdd;
    if (shadowed) shadow_ray(slot, dir, max_t);
  }
  MJ_DEV void lights_done(PathState& ps) {
    wm->nee[path] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, 0.0f);
    state(wm->nslot - 1) = kNeeActive;
  }
  template <class F>
  MJ_DEV void env(RtCtx&, PathState&, V3, V3 dir, F term) {
    const int32_t slot = wm->nslot - 1;
    const V3 t = term();
    wm->nee[(1 + slot) * wm->path_cap + path] = make_float4(t.x, t.y, t.z, 0.0f);
    state(slot) = kNeeActive | kNeePending;
    shadow_ray(slot, dir, kUnboundedShadow);
  }
};

// ---------------------------------------------------------------- next-event terms
// Adds a path's recorded next-event terms of its last shaded bounce to its radiance (the light
// terms in light order, times the bounce's throughput, then the environment term), each one only
// if its shadow ray was unoccluded, and marks the record applied. Run by the next bounce's extend
// stage before the path's next hit, and by the resolve stage for the paths that ended: the same
// additions in the same order as the persistent kernel. Returns the path's radiance field.
MJ_DEV float4 apply_nee(const PtWaveMap& wm, int32_t path) {
  float4 rad = path_field(wm, kPathRadiance, path);
  const int32_t nlights = wm.nslot - 1;  // the model's lights and the headlight
  uint8_t& env = wm.state[nlights * wm.path_cap + path];
  const uint8_t env_state = env;
  if (!(env_state & kNeeActive)) return rad;
  V3 direct = v3(0.0f);
  for (int32_t k = 0; k < nlights; ++k) {
    const uint8_t st = wm.state[k * wm.path_cap + path];
    if (st == kNeeSkip) continue;
    V3 c = v3(0.0f);
    if (st == kNeeAdd || st == kNeeVisible) {
      const float4 t = wm.nee[(1 + k) * wm.path_cap + path];
      c = V3{t.x, t.y, t.z};
    }
    direct += c;
  }
  const float4 head = wm.nee[path];
  V3 radiance{rad.x, rad.y, rad.z};
  radiance += cmul(V3{head.x, head.y, head.z}, direct);
  if ((env_state & ~kNeeActive) == kNeeVisible) {
    const float4 e = wm.nee[(1 + nlights) * wm.path_cap + path];
    radiance += V3{e.x, e.y, e.z};
  }
  rad = make_float4(radiance.x, radiance.y, radiance.z, rad.w);
  path_field(wm, kPathRadiance, path) = rad;
  env = 0;
  return rad;
}

// ---------------------------------------------------------------- cameras without RGB
template <bool kMesh>
__global__ void __launch_bounds__(kThreads) ptw_geometry_kernel(const __grid_constant__ MjpbrScene s,
                                                                const __grid_constant__ PtWaveMap wm) {
  extern __shared__ __align__(16) float smem[];
  const Stack st = wave_stack(s, smem);
  const int32_t per_world = wm.geo_base[s.nrender];
  const int32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= per_world * wm.nw) return;
  const int32_t wl = i / per_world, pix = i - wl * per_world;
  int32_t cam = 0;
  while (cam + 1 < s.nrender && pix >= wm.geo_base[cam + 1]) ++cam;
  const int32_t w = wm.w0 + wl;
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  const float* blk = world_block(s, w);
  Pixel p;
  p.cam = cam;
  p.width = s.cam_res[cam][0];
  p.height = s.cam_res[cam][1];
  p.pixelid = pix - wm.geo_base[cam];
  p.px = p.pixelid % p.width;
  p.py = p.pixelid / p.width;
  p.rec = blk + L.cam_off + cam * kCamFloats;
  const M3 R = cam_mat(p.rec);
  const V3 cpos{p.rec[0], p.rec[1], p.rec[2]};
  V3 dcam, ocam;
  float max_dist, depth_z;
  primary_ray(s, p, kSubpixel, kSubpixel / 2, kSubpixel / 2, &dcam, &ocam, &max_dist, &depth_z);
  int32_t err = 0;
  const Hit hit = trace_ray<kMesh>(s, st, blk, L, Ray{cpos + mul(R, ocam), mul(R, dcam)}, max_dist, s.settings.cull_backfaces != 0,
                                   false, &err);
  write_geometry(s, w, p, hit, depth_z);
  if (err && s.error_word) atomicOr(s.error_word, err);
}

// ---------------------------------------------------------------- extend
// Steps a lane of the traversal stages runs between refills of the warp's idle lanes.
#ifndef MJPBR_PTW_REFILL_STEPS
#define MJPBR_PTW_REFILL_STEPS 32
#endif

// Closest hits of `items` rays: start(item, &max_dist) gives a ray (and sets the lane's world block
// blk), finish(hit) stores its hit. kTogether: where lanes stride over the items, a CTA's warps start each
// round together, so that they fetch the code once: for the first bounce, whose starts and writes are much
// code and little waiting (1024 x 128 x 128 paths 2.33 -> 2.16 ms, two 256 x 256 cameras of 128 worlds 2.05 ->
// 1.93); later bounces wait for memory at different times and lose by it (2.73 -> 2.79, 2.36 -> 2.47).
template <bool kMesh, bool kScan, bool kTogether, class Start, class Finish>
MJ_DEV void closest_queue(const MjpbrScene& s, const Stack& st, const BlockLayout& L, bool cull, int64_t items,
                          unsigned long long* fetched, const float*& blk, const Start& start, const Finish& finish, int32_t* err) {
  float max_dist;
  if constexpr (kScan && !kMesh) {
    for (int64_t first = (int64_t)blockIdx.x * kThreads; first < items; first += (int64_t)gridDim.x * kThreads) {
      const int64_t i = first + threadIdx.x;
      if (i < items) {
        const Ray r = start(i, &max_dist);
        finish(scan_trace<false>(NodeBoxes{blk, &L}, s, st, blk, L, r, max_dist, cull, err));
      }
      if (kTogether) __syncthreads();
    }
  } else if constexpr (kScan) {
    ClosestWalk q;
    auto done = [&](ClosestWalk& qq) {
      if (qq.tie) qq.h = trace_ray<true>(s, st, blk, L, qq.m.r, max_dist, cull, false, err);
      finish(qq.h);
    };
    refill_loop<MJPBR_PTW_REFILL_STEPS, kFetchIdle>(
        items, fetched, q,
        [&](int64_t item, ClosestWalk& qq) {
          qq.m.r = start(item, &max_dist);
          qq.m.meshes = scan_closest<true>(qq.h, qq.tie, NodeBoxes{blk, &L}, blk, L, qq.m.r, max_dist, cull);
          qq.m.slot = -1;
          qq.m.sp = 0;
          qq.m.code = -1;
          if (qq.m.meshes) return true;
          done(qq);
          return false;
        },
        [&](ClosestWalk& qq) { return walk_closest_step(qq, s, st, blk, L, cull, err); }, [&](ClosestWalk& qq, int32_t) { done(qq); }, err);
  } else {
    ClosestQuery q;
    refill_loop<MJPBR_PTW_REFILL_STEPS>(
        items, fetched, q,
        [&](int64_t item, ClosestQuery& qq) {
          const Ray r = start(item, &max_dist);
          closest_begin(qq, st, r, max_dist, err);
          return true;
        },
        [&](ClosestQuery& qq) { return closest_step<kMesh>(qq, s, st, blk, L, cull, err); },
        [&](ClosestQuery& qq, int32_t) { finish(qq.h); }, err);
  }
}

// Closest hit of every live path; the pending next-event terms of the path's last bounce are added
// first. Scenes of up to kScanGeoms geoms are scanned (scan.cuh): without meshes the lanes stride over
// the queue, with them the meshes are traced resumably, lanes refilled from the queue (refill.cuh);
// larger scenes walk the scene BVH resumably.
template <bool kMesh, bool kScan>
__global__ void __launch_bounds__(kThreads, kScan ? kScanCtas : 3) ptw_extend_kernel(const __grid_constant__ MjpbrScene s,
                                                                 const __grid_constant__ PtWaveMap wm, int32_t parity) {
  extern __shared__ __align__(16) float smem[];
  const Stack st = wave_stack(s, smem);
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  const bool cull = s.settings.cull_backfaces != 0;
  const int64_t items = min((int64_t)wm.counters[parity], wm.path_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    wm.counters[parity ^ 1] = 0;
    wm.counters[2] = wm.counters[6] = wm.counters[7] = 0;
  }
  unsigned long long* fetched = reinterpret_cast<unsigned long long*>(wm.counters + 4);
  int32_t err = 0;
  const float* blk = nullptr;
  int32_t path = -1;
  auto start = [&](int64_t item, float* max_dist) {
    path = wm.live[item];
    apply_nee(wm, path);
    const float4 o = path_field(wm, kPathOrigin, path), d = path_field(wm, kPathDir, path);
    blk = world_block(s, wm.w0 + (path / wm.nsample) / wm.pixels);
    *max_dist = o.w;
    return Ray{V3{o.x, o.y, o.z}, V3{d.x, d.y, d.z}};
  };
  auto finish = [&](const Hit& hit) {
    // the first hits, and the geometry they write, are ptw_first_extend_kernel's
    store_hit(wm, path, hit);
    // hits and misses apart: half the secondary rays miss, which a shading warp would wait out
    const bool miss = hit.geom == -1;
    cg::coalesced_group g = cg::coalesced_threads();
    const unsigned misses = g.ballot(miss);
    const int32_t nmiss = __popc(misses), rank = __popc(misses & ((1u << g.thread_rank()) - 1u));
    int32_t at_hit = 0, at_miss = 0;
    if (g.thread_rank() == 0) {
      if (nmiss < (int32_t)g.size()) at_hit = atomicAdd(wm.counters + 3, (int32_t)g.size() - nmiss);
      if (nmiss) at_miss = atomicAdd(wm.counters + 8, nmiss);
    }
    at_hit = g.shfl(at_hit, 0) + (int32_t)g.thread_rank() - rank;
    at_miss = g.shfl(at_miss, 0) + rank;
    wm.reached[miss ? wm.path_cap - 1 - at_miss : at_hit] = path;
  };
  closest_queue<kMesh, kScan, false>(s, st, L, cull, items, fetched, blk, start, finish, &err);
  if (err && s.error_word) atomicOr(s.error_word, err);
}

// The first bounce's extend, with the start folded in: each path's camera ray is generated where
// it is traced (start_sample, pt_bounce.cuh) and the path record written once, after the hit. The shade
// stage takes the paths in their own order: neighbouring camera rays mostly hit or miss together.
template <bool kMesh, bool kScan>
__global__ void __launch_bounds__(kThreads, kScan ? kScanCtas : 3) ptw_first_extend_kernel(const __grid_constant__ MjpbrScene s, uint32_t seed,
                                                                       const __grid_constant__ PtWaveMap wm) {
  extern __shared__ __align__(16) float smem[];
  const Stack st = wave_stack(s, smem);
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  const bool cull = s.settings.cull_backfaces != 0;
  unsigned long long* fetched = reinterpret_cast<unsigned long long*>(wm.counters + 4);
  int32_t err = 0;
  const float* blk = nullptr;
  int32_t path = -1;
  // the path's start state (the same for the ray and for the record stored after the hit)
  auto start_state = [&](int32_t i, PathState& ps, Pixel& p, int32_t& w, int32_t& sample) {
    path_pixel(s, wm, i, &w, &p, &sample);
    p.rec = world_block(s, w) + L.cam_off + p.cam * kCamFloats;
    const M3 R = cam_mat(p.rec);
    const V3 cpos{p.rec[0], p.rec[1], p.rec[2]};
    start_sample(ps, s, p, pixel_seed_of(s, seed, w, p), R, cpos, sample);
  };
  auto start = [&](int64_t item, float* max_dist) {
    path = (int32_t)item;
    PathState ps;
    Pixel p;
    int32_t w, sample;
    start_state(path, ps, p, w, sample);
    blk = world_block(s, w);
    *max_dist = ps.max_dist;
    return Ray{ps.o, ps.d};
  };
  auto finish = [&](const Hit& hit) {
    store_hit(wm, path, hit);
    PathState ps;
    Pixel p;
    int32_t w, sample;
    start_state(path, ps, p, w, sample);
    float first_depth = 0.0f;
    if (sample == 0) {
      write_geometry(s, w, p, hit, ps.dcam_z);
      if (hit.geom != -1) first_depth = hit.dist * -ps.dcam_z;
    }
    store_path_radiance(wm, path, ps, first_depth);
    store_path_live(wm, path, ps);
  };
  closest_queue<kMesh, kScan, true>(s, st, L, cull, wm.npath, fetched, blk, start, finish, &err);
  if (err && s.error_word) atomicOr(s.error_word, err);
}

// ---------------------------------------------------------------- shade
template <bool kMesh, bool kTex>
__global__ void __launch_bounds__(kThreads, kTex ? MJPBR_PTW_TEX_CTAS : MJPBR_PTW_SHADE_CTAS) ptw_shade_kernel(const __grid_constant__ MjpbrScene s, uint32_t seed,
                                                                const __grid_constant__ PtWaveMap wm, int32_t parity, bool first) {
  __shared__ int32_t scan[kThreads / 32 + 1];
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  // the first bounce's paths in order, or the reached ones: the hits, then the misses
  const int32_t hits = wm.counters[3];
  const int32_t count = first ? wm.npath : (int32_t)min((int64_t)hits + wm.counters[8], wm.path_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) wm.counters[4] = wm.counters[5] = 0;
  const int32_t stride = gridDim.x * kThreads;
  const int32_t rounds = (count + stride - 1) / stride;
  int32_t err = 0;
  for (int32_t round = 0; round < rounds; ++round) {
    const int32_t i = round * stride + blockIdx.x * kThreads + threadIdx.x;
    const bool active = i < count;
    int32_t path = -1;
    bool features = false;
    using Core = PtCore<kMesh, kTex>;
    typename Core::Status status = Core::kEnded;
    typename Core::Vertex x;
    RtCtx c;
    PathState ps;
    float first_depth = 0.0f;
    uint32_t pseed = 0;
    V3 head_dir = v3(0.0f);
    if (active) {
      path = first ? i : wm.reached[i < hits ? i : (int32_t)wm.path_cap - 1 - (i - hits)];
      int32_t w, sample;
      Pixel p;
      path_pixel(s, wm, path, &w, &p, &sample);
      const float* blk = world_block(s, w);
      init_ctx(c, s, blk, L, w, kTex);
      p.rec = blk + L.cam_off + p.cam * kCamFloats;
      const M3 R = cam_mat(p.rec);
      head_dir = -V3{R.m[2], R.m[5], R.m[8]};
      pseed = pixel_seed_of(s, seed, w, p);
      ps = load_path(wm, path, &first_depth);
      // only a camera ray's bounce can set the first surface's features
      features = ps.camera_ray;
      const Hit hit = load_hit(wm, path, blk, L);
      wm.state[(wm.nslot - 1) * wm.path_cap + path] = 0;
      status = Core::reach(c, ps, hit, pseed, x);
      if (features) store_path_features(wm, path, ps);
    }
    // The CTA's warps take each phase together: the stage's code is several times the instruction cache (on
    // 1024 x 128x128 and, with environments, 128 x 2 x 256x256 paths: 8.7 -> 6.5 and 14.5 -> 10.1 ms with the
    // queues by hit and miss; 11.8 and 26.4 with no barrier at all, paths appended by warps).
    RecordedNee nee{path, v3(0.0f), &wm, &err};
    __syncthreads();
    if (status == Core::kShade) Core::lights(c, nee, ps, x, pseed, head_dir);
    __syncthreads();
    if (kTex) {
      if (status == Core::kShade) Core::env_light(c, nee, ps, x, pseed);
      __syncthreads();
    }
    bool live = status == Core::kLive;
    if (status == Core::kShade) live = !Core::proceed(c, ps, x, pseed);
    if (active) {
      store_path_radiance(wm, path, ps, first_depth);
      if (live) store_path_live(wm, path, ps);
      err |= c.err;
    }
    // the paths that continue
    const int64_t pos = cta_append(live, wm.counters + (parity ^ 1), wm.path_cap, scan, &err);
    if (pos >= 0) wm.live[pos] = path;
  }
  if (err && s.error_word) atomicOr(s.error_word, err);
}

// ---------------------------------------------------------------- shadow rays
// Any hit of every recorded shadow ray: scanned (scan.cuh; without meshes the lanes stride over the
// queue) or, past kScanGeoms geoms, by the scene BVH, lanes refilled from the queue (refill.cuh).
template <bool kMesh, bool kScan>
__global__ void __launch_bounds__(kThreads, kScan ? kScanCtas : 3) ptw_shadow_kernel(const __grid_constant__ MjpbrScene s,
                                                                 const __grid_constant__ PtWaveMap wm) {
  extern __shared__ __align__(16) float smem[];
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  const bool cull = s.settings.cull_backfaces != 0;
  const int64_t items = min((int64_t)wm.counters[2], wm.shadow_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) wm.counters[3] = wm.counters[8] = 0;
  unsigned long long* fetched = reinterpret_cast<unsigned long long*>(wm.counters + 6);
  int32_t err = 0;
  const float* blk = nullptr;
  int32_t target = -1;
  auto start = [&](int64_t item, float* max_dist) {
    const float4 o = wm.shadow[item], d = wm.shadow[wm.shadow_cap + item];
    target = __float_as_int(d.w);
    const int32_t path = target % (int32_t)wm.path_cap;
    blk = world_block(s, wm.w0 + (path / wm.nsample) / wm.pixels);
    *max_dist = o.w;
    return Ray{V3{o.x, o.y, o.z}, V3{d.x, d.y, d.z}};
  };
  auto visible = [&] { wm.state[target] += kNeeVisible - kNeePending; };  // the environment's keeps kNeeActive
  float max_dist;
  if constexpr (kScan && !kMesh) {
    uint32_t meshes;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < items; i += (int64_t)gridDim.x * kThreads) {
      const Ray r = start(i, &max_dist);
      if (!scan_any<false>(blk, L, r, max_dist, cull, &meshes)) visible();
    }
  } else if constexpr (kScan) {
    const Stack st = wave_stack(s, smem);
    MeshWalk q;
    refill_loop<MJPBR_PTW_REFILL_STEPS, kFetchIdle>(
        items, fetched, q,
        [&](int64_t item, MeshWalk& qq) {
          qq.r = start(item, &qq.cut);
          qq.sp = 0;
          qq.code = -1;
          const bool hit = scan_any<true>(blk, L, qq.r, qq.cut, cull, &qq.meshes);
          if (!hit && qq.meshes) return true;
          if (!hit) visible();
          return false;
        },
        [&](MeshWalk& qq) { return walk_any_step(qq, s, st, blk, L, &err); },
        [&](MeshWalk&, int32_t res) {
          if (res == kAnyClear) visible();
        },
        &err);
  } else {
    const Stack st = wave_stack(s, smem);
    AnyQuery q;
    refill_loop<MJPBR_PTW_REFILL_STEPS>(
        items, fetched, q,
        [&](int64_t item, AnyQuery& qq) {
          const Ray r = start(item, &max_dist);
          any_begin(qq, st, r, max_dist, &err);
          return true;
        },
        [&](AnyQuery& qq) { return any_step<kMesh>(qq, s, st, blk, L, cull, &err); },
        [&](AnyQuery&, int32_t res) {
          if (res == kAnyClear) visible();
        },
        &err);
  }
  if (err && s.error_word) atomicOr(s.error_word, err);
}

// ---------------------------------------------------------------- pixels
template <bool kTex>
__global__ void __launch_bounds__(kThreads) ptw_resolve_kernel(const __grid_constant__ MjpbrScene s, const __grid_constant__ PtWaveMap wm) {
  const int32_t pix_all = blockIdx.x * kThreads + threadIdx.x;
  if (pix_all >= wm.nw * wm.pixels) return;
  int32_t w, sample;
  Pixel p;
  path_pixel(s, wm, pix_all * wm.nsample, &w, &p, &sample);
  const BlockLayout L = block_layout(s.nbvh_geom, s.nnode, s.nlight, s.nrender);
  RtCtx c;
  init_ctx(c, s, world_block(s, w), L, w, kTex);
  PixelAcc acc;
  clear_pixel(acc);
  for (int32_t k = 0; k < wm.nsample; ++k) {
    const int32_t path = pix_all * wm.nsample + k;
    const float4 rad = apply_nee(wm, path);
    const float4 f0 = path_field(wm, kPathFeature0, path), f1 = path_field(wm, kPathFeature1, path), f2 = path_field(wm, kPathFeature2, path);
    PathState ps;
    ps.radiance = V3{rad.x, rad.y, rad.z};
    ps.sample = k;
    ps.albedo = V3{f0.x, f0.y, f0.z};
    ps.normal = V3{f0.w, f1.x, f1.y};
    ps.emission = V3{f1.z, f1.w, f2.x};
    ps.base_color = V3{f2.y, f2.z, f2.w};
    if (k == 0) acc.first_depth = rad.w;
    add_sample(acc, ps, s.settings.denoise != 0, c.exposure);
  }
  write_pixel(s, c, (int64_t)w * s.rgb_stride + s.rgb_adr[p.cam] + p.pixelid, acc, wm.nsample);
}

// ---------------------------------------------------------------- host side

int64_t align256(int64_t b) { return (b + 255) & ~int64_t(255); }

int32_t slots_of(const MjpbrScene& s) { return std::max(s.nlight, 0) + 2; }

void rgb_pixels(const MjpbrScene& s, int32_t* pix_base, int32_t* geo_base, int64_t* pixels) {
  int64_t rgb = 0, geo = 0;
  geo_base[0] = 0;
  for (int32_t c = 0; c < s.nrender; ++c) {
    const int64_t npix = (int64_t)s.cam_res[c][0] * s.cam_res[c][1];
    pix_base[c] = s.render_rgb[c] ? (int32_t)rgb : -1;
    if (s.render_rgb[c]) rgb += npix;
    if (!s.render_rgb[c] && (s.render_depth[c] || s.render_seg[c])) geo += npix;
    geo_base[c + 1] = (int32_t)geo;
  }
  for (int32_t c = s.nrender; c < MJPBR_MAX_RENDER; ++c) pix_base[c] = -1;
  *pixels = rgb;
}

int64_t layout(PtWaveMap* wm, char* base, int64_t npath, int32_t nslot) {
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    char* p = base + off;
    off += align256(bytes);
    return p;
  };
  char* counters = take(256);
  char* path = take(npath * kPathFields * 16);
  char* hit = take(npath * kHitFields * 16);
  char* nee = take(npath * (1 + (int64_t)nslot) * 16);
  char* state = take(npath * nslot);
  char* q0 = take(npath * 4);
  char* q1 = take(npath * 4);
  char* shadow = take(npath * nslot * kShadowFields * 16);
  if (wm) {
    wm->counters = reinterpret_cast<int32_t*>(counters);
    wm->path = reinterpret_cast<float4*>(path);
    wm->hit = reinterpret_cast<float4*>(hit);
    wm->nee = reinterpret_cast<float4*>(nee);
    wm->state = reinterpret_cast<uint8_t*>(state);
    wm->live = reinterpret_cast<int32_t*>(q0);
    wm->reached = reinterpret_cast<int32_t*>(q1);
    wm->shadow = reinterpret_cast<float4*>(shadow);
    wm->path_cap = npath;
    wm->shadow_cap = npath * nslot;
  }
  return off;
}

template <class K>
int resident_ctas(K kern, size_t smem) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, kThreads, smem) != cudaSuccess || n < 1) n = 1;
  return n;
}

template <class K>
int set_smem(K kern, size_t smem, const char* what) {
  return ensure_smem(reinterpret_cast<const void*>(kern), smem, what);
}

template <bool kMesh, bool kTex, bool kScan>
int launch_pt_wave(const MjpbrScene& s, uint32_t seed, cudaStream_t stream, int32_t chunk, int64_t pixels) {
  const size_t stack = (size_t)kThreads * stack_entries(s.settings.stack_depth) * 8;
  auto k_geometry = ptw_geometry_kernel<kMesh>;
  auto k_extend = ptw_extend_kernel<kMesh, kScan>;
  auto k_first = ptw_first_extend_kernel<kMesh, kScan>;
  auto k_shade = ptw_shade_kernel<kMesh, kTex>;
  auto k_shadow = ptw_shadow_kernel<kMesh, kScan>;
  auto k_resolve = ptw_resolve_kernel<kTex>;
  int rc = set_smem(k_geometry, stack, "path wavefront geometry");
  if (!rc) rc = set_smem(k_extend, stack, "path wavefront extend");
  if (!rc) rc = set_smem(k_first, stack, "path wavefront first extend");
  if (!rc) rc = set_smem(k_shadow, stack, "path wavefront shadow");
  if (rc) return rc;
  const int sms = device_sm_count();
  const int g_extend = sms * resident_ctas(k_extend, stack);
  const int g_first = sms * resident_ctas(k_first, stack);
  const int g_shade = sms * resident_ctas(k_shade, 0);
  const int g_shadow = sms * resident_ctas(k_shadow, stack);
  PtWaveMap wm;
  wm.nsample = s.settings.path_samples;
  wm.pixels = (int32_t)pixels;
  wm.nslot = slots_of(s);
  rgb_pixels(s, wm.pix_base, wm.geo_base, &pixels);
  layout(&wm, static_cast<char*>(s.wave_scratch), (int64_t)chunk * pixels * wm.nsample, wm.nslot);
  const int32_t geo_pixels = wm.geo_base[s.nrender];
  const int32_t iterations = s.settings.max_depth + 1 + (s.settings.has_transparency ? 4 * s.settings.max_layers : 0);
  for (int32_t w0 = 0; w0 < s.nworld; w0 += chunk) {
    wm.w0 = w0;
    wm.nw = std::min(chunk, s.nworld - w0);
    wm.npath = (int32_t)((int64_t)wm.nw * pixels * wm.nsample);
    if (geo_pixels > 0) {
      const int64_t n = (int64_t)geo_pixels * wm.nw;
      k_geometry<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, stack, stream>>>(s, wm);
      if ((rc = check_launch("ptw_geometry_kernel"))) return rc;
    }
    if (wm.npath == 0) continue;
    cudaError_t ez = cudaMemsetAsync(wm.counters, 0, 9 * sizeof(int32_t), stream);
    if (ez != cudaSuccess) return set_error(MJPBR_ERR_CUDA, "path wavefront counters: %s", cudaGetErrorString(ez));
    for (int32_t it = 0; it < iterations; ++it) {
      const int32_t parity = it & 1;
      if (it == 0) {
        k_first<<<g_first, kThreads, stack, stream>>>(s, seed, wm);
        if ((rc = check_launch("ptw_first_extend_kernel"))) return rc;
      } else {
        k_extend<<<g_extend, kThreads, stack, stream>>>(s, wm, parity);
        if ((rc = check_launch("ptw_extend_kernel"))) return rc;
      }
      k_shade<<<g_shade, kThreads, 0, stream>>>(s, seed, wm, parity, it == 0);
      if ((rc = check_launch("ptw_shade_kernel"))) return rc;
      // every bounce may ask for shadow rays (lights, environment)
      k_shadow<<<g_shadow, kThreads, stack, stream>>>(s, wm);
      if ((rc = check_launch("ptw_shadow_kernel"))) return rc;
    }
    const int64_t npix = (int64_t)wm.nw * pixels;
    k_resolve<<<(unsigned)((npix + kThreads - 1) / kThreads), kThreads, 0, stream>>>(s, wm);
    if ((rc = check_launch("ptw_resolve_kernel"))) return rc;
  }
  return MJPBR_OK;
}

}  // namespace

int64_t pt_wave_scratch_bytes(const MjpbrScene& s, int32_t worlds) {
  int32_t pix_base[MJPBR_MAX_RENDER], geo_base[MJPBR_MAX_RENDER + 1];
  int64_t pixels = 0;
  rgb_pixels(s, pix_base, geo_base, &pixels);
  if (worlds < 0 || s.settings.path_samples < 1) return -1;
  return layout(nullptr, nullptr, (int64_t)worlds * pixels * s.settings.path_samples, slots_of(s));
}

// The path wavefront's records pack geom slots and triangle BVH ids in 16 bits; larger scenes render
// with the persistent path kernel (the same images).
bool pt_wave_supported(const MjpbrScene& s) { return s.nbvh_geom <= 0xffff && s.nmesh + s.nhfield < 0x7fff; }

int render_pt_wave_launch(const MjpbrScene& s, uint32_t seed, cudaStream_t stream) {
  if (!pt_wave_supported(s)) {
    return set_error(MJPBR_ERR_UNSUPPORTED, "the path wavefront packs slots and triangle BVHs in 16 bits; use the grid schedule");
  }
  if (!s.wave_scratch || (reinterpret_cast<uintptr_t>(s.wave_scratch) & 255u)) {
    return set_error(MJPBR_ERR_ARG, "the path wavefront needs wave_scratch (256-byte aligned)");
  }
  int32_t pix_base[MJPBR_MAX_RENDER], geo_base[MJPBR_MAX_RENDER + 1];
  int64_t pixels = 0;
  rgb_pixels(s, pix_base, geo_base, &pixels);
  // worlds per chunk: as many as the scratch holds, with path and shadow-target indices in int32
  int32_t chunk = s.nworld;
  if (pixels > 0) {
    const int64_t per_world = pixels * s.settings.path_samples * slots_of(s);
    chunk = (int32_t)std::min<int64_t>(chunk, INT32_MAX / std::max<int64_t>(per_world, 1));
    if (pt_wave_scratch_bytes(s, chunk) > s.wave_scratch_bytes) {
      int32_t lo = 0, hi = chunk;
      while (lo < hi) {
        const int32_t mid = lo + (hi - lo + 1) / 2;
        if (pt_wave_scratch_bytes(s, mid) <= s.wave_scratch_bytes) {
          lo = mid;
        } else {
          hi = mid - 1;
        }
      }
      chunk = lo;
    }
    if (chunk < 1) {
      return set_error(MJPBR_ERR_ARG, "wave_scratch of %lld bytes holds no world (one needs %lld)", (long long)s.wave_scratch_bytes,
                       (long long)pt_wave_scratch_bytes(s, 1));
    }
  }
  const bool mesh = s.nmesh + s.nhfield > 0 && s.blas_root != nullptr;
  const bool tex = s.settings.textures || s.settings.has_env || s.settings.env_background;
  auto launch = [&](auto m, auto t) {
    constexpr bool kMesh = decltype(m)::value, kTex = decltype(t)::value;
    return s.nbvh_geom <= kScanGeoms ? launch_pt_wave<kMesh, kTex, true>(s, seed, stream, chunk, pixels)
                                     : launch_pt_wave<kMesh, kTex, false>(s, seed, stream, chunk, pixels);
  };
  if (mesh && tex) return launch(std::true_type{}, std::true_type{});
  if (mesh) return launch(std::true_type{}, std::false_type{});
  if (tex) return launch(std::false_type{}, std::true_type{});
  return launch(std::false_type{}, std::false_type{});
}

}  // namespace mjpbr

#ifdef MJPBR_COUNT_OPS
namespace mjpbr {
// Counting build: this unit's copy of the counter array pointer (see opcount.cuh).
int pt_wave_count_set(void* counts) { return cudaMemcpyToSymbol(g_op_counts, &counts, sizeof(counts)) == cudaSuccess ? 0 : 1; }
}  // namespace mjpbr
#endif
