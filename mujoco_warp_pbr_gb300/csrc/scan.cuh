// Ray queries of scenes of at most kScanGeoms geoms per world: instead of walking the scene BVH lane
// by lane, a warp tests the leaf boxes of all geoms in one branch-free loop (a bit mask of the
// geoms a lane's ray can hit), then visits the geoms some lane can hit one after the other, all
// lanes on the same geom: no stack, and one primitive type at a time, where the per-lane traversal
// (trace.cuh) has lanes at different nodes, geoms and types. Mesh geoms are left as a mask; each
// lane traces its own meshes' BVHs afterwards.
//
// The hit is trace_ray's. Which geoms are tested differs only in ones too far to win. The selection
// between hits (tolerance, higher geom id) depends on the order of the tests only when two hits lie
// within a few tolerances of each other: such a ray is marked (`tie`) and traced again by trace_ray,
// in its order. Any-hit queries do not depend on the order.
//
// What bounds these queries is instruction issue: the per-lane traversal runs 16 (camera rays), 13
// (shadow) and 7 (mirror) of 32 lanes; the scan 27-30 without meshes. Camera rays of 1024 mesh worlds
// (128 x 128, 2 x 2 samples) 13.2 -> 8.95 ms, of 300 terrain worlds (96 x 96) 1.34 -> 0.79, the walk's with
// the primitives' earlier tests.
//
// kScanGeoms = 32: one mask word, and the scan is the faster of the two up to there (256 worlds of
// 128 x 128, ms a frame, scan / BVH): primitives 0.71 / 1.62 at 4 geoms, 1.10 / 1.90 at 17, 1.38 / 2.12 at 32;
// with a third of them meshes 2.11 / 2.50, 3.56 / 4.48 and 4.60 / 5.54; path-traced 2.96 / 3.77, 4.83 /
// 5.97 and 6.08 / 6.90, with meshes 7.02 / 8.05, 14.4 / 16.3 and 17.7 / 18.8. The leaf boxes are read from the scene
// BVH's nodes (each child of a node with count 1 is a leaf; hidden geoms have none), whose bounds the leaf's
// ancestors contain, so the boxes that pass are those the traversal reaches.
#pragma once

#include "trace.cuh"

namespace mjpbr {

constexpr int32_t kScanGeoms = 32;

// Distances closer than this may be decided by the order of the tests: twice the selection's
// tolerance, and past the traversal's cut-off.
MJ_DEV float scan_window(float dist) { return 2.5f * kRayTolRel * fmaxf(dist, 1.0f); }

// The box tests are trace_ray's, reciprocals included (make_inv). An approximate reciprocal moves a slab by
// 1e-7 of its distance, which the boxes' padding, 1e-5 of their own coordinates, covers only near them: 5 of
// 204,800 camera rays from 4 km at axis-aligned boxes lost their hit by it. Three divisions a ray cost less
// than 1 % of a frame.

// The geoms a ray may hit before cut, as a mask of slots, from the scene BVH's nodes in a world block.
struct NodeBoxes {
  const float* blk;
  const BlockLayout* L;
  MJ_DEV uint32_t mask(const RayInv& ri, float cut) const {
    uint32_t mask = 0;
    const float4* nd = reinterpret_cast<const float4*>(blk + L->node_off);
#pragma unroll 2
    for (int32_t i = 0; i < L->nnode; ++i, nd += 4) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float4 lo = nd[2 * k], hi = nd[2 * k + 1];
        if (__float_as_int(hi.w) == 1) {
          MJPBR_COUNT(kOpBox);
          if (box_entry(ri, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, cut) >= 0.0f) mask |= 1u << __float_as_int(lo.w);
        }
      }
    }
    return mask;
  }
};

// The same from a CTA's own copy of the leaf boxes by slot, for the kernels that stage one world: no
// inner nodes to pass over. stage_boxes fills it (kScanGeoms x 2 float4, and *valid: the slots that
// have a box) from the staged block; every thread of the CTA calls it, between synchronisations.
struct SlotBoxes {
  const float4* box;
  uint32_t valid;
  MJ_DEV uint32_t mask(const RayInv& ri, float cut) const {
    uint32_t mask = 0;
#pragma unroll 1
    for (uint32_t v = valid; v; v &= v - 1u) {
      const int32_t slot = __ffs(v) - 1;
      const float4 lo = box[2 * slot], hi = box[2 * slot + 1];
      MJPBR_COUNT(kOpBox);
      if (box_entry(ri, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, cut) >= 0.0f) mask |= 1u << slot;
    }
    return mask;
  }
  // The slots any ray from o to within `radius` of o + to may hit: on its way such a ray stays within radius
  // of this one. radius has to cover the rounding of the tests too, the approximate reciprocals' among it.
  static MJ_DEV float around_rcp(float x) { return approx_rcp(fabsf(x) > 1.0e-30f ? x : (x >= 0.0f ? 1.0e-30f : -1.0e-30f)); }
  MJ_DEV uint32_t mask_around(V3 o, V3 to, float cut, float radius) const {
    RayInv ri;
    ri.inv = V3{around_rcp(to.x), around_rcp(to.y), around_rcp(to.z)};
    ri.oinv = cmul(o, ri.inv);
    const float gx = radius * fabsf(ri.inv.x), gy = radius * fabsf(ri.inv.y), gz = radius * fabsf(ri.inv.z);
    uint32_t mask = 0;
#pragma unroll 1
    for (uint32_t v = valid; v; v &= v - 1u) {
      const int32_t slot = __ffs(v) - 1;
      const float4 lo = box[2 * slot], hi = box[2 * slot + 1];
      MJPBR_COUNT(kOpBox);
      const float ax = __fmaf_rn(lo.x, ri.inv.x, -ri.oinv.x), bx = __fmaf_rn(hi.x, ri.inv.x, -ri.oinv.x);
      const float ay = __fmaf_rn(lo.y, ri.inv.y, -ri.oinv.y), by = __fmaf_rn(hi.y, ri.inv.y, -ri.oinv.y);
      const float az = __fmaf_rn(lo.z, ri.inv.z, -ri.oinv.z), bz = __fmaf_rn(hi.z, ri.inv.z, -ri.oinv.z);
      const float tmin = fmaxf(fmaxf(fminf(ax, bx) - gx, fminf(ay, by) - gy), fminf(az, bz) - gz);
      const float tmax = fminf(fminf(fmaxf(ax, bx) + gx, fmaxf(ay, by) + gy), fmaxf(az, bz) + gz);
      if (tmax >= fmaxf(tmin, 0.0f) && tmin < cut) mask |= 1u << slot;
    }
    return mask;
  }
};

constexpr int32_t kSlotBoxFloats = kScanGeoms * 8 + 4;

MJ_DEV void stage_boxes(const float* blk, const BlockLayout& L, float* out, int32_t nthreads) {
  uint32_t* valid = reinterpret_cast<uint32_t*>(out + kScanGeoms * 8);
  for (int32_t i = threadIdx.x; i < 2 * L.nnode; i += nthreads) {
    const float4* c = reinterpret_cast<const float4*>(blk + L.node_off) + 2 * i;
    if (__float_as_int(c[1].w) != 1) continue;
    const int32_t slot = __float_as_int(c[0].w);
    reinterpret_cast<float4*>(out)[2 * slot] = c[0];
    reinterpret_cast<float4*>(out)[2 * slot + 1] = c[1];
    atomicOr(valid, 1u << slot);
  }
}

MJ_DEV SlotBoxes staged_boxes(const float* out) {
  return SlotBoxes{reinterpret_cast<const float4*>(out), *reinterpret_cast<const uint32_t*>(out + kScanGeoms * 8)};
}

// The union of the converged lanes' masks: the lanes of a warp that call together visit its geoms
// together (any grouping gives the same results).
MJ_DEV uint32_t scan_union(uint32_t mask) { return __reduce_or_sync(__activemask(), mask); }

// trace_ray's selection between the best hit so far and a hit of geom g at d (d < 0: none).
MJ_DEV void scan_offer(Hit& h, bool& tie, const Ray& r, const float* g, int32_t slot, float d, V3 n, float u, float v, int32_t face,
                       int32_t mesh, bool cull) {
  if (cull && d >= 0.0f && dot(r.d, n) > 0.0f) d = -1.0f;
  if (d < 0.0f) return;
  const int32_t gi = __float_as_int(g[16]);
  const float tol = kRayTolRel * fmaxf(h.dist, 1.0f);
  if (h.geom >= 0 && fabsf(d - h.dist) <= scan_window(h.dist)) tie = true;
  const bool closer = (d < h.dist - tol) || (fabsf(d - h.dist) <= tol && (h.geom < 0 || gi > h.geom));
  if (closer) {
    h.dist = d;
    h.normal = n;
    h.geom = gi;
    h.slot = slot;
    h.u = u;
    h.v = v;
    h.face = face;
    h.mesh = mesh;
  }
}

// Closest hit among the primitives; returns the mask of the mesh geoms still to trace.
template <bool kMesh, class Boxes>
MJ_DEV uint32_t scan_closest(Hit& h, bool& tie, const Boxes& boxes, const float* blk, const BlockLayout& L, const Ray& r, float max_dist,
                             bool cull) {
  MJPBR_COUNT(kOpRayClosest);
  h.geom = -1;
  h.slot = -1;
  h.dist = max_dist;
  h.normal = v3(0.0f);
  h.u = 0.0f;
  h.v = 0.0f;
  h.face = -1;
  h.mesh = -1;
  tie = false;
  const uint32_t mask = boxes.mask(make_inv(r), max_dist * (1.0f + kRayTolRel) + kRayTolAbs);
  uint32_t meshes = 0;
  for (uint32_t todo = scan_union(mask); todo; todo &= todo - 1u) {
    const int32_t slot = __ffs(todo) - 1;
    if (!((mask >> slot) & 1u)) continue;
    const float* g = blk + L.geom_off + slot * kGeomFloats;
    if (kMesh && geom_bvh(g) >= 0) {
      meshes |= 1u << slot;
    } else {
      V3 n = v3(0.0f);
      const float d = intersect_primitive(g, r, &n);
      scan_offer(h, tie, r, g, slot, d, n, 0.0f, 0.0f, -1, -1, cull);
    }
  }
  return meshes;
}

// How far a mesh is traced: a little past the best hit so far, so that a hit that order could decide is
// seen and marked; without one, to trace_ray's own cut-off.
MJ_DEV float scan_cut(const Hit& h) {
  return h.geom >= 0 ? h.dist + scan_window(h.dist) : h.dist * (1.0f + kRayTolRel) + kRayTolAbs;
}

// The closest hit within max_dist (trace_ray with any = false).
template <bool kMesh, class Boxes>
MJ_DEV Hit scan_trace(const Boxes& boxes, const MjpbrScene& sc, const Stack& st, const float* blk, const BlockLayout& L, const Ray& r, float max_dist,
                      bool cull, int32_t* err) {
  Hit h;
  bool tie;
  uint32_t meshes = scan_closest<kMesh>(h, tie, boxes, blk, L, r, max_dist, cull);
  if (kMesh) {
    for (; meshes; meshes &= meshes - 1u) {
      const int32_t slot = __ffs(meshes) - 1;
      const float* g = blk + L.geom_off + slot * kGeomFloats;
      const GeomFrame f = geom_frame(g);
      const int32_t mid = __float_as_int(g[17]);
      V3 lo, ld, nl = v3(0.0f);
      float u = 0.0f, v = 0.0f;
      int32_t face = -1;
      map_local(f, r, &lo, &ld);
      const float d = mesh_query(sc, st, 0, mid, lo, ld, scan_cut(h), cull, false, &nl, &u, &v, &face, err);
      if (d >= 0.0f) scan_offer(h, tie, r, g, slot, d, mul(f.mat, nl), u, v, face, mid, cull);
    }
  }
  if (tie) h = trace_ray<kMesh>(sc, st, blk, L, r, max_dist, cull, false, err);
  return h;
}

// Any hit before max_dist among the primitives of mask; *meshes gets its mesh geoms, still to trace (0
// after a hit).
template <bool kMesh>
MJ_DEV bool scan_any(uint32_t mask, const float* blk, const BlockLayout& L, const Ray& r, float max_dist, bool cull, uint32_t* meshes) {
  MJPBR_COUNT(kOpRayAny);
  uint32_t mm = 0;
  bool found = false;
  for (uint32_t todo = scan_union(mask); todo; todo &= todo - 1u) {
    const int32_t slot = __ffs(todo) - 1;
    if (!((mask >> slot) & 1u)) continue;
    const float* g = blk + L.geom_off + slot * kGeomFloats;
    if (kMesh && geom_bvh(g) >= 0) {
      mm |= 1u << slot;
    } else {
      V3 n = v3(0.0f);
      float d = intersect_primitive(g, r, &n);
      if (cull && d >= 0.0f && dot(r.d, n) > 0.0f) d = -1.0f;
      if (d >= 0.0f && d < max_dist) {
        found = true;
        mask = 0;
        mm = 0;
      }
    }
  }
  *meshes = mm;
  return found;
}

template <bool kMesh>
MJ_DEV bool scan_any(const float* blk, const BlockLayout& L, const Ray& r, float max_dist, bool cull, uint32_t* meshes) {
  return scan_any<kMesh>(NodeBoxes{blk, &L}.mask(make_inv(r), max_dist * (1.0f + kRayTolRel) + kRayTolAbs), blk, L, r, max_dist, cull, meshes);
}

// ---------------------------------------------------------------- resumable mesh part
// The meshes of a scanned ray as a resumable query for the persistent refill loops (refill.cuh):
// scan_begin_mesh sets up the next mesh of the mask, scan_mesh_step advances by one node or leaf.
struct MeshWalk {
  Ray r;
  uint32_t meshes;  // mesh geoms still to trace
  int32_t sp;
  int32_t code;     // the node or leaf to visit, -1: the mesh (or the first one) is done
  int32_t slot;     // the mesh geom being traced, -1: none
  const float* nodes;
  const float* tris;
  WoopRay w;
  RayInv ri;
  float cut;        // hits at or past it do not count
};

// What a walk's next step does: 0 visits a node, 1 a leaf, 2 ends a mesh and takes the next.
MJ_DEV int32_t walk_kind(const MeshWalk& q) { return q.code < 0 ? 2 : ((q.code & 7) != 0 ? 1 : 0); }

MJ_DEV void walk_next(MeshWalk& q, const MjpbrScene& sc, const float* blk, const BlockLayout& L) {
  const int32_t slot = __ffs(q.meshes) - 1;
  q.meshes &= q.meshes - 1u;
  const float* g = blk + L.geom_off + slot * kGeomFloats;
  const int32_t bvh = __float_as_int(g[17]);
  V3 lo, ld;
  map_local(geom_frame(g), q.r, &lo, &ld);
  q.nodes = sc.blas_nodes + (int64_t)sc.blas_root[bvh] * kNodeFloats;
  q.tris = sc.blas_tris + (int64_t)sc.blas_tri_base[bvh] * kTriFloats;
  q.w = woop_setup(lo, ld);
  q.ri = make_inv(Ray{lo, ld});
  q.slot = slot;
  q.sp = 0;
  q.code = 0;  // the root
}

// Any hit: q.cut = max_dist.
MJ_DEV int32_t walk_any_step(MeshWalk& q, const MjpbrScene& sc, const Stack& st, const float* blk, const BlockLayout& L, int32_t* err) {
  if (q.code < 0) {
    if (!q.meshes) return kAnyClear;
    walk_next(q, sc, blk, L);
    return kAnyRunning;
  }
  const int32_t ref = q.code >> 3, cnt = q.code & 7;
  if (cnt == 0) {
    const float* nd = q.nodes + (int64_t)ref * kNodeFloats;
    if (!descend(st, q.sp, q.ri, ldg4(nd), ldg4(nd + 4), ldg4(nd + 8), ldg4(nd + 12), q.cut, &q.code, err) &&
        !pop_near(st, q.sp, 0, q.cut, &q.code)) {
      q.code = -1;
    }
    return kAnyRunning;
  }
  for (int32_t i = ref; i < ref + cnt; ++i) {
    const float* tr = q.tris + (int64_t)i * kTriFloats;
    const float4 a = ldg4(tr), b = ldg4(tr + 4), c = ldg4(tr + 8);
    float tu, tv;
    MJPBR_COUNT(kOpTri);
    if (woop_hit(q.w, V3{a.x, a.y, a.z}, V3{b.x, b.y, b.z}, V3{c.x, c.y, c.z}, q.cut, &tu, &tv) >= 0.0f) return kAnyHit;
  }
  if (!pop_near(st, q.sp, 0, q.cut, &q.code)) q.code = -1;
  return kAnyRunning;
}

// Closest hit: q.cut is the best hit's distance within the mesh being traced (at first a little past
// the best hit of all geoms).
struct ClosestWalk {
  MeshWalk m;
  Hit h;
  bool tie;
  V3 ld, n;
  float u, v;
  int32_t face;
};

MJ_DEV int32_t walk_closest_step(ClosestWalk& q, const MjpbrScene& sc, const Stack& st, const float* blk, const BlockLayout& L, bool cull,
                                 int32_t* err) {
  MeshWalk& m = q.m;
  if (m.code < 0) {
    if (m.slot >= 0) {  // the mesh is done
      if (q.face >= 0) {
        const float* g = blk + L.geom_off + m.slot * kGeomFloats;
        scan_offer(q.h, q.tie, m.r, g, m.slot, m.cut, mul(geom_frame(g).mat, normalize(q.n)), q.u, q.v, q.face, __float_as_int(g[17]), cull);
      }
      m.slot = -1;
    }
    if (!m.meshes) return kAnyClear;
    walk_next(m, sc, blk, L);
    q.ld = mul_t(geom_frame(blk + L.geom_off + m.slot * kGeomFloats).mat, m.r.d);
    m.cut = scan_cut(q.h);
    q.face = -1;
    return kAnyRunning;
  }
  const int32_t ref = m.code >> 3, cnt = m.code & 7;
  if (cnt == 0) {
    const float* nd = m.nodes + (int64_t)ref * kNodeFloats;
    if (!descend(st, m.sp, m.ri, ldg4(nd), ldg4(nd + 4), ldg4(nd + 8), ldg4(nd + 12), m.cut, &m.code, err) &&
        !pop_near(st, m.sp, 0, m.cut, &m.code)) {
      m.code = -1;
    }
    return kAnyRunning;
  }
  for (int32_t i = ref; i < ref + cnt; ++i) {
    const float* tr = m.tris + (int64_t)i * kTriFloats;
    const float4 a = ldg4(tr), b = ldg4(tr + 4), c = ldg4(tr + 8);
    const V3 v0{a.x, a.y, a.z}, v1{b.x, b.y, b.z}, v2{c.x, c.y, c.z};
    float tu, tv;
    MJPBR_COUNT(kOpTri);
    const float t = woop_hit(m.w, v0, v1, v2, m.cut, &tu, &tv);
    if (t < 0.0f) continue;
    const V3 ng = cross(v1 - v0, v2 - v0);
    if (cull && dot(q.ld, ng) > 0.0f) continue;
    m.cut = t;
    q.face = __float_as_int(a.w);
    q.n = ng;
    q.u = tu;
    q.v = tv;
  }
  if (!pop_near(st, m.sp, 0, m.cut, &m.code)) m.code = -1;
  return kAnyRunning;
}

}  // namespace mjpbr
