// Persistent ray loops with lane refill, for the traversal stages of the wavefront schedules.
//
// A warp's lanes each trace one ray of a queue as a resumable query (trace.cuh: AnyQuery,
// ClosestQuery) and take the next queue item as soon as their ray is done, instead of waiting for
// the warp's slowest ray: every trip, the idle lanes fetch items from a counter (one atomic per warp),
// then every busy lane advances its query by up to kSteps steps. The per-ray results are the
// queries' own, so they do not depend on which lane traces which ray, or when.
#pragma once

#include "trace.cuh"

namespace mjpbr {

constexpr int32_t kAnyAbort = 3;                       // a query stopped by the step bound
constexpr int32_t kMaxRaySteps = 1 << 20;              // steps of one ray: far above any traversal of a scene
// Idle lanes before a warp of the scanned stages fetches again, whose fetches trace all primitives of a ray. ms at 1,
// 4, 8 and 16: shadow rays of 1024 mesh worlds (128 x 128, 2 x 2 samples) 6.30, 6.73, 6.53, 6.31, of 300 terrain
// worlds 1.38, 1.31, 1.28, 1.26; path-traced frames of 12 and 32 geoms, a third meshes, 6.75, 6.97, 6.80, 6.66 and
// 5.53, 5.66, 5.54, 5.47. For voted_loop's see there.
constexpr int32_t kFetchIdle = 16;
constexpr uint64_t kRefillTimeLimitNs = 4000000000ull; // three orders of magnitude above the largest chunk's stage

MJ_DEV uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Runs the warp's share of `items` queue items (every lane of every warp of the launch must call
// it). fetch(item, q) sets up the query of an item and returns false when the item has no ray;
// step(q) advances the query (kAnyRunning while it runs); finish(q, result) stores a finished
// query's result (result kAnyAbort after kMaxRaySteps steps, with kErrWorkQueue in *err).
// `counter` (64-bit, zero before the launch) hands the items out. Every trip takes new items or
// advances a ray, so the loop ends; a launch still running after kRefillTimeLimitNs sets
// kErrWorkQueue and returns instead of spinning. kMinIdle: idle lanes it takes for the warp to fetch
// (with fewer, the busy lanes go on), and the warp fetches again while that many are idle: for fetches
// that do much of a ray's work, and often all of it.
template <int32_t kSteps, int32_t kMinIdle = 1, class Query, class Fetch, class Step, class Finish>
MJ_DEV void refill_loop(int64_t items, unsigned long long* counter, Query& q, const Fetch& fetch, const Step& step, const Finish& finish,
                        int32_t* err) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  bool busy = false, exhausted = false;
  int32_t steps = 0;
  const uint64_t t_start = global_ns();
  for (;;) {
    if (__any_sync(full, global_ns() - t_start > kRefillTimeLimitNs)) {
      *err |= kErrWorkQueue;
      return;
    }
    const bool need = !busy && !exhausted;
    const unsigned m = __ballot_sync(full, need);
    if (m && (kMinIdle <= 1 || __popc(m) >= kMinIdle || __ballot_sync(full, busy) == 0)) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(m));
      base = __shfl_sync(full, base, leader);
      if (need) {
        const int64_t item = (int64_t)base + __popc(m & ((1u << lane) - 1u));
        if (item >= items) {
          exhausted = true;
        } else if (fetch(item, q)) {
          busy = true;
          steps = 0;
        }
      }
      if (kMinIdle > 1 && __popc(__ballot_sync(full, !busy && !exhausted)) >= kMinIdle) continue;
    }
    if (__ballot_sync(full, busy) == 0) {
      if (__all_sync(full, exhausted)) return;
      continue;
    }
    if (busy) {
#pragma unroll 1
      for (int32_t k = 0; k < kSteps; ++k) {
        int32_t res = step(q);
        if (++steps > kMaxRaySteps && res == kAnyRunning) {
          *err |= kErrWorkQueue;
          res = kAnyAbort;
        }
        if (res != kAnyRunning) {
          finish(q, res);
          busy = false;
          break;
        }
      }
    }
  }
}

// As refill_loop, for queries whose steps differ in kind: kind(q) is what the query's next step does (0, 1
// or 2), and a trip runs the kind most of the warp's lanes wait for, on those lanes. A step of any kind
// then costs its own instructions for many lanes, where stepping every lane costs all kinds' for a few
// each (closest hits of mirror rays among meshes: 4.9 of 32 lanes on average). Lanes of the rarer kinds
// wait, so it pays where rays share little: mirror rays of 1024 mesh worlds of 128 x 128 with 2 x 2 samples
// 6.1 -> 4.1 ms; shadow rays, whose primitives are tested as they are fetched and whose walks are
// alike, go from 1.43 to 1.59 ms on terrain and stay with refill_loop. Fetches happen when kMinIdle lanes
// are idle: at 8, 4.29 ms, at 16, 4.12, at 24, 4.43.
template <int32_t kMinIdle, class Query, class Fetch, class Kind, class Step, class Finish>
MJ_DEV void voted_loop(int64_t items, unsigned long long* counter, Query& q, const Fetch& fetch, const Kind& kind, const Step& step,
                       const Finish& finish, int32_t* err) {
  constexpr int32_t kTrips = 64;  // steps between looks at the clock
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  bool busy = false, exhausted = false;
  int32_t steps = 0;
  const uint64_t t_start = global_ns();
  for (;;) {
    if (__any_sync(full, global_ns() - t_start > kRefillTimeLimitNs)) {
      *err |= kErrWorkQueue;
      return;
    }
    const bool need = !busy && !exhausted;
    const unsigned m = __ballot_sync(full, need);
    if (m && (__popc(m) >= kMinIdle || __ballot_sync(full, busy) == 0)) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(m));
      base = __shfl_sync(full, base, leader);
      if (need) {
        const int64_t item = (int64_t)base + __popc(m & ((1u << lane) - 1u));
        if (item >= items) {
          exhausted = true;
        } else if (fetch(item, q)) {
          busy = true;
          steps = 0;
        }
      }
      __syncwarp();
    }
    if (__ballot_sync(full, busy) == 0) {
      if (__all_sync(full, exhausted)) return;
      continue;
    }
#pragma unroll 1
    for (int32_t k = 0; k < kTrips; ++k) {
      const int32_t kd = busy ? kind(q) : 3;
      const int n0 = __popc(__ballot_sync(full, kd == 0)), n1 = __popc(__ballot_sync(full, kd == 1)), n2 = __popc(__ballot_sync(full, kd == 2));
      if (n0 + n1 + n2 == 0) break;
      const int32_t chosen = n0 >= n1 ? (n0 >= n2 ? 0 : 2) : (n1 >= n2 ? 1 : 2);
      if (kd == chosen) {
        int32_t res = step(q);
        if (++steps > kMaxRaySteps && res == kAnyRunning) {
          *err |= kErrWorkQueue;
          res = kAnyAbort;
        }
        if (res != kAnyRunning) {
          finish(q, res);
          busy = false;
        }
      }
      __syncwarp();
      if (__popc(__ballot_sync(full, !busy && !exhausted)) >= kMinIdle) break;
    }
  }
}

}  // namespace mjpbr
