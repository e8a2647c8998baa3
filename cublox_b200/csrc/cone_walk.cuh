// Exact ray walk of 32 neighbouring rays in step (sm_100a), used by the
// batched walk (batch.cu) and the single-grid walk (raycast_cone.cu).
//
// What bounds a walk of a thread per ray is the atomic requests the L2 takes: about
// 185 G/s however wide each is, with lanes of one instruction served
// together where they add to different words of a 32-byte sector and one
// after another where they add to the same word.  A thread per ray in input
// order sends one request per voxel visited (19.7M for a 65,536-ray scan).
// Here the rays of an item are ordered by direction, so that a warp holds a
// narrow cone of rays, and its lanes walk in step: every ray starts in the
// sensor's voxel and visits a voxel at L1 distance k on its k-th step, so
// lanes that visit the same voxel do so in the same iteration.  Runs of
// neighbouring lanes on one voxel become one addition of the run's length
// (every lane of the voxel's, in the first steps), and lanes on different
// voxels of one sector share a request: 6.8M (8.3M in one grid's smaller items),
// 62 to 76 G/s, so that a ray's chain of dependent steps and the barrier at an
// item's end are the bound now.  There is no counter cube around the sensor to
// clear and flush: a warp adds 32 rays to the sensor's voxel in one request.
#pragma once

#include <cstdint>

#include "exact_fp.cuh"
#include "far_walk.cuh"
#include "kernels.cuh"
#include "ray_walk.cuh"

namespace cublox_b200 {

// ---- a map's address terms as steps ----
// For each axis and direction, what each step of a ray adds to the voxel's
// address, from the window's far side to where the ray leaves it: the ring
// buffer's wrap and the brick arithmetic are done once per item instead of
// once per step, and a place in the table only ever moves up by one.  The
// step out of the window adds kLeave, which makes any address negative; the
// walk goes on by up to kBlock - 1 steps of zeros after it, and rests on the
// zeros at the table's end.
constexpr int kBlock = 4;  // steps walked between two looks at who is left
constexpr int kLeave = -(1 << 29);
constexpr float kConeMaxRes = 1e25f;  // cone_walk: longer voxels are walked step by step
constexpr int kConeTableMax = 8192;  // words of shared memory a table may take

CBX_HD int64_t cone_table_words(const int map[3]) {
  return 2 * (static_cast<int64_t>(map[0]) + map[1] + map[2]) + 7 * kBlock;
}

// Whether the cone walk takes a map: its table fits the shared memory set
// aside for it, and an address less one to four times -kLeave (the ray's end
// and three axes' steps out) is below zero and does not wrap around.
CBX_HD bool cone_takes(const int map[3], int64_t nalloc) {
  return cone_table_words(map) <= kConeTableMax && nalloc <= -static_cast<int64_t>(kLeave);
}

// Start of axis a's steps in the table, up (dir 0) or down (dir 1); a = 3:
// the resting place.
__device__ __forceinline__ int cone_axis_base(const RayParams &p, int a, int dir) {
  int b = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < a) b += 2 * (p.map[i] + kBlock);
  return a < 3 ? b + dir * (p.map[a] + kBlock) : b;
}

// Fills the table of the map; the whole CTA takes part and meets at the
// caller's next barrier.
__device__ __forceinline__ void cone_table(const RayParams &p, int *table) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int m = p.map[a], up = cone_axis_base(p, a, 0), down = cone_axis_base(p, a, 1);
    // slot of the window's far side: the middle's less half, around the ring
    // (win - half itself may be out of range)
    const int l0 = global_to_local(p.win[a], m, p.half[a]);
    const int s0 = l0 < 0 ? l0 + m : l0;
    for (int r = threadIdx.x; r < m + kBlock; r += blockDim.x) {
      if (r >= m) {
        table[up + r] = table[down + r] = 0;
      } else if (r == m - 1) {
        table[up + r] = table[down + r] = kLeave;
      } else {  // between the window's r-th and (r + 1)-th slot
        const int s = s0 + r >= m ? s0 + r - m : s0 + r;
        const int step = vox_axis(p.lay, a, s + 1 == m ? 0 : s + 1) - vox_axis(p.lay, a, s);
        table[up + r] = step;
        table[down + m - 2 - r] = -step;
      }
    }
  }
  if (threadIdx.x < kBlock) table[cone_axis_base(p, 3, 0) + threadIdx.x] = 0;
}

// ---- an item's rays in direction order ----
template <int kRays>
struct ConeItem {
  float x[kRays], y[kRays], z[kRays];  // the item's points, in input order
  uint32_t key[kRays];                 // being sorted: direction above, ray below
};

// Place of the ray's direction: elevation rows (512 over the sphere's
// height), azimuth along a row (2,048 over the circle); any place for
// degenerate rays.  Rows, not square cells: neighbours along a row stay on
// one level of voxels, so that they share voxels and, with bricks one voxel
// high, sectors (8 maps' walks 0.64 ms, 0.80 ms in Morton order of square
// direction cells).
__device__ __forceinline__ uint32_t cone_place(float dx, float dy, float dz) {
  const float flat = fabsf(dx) + fabsf(dy);
  const float el = dz * rsqrtf(dx * dx + dy * dy + dz * dz);
  float az = flat > 0.0f ? dx / flat : 0.0f;
  az = dy < 0.0f ? 3.0f - az : 1.0f + az;  // [0, 4): monotone around the circle
  const int row = min(max(static_cast<int>((el * 0.5f + 0.5f) * 512.0f), 0), 511);
  const int col = min(max(static_cast<int>(az * 512.0f), 0), 2047);
  return static_cast<uint32_t>(row) << 11 | static_cast<uint32_t>(col);
}

// Reads the item's points (each once: they may sit in host memory) and
// sorts its rays by direction: a bitonic sort of kKeys keys per thread (the
// places t and t + kRays / 2 of the item for two), exchanges within a warp by
// shuffle.  blockDim.x == kRays / kKeys, a power of two of at least 32.
// ray[r] is then the ray (its place in the item) that came to this thread's
// r-th place, -1 past the item's rays: a warp's threads hold 32 neighbours,
// and with two keys another 32 from half the item's rows away.  An item
// without a finite point (most of a depth image's sky) is not sorted: all its
// threads get -1.  Contains CTA barriers.
template <int kRays, int kKeys>
__device__ __forceinline__ void cone_order(const RayParams &p, int start, int count,
                                           ConeItem<kRays> &it, int (&ray)[kKeys]) {
  constexpr int kThreads = kRays / kKeys;
  static_assert((kRays & (kRays - 1)) == 0 && kThreads >= 32 && kRays <= 1024 && kKeys <= 2,
                "a CTA's worth");
  const int t = threadIdx.x;
  uint32_t key[kKeys];
  bool finite = false;
#pragma unroll
  for (int r = 0; r < kKeys; ++r) {
    const int e = t + r * kThreads;
    key[r] = 0xffffffffu;
    ray[r] = -1;
    if (e < count) {
      const size_t k = static_cast<size_t>(start + e) * p.stride;
      const float x = p.x[k], y = p.y[k], z = p.z[k];
      it.x[e] = x;
      it.y[e] = y;
      it.z[e] = z;
      key[r] = (cone_place(x - p.o[0], y - p.o[1], z - p.o[2]) << 10) | e;
      // coordinate by coordinate: the sum of finite ones may be out of range
      finite = finite || (isfinite(x) && isfinite(y) && isfinite(z));
    }
  }
  if (!__syncthreads_or(finite)) return;
#pragma unroll
  for (int len = 2; len <= kRays; len <<= 1) {
#pragma unroll
    for (int d = len >> 1; d > 0; d >>= 1) {
      if (d >= 32 && d < kThreads) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kKeys; ++r) it.key[t + r * kThreads] = key[r];
        __syncthreads();
      }
      uint32_t other[kKeys];
#pragma unroll
      for (int r = 0; r < kKeys; ++r)
        other[r] = d == kThreads ? key[kKeys - 1 - r]
                   : d >= 32     ? it.key[(t + r * kThreads) ^ d]
                                 : __shfl_xor_sync(0xffffffffu, key[r], d);
#pragma unroll
      for (int r = 0; r < kKeys; ++r) {
        const int e = t + r * kThreads;
        const bool up = (e & len) == 0, low = (e & d) == 0;
        key[r] = (up == low) ? min(key[r], other[r]) : max(key[r], other[r]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kKeys; ++r)
    ray[r] = key[r] == 0xffffffffu ? -1 : static_cast<int>(key[r] & 0x3ffu);
}

// ---- the walk ----
// An addition whose result nobody waits for.  Spelled in PTX because
// atomicAdd of a value other than a constant became an atomic with a return
// value here, which takes the way back through the crossbar as well.
__device__ __forceinline__ void red_add(uint32_t *at, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(at)), "r"(v)
               : "memory");
}

constexpr int kMatchBlocks = 2;  // first blocks merged over all lanes, not runs alone

// A warp's far state: one ray a lane.
struct ConeRay {
  float t0, t1, t2, d0, d1, d2;  // next event time per axis, and its step
  uint32_t j0, j1, j2;           // shared-memory addresses of the next steps' table words
  int h;                         // address of the current voxel, negative once the loop is over
  int he;                        // endpoint's address, -1 outside the window
  int limit;                     // loop iterations the ray may still take
  int last;                      // line flagged last
};

// kBlock loop iterations (k, k + 1, ...) of the warp's rays: each stops a
// ray at its endpoint or its step limit, counts the current voxel, then
// steps by ray_step's rule.  Lanes whose loop is over do the same on
// addresses below zero (an address in the map, less at most four times
// -kLeave), so that nothing branches.
template <bool kMatch, bool kStats>
__device__ __forceinline__ void cone_block(ConeRay &r, int k, unsigned lane, uint32_t gt,
                                           uint32_t *cnt, uint8_t *dirty, uint32_t &incs) {
#pragma unroll
  for (int i = 0; i < kBlock; ++i) {
    if (r.h >= 0 && (r.h == r.he || k + i >= r.limit)) r.h += kLeave;
    const int h = r.h;
    // one addition per run of lanes on one voxel
    uint32_t add;
    bool head;
    if (kMatch) {
      const uint32_t peers = __match_any_sync(0xffffffffu, h);
      head = (peers & ~gt) == (1u << lane);
      add = __popc(peers);
    } else {
      const int prev = __shfl_up_sync(0xffffffffu, h, 1);
      head = lane == 0 || prev != h;
      const uint32_t heads = __ballot_sync(0xffffffffu, head) & gt;
      add = __clz(__brev(heads)) - lane;
    }
    const int line = h >> kLineShift;
    head = head && h >= 0;
    if (head) red_add(cnt + h, add);
    // lanes on one line share the store
    if (h >= 0 && line != r.last) dirty[line] = 1;
    r.last = line;
    if (kStats && h >= 0) ++incs;
    asm("{\n\t"
        ".reg .pred a, x, y, xy;\n\t"
        ".reg .b32 j, v;\n\t"
        "setp.lt.f32 a, %0, %1;\n\t"
        "setp.lt.and.f32 x, %0, %2, a;\n\t"
        "setp.lt.and.f32 y, %1, %2, !a;\n\t"
        "or.pred xy, x, y;\n\t"
        "selp.b32 j, %4, %5, y;\n\t"
        "selp.b32 j, %3, j, x;\n\t"
        "ld.shared.b32 v, [j];\n\t"
        "add.s32 %6, %6, v;\n\t"
        "@x add.rn.f32 %0, %0, %7;\n\t"
        "@y add.rn.f32 %1, %1, %8;\n\t"
        "@!xy add.rn.f32 %2, %2, %9;\n\t"
        "@x add.u32 %3, %3, 4;\n\t"
        "@y add.u32 %4, %4, 4;\n\t"
        "@!xy add.u32 %5, %5, 4;\n\t"
        "}"
        : "+f"(r.t0), "+f"(r.t1), "+f"(r.t2), "+r"(r.j0), "+r"(r.j1), "+r"(r.j2), "+r"(r.h)
        : "f"(r.d0), "f"(r.d1), "f"(r.d2)
        : "memory");
  }
}

template <bool kStats>
__device__ __forceinline__ void cone_loop(ConeRay &r, uint32_t rest, uint32_t *cnt, uint8_t *dirty,
                                          uint32_t &incs) {
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t gt = 0xfffffffeu << lane;  // lanes above this one
  for (int k = 0; __any_sync(0xffffffffu, r.h >= 0); k += kBlock) {
    if (k < kMatchBlocks * kBlock)
      cone_block<true, kStats>(r, k, lane, gt, cnt, dirty, incs);
    else
      cone_block<false, kStats>(r, k, lane, gt, cnt, dirty, incs);
    if (r.h < 0) {
      r.h = kLeave;
      r.j0 = r.j1 = r.j2 = rest;
    }
  }
}

// Walks the warp's rays (one a lane, `live` lanes only) and applies their
// endpoints.  Every lane calls it; `table` is the map's (in shared memory).
// rays, incs and hits are this lane's; incs only with stats on.
__device__ __forceinline__ void cone_walk(const RayParams &p, const int *table, bool live, float ex,
                                          float ey, float ez, uint32_t &rays, uint32_t &incs,
                                          uint32_t &hits) {
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(table));
  const uint32_t rest = base + 4u * cone_axis_base(p, 3, 0);
  ConeRay r;
  r.t0 = r.t1 = r.t2 = r.d0 = r.d1 = r.d2 = 0.0f;
  r.j0 = r.j1 = r.j2 = rest;
  r.h = kLeave;
  r.he = -1;
  r.limit = 0;
  r.last = -1;
  bool hit = false;
  RayWalk w;
  if (live && ray_begin(p, ex, ey, ez, w)) {
    ++rays;
    // Where the sensor's index is 2^31 voxels or more from the window's (one of
    // them out of range), rel has wrapped around: it does not say where in the
    // table the voxel's slot is.
    bool apart = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const long long d = static_cast<long long>(w.id[a]) - p.win[a];
      apart = apart || d > INT32_MAX || d < -INT32_MAX;
    }
    r.he = end_hash(w, p);
    hit = r.he >= 0 && !w.clipped;
    // up to the window, if the sensor is outside it
    int k = 0;
    while (k < w.max_steps && !at_end(w) && !in_window(w, p)) {
      if (left_for_good(w, p)) {
        k = w.max_steps;
      } else {
        ray_step(w, p);
        ++k;
      }
    }
    // With a time that is no number (or that its first step makes one, from
    // -inf), or with none finite, ray_step's rule may pick an axis that the
    // ray does not move on, which has no steps in the table: walked here, step
    // by step.  So is a map whose steps are so long that adding them up could
    // leave no time finite (below kConeMaxRes the time of a ray's longest axis
    // grows by less than 2e25 a step, in up to 2^33 steps).
    const float inf = inf_f();
    if (apart || !(p.res < kConeMaxRes) || !(w.tM[0] > -inf) || !(w.tM[1] > -inf) || !(w.tM[2] > -inf) ||
        !(fminf(w.tM[0], fminf(w.tM[1], w.tM[2])) < inf)) {
      int last = -1;
      while (k < w.max_steps && !at_end(w) && !left_for_good(w, p)) {
        if (in_window(w, p)) {
          const int h = walk_hash(w, p);
          atomicAdd(p.cnt + h, 1u);
          mark_line(p, h, last);
          ++incs;
        }
        ray_step(w, p);
        ++k;
      }
      k = w.max_steps;
    }
    if (k < w.max_steps && !at_end(w)) {
      r.t0 = w.tM[0], r.t1 = w.tM[1], r.t2 = w.tM[2];
      r.d0 = w.tD[0], r.d1 = w.tD[1], r.d2 = w.tD[2];
      r.h = walk_hash(w, p);
      r.limit = w.max_steps - k;
      uint32_t j[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int q = p.half[a] + (w.st[a] < 0 ? -w.rel[a] : w.rel[a]);
        j[a] = w.st[a] == 0 ? rest : base + 4u * (cone_axis_base(p, a, w.st[a] < 0) + q);
      }
      r.j0 = j[0], r.j1 = j[1], r.j2 = j[2];
    }
  }
  __syncwarp();
  if (p.stats)
    cone_loop<true>(r, rest, p.cnt, p.dirty, incs);
  else
    cone_loop<false>(r, rest, p.cnt, p.dirty, incs);
  if (r.he >= 0) {  // the endpoint (kernels.cu:139-151)
    red_add(p.cnt + r.he, 1u);
    p.dirty[r.he >> kLineShift] = 1;
    ++incs;
    if (hit) {
      mark_hit(p, r.he, 1u);
      ++hits;
    }
  }
}

}  // namespace cublox_b200
