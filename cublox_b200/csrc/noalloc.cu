// Allocation-free scan integration (cublox_integrate_noalloc).
//
// For callers that may not allocate device memory once they are running:
// a robot's real-time mapping loop that reserves all GPU memory at start-up
// (a cudaMalloc there can block behind other work and blow the cycle's time
// budget), or code that runs inside a host framework which hands it only a
// stream and buffers it owns (an inference-engine plugin's enqueue step, a
// pooled multi-tenant server).  Such a caller owns the map buffers and the
// points; this entry point owns nothing but a fixed scratch area, which
// lives in a file-scope __device__ array (every GPU that loads the library
// holds it until the process exits).
//
// Maps of up to 134M voxels are walked in direction order (cone_walk.cuh) and
// folded by flagged lines (fold.cuh), with the line flags in the scratch.
// Larger ones, those too wide for that walk's step table, and arrays that are
// not 16-byte aligned take the direction-binned walk, with its sorted rays in
// the scratch, and a sweep of every counter (a 65,536-ray scan into
// 701 x 701 x 151 voxels: 505 us; in direction order 267), whose accesses are
// as wide as the arrays' alignment allows (fold_sweep).
//
// The scratch is shared by every call on a device and keeps whatever the
// last call left in it.  The line flags or the direction histogram are
// cleared at the start of each call; every other scratch word is fully
// overwritten before it is read.  Calls whose GPU work overlaps (different
// streams, or different host threads, at the same time) race on the scratch
// and must not be issued.
//
// The walks and folds used here have no device-side check that can fail
// (every index they form is in range by construction), so this entry point
// reports no device error word: the kernels are given none (RayParams::err is
// null, and none of them dereferences it).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/cublox_b200.h"
#include "cone_walk.cuh"
#include "exact_fp.cuh"
#include "kernels.cuh"

using namespace cublox_b200;

namespace {

constexpr int kMaxPoints = CUBLOX_NOALLOC_MAX_POINTS;
constexpr int kBinsWords = 4096;  // direction bins (binned_bins())
// Layout: bins[kMaxPoints] | hist[kBinsWords] | cursor[kBinsWords] |
//         sorted[3 * kMaxPoints] (16-byte aligned)
constexpr size_t kOffHist = sizeof(int) * kMaxPoints;
constexpr size_t kOffCursor = kOffHist + sizeof(int) * kBinsWords;
constexpr size_t kOffSorted = kOffCursor + sizeof(int) * kBinsWords;
static_assert(kOffSorted % 16 == 0, "sorted points must start on a 16-byte boundary");
constexpr size_t kSortBytes = kOffSorted + sizeof(float) * 3 * kMaxPoints;
// Or: flags of up to kFlagLines lines | flags of lines with a hit
constexpr size_t kFlagLines = size_t(1) << 22;
constexpr size_t kScratchBytes = 2 * kFlagLines > kSortBytes ? 2 * kFlagLines : kSortBytes;

__device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

std::mutex g_mu;
constexpr int kMaxDevices = 64;
unsigned char *g_scratch_ptr[kMaxDevices] = {};

thread_local std::string g_noalloc_err;

int noalloc_fail(int code, const std::string &msg) {
  g_noalloc_err = msg;
  return code;
}

bool aligned(const void *q, uintptr_t bytes) {
  return (reinterpret_cast<uintptr_t>(q) & (bytes - 1)) == 0;
}

// The fold of voxels [first, first + n) of the scan that `p` walked: variant 2
// by flagged lines, 1 a sweep that reads counters and stored values 16 bytes
// at a time, 0 one that reads only the counters so.
int fold(const cublox_map_view *map, const RayParams &p, int first, int n, int variant, int lines,
         cudaStream_t s) {
  ApplyParams a{};
  a.occ = map->occ + first;
  a.cnt = map->cnt + first;
  a.hit = map->hit + first;
  a.vnum = n;
  a.l_hit = map->l_hit;
  a.l_miss = map->l_miss;
  a.l_min = map->l_min;
  a.l_max = map->l_max;
  a.l_unknown = 0.0f;
  a.fp = kFpPinned;
  a.stats = nullptr;
  a.variant = variant;
  a.dirty = p.dirty;
  a.hot = p.dirty ? p.dirty + p.hot : nullptr;
  a.nlines = lines;
  launch_apply(a, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return noalloc_fail(CUBLOX_ERR_CUDA, std::string("cublox_integrate_noalloc: fold: ") +
                                             cudaGetErrorString(e));
  return CUBLOX_OK;
}

// A sweep of all voxels.  Stored values that are not 16-byte aligned are
// accessed one by one; of counters that are not, the few before the first
// aligned one are folded by a launch of their own, which has no whole group of
// four.
int fold_sweep(const cublox_map_view *map, const RayParams &p, cudaStream_t s) {
  if (aligned(map->occ, 16) && aligned(map->cnt, 16)) return fold(map, p, 0, p.vnum, 1, 0, s);
  int lead = static_cast<int>((0 - reinterpret_cast<uintptr_t>(map->cnt)) & 15) / 4;
  if (lead > p.vnum) lead = p.vnum;
  const int rc = lead ? fold(map, p, 0, lead, 0, 0, s) : CUBLOX_OK;
  return rc || lead == p.vnum ? rc : fold(map, p, lead, p.vnum - lead, 0, 0, s);
}

}  // namespace

extern "C" {

const char *cublox_noalloc_last_error(void) { return g_noalloc_err.c_str(); }

int cublox_integrate_noalloc(const cublox_map_view *map, const float *xyz_soa, int n,
                             const float sensor_origin[3], void *stream) {
  if (!map || !sensor_origin || !map->occ || !map->cnt || !map->hit)
    return noalloc_fail(CUBLOX_ERR_INVALID, "cublox_integrate_noalloc: null argument");
  if (n < 0 || n > kMaxPoints)
    return noalloc_fail(CUBLOX_ERR_INVALID,
                        "cublox_integrate_noalloc: " + std::to_string(n) +
                            " points; this entry point takes at most " +
                            std::to_string(kMaxPoints) + " per call");
  if (n > 0 && !xyz_soa)
    return noalloc_fail(CUBLOX_ERR_INVALID, "cublox_integrate_noalloc: null points");
  if (!(map->resolution > 0.0f))
    return noalloc_fail(CUBLOX_ERR_INVALID, "cublox_integrate_noalloc: resolution must be > 0");
  // 2 * half + 1 per axis and their product, in 64-bit arithmetic: every
  // factor is checked against int32 before the next multiplication, so no
  // intermediate can overflow (Grid.cpp:33, :44-50).
  int64_t vnum = 1;
  int mapsz[3];
  for (int a = 0; a < 3; ++a) {
    if (map->half_map_size[a] < 0)
      return noalloc_fail(CUBLOX_ERR_INVALID, "cublox_integrate_noalloc: negative half size");
    const int64_t ms = 2 * static_cast<int64_t>(map->half_map_size[a]) + 1;
    if (ms > 2147483647 || vnum * ms > 2147483647)
      return noalloc_fail(CUBLOX_ERR_RANGE, "cublox_integrate_noalloc: voxel count above int32");
    mapsz[a] = static_cast<int>(ms);
    vnum *= ms;
  }
  if (n == 0) return CUBLOX_OK;
  if (!aligned(map->occ, 4) || !aligned(map->cnt, 4) || !aligned(map->hit, 4) || !aligned(xyz_soa, 4))
    return noalloc_fail(CUBLOX_ERR_INVALID,
                        "cublox_integrate_noalloc: an array does not start on a 4-byte boundary");

  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return noalloc_fail(CUBLOX_ERR_CUDA, "cublox_integrate_noalloc: no current device");
  unsigned char *base = nullptr;
  {
    // First call on this device: the scratch array's device address.  In
    // host code the array's name is only a host-side stand-in, so the
    // kernels must be given this address instead.
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch_ptr[dev]) {
      void *ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if (e != cudaSuccess) {
        cudaGetLastError();
        return noalloc_fail(CUBLOX_ERR_CUDA, std::string("cublox_integrate_noalloc: "
                                                         "cudaGetSymbolAddress: ") +
                                                 cudaGetErrorString(e));
      }
      g_scratch_ptr[dev] = static_cast<unsigned char *>(ptr);
    }
    base = g_scratch_ptr[dev];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  RayParams p{};
  p.x = xyz_soa;
  p.y = xyz_soa + n;
  p.z = xyz_soa + 2 * static_cast<size_t>(n);
  p.n = n;
  p.stride = 1;
  const float res = map->resolution;
  for (int a = 0; a < 3; ++a) {
    p.o[a] = sensor_origin[a];
    p.win[a] = map->origin_index[a];
    p.half[a] = map->half_map_size[a];
    p.map[a] = mapsz[a];
  }
  p.res = res;
  p.inv = 1.0f / res;
  p.max_range = map->max_range;
  p.vnum = static_cast<int>(vnum);
  p.ctr = map->origin_at_center ? 1 : 0;
  p.fp = kFpPinned;
  p.cnt = map->cnt;
  p.hit = map->hit;
  p.stats = nullptr;
  p.err = nullptr;  // no check on this path can fail (file comment)
  // the caller's arrays are in the reference's hash order, and bring no line
  // flags
  p.lay.bs[0] = mapsz[1] * mapsz[2];
  p.lay.bs[1] = mapsz[2];
  p.lay.bs[2] = 1;
  p.dirty = nullptr;

  // lines of 32 voxels in full, and the last, partial one
  const int64_t lines = vnum >> kLineShift;
  const size_t flags = (static_cast<size_t>(lines) + 1 + 255) & ~size_t(255);
  if (flags <= kFlagLines && cone_takes(mapsz, vnum) && aligned(map->occ, 16) &&
      aligned(map->cnt, 16) && aligned(map->hit, 16)) {
    p.dirty = base;
    p.hot = static_cast<uint32_t>(flags);
    if ((e = cudaMemsetAsync(base, 0, 2 * flags, s)) == cudaSuccess) {
      launch_raycast_cone(p, s);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess)
      return noalloc_fail(CUBLOX_ERR_CUDA, std::string("cublox_integrate_noalloc: raycast: ") +
                                               cudaGetErrorString(e));
    return fold(map, p, 0, p.vnum, 2, static_cast<int>(lines), s);
  }

  BinnedScratch b{reinterpret_cast<int *>(base), reinterpret_cast<int *>(base + kOffHist),
                  reinterpret_cast<int *>(base + kOffCursor),
                  reinterpret_cast<float *>(base + kOffSorted)};
  // The direction histogram must start at zero; the sort clears it.
  launch_raycast_binned(p, b, 32, false, true, s);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return noalloc_fail(CUBLOX_ERR_CUDA, std::string("cublox_integrate_noalloc: raycast: ") +
                                             cudaGetErrorString(e));
  return fold_sweep(map, p, s);
}

}  // extern "C"
