// Single-grid walk in direction order (cone_walk.cuh): one CTA per item of
// rays, 32 neighbouring rays per warp in step.
#include <cuda_runtime.h>

#include <cstdint>

#include "cone_walk.cuh"
#include "kernels.cuh"

namespace cublox_b200 {

namespace {

template <int kRays>
__global__ void __launch_bounds__(kRays, 1024 / kRays)
    cone_walk_kernel(const __grid_constant__ RayParams p) {
  extern __shared__ int table[];
  __shared__ ConeItem<kRays> ci;
  cone_table(p, table);  // cone_order's barriers follow
  const int start = blockIdx.x * kRays;
  int ray[1];
  cone_order<kRays, 1>(p, start, min(kRays, p.n - start), ci, ray);
  const int r = ray[0];
  uint32_t rays = 0, incs = 0, hits = 0;
  cone_walk(p, table, r >= 0, r >= 0 ? ci.x[r] : 0.0f, r >= 0 ? ci.y[r] : 0.0f,
            r >= 0 ? ci.z[r] : 0.0f, rays, incs, hits);
  if (p.stats) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      rays += __shfl_down_sync(0xffffffffu, rays, off);
      incs += __shfl_down_sync(0xffffffffu, incs, off);
      hits += __shfl_down_sync(0xffffffffu, hits, off);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(p.stats + 0, static_cast<unsigned long long>(rays));
      atomicAdd(p.stats + 1, static_cast<unsigned long long>(incs));
      atomicAdd(p.stats + 2, static_cast<unsigned long long>(hits));
    }
  }
}

template <int kRays>
void launch(const RayParams &p, cudaStream_t s) {
  cone_walk_kernel<kRays><<<(p.n + kRays - 1) / kRays, kRays,
                            sizeof(int) * static_cast<size_t>(cone_table_words(p.map)), s>>>(p);
}

}  // namespace

// Rays per item: as many as leave 256 items, so that every SM has some (the
// longest ray of an item sets its time), 64 to 512.  Wider items put more
// neighbours into a warp's rows.  Walk times in us at 64 / 128 / 256 / 512 /
// 1,024 rays (the split walk with its plan: last): 16-beam scan of 16,384 rays
// 32 / 37 / 39 / 46 / - (78); 64 beams, 65,536 rays 186 / 148 / 119 / 116 /
// 179 (216); 128 beams, 262,144 rays 587 / 570 / 455 / 398 / 377 (933); 640 x
// 480 depth image, 307,200 rays 68 / 61 / 63 / 68 / 74 (205).  The rule takes
// the fastest for the first of these and is 3 us, 21 and 7 off it for the
// others: no size but 256 and 512 is near the fastest for both of the last two.
void launch_raycast_cone(const RayParams &p, cudaStream_t s) {
  if (p.n <= 0) return;
  const int fit = p.n / 256;
  if (fit >= 512)
    launch<512>(p, s);
  else if (fit >= 256)
    launch<256>(p, s);
  else if (fit >= 128)
    launch<128>(p, s);
  else
    launch<64>(p, s);
}

}  // namespace cublox_b200
