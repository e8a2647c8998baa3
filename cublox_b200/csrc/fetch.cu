// Sphere fetch over host-clipped candidate boxes (the reference's
// fetchOccupancySphereKernel, src/kernels.cu:506-562), samples in ascending
// (x, y, z) order.
//
// A lane takes one (x, y) column of the box and walks it upwards; a warp's
// lanes are the columns of a tile of 8 x 4 slots, so that a level of the tile is
// one 128-byte line of the default voxel layout's bricks.  What is the
// same for a column (its squared offset, its address terms) is computed once
// per column, and nothing is divided per candidate.  The launches:
//   count    samples per column, then a prefix over the columns of each x row
//            (a CTA takes all columns of one tile width of rows; where that
//            makes too few CTAs, several do, and a launch of its own makes the
//            prefixes) and the row's total;
//   rows     per query, a prefix over its rows, and the samples it keeps;
//   offsets  a prefix over the queries (and up to 32 queries' rows);
//   write    32 levels of a tile make 32 keep masks (kept by the count where
//            one state is wanted, else found again), and the warp writes them
//            one column after another, a lane per level, so that neighbouring
//            lanes write neighbouring samples.
// Times (cold cache), and with one candidate per thread in (x, y, z) order,
// each a sector of its own behind two 64-bit divisions: a 25 m sphere's
// OCCUPIED voxels, 30M candidates, count 74 us (319), write 15 us (190); those
// of 256 spheres of 1.5 m, 29 us (77) and 17 us (90); 1,000 spheres of 1 m,
// all 3.2M samples, 34 us (94) and 58 us (117).
#include <cuda_runtime.h>

#include <cstdint>

#include "exact_fp.cuh"
#include "kernels.cuh"

namespace cublox_b200 {

namespace {

// A column: where it is, and what its candidates share.
struct Column {
  int rx;           // row within the query's box
  long long at;     // among the query's columns in this launch
  int addr;         // address terms of x and y
  float px, py;     // centre position
  float dx, dy;     // offset from the query's centre
  float xy;         // fma(dx, dx, dy * dy)
  bool valid;
};

__device__ __forceinline__ int slot_global(const FetchParams &p, int a, int slot) {
  return p.win[a] + global_to_local(slot - p.half[a] - p.win[a], p.map[a], p.half[a]);
}

__device__ __forceinline__ void axis_offset(const FetchParams &p, int g, float c, float &pos,
                                            float &d) {
  const float t = p.ctr ? static_cast<float>(g) : fadd(static_cast<float>(g), 0.5f);
  pos = fmul(t, p.res);
  d = (p.fp & kFpFetchDFma) ? ffma(t, p.res, -c) : fsub(pos, c);
}

// The first of the columns of row r of unit `unit`'s tile.
__device__ __forceinline__ long long first_column(const FetchQuery &q, int unit, int r) {
  return static_cast<long long>(((unit - q.u0) << kFetchTileX) + r) * q.n[1];
}

// This lane's column in tile (tx, ty) of the query's box, tx unit `unit`'s.
__device__ __forceinline__ Column column_of(const FetchParams &p, const FetchQuery &q, int unit, int tx,
                                            int ty, int lane) {
  Column c;
  const int r = lane >> kFetchTileY;
  const int sx = (tx << kFetchTileX) + r;
  const int sy = (ty << kFetchTileY) + (lane & ((1 << kFetchTileY) - 1));
  c.valid = sx < p.map[0] && sy < p.map[1];
  const int gx = slot_global(p, 0, sx), gy = slot_global(p, 1, sy);
  c.rx = gx - q.g0[0];
  const int ry = gy - q.g0[1];
  c.valid = c.valid && static_cast<unsigned>(c.rx) < static_cast<unsigned>(q.n[0]) &&
            static_cast<unsigned>(ry) < static_cast<unsigned>(q.n[1]);
  c.at = first_column(q, unit, r) + ry;
  c.addr = vox_axis(p.lay, 0, sx) + vox_axis(p.lay, 1, sy);
  axis_offset(p, gx, q.c[0], c.px, c.dx);
  axis_offset(p, gy, q.c[1], c.py, c.dy);
  c.xy = ffma(c.dx, c.dx, fmul(c.dy, c.dy));
  return c;
}

// kBatch levels from gz (slot sz) of the column, n of them within the box:
// bit k of keep, occupied and free.  All loads are issued before the first
// value is looked at, so that a warp waits once per batch (one by one, the
// count of a 25 m sphere on 63 CTAs took 330 us instead of 143; batches of 16
// gain nothing on more CTAs).
// kPinned: the sphere test's sum of squares is the pinned fma(z, z, fma(x, x,
// y * y)).
constexpr int kBatch = 8;

struct Levels {
  uint32_t keep, occupied, free_;
};

template <bool kPinned>
__device__ __forceinline__ Levels column_levels(const FetchParams &p, const FetchQuery &q,
                                                const Column &c, int gz, int sz, int n) {
  float l[kBatch];
  uint32_t in = 0;
#pragma unroll
  for (int k = 0; k < kBatch; ++k) {
    float pz, dz;
    axis_offset(p, gz + k, q.c[2], pz, dz);
    const float s = kPinned ? ffma(dz, dz, c.xy)
                            : sos(c.dx, c.dy, dz, (p.fp >> kFpFetchSosShift) & 7u);
    const bool inside = c.valid && k < n && !(s > q.r2);
    int slot = sz + k;
    slot = slot >= p.map[2] ? slot - p.map[2] : slot;
    l[k] = 0.0f;
    if (inside) l[k] = p.occ[c.addr + vox_axis(p.lay, 2, slot)];
    in |= static_cast<uint32_t>(inside) << k;
  }
  Levels r{0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < kBatch; ++k) {
    const float v = fadd(l[k], p.l_unknown);
    const int st = v >= p.l_occ ? 2 : (v < p.l_free ? 1 : 0);
    const bool keep = (in >> k & 1u) && (p.filter < 0 || st == p.filter);
    r.keep |= static_cast<uint32_t>(keep) << k;
    r.occupied |= static_cast<uint32_t>(st == 2) << k;
    r.free_ |= static_cast<uint32_t>(st == 1) << k;
  }
  return r;
}

__device__ __forceinline__ int ring(int t, int n) { return t >= n ? t - n : t; }

// An exclusive prefix over n values by one warp, in place; returns their sum.
__device__ __forceinline__ int warp_prefix(int *v, int n, int lane) {
  int carry = 0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int x = i0 + lane < n ? v[i0 + lane] : 0;
    int incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (i0 + lane < n) v[i0 + lane] = carry + incl - x;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  return carry;
}

// A unit's tiles along y are shared by gridDim.y CTAs.
__device__ __forceinline__ int first_tile(const FetchQuery &q) {
  return q.nt[1] * static_cast<int>(blockIdx.y) / static_cast<int>(gridDim.y);
}
__device__ __forceinline__ int last_tile(const FetchQuery &q) {
  return q.nt[1] * static_cast<int>(blockIdx.y + 1) / static_cast<int>(gridDim.y);
}

// For each row of unit `unit`'s tile tx along x: the prefix over its columns,
// and its total.
__device__ __forceinline__ void unit_rows(const FetchParams &p, const FetchQuery &q, int unit, int tx,
                                          int warp, int warps, int lane) {
  for (int r = warp; r < 1 << kFetchTileX; r += warps) {
    const int sx = (tx << kFetchTileX) + r;
    const int rx = slot_global(p, 0, sx) - q.g0[0];
    if (sx >= p.map[0] || static_cast<unsigned>(rx) >= static_cast<unsigned>(q.n[0])) continue;
    const int sum = warp_prefix(p.col + q.col0 + first_column(q, unit, r), q.n[1], lane);
    if (lane == 0 && !p.rows_done) p.row[q.row0 + rx] = sum;
  }
}

template <bool kPinned>
__global__ void __launch_bounds__(256) fetch_count_kernel(const __grid_constant__ FetchParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int2 unit = p.units[blockIdx.x];
  const FetchQuery q = p.queries[unit.x];
  const int tiles_x = (p.map[0] + (1 << kFetchTileX) - 1) >> kFetchTileX;
  const int tiles_y = (p.map[1] + (1 << kFetchTileY) - 1) >> kFetchTileY;
  const int tx = ring(q.t0[0] + unit.y, tiles_x);
  const int s0 = global_to_local(q.g0[2], p.map[2], p.half[2]) + p.half[2];
  int *col = p.col + q.col0;
  const int j1 = last_tile(q);
  for (int j = first_tile(q) + warp; j < j1; j += warps) {
    const Column c = column_of(p, q, unit.y, tx, ring(q.t0[1] + j, tiles_y), lane);
    const int words = (q.n[2] + 31) >> 5;
    int n = 0;
    for (int k0 = 0; k0 < q.n[2]; k0 += 32) {
      uint32_t keep = 0;
      for (int k = 0; k < min(32, q.n[2] - k0); k += kBatch)
        keep |= column_levels<kPinned>(p, q, c, q.g0[2] + k0 + k, ring(s0 + k0 + k, p.map[2]),
                                       q.n[2] - k0 - k).keep << k;
      n += __popc(keep);
      if (p.mask && c.valid) p.mask[q.mask0 + c.at * words + (k0 >> 5)] = keep;
    }
    if (c.valid) col[c.at] = n;
  }
  if (gridDim.y > 1) return;  // the unit's rows are not done: fetch_columns_kernel
  __syncthreads();            // the CTA's own global writes: its rows' columns
  unit_rows(p, q, unit.y, tx, warp, warps, lane);
}

// The row prefixes of units whose columns several CTAs counted.
__global__ void __launch_bounds__(256) fetch_columns_kernel(const __grid_constant__ FetchParams p) {
  const int2 unit = p.units[blockIdx.x];
  const FetchQuery q = p.queries[unit.x];
  const int tiles_x = (p.map[0] + (1 << kFetchTileX) - 1) >> kFetchTileX;
  unit_rows(p, q, unit.y, ring(q.t0[0] + unit.y, tiles_x), threadIdx.x >> 5, blockDim.x >> 5,
            threadIdx.x & 31);
}

// Samples query i keeps, and the prefix over its rows, by one warp.
__device__ __forceinline__ void query_rows(const FetchParams &p, int i, int lane) {
  const FetchQuery q = p.queries[i];
  const int n = q.n[1] > 0 && q.n[2] > 0 ? warp_prefix(p.row + q.row0, q.n[0], lane) : 0;
  if (lane == 0) p.kept[i] = min(n, p.cap);
}

__global__ void __launch_bounds__(256) fetch_rows_kernel(const __grid_constant__ FetchParams p) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i < p.nq) query_rows(p, i, threadIdx.x & 31);
}

// One CTA: offsets[i] = samples the fetch's queries before i keep, offsets[nq]
// = those up to here.  Up to 32 queries' rows are done here too.
__global__ void __launch_bounds__(1024) fetch_offsets_kernel(const __grid_constant__ FetchParams p) {
  __shared__ long long sums[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (p.nq <= 32) {
    if (warp < p.nq) query_rows(p, warp, lane);
    __syncthreads();
  }
  long long carry = p.first ? 0 : p.offsets[0];  // written back below, the same
  for (int i0 = 0; i0 < p.nq; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const long long x = i < p.nq ? p.kept[i] : 0;
    long long incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    long long before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      before += w < warp ? sums[w] : 0;
      all += sums[w];
    }
    if (i < p.nq) p.offsets[i] = carry + before + incl - x;
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) p.offsets[p.nq] = carry;
}

template <bool kPinned>
__global__ void __launch_bounds__(256) fetch_write_kernel(const __grid_constant__ FetchParams p) {
  if (p.offsets[p.nq] > p.room) return;  // the host makes room and launches again
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;  // lanes below this one
  const int2 unit = p.units[blockIdx.x];
  const FetchQuery q = p.queries[unit.x];
  const int tiles_x = (p.map[0] + (1 << kFetchTileX) - 1) >> kFetchTileX;
  const int tiles_y = (p.map[1] + (1 << kFetchTileY) - 1) >> kFetchTileY;
  const int tx = ring(q.t0[0] + unit.y, tiles_x);
  const int s0 = global_to_local(q.g0[2], p.map[2], p.half[2]) + p.half[2];
  const long long base = p.offsets[unit.x];
  const int j1 = last_tile(q);
  for (int j = first_tile(q) + warp; j < j1; j += warps) {
    const Column c = column_of(p, q, unit.y, tx, ring(q.t0[1] + j, tiles_y), lane);
    const int words = (q.n[2] + 31) >> 5;
    int rank = p.cap;  // of the column's next sample within the query
    if (c.valid) rank = p.row[q.row0 + c.rx] + p.col[q.col0 + c.at];
    for (int k0 = 0; k0 < q.n[2]; k0 += 32) {
      // 32 levels: bit k of keep, occupied and free
      uint32_t keep = 0, occupied = 0, free_ = 0;
      if (p.mask) {  // one state wanted: the count kept the masks
        if (c.valid) keep = p.mask[q.mask0 + c.at * words + (k0 >> 5)];
        occupied = p.filter == 2 ? keep : 0u;
        free_ = p.filter == 1 ? keep : 0u;
      }
      for (int k = 0; !p.mask && k < min(32, q.n[2] - k0); k += kBatch) {
        const Levels v = column_levels<kPinned>(p, q, c, q.g0[2] + k0 + k,
                                                ring(s0 + k0 + k, p.map[2]), q.n[2] - k0 - k);
        keep |= v.keep << k;
        occupied |= v.occupied << k;
        free_ |= v.free_ << k;
      }
      float pz, dz;
      axis_offset(p, q.g0[2] + k0 + lane, q.c[2], pz, dz);
      uint32_t with = __ballot_sync(0xffffffffu, keep != 0u && rank < p.cap);
      while (with) {
        const int l = __ffs(with) - 1;
        with &= with - 1;
        const uint32_t m = __shfl_sync(0xffffffffu, keep, l);
        const uint32_t m2 = __shfl_sync(0xffffffffu, occupied, l);
        const uint32_t m1 = __shfl_sync(0xffffffffu, free_, l);
        const float px = __shfl_sync(0xffffffffu, c.px, l), py = __shfl_sync(0xffffffffu, c.py, l);
        const int r = __shfl_sync(0xffffffffu, rank, l) + __popc(m & lt);
        if ((m >> lane & 1u) && r < p.cap) {
          const long long o = base + r;
          p.out_pos[3 * o + 0] = px;
          p.out_pos[3 * o + 1] = py;
          p.out_pos[3 * o + 2] = pz;
          p.out_state[o] = static_cast<uint8_t>((m2 >> lane & 1u) ? 2 : (m1 >> lane & 1u));
        }
      }
      rank += min(__popc(keep), p.cap - rank);  // never past the cap
    }
  }
}

}  // namespace

// CTAs per unit: enough that few units (one large sphere) fill the GPU with 8
// an SM (a 25 m sphere's count: 143 us on its 63 units, 93 on 592 CTAs, 74 on
// 1,184), at most one per 8 tiles (a CTA's warps).
static int fetch_split(const FetchParams &p) {
  const int want = (p.ctas + p.nu - 1) / p.nu;
  const int most = (p.most_tiles + 7) / 8;
  return want < most ? want : most;
}

void launch_fetch_count(const FetchParams &p, cudaStream_t s) {
  if (p.nu <= 0) return;
  const dim3 grid(p.nu, fetch_split(p));
  const int block = 32 * (p.most_tiles < 8 ? p.most_tiles : 8);
  if (((p.fp >> kFpFetchSosShift) & 7u) == kSosFxFz)
    fetch_count_kernel<true><<<grid, block, 0, s>>>(p);
  else
    fetch_count_kernel<false><<<grid, block, 0, s>>>(p);
  if (grid.y > 1) fetch_columns_kernel<<<p.nu, 256, 0, s>>>(p);
}

void launch_fetch_offsets(const FetchParams &p, cudaStream_t s) {
  if (p.nq <= 0) return;
  if (p.nq > 32) fetch_rows_kernel<<<(p.nq + 7) / 8, 256, 0, s>>>(p);
  fetch_offsets_kernel<<<1, 1024, 0, s>>>(p);
}

void launch_fetch_write(const FetchParams &p, cudaStream_t s) {
  if (p.nu <= 0) return;
  const dim3 grid(p.nu, fetch_split(p));
  const int block = 32 * (p.most_tiles < 8 ? p.most_tiles : 8);
  if (((p.fp >> kFpFetchSosShift) & 7u) == kSosFxFz)
    fetch_write_kernel<true><<<grid, block, 0, s>>>(p);
  else
    fetch_write_kernel<false><<<grid, block, 0, s>>>(p);
}

}  // namespace cublox_b200
