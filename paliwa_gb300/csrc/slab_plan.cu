// Host side of the slab kernel (slab.cuh): slab groups, jobs, tensor maps and
// the single-grid launch.
#include <algorithm>
#include <cstring>
#include <vector>

#include "paliwa_gb300.h"
#include "slab_plan.hpp"

namespace pgb {

// The slab group of a grid: its trailing axes whose slab (the product of
// their extents) fits one tile, when that group holds at least two axes
// with levels to transform, or one in a grid that is a single tile: a batch
// then needs no launch of its own for it (there and back, us: FP64 6D |l|_1 =
// 9 - q 59 -> 23, FP32 3D 75 -> 63). The grid is a whole number of 1 KB boxes
// and starts on a row of the tensor map (rows of 128 bytes from map_base).
// FP32c pencils of more than 4096 points are windows that round in between
// (plan_axis), and stay so. Returns the group's first axis, or ndim for none.
int slab_start(int dtype, int ndim, int64_t const *lv, int64_t const *lmin,
               unsigned long long addr, unsigned long long map_base) {
  int const log2es = dtype_size(dtype) == 8 ? 3 : 2;
  int64_t total = 0;
  for (int d = 0; d < ndim; ++d) total += lv[d];
  if (total + log2es < 10) return ndim;  // under one 1 KB box
  if (addr < map_base || (addr - map_base) % 128 != 0) return ndim;
  int m = ndim;
  int64_t vol = 0;
  while (m > 0 && vol + lv[m - 1] + log2es <= 15) vol += lv[--m];
  int work = 0;
  for (int d = m; d < ndim; ++d) {
    work += lv[d] > lmin[d];
    if (dtype == PALIWA_GB_F32C && lv[d] > 12) return ndim;
  }
  return work >= (m == 0 ? 1 : 2) && work <= kSlabMaxAxes ? m : ndim;
}

// The slab job of a grid for its axes m..ndim-1: per axis with levels to
// transform, the pencil length, its element stride inside a tile (the
// product of the later extents) and the chunk size: 32 points (at most the
// pencil) for the contiguous last axis and for strides of 32 elements or
// more, 8 or fewer for smaller strides when the pencil's chunks then fit
// the CTA's 256 threads (distinct shared-memory banks under the swizzle).
SlabJob slab_job(int dtype, int ndim, int m, int64_t const *lv,
                 int64_t const *lmin, unsigned long long addr,
                 unsigned long long map_base) {
  int const log2es = dtype_size(dtype) == 8 ? 3 : 2;
  SlabJob job;
  std::memset(&job, 0, sizeof(job));
  int64_t total = 0;
  for (int d = 0; d < ndim; ++d) total += lv[d];
  job.log2_tile = static_cast<int>(std::min<int64_t>(total, 15 - log2es));
  job.row0 = static_cast<long long>((addr - map_base) / 128);
  int log2s = 0;
  std::vector<SlabAxis> axes;
  for (int d = ndim - 1; d >= m; --d) {
    int const log2n = static_cast<int>(lv[d]);
    int const nlev = static_cast<int>(lv[d] - lmin[d]);
    if (nlev > 0) {
      SlabAxis ax{};
      ax.log2n = static_cast<signed char>(log2n);
      ax.log2s = static_cast<signed char>(log2s);
      ax.nlevels = static_cast<signed char>(nlev);
      // Pairs of floats: FP32 throughout, FP32c for pencils that need no
      // barrier (one chunk, or chunks in one warp), in tiles of at least 16
      // points a thread. They halve the shared-memory instructions and double
      // the arithmetic of one. Measured (us, one launch, forward, hat / CDF
      // (2,2)): FP32 32^4 x 16^2 axes 766 / 869 -> 647 / 731, 2^14 x 4^6 344
      // -> 252 (hat), FP32c 32^4 x 16^2 1165 / 1572 -> 1044 / 1431, 2^16 x 8 x
      // 8 x 16 283 / 371 -> 231 / 313; FP32c with barriers 64^3 x 128 axes
      // would go from 111 to 119 (hat).
      int log2r = std::min(log2n, 5);
      if (log2s >= 1 && log2es == 2) {
        int const log2p = log2s - 1;  // inner extent in pairs
        int r = std::min(log2n, dtype == PALIWA_GB_F32C ? 4 : 5);
        if (log2p <= 3 && log2n + log2p - 3 <= 8) r = std::min(log2n, 3);
        int const log2G = log2n - r;
        if (dtype == PALIWA_GB_F32 ||
            (job.log2_tile >= 12 && (log2G == 0 || log2G + log2p <= 5))) {
          ax.pair = 1;
          log2r = r;
        }
      }
      if (ax.pair == 0 && log2s >= 1 && log2s <= 4 && log2n + log2s - 3 <= 8)
        log2r = std::min(log2n, 3);
      ax.log2r = static_cast<signed char>(log2r);
      axes.push_back(ax);
    }
    log2s += log2n;
  }
  std::reverse(axes.begin(), axes.end());
  job.naxes = static_cast<int>(axes.size());
  for (size_t i = 0; i < axes.size(); ++i) job.axis[i] = axes[i];
  return job;
}

// Whether a launch of this job is worth the kernel that works in pairs: they
// halve the threads at work, and small tiles have none to spare (FP32, all
// grids of 2^9 points in 3D, both directions: 34.3 us with them, 34.1
// without).
bool slab_pairs(SlabJob const &job) {
  for (int a = 0; a < job.naxes; ++a)
    if (job.axis[a].pair) return job.log2_tile >= 12;
  return false;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda): a 2D view [rows][128 bytes] from `base`, 1 KB boxes
// (8 rows), 128-byte swizzle.
bool encode_slab_map(CUtensorMap *map, unsigned long long base,
                     unsigned long long rows, size_t es) {
  auto const encode = tensor_map_encoder();
  if (encode == nullptr) return false;
  if (rows == 0 || rows > (1ULL << 31)) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(128 / es), rows};
  cuuint64_t strides[1] = {128};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / es), 8};
  cuuint32_t elem[2] = {1, 1};
  CUresult const r = encode(
      map, es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64
                   : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
      2, reinterpret_cast<void *>(base), dims, strides, box, elem,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

void launch_slab(int dtype, int sched, SlabParams const &p, cudaStream_t s) {
  switch (dtype) {
  case PALIWA_GB_F64: return launch_slab_f64(sched, p, s);
  case PALIWA_GB_F32: return launch_slab_f32(sched, p, s);
  case PALIWA_GB_F32C: return launch_slab_f32c(sched, p, s);
  }
  throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "unknown dtype");
}

// Measured, one call (us, hat / CDF (2,2)), slab against axis by axis:
// launches are what small grids spend their time on (FP32 4^6 15 against 31,
// 128 x 128 x 64 14 / 15 against 19 / 19; FP32c 32^2 x 64 15 / 17 against 19 /
// 20). Floats gain up to about 2^22 points (FP32c 1024 x 64 x 64 34 / 42
// against 36 / 46; 4096 x 64 x 64 130 / 159 against 120 / 152). FP32 gains
// again where the axes no longer run out of L2 (2^26 points: 331 / 361 against
// 362 / 371; 2^24: 106 / 114 against 99 / 108, on four axes 75 / 85 against 70
// / 78). Doubles: one SM's FP64 pipe holds them to 2^13 points on three or
// more axes and 2^11 on two; and a chunk is one thread's chain of updates,
// which the wide kernel cuts into more (on the device, 32 x 32 12 / 22 against
// 7 / 9, 8 x 64 8 / 14 against 6 / 8): no axis in chunks of 32, and two axes in
// chunks of 16 only up to 2^8 points (32 x 16 7 / 10 against 6 / 9; 8 x 16, as
// calls in a row, 8 / 10 against 11 / 12). Over 613 random FP64 grids that is
// 1.25x axis by axis, where the better side of each would give 1.27x.
int single_slab_start(int dtype, int ndim, int64_t const *level,
                      int64_t const *lmin, void const *grid) {
  auto const addr = reinterpret_cast<unsigned long long>(grid);
  int64_t total = 0;
  int axes = 0;
  for (int d = 0; d < ndim; ++d) {
    total += level[d];
    axes += level[d] > lmin[d];
  }
  bool gain = false;
  switch (dtype) {
  case PALIWA_GB_F64: gain = total <= (axes >= 3 ? 13 : 11); break;
  case PALIWA_GB_F32C: gain = total <= 22; break;
  case PALIWA_GB_F32: gain = total <= 22 || total >= 26; break;
  }
  if (!gain || axes < 2 || addr % 128 != 0 || tensor_map_encoder() == nullptr)
    return ndim;
  int const m = slab_start(dtype, ndim, level, lmin, addr, addr);
  if (dtype == PALIWA_GB_F64 && m < ndim) {
    SlabJob const job = slab_job(dtype, ndim, m, level, lmin, addr, addr);
    int log2r = 0;
    for (int a = 0; a < job.naxes; ++a)
      log2r = std::max(log2r, static_cast<int>(job.axis[a].log2r));
    if (log2r > 4 || (log2r == 4 && job.naxes < 3 && total > 8)) return ndim;
  }
  return m;
}

bool launch_single_slab(int dtype, int ndim, int m, int64_t const *level,
                        int64_t const *lmin, void *grid, int sched,
                        unsigned *error, cudaStream_t s) {
  auto const addr = reinterpret_cast<unsigned long long>(grid);
  size_t const es = dtype_size(dtype);
  int64_t total = 0;
  for (int d = 0; d < ndim; ++d) total += level[d];
  SlabParams p;
  std::memset(&p, 0, sizeof(p));
  if (!encode_slab_map(&p.map, addr, (es << total) / 128, es)) return false;
  p.job = slab_job(dtype, ndim, m, level, lmin, addr, addr);
  p.njobs = 1;
  p.pairs = slab_pairs(p.job);
  p.total_tiles = 1LL << (total - p.job.log2_tile);
  p.error = error;
  launch_slab(dtype, sched, p, s);
  return true;
}

} // namespace pgb
