// Host side of the slab kernel (slab.cuh).
#pragma once

#include "slab.cuh"
#include "twide_plan.hpp"

namespace pgb {

int slab_start(int dtype, int ndim, int64_t const *level, int64_t const *lmin,
               unsigned long long addr, unsigned long long map_base);
SlabJob slab_job(int dtype, int ndim, int m, int64_t const *level,
                 int64_t const *lmin, unsigned long long addr,
                 unsigned long long map_base);
bool slab_pairs(SlabJob const &job);
bool encode_slab_map(CUtensorMap *map, unsigned long long base,
                     unsigned long long rows, size_t es);

// sched = 2 * wavelet + (forward ? 1 : 0).
void launch_slab(int dtype, int sched, SlabParams const &p, cudaStream_t s);
void launch_slab_f64(int sched, SlabParams const &p, cudaStream_t s);
void launch_slab_f32(int sched, SlabParams const &p, cudaStream_t s);
void launch_slab_f32c(int sched, SlabParams const &p, cudaStream_t s);

// First axis of the trailing axes that a single grid's transform runs as one
// slab launch (ndim: none), and that launch (error: from begin_stages; false:
// the tensor map was refused and nothing was launched).
int single_slab_start(int dtype, int ndim, int64_t const *level,
                      int64_t const *lmin, void const *grid);
bool launch_single_slab(int dtype, int ndim, int m, int64_t const *level,
                        int64_t const *lmin, void *grid, int sched,
                        unsigned *error, cudaStream_t s);

} // namespace pgb
