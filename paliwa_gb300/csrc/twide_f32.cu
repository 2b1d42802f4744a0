// The TMA wide kernel (twide.cuh) for FP32 grids (rows of two columns as f32x2 pairs).
#include "twide_launch.cuh"

namespace pgb {

void launch_twide_f32(int sched, int code, TWideParams const &p,
                     cudaStream_t s) {
  with_wavelet_sched(sched, [&](auto w) {
    launch_twide_rows<RowF32x2<true>, decltype(w)>(code, p, s);
  });
}

} // namespace pgb
