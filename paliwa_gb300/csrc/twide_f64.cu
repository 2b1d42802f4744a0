// The TMA wide kernel (twide.cuh) for FP64 grids (one column per thread).
#include "twide_launch.cuh"

namespace pgb {

void launch_twide_f64(int sched, int code, TWideParams const &p,
                     cudaStream_t s) {
  with_wavelet_sched(sched, [&](auto w) {
    launch_twide_cols<ColF64<true>, decltype(w)>(code, p, s);
  });
}

} // namespace pgb
