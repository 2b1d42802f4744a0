// The TMA wide kernel (twide.cuh) with a caller's filters, for
// FP64 grids (one column per thread).
#include "twide_launch.cuh"

namespace pgb {

void launch_twide_table_f64(bool exact, int sched, int code,
                           TWideParams const &p, cudaStream_t s) {
  with_table_sched(sched, [&](auto w) {
    if (exact)
      launch_twide_cols<ColF64<true>, decltype(w)>(code, p, s);
    else
      launch_twide_cols<ColF64<false>, decltype(w)>(code, p, s);
  });
}

} // namespace pgb
