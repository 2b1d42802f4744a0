// The TMA wide kernel (twide.cuh) with a caller's filters, for
// FP32 grids (rows of two columns as f32x2 pairs).
#include "twide_launch.cuh"

namespace pgb {

void launch_twide_table_f32(bool exact, int sched, int code,
                           TWideParams const &p, cudaStream_t s) {
  with_table_sched(sched, [&](auto w) {
    if (exact)
      launch_twide_rows<RowF32x2<true>, decltype(w)>(code, p, s);
    else
      launch_twide_rows<RowF32x2<false>, decltype(w)>(code, p, s);
  });
}

} // namespace pgb
