// Plans of FP32c pencils longer than 4096 points: windows hand their chunk
// heads on only where the tensor maps of those windows are accepted (no other
// kernel takes them). Host code; without a driver every map is refused.
#include <cstdio>
#include <cstdlib>

#include "paliwa_gb300.h"
#include "twide_plan.hpp"

using namespace pgb;

#define CHECK(c)                                                            \
  do {                                                                      \
    if (!(c)) {                                                             \
      std::printf("%s:%d: %s (n 2^%d, inner 2^%d, wavelet %d, forward %d)\n", \
                  __FILE__, __LINE__, #c, n, inner, wavelet, fwd);          \
      std::exit(1);                                                         \
    }                                                                       \
  } while (0)

int main() {
  bool const device = cudaFree(nullptr) == cudaSuccess;  // and its context
  bool const maps = device && tensor_map_encoder() != nullptr;
  int with = 0, without = 0;
  for (int n : {13, 14, 16, 17})
    for (int inner : {0, 2, 7, 10})
      for (int wavelet = 0; wavelet < 3; ++wavelet)
        for (int fwd = 0; fwd < 2; ++fwd) {
          int64_t const level[2] = {n, inner};
          AxisView v = axis_view(1ULL << 32, 2, level, 0, PALIWA_GB_F32C);
          v.shadow = 2ULL << 32;
          v.heads = 3ULL << 32;
          std::vector<Stage> stages;
          plan_axis(v, level_shifts(n, 0, fwd != 0),
                    wavelet_filters(wavelet, fwd != 0), stages);
          bool const heads = maps && n <= 16 && inner >= 7;
          int windows = 0;
          for (Stage const &st : stages) {
            if (st.R >= kHeadsIn) {  // the heads' copies and levels
              CHECK(heads);
              continue;
            }
            if (st.R == kHalo || st.job.periodic) continue;
            ++windows;
            CHECK((st.heads != 0) == heads);
            CHECK(st.box == heads);
            CHECK(st.job.log2_window ==
                  (heads ? kBoxWindowLog2 : kWindowLog2));
          }
          CHECK(windows > 0);
          ++(heads ? with : without);
        }
  std::printf("plans ok: %d with heads, %d without\n", with, without);
  return 0;
}
