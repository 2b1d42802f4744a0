// Instantiation and launch of the TMA wide kernel, shared by the per-type
// translation units (compiled in parallel).
#pragma once

#include "launch.cuh"
#include "twide_box.cuh"
#include "twide_plan.hpp"

namespace pgb {

template <class A, int R, class Sched, int FORM>
void launch_twide_r(TWideParams const &p, cudaStream_t s) {
  static thread_local Occupancy occ;
  constexpr bool kLong = FORM == 2 || FORM == 5;
  constexpr bool kBox = FORM >= 6;  // 7: with heads
  constexpr int kBlock = kLong  ? kTWideThreads
                         : kBox ? box_threads(R) + 32
                                : twide_threads(R) + 32;
  auto kernel = [] {
    if constexpr (kLong)
      return twide_long_kernel<A, Sched, FORM == 5>;
    else if constexpr (kBox)
      return twide_box_kernel<A, R, Sched, FORM == 7>;
    else
      return twide_kernel<A, R, Sched, FORM>;
  }();
  size_t const smem =
      kBox ? box_smem_bytes<R>() : twide_smem_bytes<R, kLong, Sched::kTable>();
  int const dev = current_device();
  if (dev < 0 || dev >= Occupancy::kMaxDevices)
    throw StatusError(2, "device ordinal beyond the launch cache");
  int &per_sm = occ.per_sm[dev];
  int &sms = occ.sms[dev];
  if (per_sm == 0) {
    cuda_check(cudaFuncSetAttribute(
                   kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                   static_cast<int>(smem)),
               "cudaFuncSetAttribute(twide)");
    int n = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                   &n, kernel, kBlock, smem),
               "occupancy query (twide)");
    sms = device_sms();
    per_sm = n < 1 ? 1 : n;
  }
  long long const resident =
      static_cast<long long>(capped_per_sm(per_sm, p.ctas_per_sm)) * sms;
  long long const blocks = std::min(p.total_tiles, resident);
  kernel<<<static_cast<unsigned>(blocks), kBlock, smem, s>>>(p);
  cuda_check(cudaGetLastError(), "twide kernel launch");
}

// Chunks of floats (rows of two columns).
template <class A, class Sched>
void launch_twide_rows(int code, TWideParams const &p, cudaStream_t s) {
  switch (code) {
  case 2: return launch_twide_r<A, 2, Sched, 0>(p, s);
  case 4: return launch_twide_r<A, 4, Sched, 0>(p, s);
  case 8: return launch_twide_r<A, 8, Sched, 0>(p, s);
  case 16: return launch_twide_r<A, 16, Sched, 0>(p, s);
  case kTWideChunked + 16: return launch_twide_r<A, 16, Sched, 1>(p, s);
  case kTWideContig + 4: return launch_twide_r<A, 4, Sched, 3>(p, s);
  case kTWideContig + 8: return launch_twide_r<A, 8, Sched, 3>(p, s);
  case kTWideContig + 16: return launch_twide_r<A, 16, Sched, 3>(p, s);
  case kTWidePairs + 4: return launch_twide_r<A, 4, Sched, 4>(p, s);
  case kTWidePairs + 8: return launch_twide_r<A, 8, Sched, 4>(p, s);
  case kTWidePairs + 16: return launch_twide_r<A, 16, Sched, 4>(p, s);
  case kTWideLong + 16: return launch_twide_r<A, 16, Sched, 2>(p, s);
  case kTWideLongContig + 16: return launch_twide_r<A, 16, Sched, 5>(p, s);
  case kTWideBox + 16: return launch_twide_r<A, 16, Sched, 6>(p, s);
  case kTWideBoxHeads + 16:
    if constexpr (std::is_same<A, RowF32C>::value)
      return launch_twide_r<A, 16, Sched, 7>(p, s);
    break;
  case kTWide32Chunked:
    if constexpr (sizeof(typename A::V) <= 8)  // plain floats
      return launch_twide_r<A, 32, Sched, 1>(p, s);
    break;
  }
  throw StatusError(2, "twide launch with an unsupported form");
}

// Chunks of doubles (one column per thread).
template <class A, class Sched>
void launch_twide_cols(int code, TWideParams const &p, cudaStream_t s) {
  switch (code) {
  case 2: return launch_twide_r<A, 2, Sched, 0>(p, s);
  case 4: return launch_twide_r<A, 4, Sched, 0>(p, s);
  case 8: return launch_twide_r<A, 8, Sched, 0>(p, s);
  case 16: return launch_twide_r<A, 16, Sched, 0>(p, s);
  case kTWidePairs + 4: return launch_twide_r<A, 4, Sched, 4>(p, s);
  case kTWidePairs + 8: return launch_twide_r<A, 8, Sched, 4>(p, s);
  case kTWidePairs + 16: return launch_twide_r<A, 16, Sched, 4>(p, s);
  case kTWide32Dense: return launch_twide_r<A, 32, Sched, 0>(p, s);
  case kTWide32Chunked: return launch_twide_r<A, 32, Sched, 1>(p, s);
  case kTWide32Pairs: return launch_twide_r<A, 32, Sched, 4>(p, s);
  case kTWide32Box: return launch_twide_r<A, 32, Sched, 6>(p, s);
  }
  throw StatusError(2, "twide launch with an unsupported form");
}

// Calls f with the wavelet schedule of code 2 * wavelet + (forward ? 1 : 0).
template <class F> void with_wavelet_sched(int sched, F &&f) {
  switch (sched) {
  case 0: return f(WaveletSched<0, false>{});
  case 1: return f(WaveletSched<0, true>{});
  case 2: return f(WaveletSched<1, false>{});
  case 3: return f(WaveletSched<1, true>{});
  case 4: return f(WaveletSched<2, false>{});
  case 5: return f(WaveletSched<2, true>{});
  }
  throw StatusError(2, "twide kernel planned without a wavelet schedule");
}

// Calls f with the schedule of a caller's filters.
template <class F> void with_table_sched(int sched, F &&f) {
  if (sched == kTableSched) return f(TableSched<false>{});
  if (sched == kTableSched + 1) return f(TableSched<true>{});
  throw StatusError(2, "bad table schedule");
}

} // namespace pgb
