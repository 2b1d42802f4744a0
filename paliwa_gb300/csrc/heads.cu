// Chunk heads of FP32c windows (twide_box.cuh) as double-float pairs: copies
// between the grid and the heads' buffer, and the coarse levels' stage on it.
#include "launch.cuh"

namespace pgb {

namespace {

// The heads of a grid [outer][n][inner] (every 16th point along the axis, at
// job.base) and their buffer [outer][n / 16][inner / 2] of pairs of columns
// {high, high, low, low} at job.halo_base: OUT rounds the pairs to the grid,
// in takes the grid's values as high parts. Four columns per thread and step;
// memory-bound on a sixteenth of the grid.
template <bool OUT>
__global__ void __launch_bounds__(kThreads)
    heads_kernel(__grid_constant__ const LiftJob job) {
  int const log2q = job.log2_inner - 2;
  int const log2h = job.log2_n - 4;
  long long const total = (job.columns >> 2) << log2h;
  long long const step = static_cast<long long>(gridDim.x) * kThreads;
  for (long long i = static_cast<long long>(blockIdx.x) * kThreads +
                     threadIdx.x;
       i < total; i += step) {
    long long const x = i & ((1LL << log2q) - 1);
    long long const h = (i >> log2q) & ((1LL << log2h) - 1);
    long long const z = i >> (log2q + log2h);
    float4 *const grid = reinterpret_cast<float4 *>(
        reinterpret_cast<float *>(job.base) + (z << job.log2_astride) +
        (h << (4 + job.log2_kstride)) + 4 * x);
    float4 *const pair = reinterpret_cast<float4 *>(job.halo_base) + 2 * i;
    if constexpr (OUT) {
      float4 const a = pair[0], b = pair[1];
      *grid = float4{__fadd_rn(a.x, a.z), __fadd_rn(a.y, a.w),
                     __fadd_rn(b.x, b.z), __fadd_rn(b.y, b.w)};
    } else {
      float4 const v = *grid;
      pair[0] = float4{v.x, v.y, 0.0f, 0.0f};
      pair[1] = float4{v.z, v.w, 0.0f, 0.0f};
    }
  }
}

// Levels of the heads' stage: a wavelet's levels with the heads rounded to
// float where the staged kernel's split rounds them, between the fine levels
// of its 4096-point windows (the pencil's levels below 2^7, one-pass wavelets
// 2^8) and its sub-lattice of the others, so that every plan gives the same
// bits. In units of heads those are the levels below 2^KR.
template <int W, bool FWD> struct HeadSched {
  using Base = WaveletSched<W, FWD>;
  static constexpr int KR = Base::Passes::size == 1 ? 4 : 3;

  template <class A, int R, int NT, class Ctx>
  static __device__ __forceinline__ void run_levels(typename A::V (&v)[R],
                                                    Ctx &ctx, int L) {
    constexpr int LOG2R = Log2<R>::value;
    static_assert(LOG2R == 4, "KR is at most the chunk's levels");
    auto round = [&] {
      if (L <= KR) return;
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = RowF32C::load(RowF32C::store(v[j]));
    };
    auto coarse = [&] {
      if (L > LOG2R &&
          !Base::template coarse_heads<A, R, NT>(v[0], ctx, L - LOG2R)) {
        for (int i = LOG2R; i < L; ++i) {
          int const sh = FWD ? i : LOG2R + L - 1 - i;
          Base::template coarse_level<A, R, NT>(
              v, ctx, 1 << (sh - LOG2R), typename Base::Passes{});
        }
      }
    };
    if constexpr (FWD) {
      Base::template fine_up<A, R, NT, 0>(v, ctx, L < KR ? L : KR);
      round();
      Base::template fine_up<A, R, NT, KR>(v, ctx, L);
      coarse();
    } else {
      coarse();
      fine_down_to<A, R, NT, LOG2R - 1>(v, ctx, L);
      round();
      Base::template fine_down<A, R, NT, KR - 1>(v, ctx, L);
    }
  }

 private:
  // Fine levels K .. KR.
  template <class A, int R, int NT, int K, class Ctx>
  static __device__ __forceinline__ void fine_down_to(typename A::V (&v)[R],
                                                      Ctx &ctx, int L) {
    if constexpr (K >= KR) {
      if (K < L)
        Base::template fine_level<A, R, NT, K>(v, ctx,
                                               typename Base::Passes{});
      fine_down_to<A, R, NT, K - 1>(v, ctx, L);
    }
  }
};

template <int W, bool FWD>
void launch_head_levels(int R, LiftParams const &p, cudaStream_t s) {
  if (R == kHeadsTile + kTile + 16)
    launch_tile_r<RowDF, 16, HeadSched<W, FWD>, false>(p, s);
  else
    launch_tile_r<RowDF, 16, HeadSched<W, FWD>, true>(p, s);
}

} // namespace

void launch_heads(int sched, int R, LiftParams p, long long total_tiles,
                  cudaStream_t s) {
  if (R == kHeadsIn || R == kHeadsOut) {
    long long const blocks = std::min(
        (((p.job.columns >> 2) << (p.job.log2_n - 4)) + kThreads - 1) /
            kThreads,
        16LL * device_sms());
    if (R == kHeadsOut)
      heads_kernel<true>
          <<<static_cast<unsigned>(blocks), kThreads, 0, s>>>(p.job);
    else
      heads_kernel<false>
          <<<static_cast<unsigned>(blocks), kThreads, 0, s>>>(p.job);
    cuda_check(cudaGetLastError(), "heads kernel launch");
    return;
  }
  p.jobs = nullptr;
  p.njobs = 1;
  p.total_tiles = total_tiles;
  p.rounds = kRounds;
  switch (sched) {
  case 0: return launch_head_levels<0, false>(R, p, s);
  case 1: return launch_head_levels<0, true>(R, p, s);
  case 2: return launch_head_levels<1, false>(R, p, s);
  case 3: return launch_head_levels<1, true>(R, p, s);
  case 4: return launch_head_levels<2, false>(R, p, s);
  case 5: return launch_head_levels<2, true>(R, p, s);
  }
  throw StatusError(2, "heads planned without a wavelet schedule");
}

} // namespace pgb
