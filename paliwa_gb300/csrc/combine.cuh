// Combination-technique kernels: FP64 combine of component-grid surpluses
// into sparse-grid subspaces, restriction of the combined subspaces back to
// the component grids, and scatter of the subspaces into a full grid.
//
// Restates the reference's test driver
// (test/test_paliwa_combination_technique.cpp): combine :256-290
// (subspace += coefficient * grid, FP64, grids in order), scatter :293-318
// (full grid += subspace). The subspace of level vector s is
// strided_hierarchical_domain_from_level(s, lmax) (paliwa_domains.hpp:51-83):
// per dimension 2^(s-1) points at uids 2^(L-s) + j * 2^(L-s+1), or the single
// point 0 at s = 0. Inside a grid at level l the same point has the compact
// index (2 j + 1) * 2^(l - s) (0 at s = 0).
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace pgb {

constexpr int kMaxDims = 12;

struct CtSubspace {
  long long offset;      // first sparse point of this subspace
  int grid_begin;        // range in the containing-grid list
  int grid_end;
  signed char level[kMaxDims];
};

struct __align__(16) CtGrid {
  unsigned long long base;  // byte address of the grid
  double coefficient;
  signed char level[kMaxDims];
  // log2 of level 0's element step along each dimension (the dimension's
  // extent times its stride), one byte each: level s steps step - s.
  unsigned step[kMaxDims / 4];
};

// Work of one combine CTA: nsub subspaces of 2^log2p points each (their ids
// at CtParams::order + order_first; all points of each), or, for a subspace
// of more than kCtBlock points, kCtBlock of its points from `local` on.
struct CtBlock {
  long long local;
  int order_first;
  int nsub;
  int log2p;    // points of each subspace held by the CTA
  int longest;  // longest grid list among its subspaces
};

struct CtParams {
  CtSubspace const *subspaces;
  int nsubspaces;
  int const *grid_lists;  // containing grids of each subspace, in grid order
  CtGrid const *grids;
  int ndim;
  long long npoints;       // sparse points in total
  double *sparse;          // combined values (FP64)
  double *full;            // full grid at the maximum level (scatter)
  signed char max_level[kMaxDims];
  // Every coefficient times every grid value is exact in FP64 (coefficients
  // of at most 29 significant bits and moderate magnitude on FP32 grids,
  // +-1 on FP64 grids): the combine then fuses multiply and add.
  int exact_products;
  // block_sub[b]: the subspace holding point kCtBlock * b (the first point
  // of CTA b of a thread-per-point kernel), planned on the host.
  int const *block_sub;
  // Combine: its CTAs and the subspace ids they refer to.
  CtBlock const *blocks;
  int const *order;
  // Restrict: the grid of every unit of ct_unit points, each grid's first
  // unit, and its families (see ct_restrict_kernel): families[
  // family_first[g] + index of (s_1 .. s_{d-1})].
  int const *unit_grid;
  long long const *unit_first;
  long long const *families;
  long long const *family_first;
  void const *values;  // the sparse values, in the grids' type or as doubles
};

// Points (threads) per CTA of the combine and scatter kernels.
constexpr int kCtBlock = 256;
// Grid descriptors staged per batch of a combine CTA.
constexpr int kCtStage = 256;
// Grid values a combine thread loads before it adds them, and the kernel's
// CTAs per SM (48 registers). Measured, 4D |l|_1 = 19 - q and 6D 16 - q, us:
// 8 values and 5 CTAs 1567 and 997, 4 and 5 1575 and 1090, 8 and 4 1776 and
// 1008, 4 and 6 1774 and 1147, 8 and 3 1975 and 1127.
constexpr int kCtAhead = 8;
constexpr int kCtCtas = 5;
// Subspaces of up to 2^kCtLog2Few points have the longest grid lists (those of
// one point every grid): their values are loaded by every thread of the CTA,
// since one thread with kCtAhead loads in flight took 2.0 ms for 7,798 grids.
constexpr int kCtLog2Few = 3;
// Whether ct_combine_direct_kernel takes a scheme (see there): short lists,
// and points enough to hide the longest.
inline bool ct_direct(size_t element, long long npoints, int longest) {
  return longest <= 48 &&
         npoints >= longest * (element == 8 ? 1LL << 15 : 1LL << 17);
}
// Subspaces of one combine CTA, at most, by their points: the fewer, the more
// grids a batch holds.
inline int ct_max_subs(int log2p) {
  return log2p <= 1 ? 2 : log2p <= kCtLog2Few ? 4 : 8;
}
// Groups of 4 grid points per restrict thread (floats, doubles), and points
// per CTA. Eight CTAs per SM (32 registers) hide the gathers: 4D |l|_1 = 19 -
// q in floats 970 us, with the compiler's choice of six 1110, 2 groups 1176, 8
// groups 1227; 17 - q in doubles 2 groups 289, 4 groups 372.
__host__ __device__ constexpr int ct_groups(size_t element) {
  return element == 8 ? 2 : 4;
}
__host__ __device__ constexpr int ct_unit(size_t element) {
  return 4 * ct_groups(element) * kCtBlock;
}
constexpr int kCtRestrictCtas = 8;

// A family is the subspaces (s_1 .. s_{d-1}, 0 .. top) of one leading level
// vector; they lie one after another in the sparse grid. Packed as the first
// sparse point in the low 56 bits and top + 1 above (0: none kept).
constexpr int kCtFamilyShift = 56;

// float -> double without the conversion instruction, which on GB300 runs
// on the FP64 pipe: the double is the float's sign, exponent rebiased by
// 1023 - 127 and fraction shifted by 29 bits (the exact value). Subnormals are
// scaled by 2^24 first, zeros, infinities and NaNs keep their own exponent
// field. No branch holds a conversion: the compiler runs a short one for
// every value under a predicate, and one conversion per value doubled the
// combine's FP64 work.
__device__ __forceinline__ double widen(float x) {
  unsigned u = __float_as_uint(x);
  unsigned const a = u & 0x7fffffffu;
  unsigned bias = (1023u - 127u) << 20;
  if (a < 0x00800000u) {
    u = __float_as_uint(__fmul_rn(x, 16777216.0f));
    bias -= a == 0u ? bias : 24u << 20;
  }
  unsigned hi = ((u & 0x7fffffffu) >> 3) + bias;
  if (a >= 0x7f800000u) hi |= 0x7ff00000u;
  return __hiloint2double(static_cast<int>(hi | (u & 0x80000000u)),
                          static_cast<int>(u << 29));
}
__device__ __forceinline__ double widen(double x) { return x; }

// Multi-index of point `p` of subspace `sub` -> compact index inside a grid
// at level `lv` (element offset, row-major, last dimension fastest).
__device__ __forceinline__ long long ct_offset(long long p,
                                              signed char const *s,
                                              signed char const *lv,
                                              int ndim) {
  long long off = 0;
  int shift = 0;  // log2 of the element stride of the current dimension
  for (int d = ndim - 1; d >= 0; --d) {
    int const sd = s[d];
    int const ld = lv[d];
    int const ext_log2 = sd == 0 ? 0 : sd - 1;  // 2^(s-1) points, 1 at s=0
    long long const j = p & ((1LL << ext_log2) - 1);
    p >>= ext_log2;
    long long const k = sd == 0 ? 0 : ((2 * j + 1) << (ld - sd));
    off += k << shift;
    shift += ld;
  }
  return off;
}

// Combine: sparse[p] = sum over the containing grids, in grid order, of
// coefficient * value in FP64 (with exact products fma(c, v, acc) rounds
// like the reference driver's separate multiply and add, and issues one FP64
// instruction instead of two).
//
// The floor is one FP64 update per contained grid value: about two lane
// operations per clock and SM, 0.45 ms for the 273 M values of 4D |l|_1 =
// 18 - q, behind one scattered load each. A CTA takes points of subspaces of
// one size (a few subspaces, so that small ones fill its warps) and walks
// their grid lists in batches: every thread stages one descriptor (address,
// coefficient and the element step of each dimension) in shared memory, then
// each point's thread forms its addresses with one multiply-add per dimension
// and keeps kCtAhead loads in flight. Measured (FP32 grids), against a thread
// that walked list entry -> grid -> value by itself and converted each value
// on the FP64 pipe: 4D |l|_1 = 19 - q 3.60 -> 1.57 ms, 20 - q 8.5 -> 3.7, 6D
// 16 - q 7.5 -> 1.0.
template <typename S, int ND, bool Fused, bool Big>
__global__ void __launch_bounds__(kCtBlock, kCtCtas)
    ct_combine_kernel(CtParams const p) {
  using Mult = typename std::conditional<Big, unsigned long long,
                                         unsigned>::type;
  // One descriptor: 16-byte reads, one wavefront each (the lanes of a warp
  // read the same one, or a few).
  struct __align__(16) Desc {
    unsigned long long base;
    double coef;
    Mult mult[ND];
  };
  __shared__ Desc s_desc[kCtStage];
  __shared__ S s_value[1 << kCtLog2Few][kCtStage];
  int const t = threadIdx.x;
  CtBlock const blk = p.blocks[blockIdx.x];
  int const pi = t & ((1 << blk.log2p) - 1);
  int const si = t >> blk.log2p;
  bool const active = si < blk.nsub;
  // Batch: kCtStage / (subspaces rounded up to a power of two) grids each.
  int const log2subs = blk.nsub <= 1 ? 0 : 32 - __clz(blk.nsub - 1);
  int const log2k = 31 - __clz(kCtStage) - log2subs;
  int const K = 1 << log2k;
  // This thread's point, as odd multiples m_d of each dimension's step.
  int len = 0;
  long long point = 0;
  unsigned m[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) m[d] = 0;
  if (active) {
    CtSubspace const &ss = p.subspaces[p.order[blk.order_first + si]];
    len = ss.grid_end - ss.grid_begin;
    long long r = blk.local + pi;
    point = ss.offset + r;
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      int const sd = d < p.ndim ? ss.level[d] : 0;
      if (sd == 0) continue;
      m[d] = 2 * static_cast<unsigned>(r & ((1LL << (sd - 1)) - 1)) + 1;
      r >>= sd - 1;
    }
  }
  // The subspace whose grids this thread stages.
  int const st = t >> log2k;
  int st_begin = 0, st_end = 0;
  unsigned st_level[ND / 4];  // its levels, 4 dimensions per word
#pragma unroll
  for (int w = 0; w < ND / 4; ++w) st_level[w] = 0;
  if (st < blk.nsub) {
    CtSubspace const &ss = p.subspaces[p.order[blk.order_first + st]];
    st_begin = ss.grid_begin + (t & (K - 1));
    st_end = ss.grid_end;
#pragma unroll
    for (int w = 0; w < ND / 4; ++w)
      st_level[w] = reinterpret_cast<unsigned const *>(ss.level)[w];
  }
  double acc = 0.0;
  bool const staged = blk.log2p <= kCtLog2Few;
  for (int k0 = 0; k0 < blk.longest; k0 += K) {
    if (k0 > 0) __syncthreads();  // the last batch is done with
    if (st_begin + k0 < st_end) {
      CtGrid const &g = p.grids[p.grid_lists[st_begin + k0]];
      Desc desc;
      desc.base = g.base;
      desc.coef = g.coefficient;
      unsigned step[ND / 4];  // 4 dimensions' step bytes per word
#pragma unroll
      for (int w = 0; w < ND / 4; ++w) step[w] = g.step[w];
#pragma unroll
      for (int d = 0; d < ND; ++d)
        desc.mult[d] = static_cast<Mult>(1)
                       << (((step[d / 4] - st_level[d / 4]) >> (8 * (d % 4))) &
                           63u);
      s_desc[t] = desc;
      if (staged) {
        S const *const from = reinterpret_cast<S const *>(desc.base);
        S x[1 << kCtLog2Few];
#pragma unroll
        for (int i = 0; i < (1 << kCtLog2Few); ++i) {
          if (i >> blk.log2p) break;
          unsigned long long off = 0;
          unsigned r = static_cast<unsigned>(i);
#pragma unroll
          for (int d = ND - 1; d >= 0; --d) {
            unsigned const sd = (st_level[d / 4] >> (8 * (d % 4))) & 63u;
            if (sd == 0) continue;
            off += static_cast<unsigned long long>(
                       2 * (r & ((1u << (sd - 1)) - 1)) + 1) * desc.mult[d];
            r >>= sd - 1;
          }
          x[i] = from[off];
        }
#pragma unroll
        for (int i = 0; i < (1 << kCtLog2Few); ++i)
          if (!(i >> blk.log2p)) s_value[i][t] = x[i];
      }
    }
    __syncthreads();
    int const n = min(K, len - k0);
    int const e0 = si << log2k;
    auto add = [&](double coef, S x) {
      double const v = widen(x);
      if constexpr (Fused)
        acc = __fma_rn(coef, v, acc);
      else
        acc = __dadd_rn(acc, __dmul_rn(coef, v));
    };
    if (staged) {
      for (int k = 0; k < n; ++k)
        add(s_desc[e0 + k].coef, s_value[pi][e0 + k]);
      continue;
    }
    auto value = [&](int e, double &coef) {
      Desc const desc = s_desc[e];
      unsigned long long off = 0;
#pragma unroll
      for (int d = 0; d < ND; ++d)
        off += static_cast<unsigned long long>(m[d]) * desc.mult[d];
      coef = desc.coef;
      return reinterpret_cast<S const *>(desc.base)[off];
    };
    int k = 0;
    for (; k + kCtAhead <= n; k += kCtAhead) {
      S x[kCtAhead];
      double c[kCtAhead];
#pragma unroll
      for (int i = 0; i < kCtAhead; ++i) x[i] = value(e0 + k + i, c[i]);
#pragma unroll
      for (int i = 0; i < kCtAhead; ++i) add(c[i], x[i]);
    }
    for (; k < n; ++k) {
      double c;
      S const x = value(e0 + k, c);
      add(c, x);
    }
  }
  if (active) p.sparse[point] = acc;
}

// The sparse values in the grids' type, converted once per point: a
// conversion per grid value would take the FP64 pipe as long as the combine
// (and gather twice the bytes: 4D |l|_1 = 19 - q with lmin 2 365 us, 499
// converting as it gathers). Sparse grids of fewer points are converted as
// they are gathered: this launch would be what they wait for (up to 2^17
// points 1.3-2.2 us faster without, never slower; from 2^18 on either side).
constexpr long long kCtNarrow = 1LL << 17;
__global__ void __launch_bounds__(kCtBlock)
    ct_narrow_kernel(double const *in, float *out, long long n) {
  long long const step = static_cast<long long>(gridDim.x) * kCtBlock;
  for (long long i = static_cast<long long>(blockIdx.x) * kCtBlock +
                     threadIdx.x;
       i < n; i += step)
    out[i] = static_cast<float>(in[i]);
}

// Restrict: every grid point whose subspace is kept takes its combined value.
//
// Bound by memory: each grid is written once, in storage order, and the
// sparse values are gathered. (Written from the sparse side, one thread per
// sparse point over its grids, every store touched a 32-byte sector for 4
// bytes: 4D |l|_1 = 19 - q 3.17 -> 0.97 ms, 20 - q 7.7 -> 2.3, 6D 16 - q
// 2.65 -> 0.64.) Thread = 4 consecutive points 4 a .. 4 a + 3 of a last-axis row:
// levels l, l - 1, l and, for 4 a, whatever its trailing zeros say, so a warp
// gathers a few contiguous runs. The leading indices name the row's family,
// whose first point and kept levels come from a table per grid. ND: the
// dimensions (kMaxDims: any number); I: the type of point indices (32 bits
// where the grid and the sparse grid allow it: the index arithmetic issues on
// 80 % of the cycles otherwise).
template <int ND, typename I> struct CtRows {
  int lv[ND];     // levels of the leading dimensions and the last
  int radix[ND];  // of the family index
  long long const *families;
  int nd;

  __device__ __forceinline__ CtRows(CtParams const &p, int g) {
    nd = ND < kMaxDims ? ND : p.ndim;
    families = p.families + p.family_first[g];
    int r = 1;
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      lv[d] = d < nd ? p.grids[g].level[d] : 0;
      radix[d] = r;
      if (d < nd - 1) r *= lv[d] + 1;
    }
  }
  __device__ __forceinline__ int last() const {
    int l = lv[0];
#pragma unroll
    for (int d = 1; d < ND; ++d)
      if (d == nd - 1) l = lv[d];
    return l;
  }
};

// A row of the grid along its last axis.
template <typename I> struct CtRow {
  I base;   // first sparse point of its family
  I fam;    // points of the family at its coarsest level
  I pos;    // the row among them
  int top;  // highest kept level of the last axis (-1: none)

  template <int ND>
  __device__ __forceinline__ CtRow(CtRows<ND, I> const &rows, I row) {
    int fi = 0, log2fam = 0;
    pos = 0;
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
      if (d >= rows.nd - 1) continue;
      int const l = rows.lv[d];
      unsigned const k = static_cast<unsigned>(row) & ((1u << l) - 1);
      row >>= l;
      int const tz = __ffs(k | (1u << l)) - 1;
      int const s = l - tz;  // k = 0: tz = l, level 0
      fi += s * rows.radix[d];
      pos += static_cast<I>((k >> tz) >> 1) << log2fam;
      log2fam += max(s - 1, 0);
    }
    long long const e = rows.families[fi];
    base = static_cast<I>(e & ((1LL << kCtFamilyShift) - 1));
    top = static_cast<int>(e >> kCtFamilyShift) - 1;
    fam = static_cast<I>(1) << log2fam;
  }
  // Sparse point j of level s >= 1 of the row.
  __device__ __forceinline__ I at(int s, unsigned j) const {
    return base + ((fam + pos) << (s - 1)) + j;
  }
  // Sparse point of last-axis index k (its level in s).
  __device__ __forceinline__ I of(unsigned k, int l, int &s) const {
    int const tz = __ffs(k | (1u << l)) - 1;
    s = l - tz;
    return s == 0 ? base + pos : at(s, (k >> tz) >> 1);
  }
};

template <typename S, int ND, typename I, typename V>
__global__ void __launch_bounds__(kCtBlock, kCtRestrictCtas)
    ct_restrict_kernel(CtParams const p) {
  constexpr int GROUPS = ct_groups(sizeof(S));
  constexpr int UNIT = ct_unit(sizeof(S));
  int const g = p.unit_grid[blockIdx.x];
  CtRows<ND, I> const rows(p, g);
  unsigned long long const base = p.grids[g].base;
  S *const out = reinterpret_cast<S *>(base);
  V const *const values = reinterpret_cast<V const *>(p.values);
  auto val = [&](I at) { return static_cast<S>(values[at]); };
  int total = 0;
#pragma unroll
  for (int d = 0; d < ND; ++d) total += rows.lv[d];
  I const n = static_cast<I>(1) << total;
  int const l = rows.last();
  I const first =
      static_cast<I>(blockIdx.x - p.unit_first[g]) * UNIT + 4 * threadIdx.x;
  if (l >= 2) {
    bool const vec = (base & 15) == 0;
    S v[GROUPS][4];
    unsigned keep[GROUPS];
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
      I const f = first + q * 4 * kCtBlock;
      keep[q] = 0;
      if (f >= n) continue;
      CtRow<I> const r(rows, f >> l);
      unsigned const k = static_cast<unsigned>(f) & ((1u << l) - 1);
      int s;
      I const at0 = r.of(k, l, s);
      if (s <= r.top) {
        v[q][0] = val(at0);
        keep[q] = 1;
      }
      if (l - 1 <= r.top) {
        v[q][2] = val(r.at(l - 1, k >> 2));
        keep[q] |= 4;
      }
      if (l <= r.top) {
        I const at1 = r.at(l, k >> 1);
        v[q][1] = val(at1);
        v[q][3] = val(at1 + 1);
        keep[q] |= 10;
      }
    }
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
      S *const to = out + first + q * 4 * kCtBlock;
      if (keep[q] == 15u && vec) {
        constexpr int PER = 16 / sizeof(S);
#pragma unroll
        for (int i = 0; i < 4; i += PER) {
          uint4 u;
          memcpy(&u, &v[q][i], 16);
          *reinterpret_cast<uint4 *>(to + i) = u;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if ((keep[q] >> i) & 1u) to[i] = v[q][i];
      }
    }
    return;
  }
  // Rows of one or two points: each point has a row of its own. (Four points'
  // loads at once: one after another 2D grids of 2^17 points in such rows took
  // 8.3 us, 6.4 so.)
  for (int q = 0; q < GROUPS; ++q) {
    S v[4];
    unsigned keep = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      I const f = first + q * 4 * kCtBlock + i;
      if (f >= n) continue;
      CtRow<I> const r(rows, f >> l);
      int s;
      I const at = r.of(static_cast<unsigned>(f) & ((1u << l) - 1), l, s);
      if (s > r.top) continue;
      v[i] = val(at);
      keep |= 1u << i;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((keep >> i) & 1u) out[first + q * 4 * kCtBlock + i] = v[i];
  }
}

// The subspace of sparse point `point` of CTA blockIdx.x (kCtBlock points
// each). The CTA's first subspace comes from the host's table. Most CTAs lie
// inside one subspace: one load settles that. Otherwise the CTA's 256 points
// span at most 256 subspaces (each has at least one point): a binary search
// over those.
__device__ __forceinline__ CtSubspace const &
ct_subspace_of(CtParams const &p, long long point) {
  int const sub0 = p.block_sub[blockIdx.x];
  int sub = sub0;
  if (sub0 + 1 < p.nsubspaces && p.subspaces[sub0 + 1].offset <= point) {
    int lo = sub0 + 1;
    int hi = min(sub0 + kCtBlock - 1, p.nsubspaces - 1);
    while (lo < hi) {
      int const mid = (lo + hi + 1) >> 1;
      if (p.subspaces[mid].offset <= point)
        lo = mid;
      else
        hi = mid - 1;
    }
    sub = lo;
  }
  return p.subspaces[sub];
}

// Combine with few grids: a thread per sparse point walks its grid list
// itself. The packed kernel above waits out a chain of loads (work item,
// subspace, list, grid, value) per CTA, at five CTAs per SM; where the lists
// are short there is little else, and this one runs more CTAs. Measured in 2D,
// us, packed against direct: FP64 17 grids, 1.1 M points 23.3 and 18.6, 43
// grids, 11.5 M 309 and 272; FP32 3 grids, 3.1 M 26.6 and 20.9, 35 grids, 5.0
// M 87.5 and 76.9. But FP64 25 grids, 0.46 M 10.7 and 15.6, FP32 19 grids, 0.7
// M 13.0 and 14.9: the few points of the coarse subspaces then walk all grids.
template <typename S, bool Fused>
__global__ void __launch_bounds__(kCtBlock) ct_combine_direct_kernel(
    CtParams const p) {
  long long const point =
      static_cast<long long>(blockIdx.x) * kCtBlock + threadIdx.x;
  if (point >= p.npoints) return;
  CtSubspace const &ss = ct_subspace_of(p, point);
  double acc = 0.0;
  for (int gi = ss.grid_begin; gi < ss.grid_end; ++gi) {
    CtGrid const &g = p.grids[p.grid_lists[gi]];
    long long const off =
        ct_offset(point - ss.offset, ss.level, g.level, p.ndim);
    double const v = widen(reinterpret_cast<S const *>(g.base)[off]);
    if constexpr (Fused)
      acc = __fma_rn(g.coefficient, v, acc);
    else
      acc = __dadd_rn(acc, __dmul_rn(g.coefficient, v));
  }
  p.sparse[point] = acc;
}

// Scatter: full[p] += sparse[p] on the full grid at the maximum level.
__global__ void __launch_bounds__(kCtBlock) ct_scatter_kernel(
    CtParams const p) {
  long long const point =
      static_cast<long long>(blockIdx.x) * kCtBlock + threadIdx.x;
  if (point >= p.npoints) return;
  CtSubspace const &ss = ct_subspace_of(p, point);
  long long const off =
      ct_offset(point - ss.offset, ss.level, p.max_level, p.ndim);
  p.full[off] = __dadd_rn(p.full[off], p.sparse[point]);
}

} // namespace pgb
