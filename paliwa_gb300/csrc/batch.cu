// Batched transforms of many component grids and the combination-technique
// combine / restrict / scatter (include/paliwa_gb300.h).
//
// The reference transforms the component grids of a combination scheme one
// hierarchize() call each, spread over execution-space instances
// (test/test_paliwa_combination_technique.cpp:164-174). Here one plan covers
// every grid: for each axis, the per-grid stages of plan_axis() are merged
// into one launch per stage index and chunk size, whose device-side job list
// names every grid. The grids are dealt into up to kBatchGroups groups of
// about equal size, each planned on its own; a direction's launch sequences
// of the groups run on parallel branches (forked streams, joined at the
// end), so one group's launches fill the tails of another's and kernels of
// different kinds share the GPU. The whole direction is captured once into a
// CUDA graph and replayed.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <unordered_map>
#include <vector>

#include "combine.cuh"
#include "paliwa_gb300.h"
#include "plan.hpp"
#include "slab_plan.hpp"
#include "twide_plan.hpp"

using namespace pgb;

namespace {

// Groups of grids planned and run on parallel branches. Measured on the 4D
// CT workload (3,025 grids, FP32c, forward + inverse): 28.7 ms with one
// group, 26.1 with two, 25.7 with three, 25.6 with four.
constexpr int kBatchGroups = 4;

// Kernel code of a slab launch (slab.cuh); the others are plan.hpp's and
// twide_plan.hpp's.
constexpr int kSlab = 1024;

struct Launch {
  int group = 0;
  int R = 0;
  int sched = -1;
  size_t job_first = 0;  // index into the device job array
  size_t tile_first = 0;  // slab launches: index into the tile-job table
  int njobs = 0;
  long long tiles = 0;
  long long points = 0;  // grid points stored by this launch
  bool pairs = false;    // slab launches: some job is worth pairs
};

struct Direction {
  LiftParams params{};
  bool exact = true;
  bool symmetric = true;
  std::vector<Launch> launches;
  LiftJob *jobs_dev = nullptr;
  SlabJob *slab_dev = nullptr;  // jobs of the slab launches
  int *slab_tile_dev = nullptr;  // job of every tile of the slab launches
  // TMA wide launches: jobs, the job of every tile, the tensor maps.
  TWideJob *twide_dev = nullptr;
  int *twide_tile_dev = nullptr;
  CUtensorMap *maps_dev = nullptr;
  cudaGraphExec_t graph = nullptr;
  Tuning tuning;  // kernel forced per class (autotuner)
  // Slab launches where they apply (default_slabs, or the batch's setting);
  // the autotuner takes the other choice when the direction runs faster so.
  bool slabs = true;
  // TMA wide launches for the stages planned on them (the batch's setting).
  bool tma = true;
  // Classes of the plan's periodic stages: applicable kernels (bits), the
  // default choice of the first stage seen, and the points they store.
  struct ClassInfo {
    unsigned kernels = 0;
    int dflt = 0;
    long long points = 0;
  };
  std::map<int, ClassInfo> classes;
};

void free_direction(Direction &d) {
  if (d.graph) cudaGraphExecDestroy(d.graph);
  if (d.jobs_dev) cudaFree(d.jobs_dev);
  if (d.slab_dev) cudaFree(d.slab_dev);
  if (d.slab_tile_dev) cudaFree(d.slab_tile_dev);
  if (d.twide_dev) cudaFree(d.twide_dev);
  if (d.twide_tile_dev) cudaFree(d.twide_tile_dev);
  if (d.maps_dev) cudaFree(d.maps_dev);
  d.slab_tile_dev = nullptr;
  d.twide_dev = nullptr;
  d.twide_tile_dev = nullptr;
  d.maps_dev = nullptr;
  d.graph = nullptr;
  d.jobs_dev = nullptr;
  d.slab_dev = nullptr;
  d.launches.clear();
  d.classes.clear();
}

void check_grid_levels(int ndim, int ngrids, int64_t const *levels,
                       int64_t const *lmin, int64_t const *lmax) {
  if (ndim < 1 || ndim > kMaxDims)
    throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "ndim must be in [1, 12]");
  if (ngrids < 1)
    throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "no grids");
  for (int g = 0; g < ngrids; ++g) {
    int64_t total = 0;
    for (int d = 0; d < ndim; ++d) {
      int64_t const l = levels[g * ndim + d];
      if (l < 0 || l > lmax[d] || lmax[d] > 30 ||
          (lmin != nullptr && (lmin[d] < 0 || lmin[d] > l)))
        throw StatusError(
            PALIWA_GB_INVALID_ARGUMENT,
            "requires 0 <= minimum_level <= level <= maximum_level <= 30");
      total += l;
    }
    if (total > 40)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "grid too large");
  }
}

} // namespace

struct paliwa_gb_batch {
  int ndim = 0;
  int ngrids = 0;
  int dtype = 0;
  int wavelet = 0;
  long long points = 0;
  bool use_graphs = true;
  Direction dir[2];  // 0 = forward, 1 = inverse
  // The grids as created (for re-planning).
  std::vector<int64_t> levels, lmin;
  std::vector<void *> grids;
  // Halo buffers of the windowed stages (grids with pencils longer than one
  // CTA holds; a region of the grid's size per grid and axis), reused by
  // every axis of a group (a group's axes run in order); the groups, which
  // run concurrently, have disjoint regions.
  void *shadow = nullptr;
  size_t shadow_bytes = 0;
  // group[g]: the group of grid g; group_shadow[k]: byte offset of group
  // k's shadow region. Group k > 0 runs on streams[k - 1] (non-blocking),
  // forked from and joined into the caller's stream with events.
  int ngroups = 1;
  std::vector<int> group;
  std::vector<size_t> group_shadow;
  std::vector<cudaStream_t> streams;
  std::vector<cudaEvent_t> events;  // [0] fork, [k] join of group k
  // Slab launches (slab.cuh): the tensor map over the grids' memory as
  // 128-byte rows from slab_base, and the error word of their bounded waits.
  bool use_slabs = true;
  // TMA wide launches for the stages planned on them.
  bool use_tma = true;
  bool slab_map_ok = false;
  unsigned long long slab_base = 0;
  CUtensorMap slab_map{};
  unsigned *slab_error = nullptr;
  // Cap on the CTAs per SM of every launch (0: as many as fit).
  int ctas_per_sm = 0;
};

namespace {

// Whether a new batch plans slabs. They save launches, which is what small
// batches spend their time on (us, there and back, CDF (2,2): FP32c 6D |l|_1 =
// 12 - q, 2.6 M points, 67 against 240, 4D 15 - q, 19 M, 485 against 512; FP64
// 6D 12 - q 137 against 387, 4D 13 - q, 2.8 M, 320 against 335), but their
// axes are bound by barriers and latencies at about half the TMA wide kernel's
// rate for double and double-float arithmetic: FP64 from about 2^22 points on
// (4D 14 - q, 7.4 M: 597 against 518) and FP32c somewhere from 2^25 on (6D 14
// - q, 30 M: 515 against 742; 4D 16 - q, 48 M: 1040 against 1052; 5D 16 - q,
// 139 M: 2109 against 2006) are faster axis by axis. Plain FP32 is bound by
// memory either way and takes slabs throughout (5D 16 - q 1425 against 1697;
// 4D 18 - q 3108 against 3109).
bool default_slabs(int dtype, long long points) {
  switch (dtype) {
  case PALIWA_GB_F64: return points <= 1LL << 22;
  case PALIWA_GB_F32C: return points <= 1LL << 25;
  }
  return true;
}

// The tensor map over every grid of the batch (rows of 128 bytes from the
// lowest grid address, rounded down to 128 bytes).
void setup_slab_map(paliwa_gb_batch &b) {
  b.slab_map_ok = false;
  size_t const es = dtype_size(b.dtype);
  unsigned long long lo = ~0ULL, hi = 0;
  for (int g = 0; g < b.ngrids; ++g) {
    unsigned long long const a = reinterpret_cast<unsigned long long>(b.grids[g]);
    unsigned long long bytes = es;
    for (int d = 0; d < b.ndim; ++d) bytes <<= b.levels[g * b.ndim + d];
    lo = std::min(lo, a);
    hi = std::max(hi, a + bytes);
  }
  lo &= ~127ULL;
  b.slab_base = lo;
  b.slab_map_ok = encode_slab_map(&b.slab_map, lo, (hi - lo + 127) / 128, es);
}

void plan_direction(paliwa_gb_batch &b, Direction &dr, bool forward,
                    int64_t const *levels, int64_t const *lmin,
                    void *const *grid_ptrs) {
  auto const filters = wavelet_filters(b.wavelet, forward);
  dr.params = launch_params(filters);
  dr.exact = exact_scalers(filters);
  dr.symmetric = symmetric_filters(filters);
  std::vector<LiftJob> all_jobs;
  std::vector<SlabJob> all_slabs;
  std::vector<int> slab_tiles;  // per slab launch tile: its job in the launch
  std::vector<TWideJob> all_twide;
  std::vector<int> twide_tiles;  // per TMA wide launch tile: its job
  std::vector<CUtensorMap> maps;
  size_t const es = dtype_size(b.dtype);
  int const ws = wavelet_schedule(filters);
  bool const tma =
      b.use_tma && dr.tma && ws >= 0 && tensor_map_encoder() != nullptr;
  // First axis of every grid's slab group (ndim: none). A lone grid's only
  // axis saves no launch there, and its threads hold longer chunks than in its
  // own kernel (us: FP64 2^8 points, CDF (2,2), 14.4 against 6.2, FP32c hat
  // 6.2 against 4.2).
  std::vector<int> slab_from(b.ngrids, b.ndim);
  if (b.use_slabs && dr.slabs && b.slab_map_ok && ws >= 0)
    for (int g = 0; g < b.ngrids; ++g) {
      int64_t const *lv = levels + static_cast<size_t>(g) * b.ndim;
      int work = 0;
      for (int d = 0; d < b.ndim; ++d) work += lv[d] > lmin[d];
      if (b.ngrids == 1 && work == 1) continue;
      slab_from[g] = slab_start(
          b.dtype, b.ndim, lv, lmin,
          reinterpret_cast<unsigned long long>(b.grids[g]), b.slab_base);
    }
  for (int grp = 0; grp < b.ngroups; ++grp) {
    std::vector<int> members;
    for (int g = 0; g < b.ngrids; ++g)
      if (b.group[g] == grp) members.push_back(g);
    for (int d = 0; d < b.ndim; ++d) {
      // stages[i] = the ordered stages of grid members[i] along axis d
      std::vector<std::vector<Stage>> stages(members.size());
      size_t depth = 0;
      size_t shadow_off = b.group_shadow[grp];
      for (size_t i = 0; i < members.size(); ++i) {
        int const g = members[i];
        int64_t const *lv = levels + static_cast<size_t>(g) * b.ndim;
        // In the grid's slab launch; a single axis there (slab_start) still
        // has its class, and a kernel that is chosen for it (tuning) runs it.
        int work = 0;
        for (int k = 0; k < b.ndim; ++k) work += lv[k] > lmin[k];
        bool const in_slab = d >= slab_from[g];
        if (in_slab && (work > 1 || lv[d] == lmin[d])) continue;
        AxisView view =
            axis_view(reinterpret_cast<unsigned long long>(grid_ptrs[g]),
                      b.ndim, lv, d, b.dtype);
        auto const shifts = level_shifts(lv[d], lmin[d], forward);
        if (needs_shadow(view, shifts)) {
          size_t bytes = es;
          for (int k = 0; k < b.ndim; ++k) bytes <<= lv[k];
          if (shadow_off + bytes > b.shadow_bytes)
            throw StatusError(PALIWA_GB_RUNTIME_ERROR,
                              "shadow plan overflow");
          view.shadow =
              reinterpret_cast<unsigned long long>(b.shadow) + shadow_off;
          shadow_off += (bytes + 255) / 256 * 256;
        }
        plan_axis(view, shifts, filters, stages[i], &dr.tuning);
        for (Stage const &st : stages[i]) {
          if (st.kernels == 0) continue;
          auto &ci = dr.classes[st.tclass];
          if (ci.kernels == 0) {
            ci.kernels = st.kernels;
            ci.dflt = st.dflt;
          }
          ci.points += st.job.columns << st.job.log2_n;
        }
        if (in_slab) {
          bool chosen = false;
          for (Stage const &st : stages[i])
            chosen |= st.kernels != 0 && dr.tuning.choice.count(st.tclass) != 0;
          if (chosen)
            slab_from[g] = b.ndim;
          else
            stages[i].clear();
        }
        depth = std::max(depth, stages[i].size());
      }
      for (size_t k = 0; k < depth; ++k) {
        // One launch per chunk size among the k-th stages of the group;
        // strided wide stages that qualify go to the TMA wide kernel.
        std::map<int, std::vector<Stage const *>> by_r;
        for (size_t i = 0; i < members.size(); ++i)
          if (k < stages[i].size()) {
            Stage const &st = stages[i][k];
            int code = st.R;
            if (tma && canonical_shifts(st.job, (ws & 1) != 0)) {
              int const form = twide_code(st, b.dtype);
              if (form != 0) code = kTWide + form;
            }
            by_r[code].push_back(&st);
          }
        // TMA wide launches: stages that do not qualify, and all of a form
        // that are too few points together, join the launches of their own
        // kernels (3D |l|_1 = 4 - q with lmin 0, FP64: 37 launches, 43 where
        // they had launches to themselves).
        std::vector<Launch> wide;
        for (auto it = by_r.upper_bound(kTWide); it != by_r.end();
             it = by_r.erase(it)) {
          auto const &[R, list] = *it;
          Launch L;
          L.group = grp;
          L.R = R;
          L.sched = ws;
          L.job_first = all_twide.size();
          L.tile_first = twide_tiles.size();
          long long points = 0;
          bool tuned = false;
          for (Stage const *st : list) {
            points += stage_points(*st);
            tuned |= st->tuned;
          }
          bool const enough =
              tuned || twide_enough(R - kTWide, b.dtype, points);
          for (Stage const *st : list) {
            TWideJob job;
            CUtensorMap map[2];
            long long tiles = 0;
            if (!enough || !twide_job(*st, b.dtype, job, map, tiles)) {
              by_r[st->R].push_back(st);
              continue;
            }
            job.tile_begin = L.tiles;
            job.map = static_cast<int>(maps.size());
            maps.push_back(map[0]);
            if (st->box && job.win.seg_len > 0) {
              job.win.halo_map = job.map + 1;
              maps.push_back(map[1]);
            }
            all_twide.push_back(job);
            twide_tiles.insert(twide_tiles.end(), tiles, L.njobs);
            L.tiles += tiles;
            L.points += stage_points(*st);
            ++L.njobs;
          }
          if (L.njobs > 0) wide.push_back(L);
        }
        for (auto const &[R, list] : by_r) {
          Launch L;
          L.group = grp;
          L.R = R;
          L.sched = ws;
          for (Stage const *st : list)
            if (ws < 0 || !canonical_shifts(st->job, (ws & 1) != 0))
              L.sched = -1;
          L.job_first = all_jobs.size();
          L.njobs = static_cast<int>(list.size());
          for (Stage const *st : list) {
            LiftJob job = st->job;
            job.tile_begin = L.tiles;
            L.tiles += st->tiles;
            L.points += stage_points(*st);
            all_jobs.push_back(job);
          }
          if (L.R != 0 && L.tiles > 0) dr.launches.push_back(L);
        }
        dr.launches.insert(dr.launches.end(), wide.begin(), wide.end());
      }
    }
    // The group's slab launch, after every per-axis stage of its grids.
    Launch L;
    L.group = grp;
    L.R = kSlab;
    L.sched = ws;
    L.job_first = all_slabs.size();
    L.tile_first = slab_tiles.size();
    for (int g : members) {
      if (slab_from[g] >= b.ndim) continue;
      SlabJob job = slab_job(
          b.dtype, b.ndim, slab_from[g],
          levels + static_cast<size_t>(g) * b.ndim, lmin,
          reinterpret_cast<unsigned long long>(grid_ptrs[g]), b.slab_base);
      job.tile_begin = L.tiles;
      int64_t total = 0;
      for (int k = 0; k < b.ndim; ++k) total += levels[g * b.ndim + k];
      long long const tiles = 1LL << (total - job.log2_tile);
      slab_tiles.insert(slab_tiles.end(), tiles, L.njobs);
      L.tiles += tiles;
      L.points += 1LL << total;
      L.pairs |= slab_pairs(job);
      all_slabs.push_back(job);
      ++L.njobs;
    }
    if (L.njobs > 0) dr.launches.push_back(L);
  }
  if (!all_slabs.empty()) {
    size_t const bytes = all_slabs.size() * sizeof(SlabJob);
    cuda_check(cudaMalloc(&dr.slab_dev, bytes), "cudaMalloc(slab jobs)");
    cuda_check(cudaMemcpy(dr.slab_dev, all_slabs.data(), bytes,
                          cudaMemcpyHostToDevice),
               "cudaMemcpy(slab jobs)");
    size_t const tbytes = slab_tiles.size() * sizeof(int);
    cuda_check(cudaMalloc(&dr.slab_tile_dev, tbytes),
               "cudaMalloc(slab tiles)");
    cuda_check(cudaMemcpy(dr.slab_tile_dev, slab_tiles.data(), tbytes,
                          cudaMemcpyHostToDevice),
               "cudaMemcpy(slab tiles)");
  }
  if (!all_twide.empty()) {
    size_t const jb = all_twide.size() * sizeof(TWideJob);
    cuda_check(cudaMalloc(&dr.twide_dev, jb), "cudaMalloc(twide jobs)");
    cuda_check(cudaMemcpy(dr.twide_dev, all_twide.data(), jb,
                          cudaMemcpyHostToDevice),
               "cudaMemcpy(twide jobs)");
    size_t const tb = twide_tiles.size() * sizeof(int);
    cuda_check(cudaMalloc(&dr.twide_tile_dev, tb), "cudaMalloc(twide tiles)");
    cuda_check(cudaMemcpy(dr.twide_tile_dev, twide_tiles.data(), tb,
                          cudaMemcpyHostToDevice),
               "cudaMemcpy(twide tiles)");
    size_t const mb = maps.size() * sizeof(CUtensorMap);
    cuda_check(cudaMalloc(&dr.maps_dev, mb), "cudaMalloc(tensor maps)");
    cuda_check(cudaMemcpy(dr.maps_dev, maps.data(), mb,
                          cudaMemcpyHostToDevice),
               "cudaMemcpy(tensor maps)");
  }
  if (!all_jobs.empty()) {
    size_t const bytes = all_jobs.size() * sizeof(LiftJob);
    cuda_check(cudaMalloc(&dr.jobs_dev, bytes), "cudaMalloc(jobs)");
    cuda_check(cudaMemcpy(dr.jobs_dev, all_jobs.data(), bytes,
                          cudaMemcpyHostToDevice),
               "cudaMemcpy(jobs)");
  }
}

// One launch of a direction's plan: a lifting kernel or a slab kernel.
void launch_one(paliwa_gb_batch &b, Direction &dr, Launch const &L,
                cudaStream_t s) {
  if (L.R > kTWide) {
    TWideParams p;
    std::memset(&p, 0, sizeof(p));
    p.maps = dr.maps_dev;
    p.jobs = dr.twide_dev + L.job_first;
    p.tile_job = dr.twide_tile_dev + L.tile_first;
    p.total_tiles = L.tiles;
    p.error = b.slab_error;
    p.ctas_per_sm = b.ctas_per_sm;
    launch_twide(b.dtype, dr.exact, L.sched, L.R - kTWide, p, s);
    return;
  }
  if (L.R != kSlab) {
    LiftParams lp = dr.params;
    lp.ctas_per_sm = b.ctas_per_sm;
    launch_lift(b.dtype, dr.exact, dr.symmetric, L.sched, L.R, lp,
                dr.jobs_dev + L.job_first, L.njobs, L.tiles, s);
    return;
  }
  SlabParams p;
  std::memset(&p, 0, sizeof(p));
  p.ctas_per_sm = b.ctas_per_sm;
  p.map = b.slab_map;
  p.jobs = dr.slab_dev + L.job_first;
  p.tile_job = dr.slab_tile_dev + L.tile_first;
  p.njobs = L.njobs;
  p.total_tiles = L.tiles;
  p.error = b.slab_error;
  p.pairs = L.pairs;
  launch_slab(b.dtype, L.sched, p, s);
}

void run_direction(paliwa_gb_batch &b, Direction &dr, cudaStream_t s) {
  // Group 0 runs on the caller's stream, group k > 0 on streams[k - 1],
  // forked after the work already queued on `s` and joined back into it.
  auto launch_all = [&] {
    if (b.ngroups > 1)
      cuda_check(cudaEventRecord(b.events[0], s), "cudaEventRecord(fork)");
    for (int k = 1; k < b.ngroups; ++k)
      cuda_check(cudaStreamWaitEvent(b.streams[k - 1], b.events[0], 0),
                 "cudaStreamWaitEvent(fork)");
    for (auto const &L : dr.launches)
      launch_one(b, dr, L, L.group == 0 ? s : b.streams[L.group - 1]);
    for (int k = 1; k < b.ngroups; ++k) {
      cuda_check(cudaEventRecord(b.events[k], b.streams[k - 1]),
                 "cudaEventRecord(join)");
      cuda_check(cudaStreamWaitEvent(s, b.events[k], 0),
                 "cudaStreamWaitEvent(join)");
    }
  };
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (s != nullptr)
    cuda_check(cudaStreamIsCapturing(s, &status), "cudaStreamIsCapturing");
  // The legacy default stream cannot be captured; a stream that is already
  // capturing records our launches (and the fork) into the caller's graph.
  if (!b.use_graphs || s == nullptr || status != cudaStreamCaptureStatusNone) {
    launch_all();
    return;
  }
  if (dr.graph == nullptr) {
    cudaGraph_t graph = nullptr;
    cuda_check(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal),
               "cudaStreamBeginCapture");
    try {
      launch_all();
    } catch (...) {
      cudaStreamEndCapture(s, &graph);
      if (graph) cudaGraphDestroy(graph);
      throw;
    }
    cuda_check(cudaStreamEndCapture(s, &graph), "cudaStreamEndCapture");
    cudaError_t const e = cudaGraphInstantiate(&dr.graph, graph, 0);
    cudaGraphDestroy(graph);
    cuda_check(e, "cudaGraphInstantiate");
  }
  cuda_check(cudaGraphLaunch(dr.graph, s), "cudaGraphLaunch");
}

// Deals the grids, largest first, round-robin into groups, and sizes each
// group's shadow region (the largest per-axis total over the group's grids
// whose pencils along that axis need windowed stages).
void assign_groups(paliwa_gb_batch &b, int64_t const *levels,
                   int64_t const *lmin, int want) {
  size_t const es = dtype_size(b.dtype);
  std::vector<int> order(b.ngrids);
  std::vector<int> log2size(b.ngrids, 0);
  for (int g = 0; g < b.ngrids; ++g) {
    order[g] = g;
    for (int d = 0; d < b.ndim; ++d)
      log2size[g] += static_cast<int>(levels[g * b.ndim + d]);
  }
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) {
    return log2size[a] > log2size[c];
  });
  b.ngroups = std::max(1, std::min(want, b.ngrids));
  b.group.assign(b.ngrids, 0);
  for (int i = 0; i < b.ngrids; ++i) b.group[order[i]] = i % b.ngroups;
  b.group_shadow.assign(b.ngroups, 0);
  b.shadow_bytes = 0;
  for (int k = 0; k < b.ngroups; ++k) {
    size_t need = 0;
    for (int d = 0; d < b.ndim; ++d) {
      size_t total = 0;
      for (int g = 0; g < b.ngrids; ++g) {
        if (b.group[g] != k) continue;
        int64_t const *lv = levels + static_cast<size_t>(g) * b.ndim;
        if (lv[d] <= kWindowLog2 || lv[d] == lmin[d]) continue;
        size_t bytes = es;
        for (int j = 0; j < b.ndim; ++j) bytes <<= lv[j];
        total += (bytes + 255) / 256 * 256;
      }
      need = std::max(need, total);
    }
    b.group_shadow[k] = b.shadow_bytes;
    b.shadow_bytes += need;
  }
}

void free_batch_streams(paliwa_gb_batch &b) {
  for (cudaStream_t st : b.streams)
    if (st != nullptr) cudaStreamDestroy(st);
  for (cudaEvent_t ev : b.events)
    if (ev != nullptr) cudaEventDestroy(ev);
  b.streams.clear();
  b.events.clear();
}

// (Re)groups the batch into `want` groups and plans both directions (keeping
// the autotuner's choices): shadow regions, branch streams and events.
void setup_groups(paliwa_gb_batch &b, int want) {
  free_direction(b.dir[0]);
  free_direction(b.dir[1]);
  free_batch_streams(b);
  if (b.shadow) cudaFree(b.shadow);
  b.shadow = nullptr;
  assign_groups(b, b.levels.data(), b.lmin.data(), want);
  setup_slab_map(b);
  if (b.shadow_bytes)
    cuda_check(cudaMalloc(&b.shadow, b.shadow_bytes), "cudaMalloc(shadow)");
  b.events.assign(b.ngroups, nullptr);
  for (auto &ev : b.events)
    cuda_check(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming),
               "cudaEventCreate");
  b.streams.assign(b.ngroups - 1, nullptr);
  for (auto &st : b.streams)
    cuda_check(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking),
               "cudaStreamCreate");
  plan_direction(b, b.dir[0], true, b.levels.data(), b.lmin.data(),
                 b.grids.data());
  plan_direction(b, b.dir[1], false, b.levels.data(), b.lmin.data(),
                 b.grids.data());
}

} // namespace

// ---------------------------------------------------------------------------
// Combination technique.

struct paliwa_gb_ct {
  int ndim = 0;
  int ngrids = 0;
  int dtype = 0;
  long long npoints = 0;
  std::vector<std::vector<int>> subspace_levels;  // lexicographic order
  std::vector<long long> offsets;
  CtSubspace *subspaces_dev = nullptr;
  int *lists_dev = nullptr;
  CtGrid *grids_dev = nullptr;
  int *block_sub_dev = nullptr;
  CtBlock *blocks_dev = nullptr;
  int *order_dev = nullptr;
  int *unit_grid_dev = nullptr;
  long long *unit_first_dev = nullptr;
  long long *families_dev = nullptr;
  long long *family_first_dev = nullptr;
  // FP32 grids, kCtNarrow points and more: the sparse values as floats during
  // a restrict.
  float *values_dev = nullptr;
  long long ncombine = 0;   // combine CTAs
  long long nrestrict = 0;  // restrict CTAs
  bool big = false;         // a grid of 2^31 points or more
  bool direct = false;      // combine by ct_combine_direct_kernel
  CtParams params{};
};

namespace {

// Key of a level vector (<= 12 dims, levels <= 30: 5 bits each).
uint64_t level_key(int const *s, int ndim) {
  uint64_t k = 0;
  for (int d = 0; d < ndim; ++d) k = (k << 5) | static_cast<uint64_t>(s[d]);
  return k;
}

template <typename T>
void upload(T **dst, std::vector<T> const &v, char const *what) {
  if (v.empty()) return;
  size_t const bytes = v.size() * sizeof(T);
  cuda_check(cudaMalloc(reinterpret_cast<void **>(dst), bytes), what);
  cuda_check(cudaMemcpy(*dst, v.data(), bytes, cudaMemcpyHostToDevice), what);
}

// log2 of a subspace's points.
int subspace_log2(CtSubspace const &ss, int ndim) {
  int n = 0;
  for (int d = 0; d < ndim; ++d) n += std::max(0, ss.level[d] - 1);
  return n;
}

// The combine's CTAs: subspaces of fewer than kCtBlock points grouped by
// size, longest grid lists first (the lists of one CTA are then about
// equally long, and the longest chains of updates start first), then the
// larger subspaces cut into kCtBlock points in storage order (neighbouring
// CTAs share sectors of the grids).
void plan_combine(paliwa_gb_ct &ct, std::vector<CtSubspace> const &subs) {
  int const nsubs = static_cast<int>(subs.size());
  constexpr int log2block = Log2<kCtBlock>::value;
  std::vector<int> order(nsubs), log2p(nsubs);
  auto const length = [&](int i) {
    return subs[i].grid_end - subs[i].grid_begin;
  };
  for (int i = 0; i < nsubs; ++i) {
    order[i] = i;
    log2p[i] = std::min(subspace_log2(subs[i], ct.ndim), log2block);
  }
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    if (log2p[a] != log2p[b]) return log2p[a] < log2p[b];
    return log2p[a] < log2block && length(a) > length(b);
  });
  std::vector<CtBlock> blocks;
  for (int i = 0; i < nsubs;) {
    int const lp = log2p[order[i]];
    CtBlock blk{};
    blk.order_first = i;
    blk.log2p = lp;
    blk.longest = length(order[i]);
    if (lp < log2block) {
      int const most = std::min(ct_max_subs(lp), kCtBlock >> lp);
      while (blk.nsub < most && i + blk.nsub < nsubs &&
             log2p[order[i + blk.nsub]] == lp)
        ++blk.nsub;
      blocks.push_back(blk);
      i += blk.nsub;
      continue;
    }
    blk.nsub = 1;
    long long const size = 1LL << subspace_log2(subs[order[i]], ct.ndim);
    for (blk.local = 0; blk.local < size; blk.local += kCtBlock)
      blocks.push_back(blk);
    ++i;
  }
  // The lists of the small subspaces' CTAs, longest first over all sizes.
  std::stable_sort(blocks.begin(), blocks.end(),
                   [&](CtBlock const &a, CtBlock const &b) {
                     int const la = a.log2p < log2block ? a.longest : -1;
                     int const lb = b.log2p < log2block ? b.longest : -1;
                     return la > lb;
                   });
  ct.ncombine = static_cast<long long>(blocks.size());
  upload(&ct.blocks_dev, blocks, "upload combine blocks");
  upload(&ct.order_dev, order, "upload subspace order");
  ct.params.blocks = ct.blocks_dev;
  ct.params.order = ct.order_dev;
}

// The restrict's units of ct_unit points (the grid of each) and every grid's
// table of families: for the leading levels (s_1 .. s_{d-1}), 0 <= s <= l,
// last dimension fastest, the first sparse point of (s_1 .. s_{d-1}, 0) and
// the highest kept last level of the grid (a subspace's lower neighbours are
// in every grid that holds it, so the kept levels are 0 .. top).
void plan_restrict(paliwa_gb_ct &ct, std::vector<CtSubspace> const &subs,
                   int64_t const *levels) {
  int const nd = ct.ndim;
  // Leading levels -> {first sparse point, highest kept last level}: the
  // subspaces of a family are consecutive and start at last level 0.
  std::unordered_map<uint64_t, std::pair<long long, int>> family;
  std::vector<int> s(nd);
  for (auto const &ss : subs) {
    for (int d = 0; d < nd; ++d) s[d] = ss.level[d];
    auto const it =
        family.emplace(level_key(s.data(), nd - 1),
                       std::make_pair(ss.offset, -1)).first;
    it->second.second = std::max(it->second.second, s[nd - 1]);
  }
  long long const unit = ct_unit(dtype_size(ct.dtype));
  std::vector<int> unit_grid;
  std::vector<long long> unit_first(ct.ngrids), first(ct.ngrids), table;
  for (int g = 0; g < ct.ngrids; ++g) {
    int64_t const *lv = levels + static_cast<size_t>(g) * nd;
    int64_t total = 0;
    for (int d = 0; d < nd; ++d) total += lv[d];
    unit_first[g] = static_cast<long long>(unit_grid.size());
    unit_grid.insert(unit_grid.end(),
                     ((1LL << total) + unit - 1) / unit, g);
    first[g] = static_cast<long long>(table.size());
    std::fill(s.begin(), s.end(), 0);
    while (true) {
      auto const it = family.find(level_key(s.data(), nd - 1));
      long long e = 0;
      if (it != family.end()) {
        int const top =
            std::min<int>(it->second.second, static_cast<int>(lv[nd - 1]));
        e = it->second.first |
            (static_cast<long long>(top + 1) << kCtFamilyShift);
      }
      table.push_back(e);
      int d = nd - 2;
      while (d >= 0 && s[d] == lv[d]) s[d--] = 0;
      if (d < 0) break;
      ++s[d];
    }
  }
  ct.nrestrict = static_cast<long long>(unit_grid.size());
  upload(&ct.unit_grid_dev, unit_grid, "upload restrict units");
  upload(&ct.unit_first_dev, unit_first, "upload restrict unit offsets");
  upload(&ct.families_dev, table, "upload families");
  upload(&ct.family_first_dev, first, "upload family offsets");
  ct.params.unit_grid = ct.unit_grid_dev;
  ct.params.unit_first = ct.unit_first_dev;
  ct.params.families = ct.families_dev;
  ct.params.family_first = ct.family_first_dev;
  if (ct.dtype != PALIWA_GB_F64 && ct.npoints >= kCtNarrow)
    cuda_check(cudaMalloc(&ct.values_dev, ct.npoints * sizeof(float)),
               "cudaMalloc(restrict values)");
}

void free_ct(paliwa_gb_ct &ct) {
  cudaFree(ct.subspaces_dev);
  cudaFree(ct.lists_dev);
  cudaFree(ct.grids_dev);
  cudaFree(ct.block_sub_dev);
  cudaFree(ct.blocks_dev);
  cudaFree(ct.order_dev);
  cudaFree(ct.unit_grid_dev);
  cudaFree(ct.unit_first_dev);
  cudaFree(ct.families_dev);
  cudaFree(ct.family_first_dev);
  cudaFree(ct.values_dev);
}

void build_ct(paliwa_gb_ct &ct, int64_t const *levels,
              double const *coefficients, int64_t const *lmax,
              void *const *grid_ptrs, int keep_all) {
  int const nd = ct.ndim;
  // Count every hierarchical subspace 0 <= s <= l of every grid
  // (paliwa_utils.hpp:9-26; test_paliwa_combination_technique.cpp:177-192).
  std::unordered_map<uint64_t, int> count;
  std::vector<int> s(nd);
  for (int g = 0; g < ct.ngrids; ++g) {
    int64_t const *lv = levels + static_cast<size_t>(g) * nd;
    std::fill(s.begin(), s.end(), 0);
    while (true) {
      ++count[level_key(s.data(), nd)];
      int d = nd - 1;
      while (d >= 0 && s[d] == lv[d]) s[d--] = 0;
      if (d < 0) break;
      ++s[d];
    }
  }
  // Keep subspaces present in more than one grid (:212-225), ordered like
  // the reference's std::map (lexicographic on the level vector).
  std::vector<std::vector<int>> kept;
  for (auto const &[key, c] : count) {
    if (c <= 1 && !keep_all) continue;
    std::vector<int> v(nd);
    uint64_t k = key;
    for (int d = nd - 1; d >= 0; --d) {
      v[d] = static_cast<int>(k & 31);
      k >>= 5;
    }
    kept.push_back(v);
  }
  std::sort(kept.begin(), kept.end());
  std::vector<CtSubspace> subs(kept.size());
  std::vector<int> lists;
  long long off = 0;
  for (size_t i = 0; i < kept.size(); ++i) {
    CtSubspace &ss = subs[i];
    std::memset(&ss, 0, sizeof(ss));
    ss.offset = off;
    long long size = 1;
    for (int d = 0; d < nd; ++d) {
      ss.level[d] = static_cast<signed char>(kept[i][d]);
      if (kept[i][d] > 0) size <<= (kept[i][d] - 1);
    }
    off += size;
    ss.grid_begin = static_cast<int>(lists.size());
    for (int g = 0; g < ct.ngrids; ++g) {
      bool contains = true;  // :270-276
      for (int d = 0; d < nd; ++d)
        if (kept[i][d] > levels[static_cast<size_t>(g) * nd + d]) {
          contains = false;
          break;
        }
      if (contains) lists.push_back(g);
    }
    ss.grid_end = static_cast<int>(lists.size());
  }
  ct.npoints = off;
  ct.subspace_levels = kept;
  ct.offsets.resize(kept.size());
  for (size_t i = 0; i < kept.size(); ++i) ct.offsets[i] = subs[i].offset;
  std::vector<CtGrid> grids(ct.ngrids);
  for (int g = 0; g < ct.ngrids; ++g) {
    std::memset(&grids[g], 0, sizeof(CtGrid));
    grids[g].base = reinterpret_cast<unsigned long long>(grid_ptrs[g]);
    grids[g].coefficient = coefficients[g];
    int step = 0;
    for (int d = nd - 1; d >= 0; --d) {
      int const l = static_cast<int>(levels[static_cast<size_t>(g) * nd + d]);
      grids[g].level[d] = static_cast<signed char>(l);
      step += l;
      grids[g].step[d / 4] |= static_cast<unsigned>(step) << (8 * (d % 4));
    }
  }
  upload(&ct.subspaces_dev, subs, "upload subspaces");
  upload(&ct.lists_dev, lists, "upload grid lists");
  upload(&ct.grids_dev, grids, "upload grids");
  // First subspace of every CTA's 256 points (the subspace holding point
  // 256 b), so that no CTA searches the whole subspace list.
  std::vector<int> block_sub((off + kCtBlock - 1) / kCtBlock);
  {
    size_t si = 0;
    for (size_t b = 0; b < block_sub.size(); ++b) {
      long long const first = static_cast<long long>(b) * kCtBlock;
      while (si + 1 < subs.size() && subs[si + 1].offset <= first) ++si;
      block_sub[b] = static_cast<int>(si);
    }
  }
  upload(&ct.block_sub_dev, block_sub, "upload block subspaces");
  std::memset(&ct.params, 0, sizeof(ct.params));
  ct.params.subspaces = ct.subspaces_dev;
  ct.params.nsubspaces = static_cast<int>(subs.size());
  ct.params.grid_lists = ct.lists_dev;
  ct.params.grids = ct.grids_dev;
  ct.params.ndim = nd;
  ct.params.npoints = ct.npoints;
  for (int d = 0; d < nd && d < kMaxDims; ++d)
    ct.params.max_level[d] = static_cast<signed char>(lmax[d]);
  ct.params.block_sub = ct.block_sub_dev;
  int longest = 0;
  for (auto const &ss : subs)
    longest = std::max(longest, ss.grid_end - ss.grid_begin);
  ct.direct = ct_direct(dtype_size(ct.dtype), ct.npoints, longest);
  plan_combine(ct, subs);
  plan_restrict(ct, subs, levels);
  // Products c * v are exact in FP64 when c has at most 53 - 24 = 29
  // significant bits and v is a float (whose magnitude lies in
  // [2^-149, 2^128]), provided |c| stays within [2^-500, 2^500] so that the
  // product neither underflows nor overflows. For FP64 grids only |c| = 1
  // is exact for every value.
  bool exact = true;
  for (int g = 0; g < ct.ngrids && exact; ++g) {
    double const c = coefficients[g];
    if (c == 0.0) continue;
    if (!std::isfinite(c)) {
      exact = false;
      break;
    }
    if (ct.dtype == PALIWA_GB_F64) {
      exact = std::fabs(c) == 1.0;
      continue;
    }
    int e = 0;
    double m = std::frexp(std::fabs(c), &e);  // m in [0.5, 1)
    long long bits = static_cast<long long>(std::ldexp(m, 53));
    int sig = 53;
    while ((bits & 1) == 0) {
      bits >>= 1;
      --sig;
    }
    if (sig > 29 || e < -500 || e > 500) exact = false;
  }
  ct.params.exact_products = exact ? 1 : 0;
}

// Dimensions padded to 4, 8 or 12 (a padded dimension has one point).
template <typename S, bool Fused>
void launch_combine(paliwa_gb_ct const &ct, CtParams const &p,
                    cudaStream_t s) {
  unsigned const blocks = static_cast<unsigned>(ct.ncombine);
  if (ct.big)
    ct_combine_kernel<S, kMaxDims, Fused, true><<<blocks, kCtBlock, 0, s>>>(p);
  else if (ct.ndim <= 4)
    ct_combine_kernel<S, 4, Fused, false><<<blocks, kCtBlock, 0, s>>>(p);
  else if (ct.ndim <= 8)
    ct_combine_kernel<S, 8, Fused, false><<<blocks, kCtBlock, 0, s>>>(p);
  else
    ct_combine_kernel<S, kMaxDims, Fused, false><<<blocks, kCtBlock, 0, s>>>(
        p);
  cuda_check(cudaGetLastError(), "ct_combine_kernel launch");
}

void launch_combine_direct(paliwa_gb_ct const &ct, CtParams const &p,
                           cudaStream_t s) {
  unsigned const blocks =
      static_cast<unsigned>((ct.npoints + kCtBlock - 1) / kCtBlock);
  if (ct.dtype == PALIWA_GB_F64) {
    if (p.exact_products)
      ct_combine_direct_kernel<double, true><<<blocks, kCtBlock, 0, s>>>(p);
    else
      ct_combine_direct_kernel<double, false><<<blocks, kCtBlock, 0, s>>>(p);
  } else {
    if (p.exact_products)
      ct_combine_direct_kernel<float, true><<<blocks, kCtBlock, 0, s>>>(p);
    else
      ct_combine_direct_kernel<float, false><<<blocks, kCtBlock, 0, s>>>(p);
  }
  cuda_check(cudaGetLastError(), "ct_combine_direct_kernel launch");
}

void ct_combine(paliwa_gb_ct const &ct, double *sparse, cudaStream_t s) {
  if (ct.npoints == 0) return;
  CtParams p = ct.params;
  p.sparse = sparse;
  if (ct.direct) return launch_combine_direct(ct, p, s);
  if (ct.dtype == PALIWA_GB_F64)
    return p.exact_products ? launch_combine<double, true>(ct, p, s)
                            : launch_combine<double, false>(ct, p, s);
  p.exact_products ? launch_combine<float, true>(ct, p, s)
                   : launch_combine<float, false>(ct, p, s);
}

// One to six dimensions have kernels of their own while 32-bit indices hold
// every grid and the sparse grid (with a unit to spare past a grid's end);
// anything else takes the general one.
template <typename S, typename V>
void launch_restrict(paliwa_gb_ct const &ct, CtParams const &p,
                     cudaStream_t s) {
  unsigned const blocks = static_cast<unsigned>(ct.nrestrict);
  bool const small = !ct.big && ct.npoints < (1LL << 31);
  switch (small ? ct.ndim : 0) {
  case 1:
    ct_restrict_kernel<S, 1, unsigned, V><<<blocks, kCtBlock, 0, s>>>(p);
    break;
  case 2:
    ct_restrict_kernel<S, 2, unsigned, V><<<blocks, kCtBlock, 0, s>>>(p);
    break;
  case 3:
    ct_restrict_kernel<S, 3, unsigned, V><<<blocks, kCtBlock, 0, s>>>(p);
    break;
  case 4:
    ct_restrict_kernel<S, 4, unsigned, V><<<blocks, kCtBlock, 0, s>>>(p);
    break;
  case 5:
    ct_restrict_kernel<S, 5, unsigned, V><<<blocks, kCtBlock, 0, s>>>(p);
    break;
  case 6:
    ct_restrict_kernel<S, 6, unsigned, V><<<blocks, kCtBlock, 0, s>>>(p);
    break;
  default:
    ct_restrict_kernel<S, kMaxDims, unsigned long long, V>
        <<<blocks, kCtBlock, 0, s>>>(p);
  }
  cuda_check(cudaGetLastError(), "ct_restrict_kernel launch");
}

void ct_restrict(paliwa_gb_ct const &ct, double const *sparse,
                 cudaStream_t s) {
  if (ct.npoints == 0) return;
  CtParams p = ct.params;
  if (ct.dtype == PALIWA_GB_F64) {
    p.values = sparse;
    launch_restrict<double, double>(ct, p, s);
  } else if (ct.npoints < kCtNarrow) {
    p.values = sparse;
    launch_restrict<float, double>(ct, p, s);
  } else {
    long long const nb = (ct.npoints + kCtBlock - 1) / kCtBlock;
    ct_narrow_kernel<<<static_cast<unsigned>(std::min(nb, 16LL * device_sms())),
                       kCtBlock, 0, s>>>(sparse, ct.values_dev, ct.npoints);
    p.values = ct.values_dev;
    launch_restrict<float, float>(ct, p, s);
  }
}

void ct_scatter(paliwa_gb_ct const &ct, double const *sparse, double *full,
                cudaStream_t s) {
  if (ct.npoints == 0) return;
  CtParams p = ct.params;
  p.sparse = const_cast<double *>(sparse);
  p.full = full;
  ct_scatter_kernel<<<static_cast<unsigned>((ct.npoints + kCtBlock - 1) /
                                            kCtBlock),
                      kCtBlock, 0, s>>>(p);
  cuda_check(cudaGetLastError(), "ct_scatter_kernel launch");
}

} // namespace

extern "C" {

int paliwa_gb_batch_create(int ndim, int ngrids, const int64_t *levels,
                           const int64_t *minimum_level,
                           const int64_t *maximum_level, int dtype,
                           int wavelet, void *const *grid_ptrs,
                           paliwa_gb_batch **out) {
  return guarded([&] {
    if (out == nullptr || levels == nullptr || minimum_level == nullptr ||
        maximum_level == nullptr || grid_ptrs == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    check_grid_levels(ndim, ngrids, levels, minimum_level, maximum_level);
    size_t const es = dtype_size(dtype);
    wavelet_filters(wavelet, true);  // validates the id
    auto b = std::make_unique<paliwa_gb_batch>();
    b->ndim = ndim;
    b->ngrids = ngrids;
    b->dtype = dtype;
    b->wavelet = wavelet;
    b->levels.assign(levels, levels + static_cast<size_t>(ngrids) * ndim);
    b->lmin.assign(minimum_level, minimum_level + ndim);
    b->grids.assign(grid_ptrs, grid_ptrs + ngrids);
    for (int g = 0; g < ngrids; ++g) {
      if (grid_ptrs[g] == nullptr ||
          reinterpret_cast<uintptr_t>(grid_ptrs[g]) % es != 0)
        throw StatusError(PALIWA_GB_INVALID_ARGUMENT,
                          "grid pointer is null or misaligned");
      int64_t total = 0;
      for (int d = 0; d < ndim; ++d) total += levels[g * ndim + d];
      b->points += 1LL << total;
    }
    for (Direction &dr : b->dir) dr.slabs = default_slabs(dtype, b->points);
    try {
      cuda_check(cudaMalloc(&b->slab_error, sizeof(unsigned)),
                 "cudaMalloc(error word)");
      cuda_check(cudaMemset(b->slab_error, 0, sizeof(unsigned)),
                 "cudaMemset(error word)");
      setup_groups(*b, kBatchGroups);
    } catch (...) {
      free_direction(b->dir[0]);
      free_direction(b->dir[1]);
      free_batch_streams(*b);
      if (b->shadow) cudaFree(b->shadow);
      if (b->slab_error) cudaFree(b->slab_error);
      throw;
    }
    *out = b.release();
  });
}

int paliwa_gb_batch_hierarchize(paliwa_gb_batch *batch, void *stream) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    run_direction(*batch, batch->dir[0], static_cast<cudaStream_t>(stream));
  });
}

int paliwa_gb_batch_dehierarchize(paliwa_gb_batch *batch, void *stream) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    run_direction(*batch, batch->dir[1], static_cast<cudaStream_t>(stream));
  });
}

int paliwa_gb_batch_use_graphs(paliwa_gb_batch *batch, int enable) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    batch->use_graphs = enable != 0;
  });
}

int paliwa_gb_batch_set_groups(paliwa_gb_batch *batch, int ngroups) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    if (ngroups < 1)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "ngroups must be >= 1");
    cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    setup_groups(*batch, ngroups);
  });
}

int paliwa_gb_batch_use_slabs(paliwa_gb_batch *batch, int enable) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    batch->use_slabs = enable != 0;
    for (Direction &dr : batch->dir) dr.slabs = batch->use_slabs;
    setup_groups(*batch, batch->ngroups);
  });
}

int paliwa_gb_batch_use_tma(paliwa_gb_batch *batch, int enable) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    batch->use_tma = enable != 0;
    setup_groups(*batch, batch->ngroups);
  });
}

int paliwa_gb_batch_set_ctas_per_sm(paliwa_gb_batch *batch, int ctas) {
  return guarded([&] {
    if (batch == nullptr || ctas < 0)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT,
                        "null batch or negative CTA count");
    cuda_check(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    batch->ctas_per_sm = ctas;
    setup_groups(*batch, batch->ngroups);
  });
}

int paliwa_gb_batch_status(paliwa_gb_batch *batch) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    unsigned err = 0;
    cuda_check(cudaMemcpy(&err, batch->slab_error, sizeof(err),
                          cudaMemcpyDeviceToHost),
               "cudaMemcpy(error word)");
    if (err != 0) {
      cuda_check(cudaMemset(batch->slab_error, 0, sizeof(err)),
                 "cudaMemset(error word)");
      throw StatusError(PALIWA_GB_TIMEOUT,
                        "a slab kernel's bounded wait for its tile copy "
                        "gave up");
    }
  });
}

int paliwa_gb_batch_info(const paliwa_gb_batch *batch, int64_t *points,
                         int64_t *launches_forward,
                         int64_t *launches_inverse) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    if (points) *points = batch->points;
    if (launches_forward)
      *launches_forward = static_cast<int64_t>(batch->dir[0].launches.size());
    if (launches_inverse)
      *launches_inverse = static_cast<int64_t>(batch->dir[1].launches.size());
  });
}

namespace {

// Milliseconds of direction `which` (0 forward, 1 inverse), best of `reps`
// event-timed runs as the batch runs them (its groups on parallel branches,
// from a graph when graphs are on: a plan's speed depends on how its
// launches overlap); every run is followed (forward) or preceded (inverse)
// by the other direction, so that the grids return to their contents up to
// rounding.
float time_direction(paliwa_gb_batch &b, int which, int reps,
                     cudaStream_t s) {
  cudaEvent_t e0, e1;
  cuda_check(cudaEventCreate(&e0), "cudaEventCreate");
  cuda_check(cudaEventCreate(&e1), "cudaEventCreate");
  auto run = [&](Direction &dr) { run_direction(b, dr, s); };
  float best = 1e30f;
  for (int r = 0; r < reps; ++r) {
    if (which == 1) run(b.dir[0]);
    cuda_check(cudaEventRecord(e0, s), "cudaEventRecord");
    run(b.dir[which]);
    cuda_check(cudaEventRecord(e1, s), "cudaEventRecord");
    if (which == 0) run(b.dir[1]);
    cuda_check(cudaEventSynchronize(e1), "cudaEventSynchronize");
    float ms = 0;
    cuda_check(cudaEventElapsedTime(&ms, e0, e1), "cudaEventElapsedTime");
    best = std::min(best, ms);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return best;
}

void replan(paliwa_gb_batch &b, int which) {
  Direction &dr = b.dir[which];
  free_direction(dr);
  plan_direction(b, dr, which == 0, b.levels.data(), b.lmin.data(),
                 b.grids.data());
}

} // namespace

int paliwa_gb_batch_autotune(paliwa_gb_batch *batch, void *stream, int reps,
                             int *changed) {
  return guarded([&] {
    if (batch == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null batch");
    if (reps < 1) reps = 1;
    cudaStream_t const s = static_cast<cudaStream_t>(stream);
    int nchanged = 0;
    for (int which = 0; which < 2; ++which) {
      Direction &dr = batch->dir[which];
      float best = time_direction(*batch, which, reps, s);
      // Slab launches against the same axes planned one by one (either way
      // round, so that a second call can bring the slabs back).
      bool has_slab = false;
      for (auto const &L : dr.launches) has_slab |= L.R == kSlab;
      if (batch->use_slabs && batch->slab_map_ok && (has_slab || !dr.slabs)) {
        dr.slabs = !dr.slabs;
        replan(*batch, which);
        float const t = time_direction(*batch, which, reps, s);
        if (t < best * 0.99f) {
          best = t;
          ++nchanged;
        } else {
          dr.slabs = !dr.slabs;
          replan(*batch, which);
        }
      }
      // Coordinate descent over the classes of periodic stages: try every
      // kernel that applies to a class, keep the fastest whole direction.
      auto const classes = dr.classes;
      long long total = 0;
      for (auto const &kv : classes) total += kv.second.points;
      for (auto const &[tclass, info] : classes) {
        unsigned const mask = info.kernels;
        int const dflt = info.dflt;
        if ((mask & (mask - 1)) == 0) continue;  // one kernel applies
        // A class with under 2 % of the points cannot move the direction's
        // time by the 1 % a change must gain.
        if (info.points * 50 < total) continue;
        auto const it = dr.tuning.choice.find(tclass);
        int const current = it != dr.tuning.choice.end() ? it->second : dflt;
        int keep = current;
        for (int c = 0; c < kChooseCount; ++c) {
          if (c == current || !((mask >> c) & 1u)) continue;
          dr.tuning.choice[tclass] = c;
          replan(*batch, which);
          float const t = time_direction(*batch, which, reps, s);
          if (t < best * 0.99f) {
            best = t;
            keep = c;
          }
        }
        if (keep == dflt && it == dr.tuning.choice.end())
          dr.tuning.choice.erase(tclass);
        else
          dr.tuning.choice[tclass] = keep;
        if (keep != current) ++nchanged;
        replan(*batch, which);
      }
    }
    if (changed != nullptr) *changed = nchanged;
  });
}

int paliwa_gb_batch_tuning(const paliwa_gb_batch *batch, int forward,
                           int capacity, int *nclasses, int32_t *classes,
                           int32_t *kernels, int32_t *choices) {
  return guarded([&] {
    if (batch == nullptr || nclasses == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    Direction const &dr = batch->dir[forward ? 0 : 1];
    *nclasses = static_cast<int>(dr.classes.size());
    if (capacity < *nclasses || classes == nullptr || kernels == nullptr ||
        choices == nullptr)
      return;
    int i = 0;
    for (auto const &[tclass, info] : dr.classes) {
      auto const it = dr.tuning.choice.find(tclass);
      classes[i] = tclass;
      kernels[i] = static_cast<int32_t>(info.kernels);
      choices[i] = it != dr.tuning.choice.end() ? it->second : info.dflt;
      ++i;
    }
  });
}

int paliwa_gb_batch_set_tuning(paliwa_gb_batch *batch, int forward,
                               int nclasses, const int32_t *classes,
                               const int32_t *choices) {
  return guarded([&] {
    if (batch == nullptr || nclasses < 0 ||
        (nclasses > 0 && (classes == nullptr || choices == nullptr)))
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    int const which = forward ? 0 : 1;
    Direction &dr = batch->dir[which];
    // Check every entry before changing anything.
    for (int i = 0; i < nclasses; ++i) {
      auto const it = dr.classes.find(classes[i]);
      if (it == dr.classes.end())
        throw StatusError(PALIWA_GB_INVALID_ARGUMENT,
                          "no stage of the batch is in tuning class " +
                              std::to_string(classes[i]));
      if (choices[i] < 0 || choices[i] >= kChooseCount ||
          !((it->second.kernels >> choices[i]) & 1u))
        throw StatusError(PALIWA_GB_INVALID_ARGUMENT,
                          "kernel " + std::to_string(choices[i]) +
                              " does not apply to tuning class " +
                              std::to_string(classes[i]));
    }
    for (int i = 0; i < nclasses; ++i) {
      if (choices[i] == dr.classes.at(classes[i]).dflt)
        dr.tuning.choice.erase(classes[i]);
      else
        dr.tuning.choice[classes[i]] = choices[i];
    }
    replan(*batch, which);
  });
}

int paliwa_gb_batch_profile(paliwa_gb_batch *batch, int forward, void *stream,
                            int capacity, int *nlaunches, float *ms,
                            int64_t *bytes, int32_t *kernels) {
  return guarded([&] {
    if (batch == nullptr || nlaunches == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    Direction &dr = batch->dir[forward ? 0 : 1];
    cudaStream_t const s = static_cast<cudaStream_t>(stream);
    int const n = static_cast<int>(dr.launches.size());
    *nlaunches = n;
    if (capacity < n || ms == nullptr || bytes == nullptr) return;
    std::vector<cudaEvent_t> ev(n + 1);
    for (auto &e : ev) cuda_check(cudaEventCreate(&e), "cudaEventCreate");
    size_t const es = dtype_size(batch->dtype);
    cuda_check(cudaEventRecord(ev[0], s), "cudaEventRecord");
    for (int i = 0; i < n; ++i) {
      Launch const &L = dr.launches[i];
      launch_one(*batch, dr, L, s);
      cuda_check(cudaEventRecord(ev[i + 1], s), "cudaEventRecord");
      bytes[i] = static_cast<int64_t>(2 * es) * L.points;
      if (kernels != nullptr) kernels[i] = L.R;
    }
    cuda_check(cudaEventSynchronize(ev[n]), "cudaEventSynchronize");
    for (int i = 0; i < n; ++i)
      cuda_check(cudaEventElapsedTime(&ms[i], ev[i], ev[i + 1]),
                 "cudaEventElapsedTime");
    for (auto &e : ev) cudaEventDestroy(e);
  });
}

void paliwa_gb_batch_destroy(paliwa_gb_batch *batch) {
  if (batch == nullptr) return;
  free_direction(batch->dir[0]);
  free_direction(batch->dir[1]);
  free_batch_streams(*batch);
  if (batch->shadow) cudaFree(batch->shadow);
  if (batch->slab_error) cudaFree(batch->slab_error);
  delete batch;
}

int paliwa_gb_ct_create(int ndim, int ngrids, const int64_t *levels,
                        const double *coefficients,
                        const int64_t *maximum_level, int dtype,
                        void *const *grid_ptrs, int keep_all,
                        paliwa_gb_ct **out) {
  return guarded([&] {
    if (out == nullptr || levels == nullptr || coefficients == nullptr ||
        maximum_level == nullptr || grid_ptrs == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    check_grid_levels(ndim, ngrids, levels, nullptr, maximum_level);
    size_t const es = dtype_size(dtype);
    for (int g = 0; g < ngrids; ++g)
      if (grid_ptrs[g] == nullptr ||
          reinterpret_cast<uintptr_t>(grid_ptrs[g]) % es != 0)
        throw StatusError(PALIWA_GB_INVALID_ARGUMENT,
                          "grid pointer is null or misaligned");
    auto ct = std::make_unique<paliwa_gb_ct>();
    ct->ndim = ndim;
    ct->ngrids = ngrids;
    ct->dtype = dtype;
    for (int g = 0; g < ngrids; ++g) {
      int64_t total = 0;
      for (int d = 0; d < ndim; ++d) total += levels[g * ndim + d];
      ct->big |= total >= 31;
    }
    try {
      build_ct(*ct, levels, coefficients, maximum_level, grid_ptrs, keep_all);
    } catch (...) {
      free_ct(*ct);
      throw;
    }
    *out = ct.release();
  });
}

int paliwa_gb_ct_info(const paliwa_gb_ct *ct, int64_t *npoints,
                      int64_t *nsubspaces) {
  return guarded([&] {
    if (ct == nullptr) throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null ct");
    if (npoints) *npoints = ct->npoints;
    if (nsubspaces)
      *nsubspaces = static_cast<int64_t>(ct->subspace_levels.size());
  });
}

int paliwa_gb_ct_subspaces(const paliwa_gb_ct *ct, int64_t *levels,
                           int64_t *offsets) {
  return guarded([&] {
    if (ct == nullptr) throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null ct");
    for (size_t i = 0; i < ct->subspace_levels.size(); ++i) {
      if (levels)
        for (int d = 0; d < ct->ndim; ++d)
          levels[i * ct->ndim + d] = ct->subspace_levels[i][d];
      if (offsets) offsets[i] = ct->offsets[i];
    }
  });
}

int paliwa_gb_ct_combine(paliwa_gb_ct *ct, double *sparse, void *stream) {
  return guarded([&] {
    if (ct == nullptr || sparse == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    ct_combine(*ct, sparse, static_cast<cudaStream_t>(stream));
  });
}

int paliwa_gb_ct_restrict(paliwa_gb_ct *ct, const double *sparse,
                          void *stream) {
  return guarded([&] {
    if (ct == nullptr || sparse == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    ct_restrict(*ct, sparse, static_cast<cudaStream_t>(stream));
  });
}

int paliwa_gb_ct_scatter(paliwa_gb_ct *ct, const double *sparse, double *full,
                         void *stream) {
  return guarded([&] {
    if (ct == nullptr || sparse == nullptr || full == nullptr)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "null argument");
    // The full grid starts from zero (test_paliwa_combination_technique.cpp
    // :295-298); every kept subspace point is then added once.
    long long total = 0;
    for (int d = 0; d < ct->ndim; ++d) total += ct->params.max_level[d];
    if (total > 36)
      throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "full grid too large");
    cuda_check(cudaMemsetAsync(full, 0, sizeof(double) << total,
                               static_cast<cudaStream_t>(stream)),
               "cudaMemsetAsync");
    ct_scatter(*ct, sparse, full, static_cast<cudaStream_t>(stream));
  });
}

void paliwa_gb_ct_destroy(paliwa_gb_ct *ct) {
  if (ct == nullptr) return;
  free_ct(*ct);
  delete ct;
}

} // extern "C"
