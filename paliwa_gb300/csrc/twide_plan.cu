// Host side of the TMA wide kernel: stages, jobs, tensor maps and launches
// of single grids.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>

#include "launch.cuh"
#include "paliwa_gb300.h"
#include "twide_box.cuh"
#include "twide_plan.hpp"

namespace pgb {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 const encode = [] {
    cudaDriverEntryPointQueryResult q{};
    void *fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                         cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }();
  return encode;
}

namespace {

// Points per thread of the TMA wide kernel (0: it does not take the stage).
// Floats: whole pencils of up to 16 points, chunks of n / 4 points up to 64
// (a strided axis) and of 16 points beyond. Doubles: whole pencils of up to
// 32 points and chunks of 32 beyond: the FP64 pipe runs a coarse step of one
// head per chunk as a whole warp instruction, so half the chunks are half
// that waste (512 points: 140 instead of 160 DFMAs for every 128 needed).
int twide_chunk(LiftJob const &job, int dtype, bool table) {
  int const n = job.log2_n;
  bool const last = job.log2_inner == 0 && job.log2_kstride == 0;
  if (dtype == PALIWA_GB_F64) return n < 1 || n > 10 ? 0 : 1 << std::min(n, 5);
  if (n < 1 || n > (last ? 12 : 11)) return 0;
  // Plain floats: strided pencils of 1024 points in chunks of 32, which
  // exchange by shuffles (5200 GB/s against 3310-3870 in the long form and
  // 3840-4650 on the tile kernel); with a caller's filters also those of 256
  // and 512 (four passes, n = 512: 4030 against 2830; CDF (2,2): 5470 against
  // 5530).
  if (dtype == PALIWA_GB_F32 && !last && (n == 10 || (n >= 8 && n <= 9 && table)))
    return 32;
  if (n <= 4) return 1 << n;
  if (n <= 6 && !last) return 1 << (n - 2);
  return 16;
}

} // namespace

int twide_code(Stage const &st, int dtype) {
  if (st.box)
    return dtype == PALIWA_GB_F64 ? kTWide32Box
           : st.heads != 0        ? kTWideBoxHeads + 16
                                  : kTWideBox + 16;
  int const r = st.tma ? twide_chunk(st.job, dtype, st.table) : 0;
  if (r == 0) return 0;
  int const log2G = st.job.log2_n - (31 - __builtin_clz(r));
  // Inner extent in floats (see twide_job).
  int const inner = st.job.log2_inner + (dtype == PALIWA_GB_F64 ? 1 : 0);
  if (r == 32)
    return dtype == PALIWA_GB_F64 && inner == 1 ? kTWide32Pairs
           : log2G >= 3 ? kTWide32Chunked : kTWide32Dense;
  bool const last = inner == 0 && st.job.log2_kstride == 0;
  return r + (last         ? (log2G > 5 ? kTWideLongContig : kTWideContig)
              : inner == 1 ? kTWidePairs
              : log2G > 5  ? kTWideLong
              : log2G >= 3 ? kTWideChunked : 0);
}

// Measured per launch, replayed from a graph (us, against the stage's own
// kernel): FP32 n = 16 at 2^12 points 3.6 against 3.1, at 2^14 3.8 against
// 4.1; FP32c 4.6 against 3.4 and 4.8 against 6.1; FP64 at 2^10 7.5 against
// 6.5, at 2^12 7.9 against 7.6 and at 2^14 7.8 against 22.4 (few threads of
// the FP64 pipe); chunked and long forms win from their smallest launches
// (FP32 n = 128 at 2^12 4.1 against 6.7).
bool twide_enough(int code, int dtype, long long points) {
  bool const longer =
      code == kTWideBoxHeads + 16 || code == kTWideBox + 16 ||
      code == kTWide32Box || code == kTWide32Chunked ||
      code == kTWideChunked + 16 || code == kTWideLong + 16 ||
      code == kTWideLongContig + 16;
  return longer || points >= (dtype == PALIWA_GB_F64 ? 1LL << 12 : 1LL << 13);
}

// A caller's filters on pencils of 2 points, and of 4 floats, have less work
// for the same start-up (us, four passes / one, against the direct kernel:
// FP32 n = 2 at 2^18 points 5.6 / 4.4 against 3.5 / 2.7, at 2^20 6.8 / 5.3
// against 8.2 / 6.0; n = 4 5.2 / 3.7 against 4.5 / 3.0 and 6.5 / 5.1 against
// 8.0 / 5.6; FP64 n = 2 at 2^16 9.0 / 5.2 against 7.2 / 3.6, at 2^18 8.7 / 5.0
// against 11.4 / 4.6; FP64 n = 4 gains from 2^12 on).
static bool table_enough(Stage const &st, int dtype) {
  int const log2_n = st.job.log2_n;
  return !st.table || log2_n > 2 || (log2_n == 2 && dtype == PALIWA_GB_F64) ||
         stage_points(st) >= (dtype == PALIWA_GB_F64 ? 1LL << 18 : 1LL << 19);
}

namespace {

// Boxed form: the 3D view [outer][n][inner] of the grid (and of the halo
// buffer, in the same layout) in boxes of 128 bytes of columns by one chunk.
bool twide_box_job(Stage const &st, int dtype, TWideJob &job,
                   CUtensorMap map[2], long long &tiles) {
  auto const encode = tensor_map_encoder();
  LiftJob lj = st.job;
  int const r = dtype == PALIWA_GB_F64 ? 32 : 16;
  if (dtype == PALIWA_GB_F64) {  // a double column is two float columns
    ++lj.log2_inner;
    ++lj.log2_kstride;
    ++lj.log2_astride;
    lj.columns *= 2;
  }
  int const log2w = lj.periodic ? lj.log2_n : lj.log2_window;
  int const log2boxes = 31 - __builtin_clz(
                                 static_cast<unsigned>(kBoxRows / r));
  int const log2G = log2w - (31 - __builtin_clz(static_cast<unsigned>(r)));
  if (encode == nullptr || lj.log2_inner < 5 || log2w > 9 || log2G < 1 ||
      log2G > log2boxes || (lj.base | lj.halo_base) % 16 != 0 ||
      lj.log2_n > 30)
    return false;
  std::memset(&job, 0, sizeof(job));
  job.log2_n = log2w;
  job.log2_inner = lj.log2_inner;
  job.nlevels = lj.nlevels;
  job.win.halo_map = 1;
  // Tiles of 2^(log2boxes - log2G) blocks of 32 floats.
  int const log2ct = 5 + log2boxes - log2G;
  long long const ct = (lj.columns + (1LL << log2ct) - 1) >> log2ct;
  long long segments = 1;
  if (!lj.periodic) {
    if (lj.halo_base == 0 || lj.seg_len % r != 0 || lj.halo % r != 0)
      return false;
    job.win.seg_len = lj.seg_len;
    job.win.halo = lj.halo;
    job.win.log2_full = lj.log2_n;
    segments = ((1LL << lj.log2_n) + lj.seg_len - 1) / lj.seg_len;
  }
  tiles = ct * segments;
  if (tiles >= (1LL << 30)) return false;
  job.win.col_tiles = static_cast<int>(ct);
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(1) << lj.log2_inner,
                        static_cast<cuuint64_t>(1) << lj.log2_n,
                        static_cast<cuuint64_t>(lj.columns >> lj.log2_inner)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(4) << lj.log2_kstride,
                           static_cast<cuuint64_t>(4) << lj.log2_astride};
  cuuint32_t box[3] = {32, static_cast<cuuint32_t>(r), 1};
  cuuint32_t elem[3] = {1, 1, 1};
  for (int i = 0; i < (lj.periodic ? 1 : 2); ++i)
    if (encode(&map[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
               reinterpret_cast<void *>(i == 0 ? lj.base : lj.halo_base),
               dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  return true;
}

} // namespace

// Up to 4 chunks per pencil (dense): the 3D view [outer][n][inner] of the
// stage's pencils with the axis' strides and boxes {Bx, n, Sx}. 8 chunks and
// more (chunk-interleaved): the 5D view [outer][inner / X][row of chunk]
// [chunk][X columns] and one box per tile, so that shared memory holds the
// tile as [column group][row of chunk][chunk][X columns]. The last axis and
// inner extents of 2 floats: rows of 128 bytes.
bool twide_job(Stage const &st, int dtype, TWideJob &job, CUtensorMap map[2],
               long long &tiles) {
  auto encode = tensor_map_encoder();
  if (st.box) return twide_box_job(st, dtype, job, map, tiles);
  LiftJob lj = st.job;
  int const r = twide_chunk(lj, dtype, st.table);
  if (encode == nullptr || r == 0 || lj.periodic != 1 || lj.base % 16 != 0)
    return false;
  // A double column is two float columns: the grid is viewed as floats with
  // twice the inner extent (every copy moves 4-byte words).
  if (dtype == PALIWA_GB_F64) {
    ++lj.log2_inner;
    ++lj.log2_kstride;
    ++lj.log2_astride;
    lj.columns *= 2;
  }
  int const log2r = 31 - __builtin_clz(static_cast<unsigned>(r));
  int const log2G = lj.log2_n - log2r;
  int const threads = twide_threads(r);
  int const log2nt = 31 - __builtin_clz(static_cast<unsigned>(threads));
  bool const last = lj.log2_inner == 0 && lj.log2_kstride == 0;
  bool const pairs = lj.log2_inner == 1 && lj.log2_kstride == 1 &&
                     lj.log2_astride == lj.log2_n + 1;
  if (last || pairs) {
    // The last axis (contiguous layout), or a strided axis of inner extent
    // 2 whose pencil pairs lie one after another (pairs layout): the
    // stage's points as rows of 32 floats (128 bytes), boxes of the unit's
    // rows, 128-byte swizzle; units of 2 threads r floats (whole pencils).
    if (r < 4 || log2G < 0 ||
        log2G > (pairs ? (r == 32 ? 5 : 2) : 5 + 3 * (r == 16)))
      return false;
    long long const points = lj.columns << lj.log2_n;
    int const log2unit = 1 + log2nt + log2r;
    int const log2u = r >= 8 ? 0 : 3 - log2r;  // units per tile
    if (points % 32 != 0 || (points >> (log2unit + log2u)) >= (1LL << 30))
      return false;
    tiles = (points + (1LL << (log2unit + log2u)) - 1) >> (log2unit + log2u);
    std::memset(&job, 0, sizeof(job));
    job.log2_n = lj.log2_n;
    job.nlevels = lj.nlevels;
    job.chunked = pairs ? 3 : 2;
    job.nxb = 1;
    job.log2_bx = log2unit - lj.log2_n;  // box bytes = the unit
    job.log2_sx = 0;
    cuuint64_t dims[2] = {32, static_cast<cuuint64_t>(points / 32)};
    cuuint64_t strides[1] = {128};
    cuuint32_t box[2] = {32, 1u << (log2unit - 5)};
    cuuint32_t elem[2] = {1, 1};
    CUresult const res = encode(
        &map[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
        reinterpret_cast<void *>(lj.base), dims, strides, box, elem,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return res == CUDA_SUCCESS;
  }
  if (lj.log2_inner < 2 || log2G < 0 || log2G > 7 || lj.log2_n > 11 ||
      (log2G > 2 && r < 16) || (r == 32 && log2G > 5))
    return false;
  int const log2ct = log2nt + 1 - log2G;
  // Units per tile: TWideShape<R>::kUnits (16 KB tiles for chunks of up to
  // 8 points).
  int const log2u = r >= 8 ? 0 : 3 - log2r;
  std::memset(&job, 0, sizeof(job));
  job.log2_n = lj.log2_n;
  job.log2_inner = lj.log2_inner;
  job.nlevels = lj.nlevels;
  job.log2_bx = std::min(std::min(lj.log2_inner, log2ct), 8);
  job.log2_sx = std::max(0, log2ct - lj.log2_inner);
  job.nxb = 1 << (log2ct - job.log2_bx - job.log2_sx);
  job.log2_rs = job.log2_bx;
  tiles = (lj.columns + (1LL << (log2ct + log2u)) - 1) >> (log2ct + log2u);
  if (tiles >= (1LL << 30)) return false;
  long long const outer = lj.columns >> lj.log2_inner;
  if (log2G >= 3) {
    job.chunked = 1;
    job.nxb = 1;
    job.log2_bx = std::min(lj.log2_inner, log2ct);  // Bx >= 4: log2ct <= 6
    job.log2_sx = log2ct - job.log2_bx;
    // Groups of X columns: 4 (16 bytes, the least a box row may be), 8 or 16
    // where the tile and the inner extent hold them. Wider rows are fewer for
    // the tensor memory accelerator, but the chunks a warp reads together lie
    // X columns apart, on fewer banks. 8 for up to 32 chunks (the chunked
    // form 3.9 against 3.5 TB/s on the 4D batch; the long form is slower with
    // them); 16 for up to 16 chunks of plain floats, whose arithmetic is cheap
    // (n = 128 6.0 against 5.5 TB/s, n = 256 6.1 against 5.5), and for FP32c
    // where the pencils span 256 MB or more: every box row is then a page of
    // its own, at 8 clocks each (n = 128 4.75 against 3.25, n = 256 3.97
    // against 3.53 and less; below that span 4.77 against 4.84 and 3.97
    // against 4.45). A caller's filters take 8 (four passes, n = 256 3.2
    // against 2.9 TB/s).
    bool const spread =
        lj.log2_n + lj.log2_kstride + 2 >= 28 || dtype == PALIWA_GB_F32;
    int const xmax = log2G > 5 ? 2
                     : log2G <= 4 && dtype != PALIWA_GB_F64 && !st.table &&
                             spread ? 4 : 3;
    int const xlo = std::max(2, std::min({xmax, log2ct, lj.log2_inner}));
    job.log2_xlo = xlo;
    job.log2_rs = log2G + xlo;
    cuuint64_t dims[5] = {1u << xlo, static_cast<cuuint64_t>(1) << log2G,
                          static_cast<cuuint64_t>(r),
                          static_cast<cuuint64_t>(1) << (lj.log2_inner - xlo),
                          static_cast<cuuint64_t>(outer)};
    cuuint64_t strides[4] = {
        static_cast<cuuint64_t>(4 * r) << lj.log2_kstride,
        static_cast<cuuint64_t>(4) << lj.log2_kstride,
        static_cast<cuuint64_t>(4) << xlo,
        static_cast<cuuint64_t>(4) << lj.log2_astride};
    cuuint32_t box[5] = {1u << xlo, 1u << log2G, static_cast<cuuint32_t>(r),
                         1u << (job.log2_bx - xlo), 1u << job.log2_sx};
    cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    CUresult const res = encode(
        &map[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5,
        reinterpret_cast<void *>(lj.base), dims, strides, box, elem,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return res == CUDA_SUCCESS;
  }
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(1) << lj.log2_inner,
                        static_cast<cuuint64_t>(1) << lj.log2_n,
                        static_cast<cuuint64_t>(outer)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(4) << lj.log2_kstride,
                           static_cast<cuuint64_t>(4) << lj.log2_astride};
  cuuint32_t box[3] = {1u << job.log2_bx, 1u << lj.log2_n,
                       1u << job.log2_sx};
  // An outer index's n rows of `inner` columns are one contiguous block
  // when the pencil stride is the inner extent (no sub-lattice). When a
  // tile holds whole blocks (inner < Ct) and a block fits one box
  // dimension, the map takes the block as its rows: box rows of n inner
  // floats instead of inner (fewer, longer rows for the tensor memory
  // accelerator), the same bytes in the same shared-memory order, the same
  // box coordinates (x = y = 0).
  if (lj.log2_kstride == lj.log2_inner && lj.log2_inner < log2ct &&
      lj.log2_n + lj.log2_inner <= 8) {
    int const log2blk = lj.log2_n + lj.log2_inner;
    dims[0] = static_cast<cuuint64_t>(1) << log2blk;
    dims[1] = 1;
    strides[0] = static_cast<cuuint64_t>(4) << log2blk;
    box[0] = 1u << log2blk;
    box[1] = 1;
  }
  cuuint32_t elem[3] = {1, 1, 1};
  CUresult const res = encode(
      &map[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
      reinterpret_cast<void *>(lj.base), dims, strides, box, elem,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return res == CUDA_SUCCESS;
}

void launch_twide(int dtype, bool exact, int sched, int code,
                  TWideParams const &p, cudaStream_t s) {
  bool const table = sched >= kTableSched;
  switch (dtype) {
  case PALIWA_GB_F64:
    return table ? launch_twide_table_f64(exact, sched, code, p, s)
                 : launch_twide_f64(sched, code, p, s);
  case PALIWA_GB_F32:
    return table ? launch_twide_table_f32(exact, sched, code, p, s)
                 : launch_twide_f32(sched, code, p, s);
  case PALIWA_GB_F32C: return launch_twide_f32c(sched, code, p, s);
  }
  throw StatusError(PALIWA_GB_INVALID_ARGUMENT, "unknown dtype");
}

namespace {

// Error words of the single-grid launches' bounded waits, per device: one per
// stream handle, given out in order of use (once all are, further streams
// share them), and one for captured launches, whose replays may run on any
// stream. They lie in mapped host memory (one page), which the host reads
// without a copy. (By the handle, not the id: cudaStreamGetId ends a capture.)
constexpr unsigned kStreamWords = 1023;
std::atomic<unsigned *> g_error_words[Occupancy::kMaxDevices];
std::atomic<uintptr_t> g_word_streams[Occupancy::kMaxDevices][kStreamWords];

// Allocated by a device's first single-grid call (also inside a stream
// capture: the allocation is not part of the captured work); nullptr where
// that fails.
unsigned *error_words(int dev) {
  if (dev < 0 || dev >= Occupancy::kMaxDevices) return nullptr;
  unsigned *words = g_error_words[dev].load(std::memory_order_acquire);
  if (words != nullptr) return words;
  static std::mutex mutex;
  std::lock_guard<std::mutex> lock(mutex);
  words = g_error_words[dev].load(std::memory_order_acquire);
  if (words != nullptr) return words;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cuda_check(cudaThreadExchangeStreamCaptureMode(&mode),
             "cudaThreadExchangeStreamCaptureMode");
  void *p = nullptr;
  size_t const bytes = (kStreamWords + 1) * sizeof(unsigned);
  cudaError_t const e =
      cudaHostAlloc(&p, bytes, cudaHostAllocPortable | cudaHostAllocMapped);
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  std::memset(p, 0, bytes);
  words = static_cast<unsigned *>(p);
  g_error_words[dev].store(words, std::memory_order_release);
  return words;
}

unsigned stream_slot(int dev, cudaStream_t s) {
  uintptr_t const key =
      s == nullptr ? reinterpret_cast<uintptr_t>(cudaStreamLegacy)
                   : reinterpret_cast<uintptr_t>(s);
  unsigned const first = static_cast<unsigned>((key >> 4) % kStreamWords);
  for (unsigned i = 0, k = first; i < kStreamWords; ++i) {
    auto &slot = g_word_streams[dev][k];
    uintptr_t cur = slot.load(std::memory_order_relaxed);
    if (cur == key ||
        (cur == 0 && (slot.compare_exchange_strong(cur, key) || cur == key)))
      return k;
    k = k + 1 == kStreamWords ? 0 : k + 1;
  }
  return first;
}

// Whether the word was set; clears it. (A report that comes in between is
// either part of this one or stays.)
bool take_error(unsigned *word) {
  return __atomic_load_n(word, __ATOMIC_RELAXED) != 0 &&
         __atomic_exchange_n(word, 0u, __ATOMIC_ACQ_REL) != 0;
}

} // namespace

unsigned *stage_error_word(cudaStream_t s) {
  if (tensor_map_encoder() == nullptr) return nullptr;
  int const dev = current_device();
  unsigned *const words = error_words(dev);
  if (words == nullptr) return nullptr;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) cudaGetLastError();
  return words + (capture != cudaStreamCaptureStatusNone
                      ? kStreamWords
                      : stream_slot(dev, s));
}

void check_stage_errors(cudaStream_t s) {
  int const dev = current_device();
  if (dev < 0 || dev >= Occupancy::kMaxDevices) return;
  unsigned *const words = g_error_words[dev].load(std::memory_order_acquire);
  if (words == nullptr) return;
  bool const own = take_error(words + stream_slot(dev, s));
  bool const captured = take_error(words + kStreamWords);
  if (own || captured)
    throw StatusError(PALIWA_GB_TIMEOUT,
                      own ? "a bounded wait of an earlier transform's tile "
                            "copies on this stream gave up"
                          : "a bounded wait of a captured transform's tile "
                            "copies gave up");
}

unsigned *begin_stages(cudaStream_t s) {
  check_stage_errors(s);
  return stage_error_word(s);
}

void launch_stage(int dtype, bool exact, bool symmetric, int ws,
                  LiftParams const &params, Stage const &st, unsigned *error,
                  cudaStream_t s) {
  int const sched =
      ws >= 0 && canonical_shifts(st.job, (ws & 1) != 0) ? ws : -1;
  if (st.R >= kHeadsIn) {
    LiftParams p = params;
    p.job = st.job;
    return launch_heads(sched, st.R, p, st.tiles, s);
  }
  if (st.tma && error != nullptr) {
    TWideParams p;
    std::memset(&p, 0, sizeof(p));
    p.heads = reinterpret_cast<uint4 *>(st.heads);
    p.head_columns = st.job.columns;
    int tsched = sched;
    if (sched < 0) {
      tsched = kTableSched + (canonical_shifts(st.job, true) ? 1 : 0);
      p.filters.npasses = params.npasses;
      p.filters.c1_one_mask = params.c1_one_mask;
      std::copy_n(params.offsets, kMaxPasses, p.filters.offsets);
      std::copy_n(params.coeffs, kMaxPasses, p.filters.coeffs);
    }
    int const code = twide_code(st, dtype);
    if (code != 0 && twide_enough(code, dtype, stage_points(st)) &&
        table_enough(st, dtype) &&
        twide_job(st, dtype, p.job, p.map, p.total_tiles)) {
      p.error = error;
      return launch_twide(dtype, exact, tsched, code, p, s);
    }
  }
  if (st.heads != 0)  // (planned with an error word and its maps accepted)
    throw StatusError(PALIWA_GB_CUDA_ERROR,
                      "the tensor map of a windowed stage was refused");
  LiftParams p = params;
  p.job = st.job;
  launch_lift(dtype, exact, symmetric, sched, st.R, p, nullptr, 1, st.tiles,
              s);
}

} // namespace pgb
