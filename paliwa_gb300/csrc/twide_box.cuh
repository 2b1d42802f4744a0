// Boxed form of the TMA wide kernel: strided pencils of 128 to 512 points (8
// to 32 chunks of floats, 4 to 16 of doubles) in rows of 128 bytes, and the
// 512-point windows of longer pencils.
//
// A tile is 64 KB: 512 / n blocks of 128 bytes of adjacent columns (32 floats
// or 16 doubles) by the n rows of their pencils. Every chunk of a block is one
// box of the axis' 3D tensor map, {128 bytes, R rows, 1}, with the 128-byte
// swizzle (the 16-byte piece q of the row at shared-memory address a lies at
// q ^ (a / 128 mod 8)). A box takes R + 1 rows of shared memory, so the
// swizzle phase of a row advances by one from chunk to chunk, and the chunks
// a warp reads together (rows R apart) lie on different banks: at most two
// wavefronts above the minimum for 32 chunks, none for 16.
//
// Against the chunk-interleaved layout of twide_kernel (rows of 32 bytes, one
// box per tile) a box row is four times as long. That is what a box row costs
// where the rows of a pencil lie on pages of their own (see the dispatch in
// periodic_kernels), and every chunk may come from a source of its own: a
// window's segment from the grid, its halo from the halo buffer.
//
// Windows (job.win.seg_len > 0). The window of segment s is the points
// [s seg_len - halo, s seg_len - halo + 512) modulo the pencil. Its outermost
// chunks are loaded from the halo buffer (the neighbouring windows overwrite
// the grid) and not stored; the levels run as on a periodic pencil, which
// reaches only points outside the segment's dependency cone.
//
// HEADS (FP32c windows): the chunk heads, every 16th point of the pencil, are
// the points of the coarse levels' stage. A forward window also writes its
// segment's heads to p.heads as unrounded double-float pairs, and an inverse
// window takes its heads from there: rounding every 16th point to its storage
// between the two stages would be eight times the rounding of the staged
// kernel's split at every 128th.
//
// The CTA is warp-specialised as twide_kernel's, with one CTA of 512 (doubles
// 256) transform threads per SM and three tiles in flight. Lane b of the
// producer warp issues the tile's box b, load and store.
#pragma once

#include "twide.cuh"

namespace pgb {

__host__ __device__ constexpr int box_threads(int r) {
  return r >= 32 ? 256 : 512;
}
constexpr int kBoxStages = 3;
// Rows of 128 bytes per tile, and bytes of one box with its pad.
constexpr int kBoxRows = 512;
__host__ __device__ constexpr int box_bytes_padded(int r) {
  return (r + 1) * 128;
}
template <int R> constexpr size_t box_smem_bytes() {
  return size_t(kBoxStages) * (kBoxRows / R) * box_bytes_padded(R) + 1024;
}

template <class A, int R, class Sched, bool HEADS>
__global__ void __launch_bounds__(box_threads(R) + 32, 1)
    twide_box_kernel(__grid_constant__ const TWideParams p) {
  using V = typename A::V;
  using W = typename A::Store;
  static_assert(sizeof(W) == 8, "rows of 8 bytes");
  constexpr int NT = box_threads(R);
  constexpr int S = kBoxStages;
  constexpr int NB = kBoxRows / R;  // boxes per tile: one per producer lane
  static_assert(NB <= 32 && NT == 16 * NB, "16 columns of 8 bytes per box");
  constexpr int LOG2NB = Log2<NB>::value;
  constexpr int LOG2R = Log2<R>::value;
  constexpr int BOX = box_bytes_padded(R);
  constexpr int TILE = NB * BOX;
  static_assert(TILE % 1024 == 0, "swizzle phase 0 at every tile");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned const base_addr = smem_u32(smem_raw);
  unsigned char *const tiles = smem_raw + ((1024 - (base_addr & 1023)) & 1023);
  __shared__ uint64_t full[S], empty[S];
  __shared__ TWideJob sjob[S];
  __shared__ int abort_flag;  // set when a bounded wait gave up
  int volatile *const abort = &abort_flag;

  int const t = threadIdx.x;
  int const lane = t & 31;
  long long const first = blockIdx.x;
  long long const step = gridDim.x;
  if (first >= p.total_tiles) return;
  long long const ntiles = (p.total_tiles - first + step - 1) / step;

  if (t == 0) {
    for (int b = 0; b < S; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], NT);
    }
    *abort = 0;
    fence_mbar_init();
  }
  __syncthreads();  // the CTA's only barrier

  if (t >= NT) {
    // Producer warp.
    TWideJob const *const jobs = p.jobs != nullptr ? p.jobs : &p.job;
    CUtensorMap const *const maps = p.jobs != nullptr ? p.maps : p.map;
    int fenced = p.jobs != nullptr ? -1 : 0;
    // This lane's box of `tile`: its map coordinates, and whether it is the
    // tile's own (of the segment, for a window).
    auto box = [&](TWideJob const &job, long long tile, int &x, int &y,
                   int &z) {
      int const log2G = job.log2_n - LOG2R;
      int const c = lane & ((1 << log2G) - 1);
      long long ct = tile - job.tile_begin;
      int seg = 0;
      if (job.win.seg_len > 0) {
        seg = static_cast<int>(ct / job.win.col_tiles);
        ct -= static_cast<long long>(seg) * job.win.col_tiles;
      }
      long long const col =
          ((ct << (LOG2NB - log2G)) + (lane >> log2G)) << 5;
      z = static_cast<int>(col >> job.log2_inner);
      x = static_cast<int>(col & ((1LL << job.log2_inner) - 1));
      y = c << LOG2R;
      if (job.win.seg_len == 0) return true;
      int const n = 1 << job.win.log2_full;
      bool const own = static_cast<unsigned>(y - job.win.halo) <
                       static_cast<unsigned>(job.win.seg_len);
      y += seg * job.win.seg_len - job.win.halo;
      bool const in = y < n;
      y &= n - 1;
      return own && in;
    };
    auto issue_load = [&](long long k) {
      int const b = static_cast<int>(k % S);
      long long const tile = first + k * step;
      __syncwarp();  // every lane is done with the buffer's last job
      if (lane == 0) {
        sjob[b] = jobs[p.tile_job != nullptr ? p.tile_job[tile] : 0];
        mbar_expect_tx(&full[b], static_cast<unsigned>(NB * R * 128));
      }
      __syncwarp();
      TWideJob const &job = sjob[b];
      if (job.map != fenced) {
        fence_tensormap(maps + job.map);
        if (job.win.seg_len > 0) fence_tensormap(maps + job.win.halo_map);
        fenced = job.map;
      }
      if (lane < NB) {
        int x, y, z;
        bool const own = box(job, tile, x, y, z);
        tma_load_3d(tiles + b * TILE + lane * BOX,
                    maps + (own ? job.map : job.win.halo_map), x, y, z,
                    &full[b]);
      }
    };
    auto issue_store = [&](long long k) {
      int const b = static_cast<int>(k % S);
      TWideJob const &job = sjob[b];
      if (lane < NB) {
        int x, y, z;
        if (box(job, first + k * step, x, y, z))
          tma_store_3d(maps + job.map, x, y, z,
                       tiles + b * TILE + lane * BOX);
      }
      bulk_commit();
    };
    long long issued = 0;
    for (; issued < S && issued < ntiles; ++issued) issue_load(issued);
    bool failed = false;
    for (long long k = 0; k < ntiles; ++k) {
      int const b = static_cast<int>(k % S);
      bool const ok = mbar_wait_bounded(
          &empty[b], static_cast<unsigned>((k / S) & 1), abort);
      if (!__all_sync(0xffffffffu, ok)) {
        failed = true;
        break;
      }
      issue_store(k);
      if (issued < ntiles) {  // issued == k + S: the next tile for buffer b
        bulk_wait_read_all();  // this lane's store has read its box
        issue_load(issued);
        ++issued;
      }
    }
    if (failed) {
      if (lane == 0) {
        atomicExch(p.error, 1u);
        *abort = 1;
      }
      // Wait (bounded) for the last load issued into each buffer, so that
      // no copy is in flight when the CTA's shared memory goes away.
      for (long long q = issued > S ? issued - S : 0; q < issued; ++q)
        mbar_wait_bounded(&full[q % S], static_cast<unsigned>((q / S) & 1),
                          nullptr);
    }
    bulk_wait_all();
    return;
  }

  // HEADS: this thread's head in tile k (nullptr past the last column; own:
  // of the tile's segment). A launch with heads has one job of 512-point
  // windows (32 chunks, one block per tile): chunk = lane, column = warp.
  auto head_of = [&](long long k, bool &own) -> uint4 * {
    TWideJob const &job = p.job;
    long long const tile = first + k * step;
    int const seg = static_cast<int>(tile / job.win.col_tiles);
    long long const ct =
        tile - static_cast<long long>(seg) * job.win.col_tiles;
    long long const col = (ct << 5) + 2 * (t >> 5);
    long long const z = col >> job.log2_inner;
    int const x = static_cast<int>(col & ((1LL << job.log2_inner) - 1));
    int const w = lane << LOG2R;
    int y = seg * job.win.seg_len - job.win.halo + w;
    int const n = 1 << job.win.log2_full;
    own = static_cast<unsigned>(w - job.win.halo) <
              static_cast<unsigned>(job.win.seg_len) &&
          y < n;
    y &= n - 1;
    if (col >= p.head_columns) return nullptr;
    return p.heads +
           ((((z << (job.win.log2_full - LOG2R)) + (y >> LOG2R))
             << (job.log2_inner - 1)) +
            (x >> 1));
  };

  // Transform threads.
  for (long long k = 0; k < ntiles; ++k) {
    int const b = static_cast<int>(k % S);
    uint4 *head = nullptr;
    bool own = false;
    uint4 head_in = {};
    if constexpr (HEADS) {
      head = head_of(k, own);
      // (the load runs while the tile's boxes land)
      if constexpr (!Sched::kForward)
        if (head != nullptr) head_in = *head;
    }
    bool const ok = mbar_wait_bounded(
        &full[b], static_cast<unsigned>((k / S) & 1), abort);
    // A warp leaves as a whole (its lanes exchange by shuffles).
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) {
        atomicExch(p.error, 1u);
        *abort = 1;
      }
      break;
    }
    TWideJob const &job = sjob[b];
    int const log2G = job.log2_n - LOG2R;
    if (log2G >= 1 && log2G <= LOG2NB) {
      // Thread = (chunk c, column g of 8 bytes): the chunks of a column are
      // lanes 32 / G apart, columns run over the tile's blocks of 16.
      int const log2ls = 5 - log2G;
      int const c = lane >> log2ls;
      int const g = ((t >> 5) << log2ls) | (lane & ((1 << log2ls) - 1));
      int const bi = ((g >> 4) << log2G) + c;
      int const q = (g & 15) >> 1;
      unsigned char *const mine =
          tiles + b * TILE + bi * BOX + ((g & 1) << 3);
      // The rows' swizzled pieces repeat every 8 rows.
      int piece[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) piece[j] = (q ^ ((bi + j) & 7)) << 4;
      V v[R];
#pragma unroll
      for (int j = 0; j < R; ++j)
        v[j] = A::load(
            *reinterpret_cast<W const *>(mine + j * 128 + piece[j & 7]));
      if constexpr (HEADS && !Sched::kForward) v[0] = RowDF::load(head_in);
      RoundCtx<A, NT, true> ctx(t, c, 1 << log2G, log2G, lane, 1, nullptr,
                                nullptr, log2ls);
      twide_levels<Sched, A, R, NT>(v, ctx, job.nlevels, p);
      if constexpr (HEADS && Sched::kForward)
        if (own && head != nullptr) *head = RowDF::store(v[0]);
#pragma unroll
      for (int j = 0; j < R; ++j)
        *reinterpret_cast<W *>(mine + j * 128 + piece[j & 7]) =
            A::store(v[j]);
    } else if (lane == 0) {
      atomicExch(p.error, 1u);
    }
    fence_proxy_async_smem();  // the writes above, before the tile's store
    mbar_arrive(&empty[b]);
  }
}

} // namespace pgb
