// Tile-owning gridding.
//
// The grid is cut into tiles of TW (u) x TV (v) cells.  After the sort each
// tile's (visibility, tile) records are contiguous (ordered by plane where
// there are many plane groups); a tile's record range is cut into work items
// of at most `chunk` records.  k_prepare_records turns the sorted records into
// descriptors; then every warp of the persistent gridding kernel works by
// itself: it takes a band of a work item (8 lane rows by the tile's columns)
// from a queue and keeps the band's cells in registers: lane (lx, ly) owns
// column lx and kRows consecutive rows.  For every record whose footprint
// meets its rows the warp multiplies the visibility by the kernel taps of its
// own cells and accumulates -- no atomics, no shared-memory
// read-modify-write.  A tile with one item is then added to the grid in place
// with one coalesced read-modify-write per band; a tile split over several
// items writes one partial tile per item and k_reduce_partials (or
// k_reduce_phases) adds them to the grid in item order, so the result does
// not depend on scheduling.
//
// The bands of a tile are far from equally loaded where the visibilities
// crowd (in a simulation of eight warps sharing one stream of records they
// were busy 81 % of the time on 512-station tracks over 8192^2, 44 % on
// 128-station ones over 2048^2), so they are units of their own.
//
// What bounds it: each complex multiply-add needs one 8-byte tap that no
// register holds, so a warp's 32 taps cost two cycles of the SM's L1 data
// pipe, and a step (a record on a band, 8 rows) 16 at least; as about half of
// the lanes and rows of a step lie inside its footprint, about half of that
// serves no multiply-add.  The pass takes about 33 cycles a step where it
// took 40 to 50, and the instructions issued (about 65 a step) come next.
// What led there, passes in ms (8192^2: 2.2e6 points, uniform w; 7.8e6 track
// points, 339 planes; 16 grids of 2048^2, 1.1e7 points):
//                                               5.6   8.0  15.6
//   taps of long runs no longer copied into
//   shared memory first (the copies' slots took
//   the L1 capacity of all other records), rows
//   unfolded (StackView)                        5.6   5.8  11.7
//   warps of their own, plain FMAs              5.2   5.7   8.8
//   everything a lane needs of a record worked
//   out once when it is queued, packed FMAs     4.6   5.4   8.7
//   32-bit tap offsets (load_taps)              4.4   5.1   8.1
//
// Three warp shapes share the 2048-cell tile: TW = 32 (32 x 64 tiles, for
// large footprints), 16 (16 x 128) and 8 (8 x 256, for small footprints,
// where a 32-wide warp would leave most lanes outside the footprint).  Each
// lane row of the narrow ones takes its own records.
//
// Tile phases (TileGeom::tile_phases): up to eight tile grids, each offset
// by a strip of TW / phases columns from the last; every visibility's
// records are on the grid that cuts its footprint into the fewest tile
// columns, so fewer warp steps fall on footprints cut by a tile boundary.
// One launch takes all the phases of a plane group: phase 0's single-item
// tiles add to the grid as above, every other item writes a partial tile,
// and k_reduce_phases adds those per cell in phase order after the launch
// (where the grid is the caller's host memory in place, reading and writing
// it per strip as the strip's first and last passes would).
//
// The reference's equivalent is oskar_process_tiles_dynamic
// (oskar_grid_wproj_gpu.cu:840-1309), a one-warp-per-32x16-tile kernel that
// flushes with float atomics whenever its tile changes.
//
// FP32 accumulation is compensated: the records of each run of 128 are summed
// in plain FP32 FMA, then folded into a (hi, lo) pair by Knuth's TwoSum, so
// rounding error does not grow with the number of visibilities on a cell.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "gg_internal.h"
#include "gg_tiles.cuh"

namespace gg {

namespace {

// A prepared record: slice_record's descriptor and the weighted visibility.
template <typename Real>
struct alignas(16) Record {
  uint2 d;
  typename Vec2<Real>::type v;
};
// FP64: also the tile rows of the footprint (in what would be padding).
template <>
struct alignas(16) Record<double> {
  uint2 d;
  int row0, row1;
  double2 v;
};

// The lane-row groups (kRows rows each, at most 32) of a tile that a
// record's footprint meets, first | last << 5, with bit 15 set where its
// kernel is conjugated (ww > 0).
constexpr uint32_t kSpanConj = 1u << 15;
constexpr uint32_t kSpanNone = 31u;   // first 31, last 0: meets none
__device__ __forceinline__ bool span_meets(uint32_t span, int group) {
  return (int)((span >> 5) & 31u) >= group && (int)(span & 31u) <= group;
}

// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

template <typename Real>
struct GridArgs {
  const WorkItem* items;
  const uint32_t* group_items;  // queue start of each virtual group
  int group;                     // the launch's first virtual group
  int group_span;                // virtual groups in the launch
  uint32_t* counter;
  const uint32_t* rec_vis;
  const Placed<Real>* placed;
  Record<Real>* recs;       // prepared records, in sorted order
  unsigned short* spans;    // and the rows they meet
  StackView view;
  TileGeom geom;
  int grid_size;
  Real* grid;
  long long grid_stride;
  typename Vec2<Real>::type* partials;
  // Direct mode (single grid, tile_groups non-null): the caller's grid at
  // host, addressed in place.  tile_groups[tile] = first | last << 16, the
  // first and last plane group with records in the tile: the first reads
  // the tile's cells from host, the last writes them to host, the others
  // go through grid (scratch).
  Real* host;
  const uint32_t* tile_groups;
};

// Source and destination of a grid cell's read-modify-write in virtual
// group `group`: the scratch grid g, or the caller's grid h in direct mode.
// Direct mode keeps, per strip of tile_u / tile_phases columns of a tile
// row, the first and last virtual group whose tiles hold records there
// (k_tile_groups): the first reads the cells from h, the last writes them
// to h, the others go through g.
template <typename R2>
__device__ __forceinline__ void cell_ends(const uint32_t* tile_groups,
                                          const TileGeom& geom, int tv,
                                          int col, int group, R2* g, R2* h,
                                          R2*& src, R2*& dst) {
  src = g;
  dst = g;
  if (tile_groups) {
    const uint32_t fl = tile_groups[tv * geom.strips_u + (col >> geom.strip_shift)];
    if ((int)(fl & 0xFFFFu) == group) src = h;
    if ((int)(fl >> 16) == group) dst = h;
  }
}

// The first column and row of a virtual tile.
template <int TW>
__device__ __forceinline__ int2 tile_origin(const TileGeom& g, int tile) {
  using WS = WarpShape<TW>;
  const int vg = tile / g.tiles_total;   // virtual group
  const int tl = (tile - vg * g.tiles_total) % (g.tiles_u * g.tiles_v);
  return make_int2((tl % g.tiles_u) * WS::kTileU - phase_shift(g, vg),
                   (tl / g.tiles_u) * WS::kTileV);
}

// The prepared record of visibility vid in the tile that starts at `tile`.
template <typename Real, int TW>
__device__ __forceinline__ void prepare_record(const GridArgs<Real>& a,
                                               int2 tile, uint32_t vid,
                                               Record<Real>& rec,
                                               uint32_t& span) {
  const Placed<Real> pt = a.placed[vid];
  const uint32_t m = pt.meta;
  const SlicePlane plane = a.view.planes[meta_plane(m)];
  const int ou = meta_ou(m), ov = meta_ov(m), s = plane.support;
  const int gu = cell_u(pt.cell) - tile.x, gv = cell_v(pt.cell) - tile.y;
  rec.d = slice_record(slice_origin(plane, a.view.omax, abs(ou), abs(ov)), s,
                       ou, ov, gu, gv);
  rec.v = pt.v;
  if constexpr (sizeof(Real) == 8) {
    rec.row0 = gv - s;
    rec.row1 = gv + s;
  }
  // The tile meets each of its records: clipped to it.
  span = (uint32_t)(max(gv - s, 0) / kRows) |
         (uint32_t)(min(gv + s, WarpShape<TW>::kTileV - 1) / kRows) << 5 |
         (meta_conj(m) ? kSpanConj : 0u);
  if (m & kMetaOdd) span = kSpanNone;   // k_grid_odd's
}

// Prepares the records of every work item of the call: one block per item at
// a time.  HBM-bound: 4 B of index and one sector at random per record in,
// 18 B (FP64: 34 B) out.
template <typename Real, int TW>
__global__ void __launch_bounds__(128)
k_prepare_records(GridArgs<Real> a, int num_groups) {
  const int num_items = (int)a.group_items[num_groups];
  // The first gridding launch's work counter.
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.counter = 0;
  for (int it = blockIdx.x; it < num_items; it += gridDim.x) {
    const WorkItem item = a.items[it];
    const int2 tile = tile_origin<TW>(a.geom, item.tile);
    const uint32_t n = item.rec_end - item.rec_begin;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
      const uint32_t i = item.rec_begin + k;
      Record<Real> rec;
      uint32_t span;
      prepare_record<Real, TW>(a, tile, a.rec_vis[i], rec, span);
      a.recs[i] = rec;
      a.spans[i] = (unsigned short)span;
    }
  }
}

// A queued record of a lane-row group: everything the group's lanes need for
// it, worked out by the one lane that queues it.  The tap of the lane at tile
// column col in the group's row r is
//   taps[x + r * step + su * clamp(col - gu, -S, S)]
// with S = s + 1 (the clamped ends are zero taps) and step = +-2S; the record
// adds (a, d) * (t.re, t.im) to the cell's P and (c, b) * (t.re, t.im) to its
// Q, and re = P.x + Q.y, im = Q.x + P.y (two packed FMAs a cell).
struct alignas(16) Queued {
  uint32_t x;
  int gu_su;    // gu << 16 | (su & 0xFFFF)
  int S, step;
  float a, d, c, b;
};
__device__ __forceinline__ Queued queued(const Record<float>& r, uint32_t span,
                                         int group) {
  Queued q;
  const int z = (int)(short)(r.d.y & 0xFFFFu);
  const int s = (int)((r.d.y >> 16) & 0x3FFFu);
  const bool mu = (r.d.y & kMirrorU) != 0u, conj = (span & kSpanConj) != 0u;
  q.S = s + 1;
  q.step = slice_step(r.d);
  q.x = r.d.x + (uint32_t)(group * kRows * q.step + s);
  const int gu = mu ? z - s : s - z;
  q.gu_su = (int)((uint32_t)gu << 16 | (mu ? 0xFFFFu : 1u));
  q.a = r.v.x;
  q.c = r.v.y;
  q.d = conj ? -r.v.x : r.v.x;
  q.b = conj ? r.v.y : -r.v.y;
  return q;
}

// Shared memory of one warp of the gridding kernel.
template <int TW>
struct WarpSmem {
  static constexpr int kQueue = 64;
  float2 hi[kRows][32];
  float2 lo[kRows][32];
  // Records waiting for each lane-row group, a ring.
  Queued queue[WarpShape<TW>::kLanesY][kQueue];
};

constexpr int kGridWarps = 4;    // per block of the gridding kernel
constexpr int kGridThreads = kGridWarps * 32;
static_assert(kGridWarps * kBlocksPerTeam == kWarps, "a team");

// kPrepared: the records come from k_prepare_records; else (a call for which
// those do not fit the device's memory) every band's warp prepares them itself.
template <int TW, bool kWide, bool kPrepared>
__global__ void __launch_bounds__(kGridThreads, 5)
k_grid_tiles(GridArgs<float> a) {
  constexpr int kDepth = 2;   // records in flight per warp
  using R2 = float2;
  using WS = WarpShape<TW>;
  using SM = WarpSmem<TW>;
  constexpr int G = WS::kLanesY, Q = SM::kQueue;
  extern __shared__ __align__(16) unsigned char g_smem_raw[];
  const int lane = threadIdx.x & 31;
  SM& sm = reinterpret_cast<SM*>(g_smem_raw)[threadIdx.x >> 5];
  const int lx = lane % TW, ly = lane / TW;
  const R2* __restrict__ stack = (const R2*)a.view.taps;
  const uint32_t lt = (1u << lane) - 1u;
  // The launch's units: the bands of its virtual groups' items.
  const unsigned first = a.group_items[a.group];
  const unsigned units =
      (a.group_items[a.group + a.group_span] - first) * kWarps;
  unsigned next = 0;
  if (lane == 0) next = atomicAdd(a.counter, 1u);
  for (;;) {
    const unsigned unit = __shfl_sync(0xffffffffu, next, 0);
    if (unit >= units) return;
    if (lane == 0) next = atomicAdd(a.counter, 1u);   // used in the next turn
    const WorkItem item = a.items[first + unit / kWarps];
    const int band = (int)(unit % kWarps);
    const int g0 = band * G;   // first lane-row group

    R2 acc[kRows], acq[kRows];   // P and Q
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      acc[r] = acq[r] = R2{};
      sm.hi[r][lane] = sm.lo[r][lane] = R2{};
    }
    R2 tp[kDepth][kRows];
    // Queue positions: `at` the oldest record not yet added (the kDepth from
    // there on are being loaded once `primed`), tails the ends.
    int at = 0, tails[G];
    bool primed = false;
#pragma unroll
    for (int g = 0; g < G; ++g) tails[g] = 0;
    Queued* const queue = sm.queue[ly];
    auto load = [&](int i, R2 (&out)[kRows]) {
      const int4 e = *(const int4*)&queue[i & (Q - 1)];
      const int t = min(max(lx - (e.y >> 16), -e.z), e.z);
      load_taps<kWide>(stack, (uint32_t)(e.x + (int)(short)e.y * t), e.w, out);
    };
    auto add = [&](int i, const R2 (&t)[kRows]) {
      const Queued& e = queue[i & (Q - 1)];
      R2 p, q;
      p.x = e.a; p.y = e.d;
      q.x = e.c; q.y = e.b;
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        acc[r] = fma2(p, t[r], acc[r]);
        acq[r] = fma2(q, t[r], acq[r]);
      }
    };
    // Adds queued records, kDepth at a time, while every queue holds another
    // kDepth to load behind them.
    auto run = [&](int end) {
      if (!primed && end - at >= kDepth) {
#pragma unroll
        for (int d = 0; d < kDepth; ++d) load(at + d, tp[d]);
        primed = true;
      }
      for (; end - at >= 2 * kDepth; at += kDepth) {
#pragma unroll
        for (int d = 0; d < kDepth; ++d) {
          add(at + d, tp[d]);
          load(at + kDepth + d, tp[d]);
        }
      }
    };
    // Fills every queue up to `end` with records that add nothing.
    auto fill = [&](int end) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g == ly)
          for (int i = tails[g] + lx; i < end; i += TW) {
            Queued none{};
            none.x = kStackZero;
            queue[i & (Q - 1)] = none;
          }
        tails[g] = max(tails[g], end);
      }
      __syncwarp();
    };
    auto fold = [&]() {
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        R2 hi = sm.hi[r][lane], lo = sm.lo[r][lane];
        float s, e;
        two_sum(hi.x, acc[r].x + acq[r].y, s, e); hi.x = s; lo.x += e;
        two_sum(hi.y, acq[r].x + acc[r].y, s, e); hi.y = s; lo.y += e;
        sm.hi[r][lane] = hi;
        sm.lo[r][lane] = lo;
        acc[r] = acq[r] = R2{};
      }
    };

    uint32_t span = kSpanNone;
    Record<float> rec;
    // Record positions: ints below kWideRecords; in the wide kernels all 32
    // bits, where i + 32 may wrap and the distance to the end is tested (in
    // every call that took 8192^2 workloads 1 % longer, 4.82 and 4.87 ms).
    using Pos = std::conditional_t<kWide, uint32_t, int>;
    const Pos rec_end = (Pos)item.rec_end;
    auto before_end = [&](Pos i, int k) {
      if constexpr (kWide) return (uint32_t)k < rec_end - i;
      else return i + k < rec_end;
    };
    auto fetch = [&](Pos i) {
      span = kSpanNone;
      if (before_end(i, lane)) {
        if constexpr (kPrepared) {
          span = a.spans[i + lane];
          rec = a.recs[i + lane];
        } else {
          prepare_record<float, TW>(a, tile_origin<TW>(a.geom, item.tile),
                                    a.rec_vis[i + lane], rec, span);
        }
      }
    };
    fetch((Pos)item.rec_begin);
    for (Pos i = (Pos)item.rec_begin; kWide || i < rec_end; i += 32) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const bool hit = span_meets(span, g0 + g);
        const uint32_t b = __ballot_sync(0xffffffffu, hit);
        if (hit)
          sm.queue[g][(tails[g] + __popc(b & lt)) & (Q - 1)] =
              queued(rec, span, g0 + g);
        tails[g] += __popc(b);
      }
      if (before_end(i, 32)) fetch(i + 32);
      __syncwarp();
      int lo = tails[0], hi = tails[0];
#pragma unroll
      for (int g = 1; g < G; ++g) {
        lo = min(lo, tails[g]);
        hi = max(hi, tails[g]);
      }
      run(lo);
      // A queue without room for another 32 records goes on alone.
      if (G > 1 && hi - at > Q - 32) {
        fill(hi - (hi - at) % kDepth);
        run(hi - (hi - at) % kDepth);
      }
      // Plain FP32 sums of at most 128 records (and the few in flight) go
      // into the compensated (hi, lo) pair.
      if (((i - (Pos)item.rec_begin) & 96) == 96) fold();
      __syncwarp();
      if (kWide && !before_end(i, 32)) break;
    }
    int end = tails[0];
#pragma unroll
    for (int g = 1; g < G; ++g) end = max(end, tails[g]);
    if (end > at) {
      end = at + (end - at + kDepth - 1) / kDepth * kDepth;
      fill(end);
      run(end);
#pragma unroll
      for (int d = 0; d < kDepth; ++d) add(at + d, tp[d]);
    }
    __syncwarp();   // the queues are free for the next unit
    fold();
    // An owned band that no record meets stays as it is (in direct mode its
    // cells may still have to move between the host and the scratch grid).
    if (end == 0 && item.slot < 0 && !a.tile_groups) continue;

    // ---- flush the band ---------------------------------------------------
    const int tiles_per_grid = a.geom.tiles_u * a.geom.tiles_v;
    const int rt = item.tile % a.geom.tiles_total;   // real tile
    const int gi = rt / tiles_per_grid;
    const int tl = rt - gi * tiles_per_grid;
    const int vg = item.tile / a.geom.tiles_total;   // virtual group
    R2 out[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const R2 hi = sm.hi[r][lane], lo = sm.lo[r][lane];
      out[r].x = hi.x + lo.x;
      out[r].y = hi.y + lo.y;
    }
    if (item.slot < 0) {
      const int col =
          (tl % a.geom.tiles_u) * WS::kTileU - phase_shift(a.geom, vg) + lx;
      const int row0 = (tl / a.geom.tiles_u) * WS::kTileV +
                       (g0 + ly) * kRows;
      // Phase tiles reach past the grid's first and last columns.
      const bool col_in = (unsigned)col < (unsigned)a.grid_size;
      R2 *src, *dst;
      cell_ends<R2>(a.tile_groups, a.geom, tl / a.geom.tiles_u,
                    col_in ? col : 0, vg,
                    (R2*)(a.grid + (long long)gi * a.grid_stride),
                    (R2*)a.host, src, dst);
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        const int row = row0 + r;
        if (row < a.grid_size && col_in) {
          const size_t off = (size_t)row * a.grid_size + col;
          R2 old = __ldcs(src + off);
          old.x += out[r].x;
          old.y += out[r].y;
          __stcs(dst + off, old);
        }
      }
    } else {
      // Partial tile, thread-major: entry r * kConsumers + band * 32 + lane.
      R2* p = a.partials + (size_t)item.slot * kCells + band * 32 + lane;
#pragma unroll
      for (int r = 0; r < kRows; ++r) __stcs(p + r * kConsumers, out[r]);
    }
  }
}

// A queued record of the FP64 kernel: its footprint clipped to the warp's band,
// w columns of n cells, row by row.  Cell i of it lies in row i / w, column
// i % w: band cell `cell` + row * TW + column, tap x + row * step + su *
// column.  (a, d, c, b): the coefficients of t.re (a, c) and t.im (b, d) in re
// and im.
struct alignas(16) Queued64 {
  uint32_t x;
  int su, step, cell;
  int n, w;
  float inv_w;
  double a, b, c, d;
};

constexpr int kBandCells = kCells / kWarps;   // 256

struct WarpSmem64 {
  double2 acc[kBandCells];
  Queued64 queue[32];
};

// The gridding kernel in FP64.  The FP64 pipe bounds it (a warp's FMA takes
// 16 cycles of the SM however few of its lanes are active, four of them for
// 32 cells), so the lanes take a record's cells in the band packed row by row,
// whatever the footprint's position, instead of a column each: of the cells
// of a record on a band about half are inside its footprint (2048^2, 2e5
// points, 128 planes, support 4 to 24), of the packed ones 95 %.  The band's
// sums lie in shared memory, a read and a write of 16 bytes a cell that the
// pipe hides; a warp adds its records one after the other, so no two lanes
// meet in a cell.  That workload's pass: 4.1 ms with a column a lane and
// band rows in registers, 2.15 so (the multiply-adds alone 1.73).  Eight
// cells a lane in flight, three blocks: 2.15; four cells and four to six
// blocks 2.18 to 2.2, as the units in flight at the end are more.
template <int TW, bool kPrepared>
__global__ void __launch_bounds__(kGridThreads, 3)
k_grid_tiles_f64(GridArgs<double> a) {
  using WS = WarpShape<TW>;
  constexpr int kAhead = 8;   // cells of a lane in flight
  extern __shared__ __align__(16) unsigned char g_smem_raw[];
  const int lane = threadIdx.x & 31;
  WarpSmem64& sm =
      reinterpret_cast<WarpSmem64*>(g_smem_raw)[threadIdx.x >> 5];
  const double2* __restrict__ stack = (const double2*)a.view.taps;
  const unsigned first = a.group_items[a.group];
  const unsigned units =
      (a.group_items[a.group + a.group_span] - first) * kWarps;
  unsigned next = 0;
  if (lane == 0) next = atomicAdd(a.counter, 1u);
  for (;;) {
    const unsigned unit = __shfl_sync(0xffffffffu, next, 0);
    if (unit >= units) return;
    if (lane == 0) next = atomicAdd(a.counter, 1u);   // used in the next turn
    const WorkItem item = a.items[first + unit / kWarps];
    const int band = (int)(unit % kWarps);
    const int row0 = band * WS::kBand;
    for (int i = lane; i < kBandCells; i += 32) sm.acc[i] = double2{};
    bool any = false;
    uint32_t span = kSpanNone;
    Record<double> rec;
    auto fetch = [&](uint32_t i) {
      span = kSpanNone;
      if ((uint32_t)lane < item.rec_end - i) {
        if constexpr (kPrepared) {
          span = a.spans[i + lane];
          rec = a.recs[i + lane];
        } else {
          prepare_record<double, TW>(a, tile_origin<TW>(a.geom, item.tile),
                                     a.rec_vis[i + lane], rec, span);
        }
      }
    };
    fetch(item.rec_begin);
    for (uint32_t i0 = item.rec_begin;; i0 += 32) {
      // The lane's record, clipped to the band and the tile.
      const int s = (int)((rec.d.y >> 16) & 0x3FFFu);
      const bool mu = (rec.d.y & kMirrorU) != 0u;
      const int z = (int)(short)(rec.d.y & 0xFFFFu);
      const int gu = mu ? z - s : s - z;
      const int c0 = max(gu - s, 0), c1 = min(gu + s, TW - 1);
      const uint32_t g0 = (uint32_t)(band * WS::kLanesY);
      const bool hit = (int)((span >> 5) & 31u) >= (int)g0 &&
                       (int)(span & 31u) < (int)g0 + WS::kLanesY && c0 <= c1;
      const uint32_t b = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int step = slice_step(rec.d);
        const int r0 = max(rec.row0 - row0, 0);
        const int r1 = min(rec.row1 - row0, WS::kBand - 1);
        Queued64 q;
        q.w = c1 - c0 + 1;
        q.n = q.w * (r1 - r0 + 1);
        q.inv_w = 1.0f / (float)q.w;
        q.su = mu ? -1 : 1;
        q.step = step;
        q.cell = r0 * TW + c0;
        q.x = rec.d.x +
              (uint32_t)((row0 + r0) * step + (mu ? z - c0 : z + c0));
        const bool conj = (span & kSpanConj) != 0u;
        q.a = rec.v.x;
        q.c = rec.v.y;
        q.d = conj ? -rec.v.x : rec.v.x;
        q.b = conj ? rec.v.y : -rec.v.y;
        sm.queue[__popc(b & ((1u << lane) - 1u))] = q;
      }
      const int count = __popc(b);
      any |= count > 0;
      const bool more = item.rec_end - i0 > 32u;
      if (more) fetch(i0 + 32);
      __syncwarp();
      for (int k = 0; k < count; ++k) {
        const Queued64& q = sm.queue[k];
        const int n = q.n, w = q.w, step = q.step, su = q.su;
        const uint32_t x = q.x;
        const float inv_w = q.inv_w;
        const double ca = q.a, cb = q.b, cc = q.c, cd = q.d;
        double2* const acc = sm.acc + q.cell;
        // Up to eight of the lane's cells at a time: their taps' loads
        // overlap.
        for (int i = lane; i < n; i += 32 * kAhead) {
          double2 t[kAhead];
          int at[kAhead];
#pragma unroll
          for (int j = 0; j < kAhead; ++j) {
            const int e = i + 32 * j;
            const int row = (int)(((float)e + 0.5f) * inv_w);
            const int col = e - row * w;
            at[j] = row * TW + col;
            t[j] = double2{};
            if (e < n)
              t[j] = ld_tap(stack + (x + (uint32_t)(row * step + su * col)));
          }
#pragma unroll
          for (int j = 0; j < kAhead; ++j) {
            if (i + 32 * j >= n) break;
            double2 v = acc[at[j]];
            v.x = fma(cb, t[j].y, fma(ca, t[j].x, v.x));
            v.y = fma(cd, t[j].y, fma(cc, t[j].x, v.y));
            acc[at[j]] = v;
          }
        }
        __syncwarp();   // the next record may add to these cells
      }
      if (!more) break;
    }
    __syncwarp();
    // An owned band that no record meets: as in k_grid_tiles.
    if (!any && item.slot < 0 && !a.tile_groups) continue;
    const int tiles_per_grid = a.geom.tiles_u * a.geom.tiles_v;
    const int rt = item.tile % a.geom.tiles_total;   // real tile
    const int gi = rt / tiles_per_grid;
    const int tl = rt - gi * tiles_per_grid;
    const int vg = item.tile / a.geom.tiles_total;   // virtual group
    const int u0 =
        (tl % a.geom.tiles_u) * WS::kTileU - phase_shift(a.geom, vg);
    const int v0 = (tl / a.geom.tiles_u) * WS::kTileV + row0;
    for (int i = lane; i < kBandCells; i += 32) {
      const double2 out = sm.acc[i];
      const int r = i / TW, c = i % TW;
      if (item.slot < 0) {
        const int col = u0 + c, row = v0 + r;
        if (row >= a.grid_size || (unsigned)col >= (unsigned)a.grid_size)
          continue;
        double2 *src, *dst;
        cell_ends<double2>(a.tile_groups, a.geom, tl / a.geom.tiles_u, col,
                           vg,
                           (double2*)(a.grid + (long long)gi * a.grid_stride),
                           (double2*)a.host, src, dst);
        const size_t off = (size_t)row * a.grid_size + col;
        double2 old = __ldcs(src + off);
        old.x += out.x;
        old.y += out.y;
        __stcs(dst + off, old);
      } else {
        // Partial tile entry of band row r, column c (see BandCell).
        const int e = r % kRows * kConsumers + r / kRows * TW + c;
        __stcs(a.partials + (size_t)item.slot * kCells + band * 32 + e, out);
      }
    }
    __syncwarp();   // acc is free for the next unit
  }
}

// Adds the kMetaOdd points, a warp each at a time, its lanes on the footprint's
// cells.  The atomics bound it; cells that are NaN already, as nearly all soon
// are, need none (2.15e6 points on 8192^2, all of them odd: 24.3 ms a call, with
// this test 14.9, none odd 4.8; a tenth 7.2 and 6.6).
__global__ void __launch_bounds__(256)
k_grid_odd(const Placed<float>* __restrict__ placed, unsigned long long n,
           const uint32_t* __restrict__ shape, StackView v, int G, float* grid,
           long long grid_stride,
           const unsigned long long* __restrict__ grid_offsets,
           int num_grids) {
  if (shape && !(*shape & kShapeOdd)) return;
  const int lane = threadIdx.x & 31;
  const unsigned long long warps = (unsigned long long)gridDim.x * 8;
  for (unsigned long long i0 =
           ((unsigned long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 32;
       i0 < n; i0 += warps * 32) {
    const uint32_t mine = i0 + lane < n ? placed[i0 + lane].meta : 0u;
    for (uint32_t b = __ballot_sync(0xffffffffu, (mine & kMetaOdd) != 0u); b;
         b &= b - 1) {
      const unsigned long long i = i0 + (__ffs(b) - 1);
      int gi = 0;
      for (int hi = num_grids - 1; gi < hi;) {   // i's grid
        const int mid = (gi + hi + 1) >> 1;
        if (grid_offsets[mid] <= i) gi = mid; else hi = mid - 1;
      }
      const Placed<float> pt = placed[i];
      const SlicePlane plane = v.planes[meta_plane(pt.meta)];
      const int s = plane.support, F = 2 * s + 1, pitch = slice_pitch(s);
      const int ou = meta_ou(pt.meta), ov = meta_ov(pt.meta);
      const float2* const taps =
          (const float2*)v.taps + slice_origin(plane, v.omax, abs(ou), abs(ov));
      const float sgn = meta_conj(pt.meta) ? -1.0f : 1.0f;
      float* const corner =
          grid + gi * grid_stride +
          2 * ((size_t)(cell_v(pt.cell) - s) * G + (cell_u(pt.cell) - s));
      for (int e = lane; e < F * F; e += 32) {
        const int row = e / F, col = e - row * F;
        const float2 t = taps[(ov < 0 ? F - 1 - row : row) * pitch +
                              (ou < 0 ? F - 1 - col : col)];
        const float ti = sgn * t.y;
        float* const c = corner + 2 * ((size_t)row * G + col);
        const float2 was = __ldcg((const float2*)c);   // a NaN stays one
        if (!isnan(was.x)) atomicAdd(c, pt.v.x * t.x - pt.v.y * ti);
        if (!isnan(was.y)) atomicAdd(c + 1, pt.v.x * ti + pt.v.y * t.x);
      }
    }
  }
}

// host += sums where these are not zero: what the kMetaOdd points add, none of
// which is finite.  Two cells a thread.
__global__ void __launch_bounds__(256)
k_add_odd(const float4* __restrict__ sums, unsigned long long pairs,
          size_t cells, float2* __restrict__ host) {
  const unsigned long long i =
      (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs) return;
  const bool two = 2 * i + 1 < cells;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (two) {
    v = sums[i];
  } else {
    const float2 one = ((const float2*)sums)[2 * i];
    v.x = one.x; v.y = one.y;
  }
  if (v.x != 0.0f || v.y != 0.0f) {
    const float2 was = host[2 * i];
    host[2 * i] = make_float2(was.x + v.x, was.y + v.y);
  }
  if (two && (v.z != 0.0f || v.w != 0.0f)) {
    const float2 was = host[2 * i + 1];
    host[2 * i + 1] = make_float2(was.x + v.z, was.y + v.w);
  }
}

// A sum in more than the call's precision.  FP32: the sum split over three
// floats by two TwoSums an addition, as an FP64 addition takes 16 cycles of the
// SM a warp, as does the conversion of what it adds, and the tiles with
// hundreds of chunks lie on a few SMs.  Only lo's own additions round: after
// settle() mid and lo are at most 2^-24 and 2^-48 of hi, so while sixteen
// values are added |mid| < 17 * 2^-24 and |lo| < 2^9 * 2^-48 of the largest
// sum so far, and an addition loses less than 2^-63 of it, where FP64 loses
// up to 2^-53.  Calls with FP64 sums and so, ms: 2e5
// uniform points on 2048^2 0.443 and 0.409; track points, four tile phases, 1e6
// on 1024^2 1.10 and 0.74, 7.8e6 on 2048^2 5.66 and 4.98.
struct WideSum32 {
  float hi, mid, lo;
  __device__ __forceinline__ explicit WideSum32(float v)
      : hi(v), mid(0), lo(0) {}
  __device__ __forceinline__ void add(float v) {
    float e;
    two_sum(hi, v, hi, e);
    two_sum(mid, e, mid, e);
    lo += e;
  }
  __device__ __forceinline__ void settle() {
    two_sum(hi, mid, hi, mid);
    two_sum(mid, lo, mid, lo);
  }
  // The three added from the small end, rounded once (twice where the sum
  // lies within 2^-24 of its last place from a tie).
  __device__ __forceinline__ float value() const {
    float a, b, c, d;
    two_sum(hi, mid, a, b);
    two_sum(b, lo, c, d);
    two_sum(a, c, a, c);
    return a + (c + d);
  }
};
struct WideSum64 {
  double s;
  __device__ __forceinline__ explicit WideSum64(double v) : s(v) {}
  __device__ __forceinline__ void add(double v) { s += v; }
  __device__ __forceinline__ void settle() {}
  __device__ __forceinline__ double value() const { return s; }
};

// v + the n partial values at q, one per chunk, in chunk order, rounded
// once.  Loads go out sixteen at a time: a heavy tile has hundreds of chunks,
// and one load per addition would leave the pass waiting out a memory latency
// for each.
template <typename Sum, int kAhead, typename R2>
__device__ __forceinline__ R2 sum_chunks(R2 v, const R2* __restrict__ q,
                                         int n) {
  Sum sx(v.x), sy(v.y);
  int c = 0;
  for (; c + kAhead <= n; c += kAhead) {
    R2 t[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) t[j] = q[(size_t)(c + j) * kCells];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      sx.add(t[j].x);
      sy.add(t[j].y);
    }
    sx.settle();
    sy.settle();
  }
  for (; c < n; ++c) {
    const R2 t = q[(size_t)c * kCells];
    sx.add(t.x);
    sy.add(t.y);
  }
  v.x = sx.value();
  v.y = sy.value();
  return v;
}

// v += the n partial values at q.  An FP32 sum that leaves FP32's range on the
// way, or meets an infinity, is formed again in FP64: only the end counts.
template <typename R2>
__device__ __forceinline__ void add_chunks(R2& v, const R2* __restrict__ q,
                                           int n) {
  if constexpr (sizeof(R2) == 8) {
    const R2 r = sum_chunks<WideSum32, 16>(v, q, n);
    v = isfinite(r.x) && isfinite(r.y) ? r
                                       : sum_chunks<WideSum64, 1>(v, q, n);
  } else {
    v = sum_chunks<WideSum64, 8>(v, q, n);
  }
}

// The cell of thread tid in a band of a tile (one cell per thread): its row
// and column in the band, and its entry in the tile's partials less the
// band's part, band * 32 (the gridding kernel's thread-major layout).
template <int TW>
struct BandCell {
  int row, col, entry;
  __device__ __forceinline__ explicit BandCell(int tid)
      : row(tid / TW), col(tid % TW),
        entry(row % kRows * kConsumers + row / kRows * TW + col) {}
};

// grid(tile) += sum of the tile's partials in chunk order, accumulated as
// add_chunks does and rounded once, for the split tiles of one plane group (a real
// tile is split at most once per group, so the blocks of one launch never
// share a tile).  A block takes one band of a tile at a time: the chains of
// chunks of a heavy tile, which the pass waits for, run on all its bands at
// once.
template <typename Real, int TW>
__global__ void __launch_bounds__(kConsumers, 4)
k_reduce_partials(const int4* __restrict__ split_tiles,
                  const uint32_t* __restrict__ num_split,
                  const typename Vec2<Real>::type* __restrict__ partials,
                  TileGeom g, int group, int G, Real* grid,
                  long long grid_stride, Real* host,
                  const uint32_t* __restrict__ tile_groups) {
  using R2 = typename Vec2<Real>::type;
  using WS = WarpShape<TW>;
  const int tiles_per_grid = g.tiles_u * g.tiles_v;
  const int n = (int)*num_split * kWarps;
  const BandCell<TW> me(threadIdx.x);
  for (int b = blockIdx.x; b < n; b += gridDim.x) {
    const int4 d = split_tiles[b / kWarps];  // virtual tile, first slot, chunks
    if (d.x / g.tiles_total != group) continue;
    const int band = b % kWarps;
    const int rt = d.x % g.tiles_total;
    const int gi = rt / tiles_per_grid;
    const int tl = rt - gi * tiles_per_grid;
    const int tv = tl / g.tiles_u;
    const int col =
        (tl - tv * g.tiles_u) * WS::kTileU - phase_shift(g, group) + me.col;
    const int row = tv * WS::kTileV + band * WS::kBand + me.row;
    if (row >= G || (unsigned)col >= (unsigned)G) continue;
    R2 *src, *dst;
    cell_ends<R2>(tile_groups, g, tv, col, group,
                  (R2*)(grid + (long long)gi * grid_stride), (R2*)host, src,
                  dst);
    const size_t off = (size_t)row * G + col;
    R2 v = src[off];
    add_chunks(v, partials + (size_t)d.y * kCells + band * 32 + me.entry, d.z);
    dst[off] = v;
  }
}

// The partial tiles of one plane group's tile phases (virtual groups
// group0 .. group0 + P - 1, one launch of the gridding kernel), added to
// the grids in one pass: a block takes two bands of a phase-0 tile position
// at a time (two cells a thread) and adds to each cell, phase by phase, the partial tiles of the
// tile of that phase that covers it (their chunks summed by add_chunks, rounded
// once per phase) -- the additions, in the same order, that one reduction
// launch per phase makes (k_reduce_partials).  A single chunk is added in
// the grid's precision: the FP64 sum of two FP32 values rounded to FP32 is
// their correctly rounded FP32 sum.  Those loads (the grid's cells and up to
// four partials each) all go out before the first addition.
// tile_slot[virtual tile] = (first partial slot, chunks), chunks 0 when the
// tile has no partial tiles.  HBM-bound but for the heavy tiles' chains.
// With whole tiles for a block (eight cells and, for heavy tiles, eight
// chains of chunks a thread) it took 0.66 ms on 7.8e6 track points over
// 8192^2 and 0.09 ms on 4e3 points over 256^2.
// kMaxPhases >= tile_phases (4 or 8).
template <typename Real, int TW, int kMaxPhases>
__global__ void __launch_bounds__(kConsumers, kMaxPhases > 4 ? 3 : 4)
k_reduce_phases(const int2* __restrict__ tile_slot,
                const typename Vec2<Real>::type* __restrict__ partials,
                TileGeom g, int group0, int G, Real* grid,
                long long grid_stride, Real* host,
                const uint32_t* __restrict__ tile_groups,
                const uint32_t* __restrict__ tile_start) {
  using R2 = typename Vec2<Real>::type;
  using WS = WarpShape<TW>;
  const int P = g.tile_phases;
  const int sw = 1 << g.strip_shift;
  const int real_u = g.tiles_u - 1;   // phase-0 tile columns
  const int tiles_per_grid = g.tiles_u * g.tiles_v;
  constexpr int kPairs = kWarps / 2;
  const int n = g.num_grids * real_u * g.tiles_v * kPairs;
  const BandCell<TW> me(threadIdx.x);
  for (int b = blockIdx.x; b < n; b += gridDim.x) {
    const int band = b % kPairs * 2, pos = b / kPairs;
    const int gi = pos / (real_u * g.tiles_v);
    const int rem = pos - gi * real_u * g.tiles_v;
    const int tv = rem / real_u, tu = rem - tv * real_u;
    const int col = tu * TW + me.col;
    const int row = tv * WS::kTileV + band * WS::kBand + me.row;
    if (col >= G || row >= G) continue;
    const bool both = row + WS::kBand < G;
    // This column's tile in each phase: its slots and its column there.
    int2 sl[kMaxPhases];
    int cp[kMaxPhases];
    bool mine = false, several = false;
#pragma unroll
    for (int p = 0; p < kMaxPhases; ++p) {
      sl[p] = make_int2(0, 0);
      cp[p] = 0;
      if (p < P) {
        const int c = col + p * sw;
        const int tc = c / TW;
        cp[p] = c - tc * TW - me.col;
        sl[p] = tile_slot[(size_t)(group0 + p) * g.tiles_total +
                          (size_t)gi * tiles_per_grid +
                          (size_t)tv * g.tiles_u + tc];
        mine |= sl[p].y > 0;
        several |= sl[p].y > 1;
      }
    }
    if (!mine) continue;
    R2* gg = (R2*)(grid + (long long)gi * grid_stride);
    // Direct mode (the caller's grid at host in place, one grid): the
    // column's strip was last added to at host unless phase 0's tile here
    // added itself to the scratch grid in the launch (it had records, one
    // item) or an earlier plane group touched the strip; the additions
    // here are the strip's last when its last virtual group is in this
    // launch.
    R2* src = gg;
    R2* dst = gg;
    if (tile_groups) {
      const uint32_t fl =
          tile_groups[tv * g.strips_u + (col >> g.strip_shift)];
      const int first = (int)(fl & 0xFFFFu), last = (int)(fl >> 16);
      const size_t vt0 = (size_t)group0 * g.tiles_total +
                         (size_t)gi * tiles_per_grid +
                         (size_t)tv * g.tiles_u + tu;
      const bool added0 =
          sl[0].y == 0 && tile_start[vt0 + 1] > tile_start[vt0];
      if (!added0 && first >= group0) src = (R2*)host;
      if (last < group0 + P) dst = (R2*)host;
    }
    const size_t off0 = (size_t)row * G + col;
    const size_t off1 = off0 + (both ? (size_t)WS::kBand * G : 0);
    const R2* const q = partials + band * 32 + me.entry;
    R2 v0 = src[off0], v1 = src[off1];
    if (!several) {
      R2 t0[kMaxPhases], t1[kMaxPhases];
#pragma unroll
      for (int p = 0; p < kMaxPhases; ++p) {
        const R2* qp = q + (ptrdiff_t)sl[p].x * kCells + cp[p];
        t0[p] = sl[p].y ? qp[0] : R2{};
        t1[p] = sl[p].y ? qp[32] : R2{};
      }
#pragma unroll
      for (int p = 0; p < kMaxPhases; ++p) {
        if (sl[p].y == 0) continue;
        v0.x += t0[p].x;
        v0.y += t0[p].y;
        v1.x += t1[p].x;
        v1.y += t1[p].y;
      }
    } else {
#pragma unroll
      for (int p = 0; p < kMaxPhases; ++p) {
        const R2* qp = q + (ptrdiff_t)sl[p].x * kCells + cp[p];
        if (sl[p].y == 1) {
          const R2 t0 = qp[0], t1 = qp[32];
          v0.x += t0.x;
          v0.y += t0.y;
          v1.x += t1.x;
          v1.y += t1.y;
        } else if (sl[p].y > 1) {
          add_chunks(v0, qp, sl[p].y);
          add_chunks(v1, qp + 32, sl[p].y);
        }
      }
    }
    dst[off0] = v0;
    if (both) dst[off1] = v1;
  }
}

// tile_start[t] = the first record of virtual tile t or a later one, by
// binary search: the records may leave any number of tiles empty, and a
// thread per record that writes the bounds of the tiles it passes writes
// tens of thousands of them where they do (0.22 ms of a 24 ms call with four
// plane groups).
__global__ void k_tile_bounds(const uint32_t* __restrict__ keys, uint32_t n,
                              int shift, int num_tiles,
                              uint32_t* __restrict__ tile_start) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t > num_tiles) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if ((keys[mid] >> shift) < (uint32_t)t) lo = mid + 1;
    else hi = mid;
  }
  tile_start[t] = lo;
}

// Per tile row of a single grid, the strips (tile_u / tile_phases columns)
// that virtual tiles with records cover: [lo, hi).
__global__ void k_touched_spans(const uint32_t* __restrict__ tile_start,
                                int num_tiles, int tiles_total, int tiles_u,
                                int phases, int strips_u,
                                uint32_t* __restrict__ lo,
                                uint32_t* __restrict__ hi) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < num_tiles;
       t += gridDim.x * blockDim.x) {
    if (tile_start[t + 1] == tile_start[t]) continue;
    const int r = t % tiles_total;
    const int p = (t / tiles_total) % phases;
    const int a = max((r % tiles_u) * phases - p, 0);
    const int b = min((r % tiles_u) * phases - p + phases, strips_u);
    if (a >= b) continue;
    atomicMin(&lo[r / tiles_u], (uint32_t)a);
    atomicMax(&hi[r / tiles_u], (uint32_t)b);
  }
}

// out[tv * strips_u + sc] = first | last << 16: the first and last virtual
// group whose tiles hold records in strip sc (tile_u / tile_phases columns)
// of tile row tv (0xFFFF | 0xFFFF << 16 when none), for a single grid.  In
// phase p the strip lies in tile column (sc + p) / tile_phases.
// *cells += the grid cells of the strips that have records (clipped to the
// grid), the cells a direct-mode call reads and writes at host.
__global__ void k_tile_groups(const uint32_t* __restrict__ tile_start,
                              TileGeom geom, int G, uint32_t* __restrict__ out,
                              unsigned long long* cells) {
  const int P = geom.tile_phases > 1 ? geom.tile_phases : 1;
  const int sw = 1 << geom.strip_shift;
  const int strips_u = geom.strips_u;
  const int n = strips_u * geom.tiles_v;
  unsigned long long mine = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * blockDim.x) {
    const int tv = i / strips_u, sc = i % strips_u;
    uint32_t first = 0xFFFFu, last = 0xFFFFu;
    for (int g = 0; g < geom.num_groups; ++g) {
      const int tc = (sc + g % P) / P;
      const size_t v =
          (size_t)g * geom.tiles_total + (size_t)tv * geom.tiles_u + tc;
      if (tile_start[v + 1] > tile_start[v]) {
        if (first == 0xFFFFu) first = (uint32_t)g;
        last = (uint32_t)g;
      }
    }
    out[i] = first | (last << 16);
    if (first != 0xFFFFu) {
      const int u0 = sc * sw, v0 = tv * geom.tile_v;
      mine += (unsigned long long)min(sw, G - u0) * min(geom.tile_v, G - v0);
    }
  }
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(cells, mine);
}

// The failure-report probe's wait: no other kernel waits on a barrier.
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(count)
               : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Acquire-wait for the completion of the phase with the given parity;
// false when `limit` probes have failed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          unsigned limit) {
  for (unsigned i = 0; i < limit; ++i) {
    if (mbar_test(bar, parity)) return true;
    if (i >= 32) __nanosleep(64);
  }
  return false;
}
// Failure-report probe: every thread waits, bounded by `limit` probes, on an
// mbarrier that nothing arrives at, so the wait runs out, the kernel sets the
// error flag and returns.
__global__ void k_wait_probe(unsigned limit, uint32_t* __restrict__ error) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  const bool ok = mbar_wait(&bar, 0, limit);
  if (!ok && threadIdx.x == 0) atomicExch(error, 1u);
}

// Virtual tile at queue rank i (see ItemBuffers::tile_order).
__device__ __forceinline__ int tile_at_rank(int i, int T,
                                            const int* __restrict__ order) {
  if (!order) return i;
  const int g = i / T;
  return g * T + order[i - g * T];
}

// Counts per queue rank i (tile t = tile_at_rank(i)):
// A[i] = chunks of t if it writes partial tiles (more than one chunk, or
// any chunk of a later tile phase), else 0;
// B[i] = 1 if t owns its tile in one chunk.
__global__ void k_item_counts(const uint32_t* __restrict__ tile_start,
                              int num_tiles, int num_groups,
                              const int* __restrict__ order, uint32_t chunk,
                              int partial_phases,
                              uint32_t* __restrict__ A,
                              uint32_t* __restrict__ B,
                              uint32_t* __restrict__ num_split) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *num_split = 0;   // k_item_emit counts from here
  if (i >= num_tiles) return;
  const int T = num_tiles / num_groups;
  const int t = tile_at_rank(i, T, order);
  const uint32_t c = tile_start[t + 1] - tile_start[t];
  const uint32_t chunks = num_chunks(c, chunk);
  // Later tile phases always write partial tiles (see ItemBuffers).
  const bool split = chunks > 1 || (chunks == 1 && (i / T) % partial_phases);
  A[i] = split ? chunks : 0;
  B[i] = split ? 0 : chunks;
}

// The queue is group-major (see ItemBuffers); within virtual group g the
// chunks of split tiles (every tile of a later tile phase counts as split)
// come first (they are the largest items), then the single-chunk tiles,
// each part in rank order.  With exclusive scans sA
// (split chunks) and sB (single-chunk tiles) over the ranks, group g
// starts at sA[gT] + sB[gT] (T = tiles per group), split chunk j of rank i
// sits at sA[i] + sB[gT] + j and single rank i at sA[(g+1)T] + sB[i].
// Partial slot of a split chunk = sA[i] + j.
__global__ void k_item_emit(const uint32_t* __restrict__ tile_start,
                            int num_tiles, int num_groups,
                            const int* __restrict__ order, uint32_t chunk,
                            int partial_phases,
                            const uint32_t* __restrict__ sA,
                            const uint32_t* __restrict__ sB,
                            const uint32_t* __restrict__ totA,
                            const uint32_t* __restrict__ totB,
                            WorkItem* __restrict__ items,
                            int4* __restrict__ split_tiles,
                            uint32_t* __restrict__ num_split,
                            uint32_t* __restrict__ num_items,
                            uint32_t* __restrict__ group_items,
                            int2* __restrict__ tile_slot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int T = num_tiles / num_groups;
  auto scanA = [&](int r) { return r < num_tiles ? sA[r] : *totA; };
  auto scanB = [&](int r) { return r < num_tiles ? sB[r] : *totB; };
  if (i == 0) *num_items = *totA + *totB;
  if (i <= num_groups) group_items[i] = scanA(i * T) + scanB(i * T);
  if (i >= num_tiles) return;
  const int g = i / T;
  const int t = tile_at_rank(i, T, order);
  const uint32_t s0 = tile_start[t], s1 = tile_start[t + 1];
  const uint32_t c = s1 - s0;
  const uint32_t chunks = num_chunks(c, chunk);
  const bool owns = chunks == 1 && g % partial_phases == 0;
  if (tile_slot)
    tile_slot[t] = c == 0 || owns ? make_int2(0, 0)
                                  : make_int2((int)sA[i], (int)chunks);
  if (c == 0) return;
  if (owns) {
    items[scanA((g + 1) * T) + sB[i]] = chunk_item(t, s0, s1, chunk, 0, -1);
  } else {
    const uint32_t first = sA[i];
    const uint32_t pos = first + scanB(g * T);
    for (uint32_t j = 0; j < chunks; ++j)
      items[pos + j] = chunk_item(t, s0, s1, chunk, j, (int)(first + j));
    const uint32_t k = atomicAdd(num_split, 1u);
    split_tiles[k] = make_int4(t, (int)first, (int)chunks, 0);
  }
}

// The kernels take 24 to 48 KB of dynamic shared memory: set before querying
// occupancy or launching, once per device, so later launches (replays captured
// in a CUDA graph among them) make no attribute call.
template <typename Real, int TW, bool kWide, bool kPrepared>
cudaError_t prepare_grid_kernel(void** fn, size_t* smem) {
  static std::atomic<unsigned long long> opted_in{0};
  if constexpr (sizeof(Real) == 4) {
    *fn = (void*)k_grid_tiles<TW, kWide, kPrepared>;
    *smem = kGridWarps * sizeof(WarpSmem<TW>);
  } else {
    *fn = (void*)k_grid_tiles_f64<TW, kPrepared>;
    *smem = kGridWarps * sizeof(WarpSmem64);
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev < 64 && (opted_in.load() & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(*fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)*smem);
  if (e == cudaSuccess && dev < 64) opted_in.fetch_or(bit);
  return e;
}

template <typename Real, bool kWide, bool kPrepared>
cudaError_t prepare_grid_kernel_of(int tile_u, void** fn, size_t* smem) {
  return tile_u == 32
             ? prepare_grid_kernel<Real, 32, kWide, kPrepared>(fn, smem)
         : tile_u == 16
             ? prepare_grid_kernel<Real, 16, kWide, kPrepared>(fn, smem)
             : prepare_grid_kernel<Real, 8, kWide, kPrepared>(fn, smem);
}

// Unprepared records: the wide kernel, which takes every call.
template <typename Real>
cudaError_t prepare_grid_kernel_for(int tile_u, bool wide, bool prepared,
                                    void** fn, size_t* smem) {
  constexpr bool kF32 = sizeof(Real) == 4;
  if (!prepared)
    return prepare_grid_kernel_of<Real, kF32, false>(tile_u, fn, smem);
  return wide ? prepare_grid_kernel_of<Real, kF32, true>(tile_u, fn, smem)
              : prepare_grid_kernel_of<Real, false, true>(tile_u, fn, smem);
}

}  // namespace

cudaError_t launch_tile_bounds(const uint32_t* keys, uint32_t n, int shift,
                               int num_tiles, uint32_t* tile_start,
                               cudaStream_t s) {
  // A tile per thread, and one more for the end.
  const int blocks = num_tiles / 256 + 1;
  k_tile_bounds<<<blocks, 256, 0, s>>>(keys, n, shift, num_tiles, tile_start);
  return cudaGetLastError();
}

cudaError_t launch_grid_odd(const void* placed, unsigned long long n,
                            const uint32_t* shape, StackView view, int grid_size,
                            float* grid, long long grid_stride,
                            const unsigned long long* grid_offsets,
                            int num_grids, cudaStream_t s, float* host) {
  const size_t cells = (size_t)grid_size * grid_size;
  if (host) {
    const cudaError_t e =
        cudaMemsetAsync(grid, 0, cells * sizeof(float2), s);
    if (e != cudaSuccess) return e;
  }
  const unsigned long long blocks = std::min<unsigned long long>(
      (n + 255) / 256, 1216);
  if (blocks == 0) return cudaSuccess;
  k_grid_odd<<<(unsigned)blocks, 256, 0, s>>>(
      (const Placed<float>*)placed, n, shape, view, grid_size, grid, grid_stride,
      grid_offsets, num_grids);
  if (host) {
    const unsigned long long pairs = (cells + 1) / 2;
    k_add_odd<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>(
        (const float4*)grid, pairs, cells, (float2*)host);
  }
  return cudaGetLastError();
}

cudaError_t launch_wait_probe(unsigned limit, uint32_t* error,
                              cudaStream_t s) {
  k_wait_probe<<<1, 64, 0, s>>>(limit, error);
  return cudaGetLastError();
}

cudaError_t launch_tile_groups(const uint32_t* tile_start,
                               const TileGeom& geom, int grid_size,
                               uint32_t* out, unsigned long long* cells,
                               cudaStream_t s) {
  const int n = num_strips(geom);
  const int blocks = std::min(1024, (n + 255) / 256);
  k_tile_groups<<<blocks < 1 ? 1 : blocks, 256, 0, s>>>(tile_start, geom,
                                                        grid_size, out, cells);
  return cudaGetLastError();
}

cudaError_t launch_touched_spans(const uint32_t* tile_start, int num_tiles,
                                 const TileGeom& geom, int grid_size,
                                 uint32_t* lo, uint32_t* hi, cudaStream_t s) {
  (void)grid_size;
  const int P = geom.tile_phases > 1 ? geom.tile_phases : 1;
  const int blocks = std::max(1, std::min((num_tiles + 255) / 256, 4096));
  k_touched_spans<<<blocks, 256, 0, s>>>(tile_start, num_tiles,
                                         geom.tiles_total, geom.tiles_u, P,
                                         geom.strips_u, lo, hi);
  return cudaGetLastError();
}

cudaError_t launch_build_items(const uint32_t* tile_start, int num_tiles,
                               uint32_t chunk, ItemBuffers b,
                               cudaStream_t s) {
  uint32_t* A = b.chunks;
  uint32_t* B = b.split_chunks;
  const int blocks = (num_tiles + 256) / 256;   // one more thread: bounds
  const int pp = b.partial_phases > 1 ? b.partial_phases : 1;
  k_item_counts<<<blocks, 256, 0, s>>>(tile_start, num_tiles, b.num_groups,
                                       b.tile_order, chunk, pp, A, B,
                                       b.num_split);
  // The work counter doubles as scratch for B's total until k_item_emit.
  cudaError_t e = exclusive_scan_pair_u32(A, B, num_tiles, b.num_slots,
                                          b.counter, b.scan_tmp, s);
  if (e != cudaSuccess) return e;
  k_item_emit<<<blocks, 256, 0, s>>>(tile_start, num_tiles, b.num_groups,
                                     b.tile_order, chunk, pp, A, B,
                                     b.num_slots,
                                     b.counter,
                                     b.items, b.split_tiles, b.num_split,
                                     b.num_items, b.group_items,
                                     b.tile_slot);
  return cudaGetLastError();
}

template <typename Real>
int grid_tiles_ctas_per_sm(int tile_u, bool wide) {
  void* fn = nullptr;
  size_t smem = 0;
  int n = 0;
  if (prepare_grid_kernel_for<Real>(tile_u, wide, true, &fn, &smem) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kGridThreads,
                                                    smem) != cudaSuccess)
    n = 1;
  return n < 1 ? 1 : n;
}

int grid_teams(int num_ctas) {
  return std::max(1, num_ctas / kBlocksPerTeam);
}

template <typename Real>
size_t prepared_record_bytes() {
  return sizeof(Record<Real>);
}
template size_t prepared_record_bytes<float>();
template size_t prepared_record_bytes<double>();

template <typename Real>
cudaError_t launch_reduce_phases(const int2* tile_slot, const Real* partials,
                                 TileGeom geom, int group0, int grid_size,
                                 Real* grid, long long grid_stride,
                                 Real* host, const uint32_t* tile_groups,
                                 const uint32_t* tile_start, cudaStream_t s) {
  const long long n =
      (long long)geom.num_grids * (geom.tiles_u - 1) * geom.tiles_v * kWarps /
      2;
  if (n <= 0) return cudaSuccess;
  if (geom.tile_phases > 8) return cudaErrorInvalidValue;
  const int blocks = (int)std::min<long long>(n, 65535);
  using P2 = const typename Vec2<Real>::type*;
  const bool eight = geom.tile_phases > 4;
#define GG_REDUCE_PHASES(TW_, MP_)                                          \
  k_reduce_phases<Real, TW_, MP_><<<blocks, 256, 0, s>>>(                   \
      tile_slot, (P2)partials, geom, group0, grid_size, grid, grid_stride, \
      host, tile_groups, tile_start)
  switch (geom.tile_u) {
    case 32:
      if (eight) GG_REDUCE_PHASES(32, 8); else GG_REDUCE_PHASES(32, 4);
      break;
    case 16:
      if (eight) GG_REDUCE_PHASES(16, 8); else GG_REDUCE_PHASES(16, 4);
      break;
    case 8:
      if (eight) GG_REDUCE_PHASES(8, 8); else GG_REDUCE_PHASES(8, 4);
      break;
    default: return cudaErrorInvalidValue;
  }
#undef GG_REDUCE_PHASES
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_reduce_group(const int4* split_tiles,
                                const uint32_t* num_split, int max_split,
                                const Real* partials, TileGeom geom, int group,
                                int grid_size, Real* grid,
                                long long grid_stride, Real* host,
                                const uint32_t* tile_groups, cudaStream_t s) {
  if (max_split <= 0) return cudaSuccess;
  const int blocks = (int)std::min(8LL * max_split, 2432LL);
  using P2 = const typename Vec2<Real>::type*;
  switch (geom.tile_u) {
    case 32: k_reduce_partials<Real, 32><<<blocks, 256, 0, s>>>(
        split_tiles, num_split, (P2)partials, geom, group, grid_size, grid,
        grid_stride, host, tile_groups); break;
    case 16: k_reduce_partials<Real, 16><<<blocks, 256, 0, s>>>(
        split_tiles, num_split, (P2)partials, geom, group, grid_size, grid,
        grid_stride, host, tile_groups); break;
    case 8: k_reduce_partials<Real, 8><<<blocks, 256, 0, s>>>(
        split_tiles, num_split, (P2)partials, geom, group, grid_size, grid,
        grid_stride, host, tile_groups); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_grid_tiles(const WorkItem* items,
                              const uint32_t* group_items,
                              uint32_t* counter, void* recs,
                              unsigned short* spans, const uint32_t* rec_vis,
                              const void* placed, StackView view,
                              TileGeom geom, int grid_size, Real* grid,
                              long long grid_stride,
                              Real* partials, const int4* split_tiles,
                              const uint32_t* num_split, int max_split,
                              int num_ctas, cudaStream_t s,
                              const cudaEvent_t* wait_before,
                              const cudaEvent_t* record_after,
                              Real* host_grid, const uint32_t* tile_groups,
                              int group_span, const int2* tile_slot,
                              const uint32_t* tile_start) {
  GridArgs<Real> a;
  a.items = items;
  a.group_items = group_items;
  a.group = 0;
  a.counter = counter;
  a.recs = (Record<Real>*)recs;
  a.spans = spans;
  a.rec_vis = rec_vis;
  a.placed = (const Placed<Real>*)placed;
  a.view = view;
  a.geom = geom;
  a.grid_size = grid_size;
  a.grid = grid;
  a.grid_stride = grid_stride;
  a.partials = (typename Vec2<Real>::type*)partials;
  a.host = tile_groups ? host_grid : grid;
  a.tile_groups = tile_groups;
  if (geom.tile_u != 32 && geom.tile_u != 16 && geom.tile_u != 8)
    return cudaErrorInvalidValue;
  void* fn = nullptr;
  size_t smem = 0;
  cudaError_t e = prepare_grid_kernel_for<Real>(
      geom.tile_u, view.wide, recs != nullptr, &fn, &smem);
  if (e != cudaSuccess) return e;
  const int span = group_span > 1 ? group_span : 1;
  a.group_span = span;
  int num_groups = geom.num_groups;
  void* prep_args[] = {&a, &num_groups};
  if (recs) {
    e = cudaLaunchKernel(geom.tile_u == 32 ? (void*)k_prepare_records<Real, 32>
                         : geom.tile_u == 16
                             ? (void*)k_prepare_records<Real, 16>
                             : (void*)k_prepare_records<Real, 8>,
                         dim3(8 * num_ctas), dim3(128), prep_args, 0, s);
    if (e != cudaSuccess) return e;
  }
  void* args[] = {&a};
  for (int g = 0; g < geom.num_groups; g += span) {
    a.group = g;
    if (wait_before && wait_before[g]) {
      e = cudaStreamWaitEvent(s, wait_before[g], 0);
      if (e != cudaSuccess) return e;
    }
    if (g > 0 || !recs) {
      e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
      if (e != cudaSuccess) return e;
    }
    e = cudaLaunchKernel(fn, dim3(num_ctas), dim3(kGridThreads), args, smem, s);
    if (e != cudaSuccess) return e;
    if (span > 1 && tile_slot) {
      e = launch_reduce_phases<Real>(tile_slot, partials, geom, g, grid_size,
                                     grid, grid_stride, a.host, tile_groups,
                                     tile_start, s);
      if (e != cudaSuccess) return e;
    } else {
      for (int p = 0; p < span; ++p) {
        e = launch_reduce_group<Real>(split_tiles, num_split, max_split,
                                      partials, geom, g + p, grid_size, grid,
                                      grid_stride, a.host, tile_groups, s);
        if (e != cudaSuccess) return e;
      }
    }
    if (record_after && record_after[g + span - 1]) {
      e = cudaEventRecord(record_after[g + span - 1], s);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

template int grid_tiles_ctas_per_sm<float>(int, bool);
template int grid_tiles_ctas_per_sm<double>(int, bool);
template cudaError_t launch_grid_tiles<float>(
    const WorkItem*, const uint32_t*, uint32_t*, void*, unsigned short*,
    const uint32_t*, const void*, StackView, TileGeom, int,
    float*, long long, float*, const int4*, const uint32_t*, int, int,
    cudaStream_t, const cudaEvent_t*, const cudaEvent_t*, float*,
    const uint32_t*, int, const int2*, const uint32_t*);
template cudaError_t launch_grid_tiles<double>(
    const WorkItem*, const uint32_t*, uint32_t*, void*, unsigned short*,
    const uint32_t*, const void*, StackView, TileGeom, int,
    double*, long long, double*, const int4*, const uint32_t*, int, int,
    cudaStream_t, const cudaEvent_t*, const cudaEvent_t*, double*,
    const uint32_t*, int, const int2*, const uint32_t*);

}  // namespace gg
