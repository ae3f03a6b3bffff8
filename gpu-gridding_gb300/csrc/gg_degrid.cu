// Adjoint of the gridding map (degridding): grid -> visibilities.
//
// Forward gridding adds v_i * c~_i(cell) to every cell of visibility i's
// footprint (oskar_grid_wproj.c:190-209), with c~ the kernel tap whose
// imaginary part is negated for ww > 0.  Its exact adjoint is the gather
//   out_i = sum over the footprint of conj(c~_i(cell)) * grid(cell).
//
// It runs on the gridder's records: after placement, emission and the sort,
// each 32 x 64-cell tile's (visibility, tile) records are contiguous, tiles in
// queue order.  Every warp works by itself: it takes a unit of up to 128
// consecutive records, prepares them in its shared memory, and goes through
// the tile's eight bands with the band's grid values in registers (lane =
// column, kRows rows per lane, as in the gridder): for each record that meets
// the band it multiplies them by the record's taps, sums over the warp and
// adds that to the record's sum.  Each record's sum goes to its emission slot
// (rec_offset[visibility] + its tile's rank among the visibility's tiles);
// k_degrid_finish then adds each visibility's partial results in emission
// order.  Nothing is accumulated with atomics, and a record's sums are formed
// alike whatever unit it is in, so the result does not depend on scheduling.
// With tile phases (see gg_grid.cu) a visibility's records are on its phase's
// tiles; the degridder only reads the grid, so the tiles of all phases share
// its one launch.
//
// What bounds it: the instructions issued, some 100 a record and band (issue
// slots 65 % in use, the L1 data pipe 52 %), of which the sum over the warp
// is a dozen.  In FP64 the FP64 pipe (16 cycles of the SM for a warp's FMA).
// Calls in ms, with a block of eight band warps and a producer sharing a
// stream of records -> warps of their own: 2e5 points on 2048^2 0.513 ->
// 0.467; 7.8e6 track points on 8192^2 (support 4 to 72) 7.9 -> 6.8; the
// former in FP64 5.4 -> 2.8 (the multiply-adds alone 1.7); and with a tile's
// records in visibility order 0.449 and 6.4.
//
// The reference has no degridder; this one is pinned by the dot-product
// identity <G x, y> = <x, G^H y> against the forward kernel and by the FP64
// oracle.
#include <algorithm>
#include <atomic>

#include "gg_internal.h"
#include "gg_tiles.cuh"

namespace gg {

namespace {

constexpr int kDegridTileU = 32;
using DegridShape = WarpShape<kDegridTileU>;
constexpr int kDegridWarps = 4;    // per block
constexpr int kDegridThreads = kDegridWarps * 32;
static_assert(kDegridWarps * kBlocksPerTeam == kWarps, "a team");
constexpr int kUnit = 128;         // records of a unit, at most
constexpr int kPerLane = kUnit / 32;
// A unit with fewer records a tile than this takes its records' grid values
// one by one: tile by tile, each band would wait out a memory latency for a
// record or two.  2e5 points on 2048^2: 0.485 ms so, 0.53 tile by tile; 3, 6
// and 12 records a tile as the line measure the same within 1 %.
constexpr int kSparse = 6;
constexpr uint32_t kConj = 1u << 31;

// The records are cut into units of 128, then (from record `begin64` on) of
// 64, then (from `begin32` on) of 32, two of 32 and four of 64 a warp: a
// launch ends with units that are short for the warps that still have one
// (2e5 points on 2048^2, 6.6e5 records: 0.47 ms, half as many
// short units 0.475 to 0.48, none of 32 0.50; 1.5e7 records: no difference).
struct DegridUnits {
  uint32_t total;              // records
  uint32_t begin64, begin32;   // multiples of 128
};
__device__ __forceinline__ uint2 degrid_unit(const DegridUnits& c,
                                             uint32_t unit) {
  const uint32_t n128 = c.begin64 / 128, n64 = (c.begin32 - c.begin64) / 64;
  uint32_t b, n;
  if (unit < n128) {
    b = unit * 128; n = 128;
  } else if (unit - n128 < n64) {
    b = c.begin64 + (unit - n128) * 64; n = 64;
  } else {
    b = c.begin32 + (unit - n128 - n64) * 32; n = 32;
  }
  return make_uint2(b, min(b + n, c.total));
}

template <typename Real>
struct DegridArgs {
  DegridUnits cut;
  uint32_t num_units;
  uint32_t* counter;
  const uint32_t* rec_key;    // sorted records: keys (tile << low_bits | ...)
  const uint32_t* rec_vis;    // and visibility indices
  int low_bits;
  const int* tile_order;      // tile at each place of the queue order
  const void* points;         // per visibility: cell, meta, emission slot; or,
  const uint32_t* rec_offset; // where given, the slots, points cell and meta
  StackView view;
  TileGeom geom;
  int grid_size;
  const Real* grid;
  typename Vec2<Real>::type* rec_out;  // partial result per emission slot
  // A grid in the caller's host memory, or null: read in place where
  // stays_at_host, else `grid` holds the cells that the tiles cover.
  const Real* host;
  const uint32_t* marked;     // strips of the tiles with records
};

// Whether a grid in host memory is read there unit by unit.  Every unit reads its
// tiles' values anew, over the link in that case, but those of its records'
// bands alone and beside its work, so calls of less than nine records a tile of
// cells to be brought over do (tile_phases strips; tiles of several phases share
// theirs).  Host calls in ms, so and with the tiles brought over first; on
// 8192^2, support 2 to 8: 2e4 points (4.4 records) 0.65 and 0.81, 5e4 (7.9) 1.04
// and 1.03, 4e5 2.97 and 1.76; 8 to 20: 5e3 (3.4) 0.52 and 0.68, 2e4 (7.9) 0.91
// and 1.03, 5e4 (15) 1.36 and 1.26; 20 to 36: 5e3 (4.9) 0.72 and 0.84, 2e4 (12)
// 1.28 and 1.22; 40 to 72: 2e3 (4.8) 0.78 and 0.87, 5e3 (8.8) 1.12 and 1.11, 2e4
// 1.87 and 1.57; on 2048^2, 2 to 8: 2e3 (5.7) 0.23 and 0.24, 2e4 (32) 0.38 and
// 0.33; 4 to 24: 2e5 1.51 and 0.75.
__device__ __forceinline__ bool stays_at_host(uint32_t marked, uint32_t total,
                                              int phases) {
  return 9ull * marked > (unsigned long long)total * (unsigned)phases;
}

// Marks the strips (TileGeom) of the tiles with records, a byte each, and counts
// them.  tile_start: by place in the queue order.
__global__ void k_mark_strips(const uint32_t* __restrict__ tile_start,
                              const int* __restrict__ tile_order, TileGeom g,
                              int num_tiles, uint32_t* __restrict__ marks,
                              uint32_t* __restrict__ marked) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t n = 0;
  if (t < num_tiles && tile_start[t + 1] > tile_start[t]) {
    const int vg = t / g.tiles_total, P = g.tile_phases;
    const int tl = tile_order[t - vg * g.tiles_total];
    const int tv = tl / g.tiles_u, tu = tl - tv * g.tiles_u;
    const int first = tu * P - (vg & (P - 1));
    for (int s = max(first, 0); s < min(first + P, g.strips_u); ++s) {
      const size_t at = (size_t)tv * g.strips_u + s;
      const uint32_t bit = 1u << (8 * (at & 3));
      n += (atomicOr(marks + at / 4, bit) & bit) == 0u;
    }
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(marked, n);
}

// Brings the marked strips' cells from the caller's host memory, grid row by
// grid row, each over the link once.  The link bounds it (16 blocks of 1024
// threads are too few, 48 to 300 the same); beside the binning, on a stream of
// its own, it got in the way of the cube's transfer (2e5 points on 2048^2 1.09
// ms a call instead of 0.76).
template <typename R2>
__global__ void __launch_bounds__(256)
k_gather_strips(const unsigned char* __restrict__ marks,
                const uint32_t* __restrict__ marked, uint32_t total,
                TileGeom g, int G, const R2* __restrict__ src,
                R2* __restrict__ dst) {
  constexpr int kAhead = 4;
  if (stays_at_host(*marked, total, g.tile_phases)) return;
  for (int row = blockIdx.x; row < G; row += gridDim.x) {
    const unsigned char* mark = marks + (size_t)(row / g.tile_v) * g.strips_u;
    const size_t at = (size_t)row * G;
    for (int c0 = threadIdx.x; c0 < G; c0 += kAhead * blockDim.x) {
      R2 v[kAhead];
      bool on[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int c = c0 + k * (int)blockDim.x;
        on[k] = c < G && mark[c >> g.strip_shift];
        if (on[k]) v[k] = src[at + c];
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k)
        if (on[k]) dst[at + c0 + k * blockDim.x] = v[k];
    }
  }
}

// Shared memory of one warp.  A record's int4: the tap index of the footprint
// centre's column in the slice row of tile row 0; conjugated << 31 | columns
// mirrored << 30 | the centre's tile column (16 bits); support + 1; taps from
// one tile row to the next.  Record kUnit adds nothing.
template <typename Real>
struct DegridWarp {
  using R2 = typename Vec2<Real>::type;
  int4 rec[kUnit + 1];
  R2 sum[kUnit];
  uint32_t out[kUnit];          // emission slot
  int2 origin[kUnit + 1];       // grid column and row of the tile's first cell
  // FP32: the tile's place, the bands it meets (first | last << 8), and the
  // records that meet a band with fillers up to a multiple of four.
  uint32_t tile[kUnit];
  unsigned short span[kUnit];
  alignas(4) unsigned char queue[kUnit + 4];
  short row0[kUnit];            // FP64: the footprint's first tile row
};

// v[2 j + c] summed over the warp for c = 0, 1 of the four records j: the
// lane's result is that of j = lane >> 3, c = (lane >> 2) & 1.  Halving the
// values a lane holds at each of the first three steps takes 9 shuffles
// where a tree per value takes 40.
template <typename Real>
__device__ __forceinline__ Real warp_sum_4x2(const Real (&v)[8], int lane) {
  Real a[4], b[2];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool up = (lane & 16) != 0;
    a[j] = up ? v[j + 4] : v[j];
    a[j] += __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + 4], 16);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const bool up = (lane & 8) != 0;
    b[j] = up ? a[j + 2] : a[j];
    b[j] += __shfl_xor_sync(0xffffffffu, up ? a[j] : a[j + 2], 8);
  }
  const bool up = (lane & 4) != 0;
  Real r = up ? b[1] : b[0];
  r += __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

// This lane's share of conj(c~) * g over its kRows cells, with g = (re, im)
// and gs = (im, re): X = sum (t.re g.re, t.im g.im) and Y = sum (t.re g.im,
// t.im g.re), so with c~ = (t.re, sgn * t.im)
//   re = X.x + sgn * X.y,  im = Y.x - sgn * Y.y.
__device__ __forceinline__ void dot_record(const float2 (&t)[kRows],
                                           const float2 (&g)[kRows],
                                           const float2 (&gs)[kRows],
                                           int flags, float& re, float& im) {
  float2 X{}, Y{};
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    X = fma2(t[r], g[r], X);
    Y = fma2(t[r], gs[r], Y);
  }
  const float sgn = __int_as_float(((uint32_t)flags & kConj) | 0x3F800000u);
  re = fmaf(sgn, X.y, X.x);
  im = fmaf(-sgn, Y.y, Y.x);
}

// kHost: the grid may be read in the caller's memory.  In the kernel of every
// call this choice took degridding 5 to 8 % longer (2e5 points on 2048^2 0.449
// and 0.470 ms, 3.1e7 track points on 8192^2 6.17 and 6.65).
template <typename Real, bool kWide, bool kHost>
__global__ void __launch_bounds__(kDegridThreads, sizeof(Real) == 4 ? 4 : 3)
k_degrid_tiles(DegridArgs<Real> a) {
  using R2 = typename Vec2<Real>::type;
  using SM = DegridWarp<Real>;
  constexpr bool kPacked = sizeof(Real) == 8;
  extern __shared__ __align__(16) unsigned char g_smem_raw[];
  const int lane = threadIdx.x & 31;
  SM& sm = reinterpret_cast<SM*>(g_smem_raw)[threadIdx.x >> 5];
  const int G = a.grid_size;
  const R2* __restrict__ taps = (const R2*)a.view.taps;
  const R2* __restrict__ grid = (const R2*)a.grid;
  if constexpr (kHost)
    if (stays_at_host(*a.marked, a.cut.total, a.geom.tile_phases))
      grid = (const R2*)a.host;
  const uint32_t lt = (1u << lane) - 1u;
  if (lane == 0) {
    sm.rec[kUnit] = make_int4((int)kStackZero, 0, 0, 0);
    sm.origin[kUnit] = make_int2(0, 0);
  }
  unsigned next = 0;
  if (lane == 0) next = atomicAdd(a.counter, 1u);
  for (;;) {
    const unsigned unit = __shfl_sync(0xffffffffu, next, 0);
    if (unit >= a.num_units) return;
    if (lane == 0) next = atomicAdd(a.counter, 1u);   // used in the next turn
    const uint2 range = degrid_unit(a.cut, unit);
    const int nb = (int)(range.y - range.x);
    // Prepare the records.
    uint4 pt[kPerLane];
    uint32_t key[kPerLane];
#pragma unroll
    for (int q = 0; q < kPerLane; ++q) {
      const int t = q * 32 + lane;
      if (t < nb) {
        key[q] = a.rec_key[range.x + t];
        const uint32_t vid = a.rec_vis[range.x + t];
        if (a.rec_offset) {
          const uint2 c = ((const uint2*)a.points)[vid];
          pt[q] = make_uint4(c.x, c.y, a.rec_offset[vid], 0u);
        } else {
          pt[q] = ((const uint4*)a.points)[vid];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kPerLane; ++q) {
      const int t = q * 32 + lane;
      if (t < nb) {
        const uint32_t tile = key[q] >> a.low_bits;
        const int vg = (int)(tile / (uint32_t)a.geom.tiles_total);
        const int tl =
            a.tile_order[tile - (uint32_t)vg * (uint32_t)a.geom.tiles_total];
        const int tv = tl / a.geom.tiles_u, tu = tl - tv * a.geom.tiles_u;
        const int sh = phase_shift(a.geom, vg);
        const int u0 = tu * DegridShape::kTileU - sh;
        const int v0 = tv * DegridShape::kTileV;
        const uint32_t m = pt[q].y;
        const SlicePlane plane = a.view.planes[meta_plane(m)];
        const int s = plane.support;
        const int gu = cell_u(pt[q].x), gv = cell_v(pt[q].x);
        const int ou = meta_ou(m), ov = meta_ov(m);
        const uint2 d = slice_record(
            slice_origin(plane, a.view.omax, abs(ou), abs(ov)), s, ou, ov,
            gu - u0, gv - v0);
        sm.rec[t] = make_int4(
            (int)(d.x + (uint32_t)s),
            (int)(((uint32_t)(gu - u0) & 0xFFFFu) | (d.y & kMirrorU) |
                  (meta_conj(m) ? kConj : 0u)),
            s + 1, slice_step(d));
        sm.origin[t] = make_int2(u0, v0);
        const int top = gv - s - v0;
        if constexpr (kPacked) {
          sm.row0[t] = (short)top;
        } else {
          sm.tile[t] = tile;
          sm.span[t] = (unsigned short)(
              (uint32_t)(max(top, 0) / kRows) |
              (uint32_t)(min(top + 2 * s, DegridShape::kTileV - 1) / kRows)
                  << 8);
        }
        sm.sum[t] = R2{};
        // Rank of this tile among the visibility's tiles, in the order
        // k_emit writes them (tile rows outer, tile columns inner, on the
        // visibility's tile phase).
        const int tu0 = (gu - s + sh) / DegridShape::kTileU;
        const int tu1 = (gu + s + sh) / DegridShape::kTileU;
        const int tv0 = (gv - s) / DegridShape::kTileV;
        sm.out[t] = pt[q].z +
                    (uint32_t)((tv - tv0) * (tu1 - tu0 + 1) + (tu - tu0));
      }
    }
    __syncwarp();
    // Adds the warp sums of the four records named by the bytes of w.
    auto store = [&](uint32_t w, const Real (&v)[8]) {
      const Real r = warp_sum_4x2(v, lane);
      const uint32_t t = w >> (lane >> 3 << 3) & 0xFFu;
      if ((lane & 3) == 0 && t < kUnit)
        ((Real*)sm.sum)[2 * t + ((lane >> 2) & 1)] += r;
    };
    if constexpr (kPacked) {
      // As in the FP64 gridder the lanes take a record's cells packed row by
      // row; the grid values come straight from the grid.
      constexpr int kAhead = 8;   // cells of a lane in flight
      for (int t0 = 0; t0 < nb; t0 += 4) {
        uint32_t word = 0;
        Real v[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = min(t0 + j, kUnit);
          word |= (uint32_t)(t < nb ? t : kUnit) << (8 * j);
          // As dot_record's sums, eight cells of a lane at a time: one chain
          // of additions over all of a lane's cells left up to half as much
          // error again (supports of 30 to 60), and took longer: 2e5 points
          // of support 4 to 24 on 2048^2 2.82 ms, so 2.77; 6e4 of 10 to 60
          // 4.73 and 4.24.
          R2 X{}, Y{};
          bool conj = false;
          if (t < nb) {
            const int4 e = sm.rec[t];
            const int gu = (int)(short)e.y, s = e.z - 1;
            const int su = e.y & kMirrorU ? -1 : 1;
            conj = e.y < 0;
            const int c0 = max(gu - s, 0);
            const int w = min(gu + s, kDegridTileU - 1) - c0 + 1;
            const int top = sm.row0[t];
            const int r0 = max(top, 0);
            const int n =
                w * (min(top + 2 * s, DegridShape::kTileV - 1) - r0 + 1);
            const float inv_w = 1.0f / (float)w;
            const uint32_t x = (uint32_t)(e.x + r0 * e.w + su * (c0 - gu));
            const int2 o = sm.origin[t];
            const R2* const cells = grid + (size_t)(o.y + r0) * G + o.x + c0;
            auto add = [&](int k, R2& PX, R2& PY) {
              R2 tap[kAhead], cell[kAhead];
#pragma unroll
              for (int h = 0; h < kAhead; ++h) {
                const int l = k + 32 * h;
                const int row = (int)(((float)l + 0.5f) * inv_w);
                const int c = l - row * w;
                tap[h] = cell[h] = R2{};
                if (l < n) {
                  tap[h] =
                      ld_tap(taps + (x + (uint32_t)(row * e.w + su * c)));
                  cell[h] = cells[(size_t)row * G + c];
                }
              }
#pragma unroll
              for (int h = 0; h < kAhead; ++h) {
                if (k + 32 * h >= n) break;
                PX.x = fma(tap[h].x, cell[h].x, PX.x);
                PX.y = fma(tap[h].y, cell[h].y, PX.y);
                PY.x = fma(tap[h].x, cell[h].y, PY.x);
                PY.y = fma(tap[h].y, cell[h].x, PY.y);
              }
            };
            if (lane < n) add(lane, X, Y);
            for (int k = lane + 32 * kAhead; k < n; k += 32 * kAhead) {
              R2 PX{}, PY{};
              add(k, PX, PY);
              X.x += PX.x;
              X.y += PX.y;
              Y.x += PY.x;
              Y.y += PY.y;
            }
          }
          v[2 * j] = X.x + (conj ? -X.y : X.y);
          v[2 * j + 1] = Y.x - (conj ? -Y.y : Y.y);
        }
        __syncwarp();
        store(word, v);
      }
    } else {
      R2 g[kRows], gs[kRows];   // grid values (re, im) and (im, re)
      int band = 0;
      auto load_grid = [&](int2 o) {
        const int row0 = o.y + band * kRows, col = o.x + lane;
        // Tiles of later phases start left of phase 0's (and may reach past
        // either edge of the grid).
        const bool col_in = (unsigned)col < (unsigned)G;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          g[r] = R2{};
          if (row0 + r < G && col_in) g[r] = grid[(size_t)(row0 + r) * G + col];
        }
      };
      auto swap_grid = [&]() {
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          gs[r].x = g[r].y;
          gs[r].y = g[r].x;
        }
      };
      auto load = [&](uint32_t t, R2 (&out)[kRows], int& y) {
        const int4 e = sm.rec[t & 0xFFu];
        const int c = min(max(lane - (int)(short)e.y, -e.z), e.z);
        y = e.y;
        load_taps<kWide>(
            taps,
            (uint32_t)(e.x + band * kRows * e.w + (e.y & kMirrorU ? -c : c)), e.w,
            out);
      };
      // Queues the records from `begin` on, of the same tile if `tile` is
      // set, that meet the band; returns how many, fillers included.
      auto enqueue = [&](int begin, bool same) {
        const uint32_t tile = sm.tile[begin];
        int count = 0;
        __syncwarp();
        for (int t = begin + lane; t - lane < nb; t += 32) {
          const uint32_t span = t < nb ? sm.span[t] : 0xFFu;
          const bool hit = (int)(span & 0xFFu) <= band &&
                           (int)(span >> 8) >= band &&
                           (!same || sm.tile[t] == tile);
          const uint32_t b = __ballot_sync(0xffffffffu, hit);
          if (hit) sm.queue[count + __popc(b & lt)] = (unsigned char)t;
          count += __popc(b);
        }
        const int end = (count + 3) & ~3;
        if (count + lane < end) sm.queue[count + lane] = kUnit;
        __syncwarp();
        return end;
      };
      const uint32_t* const queue = (const uint32_t*)sm.queue;
      int tiles = 0;
      for (int t = lane; t - lane < nb; t += 32)
        tiles += __popc(__ballot_sync(
            0xffffffffu,
            t < nb && (t == 0 || sm.tile[t] != sm.tile[t - 1])));
      if (tiles * kSparse > nb) {
        // Few records a tile: band by band over all of them, each with its
        // own grid values.
        for (band = 0; band < kWarps; ++band) {
          const int end = enqueue(0, false);
          for (int i = 0; i < end; i += 4) {
            const uint32_t w = queue[i / 4];
            Real v[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              R2 t[kRows];
              int y;
              load(w >> (8 * j), t, y);
              load_grid(sm.origin[w >> (8 * j) & 0xFFu]);
              swap_grid();
              dot_record(t, g, gs, y, v[2 * j], v[2 * j + 1]);
            }
            store(w, v);
          }
        }
      } else {
        for (int begin = 0; begin < nb;) {
          for (band = 0; band < kWarps; ++band) {
            const int end = enqueue(begin, true);
            if (end == 0) continue;
            R2 ta[kRows], tb[kRows];   // two records' taps in flight
            int ya = 0, yb = 0;
            uint32_t w = queue[0];
            load_grid(sm.origin[begin]);
            load(w, ta, ya);
            load(w >> 8, tb, yb);
            swap_grid();
            for (int i = 4;; i += 4) {
              const uint32_t wn = i < end ? queue[i / 4] : w;
              Real v[8];
              dot_record(ta, g, gs, ya, v[0], v[1]);
              load(w >> 16, ta, ya);
              dot_record(tb, g, gs, yb, v[2], v[3]);
              load(w >> 24, tb, yb);
              dot_record(ta, g, gs, ya, v[4], v[5]);
              if (i < end) load(wn, ta, ya);
              dot_record(tb, g, gs, yb, v[6], v[7]);
              if (i < end) load(wn >> 8, tb, yb);
              store(w, v);
              if (i >= end) break;
              w = wn;
            }
          }
          const uint32_t tile = sm.tile[begin];
          int same = 0;
          for (int t = begin + lane; t - lane < nb; t += 32)
            same += __popc(__ballot_sync(0xffffffffu,
                                         t < nb && sm.tile[t] == tile));
          begin += same;
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kPerLane; ++q) {
      const int t = q * 32 + lane;
      if (t < nb) a.rec_out[sm.out[t]] = sm.sum[t];
    }
    __syncwarp();
  }
}

// out[i] = sum of visibility i's partial results in emission order, in the
// call's precision (a visibility has a handful of records: its footprint's
// tiles); skipped visibilities have no records and get 0.
template <typename Real>
__global__ void k_degrid_finish(const uint32_t* __restrict__ count,
                                const uint32_t* __restrict__ offset,
                                const typename Vec2<Real>::type* __restrict__
                                    rec_out,
                                unsigned long long n, Real* __restrict__ out) {
  using R2 = typename Vec2<Real>::type;
  const unsigned long long i =
      (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t c = count[i], o = offset[i];
  R2 acc;
  acc.x = acc.y = 0;
  for (uint32_t k = 0; k < c; ++k) {
    const R2 v = rec_out[o + k];
    acc.x += v.x;
    acc.y += v.y;
  }
  ((R2*)out)[i] = acc;
}

template <typename Real, bool kWide, bool kHost>
cudaError_t prepare_degrid_kernel(void** fn, size_t* smem) {
  static std::atomic<unsigned long long> opted_in{0};
  *fn = (void*)k_degrid_tiles<Real, kWide, kHost>;
  *smem = kDegridWarps * sizeof(DegridWarp<Real>);
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

template <typename Real>
cudaError_t prepare_degrid_kernel_for(bool wide, bool host, void** fn,
                                      size_t* smem) {
  if (host)
    return wide ? prepare_degrid_kernel<Real, true, true>(fn, smem)
                : prepare_degrid_kernel<Real, false, true>(fn, smem);
  return wide ? prepare_degrid_kernel<Real, true, false>(fn, smem)
              : prepare_degrid_kernel<Real, false, false>(fn, smem);
}

}  // namespace

template <typename Real>
int degrid_tiles_ctas_per_sm(bool wide) {
  void* fn = nullptr;
  size_t smem = 0;
  int n = 0;
  if (prepare_degrid_kernel_for<Real>(wide, false, &fn, &smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kDegridThreads,
                                                    smem) !=
          cudaSuccess)
    n = 1;
  return n < 1 ? 1 : n;
}

template <typename Real>
cudaError_t launch_degrid_tiles(const uint32_t* rec_key,
                                const uint32_t* rec_vis, uint32_t total,
                                int low_bits, const int* tile_order,
                                PlacedPoints points,
                                const uint32_t* rec_offset, uint32_t* counter,
                                StackView view, TileGeom geom, int grid_size,
                                const Real* grid, const Real* host,
                                const uint32_t* marked, void* rec_out,
                                int num_ctas, cudaStream_t s) {
  if (geom.tile_u != kDegridTileU || geom.tile_v != DegridShape::kTileV)
    return cudaErrorInvalidValue;
  DegridArgs<Real> a;
  const uint32_t warps = (uint32_t)num_ctas * kDegridWarps;
  a.cut.total = total;
  a.cut.begin32 = (total - std::min(total, 64 * warps)) / 128 * 128;
  a.cut.begin64 =
      (a.cut.begin32 - std::min(a.cut.begin32, 256 * warps)) / 128 * 128;
  a.num_units = a.cut.begin64 / 128 + (a.cut.begin32 - a.cut.begin64) / 64 +
                (total - a.cut.begin32 + 31) / 32;
  a.counter = counter;
  a.rec_key = rec_key;
  a.rec_vis = rec_vis;
  a.low_bits = low_bits;
  a.tile_order = tile_order;
  a.points = points.p;
  a.rec_offset = points.stride == 16 ? nullptr : rec_offset;
  a.view = view;
  a.geom = geom;
  a.grid_size = grid_size;
  a.grid = grid;
  a.host = host;
  a.marked = marked;
  a.rec_out = (typename Vec2<Real>::type*)rec_out;
  void* fn = nullptr;
  size_t smem = 0;
  cudaError_t e = prepare_degrid_kernel_for<Real>(view.wide, host != nullptr,
                                                  &fn, &smem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchKernel(fn, dim3(num_ctas), dim3(kDegridThreads), args, smem,
                          s);
}

template <typename Real>
cudaError_t launch_gather_tiles(const uint32_t* tile_start,
                                const int* tile_order, TileGeom geom,
                                int num_tiles, uint32_t total,
                                uint32_t* marks, uint32_t* marked,
                                int grid_size, const Real* host, Real* grid,
                                int num_sms, cudaStream_t s) {
  using R2 = typename Vec2<Real>::type;
  cudaError_t e = cudaMemsetAsync(marked, 0, sizeof(uint32_t), s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(marks, 0, strip_mark_bytes(geom), s);
  if (e != cudaSuccess) return e;
  k_mark_strips<<<(num_tiles + 255) / 256, 256, 0, s>>>(
      tile_start, tile_order, geom, num_tiles, marks, marked);
  k_gather_strips<R2><<<std::min(grid_size, 8 * num_sms), 256, 0, s>>>(
      (const unsigned char*)marks, marked, total, geom, grid_size,
      (const R2*)host, (R2*)grid);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_degrid_finish(const uint32_t* count, const uint32_t* offset,
                                 const void* rec_out, unsigned long long n,
                                 Real* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned long long blocks = (n + 255) / 256;
  k_degrid_finish<Real><<<(unsigned)blocks, 256, 0, s>>>(
      count, offset, (const typename Vec2<Real>::type*)rec_out, n, out);
  return cudaGetLastError();
}

template int degrid_tiles_ctas_per_sm<float>(bool);
template int degrid_tiles_ctas_per_sm<double>(bool);
template cudaError_t launch_degrid_tiles<float>(
    const uint32_t*, const uint32_t*, uint32_t, int, const int*, PlacedPoints,
    const uint32_t*, uint32_t*, StackView, TileGeom, int, const float*,
    const float*, const uint32_t*, void*, int, cudaStream_t);
template cudaError_t launch_degrid_tiles<double>(
    const uint32_t*, const uint32_t*, uint32_t, int, const int*, PlacedPoints,
    const uint32_t*, uint32_t*, StackView, TileGeom, int, const double*,
    const double*, const uint32_t*, void*, int, cudaStream_t);
template cudaError_t launch_gather_tiles<float>(
    const uint32_t*, const int*, TileGeom, int, uint32_t, uint32_t*,
    uint32_t*, int, const float*, float*, int, cudaStream_t);
template cudaError_t launch_gather_tiles<double>(
    const uint32_t*, const int*, TileGeom, int, uint32_t, uint32_t*,
    uint32_t*, int, const double*, double*, int, cudaStream_t);
template cudaError_t launch_degrid_finish<float>(const uint32_t*,
                                                 const uint32_t*, const void*,
                                                 unsigned long long, float*,
                                                 cudaStream_t);
template cudaError_t launch_degrid_finish<double>(const uint32_t*,
                                                  const uint32_t*, const void*,
                                                  unsigned long long, double*,
                                                  cudaStream_t);

}  // namespace gg
