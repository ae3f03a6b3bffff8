// Shared definitions of the GB300 gridder's CUDA sources.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

namespace gg {

// ---------------------------------------------------------------------------
// Limits of this build.
// ---------------------------------------------------------------------------
// Cell coordinates are packed as two 16-bit fields, so grid_size <= 65535.
constexpr int kMaxGridSize = 65535;
// Oversampled offsets are stored biased by 8 in 4-bit fields: |off| <= 7,
// i.e. oversample <= 14 (|off| <= (oversample + 1) / 2).
constexpr int kMaxOversample = 14;
// W-plane index is a 16-bit field.
constexpr int kMaxPlanes = 65535;

// Packed placement of one visibility (written by the placement kernel).
//   cell: u in bits 0-15, v in bits 16-31
//   meta: plane in bits 0-15, (off_u + 8) in 16-19, (off_v + 8) in 20-23,
//         conj_neg in bit 24, skipped in bit 25, kMetaOdd in bit 26
__host__ __device__ inline uint32_t pack_cell(int u, int v) {
  return (uint32_t)(u & 0xFFFF) | ((uint32_t)(v & 0xFFFF) << 16);
}
__host__ __device__ inline int cell_u(uint32_t c) { return (int)(c & 0xFFFF); }
__host__ __device__ inline int cell_v(uint32_t c) { return (int)(c >> 16); }
__host__ __device__ inline uint32_t pack_meta(int plane, int ou, int ov,
                                              int conj_neg, int skipped) {
  return (uint32_t)plane | ((uint32_t)(ou + 8) << 16) |
         ((uint32_t)(ov + 8) << 20) | ((uint32_t)conj_neg << 24) |
         ((uint32_t)skipped << 25);
}
// A gridded FP32 point whose weighted visibility is infinite or not a number:
// added cell by cell (launch_grid_odd), as the tile kernel's lanes outside its
// footprint would make NaNs of their zero taps.
constexpr uint32_t kMetaOdd = 1u << 26;
__host__ __device__ inline int meta_plane(uint32_t m) { return (int)(m & 0xFFFF); }
__host__ __device__ inline int meta_ou(uint32_t m) { return (int)((m >> 16) & 0xF) - 8; }
__host__ __device__ inline int meta_ov(uint32_t m) { return (int)((m >> 20) & 0xF) - 8; }
__host__ __device__ inline int meta_conj(uint32_t m) { return (int)((m >> 24) & 1); }
__host__ __device__ inline int meta_skipped(uint32_t m) { return (int)((m >> 25) & 1); }

// Two-component vector of the call's precision (complex value, re/im).
template <typename Real>
struct Vec2;
template <>
struct Vec2<float> { using type = float2; };
template <>
struct Vec2<double> { using type = double2; };

// A placed visibility as the gridding kernel's records gather it: cell, meta
// and the weighted visibility together, so that the gather of a record, in
// tile order and so at random, is one sector of HBM and not three (3.1e7 track
// points, 5.9e7 records: 2.55 ms with three, 1.10 with one).
template <typename Real>
struct alignas(4 * sizeof(Real)) Placed {
  uint32_t cell, meta;
  typename Vec2<Real>::type v;
};

// The placed points of a call: cell and meta of point i at p + i * stride.
// Gridding's are Placed; degridding's pairs are 16 bytes apart, with room for
// the point's first emission slot behind them, or 8 where memory is short.
struct PlacedPoints {
  unsigned char* p;
  unsigned stride;
  __device__ __forceinline__ uint2 at(unsigned long long i) const {
    return *(const uint2*)(p + i * stride);
  }
};

// ---------------------------------------------------------------------------
// Re-laid kernel stack: one dense slice per (plane, |offset| class).
// ---------------------------------------------------------------------------
// The reference stores, per plane, the first quadrant K[t][c] of an
// oversampled kernel and reads the tap of footprint cell (j, k) at
// t = |off_v + j*os|, c = |off_u + k*os| (oskar_grid_wproj.c:196-203).  For
// a given offset those taps form a (2s+1)^2 matrix; the device copy stores
// that matrix explicitly, for every plane and every absolute offset class
// (cu, cv) in [0, omax]^2:
//   S[jj][kk] = K[|cv + (jj - s)*os|][|cu + (kk - s)*os|],  jj, kk in [0, 2s]
// A negative offset reads the mirrored slice: |-c + k*os| = |c + (-k)*os|,
// so the tap of (j, k) for offsets (ou, ov) is
//   S_{|ou|,|ov|}[s + sgn(ov)*j][s + sgn(ou)*k].
// A warp whose lanes hold consecutive k thus reads one contiguous run of a
// row, whatever the offset: two 128-byte wavefronts per 32 taps, where a row
// folded at off_u + k*os = 0 (two runs, each across line boundaries) took
// 2.7 to 3.0 (measured with the taps in L1).  Every row ends in one zero tap
// (row pitch 2s + 2), so a lane left or right of the footprint reads the zero
// tap beside the row's own taps -- the end of the row above, or of the row
// itself -- and kSlicePad zero rows lie above and below every slice (shared
// by neighbours), so a lane whose kRows consecutive cells straddle the
// footprint's top or bottom edge reads zeros there instead of testing each
// row.
constexpr int kSlicePad = 7;
// Zero taps before the first plane, and one of them from which kRows rows of
// the smallest pitch (2) and one column may be read either way: a record, or
// a lane, that adds nothing.
constexpr int kStackLead = 40;
constexpr int kStackZero = 20;

// One plane's slices, as the producers of the tile kernels look them up.
struct alignas(16) SlicePlane {
  long long origin;   // tap S[0][0] of the slice of class (0, 0)
  int stride;         // taps from one class's slice to the next
  int support;
};

// From here on FP32 gridding takes record positions as unsigned (wide view).
constexpr uint32_t kWideRecords = (1u << 31) - 64;

struct StackView {
  int num_planes;
  int oversample;
  int omax;                 // (oversample + 1) / 2: largest |offset|
  int conv_size_half;
  const int* support;       // [P]
  const SlicePlane* planes; // [P]
  const void* taps;         // float2 or double2
  bool wide;                // more than 4 GiB of taps (load_taps), or a call
                            // with kWideRecords records or more
  const double* tap_sum;    // [P][2*omax+1][2*omax+1] sum of Re(tap), FP64
};

// Row pitch of a slice: its 2s + 1 taps and a zero (even, so every row
// starts 16-byte aligned).
__host__ __device__ inline int slice_pitch(int s) { return 2 * s + 2; }
// Taps from one slice of a plane to the next: its rows and the pad rows.
__host__ __device__ inline long long slice_stride(int s) {
  return (long long)(2 * s + 1 + kSlicePad) * slice_pitch(s);
}
// Taps of a plane: pad rows, then the slices, each followed by pad rows.
__host__ __device__ inline long long plane_taps(int s, int omax) {
  return (long long)kSlicePad * slice_pitch(s) +
         (long long)(omax + 1) * (omax + 1) * slice_stride(s);
}
// Index of tap S[0][0] of the plane's slice for absolute offsets (cu, cv).
__host__ __device__ inline long long slice_origin(const SlicePlane& p,
                                                  int omax, int cu, int cv) {
  return p.origin + (long long)(cu * (omax + 1) + cv) * p.stride;
}

// Rows and columns of a plane's quadrant cube that the stack preparation may
// read (|off| + s*os with |off| <= omax, rounded up to whole oversampling
// steps): the square [0, E)^2.
__host__ __device__ inline int cube_read_extent(int s, int os, int omax,
                                                int csh) {
  const int a = s * os + omax + 1, b = (s + 1 + (omax >= os ? 1 : 0)) * os;
  const int e = a > b ? a : b;
  return e < csh ? e : csh;
}

// ---------------------------------------------------------------------------
// Call parameters.
// ---------------------------------------------------------------------------
template <typename Real>
struct PlaceParams {
  const Real* uu;
  const Real* vv;
  const Real* ww;
  const Real* vis;      // interleaved
  const Real* weight;
  Real grid_scale;      // grid_size * cell_size_rad, in the call's precision
  Real w_scale;
  int grid_size;
  int grid_centre;
  unsigned long long num_points;
  // Norm terms left to launch_norm_terms (the kernel stack's tap sums are
  // not ready yet when placement runs).
  bool defer_norm = false;
};

// Tile geometry shared by the binning and gridding kernels.
// With plane groups (num_groups > 1) the records of a call are gridded in
// one pass per group of consecutive w-planes, each group's kernel slices
// small enough to stay in L2 during its pass; the sort key's tile field is
// then the virtual tile group * tiles_total + tile.
struct TileGeom {
  int tile_u, tile_v;        // cells per tile
  int tiles_u, tiles_v;      // tiles per grid side
  int num_grids;
  int plane_bits;            // key bits of the plane, below the tile index
  int num_groups;            // plane groups (passes), >= 1
  int tiles_total;           // num_grids * tiles_u * tiles_v
  const int* plane_group;    // [P] group of each plane (num_groups > 1)
  // > 0: plane groups are gridded in two passes by tile rows (rows below
  // split_tv first) -- the first plane group when bit 0 of split_mask is
  // set, the last one when bit 1 is (single-grid calls).  Virtual groups:
  // [first upper, first lower,] middle groups..., [last upper, last lower];
  // num_groups counts them all.
  int split_tv;
  int split_mask;
  // Tile phases (1, 2, 4 or 8): the tile columns of phase p start p * tile_u /
  // tile_phases cells to the left of phase 0's, and each visibility is
  // gridded on the phase whose tiles cut its footprint into the fewest
  // columns (footprint_phase).  Tiles of different phases overlap, so each
  // phase is a pass of its own: virtual group = group * tile_phases +
  // phase.  With more than one phase tiles_u counts one more column (phase
  // p's first column starts left of the grid, its last may end past it).
  int tile_phases;
  // Strips of tile_u / tile_phases columns (a power of two, 1 << strip_shift)
  // by tile rows: the units in which a single-grid call records which
  // passes touch which cells (strips_u strips per tile row).
  int strip_shift;
  int strips_u;
};

// Columns of the tile grid of virtual group `group` left of phase 0's
// (tile_phases a power of two >= 1; a phase is one strip, 1 << strip_shift
// columns).
__host__ __device__ inline int phase_shift(const TileGeom& g, int group) {
  return (group & (g.tile_phases - 1)) << g.strip_shift;
}

// Phase of a footprint spanning cells [c0, c1] (c0 >= 0) on tiles of
// 1 << tile_shift columns: the one whose tile columns cut it into the
// fewest pieces, the lowest on ties.  Phase p's columns start p strips
// (1 << strip_shift columns) left of phase 0's.
__host__ __device__ inline int footprint_phase(int c0, int c1,
                                               int tile_shift,
                                               int strip_shift, int phases) {
  int best = 0, fewest = (c1 >> tile_shift) - (c0 >> tile_shift);
  for (int p = 1; p < phases; ++p) {
    const int sh = p << strip_shift;
    const int n = ((c1 + sh) >> tile_shift) - ((c0 + sh) >> tile_shift);
    if (n < fewest) {
      fewest = n;
      best = p;
    }
  }
  return best;
}

// Work item of the gridding kernel: a range of sorted records of one tile.
// Record positions take all 32 bits (a call has up to 2^32 - 16 records): a
// position plus a stride may wrap, so loops from kWideRecords on test the
// distance to rec_end.  No item is empty.
struct WorkItem {
  int tile;        // global tile index (grid * tiles_per_grid + tile)
  uint32_t rec_begin;
  uint32_t rec_end;
  int slot;        // partial-tile slot, or -1 when the item owns the tile
};

// Chunks of at most `chunk` records that `count` records make, and the item of
// chunk j of the records [begin, end).
__host__ __device__ inline uint32_t num_chunks(uint32_t count,
                                               uint32_t chunk) {
  return count / chunk + (count % chunk != 0 ? 1u : 0u);
}
__host__ __device__ inline WorkItem chunk_item(int tile, uint32_t begin,
                                               uint32_t end, uint32_t chunk,
                                               uint32_t j, int slot) {
  WorkItem w;
  w.tile = tile;
  w.rec_begin = begin + j * chunk;
  const uint32_t left = end - w.rec_begin;
  w.rec_end = w.rec_begin + (left < chunk ? left : chunk);
  w.slot = slot;
  return w;
}

}  // namespace gg
