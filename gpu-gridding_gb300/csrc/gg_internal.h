// Host-side declarations shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stddef.h>

#include "gg_common.cuh"

struct gg_kernels;  // kernel-stack handle of the C ABI (gg_api.cu)

namespace gg {

// ---- device-wide exclusive scan of uint32 (gg_sort.cu) --------------------
// out[i] = in[0] + ... + in[i-1]; *d_total (if non-null) = sum of all n.
// in and out may alias.  tmp must hold scan_temp_bytes(n).
size_t scan_temp_bytes(size_t n);
cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, size_t n,
                               uint32_t* d_total, void* tmp, cudaStream_t s);
// The same for two arrays of n entries, in place and in the same launches
// (tmp: scan_temp_bytes(n)).
cudaError_t exclusive_scan_pair_u32(uint32_t* a, uint32_t* b, size_t n,
                                    uint32_t* total_a, uint32_t* total_b,
                                    void* tmp, cudaStream_t s);
// *total (device) = sum of in[0..n) in 64 bits.
cudaError_t sum_u32(const uint32_t* in, size_t n, unsigned long long* total,
                    cudaStream_t s);

// ---- stable LSD radix sort of (key, value) pairs (gg_sort.cu) -------------
// Sorts the first n pairs by key bits [0, end_bit).  Ping-pongs between
// (keys, vals) and (keys_alt, vals_alt); on return *in_alt tells which pair
// of buffers holds the result.  tmp must hold radix_temp_bytes(n).
// Kernel launches of a scan of n entries (one array or a pair), and of a sort.
int scan_launches(size_t n);
int radix_passes(int end_bit);
int radix_launches(size_t n, int end_bit);
size_t radix_temp_bytes(size_t n);
cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals,
                             uint32_t* keys_alt, uint32_t* vals_alt, size_t n,
                             int end_bit, void* tmp, cudaStream_t s,
                             bool* in_alt);

// ---- kernel stack preparation (gg_stack.cu) -------------------------------
// Re-lays conv_func (device, [P][csh][csh] complex) into the slices of
// StackView and forms the FP64 tap sums in the reference's summation order.
// With `changed` given, each of these kernels returns at once while
// *changed == 0 (a cube equal to the one the outputs were made from).
template <typename Real>
cudaError_t launch_stack_relayout(const Real* d_conv_func, StackView view,
                                  void* d_taps_out, cudaStream_t s,
                                  const int* changed = nullptr);
// support_max: the largest support of the stack (sizes the row window).
template <typename Real>
cudaError_t launch_tap_sums(StackView view, double* d_tap_sum,
                            int support_max, cudaStream_t s,
                            const int* changed = nullptr);
// *changed = 1 when the read squares of cubes a and b (device) differ in
// any bit; *changed is left as it is otherwise.
template <typename Real>
cudaError_t launch_cube_compare(const Real* a, const Real* b, StackView view,
                                int* changed, cudaStream_t s);
// dst[p] = src[p] over each plane's read square [0, cube_read_extent)^2;
// src is a cube in host memory that the device addresses (view.support must
// already be on the device).
template <typename Real>
cudaError_t launch_cube_gather(const Real* src, StackView view, Real* dst,
                               cudaStream_t s);

// ---- placement and binning (gg_place.cu) ----------------------------------
// Tile shapes of the gridding kernel: every tile holds 2048 cells, tile_u
// columns by 2048 / tile_u rows.  Shape index 0, 1, 2 = tile_u 32, 16, 8.
constexpr int kNumTileShapes = 3;
__host__ __device__ inline int tile_u_of_shape(int shape) {
  return 32 >> shape;
}
__host__ __device__ inline int tile_v_of_shape(int shape) {
  return 2048 / (32 >> shape);
}

// Tile shape and tile phases for a call, from its mean footprint side
// sqrt(macs / gridded points): narrow tiles only for tiny footprints (a
// 32-wide warp would leave most lanes outside them); tile phases (bits 12 and
// 13: log2 of 1, 2, 4 or 8) four when footprints are narrower than the tile,
// where offset tile grids save the most tile crossings, and the call has
// enough of them for its `tiles` tiles, else one.  What four phases save
// grows with the MACs (more per MAC in narrow tiles), what they cost (the
// partial tiles of the later phases and their addition) with the tiles, and
// there is a fixed cost of 30 to 40 us (a second wait for the host, which sizes
// the partial tiles, and the reduction), 1.5e8 of them: 256^2, support 8 to 13,
// 1.1e8 MACs 0.346 and 0.375, 2.3e8 0.511 and 0.498; 1024^2 0.298 and 0.327,
// 0.454 and 0.426; 16-wide tiles, support 5 and 6, 512^2, 6.3e7 MACs 0.332 and
// 0.347, 1.3e8 0.503 and 0.481.
// Measured, ms with one and four phases (track points, 32-wide tiles where
// support reaches 44, 16-wide for 18): 7.8e6 on 2048^2, support 44 6.85 and
// 5.17, 18 3.09 and 2.50; on 8192^2 6.57 and 5.69, 3.07 and 3.03; 1e6 on
// 2048^2 1.16 and 1.05, 0.63 and 0.64; on 8192^2 1.26 and 1.61, 0.75 and
// 1.17; 4e3 uniform points on 256^2 0.14 and 0.17.
// tiles < 0: degridding, whose phases cost nothing and save 10 % of large
// calls.
// forced_shape >= 0 overrides the shape, phases > 0 the phases.
__host__ __device__ inline uint32_t choose_shape(unsigned long long macs,
                                                 unsigned long long gridded,
                                                 int forced_shape,
                                                 int phases = 1,
                                                 long long tiles = -1) {
  const double side = gridded ? sqrt((double)macs / (double)gridded) : 0.0;
  int shape = forced_shape;
  if (shape < 0) shape = side >= 16.0 ? 0 : (side >= 8.0 ? 1 : 2);
  const int tu = tile_u_of_shape(shape);
  if (phases <= 0)
    phases = side < (double)tu &&
                     (tiles < 0 || (double)macs * (32 / tu) >
                                       7e4 * (double)tiles + 1.5e8)
                 ? 4
                 : 1;
  const uint32_t pbits =
      phases >= 8 ? 3u : (phases >= 4 ? 2u : (phases >= 2 ? 1u : 0u));
  return (uint32_t)shape | (pbits << 12);
}
// In a shape word: the call has kMetaOdd points.
constexpr uint32_t kShapeOdd = 1u << 31;
// Tile phases of a shape word made by choose_shape.
__host__ __device__ inline int phases_of_shape(uint32_t word) {
  return 1 << ((word >> 12) & 3u);
}

struct PlaceOut {
  PlacedPoints points;        // [N] Placed<Real>, or pairs for degridding
  uint32_t* rec_count;        // [N] records (tiles touched) per visibility
  double* blk_norm;           // [num_blocks]
  unsigned long long* blk_skip;   // [num_blocks] skipped + kOneOdd * odd
  unsigned long long* blk_macs;   // [num_blocks]
};
// One kMetaOdd point in the skip counts' upper halves (a call has fewer than
// 2^32 points).
constexpr unsigned long long kOneOdd = 1ull << 32;
// Points per block of the placement kernel (its per-block partials).
constexpr int kPlaceBlock = 256;
int place_num_blocks(unsigned long long n);
template <typename Real>
cudaError_t launch_place(PlaceParams<Real> p, StackView view, TileGeom geom,
                         int grid_index, unsigned long long vis_offset,
                         PlaceOut out, cudaStream_t s);
// *p = v on stream s (device p), without a copy-engine transfer.
cudaError_t launch_store_f64(double* p, double v, cudaStream_t s);
// For a placement made with PlaceParams::defer_norm: the norm terms from
// the placed meta and the stack's tap sums, reduced in k_place's block
// order, then *d_norm += their sum exactly as launch_place_finalize would.
template <typename Real>
cudaError_t launch_norm_terms(PlacedPoints points, const Real* weight,
                              unsigned long long n, StackView view,
                              double* blk_norm, double* d_norm,
                              cudaStream_t s);
// Sums the per-block partials: *d_norm += norm, *d_num_skipped = skips,
// *d_macs = macs (all device pointers), and picks the tile shape and tile
// phases for the call into *d_shape (choose_shape): forced_shape if >= 0,
// phases if > 0, else from the mean footprint area (macs / gridded points).
// kShapeOdd is set in *d_shape where the call has kMetaOdd points.
cudaError_t launch_place_finalize(const double* blk_norm,
                                  const unsigned long long* blk_skip,
                                  const unsigned long long* blk_macs,
                                  int num_blocks, unsigned long long n,
                                  int forced_shape, double* d_norm,
                                  unsigned long long* d_num_skipped,
                                  unsigned long long* d_macs,
                                  uint32_t* d_shape, cudaStream_t s,
                                  int phases = 1, long long tiles = -1);
// use[b] = how many of up to 8192 placed points, evenly spread, are gridded with
// planes p of bin b = p * kPlaneBins / num_planes.
constexpr int kPlaneBins = 256;
cudaError_t launch_plane_use(PlacedPoints points, unsigned long long n,
                             int num_planes, uint32_t* use, cudaStream_t s);
// count[i] = tiles of shape *d_shape touched by visibility i on its tile
// phase (footprint_phase; 0 if skipped).
cudaError_t launch_count_records(PlacedPoints points, unsigned long long n,
                                 StackView view, const uint32_t* d_shape,
                                 uint32_t* count, cudaStream_t s);
template <typename Real>
cudaError_t launch_place_only(PlaceParams<Real> p, StackView view, int* out,
                              cudaStream_t s);
cudaError_t launch_emit_records(PlacedPoints points,
                                const uint32_t* rec_offset,
                                unsigned long long n, StackView view,
                                TileGeom geom, int grid_index,
                                unsigned long long vis_offset, uint32_t* keys,
                                uint32_t* vals, cudaStream_t s,
                                const unsigned long long* grid_offsets =
                                    nullptr,
                                int num_grids = 1,
                                const int* tile_rank = nullptr,
                                bool write_slots = false);
// grid_offsets (device, num_grids + 1): batched calls, where visibility i
// belongs to the grid g with grid_offsets[g] <= i < grid_offsets[g + 1].
// tile_rank (device; degridding): keys hold each tile's tile_rank[tile] in
// place of its index.  write_slots: every gridded point's first emission slot
// goes behind its cell and meta (points 16 bytes apart).

// ---- batched calls (gg_batch.cu) ------------------------------------------
// Per-visibility placement for a batched call: like launch_place, but the
// FP64 norm term of every visibility goes to nterm[i] (0 if skipped) so the
// norm can be reduced per grid.
template <typename Real>
cudaError_t launch_place_batched(PlaceParams<Real> p, StackView view,
                                 PlaceOut out, double* nterm, cudaStream_t s);
// Weighted visibilities and norm terms for new amplitudes and weights on
// an existing placement.
template <typename Real>
cudaError_t launch_revalue(const Real* vis, const Real* weight,
                           StackView view, unsigned long long n, void* placed,
                           double* nterm, cudaStream_t s);
// Deterministic per-grid totals over a chunk table (chunk c covers
// visibilities [chunk_begin[c], chunk_begin[c+1]) of grid chunk_grid[c];
// grid g owns chunks [grid_chunk0[g], grid_chunk0[g+1])):
// d_norm[g] += sum of nterm, d_num_skipped[g] = skips, *d_macs = total
// MACs, *d_shape = choose_shape(total MACs, gridded, forced_shape).
cudaError_t launch_batch_totals(PlacedPoints points, const double* nterm,
                                StackView view, int num_chunks,
                                const unsigned long long* chunk_begin,
                                int num_grids, const int* grid_chunk0,
                                double* chunk_norm,
                                unsigned long long* chunk_skip,
                                unsigned long long* chunk_macs,
                                int forced_shape, double* d_norm,
                                unsigned long long* d_num_skipped,
                                unsigned long long* d_macs, uint32_t* d_shape,
                                cudaStream_t s, int phases = 1,
                                long long tiles = -1);

// ---- work decomposition and gridding (gg_grid.cu) -------------------------
cudaError_t launch_tile_bounds(const uint32_t* keys, uint32_t n, int shift,
                               int num_tiles, uint32_t* tile_start,
                               cudaStream_t s);
// One block whose threads wait, bounded by `limit` probes, on an mbarrier
// that nothing arrives at, then set *error (see gg_plan_probe_bounded_wait).
cudaError_t launch_wait_probe(unsigned limit, uint32_t* error,
                              cudaStream_t s);
// Touched spans of a single-grid call, in strips of tile_u / tile_phases
// columns: for every virtual tile t holding records (tile_start[t + 1] >
// tile_start[t]) of tile row r, lo[r] takes the first strip it covers and
// hi[r] the last + 1.  lo must start at 0xFFFFFFFF and hi at 0.
cudaError_t launch_touched_spans(const uint32_t* tile_start, int num_tiles,
                                 const TileGeom& geom, int grid_size,
                                 uint32_t* lo, uint32_t* hi, cudaStream_t s);
// Strips of tile_u / tile_phases columns by tile rows of a single grid: the
// units of the direct-mode group table and of the touched spans.
inline int num_strips(const TileGeom& g) { return g.strips_u * g.tiles_v; }
// Sets the strip fields of g (tile_u, tile_phases set) for a grid side.
inline void set_strips(TileGeom& g, int grid_size) {
  const int P = g.tile_phases > 1 ? g.tile_phases : 1;
  int sh = 0;
  while ((1 << (sh + 1)) <= g.tile_u / P) ++sh;
  g.strip_shift = sh;
  g.strips_u = (grid_size + (1 << sh) - 1) >> sh;
}
// Work-item queue of a call.  Tiles are virtual tiles (group * tiles_total
// + tile, see TileGeom); the queue is group-major, and within a group the
// chunks of split tiles come first.  group_items[g] .. group_items[g+1] is
// the queue range of plane group g (num_groups + 1 entries).
struct ItemBuffers {
  uint32_t* chunks;       // [num_tiles] chunks per tile (then offsets)
  uint32_t* split_chunks; // [num_tiles] chunks of split tiles (then slots)
  uint32_t* group_items;  // [num_groups + 1]
  int num_groups;
  uint32_t* num_items;    // [1]
  uint32_t* num_slots;    // [1]
  WorkItem* items;        // [capacity]
  int4* split_tiles;      // [num_tiles] (tile, first slot, chunks, -)
  uint32_t* num_split;    // [1]
  uint32_t* counter;      // [1] work counter of the persistent kernel
  void* scan_tmp;
  // Queue order of the tiles within a group: rank r of group g is virtual
  // tile g * T + tile_order[r] (T = tiles per group); null = tile order.
  const int* tile_order = nullptr;
  // > 1: the tiles of virtual groups g with g % partial_phases != 0 (tile
  // phases after the first) write partial tiles even when they have one
  // chunk, so that all the phases of a plane group share one launch.
  int partial_phases = 1;
  // [num_tiles] (first partial slot, chunks) of each virtual tile, chunks 0
  // when it writes none (filled when not null).
  int2* tile_slot = nullptr;
};
cudaError_t launch_build_items(const uint32_t* tile_start, int num_tiles,
                               uint32_t chunk, ItemBuffers b,
                               cudaStream_t s);
// Bytes of a prepared record (launch_grid_tiles' recs, one per record; spans
// takes two more).
template <typename Real>
size_t prepared_record_bytes();
// Prepares the records of every item (recs, spans; without recs the gridding
// kernel prepares them itself, for each band anew), then persistent launches in virtual-group order, each over the work items of
// group_span consecutive virtual groups: with group_span = tile_phases one
// launch per plane group takes all its tile phases (the items were built
// with ItemBuffers::partial_phases = tile_phases: the first phase's
// single-chunk tiles are added to the grid by the launch, every other item
// writes a partial tile); with group_span = 1 one launch per virtual group.
// Each launch is followed by the reduction of its virtual groups' partial
// tiles in group order (grid += their partials in chunk order; all
// the phases of a launch in one pass over the grid when tile_slot, the
// item builder's map, is given): the grid takes the groups' and phases'
// contributions in order.
// wait_before[v] / record_after[v] (arrays of num_groups events, entries
// may be null): s waits for the first before the launch that starts with
// virtual group v and records the second after the launch (and its
// reductions) that ends with v.
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
                              const cudaEvent_t* wait_before = nullptr,
                              const cudaEvent_t* record_after = nullptr,
                              Real* host_grid = nullptr,
                              const uint32_t* tile_groups = nullptr,
                              int group_span = 1,
                              const int2* tile_slot = nullptr,
                              const uint32_t* tile_start = nullptr);
// After launch_grid_tiles, whose kernel leaves kMetaOdd points out: adds these
// to the grid cell by cell, atomically; the cells they reach come out infinite or
// as NaN whatever the order.  With host given, the caller's grid in host memory,
// they are added in `grid`, whose cells are no longer needed, and these sums then
// to host, whose atomics would each cross the link (a tenth of 2.15e6 points on
// 8192^2: 107 ms a call, so 13).  Returns at
// once where the shape word at `shape` (if given) lacks kShapeOdd.
// grid_offsets as in launch_emit_records.
cudaError_t launch_grid_odd(const void* placed, unsigned long long n,
                            const uint32_t* shape, StackView view, int grid_size,
                            float* grid, long long grid_stride,
                            const unsigned long long* grid_offsets,
                            int num_grids, cudaStream_t s,
                            float* host = nullptr);
// Direct mode of a single-grid call: per strip (num_strips), the first and
// last virtual group (plane group and tile phase) with records there
// (first | last << 16, 0xFFFF when none), and *cells += the grid cells of
// the strips with records.  With tile_groups given, launch_grid_tiles reads
// each such strip's cells from host_grid in its first group's pass, writes
// them back there in its last group's, and keeps the sums in between in
// grid: every cell takes the same additions in the same order as when grid
// holds a copy of host_grid.
cudaError_t launch_tile_groups(const uint32_t* tile_start,
                               const TileGeom& geom, int grid_size,
                               uint32_t* out, unsigned long long* cells,
                               cudaStream_t s);
// Blocks of the tile kernels that make a team: a warp for each of a tile's
// eight bands.  What a caller sets and reads are teams (ctas_per_sm, num_ctas),
// as a block of the kernels before these had those eight warps.
constexpr int kBlocksPerTeam = 2;
// Resident blocks per SM (wide: StackView::wide), and the teams that num_ctas
// blocks make.
template <typename Real>
int grid_tiles_ctas_per_sm(int tile_u, bool wide);
int grid_teams(int num_ctas);

// ---- accessors defined in gg_api.cu ---------------------------------------
// Records a failure for gg_last_error() on this thread; returns code.
int record_error(int code, const char* message);
// The device view and properties of a kernel-stack handle.
bool kernels_info(const gg_kernels* k, StackView* view, int* device,
                  bool* is_double, int* num_planes);

// Slice bytes that a gridding pass's taps may come from without leaving an L2
// cache of l2 bytes: three quarters of it (the grid and the records stream
// through the rest).
inline long long cache_budget(int l2) {
  const long long b = (long long)l2 / 4 * 3;
  return b > (1 << 20) ? b : 1 << 20;
}

// ---- uniform weighting (gg_weights.cu) -------------------------------------
// Keys each point by its density cell (grid_size^2 when off the grid), its
// value the weight's bits (FP32) or its index, and counts the off-grid points
// into *d_num_skipped (which must start at 0).
template <typename Real>
cudaError_t launch_weight_keys(const Real* uu, const Real* vv,
                               const Real* weight, unsigned long long n,
                               Real cell_size_rad,
                               int grid_size, uint32_t* keys, uint32_t* vals,
                               unsigned long long* d_num_skipped,
                               cudaStream_t s);
// grid[cell] += the weights of the cell's points, in the order of the
// stably sorted (keys, vals).
template <typename Real>
cudaError_t launch_weight_runs(const uint32_t* keys, const uint32_t* vals,
                               unsigned long long n, const Real* weight,
                               int grid_size, Real* grid, cudaStream_t s);
template <typename Real>
cudaError_t launch_weights_read(const Real* uu, const Real* vv,
                                const Real* w_in, Real* w_out,
                                unsigned long long n, Real cell_size_rad,
                                int grid_size, const Real* grid,
                                unsigned long long* d_num_skipped,
                                cudaStream_t s);

// ---- W-kernel generation (gg_kgen.cu) -------------------------------------
// Writes the taper x chirp cube [P][csh][csh] complex into d_cube; d_total
// holds P complex FP64 normalisation sums (16 B each).
template <typename Real>
cudaError_t launch_kernel_generate(int num_planes, const int* d_support,
                                   const double* d_w_planes, int oversample,
                                   int conv_size_half, void* d_total,
                                   Real* d_cube, cudaStream_t s);

// ---- FP32 FMA throughput probe (gg_calib.cu) ------------------------------
cudaError_t measure_fp32_fma(int num_sms, double* tflops_best, float* ms_out);

// ---- adjoint (gg_degrid.cu) -----------------------------------------------
// Resident CTAs per SM of the degridding kernel.
template <typename Real>
int degrid_tiles_ctas_per_sm(bool wide);
// One persistent launch over all `total` records, sorted by (tile's place in
// the queue order tile_order, ...) with the tile's place above the keys'
// low_bits (32 x 64-cell tiles only): rec_out[rec_offset[v] + rank] = the
// record's share of conj(tap) * grid for every record, rank = the record's
// tile among visibility v's tiles in emission order.  points: 16 bytes apart
// with the slots that launch_emit_records wrote, or 8 bytes apart.
template <typename Real>
cudaError_t launch_degrid_tiles(const uint32_t* rec_key,
                                const uint32_t* rec_vis, uint32_t total,
                                int low_bits, const int* tile_order,
                                PlacedPoints points,
                                const uint32_t* rec_offset, uint32_t* counter,
                                StackView view, TileGeom geom, int grid_size,
                                const Real* grid, const Real* host,
                                const uint32_t* marked, void* rec_out,
                                int num_ctas, cudaStream_t s);
// For a grid at `host`, in the caller's host memory: the cells of the tiles
// with records (tile_start by place in the queue order) come to `grid`, unless
// the records are so few a tile that launch_degrid_tiles (given host and
// marked) reads them there.  marks: strip_mark_bytes; marked: one word.
inline size_t strip_mark_bytes(const TileGeom& g) {
  return ((size_t)num_strips(g) + 3) / 4 * 4;
}
template <typename Real>
cudaError_t launch_gather_tiles(const uint32_t* tile_start,
                                const int* tile_order, TileGeom geom,
                                int num_tiles, uint32_t total,
                                uint32_t* marks, uint32_t* marked,
                                int grid_size, const Real* host, Real* grid,
                                int num_sms, cudaStream_t s);
// out[v] = the sum of visibility v's count[v] partial results from
// rec_out[offset[v]] on, in order.
template <typename Real>
cudaError_t launch_degrid_finish(const uint32_t* count, const uint32_t* offset,
                                 const void* rec_out, unsigned long long n,
                                 Real* out, cudaStream_t s);

}  // namespace gg
