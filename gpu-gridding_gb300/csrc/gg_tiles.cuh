// Pieces shared by the tile-owning kernels (gridding in gg_grid.cu,
// degridding in gg_degrid.cu): the tile shape (2048 cells in eight bands,
// lane = column, kRows rows per lane), tap loads and the slice descriptor of a
// record.
#pragma once

#include "gg_internal.h"

namespace gg {

namespace {

constexpr int kRows = 8;          // rows per lane (registers)
constexpr int kWarps = 8;         // bands of a tile, one warp each
constexpr int kConsumers = kWarps * 32;
constexpr int kCells = kConsumers * kRows; // 2048 cells per tile
static_assert(kRows - 1 <= kSlicePad, "slices need kRows-1 padding rows");
template <int TW>
struct WarpShape {
  static constexpr int kLanesY = 32 / TW;          // lane rows per warp
  static constexpr int kBand = kLanesY * kRows;    // rows per warp band
  static constexpr int kTileU = TW;
  static constexpr int kTileV = kWarps * kBand;
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  return __ffma2_rn(a, b, c);
}
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}

// Read-only tap load.
__device__ __forceinline__ float2 ld_tap(const float2* p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];"
               : "=f"(v.x), "=f"(v.y)
               : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_tap(const double2* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "l"(p));
  return v;
}

// Descriptor of a record (plane with support s, offsets ou, ov; footprint
// centre at tile-relative column gu, row gv) for its slice, tap S[0][0] at
// index `origin`, row pitch `pitch`:
//   x: tap index of slice column 0 in the slice row of tile row 0 (which
//      may lie outside the stack, or wrap: only sums are tap indices)
//   y: slice column of tile column 0 (bits 0-15, signed), s (16-29), and
//      bits 30 and 31 where the columns (ou < 0) and rows (ov < 0) are
//      mirrored
// so with z and s from y and su, sv = -1 where mirrored, else 1, the tap of
// tile cell (row, col) is
//   taps[x + sv * row * pitch + clamp(z + su * col, -1, 2s + 1)]
// where the clamped ends are zero taps.
constexpr uint32_t kMirrorU = 1u << 30, kMirrorV = 1u << 31;
__device__ __forceinline__ uint2 slice_record(long long origin, int s, int ou,
                                              int ov, int gu, int gv) {
  const int pitch = slice_pitch(s);
  const int z = ou < 0 ? s + gu : s - gu;
  const int row = ov < 0 ? s + gv : s - gv;
  return make_uint2((uint32_t)(origin + (long long)row * pitch),
                    ((uint32_t)z & 0xFFFFu) | (uint32_t)s << 16 |
                        (ou < 0 ? kMirrorU : 0u) |
                        (ov < 0 ? kMirrorV : 0u));
}

// Taps from one tile row to the next of descriptor d.
__device__ __forceinline__ int slice_step(uint2 d) {
  const int pitch = 2 * (int)((d.y >> 16) & 0x3FFFu) + 2;
  return (int)d.y < 0 ? -pitch : pitch;
}
// kRows taps from `at` on, `step` taps apart.  kWide: the stack holds more
// than 4 GiB; below that its byte offsets fit 32 bits, and each row costs one
// 32-bit addition to a common base instead of a 64-bit one (5 % of the
// gridding passes on 8192^2 workloads).
template <bool kWide, typename R2>
__device__ __forceinline__ void load_taps(const R2* __restrict__ taps,
                                          uint32_t at, int step,
                                          R2 (&out)[kRows]) {
  if constexpr (kWide) {
    const R2* p = taps + at;
#pragma unroll
    for (int r = 0; r < kRows; ++r) out[r] = ld_tap(p + (long long)r * step);
  } else {
    const uint32_t first = at * (uint32_t)sizeof(R2);
    const uint32_t bytes = (uint32_t)step * (uint32_t)sizeof(R2);
#pragma unroll
    for (int r = 0; r < kRows; ++r)
      out[r] = ld_tap(
          (const R2*)((const char*)taps + (size_t)(first + r * bytes)));
  }
}

}  // namespace

}  // namespace gg
