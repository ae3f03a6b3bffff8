// Pieces shared by the tile-owning kernels (gridding in gg_grid.cu,
// degridding in gg_degrid.cu): the tile shape (2048 cells in eight bands,
// lane = column, kRows rows per lane), bounded mbarrier waits, tap loads and
// the slice descriptor of a record.
#pragma once

#include "gg_internal.h"

namespace gg {

namespace {

constexpr int kRows = 8;          // rows per lane (registers)
constexpr int kWarps = 8;         // consumer warps per CTA
constexpr int kConsumers = kWarps * 32;
constexpr int kCells = kConsumers * kRows; // 2048 cells per tile
static_assert(kRows - 1 <= kSlicePad, "slices need kRows-1 padding rows");
// Bound on every mbarrier wait (each failed probe sleeps ~100 ns): a wait
// that runs out (> ~1 s) sets the error flag and the CTA returns.
constexpr unsigned kWaitLimit = 1u << 24;

template <int TW>
struct WarpShape {
  static constexpr int kLanesY = 32 / TW;          // lane rows per warp
  static constexpr int kBand = kLanesY * kRows;    // rows per warp band
  static constexpr int kTileU = TW;
  static constexpr int kTileV = kWarps * kBand;
};

// ---- mbarrier helpers (shared::cta) --------------------------
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
                                          unsigned limit = kWaitLimit) {
  for (unsigned i = 0; i < limit; ++i) {
    if (mbar_test(bar, parity)) return true;
    if (i >= 32) __nanosleep(64);
  }
  return false;
}
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
// Tap index of tile cell (0, col) of descriptor d with that step.
__device__ __forceinline__ uint32_t slice_tap(uint2 d, int step, int col) {
  const int z = (int)(short)(d.y & 0xFFFFu);
  const int c = d.y & kMirrorU ? z - col : z + col;
  return d.x + (uint32_t)min(max(c, -1), abs(step) - 1);
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
