// Kernels of the batched (multi-channel) gridding call: many grids -- e.g.
// the frequency channels or snapshots of an observation, each with its own
// number of visibilities -- gridded by one placement pass, one sort and one
// persistent tile-gridding launch.  The reference grids one channel per call
// (main.cpp:243-381 loops over blocks and calls oskar_grid_wproj_f for
// each); a batched call returns, per grid, exactly what that call returns.
//
// Per-grid norm and skip counts are reduced deterministically: every
// visibility's FP64 norm term is stored, chunks of a grid are summed by
// separate blocks in a fixed order, and each grid's chunk sums are then
// added in chunk order.
#include "gg_internal.h"
#include "gg_placement.cuh"

namespace gg {

namespace {

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}

template <typename T>
__device__ __forceinline__ T block_sum(T x) {
  __shared__ T s[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  x = warp_sum(x);
  if (lane == 0) s[warp] = x;
  __syncthreads();
  T r = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kThreads / 32; ++w) r += s[w];
  __syncthreads();
  return r;  // valid in thread 0
}

template <typename Real>
__global__ void __launch_bounds__(kThreads)
k_place_batched(PlaceParams<Real> p, StackView v, PlaceOut out,
                double* __restrict__ nterm) {
  const unsigned long long i =
      (unsigned long long)blockIdx.x * kThreads + threadIdx.x;
  if (i >= p.num_points) return;
  const Placement r = place_one(p, v, i);
  const Real w = p.weight[i];
  Placed<Real> o;
  o.cell = pack_cell(r.gu, r.gv);
  o.meta = pack_meta(r.plane, r.ou, r.ov, r.conj_neg, r.skipped);
  o.v.x = rmul(w, p.vis[2 * i]);
  o.v.y = rmul(w, p.vis[2 * i + 1]);
  o.meta |= odd_bit(o.v, r.skipped);
  ((Placed<Real>*)out.points.p)[i] = o;
  double t = 0.0;
  if (!r.skipped) {
    const int side = 2 * v.omax + 1;
    const double ts = v.tap_sum[((size_t)r.plane * side + (r.ou + v.omax)) *
                                    side + (r.ov + v.omax)];
    // oskar_grid_wproj.c:210: *norm += sum * weight_i (FP64).
    t = __dmul_rn(ts, (double)w);
  }
  nterm[i] = t;
}

// New amplitudes and weights on a kept geometry: weighted visibilities and
// FP64 norm terms from the stored placement (meta), no re-placement.
template <typename Real>
__global__ void __launch_bounds__(kThreads)
k_revalue(const Real* __restrict__ vis, const Real* __restrict__ weight,
          StackView v, unsigned long long n, Placed<Real>* __restrict__ placed,
          double* __restrict__ nterm) {
  using R2 = typename Vec2<Real>::type;
  const unsigned long long i =
      (unsigned long long)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const Real w = weight[i];
  R2 o;
  o.x = rmul(w, vis[2 * i]);
  o.y = rmul(w, vis[2 * i + 1]);
  const uint32_t m = placed[i].meta;
  placed[i].v = o;
  if constexpr (sizeof(Real) == 4)
    placed[i].meta = (m & ~kMetaOdd) | odd_bit(o, meta_skipped(m));
  double t = 0.0;
  if (!meta_skipped(m)) {
    const int side = 2 * v.omax + 1;
    const double ts =
        v.tap_sum[((size_t)meta_plane(m) * side + (meta_ou(m) + v.omax)) *
                      side + (meta_ov(m) + v.omax)];
    t = __dmul_rn(ts, (double)w);
  }
  nterm[i] = t;
}

// One block per chunk of one grid.
__global__ void __launch_bounds__(kThreads)
k_chunk_totals(PlacedPoints points,
               const double* __restrict__ nterm, StackView v,
               const unsigned long long* __restrict__ chunk_begin,
               double* __restrict__ chunk_norm,
               unsigned long long* __restrict__ chunk_skip,
               unsigned long long* __restrict__ chunk_macs) {
  const int c = blockIdx.x;
  const unsigned long long b = chunk_begin[c], e = chunk_begin[c + 1];
  // A thread's points in flight: a chunk is one block, so that the latency of
  // its loads bounds it (16 grids of 62 500 points: 89 us one at a time).
  constexpr int kAhead = 8;
  double n = 0.0;
  unsigned long long skip = 0, macs = 0;
  uint32_t odd = 0;
  for (unsigned long long i0 = b + threadIdx.x; i0 < e;
       i0 += kAhead * kThreads) {
    uint32_t m[kAhead];
    double t[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const unsigned long long i = i0 + j * kThreads;
      m[j] = i < e ? points.at(i).y : 0u;
      t[j] = i < e ? nterm[i] : 0.0;   // 0 for a skipped point
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      if (i0 + j * kThreads >= e) break;
      odd |= m[j] & kMetaOdd;
      n += t[j];
      if (meta_skipped(m[j])) {
        ++skip;
      } else {
        const unsigned long long f = 2ull * v.support[meta_plane(m[j])] + 1;
        macs += f * f;
      }
    }
  }
  n = block_sum(n);
  // Threads with an odd point count as one (only none or some matters).
  skip = block_sum(skip + (odd ? kOneOdd : 0ull));
  macs = block_sum(macs);
  if (threadIdx.x == 0) {
    chunk_norm[c] = n;
    chunk_skip[c] = skip;
    chunk_macs[c] = macs;
  }
}

// One block: thread g adds grid g's chunks in order; the totals choose the
// tile shape of the call.
__global__ void __launch_bounds__(kThreads)
k_batch_finalize(int num_grids, const int* __restrict__ grid_chunk0,
                 const unsigned long long* __restrict__ chunk_begin,
                 const double* __restrict__ chunk_norm,
                 const unsigned long long* __restrict__ chunk_skip,
                 const unsigned long long* __restrict__ chunk_macs,
                 int forced_shape, int phases, long long tiles, double* d_norm,
                 unsigned long long* d_num_skipped,
                 unsigned long long* d_macs, uint32_t* d_shape) {
  unsigned long long points = 0, skips = 0, macs = 0;
  for (int g = threadIdx.x; g < num_grids; g += kThreads) {
    double n = 0.0;
    unsigned long long sk = 0;
    for (int c = grid_chunk0[g]; c < grid_chunk0[g + 1]; ++c) {
      n += chunk_norm[c];
      sk += chunk_skip[c];
      macs += chunk_macs[c];
      points += chunk_begin[c + 1] - chunk_begin[c];
    }
    if (d_norm) d_norm[g] += n;
    if (d_num_skipped) d_num_skipped[g] = sk % kOneOdd;
    skips += sk;
  }
  points = block_sum(points);
  skips = block_sum(skips);
  macs = block_sum(macs);
  if (threadIdx.x == 0) {
    const uint32_t odd = skips >= kOneOdd ? kShapeOdd : 0u;
    skips %= kOneOdd;
    *d_macs = macs;
    *d_shape = choose_shape(macs, points - skips, forced_shape, phases, tiles) |
               odd;
  }
}

}  // namespace

template <typename Real>
cudaError_t launch_place_batched(PlaceParams<Real> p, StackView view,
                                 PlaceOut out, double* nterm, cudaStream_t s) {
  if (p.num_points == 0) return cudaSuccess;
  const unsigned nb = (unsigned)((p.num_points + kThreads - 1) / kThreads);
  k_place_batched<Real><<<nb, kThreads, 0, s>>>(p, view, out, nterm);
  return cudaGetLastError();
}

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
                                cudaStream_t s, int phases, long long tiles) {
  if (num_chunks > 0)
    k_chunk_totals<<<num_chunks, kThreads, 0, s>>>(
        points, nterm, view, chunk_begin, chunk_norm, chunk_skip, chunk_macs);
  k_batch_finalize<<<1, kThreads, 0, s>>>(
      num_grids, grid_chunk0, chunk_begin, chunk_norm, chunk_skip,
      chunk_macs, forced_shape, phases, tiles, d_norm, d_num_skipped, d_macs,
      d_shape);
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_revalue(const Real* vis, const Real* weight,
                           StackView view, unsigned long long n, void* placed,
                           double* nterm, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned nb = (unsigned)((n + kThreads - 1) / kThreads);
  k_revalue<Real><<<nb, kThreads, 0, s>>>(
      vis, weight, view, n, (Placed<Real>*)placed, nterm);
  return cudaGetLastError();
}
template cudaError_t launch_revalue<float>(const float*, const float*,
                                           StackView, unsigned long long,
                                           void*, double*, cudaStream_t);
template cudaError_t launch_revalue<double>(const double*, const double*,
                                            StackView, unsigned long long,
                                            void*, double*, cudaStream_t);

template cudaError_t launch_place_batched<float>(PlaceParams<float>,
                                                 StackView, PlaceOut, double*,
                                                 cudaStream_t);
template cudaError_t launch_place_batched<double>(PlaceParams<double>,
                                                  StackView, PlaceOut,
                                                  double*, cudaStream_t);

}  // namespace gg
