// Device-wide exclusive scan and stable LSD radix sort of (key, value)
// pairs.  These order the (visibility, tile) records by (grid, tile), some
// calls' by plane too, so the gridding kernel sees each tile's records
// contiguously.  The reference bins with an atomic bucket
// scatter whose in-bucket order changes from run to run
// (oskar_grid_wproj_gpu.cu:520-649); this sort is stable, so the record
// order -- and with it the accumulation order -- is the same on every call.
#include "gg_internal.h"

namespace gg {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t x,
                                                         uint32_t* total) {
  __shared__ uint32_t warp_sums[33];  // [32] holds the block total
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  uint32_t inc = warp_inclusive_scan(x);
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < nwarps ? warp_sums[lane] : 0;
    uint32_t wi = warp_inclusive_scan(w);
    if (lane < nwarps) warp_sums[lane] = wi - w;
    if (lane == nwarps - 1) warp_sums[32] = wi;
  }
  __syncthreads();
  uint32_t result = warp_sums[warp] + inc - x;
  *total = warp_sums[32];
  __syncthreads();
  return result;
}

// The arrays of one scan launch: blockIdx.y takes one of two.
struct ScanArrays {
  const uint32_t* in[2];
  uint32_t* out[2];
  uint32_t* total[2];   // may be null
};

__global__ void k_scan_reduce(ScanArrays a, size_t n,
                              uint32_t* __restrict__ block_sums) {
  const uint32_t* __restrict__ in = a.in[blockIdx.y];
  const size_t base = (size_t)blockIdx.x * kScanTile;
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    size_t idx = base + (size_t)i * kScanThreads + threadIdx.x;
    if (idx < n) s += in[idx];
  }
  uint32_t total;
  block_exclusive_scan(s, &total);
  if (threadIdx.x == 0)
    block_sums[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = total;
}

// Exclusive scan of the block sums in place by one block, chunk by chunk.
__global__ void k_scan_top(uint32_t* __restrict__ sums, size_t nb,
                           ScanArrays a) {
  sums += (size_t)blockIdx.y * nb;
  uint32_t carry = 0;
  for (size_t base = 0; base < nb; base += blockDim.x) {
    size_t idx = base + threadIdx.x;
    uint32_t x = idx < nb ? sums[idx] : 0;
    uint32_t total;
    uint32_t ex = block_exclusive_scan(x, &total);
    if (idx < nb) sums[idx] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0 && a.total[blockIdx.y]) *a.total[blockIdx.y] = carry;
}

// One kScanTile of a scan by kThreads_ threads; returns the tile's sum.
template <int kThreads_>
__device__ __forceinline__ uint32_t scan_tile(const uint32_t* in,
                                              uint32_t* out, size_t base,
                                              size_t n, uint32_t before,
                                              uint32_t* tile) {
  constexpr int kItems = kScanTile / kThreads_;
  // Striped, coalesced load into shared memory.
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    int t = i * kThreads_ + threadIdx.x;
    size_t idx = base + t;
    tile[t] = idx < n ? in[idx] : 0;
  }
  __syncthreads();
  // Each thread scans its kItems consecutive entries.
  uint32_t v[kItems];
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    v[i] = tile[threadIdx.x * kItems + i];
    s += v[i];
  }
  uint32_t total;
  uint32_t pre = block_exclusive_scan(s, &total) + before;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    tile[threadIdx.x * kItems + i] = pre;
    pre += v[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    int t = i * kThreads_ + threadIdx.x;
    size_t idx = base + t;
    if (idx < n) out[idx] = tile[t];
  }
  __syncthreads();
  return total;
}

__global__ void k_scan_down(ScanArrays a, size_t n,
                            const uint32_t* __restrict__ block_offsets) {
  __shared__ uint32_t tile[kScanTile];
  scan_tile<kScanThreads>(
      a.in[blockIdx.y], a.out[blockIdx.y], (size_t)blockIdx.x * kScanTile, n,
      block_offsets[(size_t)blockIdx.y * gridDim.x + blockIdx.x], tile);
}

// A whole scan by one block (n <= kScanOneBlock): one launch instead of
// three, which is what a short scan costs (3 to 4 us each in a small call).
constexpr size_t kScanOneBlock = 8 * kScanTile;
__global__ void __launch_bounds__(1024) k_scan_one(ScanArrays a, size_t n) {
  __shared__ uint32_t tile[kScanTile];
  uint32_t sum = 0;
  for (size_t base = 0; base < n; base += kScanTile)
    sum += scan_tile<1024>(a.in[blockIdx.y], a.out[blockIdx.y], base, n, sum,
                           tile);
  if (threadIdx.x == 0 && a.total[blockIdx.y]) *a.total[blockIdx.y] = sum;
}

// ---------------------------------------------------------------------------
// Radix sort: digits of 8 bits, or of 9 where that saves a pass (9, 17, 18 and
// 25 to 27 key bits), 4096 keys per block, reduce-then-scan per pass.  A pass
// of 9 bits writes shorter runs (8 keys of a digit a block on average, one
// sector).  7.8e6 points sorted by the cells of an 8192^2 grid (uniform
// weighting, 27 bits, the whole call): 0.55 ms with three passes, 0.60 with four.
// ---------------------------------------------------------------------------
constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixRounds = 16;
constexpr int kRadixTile = kRadixThreads * kRadixRounds;  // 4096
inline int radix_digit_bits(int end_bit) {
  return (end_bit + 8) / 9 < (end_bit + 7) / 8 ? 9 : 8;
}
// Up to this many blocks the scatter kernel works out its run starts from the
// histograms itself (num_blocks loads a thread, from L2): two launches a pass
// instead of five.
constexpr int kFewBlocks = 192;

template <bool kFew, int kBits>
__global__ void __launch_bounds__(kRadixThreads)
k_radix_hist(const uint32_t* __restrict__ keys, size_t n, int shift,
             int num_blocks, uint32_t* __restrict__ hist) {
  constexpr int kDigits = 1 << kBits;
  __shared__ uint32_t h[kDigits];
  for (int d = threadIdx.x; d < kDigits; d += kRadixThreads) h[d] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * kRadixTile;
  // All loads first (independent, in flight together), then the counts.
  uint32_t k[kRadixRounds];
#pragma unroll
  for (int r = 0; r < kRadixRounds; ++r) {
    const size_t idx = base + (size_t)r * kRadixThreads + threadIdx.x;
    k[r] = idx < n ? keys[idx] : 0u;
  }
#pragma unroll
  for (int r = 0; r < kRadixRounds; ++r) {
    const size_t idx = base + (size_t)r * kRadixThreads + threadIdx.x;
    if (idx < n) atomicAdd(&h[(k[r] >> shift) & (kDigits - 1)], 1u);
  }
  __syncthreads();
  // Digit-major layout: the scan then yields, for each (digit, block), the
  // global position of that block's first key with that digit.  Without a
  // scan (kFew) block-major, so that a block's threads read the counts
  // of a digit each, block by block.
  for (int d = threadIdx.x; d < kDigits; d += kRadixThreads)
    hist[kFew ? (size_t)blockIdx.x * kDigits + d
              : (size_t)d * num_blocks + blockIdx.x] = h[d];
}

// Stable scatter of one 4096-key block: the keys are first ordered by digit
// in shared memory (in block order within a digit), then written out in
// that order, so keys with the same digit go to consecutive addresses and a
// warp's stores form a few contiguous runs instead of 32 scattered words.
// Warp w ranks its own 512 consecutive keys (lane l's j-th key is key
// w * 512 + j * 32 + l of the block) against warp-private digit counters,
// so the ranking needs no block barrier; one per-digit prefix over the
// warps then places every key.  hist holds the block's digit counts
// (as k_radix_hist wrote them) and offsets, unless kFew, their exclusive scan (global start of each (digit, block) run).
template <bool kFew, int kBits>
__global__ void __launch_bounds__(kRadixThreads, 3)
k_radix_scatter(const uint32_t* __restrict__ keys,
                const uint32_t* __restrict__ vals, size_t n, int shift,
                int num_blocks, const uint32_t* __restrict__ hist,
                const uint32_t* __restrict__ offsets,
                uint32_t* __restrict__ keys_out,
                uint32_t* __restrict__ vals_out) {
  constexpr int kPerWarp = kRadixTile / kRadixWarps;   // 512
  __shared__ uint32_t s_keys[kRadixTile];
  __shared__ uint32_t s_vals[kRadixTile];
  constexpr int kDigits = 1 << kBits;
  constexpr uint32_t kMask = kDigits - 1;
  // Thread t owns digits t * kOwn to t * kOwn + kOwn - 1.
  constexpr int kOwn = kDigits / kRadixThreads;
  __shared__ uint32_t digit_base[kDigits];        // global run start
  __shared__ unsigned short local_start[kDigits]; // block-local run start
  // Per warp and digit: the warp's count, then the keys of the digit in
  // the warps before it.
  __shared__ unsigned short warp_count[kRadixWarps][kDigits];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t total, count[kOwn], sum = 0;
  if constexpr (kFew) {
    uint32_t before[kOwn], all[kOwn], every = 0;
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const uint32_t* h = hist + threadIdx.x * kOwn + o;
      before[o] = all[o] = 0;
      count[o] = h[(size_t)blockIdx.x * kDigits];
#pragma unroll 8
      for (int b = 0; b < num_blocks; ++b) {
        const uint32_t c = h[(size_t)b * kDigits];
        all[o] += c;
        if (b < (int)blockIdx.x) before[o] += c;
      }
      every += all[o];
    }
    uint32_t at = block_exclusive_scan(every, &total);
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      digit_base[threadIdx.x * kOwn + o] = at + before[o];
      at += all[o];
    }
  } else {
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const size_t cell =
          (size_t)(threadIdx.x * kOwn + o) * num_blocks + blockIdx.x;
      digit_base[threadIdx.x * kOwn + o] = offsets[cell];
      count[o] = hist[cell];
    }
  }
#pragma unroll
  for (int w = 0; w < kRadixWarps; ++w)
#pragma unroll
    for (int o = 0; o < kOwn; ++o) warp_count[w][threadIdx.x * kOwn + o] = 0;
#pragma unroll
  for (int o = 0; o < kOwn; ++o) sum += count[o];
  // (block_exclusive_scan ends with a barrier: the counters are zeroed.)
  uint32_t start = block_exclusive_scan(sum, &total);
#pragma unroll
  for (int o = 0; o < kOwn; ++o) {
    local_start[threadIdx.x * kOwn + o] = (unsigned short)start;
    start += count[o];
  }
  const uint32_t lt_mask = (1u << lane) - 1u;
  const size_t base = (size_t)blockIdx.x * kRadixTile;
  const int valid_n = (int)min((size_t)kRadixTile, n - base);
  const int wbase = warp * kPerWarp;
  // The warp's keys and values, all loads in flight together.
  uint32_t kr[kRadixRounds], vr[kRadixRounds];
#pragma unroll
  for (int j = 0; j < kRadixRounds; ++j) {
    const int t = wbase + j * 32 + lane;
    kr[j] = t < valid_n ? keys[base + t] : 0u;
    vr[j] = t < valid_n ? vals[base + t] : 0u;
  }
  // Ranks within the warp, in key order: the digit's keys in the warp's
  // earlier rounds plus the lower lanes of this round with the same digit.
  unsigned short* cnt = warp_count[warp];
#pragma unroll
  for (int j = 0; j < kRadixRounds; ++j) {
    const bool valid = wbase + j * 32 + lane < valid_n;
    // Invalid lanes take digit kDigits so they never match a valid one.
    const uint32_t digit = valid ? ((kr[j] >> shift) & kMask) : kDigits;
    const uint32_t peers = __match_any_sync(0xffffffffu, digit);
    // The counter is read at digit & kMask: the load may be issued for
    // invalid lanes too, and digit kDigits would lie past the warp's row (past
    // the whole array for the last warp).
    const uint32_t c_before = cnt[digit & kMask];
    const uint32_t before = valid ? c_before : 0u;
    // The rank waits in s_keys at the key's own index (free until the
    // placement below, which reads it back first).
    s_keys[wbase + j * 32 + lane] = before + __popc(peers & lt_mask);
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1)
      cnt[digit & kMask] = (unsigned short)(before + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  // Per digit: the keys in the warps before each.
#pragma unroll
  for (int o = 0; o < kOwn; ++o) {
    const int d = threadIdx.x * kOwn + o;
    uint32_t running = 0;
#pragma unroll
    for (int w = 0; w < kRadixWarps; ++w) {
      const uint32_t c = warp_count[w][d];
      warp_count[w][d] = (unsigned short)running;
      running += c;
    }
  }
  __syncthreads();   // every digit's prefix written before any is read
  uint32_t pos[kRadixRounds];
#pragma unroll
  for (int j = 0; j < kRadixRounds; ++j) {
    const uint32_t d = (kr[j] >> shift) & kMask;
    pos[j] = local_start[d] + warp_count[warp][d] + s_keys[wbase + j * 32 + lane];
  }
  __syncthreads();   // every rank read before any key lands in s_keys
#pragma unroll
  for (int j = 0; j < kRadixRounds; ++j) {
    // pos < valid_n for every valid key (the ranks of a digit fill its
    // block-local run); the bound also keeps a stray rank in the array.
    if (wbase + j * 32 + lane < valid_n && pos[j] < (uint32_t)kRadixTile) {
      s_keys[pos[j]] = kr[j];
      s_vals[pos[j]] = vr[j];
    }
  }
  __syncthreads();
  // Write the block out in digit order.
  for (int i = threadIdx.x; i < valid_n; i += kRadixThreads) {
    const uint32_t key = s_keys[i];
    const uint32_t d = (key >> shift) & kMask;
    const uint32_t pos = digit_base[d] + ((uint32_t)i - local_start[d]);
    keys_out[pos] = key;
    vals_out[pos] = s_vals[i];
  }
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

size_t scan_temp_bytes(size_t n) {
  size_t nb = (n + kScanTile - 1) / kScanTile;
  return align_up(2 * (nb + 1) * sizeof(uint32_t), 256);
}

// `arrays` scans of n entries each in the same launches; tmp holds
// scan_temp_bytes(n) for each.
static cudaError_t scan_impl(const ScanArrays& a, int arrays, size_t n,
                             void* tmp, cudaStream_t s) {
  if (n == 0) {
    for (int i = 0; i < arrays; ++i)
      if (a.total[i]) {
        cudaError_t e = cudaMemsetAsync(a.total[i], 0, sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
      }
    return cudaSuccess;
  }
  if (n <= kScanOneBlock) {
    k_scan_one<<<dim3(1, arrays), 1024, 0, s>>>(a, n);
    return cudaGetLastError();
  }
  size_t nb = (n + kScanTile - 1) / kScanTile;
  uint32_t* sums = (uint32_t*)tmp;
  k_scan_reduce<<<dim3((unsigned)nb, arrays), kScanThreads, 0, s>>>(a, n,
                                                                    sums);
  k_scan_top<<<dim3(1, arrays), 1024, 0, s>>>(sums, nb, a);
  k_scan_down<<<dim3((unsigned)nb, arrays), kScanThreads, 0, s>>>(a, n, sums);
  return cudaGetLastError();
}

// *total = sum of in[0..n) in 64 bits (the scan's 32-bit total wraps).
__global__ void k_sum_u32(const uint32_t* __restrict__ in, size_t n,
                          unsigned long long* __restrict__ total) {
  unsigned long long v = 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    v += in[i];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __shared__ unsigned long long w[32];
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < (blockDim.x >> 5) ? w[threadIdx.x] : 0ull;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0 && v) atomicAdd(total, v);
  }
}

cudaError_t sum_u32(const uint32_t* in, size_t n, unsigned long long* total,
                    cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(total, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  if (n == 0) return cudaSuccess;
  const size_t blocks = (n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096;
  k_sum_u32<<<(unsigned)blocks, 256, 0, s>>>(in, n, total);
  return cudaGetLastError();
}

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, size_t n,
                               uint32_t* d_total, void* tmp, cudaStream_t s) {
  return scan_impl({{in, nullptr}, {out, nullptr}, {d_total, nullptr}}, 1, n,
                   tmp, s);
}

cudaError_t exclusive_scan_pair_u32(uint32_t* a, uint32_t* b, size_t n,
                                    uint32_t* total_a, uint32_t* total_b,
                                    void* tmp, cudaStream_t s) {
  return scan_impl({{a, b}, {a, b}, {total_a, total_b}}, 2, n, tmp, s);
}

int scan_launches(size_t n) {
  return n == 0 ? 0 : n <= kScanOneBlock ? 1 : 3;
}
int radix_passes(int end_bit) {
  const int bits = radix_digit_bits(end_bit);
  return end_bit <= 0 ? 0 : (end_bit + bits - 1) / bits;
}
int radix_launches(size_t n, int end_bit) {
  if (n <= 1 || end_bit <= 0) return 0;
  const size_t nb = (n + kRadixTile - 1) / kRadixTile;
  return radix_passes(end_bit) *
         (nb > kFewBlocks
              ? 2 + scan_launches(nb << radix_digit_bits(end_bit))
              : 2);
}

size_t radix_temp_bytes(size_t n) {
  size_t nb = (n + kRadixTile - 1) / kRadixTile;
  if (nb == 0) nb = 1;
  const size_t cells = nb << 9;   // the longest digit's
  return 2 * align_up(cells * sizeof(uint32_t), 256) + scan_temp_bytes(cells);
}

template <int kBits>
static cudaError_t radix_pass(const uint32_t* k_in, const uint32_t* v_in,
                              size_t n, int shift, int nb, uint32_t* hist,
                              uint32_t* offs, void* scan_tmp, uint32_t* k_out,
                              uint32_t* v_out, cudaStream_t s) {
  if (nb <= kFewBlocks) {
    k_radix_hist<true, kBits><<<nb, kRadixThreads, 0, s>>>(k_in, n, shift, nb,
                                                           hist);
    k_radix_scatter<true, kBits><<<nb, kRadixThreads, 0, s>>>(
        k_in, v_in, n, shift, nb, hist, offs, k_out, v_out);
    return cudaGetLastError();
  }
  k_radix_hist<false, kBits><<<nb, kRadixThreads, 0, s>>>(k_in, n, shift, nb,
                                                          hist);
  const cudaError_t e = exclusive_scan_u32(hist, offs, (size_t)nb << kBits,
                                           nullptr, scan_tmp, s);
  if (e != cudaSuccess) return e;
  k_radix_scatter<false, kBits><<<nb, kRadixThreads, 0, s>>>(
      k_in, v_in, n, shift, nb, hist, offs, k_out, v_out);
  return cudaGetLastError();
}

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals,
                             uint32_t* keys_alt, uint32_t* vals_alt, size_t n,
                             int end_bit, void* tmp, cudaStream_t s,
                             bool* in_alt) {
  *in_alt = false;
  if (n <= 1 || end_bit <= 0) return cudaSuccess;
  size_t nb = (n + kRadixTile - 1) / kRadixTile;
  const int bits = radix_digit_bits(end_bit);
  const size_t cells = nb << bits;
  size_t hist_bytes = align_up(cells * sizeof(uint32_t), 256);
  uint32_t* hist = (uint32_t*)tmp;
  uint32_t* offs = (uint32_t*)((char*)tmp + hist_bytes);
  void* scan_tmp = (char*)tmp + 2 * hist_bytes;
  uint32_t *k_in = keys, *v_in = vals, *k_out = keys_alt, *v_out = vals_alt;
  for (int shift = 0; shift < end_bit; shift += bits) {
    const cudaError_t e =
        bits == 9 ? radix_pass<9>(k_in, v_in, n, shift, (int)nb, hist, offs,
                                  scan_tmp, k_out, v_out, s)
                  : radix_pass<8>(k_in, v_in, n, shift, (int)nb, hist, offs,
                                  scan_tmp, k_out, v_out, s);
    if (e != cudaSuccess) return e;
    uint32_t* t;
    t = k_in; k_in = k_out; k_out = t;
    t = v_in; v_in = v_out; v_out = t;
    *in_alt = !*in_alt;
  }
  return cudaGetLastError();
}

}  // namespace gg
