// Stable LSD radix sort of 64-bit keys (8-bit digits, a pass for each digit
// in use).
//
// Used by the sampler to sort its targets (the reference sorts them with
// rayon's par_sort_unstable_by(f64::total_cmp), src/measure.rs:125-126; the
// keys here are the doubles' total-order bit patterns, so equal keys are
// equal doubles and stability does not change the result).
//
// Per pass: per-tile digit histograms (and the digits' totals), the tiles'
// places in each digit's run, then a stable scatter. In L2 throughout, so
// latency bounds it: a thread has its 16 keys loaded at once, a warp ranks its
// own 512 with __match_any_sync and meets the block's others twice, and each
// digit's row of tiles is scanned by a warp of its own. A million keys, per
// pass: 10.6 + 13.2 + 23.5 us (a round of 256 keys at a time with four
// barriers; one block scanning all rows) -> 5.0 + 4.2 + 16.3 us.
//
// Up to 4096 keys are sorted by one block in shared memory, a bitonic network
// (equal keys are equal bits, so stability makes no difference): 24 launches
// become one (a thousand shots of 28 qubits: 0.94 -> 0.85 ms).

#include <cuda_runtime.h>

#include <algorithm>

#include "engine.hpp"

namespace qvdg {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTile = 4096;  // keys per tile
constexpr int kRounds = kTile / kThreads;

// The keys of a thread: a warp's are consecutive, 32 a round.
__device__ __forceinline__ size_t first_key() {
  return size_t(blockIdx.x) * kTile + (threadIdx.x >> 5) * (kTile / kWarps) + (threadIdx.x & 31);
}

// hist[digit * pitch + tile], and each digit's total.
__global__ void __launch_bounds__(kThreads) k_hist(const uint64_t* __restrict__ keys, size_t n, int shift,
                                                   uint32_t* __restrict__ hist, uint32_t pitch,
                                                   uint32_t* __restrict__ totals) {
  __shared__ uint32_t counts[256];
  counts[threadIdx.x] = 0;
  __syncthreads();
  const size_t first = first_key();
  uint64_t key[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (first + r * 32 < n) key[r] = keys[first + r * 32];
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (first + r * 32 < n) atomicAdd(&counts[(key[r] >> shift) & 255], 1u);
  __syncthreads();
  const uint32_t c = counts[threadIdx.x];
  hist[size_t(threadIdx.x) * pitch + blockIdx.x] = c;
  if (c) atomicAdd(totals + threadIdx.x, c);
}

// Each row of `hist` to its exclusive sums, after all smaller digits' totals.
// A warp takes a row, 128 tiles at a time (what lies past the last tile, up to
// `pitch`, a multiple of 4, reaches no sum that is used).
__global__ void __launch_bounds__(kThreads) k_scan(uint32_t* __restrict__ hist, uint32_t pitch,
                                                   const uint32_t* __restrict__ totals) {
  __shared__ uint32_t warp_sums[kWarps];
  __shared__ uint32_t start[256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto warp_scan = [&](uint32_t v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += y;
    }
    return v;
  };
  const uint32_t total = totals[threadIdx.x];
  const uint32_t incl = warp_scan(total);
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  uint32_t before = incl - total;
  for (int w = 0; w < warp; ++w) before += warp_sums[w];
  start[threadIdx.x] = before;
  __syncthreads();
  const uint32_t digit = blockIdx.x * kWarps + warp;
  uint32_t run = start[digit];
  uint4* row = reinterpret_cast<uint4*>(hist + size_t(digit) * pitch);
  const uint32_t vecs = pitch / 4;
  uint4 ahead = uint32_t(lane) < vecs ? row[lane] : make_uint4(0, 0, 0, 0);
  for (uint32_t v0 = 0; v0 < vecs; v0 += 32) {
    const uint4 x = ahead;
    if (v0 + 32 + lane < vecs) ahead = row[v0 + 32 + lane];
    const uint32_t sum = x.x + x.y + x.z + x.w;
    const uint32_t upto = warp_scan(sum);
    const uint32_t base = run + upto - sum;
    if (v0 + lane < vecs) row[v0 + lane] = make_uint4(base, base + x.x, base + x.x + x.y, base + x.x + x.y + x.z);
    run += __shfl_sync(0xffffffffu, upto, 31);
  }
}

__global__ void __launch_bounds__(kThreads) k_scatter(const uint64_t* __restrict__ in, uint64_t* __restrict__ out,
                                                      size_t n, int shift, const uint32_t* __restrict__ hist,
                                                      uint32_t pitch) {
  __shared__ uint32_t place[kWarps][256];  // counts, then where each warp's keys of a digit go
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const size_t first = first_key();
  uint64_t key[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) key[r] = first + r * 32 < n ? in[first + r * 32] : 0;
  uint32_t base = hist[size_t(threadIdx.x) * pitch + blockIdx.x];
#pragma unroll
  for (int i = 0; i < 256; i += 32) place[warp][i + lane] = 0;
  __syncwarp();
  uint32_t rank[kRounds];  // among the warp's keys of the same digit
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const bool valid = first + r * 32 < n;
    const uint32_t d = valid ? uint32_t(key[r] >> shift) & 255u : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const uint32_t earlier = valid ? place[warp][d] : 0;
    __syncwarp();
    rank[r] = earlier + __popc(peers & lt);
    if (valid && !(peers & lt)) place[warp][d] = earlier + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const uint32_t c = place[w][threadIdx.x];
    place[w][threadIdx.x] = base;
    base += c;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (first + r * 32 < n) out[place[warp][uint32_t(key[r] >> shift) & 255u] + rank[r]] = key[r];
}

// Up to kTile keys in place; `size` is the power of two from them on.
__global__ void __launch_bounds__(1024) k_sort_block(uint64_t* __restrict__ keys, uint32_t count, uint32_t size) {
  __shared__ uint64_t key[kTile];
  for (uint32_t i = threadIdx.x; i < size; i += blockDim.x) key[i] = i < count ? keys[i] : ~uint64_t(0);
  for (uint32_t k = 2; k <= size; k <<= 1)
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (uint32_t t = threadIdx.x; t < size / 2; t += blockDim.x) {
        const uint32_t a = 2 * t - (t & (j - 1)), b = a + j;
        const uint64_t x = key[a], y = key[b];
        if ((x > y) == ((a & k) == 0)) {
          key[a] = y;
          key[b] = x;
        }
      }
    }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) keys[i] = key[i];
}

}  // namespace

void radix_sort_u64(uint64_t* keys, uint64_t* tmp, size_t count, DeviceScratch& work, cudaStream_t stream, int bits) {
  if (count <= 1) return;
  if (count <= size_t(kTile)) {
    uint32_t size = 2;
    while (size < count) size *= 2;
    k_sort_block<<<1, std::max(32u, std::min(1024u, size / 2)), 0, stream>>>(keys, uint32_t(count), size);
    QVDG_LAUNCH_CHECK();
    return;
  }
  const int end = (bits + 15) / 16 * 16;  // an even number of passes: the result is back in `keys`
  if (count > size_t(0xFFFFFFFFu)) throw Error(1, "too many keys to sort");
  const uint32_t tiles = uint32_t((count + kTile - 1) / kTile), pitch = (tiles + 3) & ~3u;
  const size_t total_bytes = size_t(8) * 256 * sizeof(uint32_t);  // of every pass
  uint32_t* totals = static_cast<uint32_t*>(work.get(total_bytes + size_t(256) * pitch * sizeof(uint32_t)));
  uint32_t* hist = totals + 8 * 256;
  QVDG_CUDA(cudaMemsetAsync(totals, 0, total_bytes, stream));
  uint64_t* src = keys;
  uint64_t* dst = tmp;
  for (int shift = 0; shift < end; shift += 8, totals += 256) {
    k_hist<<<tiles, kThreads, 0, stream>>>(src, count, shift, hist, pitch, totals);
    QVDG_LAUNCH_CHECK();
    k_scan<<<256 / kWarps, kThreads, 0, stream>>>(hist, pitch, totals);
    QVDG_LAUNCH_CHECK();
    k_scatter<<<tiles, kThreads, 0, stream>>>(src, dst, count, shift, hist, pitch);
    QVDG_LAUNCH_CHECK();
    std::swap(src, dst);
  }
}

}  // namespace qvdg
