// Stable LSD radix sort of 64-bit keys (8-bit digits, a pass for each digit
// in use).
//
// Used by the sampler to sort its targets (the reference sorts them with
// rayon's par_sort_unstable_by(f64::total_cmp), src/measure.rs:125-126; the
// keys here are the doubles' total-order bit patterns, so equal keys are
// equal doubles and stability does not change the result).
//
// Per pass: per-tile digit histograms, one exclusive scan over them in
// digit-major order, then a stable scatter in which each warp ranks equal
// digits with __match_any_sync and warps are combined through shared memory.

#include <cuda_runtime.h>

#include "engine.hpp"

namespace qvdg {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTile = 4096;  // keys per tile
constexpr int kRounds = kTile / kThreads;

__global__ void __launch_bounds__(kThreads) k_hist(const uint64_t* __restrict__ keys, size_t n, int shift,
                                                   uint32_t* __restrict__ hist, uint32_t tiles) {
  __shared__ uint32_t counts[256];
  counts[threadIdx.x] = 0;
  __syncthreads();
  const size_t base = size_t(blockIdx.x) * kTile;
  for (int r = 0; r < kRounds; ++r) {
    const size_t i = base + size_t(r) * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&counts[(keys[i] >> shift) & 255], 1u);
  }
  __syncthreads();
  hist[size_t(threadIdx.x) * tiles + blockIdx.x] = counts[threadIdx.x];
}

// Exclusive scan of `count` values in place, one block of 1024 threads, 4096
// consecutive values at a time, the next ones loaded while these are scanned
// (a contiguous segment per thread, read with a stride between lanes, took
// 53 us for a million keys' 62,720 values).
__global__ void __launch_bounds__(1024) k_scan(uint32_t* __restrict__ v, size_t count) {
  __shared__ uint32_t warp_sums[2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto load = [&](size_t first) {
    const size_t i = first + size_t(threadIdx.x) * 4;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (i + 4 <= count) {
      x = *reinterpret_cast<const uint4*>(v + i);
    } else if (i < count) {
      x.x = v[i];
      if (i + 1 < count) x.y = v[i + 1];
      if (i + 2 < count) x.z = v[i + 2];
    }
    return x;
  };
  uint32_t before = 0;
  uint4 ahead = load(0);
  int turn = 0;
  for (size_t first = 0; first < count; first += 4096, turn ^= 1) {
    const uint4 x = ahead;
    if (first + 4096 < count) ahead = load(first + 4096);
    const uint32_t sum = x.x + x.y + x.z + x.w;
    uint32_t run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += y;
    }
    if (lane == 31) warp_sums[turn][warp] = run;
    __syncthreads();
    const uint32_t mine = warp_sums[turn][lane];
    uint32_t all = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, all, o);
      if (lane >= o) all += y;
    }
    const uint32_t base = before + __shfl_sync(0xffffffffu, all - mine, warp) + run - sum;
    before += __shfl_sync(0xffffffffu, all, 31);
    const size_t i = first + size_t(threadIdx.x) * 4;
    const uint4 out = make_uint4(base, base + x.x, base + x.x + x.y, base + x.x + x.y + x.z);
    if (i + 4 <= count) {
      *reinterpret_cast<uint4*>(v + i) = out;
    } else if (i < count) {
      v[i] = out.x;
      if (i + 1 < count) v[i + 1] = out.y;
      if (i + 2 < count) v[i + 2] = out.z;
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_scatter(const uint64_t* __restrict__ in, uint64_t* __restrict__ out,
                                                      size_t n, int shift, const uint32_t* __restrict__ hist,
                                                      uint32_t tiles) {
  __shared__ uint32_t base[256];
  __shared__ uint32_t wcount[kWarps][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  base[threadIdx.x] = hist[size_t(threadIdx.x) * tiles + blockIdx.x];
  const size_t tile = size_t(blockIdx.x) * kTile;
  const unsigned lt = (1u << lane) - 1u;
  for (int r = 0; r < kRounds; ++r) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) wcount[w][threadIdx.x] = 0;
    __syncthreads();
    const size_t i = tile + size_t(r) * kThreads + threadIdx.x;
    const bool valid = i < n;
    const uint64_t key = valid ? in[i] : 0;
    const uint32_t d = valid ? uint32_t((key >> shift) & 255) : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const uint32_t rank = __popc(peers & lt);
    if (valid && rank == 0) wcount[warp][d] = __popc(peers);
    __syncthreads();
    if (valid) {
      uint32_t off = base[d] + rank;
      for (int w = 0; w < warp; ++w) off += wcount[w][d];
      out[off] = key;
    }
    __syncthreads();
    uint32_t add = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) add += wcount[w][threadIdx.x];
    base[threadIdx.x] += add;
    __syncthreads();
  }
}

}  // namespace

void radix_sort_u64(uint64_t* keys, uint64_t* tmp, size_t count, DeviceScratch& work, cudaStream_t stream, int bits) {
  if (count <= 1) return;
  const int end = (bits + 15) / 16 * 16;  // an even number of passes: the result is back in `keys`
  if (count > size_t(0xFFFFFFFFu)) throw Error(1, "too many keys to sort");
  const uint32_t tiles = uint32_t((count + kTile - 1) / kTile);
  uint32_t* hist = static_cast<uint32_t*>(work.get(size_t(256) * tiles * sizeof(uint32_t)));
  uint64_t* src = keys;
  uint64_t* dst = tmp;
  for (int shift = 0; shift < end; shift += 8) {
    k_hist<<<tiles, kThreads, 0, stream>>>(src, count, shift, hist, tiles);
    QVDG_LAUNCH_CHECK();
    k_scan<<<1, 1024, 0, stream>>>(hist, size_t(256) * tiles);
    QVDG_LAUNCH_CHECK();
    k_scatter<<<tiles, kThreads, 0, stream>>>(src, dst, count, shift, hist, tiles);
    QVDG_LAUNCH_CHECK();
    uint64_t* t = src;
    src = dst;
    dst = t;
  }
}

}  // namespace qvdg
