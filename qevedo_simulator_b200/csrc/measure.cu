// Measurement on the device: FP64 reductions and the two-pass sampler.
//
// Reductions (norm, per-bit probabilities) accumulate in double precision in
// a fixed order per launch shape, so repeated calls give identical results.
//
// The sampler restates StateVector::sample_unordered (src/measure.rs:104-174)
// so that, for the same amplitudes and the same uniforms, every outcome is
// bit-identical to the reference's:
//   - the state is cut into chunks of CHUNK_BLOCKS * LANES amplitudes
//     (4096 * 8 = 32768 for complex64, 4096 * 4 = 16384 for complex128,
//     src/measure.rs:13 and src/simd.rs:71-97), in physical index order;
//   - p = re*re + im*im in f64 without contraction (__dmul_rn/__dadd_rn);
//   - each chunk sum is one sequential left fold in index order (one lane
//     owns a chunk);
//   - the chunk prefix is sequential; targets = u * total are sorted in f64
//     total order; bounds are partition points of the prefix;
//   - the walk adds p in index order from prefix[chunk] and emits the first
//     index whose running sum exceeds the target, or the last nonzero index.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <mutex>
#include <vector>

#include "engine.hpp"
#include "qvdg.h"

namespace qvdg {

namespace {

constexpr int kThreads = 256;

__host__ __device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

template <typename T>
__device__ __forceinline__ double prob(const cplx_t<T>& a) {
  const double re = double(a.x), im = double(a.y);
  return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic block sum (result valid in thread 0).
__device__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t += red[w];
  return t;
}

// The grid's total of each block's `mine` (in thread 0), in block order, by
// whichever block finishes last: true there, with the total in thread 0. One
// launch instead of two: most of an expectation's time on a small state is
// launches. `ticket` is 0 between launches on a state's stream.
__device__ bool grid_sum(double mine, double* __restrict__ partials, unsigned* ticket, double* red, double& total) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = mine;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double t = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) t += __ldcg(partials + i);
  total = block_sum(t, red);
  if (threadIdx.x == 0) *ticket = 0;
  return true;
}

// The amplitudes of a 16-byte vector: two of complex64, one of complex128.
template <typename T>
constexpr int kPerVec = sizeof(T) == 4 ? 2 : 1;

template <typename T>
__device__ __forceinline__ void unpack(const float4& v, cplx_t<T>* a) {
  if constexpr (sizeof(T) == 4) {
    a[0] = make_float2(v.x, v.y);
    a[1] = make_float2(v.z, v.w);
  } else {
    a[0] = *reinterpret_cast<const double2*>(&v);
  }
}

// Vectors a thread of a whole-state reduction has in flight. These passes
// read the state once (HBM bounds them); with one 8-byte load in flight per
// thread they ran at half the copy rate.
constexpr int kReduceUnroll = 4;
// Blocks of a reduction that an SM holds; its grid has no more. With 8 an SM
// the last ones ran alone: norm of 27 qubits complex64 0.183 -> 0.160 ms, of 26
// qubits complex128 0.263 -> 0.195, a Z string 0.182 -> 0.173 and 0.208 ->
// 0.178, a host's 10 us included.
constexpr int kSumBlocks = 6;
template <bool kPairs>
constexpr int kPauliBlocks = kPairs ? 4 : 5;

// A sum in mapped host memory and, stored after it, that it is there. A host
// that polls `done` has it about 2 us before a synchronisation with the
// stream returns (a 13-qubit circuit and 25 expectations: 1.13 -> 1.08 ms).
struct HostSum {
  double sum;
  unsigned done;
};
__device__ __forceinline__ void post(HostSum* out, double sum) {
  out->sum = sum;
  __threadfence_system();
  *reinterpret_cast<volatile unsigned*>(&out->done) = 1;
}

// What k_sumsq leaves: the sum, or, with `gate`, a
// measurement's outcome for `uniform` where the sum is P(1)
// (src/measure.rs:68-80) and the gate that collapses the state on it, as the
// gate kernels read it: the diagonal (keep, 0) or (0, keep), or, for a reset,
// the matrix that also moves the kept amplitude to |0>.
template <typename T>
struct SumResult {
  HostSum* sum = nullptr;
  cplx_t<T>* gate = nullptr;
  double uniform = 0.0;
  int reset = 0;
  int* outcome = nullptr;
};

// Sum of |a|^2 over the vectors (of a state of at least one vector) whose
// index has bit `bit` set, or over all of them (bit < 0); with `odd`, over
// each vector's second amplitude alone.
template <typename T>
__global__ void __launch_bounds__(kThreads, kSumBlocks)
    k_sumsq(const float4* __restrict__ psi, uint64_t count, int bit, int odd, double* __restrict__ partials,
            unsigned* ticket, const SumResult<T> result) {
  __shared__ double red[32];
  double acc = 0.0;
  const uint64_t step = uint64_t(gridDim.x) * kThreads;
  const uint64_t low = bit < 0 ? 0 : (uint64_t(1) << bit) - 1;
  auto at = [&](uint64_t i) { return bit < 0 ? i : (((i & ~low) << 1) | (uint64_t(1) << bit) | (i & low)); };
  for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < count; i += step * kReduceUnroll) {
    float4 v[kReduceUnroll];
#pragma unroll
    for (int u = 0; u < kReduceUnroll; ++u)
      if (i + u * step < count) v[u] = __ldcs(psi + at(i + u * step));
#pragma unroll
    for (int u = 0; u < kReduceUnroll; ++u) {
      if (i + u * step >= count) break;
      cplx_t<T> a[kPerVec<T>];
      unpack<T>(v[u], a);
#pragma unroll
      for (int e = 0; e < kPerVec<T>; ++e)
        if (e == 1 || !odd) acc += prob<T>(a[e]);
    }
  }
  double t;
  if (!grid_sum(block_sum(acc, red), partials, ticket, red, t) || threadIdx.x) return;
  if (!result.gate) {
    post(result.sum, t);
    return;
  }
  double p1 = t < 0.0 ? 0.0 : t;
  p1 = 1.0 < p1 ? 1.0 : p1;
  const bool one = result.uniform < p1;
  const cplx_t<T> keep = make_c<T>(T(1.0 / sqrt(one ? p1 : 1.0 - p1)), T(0)), zero = make_c<T>(T(0), T(0));
  result.gate[0] = one ? zero : keep;
  result.gate[1] = one ? keep : zero;
  if (result.reset) result.gate[2] = result.gate[3] = zero;
  *result.outcome = one ? 1 : 0;
}

// Sums `count` vectors of `width` doubles (vector i at partials + i*width),
// one block per component in a fixed order, into out[0..width): device or
// mapped host memory. A single thread per component took longer than the
// reduction before it on states that fit in L2.
__global__ void __launch_bounds__(kThreads) k_sum_columns(const double* __restrict__ partials, int count, int width,
                                                          double* __restrict__ out) {
  __shared__ double red[32];
  double t = 0.0;
  for (int i = threadIdx.x; i < count; i += kThreads) t += partials[size_t(i) * width + blockIdx.x];
  t = block_sum(t, red);
  if (threadIdx.x == 0) out[blockIdx.x] = t;
}

// Per-bit probabilities. A segment is 1024 consecutive amplitudes: bits 0-1
// inside a thread (4 elements), bits 2-9 from the thread index; a group is
// 2^var_bits consecutive segments, and blocks take groups in turn, so that
// the grid need not be a power of two and fills the SMs evenly. A thread
// keeps one sum per varying segment bit of the group (kSegmentBits at most);
// the group's sum goes to its index bits in lane b of each warp for bit b.
// Each block writes P(bit = 1) for every bit, then the total, to
// partials[block * (n + 1) + ...]. `aligned`: psi lies on a 16-byte boundary
// (a caller's own complex64 buffer may not).
constexpr int kSegmentBits = 6;

template <typename T>
__global__ void __launch_bounds__(kThreads, 4) k_bit_probs(const cplx_t<T>* __restrict__ psi, int n, uint64_t groups,
                                                           int var_bits, bool aligned,
                                                           double* __restrict__ partials) {
  constexpr int kVecs = 4 / kPerVec<T>;  // vectors of a thread's 4 amplitudes
  constexpr int kWarps = kThreads / 32;
  __shared__ double own[kWarps][10 + kSegmentBits];  // bits 0..9 and the segment bits
  __shared__ double index[kWarps][32];               // the group index bits
  __shared__ double totals[kWarps];
  const uint64_t len = uint64_t(1) << n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double tot = 0.0, lo0 = 0.0, lo1 = 0.0, hacc = 0.0;
  double hv[kSegmentBits];
#pragma unroll
  for (int b = 0; b < kSegmentBits; ++b) hv[b] = 0.0;
  for (uint64_t g = blockIdx.x; g < groups; g += gridDim.x) {
    double sum = 0.0;
#pragma unroll 2
    for (uint32_t i = 0; i < (1u << var_bits); ++i) {
      const uint64_t first = (((g << var_bits) + i) << 10) + uint64_t(threadIdx.x) * 4;
      double p[4];
      if (aligned && first + 4 <= len) {
        float4 v[kVecs];
#pragma unroll
        for (int e = 0; e < kVecs; ++e) v[e] = reinterpret_cast<const float4*>(psi + first)[e];
#pragma unroll
        for (int e = 0; e < kVecs; ++e) {
          cplx_t<T> a[kPerVec<T>];
          unpack<T>(v[e], a);
#pragma unroll
          for (int f = 0; f < kPerVec<T>; ++f) p[e * kPerVec<T> + f] = prob<T>(a[f]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = first + e < len ? prob<T>(psi[first + e]) : 0.0;
      }
      lo0 += p[1] + p[3];
      lo1 += p[2] + p[3];
      const double st = (p[0] + p[1]) + (p[2] + p[3]);
      sum += st;
#pragma unroll
      for (int b = 0; b < kSegmentBits; ++b)
        if ((i >> b) & 1) hv[b] += st;
    }
    tot += sum;
    double w = sum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if ((g >> lane) & 1) hacc += w;
  }
  auto put = [&](int bit, double v) {
    const double s = warp_sum(v);
    if (lane == 0) own[warp][bit] = s;
  };
  put(0, lo0);
  put(1, lo1);
#pragma unroll
  for (int b = 2; b < 10; ++b) put(b, ((threadIdx.x >> (b - 2)) & 1) ? tot : 0.0);
#pragma unroll
  for (int b = 0; b < kSegmentBits; ++b) put(10 + b, hv[b]);
  const double t = warp_sum(tot);
  if (lane == 0) totals[warp] = t;
  index[warp][lane] = hacc;
  __syncthreads();
  double* out = partials + size_t(blockIdx.x) * (n + 1);
  for (int bit = threadIdx.x; bit <= n; bit += kThreads) {
    double s = 0.0;
    for (int w = 0; w < kWarps; ++w)
      s += bit == n ? totals[w] : (bit < 10 + var_bits ? own[w][bit] : index[w][bit - 10 - var_bits]);
    out[bit] = s;
  }
}

// The shape of a k_bit_probs launch on at most `most` blocks: groups of up
// to 2^kSegmentBits segments, smaller ones where the state would not give
// every block several.
struct BitProbsShape {
  uint64_t groups;
  int var_bits;
  unsigned blocks;
};
BitProbsShape bit_probs_shape(uint32_t n, uint64_t most) {
  const int seg_bits = n > 10 ? int(n) - 10 : 0;
  BitProbsShape s{};
  s.var_bits = std::min(seg_bits, kSegmentBits);
  while (s.var_bits > 0 && (uint64_t(1) << (seg_bits - s.var_bits)) < 4 * most) --s.var_bits;
  s.groups = uint64_t(1) << (seg_bits - s.var_bits);
  s.blocks = unsigned(std::min(s.groups, most));
  return s;
}

template <typename T>
__global__ void k_probs(const cplx_t<T>* __restrict__ psi, double* __restrict__ out, uint64_t first, uint64_t count,
                        const uint64_t* __restrict__ tables, int ntables) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < count; t += stride) {
    uint64_t i = first + t, p = i;
    if (ntables) {
      p = 0;
      for (int b = 0; b < ntables; ++b) p |= tables[b * 256 + ((i >> (8 * b)) & 255)];
    }
    const cplx_t<T> a = psi[p];
    out[t] = double(a.x) * double(a.x) + double(a.y) * double(a.y);
  }
}

// ---------------------------------------------------------------- sampler
__device__ __forceinline__ void cp_async16_s(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// prob<T> in fewer instructions: for a complex64 amplitude re*re and im*im
// are exact in f64 (24-bit significands), so re*re + im*im rounded once, as
// one fused multiply-add, equals the sum of the two rounded products.
template <typename T>
__device__ __forceinline__ double prob_fast(const cplx_t<T>& a) {
  if constexpr (sizeof(T) == 4) {
    const double re = double(a.x), im = double(a.y);
    return __fma_rn(re, re, __dmul_rn(im, im));
  } else {
    return prob<T>(a);
  }
}

// Sequential f64 folds of p over chunks, in index order: each chunk's sum
// from +0 (src/measure.rs:110-118), or, with `checkpoints`, the running sum
// from prefix[chunk] of the chunks listed in `active`, written down after
// every kCheckpoint amplitudes (the walk of src/measure.rs:134-167 without
// its emissions).
//
// The order of the additions is fixed (bit-exactness), so a chunk's chain of
// 32768 (complex64) dependent additions, 8.4 cycles each, bounds a state of
// few chunks (0.15 ms) and HBM one of many. Warp 0 does nothing but the
// chains, lane c folding chunk c of the block's kFoldChunks; the other warps
// turn amplitudes into probabilities beside it (the f32 to f64 conversions,
// 16 a cycle and SM, took twice the chain's time when the folding lanes did
// them: 0.63 ms for the sums of 26 qubits). Amplitudes come in windows of 512
// bytes a chunk, copied with cp.async kFoldStages - 1 windows ahead;
// probabilities go through two buffers, rows padded by 16 bytes so that the
// chains' 16-byte reads (one row per lane) hit distinct banks. One block
// barrier a window. Past the state's end the windows hold zeros: adding +0
// changes nothing.
constexpr int kFoldChunks = 16;
constexpr int kFoldWarps = 5;    // the chains' and four that convert
constexpr int kFoldStages = 4;
constexpr int kFoldWindow = 512;  // bytes per chunk per window
constexpr int kCheckpoint = 64;  // amplitudes

template <typename T>
constexpr int fold_smem() {
  constexpr int amps = kFoldWindow / int(sizeof(cplx_t<T>));
  return kFoldStages * kFoldChunks * kFoldWindow + 2 * kFoldChunks * (amps * 8 + 16);
}

template <typename T>
__global__ void __launch_bounds__(32 * kFoldWarps) k_fold(const cplx_t<T>* __restrict__ psi, uint64_t len,
                                                          uint64_t chunk_len, uint64_t count,
                                                          const uint32_t* __restrict__ active,
                                                          const double* __restrict__ prefix,
                                                          double* __restrict__ out, int checkpoints) {
  constexpr int kAmp = int(sizeof(cplx_t<T>));
  constexpr int kAmps = kFoldWindow / kAmp;      // per chunk per window
  constexpr int kRow = kAmps * 8 + 16;           // bytes of a row of probabilities
  constexpr int kVecs = kFoldWindow / 16;        // 16-byte vectors per chunk per window
  constexpr int kWorkers = 32 * (kFoldWarps - 1);
  constexpr int kEach = kFoldChunks * kVecs / kWorkers;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* raw = smem;                                                // [stage][chunk][window]
  unsigned char* rows = smem + kFoldStages * kFoldChunks * kFoldWindow;     // [2][chunk][row]
  __shared__ uint64_t first[kFoldChunks];
  const uint64_t item0 = uint64_t(blockIdx.x) * kFoldChunks;
  const int live = int(umin64(kFoldChunks, count - item0));
  if (threadIdx.x < uint32_t(kFoldChunks))
    first[threadIdx.x] = int(threadIdx.x) < live
                             ? (active ? uint64_t(active[item0 + threadIdx.x]) : item0 + threadIdx.x) * chunk_len
                             : len;
  __syncthreads();
  const uint64_t windows = (umin64(chunk_len, len) + kAmps - 1) / kAmps;
  const int worker = int(threadIdx.x) - 32;
  const unsigned char* bytes = reinterpret_cast<const unsigned char*>(psi);
  const uint64_t end_b = len * kAmp;
  const uint32_t raw_s = static_cast<uint32_t>(__cvta_generic_to_shared(raw));
  auto issue = [&](uint64_t w) {
    if (w < windows)
#pragma unroll
      for (int i = 0; i < kEach; ++i) {
        const int v = worker + i * kWorkers, c = v / kVecs, o = v % kVecs;
        const uint64_t at = (first[c] * kAmp) + w * kFoldWindow + uint64_t(o) * 16;
        const uint32_t dst = uint32_t(int(w % kFoldStages) * kFoldChunks * kFoldWindow + v * 16);
        if (at < end_b)
          cp_async16_s(raw_s + dst, bytes + at);
        else
          *reinterpret_cast<float4*>(raw + dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    cp_async_commit();
  };
  // Window w's probabilities into its row buffer (this worker's own copies).
  auto convert = [&](uint64_t w) {
    cp_async_wait<kFoldStages - 2>();
#pragma unroll
    for (int i = 0; i < kEach; ++i) {
      const int v = worker + i * kWorkers, c = v / kVecs, o = v % kVecs;
      const float4 x = *reinterpret_cast<const float4*>(raw + int(w % kFoldStages) * kFoldChunks * kFoldWindow + v * 16);
      unsigned char* row = rows + (int(w & 1) * kFoldChunks + c) * kRow;
      if constexpr (sizeof(T) == 4) {
        const double p0 = prob_fast<float>(make_float2(x.x, x.y)), p1 = prob_fast<float>(make_float2(x.z, x.w));
        *reinterpret_cast<double2*>(row + o * 16) = make_double2(p0, p1);
      } else {
        *reinterpret_cast<double*>(row + o * 8) = prob_fast<double>(*reinterpret_cast<const double2*>(&x));
      }
    }
  };
  const int lane = int(threadIdx.x);
  double s = 0.0;
  double* mine = nullptr;
  if (worker >= 0) {
    for (int w = 0; w < kFoldStages - 1; ++w) issue(uint64_t(w));
    convert(0);
  } else if (checkpoints && lane < live) {
    s = prefix[active[item0 + lane]];
    mine = out + (item0 + lane) * (chunk_len / kCheckpoint);
  }
  __syncthreads();
  for (uint64_t w = 0; w < windows; ++w) {
    if (worker >= 0) {
      issue(w + kFoldStages - 1);
      if (w + 1 < windows) convert(w + 1);
    } else if (lane < kFoldChunks) {
      const double2* row = reinterpret_cast<const double2*>(rows + (int(w & 1) * kFoldChunks + lane) * kRow);
#pragma unroll
      for (int j = 0; j < kAmps / 2; ++j) {
        const double2 p = row[j];
        s = __dadd_rn(s, p.x);
        s = __dadd_rn(s, p.y);
      }
      if (mine && ((w + 1) * kAmps) % kCheckpoint == 0) mine[(w + 1) * kAmps / kCheckpoint - 1] = s;
    }
    __syncthreads();
  }
  if (worker < 0 && lane < live) {
    if (!checkpoints)
      out[item0 + lane] = s;
    else if ((windows * kAmps) % kCheckpoint != 0)  // a state shorter than a checkpoint
      mine[windows * kAmps / kCheckpoint] = s;
  }
  cp_async_wait<0>();  // no copy outlives the kernel's shared memory
}

// prefix[0] = 0, prefix[c + 1] = prefix[c] + sums[c], sequentially
// (src/measure.rs:119-124). A chain of dependent additions (8.4 cycles each)
// in one thread: it works on registers, 16 sums read ahead of their additions,
// and the block copies in and out. 8192 chunks: 70 us with a global store per
// addition, 47 now (a thousand shots of 30 qubits: 2.07 -> 1.97 ms).
__global__ void __launch_bounds__(256) k_prefix(const double* __restrict__ sums, uint64_t nchunks,
                                                double* __restrict__ prefix) {
  constexpr int kTile = 2048, kAhead = 16;
  __shared__ __align__(16) double tile[kTile];
  double p = 0.0;
  if (threadIdx.x == 0) prefix[0] = 0.0;
  for (uint64_t t0 = 0; t0 < nchunks; t0 += kTile) {
    const int n = int(umin64(kTile, nchunks - t0));
    for (int i = threadIdx.x; i < kTile; i += blockDim.x) tile[i] = i < n ? sums[t0 + i] : 0.0;
    __syncthreads();
    if (threadIdx.x == 0) {
      double2* v = reinterpret_cast<double2*>(tile);
      double2 next[kAhead / 2];
#pragma unroll
      for (int e = 0; e < kAhead / 2; ++e) next[e] = v[e];
      for (int i = 0; i < n; i += kAhead) {
        double2 x[kAhead / 2];
#pragma unroll
        for (int e = 0; e < kAhead / 2; ++e) x[e] = next[e];
        const int j = (i + kAhead < kTile ? i + kAhead : 0) / 2;
#pragma unroll
        for (int e = 0; e < kAhead / 2; ++e) next[e] = v[j + e];
#pragma unroll
        for (int e = 0; e < kAhead / 2; ++e) {
          x[e].x = p = __dadd_rn(p, x[e].x);
          x[e].y = p = __dadd_rn(p, x[e].y);
          v[i / 2 + e] = x[e];
        }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) prefix[t0 + i + 1] = tile[i];
    __syncthreads();
  }
}

// Total-order key of a double (f64::total_cmp order as unsigned integers).
__device__ __forceinline__ uint64_t order_key(double x) {
  const uint64_t b = uint64_t(__double_as_longlong(x));
  return (b >> 63) ? ~b : (b | (uint64_t(1) << 63));
}
__device__ __forceinline__ double from_key(uint64_t k) {
  const uint64_t b = (k >> 63) ? (k & ~(uint64_t(1) << 63)) : ~k;
  return __longlong_as_double((long long)b);
}

// targets = u * total (src/measure.rs:125), as sort keys.
__global__ void k_target_keys(const double* __restrict__ uniforms, size_t shots, const double* __restrict__ total,
                              uint64_t* __restrict__ keys) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < shots) keys[i] = order_key(__dmul_rn(uniforms[i], *total));
}

__global__ void k_keys_to_targets(const uint64_t* __restrict__ keys, size_t shots, double* __restrict__ targets) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < shots) targets[i] = from_key(keys[i]);
}

// bounds[c] = number of targets < prefix[c] (partition_point,
// src/measure.rs:128-131); chunks that hold shots are appended to `active`.
__global__ void k_bounds(const double* __restrict__ targets, size_t shots, const double* __restrict__ prefix,
                         uint64_t nchunks, uint64_t* __restrict__ bounds) {
  const uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c > nchunks) return;
  const double p = prefix[c];
  size_t lo = 0, hi = shots;
  while (lo < hi) {
    const size_t mid = (lo + hi) >> 1;
    if (targets[mid] < p)
      lo = mid + 1;
    else
      hi = mid;
  }
  bounds[c] = lo;
}

// Chunks that hold shots, in any order, and each one's place among them.
__global__ void k_active(const uint64_t* __restrict__ bounds, uint64_t nchunks, size_t shots,
                         uint32_t* __restrict__ active, uint32_t* __restrict__ place, uint32_t* __restrict__ count) {
  const uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= nchunks) return;
  const uint64_t lo = bounds[c], hi = umin64(bounds[c + 1], shots);
  if (lo < hi) {
    const uint32_t a = atomicAdd(count, 1u);
    active[a] = uint32_t(c);
    place[c] = a;
  }
}

// Pass 2: the outcome of each sorted target (src/measure.rs:134-167), one
// thread per shot. Its chunk is the one whose bounds hold the shot; the
// reference walks that chunk from prefix[chunk] and emits the first index
// whose running sum exceeds the target. The sums never decrease (p >= +0), so
// the checkpoints (the same sums) tell which kCheckpoint amplitudes hold it,
// and only those are added again, from the checkpoint before them. Targets
// beyond the chunk's last sum get its last nonzero index. (A million shots of
// 28 qubits: one warp walking and emitting per chunk 2.17 ms; the fold 0.40 ms
// and this about 0.15.) Chunks whose place
// among the active ones is outside [a0, a1) are another launch's.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_emit(const cplx_t<T>* __restrict__ psi, uint64_t len,
                                                   uint64_t chunk_len, uint64_t nchunks,
                                                   const uint32_t* __restrict__ place, uint32_t a0, uint32_t a1,
                                                   const double* __restrict__ prefix,
                                                   const uint64_t* __restrict__ bounds, size_t found,
                                                   const double* __restrict__ checkpoints,
                                                   const double* __restrict__ targets, uint64_t* __restrict__ out) {
  const size_t shot = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (shot >= found) return;
  if (shot < bounds[0]) {  // a negative target: in no chunk
    out[shot] = 0;
    return;
  }
  uint64_t lo = 0, hi = nchunks;  // bounds[lo] <= shot < bounds[hi]
  while (hi - lo > 1) {
    const uint64_t mid = (lo + hi) >> 1;
    if (bounds[mid] <= shot)
      lo = mid;
    else
      hi = mid;
  }
  const uint64_t chunk = lo;
  const uint32_t a = place[chunk];
  if (a < a0 || a >= a1) return;
  const uint64_t base = chunk * chunk_len, end = umin64(chunk_len, len - base);
  const uint64_t blocks = (end + kCheckpoint - 1) / kCheckpoint;
  const double* sums = checkpoints + uint64_t(a - a0) * (chunk_len / kCheckpoint);
  const double target = targets[shot];
  uint64_t k = 0, top = blocks;  // the first block whose last sum exceeds the target
  while (k < top) {
    const uint64_t mid = (k + top) >> 1;
    if (target < sums[mid])
      top = mid;
    else
      k = mid + 1;
  }
  if (k < blocks) {
    double s = k ? sums[k - 1] : prefix[chunk];
    const uint64_t first = base + k * kCheckpoint, last = umin64(first + kCheckpoint, base + end);
    for (uint64_t i = first; i < last; ++i) {
      s = __dadd_rn(s, prob_fast<T>(psi[i]));
      if (target < s) {
        out[shot] = i;
        return;
      }
    }
  }
  uint64_t i = base + end;
  while (i > base && !(prob_fast<T>(psi[i - 1]) != 0.0)) --i;
  out[shot] = umin64(i > base ? i - 1 : base, len - 1);
}

// Physical -> logical index through byte tables.
__global__ void k_remap(uint64_t* __restrict__ out, size_t count, const uint64_t* __restrict__ tables, int ntables) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint64_t x = out[i];
  uint64_t l = 0;
  for (int b = 0; b < ntables; ++b) l |= tables[b * 256 + ((x >> (8 * b)) & 255)];
  out[i] = l;
}

template <typename TA, typename TB>
__global__ void __launch_bounds__(kThreads) k_max_diff(const cplx_t<TA>* __restrict__ a,
                                                       const cplx_t<TB>* __restrict__ b, uint64_t len,
                                                       const uint64_t* __restrict__ ta, int nta,
                                                       const uint64_t* __restrict__ tb, int ntb,
                                                       double* __restrict__ partials) {
  __shared__ double red[32];
  double m = 0.0;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < len; i += stride) {
    uint64_t pa = i, pb = i;
    if (nta) {
      pa = 0;
      for (int k = 0; k < nta; ++k) pa |= ta[k * 256 + ((i >> (8 * k)) & 255)];
    }
    if (ntb) {
      pb = 0;
      for (int k = 0; k < ntb; ++k) pb |= tb[k * 256 + ((i >> (8 * k)) & 255)];
    }
    const cplx_t<TA> x = a[pa];
    const cplx_t<TB> y = b[pb];
    const double dr = double(x.x) - double(y.x), di = double(x.y) - double(y.y);
    m = fmax(m, sqrt(dr * dr + di * di));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t = fmax(t, red[w]);
    partials[blockIdx.x] = t;
  }
}

unsigned blocks_for(uint64_t items, int threads) { return unsigned(std::max<uint64_t>(1, (items + threads - 1) / threads)); }

// grid_sum's counter: a word of the state's status buffer, 0 when it is made.
unsigned* ticket(const StateImpl& s) { return reinterpret_cast<unsigned*>(s.status) + 32; }

// The launch of k_sumsq over the amplitudes with physical bit `bit` set
// (bit < 0: all of them).
struct SumShape {
  uint64_t count;
  int vec_bit, odd;
  unsigned blocks;
};
template <typename T>
SumShape sum_shape(const StateImpl& s, int bit) {
  // Bits inside a vector: every vector, complex64's second amplitudes.
  const int shift = kPerVec<T> == 2 ? 1 : 0;
  SumShape h{};
  h.odd = bit >= 0 && bit < shift ? 1 : 0;
  h.vec_bit = bit < shift ? -1 : bit - shift;
  h.count = (s.amp_bytes / 16) >> (h.vec_bit < 0 ? 0 : 1);
  h.blocks = unsigned(std::max<uint64_t>(
      1, umin64(uint64_t(s.sms) * kSumBlocks, (h.count + kThreads * kReduceUnroll - 1) / (kThreads * kReduceUnroll))));
  return h;
}

HostSum* host_sum(StateImpl& s) {
  HostSum* h = static_cast<HostSum*>(s.host.get(sizeof(HostSum)));
  h->done = 0;
  return h;
}

// The sum that the kernel just launched posts. Nothing of the state is read
// or written after that, so what is left of the launch needs no waiting for.
// Up to 10 ms, longer than one of 32 qubits takes; a sum that takes longer, or
// never comes because the launch failed, is waited for by the stream.
double await_sum(StateImpl& s, const HostSum* h) {
  const volatile unsigned* done = &h->done;
  const auto limit = std::chrono::steady_clock::now() + std::chrono::milliseconds(10);
  while (!*done && std::chrono::steady_clock::now() < limit) {
  }
  if (!*done) QVDG_CUDA(cudaStreamSynchronize(s.stream));
  std::atomic_thread_fence(std::memory_order_acquire);
  return h->sum;
}

// Sum of |a|^2 over those amplitudes.
template <typename T>
double sumsq_t(StateImpl& s, int bit) {
  HostSum* h = host_sum(s);
  const SumShape shape = sum_shape<T>(s, bit);
  double* d = static_cast<double*>(s.work.get(shape.blocks * sizeof(double)));
  SumResult<T> result;
  result.sum = h;
  k_sumsq<T><<<shape.blocks, kThreads, 0, s.stream>>>(static_cast<const float4*>(s.amp), shape.count, shape.vec_bit,
                                                      shape.odd, d, ticket(s), result);
  QVDG_LAUNCH_CHECK();
  return await_sum(s, h);
}

// P(1) of the bit with the outcome, and the collapse: two launches and one
// synchronisation.
template <typename T>
int measure_t(StateImpl& s, uint32_t bit, double uniform, bool reset) {
  int* h = static_cast<int*>(s.host.get(sizeof(int)));
  const SumShape shape = sum_shape<T>(s, int(bit));
  char* w = static_cast<char*>(s.work.get(256 + shape.blocks * sizeof(double)));
  cplx_t<T>* gate = reinterpret_cast<cplx_t<T>*>(w);
  double* d = reinterpret_cast<double*>(w + 256);
  SumResult<T> result;
  result.gate = gate;
  result.uniform = uniform;
  result.reset = reset ? 1 : 0;
  result.outcome = h;
  k_sumsq<T><<<shape.blocks, kThreads, 0, s.stream>>>(static_cast<const float4*>(s.amp), shape.count, shape.vec_bit,
                                                      shape.odd, d, ticket(s), result);
  QVDG_LAUNCH_CHECK();
  PlainGate g;
  g.diagonal = !reset;
  g.targets = {bit};
  launch_plain_gate(s, g, gate);
  QVDG_CUDA(cudaStreamSynchronize(s.stream));
  return *h;
}

template <typename T>
void bit_probs_t(StateImpl& s, std::vector<double>& p1, double& total) {
  const int n = int(s.n);
  const BitProbsShape shape = bit_probs_shape(s.n, uint64_t(s.sms) * 4);
  const size_t width = size_t(n) + 1;
  double* d = static_cast<double*>(s.work.get(size_t(shape.blocks) * width * sizeof(double)));
  double* h = static_cast<double*>(s.host.get(width * sizeof(double)));
  k_bit_probs<T><<<shape.blocks, kThreads, 0, s.stream>>>(static_cast<const cplx_t<T>*>(s.amp), n, shape.groups,
                                                          shape.var_bits, true, d);
  QVDG_LAUNCH_CHECK();
  k_sum_columns<<<unsigned(width), kThreads, 0, s.stream>>>(d, int(shape.blocks), int(width), h);
  QVDG_LAUNCH_CHECK();
  QVDG_CUDA(cudaStreamSynchronize(s.stream));
  p1.assign(h, h + n);
  total = h[n];
}

// Byte tables mapping an index through a bit permutation: table bit q of
// the input -> bit perm[q] of the output.
int permutation_tables(StateImpl& s, const std::vector<uint32_t>& perm, uint64_t* dev) {
  const int ntables = int((s.n + 7) / 8);
  std::vector<uint64_t> t(size_t(std::max(ntables, 1)) * 256, 0);
  for (int b = 0; b < ntables; ++b)
    for (int v = 0; v < 256; ++v) {
      uint64_t p = 0;
      for (int bit = 0; bit < 8; ++bit) {
        const uint32_t q = uint32_t(8 * b + bit);
        if (q < s.n && ((v >> bit) & 1)) p |= uint64_t(1) << perm[q];
      }
      t[size_t(b) * 256 + v] = p;
    }
  QVDG_CUDA(cudaMemcpyAsync(dev, t.data(), t.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, s.stream));
  QVDG_CUDA(cudaStreamSynchronize(s.stream));
  return ntables;
}

template <typename T>
void probabilities_t(StateImpl& s, double* out_host) {
  uint64_t* tables = nullptr;
  int nt = 0;
  if (!s.identity_layout()) {
    tables = static_cast<uint64_t*>(s.work2.get(size_t((s.n + 7) / 8) * 256 * sizeof(uint64_t)));
    nt = permutation_tables(s, s.layout, tables);
  }
  const uint64_t chunk = uint64_t(1) << 24;
  const uint64_t len = s.size();
  double* d = static_cast<double*>(s.work.get(std::min(chunk, len) * sizeof(double)));
  for (uint64_t first = 0; first < len; first += chunk) {
    const uint64_t count = std::min(chunk, len - first);
    k_probs<T><<<unsigned(umin64(blocks_for(count, kThreads), uint64_t(s.sms) * 16)), kThreads, 0,
                 s.stream>>>(static_cast<const cplx_t<T>*>(s.amp), d, first, count, tables, nt);
    QVDG_LAUNCH_CHECK();
    copy_to_host(s, out_host + first, d, count * sizeof(double));
  }
}

// The sampler's outcomes (logical indices) left in the workspace at *out_dev;
// returns their number. The workspace's `keys` and `tmp` regions (shots
// entries each) are free afterwards and returned for reuse.
template <typename T>
size_t sample_device_t(StateImpl& s, size_t shots, const double* uniforms_host, uint64_t** out_dev,
                       uint64_t** keys_dev, uint64_t** tmp_dev) {
  const uint64_t len = s.size();
  // CHUNK_BLOCKS (4096) blocks of LANES amplitudes (8 for f32, 4 for f64).
  const uint64_t chunk_len = sizeof(T) == 4 ? 32768 : 16384;
  const uint64_t nchunks = (len + chunk_len - 1) / chunk_len;
  auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t o_sums = 0;
  const size_t o_prefix = o_sums + align(nchunks * 8);
  const size_t o_bounds = o_prefix + align((nchunks + 1) * 8);
  const size_t o_active = o_bounds + align((nchunks + 1) * 8);
  const size_t o_place = o_active + align(nchunks * 4);
  const size_t o_count = o_place + align(nchunks * 4);
  const size_t o_uni = o_count + 256;
  const size_t o_keys = o_uni + align(shots * 8);
  const size_t o_tmp = o_keys + align(shots * 8);
  const size_t o_targets = o_tmp + align(shots * 8);
  const size_t o_out = o_targets + align(shots * 8);
  const size_t o_tables = o_out + align(shots * 8);
  // Checkpoints of the chunks that hold shots, at most 64 MB at a time.
  const size_t per_chunk = size_t(chunk_len / kCheckpoint) * 8;
  const size_t batch = std::min<size_t>(std::min<uint64_t>(nchunks, shots), (size_t(64) << 20) / per_chunk);
  const size_t o_sumsat = o_tables + align(size_t((s.n + 7) / 8 + 1) * 256 * 8);
  const size_t total_bytes = o_sumsat + align(batch * per_chunk);
  char* w = static_cast<char*>(s.work.get(total_bytes));
  double* sums = reinterpret_cast<double*>(w + o_sums);
  double* prefix = reinterpret_cast<double*>(w + o_prefix);
  uint64_t* bounds = reinterpret_cast<uint64_t*>(w + o_bounds);
  uint32_t* active = reinterpret_cast<uint32_t*>(w + o_active);
  uint32_t* place = reinterpret_cast<uint32_t*>(w + o_place);
  double* checkpoints = reinterpret_cast<double*>(w + o_sumsat);
  uint32_t* count = reinterpret_cast<uint32_t*>(w + o_count);
  double* uni = reinterpret_cast<double*>(w + o_uni);
  uint64_t* keys = reinterpret_cast<uint64_t*>(w + o_keys);
  uint64_t* tmp = reinterpret_cast<uint64_t*>(w + o_tmp);
  double* targets = reinterpret_cast<double*>(w + o_targets);
  uint64_t* out = reinterpret_cast<uint64_t*>(w + o_out);
  uint64_t* tables = reinterpret_cast<uint64_t*>(w + o_tables);
  const cplx_t<T>* psi = static_cast<const cplx_t<T>*>(s.amp);

  static OncePerDevice once;  // per instantiation
  once(s.device, [] {
    QVDG_CUDA(cudaFuncSetAttribute(k_fold<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, fold_smem<T>()));
  });
  auto fold = [&](uint64_t items, const uint32_t* which, double* to, int at_checkpoints) {
    k_fold<T><<<unsigned((items + kFoldChunks - 1) / kFoldChunks), 32 * kFoldWarps, fold_smem<T>(), s.stream>>>(
        psi, len, chunk_len, items, which, prefix, to, at_checkpoints);
    QVDG_LAUNCH_CHECK();
  };
  fold(nchunks, nullptr, sums, 0);
  k_prefix<<<1, 256, 0, s.stream>>>(sums, nchunks, prefix);
  QVDG_LAUNCH_CHECK();
  // Staged while the chunks are summed.
  copy_to_device(s, uni, uniforms_host, shots * 8);
  k_target_keys<<<blocks_for(shots, kThreads), kThreads, 0, s.stream>>>(uni, shots, prefix + nchunks, keys);
  QVDG_LAUNCH_CHECK();
  DeviceScratch& sort_work = s.work2;
  radix_sort_u64(keys, tmp, shots, sort_work, s.stream);
  k_keys_to_targets<<<blocks_for(shots, kThreads), kThreads, 0, s.stream>>>(keys, shots, targets);
  QVDG_LAUNCH_CHECK();
  k_bounds<<<blocks_for(nchunks + 1, kThreads), kThreads, 0, s.stream>>>(targets, shots, prefix, nchunks, bounds);
  QVDG_LAUNCH_CHECK();
  QVDG_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), s.stream));
  k_active<<<blocks_for(nchunks, kThreads), kThreads, 0, s.stream>>>(bounds, nchunks, shots, active, place, count);
  QVDG_LAUNCH_CHECK();
  // Shots that land in chunks: min(bounds[nchunks], shots).
  uint64_t* hb = static_cast<uint64_t*>(s.host.get(16));
  QVDG_CUDA(cudaMemcpyAsync(hb, bounds + nchunks, 8, cudaMemcpyDeviceToHost, s.stream));
  uint32_t* hc = reinterpret_cast<uint32_t*>(hb + 1);
  QVDG_CUDA(cudaMemcpyAsync(hc, count, 4, cudaMemcpyDeviceToHost, s.stream));
  QVDG_CUDA(cudaStreamSynchronize(s.stream));
  const size_t found = size_t(umin64(hb[0], shots));
  const uint32_t num_active = *hc;
  for (size_t a0 = 0; a0 < num_active; a0 += batch) {
    const size_t a1 = std::min<size_t>(num_active, a0 + batch);
    fold(a1 - a0, active + a0, checkpoints, 1);
    k_emit<T><<<blocks_for(found, kThreads), kThreads, 0, s.stream>>>(psi, len, chunk_len, nchunks, place, uint32_t(a0),
                                                                     uint32_t(a1), prefix, bounds, found, checkpoints,
                                                                     targets, out);
    QVDG_LAUNCH_CHECK();
  }
  if (!s.identity_layout() && found > 0) {
    // physical bit p holds logical qubit q: inverse of the layout
    std::vector<uint32_t> inverse(s.n);
    for (uint32_t q = 0; q < s.n; ++q) inverse[s.layout[q]] = q;
    const int nt = permutation_tables(s, inverse, tables);
    k_remap<<<blocks_for(found, kThreads), kThreads, 0, s.stream>>>(out, found, tables, nt);
    QVDG_LAUNCH_CHECK();
  }
  *out_dev = out;
  *keys_dev = keys;
  *tmp_dev = tmp;
  return found;
}

template <typename T>
size_t sample_t(StateImpl& s, size_t shots, const double* uniforms_host, uint64_t* out_host) {
  if (shots == 0) return 0;
  uint64_t *out = nullptr, *keys = nullptr, *tmp = nullptr;
  const size_t found = sample_device_t<T>(s, shots, uniforms_host, &out, &keys, &tmp);
  if (found > 0) copy_to_host(s, out_host, out, found * 8);
  return found;
}

// Classical keys of outcomes: bit c of key i = bit q of outcome i for each
// (q, c) measurement (count_outcomes, src/simulator.rs:187-230).
struct MeasureMap {
  uint8_t q[64], c[64];
  int32_t n;
};

__global__ void k_outcome_keys(const uint64_t* __restrict__ out, size_t found, const MeasureMap m,
                               uint64_t* __restrict__ keys) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= found) return;
  const uint64_t o = out[i];
  uint64_t k = 0;
  for (int j = 0; j < m.n; ++j) k |= ((o >> m.q[j]) & 1ull) << m.c[j];
  keys[i] = k;
}

__device__ __forceinline__ bool run_head(const uint64_t* keys, size_t count, size_t i) {
  return i < count && (i == 0 || keys[i] != keys[i - 1]);
}

// Runs of equal sorted keys that begin in each block's kThreads keys.
__global__ void __launch_bounds__(kThreads) k_run_heads(const uint64_t* __restrict__ keys, size_t count,
                                                        uint32_t* __restrict__ heads) {
  const size_t i = size_t(blockIdx.x) * kThreads + threadIdx.x;
  const int n = __syncthreads_count(run_head(keys, count, i));
  if (threadIdx.x == 0) heads[blockIdx.x] = uint32_t(n);
}

// Exclusive prefix sums of `count` values in place, their total to *total
// (mapped host memory); one block of 1024 threads, 1024 values at a time.
__global__ void __launch_bounds__(1024) k_run_offsets(uint32_t* __restrict__ v, unsigned count,
                                                      uint32_t* __restrict__ total) {
  __shared__ uint32_t warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t before = 0;
  for (unsigned first = 0; first < count; first += 1024) {
    const unsigned i = first + threadIdx.x;
    const uint32_t x = i < count ? v[i] : 0u;
    uint32_t run = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += y;
    }
    if (lane == 31) warp_sums[warp] = run;
    __syncthreads();
    uint32_t base = before, all = before;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) base += warp_sums[w];
      all += warp_sums[w];
    }
    if (i < count) v[i] = base + run - x;
    before = all;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = before;
}

// Each run's key and the place of its first one, in order.
__global__ void __launch_bounds__(kThreads) k_run_starts(const uint64_t* __restrict__ keys, size_t count,
                                                         const uint32_t* __restrict__ offsets,
                                                         uint64_t* __restrict__ run_keys,
                                                         uint64_t* __restrict__ starts) {
  __shared__ uint32_t warp_heads[kThreads / 32];
  const size_t i = size_t(blockIdx.x) * kThreads + threadIdx.x;
  const bool head = run_head(keys, count, i);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned mask = __ballot_sync(0xffffffffu, head);
  if (lane == 0) warp_heads[warp] = __popc(mask);
  __syncthreads();
  if (!head) return;
  uint32_t at = offsets[blockIdx.x] + __popc(mask & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) at += warp_heads[w];
  run_keys[at] = keys[i];
  starts[at] = i;
}

template <typename T>
size_t counts_t(StateImpl& s, size_t shots, const double* uniforms_host, const MeasureMap& m,
                std::vector<uint64_t>& keys_out, std::vector<uint64_t>& counts_out) {
  keys_out.clear();
  counts_out.clear();
  if (shots == 0) return 0;
  uint64_t *out = nullptr, *keys = nullptr, *tmp = nullptr;
  const size_t found = sample_device_t<T>(s, shots, uniforms_host, &out, &keys, &tmp);
  if (found == 0) return 0;
  k_outcome_keys<<<blocks_for(found, kThreads), kThreads, 0, s.stream>>>(out, found, m, keys);
  QVDG_LAUNCH_CHECK();
  int bits = 0;  // of a key
  for (int j = 0; j < m.n; ++j) bits = std::max(bits, int(m.c[j]) + 1);
  radix_sort_u64(keys, tmp, found, s.work2, s.stream, bits);
  // The sorted keys' runs: where each begins, found on the device, so that
  // only the distinct keys and their places come back (8 MB and a pass over
  // them on the host for a million shots otherwise).
  const unsigned blocks = blocks_for(found, kThreads);
  uint32_t* heads = static_cast<uint32_t*>(s.work2.get((size_t(blocks) + 1) * sizeof(uint32_t)));
  uint32_t* total = static_cast<uint32_t*>(s.host.get(sizeof(uint32_t)));
  k_run_heads<<<blocks, kThreads, 0, s.stream>>>(keys, found, heads);
  QVDG_LAUNCH_CHECK();
  k_run_offsets<<<1, 1024, 0, s.stream>>>(heads, blocks, total);
  QVDG_LAUNCH_CHECK();
  // `out` (the outcomes) and `tmp` are free now.
  k_run_starts<<<blocks, kThreads, 0, s.stream>>>(keys, found, heads, tmp, out);
  QVDG_LAUNCH_CHECK();
  QVDG_CUDA(cudaStreamSynchronize(s.stream));
  const size_t runs = *total;
  uint64_t* h = static_cast<uint64_t*>(s.host.get(2 * runs * sizeof(uint64_t)));
  QVDG_CUDA(cudaMemcpyAsync(h, tmp, runs * sizeof(uint64_t), cudaMemcpyDeviceToHost, s.stream));
  QVDG_CUDA(cudaMemcpyAsync(h + runs, out, runs * sizeof(uint64_t), cudaMemcpyDeviceToHost, s.stream));
  QVDG_CUDA(cudaStreamSynchronize(s.stream));
  keys_out.assign(h, h + runs);
  counts_out.resize(runs);
  for (size_t i = 0; i < runs; ++i) counts_out[i] = (i + 1 < runs ? h[runs + i + 1] : uint64_t(found)) - h[runs + i];
  return found;
}

// <psi|P|psi> for a Pauli string with X/Y on the bits of x, Z/Y on the bits of
// z (physical): P|j> = i^nY (-1)^popc(j & z) |j ^ x>, so the value is
// i^nY * sum_j conj(psi[j ^ x]) psi[j] (-1)^popc(j & z). The terms of j and
// j ^ x are complex conjugates up to the sign (-1)^nY, so the sum is real
// (nY even) or imaginary (nY odd), and one of the two terms gives both. Each
// pair of amplitudes is then read once: j runs over the vectors whose x has
// its top bit clear, with the partner vector beside it (HBM bounds the pass;
// reading every amplitude twice and summing both parts of both terms took
// 0.42 ms at 27 qubits in complex64, whose 1 GiB takes 0.16 ms).
// Per-block sums in double precision, summed in a fixed order.
// kPairs: x reaches beyond a vector (partner vectors at v ^ xv); otherwise
// x is 0 or, in complex64, 1 (both amplitudes of a pair in one vector).
template <typename T, bool kPairs>
__global__ void __launch_bounds__(kThreads, kPauliBlocks<kPairs>)
    k_pauli(const float4* __restrict__ psi, uint64_t count, uint64_t x, uint64_t z, int top, int imaginary,
            double* __restrict__ partials, unsigned* ticket, HostSum* __restrict__ out) {
  constexpr int V = kPerVec<T>;
  __shared__ double red[32];
  double acc = 0.0;
  const uint64_t step = uint64_t(gridDim.x) * kThreads;
  const uint64_t low = kPairs ? (uint64_t(1) << top) - 1 : 0;
  const uint64_t xv = x / V;  // x on vector indices
  auto at = [&](uint64_t i) { return kPairs ? (((i & ~low) << 1) | (i & low)) : i; };
  // Sign of amplitude j, from its vector's sign and its place in it.
  const double second = (V == 2 && (z & 1)) ? -1.0 : 1.0;
  for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < count; i += step * kReduceUnroll) {
    float4 u[kReduceUnroll], w[kReduceUnroll];
#pragma unroll
    for (int k = 0; k < kReduceUnroll; ++k)
      if (i + k * step < count) {
        const uint64_t v = at(i + k * step);
        u[k] = __ldcs(psi + v);
        if (kPairs) w[k] = __ldcs(psi + (v ^ xv));
      }
#pragma unroll
    for (int k = 0; k < kReduceUnroll; ++k) {
      if (i + k * step >= count) break;
      const uint64_t v = at(i + k * step);
      cplx_t<T> a[V], b[V];
      unpack<T>(u[k], a);
      unpack<T>(kPairs ? w[k] : u[k], b);
      double t = 0.0;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        // The partner of amplitude e: place e ^ (x & 1) of the other vector.
        const cplx_t<T> c = (V == 2 && (x & 1)) ? b[V - 1 - e] : b[e];
        // conj(c) * a, its real or imaginary part
        const double p = imaginary ? double(c.x) * double(a[e].y) - double(c.y) * double(a[e].x)
                                   : double(c.x) * double(a[e].x) + double(c.y) * double(a[e].y);
        t += e == 1 ? second * p : p;
      }
      acc += (__popcll((v * V) & z) & 1) ? -t : t;
    }
  }
  double t;
  if (grid_sum(block_sum(acc, red), partials, ticket, red, t) && threadIdx.x == 0) post(out, kPairs ? 2.0 * t : t);
}

template <typename T>
double pauli_t(StateImpl& s, uint64_t x, uint64_t z, int ny) {
  const uint64_t xv = x / kPerVec<T>;
  const int top = xv ? 63 - __builtin_clzll(xv) : 0;
  const uint64_t count = (s.amp_bytes / 16) >> (xv ? 1 : 0);
  const unsigned blocks = unsigned(std::max<uint64_t>(
      1, umin64(uint64_t(s.sms) * (xv ? kPauliBlocks<true> : kPauliBlocks<false>),
                (count + kThreads * kReduceUnroll - 1) / (kThreads * kReduceUnroll))));
  double* d = static_cast<double*>(s.work.get(blocks * sizeof(double)));
  HostSum* h = host_sum(s);
  const float4* psi = static_cast<const float4*>(s.amp);
  if (xv)
    k_pauli<T, true><<<blocks, kThreads, 0, s.stream>>>(psi, count, x, z, top, ny & 1, d, ticket(s), h);
  else
    k_pauli<T, false><<<blocks, kThreads, 0, s.stream>>>(psi, count, x, z, top, ny & 1, d, ticket(s), h);
  QVDG_LAUNCH_CHECK();
  const double sum = await_sum(s, h);  // i^nY times it is the value
  switch (ny & 3) {
    case 0: return sum;
    case 1: return -sum;
    case 2: return -sum;
    default: return sum;
  }
}

}  // namespace

double max_abs_diff(StateImpl& a, StateImpl& b) {
  if (a.n != b.n) throw Error(1, "states of different sizes");
  const int nt = int((a.n + 7) / 8);
  const size_t tbytes = size_t(nt) * 256 * sizeof(uint64_t);
  uint64_t* ta = static_cast<uint64_t*>(a.work2.get(tbytes));
  uint64_t* tb = static_cast<uint64_t*>(b.work2.get(tbytes));
  const int nta = a.identity_layout() ? 0 : permutation_tables(a, a.layout, ta);
  const int ntb = b.identity_layout() ? 0 : permutation_tables(b, b.layout, tb);
  QVDG_CUDA(cudaStreamSynchronize(b.stream));
  const unsigned blocks = unsigned(umin64(uint64_t(a.sms) * 8, std::max<uint64_t>(1, a.size() / kThreads)));
  double* d = static_cast<double*>(a.work.get(blocks * sizeof(double)));
  if (a.bits == 32 && b.bits == 32)
    k_max_diff<float, float><<<blocks, kThreads, 0, a.stream>>>(static_cast<const float2*>(a.amp),
        static_cast<const float2*>(b.amp), a.size(), ta, nta, tb, ntb, d);
  else if (a.bits == 32)
    k_max_diff<float, double><<<blocks, kThreads, 0, a.stream>>>(static_cast<const float2*>(a.amp),
        static_cast<const double2*>(b.amp), a.size(), ta, nta, tb, ntb, d);
  else if (b.bits == 32)
    k_max_diff<double, float><<<blocks, kThreads, 0, a.stream>>>(static_cast<const double2*>(a.amp),
        static_cast<const float2*>(b.amp), a.size(), ta, nta, tb, ntb, d);
  else
    k_max_diff<double, double><<<blocks, kThreads, 0, a.stream>>>(static_cast<const double2*>(a.amp),
        static_cast<const double2*>(b.amp), a.size(), ta, nta, tb, ntb, d);
  QVDG_LAUNCH_CHECK();
  std::vector<double> h(blocks);
  QVDG_CUDA(cudaMemcpyAsync(h.data(), d, blocks * sizeof(double), cudaMemcpyDeviceToHost, a.stream));
  QVDG_CUDA(cudaStreamSynchronize(a.stream));
  double m = 0.0;
  for (double x : h) m = std::max(m, x);
  return m;
}

double norm_sqr(StateImpl& s) { return s.bits == 32 ? sumsq_t<float>(s, -1) : sumsq_t<double>(s, -1); }

void bit_probabilities(StateImpl& s, std::vector<double>& p1, double& total) {
  if (s.bits == 32)
    bit_probs_t<float>(s, p1, total);
  else
    bit_probs_t<double>(s, p1, total);
}

double probability_one(StateImpl& s, uint32_t physical_bit) {
  return s.bits == 32 ? sumsq_t<float>(s, int(physical_bit)) : sumsq_t<double>(s, int(physical_bit));
}

int measure(StateImpl& s, uint32_t physical_bit, double uniform, bool reset) {
  return s.bits == 32 ? measure_t<float>(s, physical_bit, uniform, reset)
                      : measure_t<double>(s, physical_bit, uniform, reset);
}

void probabilities(StateImpl& s, double* out_host) {
  if (s.bits == 32)
    probabilities_t<float>(s, out_host);
  else
    probabilities_t<double>(s, out_host);
}

size_t sample_counts(StateImpl& s, size_t shots, const double* uniforms_host, const uint32_t* qubits,
                     const uint32_t* clbits, size_t nm, std::vector<uint64_t>& keys, std::vector<uint64_t>& counts) {
  MeasureMap m{};
  // Every pair ORs its bit into the key, as the reference's keyed counting
  // does (src/simulator.rs:204-210); pairs repeated exactly are kept once.
  for (size_t i = 0; i < nm && m.n < 64; ++i) {
    bool dup = false;
    for (int j = 0; j < m.n; ++j) dup = dup || (m.q[j] == qubits[i] && m.c[j] == clbits[i]);
    if (dup) continue;
    m.q[m.n] = uint8_t(qubits[i]);
    m.c[m.n] = uint8_t(clbits[i]);
    ++m.n;
  }
  return s.bits == 32 ? counts_t<float>(s, shots, uniforms_host, m, keys, counts)
                      : counts_t<double>(s, shots, uniforms_host, m, keys, counts);
}

double expect_pauli(StateImpl& s, uint64_t x, uint64_t z, int ny) {
  return s.bits == 32 ? pauli_t<float>(s, x, z, ny) : pauli_t<double>(s, x, z, ny);
}

size_t sample_unordered(StateImpl& s, size_t shots, const double* uniforms_host, uint64_t* out_host) {
  return s.bits == 32 ? sample_t<float>(s, shots, uniforms_host, out_host)
                      : sample_t<double>(s, shots, uniforms_host, out_host);
}


// ---------------------------------------------------------------------------
// Per-bit probabilities with no allocation (qvdg_bit_probabilities_noalloc).
//
// For callers that cannot allocate device memory: the k_bit_probs partials
// and their column sums live in one file-scope device array instead of the
// state's workspace. At most kNoAllocMaxBlocks blocks of k_bit_probs, each
// writing kNoAllocMaxQubits + 1 doubles, plus one row of totals:
// (512 + 1) * 36 doubles = 147,744 bytes, held on every device that loads
// this library until the process exits. Every row the kernels read is
// written earlier in the same call, so nothing needs clearing; calls that
// overlap on the GPU share the array and race.
constexpr uint32_t kNoAllocMaxQubits = 35;
constexpr uint64_t kNoAllocMaxBlocks = 512;
constexpr int kNoAllocMaxDevices = 64;
static __device__ __align__(256) double g_noalloc_scratch[(kNoAllocMaxBlocks + 1) * (kNoAllocMaxQubits + 1)];

namespace {

std::mutex g_noalloc_mutex;
double* g_noalloc_address[kNoAllocMaxDevices] = {};

// The device address of g_noalloc_scratch on `device` (the current device).
// In host code g_noalloc_scratch only names the symbol; its address on a
// device comes from cudaGetSymbolAddress, looked up once per device.
double* noalloc_scratch(int device) {
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_address[device] == nullptr) {
    void* p = nullptr;
    QVDG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_address[device] = static_cast<double*>(p);
  }
  return g_noalloc_address[device];
}

template <typename T>
void bit_probs_noalloc_t(const void* amplitudes, uint32_t n, cudaStream_t stream, double* p1, double* total) {
  int device = 0;
  QVDG_CUDA(cudaGetDevice(&device));
  if (device < 0 || device >= kNoAllocMaxDevices)
    throw Error(QVDG_ERR_UNSUPPORTED, "device index beyond the no-allocation limit of 64 devices");
  double* d = noalloc_scratch(device);
  int sms = 0;
  QVDG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const BitProbsShape shape = bit_probs_shape(n, umin64(uint64_t(sms) * 4, kNoAllocMaxBlocks));
  const size_t width = size_t(n) + 1;
  k_bit_probs<T><<<shape.blocks, kThreads, 0, stream>>>(static_cast<const cplx_t<T>*>(amplitudes), int(n),
                                                        shape.groups, shape.var_bits,
                                                        reinterpret_cast<uintptr_t>(amplitudes) % 16 == 0, d);
  QVDG_LAUNCH_CHECK();
  double* sum = d + size_t(shape.blocks) * width;
  k_sum_columns<<<unsigned(width), kThreads, 0, stream>>>(d, int(shape.blocks), int(width), sum);
  QVDG_LAUNCH_CHECK();
  QVDG_CUDA(cudaMemcpyAsync(p1, sum, n * sizeof(double), cudaMemcpyDeviceToHost, stream));
  QVDG_CUDA(cudaMemcpyAsync(total, sum + n, sizeof(double), cudaMemcpyDeviceToHost, stream));
  QVDG_CUDA(cudaStreamSynchronize(stream));
}

}  // namespace

void bit_probabilities_noalloc(const void* amplitudes, uint32_t num_qubits, uint32_t precision_bits,
                               cudaStream_t stream, double* p1, double* total) {
  if (num_qubits > kNoAllocMaxQubits)
    throw Error(QVDG_ERR_UNSUPPORTED, "num_qubits " + std::to_string(num_qubits) +
                                          " exceeds the no-allocation limit of 35 qubits");
  if (precision_bits == 32)
    bit_probs_noalloc_t<float>(amplitudes, num_qubits, stream, p1, total);
  else
    bit_probs_noalloc_t<double>(amplitudes, num_qubits, stream, p1, total);
}

}  // namespace qvdg
