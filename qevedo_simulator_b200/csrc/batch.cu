// Batched layered circuits: thousands of small parameterised circuits of
// uneven width, each layer one 2x2 gate per qubit followed by an optional
// entangler ladder (CX or CZ on (q, q+1) for q = 0..n-2, in that order), run
// to <Z_q> for every qubit of every circuit in ONE persistent launch that is
// captured in a CUDA graph and replayed.
//
// There is no batched path in the reference: each circuit there is a run of
// apply_ops (src/simulator.rs:122-147) on its own StateVector, followed by
// probability_one per qubit (src/measure.rs:43-65). This file computes the
// same quantities, <Z_q> = total - 2 * P(q = 1) with sums in f64, for a whole
// batch at once.
//
// Work distribution: tasks are handed out in order through an atomic counter
// to persistent CTAs. A circuit of n <= L qubits (L = tile qubits, 12-14,
// chosen by the autotuner) is one task and lives in shared memory for its
// whole run. A wider one lives in a slot in HBM; each of its tile passes is
// cut into tasks of a few tiles, so that all SMs share it (one CTA per wide
// circuit left a batch waiting for its widest one). A task waits, in its
// CTA, until the earlier tasks of its circuit that it reads from have
// counted themselves done; those are earlier in the order, held by running
// CTAs that wait only for still earlier ones, so every wait ends whatever
// the number of resident CTAs. The waits are bounded all the same.
//
// Tile passes of a wide circuit: pass A over tiles of the low Lw qubits
// (0..Lw-1), pass B over tiles of the high qubits h0..n-1 and the low r ones
// (rows of 2^r amplitudes). The two overlap in qubits h0..Lw-1, and a layer's
// ladder only ties a qubit to its neighbours, so one A and one B pass apply
// several layers: after layer l on qubits 0..Lw-1, whose gate CX(Lw-1, Lw)
// is still to come, A applies layer l+1 on qubits 0..Lw-2, layer l+2 on
// 0..Lw-3 and so on; B then takes layer l from qubit Lw up, layer l+1 from
// Lw-1 up, down to qubit h0: Lw - h0 + 1 layers for two passes over HBM.
//
// Gates are applied in registers, four qubits at a time: a thread loads the
// 16 amplitudes of a subcube, applies the four 2x2 gates, then the part of
// the entangler ladder that lands in those qubits. A unitary 2x2 gate is
// diag(p) R diag(q) with R real and orthogonal; each row of R is divided by
// its entry of larger magnitude, which goes into p, so a rotation costs one
// (packed) multiply-add per amplitude, and the group's p factors (and CZ
// signs) are one complex multiply per amplitude from a table. CX gates cost
// nothing: those inside the group permute where registers are stored, the
// one into its first qubit, controlled from outside, flips the stores'
// addresses. Ladder order is preserved: groups run in ascending qubit order
// and a ladder gate only touches the qubits of its own and the previous
// group.
//
// Shared-memory and integer issue bound it (384 circuits of 10-22 qubits, 4-12
// layers: ALU pipe 61 % busy, shared memory 49 %, FMA 14 %, HBM 9 %): one CTA
// per wide circuit, a layer per two passes and four multiply-adds a rotation
// took 112 ms, this 11.4.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <numeric>
#include <string>
#include <vector>

#include "batch.hpp"

namespace qvdg {

namespace {

constexpr int kVec = 16;        // >= max tile qubits + 1 (reduction vector)
constexpr int kGroup = 4;       // qubits of a register group
constexpr int kMaxSteps = 16;   // groups whose tables shared memory holds at a time
constexpr long long kTaskWaitCycles = 4000000000ll;  // about two seconds

using u64 = unsigned long long;

// Shared-memory position of tile element e: bits 5-7 are folded into bits
// 1-3 and bit 4 into bit 3, so that the lanes of every register group's
// accesses (8 bytes, or 16 bytes for the group on the lowest bits) reach all
// banks; bit 0 is kept, so element pairs 2v, 2v+1 stay one 16-byte slot
// (cp.async). Linear over XOR.
__device__ __forceinline__ uint32_t swz(uint32_t e) { return e ^ ((e >> 4) & 14u) ^ ((e >> 1) & 8u); }

struct TileMap {
  int low;    // index bits kept below the tile's number
  int high;   // index bit of the element bits above them
  uint32_t tile;
  __device__ __forceinline__ uint32_t global(uint32_t e) const {
    const uint32_t l = e & ((1u << low) - 1u);
    return l | (tile << low) | ((e >> low) << high);
  }
};
// Tiles of the low `bits` qubits.
__device__ __forceinline__ TileMap low_map(int bits, uint32_t tile) { return TileMap{bits, 31, tile}; }

// A register group of a pass: G gates of one layer on local bits
// lq..lq+G-1, which hold qubits q..q+G-1.
// Gates whose rows are led by their off-diagonal entries (`flip`, a bit
// each) are an X and then the diagonal form: the X is only where the subcube
// is read from.
struct Step {
  int32_t G, lq, q;
  uint32_t layer, flip;
};

struct Tables {
  Step step[kMaxSteps];
  float2 gate[kMaxSteps][kGroup][4];          // per gate: (a, b), or the 2x2 matrix
  float2 left[kMaxSteps][2][1 << kGroup];     // factors after the rotations, by the outside control's value
  float2 right[kMaxSteps][1 << kGroup];       // factors before them
};

__device__ __forceinline__ u64 pack(float2 v) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
  return r;
}
__device__ __forceinline__ float2 unpack(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
// a * b + c on both halves.
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ u64 cmul(u64 a, float2 b) { return pack(cmul(unpack(a), b)); }
__device__ __forceinline__ float2 cfma2(float2 m0, float2 x0, float2 m1, float2 x1) {
  float2 o;
  o.x = fmaf(m0.x, x0.x, fmaf(-m0.y, x0.y, fmaf(m1.x, x1.x, -m1.y * x1.y)));
  o.y = fmaf(m0.x, x0.y, fmaf(m0.y, x0.x, fmaf(m1.x, x1.y, m1.y * x1.x)));
  return o;
}

// Where the CX ladder inside a group of G qubits (after the gate into its
// first qubit) sends element j: bit g becomes the parity of bits 0..g; and
// the element that comes to place j.
__host__ __device__ constexpr int ladder_to(int j) {
  int out = 0, c = 0;
  for (int g = 0; g < kGroup; ++g) {
    c ^= (j >> g) & 1;
    out |= c << g;
  }
  return out;
}
__host__ __device__ constexpr int ladder_from(int j) { return j ^ ((j << 1) & ((1 << kGroup) - 1)); }

// Shared-memory accesses by 32-bit address: through a pointer chosen between
// two tile buffers they become generic ones, with 64-bit address arithmetic
// for every amplitude.
__device__ __forceinline__ u64 lds64(uint32_t a) {
  u64 v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ ulonglong2 lds128(uint32_t a) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts64(uint32_t a, u64 v) {
  asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, u64 x, u64 y) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}

// One step on every subcube of the 2^nb-element tile. kLow: the group on the
// lowest bits (lq = 0: its subcubes are contiguous, moved 16 bytes at a
// time; nothing outside controls qubit 0).
template <int G, bool kLow>
__device__ __forceinline__ void apply_step(uint32_t tile, int nb, const Tables& tab, int si, uint32_t form,
                                           int entangler, const TileMap& map) {
  constexpr int S = 1 << G;
  const int lq = kLow ? 0 : tab.step[si].lq, q = tab.step[si].q;
  const uint32_t subcubes = 1u << (nb - G);
  const uint32_t low_mask = (1u << lq) - 1u;
  const bool cx = entangler == QVDG_ENTANGLE_CX_LADDER;
  uint32_t place[G];  // byte distance of the group's bits
#pragma unroll
  for (int g = 0; g < G; ++g) place[g] = swz(1u << (lq + g)) * 8u;
  auto at = [&](int j) {
    uint32_t o = 0;
#pragma unroll
    for (int g = 0; g < G; ++g)
      if ((j >> g) & 1) o ^= place[g];
    return o;
  };
  const uint32_t all = at(S - 1);
  uint32_t flip = 0;
#pragma unroll
  for (int g = 0; g < G; ++g)
    if ((tab.step[si].flip >> g) & 1u) flip ^= place[g];
  for (uint32_t b = threadIdx.x; b < subcubes; b += blockDim.x) {
    const uint32_t e = ((b & ~low_mask) << G) | (b & low_mask);
    const uint32_t base = swz(e) * 8u;
    u64 a[S];
    const uint32_t from = base ^ flip;
    if constexpr (kLow && G > 0) {
      // (16-byte pairs: a flip of bit 0 swaps each one's halves.)
      const uint32_t pair = from & ~8u;
      const bool odd = (from & 8u) != 0;
#pragma unroll
      for (int j = 0; j < S; j += 2) {
        const ulonglong2 v = lds128(tile + (pair ^ at(j)));
        a[j] = odd ? v.y : v.x;
        a[j + 1] = odd ? v.x : v.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < S; ++j) a[j] = lds64(tile + (from ^ at(j)));
    }
    // The ladder's gate into the group's first qubit is controlled by a bit
    // outside it: constant for the subcube.
    const bool ctrl = !kLow && q > 0 && ((map.global(e) >> (q - 1)) & 1u);
    if (form & kBatchShear) {
      if (form & kBatchRight)
#pragma unroll
        for (int j = 0; j < S; ++j) a[j] = cmul(a[j], tab.right[si][j]);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float2 r = tab.gate[si][g][0];
        const u64 ra = pack(make_float2(r.x, r.x)), rb = pack(make_float2(r.y, r.y));
#pragma unroll
        for (int j = 0; j < S; ++j) {
          if (j & (1 << g)) continue;
          const u64 x0 = a[j], x1 = a[j | (1 << g)];
          a[j] = fma2(ra, x1, x0);
          a[j | (1 << g)] = fma2(rb, x0, x1);
        }
      }
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float2 m00 = tab.gate[si][g][0], m01 = tab.gate[si][g][1];
        const float2 m10 = tab.gate[si][g][2], m11 = tab.gate[si][g][3];
#pragma unroll
        for (int j = 0; j < S; ++j) {
          if (j & (1 << g)) continue;
          const float2 x0 = unpack(a[j]), x1 = unpack(a[j | (1 << g)]);
          a[j] = pack(cfma2(m00, x0, m01, x1));
          a[j | (1 << g)] = pack(cfma2(m10, x0, m11, x1));
        }
      }
    }
    if ((form & kBatchShear) || entangler == QVDG_ENTANGLE_CZ_LADDER) {
      const float2* left = tab.left[si][ctrl ? 1 : 0];
#pragma unroll
      for (int j = 0; j < S; ++j) a[j] = cmul(a[j], left[j]);
    }
    if (cx) {
      const uint32_t to = ctrl ? base ^ all : base;
      if constexpr (kLow && G > 1) {
#pragma unroll
        for (int j = 0; j < S; j += 2)
          sts128(tile + (to ^ at(j)), a[ladder_from(j) & (S - 1)], a[ladder_from(j + 1) & (S - 1)]);
      } else {
#pragma unroll
        for (int j = 0; j < S; ++j) sts64(tile + (to ^ at(ladder_to(j) & (S - 1))), a[j]);
      }
    } else if constexpr (kLow && G > 0) {
#pragma unroll
      for (int j = 0; j < S; j += 2)
        sts128(tile + (base ^ at(j)), a[j], a[j + 1]);
    } else {
#pragma unroll
      for (int j = 0; j < S; ++j) sts64(tile + (base ^ at(j)), a[j]);
    }
  }
}

__device__ __forceinline__ void run_step(uint32_t tile, int nb, const Tables& tab, int si, uint32_t form,
                                         int entangler, const TileMap& map) {
  const int G = tab.step[si].G;
  if (tab.step[si].lq == 0) {
    switch (G) {
      case 4: return apply_step<4, true>(tile, nb, tab, si, form, entangler, map);
      case 3: return apply_step<3, true>(tile, nb, tab, si, form, entangler, map);
      case 2: return apply_step<2, true>(tile, nb, tab, si, form, entangler, map);
      default: return apply_step<1, true>(tile, nb, tab, si, form, entangler, map);
    }
  }
  switch (G) {
    case 4: return apply_step<4, false>(tile, nb, tab, si, form, entangler, map);
    case 3: return apply_step<3, false>(tile, nb, tab, si, form, entangler, map);
    case 2: return apply_step<2, false>(tile, nb, tab, si, form, entangler, map);
    default: return apply_step<1, false>(tile, nb, tab, si, form, entangler, map);
  }
}

// Adds the groups of layer `layer` on qubits q0..q1-1 (local bit of qubit q:
// q - q0 + lq0), up to four qubits each, split as evenly as possible (13
// qubits: 4 + 3 + 3 + 3), to the steps (thread 0).
__device__ void add_steps(Tables& tab, int& count, uint32_t layer, int q0, int q1, int lq0) {
  const int m = q1 - q0;
  if (m <= 0) return;
  const int groups = (m + kGroup - 1) / kGroup, small = m / groups, extra = m % groups;
  int q = q0;
  for (int g = 0; g < groups; ++g) {
    const int size = small + (g < extra ? 1 : 0);
    tab.step[count++] = Step{size, lq0 + q - q0, q, layer, 0u};
    q += size;
  }
}

// The steps' gate records and tables (every thread; a barrier before and
// after). `gates`: the circuit's records.
__device__ void build_tables(Tables& tab, int count, const float2* __restrict__ gates, int n, uint32_t form,
                             int entangler) {
  for (int i = threadIdx.x; i < count * kGroup; i += blockDim.x) {
    const Step s = tab.step[i / kGroup];
    const int g = i % kGroup;
    if (g >= s.G) continue;
    const float2* rec = gates + size_t(kBatchGateSlots) * (size_t(s.layer) * n + s.q + g);
    for (int k = 0; k < 4; ++k)
      if (k < 1 || !(form & kBatchShear)) tab.gate[i / kGroup][g][k] = rec[k];
  }
  for (int i = threadIdx.x; i < count << kGroup; i += blockDim.x) {
    const int si = i >> kGroup, j = i & ((1 << kGroup) - 1);
    const Step s = tab.step[si];
    if (j >= (1 << s.G)) continue;
    float2 l = make_float2(1.f, 0.f), r = make_float2(1.f, 0.f);
    uint32_t flip = 0;
    if (form & kBatchShear)
      for (int b = 0; b < s.G; ++b) {
        const float2* rec = gates + size_t(kBatchGateSlots) * (size_t(s.layer) * n + s.q + b);
        const int bit = (j >> b) & 1, off = rec[1].x != 0.f ? 1 : 0;
        flip |= uint32_t(off) << b;
        l = cmul(l, rec[2 + bit]);
        r = cmul(r, rec[4 + (bit ^ off)]);
      }
    if (j == 0) tab.step[si].flip = flip;
    float2 l1 = l;
    if (entangler == QVDG_ENTANGLE_CZ_LADDER) {
      if (__popc(j & (j >> 1)) & 1) l = make_float2(-l.x, -l.y);
      l1 = (j & 1) ? make_float2(-l.x, -l.y) : l;
    }
    tab.left[si][0][j] = l;
    tab.left[si][1][j] = l1;
    tab.right[si][j] = r;
  }
}

// Sums over the tile of |a|^2 (out[0]) and of |a|^2 where local bit b is set
// (out[1 + b]), valid in every thread after the call. Thread i visits
// elements i, i + T, i + 2T, ...: the local bits below log2(T) are fixed per
// thread and the others vary.
__device__ void reduce_tile(const unsigned char* tile, int nb, double* red, double* out) {
  double v[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) v[i] = 0.0;
  const uint32_t count = 1u << nb;
  const int tbits = 31 - __clz(blockDim.x);
  for (uint32_t e = threadIdx.x; e < count; e += blockDim.x) {
    const float2 a = *reinterpret_cast<const float2*>(tile + swz(e) * 8u);
    const double p = __dadd_rn(__dmul_rn(double(a.x), double(a.x)), __dmul_rn(double(a.y), double(a.y)));
    v[0] += p;
#pragma unroll
    for (int bit = 7; bit < kVec - 1; ++bit)  // tbits >= 7
      if (bit >= tbits && bit < nb && ((e >> bit) & 1u)) v[1 + bit] += p;
  }
#pragma unroll
  for (int bit = 0; bit < kVec - 1; ++bit)
    if (bit < tbits && bit < nb && ((threadIdx.x >> bit) & 1u)) v[1 + bit] = v[0];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    double x = v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp * kVec + i] = x;
  }
  __syncthreads();
  if (threadIdx.x < kVec) {
    double t = 0.0;
    for (int w = 0; w < warps; ++w) t += red[w * kVec + threadIdx.x];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// The first 2^bits elements of a tile copied in asynchronously, 16 bytes at
// a time (element pairs are adjacent in the slot because every tile keeps
// index bit 0, and one aligned place in shared memory because swz keeps it).
__device__ void issue_tile(unsigned char* tile, const float2* __restrict__ slot, const TileMap& map, int bits) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(tile));
  for (uint32_t u = threadIdx.x; u < (1u << (bits - 1)); u += blockDim.x)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + swz(2 * u) * 8u), "l"(slot + map.global(2 * u))
                 : "memory");
}

__device__ void store_tile(const unsigned char* tile, float2* __restrict__ slot, const TileMap& map, int nb) {
  for (uint32_t u = threadIdx.x; u < (1u << (nb - 1)); u += blockDim.x)
    __stcg(reinterpret_cast<float4*>(slot + map.global(2 * u)),
           *reinterpret_cast<const float4*>(tile + swz(2 * u) * 8u));
}

// Waits until `*count` has reached `need` (thread 0, then the CTA). False
// when the launch has been given up.
__device__ bool wait_for(const uint32_t* count, uint32_t need, int* status, volatile int* ok) {
  if (threadIdx.x == 0) {
    int good = 1;
    const long long t0 = clock64();
    for (;;) {
      uint32_t have;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(have) : "l"(count) : "memory");
      if (have >= need) break;
      if (*reinterpret_cast<volatile int*>(status)) {
        good = 0;
        break;
      }
      if (clock64() - t0 > kTaskWaitCycles) {
        atomicExch(status, 1);
        good = 0;
        break;
      }
      __nanosleep(200);
    }
    *ok = good;
  }
  __syncthreads();
  const bool good = *ok != 0;
  __syncthreads();  // `ok` may be written again
  return good;
}

// Counts `n` tiles of the CTA's circuit done, after every thread's stores.
__device__ void count_done(uint32_t* count, uint32_t n) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, n);
  }
}

template <int kThreadsPer, int kMinBlocks>
__global__ void __launch_bounds__(kThreadsPer, kMinBlocks) k_batch(const BatchLaunch p) {
  extern __shared__ __align__(16) unsigned char tiles[];
  __shared__ Tables tab;
  __shared__ double red[(kThreadsPer / 32) * kVec];
  __shared__ double sums[kVec];
  __shared__ uint32_t item;
  __shared__ int ok;
  __shared__ int steps;
  const int L = p.tile_qubits;
  const uint32_t tiles_s = static_cast<uint32_t>(__cvta_generic_to_shared(tiles));
  for (;;) {
    if (threadIdx.x == 0) item = *reinterpret_cast<volatile int*>(p.status) ? p.count : atomicAdd(p.queue, 1u);
    __syncthreads();
    const uint32_t it = item;
    if (it >= p.count) break;
    const BatchTask task = p.tasks[it];
    const BatchCircuit c = p.circuits[task.circuit];
    const int n = int(c.num_qubits), entangler = int(c.entangler);
    const float2* gates = p.gates + size_t(kBatchGateSlots) * c.gates;
    if (n <= L) {
      // Whole state in shared memory, as many layers as the tables hold at
      // a time.
      const uint32_t size = 1u << n;
      for (uint32_t e = threadIdx.x; e < size; e += blockDim.x)
        *reinterpret_cast<float2*>(tiles + swz(e) * 8u) = make_float2(e == 0 ? 1.f : 0.f, 0.f);
      const TileMap map = low_map(n, 0);
      const uint32_t chunk = uint32_t(kMaxSteps / ((n + kGroup - 1) / kGroup));
      for (uint32_t l0 = 0; l0 < c.num_layers; l0 += chunk) {
        __syncthreads();
        if (threadIdx.x == 0) {
          steps = 0;
          int count = 0;
          for (uint32_t l = l0; l < c.num_layers && l < l0 + chunk; ++l) add_steps(tab, count, l, 0, n, 0);
          steps = count;
        }
        __syncthreads();
        build_tables(tab, steps, gates, n, c.form, entangler);
        __syncthreads();
        for (int si = 0; si < steps; ++si) {
          run_step(tiles_s, n, tab, si, c.form, entangler, map);
          __syncthreads();
        }
      }
      __syncthreads();
      reduce_tile(tiles, n, red, sums);
      if (threadIdx.x < uint32_t(n)) p.out[c.out + threadIdx.x] = sums[0] - 2.0 * sums[1 + threadIdx.x];
      __syncthreads();
      continue;
    }
    const BatchWide w = p.wide[c.wide];
    const int Lw = w.tile_bits, h0 = w.high, r = w.low;
    const uint32_t phases = w.phases;
    uint32_t* done = p.done + c.wide;
    double* partials = p.partials + w.partials;
    if (task.phase == phases) {
      // Every tile of the last pass has written its sums: <Z> of qubit q
      // from the tiles' sums over it, local bit or tile-number bit.
      if (!wait_for(done, w.before(task.phase), p.status, &ok)) break;
      for (int q = int(threadIdx.x >> 5); q < n; q += int(blockDim.x >> 5)) {
        const int lane = threadIdx.x & 31;
        const int local = q < r ? q : (q >= h0 ? q - h0 + r : -1);
        double total = 0.0, one = 0.0;
        for (uint32_t t = lane; t < w.tiles; t += 32) {
          const double s = __ldcg(partials + size_t(t) * kVec);
          total += s;
          if (local >= 0)
            one += __ldcg(partials + size_t(t) * kVec + 1 + local);
          else if ((t >> (q - r)) & 1u)
            one += s;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          total += __shfl_down_sync(0xffffffffu, total, o);
          one += __shfl_down_sync(0xffffffffu, one, o);
        }
        // A circuit without layers is |0...0>: no pass has summed it.
        if (lane == 0) p.out[c.out + q] = phases ? total - 2.0 * one : 1.0;
      }
      count_done(done, 1);
      __syncthreads();
      continue;
    }
    const bool high = task.phase & 1;
    const uint32_t super = task.phase / 2, l0 = super * w.layers;
    const uint32_t depth = min(w.layers, c.num_layers - l0);
    const bool last = task.phase + 1 == phases;
    if (threadIdx.x == 0) {
      int count = 0;
      for (uint32_t j = 0; j < depth; ++j) {
        if (high)
          add_steps(tab, count, l0 + j, Lw - int(j), n, Lw - int(j) - h0 + r);
        else
          add_steps(tab, count, l0 + j, 0, Lw - int(j), 0);
      }
      steps = count;
    }
    __syncthreads();
    build_tables(tab, steps, gates, n, c.form, entangler);
    // The first pass of a circuit takes its slot over from an earlier one.
    bool go = task.phase > 0 || w.previous < 0 ||
              wait_for(p.done + w.previous, p.wide[w.previous].before(p.wide[w.previous].phases) + 1, p.status, &ok);
    if (go && task.phase > 0) go = wait_for(done, w.before(task.phase), p.status, &ok);
    if (!go) break;
    float2* slot = p.slots + w.slot;
    // From |0...0> only tile 0 of the first A pass is not zero: it is all
    // that pass runs, and the first B pass reads only from it.
    const int bits = task.phase == 1 ? r + Lw - h0 : Lw;
    const uint32_t size = 1u << Lw;
    auto map_of = [&](uint32_t t) { return high ? TileMap{r, h0, t} : low_map(Lw, t); };
    auto fetch = [&](unsigned char* buf, uint32_t t) {
      if (task.phase == 0) {
        for (uint32_t e = threadIdx.x; e < size; e += blockDim.x)
          *reinterpret_cast<float2*>(buf + swz(e) * 8u) = make_float2(e == 0 ? 1.f : 0.f, 0.f);
      } else {
        issue_tile(buf, slot, map_of(t), bits);
        for (uint32_t e = (1u << bits) + threadIdx.x; e < size; e += blockDim.x)
          *reinterpret_cast<float2*>(buf + swz(e) * 8u) = make_float2(0.f, 0.f);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // Two buffers where the shared tile holds two of the pass's tiles: the
    // next one's copies fly while the current one is computed. Otherwise
    // other CTAs of the SM cover them.
    const bool two = (1u << L) >= 2 * size;
    unsigned char* buf[2] = {tiles, two ? tiles + size * 8u : tiles};
    const uint32_t t0 = task.tile, t1 = task.tile + task.count;
    fetch(buf[0], t0);
    for (uint32_t t = t0; t < t1; ++t) {
      const uint32_t k = (t - t0) & 1u;
      const bool ahead = two && t + 1 < t1;
      if (ahead) {
        fetch(buf[k ^ 1], t + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      const TileMap map = map_of(t);
      unsigned char* cur = buf[two ? k : 0];
      for (int si = 0; si < steps; ++si) {
        run_step(tiles_s + uint32_t(cur - tiles), Lw, tab, si, c.form, entangler, map);
        __syncthreads();
      }
      if (last) {
        reduce_tile(cur, Lw, red, sums);
        if (threadIdx.x < kVec) __stcg(partials + size_t(t) * kVec + threadIdx.x, sums[threadIdx.x]);
      } else {
        store_tile(cur, slot, map, Lw);
      }
      __syncthreads();
      if (!two && t + 1 < t1) fetch(cur, t + 1);
    }
    count_done(done, t1 - t0);
    __syncthreads();
  }
}

// ---- Gate records from 2x2 complex128 matrices

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double zabs(double2 a) { return hypot(a.x, a.y); }
__device__ __forceinline__ double2 zunit(double2 a) {
  const double m = zabs(a);
  return make_double2(a.x / m, a.y / m);
}
// a / b for a unit b.
__device__ __forceinline__ double2 zover(double2 a, double2 b) { return zmul(a, make_double2(b.x, -b.y)); }

// U = diag(p0, p1) R diag(q0, q1) with R real and unit p, q: rows with one
// common phase (q = 1) or columns with one (p = 1) when possible, otherwise
// p0 = 1 and the rest from U's entries (all four nonzero for a unitary that
// is neither diagonal nor anti-diagonal). Each row of R is then divided by
// its diagonal entries (or, for both rows, its off-diagonal ones) where
// those are the larger, which go into p. False when U has no such form.
__device__ bool shear_form(const double2* u, float2* rec, bool& right) {
  const double tol = 1e-9;
  const double2 one = make_double2(1.0, 0.0);
  double r[4];
  double2 p[2] = {one, one}, q[2] = {one, one};
  auto real_of = [&](double2 c, double& out) {
    out = c.x;
    return fabs(c.y) <= tol;
  };
  auto rows = [&]() {
    for (int i = 0; i < 2; ++i) {
      const int k = zabs(u[2 * i]) >= zabs(u[2 * i + 1]) ? 0 : 1;
      if (zabs(u[2 * i + k]) == 0.0) return false;
      p[i] = zunit(u[2 * i + k]);
      if (!real_of(zover(u[2 * i], p[i]), r[2 * i]) || !real_of(zover(u[2 * i + 1], p[i]), r[2 * i + 1])) return false;
    }
    q[0] = q[1] = one;
    return true;
  };
  auto cols = [&]() {
    for (int j = 0; j < 2; ++j) {
      const int k = zabs(u[j]) >= zabs(u[2 + j]) ? 0 : 1;
      if (zabs(u[2 * k + j]) == 0.0) return false;
      q[j] = zunit(u[2 * k + j]);
      if (!real_of(zover(u[j], q[j]), r[j]) || !real_of(zover(u[2 + j], q[j]), r[2 + j])) return false;
    }
    p[0] = p[1] = one;
    return true;
  };
  auto general = [&]() {
    for (int i = 0; i < 4; ++i)
      if (zabs(u[i]) == 0.0) return false;
    p[0] = one;
    q[0] = zunit(u[0]);
    q[1] = zunit(u[1]);
    p[1] = zunit(zover(u[2], q[0]));
    for (int i = 0; i < 2; ++i)
      for (int j = 0; j < 2; ++j)
        if (!real_of(zover(u[2 * i + j], zmul(p[i], q[j])), r[2 * i + j])) return false;
    return true;
  };
  if (!rows() && !cols() && !general()) return false;
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) {
      const double2 v = zmul(p[i], q[j]);
      if (!(hypot(v.x * r[2 * i + j] - u[2 * i + j].x, v.y * r[2 * i + j] - u[2 * i + j].y) <= tol)) return false;
    }
  const bool diag = fabs(r[0]) >= fabs(r[1]) && fabs(r[3]) >= fabs(r[2]);
  const bool off = fabs(r[1]) >= fabs(r[0]) && fabs(r[2]) >= fabs(r[3]);
  const double s0 = diag ? r[0] : r[1], s1 = diag ? r[3] : r[2];
  if (!(diag || off) || s0 == 0.0 || s1 == 0.0) return false;
  rec[0] = make_float2(float((diag ? r[1] : r[0]) / s0), float((diag ? r[2] : r[3]) / s1));
  rec[1] = make_float2(diag ? 0.f : 1.f, 0.f);
  rec[2] = make_float2(float(p[0].x * s0), float(p[0].y * s0));
  rec[3] = make_float2(float(p[1].x * s1), float(p[1].y * s1));
  rec[4] = make_float2(float(q[0].x), float(q[0].y));
  rec[5] = make_float2(float(q[1].x), float(q[1].y));
  right = q[0].x != 1.0 || q[0].y != 0.0 || q[1].x != 1.0 || q[1].y != 0.0;
  return true;
}

// One block per circuit: its records and form, sheared when every matrix has
// that form, else the generic matrices.
__global__ void __launch_bounds__(128) k_batch_encode(BatchCircuit* __restrict__ circuits,
                                                      const double2* __restrict__ matrices,
                                                      float2* __restrict__ gates) {
  BatchCircuit& c = circuits[blockIdx.x];
  const uint32_t count = c.num_layers * c.num_qubits;
  const double2* m = matrices + 4 * c.gates;
  float2* rec = gates + size_t(kBatchGateSlots) * c.gates;
  bool shear = true, right = false;
  for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
    bool r = false;
    double2 u[4];
    for (int k = 0; k < 4; ++k) u[k] = m[4 * size_t(i) + k];
    shear = shear && shear_form(u, rec + size_t(kBatchGateSlots) * i, r);
    right = right || r;
  }
  const bool all = __syncthreads_and(shear), any = __syncthreads_or(right);
  if (!all)
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x)
      for (int k = 0; k < 4; ++k)
        rec[size_t(kBatchGateSlots) * i + k] = make_float2(float(m[4 * size_t(i) + k].x), float(m[4 * size_t(i) + k].y));
  if (threadIdx.x == 0) c.form = all ? kBatchShear | (any ? kBatchRight : 0u) : 0u;
}

template <int T, int B>
int occupancy_of(size_t smem) {
  int blocks = 0;
  // Allow the largest tile once, so that launches (also under stream
  // capture) need no attribute change.
  if (cudaFuncSetAttribute(k_batch<T, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(float2) << 14)) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_batch<T, B>, cudaFuncAttributePreferredSharedMemoryCarveout,
                           int(cudaSharedmemCarveoutMaxShared)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_batch<T, B>, T, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return blocks;
}

}  // namespace

int batch_kernel_occupancy(int threads, int tile_qubits) {
  const size_t smem = sizeof(float2) << tile_qubits;
  switch (threads) {
    case 128: return occupancy_of<128, 4>(smem);
    case 256: return occupancy_of<256, 3>(smem);
    default: return occupancy_of<512, 1>(smem);
  }
}

void launch_batch_encode(const BatchLaunch& b, const double* matrices, uint32_t circuits, cudaStream_t stream) {
  k_batch_encode<<<circuits, 128, 0, stream>>>(const_cast<BatchCircuit*>(b.circuits),
                                               reinterpret_cast<const double2*>(matrices),
                                               const_cast<float2*>(b.gates));
  QVDG_LAUNCH_CHECK();
}

void launch_batch(const BatchLaunch& b, cudaStream_t stream) {
  const size_t smem = sizeof(float2) << b.tile_qubits;
  QVDG_CUDA(cudaMemsetAsync(b.queue, 0, b.queue_bytes, stream));
  switch (b.threads) {
    case 128: k_batch<128, 4><<<b.ctas, 128, smem, stream>>>(b); break;
    case 256: k_batch<256, 3><<<b.ctas, 256, smem, stream>>>(b); break;
    default: k_batch<512, 1><<<b.ctas, 512, smem, stream>>>(b); break;
  }
  QVDG_LAUNCH_CHECK();
}

}  // namespace qvdg
