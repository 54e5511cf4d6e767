// Plain-path gate kernels: one pass over the state per fused gate.
//
// These replace the reference's AVX2 sweeps (src/kernels.rs:252-473). The
// state is interleaved complex in physical index order; a gate on physical
// target bits t_0..t_{k-1} with controls acts on groups of 2^k amplitudes
// whose index differs only in the target bits and whose control bits hold.
// Group bases are enumerated by inserting zero bits at the (sorted) target
// and control positions of a running counter, so a controlled gate touches
// only the 2^-c of the state its controls select (the reference's
// `free_mask`/`control_value`, src/kernels.rs:78-135). Consecutive threads
// take consecutive bases: when bit 0 is free, a warp's loads of each group
// member are one contiguous 256-byte (complex64) or 512-byte (complex128)
// run, and complex64 threads take two neighbouring groups with one 16-byte
// load per member.

#include <cuda_runtime.h>

#include <algorithm>

#include "dense_wide.hpp"
#include "engine.hpp"

namespace qvdg {

namespace {

constexpr int kThreads = 256;

// A gate's matrix as a kernel gets it: on the device, or in the launch's own
// parameters. A single gate on a small state is mostly latency (17 qubits
// complex128: 30 us a call), and the copy ahead of the kernel took 2-3 us of
// it: 40 gates of 1-6 qubits 1.22 -> 1.16 ms. At most 1 KB; a 4-qubit matrix
// of complex128 would fill the 4 KB that every launch can carry.
template <typename T>
struct MatDevice {
  const cplx_t<T>* p;
  __device__ const cplx_t<T>& operator[](int i) const { return p[i]; }
};
template <typename T, int N>
struct MatInline {
  cplx_t<T> v[N];
  __device__ const cplx_t<T>& operator[](int i) const { return v[i]; }
};
template <typename T, int N>
MatInline<T, N> mat_inline(const double* host, int count) {
  MatInline<T, N> m{};
  for (int i = 0; i < count; ++i) m.v[i] = make_c<T>(T(host[2 * i]), T(host[2 * i + 1]));
  return m;
}
constexpr int kInlineDense = 3;     // qubits of a dense gate that goes inline
constexpr int kInlineDiagonal = 6;  // and of a diagonal one

struct DenseGeom {
  uint64_t n_iter;         // number of groups
  uint64_t control_value;  // control bits that must be 1
  uint64_t offsets[64];    // index offset of each group member (matrix index order)
  uint8_t fixed[40];       // sorted target and control positions
  int32_t num_fixed;
};

// Threads of a k_dense block and the rows it computes at a time. From four
// qubits on the multiply-adds count as much as HBM (six: 1.9 ms of them at
// full rate for 28 qubits of complex64, 0.66 ms of HBM), and one whose three
// operands are all new registers runs at two thirds of the rate. Two rows
// (four for K = 4) at a time share each amplitude, two groups share each
// matrix entry, and complex64 reads two entries at once; small blocks leave
// the wide gates' registers three of them per SM. 28 qubits complex64: K = 4
// 0.83-0.92 -> 0.82 ms, K = 5 1.70-1.85 -> 1.36, K = 6 3.28 -> 2.87.
template <typename T, int K>
constexpr int kDenseThreads = sizeof(T) == 4 && K >= 5 ? 128 : kThreads;
template <typename T, int K>
constexpr int kDenseRows = sizeof(T) == 4 ? (K == 4 ? 4 : 2) : 1;

template <typename T, int K, int G, bool VEC, typename M>
__global__ void __launch_bounds__(kDenseThreads<T, K>, sizeof(T) == 4 && K >= 5 ? 3 : 1)
    k_dense(cplx_t<T>* __restrict__ psi, const __grid_constant__ DenseGeom g, const __grid_constant__ M mat) {
  constexpr int D = 1 << K, ROWS = kDenseRows<T, K>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx_t<T>* sm = reinterpret_cast<cplx_t<T>*>(smem_raw);
  __shared__ uint8_t fixed[40];
  for (int i = threadIdx.x; i < D * D; i += blockDim.x) sm[i] = mat[i];
  if (threadIdx.x < 40) fixed[threadIdx.x] = g.fixed[threadIdx.x];
  __syncthreads();
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x * G;
  for (uint64_t it = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * G; it < g.n_iter; it += stride) {
    uint64_t base[G];
#pragma unroll
    for (int q = 0; q < G; ++q) base[q] = insert_zeros(it + q, fixed, g.num_fixed) | g.control_value;
    cplx_t<T> x[G][D];
    if constexpr (VEC) {
      // complex64 with bit 0 free: groups it and it+1 are neighbours.
#pragma unroll
      for (int h = 0; h < D; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(psi + base[0] + g.offsets[h]);
        x[0][h] = make_c<T>(v.x, v.y);
        x[G - 1][h] = make_c<T>(v.z, v.w);
      }
    } else {
#pragma unroll
      for (int h = 0; h < D; ++h)
#pragma unroll
        for (int q = 0; q < G; ++q) x[q][h] = psi[base[q] + g.offsets[h]];
    }
#pragma unroll 1
    for (int r = 0; r < D; r += ROWS) {
      cplx_t<T> acc[ROWS][G];
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int q = 0; q < G; ++q) acc[i][q] = make_c<T>(T(0), T(0));
      if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int c = 0; c < D; c += 2) {
          float4 m[ROWS];
#pragma unroll
          for (int i = 0; i < ROWS; ++i) m[i] = *reinterpret_cast<const float4*>(sm + (r + i) * D + c);
#pragma unroll
          for (int q = 0; q < G; ++q) {
#pragma unroll
            for (int i = 0; i < ROWS; ++i) cmac<T>(acc[i][q], make_float2(m[i].x, m[i].y), x[q][c]);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) cmac<T>(acc[i][q], make_float2(m[i].z, m[i].w), x[q][c + 1]);
          }
        }
      } else {
#pragma unroll
        for (int c = 0; c < D; ++c) {
          const cplx_t<T> m = sm[r * D + c];
#pragma unroll
          for (int q = 0; q < G; ++q) cmac<T>(acc[0][q], m, x[q][c]);
        }
      }
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        if constexpr (VEC) {
          *reinterpret_cast<float4*>(psi + base[0] + g.offsets[r + i]) =
              make_float4(acc[i][0].x, acc[i][0].y, acc[i][G - 1].x, acc[i][G - 1].y);
        } else {
#pragma unroll
          for (int q = 0; q < G; ++q) psi[base[q] + g.offsets[r + i]] = acc[i][q];
        }
      }
    }
  }
}

// Dense gates whose targets all lie in index bits 0-4 (the lane bits of a
// warp row of 32 consecutive amplitudes), with controls above them: the
// GPU form of the reference's in-register lane permutations for targets
// inside a SIMD vector (src/kernels.rs:185, 273, xor_perm). A warp takes
// whole rows, lane l holding amplitude l of the row (one coalesced 256- or
// 512-byte access); the other members of its group are in the lanes whose
// target bits differ, and come over by warp shuffles. Lane l computes its
// own output, row r(l) of the gate (r = its target bits in matrix order),
// held in registers, so neither shared memory nor a second pass over the
// row is needed. Each thread keeps R rows in flight.
struct LaneGeom {
  uint64_t rows;           // warp rows of 32 amplitudes the controls select
  uint64_t control_value;  // control bits that must be 1
  uint8_t fixed[40];       // the control positions in the row's number, ascending
  int32_t num_fixed;
  uint8_t targets[4];      // target positions (matrix bit order), all below 5
};

template <typename T, int K, int R, typename M>
__global__ void __launch_bounds__(kThreads) k_dense_lanes(cplx_t<T>* __restrict__ psi,
                                                          const __grid_constant__ LaneGeom g,
                                                          const __grid_constant__ M mat) {
  constexpr int D = 1 << K;
  __shared__ uint8_t fixed[40];
  if (threadIdx.x < 40) fixed[threadIdx.x] = g.fixed[threadIdx.x];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t tmask = 0, row = 0;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    tmask |= 1u << g.targets[j];
    row |= ((lane >> g.targets[j]) & 1u) << j;
  }
  cplx_t<T> m[D];
  int src[D];
#pragma unroll
  for (int c = 0; c < D; ++c) {
    m[c] = mat[row * D + c];
    uint32_t p = lane & ~tmask;
#pragma unroll
    for (int j = 0; j < K; ++j) p |= uint32_t((c >> j) & 1) << g.targets[j];
    src[c] = int(p);
  }
  const uint64_t warps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  const uint64_t first = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  for (uint64_t w0 = first * R; w0 < g.rows; w0 += warps * R) {
    uint64_t base[R];
    cplx_t<T> x[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      base[q] = w0 + q < g.rows ? ((insert_zeros(w0 + q, fixed, g.num_fixed) << 5) | g.control_value) + lane : ~uint64_t(0);
      if (base[q] != ~uint64_t(0)) x[q] = psi[base[q]];
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      cplx_t<T> acc = make_c<T>(T(0), T(0));
#pragma unroll
      for (int c = 0; c < D; ++c) {
        cplx_t<T> y;
        y.x = __shfl_sync(0xffffffffu, x[q].x, src[c]);
        y.y = __shfl_sync(0xffffffffu, x[q].y, src[c]);
        cmac<T>(acc, m[c], y);
      }
      if (base[q] != ~uint64_t(0)) psi[base[q]] = acc;
    }
  }
}

// Dense gates with targets among the low index bits: each thread's group is
// then a short contiguous run and a warp's loads stride by the run length.
// Instead, a block stages a tile of 2^13 amplitudes -- index bits 0..Lb-1
// (contiguous runs of 2^Lb) plus the targets above them -- in shared memory
// with coalesced 16-byte accesses, applies the gate to the tile's 2^(13-K)
// groups there (two per thread, so each matrix entry read serves both) and
// stores the tile back.
constexpr int kTileBits = 13;

struct DenseTileGeom {
  uint64_t tiles;
  int32_t lb;             // contiguous low bits of the tile
  int32_t nhigh;          // targets at or above lb
  uint8_t high[8];        // physical positions of those targets (ascending)
  uint8_t fixed_tile[8];  // tile-local positions of all targets (ascending)
  uint16_t offsets[64];   // tile-local offset of group member h (matrix index order)
};

// Shared-memory position of tile element e (bits 4-7 folded into 1-3; bit 0
// kept so 16-byte element pairs stay together).
__device__ __forceinline__ uint32_t dswz(uint32_t e) { return e ^ ((e >> 4) & 14u); }

template <int K>
__global__ void __launch_bounds__(kThreads) k_dense_tile(float2* __restrict__ psi, const DenseTileGeom g,
                                                         const float2* __restrict__ mat) {
  constexpr int D = 1 << K;
  constexpr uint32_t kTile = 1u << kTileBits;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tile = reinterpret_cast<float2*>(smem_raw);
  float2* sm = tile + kTile;
  __shared__ uint8_t fixed[8];
  __shared__ uint16_t off[64];
  for (int i = threadIdx.x; i < D * D; i += blockDim.x) sm[i] = mat[i];
  if (threadIdx.x < 8) fixed[threadIdx.x] = g.fixed_tile[threadIdx.x];
  if (threadIdx.x < 64) off[threadIdx.x] = g.offsets[threadIdx.x];
  __syncthreads();
  const uint32_t lowmask = (1u << g.lb) - 1u;
  for (uint64_t t = blockIdx.x; t < g.tiles; t += gridDim.x) {
    // Tile t: its bits above lb, with zeros at the high targets, give the
    // base index; element e adds its low bits and the high targets.
    uint64_t base = t << g.lb;
    for (int i = 0; i < g.nhigh; ++i) {
      const uint32_t p = g.high[i];
      base = ((base >> p) << (p + 1)) | (base & ((uint64_t(1) << p) - 1));
    }
    auto global_of = [&](uint32_t e) -> uint64_t {
      uint64_t x = base | (e & lowmask);
      uint32_t h = e >> g.lb;
      for (int i = 0; i < g.nhigh; ++i) x |= uint64_t((h >> i) & 1u) << g.high[i];
      return x;
    };
    // Every 16-byte copy of the tile in flight at once (cp.async).
    for (uint32_t u = threadIdx.x; u < kTile / 2; u += blockDim.x) {
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(tile + dswz(2 * u)));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(psi + global_of(2 * u)) : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    constexpr uint32_t kGroups = kTile >> K;
    for (uint32_t q = threadIdx.x; q < kGroups / 2; q += blockDim.x) {
      uint32_t b[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        uint32_t x = q + s * (kGroups / 2);
#pragma unroll
        for (int i = 0; i < K; ++i) {
          const uint32_t p = fixed[i];
          x = ((x >> p) << (p + 1)) | (x & ((1u << p) - 1u));
        }
        b[s] = x;
      }
      float2 x[2][D];
#pragma unroll
      for (int h = 0; h < D; ++h) {
        x[0][h] = tile[dswz(b[0] | off[h])];
        x[1][h] = tile[dswz(b[1] | off[h])];
      }
#pragma unroll 1
      for (int r = 0; r < D; ++r) {
        float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < D; c += 2) {
          const float4 m = *reinterpret_cast<const float4*>(sm + r * D + c);
          const float2 m0 = make_float2(m.x, m.y), m1 = make_float2(m.z, m.w);
          cmac<float>(a0, m0, x[0][c]);
          cmac<float>(a1, m0, x[1][c]);
          cmac<float>(a0, m1, x[0][c + 1]);
          cmac<float>(a1, m1, x[1][c + 1]);
        }
        tile[dswz(b[0] | off[r])] = a0;
        tile[dswz(b[1] | off[r])] = a1;
      }
    }
    __syncthreads();
    for (uint32_t u = threadIdx.x; u < kTile / 2; u += blockDim.x)
      *reinterpret_cast<float4*>(psi + global_of(2 * u)) = *reinterpret_cast<const float4*>(tile + dswz(2 * u));
    __syncthreads();
  }
}

struct DiagGeom {
  uint64_t n_iter;         // amplitudes in the controlled subspace
  uint64_t control_value;
  uint8_t ctrl[40];        // sorted control positions
  int32_t num_ctrl;
  uint8_t targets[16];     // diagonal index bit j = targets[j]
  int32_t k;
};

template <typename T, int G, typename M>
__global__ void __launch_bounds__(kThreads) k_diag(cplx_t<T>* __restrict__ psi, const __grid_constant__ DiagGeom g,
                                                   const __grid_constant__ M diag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx_t<T>* sm = reinterpret_cast<cplx_t<T>*>(smem_raw);
  __shared__ uint8_t ctrl[40], tgt[16];
  for (int i = threadIdx.x; i < (1 << g.k); i += blockDim.x) sm[i] = diag[i];
  if (threadIdx.x < 40) ctrl[threadIdx.x] = g.ctrl[threadIdx.x];
  if (threadIdx.x < 16) tgt[threadIdx.x] = g.targets[threadIdx.x];
  __syncthreads();
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x * G;
  for (uint64_t it = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * G; it < g.n_iter; it += stride) {
    // With G == 2, bit 0 is not a control: indices i and i+1 are neighbours.
    const uint64_t i = insert_zeros(it, ctrl, g.num_ctrl) | g.control_value;
    uint32_t d[G];
#pragma unroll
    for (int q = 0; q < G; ++q) {
      d[q] = 0;
      for (int j = 0; j < g.k; ++j) d[q] |= uint32_t(((i + q) >> tgt[j]) & 1) << j;
    }
    if constexpr (G == 2 && sizeof(T) == 4) {
      float4 v = *reinterpret_cast<float4*>(psi + i);
      const cplx_t<T> a = cmul<T>(sm[d[0]], make_c<T>(v.x, v.y));
      const cplx_t<T> b = cmul<T>(sm[d[1]], make_c<T>(v.z, v.w));
      *reinterpret_cast<float4*>(psi + i) = make_float4(a.x, a.y, b.x, b.y);
    } else {
#pragma unroll
      for (int q = 0; q < G; ++q) psi[i + q] = cmul<T>(sm[d[q]], psi[i + q]);
    }
  }
}

// Several diagonal gates in one pass, each amplitude multiplied by their
// factors in order (the same products and roundings as one pass per gate).
// HBM bounds a diagonal pass, so gates that share one cost little more than
// one of them, as long as finding each gate's factor stays cheap: the bits
// of an amplitude's index that a gate reads are gathered into its table
// index by parts, from the thread's low bits (once), from the vector's place
// in the block's tile (constants) and from the tile's number (through byte
// tables in shared memory), each part holding all eight gates' indices as
// 16-bit fields of one 16-byte word. A thread moves 16-byte vectors, four
// in flight. 28-qubit QFT of a general state: 27 diagonal passes of 0.79 ms
// become 9, three alone and six of 0.75-1.15 ms, 31.7 -> 16.5 ms in all.
constexpr int kRunUnroll = 4;
constexpr int kRunTileBits = 10;  // vectors of a block's tile: kThreads * kRunUnroll

__device__ __forceinline__ uint4 or4(const uint4& a, const uint4& b) {
  return make_uint4(a.x | b.x, a.y | b.y, a.z | b.z, a.w | b.w);
}
__device__ __forceinline__ uint32_t field16(const uint4& v, int o) {
  const uint32_t w = o < 2 ? v.x : (o < 4 ? v.y : (o < 6 ? v.z : v.w));
  return (o & 1) ? w >> 16 : w & 0xffffu;
}

// All gates' table indices that the set bits of `x`, standing `shift` bits
// up in an amplitude's index, give.
__device__ __forceinline__ uint4 run_index(const DiagRun& g, uint64_t x, int shift) {
  uint32_t w[4] = {0, 0, 0, 0};
  const uint64_t i = x << shift;
#pragma unroll
  for (int o = 0; o < kDiagRunGates; ++o) {
    if (o >= g.count) break;
    uint32_t d = 0;
    for (int j = 0; j < g.k[o]; ++j) d |= uint32_t((i >> g.targets[o][j]) & 1u) << j;
    w[o >> 1] |= d << (16 * (o & 1));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_diag_run(cplx_t<T>* __restrict__ psi, uint64_t vectors, int pieces,
                                                       const __grid_constant__ DiagRun g,
                                                       const cplx_t<T>* __restrict__ mats) {
  constexpr int V = sizeof(T) == 4 ? 2 : 1;       // amplitudes of a vector
  constexpr int kLow = sizeof(T) == 4 ? 1 : 0;    // index bits inside one
  constexpr int kTile = kLow + kRunTileBits;      // index bits inside a tile
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx_t<T>* tables = reinterpret_cast<cplx_t<T>*>(smem_raw);
  uint4* high = reinterpret_cast<uint4*>(smem_raw + ((size_t(g.entries) * sizeof(cplx_t<T>) + 15) & ~size_t(15)));
  for (int o = 0; o < g.count; ++o)
    for (int i = threadIdx.x; i < (1 << g.k[o]); i += kThreads) tables[g.table[o] + i] = mats[g.matrix[o] + i];
  for (int p = 0; p < pieces; ++p) high[p * 256 + threadIdx.x] = run_index(g, threadIdx.x, kTile + 8 * p);
  const uint4 low = run_index(g, threadIdx.x, kLow);
  uint4 place[kRunUnroll];
#pragma unroll
  for (int u = 0; u < kRunUnroll; ++u) place[u] = run_index(g, uint64_t(u), kLow + 8);
  uint4 odd = make_uint4(0, 0, 0, 0);  // index bit 0 (complex64: the vector's second amplitude)
  if constexpr (V == 2) odd = run_index(g, 1, 0);
  __syncthreads();
  const uint64_t tiles = (vectors + (1u << kRunTileBits) - 1) >> kRunTileBits;
  for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint64_t v0 = (t << kRunTileBits) + threadIdx.x;
    float4 raw[kRunUnroll];
#pragma unroll
    for (int u = 0; u < kRunUnroll; ++u)
      if (v0 + u * kThreads < vectors) raw[u] = reinterpret_cast<const float4*>(psi)[v0 + u * kThreads];
    uint4 base = low;
    for (int p = 0; p < pieces; ++p) base = or4(base, high[p * 256 + ((t >> (8 * p)) & 255)]);
#pragma unroll
    for (int u = 0; u < kRunUnroll; ++u) {
      const uint64_t v = v0 + u * kThreads;
      if (v >= vectors) break;
      const uint4 index = or4(base, place[u]);
      cplx_t<T> a[V];
      if constexpr (V == 2) {
        a[0] = make_float2(raw[u].x, raw[u].y);
        a[V - 1] = make_float2(raw[u].z, raw[u].w);
      } else {
        a[0] = *reinterpret_cast<const cplx_t<T>*>(&raw[u]);
      }
#pragma unroll
      for (int o = 0; o < kDiagRunGates; ++o) {
        if (o >= g.count) break;
        const uint32_t d = field16(index, o), second = V == 2 ? field16(odd, o) : 0u;
        const cplx_t<T>* table = tables + g.table[o];
        const cplx_t<T> f0 = table[d];
        cplx_t<T> f1 = f0;
        if (V == 2 && second) f1 = table[d | second];
        if (g.control_mask[o]) {
          const uint64_t i = v << kLow;
          if ((i & g.control_mask[o]) == g.control_value[o]) a[0] = cmul<T>(f0, a[0]);
          if (V == 2 && ((i | 1) & g.control_mask[o]) == g.control_value[o]) a[V - 1] = cmul<T>(f1, a[V - 1]);
        } else {
          a[0] = cmul<T>(f0, a[0]);
          if (V == 2) a[V - 1] = cmul<T>(f1, a[V - 1]);
        }
      }
      if constexpr (V == 2)
        reinterpret_cast<float4*>(psi)[v] = make_float4(a[0].x, a[0].y, a[V - 1].x, a[V - 1].y);
      else
        psi[v] = a[0];
    }
  }
}

// Swapping physical bit pairs in place: amplitude j moves to pi(j), pi an
// involution on index bits. What bounds it is HBM (every amplitude that
// moves is read and written once, as long as both accesses are coalesced):
// a swap of a low bit with a high one scatters single amplitudes, 8 bytes
// of a 32-byte sector. So a block moves whole tiles: the tile's bits are the
// low `m` bits, their images under pi, and more bits up to kSwapMaxBits,
// closed under pi. Then pi maps tile t to the tile t' whose index bits are
// swapped and element e of it to image(e), and a block reads both tiles of a
// pair as rows of 2^m contiguous amplitudes (256 bytes), and writes each
// from the other's copy in shared memory, in rows again. Tiles that pi
// leaves as they are (t = t', image the identity) are not touched. The next
// pair's loads fly while the present one is written.
// Element e lies at e with its row bits folded into its low bits: row bit i
// is the image of low bit i where that leaves the row, so lanes that step
// over low bits hit distinct banks both when they write rows (low bits
// vary) and when they read mapped elements (row bits vary). All three maps
// of e are linear in its bits, so a thread's elements are its first one's
// plus constants. A random swap pass at 30 qubits: about 17 ms with one thread
// per amplitude, 3.7 ms now (0.70 of the copy rate; 27 qubits 0.83).
// Tiles of 16 KB: with 8 KB ones a complex64 pass ran at 0.51-0.54 of the
// copy rate (complex128, 16 KB, at 0.76-0.83).
// A complex64 state of 2^32 bytes or more whose rows scatter (four low bits
// or more leave the row) takes 512-byte rows and 32 KB tiles instead: half as
// many pages a byte (30 qubits, random swaps 5.2 -> 3.8 ms); one block per SM
// makes them slower elsewhere (27 qubits 0.40 -> 0.49 ms).
constexpr int kSwapMaxBits = 12;
constexpr int kSwapElems = 8;  // of a tile per thread (complex128: 4)

struct SwapGeom {
  uint64_t tiles;                 // 2^(n - k)
  int32_t k, m;                   // tile bits, low bits of a row
  int32_t np;                     // swapped pairs of tile-index bits
  int32_t moves;                  // image is not the identity
  uint8_t a[32], b[32];           // those pairs
  uint8_t fixed[kSwapMaxBits];   // the tile's physical bits, ascending
  uint8_t bit[kSwapMaxBits];     // physical bit of element bit i (the low m ones are 0..m-1)
  uint8_t image[kSwapMaxBits];   // element bit that element bit i moves to
  // Element i * threads: its offset in the state, its place in shared
  // memory and the place of its image.
  uint64_t off[kSwapElems];
  uint16_t pos[kSwapElems], from[kSwapElems];
};

__host__ __device__ __forceinline__ uint32_t swap_pos(uint32_t e, int m) {
  return e ^ ((e >> m) & ((1u << m) - 1u));
}

template <typename T, int kSwapThreads>
__global__ void __launch_bounds__(kSwapThreads) k_swap_bits(cplx_t<T>* __restrict__ psi,
                                                        const __grid_constant__ SwapGeom g) {
  constexpr int E = sizeof(T) == 4 ? kSwapElems : kSwapElems / 2;  // elements of a tile per thread
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx_t<T>(*buf)[E * kSwapThreads] = reinterpret_cast<cplx_t<T>(*)[E * kSwapThreads]>(smem_raw);
  __shared__ uint8_t fixed[kSwapMaxBits];
  if (threadIdx.x < kSwapMaxBits) fixed[threadIdx.x] = g.fixed[threadIdx.x];
  __syncthreads();
  uint64_t off = 0;
  uint32_t x0 = 0;
  for (int j = 0; j < g.k; ++j) {
    off |= uint64_t((threadIdx.x >> j) & 1u) << g.bit[j];
    x0 |= ((threadIdx.x >> j) & 1u) << g.image[j];
  }
  const uint32_t pos = swap_pos(threadIdx.x, g.m), from = swap_pos(x0, g.m);
  auto live = [&](int i) { return threadIdx.x + uint32_t(i) * kSwapThreads < (1u << g.k); };
  auto partner = [&](uint64_t t) {
    uint64_t t2 = t;
    for (int p = 0; p < g.np; ++p) {
      const uint64_t d = ((t >> g.a[p]) ^ (t >> g.b[p])) & 1u;
      t2 ^= (d << g.a[p]) | (d << g.b[p]);
    }
    return t2;
  };
  // The block's next tile from t on that moves, with its partner.
  auto next = [&](uint64_t& t, uint64_t& t2) {
    for (; t < g.tiles; t += gridDim.x) {
      t2 = partner(t);
      if (t2 > t || (t2 == t && g.moves)) return true;
    }
    return false;
  };
  cplx_t<T> x[E], y[E];
  cplx_t<T>*p1 = psi, *p2 = psi;  // this thread's first element of the two tiles
  auto load = [&](uint64_t t, uint64_t t2) {
    p1 = psi + (insert_zeros(t, fixed, g.k) + off);
    p2 = psi + (insert_zeros(t2, fixed, g.k) + off);
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (live(i)) x[i] = p1[g.off[i]];
    if (t2 != t)
#pragma unroll
      for (int i = 0; i < E; ++i)
        if (live(i)) y[i] = p2[g.off[i]];
  };
  uint64_t t = blockIdx.x, t2 = 0;
  bool more = next(t, t2);
  if (more) load(t, t2);
  while (more) {
    cplx_t<T>*w1 = p1, *w2 = p2;
    const bool two = w2 != w1;
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (live(i)) {
        buf[0][pos ^ g.pos[i]] = x[i];
        if (two) buf[1][pos ^ g.pos[i]] = y[i];
      }
    __syncthreads();
    t += gridDim.x;
    more = next(t, t2);
    if (more) load(t, t2);
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (live(i)) {
        w1[g.off[i]] = buf[two ? 1 : 0][from ^ g.from[i]];
        if (two) w2[g.off[i]] = buf[0][from ^ g.from[i]];
      }
    __syncthreads();
  }
}

template <typename T>
__global__ void k_set_one(cplx_t<T>* psi) {
  psi[0] = make_c<T>(T(1), T(0));
}

// Logical index -> physical index through per-byte lookup tables.
__device__ __forceinline__ uint64_t to_physical(uint64_t i, const uint64_t* tables, int ntables) {
  if (ntables == 0) return i;
  uint64_t p = 0;
  for (int b = 0; b < ntables; ++b) p |= tables[b * 256 + ((i >> (8 * b)) & 255)];
  return p;
}

template <typename T>
__global__ void k_export(const cplx_t<T>* __restrict__ psi, double2* __restrict__ out, uint64_t first,
                         uint64_t count, const uint64_t* __restrict__ tables, int ntables) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < count; t += stride) {
    const cplx_t<T> a = psi[to_physical(first + t, tables, ntables)];
    out[t] = make_double2(double(a.x), double(a.y));
  }
}

template <typename T>
__global__ void k_import(cplx_t<T>* __restrict__ psi, const double2* __restrict__ in, uint64_t first,
                         uint64_t count, const uint64_t* __restrict__ tables, int ntables) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < count; t += stride) {
    const double2 a = in[t];
    psi[to_physical(first + t, tables, ntables)] = make_c<T>(T(a.x), T(a.y));
  }
}

template <typename T>
__global__ void k_scale(cplx_t<T>* __restrict__ psi, uint64_t len, double factor) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < len; i += stride) {
    cplx_t<T> a = psi[i];
    a.x = T(double(a.x) * factor);
    a.y = T(double(a.y) * factor);
    psi[i] = a;
  }
}

unsigned grid_for(const StateImpl& s, uint64_t work_items) {
  const uint64_t blocks = (work_items + kThreads - 1) / kThreads;
  return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(blocks, uint64_t(s.sms) * 16)));
}

// The grid of a gate pass. A state that gives every SM 128 blocks is covered
// by `many` of them per SM, started in order, so that the SMs read and write
// neighbouring memory; 16 per SM stride over all of it. Each block sets its
// tables up, which smaller states and wider gates do not make up for. 16 per
// SM and many: 28 qubits complex64, gates on 1, 2, 3 qubits 0.700, 0.700, 0.685
// and 0.668, 0.658, 0.650 ms; 26 qubits complex128 0.371, 0.360, 0.354 and
// 0.340, 0.338, 0.339, a 2-qubit diagonal 0.394 and 0.347; low targets (64 per
// SM) 0.695, 0.727 and 0.671, 0.683, 0.361, 0.365 and 0.343, 0.357. 4-qubit
// gates and 3-qubit ones on low targets are slower so, and 22 qubits too (a
// diagonal 0.032 and 0.035 ms).
unsigned gate_grid(const StateImpl& s, uint64_t blocks, int many) {
  const uint64_t per_sm = blocks >= uint64_t(s.sms) * 128 ? uint64_t(many) : 16;
  return unsigned(std::max<uint64_t>(1, std::min(blocks, uint64_t(s.sms) * per_sm)));
}

template <typename T, int K, int G, bool VEC>
void dense_launch(StateImpl& s, const DenseGeom& g, const void* mat, const double* host) {
  constexpr int threads = kDenseThreads<T, K>;
  const size_t smem = size_t(1) << (2 * K);
  const size_t bytes = smem * sizeof(cplx_t<T>);
  const uint64_t blocks = (g.n_iter / G + threads - 1) / threads;
  const unsigned grid = gate_grid(s, blocks, K <= 3 ? 128 : 16);
  auto* psi = static_cast<cplx_t<T>*>(s.amp);
  if constexpr (K <= kInlineDense) {
    if (host) {
      using M = MatInline<T, 1 << (2 * K)>;
      k_dense<T, K, G, VEC, M><<<grid, threads, bytes, s.stream>>>(psi, g, mat_inline<T, 1 << (2 * K)>(host, 1 << (2 * K)));
      QVDG_LAUNCH_CHECK();
      return;
    }
  }
  using M = MatDevice<T>;
  if constexpr (K == 6) {  // more than the default 48 KB
    static OncePerDevice once;  // per instantiation
    once(s.device, [&] {
      QVDG_CUDA(
          cudaFuncSetAttribute(k_dense<T, K, G, VEC, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
    });
  }
  k_dense<T, K, G, VEC, M><<<grid, threads, bytes, s.stream>>>(psi, g, M{static_cast<const cplx_t<T>*>(mat)});
  QVDG_LAUNCH_CHECK();
}

template <typename T, int K>
void dense_pick(StateImpl& s, const DenseGeom& g, const void* mat, const double* host, bool bit0_free) {
  // Two groups per thread (two neighbours as one 16-byte load) as far as
  // their amplitudes fit the registers.
  if constexpr (K <= 4 || (K == 5 && sizeof(T) == 4)) {
    if (g.n_iter >= 2) {
      if constexpr (sizeof(T) == 4)
        if (bit0_free) return dense_launch<T, K, 2, true>(s, g, mat, host);
      return dense_launch<T, K, 2, false>(s, g, mat, host);
    }
  }
  dense_launch<T, K, 1, false>(s, g, mat, host);
}

template <typename T, int K>
void lanes_launch(StateImpl& s, const LaneGeom& g, const void* mat, const double* host) {
  constexpr int R = 4;
  const uint64_t blocks = ((g.rows + R - 1) / R * 32 + kThreads - 1) / kThreads;
  const unsigned grid = gate_grid(s, blocks, K <= 2 ? 64 : 16);
  auto* psi = static_cast<cplx_t<T>*>(s.amp);
  constexpr int kEntries = 1 << (2 * K);
  if (host)
    k_dense_lanes<T, K, R, MatInline<T, kEntries>>
        <<<grid, kThreads, 0, s.stream>>>(psi, g, mat_inline<T, kEntries>(host, kEntries));
  else
    k_dense_lanes<T, K, R, MatDevice<T>>
        <<<grid, kThreads, 0, s.stream>>>(psi, g, MatDevice<T>{static_cast<const cplx_t<T>*>(mat)});
  QVDG_LAUNCH_CHECK();
}

template <typename T>
void lanes_pick(StateImpl& s, const PlainGate& pg, uint64_t control_value, const std::vector<uint8_t>& ctrl,
                const void* mat, const double* host) {
  LaneGeom g{};
  g.rows = uint64_t(1) << (s.n - 5 - ctrl.size());
  g.control_value = control_value;
  g.num_fixed = int(ctrl.size());  // ascending
  for (size_t i = 0; i < ctrl.size(); ++i) g.fixed[i] = uint8_t(ctrl[i] - 5);
  for (size_t j = 0; j < pg.targets.size(); ++j) g.targets[j] = uint8_t(pg.targets[j]);
  switch (pg.targets.size()) {
    case 1: return lanes_launch<T, 1>(s, g, mat, host);
    case 2: return lanes_launch<T, 2>(s, g, mat, host);
    default: return lanes_launch<T, 3>(s, g, mat, host);
  }
}

template <typename T>
void plain_gate(StateImpl& s, const PlainGate& pg, const void* matrices, const double* host) {
  const int k = int(pg.targets.size());
  const int c = int(pg.controls.size());
  uint64_t control_value = 0;
  std::vector<uint8_t> ctrl;
  for (auto& cv : pg.controls) {
    ctrl.push_back(uint8_t(cv.first));
    if (cv.second) control_value |= uint64_t(1) << cv.first;
  }
  std::sort(ctrl.begin(), ctrl.end());
  const cplx_t<T>* mat = matrices ? static_cast<const cplx_t<T>*>(matrices) + pg.matrix_offset : nullptr;
  if (pg.diagonal) {
    DiagGeom g{};
    g.n_iter = uint64_t(1) << (s.n - c);
    g.control_value = control_value;
    g.num_ctrl = c;
    for (int i = 0; i < c; ++i) g.ctrl[i] = ctrl[i];
    g.k = k;
    for (int j = 0; j < k; ++j) g.targets[j] = uint8_t(pg.targets[j]);
    const bool bit0_ctrl = c > 0 && ctrl[0] == 0;
    const size_t bytes = (size_t(1) << k) * sizeof(cplx_t<T>);
    auto* psi = static_cast<cplx_t<T>*>(s.amp);
    auto launch = [&](const auto& m) {
      using M = std::decay_t<decltype(m)>;
      if (g.n_iter >= 2 && !bit0_ctrl)
        k_diag<T, 2, M><<<gate_grid(s, (g.n_iter / 2 + kThreads - 1) / kThreads, 128), kThreads, bytes, s.stream>>>(psi, g, m);
      else
        k_diag<T, 1, M><<<gate_grid(s, (g.n_iter + kThreads - 1) / kThreads, 128), kThreads, bytes, s.stream>>>(psi, g, m);
    };
    if (host)
      launch(mat_inline<T, 1 << kInlineDiagonal>(host, 1 << k));
    else
      launch(MatDevice<T>{mat});
    QVDG_LAUNCH_CHECK();
    return;
  }
  DenseGeom g{};
  g.n_iter = uint64_t(1) << (s.n - k - c);
  g.control_value = control_value;
  std::vector<uint8_t> fixed(ctrl);
  for (uint32_t t : pg.targets) fixed.push_back(uint8_t(t));
  std::sort(fixed.begin(), fixed.end());
  g.num_fixed = int(fixed.size());
  for (size_t i = 0; i < fixed.size(); ++i) g.fixed[i] = fixed[i];
  for (int h = 0; h < (1 << k); ++h) {
    uint64_t o = 0;
    for (int j = 0; j < k; ++j) o |= uint64_t((h >> j) & 1) << pg.targets[j];
    g.offsets[h] = o;
  }
  const bool bit0_free = fixed.empty() || fixed[0] != 0;
  // Targets all in the lane bits 0-4 (controls above them): warp shuffles.
  {
    bool lanes = k <= 3 && s.n >= 5;
    for (uint32_t t : pg.targets) lanes = lanes && t < 5;
    for (uint8_t cq : ctrl) lanes = lanes && cq >= 5;
    if (lanes) return lanes_pick<T>(s, pg, control_value, ctrl, mat, host);
  }
  // complex64, 4 qubits, no controls, targets (nearly) all among bits 0-3 --
  // each group one short contiguous run -- and a state of at least one tile:
  // stage tiles through shared memory (coalesced) instead. With fewer low
  // targets the direct kernel's accesses are coalesced enough and it is faster.
  int low_targets = 0;
  for (uint32_t t : pg.targets) low_targets += t < 4 ? 1 : 0;
  if (sizeof(T) == 4 && c == 0 && k == 4 && low_targets >= 3 &&
      s.n >= uint32_t(kTileBits) + 1) {
    DenseTileGeom tg{};
    int lb = kTileBits, nhigh = 0;
    for (int iter = 0; iter < 8; ++iter) {
      nhigh = 0;
      for (uint32_t t : pg.targets) nhigh += t >= uint32_t(lb) ? 1 : 0;
      const int next = kTileBits - nhigh;
      if (next == lb) break;
      lb = next;
    }
    std::vector<uint32_t> high;
    for (uint32_t t : pg.targets)
      if (t >= uint32_t(lb)) high.push_back(t);
    std::sort(high.begin(), high.end());
    if (int(high.size()) == nhigh && lb + nhigh == kTileBits) {
      tg.lb = lb;
      tg.nhigh = nhigh;
      tg.tiles = uint64_t(1) << (s.n - kTileBits);
      for (int i = 0; i < nhigh; ++i) tg.high[i] = uint8_t(high[i]);
      auto local = [&](uint32_t t) -> uint32_t {
        if (t < uint32_t(lb)) return t;
        return uint32_t(lb) + uint32_t(std::find(high.begin(), high.end(), t) - high.begin());
      };
      std::vector<uint8_t> ft;
      for (uint32_t t : pg.targets) ft.push_back(uint8_t(local(t)));
      std::sort(ft.begin(), ft.end());
      for (size_t i = 0; i < ft.size(); ++i) tg.fixed_tile[i] = ft[i];
      for (int h = 0; h < (1 << k); ++h) {
        uint32_t o = 0;
        for (int j = 0; j < k; ++j) o |= uint32_t((h >> j) & 1) << local(pg.targets[j]);
        tg.offsets[h] = uint16_t(o);
      }
      const size_t bytes = (size_t(1) << kTileBits) * sizeof(float2) + (size_t(1) << (2 * k)) * sizeof(float2);
      const unsigned grid = unsigned(std::min<uint64_t>(tg.tiles, uint64_t(s.sms) * 3));
      auto* psi = static_cast<float2*>(s.amp);
      auto* m = reinterpret_cast<const float2*>(mat);
      static OncePerDevice once;
      once(s.device, [&] {
        QVDG_CUDA(cudaFuncSetAttribute(k_dense_tile<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
      });
      k_dense_tile<4><<<grid, kThreads, bytes, s.stream>>>(psi, tg, m);
      QVDG_LAUNCH_CHECK();
      return;
    }
  }
  // 5-6 qubits: matrix products on tiles, unless too few amplitudes are
  // selected for one.
  if (launch_dense_wide(s, pg, mat)) return;
  switch (k) {
    case 1: return dense_pick<T, 1>(s, g, mat, host, bit0_free);
    case 2: return dense_pick<T, 2>(s, g, mat, host, bit0_free);
    case 3: return dense_pick<T, 3>(s, g, mat, host, bit0_free);
    case 4: return dense_pick<T, 4>(s, g, mat, host, bit0_free);
    case 5: return dense_pick<T, 5>(s, g, mat, host, bit0_free);
    case 6: return dense_pick<T, 6>(s, g, mat, host, bit0_free);
    default: throw Error(4, "dense gates on more than 6 qubits are not supported");
  }
}

// Byte-wise logical->physical tables for a non-identity layout (uploaded to
// the workspace); returns the number of tables (0 for the identity).
int layout_tables(StateImpl& s, uint64_t** dev_tables) {
  if (s.identity_layout()) {
    *dev_tables = nullptr;
    return 0;
  }
  const int ntables = int((s.n + 7) / 8);
  std::vector<uint64_t> t(size_t(ntables) * 256, 0);
  for (int b = 0; b < ntables; ++b)
    for (int v = 0; v < 256; ++v) {
      uint64_t p = 0;
      for (int bit = 0; bit < 8; ++bit) {
        const uint32_t q = uint32_t(8 * b + bit);
        if (q < s.n && ((v >> bit) & 1)) p |= uint64_t(1) << s.layout[q];
      }
      t[size_t(b) * 256 + v] = p;
    }
  uint64_t* d = static_cast<uint64_t*>(s.work2.get(t.size() * sizeof(uint64_t)));
  QVDG_CUDA(cudaMemcpyAsync(d, t.data(), t.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, s.stream));
  QVDG_CUDA(cudaStreamSynchronize(s.stream));  // `t` is pageable and goes out of scope
  *dev_tables = d;
  return ntables;
}

}  // namespace

void launch_plain_gate(StateImpl& s, const PlainGate& g, const void* matrices) {
  if (s.bits == 32)
    plain_gate<float>(s, g, matrices, nullptr);
  else
    plain_gate<double>(s, g, matrices, nullptr);
}

bool launch_plain_gate_inline(StateImpl& s, const PlainGate& g, const double* matrix) {
  if (g.tensor || g.targets.size() > size_t(g.diagonal ? kInlineDiagonal : kInlineDense)) return false;
  if (s.bits == 32)
    plain_gate<float>(s, g, nullptr, matrix);
  else
    plain_gate<double>(s, g, nullptr, matrix);
  return true;
}

bool diag_run_fits(const DiagRun& run, const PlainGate& g, int bits) {
  return run.count < kDiagRunGates && g.targets.size() <= size_t(kDiagRunTargets) &&
         run.entries + (1u << g.targets.size()) <= diag_run_entries(bits) &&
         g.matrix_offset + (size_t(1) << g.targets.size()) <= ~uint32_t(0);
}

void diag_run_add(DiagRun& run, const PlainGate& g) {
  const int o = run.count++;
  run.matrix[o] = uint32_t(g.matrix_offset);
  run.table[o] = uint16_t(run.entries);
  run.k[o] = uint8_t(g.targets.size());
  for (size_t j = 0; j < g.targets.size(); ++j) run.targets[o][j] = uint8_t(g.targets[j]);
  for (auto& c : g.controls) {
    run.control_mask[o] |= uint64_t(1) << c.first;
    if (c.second) run.control_value[o] |= uint64_t(1) << c.first;
  }
  run.entries += 1u << g.targets.size();
}

void launch_diag_run(StateImpl& s, const DiagRun& run, const void* matrices) {
  const uint64_t vectors = s.amp_bytes / 16;  // a state has at least one (n >= 1)
  const int index_bits = int(s.n) - (s.bits == 32 ? 1 : 0) - kRunTileBits;  // of the tile's number
  const int pieces = index_bits > 0 ? (index_bits + 7) / 8 : 0;
  const size_t smem = ((size_t(run.entries) * s.elem_bytes() + 15) & ~size_t(15)) + size_t(pieces) * 256 * 16;
  const uint64_t tiles = (vectors + (uint64_t(1) << kRunTileBits) - 1) >> kRunTileBits;
  const unsigned grid = unsigned(std::min<uint64_t>(tiles, uint64_t(s.sms) * 8));
  if (s.bits == 32)
    k_diag_run<float><<<grid, kThreads, smem, s.stream>>>(static_cast<float2*>(s.amp), vectors, pieces, run,
                                                          static_cast<const float2*>(matrices));
  else
    k_diag_run<double><<<grid, kThreads, smem, s.stream>>>(static_cast<double2*>(s.amp), vectors, pieces, run,
                                                           static_cast<const double2*>(matrices));
  QVDG_LAUNCH_CHECK();
}

void launch_swap_bits(StateImpl& s, const std::vector<std::pair<uint32_t, uint32_t>>& pairs) {
  if (pairs.empty()) return;
  std::vector<uint32_t> pi(s.n);
  for (uint32_t q = 0; q < s.n; ++q) pi[q] = q;
  for (auto& pr : pairs) std::swap(pi[pr.first], pi[pr.second]);
  SwapGeom g{};
  // 256-byte rows and 16 KB tiles, or 512 bytes and 32 KB.
  int scattered = 0;
  for (uint32_t q = 0; q < 5 && q < s.n; ++q) scattered += pi[q] > 5 ? 1 : 0;
  const bool large = s.bits == 32 && s.amp_bytes >= (size_t(1) << 32) && scattered >= 4;
  const uint32_t m = std::min<uint32_t>(s.bits == 32 ? (large ? 6 : 5) : 4, s.n);
  const uint32_t most = std::min<uint32_t>(s.bits == 32 ? (large ? 12 : 11) : 10, s.n);
  const uint32_t threads = large ? 512 : 256;
  // Element bits: the low bits, each one's image outside them next to it
  // (row bit i for low bit i as far as that goes), then more bits or pairs.
  std::vector<uint32_t> bits;
  std::vector<bool> in(s.n, false);
  auto add = [&](uint32_t q) {
    if (!in[q]) bits.push_back(q);
    in[q] = true;
  };
  for (uint32_t q = 0; q < m; ++q) add(q);
  std::vector<uint32_t> rows(m, ~0u), more;
  size_t count = m;
  for (uint32_t q = 0; q < m; ++q)
    if (pi[q] >= m) {
      rows[q] = pi[q];
      in[pi[q]] = true;
      ++count;
    }
  for (uint32_t q = m; q < s.n; ++q) {
    if (in[q]) continue;
    const uint32_t need = pi[q] == q ? 1 : 2;
    if (count + need > most) continue;
    more.push_back(q);
    in[q] = true;
    if (need == 2) {
      more.push_back(pi[q]);
      in[pi[q]] = true;
    }
    count += need;
  }
  size_t next = 0;
  for (uint32_t q = 0; q < m; ++q) {
    if (rows[q] != ~0u)
      bits.push_back(rows[q]);
    else if (next < more.size())
      bits.push_back(more[next++]);
  }
  while (next < more.size()) bits.push_back(more[next++]);
  // A gap (a low bit whose image stays low, and no bit to fill it) would
  // only cost bank conflicts: the order of the row bits is free.
  g.k = int(bits.size());
  g.m = int(m);
  g.tiles = uint64_t(1) << (s.n - bits.size());
  std::vector<uint32_t> sorted(bits);
  std::sort(sorted.begin(), sorted.end());
  for (size_t i = 0; i < bits.size(); ++i) {
    g.fixed[i] = uint8_t(sorted[i]);
    g.bit[i] = uint8_t(bits[i]);
    g.image[i] = uint8_t(std::find(bits.begin(), bits.end(), pi[bits[i]]) - bits.begin());
    if (pi[bits[i]] != bits[i]) g.moves = 1;
  }
  for (uint32_t i = 0; i < uint32_t(kSwapElems) && i * threads < (1u << g.k); ++i) {
    uint32_t image = 0;
    for (int j = 0; j < g.k; ++j)
      if ((i * threads >> j) & 1u) {
        g.off[i] |= uint64_t(1) << g.bit[j];
        image |= 1u << g.image[j];
      }
    g.pos[i] = uint16_t(swap_pos(i * threads, g.m));
    g.from[i] = uint16_t(swap_pos(image, g.m));
  }
  // Tile-index bit of a physical bit outside the tile.
  auto outer = [&](uint32_t q) {
    uint32_t o = q;
    for (uint32_t b : bits) o -= b < q ? 1 : 0;
    return uint8_t(o);
  };
  for (auto& pr : pairs)
    if (!in[pr.first]) {
      g.a[g.np] = outer(pr.first);
      g.b[g.np] = outer(pr.second);
      ++g.np;
    }
  const unsigned grid = unsigned(std::min<uint64_t>(g.tiles, uint64_t(s.sms) * 16));
  const size_t smem = size_t(large ? 64 : 32) << 10;  // two tiles
  if (large) {
    static OncePerDevice once;
    once(s.device, [&] {
      QVDG_CUDA(cudaFuncSetAttribute(k_swap_bits<float, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    });
    k_swap_bits<float, 512><<<grid, 512, smem, s.stream>>>(static_cast<float2*>(s.amp), g);
  } else if (s.bits == 32) {
    k_swap_bits<float, 256><<<grid, 256, smem, s.stream>>>(static_cast<float2*>(s.amp), g);
  } else {
    k_swap_bits<double, 256><<<grid, 256, smem, s.stream>>>(static_cast<double2*>(s.amp), g);
  }
  QVDG_LAUNCH_CHECK();
}

void launch_zero(StateImpl& s) {
  QVDG_CUDA(cudaMemsetAsync(s.amp, 0, s.amp_bytes, s.stream));
  if (s.bits == 32)
    k_set_one<float><<<1, 1, 0, s.stream>>>(static_cast<float2*>(s.amp));
  else
    k_set_one<double><<<1, 1, 0, s.stream>>>(static_cast<double2*>(s.amp));
  QVDG_LAUNCH_CHECK();
}

void launch_export(StateImpl& s, uint64_t first, uint64_t count, double* out_dev) {
  uint64_t* tables;
  const int nt = layout_tables(s, &tables);
  if (s.bits == 32)
    k_export<float><<<grid_for(s, count), kThreads, 0, s.stream>>>(static_cast<const float2*>(s.amp),
                                                                    reinterpret_cast<double2*>(out_dev), first,
                                                                    count, tables, nt);
  else
    k_export<double><<<grid_for(s, count), kThreads, 0, s.stream>>>(static_cast<const double2*>(s.amp),
                                                                     reinterpret_cast<double2*>(out_dev), first,
                                                                     count, tables, nt);
  QVDG_LAUNCH_CHECK();
}

void launch_import(StateImpl& s, uint64_t first, uint64_t count, const double* in_dev) {
  uint64_t* tables;
  const int nt = layout_tables(s, &tables);
  if (s.bits == 32)
    k_import<float><<<grid_for(s, count), kThreads, 0, s.stream>>>(static_cast<float2*>(s.amp),
                                                                    reinterpret_cast<const double2*>(in_dev), first,
                                                                    count, tables, nt);
  else
    k_import<double><<<grid_for(s, count), kThreads, 0, s.stream>>>(static_cast<double2*>(s.amp),
                                                                     reinterpret_cast<const double2*>(in_dev),
                                                                     first, count, tables, nt);
  QVDG_LAUNCH_CHECK();
}

void launch_scale(StateImpl& s, double factor) {
  if (s.bits == 32)
    k_scale<float><<<grid_for(s, s.size()), kThreads, 0, s.stream>>>(static_cast<float2*>(s.amp), s.size(), factor);
  else
    k_scale<double><<<grid_for(s, s.size()), kThreads, 0, s.stream>>>(static_cast<double2*>(s.amp), s.size(),
                                                                       factor);
  QVDG_LAUNCH_CHECK();
}

}  // namespace qvdg
