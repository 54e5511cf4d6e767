// Dense gates on 5 and 6 qubits on the CUDA cores, in the state's own
// precision: one pass over the state per gate (the reference's wide dense
// kernels, src/kernels.rs:330-473).
//
// A gate on k qubits costs 4 * 2^k multiply-adds per amplitude, so from five
// qubits on the arithmetic bounds the pass (6 qubits, 28-qubit complex64
// state: 1.9 ms of multiply-adds at full rate, 0.66 ms of HBM). One thread
// per group of 2^k amplitudes reads a matrix entry from shared memory for
// every four multiply-adds, and its 2^k amplitudes leave few warps (complex128:
// not even registers). Here the gate is a matrix product over a tile:
// NG groups side by side are a 2^k x NG matrix in shared memory, and a thread
// computes R rows of GQ groups in registers, reading R + GQ values for
// 4 * R * GQ multiply-adds.
//
// The tile's index bits are the targets and the lowest free bits, so that a
// block reads and writes it in contiguous runs (16 bytes a lane where bit 0
// is free of controls) whatever the targets are. Amplitude (c, g) of the tile
// (matrix column c, group g) lies at c * NG + (g ^ fold(c)); fold, chosen on
// the host, is linear and gives the index bits that a warp's lanes step over
// when they copy distinct banks.

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "dense_wide.hpp"

namespace qvdg {

namespace {

constexpr int kWideMaxItems = 32;  // elements a thread copies

struct WideGeom {
  uint64_t tiles;
  uint64_t control_value;
  int32_t num_fixed;             // tile bits and controls
  int32_t pairs;                 // bit 0 lies in the tile: elements 2i, 2i + 1 are one 16-byte access (complex64)
  uint8_t fixed[48];             // their positions, ascending
  uint8_t bit[16];               // physical bit of element bit i (ascending)
  uint16_t place[16];            // place of element bit i in shared memory (linear)
  uint64_t off[kWideMaxItems];   // element i * threads (of elements or pairs): offset in the state
  uint16_t pos[kWideMaxItems];   // and place
  uint8_t fold[8];               // place (group bits) that column bit j is folded into
};

// Threads of a block, one per R x GQ block of the product.
template <int K, int NG, int R, int GQ>
constexpr int kWideThreads = ((1 << K) / R) * (NG / GQ);

template <typename T, int K, int NG, int R, int GQ>
__global__ void __launch_bounds__(kWideThreads<K, NG, R, GQ>, 2)
    k_dense_wide(cplx_t<T>* __restrict__ psi, const __grid_constant__ WideGeom g, const cplx_t<T>* __restrict__ mat) {
  using C2 = cplx_t<T>;
  constexpr int D = 1 << K, kElems = D * NG, kLanes = NG / GQ, kThreads = kWideThreads<K, NG, R, GQ>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2* tile = reinterpret_cast<C2*>(smem_raw);
  C2* mt = tile + kElems;  // mt[c * D + r]
  __shared__ uint8_t fixed[48];
  if (threadIdx.x < 48) fixed[threadIdx.x] = g.fixed[threadIdx.x];
  for (int i = threadIdx.x; i < D * D; i += kThreads) mt[i] = mat[(i & (D - 1)) * D + (i >> K)];
  // This thread's first element of a tile: offset in the state and place.
  const bool pairs = sizeof(T) == 4 && g.pairs;
  uint64_t off = 0;
  uint32_t pos = 0;
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    const uint32_t e = threadIdx.x << (pairs ? 1 : 0);
    if ((e >> i) & 1u) {
      off |= uint64_t(1) << g.bit[i];
      pos ^= g.place[i];
    }
  }
  // Where this thread's groups of column c lie: c * NG + (group ^ fold(c)).
  const uint32_t gl = threadIdx.x % kLanes, r0 = (threadIdx.x / kLanes) * R;
  uint32_t fold[K];
#pragma unroll
  for (int j = 0; j < K; ++j) fold[j] = g.fold[j];
  __syncthreads();
  for (uint64_t t = blockIdx.x; t < g.tiles; t += gridDim.x) {
    C2* base = psi + ((insert_zeros(t, fixed, g.num_fixed) | g.control_value) + off);
    if (pairs) {
      if constexpr (sizeof(T) == 4) {
        constexpr int N = kElems / 2 / kThreads;
        float4 v[N < 8 ? N : 8];
#pragma unroll
        for (int i0 = 0; i0 < N; i0 += 8) {
#pragma unroll
          for (int i = 0; i < 8 && i0 + i < N; ++i) v[i] = *reinterpret_cast<const float4*>(base + g.off[i0 + i]);
#pragma unroll
          for (int i = 0; i < 8 && i0 + i < N; ++i) {
            const uint32_t q = pos ^ g.pos[i0 + i];
            tile[q] = make_float2(v[i].x, v[i].y);
            tile[q ^ g.place[0]] = make_float2(v[i].z, v[i].w);
          }
        }
      }
    } else {
      constexpr int N = kElems / kThreads;
      C2 v[N < 8 ? N : 8];
#pragma unroll
      for (int i0 = 0; i0 < N; i0 += 8) {
#pragma unroll
        for (int i = 0; i < 8 && i0 + i < N; ++i) v[i] = base[g.off[i0 + i]];
#pragma unroll
        for (int i = 0; i < 8 && i0 + i < N; ++i) tile[pos ^ g.pos[i0 + i]] = v[i];
      }
    }
    __syncthreads();
    C2 acc[R][GQ];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int q = 0; q < GQ; ++q) acc[r][q] = make_c<T>(T(0), T(0));
#pragma unroll 4
    for (int c = 0; c < D; ++c) {
      uint32_t f = 0;
#pragma unroll
      for (int j = 0; j < K; ++j) f ^= ((c >> j) & 1) ? fold[j] : 0u;
      C2 x[GQ], m[R];
      const C2* col = tile + c * NG;
#pragma unroll
      for (int q = 0; q < GQ; ++q) x[q] = col[(gl + q * kLanes) ^ f];
#pragma unroll
      for (int r = 0; r < R; ++r) m[r] = mt[c * D + r0 + r];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < GQ; ++q) cmac<T>(acc[r][q], m[r], x[q]);
    }
    __syncthreads();  // every column has been read
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint32_t f = 0;
#pragma unroll
      for (int j = 0; j < K; ++j) f ^= (((r0 + r) >> j) & 1) ? fold[j] : 0u;
#pragma unroll
      for (int q = 0; q < GQ; ++q) tile[(r0 + r) * NG + ((gl + q * kLanes) ^ f)] = acc[r][q];
    }
    __syncthreads();
    if (pairs) {
      if constexpr (sizeof(T) == 4) {
#pragma unroll 4
        for (int i = 0; i < kElems / 2 / kThreads; ++i) {
          const uint32_t q = pos ^ g.pos[i];
          const float2 a = tile[q], b = tile[q ^ g.place[0]];
          *reinterpret_cast<float4*>(base + g.off[i]) = make_float4(a.x, a.y, b.x, b.y);
        }
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < kElems / kThreads; ++i) base[g.off[i]] = tile[pos ^ g.pos[i]];
    }
    __syncthreads();
  }
}

template <typename T, int K, int NG, int R, int GQ>
void launch(StateImpl& s, const PlainGate& pg, const void* mat) {
  constexpr int D = 1 << K, kElems = D * NG, kThreads = kWideThreads<K, NG, R, GQ>;
  static_assert(kElems / kThreads <= kWideMaxItems, "a thread's elements");
  WideGeom g{};
  std::vector<uint32_t> ctrl;
  uint64_t taken = 0;  // targets and controls
  for (auto& c : pg.controls) {
    ctrl.push_back(c.first);
    taken |= uint64_t(1) << c.first;
    if (c.second) g.control_value |= uint64_t(1) << c.first;
  }
  uint64_t targets = 0;
  for (uint32_t t : pg.targets) targets |= uint64_t(1) << t;
  taken |= targets;
  // The tile's bits: the targets and the lowest free bits.
  uint64_t in = targets;
  std::vector<uint32_t> groups;
  for (uint32_t q = 0; (1 << groups.size()) < NG; ++q)
    if (!((taken >> q) & 1)) {
      groups.push_back(q);
      in |= uint64_t(1) << q;
    }
  std::vector<uint32_t> bits, fixed(ctrl);
  for (uint32_t q = 0; q < s.n; ++q)
    if ((in >> q) & 1) bits.push_back(q);
  fixed.insert(fixed.end(), bits.begin(), bits.end());
  std::sort(fixed.begin(), fixed.end());
  g.num_fixed = int(fixed.size());
  for (size_t i = 0; i < fixed.size(); ++i) g.fixed[i] = uint8_t(fixed[i]);
  g.tiles = uint64_t(1) << (s.n - fixed.size());
  g.pairs = sizeof(T) == 4 && bits[0] == 0;
  // The element bits that the lanes of one shared-memory access step over
  // (128 bytes: 16 lanes of 8-byte elements, 8 of 16): group bits take their
  // own place, target bits are folded into the places left.
  constexpr uint32_t kLaneBits = sizeof(T) == 4 ? 4 : 3;
  const size_t skip = g.pairs ? 1 : 0;
  uint32_t used = 0;
  for (size_t i = skip; i < bits.size() && i < skip + kLaneBits; ++i) {
    const auto it = std::find(groups.begin(), groups.end(), bits[i]);
    if (it != groups.end()) used |= 1u << (it - groups.begin());
  }
  for (size_t i = skip; i < bits.size() && i < skip + kLaneBits; ++i) {
    const auto it = std::find(pg.targets.begin(), pg.targets.end(), bits[i]);
    if (it == pg.targets.end()) continue;
    for (uint32_t p = 0; p < kLaneBits && (1 << p) < NG; ++p)
      if (!((used >> p) & 1)) {
        used |= 1u << p;
        g.fold[it - pg.targets.begin()] = uint8_t(1u << p);
        break;
      }
  }
  for (size_t i = 0; i < bits.size(); ++i) {
    g.bit[i] = uint8_t(bits[i]);
    const auto it = std::find(groups.begin(), groups.end(), bits[i]);
    if (it != groups.end()) {
      g.place[i] = uint16_t(1u << (it - groups.begin()));
    } else {
      const size_t j = size_t(std::find(pg.targets.begin(), pg.targets.end(), bits[i]) - pg.targets.begin());
      g.place[i] = uint16_t((1u << j) * NG ^ g.fold[j]);
    }
  }
  const uint32_t items = uint32_t(kElems / kThreads) >> skip;
  for (uint32_t i = 0; i < items; ++i) {
    const uint32_t e = (i * kThreads) << skip;
    for (size_t j = 0; j < bits.size(); ++j)
      if ((e >> j) & 1u) {
        g.off[i] |= uint64_t(1) << bits[j];
        g.pos[i] ^= g.place[j];
      }
  }
  const size_t smem = (size_t(kElems) + size_t(D) * D) * sizeof(cplx_t<T>);
  static OncePerDevice once;  // per instantiation
  once(s.device, [&] {
    QVDG_CUDA(cudaFuncSetAttribute(k_dense_wide<T, K, NG, R, GQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(smem)));
  });
  const unsigned grid = unsigned(std::min<uint64_t>(g.tiles, uint64_t(s.sms) * (smem <= 113 * 1024 ? 2 : 1)));
  k_dense_wide<T, K, NG, R, GQ><<<grid, kThreads, smem, s.stream>>>(static_cast<cplx_t<T>*>(s.amp), g,
                                                                       static_cast<const cplx_t<T>*>(mat));
  QVDG_LAUNCH_CHECK();
}

}  // namespace

// Which gates take the tile product.
//   - All 6-qubit gates of complex128: a group per thread does not fit its
//     registers (26 qubits 2.76 ms; tiles with 4 x 2 a thread 1.92, 8 x 4
//     1.67).
//   - Gates on states where one thread per group would leave SMs idle (fewer
//     than two blocks of groups per SM).
//   - Gates that leave none of the lowest bits free: neighbouring threads'
//     groups then lie 8 amplitudes or more apart (complex128: 4), and the
//     group kernel's loads fetch a sector for each lane. 28 qubits complex64,
//     targets 0, 1, 2 and others, group kernel and tiles: 5 qubits 2.64 and
//     1.87 ms, 6 qubits 3.37-4.17 and 3.22; 26 qubits complex128, 5 qubits,
//     targets 0, 1 and others 0.93 and 0.89, with 2 too 1.13 and 0.91.
// For the other gates on larger states the group kernel is faster (28 qubits
// complex64: 1.35-1.7 and 2.9-3.05 ms for 5 and 6 qubits, tiles 1.9-2.0 and
// 3.25-3.4; 26 qubits complex128, 5 qubits: 0.86 ms, tiles 0.89).
bool launch_dense_wide(StateImpl& s, const PlainGate& pg, const void* mat) {
  const size_t k = pg.targets.size();
  const int free_bits = int(s.n) - int(pg.controls.size());  // index bits of the selected amplitudes
  if ((k != 5 && k != 6) || free_bits < (s.bits == 32 ? 11 : 10)) return false;
  const bool few = (uint64_t(1) << (free_bits - int(k))) < uint64_t(s.sms) * 2 * 256;
  uint64_t taken = 0;
  for (uint32_t t : pg.targets) taken |= uint64_t(1) << t;
  for (auto& c : pg.controls) taken |= uint64_t(1) << c.first;
  const uint64_t lowest = s.bits == 32 ? 7 : 3;
  const bool scattered = (taken & lowest) == lowest;
  if (s.bits == 32) {
    if (few) {
      if (k == 6)
        launch<float, 6, 32, 4, 2>(s, pg, mat);
      else
        launch<float, 5, 64, 4, 2>(s, pg, mat);
    } else {
      if (!scattered) return false;
      if (k == 6)
        launch<float, 6, 64, 16, 2>(s, pg, mat);
      else
        launch<float, 5, 128, 16, 2>(s, pg, mat);
    }
  } else if (k == 6) {
    // Tiles of 2048 amplitudes once they give every SM two.
    if (free_bits >= 11 && (uint64_t(1) << (free_bits - 11)) >= uint64_t(s.sms) * 2)
      launch<double, 6, 32, 8, 4>(s, pg, mat);
    else
      launch<double, 6, 16, 4, 1>(s, pg, mat);
  } else if (few) {
    launch<double, 5, 32, 4, 1>(s, pg, mat);
  } else {
    if (!scattered) return false;
    launch<double, 5, 128, 8, 4>(s, pg, mat);
  }
  return true;
}

}  // namespace qvdg
