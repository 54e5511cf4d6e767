// Register-blocked stage kernel: the staged tile pass on the CUDA cores,
// gate by gate without fusing matrices.
//
// A stage (the reference's cache-blocked stage, src/blocking.rs:57-302) runs
// over tiles of 2^L amplitudes held in shared memory. Within a tile the
// stage's gates are cut into *register passes*: each names four tile bits G;
// a thread loads the 16 amplitudes of one G-subcube into registers, applies
// every gate of the pass there and stores them back. A register pass takes
// the gates, in dependency order, whose dense targets lie in G (controls may
// be anywhere: outside G they are a per-thread or per-tile predicate, inside
// a mask of active register groups) and every diagonal gate that is ready
// (a diagonal reads bits inside G per register and bits outside G from the
// thread's subcube base). So one shared-memory round trip serves several
// gates, and no matrix is ever multiplied out. A 1-qubit gate whose rows'
// larger entries lie on the diagonal and agree up to sign (rotations, H, SX,
// the square roots of X, Y and W) is divided by them: x0 + a x1 and
// x1 + b x0, two multiply-adds per amplitude for real or imaginary a and b,
// four for complex ones, half of what the matrix takes. The stage's last
// register pass multiplies by the product of the divisors, an earlier one where
// that product would leave the numbers' range, and their signs join the sign
// flips. A +-1 diagonal (CZ and the like) only toggles sign
// bits, consecutive ones together; a (controlled) X moves registers.
//
// A tile's 16-byte cp.async copies and its stores back to HBM are covered by
// another CTA's computation: two CTAs per SM, one tile buffer each. What
// bounds the kernel is the latency of each gate's chain (its record, then
// its matrix, then the arithmetic), so warps count for more than a second
// buffer: one CTA with two buffers left a complex128 stage 8 warps per SM.
// (26-qubit complex128 grid circuit of depth 20, 14 stages: 43.7 ms then,
// 23.7 now, of which sheared gates and sign flips are a fifth.)
// Only a pass whose gate data leave no room for a second CTA keeps two
// buffers, the next tile's copies in flight while the current is computed.

#include <cuda_runtime.h>

#include <algorithm>
#include <complex>
#include <cstring>
#include <vector>

#include "program.hpp"
#include "stage_kernel.hpp"

namespace qvdg {

namespace {

constexpr int kRegThreads = 512;
constexpr size_t kRegBlobBudget = 64 * 1024;
// How far the product of the divisors left out may go from 1 (a power of two)
// before the state is multiplied by it: until then the amplitudes are off by
// its inverse, and 200 gates with a divisor of 1/2 would take complex64 ones
// past 2^128. 2^40 (complex128: 2^200) leaves a state that is not normalised
// the rest of the range; unitary gates (divisors from 1/sqrt 2) reach it once
// in 80 of them.
bool scale_far(const std::complex<long double>& scale, int bits) {
  const long double size = scale.real() * scale.real() + scale.imag() * scale.imag();
  const long double limit = bits == 32 ? 0x1p80L : 0x1p400L;
  return size > limit || size * limit < 1.0L;
}

enum : uint8_t { kRegDense1 = 0, kRegDense2 = 1, kRegSign = 2, kRegPhase = 3, kRegSign2 = 4 };
enum : uint8_t { kFormGeneral = 0, kFormReal = 1, kFormImag = 2, kFormComplex = 3, kFormX = 4 };

// Shared-memory position of tile element e, XOR-linear. complex64: bits 1-3
// XORed with bits 5-7, 9-11 and 13-15 (bit 0 is kept, so element pairs 2v,
// 2v+1 stay one 16-byte slot for cp.async). complex128, whose elements are
// 16 bytes and go eight lanes at a time: bits 0-2 XORed with every higher
// three, so that any three neighbouring bits reach all eight places.
template <typename T>
__device__ __forceinline__ uint32_t reg_swz(uint32_t e) {
  if (sizeof(T) == 8) return e ^ (((e >> 3) ^ (e >> 6) ^ (e >> 9)) & 7u);
  return e ^ (((e >> 4) ^ (e >> 8) ^ (e >> 12)) & 14u);
}

struct RegPassHdr {
  uint8_t g[4];         // tile bits held in registers, ascending: register index bit i <-> tile bit g[i]
  uint16_t num_gates;
  uint16_t pair;        // g[0] == 0: registers j, j^1 are one 16-byte slot (complex64)
  uint32_t first_gate;  // index of the pass's first gate
  uint32_t pad;
};
static_assert(sizeof(RegPassHdr) == 16, "header layout");

// Dispatch codes of the register kernel (one switch per gate).
enum : uint16_t {
  kOpShear = 0,    // + 4 * (form - kFormReal) + target register bit (12 codes): (a, b)
  kOpX = 12,       // + target register bit: X where `pmask` says
  kOpDense1 = 16,  // + target register bit: any matrix, where `pmask` says
  kOpDense2 = 20,
  kOpSign2 = 21,
  kOpSign = 22,
  kOpPhase = 23,
  kOpScale = 24,   // multiply by a number
};

struct RegGate {
  // Hot: the first 16 bytes, read with one 16-byte load per gate.
  uint16_t op;        // kOp* dispatch code
  uint16_t pmask;     // dense: register bases j (target bits clear) whose group is active (0xffff: all)
  uint8_t t0, t1;     // dense: register bits of matrix bits 0 and 1; kOpSign2: bit of index bits 0, 1 in the
                      // word (tile base | subcube base << 48), 63: none
  uint8_t pred;       // 1 when the gate has controls outside the registers (gcm/lcm)
  uint8_t k;          // diagonal: targets
  uint32_t data;      // byte offset in the pass blob: matrix, diagonal entries or sign masks
  uint32_t table;     // diagonal: byte offset of the 16 register index parts (uint16)
  // Cold.
  uint32_t lcm, lcv;  // controls on tile bits outside the registers (per-thread predicate)
  uint64_t gcm, gcv;  // controls on global bits (per-tile predicate)
  uint8_t tgt[16];    // diagonal target i: 0x40|j register bit j, l < 0x40 tile bit, 0x80|p global bit p
  uint8_t kind, spec; // host bookkeeping
  uint8_t pad1[6];
};
static_assert(sizeof(RegGate) == 64, "gate layout");

// ---------------------------------------------------------------------------
// Device side.

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ cplx_t<T> neg_c(cplx_t<T> a) {
  return make_c<T>(-a.x, -a.y);
}

template <typename T>
__device__ __forceinline__ cplx_t<T> mul_c(cplx_t<T> m, cplx_t<T> x) {
  return make_c<T>(fma(m.x, x.x, -m.y * x.y), fma(m.x, x.y, m.y * x.x));
}

// x + m * y for real, imaginary or complex m.
template <typename T, int FORM>
__device__ __forceinline__ cplx_t<T> shear(cplx_t<T> x, cplx_t<T> m, cplx_t<T> y) {
  if (FORM == kFormReal) return make_c<T>(fma(m.x, y.x, x.x), fma(m.x, y.y, x.y));
  if (FORM == kFormImag) return make_c<T>(fma(-m.y, y.y, x.x), fma(m.y, y.x, x.y));
  return make_c<T>(fma(m.x, y.x, fma(-m.y, y.y, x.x)), fma(m.x, y.y, fma(m.y, y.x, x.y)));
}

// Sign flip of a complex value where `bit` is 1, on the sign bits.
// (bit 31 of `t` set: negate).
__device__ __forceinline__ void flip(float2& x, uint32_t t) {
  const uint32_t s = t & 0x80000000u;
  x.x = __uint_as_float(__float_as_uint(x.x) ^ s);
  x.y = __uint_as_float(__float_as_uint(x.y) ^ s);
}
__device__ __forceinline__ void flip(double2& x, uint32_t t) {
  const unsigned long long s = (unsigned long long)(t & 0x80000000u) << 32;
  x.x = __longlong_as_double(__double_as_longlong(x.x) ^ s);
  x.y = __longlong_as_double(__double_as_longlong(x.y) ^ s);
}

template <typename T, int TB, int FORM>
__device__ __forceinline__ void apply_shear(cplx_t<T> (&a)[16], const cplx_t<T>* m) {
  const cplx_t<T> m0 = m[0], m1 = m[1];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j & (1 << TB)) continue;
    const cplx_t<T> x0 = a[j], x1 = a[j | (1 << TB)];
    a[j] = shear<T, FORM>(x0, m0, x1);
    a[j | (1 << TB)] = shear<T, FORM>(x1, m1, x0);
  }
}

template <typename T, int TB>
__device__ __forceinline__ void apply_x(cplx_t<T> (&a)[16], uint32_t pmask) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j & (1 << TB)) continue;
    const bool on = (pmask >> j) & 1u;
    const cplx_t<T> x0 = a[j], x1 = a[j | (1 << TB)];
    a[j] = on ? x1 : x0;
    a[j | (1 << TB)] = on ? x0 : x1;
  }
}

// A matrix entry from shared memory, read where it is used (volatile: kept in
// registers over the pairs, the entries would spill).
__device__ __forceinline__ float2 entry(const float2* m) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_u32(m)));
  return v;
}
__device__ __forceinline__ double2 entry(const double2* m) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(smem_u32(m)));
  return v;
}

template <typename T, int TB>
__device__ __forceinline__ void apply_dense1(cplx_t<T> (&a)[16], const cplx_t<T>* m, uint32_t pmask) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j & (1 << TB)) continue;
    const cplx_t<T> x0 = a[j], x1 = a[j | (1 << TB)];
    cplx_t<T> y0 = mul_c<T>(entry(m + 1), x1), y1 = mul_c<T>(entry(m + 3), x1);
    cmac<T>(y0, entry(m), x0);
    cmac<T>(y1, entry(m + 2), x0);
    const bool on = (pmask >> j) & 1u;
    a[j] = on ? y0 : x0;
    a[j | (1 << TB)] = on ? y1 : x1;
  }
}

// Dense 2-qubit gate on the subcube at `place` in the tile, on the register
// bits whose byte distances are b0 and b1 (the others c0 and c1), for the
// groups active in `groups` (bit k: the others' values). It works on the
// thread's own subcube in shared memory, one group at a time: six pairs of
// target bits as code on the registers would take more of them than two CTAs
// per SM leave.
template <typename T>
__device__ __noinline__ void apply2(unsigned char* tile, uint32_t place, uint32_t b0, uint32_t b1, uint32_t c0,
                                    uint32_t c1, uint32_t groups, const cplx_t<T>* m) {
#pragma unroll 1
  for (uint32_t k = 0; k < 4; ++k) {
    if (!((groups >> k) & 1u)) continue;
    const uint32_t o = place ^ ((k & 1u) ? c0 : 0u) ^ ((k & 2u) ? c1 : 0u);
    cplx_t<T>* p[4] = {reinterpret_cast<cplx_t<T>*>(tile + o), reinterpret_cast<cplx_t<T>*>(tile + (o ^ b0)),
                       reinterpret_cast<cplx_t<T>*>(tile + (o ^ b1)),
                       reinterpret_cast<cplx_t<T>*>(tile + (o ^ b0 ^ b1))};
    const cplx_t<T> x[4] = {*p[0], *p[1], *p[2], *p[3]};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      cplx_t<T> acc = make_c<T>(T(0), T(0));
#pragma unroll
      for (int c = 0; c < 4; ++c) cmac<T>(acc, m[r * 4 + c], x[c]);
      *p[r] = acc;
    }
  }
}

template <typename T>
__device__ __forceinline__ void flip_mask(cplx_t<T> (&a)[16], uint32_t mask) {
#pragma unroll
  for (int j = 0; j < 16; ++j) flip(a[j], mask << (31 - j));
}

// Index bits of a diagonal gate that do not come from the registers.
__device__ __forceinline__ uint32_t diag_fixed(const RegGate& g, uint32_t eb, uint64_t tile_base) {
  uint32_t idx = 0;
  for (int i = 0; i < g.k; ++i) {
    const uint32_t t = g.tgt[i];
    if (t & 0x80)
      idx |= uint32_t((tile_base >> (t & 0x7f)) & 1u) << i;
    else if (!(t & 0x40))
      idx |= ((eb >> t) & 1u) << i;
  }
  return idx;
}

template <typename T>
__device__ void run_register_pass(cplx_t<T>* tile, const RegPassHdr& h, const RegGate* gates,
                                  const unsigned char* blob, int L, uint64_t tile_base) {
  using C2 = cplx_t<T>;
  const uint32_t nsub = 1u << (L - 4);
  uint32_t bit[4];  // byte distance (swizzled) of each register bit
#pragma unroll
  for (int i = 0; i < 4; ++i)  // a reduction of equal lanes: in uniform registers (24.3 -> 23.7 ms)
    bit[i] = __reduce_or_sync(0xffffffffu, reg_swz<T>(1u << h.g[i]) * uint32_t(sizeof(C2)));
  const uint32_t first = h.first_gate, last = first + h.num_gates;
  for (uint32_t s = threadIdx.x; s < nsub; s += blockDim.x) {
    uint32_t eb = s;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t p = h.g[i];
      eb = ((eb >> p) << (p + 1)) | (eb & ((1u << p) - 1u));
    }
    // Register j at the subcube's place XOR the places of j's bits (the
    // swizzle is XOR-linear).
    unsigned char* const bytes = reinterpret_cast<unsigned char*>(tile);
    const uint32_t place = reg_swz<T>(eb) * uint32_t(sizeof(C2));
    auto at = [&](int j) {
      uint32_t o = place;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if ((j >> i) & 1) o ^= bit[i];
      return bytes + o;
    };
    C2 a[16];
    auto fetch = [&] {
      if (sizeof(C2) == 8 && h.pair) {
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float4 v = *reinterpret_cast<const float4*>(at(j));
          a[j] = make_c<T>(T(v.x), T(v.y));
          a[j + 1] = make_c<T>(T(v.z), T(v.w));
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) a[j] = *reinterpret_cast<const C2*>(at(j));
      }
    };
    auto save = [&] {
      if (sizeof(C2) == 8 && h.pair) {
#pragma unroll
        for (int j = 0; j < 16; j += 2)
          *reinterpret_cast<float4*>(at(j)) =
              make_float4(float(a[j].x), float(a[j].y), float(a[j + 1].x), float(a[j + 1].y));
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) *reinterpret_cast<C2*>(at(j)) = a[j];
      }
    };
    fetch();
    // Bits a sign gate reads outside the registers: the tile's global bits
    // and the subcube's tile bits (at 48 and up).
    const uint64_t where = tile_base | (uint64_t(eb) << 48);
    uint32_t flips = 0;   // registers to negate
    bool signs = false;   // some gate has set it (the same in every thread)
    // The next gate's record is read while the present one is applied.
    uint4 ahead = *reinterpret_cast<const uint4*>(&gates[first]);
    for (uint32_t gi = first; gi < last; ++gi) {
      const RegGate& g = gates[gi];
      const uint4 hot = ahead;
      ahead = *reinterpret_cast<const uint4*>(&gates[gi + 1 < last ? gi + 1 : gi]);
      const uint32_t op = hot.x & 0xffffu, pmask = hot.x >> 16;
      const uint32_t t0 = hot.y & 0xffu, t1 = (hot.y >> 8) & 0xffu;
      if ((hot.y >> 16) & 0xffu)
        if ((tile_base & g.gcm) != g.gcv || (eb & g.lcm) != g.lcv) continue;
      const unsigned char* data = blob + hot.z;
      const C2* m = reinterpret_cast<const C2*>(data);
      if (op < kOpSign2 && signs) {
        // Sign flips up to here, all at once (diagonals commute with them).
        flip_mask<T>(a, flips);
        flips = 0;
        signs = false;
      }
      switch (op) {
#define QVDG_SHEAR(form, bit_) \
  case kOpShear + 4 * (form - kFormReal) + bit_: apply_shear<T, bit_, form>(a, m); break;
        QVDG_SHEAR(kFormReal, 0)
        QVDG_SHEAR(kFormReal, 1)
        QVDG_SHEAR(kFormReal, 2)
        QVDG_SHEAR(kFormReal, 3)
        QVDG_SHEAR(kFormImag, 0)
        QVDG_SHEAR(kFormImag, 1)
        QVDG_SHEAR(kFormImag, 2)
        QVDG_SHEAR(kFormImag, 3)
        QVDG_SHEAR(kFormComplex, 0)
        QVDG_SHEAR(kFormComplex, 1)
        QVDG_SHEAR(kFormComplex, 2)
        QVDG_SHEAR(kFormComplex, 3)
#undef QVDG_SHEAR
        case kOpX + 0: apply_x<T, 0>(a, pmask); break;
        case kOpX + 1: apply_x<T, 1>(a, pmask); break;
        case kOpX + 2: apply_x<T, 2>(a, pmask); break;
        case kOpX + 3: apply_x<T, 3>(a, pmask); break;
        case kOpDense1 + 0: apply_dense1<T, 0>(a, m, pmask); break;
        case kOpDense1 + 1: apply_dense1<T, 1>(a, m, pmask); break;
        case kOpDense1 + 2: apply_dense1<T, 2>(a, m, pmask); break;
        case kOpDense1 + 3: apply_dense1<T, 3>(a, m, pmask); break;
        case kOpDense2: {
          save();
          // The register bits that are not targets, and the groups (by their
          // values) that are active.
          const uint32_t rest = 15u & ~((1u << t0) | (1u << t1));
          const uint32_t r0 = __ffs(rest) - 1u, r1 = 31u - __clz(rest);
          uint32_t groups = 0;
          for (uint32_t k = 0; k < 4; ++k)
            groups |= ((pmask >> (((k & 1u) << r0) | ((k >> 1) << r1))) & 1u) << k;
          auto dist = [&](uint32_t i) { return i == 0 ? bit[0] : (i == 1 ? bit[1] : (i == 2 ? bit[2] : bit[3])); };
          apply2<T>(bytes, place, dist(t0), dist(t1), dist(r0), dist(r1), groups, m);
          fetch();
          break;
        }
        case kOpSign2: {
          const uint16_t* masks = reinterpret_cast<const uint16_t*>(data);
          flips ^= masks[uint32_t((where >> t0) & 1u) | (uint32_t((where >> t1) & 1u) << 1)];
          signs = true;
          break;
        }
        case kOpSign: {
          const uint16_t* masks = reinterpret_cast<const uint16_t*>(data);
          flips ^= masks[diag_fixed(g, eb, tile_base)];
          signs = true;
          break;
        }
        case kOpPhase: {
          const uint16_t* ridx = reinterpret_cast<const uint16_t*>(blob + hot.w);
          const uint32_t f = diag_fixed(g, eb, tile_base);
#pragma unroll
          for (int j = 0; j < 16; ++j) a[j] = mul_c<T>(m[f | ridx[j]], a[j]);
          break;
        }
        default: {  // kOpScale
          const C2 f = m[0];
          if (f.y == T(0)) {
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = make_c<T>(f.x * a[j].x, f.x * a[j].y);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = mul_c<T>(f, a[j]);
          }
          break;
        }
      }
    }
    if (signs) flip_mask<T>(a, flips);
    save();
  }
  __syncthreads();
}

// complex128 tiles are 2^12 amplitudes (256 subcubes): 256 threads, which
// leaves room for twice the registers.
template <typename T>
constexpr int reg_threads() {
  return sizeof(T) == 4 ? kRegThreads : kRegThreads / 2;
}

template <typename T>
__global__ void __launch_bounds__(reg_threads<T>(), 2)
    k_stage_reg(cplx_t<T>* __restrict__ psi, const TileGeom geo, const unsigned char* __restrict__ blob_all,
                int buffers) {
  using C2 = cplx_t<T>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint8_t tile_bits[48];
  __shared__ uint64_t map_lo[32], map_hi[32];
  const int tid = threadIdx.x;
  const int L = geo.L, B = geo.B;
  const uint32_t n_el = 1u << L;
  C2* const buf0 = reinterpret_cast<C2*>(smem);  // tiles at buf0 (and buf0 + n_el)
  unsigned char* blob = smem + size_t(buffers) * sizeof(C2) * n_el;

  for (int i = tid; i < 48; i += blockDim.x) tile_bits[i] = geo.tile_bits[i];
  {
    const uint4* src = reinterpret_cast<const uint4*>(blob_all + geo.tc_offset);
    uint4* dst = reinterpret_cast<uint4*>(blob);
    for (uint32_t i = tid; i < geo.tc_bytes / 16; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  // Tile element e -> physical index offset: the low B bits are physical
  // bits 0..B-1; the others go through two tables of their set bits.
  const int nfree = L - B, nlo = nfree < 5 ? nfree : 5;
  for (int i = tid; i < 32; i += blockDim.x) {
    uint64_t a = 0, b = 0;
    for (int j = 0; j < nlo; ++j)
      if ((i >> j) & 1) a |= uint64_t(1) << tile_bits[B + j];
    for (int j = nlo; j < nfree; ++j)
      if ((i >> (j - nlo)) & 1) b |= uint64_t(1) << tile_bits[B + j];
    map_lo[i] = a;
    map_hi[i] = b;
  }
  __syncthreads();
  const uint32_t lowmask = (1u << B) - 1u;
  auto phys = [&](uint64_t base, uint32_t e) -> uint64_t {
    const uint32_t r = e >> B;
    return base | map_lo[r & 31] | map_hi[r >> nlo] | (e & lowmask);
  };
  constexpr uint32_t per16 = 16 / sizeof(C2);  // elements per 16-byte copy
  const uint32_t units = n_el / per16;
  const RegPassHdr* hdrs = reinterpret_cast<const RegPassHdr*>(blob);
  const RegGate* gates = reinterpret_cast<const RegGate*>(blob + sizeof(RegPassHdr) * geo.num_gates);

  auto issue = [&](uint64_t t, C2* dst) {
    const uint64_t base = insert_zeros(t, tile_bits, L);
    for (uint32_t u = tid; u < units; u += blockDim.x) {
      const uint32_t e = u * per16;
      cp_async16(smem_u32(dst + reg_swz<T>(e)), psi + phys(base, e));
    }
  };

  uint64_t t = blockIdx.x;
  int cur = 0;
  const int other = buffers - 1;  // 0: one buffer
  if (t < geo.num_tiles && other) issue(t, buf0);
  cp_async_commit();
  for (; t < geo.num_tiles; t += gridDim.x) {
    const uint64_t next = t + gridDim.x;
    if (!other) {
      issue(t, buf0);
      cp_async_commit();
      cp_async_wait0();
    } else {
      if (next < geo.num_tiles) issue(next, buf0 + (cur ^ 1) * n_el);
      cp_async_commit();
      cp_async_wait1();
    }
    __syncthreads();
    C2* tile = buf0 + cur * n_el;
    const uint64_t base = insert_zeros(t, tile_bits, L);
    for (int p = 0; p < geo.num_gates; ++p) run_register_pass<T>(tile, hdrs[p], gates, blob, L, base);
    for (uint32_t u = tid; u < units; u += blockDim.x) {
      const uint32_t e = u * per16;
      *reinterpret_cast<uint4*>(psi + phys(base, e)) = *reinterpret_cast<const uint4*>(tile + reg_swz<T>(e));
    }
    __syncthreads();
    cur ^= other;
  }
  cp_async_wait0();
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side: lowering a stage to register passes.

namespace {

struct RegOp {
  bool dense = false;
  std::vector<int> tgt;                      // dense: tile bits; diagonal: encoded as RegGate::tgt (before registers)
  std::vector<int> dtgt_local;               // diagonal: tile bit of target i, or -1
  std::vector<int> dtgt_global;              // diagonal: physical bit of target i, or -1
  uint32_t local_ctl_mask = 0, local_ctl_val = 0;
  uint64_t gcm = 0, gcv = 0;
  uint32_t qmask = 0;                        // tile bits touched (dependencies)
  std::vector<C> entries;                    // dense matrix (row-major) or diagonal entries
};

bool is_pm_one(const C& c) { return c.im == 0.0 && (c.re == 1.0 || c.re == -1.0); }

template <typename V>
size_t put(std::vector<uint8_t>& blob, const V* p, size_t n) {
  blob.resize((blob.size() + 15) & ~size_t(15), 0);
  const size_t off = blob.size();
  blob.resize(off + n * sizeof(V));
  std::memcpy(blob.data() + off, p, n * sizeof(V));
  return off;
}

size_t put_complex(std::vector<uint8_t>& blob, const std::vector<C>& v, int bits) {
  if (bits == 32) {
    std::vector<float> f;
    for (const C& c : v) {
      f.push_back(float(c.re));
      f.push_back(float(c.im));
    }
    return put(blob, f.data(), f.size());
  }
  std::vector<double> d;
  for (const C& c : v) {
    d.push_back(c.re);
    d.push_back(c.im);
  }
  return put(blob, d.data(), d.size());
}

// How a 1-qubit gate is applied: X, sheared (m becomes (a, b), its divisor
// goes into `scale`; `negate`: the second row's has the other sign), or by
// its matrix. Only a gate applied everywhere can be sheared, and only by a
// divisor of ordinary size (a user's matrix need not be unitary).
uint8_t dense1_form(std::vector<C>& m, bool everywhere, std::complex<long double>& scale, bool& negate) {
  using Cd = std::complex<double>;
  const Cd u[4] = {{m[0].re, m[0].im}, {m[1].re, m[1].im}, {m[2].re, m[2].im}, {m[3].re, m[3].im}};
  if (u[0] == 0.0 && u[3] == 0.0 && u[1] == 1.0 && u[2] == 1.0) return kFormX;
  const double d = std::abs(u[0]);
  if (!everywhere || !(d >= 0.5 && d <= 2.0)) return kFormGeneral;
  const double eps = 2.3e-16 * d;
  const bool same = std::abs(u[3] - u[0]) <= eps, opposite = std::abs(u[3] + u[0]) <= eps;
  if (!(same || opposite) || !(std::abs(u[1]) <= 1.0001 * d) || !(std::abs(u[2]) <= 1.0001 * d)) return kFormGeneral;
  const Cd a = u[1] / u[0], b = u[2] / u[3];
  // a and b are rounded: the divisor that keeps the rows' norms takes half of
  // that back (equal gates would add it up).
  using Cl = std::complex<long double>;
  const Cl l[4] = {Cl(u[0]), Cl(u[1]), Cl(u[2]), Cl(u[3])};
  auto off = [&](const Cd& ratio, const Cl& entry, const Cl& div) {  // of an entry, times its share of the row
    return entry == Cl(0) ? Cl(0) : (Cl(ratio) * div / entry - Cl(1)) * (std::norm(entry) / (std::norm(entry) + std::norm(div)));
  };
  scale *= l[0] * (Cl(1) - (off(a, l[1], l[0]) + off(b, l[2], l[3])) / Cl(2));
  negate = opposite;
  m = {C{a.real(), a.imag()}, C{b.real(), b.imag()}};
  if (a.imag() == 0.0 && b.imag() == 0.0) return kFormReal;
  if (a.real() == 0.0 && b.real() == 0.0) return kFormImag;
  return kFormComplex;
}

}  // namespace

bool register_pass_ok(const Target& s, const PlannedPass& p) {
  if (!p.staged || p.tile_bits.size() < 5 || p.tile_bits.size() > 14) return false;
  for (const HOp& op : p.ops) {
    if (op.diagonal) {
      if (op.targets.size() + op.controls.size() > QVDG_MAX_DIAGONAL_QUBITS) return false;
    } else if (op.targets.size() > 2) {
      return false;
    }
  }
  (void)s;
  return true;
}

namespace {

// False when the pass's blob is too large (nothing is uploaded then).
bool lower_register(const Target& s, const PlannedPass& p, const StageConfig& cfg, StageUpload& up, bool shear,
                    LoweredPass& lp) {
  lp.staged = true;
  TileGeom& geo = lp.geo;
  const int L = int(p.tile_bits.size());
  geo.L = L;
  geo.B = int(cfg.low_bits);
  geo.num_tiles = uint64_t(1) << (s.n - uint32_t(L));
  geo.tensor = 2;
  for (size_t j = 0; j < p.tile_bits.size(); ++j) geo.tile_bits[j] = uint8_t(p.tile_bits[j]);
  std::vector<int> local(s.n, -1);
  for (size_t j = 0; j < p.tile_bits.size(); ++j) local[p.tile_bits[j]] = int(j);

  // Ops on tile bits. A controlled diagonal becomes a diagonal on its
  // controls and targets.
  std::vector<RegOp> ops;
  for (const HOp& op : p.ops) {
    RegOp r;
    if (op.diagonal) {
      std::vector<uint32_t> qs;
      HMatrix full;
      op.full(qs, full);  // qs = controls then targets
      r.entries = full.diagonal_entries();
      for (uint32_t q : qs) {
        const uint32_t ph = s.layout[q];
        r.dtgt_local.push_back(local[ph]);
        r.dtgt_global.push_back(local[ph] >= 0 ? -1 : int(ph));
        if (local[ph] >= 0) r.qmask |= 1u << local[ph];
      }
    } else {
      r.dense = true;
      for (uint32_t q : op.targets) {
        const int l = local[s.layout[q]];
        if (l < 0) throw Error(QVDG_ERR_INVALID, "internal: dense stage gate with a global target");
        r.tgt.push_back(l);
        r.qmask |= 1u << l;
      }
      for (auto& c : op.controls) {
        const uint32_t ph = s.layout[c.first];
        if (local[ph] >= 0) {
          r.local_ctl_mask |= 1u << local[ph];
          if (c.second) r.local_ctl_val |= 1u << local[ph];
          r.qmask |= 1u << local[ph];
        } else {
          r.gcm |= uint64_t(1) << ph;
          if (c.second) r.gcv |= uint64_t(1) << ph;
        }
      }
      r.entries = op.matrix.a;
    }
    ops.push_back(std::move(r));
  }

  // Register passes: one scan in program order takes every op that commutes
  // with all ops skipped before it and, if dense, whose targets fit in the
  // pass's four register bits (grown from the first dense ops).
  struct Pass {
    uint32_t gmask = 0;
    std::vector<size_t> ops;
  };
  std::vector<Pass> passes;
  std::vector<bool> done(ops.size(), false);
  size_t remaining = ops.size();
  while (remaining > 0) {
    Pass ps;
    uint32_t block_dense = 0, block_any = 0;
    for (size_t i = 0; i < ops.size(); ++i) {
      if (done[i]) continue;
      const RegOp& r = ops[i];
      if (r.dense) {
        uint32_t want = ps.gmask;
        for (int b : r.tgt) want |= 1u << b;
        if ((r.qmask & block_any) == 0 && __builtin_popcount(want) <= 4) {
          ps.gmask = want;
          ps.ops.push_back(i);
        } else {
          block_any |= r.qmask;
          block_dense |= r.qmask;
        }
      } else if ((r.qmask & block_dense) == 0) {
        ps.ops.push_back(i);
      } else {
        block_any |= r.qmask;
      }
    }
    for (size_t i : ps.ops) done[i] = true;
    remaining -= ps.ops.size();
    // Fill the register bits up to four with the lowest free tile bits.
    for (int b = 0; b < L && __builtin_popcount(ps.gmask) < 4; ++b) ps.gmask |= 1u << b;
    passes.push_back(std::move(ps));
  }

  // The pass blob: headers, gates, data.
  std::vector<uint8_t> blob(sizeof(RegPassHdr) * passes.size(), 0);
  std::vector<RegGate> gates;
  std::vector<uint8_t> data;  // appended after the gates; offsets fixed up below
  struct Fix {
    size_t gate;
    size_t data_off, table_off;
    bool has_table;
  };
  std::vector<Fix> fixes;
  std::complex<long double> scale = 1.0L;  // product of the sheared gates' divisors so far left out
  auto put_scale = [&] {
    RegGate f{};
    f.op = kOpScale;
    Fix fx{gates.size(), put_complex(data, {C{double(scale.real()), double(scale.imag())}}, s.bits), 0, false};
    gates.push_back(f);
    fixes.push_back(fx);
    scale = 1.0L;
  };
  for (size_t pi = 0; pi < passes.size(); ++pi) {
    const Pass& ps = passes[pi];
    RegPassHdr h{};
    int reg_of[64];
    std::fill(reg_of, reg_of + 64, -1);
    int gi = 0;
    for (int b = 0; b < L; ++b)
      if ((ps.gmask >> b) & 1u) {
        h.g[gi] = uint8_t(b);
        reg_of[b] = gi++;
      }
    h.pair = h.g[0] == 0 ? 1 : 0;
    h.first_gate = uint32_t(gates.size());
    for (size_t oi : ps.ops) {
      const RegOp& r = ops[oi];
      RegGate g{};
      Fix fx{gates.size(), 0, 0, false};
      bool sign_after = false;
      g.gcm = r.gcm;
      g.gcv = r.gcv;
      if (r.dense) {
        g.kind = r.tgt.size() == 1 ? kRegDense1 : kRegDense2;
        // Register controls become the mask of active bases, outside ones a predicate.
        uint32_t rcm = 0, rcv = 0;
        for (int b = 0; b < L; ++b) {
          if (!((r.local_ctl_mask >> b) & 1u)) continue;
          const bool v = (r.local_ctl_val >> b) & 1u;
          if (reg_of[b] >= 0) {
            rcm |= 1u << reg_of[b];
            if (v) rcv |= 1u << reg_of[b];
          } else {
            g.lcm |= 1u << b;
            if (v) g.lcv |= 1u << b;
          }
        }
        std::vector<C> m = r.entries;
        int t0 = reg_of[r.tgt[0]], t1 = r.tgt.size() > 1 ? reg_of[r.tgt[1]] : -1;
        if (t1 >= 0 && t1 < t0) {
          // Swap matrix bits 0 and 1 so that t0 < t1.
          std::vector<C> w(16);
          auto sw = [](int x) { return ((x & 1) << 1) | ((x >> 1) & 1); };
          for (int rr = 0; rr < 4; ++rr)
            for (int cc = 0; cc < 4; ++cc) w[sw(rr) * 4 + sw(cc)] = m[rr * 4 + cc];
          m = w;
          std::swap(t0, t1);
        }
        g.t0 = uint8_t(t0);
        g.t1 = uint8_t(t1 < 0 ? 0 : t1);
        const uint32_t tmask = (1u << t0) | (t1 >= 0 ? 1u << t1 : 0u);
        uint32_t pm = 0;
        for (uint32_t j = 0; j < 16; ++j)
          if (!(j & tmask) && (j & rcm) == rcv) pm |= 1u << j;
        g.pmask = rcm == 0 ? uint16_t(0xffffu) : uint16_t(pm);  // 0xffff: no register controls
        if (g.kind == kRegDense1) {
          const bool everywhere = shear && r.local_ctl_mask == 0 && r.gcm == 0;
          g.spec = dense1_form(m, everywhere, scale, sign_after);
        }
        fx.data_off = put_complex(data, m, s.bits);
      } else {
        const size_t k = r.dtgt_local.size();
        g.k = uint8_t(k);
        uint32_t reg_idx_mask = 0;
        for (size_t i = 0; i < k; ++i) {
          if (r.dtgt_local[i] >= 0) {
            const int b = r.dtgt_local[i];
            if (reg_of[b] >= 0) {
              g.tgt[i] = uint8_t(0x40 | reg_of[b]);
              reg_idx_mask |= 1u << i;
            } else {
              g.tgt[i] = uint8_t(b);
            }
          } else {
            g.tgt[i] = uint8_t(0x80 | r.dtgt_global[i]);
          }
        }
        // Register part of the diagonal index for each register j.
        uint16_t ridx[16];
        for (uint32_t j = 0; j < 16; ++j) {
          uint32_t idx = 0;
          for (size_t i = 0; i < k; ++i)
            if ((reg_idx_mask >> i) & 1u)
              if ((j >> (g.tgt[i] & 0x3f)) & 1u) idx |= 1u << i;
          ridx[j] = uint16_t(idx);
        }
        const bool sign = k <= 4 && std::all_of(r.entries.begin(), r.entries.end(), is_pm_one);
        if (sign) {
          g.kind = kRegSign;
          if (k <= 2 && s.n <= 48) {
            // Index bits from two shifts of (tile base | subcube base << 48);
            // register bits read bit 63, which is always 0.
            auto where = [&](size_t i) -> uint8_t {
              if (i >= k || (g.tgt[i] & 0x40)) return 63;
              if (g.tgt[i] & 0x80) return uint8_t(g.tgt[i] & 0x7f);
              return uint8_t(48 + g.tgt[i]);
            };
            g.kind = kRegSign2;
            g.t0 = where(0);
            g.t1 = where(1);
          }
          // For each value of the non-register index bits: the registers to negate.
          std::vector<uint16_t> masks(size_t(1) << k, 0);
          for (uint32_t f = 0; f < (1u << k); ++f) {
            if (f & reg_idx_mask) continue;
            uint16_t mk = 0;
            for (uint32_t j = 0; j < 16; ++j)
              if (r.entries[f | ridx[j]].re < 0) mk |= uint16_t(1u << j);
            masks[f] = mk;
          }
          fx.data_off = put(data, masks.data(), masks.size());
        } else {
          g.kind = kRegPhase;
          fx.data_off = put_complex(data, r.entries, s.bits);
          fx.table_off = put(data, ridx, 16);
          fx.has_table = true;
        }
      }
      g.pred = (g.gcm != 0 || g.lcm != 0) ? 1 : 0;
      if (g.kind == kRegDense1)
        g.op = uint16_t(g.t0 + (g.spec == kFormGeneral ? kOpDense1
                                                       : (g.spec == kFormX ? kOpX : kOpShear + 4 * (g.spec - kFormReal))));
      else if (g.kind == kRegDense2)
        g.op = kOpDense2;
      else if (g.kind == kRegSign2)
        g.op = kOpSign2;
      else if (g.kind == kRegSign)
        g.op = kOpSign;
      else
        g.op = kOpPhase;
      gates.push_back(g);
      fixes.push_back(fx);
      if (g.op < kOpX && scale_far(scale, s.bits)) put_scale();
      if (sign_after) {
        // Divisors of opposite sign: -1 where the target is 1.
        RegGate z{};
        z.kind = kRegSign2;
        z.op = kOpSign2;
        z.t0 = z.t1 = 63;
        uint16_t mask = 0;
        for (uint32_t j = 0; j < 16; ++j)
          if ((j >> g.t0) & 1u) mask |= uint16_t(1u << j);
        const uint16_t masks[4] = {mask, mask, mask, mask};
        Fix zx{gates.size(), put(data, masks, 4), 0, false};
        gates.push_back(z);
        fixes.push_back(zx);
      }
    }
    if (pi + 1 == passes.size() && scale != std::complex<long double>(1.0L)) put_scale();
    h.num_gates = uint16_t(gates.size() - h.first_gate);
    std::memcpy(blob.data() + pi * sizeof(RegPassHdr), &h, sizeof(h));
  }
  const size_t gates_off = blob.size();  // a multiple of 16
  const size_t data_base = gates_off + gates.size() * sizeof(RegGate);
  for (const Fix& fx : fixes) {
    gates[fx.gate].data = uint32_t(data_base + fx.data_off);
    if (fx.has_table) gates[fx.gate].table = uint32_t(data_base + fx.table_off);
  }
  blob.resize(data_base);
  std::memcpy(blob.data() + gates_off, gates.data(), gates.size() * sizeof(RegGate));
  blob.insert(blob.end(), data.begin(), data.end());
  blob.resize((blob.size() + 15) & ~size_t(15), 0);
  if (blob.size() > kRegBlobBudget) return false;

  up.tc.resize((up.tc.size() + 15) & ~size_t(15), 0);
  geo.tc_offset = up.tc.size();
  geo.tc_bytes = uint32_t(blob.size());
  geo.num_gates = int(passes.size());
  up.tc.insert(up.tc.end(), blob.begin(), blob.end());
  lp.gate_offset = up.gates.size();
  return true;
}

}  // namespace

LoweredPass lower_register_pass(const Target& s, const PlannedPass& p, const StageConfig& cfg, StageUpload& up) {
  // The signs and the factor that sheared gates leave take some room of
  // their own.
  for (const bool shear : {true, false}) {
    LoweredPass lp;
    if (lower_register(s, p, cfg, up, shear, lp)) return lp;
  }
  throw Error(QVDG_ERR_UNSUPPORTED, "internal: register stage program too large");
}

bool register_pass_fits(const Target& s, const PlannedPass& p, const StageConfig& cfg) {
  // At most: a register pass's header, the record and the matrix, or the
  // diagonal with its controls and the index parts, of each gate.
  const size_t elem = s.bits == 32 ? 8 : 16;
  size_t bytes = 0;
  for (const HOp& op : p.ops) {
    const size_t k = op.targets.size();
    const size_t data = op.diagonal ? (elem << (k + op.controls.size())) + 32 : elem << (2 * k);
    bytes += sizeof(RegPassHdr) + sizeof(RegGate) + ((data + 15) & ~size_t(15));
  }
  if (bytes <= kRegBlobBudget) return true;
  // Sheared or not, as lower_register_pass tries them.
  for (const bool shear : {true, false}) {
    LoweredPass lp;
    StageUpload up;
    if (lower_register(s, p, cfg, up, shear, lp)) return true;
  }
  return false;
}

void launch_stage_reg(StateImpl& s, const LoweredPass& lp, const DeviceUpload& dev) {
  const size_t tile_bytes = (s.bits == 32 ? 8 : 16) << lp.geo.L;
  // Two CTAs per SM where they fit beside each other (227 KB of shared
  // memory, a few hundred bytes of each CTA static, 1 KB reserved).
  const int buffers = tile_bytes + lp.geo.tc_bytes + 2048 <= 227 * 1024 / 2 ? 1 : 2;
  const size_t smem = buffers * tile_bytes + lp.geo.tc_bytes;
  // One thread per register subcube, at least one full warp (the set-up
  // loops are strided, so any count works).
  const int cap = s.bits == 32 ? reg_threads<float>() : reg_threads<double>();
  const int threads = std::max(32, std::min(cap, 1 << (lp.geo.L - 4)));
  const uint64_t grid = std::min<uint64_t>(lp.geo.num_tiles, uint64_t(s.sms) * (buffers == 1 ? 2 : 1));
  auto launch = [&](auto* psi, auto kernel, OncePerDevice& once) {
    once(s.device, [&] {
      // Two tiles and the largest program, the most any pass takes.
      QVDG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     int(2 * (size_t(8) << 13) + kRegBlobBudget)));
    });
    kernel<<<unsigned(grid), threads, smem, s.stream>>>(psi, lp.geo, dev.tc, buffers);
  };
  static OncePerDevice once[2];
  if (s.bits == 32)
    launch(static_cast<float2*>(s.amp), k_stage_reg<float>, once[0]);
  else
    launch(static_cast<double2*>(s.amp), k_stage_reg<double>, once[1]);
  QVDG_LAUNCH_CHECK();
}

}  // namespace qvdg
