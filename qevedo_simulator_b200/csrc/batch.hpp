// Batched layered circuits (one persistent launch for many small circuits).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "qvdg.h"

namespace qvdg {

constexpr int kBatchMaxQubits = QVDG_BATCH_MAX_QUBITS;

// One circuit of the batch on the device.
struct BatchCircuit {
  uint32_t num_qubits, num_layers, entangler;
  uint32_t form;   // kBatchShear | kBatchRight, or 0: generic 2x2 matrices
  uint64_t gates;  // index of its first gate record (kBatchGateSlots complex64 each) in the gate buffer
  uint64_t out;    // index of its first <Z> output
  uint32_t wide;   // its BatchWide, where it is wider than the tile
  uint32_t reserved;
};

// A circuit wider than the shared-memory tile, for one tile shape.
struct BatchWide {
  uint64_t slot, partials;  // first amplitude of its slot, first of its tiles' sums
  uint32_t tiles;           // of a pass
  uint32_t phases;          // tile passes: A and B in turn
  uint32_t layers;          // of an A and a B pass together
  int32_t previous;         // the wide circuit with layers that had the slot before (-1: none)
  int32_t tile_bits, low, high;  // tile qubits; pass B's low qubits and first high one
  int32_t reserved;
  // Tiles of the circuit that are done before phase p begins (the first A
  // pass runs its tile 0 alone).
  __host__ __device__ uint32_t before(uint32_t p) const { return p == 0 ? 0 : 1 + (p - 1) * tiles; }
};

// A piece of work: a whole circuit, or `count` tiles from `tile` of a wide
// circuit's tile pass `phase` (phase = its number of passes: the results).
struct BatchTask {
  uint32_t circuit, phase, tile, count;
};

// A gate record: the 2x2 matrix (m00, m01, m10, m11) in slots 0-3 for a
// generic circuit. For a sheared one U = diag(p0, p1) R diag(q0, q1) with R
// real, its rows divided by their larger entries: slots (a, b), (off, 0),
// p0, p1, q0, q1, where R maps (x0, x1) to (x0 + a x1, x1 + b x0), or, off
// set, to (x1 + a x0, x0 + b x1).
constexpr int kBatchGateSlots = 6;
constexpr uint32_t kBatchShear = 1, kBatchRight = 2;

// Everything one launch of the batch kernel reads.
struct BatchLaunch {
  const BatchCircuit* circuits = nullptr;
  const BatchWide* wide = nullptr;
  const BatchTask* tasks = nullptr;  // in the order CTAs take them
  uint32_t count = 0;
  const float2* gates = nullptr;
  float2* slots = nullptr;      // HBM states of wide circuits
  double* partials = nullptr;   // their last pass's sums per tile
  double* out = nullptr;
  // Reset by each launch (queue_bytes from `queue` on): the work counter,
  // the give-up status, and each wide circuit's count of tiles done.
  uint32_t* queue = nullptr;
  int* status = nullptr;
  uint32_t* done = nullptr;
  size_t queue_bytes = 0;
  int tile_qubits = 13;
  int threads = 256;
  int ctas = 0;
};

// Resident CTAs per SM of the batch kernel for a shape (0 if it cannot run).
int batch_kernel_occupancy(int threads, int tile_qubits);
// Write the circuits' gate records and forms from their matrices (2x2
// complex128, one circuit after another) on the device.
void launch_batch_encode(const BatchLaunch& b, const double* matrices, uint32_t circuits, cudaStream_t stream);
// Reset the work counter and launch the persistent kernel on `stream`.
void launch_batch(const BatchLaunch& b, cudaStream_t stream);

}  // namespace qvdg

// Host side (batch_host.cpp), called by the C ABI in api.cpp.
namespace qvdg {
qvdg_batch* batch_create(const qvdg_layered_circuit* circuits, size_t count, const qvdg_batch_options* options);
void batch_destroy(qvdg_batch* b);
void batch_set_gates(qvdg_batch* b, const double* gates, size_t num_matrices);
void batch_run(qvdg_batch* b, double* expect_z, size_t count, double* seconds);
void batch_info(const qvdg_batch* b, qvdg_batch_summary* info);
size_t batch_tuning(const qvdg_batch* b, uint32_t* tile_qubits, uint32_t* threads, double* seconds, size_t capacity);
}  // namespace qvdg
