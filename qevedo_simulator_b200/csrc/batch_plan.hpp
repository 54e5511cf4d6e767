// The order of a batch's work (host only).
#pragma once

#include <cstddef>
#include <vector>

#include "batch.hpp"

namespace qvdg {

// The work of a set of circuits on tiles of L qubits, in the order CTAs take
// it: waves of wide circuits, as many as there are slots, each wave pass by
// pass; then the circuits that fit a tile.
struct BatchWork {
  std::vector<BatchWide> wide;
  std::vector<uint32_t> wide_of;  // per circuit
  std::vector<BatchTask> tasks;
  uint64_t partials = 0;          // doubles
};

// Circuits of `order` wider than a tile of L qubits.
size_t wide_count(const std::vector<BatchCircuit>& circuits, const std::vector<uint32_t>& order, int L);

// `slots` >= 1 slots of `slot_elems` amplitudes hold the wide circuits' states.
BatchWork plan_batch(const std::vector<BatchCircuit>& circuits, const std::vector<uint32_t>& order, int L, int ctas,
                     size_t slots, uint64_t slot_elems);

}  // namespace qvdg
