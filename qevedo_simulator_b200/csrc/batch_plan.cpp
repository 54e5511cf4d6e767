// The order of a batch's work: which slot each circuit wider than a tile takes,
// and the tile passes as tasks.

#include "batch_plan.hpp"

#include <algorithm>

namespace qvdg {

namespace {

constexpr uint32_t kMaxDepth = 5;  // layers of an A and B pass (their tables fit the kernel's steps)
constexpr uint64_t kPartialRow = 16;  // doubles per tile

// Wide circuits run on tiles of 13 qubits (the largest tile leaves two of
// them per CTA, so that copies fly under the computation), or the tile's own
// 12. Pass B keeps 2^r contiguous amplitudes: 64 bytes, or a 32-byte sector
// where that lets an A and B pass take a layer more.
void wide_shape(uint32_t n, int L, BatchWide& w) {
  w.tile_bits = std::min(L, 13);
  w.low = 2 * w.tile_bits - 3 - int(n) >= 2 ? 3 : 2;
  w.high = int(n) - (w.tile_bits - w.low);
  w.layers = std::min<uint32_t>(uint32_t(w.tile_bits - w.high) + 1, kMaxDepth);
  w.tiles = uint32_t(1) << (n - uint32_t(w.tile_bits));
}

}  // namespace

size_t wide_count(const std::vector<BatchCircuit>& circuits, const std::vector<uint32_t>& order, int L) {
  size_t k = 0;
  for (uint32_t i : order) k += circuits[i].num_qubits > uint32_t(L);
  return k;
}

BatchWork plan_batch(const std::vector<BatchCircuit>& circuits, const std::vector<uint32_t>& order, int L, int ctas,
                     size_t slots, uint64_t slot_elems) {
  BatchWork w;
  w.wide_of.assign(circuits.size(), 0);
  std::vector<uint32_t> wide;  // circuits, largest first as in `order`
  // Those of them that hold a slot, in turn. A circuit without layers is
  // |0...0>: its results wait for nobody, so it must not stand between a
  // slot's holders, who wait only for the one before them.
  std::vector<uint32_t> holders;
  uint64_t pass_tiles = 0;
  for (uint32_t i : order)
    if (circuits[i].num_qubits > uint32_t(L)) {
      BatchWide x{};
      const uint32_t k = uint32_t(wide.size());
      wide_shape(circuits[i].num_qubits, L, x);
      x.phases = 2 * ((circuits[i].num_layers + x.layers - 1) / x.layers);
      x.previous = -1;
      if (x.phases) {
        const size_t h = holders.size();
        x.slot = (h % slots) * slot_elems;
        if (h >= slots) x.previous = int32_t(holders[h - slots]);
        if (h < slots) pass_tiles += x.tiles;
        holders.push_back(k);
      }
      x.partials = w.partials;
      w.partials += uint64_t(x.tiles) * kPartialRow;
      w.wide_of[i] = k;
      w.wide.push_back(x);
      wide.push_back(i);
    }
  // Tiles of a task: several where that still leaves every CTA a few tasks
  // of each pass (a task builds its gate tables once).
  uint32_t grain = 1;
  while (grain < 8 && pass_tiles >= uint64_t(grain) * 2 * 6 * uint64_t(ctas)) grain *= 2;
  for (size_t first = 0; first < wide.size(); first += slots) {
    const size_t end = std::min(wide.size(), first + slots);
    uint32_t phases = 0;
    for (size_t k = first; k < end; ++k) phases = std::max(phases, w.wide[k].phases);
    for (uint32_t p = 0; p <= phases; ++p)
      for (size_t k = first; k < end; ++k) {
        const BatchWide& x = w.wide[k];
        if (p > x.phases) continue;
        if (p == x.phases || p == 0) {
          w.tasks.push_back({wide[k], p, 0, 1});
          continue;
        }
        const uint32_t g = std::min(grain, x.tiles);
        for (uint32_t t = 0; t < x.tiles; t += g) w.tasks.push_back({wide[k], p, t, g});
      }
  }
  for (uint32_t i : order)
    if (circuits[i].num_qubits <= uint32_t(L)) w.tasks.push_back({i, 0, 0, 1});
  return w;
}

}  // namespace qvdg
