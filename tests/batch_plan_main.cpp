// Prints a batch's work: reads "L ctas slots" and then "qubits layers" a
// circuit, in the order given.
#include <cstdio>
#include <numeric>

#include "batch_plan.hpp"

int main() {
  int L, ctas;
  unsigned long slots;
  if (std::scanf("%d %d %lu", &L, &ctas, &slots) != 3) return 1;
  std::vector<qvdg::BatchCircuit> circuits;
  unsigned n, layers;
  while (std::scanf("%u %u", &n, &layers) == 2) {
    qvdg::BatchCircuit c{};
    c.num_qubits = n;
    c.num_layers = layers;
    circuits.push_back(c);
  }
  std::vector<uint32_t> order(circuits.size());
  std::iota(order.begin(), order.end(), 0u);
  const qvdg::BatchWork w = qvdg::plan_batch(circuits, order, L, ctas, slots, uint64_t(1) << 24);
  for (size_t i = 0; i < circuits.size(); ++i) {
    if (circuits[i].num_qubits <= unsigned(L)) continue;
    const qvdg::BatchWide& x = w.wide[w.wide_of[i]];
    std::printf("wide %zu %u %llu %d %u %u\n", i, w.wide_of[i], (unsigned long long)(x.slot >> 24), x.previous,
                x.phases, x.tiles);
  }
  for (const qvdg::BatchTask& t : w.tasks) std::printf("task %u %u %u %u\n", t.circuit, t.phase, t.tile, t.count);
}
