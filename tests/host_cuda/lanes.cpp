// A batch's lanes with little memory: prints what tests/test_lane_memory.py reads.
#include <cstdio>
#include <cstring>

#include "../../qmetal_gb300/csrc/batch.hpp"
#include "../../qmetal_gb300/csrc/simulator.hpp"
#include "fake_device.hpp"

using namespace qmetal;

namespace {

Circuit ladders(uint32_t n) {
  Circuit c;
  c.num_qubits = n;
  for (int layer = 0; layer < 3; layer++) {
    for (uint32_t q = 0; q < n; q++) c.add(g1p(G_RY, q, 0.1 + q));
    for (uint32_t q = 0; q + 1 < n; q++) c.add(g2(G_CX, q, q + 1));
  }
  return c;
}

}  // namespace

int main(int argc, char **argv) {
  const char *what = argc > 1 ? argv[1] : "";
  auto mode = [&](const char *m) { return std::strcmp(what, m) == 0; };
  if (mode("create")) {   // device memory of a simulator of 12 qubits, and after a run and a gradient
    Simulator sim(12);
    const size_t made = fake::used;
    const Circuit c = ladders(12);
    Hamiltonian h;
    h.add(1.0, PauliString::single('Z', 0));
    sim.run(c);
    const size_t ran = fake::used;
    sim.energy_and_gradient(c, h);
    std::printf("made %zu ran %zu gradient %zu small %d overlaps %d\n", made, ran, fake::used,
                fake::small_runs, fake::overlaps);
    return 0;
  }
  std::vector<uint32_t> widths = {20, 16};
  if (mode("narrow")) widths = {20, 13, 12, 12, 11, 6, 1};
  std::vector<Circuit> circuits;
  for (uint32_t n : widths) circuits.push_back(ladders(n));
  Hamiltonian h;
  h.add(1.0, PauliString::single('Z', 0));
  std::vector<std::vector<double>> grads;
  std::vector<BatchItem> items(widths.size());
  for (const Circuit &c : circuits) grads.emplace_back(c.size());
  for (size_t k = 0; k < items.size(); k++) {
    items[k].circuit = &circuits[k];
    items[k].hamiltonian = &h;
    items[k].grad = grads[k].data();
  }
  if (mode("pinned")) fake::fail_pinned = 1;
  // The lane's memory, 2 GiB of headroom, and room for a second buffer of 16
  // qubits (512 KiB) but not of 20 (8 MiB).
  if (mode("scratch"))
    fake::total = Simulator::lane_device_bytes(20, circuits[0].size(), 0) + (size_t(2) << 30) + (4u << 20);
  run_batch(items, BatchMode::Lanes, 1);
  std::printf("wide %d narrow %d held %zu left %zu small %d overlaps %d\n",
              fake::permutations[20], fake::permutations[16], fake::used_after_failed_pinned,
              fake::used, fake::small_runs, fake::overlaps);
  return 0;
}
