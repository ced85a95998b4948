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
  const Circuit wide = ladders(20), narrow = ladders(std::strcmp(what, "narrow") ? 16 : 12);
  Hamiltonian h;
  h.add(1.0, PauliString::single('Z', 0));
  std::vector<double> g0(wide.size()), g1(narrow.size());
  std::vector<BatchItem> items(2);
  items[0].circuit = &wide;
  items[0].grad = g0.data();
  items[1].circuit = &narrow;
  items[1].grad = g1.data();
  for (BatchItem &it : items) it.hamiltonian = &h;
  if (!std::strcmp(what, "pinned")) fake::fail_pinned = 1;
  // The lane's memory, 2 GiB of headroom, and room for a second buffer of 16
  // qubits (512 KiB) but not of 20 (8 MiB).
  if (!std::strcmp(what, "scratch"))
    fake::total = Simulator::lane_device_bytes(20, wide.size(), 0) + (size_t(2) << 30) + (4u << 20);
  run_batch(items, BatchMode::Lanes, 1);
  std::printf("wide %d narrow %d held %zu left %zu small %d overlaps %d\n",
              fake::permutations[20], fake::permutations[16], fake::used_after_failed_pinned,
              fake::used, fake::small_runs, fake::overlaps);
  return 0;
}
