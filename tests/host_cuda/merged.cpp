// Host time of a merged run and of its gather schedule alone, for
// tests/test_merged_host_time.py.
#include <chrono>
#include <cstdio>

#include "../../qmetal_gb300/csrc/schedule.hpp"
#include "../../qmetal_gb300/csrc/simulator.hpp"

using namespace qmetal;

namespace {

template <typename F>
double best_us(F &&f) {
  double best = 1e30;
  for (int k = 0; k < 50; k++) {
    const auto t0 = std::chrono::steady_clock::now();
    f();
    best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
  }
  return 1e6 * best;
}

}  // namespace

int main() {
  Circuit c;
  c.num_qubits = 21;
  uint32_t x = 1;
  auto random = [&](uint32_t n) { return (x = x * 1664525u + 1013904223u) / 65536u % n; };
  for (int k = 0; k < 400; k++) {
    const uint32_t a = random(21), b = (a + 1 + random(20)) % 21;
    c.add(g2(k % 4 ? G_CX : G_SWAP, a, b));
  }
  const Plan p = build_plan(c);
  Simulator sim(21);
  std::printf("run %d schedule %d\n", static_cast<int>(best_us([&] { sim.run_merged(p); })),
              static_cast<int>(best_us([&] { merged_schedule(p); })));
  return 0;
}
