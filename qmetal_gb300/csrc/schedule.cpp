// schedule.cpp -- merged forward, co-state and backward-sweep schedules.
#include "schedule.hpp"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <map>
#include <stdexcept>

namespace qmetal {
namespace {

uint32_t popc(uint64_t x) { return static_cast<uint32_t>(__builtin_popcountll(x)); }

constexpr uint32_t kWindowOps = 16;     // ops per window pass below 6 qubits
constexpr uint32_t kWideWindowOps = 32;  // ops per warp-tile window pass
constexpr uint32_t kWindowGrads = 16;   // gradients per window pass
// ... and in the compile-time tile of wire 0, wires 1..5 and four wires >= 6
// that all carry RZ then RY (undo order): the first tile of a
// hardware-efficient layer.
constexpr uint32_t kWideUniformGrads = 20;
constexpr uint32_t kSigRzRy = 6;          // uniform_signature of RZ then RY

// The structure the kernel layer finds in a 2x2 once narrowed to float (the
// kMat* classes of kcommon.cuh): 3 diagonal, 1 real, 2 RX-like, 0 general.
int narrowed_class(const cdouble m[4]) {
  float f[8];
  for (int k = 0; k < 4; k++) {
    f[2 * k] = static_cast<float>(m[k].real());
    f[2 * k + 1] = static_cast<float>(m[k].imag());
  }
  if (f[2] == 0.0f && f[3] == 0.0f && f[4] == 0.0f && f[5] == 0.0f) return 3;
  if (f[1] == 0.0f && f[3] == 0.0f && f[5] == 0.0f && f[7] == 0.0f) return 1;
  if (f[1] == 0.0f && f[7] == 0.0f && f[2] == 0.0f && f[4] == 0.0f) return 2;
  return 0;
}

}  // namespace

Affine::Affine(uint32_t n) : cols(n) {
  for (uint32_t j = 0; j < n; j++) cols[j] = 1ull << j;
}

void Affine::then_cx(uint32_t c, uint32_t t) {
  auto f = [&](uint64_t v) { return v ^ (((v >> c) & 1ull) << t); };
  for (uint64_t &v : cols) v = f(v);
  off = f(off);
}

void Affine::then_swap(uint32_t a, uint32_t b) {
  auto f = [&](uint64_t v) {
    const uint64_t d = ((v >> a) ^ (v >> b)) & 1ull;
    return v ^ (d << a) ^ (d << b);
  };
  for (uint64_t &v : cols) v = f(v);
  off = f(off);
}

uint32_t Affine::sectors() const {
  std::vector<uint64_t> s;
  for (uint64_t y = 0; y < 64 && y < (1ull << cols.size()); y++) {
    uint64_t x = off;
    for (uint32_t j = 0; j < cols.size() && j < 6; j++)
      if ((y >> j) & 1) x ^= cols[j];
    s.push_back(x >> 2);
  }
  std::sort(s.begin(), s.end());
  return static_cast<uint32_t>(std::unique(s.begin(), s.end()) - s.begin());
}

// Every gate of a run is an involution, so undoing the run composes its gates
// first to last, and applying it composes them last to first.
Affine run_map(uint32_t n, const std::vector<PermGate> &run, bool undo) {
  Affine m(n);
  auto step = [&](const PermGate &g) {
    if (g.swap) m.then_swap(g.a, g.b);
    else m.then_cx(g.a, g.b);
  };
  if (undo) {
    for (const PermGate &g : run) step(g);
  } else {
    for (size_t k = run.size(); k-- > 0;) step(run[k]);
  }
  return m;
}

// A gather pass moves 2S, more when the warp's sources scatter; the run's
// gates move S each (half the state read and written per CX, all of it
// crossing for a SWAP, counted as S by the roofline model).
bool permutation_pays(const Affine &m, size_t gates) {
  const double pass = 2.0 * std::max(1.0, m.sectors() / 16.0);
  return pass * 1.25 < static_cast<double>(gates);
}

Gate invert(const Gate &g) {
  Gate inv = g;
  switch (g.kind) {
    case G_RX: case G_RY: case G_RZ: case G_P: case G_CP:
      inv.params[0] = -g.params[0];
      break;
    case G_S: inv.kind = G_SDG; break;
    case G_SDG: inv.kind = G_S; break;
    case G_T: inv.kind = G_TDG; break;
    case G_TDG: inv.kind = G_T; break;
    case G_U3:   // U3(t, f, l)^-1 = U3(-t, -l, -f)
      inv.params[0] = -g.params[0];
      inv.params[1] = -g.params[2];
      inv.params[2] = -g.params[1];
      break;
    default: break;
  }
  return inv;
}

int generator_of(const Gate &g) {
  switch (g.kind) {
    case G_RX: return 1;
    case G_RY: return 2;
    case G_RZ: return 3;
    default: return 0;
  }
}

// ---------------------------------------------------------------------------

namespace {

// Wires 0..5 (wire 0 apart), and wires >= 6, that one group pass may hold.
bool group_fits(uint32_t n, bool zero, size_t lane, size_t high) {
  (void)zero;
  if (lane >= 1 && high <= 4 && n >= 6 + high) return true;
  if (lane == 0 && high >= 6 && high <= 7 && n >= 6 + high) return true;   // block groups
  return lane + high <= 5;
}

// Most wires >= 6 one pass of such wires alone may hold.
uint32_t high_cap(uint32_t n) { return n >= 13 ? 7 : n >= 12 ? 6 : 5; }

// One-wire ops on distinct wires, not yet issued.
struct WireRun {
  std::vector<uint32_t> wires;
  std::vector<cdouble> mats;
  bool holds(uint32_t q) const { return std::find(wires.begin(), wires.end(), q) != wires.end(); }
  void add(uint32_t q, const cdouble *m) {
    wires.push_back(q);
    mats.insert(mats.end(), m, m + 4);
  }
  void clear() {
    wires.clear();
    mats.clear();
  }
};

// The run's ops (they all commute) as the fewest group passes: wires 0..5
// take k wires >= 6 along, the rest go up to seven a pass in order. Where a
// lane wire's matrix is general, the pass of the lane wires is bound by its
// multiply-adds: of the k that give the fewest passes the least is kept, but
// at least one where there is one (a pass of the lane wires alone has too
// little work per thread to hide its loads), so an HEA layer at 28 qubits
// goes as 6 + 1, 7, 7, 7 wires instead of 6 + 4, 7, 7, 4. Narrow matrices
// (real, RX-like, diagonal) halve the lane pass's multiply-adds: it then
// keeps as many wires >= 6 as fit. Returns each pass's entries of the run.
std::vector<std::vector<size_t>> split_run(uint32_t n, const WireRun &run) {
  std::vector<size_t> low, high;
  for (size_t i = 0; i < run.wires.size(); i++) (run.wires[i] < 6 ? low : high).push_back(i);
  size_t lane = 0;
  bool zero = false, general = false;
  for (size_t i : low) {
    if (run.wires[i] == 0) zero = true;
    else lane++;
    general = general || narrowed_class(&run.mats[4 * i]) == 0;
  }
  const size_t cap = high_cap(n);
  size_t best_k = 0, best = SIZE_MAX;
  for (size_t k = low.empty() ? 0 : std::min<size_t>(1, high.size()); k <= high.size(); k++) {
    const bool some = !low.empty() || k > 0;
    if (some && !group_fits(n, zero, lane, k)) break;
    const size_t passes = (some ? 1 : 0) + (high.size() - k + cap - 1) / cap;
    if (passes < best || (!general && passes == best)) {
      best = passes;
      best_k = k;
    }
  }
  std::vector<std::vector<size_t>> out;
  std::vector<size_t> first = low;
  first.insert(first.end(), high.begin(), high.begin() + best_k);
  if (!first.empty()) out.push_back(std::move(first));
  for (size_t j = best_k; j < high.size(); j += cap)
    out.emplace_back(high.begin() + j, high.begin() + std::min(high.size(), j + cap));
  for (auto &pass : out)
    std::sort(pass.begin(), pass.end(),
              [&](size_t a, size_t b) { return run.wires[a] < run.wires[b]; });
  return out;
}

ForwardStep group_step(const WireRun &run, const std::vector<size_t> &idx) {
  ForwardStep s;
  s.kind = ForwardStep::Group;
  for (size_t i : idx) s.wires.push_back(run.wires[i]);
  s.mats.reserve(4 * idx.size());
  for (size_t i : idx)
    s.mats.insert(s.mats.end(), run.mats.begin() + 4 * i, run.mats.begin() + 4 * i + 4);
  return s;
}

// A plan op that only moves amplitudes between two wires.
bool is_wire_move(const PlanOp &op, uint32_t n) {
  const bool cx = op.kind == PlanOp::Kind::Controlled1q && op.matrix[0] == 0.0 &&
                  op.matrix[1] == 1.0 && op.matrix[2] == 1.0 && op.matrix[3] == 0.0;
  return (cx || op.kind == PlanOp::Kind::Swap) && op.qubits[0] < n && op.qubits[1] < n &&
         op.qubits[0] != op.qubits[1];
}

// The wires and matrices of a one-qubit plan op; false for any other op.
bool one_wire_op(const PlanOp &op, uint32_t n, const uint32_t *&wires, const cdouble *&mats,
                 size_t &count) {
  if (op.kind == PlanOp::Kind::Dense1q) {
    wires = op.qubits;
    mats = op.matrix;
    count = 1;
  } else if (op.kind == PlanOp::Kind::Dense1qGroup) {
    wires = op.group_qubits.data();
    mats = op.group_matrices.data();
    count = op.group_qubits.size();
  } else {
    return false;
  }
  for (size_t j = 0; j < count; j++)
    if (wires[j] >= n) throw std::runtime_error("qubit index out of range");
  return true;
}

}  // namespace

std::vector<ForwardStep> merged_schedule(const Plan &p) {
  const uint32_t n = p.num_qubits;
  std::vector<ForwardStep> out;
  WireRun held;
  auto flush = [&]() {
    if (held.wires.empty()) return;
    for (const auto &pass : split_run(n, held)) out.push_back(group_step(held, pass));
    held.clear();
  };
  std::vector<PermGate> run;
  std::vector<size_t> run_ops;
  auto flush_run = [&]() {
    if (run.empty()) return;
    const Affine map = run.size() >= 2 ? run_map(n, run, false) : Affine(0);
    if (run.size() >= 2 && permutation_pays(map, run.size())) {
      ForwardStep s;
      s.kind = ForwardStep::Permute;
      s.cols = map.cols;
      s.off = map.off;
      s.ops = run_ops;
      out.push_back(std::move(s));
    } else {
      for (size_t i : run_ops) {
        ForwardStep s;
        s.ops = {i};
        out.push_back(std::move(s));
      }
    }
    run.clear();
    run_ops.clear();
  };
  for (size_t i = 0; i < p.ops.size(); i++) {
    const PlanOp &op = p.ops[i];
    if (is_wire_move(op, n)) {
      flush();
      run.push_back({op.kind == PlanOp::Kind::Swap, op.qubits[0], op.qubits[1]});
      run_ops.push_back(i);
      continue;
    }
    flush_run();
    const uint32_t *w = nullptr;
    const cdouble *m = nullptr;
    size_t count = 0;
    if (!one_wire_op(op, n, w, m, count)) {
      flush();
      ForwardStep s;
      s.ops = {i};
      out.push_back(std::move(s));
      continue;
    }
    bool overlap = false;
    for (size_t j = 0; j < count; j++) overlap = overlap || held.holds(w[j]);
    if (overlap) flush();
    // The group's wires commute with each other and with the pending ones:
    // they join the pending run, which is split into passes when it ends.
    for (size_t j = 0; j < count; j++) held.add(w[j], m + 4 * j);
  }
  flush();
  flush_run();
  return out;
}

// ---------------------------------------------------------------------------

namespace {

// One way to issue a pending run of one-wire ops and the CX / SWAP gates that
// follow it: passes of at most `cap` wires >= 6 each (at most four beside
// wires 0..5), every pass with the gates, in order, that it holds both wires
// of and that no gate left for later has a wire of. Empty where that takes
// `most` passes or more.
std::vector<ForwardStep> move_passes(const WireRun &held, const std::vector<PermGate> &run,
                                     const std::vector<size_t> &run_ops, uint32_t cap,
                                     size_t most) {
  std::vector<ForwardStep> out;
  std::vector<size_t> todo(run.size());   // the run's gates not yet in a pass
  for (size_t k = 0; k < todo.size(); k++) todo[k] = k;
  std::vector<bool> wire_done(held.wires.size(), false);
  size_t wires_left = held.wires.size();
  uint64_t used = 0;   // by any gate
  for (const PermGate &g : run) used |= (1ull << g.a) | (1ull << g.b);
  while (!todo.empty() || wires_left) {
    if (out.size() + 1 >= most) return {};
    uint64_t tile = 0, blocked = 0;
    uint32_t high = 0;
    bool low = false;
    auto admit = [&](uint64_t wires) {
      uint32_t add = 0;
      bool lo = low;
      for (uint64_t m = wires & ~tile; m; m &= m - 1) {
        if (__builtin_ctzll(m) < 6) lo = true;
        else add++;
      }
      if (high + add > (lo ? std::min(cap, 4u) : cap)) return false;
      tile |= wires;
      high += add;
      low = lo;
      return true;
    };
    // Wires that a further gate of this pass could have: gates after the point
    // where there are fewer than two need no look.
    auto usable = [&]() {
      uint64_t m = tile;
      if (high < (low ? std::min(cap, 4u) : cap)) m |= ~63ull;
      if (high <= std::min(cap, 4u)) m |= 63ull;
      return m & ~blocked;
    };
    ForwardStep s;
    s.kind = ForwardStep::Moves;
    size_t at = 0, left = 0;
    for (; at < todo.size(); at++) {
      const size_t k = todo[at];
      const uint64_t w = (1ull << run[k].a) | (1ull << run[k].b);
      if ((w & blocked) || !admit(w)) {
        blocked |= w;
        todo[left++] = k;
        if (popc(usable() & used) < 2) {
          at++;
          break;
        }
        continue;
      }
      s.moves.push_back(run[k]);
      s.ops.push_back(run_ops[k]);
    }
    todo.erase(todo.begin() + left, todo.begin() + at);
    std::vector<size_t> idx;
    for (size_t i = 0; i < held.wires.size(); i++) {
      if (wire_done[i] || !admit(1ull << held.wires[i])) continue;
      wire_done[i] = true;
      idx.push_back(i);
      wires_left--;
    }
    std::sort(idx.begin(), idx.end(),
              [&](size_t a, size_t b) { return held.wires[a] < held.wires[b]; });
    ForwardStep g = group_step(held, idx);
    s.wires = std::move(g.wires);
    s.mats = std::move(g.mats);
    if (s.moves.empty()) s.kind = ForwardStep::Group;
    out.push_back(std::move(s));
  }
  return out;
}

}  // namespace

namespace {

// The wires every mask of a diagonal layer holds, if it is a fan: one or two
// wires a mask, finite angles, no constant phase. 0 otherwise.
uint64_t fan_centres(const PlanOp &op, uint32_t n) {
  if (op.kind != PlanOp::Kind::DiagonalLayer || op.global_phase != 0.0 || op.masks.empty() ||
      op.angles.size() != op.masks.size())
    return 0;
  uint64_t common = ~0ull;
  for (size_t t = 0; t < op.masks.size(); t++) {
    const uint64_t m = op.masks[t];
    // (angles that a sum with others of their wire keeps finite)
    if (popc(m) < 1 || popc(m) > 2 || (m >> n) || !(std::abs(op.angles[t]) <= 1e300)) return 0;
    common &= m;
  }
  return common;
}

// The longest pass of stages from plan op `first` on. Returns the plan ops it
// takes, 0 where they are better off by themselves.
size_t match_stages(const Plan &p, size_t first, ForwardStep &step) {
  const uint32_t n = p.num_qubits;
  step = ForwardStep{};
  step.kind = ForwardStep::Stages;
  std::vector<Stage> &st = step.stages;
  uint64_t held = 0;
  uint32_t high = 0;
  bool low = false;
  double alone = 0.0;   // in S
  auto open = [&](uint32_t w) {
    if ((held >> w) & 1ull) return false;
    if (w >= 6 ? low || high == 7 : high > 4) return false;
    held |= 1ull << w;
    if (w >= 6) high++;
    else low = true;
    st.emplace_back();
    st.back().wire = w;
    return true;
  };
  size_t k = first;
  for (; k < p.ops.size(); k++) {
    const PlanOp &op = p.ops[k];
    if (op.kind == PlanOp::Kind::Dense1q) {
      const uint32_t w = op.qubits[0];
      if (w >= n) break;
      const bool joins = !st.empty() && st.back().wire == w && !st.back().has_matrix;
      if (!joins && !open(w)) break;
      st.back().has_matrix = true;
      std::copy(op.matrix, op.matrix + 4, st.back().m);
      alone += 2.0;
      continue;
    }
    const uint64_t centres = fan_centres(op, n);
    if (!centres) break;
    const bool after = !st.empty() && st.back().phase == 0 && ((centres >> st.back().wire) & 1ull);
    if (!after && !open(static_cast<uint32_t>(63 - __builtin_clzll(centres)))) break;
    Stage &s = st.back();
    s.phase = after ? 1 : 2;
    s.angles.assign(n, 0.0);
    for (size_t t = 0; t < op.masks.size(); t++) {
      const uint64_t other = op.masks[t] & ~(1ull << s.wire);
      s.angles[other ? static_cast<uint32_t>(__builtin_ctzll(other)) : s.wire] += op.angles[t];
    }
    alone += op.masks.size() == 1 ? 0.5 : 1.0;
  }
  for (size_t i = first; i < k; i++) step.ops.push_back(i);
  return alone >= 4.0 && st.size() >= 2 ? k - first : 0;
}

}  // namespace

namespace {

double step_cost(const Plan &p, const ForwardStep &st) {
  if (st.kind == ForwardStep::Stages) return 2.7;
  if (st.kind != ForwardStep::Op) return 2.0;
  const PlanOp &op = p.ops[st.ops[0]];
  const bool half = op.kind == PlanOp::Kind::Controlled1q || op.kind == PlanOp::Kind::Swap ||
                    fan_centres(op, p.num_qubits) != 0;
  return op.kind == PlanOp::Kind::CCX ? 0.5 : half ? 1.0 : 2.0;
}

}  // namespace

double schedule_cost(const Plan &p, const std::vector<ForwardStep> &steps) {
  double cost = 0.0;
  for (const ForwardStep &st : steps) cost += step_cost(p, st);
  return cost;
}

namespace {

// inplace_schedule() before diagonal layers take wires along; false, with `out`
// unfinished, once it costs `most` or more.
bool inplace_steps(const Plan &p, double most, std::vector<ForwardStep> &out) {
  const uint32_t n = p.num_qubits;
  double spent = 0.0;
  auto emit = [&](ForwardStep &&s) {
    spent += step_cost(p, s);
    out.push_back(std::move(s));
  };
  WireRun held;
  std::vector<PermGate> run;
  std::vector<size_t> run_ops;
  auto flush = [&]() {
    // A long run in pieces, which keeps the search for passes linear in it.
    for (size_t from = 0; from < run.size() || !held.wires.empty(); from += kMovesPiece) {
      const size_t to = std::min(run.size(), from + kMovesPiece);
      const std::vector<PermGate> piece(run.begin() + from, run.begin() + to);
      const std::vector<size_t> ops(run_ops.begin() + from, run_ops.begin() + to);
      const auto groups = split_run(n, held);
      // A pass reads and writes the state (2 S); a CX or SWAP of its own moves S.
      std::vector<ForwardStep> best;
      if (!piece.empty() && n >= kMovesMinQubits) {
        double passes = static_cast<double>(groups.size() + piece.size() / 2 + 1);
        passes = std::min(passes, std::max(0.0, std::ceil((most - spent) / 2.0)));
        size_t fewer = static_cast<size_t>(passes);   // than so many
        for (uint32_t cap = 4; cap <= 7; cap++) {
          std::vector<ForwardStep> t = move_passes(held, piece, ops, cap, fewer);
          if (t.empty()) continue;
          fewer = t.size();
          best = std::move(t);
        }
      }
      if (!best.empty()) {
        for (ForwardStep &s : best) emit(std::move(s));
      } else {
        if (spent + 2.0 * groups.size() + piece.size() >= most) return false;
        for (const auto &pass : groups) emit(group_step(held, pass));
        for (size_t i : ops) {
          ForwardStep s;
          s.ops = {i};
          emit(std::move(s));
        }
      }
      held.clear();
    }
    run.clear();
    run_ops.clear();
    return spent < most;
  };
  for (size_t i = 0; i < p.ops.size(); i++) {
    const PlanOp &op = p.ops[i];
    ForwardStep stages;
    if (n >= kStagesMinQubits && i + 1 < p.ops.size() &&
        (op.kind == PlanOp::Kind::Dense1q || op.kind == PlanOp::Kind::DiagonalLayer)) {
      if (const size_t taken = match_stages(p, i, stages)) {
        if (!flush()) return false;
        emit(std::move(stages));
        i += taken - 1;
        continue;
      }
    }
    if (is_wire_move(op, n)) {
      run.push_back({op.kind == PlanOp::Kind::Swap, op.qubits[0], op.qubits[1]});
      run_ops.push_back(i);
      continue;
    }
    const uint32_t *w = nullptr;
    const cdouble *m = nullptr;
    size_t count = 0;
    if (!one_wire_op(op, n, w, m, count)) {
      if (!flush()) return false;
      ForwardStep s;
      s.ops = {i};
      emit(std::move(s));
      continue;
    }
    bool later = !run.empty();
    for (size_t j = 0; j < count; j++) later = later || held.holds(w[j]);
    if (later && !flush()) return false;
    for (size_t j = 0; j < count; j++) held.add(w[j], m + 4 * j);
  }
  return flush();
}

// Does inplace_schedule() do anything that merged_schedule() does not: carry
// moves, or take single gates and fans as stages?
bool inplace_differs(const Plan &p) {
  bool before = false;   // a single gate or a fan was the last op
  for (const PlanOp &op : p.ops) {
    if (is_wire_move(op, p.num_qubits)) return true;
    const bool stage = op.kind == PlanOp::Kind::Dense1q || fan_centres(op, p.num_qubits) != 0;
    if (stage && before) return true;
    before = stage;
  }
  return false;
}

}  // namespace

std::vector<ForwardStep> inplace_schedule(const Plan &p) {
  std::vector<ForwardStep> out;
  inplace_steps(p, HUGE_VAL, out);
  return fold_diagonals(p, std::move(out));
}

namespace {

// The runs that a plan falls into, each of single gates and then CX / SWAP moves,
// or one other op; counted as far as most + 1.
size_t plan_runs(const Plan &p, size_t most) {
  enum { None, Single, Move } last = None;
  size_t runs = 0;
  for (const PlanOp &op : p.ops) {
    if (runs > most) break;
    if (is_wire_move(op, p.num_qubits)) {
      runs += last == None;
      last = Move;
    } else if (op.kind == PlanOp::Kind::Dense1q || op.kind == PlanOp::Kind::Dense1qGroup) {
      runs += last != Single;
      last = Single;
    } else {
      runs++;
      last = None;
    }
  }
  return runs;
}

}  // namespace

std::vector<ForwardStep> run_merged_schedule(const Plan &p) {
  std::vector<ForwardStep> steps = fold_diagonals(p, merged_schedule(p));
  if (!inplace_differs(p)) return steps;
  const double cost = schedule_cost(p, steps);
  // One run of single gates and moves goes in passes of up to seven wires >= 6.
  if (plan_runs(p, 1) == 1) {
    uint64_t wires = 0;
    for (const PlanOp &op : p.ops) {
      if (is_wire_move(op, p.num_qubits)) wires |= (1ull << op.qubits[0]) | (1ull << op.qubits[1]);
      else if (op.kind == PlanOp::Kind::Dense1q) wires |= 1ull << op.qubits[0];
      else for (uint32_t w : op.group_qubits) wires |= 1ull << w;
    }
    if (2.0 * std::max(1u, (popc(wires >> 6) + 6) / 7) >= cost) return steps;
  }
  double folds = 0.0;   // what the folding of layers may still save
  for (const PlanOp &op : p.ops) folds += op.kind == PlanOp::Kind::DiagonalLayer ? 4.0 : 0.0;
  std::vector<ForwardStep> inplace;
  if (!inplace_steps(p, cost + folds, inplace)) return steps;
  inplace = fold_diagonals(p, std::move(inplace));
  return schedule_cost(p, inplace) < cost ? inplace : steps;
}


std::vector<ForwardStep> fold_diagonals(const Plan &p, std::vector<ForwardStep> steps) {
  const uint32_t n = p.num_qubits;
  if (n <= kDiagGroupMinWire) return steps;
  auto layer = [&](const ForwardStep &st) {
    if (st.kind != ForwardStep::Op) return false;
    const PlanOp &op = p.ops[st.ops[0]];
    if (op.kind != PlanOp::Kind::DiagonalLayer || op.masks.empty() ||
        op.angles.size() != op.masks.size() || fan_centres(op, n))
      return false;
    for (uint64_t m : op.masks)
      if ((m >> n) || popc(m) > 2) return false;
    return op.masks.size() > 1 || op.global_phase != 0.0;   // (one term is a masked phase)
  };
  std::vector<ForwardStep> out;
  for (size_t i = 0; i < steps.size(); i++) {
    if (!layer(steps[i])) {
      out.push_back(std::move(steps[i]));
      continue;
    }
    // The group passes that follow, as far as their wires differ.
    WireRun run;
    size_t j = i + 1;
    for (; j < steps.size() && steps[j].kind == ForwardStep::Group; j++) {
      bool again = false;
      for (uint32_t w : steps[j].wires) again = again || run.holds(w);
      if (again) break;
      for (size_t k = 0; k < steps[j].wires.size(); k++)
        run.add(steps[j].wires[k], &steps[j].mats[4 * k]);
    }
    std::vector<size_t> order(run.wires.size());
    for (size_t k = 0; k < order.size(); k++) order[k] = k;
    std::sort(order.begin(), order.end(),
              [&](size_t a, size_t b) { return run.wires[a] < run.wires[b]; });
    size_t best = j - i - 1, take = 0;
    std::vector<std::vector<size_t>> passes;
    WireRun left;
    for (size_t k = 1; k <= kDiagGroupWires && k <= order.size(); k++) {
      if (run.wires[order[order.size() - k]] < kDiagGroupMinWire) break;
      WireRun rest;
      for (size_t m = 0; m + k < order.size(); m++)
        rest.add(run.wires[order[m]], &run.mats[4 * order[m]]);
      auto split = split_run(n, rest);
      if (split.size() >= best) continue;
      best = split.size();
      take = k;
      passes = std::move(split);
      left = std::move(rest);
    }
    if (!take) {
      out.push_back(std::move(steps[i]));
      continue;
    }
    ForwardStep s = group_step(run, {order.end() - take, order.end()});
    s.kind = ForwardStep::DiagGroup;
    s.ops = steps[i].ops;
    out.push_back(std::move(s));
    for (const auto &pass : passes) out.push_back(group_step(left, pass));
    i = j - 1;
  }
  return out;
}

// ---------------------------------------------------------------------------

std::vector<ForwardStep> small_schedule(const Plan &p) {
  const uint32_t n = p.num_qubits;
  std::vector<ForwardStep> out;
  WireRun held;
  std::vector<PermGate> run;
  std::vector<size_t> run_ops;
  auto flush = [&]() {
    std::vector<size_t> idx(held.wires.size());
    for (size_t i = 0; i < idx.size(); i++) idx[i] = i;
    std::sort(idx.begin(), idx.end(),
              [&](size_t a, size_t b) { return held.wires[a] < held.wires[b]; });
    for (size_t b = 0; b < idx.size(); b += 3)
      out.push_back(group_step(held, {idx.begin() + b, idx.begin() + std::min(idx.size(), b + 3)}));
    held.clear();
    if (run.empty()) return;
    const Affine map = run_map(n, run, false);
    ForwardStep s;
    s.kind = ForwardStep::Permute;
    s.cols = map.cols;
    s.off = map.off;
    s.ops = std::move(run_ops);
    out.push_back(std::move(s));
    run.clear();
    run_ops.clear();
  };
  for (size_t i = 0; i < p.ops.size(); i++) {
    const PlanOp &op = p.ops[i];
    if (is_wire_move(op, n)) {
      run.push_back({op.kind == PlanOp::Kind::Swap, op.qubits[0], op.qubits[1]});
      run_ops.push_back(i);
      continue;
    }
    const uint32_t *w = nullptr;
    const cdouble *m = nullptr;
    size_t count = 0;
    if (!one_wire_op(op, n, w, m, count)) {
      flush();
      ForwardStep s;
      s.ops = {i};
      out.push_back(std::move(s));
      continue;
    }
    bool later = !run.empty();
    for (size_t j = 0; j < count; j++) later = later || held.holds(w[j]);
    if (later) flush();
    for (size_t j = 0; j < count; j++) held.add(w[j], m + 4 * j);
  }
  flush();
  return out;
}

bool undone_by(const Plan &p, const ForwardStep &gather, const std::vector<size_t> &gates) {
  if (gather.ops.size() != gates.size()) return false;
  for (size_t k = 0; k < gates.size(); k++)
    if (p.ops[gather.ops[k]].gate != gates[gates.size() - 1 - k]) return false;
  return true;
}

// ---------------------------------------------------------------------------

namespace {

struct FlipGroup {
  uint64_t flip;
  std::vector<size_t> terms;
};

std::vector<FlipGroup> group_by_flip(const std::vector<const PauliTerm *> &terms) {
  std::vector<FlipGroup> out;
  std::map<uint64_t, size_t> where;
  for (size_t t = 0; t < terms.size(); t++) {
    const PauliString &p = terms[t]->pauli;
    const uint64_t f = p.x_mask | p.y_mask;
    auto it = where.find(f);
    if (it == where.end()) {
      where[f] = out.size();
      out.push_back({f, {t}});
    } else {
      out[it->second].terms.push_back(t);
    }
  }
  return out;
}

}  // namespace

// Z strings of <= 2 bits go as one quadratic-form pass; plain X_w terms
// (a transverse field) go as block passes of up to seven wires >= 6 with any
// of wires 0..5, the terms on one wire summed; other terms that flip one wire
// pack many wires per pass (wires 0..5 ride along in every pass, at most
// four wires >= 6 and 16 terms a pass); anything else goes one pass per flip
// mask, 16 terms at a time. When every term is of the first two kinds their
// passes also sum the energy, and no separate energy pass follows.
std::vector<CostateStep> costate_schedule(const Hamiltonian &h, uint32_t n) {
  std::vector<CostateStep> out;
  std::vector<const PauliTerm *> zpart, xfield, local, rest;
  for (const PauliTerm &t : h.terms) {
    const uint64_t flip = t.pauli.x_mask | t.pauli.y_mask;
    if (!flip && popc(t.pauli.z_mask) <= 2) zpart.push_back(&t);
    else if (popc(flip) == 1 && !t.pauli.y_mask && !t.pauli.z_mask && n >= kXFieldMinQubits)
      xfield.push_back(&t);
    else if (popc(flip) == 1 && n >= 6) local.push_back(&t);
    else rest.push_back(&t);
  }
  const bool fused_energy = local.empty() && rest.empty() && !h.terms.empty();
  bool first = true;
  if (!zpart.empty()) {
    CostateStep s;
    s.kind = CostateStep::ZDiag;
    s.overwrite = true;
    for (const PauliTerm *t : zpart) {
      s.masks.push_back(t->pauli.z_mask);
      s.coeffs.push_back(t->coefficient);
    }
    out.push_back(std::move(s));
    first = false;
  }
  if (!xfield.empty()) {
    std::map<uint32_t, double> coef;   // wire -> summed coefficient, ascending
    for (const PauliTerm *t : xfield)
      coef[static_cast<uint32_t>(__builtin_ctzll(t->pauli.x_mask))] += t->coefficient;
    std::vector<uint32_t> low, high;
    for (const auto &wc : coef) (wc.first < 6 ? low : high).push_back(wc.first);
    // ceil(H / 7) passes, as even as possible (22 wires: 6, 6, 5, 5); wires
    // 0..5 join the last, which is among the smallest.
    const size_t passes = std::max<size_t>(
        1, (high.size() + kXFieldHighPerPass - 1) / kXFieldHighPerPass);
    size_t at = 0;
    for (size_t p = 0; p < passes; p++) {
      const size_t take = high.size() / passes + (p < high.size() % passes ? 1 : 0);
      CostateStep s;
      s.kind = CostateStep::XField;
      s.overwrite = first;
      if (fused_energy) s.energy = first ? 1 : 2;
      first = false;
      if (p + 1 == passes)
        for (uint32_t w : low) {
          s.wires.push_back(w);
          s.coeffs.push_back(coef[w]);
        }
      for (size_t j = 0; j < take; j++, at++) {
        s.wires.push_back(high[at]);
        s.coeffs.push_back(coef[high[at]]);
      }
      out.push_back(std::move(s));
    }
  }
  if (fused_energy) return out;
  if (!local.empty()) {
    auto wire_of = [&](const PauliTerm *t) {
      return static_cast<uint32_t>(__builtin_ctzll(t->pauli.x_mask | t->pauli.y_mask));
    };
    std::stable_sort(local.begin(), local.end(),
                     [&](const PauliTerm *a, const PauliTerm *b) { return wire_of(a) < wire_of(b); });
    const uint32_t max_high = std::min<uint32_t>(4, n - 6);
    CostateStep s;
    std::vector<uint32_t> highs;
    auto flush = [&]() {
      if (s.wires.empty()) return;
      s.kind = CostateStep::Local;
      s.overwrite = first;
      first = false;
      out.push_back(std::move(s));
      s = CostateStep{};
      highs.clear();
    };
    for (const PauliTerm *t : local) {
      const uint32_t w = wire_of(t);
      const bool new_high = w >= 6 && std::find(highs.begin(), highs.end(), w) == highs.end();
      if (s.wires.size() == kCostateTermsPerPass || (new_high && highs.size() == max_high)) flush();
      if (w >= 6 && std::find(highs.begin(), highs.end(), w) == highs.end()) highs.push_back(w);
      s.wires.push_back(w);
      s.masks.push_back(t->pauli.y_mask | t->pauli.z_mask);
      s.nys.push_back(popc(t->pauli.y_mask));
      s.coeffs.push_back(t->coefficient);
    }
    flush();
  }
  for (const FlipGroup &g : group_by_flip(rest)) {
    for (size_t b = 0; b < g.terms.size(); b += kCostateTermsPerPass) {
      const size_t take = std::min<size_t>(kCostateTermsPerPass, g.terms.size() - b);
      CostateStep s;
      s.kind = CostateStep::Flip;
      s.overwrite = first;
      s.flip = g.flip;
      for (size_t j = 0; j < take; j++) {
        const PauliTerm &t = *rest[g.terms[b + j]];
        s.masks.push_back(t.pauli.y_mask | t.pauli.z_mask);
        s.nys.push_back(popc(t.pauli.y_mask));
        s.coeffs.push_back(t.coefficient);
      }
      out.push_back(std::move(s));
      first = false;
    }
  }
  if (first) out.push_back(CostateStep{});
  CostateStep dot;
  dot.kind = CostateStep::Dot;
  out.push_back(std::move(dot));
  return out;
}

// ---------------------------------------------------------------------------

namespace {

// A run of the circuit that the sweep undoes as a unit.
struct Segment {
  enum Kind { Window, Diag, Single } kind = Single;
  size_t begin = 0, end = 0;
  bool has_param = false;
  // Diag: the block's forward phase terms and its Z-string generators.
  std::vector<uint64_t> masks;
  std::vector<double> angles;
  double gphase = 0.0;
  std::vector<uint64_t> gens;
  std::vector<uint32_t> slots;
};

// Forward segmentation: a maximal run of one-qubit gates is a window; a run
// of ZZ couplings (CX.RZ.CX) and two-qubit diagonal gates is a diagonal block;
// anything else stands alone.
std::vector<Segment> segment_circuit(const Circuit &c) {
  std::vector<Segment> segs;
  const size_t G = c.ops.size();
  size_t i = 0;
  while (i < G) {
    const Gate &g = c.ops[i];
    Segment s;
    s.begin = i;
    uint32_t a, b;
    double t;
    if (g.num_qubits == 1) {
      s.kind = Segment::Window;
      size_t j = i;
      for (; j < G && c.ops[j].num_qubits == 1; j++)
        if (c.ops[j].num_params) s.has_param = true;
      s.end = j;
    } else if (zz_coupling_at(c, i, &a, &b, &t) || (g.num_qubits == 2 && is_diagonal(g))) {
      s.kind = Segment::Diag;
      size_t j = i;
      while (j < G) {
        if (zz_coupling_at(c, j, &a, &b, &t)) {
          const uint64_t ma = 1ull << a, mb = 1ull << b;
          s.masks.insert(s.masks.end(), {ma, mb, ma | mb});
          s.angles.insert(s.angles.end(), {t, t, -2.0 * t});
          s.gphase += -t / 2.0;
          if (c.ops[j + 1].num_params) {
            s.gens.push_back(ma | mb);   // exp(-i t/2 Z_a Z_b)
            s.slots.push_back(static_cast<uint32_t>(j + 1));
            s.has_param = true;
          }
          j += 3;
        } else if (c.ops[j].num_qubits == 2 && is_diagonal(c.ops[j])) {
          s.gphase += diagonal_term(c.ops[j], s.masks, s.angles);
          if (c.ops[j].num_params) s.has_param = true;
          j++;
        } else {
          break;
        }
      }
      s.end = j;
    } else {
      s.kind = Segment::Single;
      s.end = i + 1;
      s.has_param = g.num_params > 0;
    }
    i = s.end;
    segs.push_back(std::move(s));
  }
  return segs;
}

}  // namespace

// Every gradient of a commuting block is read at the block boundary and the
// block is undone on both states in the same pass. Blocks before the first
// parameterised one are never undone.
namespace {

// A wire's ops (in undo order) as one of the rotation sequences the block
// tiles compile in: one RX, RY or RZ, or RZ then RY, or RY then RZ. Returns
// a nonzero code for each such sequence, 0 for any other.
uint32_t uniform_signature(const std::vector<WireOp> &ops) {
  if (ops.empty() || ops.size() > 2) return 0;
  int kind[2];
  for (size_t k = 0; k < ops.size(); k++) {
    const int cls = narrowed_class(ops[k].minv), gen = ops[k].gen;
    if (cls == 2 && gen == 1) kind[k] = 0;        // RX
    else if (cls == 1 && gen == 2) kind[k] = 1;   // RY
    else if (cls == 3 && gen == 3) kind[k] = 2;   // RZ
    else return 0;
  }
  if (ops.size() == 1) return 1 + kind[0];
  if ((kind[0] == 2 && kind[1] == 1) || (kind[0] == 1 && kind[1] == 2))
    return 4 + kind[0];
  return 0;
}

}  // namespace

std::vector<BackwardStep> backward_schedule(const Circuit &c, uint32_t tile_high) {
  const uint32_t n = c.num_qubits;
  tile_high = std::min<uint32_t>(std::max<uint32_t>(tile_high, 1), kMaxTileHigh);
  std::vector<BackwardStep> out;
  const auto segs = segment_circuit(c);
  size_t first = segs.size();
  for (size_t s = 0; s < segs.size(); s++)
    if (segs[s].has_param) {
      first = s;
      break;
    }
  for (size_t s = segs.size(); s-- > first;) {
    const Segment &seg = segs[s];
    const bool undo = s > first;
    if (seg.kind == Segment::Single) {
      // A run of CX / SWAP gates, all undone here, goes as one gather pass
      // per state when that moves fewer bytes.
      auto perm_gate = [&](size_t k) {
        const Gate &g = c.ops[segs[k].begin];
        return segs[k].kind == Segment::Single && (g.kind == G_CX || g.kind == G_SWAP) &&
               g.qubits[0] < n && g.qubits[1] < n && g.qubits[0] != g.qubits[1];
      };
      if (undo && perm_gate(s)) {
        size_t lo = s;
        while (lo - 1 > first && perm_gate(lo - 1)) lo--;
        if (s > lo) {
          std::vector<PermGate> run;
          for (size_t k = lo; k <= s; k++) {
            const Gate &g = c.ops[segs[k].begin];
            run.push_back({g.kind == G_SWAP, g.qubits[0], g.qubits[1]});
          }
          const Affine map = run_map(n, run, true);
          if (permutation_pays(map, run.size())) {
            BackwardStep st;
            st.kind = BackwardStep::PermuteUndo;
            st.cols = map.cols;
            st.off = map.off;
            for (size_t k = s + 1; k-- > lo;) st.gates.push_back(segs[k].begin);
            out.push_back(std::move(st));
            s = lo;
            continue;
          }
        }
      }
      if (undo) {
        BackwardStep st;
        st.gates = {seg.begin};
        out.push_back(std::move(st));
      }
      continue;
    }
    if (seg.kind == Segment::Diag) {
      const uint32_t ng = static_cast<uint32_t>(seg.gens.size());
      if (ng == 0 && !undo) continue;
      uint32_t done = 0;
      do {
        const uint32_t take = std::min(kDiagGensPerPass, ng - done);
        BackwardStep st;
        st.kind = BackwardStep::Diag;
        st.masks = seg.masks;
        st.angles = seg.angles;
        st.gphase = seg.gphase;
        st.gens.assign(seg.gens.begin() + done, seg.gens.begin() + done + take);
        st.slots.assign(seg.slots.begin() + done, seg.slots.begin() + done + take);
        st.undo = done + take == ng && undo;
        out.push_back(std::move(st));
        done += take;
      } while (done < ng);
      continue;
    }
    // Window: each wire's gates last to first, a few wires per pass. Gates
    // on different wires commute, and a generator on one wire commutes with
    // every gate on the others, so the order across wires is free.
    std::vector<std::vector<size_t>> per_wire(n);
    for (size_t k = seg.begin; k < seg.end; k++) per_wire[c.ops[k].qubits[0]].push_back(k);
    std::vector<WireOp> tile;
    uint32_t others = 0, highs = 0, grads = 0;
    bool tile_has_param = false;
    bool tile_low = false;     // the tile holds a wire below 6
    uint32_t tile_sig = 0;     // the rotation sequence all its wires share (0: none)
    const bool wide = n >= 6;
    const uint32_t max_ops = wide ? kWideWindowOps : kWindowOps;
    // Up to four wires >= 6 per pass in a warp tile; five or six in a block
    // tile, which holds only wires >= 6 that all carry one rotation sequence.
    const uint32_t max_high = wide ? std::min<uint32_t>(std::min<uint32_t>(tile_high, 4), n - 6) : 0;
    const uint32_t max_high_blk = wide ? std::min<uint32_t>(tile_high, n - 6) : 0;
    auto flush = [&]() {
      if (tile.empty()) return;
      if (undo || tile_has_param) {
        BackwardStep st;
        st.kind = BackwardStep::Window;
        st.tile = tile;
        out.push_back(std::move(st));
      }
      tile.clear();
      others = highs = grads = 0;
      tile_has_param = false;
      tile_low = false;
      tile_sig = 0;
    };
    // Each wire's ops in undo order, and the rotation sequence they form.
    std::vector<std::vector<WireOp>> wire_ops(n);
    std::vector<uint32_t> wire_sig(n, 0);
    for (uint32_t w = 0; w < n; w++) {
      for (size_t r = per_wire[w].size(); r-- > 0;) {
        const size_t k = per_wire[w][r];
        const Gate &g = c.ops[k];
        const Gate inv = invert(g);
        WireOp o{};
        o.wire = w;
        gate_matrix_1q(inv.kind, inv.params, o.minv);
        o.gen = g.num_params > 0 ? generator_of(g) : 0;
        o.slot = static_cast<uint32_t>(k);
        wire_ops[w].push_back(o);
      }
      wire_sig[w] = uniform_signature(wire_ops[w]);
    }
    // The block tiles of a run of wires sharing one rotation sequence split
    // it evenly: a run of R wires takes ceil(R / tile_high) passes of at most
    // ceil(R / passes) wires each (twenty wires: five passes of four become
    // four of five, not three of six and one of two).
    uint32_t blk_cap = max_high_blk;
    auto balanced_cap = [&](uint32_t w) {
      uint32_t run = 0;
      for (uint32_t v = w; v < n; v++) {
        if (wire_ops[v].empty()) continue;
        if (wire_sig[v] != wire_sig[w]) break;
        run++;
      }
      if (run == 0 || max_high_blk == 0) return max_high_blk;
      const uint32_t passes = (run + max_high_blk - 1) / max_high_blk;
      return (run + passes - 1) / passes;
    };
    // When every wire >= 6 of the window carries one rotation (one op per
    // wire), the block tiles take them more cheaply than the tile of wires
    // 0..5 (whose lane wires trade by shuffle): that first tile keeps only as
    // many wires >= 6 as leave the number of passes at its least, and at
    // least one, so it stays a compile-time tile (measured: 379 -> 394
    // MaxCut requests/s). With two ops per wire the first tile's share
    // moved to the block tiles costs more than it saves (the 28-qubit HEA
    // gradient 0.108 -> 0.120 s), so there it keeps what fits.
    uint32_t first_high = max_high;
    bool wide_first = false;
    {
      uint32_t run = 0, sig0 = 0, low_grads = 0, high_grads = 0;
      bool uniform = true, low = false;
      for (uint32_t w = 0; w < n; w++) {
        if (per_wire[w].empty()) continue;
        uint32_t g = 0;
        for (const WireOp &o : wire_ops[w]) g += o.gen != 0;
        if (w < 6) {
          low = true;
          low_grads += g;
          continue;
        }
        if (run == 0) {
          sig0 = wire_sig[w];
          high_grads = g;
        }
        uniform &= wire_sig[w] != 0 && wire_sig[w] == sig0;
        run++;
      }
      // The first tile of an RZ-then-RY layer takes four wires >= 6 (twenty
      // gradients, where sixteen allow two) when that saves a block pass: at
      // 28 qubits 2 + 5, 5, 5, 5 wires >= 6 become 4 + 6, 6, 6.
      bool low_rzry = n >= 10;
      for (uint32_t w = 0; w < 6 && w < n; w++) low_rzry &= wire_sig[w] == kSigRzRy;
      if (low_rzry && uniform && sig0 == kSigRzRy && run >= 4 && max_high >= 4 &&
          max_high_blk >= 5) {
        const uint32_t before = (run - 2 + max_high_blk - 1) / max_high_blk;
        const uint32_t after = (run - 4 + max_high_blk - 1) / max_high_blk;
        wide_first = after < before;
      }
      if (low && uniform && run > 0 && max_high_blk >= 5 && high_grads <= 1) {
        // as many as the first tile's gradient slots allow
        uint32_t room = max_high;
        if (high_grads > 0)
          room = low_grads >= kWindowGrads ? 0 : std::min(room, (kWindowGrads - low_grads) / high_grads);
        uint32_t best = ~0u;
        for (uint32_t k = std::min<uint32_t>(1, std::min(room, run)); k <= std::min(room, run);
             k++) {
          const uint32_t passes = (run - k + max_high_blk - 1) / max_high_blk;
          if (passes < best) {
            best = passes;
            first_high = k;
          }
        }
      }
    }
    for (uint32_t w = 0; w < n; w++) {
      if (per_wire[w].empty()) continue;
      const std::vector<WireOp> &ops = wire_ops[w];
      uint32_t wgrads = 0;
      for (const WireOp &o : ops) wgrads += o.gen != 0;
      const uint32_t need_other = w != 0 ? 1u : 0u, need_high = w >= 6 ? 1u : 0u;
      if (ops.size() > max_ops || wgrads > kWindowGrads) {
        flush();
        for (size_t b = 0; b < ops.size(); b += kWindowOps) {
          const size_t e = std::min<size_t>(ops.size(), b + kWindowOps);
          tile.assign(ops.begin() + b, ops.begin() + e);
          for (const WireOp &o : tile) tile_has_param |= o.gen != 0;
          flush();
        }
        continue;
      }
      bool full;
      const uint32_t sig = wire_sig[w];
      if (wide) {
        // Warp tiles: wire 0, wires 1..5 in the lanes, up to four wires >= 6;
        // block tiles: five or six wires >= 6 of one rotation sequence.
        const bool blk = !tile_low && w >= 6 && sig != 0 && (tile.empty() || sig == tile_sig);
        if (blk && tile.empty()) blk_cap = balanced_cap(w);
        // A tile of wire 0 and wires 1..5 that all carry RZ then RY takes four
        // wires >= 6 with the same ops (twenty gradients) where that saves a pass.
        const bool wide_rzry = wide_first && tile_low && others == 5 + highs &&
                               tile.size() == 12 + 2 * highs && tile_sig == kSigRzRy &&
                               sig == kSigRzRy;
        full = tile.size() + ops.size() > max_ops ||
               highs + need_high >
                   (blk ? std::max(blk_cap, max_high) : (tile_low ? first_high : max_high)) ||
               grads + wgrads > (wide_rzry ? kWideUniformGrads : kWindowGrads);
        if (!full && !blk && highs > max_high) full = true;   // a block tile takes no other wire
      } else {
        const uint32_t cap = (others + need_other >= 3) ? 8u : 16u;
        full = tile.size() + ops.size() > kWindowOps || others + need_other > 3 ||
               grads + wgrads > cap;
      }
      if (full) flush();
      if (tile.empty() && w >= 6 && sig != 0) blk_cap = balanced_cap(w);   // a new tile opens
      tile_sig = tile.empty() ? sig : (sig == tile_sig ? sig : 0);
      tile_low |= w < 6;
      tile.insert(tile.end(), ops.begin(), ops.end());
      others += need_other;
      highs += need_high;
      grads += wgrads;
      tile_has_param |= wgrads > 0;
    }
    flush();
  }
  return out;
}

// ---------------------------------------------------------------------------

namespace {

void put_map(std::vector<double> &v, uint32_t n, const std::vector<uint64_t> &cols, uint64_t off) {
  v.push_back(n);
  for (uint32_t j = 0; j < n; j++) v.push_back(static_cast<double>(cols[j]));
  v.push_back(static_cast<double>(off));
}

void put_mat(std::vector<double> &v, const cdouble *m) {
  for (int k = 0; k < 4; k++) {
    v.push_back(m[k].real());
    v.push_back(m[k].imag());
  }
}

}  // namespace

void serialise_schedule(const std::vector<ForwardStep> &s, uint32_t n, std::vector<double> &v) {
  v.push_back(static_cast<double>(s.size()));
  for (const ForwardStep &st : s) {
    v.push_back(st.kind);
    if (st.kind == ForwardStep::Group || st.kind == ForwardStep::Moves ||
        st.kind == ForwardStep::DiagGroup) {
      if (st.kind == ForwardStep::DiagGroup) v.push_back(static_cast<double>(st.ops.at(0)));
      v.push_back(static_cast<double>(st.wires.size()));
      for (size_t i = 0; i < st.wires.size(); i++) {
        v.push_back(st.wires[i]);
        put_mat(v, &st.mats[4 * i]);
      }
      if (st.kind == ForwardStep::Moves) {
        v.push_back(static_cast<double>(st.moves.size()));
        for (const PermGate &m : st.moves) {
          v.push_back(m.swap ? 1.0 : 0.0);
          v.push_back(m.a);
          v.push_back(m.b);
        }
      }
    } else if (st.kind == ForwardStep::Stages) {
      v.push_back(static_cast<double>(st.stages.size()));
      for (const Stage &s : st.stages) {
        v.push_back(s.wire);
        v.push_back(s.has_matrix ? 1.0 : 0.0);
        put_mat(v, s.m);
        v.push_back(s.phase);
        for (uint32_t w = 0; w < n; w++) v.push_back(s.phase ? s.angles[w] : 0.0);
      }
    } else if (st.kind == ForwardStep::Permute) {
      put_map(v, n, st.cols, st.off);
      v.push_back(static_cast<double>(st.ops.size()));
      for (size_t i : st.ops) v.push_back(static_cast<double>(i));
    } else {
      v.push_back(static_cast<double>(st.ops.at(0)));
    }
  }
}

void serialise_schedule(const std::vector<CostateStep> &s, std::vector<double> &v) {
  v.push_back(static_cast<double>(s.size()));
  for (const CostateStep &st : s) {
    v.push_back(st.kind);
    switch (st.kind) {
      case CostateStep::ZDiag:
        v.push_back(static_cast<double>(st.masks.size()));
        for (size_t i = 0; i < st.masks.size(); i++) {
          v.push_back(static_cast<double>(st.masks[i]));
          v.push_back(st.coeffs[i]);
        }
        break;
      case CostateStep::Local:
        v.push_back(st.overwrite ? 1.0 : 0.0);
        v.push_back(static_cast<double>(st.wires.size()));
        for (size_t i = 0; i < st.wires.size(); i++) {
          v.push_back(st.wires[i]);
          v.push_back(static_cast<double>(st.masks[i]));
          v.push_back(st.nys[i]);
          v.push_back(st.coeffs[i]);
        }
        break;
      case CostateStep::Flip:
        v.push_back(st.overwrite ? 1.0 : 0.0);
        v.push_back(static_cast<double>(st.flip));
        v.push_back(static_cast<double>(st.masks.size()));
        for (size_t i = 0; i < st.masks.size(); i++) {
          v.push_back(static_cast<double>(st.masks[i]));
          v.push_back(st.nys[i]);
          v.push_back(st.coeffs[i]);
        }
        break;
      case CostateStep::XField:
        v.push_back(st.overwrite ? 1.0 : 0.0);
        v.push_back(st.energy);
        v.push_back(static_cast<double>(st.wires.size()));
        for (size_t i = 0; i < st.wires.size(); i++) {
          v.push_back(st.wires[i]);
          v.push_back(st.coeffs[i]);
        }
        break;
      default:
        break;
    }
  }
}

void serialise_schedule(const std::vector<BackwardStep> &s, uint32_t n, std::vector<double> &v) {
  v.push_back(static_cast<double>(s.size()));
  for (const BackwardStep &st : s) {
    v.push_back(st.kind);
    switch (st.kind) {
      case BackwardStep::Window:
        v.push_back(static_cast<double>(st.tile.size()));
        for (const WireOp &o : st.tile) {
          v.push_back(o.wire);
          put_mat(v, o.minv);
          v.push_back(o.gen);
          v.push_back(o.slot);
        }
        break;
      case BackwardStep::Diag:
        v.push_back(st.undo ? 1.0 : 0.0);
        v.push_back(static_cast<double>(st.masks.size()));
        for (size_t i = 0; i < st.masks.size(); i++) {
          v.push_back(static_cast<double>(st.masks[i]));
          v.push_back(st.angles[i]);
        }
        v.push_back(st.gphase);
        v.push_back(static_cast<double>(st.gens.size()));
        for (size_t i = 0; i < st.gens.size(); i++) {
          v.push_back(static_cast<double>(st.gens[i]));
          v.push_back(st.slots[i]);
        }
        break;
      case BackwardStep::PermuteUndo:
        put_map(v, n, st.cols, st.off);
        v.push_back(static_cast<double>(st.gates.size()));
        for (size_t g : st.gates) v.push_back(static_cast<double>(g));
        break;
      case BackwardStep::GateUndo:
        v.push_back(static_cast<double>(st.gates.at(0)));
        break;
    }
  }
}

}  // namespace qmetal
