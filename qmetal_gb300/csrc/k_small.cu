// k_small.cu -- a whole circuit on a narrow state (up to 13 qubits) in one
// launch.
//
// A state of 2^n amplitudes, n <= 13, fits one multiprocessor's shared memory
// (64 KiB at 13), where an op costs a barrier and a few hundred cycles. As
// launches of their own, a circuit's ops cost 2 to 5 us each whatever their
// size (the 52 ops of a 9-qubit U3 circuit: 200 us). One block loads the
// state, runs the ops one after another and stores it; the ops come as kernel
// arguments, so nothing is staged or kept. The phases of all the circuit's
// diagonal layers are tabulated first by one launch over the whole chip: their
// FP64 sums and sincos would take one multiprocessor far longer than the
// circuit.
//
// A gradient runs the same way: the block then holds the co-state beside the
// state, forms it after the forward ops, and takes each backward step's
// gradients while it undoes both.
//
// Bound by latency: a barrier, shared-memory round trip and up to three
// dependent 2x2s an op. The 9-qubit U3 circuit of depth 10 with its read-out:
// 310 -> 77 us; gradients of four HEA layers, host work and read-out in, at 6, 10
// and 12 qubits 213 -> 108, 233 -> 157 and 304 -> 247 us. At 13 qubits, where one
// block took 360 us and the launches take 297, a gradient goes by launches.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <vector>

#include "kadjoint.cuh"
#include "../../include/qmetal/qmetal_kernels.h"

using namespace qmk;
using qmk_host::grid_for;
using qmk_host::launch_status;

namespace {

constexpr uint32_t kMaxN = QMK_SMALL_MAX_QUBITS, kMaxN2 = QMK_SMALL_MAX_ADJOINT;
// Most phase tables per launch, and states kept.
constexpr uint32_t kMaxLayers = 32;
constexpr uint32_t layers_of(uint32_t n) { return n >= 13 ? 16 : kMaxLayers; }
constexpr uint32_t saves_of(uint32_t n) { return n > kMaxN2 ? 0 : n >= 12 ? 16 : 32; }
// Widest blocks: eight amplitudes a thread at 13 qubits, eight of each state at
// 12 with the co-state.
constexpr unsigned kSmallThreads = 1024, kSmallThreads2 = 512;
// Warps beside a gradient's threads (while those are at most 256) that add up
// the rows of partial sums, so that no working warp waits for them (6 qubits,
// four HEA layers: 32 us less).
constexpr unsigned kHelpers = 4;
constexpr int kRows = 12;                  // gradients per step

// The ops as words, in four sizes of kernel arguments up to their limit of
// 32 KiB (10 qubits, four
// HEA layers, a gradient: 11 us less with four sizes than with two). An op's first word and each of its
// matrices start on 16 bytes. The block copies them into shared memory first.
template <int WORDS>
struct Code {
  uint32_t count;        // words used
  uint32_t w[WORDS];
};
constexpr int kCode1 = 960, kCode2 = 1920, kCode3 = 3840, kLongCode = 7936;
constexpr uint32_t kOpHead = 4;   // words before an op's matrices
// A matrix: eight words narrowed to FP32, eight of what they lack. The narrowing
// errors of one angle add up over wires and layers, and forward and back (ten
// qubits, eight Trotter layers: most of a gradient's 2e-6); the low parts cost a
// few multiply-adds in a kernel that waits for latency.
constexpr uint32_t kMatWords = 16;
constexpr uint32_t kItemWords = kOpHead + kMatWords;

// A phase layer of the first launch: merged terms and the constant.
template <int TERMS>
struct Layers {
  uint32_t count;
  uint32_t real;         // bit l: layer l tabulates sum of angle (-1)^parity(i & mask)
  uint16_t first[kMaxLayers + 1];
  uint16_t mask[TERMS];
  double g[kMaxLayers];
  double angle[TERMS];
};
constexpr int kShortTerms = 320, kLongTerms = 3000;

enum : uint32_t {
  kGroup = 0, kPhase = 1, kControlled = 2, kMap = 3, kLayer = 4,
  kWindow = 5, kCostate = 6, kDiagGrad = 7
};
constexpr uint32_t kBoth = 1u << 28;   // on the state and the co-state
constexpr uint32_t kConj = 1u << 29;   // the conjugate of the layer's phases

// Bound by its FP64 sums and sincos: two-warp blocks spread it over the chip.
template <int TERMS>
__global__ void __launch_bounds__(64)
k_small_tables(uint32_t n, const Layers<TERMS> ls, float2 *__restrict__ tables) {
  const uint32_t i = blockIdx.x * 64 + threadIdx.x, l = blockIdx.y;
  if (i >= (1u << n)) return;
  double f = ls.g[l];
  if ((ls.real >> l) & 1u) {
    for (uint32_t t = ls.first[l]; t < ls.first[l + 1]; t++)
      f += (__popc(i & ls.mask[t]) & 1) ? -ls.angle[t] : ls.angle[t];
    tables[(static_cast<size_t>(l) << n) + i] = make_float2(static_cast<float>(f), 0.0f);
    return;
  }
  for (uint32_t t = ls.first[l]; t < ls.first[l + 1]; t++)
    if ((i & ls.mask[t]) == ls.mask[t]) f += ls.angle[t];
  double s, c;
  sincos(f, &s, &c);
  tables[(static_cast<size_t>(l) << n) + i] =
      make_float2(static_cast<float>(c), static_cast<float>(s));
}

// Slot of amplitude i: the low four bits (one shared-memory wavefront holds
// sixteen amplitudes) folded with the next eight, so that threads whose
// amplitudes are 8 or 16 apart fall on different banks.
__device__ __forceinline__ uint32_t slot(uint32_t i) {
  return i ^ ((i >> 4) & 15u) ^ ((i >> 8) & 15u);
}

__device__ __forceinline__ uint32_t ins0s(uint32_t x, uint32_t p) {
  const uint32_t low = x & ((1u << p) - 1u);
  return ((x >> p) << (p + 1)) | low;
}

__device__ __forceinline__ M2 m2(const uint32_t *w) {   // on 16 bytes
  const float4 a = *reinterpret_cast<const float4 *>(w);
  const float4 b = *reinterpret_cast<const float4 *>(w + 4);
  return {lo2(a), hi2(a), lo2(b), hi2(b)};
}

// A 2x2 in two parts, of the class of its high part.
struct M2x {
  M2 hi, lo;
};
__device__ __forceinline__ M2x m2x(const uint32_t *w) { return {m2(w), m2(w + 8)}; }

__device__ __forceinline__ float2 cmul_add(float2 a, float2 x, float2 c) {   // a x + c
  return make_float2(fmaf(a.x, x.x, fmaf(-a.y, x.y, c.x)), fmaf(a.x, x.y, fmaf(a.y, x.x, c.y)));
}
// s u + t v, s and t of a class-CLS matrix (cmac2c's forms).
template <int CLS>
__device__ __forceinline__ float2 row_of(float2 s, float2 sl, float2 u, float2 t, float2 tl,
                                         float2 v) {
  if (CLS == kMatReal)
    return make_float2(fmaf(s.x, u.x, fmaf(t.x, v.x, fmaf(sl.x, u.x, tl.x * v.x))),
                       fmaf(s.x, u.y, fmaf(t.x, v.y, fmaf(sl.x, u.y, tl.x * v.y))));
  if (CLS == kMatRx)
    return make_float2(fmaf(s.x, u.x, fmaf(-t.y, v.y, fmaf(sl.x, u.x, -tl.y * v.y))),
                       fmaf(s.x, u.y, fmaf(t.y, v.x, fmaf(sl.x, u.y, tl.y * v.x))));
  if (CLS == kMatDiag) return cmul_add(s, u, cmul(sl, u));
  return cmul_add(s, u, cmul_add(t, v, cmul_add(sl, u, cmul(tl, v))));
}
template <int CLS>
__device__ __forceinline__ void apply2x(const M2x &m, float2 &u, float2 &v) {
  const float2 nu = row_of<CLS>(m.hi.a, m.lo.a, u, m.hi.b, m.lo.b, v);
  const float2 nv = row_of<CLS>(m.hi.d, m.lo.d, v, m.hi.c, m.lo.c, u);
  u = nu;
  v = nv;
}

// K 2x2s on distinct wires q[0] < q[1] < q[2]: 2^K amplitudes in registers.
template <int K, int CLS>
__device__ __forceinline__ void group(float2 *amp, uint32_t n, const uint32_t *w, uint32_t me,
                                      uint32_t step) {
  uint32_t q[K];
#pragma unroll
  for (int j = 0; j < K; j++) q[j] = (w[0] >> (8 + 5 * j)) & 31u;
  for (uint32_t s = me; s < (1u << (n - K)); s += step) {
    uint32_t base = s;
#pragma unroll
    for (int j = 0; j < K; j++) base = ins0s(base, q[j]);
    uint32_t at[1 << K];
    float2 r[1 << K];
#pragma unroll
    for (int l = 0; l < (1 << K); l++) {
      uint32_t i = base;
#pragma unroll
      for (int j = 0; j < K; j++)
        if ((l >> j) & 1) i |= 1u << q[j];
      at[l] = slot(i);
      r[l] = amp[at[l]];
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
      const M2x m = m2x(w + kOpHead + kMatWords * j);
#pragma unroll
      for (int l = 0; l < (1 << K); l++)
        if (!((l >> j) & 1)) apply2x<CLS>(m, r[l], r[l | (1 << j)]);
    }
#pragma unroll
    for (int l = 0; l < (1 << K); l++) amp[at[l]] = r[l];
  }
}

template <int K>
__device__ __forceinline__ void group_cls(float2 *amp, uint32_t n, const uint32_t *w, uint32_t me,
                                          uint32_t step) {
  switch ((w[0] >> 6) & 3u) {
    case kMatReal: group<K, kMatReal>(amp, n, w, me, step); break;
    case kMatRx: group<K, kMatRx>(amp, n, w, me, step); break;
    default: group<K, kMatGeneral>(amp, n, w, me, step); break;
  }
}

// The threads' partial sums of one result, added by one warp in a fixed order.
__device__ __forceinline__ double row_sum(const float *row, uint32_t count) {
  const uint32_t lane = threadIdx.x & 31;
  Two v = {0.0f, 0.0f};
  for (uint32_t t = lane; t < count; t += 32) v = add(v, Two{row[t], 0.0f});
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = add(v, shfl_xor(v, o));
  return widen(v);
}

// Im(conj(lambda) P psi) over the register pairs of wire bit J.
template <int K, int J, int GEN>
__device__ __forceinline__ float window_overlap(const float2 (&p)[1 << K], const float2 (&l)[1 << K]) {
  float s[2] = {0.0f, 0.0f};
  int at = 0;
#pragma unroll
  for (int k = 0; k < (1 << K); k++)
    if (!((k >> J) & 1))
      s[at++ & 1] += qmk_adj::overlap(GEN, p[k], p[k | (1 << J)], l[k], l[k | (1 << J)]);
  return s[0] + s[1];
}
template <int K, int J, int CLS>
__device__ __forceinline__ void window_apply(float2 (&p)[1 << K], float2 (&l)[1 << K], const M2x &m) {
#pragma unroll
  for (int k = 0; k < (1 << K); k++) {
    if ((k >> J) & 1) continue;
    apply2x<CLS>(m, p[k], p[k | (1 << J)]);
    apply2x<CLS>(m, l[k], l[k | (1 << J)]);
  }
}
template <int K, int J>
__device__ __forceinline__ float window_op(float2 (&p)[1 << K], float2 (&l)[1 << K], uint32_t gen,
                                           uint32_t cls, const M2x &m) {
  float s = 0.0f;
  if (gen == 1) s = window_overlap<K, J, 1>(p, l);
  else if (gen == 2) s = window_overlap<K, J, 2>(p, l);
  else if (gen == 3) s = window_overlap<K, J, 3>(p, l);
  switch (cls) {
    case kMatReal: window_apply<K, J, kMatReal>(p, l, m); break;
    case kMatRx: window_apply<K, J, kMatRx>(p, l, m); break;
    case kMatDiag: window_apply<K, J, kMatDiag>(p, l, m); break;
    default: window_apply<K, J, kMatGeneral>(p, l, m); break;
  }
  return s;
}

// Up to three wires' gates, last to first on each: an op's gradient, then its
// undo, both states in registers. part: one row of thread sums per gradient.
template <int K>
__device__ __forceinline__ void window(float2 *psi, float2 *lam, uint32_t n, const uint32_t *w,
                                       float *part, uint32_t me, uint32_t step) {
  uint32_t q[K];
#pragma unroll
  for (int j = 0; j < K; j++) q[j] = (w[0] >> (8 + 5 * j)) & 31u;
  const uint32_t nops = w[1];
  bool first = true;
  for (uint32_t s = me; s < (1u << (n - K)) || (first && s < step); s += step) {
    const bool active = s < (1u << (n - K));   // an idle thread leaves zero sums
    uint32_t base = s;
#pragma unroll
    for (int j = 0; j < K; j++) base = ins0s(base, q[j]);
    uint32_t at[1 << K];
    float2 p[1 << K], l[1 << K];
#pragma unroll
    for (int k = 0; k < (1 << K); k++) {
      uint32_t i = base;
#pragma unroll
      for (int j = 0; j < K; j++)
        if ((k >> j) & 1) i |= 1u << q[j];
      at[k] = slot(i);
      p[k] = active ? psi[at[k]] : make_float2(0.0f, 0.0f);
      l[k] = active ? lam[at[k]] : make_float2(0.0f, 0.0f);
    }
    uint32_t row = 0;
    for (uint32_t o = 0; o < nops; o++) {
      const uint32_t *op = w + kOpHead + kItemWords * o;
      const uint32_t j = op[0] & 3u, gen = (op[0] >> 2) & 3u, cls = op[0] >> 4;
      const M2x m = m2x(op + kOpHead);
      float v;
      if (K > 2 && j == 2) v = window_op<K, (K > 2 ? 2 : 0)>(p, l, gen, cls, m);
      else if (K > 1 && j == 1) v = window_op<K, (K > 1 ? 1 : 0)>(p, l, gen, cls, m);
      else v = window_op<K, 0>(p, l, gen, cls, m);
      if (gen) {
        float *mine = part + row * step + me;
        *mine = first ? v : *mine + v;
        row++;
      }
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < (1 << K); k++) {
        psi[at[k]] = p[k];
        lam[at[k]] = l[k];
      }
    }
    first = false;
  }
}

// (h, l) (a, b) in two parts.
__device__ __forceinline__ void times(float2 h, float2 l, float2 a, float2 b, float2 &rh,
                                      float2 &rl) {
  const float xx = __fmul_rn(h.x, a.x), yy = __fmul_rn(h.y, a.y);
  const float xy = __fmul_rn(h.x, a.y), yx = __fmul_rn(h.y, a.x);
  const float re = __fadd_rn(xx, -yy), im = __fadd_rn(xy, yx);
  // what the products and their sum lost, then the cross terms
  const float er = (fmaf(h.x, a.x, -xx) - fmaf(h.y, a.y, -yy)) +
                   add(Two{xx, 0.0f}, Two{-yy, 0.0f}).lo;
  const float ei = (fmaf(h.x, a.y, -xy) + fmaf(h.y, a.x, -yx)) +
                   add(Two{xy, 0.0f}, Two{yx, 0.0f}).lo;
  const float2 c = cmul_add(h, b, cmul(l, a));
  rh = make_float2(re, im);
  rl = make_float2(er + c.x, ei + c.y);
}

// The same where every wire has one RX (SIG 1) or RZ then RY (SIG 2), with
// their gradients: no dispatch per op, and the wires' RZ in one go -- their
// gradients from one Im(conj(lambda) psi) an amplitude, their undo one phase an
// amplitude.
template <int K, int SIG>
__device__ __forceinline__ void window_uniform(float2 *psi, float2 *lam, uint32_t n,
                                               const uint32_t *w, float *part, uint32_t me,
                                               uint32_t step) {
  constexpr int A = 1 << K;
  uint32_t q[K];
#pragma unroll
  for (int j = 0; j < K; j++) q[j] = (w[0] >> (8 + 5 * j)) & 31u;
  auto matrix = [&](int item) { return m2x(w + 2 * kOpHead + kItemWords * item); };
  auto add_to = [&](int row, float v, bool first) {
    float *mine = part + row * step + me;
    *mine = first ? v : *mine + v;
  };
  bool first = true;
  for (uint32_t s = me; s < (1u << (n - K)) || (first && s < step); s += step) {
    const bool active = s < (1u << (n - K));   // an idle thread leaves zero sums
    uint32_t base = s;
#pragma unroll
    for (int j = 0; j < K; j++) base = ins0s(base, q[j]);
    uint32_t at[A];
    float2 p[A], l[A];
#pragma unroll
    for (int k = 0; k < A; k++) {
      uint32_t i = base;
#pragma unroll
      for (int j = 0; j < K; j++)
        if ((k >> j) & 1) i |= 1u << q[j];
      at[k] = slot(i);
      p[k] = active ? psi[at[k]] : make_float2(0.0f, 0.0f);
      l[k] = active ? lam[at[k]] : make_float2(0.0f, 0.0f);
    }
    if (SIG == 2) {
      float f[A];
#pragma unroll
      for (int k = 0; k < A; k++) f[k] = l[k].x * p[k].y - l[k].y * p[k].x;
#pragma unroll
      for (int j = 0; j < K; j++) {
        float lo = 0.0f, hi = 0.0f;
#pragma unroll
        for (int k = 0; k < A; k++) {
          if ((k >> j) & 1) hi += f[k];
          else lo += f[k];
        }
        add_to(2 * j, lo - hi, first);
      }
      float2 ph[A], pl[A];   // high and low parts
#pragma unroll
      for (int j = 0; j < K; j++) {
        const M2x m = matrix(2 * j);
        if (j == 0) {
          ph[0] = m.hi.a;
          ph[1] = m.hi.d;
          pl[0] = m.lo.a;
          pl[1] = m.lo.d;
        } else {
#pragma unroll
          for (int k = 0; k < (1 << j); k++) {
            times(ph[k], pl[k], m.hi.d, m.lo.d, ph[k | (1 << j)], pl[k | (1 << j)]);
            times(ph[k], pl[k], m.hi.a, m.lo.a, ph[k], pl[k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < A; k++) {
        p[k] = cmul_add(ph[k], p[k], cmul(pl[k], p[k]));
        l[k] = cmul_add(ph[k], l[k], cmul(pl[k], l[k]));
      }
    }
#pragma unroll
    for (int j = 0; j < K; j++) {
      const M2x m = matrix(SIG == 2 ? 2 * j + 1 : j);
      float v[2] = {0.0f, 0.0f};
      int pair = 0;
#pragma unroll
      for (int k = 0; k < A; k++) {
        if ((k >> j) & 1) continue;
        const int h = k | (1 << j);
        v[pair++ & 1] += qmk_adj::overlap(SIG == 2 ? 2 : 1, p[k], p[h], l[k], l[h]);
        apply2x<SIG == 2 ? kMatReal : kMatRx>(m, p[k], p[h]);
        apply2x<SIG == 2 ? kMatReal : kMatRx>(m, l[k], l[h]);
      }
      add_to(SIG == 2 ? 2 * j + 1 : j, v[0] + v[1], first);
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < A; k++) {
        psi[at[k]] = p[k];
        lam[at[k]] = l[k];
      }
    }
    first = false;
  }
}

struct SmallOut {
  float2 *lam;         // co-state
  double *grad;        // gradient slots
  double *energy;
  float2 *saves;       // states kept at MAP ops
};

// TWO: the co-state sits behind the state in shared memory, then the rows of
// partial sums, in two sets so that a step's rows are added up while the next
// step runs.
template <int WORDS, bool TWO>
__global__ void __launch_bounds__(TWO ? kSmallThreads2 : kSmallThreads)
k_small(float2 *__restrict__ st, uint32_t n, uint32_t step,
        const __grid_constant__ Code<WORDS> code, const float2 *__restrict__ tables, SmallOut out) {
  extern __shared__ __align__(16) float2 amp[];
  constexpr int E = 8;   // most amplitudes a thread
  const uint32_t dim = 1u << n;
  // A helper warp's index is past every loop over amplitudes.
  const bool helper = TWO && threadIdx.x >= step;
  const uint32_t me = helper ? 1u << 30 : threadIdx.x;
  float2 *lam = amp + dim;
  float *part = reinterpret_cast<float *>(amp + (TWO ? 2 : 1) * dim);
  uint32_t *ops = reinterpret_cast<uint32_t *>(part + (TWO ? 2 * kRows * step : 0));
  {
    const uint32_t *from = code.w;
    asm volatile("" : "+l"(from));   // an address: loads of many words at once, not constants
    for (uint32_t i = threadIdx.x; i < code.count; i += blockDim.x) ops[i] = from[i];
  }
  uint32_t set = 0;
  // The rows of this step, each added up by one warp (a helper where there are
  // any). The barrier ends the step's writes to the states; the next step
  // fills the other set of rows.
  auto add_rows = [&](uint32_t rows, const uint32_t *slots, uint32_t stride, double *to) {
    const float *p = part + set * kRows * step;
    __syncthreads();
    const bool own = blockDim.x == step;
    if (own || helper) {
      const uint32_t first = own ? 0 : step / 32, warps = blockDim.x / 32 - first;
      for (uint32_t r = (threadIdx.x >> 5) - first; r < rows; r += warps) {
        const double v = row_sum(p + r * step, step);
        if ((threadIdx.x & 31) == 0) to[slots ? slots[stride * r] : 0] = v;
      }
    }
    set ^= 1u;
  };
  for (uint32_t i = me; i < dim; i += step) {
    amp[slot(i)] = st[i];
    if (TWO) lam[slot(i)] = out.lam[i];
  }
  __syncthreads();
  for (uint32_t at = 0; at < code.count;) {
    const uint32_t *w = ops + at;
    const uint32_t head = w[0];
    const uint32_t states = TWO && (head & kBoth) ? 2u : 1u;
    switch (head & 7u) {
      case kGroup: {
        const uint32_t k = (head >> 3) & 7u;
        for (uint32_t a = 0; a < states; a++) {
          float2 *x = amp + a * dim;
          if (k == 3) group_cls<3>(x, n, w, me, step);
          else if (k == 2) group_cls<2>(x, n, w, me, step);
          else group_cls<1>(x, n, w, me, step);
        }
        at += kOpHead + kMatWords * k;
        break;
      }
      case kPhase: {   // amplitudes with every mask bit set, by FP32 high and low parts
        const uint32_t mask = (head >> 8) & 0x3fffu;
        const float4 f = *reinterpret_cast<const float4 *>(w + kOpHead);
        const float2 hi = lo2(f), lo = hi2(f);
        for (uint32_t i = me; i < dim * states; i += step) {
          if ((i & mask) != mask) continue;
          float2 *a = amp + (i & dim) + slot(i & (dim - 1));
          const float2 x = *a;
          *a = make_float2(
              fmaf(hi.x, x.x, fmaf(-hi.y, x.y, fmaf(lo.x, x.x, -lo.y * x.y))),
              fmaf(hi.x, x.y, fmaf(hi.y, x.x, fmaf(lo.x, x.y, lo.y * x.x))));
        }
        at += kOpHead + 4;
        break;
      }
      case kControlled: {
        const uint32_t ctrl = (head >> 8) & 0x3fffu, q = w[1];
        const M2 m = m2(w + kOpHead);
        for (uint32_t s = me; s < dim / 2 * states; s += step) {
          const uint32_t i = ins0s(s & (dim / 2 - 1), q);
          if ((i & ctrl) != ctrl) continue;
          float2 *b = amp + ((s & (dim / 2)) << 1);
          float2 x = b[slot(i)], y = b[slot(i | (1u << q))];
          apply2(m, x, y);
          b[slot(i)] = x;
          b[slot(i | (1u << q))] = y;
        }
        at += kOpHead + 8;
        break;
      }
      case kMap: {     // amplitude y comes from the XOR of column words over y's bits
        const uint32_t save = (head >> 8) & 63u;   // 1 + the kept state's number
        float2 *kept = TWO && save ? out.saves + (static_cast<size_t>(save - 1) << n) : nullptr;
        // The image of this thread's first amplitude; the others are the first
        // one's with bits from the block's size up.
        uint32_t base = 0;
        for (uint32_t j = 0; j < n; j++)
          if ((me >> j) & 1u) base ^= w[kOpHead + j];
        const uint32_t *high = w + kOpHead + (31 - __clz(step));
        for (uint32_t a = 0; a < states; a++) {
          float2 *x = amp + a * dim;
          float2 r[E];
#pragma unroll
          for (int e = 0; e < E; e++) {
            const uint32_t y = me + e * step;
            if (y >= dim) break;
            if (TWO && a == 0 && kept && states == 2) {   // the state as it was kept
              r[e] = kept[y];
              continue;
            }
            if (TWO && kept && states == 1) kept[y] = x[slot(y)];
            uint32_t from = base;
#pragma unroll
            for (int j = 0; j < 3; j++)
              if ((e >> j) & 1) from ^= high[j];
            r[e] = x[slot(from)];
          }
          __syncthreads();
#pragma unroll
          for (int e = 0; e < E; e++) {
            const uint32_t y = me + e * step;
            if (y >= dim) break;
            x[slot(y)] = r[e];
          }
        }
        at += kOpHead + ((n + 3) & ~3u);
        break;
      }
      case kLayer: {   // a phase layer's table
        const float2 *t = tables + (static_cast<size_t>((head >> 8) & 63u) << n);
        const float sg = TWO && (head & kConj) ? -1.0f : 1.0f;
        constexpr int L = TWO ? 4 : 8;   // reads of the table in flight
#pragma unroll 1
        for (uint32_t i0 = me; i0 < dim; i0 += L * step) {
          float2 f[L];
#pragma unroll
          for (int e = 0; e < L; e++)
            if (i0 + e * step < dim) f[e] = t[i0 + e * step];
#pragma unroll
          for (int e = 0; e < L; e++) {
            if (i0 + e * step >= dim) continue;
            const uint32_t a = slot(i0 + e * step);
            f[e].y *= sg;
            amp[a] = cmul(f[e], amp[a]);
            if (TWO && states == 2) lam[a] = cmul(f[e], lam[a]);
          }
        }
        at += kOpHead;
        break;
      }
      default:
        if constexpr (TWO) {
          float *rows = part + set * kRows * step;
          if ((head & 7u) == kWindow) {
            const uint32_t k = (head >> 3) & 7u, nops = w[1];
            const uint32_t sig = w[2];
            if (k == 3 && sig == 2) window_uniform<3, 2>(amp, lam, n, w, rows, me, step);
            else if (k == 3 && sig == 1) window_uniform<3, 1>(amp, lam, n, w, rows, me, step);
            else if (k == 3) window<3>(amp, lam, n, w, rows, me, step);
            else if (k == 2 && sig == 2) window_uniform<2, 2>(amp, lam, n, w, rows, me, step);
            else if (k == 2 && sig == 1) window_uniform<2, 1>(amp, lam, n, w, rows, me, step);
            else if (k == 2) window<2>(amp, lam, n, w, rows, me, step);
            else window<1>(amp, lam, n, w, rows, me, step);
            add_rows(w[3], w + kOpHead + kItemWords * nops, 1, out.grad);
            at += kOpHead + kItemWords * nops + ((w[3] + 3) & ~3u);
            continue;
          } else if ((head & 7u) == kCostate) {
            // lambda = H psi: the Z strings' tabulated sum, then string by string.
            const uint32_t table = (head >> 8) & 63u, nt = w[1];   // 1 + the table's number
            const float2 *z = tables + (static_cast<size_t>(table - (table != 0)) << n);
            float e = 0.0f;
            for (uint32_t i = me; i < dim; i += step) {
              const float2 x = amp[slot(i)];
              const float d = table ? z[i].x : 0.0f;
              float2 s = make_float2(d * x.x, d * x.y);
              for (uint32_t t = 0; t < nt; t++) {
                const uint32_t ms = w[kOpHead + 2 * t];
                const uint32_t j = i ^ (ms & 0x1fffu);
                const float2 y = amp[slot(j)];
                const float c0 = __uint_as_float(w[kOpHead + 2 * t + 1]);
                const float c = (__popc(j & ((ms >> 13) & 0x1fffu)) & 1) != ((ms >> 27) & 1u)
                                    ? -c0 : c0;
                if ((ms >> 26) & 1u) {   // an odd number of Y
                  s.x = fmaf(-c, y.y, s.x);
                  s.y = fmaf(c, y.x, s.y);
                } else {
                  s.x = fmaf(c, y.x, s.x);
                  s.y = fmaf(c, y.y, s.y);
                }
              }
              lam[slot(i)] = s;
              e += x.x * s.x + x.y * s.y;
            }
            if (!helper) rows[me] = e;
            add_rows(1, nullptr, 0, out.energy);
            at += kOpHead + ((2 * nt + 3) & ~3u);
            continue;
          } else {
            // Gradients of Z strings, eight a step: signed sums of Im(conj(lambda) psi).
            const uint32_t ng = w[1];
            for (uint32_t g0 = 0; g0 < ng; g0 += 8) {
              rows = part + set * kRows * step;
              float s[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
              const uint32_t take = min(8u, ng - g0);
              for (uint32_t i = me; i < dim; i += step) {
                const float2 p = amp[slot(i)], l = lam[slot(i)];
                const float f = l.x * p.y - l.y * p.x;
#pragma unroll
                for (uint32_t g = 0; g < 8; g++)
                  if (g < take) s[g] += (__popc(i & w[kOpHead + 2 * (g0 + g)]) & 1) ? -f : f;
              }
#pragma unroll
              for (uint32_t g = 0; g < 8; g++)
                if (g < take && !helper) rows[g * step + me] = s[g];
              add_rows(take, w + kOpHead + 2 * g0 + 1, 2, out.grad);
            }
            at += kOpHead + ((2 * ng + 3) & ~3u);
            continue;
          }
        }
        break;
    }
    __syncthreads();
  }
  for (uint32_t i = me; i < dim; i += step) {
    st[i] = amp[slot(i)];
    if (TWO) out.lam[i] = lam[slot(i)];
  }
}

template <int WORDS, bool TWO>
int launch_small(float *state, uint32_t n, const std::vector<uint32_t> &code, const float2 *tables,
                 const SmallOut &out, cudaStream_t s) {
  static std::atomic<bool> opted[64];   // zero-initialised: false
  const unsigned most = TWO ? kSmallThreads2 : kSmallThreads;
  const unsigned threads = std::min(most, std::max(32u, (1u << n) / 8));
  auto bytes = [](uint32_t width, unsigned t) {
    return std::max<size_t>(16, (sizeof(float2) << width) * (TWO ? 2 : 1)) +
           (TWO ? 2 * kRows * t * sizeof(float) : 0) + WORDS * sizeof(uint32_t);
  };
  const size_t smem = bytes(n, threads);
  if (smem > 48 * 1024) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    if (!opted[dev]) {   // the opt-in above 48 KiB is per device
      const cudaError_t e =
          cudaFuncSetAttribute(k_small<WORDS, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(bytes(TWO ? kMaxN2 : kMaxN, most)));
      if (e != cudaSuccess) return static_cast<int>(e);
      opted[dev] = true;
    }
  }
  Code<WORDS> c;
  c.count = static_cast<uint32_t>(code.size());
  std::copy(code.begin(), code.end(), c.w);
  const unsigned all = threads + (TWO && threads <= 256 ? 32 * kHelpers : 0);
  k_small<WORDS, TWO><<<1, all, smem, s>>>(reinterpret_cast<float2 *>(state), n, threads, c, tables,
                                           out);
  return launch_status();
}

template <bool TWO>
int launch_code(float *state, uint32_t n, const std::vector<uint32_t> &code, const float2 *tables,
                const SmallOut &out, cudaStream_t s) {
  const int words = static_cast<int>(code.size());
  if (words <= kCode1) return launch_small<kCode1, TWO>(state, n, code, tables, out, s);
  if (words <= kCode2) return launch_small<kCode2, TWO>(state, n, code, tables, out, s);
  if (words <= kCode3) return launch_small<kCode3, TWO>(state, n, code, tables, out, s);
  return launch_small<kLongCode, TWO>(state, n, code, tables, out, s);
}

template <int TERMS>
int launch_tables(uint32_t n, const std::vector<qmk_phase_layer> &layers, uint32_t real,
                  float2 *tables, cudaStream_t s) {
  Layers<TERMS> ls;
  ls.count = static_cast<uint32_t>(layers.size());
  ls.real = real;
  uint32_t at = 0;
  for (uint32_t l = 0; l < ls.count; l++) {
    ls.first[l] = static_cast<uint16_t>(at);
    ls.g[l] = layers[l].global_phase;
    for (uint32_t t = 0; t < layers[l].num_terms; t++, at++) {
      ls.mask[at] = static_cast<uint16_t>(layers[l].masks[t]);
      ls.angle[at] = layers[l].angles[t];
    }
  }
  ls.first[ls.count] = static_cast<uint16_t>(at);
  k_small_tables<TERMS><<<dim3(grid_for(1u << n, 64), ls.count), 64, 0, s>>>(n, ls, tables);
  return launch_status();
}

bool same_layer(const qmk_phase_layer &a, const qmk_phase_layer &b) {
  return a.num_terms == b.num_terms && a.global_phase == b.global_phase &&
         std::equal(a.masks, a.masks + a.num_terms, b.masks) &&
         std::equal(a.angles, a.angles + a.num_terms, b.angles);
}

void put(std::vector<uint32_t> &code, const float *f, int count) {
  for (int k = 0; k < count; k++) {
    uint32_t u;
    std::memcpy(&u, f + k, 4);
    code.push_back(u);
  }
}

}  // namespace

extern "C" size_t qmk_small_workspace_bytes(uint32_t n) {
  return n >= 1 && n <= kMaxN ? (sizeof(float2) << n) * (layers_of(n) + saves_of(n)) : 0;
}

extern "C" uint32_t qmk_small_saves(uint32_t n) { return n >= 1 && n <= kMaxN ? saves_of(n) : 0; }

extern "C" uint32_t qmk_small_tables(uint32_t n) { return n >= 1 && n <= kMaxN ? layers_of(n) : 0; }

static bool needs_table(const qmk_small_op &o) {
  return o.kind == QMK_SMALL_LAYER || (o.kind == QMK_SMALL_COSTATE && o.layer.num_terms);
}

// Checks of one op; two: the ops that need the co-state are allowed; room for so
// many phase tables and kept states.
static bool small_op_ok(const qmk_small_op &o, uint32_t n, bool two, uint32_t tables,
                        uint32_t saves) {
  auto layer_ok = [&]() {
    if (o.layer.num_terms > QMK_SMALL_MAX_TERMS || (!tables && needs_table(o)) ||
        (o.layer.num_terms && (!o.layer.masks || !o.layer.angles)))
      return false;
    for (uint32_t t = 0; t < o.layer.num_terms; t++)
      if (o.layer.masks[t] >> n) return false;
    return true;
  };
  if ((o.both || o.save || o.kind >= QMK_SMALL_WINDOW) && !two) return false;
  switch (o.kind) {
    case QMK_SMALL_GROUP:
      if (o.count < 1 || o.count > 3 || !o.mats) return false;
      for (uint32_t j = 0; j < o.count; j++)
        if (o.q[j] >= n || (j && o.q[j] <= o.q[j - 1])) return false;
      return true;
    case QMK_SMALL_PHASE:
      return o.mask && !(o.mask >> n);
    case QMK_SMALL_CONTROLLED:
      return o.q[0] < n && !(o.mask >> n) && !((o.mask >> o.q[0]) & 1ull) && o.mats;
    case QMK_SMALL_MAP:
      if (!o.cols || o.save > saves) return false;
      for (uint32_t j = 0; j < n; j++)
        if (o.cols[j] >> n) return false;
      return true;
    case QMK_SMALL_LAYER:
      return layer_ok();
    case QMK_SMALL_WINDOW: {
      if (o.count < 1 || o.count > 3 || !o.num_items || o.num_items > QMK_SMALL_MAX_WINDOW ||
          !o.mats || !o.items)
        return false;
      for (uint32_t j = 0; j < o.count; j++)
        if (o.q[j] >= n || (j && o.q[j] <= o.q[j - 1])) return false;
      uint32_t grads = 0;
      for (uint32_t k = 0; k < o.num_items; k++) {
        if (o.items[3 * k] >= o.count || o.items[3 * k + 1] > 3) return false;
        grads += o.items[3 * k + 1] != 0;
      }
      return grads <= kRows;
    }
    case QMK_SMALL_COSTATE:
      if (!layer_ok() || o.num_items > QMK_SMALL_MAX_TERMS || (o.num_items && (!o.items || !o.mats)))
        return false;
      for (uint32_t t = 0; t < o.num_items; t++)
        if ((o.items[3 * t] >> n) || (o.items[3 * t + 1] >> n)) return false;
      return true;
    case QMK_SMALL_DIAG_GRAD:
      if (o.num_items > QMK_SMALL_MAX_TERMS || (o.num_items && !o.items)) return false;
      for (uint32_t t = 0; t < o.num_items; t++)
        if (o.items[2 * t] >> n) return false;
      return true;
    default:
      return false;
  }
}

extern "C" int qmk_run_small(float *state, uint32_t n, size_t num_ops, const qmk_small_op *ops,
                             const qmk_small_adjoint *adjoint, void *ws, size_t ws_bytes,
                             void *stream) {
  if (!ws || n < 1 || n > kMaxN || ws_bytes < qmk_small_workspace_bytes(n)) return -1;
  const size_t table = sizeof(float2) << n;
  uint32_t launches = 0;
  return qmk_run_small_counted(state, n, num_ops, ops, adjoint, ws, table * layers_of(n),
                               reinterpret_cast<float *>(static_cast<uint8_t *>(ws) +
                                                         table * layers_of(n)),
                               saves_of(n), stream, &launches);
}

extern "C" int qmk_run_small_counted(float *state, uint32_t n, size_t num_ops,
                                     const qmk_small_op *ops, const qmk_small_adjoint *adjoint,
                                     void *table_area, size_t table_bytes, float *saves,
                                     uint32_t num_saves, void *stream, uint32_t *launches) {
  if (!launches) return -1;
  *launches = 0;
  if (!state || n < 1 || n > kMaxN || (num_ops && !ops) ||
      (num_saves && (!saves || num_saves > saves_of(n))))
    return -1;
  const uint32_t most = static_cast<uint32_t>(std::min<size_t>(
      layers_of(n), table_area ? table_bytes / (sizeof(float2) << n) : 0));
  if (adjoint && (n > kMaxN2 || !adjoint->costate || !adjoint->grad || !adjoint->energy)) return -1;
  // Everything is checked before anything is launched.
  for (size_t k = 0; k < num_ops; k++) {
    if (!small_op_ok(ops[k], n, adjoint != nullptr, most, num_saves)) return -1;
    if (ops[k].kind == QMK_SMALL_WINDOW)
      for (uint32_t i = 0; i < ops[k].num_items; i++)
        if (ops[k].items[3 * i + 1] && ops[k].items[3 * i + 2] >= adjoint->num_grad) return -1;
    if (ops[k].kind == QMK_SMALL_DIAG_GRAD)
      for (uint32_t i = 0; i < ops[k].num_items; i++)
        if (ops[k].items[2 * i + 1] >= adjoint->num_grad) return -1;
  }
  cudaStream_t s = (cudaStream_t)stream;
  float2 *tables = static_cast<float2 *>(table_area);
  SmallOut out{};
  if (adjoint)
    out = {reinterpret_cast<float2 *>(adjoint->costate), adjoint->grad, adjoint->energy,
           reinterpret_cast<float2 *>(saves)};
  std::vector<uint32_t> code;
  std::vector<qmk_phase_layer> layers;
  uint32_t terms = 0, real = 0;
  auto flush = [&]() -> int {
    if (code.empty()) return 0;
    int rc = 0;
    *launches += layers.empty() ? 1 : 2;
    if (!layers.empty())
      rc = terms <= static_cast<uint32_t>(kShortTerms)
               ? launch_tables<kShortTerms>(n, layers, real, tables, s)
               : launch_tables<kLongTerms>(n, layers, real, tables, s);
    if (!rc)
      rc = adjoint ? launch_code<true>(state, n, code, tables, out, s)
                   : launch_code<false>(state, n, code, tables, out, s);
    code.clear();
    layers.clear();
    terms = real = 0;
    return rc;
  };
  // The layer's table in this launch; layers with the same terms share one.
  auto table_of = [&](const qmk_phase_layer &layer, bool is_real, uint32_t &l) -> int {
    l = 0;
    while (l < layers.size() &&
           !(((real >> l) & 1u) == (is_real ? 1u : 0u) && same_layer(layers[l], layer)))
      l++;
    if (l == layers.size()) {
      if (l == most || terms + layer.num_terms > static_cast<uint32_t>(kLongTerms)) {
        if (const int rc = flush()) return rc;
        l = 0;
      }
      layers.push_back(layer);
      if (is_real) real |= 1u << l;
      terms += layer.num_terms;
    }
    return 0;
  };
  auto matrix_class = [](const float *m) {
    return static_cast<uint32_t>(m2_class(m2_from(m)));
  };
  // An op's first words, filled up to kOpHead.
  auto start_op = [&](uint32_t head, uint32_t second = 0, uint32_t third = 0,
                      uint32_t fourth = 0) {
    code.insert(code.end(), {head, second, third, fourth});
  };
  auto put_matrix = [&](const qmk_small_op &o, uint32_t k) {
    put(code, o.mats + 8 * k, 8);
    const float none[8] = {};
    put(code, o.mats_lo ? o.mats_lo + 8 * k : none, 8);
  };
  // 1: one RX on every wire, 2: RZ then RY, each with its gradient; 0: any other.
  auto window_signature = [&](const qmk_small_op &o) -> uint32_t {
    const uint32_t per = o.num_items / o.count;
    if (per < 1 || per > 2 || per * o.count != o.num_items) return 0;
    for (uint32_t i = 0; i < o.num_items; i++) {
      const uint32_t gen = o.items[3 * i + 1], cls = matrix_class(o.mats + 8 * i);
      if (o.items[3 * i] != i / per) return 0;
      if (per == 1 && (gen != 1 || cls != kMatRx)) return 0;
      if (per == 2 && (i % 2 ? gen != 2 || cls != kMatReal : gen != 3 || cls != kMatDiag)) return 0;
    }
    return per;
  };
  for (size_t k = 0; k < num_ops; k++) {
    const qmk_small_op &o = ops[k];
    const uint32_t both = o.both ? kBoth : 0u;
    const size_t need = kOpHead + 3 * kMatWords + 16 + (o.kind == QMK_SMALL_WINDOW ? kItemWords + 1 : 2) * static_cast<size_t>(o.num_items);
    if (code.size() + need > static_cast<size_t>(kLongCode))
      if (const int rc = flush()) return rc;
    switch (o.kind) {
      case QMK_SMALL_GROUP: {
        bool rx = true, real_m = true;
        for (uint32_t j = 0; j < o.count; j++) {
          const float *m = o.mats + 8 * j;
          real_m = real_m && m[1] == 0.0f && m[3] == 0.0f && m[5] == 0.0f && m[7] == 0.0f;
          rx = rx && m[1] == 0.0f && m[7] == 0.0f && m[2] == 0.0f && m[4] == 0.0f;
        }
        uint32_t head = kGroup | (o.count << 3) | both |
                        (static_cast<uint32_t>(real_m ? kMatReal : rx ? kMatRx : kMatGeneral) << 6);
        for (uint32_t j = 0; j < o.count; j++) head |= o.q[j] << (8 + 5 * j);
        start_op(head);
        for (uint32_t j = 0; j < o.count; j++) put_matrix(o, j);
        break;
      }
      case QMK_SMALL_PHASE: {
        const float hi[2] = {static_cast<float>(o.phase[0]), static_cast<float>(o.phase[1])};
        const float lo[2] = {static_cast<float>(o.phase[0] - hi[0]),
                             static_cast<float>(o.phase[1] - hi[1])};
        start_op(kPhase | (static_cast<uint32_t>(o.mask) << 8) | both);
        put(code, hi, 2);
        put(code, lo, 2);
        break;
      }
      case QMK_SMALL_CONTROLLED:
        start_op(kControlled | (static_cast<uint32_t>(o.mask) << 8) | both, o.q[0]);
        put(code, o.mats, 8);
        break;
      case QMK_SMALL_MAP:
        start_op(kMap | (o.save << 8) | both);
        for (uint32_t j = 0; j < n; j++) code.push_back(static_cast<uint32_t>(o.cols[j]));
        break;
      case QMK_SMALL_LAYER: {
        uint32_t l = 0;
        if (const int rc = table_of(o.layer, false, l)) return rc;
        start_op(kLayer | (l << 8) | both | (o.conj ? kConj : 0u));
        break;
      }
      case QMK_SMALL_WINDOW: {
        uint32_t head = kWindow | (o.count << 3);
        for (uint32_t j = 0; j < o.count; j++) head |= o.q[j] << (8 + 5 * j);
        uint32_t grads = 0;
        for (uint32_t i = 0; i < o.num_items; i++) grads += o.items[3 * i + 1] != 0;
        start_op(head, o.num_items, window_signature(o), grads);
        for (uint32_t i = 0; i < o.num_items; i++) {
          const float *m = o.mats + 8 * i;
          start_op(o.items[3 * i] | (o.items[3 * i + 1] << 2) | (matrix_class(m) << 4));
          put_matrix(o, i);
        }
        for (uint32_t i = 0; i < o.num_items; i++)   // each row's gradient slot
          if (o.items[3 * i + 1]) code.push_back(o.items[3 * i + 2]);
        break;
      }
      case QMK_SMALL_COSTATE: {
        uint32_t l = 0;
        const bool z = o.layer.num_terms != 0;
        if (z)
          if (const int rc = table_of(o.layer, true, l)) return rc;
        start_op(kCostate | ((z ? l + 1 : 0u) << 8), o.num_items);
        for (uint32_t t = 0; t < o.num_items; t++) {
          code.push_back(o.items[3 * t] | (o.items[3 * t + 1] << 13) | ((o.items[3 * t + 2] & 3u) << 26));
          put(code, o.mats + t, 1);
        }
        break;
      }
      default:
        start_op(kDiagGrad, o.num_items);
        for (uint32_t t = 0; t < 2 * o.num_items; t++) code.push_back(o.items[t]);
        break;
    }
    code.resize((code.size() + 3) & ~size_t(3));
  }
  return flush();
}
