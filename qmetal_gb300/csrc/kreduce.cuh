// kreduce.cuh -- the deterministic device-wide reduction used by every
// kernel that returns numbers (norms, expectations, energies, gradients).
//
// Each block reduces its accumulators, FP64 or FP32 pairs (warp shuffles, then shared
// memory) into per-block partials in the workspace; the last block to finish
// (atomic ticket) sums the partials in a fixed order and hands each total to
// an output functor. A result depends only on the grid size, never on timing.
#pragma once

#include <algorithm>

#include "kcommon.cuh"

size_t qmk_reduce_area_offset();  // k_diag.cu

namespace qmk {

constexpr uint32_t kMaxBlocks = 1024;

struct Area {
  double *partials;   // kMaxBlocks x 32
  unsigned *counter;  // last-block ticket, back to 0 after each reduction
  unsigned *waits;    // bounded waits that gave up in passes on this workspace
  unsigned *polls;    // 0: waits take the full bound; k > 0: they give up after k - 1 polls
};

inline Area area_of(void *ws) {
  uint8_t *b = static_cast<uint8_t *>(ws) + qmk_reduce_area_offset();
  Area a;
  a.partials = reinterpret_cast<double *>(b);
  a.counter = reinterpret_cast<unsigned *>(b + kMaxBlocks * 32 * sizeof(double));
  a.waits = a.counter + 16;  // 64 bytes into the 256-byte tail, its own line
  a.polls = a.counter + 32;  // 128 bytes in: a test's poll limit for those waits
  return a;
}

inline unsigned reduce_grid() {
  return std::min<unsigned>(kMaxBlocks, static_cast<unsigned>(qmk_host::num_sms()) * 4);
}

// out[t] = s (or out[t] += s).
struct OutContig {
  double *p;
  bool add;
  __device__ void operator()(int t, double s) const { p[t] = add ? p[t] + s : s; }
};

// out[slot[t]] = s: results scattered to their gate's gradient entry.
template <int T>
struct OutSlots {
  double *p;
  uint32_t slot[T];
  __device__ void operator()(int t, double s) const { p[slot[t]] = s; }
};

// A sum as FP32 high and low parts, exact to about 2^-46, for sums of FP32
// values: an FP64 add or conversion holds a multiprocessor's FP64 unit for 16
// cycles a warp, these dozen FP32 operations three. An infinite sum has no low
// part.
struct Two {
  float hi, lo;
};
__device__ __forceinline__ Two add(Two a, Two b) {
  const float s = __fadd_rn(a.hi, b.hi), t = __fadd_rn(s, -a.hi);
  const float e = __fadd_rn(__fadd_rn(a.hi, -__fadd_rn(s, -t)), __fadd_rn(b.hi, -t));
  float lo = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
  if (isinf(s)) lo = 0.0f;
  const float hi = __fadd_rn(s, lo);
  lo = __fadd_rn(lo, -__fadd_rn(hi, -s));
  if (isinf(hi)) lo = 0.0f;
  return {hi, lo};
}
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ double widen(Two v) {
  return static_cast<double>(v.hi) + static_cast<double>(v.lo);
}
// a + v for a long run of FP32 values, seven operations: the low part collects
// what each sum loses and is settled once, at the run's end.
__device__ __forceinline__ Two gather(Two a, float v) {
  const float s = __fadd_rn(a.hi, v), t = __fadd_rn(s, -a.hi);
  const float e = __fadd_rn(__fadd_rn(a.hi, -__fadd_rn(s, -t)), __fadd_rn(v, -t));
  return {s, __fadd_rn(a.lo, e)};
}
__device__ __forceinline__ Two settle(Two a) {
  if (!isfinite(a.hi)) a.lo = 0.0f;
  return add(a, Two{0.0f, 0.0f});
}
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ Two shfl_xor(Two v, int mask) {
  return {__shfl_xor_sync(0xffffffffu, v.hi, mask), __shfl_xor_sync(0xffffffffu, v.lo, mask)};
}
__device__ __forceinline__ double shfl_xor(double v, int mask) {
  return __shfl_xor_sync(0xffffffffu, v, mask);
}
__device__ __forceinline__ Two load_partial(const Two *p) {
  const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
  return {v.x, v.y};
}
__device__ __forceinline__ double load_partial(const double *p) { return __ldcg(p); }

__host__ __device__ constexpr int pow2_at_least(int t) {
  return t <= 1 ? 1 : 2 * pow2_at_least((t + 1) / 2);
}

// Transposed butterfly over P = 2^k slots: each step halves the slots a lane
// carries and trades the other half with its partner, so lane l ends with
// slot l % P summed over the warp: P - 1 exchanges for P slots instead of
// 5 P (FP64 adds run at a small fraction of the FP32 rate on this part).
template <int P, typename V>
__device__ __forceinline__ V warp_slot_sums(V (&v)[P], int l) {
#pragma unroll
  for (int h = P / 2; h >= 1; h >>= 1) {
    const bool upper = (l & h) != 0;
#pragma unroll
    for (int j = 0; j < h; j++) {
      const V send = upper ? v[j] : v[j + h];
      const V keep = upper ? v[j + h] : v[j];
      v[j] = add(keep, shfl_xor(send, h));
    }
  }
#pragma unroll
  for (int o = P; o < 32; o <<= 1) v[0] = add(v[0], shfl_xor(v[0], o));
  return v[0];
}

// Partials per block: 32 doubles, or 64 for reductions of more than 32
// results (their grids stay within kMaxBlocks / 2 blocks).
template <int T>
constexpr int partial_stride() {
  return T > 32 ? 64 : 32;
}

// V: double, or Two for threads that hold FP32 sums (the adjoint passes; with
// FP64 adds and conversions there, a block's end took 6100 cycles of its
// multiprocessor for sixteen results, of 24 us in all at 20 qubits).
template <int T, typename V, typename Out>
__device__ __forceinline__ void finish_as(const V (&acc)[T], int nt, Area a, const Out &out) {
  static_assert(T >= 1 && T <= 64, "at most 64 results per reduction");
  static_assert(sizeof(V) == sizeof(double), "the partials' slots hold eight bytes");
  constexpr int kStride = partial_stride<T>();
  __shared__ V red[kThreads / 32][T];
  __shared__ unsigned ticket;
  V *partials = reinterpret_cast<V *>(a.partials);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  {
    // Slots 0..31, then 32..T-1, one butterfly each.
    constexpr int T0 = T < 32 ? T : 32;
    constexpr int P = pow2_at_least(T0);
    V v[P];
#pragma unroll
    for (int t = 0; t < P; t++) v[t] = t < T0 ? acc[t < T0 ? t : 0] : V{};
    const V sum = warp_slot_sums(v, l);
    if (l < T0) red[w][l] = sum;
    if constexpr (T > 32) {
      constexpr int T1 = T - 32;
      constexpr int P1 = pow2_at_least(T1);
      V u[P1];
#pragma unroll
      for (int t = 0; t < P1; t++) u[t] = t < T1 ? acc[t < T1 ? 32 + t : 0] : V{};
      const V more = warp_slot_sums(u, l);
      if (l < T1) red[w][32 + l] = more;
    }
  }
  __syncthreads();
  if (threadIdx.x < static_cast<unsigned>(nt)) {
    V s = V{};
    for (int k = 0; k < kThreads / 32; k++) s = add(s, red[k][threadIdx.x]);
    partials[blockIdx.x * kStride + threadIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) ticket = atomicAdd(a.counter, 1u);
  __syncthreads();
  if (ticket != gridDim.x - 1) return;
  __threadfence();
  // The last block: kThreads / P threads a result, four partials in flight
  // each, then a shared-memory tree. One thread a result (608 dependent FP64
  // adds at this part's FP64 rate) took 14-40 us of every reducing pass.
  constexpr int P = pow2_at_least(T);
  constexpr unsigned G = kThreads / P;
  __shared__ V tail[kThreads];
  const unsigned t = threadIdx.x % P, g = threadIdx.x / P;
  V s[4] = {};
  if (t < static_cast<unsigned>(nt)) {
    for (unsigned b = g; b < gridDim.x; b += 4 * G) {
      V x[4];
#pragma unroll
      for (unsigned k = 0; k < 4; k++)
        x[k] = b + k * G < gridDim.x ? load_partial(&partials[(b + k * G) * kStride + t]) : V{};
#pragma unroll
      for (unsigned k = 0; k < 4; k++) s[k] = add(s[k], x[k]);
    }
  }
  tail[threadIdx.x] = add(add(s[0], s[1]), add(s[2], s[3]));
  __syncthreads();
  for (unsigned h = G / 2; h >= 1; h /= 2) {
    if (g < h) tail[threadIdx.x] = add(tail[threadIdx.x], tail[threadIdx.x + h * P]);
    __syncthreads();
  }
  if (threadIdx.x < static_cast<unsigned>(nt))
    out(static_cast<int>(threadIdx.x), widen(tail[threadIdx.x]));
  if (threadIdx.x == 0) *a.counter = 0u;
}

template <int T, typename Out>
__device__ __forceinline__ void finish(double (&acc)[T], int nt, Area a, const Out &out) {
  finish_as<T, double>(acc, nt, a, out);
}

// For threads that hold what gather() adds up.
template <int T, typename Out>
__device__ __forceinline__ void finish(Two (&acc)[T], int nt, Area a, const Out &out) {
  Two v[T];
#pragma unroll
  for (int t = 0; t < T; t++) v[t] = settle(acc[t]);
  finish_as<T, Two>(v, nt, a, out);
}

// For threads that hold FP32 sums.
template <int T, typename Out>
__device__ __forceinline__ void finish(float (&acc)[T], int nt, Area a, const Out &out) {
  Two v[T];
#pragma unroll
  for (int t = 0; t < T; t++) v[t] = {acc[t], 0.0f};
  finish_as<T, Two>(v, nt, a, out);
}

}  // namespace qmk
