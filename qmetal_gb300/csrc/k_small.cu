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
// Bound by latency: a barrier, shared-memory round trip and up to three
// dependent 2x2s an op. The 9-qubit U3 circuit of depth 10 with its read-out:
// 310 -> 75 us; where the line of 13 qubits lies a 13-wire layer takes what
// its two group launches took, above it the state no longer fits twice.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <vector>

#include "kcommon.cuh"
#include "../../include/qmetal/qmetal_kernels.h"

using namespace qmk;
using qmk_host::grid_for;
using qmk_host::launch_status;

namespace {

constexpr uint32_t kMaxN = QMK_SMALL_MAX_QUBITS;
constexpr uint32_t kMaxLayers = 32;        // phase tables per launch
constexpr unsigned kSmallThreads = 1024;   // widest block: eight amplitudes a thread at 13 qubits

// The ops as words, in two sizes of kernel arguments (4 KiB and the limit of
// 32 KiB; the smaller one launches faster).
template <int WORDS>
struct Code {
  uint32_t count;        // words used
  uint32_t w[WORDS];
};
constexpr int kShortCode = 960, kLongCode = 8000;

// A phase layer of the first launch: merged terms and the constant.
template <int TERMS>
struct Layers {
  uint32_t count;
  uint16_t first[kMaxLayers + 1];
  uint16_t mask[TERMS];
  double g[kMaxLayers];
  double angle[TERMS];
};
constexpr int kShortTerms = 320, kLongTerms = 3000;

enum : uint32_t { kGroup = 0, kPhase = 1, kControlled = 2, kMap = 3, kLayer = 4 };

// Bound by its FP64 sums and sincos: two-warp blocks spread it over the chip.
template <int TERMS>
__global__ void __launch_bounds__(64)
k_small_tables(uint32_t n, const Layers<TERMS> ls, float2 *__restrict__ tables) {
  const uint32_t i = blockIdx.x * 64 + threadIdx.x, l = blockIdx.y;
  if (i >= (1u << n)) return;
  double f = ls.g[l];
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

__device__ __forceinline__ float2 f2(const uint32_t *w) {
  return make_float2(__uint_as_float(w[0]), __uint_as_float(w[1]));
}
__device__ __forceinline__ M2 m2(const uint32_t *w) {
  return {f2(w), f2(w + 2), f2(w + 4), f2(w + 6)};
}

// K 2x2s on distinct wires q[0] < q[1] < q[2]: 2^K amplitudes in registers.
template <int K, int CLS>
__device__ __forceinline__ void group(float2 *amp, uint32_t n, const uint32_t *w) {
  uint32_t q[K];
#pragma unroll
  for (int j = 0; j < K; j++) q[j] = (w[0] >> (8 + 5 * j)) & 31u;
  for (uint32_t s = threadIdx.x; s < (1u << (n - K)); s += blockDim.x) {
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
      const M2 m = m2(w + 1 + 8 * j);
#pragma unroll
      for (int l = 0; l < (1 << K); l++)
        if (!((l >> j) & 1)) apply2c(CLS, m, r[l], r[l | (1 << j)]);
    }
#pragma unroll
    for (int l = 0; l < (1 << K); l++) amp[at[l]] = r[l];
  }
}

template <int K>
__device__ __forceinline__ void group_cls(float2 *amp, uint32_t n, const uint32_t *w) {
  switch ((w[0] >> 6) & 3u) {
    case kMatReal: group<K, kMatReal>(amp, n, w); break;
    case kMatRx: group<K, kMatRx>(amp, n, w); break;
    default: group<K, kMatGeneral>(amp, n, w); break;
  }
}

template <int WORDS>
__global__ void __launch_bounds__(kSmallThreads)
k_small(float2 *__restrict__ st, uint32_t n, const __grid_constant__ Code<WORDS> code,
        const float2 *__restrict__ tables) {
  extern __shared__ __align__(16) float2 amp[];
  const uint32_t dim = 1u << n, step = blockDim.x;
  for (uint32_t i = threadIdx.x; i < dim; i += step) amp[slot(i)] = st[i];
  __syncthreads();
  for (uint32_t at = 0; at < code.count;) {
    const uint32_t *w = code.w + at;
    const uint32_t head = w[0];
    switch (head & 7u) {
      case kGroup: {
        const uint32_t k = (head >> 3) & 7u;
        if (k == 3) group_cls<3>(amp, n, w);
        else if (k == 2) group_cls<2>(amp, n, w);
        else group_cls<1>(amp, n, w);
        at += 1 + 8 * k;
        break;
      }
      case kPhase: {   // amplitudes with every mask bit set, by FP32 high and low parts
        const uint32_t mask = head >> 8;
        const float2 hi = f2(w + 1), lo = f2(w + 3);
        for (uint32_t i = threadIdx.x; i < dim; i += step) {
          if ((i & mask) != mask) continue;
          const float2 x = amp[slot(i)];
          amp[slot(i)] = make_float2(
              fmaf(hi.x, x.x, fmaf(-hi.y, x.y, fmaf(lo.x, x.x, -lo.y * x.y))),
              fmaf(hi.x, x.y, fmaf(hi.y, x.x, fmaf(lo.x, x.y, lo.y * x.x))));
        }
        at += 5;
        break;
      }
      case kControlled: {
        const uint32_t ctrl = head >> 8, q = w[1];
        const M2 m = m2(w + 2);
        for (uint32_t s = threadIdx.x; s < dim / 2; s += step) {
          const uint32_t i = ins0s(s, q);
          if ((i & ctrl) != ctrl) continue;
          const uint32_t a = slot(i), b = slot(i | (1u << q));
          float2 x = amp[a], y = amp[b];
          apply2(m, x, y);
          amp[a] = x;
          amp[b] = y;
        }
        at += 10;
        break;
      }
      case kMap: {     // amplitude y comes from the XOR of column words over y's bits
        float2 r[8];   // dim / blockDim.x is at most 8
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const uint32_t y = threadIdx.x + e * step;
          if (y >= dim) break;
          uint32_t x = 0;
          for (uint32_t j = 0; j < n; j++)
            if ((y >> j) & 1u) x ^= w[1 + j];
          r[e] = amp[slot(x)];
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const uint32_t y = threadIdx.x + e * step;
          if (y >= dim) break;
          amp[slot(y)] = r[e];
        }
        at += 1 + n;
        break;
      }
      default: {       // a phase layer's table
        const float2 *t = tables + (static_cast<size_t>(head >> 8) << n);
        for (uint32_t i = threadIdx.x; i < dim; i += step) {
          const uint32_t a = slot(i);
          amp[a] = cmul(t[i], amp[a]);
        }
        at += 1;
        break;
      }
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < dim; i += step) st[i] = amp[slot(i)];
}

template <int WORDS>
int launch_small(float *state, uint32_t n, const std::vector<uint32_t> &code, const float2 *tables,
                 cudaStream_t s) {
  static std::atomic<bool> opted[64];   // zero-initialised: false
  const size_t smem = sizeof(float2) << n;
  if (smem > 48 * 1024) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    if (!opted[dev]) {   // the opt-in above 48 KiB is per device
      const cudaError_t e = cudaFuncSetAttribute(
          k_small<WORDS>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(float2) << kMaxN);
      if (e != cudaSuccess) return static_cast<int>(e);
      opted[dev] = true;
    }
  }
  Code<WORDS> c;
  c.count = static_cast<uint32_t>(code.size());
  std::copy(code.begin(), code.end(), c.w);
  const unsigned threads = std::min(kSmallThreads, std::max(32u, (1u << n) / 8));
  k_small<WORDS><<<1, threads, smem, s>>>(reinterpret_cast<float2 *>(state), n, c, tables);
  return launch_status();
}

template <int TERMS>
int launch_tables(uint32_t n, const std::vector<qmk_phase_layer> &layers, float2 *tables,
                  cudaStream_t s) {
  Layers<TERMS> ls;
  ls.count = static_cast<uint32_t>(layers.size());
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
  return n >= 1 && n <= kMaxN ? (sizeof(float2) << n) * kMaxLayers : 0;
}

extern "C" int qmk_run_small(float *state, uint32_t n, size_t num_ops, const qmk_small_op *ops,
                             void *ws, size_t ws_bytes, void *stream) {
  if (!state || n < 1 || n > kMaxN || (num_ops && !ops) || !ws ||
      ws_bytes < qmk_small_workspace_bytes(n))
    return -1;
  // Everything is checked before anything is launched.
  for (size_t k = 0; k < num_ops; k++) {
    const qmk_small_op &o = ops[k];
    switch (o.kind) {
      case QMK_SMALL_GROUP:
        if (o.count < 1 || o.count > 3 || !o.mats) return -1;
        for (uint32_t j = 0; j < o.count; j++)
          if (o.q[j] >= n || (j && o.q[j] <= o.q[j - 1])) return -1;
        break;
      case QMK_SMALL_PHASE:
        if (!o.mask || (o.mask >> n)) return -1;
        break;
      case QMK_SMALL_CONTROLLED:
        if (o.q[0] >= n || (o.mask >> n) || ((o.mask >> o.q[0]) & 1ull) || !o.mats) return -1;
        break;
      case QMK_SMALL_MAP:
        if (!o.cols) return -1;
        for (uint32_t j = 0; j < n; j++)
          if (o.cols[j] >> n) return -1;
        break;
      case QMK_SMALL_LAYER:
        if (o.layer.num_terms > QMK_SMALL_MAX_TERMS ||
            (o.layer.num_terms && (!o.layer.masks || !o.layer.angles)))
          return -1;
        for (uint32_t t = 0; t < o.layer.num_terms; t++)
          if (o.layer.masks[t] >> n) return -1;
        break;
      default:
        return -1;
    }
  }
  cudaStream_t s = (cudaStream_t)stream;
  float2 *tables = static_cast<float2 *>(ws);
  std::vector<uint32_t> code;
  std::vector<qmk_phase_layer> layers;
  uint32_t terms = 0;
  auto flush = [&]() -> int {
    if (code.empty()) return 0;
    int rc = 0;
    if (!layers.empty())
      rc = terms <= static_cast<uint32_t>(kShortTerms)
               ? launch_tables<kShortTerms>(n, layers, tables, s)
               : launch_tables<kLongTerms>(n, layers, tables, s);
    if (!rc)
      rc = code.size() <= static_cast<size_t>(kShortCode)
               ? launch_small<kShortCode>(state, n, code, tables, s)
               : launch_small<kLongCode>(state, n, code, tables, s);
    code.clear();
    layers.clear();
    terms = 0;
    return rc;
  };
  for (size_t k = 0; k < num_ops; k++) {
    const qmk_small_op &o = ops[k];
    if (code.size() + 32 > static_cast<size_t>(kLongCode))
      if (const int rc = flush()) return rc;
    switch (o.kind) {
      case QMK_SMALL_GROUP: {
        bool rx = true, real = true;
        for (uint32_t j = 0; j < o.count; j++) {
          const float *m = o.mats + 8 * j;
          real = real && m[1] == 0.0f && m[3] == 0.0f && m[5] == 0.0f && m[7] == 0.0f;
          rx = rx && m[1] == 0.0f && m[7] == 0.0f && m[2] == 0.0f && m[4] == 0.0f;
        }
        uint32_t head = kGroup | (o.count << 3) |
                        (static_cast<uint32_t>(real ? kMatReal : rx ? kMatRx : kMatGeneral) << 6);
        for (uint32_t j = 0; j < o.count; j++) head |= o.q[j] << (8 + 5 * j);
        code.push_back(head);
        put(code, o.mats, static_cast<int>(8 * o.count));
        break;
      }
      case QMK_SMALL_PHASE: {
        const float hi[2] = {static_cast<float>(o.phase[0]), static_cast<float>(o.phase[1])};
        const float lo[2] = {static_cast<float>(o.phase[0] - hi[0]),
                             static_cast<float>(o.phase[1] - hi[1])};
        code.push_back(kPhase | (static_cast<uint32_t>(o.mask) << 8));
        put(code, hi, 2);
        put(code, lo, 2);
        break;
      }
      case QMK_SMALL_CONTROLLED:
        code.push_back(kControlled | (static_cast<uint32_t>(o.mask) << 8));
        code.push_back(o.q[0]);
        put(code, o.mats, 8);
        break;
      case QMK_SMALL_MAP:
        code.push_back(kMap);
        for (uint32_t j = 0; j < n; j++) code.push_back(static_cast<uint32_t>(o.cols[j]));
        break;
      default: {
        // Layers with the same terms share a table.
        size_t l = 0;
        while (l < layers.size() && !same_layer(layers[l], o.layer)) l++;
        if (l == layers.size()) {
          if (l == kMaxLayers || terms + o.layer.num_terms > static_cast<uint32_t>(kLongTerms)) {
            if (const int rc = flush()) return rc;
            l = 0;
          }
          layers.push_back(o.layer);
          terms += o.layer.num_terms;
        }
        code.push_back(kLayer | (static_cast<uint32_t>(l) << 8));
        break;
      }
    }
  }
  return flush();
}
