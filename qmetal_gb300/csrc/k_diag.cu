// k_diag.cu -- the fused diagonal layer: amplitude i *= exp(i phi(i)),
//   phi(i) = g + sum_t angle_t [mask_t fully set in i].
//
// Every mask the plan builder emits has one or two bits (Z/S/T/P/RZ, CZ/CP,
// and the three terms of a ZZ coupling), so after merging equal masks phi is
// a quadratic form in the index bits:
//   phi(i) = g + sum_q a_q x_q + sum_{q<r} b_qr x_q x_r .
// The reference evaluates every term per amplitude in FP32 (kernels.metal:
// 203-218), which stops being bandwidth bound near 75 terms. Here the index
// splits into a tile of W low bits (lo) and the tile number (hi):
//   phi = [g + phi_H(hi)] + sum_{r<W} x_r c_r(hi) + phi_L(lo)
// with c_r(hi) = sum of b_rq over partners q >= W set in hi (cross pairs).
//   * phi_L (low singles + low-low pairs) is the same for every tile: a prep
//     kernel tabulates TL[lo] = e^{i phi_L(lo)} once per layer (FP64 sums,
//     double sincos).
//   * per tile, the FP64 sums c_r(hi) and g + phi_H(hi) are formed once and
//     turned into factors f_r = e^{i c_r}, eH = e^{i(g+phi_H)}; the linear
//     part splits over bits 0..5 and 6..W-1 into two small tables Y1, Y2.
//   * per amplitude: factor = TL[lo] * Y1[lo & 63] * Y2[lo >> 6], then one
//     complex multiply of the amplitude.
// Where every mask holds a common wire (a QFT stage: CP(k, j) for all k < j)
// the half of the state with that bit clear keeps its phase and is not read.
// A layer of one term is a masked phase: no table, and only the amplitudes
// the mask picks (a 22-qubit QFT gate by gate, 231 CP: 6.25 -> 2.88 ms).
// Masks of three or more bits (never produced by the plan passes) go through
// a direct per-amplitude FP64 kernel.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "kquad.cuh"
#include "../../include/qmetal/qmetal_kernels.h"

using namespace qmk;
using qmk_host::grid_for;
using qmk_host::launch_status;

// Offsets shared with the reduction kernels.
size_t qmk_reduce_area_offset() { return kDescBytes + kTableBytes; }

namespace {

__global__ void __launch_bounds__(kThreads)
k_diag(float4 *__restrict__ st, const DiagDesc *__restrict__ d,
       const float4 *__restrict__ table4, uint64_t nparts, uint32_t part_bits, int tile_bit,
       int vec_bit) {
  __shared__ float2 f[kWMax];
  __shared__ float2 eH;
  __shared__ __align__(16) float2 Y1[64];
  __shared__ float2 Y2[1 << (kWMax - 6)];
  const uint32_t W = d->W;
  const uint32_t tid = threadIdx.x;
  // tile_bit / vec_bit >= 0: only tiles / vectors with that bit set. A block
  // takes one of the 2^part_bits equal parts of a tile's vectors.
  const uint32_t nv = 1u << ((vec_bit < 0 ? W - 1 : W - 2) - part_bits);
  auto vec = [&](uint32_t e) {
    return vec_bit < 0 ? e : static_cast<uint32_t>(ins0(e, vec_bit)) | (1u << vec_bit);
  };
  for (uint64_t kp = blockIdx.x; kp < nparts; kp += gridDim.x) {
    const uint64_t k = kp >> part_bits;
    const uint32_t first = (static_cast<uint32_t>(kp) & ((1u << part_bits) - 1u)) * nv;
    const uint64_t tile = tile_bit < 0 ? k : ins0(k, tile_bit) | (1ull << tile_bit);
    tile_coeffs<true>(d, tile, f, &eH, nullptr, nullptr, false);
    __syncthreads();
    tile_phase_tables(W, f, eH, Y1, Y2);
    __syncthreads();
    const uint64_t base = tile << (W - 1);
    constexpr int UU = 4;
    for (uint32_t e0 = tid; e0 < nv; e0 += kThreads * UU) {
      float4 x[UU], t[UU];
#pragma unroll
      for (int k = 0; k < UU; k++) {
        const uint32_t e = e0 + k * kThreads;
        if (e < nv) {
          x[k] = st[base + vec(first + e)];
          t[k] = table4[vec(first + e)];
        }
      }
#pragma unroll
      for (int k = 0; k < UU; k++) {
        const uint32_t e = e0 + k * kThreads;
        if (e >= nv) continue;
        const uint32_t lo = 2 * vec(first + e);
        const float4 y1 = *reinterpret_cast<const float4 *>(&Y1[lo & 63]);
        const float2 y2 = Y2[lo >> 6];
        const float2 f0 = cmul(cmul(lo2(t[k]), lo2(y1)), y2);
        const float2 f1 = cmul(cmul(hi2(t[k]), hi2(y1)), y2);
        st[base + vec(first + e)] = pack4(cmul(f0, lo2(x[k])), cmul(f1, hi2(x[k])));
      }
    }
    __syncthreads();
  }
}

constexpr int kGenericTerms = 64;
struct GenericTerms {
  uint32_t count;
  uint64_t mask[kGenericTerms];
  double angle[kGenericTerms];
};

// Direct evaluation, one amplitude per thread: only for masks of >= 3 bits.
__global__ void k_diag_generic(float2 *__restrict__ st, uint64_t dim, GenericTerms g) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= dim) return;
  double phi = 0.0;
  for (uint32_t t = 0; t < g.count; t++)
    if ((i & g.mask[t]) == g.mask[t]) phi += g.angle[t];
  st[i] = cmul(expi_reduced(phi), st[i]);
}

// A diagonal layer and then 2x2s on K wires >= 13 in one pass. A thread holds
// the 2^K vectors that the wires pick, one of each of 2^K tiles, so the layer's
// table is read once for all of them and the 2x2s pair registers. The same
// arithmetic in the same order as the layer's pass and then a group's.
//
// A Trotter step of 25 wires is then four passes instead of five (the layer,
// 10 + 7 + 7 + 1 wires), a QAOA layer of 28 wires too (10 + 7 + 7 + 4). Bound by
// the state's read and write: at 28 qubits the layer alone takes 646 us, the
// group of one to four wires 607 to 619, both in one pass 661 to 698 (0.95 to
// 0.91 of the copy rate); at 20 qubits 14.6, 5.1 to 5.4, and 14.7 to 19.0.
constexpr int kDiagWires = 4;
struct DiagGroupArgs {
  uint32_t pos[kDiagWires];   // tile-number bits (wire - 13), ascending
  M2 m[kDiagWires];
};

__host__ __device__ constexpr int diag_group_unroll(int k) { return k == 1 ? 2 : k == 2 ? 1 : 0; }

template <int K, int CLS>
__global__ void __launch_bounds__(kThreads, K == 4 ? 2 : 3)
k_diag_group(float4 *__restrict__ st, const DiagDesc *__restrict__ d,
             const float4 *__restrict__ table4, uint64_t nparts, uint32_t part_bits,
             DiagGroupArgs g) {
  constexpr int NT = 1 << K;
  constexpr int UN = 1 << diag_group_unroll(K);   // vectors of each tile in flight
  constexpr uint32_t kVecs = 1u << (kWMax - 1);
  __shared__ float2 f[NT][kWMax];
  __shared__ float2 eH[NT];
  __shared__ __align__(16) float2 Y1[NT][64];
  __shared__ float2 Y2[NT][1 << (kWMax - 6)];
  __shared__ uint64_t off[NT];   // vector t of a thread against vector 0
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  if (tid < NT) {
    uint64_t v = 0;
#pragma unroll
    for (int j = 0; j < K; j++)
      if ((tid >> j) & 1u) v |= static_cast<uint64_t>(kVecs) << g.pos[j];
    off[tid] = v;
  }
  // A block takes one of the 2^part_bits equal parts of the tiles' vectors.
  const uint32_t nv = kVecs >> part_bits;
  for (uint64_t sp = blockIdx.x; sp < nparts; sp += gridDim.x) {
    const uint32_t first = (static_cast<uint32_t>(sp) & ((1u << part_bits) - 1u)) * nv;
    uint64_t tile0 = sp >> part_bits;
#pragma unroll
    for (int j = 0; j < K; j++) tile0 = ins0(tile0, g.pos[j]);
    auto tile_of = [&](int t) {
      uint64_t tile = tile0;
#pragma unroll
      for (int j = 0; j < K; j++)
        if ((t >> j) & 1) tile |= 1ull << g.pos[j];
      return tile;
    };
    for (int t = static_cast<int>(warp); t < NT; t += kThreads / 32)
      warp_tile_coeffs(d, tile_of(t), f[t], &eH[t]);
    __syncthreads();
    for (int t = 0; t < NT; t++) tile_phase_tables(kWMax, f[t], eH[t], Y1[t], Y2[t]);
    __syncthreads();
    float4 *row0 = st + tile0 * kVecs;
    for (uint32_t e0 = first + tid; e0 < first + nv; e0 += kThreads * UN) {
      float4 r[UN][NT], x[UN];
#pragma unroll
      for (int u = 0; u < UN; u++) {
        x[u] = table4[e0 + u * kThreads];
#pragma unroll
        for (int t = 0; t < NT; t++) r[u][t] = row0[off[t] + e0 + u * kThreads];
      }
#pragma unroll
      for (int u = 0; u < UN; u++) {
        const uint32_t lo = 2 * (e0 + u * kThreads);
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const float4 y1 = *reinterpret_cast<const float4 *>(&Y1[t][lo & 63]);
          const float2 y2 = Y2[t][lo >> 6];
          const float2 f0 = cmul(cmul(lo2(x[u]), lo2(y1)), y2);
          const float2 f1 = cmul(cmul(hi2(x[u]), hi2(y1)), y2);
          r[u][t] = pack4(cmul(f0, lo2(r[u][t])), cmul(f1, hi2(r[u][t])));
          if (NT >= 8 && t % 4 == 3) asm volatile("" ::: "memory");   // factors four at a time
        }
#pragma unroll
        for (int j = 0; j < K; j++) {
#pragma unroll
          for (int t = 0; t < NT; t++) {
            if ((t >> j) & 1) continue;
            float4 &a = r[u][t], &b = r[u][t | (1 << j)];
            float2 a0 = lo2(a), b0 = lo2(b), a1 = hi2(a), b1 = hi2(b);
            apply2c(CLS, g.m[j], a0, b0);
            apply2c(CLS, g.m[j], a1, b1);
            a = pack4(a0, a1);
            b = pack4(b0, b1);
          }
        }
#pragma unroll
        for (int t = 0; t < NT; t++) row0[off[t] + e0 + u * kThreads] = r[u][t];
      }
    }
    __syncthreads();
  }
}

template <int K>
void launch_diag_group(int cls, float4 *st, const DiagDesc *d, const float4 *table4,
                       uint64_t nsuper, const DiagGroupArgs &g, cudaStream_t s) {
  const uint32_t bits = tile_part_bits(nsuper, kWMax - 1, 8 + diag_group_unroll(K));
  const uint64_t np = nsuper << bits;
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(
      np, static_cast<uint64_t>(qmk_host::num_sms()) * (K == 4 ? 2 : 3)));
  switch (cls) {
    case kMatReal: k_diag_group<K, kMatReal><<<grid, kThreads, 0, s>>>(st, d, table4, np, bits, g); break;
    case kMatRx: k_diag_group<K, kMatRx><<<grid, kThreads, 0, s>>>(st, d, table4, np, bits, g); break;
    default: k_diag_group<K, kMatGeneral><<<grid, kThreads, 0, s>>>(st, d, table4, np, bits, g); break;
  }
}

// One term of one to three wires and no global phase.
bool diagonal_is_phase(uint32_t n, uint32_t nt, const uint64_t *masks, double global_phase) {
  return nt == 1 && global_phase == 0.0 && masks[0] && !(masks[0] >> n) &&
         __builtin_popcountll(masks[0]) <= 3;
}

}  // namespace

extern "C" size_t qmk_workspace_bytes(uint32_t n) {
  (void)n;
  // Reduction area: 1024 blocks x 32 doubles of partials, then a counter.
  return kDescBytes + kTableBytes + 1024 * 32 * sizeof(double) + 256;
}

extern "C" size_t qmk_workspace_scratch_bytes(uint32_t n) {
  return n >= 1 ? qmk_workspace_bytes(n) - 256 : 0;   // all but the counters of the reductions
}

extern "C" int qmk_workspace_init(void *ws, size_t bytes, void *stream) {
  if (!ws || bytes < qmk_workspace_bytes(0)) return -1;
  cudaError_t e = cudaMemsetAsync(ws, 0, bytes, (cudaStream_t)stream);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

extern "C" int qmk_apply_diagonal(float *state, uint32_t n, uint32_t nt,
                                  const uint64_t *masks, const double *angles,
                                  double global_phase, void *ws,
                                  size_t ws_bytes, void *stream) {
  if (!state || n < 1 || n > 40 || (nt && (!masks || !angles))) return -1;
  if (!ws || ws_bytes < qmk_workspace_bytes(n)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  if (diagonal_is_phase(n, nt, masks, global_phase))
    return qmk_apply_phase64(state, n, masks[0], std::cos(angles[0]), std::sin(angles[0]), stream);
  const uint32_t W = std::min<uint32_t>(n, kWMax);
  DiagDesc d;
  std::vector<uint64_t> gm;
  std::vector<double> ga;
  if (build_quad_desc(n, nt, masks, angles, global_phase, d, &gm, &ga) != 0) return -1;

  uint8_t *base = static_cast<uint8_t *>(ws);
  DiagDesc *dd = reinterpret_cast<DiagDesc *>(base);
  float2 *table = reinterpret_cast<float2 *>(base + kDescBytes);
  k_quad_prep<true><<<grid_for(1u << W, kPrepThreads), kPrepThreads, 0, s>>>(d, dd, table);
  int rc = launch_status();
  if (rc) return rc;
  // The highest wire that every mask holds (wires 0 and 1 save no sectors).
  uint64_t common = nt && global_phase == 0.0 ? ~0ull : 0;
  for (uint32_t t = 0; t < nt; t++) common &= masks[t];
  common &= ~3ull;
  const int q = common ? 63 - __builtin_clzll(common) : -1;
  const int tile_bit = q >= static_cast<int>(W) ? q - static_cast<int>(W) : -1;
  const int vec_bit = q >= 0 && q < static_cast<int>(W) ? q - 1 : -1;
  const uint64_t ntiles = 1ull << (n - W - (tile_bit >= 0 ? 1 : 0));
  const uint64_t cap = static_cast<uint64_t>(qmk_host::num_sms()) * 8;
  const uint32_t part_bits = tile_part_bits(ntiles, vec_bit < 0 ? W - 1 : W - 2);
  const uint64_t nparts = ntiles << part_bits;
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(nparts, cap));
  k_diag<<<grid, kThreads, 0, s>>>(reinterpret_cast<float4 *>(state), dd,
                                   reinterpret_cast<const float4 *>(table), nparts, part_bits,
                                   tile_bit, vec_bit);
  rc = launch_status();
  if (rc) return rc;
  for (size_t b = 0; b < gm.size(); b += kGenericTerms) {
    GenericTerms g{};
    g.count = static_cast<uint32_t>(std::min<size_t>(kGenericTerms, gm.size() - b));
    for (uint32_t k = 0; k < g.count; k++) {
      g.mask[k] = gm[b + k];
      g.angle[k] = ga[b + k];
    }
    const uint64_t dim = 1ull << n;
    k_diag_generic<<<grid_for(dim, kThreads), kThreads, 0, s>>>(
        reinterpret_cast<float2 *>(state), dim, g);
    rc = launch_status();
    if (rc) return rc;
  }
  return 0;
}

extern "C" int qmk_apply_diagonal_group(float *state, uint32_t n, uint32_t nt,
                                        const uint64_t *masks, const double *angles,
                                        double global_phase, uint32_t k, const uint32_t *wires,
                                        const float *mats, void *ws, size_t ws_bytes,
                                        void *stream) {
  if (!state || (reinterpret_cast<uintptr_t>(state) & 15u) || n < kWMax + 1 || n > 40 ||
      (nt && (!masks || !angles)) || k < 1 || k > static_cast<uint32_t>(kDiagWires) || !wires || !mats)
    return -1;
  if (!ws || ws_bytes < qmk_workspace_bytes(n)) return -1;
  DiagGroupArgs g{};
  bool rx = true, real = true;
  for (uint32_t j = 0; j < k; j++) {
    if (wires[j] < kWMax || wires[j] >= n || (j && wires[j] <= wires[j - 1])) return -1;
    g.pos[j] = wires[j] - kWMax;
    g.m[j] = m2_from(mats + 8 * j);
    const M2 &m = g.m[j];
    real = real && m.a.y == 0.0f && m.b.y == 0.0f && m.c.y == 0.0f && m.d.y == 0.0f;
    rx = rx && m.a.y == 0.0f && m.d.y == 0.0f && m.b.x == 0.0f && m.c.x == 0.0f;
  }
  DiagDesc d;
  if (build_quad_desc(n, nt, masks, angles, global_phase, d, nullptr, nullptr) != 0) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  uint8_t *base = static_cast<uint8_t *>(ws);
  DiagDesc *dd = reinterpret_cast<DiagDesc *>(base);
  k_quad_prep<true><<<grid_for(1u << d.W, kPrepThreads), kPrepThreads, 0, s>>>(d, dd,
                                                                               base + kDescBytes);
  const int rc = launch_status();
  if (rc) return rc;
  const int cls = real ? kMatReal : rx ? kMatRx : kMatGeneral;
  const uint64_t nsuper = 1ull << (n - kWMax - k);
  float4 *st = reinterpret_cast<float4 *>(state);
  const float4 *table = reinterpret_cast<const float4 *>(base + kDescBytes);
  switch (k) {
    case 1: launch_diag_group<1>(cls, st, dd, table, nsuper, g, s); break;
    case 2: launch_diag_group<2>(cls, st, dd, table, nsuper, g, s); break;
    case 3: launch_diag_group<3>(cls, st, dd, table, nsuper, g, s); break;
    default: launch_diag_group<4>(cls, st, dd, table, nsuper, g, s); break;
  }
  return launch_status();
}
