// k_stages.cu -- runs of one-wire gates and fans of controlled phases in one
// in-place pass.
//
// A Fourier transform is n stages: a Hadamard on a wire, then controlled
// phases from that wire to all lower ones. A stage took a read and a write of
// the state for its gate and one of half the state for its phases. A fan's
// phase is a product over the index bits, so a pass that holds the stages'
// own wires can apply all of them, whatever other wires the fans reach: for an
// amplitude with the stage's wire set it is the product of factors of its site
// (the wires outside the pass), its row and its lane. Their angles are exact
// integer sums of turns and each factor is rounded once, so that a phase costs
// no more accuracy than the diagonal layers' tables do. A 28-qubit transform
// is then four passes for its 28 stages: 26.8 -> 4.4 ms, and
// its error against 64 bits half of what it was (22 qubits: 4.4e-7 -> 2.2e-7).
//
// Seven stages on wires >= 6 are bound about equally by the state's read and
// write and by their multiply-adds; the pass of wires 0..5 by its
// multiply-adds and shuffles.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

#include "kcommon.cuh"
#include "../../include/qmetal/qmetal_kernels.h"

using namespace qmk;
using qmk_host::grid_for;
using qmk_host::launch_status;

namespace {

constexpr int kHigh = 7;       // stages of a pass on wires >= 6
constexpr int kRegs = 4;       // wires >= 6 beside wires 0..5
constexpr int kLow = kRegs + 6;
constexpr int kMaxOuter = 34;  // wires outside a pass

// What the stages of a pass share: S of them, on a site of 2^B rows.
template <int S, int B>
struct StageArgs {
  uint32_t act, before, after;   // bit s: stage s has a 2x2 / a phase before / after it
  M2 m[S];
  float lo[S];                   // kHadamard: what m[s].a.x lacks
  // Turns (2^-64) of each of wires 0..5, each row bit, each site-number bit.
  uint64_t lane[S][6], row[S][B], outer[S][kMaxOuter];
  uint32_t nouter;
};

// e^{2 pi i t}, t in units of 2^-64, within 0.7 ulp (rms that of one
// rounding): reduced to an eighth of a
// turn in integers, the rest in radians as FP32 high and low parts, Taylor sums
// to x^9 and x^10 (their remainders are below 2e-9), each result's leading terms
// added last.
__device__ __forceinline__ float2 unit_of(uint64_t t) {
  const uint32_t quarter = static_cast<uint32_t>((t + (1ull << 61)) >> 62);
  const long long r = static_cast<long long>(t - (static_cast<uint64_t>(quarter) << 62));
  const float hi = __ll2float_rn(r);
  const float lo = __ll2float_rn(r - static_cast<long long>(hi));
  // 2 pi 2^-64 in two parts
  constexpr double k = 6.283185307179586476925286766559 / 18446744073709551616.0;
  constexpr float kh = static_cast<float>(k), kl = static_cast<float>(k - static_cast<double>(kh));
  const float x = hi * kh;
  const float xl = fmaf(hi, kh, -x) + fmaf(hi, kl, lo * kh);
  const float z = x * x, zl = fmaf(x, x, -z), half = 0.5f * z;
  const float ps =
      z * fmaf(z, fmaf(z, fmaf(z, 1.0f / 362880.0f, -1.0f / 5040.0f), 1.0f / 120.0f), -1.0f / 6.0f);
  const float s = x + fmaf(x, ps, xl * (1.0f - half));
  const float pc = fmaf(z, fmaf(z, fmaf(z, -1.0f / 3628800.0f, 1.0f / 40320.0f), -1.0f / 720.0f),
                        1.0f / 24.0f);
  const float w = 1.0f - half;
  const float c = w + (((1.0f - w) - half) + fmaf(z * z, pc, fmaf(-x, xl, -0.5f * zl)));
  const float a = (quarter & 1u) ? s : c, b = (quarter & 1u) ? c : s;
  return make_float2(((quarter + 1u) & 2u) ? -a : a, (quarter & 2u) ? -b : b);
}

// The turns of the set bits of x.
template <int B>
__device__ __forceinline__ uint64_t sum_turns(const uint64_t (&turns)[B], uint32_t x) {
  uint64_t t = 0;
#pragma unroll
  for (int j = 0; j < B; j++) t += ((x >> j) & 1u) ? turns[j] : 0ull;
  return t;
}

// Stage s's turns of the wires outside the pass.
template <int S>
__device__ __forceinline__ uint64_t site_turns(const uint64_t (&outer)[S][kMaxOuter],
                                               uint32_t nouter, int s, uint64_t site) {
  uint64_t t = 0;
  for (uint32_t k = 0; k < nouter; k++) t += (site >> k & 1ull) ? outer[s][k] : 0ull;
  return t;
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// c [[1, 1], [1, -1]], c as FP32 high and low parts: 1/sqrt(2) narrowed to FP32
// is off by 1.7e-8, in the same direction at every stage, which was most of a
// transform's error (22 qubits: 3.7e-7 of 4.4e-7).
constexpr int kHadamard = 4;

template <int CLS>
__device__ __forceinline__ void stage_pair(const M2 &m, float lo, float2 &u, float2 &v) {
  if (CLS == kHadamard) {
    const float2 p = make_float2(u.x + v.x, u.y + v.y), q = make_float2(u.x - v.x, u.y - v.y);
    u = make_float2(fmaf(m.a.x, p.x, lo * p.x), fmaf(m.a.x, p.y, lo * p.y));
    v = make_float2(fmaf(m.a.x, q.x, lo * q.x), fmaf(m.a.x, q.y, lo * q.y));
  } else {
    apply2c(CLS, m, u, v);
  }
}

// One side of the pair: the amplitude whose wire is `one`.
template <int CLS>
__device__ __forceinline__ float2 stage_side(const M2 &m, float lo, bool one, float2 own,
                                             float2 other) {
  if (CLS == kHadamard) {
    const float2 t = one ? make_float2(other.x - own.x, other.y - own.y)
                         : make_float2(own.x + other.x, own.y + other.y);
    return make_float2(fmaf(m.a.x, t.x, lo * t.x), fmaf(m.a.x, t.y, lo * t.y));
  }
  return cmac2c(CLS, one ? m.d : m.a, own, one ? m.c : m.b, other);
}

// The vector times the two amplitudes' factors.
__device__ __forceinline__ float4 turned(const float4 &x, float2 f, const float4 &lanes) {
  return pack4(cmul(cmul(f, lo2(lanes)), lo2(x)), cmul(cmul(f, hi2(lanes)), hi2(x)));
}

// Up to seven stages on wires >= 6, in order: row bit j is stage j's wire. The
// block tile of k_group_blk: stages 0..3 pair registers in the first layout,
// stages 4..6 in the second, one shared-memory transpose between; the next
// site streams in meanwhile.
struct HighSite {
  uint32_t pos[kHigh];   // vector bit (wire - 1) of each row bit
  uint32_t asc[kHigh];   // the same, ascending
};

// ALL: seven stages, each a 2x2 and then its phase, without a test of each.
template <int CLS, bool ALL>
__global__ void __launch_bounds__(kThreads, 2)
k_stages_high(float4 *__restrict__ st, uint64_t nsites, HighSite h, StageArgs<kHigh, kHigh> g) {
  constexpr int NV = 16;
  extern __shared__ __align__(16) float4 site[];   // [row][32 lanes]
  __shared__ uint64_t outer[kHigh][kMaxOuter];
  __shared__ __align__(16) float2 lanes[kHigh][64];
  __shared__ uint64_t row_turns[kHigh][1 << kHigh];
  __shared__ uint64_t turns[2][kHigh];                 // of a site, two sites ahead
  __shared__ float2 rows[2][kHigh][1 << kHigh];        // factors of a site and its rows
  __shared__ uint64_t row_off[kThreads / 32][2][NV];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto row_a = [&](int l) { return static_cast<uint32_t>(l) | (warp << 4); };
  auto row_b = [&](int l) {
    return warp | ((static_cast<uint32_t>(l) >> 3) << 3) | ((static_cast<uint32_t>(l) & 7u) << 4);
  };
  {
    const int l = lane & (NV - 1);
    const uint32_t row = lane < NV ? row_a(l) : row_b(l);
    uint64_t v = 0;
#pragma unroll
    for (int j = 0; j < kHigh; j++)
      if ((row >> j) & 1u) v |= 1ull << h.pos[j];
    row_off[warp][lane / NV][l] = v;
  }
#pragma unroll
  for (int s = 0; s < kHigh; s++) {
    if (tid < 64) lanes[s][tid] = unit_of(sum_turns(g.lane[s], tid));
    else if (tid < 192) row_turns[s][tid - 64] = sum_turns(g.row[s], tid - 64);
    else if (tid - 192 < kMaxOuter) outer[s][tid - 192] = g.outer[s][tid - 192];
  }
  auto base_of = [&](uint64_t sidx) {
    uint64_t b = sidx * 32 + lane;
#pragma unroll
    for (int j = 0; j < kHigh; j++) b = ins0(b, h.asc[j]);
    return b;
  };
  auto prefetch = [&](uint64_t sidx) {
    if (sidx < nsites) {
      const uint64_t base = base_of(sidx);
#pragma unroll
      for (int l = 0; l < NV; l++)
        cp_async16(site + row_a(l) * 32 + lane, st + (base | row_off[warp][0][l]));
    }
    cp_async_commit();
  };
  auto form_turns = [&](uint64_t sidx, uint32_t to) {
    if (tid < kHigh && sidx < nsites) turns[to][tid] = site_turns(outer, g.nouter, tid, sidx);
  };
  auto form_rows = [&](uint32_t to) {   // from turns[to]
    for (uint32_t e = tid; e < (kHigh << kHigh); e += kThreads) {
      const uint32_t s = e >> kHigh, row = e & ((1u << kHigh) - 1u);
      if (ALL || (((g.before | g.after) >> s) & 1u))
        rows[to][s][row] = unit_of(turns[to][s] + row_turns[s][row]);
    }
  };
  uint32_t set = 0;
  __syncthreads();   // the tables
  prefetch(blockIdx.x);
  form_turns(blockIdx.x, 0);
  form_turns(static_cast<uint64_t>(blockIdx.x) + gridDim.x, 1);
  __syncthreads();
  form_rows(0);
  for (uint64_t sidx = blockIdx.x; sidx < nsites; sidx += gridDim.x) {
    float4 r[NV];
    cp_async_wait_all();   // this thread's copies of this site
    __syncthreads();       // the site's factors, the next one's turns
    auto phase = [&](int bit, int s, auto &&row_of) {
      const float4 two = *reinterpret_cast<const float4 *>(&lanes[s][2 * lane]);
#pragma unroll
      for (int l = 0; l < NV; l++)
        if ((l >> bit) & 1) r[l] = turned(r[l], rows[set][s][row_of(l)], two);
    };
    auto stage = [&](int bit, int s, auto &&row_of) {
      if (!ALL && ((g.before >> s) & 1u)) phase(bit, s, row_of);
      if (ALL || ((g.act >> s) & 1u)) {
#pragma unroll
        for (int l = 0; l < NV; l++) {
          if ((l >> bit) & 1) continue;
          const int u = l | (1 << bit);
          float2 a0 = lo2(r[l]), b0 = lo2(r[u]), a1 = hi2(r[l]), b1 = hi2(r[u]);
          stage_pair<CLS>(g.m[s], g.lo[s], a0, b0);
          stage_pair<CLS>(g.m[s], g.lo[s], a1, b1);
          r[l] = pack4(a0, a1);
          r[u] = pack4(b0, b1);
        }
      }
      if (ALL || ((g.after >> s) & 1u)) phase(bit, s, row_of);
    };
#pragma unroll
    for (int l = 0; l < NV; l++) r[l] = site[row_a(l) * 32 + lane];
#pragma unroll
    for (int s = 0; s < 4; s++) stage(s, s, row_a);
#pragma unroll
    for (int l = 0; l < NV; l++) site[row_a(l) * 32 + lane] = r[l];
    __syncthreads();   // the first layout is written back
#pragma unroll
    for (int l = 0; l < NV; l++) r[l] = site[row_b(l) * 32 + lane];
    __syncthreads();   // every warp has read its second layout: the slots are free
    const uint64_t next = sidx + gridDim.x;
    prefetch(next);
    if (next < nsites) form_rows(set ^ 1u);
    form_turns(next + gridDim.x, set);
#pragma unroll
    for (int s = 4; s < kHigh; s++) stage(s - 4, s, row_b);
    const uint64_t base = base_of(sidx);
#pragma unroll
    for (int l = 0; l < NV; l++) st[base | row_off[warp][1][l]] = r[l];
    set ^= 1u;
  }
  cp_async_wait_all();
}

// Up to four stages on wires >= 6, then up to six on wires 0..5 in any order:
// a warp tile (lanes = wires 1..5), no barrier after the tables are made.
struct LowSite {
  uint32_t pos[kRegs];   // site-number bit (wire - 6) of each row bit
  uint32_t asc[kRegs];
  uint32_t nlow;
  uint32_t wire[6];      // the low stages' wires: stages kRegs..
};

template <int CLS>
__global__ void __launch_bounds__(kThreads, 2)
k_stages_low(float4 *__restrict__ st, uint64_t nsites, LowSite h, StageArgs<kLow, kRegs> g) {
  constexpr int NV = 1 << kRegs;
  __shared__ uint64_t outer[kLow][kMaxOuter];
  __shared__ __align__(16) float2 lanes[kLow][64];
  __shared__ float2 rows[kLow][NV];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
#pragma unroll
  for (int s = 0; s < kLow; s++) {
    if (tid < 64) lanes[s][tid] = unit_of(sum_turns(g.lane[s], tid));
    else if (tid < 64 + NV) rows[s][tid - 64] = unit_of(sum_turns(g.row[s], tid - 64));
    else if (tid >= 96 && tid - 96 < kMaxOuter) outer[s][tid - 96] = g.outer[s][tid - 96];
  }
  __syncthreads();
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (kThreads / 32);
  for (uint64_t ws = (static_cast<uint64_t>(blockIdx.x) * kThreads + tid) >> 5; ws < nsites;
       ws += warps) {
    uint64_t b = ws;
#pragma unroll
    for (int j = 0; j < kRegs; j++) b = ins0(b, h.asc[j]);
    const uint64_t base = (b << 5) | lane;
    auto vec_of = [&](int l) {
      uint64_t v = base;
#pragma unroll
      for (int j = 0; j < kRegs; j++)
        if ((l >> j) & 1) v |= 1ull << (h.pos[j] + 5);
      return v;
    };
    float4 r[NV];
#pragma unroll
    for (int l = 0; l < NV; l++) r[l] = st[vec_of(l)];
    const float2 mine = lane < kLow ? unit_of(site_turns(outer, g.nouter, lane, ws))
                                    : make_float2(1.0f, 0.0f);
    // Stage s's factor where its wire is set: low wire q, or register bit `bit`.
    auto phase = [&](int s, int bit, uint32_t q) {
      const float2 f = make_float2(__shfl_sync(0xffffffffu, mine.x, s),
                                   __shfl_sync(0xffffffffu, mine.y, s));
      float4 two = *reinterpret_cast<const float4 *>(&lanes[s][2 * lane]);
      if (bit >= 0) {
#pragma unroll
        for (int l = 0; l < NV; l++)
          if ((l >> bit) & 1) r[l] = turned(r[l], cmul(f, rows[s][l]), two);
      } else if (q == 0) {   // the odd amplitude of each vector
#pragma unroll
        for (int l = 0; l < NV; l++)
          r[l] = pack4(lo2(r[l]), cmul(cmul(cmul(f, rows[s][l]), hi2(two)), hi2(r[l])));
      } else if ((lane >> (q - 1)) & 1u) {
#pragma unroll
        for (int l = 0; l < NV; l++) r[l] = turned(r[l], cmul(f, rows[s][l]), two);
      }
      __syncwarp();
    };
#pragma unroll
    for (int s = 0; s < kRegs; s++) {
      if ((g.before >> s) & 1u) phase(s, s, 0);
      if ((g.act >> s) & 1u) {
#pragma unroll
        for (int l = 0; l < NV; l++) {
          if ((l >> s) & 1) continue;
          const int u = l | (1 << s);
          float2 a0 = lo2(r[l]), b0 = lo2(r[u]), a1 = hi2(r[l]), b1 = hi2(r[u]);
          stage_pair<CLS>(g.m[s], g.lo[s], a0, b0);
          stage_pair<CLS>(g.m[s], g.lo[s], a1, b1);
          r[l] = pack4(a0, a1);
          r[u] = pack4(b0, b1);
        }
      }
      if ((g.after >> s) & 1u) phase(s, s, 0);
    }
#pragma unroll 1
    for (uint32_t i = 0; i < h.nlow; i++) {
      const int s = kRegs + static_cast<int>(i);
      const uint32_t q = h.wire[i];
      if ((g.before >> s) & 1u) phase(s, -1, q);
      if ((g.act >> s) & 1u) {
        const M2 m = g.m[s];
        const float lo = g.lo[s];
        if (q == 0) {
#pragma unroll
          for (int l = 0; l < NV; l++) {
            float2 x = lo2(r[l]), y = hi2(r[l]);
            stage_pair<CLS>(m, lo, x, y);
            r[l] = pack4(x, y);
          }
        } else {
          const bool one = (lane >> (q - 1)) & 1u;
#pragma unroll
          for (int l = 0; l < NV; l++) {
            const float4 o = shfl4(r[l], 1 << (q - 1));
            r[l] = pack4(stage_side<CLS>(m, lo, one, lo2(r[l]), lo2(o)),
                         stage_side<CLS>(m, lo, one, hi2(r[l]), hi2(o)));
          }
        }
      }
      if ((g.after >> s) & 1u) phase(s, -1, q);
    }
#pragma unroll
    for (int l = 0; l < NV; l++) st[vec_of(l)] = r[l];
  }
}

// An angle as turns in units of 2^-64. The quotient's rounding is 2^-52 of it: of
// many turns, the angle within one turn comes from its cosine and sine, which
// the C library reduces without loss.
uint64_t turns(double angle) {
  if (std::abs(angle) > 1024.0) angle = std::atan2(std::sin(angle), std::cos(angle));
  double t = angle / (2.0 * 3.14159265358979323846);
  t -= std::floor(t);
  const double x = std::ldexp(t, 64);
  return x >= 18446744073709551616.0 ? 0 : static_cast<uint64_t>(x);
}

// Stage o as stage s of a pass: bit_of[w] is wire w's bit of the (site, site
// number) index, 0..5 wires 0..5, then B row bits, then the site number's.
template <int S, int B>
void put_stage(StageArgs<S, B> &g, int s, const qmk_stage &o, uint32_t n, const uint32_t *bit_of) {
  if (o.has_matrix) {
    g.act |= 1u << s;
    g.m[s] = m2_from(o.m);
    g.lo[s] = o.m_lo;
  }
  if (!o.phase) return;
  (o.phase == 1 ? g.after : g.before) |= 1u << s;
  for (uint32_t w = 0; w < n; w++) {
    const uint32_t b = bit_of[w];
    const uint64_t t = turns(o.angles[w]);
    if (b < 6) g.lane[s][b] = t;
    else if (b < 6 + B) g.row[s][b - 6] = t;
    else g.outer[s][b - 6 - B] = t;
  }
}

// The class all matrices of a pass share.
int stage_class(uint32_t count, const qmk_stage *stages) {
  bool real = true, hadamard = true;
  for (uint32_t k = 0; k < count; k++) {
    if (!stages[k].has_matrix) continue;
    const M2 m = m2_from(stages[k].m);
    real = real && m.a.y == 0.0f && m.b.y == 0.0f && m.c.y == 0.0f && m.d.y == 0.0f;
    hadamard = hadamard && real && m.b.x == m.a.x && m.c.x == m.a.x && m.d.x == -m.a.x;
  }
  return hadamard ? kHadamard : real ? kMatReal : kMatGeneral;
}

template <int CLS>
int launch_low(float4 *st, uint64_t nsites, const LowSite &h, const StageArgs<kLow, kRegs> &g,
               cudaStream_t s) {
  const unsigned grid = std::min(grid_for(nsites, kThreads / 32),
                                 static_cast<unsigned>(qmk_host::num_sms()) * 2);
  k_stages_low<CLS><<<grid, kThreads, 0, s>>>(st, nsites, h, g);
  return launch_status();
}

template <int CLS, bool ALL>
int launch_high_as(float4 *st, uint64_t nsites, const HighSite &h, const StageArgs<kHigh, kHigh> &g,
                cudaStream_t s) {
  constexpr size_t smem = (size_t(1) << kHigh) * 32 * sizeof(float4);
  static std::atomic<bool> opted[64];   // zero-initialised: false
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!opted[dev]) {   // the opt-in above 48 KiB is per device
    const cudaError_t e = cudaFuncSetAttribute(
        k_stages_high<CLS, ALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    opted[dev] = true;
  }
  const unsigned grid = static_cast<unsigned>(
      std::min<uint64_t>(nsites, static_cast<uint64_t>(qmk_host::num_sms()) * 2));
  k_stages_high<CLS, ALL><<<grid, kThreads, smem, s>>>(st, nsites, h, g);
  return launch_status();
}

template <int CLS>
int launch_high(float4 *st, uint64_t nsites, const HighSite &h, const StageArgs<kHigh, kHigh> &g,
                cudaStream_t s) {
  constexpr uint32_t every = (1u << kHigh) - 1u;
  return g.act == every && g.after == every && !g.before
             ? launch_high_as<CLS, true>(st, nsites, h, g, s)
             : launch_high_as<CLS, false>(st, nsites, h, g, s);
}

}  // namespace

extern "C" int qmk_apply_stages(float *state, uint32_t n, uint32_t count, const qmk_stage *stages,
                                void *stream) {
  if (!state || (reinterpret_cast<uintptr_t>(state) & 15u) || n < 13 || n > 40 || count < 1 ||
      count > kLow || !stages)
    return -1;
  uint64_t high = 0, seen = 0;
  uint32_t nhigh = 0;
  for (uint32_t k = 0; k < count; k++) {
    const qmk_stage &o = stages[k];
    if (o.wire >= n || ((seen >> o.wire) & 1ull) || o.phase > 2 || (o.phase && !o.angles)) return -1;
    for (uint32_t w = 0; o.phase && w < n; w++)
      if (!std::isfinite(o.angles[w])) return -1;
    seen |= 1ull << o.wire;
    if (o.wire >= 6) {
      if (nhigh != k) return -1;   // wires >= 6 come first
      high |= 1ull << o.wire;
      nhigh++;
    }
  }
  const bool low = nhigh < count;
  const uint32_t rows = low ? kRegs : kHigh;
  if (nhigh > rows) return -1;
  // Row bit j is stage j's wire; the lowest free wires >= 6 fill up.
  std::vector<uint32_t> row_wire;
  for (uint32_t k = 0; k < nhigh; k++) row_wire.push_back(stages[k].wire);
  for (uint32_t w = 6; row_wire.size() < rows; w++)
    if (!((high >> w) & 1ull)) row_wire.push_back(w);
  std::vector<uint32_t> bit_of(n, 0), sorted = row_wire;
  std::sort(sorted.begin(), sorted.end());
  uint32_t out = 6 + rows;
  for (uint32_t w = 0; w < n; w++) {
    if (w < 6) {
      bit_of[w] = w;
      continue;
    }
    const auto it = std::find(row_wire.begin(), row_wire.end(), w);
    bit_of[w] = it == row_wire.end() ? out++ : 6 + static_cast<uint32_t>(it - row_wire.begin());
  }
  const uint32_t nouter = n - 6 - rows;
  if (nouter > static_cast<uint32_t>(kMaxOuter)) return -1;
  const uint64_t nsites = 1ull << nouter;
  const int cls = stage_class(count, stages);
  float4 *st = reinterpret_cast<float4 *>(state);
  cudaStream_t s = (cudaStream_t)stream;
  if (low) {
    LowSite h{};
    StageArgs<kLow, kRegs> g{};
    g.nouter = nouter;
    for (int j = 0; j < kRegs; j++) {
      h.pos[j] = row_wire[j] - 6;
      h.asc[j] = sorted[j] - 6;
    }
    for (uint32_t k = 0; k < count; k++) {
      const int at = k < nhigh ? static_cast<int>(k) : kRegs + static_cast<int>(k - nhigh);
      put_stage(g, at, stages[k], n, bit_of.data());
      if (k >= nhigh) h.wire[h.nlow++] = stages[k].wire;
    }
    switch (cls) {
      case kHadamard: return launch_low<kHadamard>(st, nsites, h, g, s);
      case kMatReal: return launch_low<kMatReal>(st, nsites, h, g, s);
      default: return launch_low<kMatGeneral>(st, nsites, h, g, s);
    }
  }
  HighSite h{};
  StageArgs<kHigh, kHigh> g{};
  g.nouter = nouter;
  for (int j = 0; j < kHigh; j++) {
    h.pos[j] = row_wire[j] - 1;
    h.asc[j] = sorted[j] - 1;
  }
  for (uint32_t k = 0; k < count; k++) put_stage(g, static_cast<int>(k), stages[k], n, bit_of.data());
  switch (cls) {
    case kHadamard: return launch_high<kHadamard>(st, nsites, h, g, s);
    case kMatReal: return launch_high<kMatReal>(st, nsites, h, g, s);
    default: return launch_high<kMatGeneral>(st, nsites, h, g, s);
  }
}
