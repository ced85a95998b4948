// k_expect.cu -- expectation values of many Pauli strings at once: Z strings
// (one read of the state for up to 32), single X terms (one read for up to
// seven wires >= 6 and wires 0..5), and narrow states (one block per string,
// one launch for all).
//
// Precision: an amplitude's or a pair's product is rounded to FP32, and sums of
// them are FP32 high and low parts from there (gather(), then the block and grid
// sums of finish()). Sums of 128 and 32 products in FP32 first had two to four
// times the error (15 qubits, rms: Z strings 7.0e-9, now 1.9e-9; X terms 4.3e-9,
// now 1.1e-9). X terms from 22 qubits on add four pairs in FP32 first: errors of
// 6e-10 and less, where sums of eight pairs and FP64 from there had the same.
#include <algorithm>
#include <atomic>
#include <vector>

#include "kreduce.cuh"
#include "../../include/qmetal/qmetal_kernels.h"

using namespace qmk;
using qmk_host::grid_for;
using qmk_host::launch_status;

namespace {

// ---------------------------------------------------------------------------
// Z strings. A thread takes 32 amplitudes -- amplitude bit 0 and vector bits
// 5..8 (wires 0 and 6..9), so a warp's loads are whole 512-byte rows -- and
// transforms their probabilities by a 32-point Walsh-Hadamard transform in
// registers: entry c is then the sum over the 32 with the sign of the bits of
// c, so each string costs one entry and one sign instead of 32 signed adds.
// Each probability goes in two parts: its multiple of 2^-18 of a power of two
// above the thread's largest, whose sums of 32 are exact in FP32, and the rest,
// whose transform rounds 2^-19 lower.
// Strings by the sign word: bit t is the parity of string t over the thread's
// lane bits (once per kernel) and over the warp's site number (one string per
// lane, a ballot per site).
//
// One block a multiprocessor: the sums take 64 registers a thread, the next
// site's vectors 64 while they arrive. Bound by the read of the state and the
// transforms' adds about equally.

constexpr int kZTerms = 32;

struct ZTermArgs {
  uint32_t nt;
  uint32_t hi[kZTerms][2];      // mask over the site number (wires 10..), 64 bits
  uint8_t lane[kZTerms];        // mask over lane bits (wires 1..5)
  uint8_t coef[kZTerms];        // transform entry: wire 0, wires 6..9
};

__device__ __forceinline__ void transform32(float (&p)[32]) {
#pragma unroll
  for (int h = 1; h < 32; h <<= 1) {
#pragma unroll
    for (int i = 0; i < 32; i++) {
      if (i & h) continue;
      const float u = p[i], v = p[i | h];
      p[i] = u + v;
      p[i | h] = u - v;
    }
  }
}

template <int T>
__global__ void __launch_bounds__(kThreads, 1)
k_zterms(const float4 *__restrict__ st, uint64_t nwsites, ZTermArgs z, Area a, OutContig out) {
  extern __shared__ __align__(16) float2 zsm[];
  float2 *w = zsm + threadIdx.x;   // [32][kThreads]
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t gw = (static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5;
  const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (kThreads / 32);
  uint32_t lsign = 0;
#pragma unroll
  for (int t = 0; t < T; t++)
    lsign |= (static_cast<uint32_t>(__popc(lane & z.lane[t])) & 1u) << t;
  const uint64_t mine =   // the site mask of the string this lane answers for
      lane < T ? (static_cast<uint64_t>(z.hi[lane][1]) << 32) | z.hi[lane][0] : 0ull;
  Two acc[T] = {};
  float4 x[16];
  auto load = [&](uint64_t ws) {
    const float4 *row = st + (ws << 9) + lane;
#pragma unroll
    for (int l = 0; l < 16; l++) x[l] = row[l * 32];
  };
  if (gw < nwsites) load(gw);
  for (uint64_t ws = gw; ws < nwsites; ws += nwarps) {
    float h[32], r[32], most = 0.0f;
#pragma unroll
    for (int l = 0; l < 16; l++) {
      r[2 * l] = fmaf(x[l].x, x[l].x, x[l].y * x[l].y);
      r[2 * l + 1] = fmaf(x[l].z, x[l].z, x[l].w * x[l].w);
      most = fmaxf(most, fmaxf(r[2 * l], r[2 * l + 1]));
    }
    if (ws + nwarps < nwsites) load(ws + nwarps);
    // c = 1.5 * 2^(e + 6) for most in [2^e, 2^(e + 1)): adding it rounds to a
    // multiple of 2^(e - 17). Without a part where that or a sum would overflow.
    const uint32_t e = __float_as_uint(most) & 0x7f800000u;
    const bool parts = e < (240u << 23);
    const float c = parts ? __uint_as_float((e + (6u << 23)) | 0x400000u) : 0.0f;
#pragma unroll
    for (int i = 0; i < 32; i++) {
      h[i] = __fadd_rn(__fadd_rn(r[i], c), -c);
      r[i] = __fadd_rn(r[i], -h[i]);
    }
    if (!parts) {
#pragma unroll
      for (int i = 0; i < 32; i++) r[i] = 0.0f;
    }
    transform32(h);
    transform32(r);
#pragma unroll
    for (int i = 0; i < 32; i++) w[i * kThreads] = make_float2(h[i], r[i]);
    const uint32_t sign = lsign ^ __ballot_sync(0xffffffffu, parity64(ws & mine));
#pragma unroll
    for (int t = 0; t < T; t++) {
      const float2 v = w[z.coef[t] * kThreads];
      const uint32_t minus = (sign << (31 - t)) & 0x80000000u;
      acc[t] = gather(acc[t], __uint_as_float(__float_as_uint(v.x) ^ minus));
      acc[t].lo = __fadd_rn(acc[t].lo, __uint_as_float(__float_as_uint(v.y) ^ minus));
    }
  }
  finish<T>(acc, static_cast<int>(z.nt), a, out);
}

template <typename K>
int opt_in(K kernel, size_t smem, std::atomic<bool> (&opted)[64]) {
  // The opt-in above 48 KiB is per device; set it once on each.
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!opted[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    opted[dev] = true;
  }
  return 0;
}

template <int T>
int launch_z(const float4 *st, uint64_t nwsites, const ZTermArgs &z, Area a, OutContig out,
             cudaStream_t s) {
  static std::atomic<bool> opted[64];   // zero-initialised: false
  const size_t smem = kThreads * 32 * sizeof(float2);
  if (const int rc = opt_in(k_zterms<T>, smem, opted)) return rc;
  const unsigned grid = std::min<unsigned>(grid_for(nwsites, kThreads / 32),
                                           static_cast<unsigned>(qmk_host::num_sms()));
  k_zterms<T><<<grid, kThreads, smem, s>>>(st, nwsites, z, a, out);
  return launch_status();
}

// ---------------------------------------------------------------------------
// Single X terms: out[k] = sum over pairs (i, i ^ (1 << w)) of Re(conj(psi_i)
// psi_j), each pair once. A site is 2^(4 + WB) rows of 32 vectors picked by
// the pass's wires >= 6, in shared memory (streamed in by cp.async while the
// block works on the site before); a warp holds sixteen of the rows in
// registers. Pairs across the four wires that pick a warp's rows are register
// pairs; across the others one vector of each pair is read from the partner
// warp's rows, the pair going to the warp whose bit equals the row's parity
// bit so that both do half; wires 1..5 read the partner lane, wire 0 is the
// other half of the vector.
//
// Bound by the read of the state and its adds about equally: a pass reads the
// state once for up to 13 wires where one wire at a time read it 13 times.

struct XTermArgs {
  uint32_t pos[7];     // vector bits (wire - 1) of the site's wires >= 6, ascending
};

// out[slot[t]] = s where the caller asked for wire t.
template <int T>
struct OutWanted {
  double *p;
  int8_t slot[T];
  __device__ void operator()(int t, double s) const {
    if (slot[t] >= 0) p[slot[t]] = s;
  }
};

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

__device__ __forceinline__ float re_dot(const float4 &x, const float4 &y) {
  return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, x.w * y.w)));
}

// Where a thread's products go. RUNS: four pairs (two vectors) are added in
// FP32, then the run to the sum; otherwise every pair by itself.
template <bool RUNS>
struct XSum {
  Two &acc;
  float run = 0.0f;
  __device__ __forceinline__ explicit XSum(Two &a) : acc(a) {}
  __device__ __forceinline__ void vectors(const float4 &x, const float4 &y) {
    if (RUNS) {
      run += re_dot(x, y);
    } else {
      acc = gather(acc, fmaf(x.x, y.x, x.y * y.y));
      acc = gather(acc, fmaf(x.z, y.z, x.w * y.w));
    }
  }
  __device__ __forceinline__ void halves(const float4 &x) {   // wire 0
    const float v = fmaf(x.x, x.z, x.y * x.w);
    if (RUNS) run += v;
    else acc = gather(acc, v);
  }
  __device__ __forceinline__ void end_run() {
    if (!RUNS) return;
    acc = gather(acc, run);
    run = 0.0f;
  }
};

template <int WB, bool LOW, bool RUNS>
__global__ void __launch_bounds__(kThreads, 2)
k_xterms(const float4 *__restrict__ st, uint64_t nsites, XTermArgs c, Area a,
         OutWanted<4 + WB + (LOW ? 6 : 0)> out) {
  constexpr int NV = 16;
  constexpr int KB = 4 + WB;                  // wires >= 6 in the site
  constexpr int T = KB + (LOW ? 6 : 0);       // results: those wires, then 0..5
  constexpr int NW = 1 << WB;                 // warps per site
  constexpr int SPB = (kThreads / 32) / NW;   // sites per block
  constexpr int ROWS = NV * NW;
  extern __shared__ __align__(16) float4 xt[];   // [site][row][32 lanes]
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t sib = warp / NW, wsl = warp % NW;
  float4 *site = xt + static_cast<size_t>(sib) * ROWS * 32;
  const uint64_t per_round = static_cast<uint64_t>(gridDim.x) * SPB;
  const uint64_t rounds = (nsites + per_round - 1) / per_round;
  __shared__ uint64_t row_off[kThreads / 32][NV];
  if (lane < NV) {
    const uint32_t row = lane | (wsl << 4);
    uint64_t v = 0;
#pragma unroll
    for (int j = 0; j < KB; j++)
      if ((row >> j) & 1u) v |= 1ull << c.pos[j];
    row_off[warp][lane] = v;
  }
  __syncwarp();
  auto site_of = [&](uint64_t r) {
    return r * per_round + static_cast<uint64_t>(blockIdx.x) * SPB + sib;
  };
  auto site_sync = [&]() {
    if constexpr (SPB == 1) {
      __syncthreads();
    } else {
      asm volatile("bar.sync %0, %1;" ::"r"(sib + 1), "r"(NW * 32) : "memory");
    }
  };
  auto prefetch = [&](uint64_t r) {
    const uint64_t sidx = site_of(r);
    if (r < rounds && sidx < nsites) {
      uint64_t base = sidx * 32 + lane;
#pragma unroll
      for (int j = 0; j < KB; j++) base = ins0(base, c.pos[j]);
#pragma unroll
      for (int l = 0; l < NV; l++)
        cp_async16(site + ((l | (wsl << 4)) * 32 + lane), st + (base | row_off[warp][l]));
    }
    cp_async_commit();
  };
  Two acc[T] = {};
  prefetch(0);
  for (uint64_t r = 0; r < rounds; r++) {
    const bool active = site_of(r) < nsites;   // uniform over the site's warps
    cp_async_wait_all();
    site_sync();   // every warp's rows of this site have landed
    if (active) {
      float4 own[NV];
#pragma unroll
      for (int l = 0; l < NV; l++) own[l] = site[(l | (wsl << 4)) * 32 + lane];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        XSum<RUNS> s(acc[j]);
        int k = 0;
#pragma unroll
        for (int l = 0; l < NV; l++) {
          if ((l >> j) & 1) continue;
          s.vectors(own[l], own[l | (1 << j)]);
          if (++k % 2 == 0) s.end_run();
        }
      }
#pragma unroll
      for (int j = 0; j < WB; j++) {
        const uint32_t b = (wsl >> j) & 1u;   // this warp takes the rows with bit 0 == b
        XSum<RUNS> s(acc[4 + j]);
#pragma unroll
        for (int l = 0; l < NV; l += 2) {
          const float4 x = b ? own[l + 1] : own[l];
          s.vectors(x, site[((l | b) | ((wsl ^ (1u << j)) << 4)) * 32 + lane]);
          if (l % 4 == 2) s.end_run();
        }
      }
      if constexpr (LOW) {
        XSum<RUNS> s0(acc[KB]);
#pragma unroll
        for (int l = 0; l < NV; l++) {
          s0.halves(own[l]);
          if (l % 4 == 3) s0.end_run();
        }
#pragma unroll
        for (int k = 0; k < 5; k++) {
          const uint32_t b = (lane >> k) & 1u;   // this lane takes the rows with bit 0 == b
          XSum<RUNS> s(acc[KB + 1 + k]);
#pragma unroll
          for (int l = 0; l < NV; l += 2) {
            const float4 x = b ? own[l + 1] : own[l];
            s.vectors(x, site[((l | b) | (wsl << 4)) * 32 + (lane ^ (1u << k))]);
            if (l % 4 == 2) s.end_run();
          }
        }
      }
    }
    site_sync();   // every warp has read the site: its slots take the next one
    prefetch(r + 1);
  }
  cp_async_wait_all();
  finish<T>(acc, T, a, out);
}

template <int WB, bool LOW, bool RUNS>
int launch_x_as(const float4 *st, uint64_t nsites, const XTermArgs &c, Area a, double *d_out,
             const int8_t (&slot)[13], cudaStream_t s) {
  constexpr int SPB = (kThreads / 32) >> WB;
  static std::atomic<bool> opted[64];   // zero-initialised: false
  const size_t smem = static_cast<size_t>(kThreads / 32) * 16 * 32 * sizeof(float4);
  if (const int rc = opt_in(k_xterms<WB, LOW, RUNS>, smem, opted)) return rc;
  OutWanted<4 + WB + (LOW ? 6 : 0)> out;
  out.p = d_out;
  for (int t = 0; t < 4 + WB + (LOW ? 6 : 0); t++) out.slot[t] = slot[t];
  const unsigned grid = std::min<unsigned>(grid_for(nsites, SPB),
                                           static_cast<unsigned>(qmk_host::num_sms()) * 2);
  k_xterms<WB, LOW, RUNS><<<grid, kThreads, smem, s>>>(st, nsites, c, a, out);
  return launch_status();
}

// From 22 qubits on four pairs at a time in FP32: by then their errors average
// out over 2^18 such sums. At 27 qubits all X terms, 27 ZZ and four longer
// strings take 1.86 ms so, 2.04 with every pair by itself.
constexpr uint32_t kXRunQubits = 22;

template <int WB, bool LOW>
int launch_x(const float4 *st, uint64_t nsites, const XTermArgs &c, Area a, double *d_out,
             const int8_t (&slot)[13], cudaStream_t s) {
  return nsites >> (kXRunQubits - 10 - WB)
             ? launch_x_as<WB, LOW, true>(st, nsites, c, a, d_out, slot, s)
             : launch_x_as<WB, LOW, false>(st, nsites, c, a, d_out, slot, s);
}

// ---------------------------------------------------------------------------
// Narrow states: a block per string, any masks, one launch. The state is in
// L2 (128 KiB at 14 qubits).

constexpr int kSmallTerms = 64;
struct SmallArgs {
  uint64_t flip[kSmallTerms], sign[kSmallTerms];
  uint64_t useim;      // bit t: string t reads Im z (odd Y count)
};

__global__ void __launch_bounds__(kThreads)
k_expect_small(const float2 *__restrict__ st, uint32_t n, SmallArgs p, double *out) {
  __shared__ double sm[kThreads / 32];
  const uint32_t t = blockIdx.x;
  const uint64_t flip = p.flip[t], sign = p.sign[t];
  const bool im = (p.useim >> t) & 1ull;
  const uint32_t hbit = flip ? 63 - __clzll(flip) : 0;
  const uint32_t items = flip ? 1u << (n - 1) : 1u << n;
  Two acc = {};
  for (uint32_t u0 = threadIdx.x; u0 < items; u0 += kThreads * 8) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const uint32_t u = u0 + k * kThreads;
      if (u < items) {
        const uint64_t i = flip ? ins0(u, hbit) : u;
        const float2 x = st[i], y = st[i ^ flip];
        const float v = im ? x.x * y.y - x.y * y.x : x.x * y.x + x.y * y.y;
        acc = gather(acc, parity64(i & sign) ? -v : v);
      }
    }
  }
  const double sum = block_sum(widen(settle(acc)), sm);
  if (threadIdx.x == 0) out[t] = sum;
}

bool ok_state(const float *p) { return p && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

bool ok_ws(void *ws, size_t bytes, uint32_t n) {
  return ws && bytes >= qmk_workspace_bytes(n);
}

}  // namespace

extern "C" int qmk_z_expect(const float *state, uint32_t n, uint32_t nt, const uint64_t *masks,
                            double *d_out, void *ws, size_t ws_bytes, void *stream) {
  if (!ok_state(state) || !d_out || n < 10 || n > 40 || nt < 1 || nt > kZTerms || !masks ||
      !ok_ws(ws, ws_bytes, n))
    return -1;
  ZTermArgs z{};
  z.nt = nt;
  for (uint32_t t = 0; t < nt; t++) {
    const uint64_t m = masks[t];
    if (m >> n) return -1;
    z.lane[t] = static_cast<uint8_t>((m >> 1) & 31u);
    z.coef[t] = static_cast<uint8_t>((m & 1u) | (((m >> 6) & 15u) << 1));
    z.hi[t][0] = static_cast<uint32_t>(m >> 10);
    z.hi[t][1] = static_cast<uint32_t>(m >> 42);
  }
  const uint64_t nwsites = 1ull << (n - 10);
  const float4 *st = reinterpret_cast<const float4 *>(state);
  const Area a = area_of(ws);
  const OutContig out{d_out, false};
  cudaStream_t s = (cudaStream_t)stream;
  if (nt <= 4) return launch_z<4>(st, nwsites, z, a, out, s);
  if (nt <= 16) return launch_z<16>(st, nwsites, z, a, out, s);
  return launch_z<32>(st, nwsites, z, a, out, s);
}

extern "C" int qmk_x_expect(const float *state, uint32_t n, uint32_t num_wires,
                            const uint32_t *wires, double *d_out, void *ws, size_t ws_bytes,
                            void *stream) {
  if (!ok_state(state) || !d_out || n < 10 || n > 40 || num_wires < 1 || num_wires > 13 || !wires ||
      !ok_ws(ws, ws_bytes, n))
    return -1;
  std::vector<uint32_t> high;
  std::vector<int8_t> slot_of(n, -1);
  bool low = false;
  for (uint32_t t = 0; t < num_wires; t++) {
    const uint32_t w = wires[t];
    if (w >= n || slot_of[w] >= 0) return -1;   // each wire once
    slot_of[w] = static_cast<int8_t>(t);
    if (w < 6) low = true;
    else high.push_back(w);
  }
  if (high.size() > 7) return -1;
  // A site holds at least four wires >= 6: the lowest free ones fill it up.
  for (uint32_t w = 6; w < n && high.size() < 4; w++)
    if (std::find(high.begin(), high.end(), w) == high.end()) high.push_back(w);
  std::sort(high.begin(), high.end());
  const uint32_t kb = static_cast<uint32_t>(high.size());
  XTermArgs c{};
  int8_t slot[13];
  for (int8_t &s : slot) s = -1;
  for (uint32_t j = 0; j < kb; j++) {
    c.pos[j] = high[j] - 1;
    slot[j] = slot_of[high[j]];
  }
  if (low)
    for (uint32_t w = 0; w < 6; w++) slot[kb + w] = slot_of[w];
  const uint64_t nsites = 1ull << (n - 6 - kb);
  const float4 *st = reinterpret_cast<const float4 *>(state);
  const Area a = area_of(ws);
  cudaStream_t s = (cudaStream_t)stream;
  switch (kb) {
    case 4: return low ? launch_x<0, true>(st, nsites, c, a, d_out, slot, s)
                       : launch_x<0, false>(st, nsites, c, a, d_out, slot, s);
    case 5: return low ? launch_x<1, true>(st, nsites, c, a, d_out, slot, s)
                       : launch_x<1, false>(st, nsites, c, a, d_out, slot, s);
    case 6: return low ? launch_x<2, true>(st, nsites, c, a, d_out, slot, s)
                       : launch_x<2, false>(st, nsites, c, a, d_out, slot, s);
    default: return low ? launch_x<3, true>(st, nsites, c, a, d_out, slot, s)
                        : launch_x<3, false>(st, nsites, c, a, d_out, slot, s);
  }
}

extern "C" int qmk_expect_small(const float *state, uint32_t n, uint32_t nt, const uint64_t *flips,
                                const uint64_t *signs, const uint32_t *ny, double *d_out,
                                void *stream) {
  if (!state || !d_out || n < 1 || n > 14 || nt < 1 || nt > kSmallTerms || !flips || !signs || !ny)
    return -1;
  SmallArgs p{};
  for (uint32_t t = 0; t < nt; t++) {
    if (flips[t] >> n) return -1;
    p.flip[t] = flips[t];
    p.sign[t] = signs[t];
    if (ny[t] & 1u) p.useim |= 1ull << t;
  }
  k_expect_small<<<nt, kThreads, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const float2 *>(state), n, p, d_out);
  return launch_status();
}
