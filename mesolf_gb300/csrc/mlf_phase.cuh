// Lines of the MATLAB-layout volume <-> the phase-major volume, through shared memory.
//
// Line (c, z) holds element N*a + alpha at X[ch(alpha, beta, z)][b][a], beta = c mod N, b = c / N: for
// a fixed alpha its elements are consecutive floats of one channel row, a run.  In shared memory a
// line is contiguous and a run has stride N (odd at the lenslet pitches in use: no bank conflicts), so
// both sides of the transposition are coalesced.
#pragma once

#include "mlf_internal.h"

namespace mlf {

constexpr int kPhaseRuns = 8;

// Channel row of run p = (line l, alpha) of the nl lines from (c0, z): offset in X of its element a = 0.
__device__ __forceinline__ int64_t phase_run(const PatchGeo& g, int c0, int z, int l, int alpha) {
  const int c = c0 + l, b = c / g.N;
  return geo_channel(g, alpha, c - b * g.N, z) * g.plane + (int64_t)b * g.Pa;
}

// A warp takes runs, eight at a time so that eight loads are in flight, its lanes along a.
// Lenslets a_lo .. a_lo + na - 1 of nl lines from (c0, z) into sm: element N*a + alpha of line l at
// sm[(N*(a - a_lo) + alpha) * si + l * sl].  use(v) sees every value once.
template <class Use>
__device__ __forceinline__ void phase_gather(const float* __restrict__ X, const PatchGeo& g, int c0, int z, int nl,
                                             int a_lo, int na, float* sm, int si, int sl, Use use) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int runs = nl * g.N;
  for (int p0 = warp; p0 < runs; p0 += kPhaseRuns * nwarps) {
    const float* src[kPhaseRuns];
    float* dst[kPhaseRuns];
#pragma unroll
    for (int u = 0; u < kPhaseRuns; ++u) {
      const int p = min(p0 + u * nwarps, runs - 1), l = p / g.N, alpha = p - l * g.N;
      src[u] = X + phase_run(g, c0, z, l, alpha) + a_lo;
      dst[u] = sm + alpha * si + l * sl;
    }
    for (int a = lane; a < na; a += 32) {
      float v[kPhaseRuns];
#pragma unroll
      for (int u = 0; u < kPhaseRuns; ++u) v[u] = p0 + u * nwarps < runs ? __ldg(src[u] + a) : 0.f;
#pragma unroll
      for (int u = 0; u < kPhaseRuns; ++u)
        if (p0 + u * nwarps < runs) {
          dst[u][g.N * a * si] = v[u];
          use(v[u]);
        }
    }
  }
}

// The same for up to kPhaseLines lines, sm[l * pitch + N*(a - a_lo) + alpha], in either direction:
// the block's threads walk the elements of all runs in one sequence, so that short runs leave no
// lanes idle, with eight of them in flight per thread.  tab: phase_tab_floats(N) floats.  Ends
// without a barrier; the caller has one between the table's use and the next call.
constexpr int kPhaseLines = 4;
struct PhaseRun {
  int64_t x;  // offset in X of the run's element a_lo
  int sm, pad;
};
__host__ __device__ constexpr int phase_tab_floats(int N) { return kPhaseLines * N * (int)(sizeof(PhaseRun) / sizeof(float)); }

__device__ __forceinline__ void phase_table(const PatchGeo& g, int c0, int z, int nl, int a_lo, int pitch, float* tab) {
  for (int p = threadIdx.x; p < nl * g.N; p += blockDim.x) {
    const int l = p / g.N, alpha = p - l * g.N;
    reinterpret_cast<PhaseRun*>(tab)[p] = PhaseRun{phase_run(g, c0, z, l, alpha) + a_lo, l * pitch + alpha, 0};
  }
}

// step(e, run, a): element a of the run, e = 0 .. kPhaseRuns - 1 within a batch; flush() after each batch
template <class Step, class Flush>
__device__ __forceinline__ void phase_walk(int runs, int na, const float* tab, Step step, Flush flush) {
  const PhaseRun* t = reinterpret_cast<const PhaseRun*>(tab);
  const int nthr = blockDim.x;
  int p = threadIdx.x / na, a = threadIdx.x - p * na;
  const int dp = nthr / na, da = nthr - dp * na;
  while (p < runs) {
#pragma unroll
    for (int e = 0; e < kPhaseRuns; ++e) {
      if (p < runs) step(e, t[p], a);
      a += da;
      p += dp;
      if (a >= na) {
        a -= na;
        ++p;
      }
    }
    flush();
  }
}

__device__ __forceinline__ void phase_lines_in(const float* __restrict__ X, const PatchGeo& g, int nl, int na,
                                               const float* tab, float* sm) {
  float v[kPhaseRuns];
  int at[kPhaseRuns];
#pragma unroll
  for (int e = 0; e < kPhaseRuns; ++e) at[e] = -1;
  phase_walk(
      nl * g.N, na, tab,
      [&](int e, const PhaseRun& r, int a) {
        v[e] = __ldg(X + r.x + a);
        at[e] = r.sm + g.N * a;
      },
      [&]() {
#pragma unroll
        for (int e = 0; e < kPhaseRuns; ++e) {
          if (at[e] >= 0) sm[at[e]] = v[e];
          at[e] = -1;
        }
      });
}

template <class F>
__device__ __forceinline__ void phase_lines_out(float* __restrict__ X, const PatchGeo& g, int nl, int na,
                                                const float* tab, const float* sm, F f) {
  phase_walk(
      nl * g.N, na, tab, [&](int, const PhaseRun& r, int a) { X[r.x + a] = f(sm[r.sm + g.N * a]); }, []() {});
}

}  // namespace mlf
