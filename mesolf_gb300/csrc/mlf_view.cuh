// Per-view phase-space RL kernel (plain FP32 path).
//
// The volume lives in phase-major layout: channel ch = (beta*N + alpha)*Z + z holds the
// coarse plane P_ch[b][a] = X(N*a + alpha, N*b + beta, z) (row pitch Pa).  In that layout
// the reference's per-view operators (recon_theory_phase_space_LFM_with_filter.m:211-249)
// become, per channel, small dense correlations on the lenslet grid:
//
//   forward  (:243-249)  HX[j][i]  += sum_{db,da} P_ch[j+db-q][i+da-q] * wf_ch[db][da]
//   backward (:211-220)  C_ch[b][a] = sum_{dj,di} R[b+sb-q+dj][a+sa-q+di] * wb_ch[dj][di]
//   D        (:123)      D_ch[b][a] = the same sum over the taps that land inside R
//   update   (:130-137)  X <- w*clean(X*C/D) + (1-w)*X, clamped at 0
//
// with sa = floor((alpha-u+h)/N), sb = floor((beta-v+h)/N).  One CTA owns one or more
// channel slots (two for the 67 x 67 lenslet patch, sharing one staged ratio image); each
// thread of a slot owns a 4 (b) x 8 (a) output tile.  Inputs are staged in shared memory
// with zero halos, so the tap loops need no bounds checks; the sliding windows are read
// with aligned 128-bit shared loads, each input row once per tile (conv_rows).  The X tile
// of a channel is copied with cp.async straight into the forward-input plane and updated
// there in place.  Each slot adds its channels' forward projections into its own partial
// plane in global memory (L2-resident, tile rows 32-byte aligned), in channel order; a
// second kernel reduces the planes in a fixed order.  Keeping those sums out of registers
// leaves each thread under 96 registers, so two CTAs of two slots (20 warps) fit an SM.
// A channel needs two CTA barriers: after the update (the forward projection reads the
// neighbouring tiles' updated X) and at its end (the next channel's X overwrites the
// plane).  The next channel's D table is built between them: its row sums read the taps
// from global memory while the back projection runs, its table after the first barrier.
#pragma once

#include <cuda_runtime.h>

#include "mlf_internal.h"

namespace mlf {

// Tile of conv_tile (8 b x 4 a), used by the allocation-free forward projection
// (mlf_noalloc.cu).
constexpr int VT_TY = 8;  // tile rows (b direction)
constexpr int VT_TX = 4;  // tile cols (a direction)

// acc[ty][tx] += sum_{dy<T, dx<T} in[(ty+dy)*pitch + OFF + tx + dx] * w[dy*WP+dx]
// `in` must be 16-byte aligned and pitch a multiple of 4.  Tap rows are WP floats apart;
// when WP is a multiple of 4 a row is read with 16-byte loads (the padding is not used).
// For a fixed output the products are added in the order dy, then dx.
template <int T, int OFF, int WP = T>
__device__ __forceinline__ void conv_tile(const float* __restrict__ in, int pitch,
                                          const float* __restrict__ w,
                                          float (&acc)[VT_TY][VT_TX]) {
  constexpr int NW = view_nw(T);
  static_assert(OFF + VT_TX + T - 1 <= 4 * NW, "window too short");
#pragma unroll 1
  for (int dy = 0; dy < T; ++dy) {
    float wr[T];
    if constexpr (WP % 4 == 0) {
      const float4* w4 = reinterpret_cast<const float4*>(w + dy * WP);
#pragma unroll
      for (int k = 0; k < (T + 3) / 4; ++k) {
        const float4 t4 = w4[k];
        wr[4 * k] = t4.x;
        if (4 * k + 1 < T) wr[4 * k + 1] = t4.y;
        if (4 * k + 2 < T) wr[4 * k + 2] = t4.z;
        if (4 * k + 3 < T) wr[4 * k + 3] = t4.w;
      }
    } else {
#pragma unroll
      for (int dx = 0; dx < T; ++dx) wr[dx] = w[dy * WP + dx];
    }
    const float* rowp = in + dy * pitch;
#pragma unroll
    for (int ty = 0; ty < VT_TY; ++ty) {
      float win[4 * NW];
      const float4* r4 = reinterpret_cast<const float4*>(rowp + ty * pitch);
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        float4 t4 = r4[k];
        win[4 * k + 0] = t4.x;
        win[4 * k + 1] = t4.y;
        win[4 * k + 2] = t4.z;
        win[4 * k + 3] = t4.w;
      }
#pragma unroll
      for (int dx = 0; dx < T; ++dx)
#pragma unroll
        for (int tx = 0; tx < VT_TX; ++tx)
          acc[ty][tx] = fmaf(win[OFF + tx + dx], wr[dx], acc[ty][tx]);
    }
  }
}

// acc[ty][tx] += sum_{dy<T, dx<T} in[(ty+dy)*pitch + col(OFF + tx + dx)] * w[dy*WP+dx]
// for a TY x TX tile of the view kernel, on a plane whose columns are swizzled in 16-byte
// chunks: chunk k of this thread's window (columns a0 + 4k .. a0 + 4k + 3) starts at column
// view_pcol(a0 + 4k, pitch) of a row.  Walks the TY + T - 1 input rows once: row r is loaded
// into registers once and serves every output row ty with a tap row dy = r - ty (tap rows
// come from shared memory as broadcast 16-byte loads), so the input window is read once
// per tile instead of once per tap row.  Per output the products are added in the order
// dy, then dx -- the order of conv_tile -- so the results are the same bit for bit.
// `in` 16-byte aligned, a0 and pitch multiples of 4, WP a multiple of 4.
template <int T, int OFF, int WP, int TY, int TX>
__device__ __forceinline__ void conv_rows(const float* __restrict__ in, int pitch, int a0,
                                          const float* __restrict__ w, float (&acc)[TY][TX]) {
  constexpr int NW = view_nw(T, TX);
  static_assert(OFF + TX + T - 1 <= 4 * NW, "window too short");
  static_assert(WP % 4 == 0, "tap rows must be 16-byte aligned");
  int off[NW];
#pragma unroll
  for (int k = 0; k < NW; ++k) off[k] = view_pcol(a0 + 4 * k, pitch);
#pragma unroll 1
  for (int r = 0; r < TY + T - 1; ++r) {
    float win[4 * NW];
    const float* row = in + r * pitch;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const float4 t4 = *reinterpret_cast<const float4*>(row + off[k]);
      win[4 * k + 0] = t4.x;
      win[4 * k + 1] = t4.y;
      win[4 * k + 2] = t4.z;
      win[4 * k + 3] = t4.w;
    }
#pragma unroll
    for (int ty = 0; ty < TY; ++ty) {
      const int dy = r - ty;
      if (dy < 0 || dy >= T) continue;
      float wr[T];
      const float4* w4 = reinterpret_cast<const float4*>(w + dy * WP);
#pragma unroll
      for (int k = 0; k < (T + 3) / 4; ++k) {
        const float4 t4 = w4[k];
        wr[4 * k] = t4.x;
        if (4 * k + 1 < T) wr[4 * k + 1] = t4.y;
        if (4 * k + 2 < T) wr[4 * k + 2] = t4.z;
        if (4 * k + 3 < T) wr[4 * k + 3] = t4.w;
      }
#pragma unroll
      for (int dx = 0; dx < T; ++dx)
#pragma unroll
        for (int tx = 0; tx < TX; ++tx) acc[ty][tx] = fmaf(win[OFF + tx + dx], wr[dx], acc[ty][tx]);
    }
  }
}

__device__ __forceinline__ int floor_div(int a, int b) {
  int q = a / b;
  return (a % b != 0 && ((a < 0) != (b < 0))) ? q - 1 : q;
}

__device__ __forceinline__ void cp_async16(float* smem, const float* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// D table of channel ch, in two steps separated by a CTA barrier (lt = thread within the
// slot, tps = threads per slot).  Row sums, read from the channel's taps in global memory:
//   rowp[dj][ca] = sum_{di in rngA[sa][ca]} wb[ch][dj][di]
// then the table:
//   dtab[cb][ca] = sum_{dj in rngB[sb][cb]} rowp[dj][ca]
// Both add in index order, so the values do not depend on the launch shape.
template <int T>
__device__ __forceinline__ void view_d_rows(const ViewArgs& A, int ch, int lt, float* rowp) {
  const int h = (A.N - 1) / 2;
  const int alpha = (int)((ch / A.Z) % A.N);
  const int sa = floor_div(alpha - A.u + h, A.N);
  const int* rA = A.rngA + (sa + 1) * A.maxc * 2;
  const float* w = A.wb + ch * (T * T);
  for (int i = lt; i < T * A.maxc; i += A.tps) {
    const int dj = i / A.maxc, ca = i - dj * A.maxc;
    const int lo = __ldg(rA + 2 * ca), hi = __ldg(rA + 2 * ca + 1);
    float v[T];  // the whole tap row in flight at once; the sum takes [lo, hi] in order
#pragma unroll
    for (int di = 0; di < T; ++di) v[di] = __ldg(w + dj * T + di);
    float s = 0.f;
#pragma unroll
    for (int di = 0; di < T; ++di)
      if (di >= lo && di <= hi) s += v[di];
    rowp[i] = s;
  }
}
template <int T>
__device__ __forceinline__ void view_d_table(const ViewArgs& A, int ch, int lt, const float* rowp,
                                             float* dtab) {
  const int h = (A.N - 1) / 2;
  const int beta = ch / (A.Z * A.N);
  const int sb = floor_div(beta - A.v + h, A.N);
  const int* rB = A.rngB + (sb + 1) * A.maxc * 2;
  for (int i = lt; i < A.maxc * A.maxc; i += A.tps) {
    const int cb = i / A.maxc, ca = i - cb * A.maxc;
    const int lo = __ldg(rB + 2 * cb), hi = __ldg(rB + 2 * cb + 1);
    float v[T];
#pragma unroll
    for (int dj = 0; dj < T; ++dj) v[dj] = rowp[dj * A.maxc + ca];
    float s = 0.f;
#pragma unroll
    for (int dj = 0; dj < T; ++dj)
      if (dj >= lo && dj <= hi) s += v[dj];
    dtab[i] = s;
  }
}

// At most kViewMaxThreads threads and two CTAs per SM: 96 registers per thread.
template <int T, int MODE, int TY, int TX>
__global__ void __launch_bounds__(kViewMaxThreads, 2) k_view(ViewArgs A) {
  static_assert(TX % 4 == 0, "tile rows are whole 16-byte chunks");
  constexpr int NC = TX / 4;             // 16-byte chunks of a tile row
  extern __shared__ __align__(16) float sm[];
  constexpr int TT = T * T;
  constexpr int TW = view_tap_pitch(T);  // tap-row pitch in shared memory
  constexpr int TTW = T * TW;
  constexpr int Q = (T - 1) / 2;
  constexpr int QP = view_qpad(Q);      // column of the forward-input interior
  constexpr bool BWD = (MODE != MODE_FWD);
  constexpr bool XIN = (MODE != MODE_BWDC);
  // The next channel's taps are requested at the start of a channel: 31 x 40 x 26 lenslets, T 9, forward
  // 46.7 -> 43.4 us per view with the second X plane, 28 x 21 x 25, T 11 solve 20.0 -> 19.4 ms.  The
  // small tile's few channels per slot gain nothing (11 x 11 x 21: 10.98 ms -> 11.05) and load them at
  // the end.
  constexpr bool AHEAD = TX == VW_TX;
  const int tid = threadIdx.x;
  const int slot = tid / A.tstride;          // slots start at multiples of tstride >= tps
  const int lt = tid - slot * A.tstride;     // thread index within slot
  const bool slot_ok = slot < A.slots && lt < A.tps;
  // tile of this thread: with more than 8 tile columns, lanes 8k .. 8k+7 take columns 0..7
  // of one tile row (a 64-float span, so a warp's window loads spread over all banks) and
  // the remaining columns follow; fewer columns: row-major
  int ta, tb;
  if (A.tilesA > 8 && lt >= 8 * A.tilesB) {
    const int w2 = A.tilesA - 8, l2 = lt - 8 * A.tilesB;
    ta = 8 + l2 % w2;
    tb = l2 / w2;
  } else if (A.tilesA > 8) {
    ta = lt & 7;
    tb = lt >> 3;
  } else {
    ta = lt % A.tilesA;
    tb = lt / A.tilesA;
  }
  const int a0 = ta * TX, b0 = tb * TY;
  int xc[NC];  // swizzled columns of this tile's X chunks in the forward-input plane
#pragma unroll
  for (int k = 0; k < NC; ++k) xc[k] = view_pcol(a0 + QP + 4 * k, A.XP);

  // ---- a cancelled solve: the rest of its view steps return at once (CTA-uniform, at the first
  // barrier; until then nothing but shared memory and the stop words is written).  Read before
  // pdl_wait, beside the loads below: the kernel that launched this one early, the reduction, does so
  // after its own wait, when the view kernel before has ended, so no view step is left half done by a
  // stop word that the next one sets.
  __shared__ int s_stop;
  if (tid == 0) s_stop = cancel_entry(A.cancel);

  // ---- shared memory carve-up
  float* rs = sm;                                              // [RProws][RP] (BWD only)
  float* slot_base = rs + (BWD ? A.RProws * A.RP : 0);
  // forward only: two X planes where they fit, so that the next channel's loads overlap this one's
  // projection (elsewhere they overlap the back projection)
  const bool xtwo = MODE == MODE_FWD && AHEAD && A.xtwo;
  const int xplane = A.XProws * A.XP;
  float* xin = slot_base + (slot_ok ? slot : 0) * A.slot_floats;  // [1 or 2][XProws][XP]
  float* taps = xin + (xtwo ? 2 : 1) * xplane;                 // [2 buffers][wb | wf]
  float* dtab = taps + 4 * TTW;                                // [maxc][maxc]
  float* rowp = dtab + A.maxc * A.maxc;                        // [T][maxc]

  // ---- zero the forward-input planes (halos must be zero)
  {
    if (XIN) {
      const int n4 = (xtwo ? 2 : 1) * xplane / 4, total = A.slots * n4;
      for (int i = tid; i < total; i += blockDim.x) {
        const int sl = i / n4;
        reinterpret_cast<float4*>(slot_base + sl * A.slot_floats)[i - sl * n4] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }

  constexpr bool DT = (MODE == MODE_STEP);  // the update needs D
  const int h = (A.N - 1) / 2;
  // channel indices and tap offsets (nch * T * T) fit in 32 bits: checked by the solver
  const int nch = (int)A.nch;
  const int step = (int)gridDim.x * A.slots;
  const int first = (int)blockIdx.x * A.slots + slot;
  // this thread's tile in its slot's forward partial plane [tilesB*TY][tilesA*TX]
  // (tile rows 32-byte aligned); recomputed where used rather than held across the loop
  auto hx_tile = [&]() {
    const int HP = A.tilesA * TX;
    return A.part + ((int64_t)blockIdx.x * A.slots + (slot_ok ? slot : 0)) * ((int64_t)A.tilesB * TY * HP) +
           (int64_t)b0 * HP + a0;
  };
  bool hx_written = false;
  auto load_taps = [&](int ch, int b) {
    float* dst = taps + b * 2 * TTW;
    for (int i = lt; i < TT; i += A.tps) {
      const int j = (i / T) * TW + i % T;
      if (AHEAD) {
        if (BWD) cp_async4(dst + j, A.wb + ch * TT + i);
        if (XIN) cp_async4(dst + TTW + j, A.wf + ch * TT + i);
      } else {
        if (BWD) dst[j] = __ldg(A.wb + ch * TT + i);
        if (XIN) dst[TTW + j] = __ldg(A.wf + ch * TT + i);
      }
    }
  };
  // X tile -> forward-input plane (interior at rows +Q, cols +QP).  A plane row has Pa (a multiple
  // of 4) floats: a 16-byte chunk of the last tile may lie past it and is then not copied (its
  // shared-memory cells stay zero).
  auto load_x = [&](int ch, float* plane) {
    const float* Xch = A.X + ch * A.plane;
#pragma unroll
    for (int y = 0; y < TY; ++y) {
      const int b = b0 + y;
      if (b >= A.Lj) continue;
#pragma unroll
      for (int k = 0; k < NC; ++k)
        if (a0 + 4 * k < A.Pa) cp_async16(plane + (b + Q) * A.XP + xc[k], Xch + (int64_t)b * A.Pa + a0 + 4 * k);
    }
  };

  // taps of the first channel into buffer 0, its D row sums; the table after the barrier
  // (the row sums come from other threads)
  if (slot_ok && first < nch) {
    load_taps(first, 0);
    if (DT) view_d_rows<T>(A, first, lt, rowp);
  }
  // Everything above depends on the PSF alone and overlaps the end of the kernel before (the
  // reduction that forms this view's ratio image); the rest reads what that kernel wrote.  The
  // kernel after may be launched now: it waits here in turn.
  pdl_launch_dependents();
  pdl_wait();
  if (BWD) {
    const int nr = A.RProws * A.RP;
    const float4* src = reinterpret_cast<const float4*>(A.rpad);
    float4* dst = reinterpret_cast<float4*>(rs);
    for (int i = tid; i < nr / 4; i += blockDim.x) dst[i] = src[i];
  }
  if (xtwo) {
    __syncthreads();  // the planes are zeroed
    if (slot_ok && first < nch) load_x(first, xin);
  }
  if (AHEAD) cp_async_wait_all();
  __syncthreads();
  if (s_stop) return;
  if (DT && slot_ok && first < nch) view_d_table<T>(A, first, lt, rowp, dtab);
  __syncthreads();

  int buf = 0;
  for (int base = (int)blockIdx.x * A.slots; base < nch; base += step, buf ^= 1) {
    const int ch = base + slot;
    const int nxt = ch + step;
    const bool active = slot_ok && ch < nch;
    const bool more = slot_ok && nxt < nch;
    const int alpha = active ? (int)((ch / A.Z) % A.N) : 0;
    const int beta = active ? ch / (A.Z * A.N) : 0;
    const int sa = floor_div(alpha - A.u + h, A.N);
    const int sb = floor_div(beta - A.v + h, A.N);
    const float* wbs = taps + buf * 2 * TTW;
    const float* wfs = wbs + TTW;

    // this channel's X (or, with two planes, the next one's) and the next channel's taps,
    // asynchronously: the buffers they go to were last read before the barrier at the loop's end
    float* const xcur = xin + (xtwo ? buf * xplane : 0);
    if (XIN && active && !xtwo) load_x(ch, xin);
    if (more) {
      if (AHEAD) load_taps(nxt, buf ^ 1);
      if (xtwo) load_x(nxt, xin + (buf ^ 1) * xplane);
    }

    // One correlation call site for both phases (back projection of view k, forward
    // projection of view k+1), so that a single unrolled body per window offset is hot.
#pragma unroll 1
    for (int ph = 0; ph < 2; ++ph) {
      if (ph == 1 && !(XIN && (MODE == MODE_FWD || A.do_fwd))) break;
      if (active && ph == 0 && !BWD) {
        if (!xtwo) cp_async_wait_all();  // forward only: this thread's X tile has landed in xin
      } else if (active) {
        float acc[TY][TX];
#pragma unroll
        for (int y = 0; y < TY; ++y)
#pragma unroll
          for (int x = 0; x < TX; ++x) acc[y][x] = 0.f;
        if (ph == 1 && hx_written) {  // this tile's forward partials into L1 for the add below
          const float* hxp = hx_tile();
#pragma unroll
          for (int y = 0; y < TY; ++y)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(hxp + y * A.tilesA * TX));
        }
        const float* in = ph == 0 ? rs + (b0 + sb + 1) * A.RP : xcur + b0 * A.XP;
        const int pitch = ph == 0 ? A.RP : A.XP;
        const float* wsel = ph == 0 ? wbs : wfs;
        switch (ph == 0 ? sa + 1 : QP - Q) {
          case 0: conv_rows<T, 0, TW, TY, TX>(in, pitch, a0, wsel, acc); break;
          case 1: conv_rows<T, 1, TW, TY, TX>(in, pitch, a0, wsel, acc); break;
          case 2: conv_rows<T, 2, TW, TY, TX>(in, pitch, a0, wsel, acc); break;
          default:
            if constexpr (QP - Q == 3) conv_rows<T, 3, TW, TY, TX>(in, pitch, a0, wsel, acc);
            break;
        }
        if (ph == 0) {
          if (MODE == MODE_BWDC) {
#pragma unroll
            for (int y = 0; y < TY; ++y) {
              const int b = b0 + y;
              if (b >= A.Lj) continue;
#pragma unroll
              for (int x = 0; x < TX; ++x)
                if (a0 + x < A.Li) A.Cout[(int64_t)ch * A.plane + (int64_t)b * A.Pa + a0 + x] = acc[y][x];
            }
          } else {
            cp_async_wait_all();  // this thread's X tile has landed in xin
            const int* cA = A.clsA + (sa + 1) * A.Li;
            const int* cB = A.clsB + (sb + 1) * A.Lj;
            float* Xch = A.X + ch * A.plane;
#pragma unroll
            for (int y = 0; y < TY; ++y) {
              const int b = b0 + y;
              if (b >= A.Lj) continue;
              const int cb = __ldg(cB + b);
              float* xrow = xin + (b + Q) * A.XP;
              float xo8[TX], xn8[TX];
#pragma unroll
              for (int k = 0; k < NC; ++k) {
                const float4 v = *reinterpret_cast<const float4*>(xrow + xc[k]);
                xo8[4 * k] = v.x;
                xo8[4 * k + 1] = v.y;
                xo8[4 * k + 2] = v.z;
                xo8[4 * k + 3] = v.w;
              }
#pragma unroll
              for (int x = 0; x < TX; ++x) {
                const int a = a0 + x;
                const float xo = xo8[x];
                xn8[x] = xo;  // columns past the patch keep their (zero) value
                if (a >= A.Li) continue;
                const float c = acc[y][x];
                const float d = dtab[cb * A.maxc + __ldg(cA + a)];
                float xc = xo * c / (d + A.d_eps);           // :130  X .* C ./ D
                if (!(xc >= 0.f) || isinf(xc)) xc = 0.f;     // :132-134 NaN, Inf, < 0
                float xn = __fmaf_rn(xc, A.w, __fmul_rn(1.f - A.w, xo));  // :136
                if (xn < 0.f) xn = 0.f;                      // :137
                xn8[x] = xn;
              }
              // the plane row has Pa (a multiple of 4) floats: its padding columns get back
              // their own values; a chunk past the row is not written
              float4* g = reinterpret_cast<float4*>(Xch + (int64_t)b * A.Pa + a0);
#pragma unroll
              for (int k = 0; k < NC; ++k)
                *reinterpret_cast<float4*>(xrow + xc[k]) =
                    make_float4(xn8[4 * k], xn8[4 * k + 1], xn8[4 * k + 2], xn8[4 * k + 3]);
              g[0] = make_float4(xn8[0], xn8[1], xn8[2], xn8[3]);
#pragma unroll
              for (int k = 1; k < NC; ++k)
                if (a0 + 4 * k < A.Pa) g[k] = make_float4(xn8[4 * k], xn8[4 * k + 1], xn8[4 * k + 2], xn8[4 * k + 3]);
            }
          }
        } else {
          // forward partials: plane += this channel's projection (tile rows are 16-byte chunks)
          float* hxp = hx_tile();
          const int HP = A.tilesA * TX;
#pragma unroll
          for (int y = 0; y < TY; ++y) {
            float4* p4 = reinterpret_cast<float4*>(hxp + y * HP);
            float4 v[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k)
              v[k] = make_float4(acc[y][4 * k], acc[y][4 * k + 1], acc[y][4 * k + 2], acc[y][4 * k + 3]);
            if (hx_written) {
              float4 o[NC];
#pragma unroll
              for (int k = 0; k < NC; ++k) o[k] = p4[k];
#pragma unroll
              for (int k = 0; k < NC; ++k) {
                v[k].x = o[k].x + v[k].x;
                v[k].y = o[k].y + v[k].y;
                v[k].z = o[k].z + v[k].z;
                v[k].w = o[k].w + v[k].w;
              }
            }
#pragma unroll
            for (int k = 0; k < NC; ++k) p4[k] = v[k];
          }
          hx_written = true;
        }
      }
      if (ph == 0) {
        // the next channel's D row sums (global taps) while other warps still correlate;
        // the table below reads them after the barrier, once dtab has been read
        if (DT && more) view_d_rows<T>(A, nxt, lt, rowp);
        if (!xtwo) __syncthreads();
      }
    }
    if (DT && more) view_d_table<T>(A, nxt, lt, rowp, dtab);  // the next channel's D table
    if (!AHEAD && more) load_taps(nxt, buf ^ 1);
    if (AHEAD) cp_async_wait_all();
    __syncthreads();
  }

  // More than two slots: their partial planes are added here (slot order) into the first one, so
  // that the reduction kernel reads one plane per CTA.  With 32 slots of the smallest patches it had
  // 4725 planes to add for 121 positions, 50 us of the 69 us a view step took at 11 x 11
  // lenslets; the planes are in L2, and a CTA adds its own in about 1 us
  // (11 x 11 x 21, 8 iterations: 53.7 -> 20.0 ms).  Two slots (67 x 67 lenslets) gain nothing:
  // 501.6 ms either way, so the reduction reads both planes.  Slot s of this CTA
  // has projected channels when blockIdx * slots + s < nch; the loop's last barrier orders its
  // writes before these reads.
  if ((MODE == MODE_FWD || (MODE == MODE_STEP && A.do_fwd)) && view_sums_slots(A.slots)) {
    const int n4 = A.tilesB * TY * A.tilesA * TX / 4;
    const int used = min(A.slots, nch - (int)blockIdx.x * A.slots);
    float4* p0 = reinterpret_cast<float4*>(A.part) + (int64_t)blockIdx.x * A.slots * n4;
    for (int i = tid; i < n4; i += blockDim.x) {
      float4 v = p0[i];
#pragma unroll 8
      for (int sl = 1; sl < used; ++sl) {
        const float4 t = p0[(int64_t)sl * n4 + i];
        v.x += t.x;
        v.y += t.y;
        v.z += t.z;
        v.w += t.w;
      }
      p0[i] = v;
    }
  }
}

#define MLF_VIEW_TILE(T, MODE, SMALL) \
  ((SMALL) ? (const void*)k_view<(T), MODE, VWS_TY, VWS_TX> : (const void*)k_view<(T), MODE, VW_TY, VW_TX>)

#define MLF_INSTANTIATE_VIEW(T)                                                                  \
  int prepare_view_T##T(bool small) {                                                           \
    MLF_TRY(allow_max_dyn_smem(MLF_VIEW_TILE(T, MODE_FWD, small)));                              \
    MLF_TRY(allow_max_dyn_smem(MLF_VIEW_TILE(T, MODE_STEP, small)));                             \
    return allow_max_dyn_smem(MLF_VIEW_TILE(T, MODE_BWDC, small));                               \
  }                                                                                             \
  int occupancy_view_T##T(bool small, int threads, size_t smem, int* blocks) {                  \
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(                              \
        blocks, MLF_VIEW_TILE(T, MODE_STEP, small), threads, smem);                              \
    if (e != cudaSuccess)                                                                       \
      return fail(MLF_ERR_CUDA, std::string("occupancy: ") + cudaGetErrorString(e));            \
    return MLF_OK;                                                                              \
  }                                                                                             \
  int launch_view_T##T(int mode, const ViewArgs& a, int grid, int threads, size_t smem,         \
                       cudaStream_t st) {                                                       \
    const void* f = mode == MODE_FWD ? MLF_VIEW_TILE(T, MODE_FWD, a.small)                      \
                    : mode == MODE_STEP ? MLF_VIEW_TILE(T, MODE_STEP, a.small)                  \
                                        : MLF_VIEW_TILE(T, MODE_BWDC, a.small);                 \
    ViewArgs v = a;                                                                             \
    void* args[] = {&v};                                                                        \
    cudaError_t e = launch_pdl(f, grid, threads, args, smem, st);                               \
    if (e != cudaSuccess)                                                                       \
      return fail(MLF_ERR_CUDA, std::string("view kernel launch: ") + cudaGetErrorString(e));   \
    return MLF_OK;                                                                              \
  }

}  // namespace mlf
