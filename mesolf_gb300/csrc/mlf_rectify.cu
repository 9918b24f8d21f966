// Rectification of raw sensor frames onto the lenslet-aligned grid, the input step of the
// pipeline: src/module/image_load_module_aug.m:19-164 (frame selection and averaging,
// raw-patch cut, img_rectify_mod, division by the movie max).
//
// img_rectify_mod (:126-164) resamples a raw patch with griddedInterpolant (bilinear, linear
// extrapolation, 1-based sample coordinates 1..H, 1..W) onto the grid
//   R = [fliplr(c : -dx/M : -dx/M), c+dx/M : dx/M : size+0.9]
// per axis (c = lenslet centre inside the patch), drops the first mod(idx(c) - floor(M/2), M)
// grid points so that lenslets start on a multiple of M, evaluates, and keeps the first
// M*floor(n/M) rows and columns.  The grids are computed here on the host in FP64 and turned
// into per-row and per-column (cell, weight) tables; the kernel gathers the four neighbours of
// every output pixel of every output frame, averaging the selected input frames first (the
// interpolation is linear, so this is the reference's mean-then-rectify).
//
// One launch covers all output frames.  Frame averaging (k_rectify): thread per output row
// of one column (coalesced along the fast axis of the output, which maps to
// near-consecutive raw rows) and 8 output frames, with all 32 neighbour loads of the 8
// frames in flight before the interpolation.  One input frame per output frame
// (k_rectify_rows): the raw tile of a block is staged in shared memory by 16-byte copies
// and the next frame chunk is prefetched while the current one is interpolated.
//
// The division by the movie's maximum needs the maximum first.  One input frame per output
// frame: the interpolation runs twice, first for the maximum alone (reads the raw cut, writes
// nothing), then writing the divided values, so the movie is written once and never read back:
// 2 x 2 + 4 bytes per pixel of 16-bit frames where write, maximum and scaling passes moved 18.
// Averaged frames read navg frames per output, so there the write pass takes the maximum and a
// scaling pass follows (2 navg + 12 bytes).
#include "mlf_f32x2.cuh"
#include "mlf_internal.h"

#include <algorithm>
#include <climits>
#include <cmath>

namespace mlf {

namespace {


template <typename TIn>
__device__ __forceinline__ float ldv(const TIn* p) {
  return (float)__ldg(p);
}

// out[(r + oh*c) + P*i] = bilinear(mean of frames f0 + i*fstep + j, j < navg_i) at row cell
// iy[r] (weight wy[r]) and column cell ix[c] (weight wx[c]).  Frame f of the input is at
// raw + f*fstride; element (row, col) of the cut at (row0 + row) + cstride*(col0 + col).
// Block: RC_ROWS output rows x RC_COLS columns (threadIdx.y), output frames in chunks of
// RC_FCH (all 4*RC_FCH neighbour loads of a chunk in flight before the interpolation), RC_NCH
// chunks per block; the tables are read once per thread.
// max_part (nullable): the largest value of each block.
constexpr int RC_ROWS = 128, RC_COLS = 4, RC_FCH = 8, RC_NCH = 8;

// Maximum over the block (fmaxf: NaN only where every value is NaN), valid in thread 0.
__device__ __forceinline__ float rc_block_max(float m, float* sh) {
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) sh[tid >> 5] = m;
  __syncthreads();
  if (tid == 0)
    for (int w = 1; w < (int)(blockDim.x * blockDim.y >> 5); ++w) m = fmaxf(m, sh[w]);
  return m;
}

// AVG: averaged frames (navg > 1).  With the block maximum one kernel for both takes 84 to 92 registers,
// one block on an SM; the two take 40 and 54.  Per call: 1100 x 1100 px, 600 16-bit frames in threes 4345 ->
// 2313 us, 600 x 600, 400 32-bit frames in pairs 1169 -> 731, 1000 x 1000, 300 16-bit frames one by one at
// pitch 2.0 1051 -> 751 (4094, 1243 and 887 before the maximum was taken here).
template <typename TIn, bool AVG>
__global__ void __launch_bounds__(RC_ROWS * RC_COLS)
k_rectify(const TIn* __restrict__ raw, int64_t fstride, int64_t cstride, int64_t row0, int64_t col0,
          const int* __restrict__ iy, const float* __restrict__ wy, int oh, const int* __restrict__ ix,
          const float* __restrict__ wx, int ow, int64_t f0, int64_t fstep, int navg, int64_t flast, int64_t n_out,
          float* __restrict__ out, float* __restrict__ max_part) {
  __shared__ float mx_sh[32];
  const int r = blockIdx.x * RC_ROWS + threadIdx.x;
  const int c = blockIdx.y * RC_COLS + threadIdx.y;
  float mx = -INFINITY;
  if (r < oh && c < ow) {
  const int64_t P = (int64_t)oh * ow;
  const int i0 = __ldg(iy + r), j0 = __ldg(ix + c);
  const float fy = __ldg(wy + r), fx = __ldg(wx + c);
  const int64_t o00 = (row0 + i0) + cstride * (col0 + j0);
  const int64_t o01 = o00 + cstride;
  float* op = out + r + (int64_t)oh * c;
  for (int ch = 0; ch < RC_NCH; ++ch) {
    const int64_t ib = ((int64_t)blockIdx.z * RC_NCH + ch) * RC_FCH;
    if (ib >= n_out) break;
    const int ni = (int)(n_out - ib < RC_FCH ? n_out - ib : RC_FCH);
    if (!AVG) {
      float v[RC_FCH][4];
#pragma unroll
      for (int q = 0; q < RC_FCH; ++q) {
        if (q < ni) {
          const TIn* fr = raw + (f0 + (ib + q) * fstep) * fstride;
          v[q][0] = ldv(fr + o00);
          v[q][1] = ldv(fr + o00 + 1);
          v[q][2] = ldv(fr + o01);
          v[q][3] = ldv(fr + o01 + 1);
        }
      }
#pragma unroll
      for (int q = 0; q < RC_FCH; ++q) {
        if (q < ni) {
          const float a = fmaf(fx, v[q][2] - v[q][0], v[q][0]), b = fmaf(fx, v[q][3] - v[q][1], v[q][1]);
          const float o = fmaf(fy, b - a, a);
          mx = fmaxf(mx, o);
          __stcs(op + P * (ib + q), o);
        }
      }
      continue;
    }
    for (int q = 0; q < ni; ++q) {
      const int64_t fa = f0 + (ib + q) * fstep;
      const int64_t fb = min(fa + navg - 1, flast);
      float v00 = 0.f, v10 = 0.f, v01 = 0.f, v11 = 0.f;
      for (int64_t f = fa; f <= fb; ++f) {
        const TIn* fr = raw + f * fstride;
        v00 += ldv(fr + o00);
        v10 += ldv(fr + o00 + 1);
        v01 += ldv(fr + o01);
        v11 += ldv(fr + o01 + 1);
      }
      const float rn = 1.f / (float)(fb - fa + 1);
      const float a = fmaf(fx, v01 - v00, v00), b = fmaf(fx, v11 - v10, v10);
      const float o = fmaf(fy, b - a, a) * rn;
      mx = fmaxf(mx, o);
      __stcs(op + P * (ib + q), o);
    }
  }
  }
  if (max_part) {
    const float m = rc_block_max(mx, mx_sh);
    if (threadIdx.x == 0 && threadIdx.y == 0)
      max_part[((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = m;
  }
}

// One input frame per output frame, with the raw tile of each block staged in shared memory by
// 16-byte loads.  Block = blockDim.x output rows (32 .. RR_MAX_ROWS) x RR_COLS output columns; stages of
// RR_SF output frames, two per thread (threadIdx.y picks the pair).  For frame q and raw column
// k of the block's footprint (raw columns ix[c0] .. ix[c1]+1, rows iy[r0] .. iy[r1]+1) the
// column segment is loaded from the 16-byte boundary at or below its first element into slot
// [q][k] (`slot` elements).  raw must be 16-byte aligned; `total` = elements of the frame buffer
// (bytes past its end are zero-filled, never read).
//
// Bound: instruction issue (82 % of the slots with one thread per output pixel, which took all
// four neighbours per output: 20 instructions), then HBM.  So a thread walks RR_COLS output
// columns of its row: the interpolation along the row axis is done once per raw column and
// serves the outputs on both sides of it, and its two frames share addresses, tables and packed
// FP32 instructions.  2000 frames of 1100 x 1100 16-bit pixels to 1065 x 1065: maximum pass
// 1.92 ms (issue 84 %), 1.24 with most stages skipped (rr_key), writing pass 2.95 ms (4.6 TB/s);
// before, interpolation 3.35, maximum 1.51 and scaling 5.03 ms.
constexpr int RR_COLS = 16, RR_SF = 4, RR_MAX_ROWS = 160;
enum RectifyMode { RR_PLAIN = 0, RR_MAX = 1, RR_DIV = 2 };

// exact uint16 -> float: the bits 0x4B000000 | x are the float 2^23 + x (x < 2^23 fits the
// mantissa), and 2^23 is taken out where the value itself is needed
__device__ __forceinline__ float rr_raw(uint16_t x) { return __uint_as_float(0x4B000000u | x); }
__device__ __forceinline__ float rr_raw(float x) { return x; }

__device__ __forceinline__ void rc_cp_async16(void* smem, const void* gmem, int src_bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(src_bytes) : "memory");
}

struct RectifyRows {
  int64_t total, fstride, cstride, row0, col0;
  const int* iy;
  const float* wy;
  const int* ix;
  const float* wx;
  int oh, ow;
  int64_t f0, fstep, n_out;
  int slot, maxc;
  const float* mx;   // RR_DIV: the movie's maximum
  float* max_part;   // RR_MAX: largest value per block
  int* best;         // RR_MAX: largest value of any block so far (rr_key)
};

// An output inside the raw cut is a convex combination of four raw pixels, so no output of a stage
// exceeds the largest raw value of its tile but by rounding.  The maximum pass therefore interpolates
// only stages whose raw values, with that margin, exceed the largest output seen so far by any block;
// the result is the same maximum.  Raw values cost a packed comparison per pair where the
// interpolation takes about ten instructions per output: 1.92 -> 1.24 ms for 2000 frames of 1100 x
// 1100 pixels of noise on a random pattern; a movie whose every stage holds the same largest value at
// a grid point gains nothing and pays the comparisons.
// rr_key: a float's place in the order as an int.
__device__ __forceinline__ int rr_key(float x) {
  const int i = __float_as_int(x);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float rr_unkey(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7fffffff); }

// Range of the raw values of one or more 16-byte vectors.
template <typename TIn>
struct RawRange;
template <>
struct RawRange<uint16_t> {
  unsigned hi = 0;
  __device__ __forceinline__ void add(const uint16_t* p) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    hi = __vmaxu2(hi, __vmaxu2(__vmaxu2(v.x, v.y), __vmaxu2(v.z, v.w)));
  }
  // whether an interpolated value may exceed `best`: the values are exact and not negative, each of
  // the two interpolations rounds twice at most
  __device__ __forceinline__ bool may_exceed(float best) const {
    const float m = (float)max(hi & 0xffffu, hi >> 16);
    return !(m * (1.f + 0x1p-20f) <= best);
  }
};
template <>
struct RawRange<float> {
  float hi = -INFINITY, lo = INFINITY;
  __device__ __forceinline__ void add(const float* p) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    hi = fmaxf(hi, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
    lo = fminf(lo, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
  }
  // NaN pixels give NaN outputs, which the maximum ignores; infinities and differences that may
  // overflow are interpolated
  __device__ __forceinline__ bool may_exceed(float best) const {
    const float a = fmaxf(fabsf(hi), fabsf(lo));
    return !(a < 1e38f && best > -1e38f && fmaf(a, 0x1p-20f, hi) <= best);
  }
};

// Persistent over stages z = blockIdx.z, blockIdx.z + gridDim.z, ...: the raw tile of stage z+1
// is copied into the second buffer (16-byte zero-filling cp.async, no register round trip)
// while stage z is interpolated, so DRAM loads stay in flight.  SAME: every frame starts at the
// same offset from a 16-byte boundary, so a column's place in its slot is one table entry.
template <typename TIn, int MODE, bool SAME>
__global__ void __launch_bounds__(2 * RR_MAX_ROWS)
k_rectify_rows(const TIn* __restrict__ raw, RectifyRows A, float* __restrict__ out) {
  constexpr int VEC = 16 / sizeof(TIn);
  extern __shared__ __align__(16) unsigned char rc_smem[];
  TIn* tiles = reinterpret_cast<TIn*>(rc_smem);  // [2 buffers][RR_SF][maxc][slot]
  __shared__ int2 colt[RR_COLS];                 // per output: left raw column, weight; bit 31 of the
                                                 // column: it is not the previous output's right one
  __shared__ float mx_sh[32];
  const int rows = blockDim.x, nthr = 2 * rows;
  const int tid = threadIdx.y * rows + threadIdx.x;
  const int r0 = blockIdx.x * rows, c0 = blockIdx.y * RR_COLS;
  const int r1 = min(r0 + rows, A.oh) - 1, cn = min(RR_COLS, A.ow - c0);
  const int rlo = __ldg(A.iy + r0), nrow = __ldg(A.iy + r1) + 2 - rlo;
  const int clo = __ldg(A.ix + c0), ncol = __ldg(A.ix + c0 + cn - 1) + 2 - clo;  // <= maxc (host bound)
  const int nv = (nrow + 2 * VEC - 2) / VEC;                                     // vectors per column segment
  const int64_t stages = (A.n_out + RR_SF - 1) / RR_SF;
  const int per = A.maxc * A.slot;  // elements per staged frame
  const int64_t base0 = (A.row0 + rlo) + A.cstride * (A.col0 + clo);
  if (tid < cn) {
    const int lc = __ldg(A.ix + c0 + tid) - clo;
    const int prev = tid > 0 ? __ldg(A.ix + c0 + tid - 1) - clo : -2;
    colt[tid] = make_int2(lc | (lc == prev + 1 ? 0 : (int)0x80000000), __float_as_int(__ldg(A.wx + c0 + tid)));
  }
  // vector e of a stage = (frame q, column k, vector v), e = tid, tid + nthr, ...: the first one
  // and the step from one to the next are divided once
  const int cnv = ncol * nv;
  const int q_0 = tid / cnv, k_0 = (tid - q_0 * cnv) / nv, v_0 = tid - q_0 * cnv - k_0 * nv;
  const int dq = nthr / cnv, dk = (nthr - dq * cnv) / nv, dv = nthr - dq * cnv - dk * nv;
  auto each_vector = [&](int nf, auto use) {
    int q = q_0, k = k_0, v = v_0;
    while (q < nf) {
      use(q, k, v);
      v += dv;
      k += dk;
      q += dq;
      if (v >= nv) {
        v -= nv;
        ++k;
      }
      if (k >= ncol) {
        k -= ncol;
        ++q;
      }
    }
  };
  auto stage = [&](int64_t z, int b) {
    const int64_t ib = z * RR_SF;
    const int nf = (int)(A.n_out - ib < RR_SF ? A.n_out - ib : RR_SF);
    const int64_t e0 = (A.f0 + ib * A.fstep) * A.fstride + base0;
    TIn* const buf = tiles + (int64_t)b * RR_SF * per;
    each_vector(nf, [&](int q, int k, int v) {
      const int64_t e = e0 + q * A.fstep * A.fstride + k * A.cstride;
      const int64_t src = (e & ~(int64_t)(VEC - 1)) + v * VEC;
      const int64_t avail = A.total - src;  // elements of the frame buffer left from src
      const int nbytes = avail >= VEC ? 16 : (avail > 0 ? (int)avail * (int)sizeof(TIn) : 0);
      rc_cp_async16(buf + q * per + k * A.slot + v * VEC, nbytes > 0 ? (const void*)(raw + src) : (const void*)raw,
                    nbytes);
    });
  };
  const int r = r0 + threadIdx.x;
  const bool mine = r < A.oh;
  const int lr = mine ? __ldg(A.iy + r) - rlo : 0;
  const float fy = mine ? __ldg(A.wy + r) : 0.f;
  const f32x2 fy2 = pack2(fy, fy);
  const int64_t P = (int64_t)A.oh * A.ow;
  const int cs = (int)(A.cstride & (VEC - 1));
  float mx = MODE == RR_DIV ? __ldg(A.mx) : -INFINITY;
  // RR_MAX: outputs of this block outside the raw cut are extrapolated and bounded by nothing
  bool extra = false;
  if (MODE == RR_MAX) {
    const float fxc = __ldg(A.wx + c0 + (tid < cn ? tid : 0));
    extra = __syncthreads_or(fy < 0.f || fy > 1.f || fxc < 0.f || fxc > 1.f);
  }
  // Division by the maximum.  16-bit frames: q = v * (1/mx), then the correction of q by its
  // residual, fma(fma(-q, mx, v), 1/mx, q), which is the correctly rounded quotient for a
  // correctly rounded reciprocal (P. Markstein, IBM J. Res. Dev. 34, 1990) while nothing
  // overflows or underflows: the values are interpolated integers, and a maximum outside
  // [2^-10, 2^20] takes the division, as do 32-bit frames.
  const bool fast_div = MODE == RR_DIV && sizeof(TIn) == 2 && mx >= 0x1p-10f && mx <= 0x1p20f;
  const float rm = fast_div ? 1.f / mx : 0.f;
  const f32x2 rm2 = pack2(rm, rm), nmx2 = pack2(-mx, -mx);
  int b = 0;
  if (blockIdx.z < stages) stage(blockIdx.z, 0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  for (int64_t z = blockIdx.z; z < stages; z += gridDim.z, b ^= 1) {
    const int64_t zn = z + gridDim.z;
    if (zn < stages) stage(zn, b ^ 1);  // the other buffer was last read before the barrier below
    int best = MODE == RR_MAX ? *reinterpret_cast<const volatile int*>(A.best) : 0;
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;\n" ::: "memory");
    const int64_t ib = z * RR_SF;
    bool wanted = true;
    if (MODE == RR_MAX) {  // the range of the vectors that this thread has copied
      RawRange<TIn> range;
      const int nf = (int)(A.n_out - ib < RR_SF ? A.n_out - ib : RR_SF);
      each_vector(nf, [&](int q, int k, int v) {
        range.add(tiles + ((int64_t)b * RR_SF + q) * per + k * A.slot + v * VEC);
      });
      wanted = __syncthreads_or(extra || range.may_exceed(rr_unkey(best)));
    } else {
      __syncthreads();  // stage z copied by every thread
    }
    const int qa = 2 * threadIdx.y;
    const int na = (int)(A.n_out - ib < RR_SF ? A.n_out - ib : RR_SF) - qa;  // frames of this thread
    if (wanted && mine && na > 0) {
      // the second frame repeats the first when there is none (its outputs are not stored)
      const int sec = na > 1 ? 1 : 0;
      const TIn* pa = tiles + ((int64_t)b * RR_SF + qa) * per + lr;
      const TIn* pb = pa + sec * per;
      const int64_t ea = (A.f0 + (ib + qa) * A.fstep) * A.fstride + base0;
      const int la = (int)(ea & (VEC - 1)), lb = (int)((ea + sec * A.fstep * A.fstride) & (VEC - 1));
      // raw column k interpolated along the rows, both frames
      auto column = [&](int k) {
        const int oa = k * A.slot + ((la + k * cs) & (VEC - 1));
        const int ob = SAME ? oa : k * A.slot + ((lb + k * cs) & (VEC - 1));
        const f32x2 x0 = pack2(rr_raw(pa[oa]), rr_raw(pb[ob])), x1 = pack2(rr_raw(pa[oa + 1]), rr_raw(pb[ob + 1]));
        const f32x2 a = sizeof(TIn) == 2 ? add2(x0, pack2(-8388608.f, -8388608.f)) : x0;
        return fma2(sub2(x1, x0), fy2, a);
      };
      float* op = out + r + (int64_t)A.oh * c0 + P * (ib + qa);
      f32x2 left = 0, right = 0;
      // few iterations in flight per thread keep the stores of a block close together in memory:
      // 3.76 / 3.13 / 2.93 ms for the writing pass unrolled 8 / 4 / 2 times
#pragma unroll(MODE == RR_MAX ? 4 : 2)
      for (int c = 0; c < cn; ++c) {
        const int2 t = colt[c];
        const int lc = t.x & 0x7fffffff;
        left = right;
        if (t.x < 0) left = column(lc);  // block-uniform: a raw column was skipped or repeated
        right = column(lc + 1);
        const float fx = __int_as_float(t.y);
        const f32x2 o2 = fma2(sub2(right, left), pack2(fx, fx), left);
        if (MODE == RR_MAX) {
          const float2 o = unpack2(o2);
          mx = fmaxf(mx, fmaxf(o.x, o.y));
        } else {
          float2 o;
          if (MODE == RR_DIV && fast_div) {
            const f32x2 q2 = mul2(o2, rm2);
            o = unpack2(fma2(fma2(q2, nmx2, o2), rm2, q2));
          } else {
            o = unpack2(o2);
            if (MODE == RR_DIV) {
              o.x = o.x / mx;
              o.y = o.y / mx;
            }
          }
          __stcs(op, o.x);
          if (sec) __stcs(op + P, o.y);
          op += A.oh;
        }
      }
    }
    if (MODE == RR_MAX && wanted) {
      const int m = __reduce_max_sync(0xffffffffu, mx == mx ? rr_key(mx) : INT_MIN);
      if ((tid & 31) == 0 && m > best) atomicMax(A.best, m);
    }
    __syncthreads();  // buffer b is read: the next iteration may stage into it
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (MODE == RR_MAX) {
    const float m = rc_block_max(mx, mx_sh);
    if (tid == 0) A.max_part[((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = m;
  }
}

// One block: mx = max(part[0..n))
__global__ void __launch_bounds__(1024) k_rc_max(const float* __restrict__ part, int64_t n, float* __restrict__ mx) {
  __shared__ float sh[32];
  float m = -INFINITY;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, part[i]);
  m = rc_block_max(m, sh);
  if (threadIdx.x == 0) *mx = m;
}

// a /= *mx: 4 elements per thread and step (VEC: n % 4 == 0 and a 16-byte aligned).
template <bool VEC>
__global__ void __launch_bounds__(256) k_rc_scale(float* __restrict__ a, int64_t n, const float* __restrict__ mx) {
  const float m = __ldg(mx);
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  if (VEC) {
    float4* a4 = reinterpret_cast<float4*>(a);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n / 4; i += step) {
      float4 v = a4[i];
      v.x = v.x / m;
      v.y = v.y / m;
      v.z = v.z / m;
      v.w = v.w / m;
      a4[i] = v;
    }
  } else {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) a[i] = a[i] / m;
  }
}

template <typename TIn, int MODE>
int launch_rows(const void* raw, const RectifyRows& A, bool same, dim3 grid, dim3 block, size_t smem, float* out,
                cudaStream_t st) {
  auto kf = same ? k_rectify_rows<TIn, MODE, true> : k_rectify_rows<TIn, MODE, false>;
  MLF_TRY(allow_max_dyn_smem((const void*)kf));
  kf<<<grid, block, smem, st>>>(static_cast<const TIn*>(raw), A, out);
  MLF_LAUNCHED();
  return MLF_OK;
}
template <int MODE>
int launch_rows(int dtype, const void* raw, const RectifyRows& A, bool same, dim3 grid, dim3 block, size_t smem,
                float* out, cudaStream_t st) {
  return dtype == MLF_DTYPE_U16 ? launch_rows<uint16_t, MODE>(raw, A, same, grid, block, smem, out, st)
                                : launch_rows<float, MODE>(raw, A, same, grid, block, smem, out, st);
}

// MATLAB a:d:b (d != 0): count floor((b-a)/d) + 1 with a relative tolerance of 1e-10
int64_t colon_count(double a, double d, double b) {
  const double q = (b - a) / d;
  const double tol = 1e-10 * std::max(1.0, std::fabs(q));
  if (q < -tol) return 0;
  return (int64_t)std::floor(q + tol) + 1;
}

}  // namespace

// One axis of img_rectify_mod: query coordinates of the kept grid (before the cut to whole
// lenslets), 1-based.  lo = -dx/M, hi = n + 0.9.
std::vector<double> rectify_axis_query(double center, double lo, double hi, int M, double dx) {
  const double s = dx / M;
  const int64_t nl = colon_count(center, -s, lo), nr = colon_count(center + s, s, hi);
  std::vector<double> R;
  R.reserve((size_t)(nl + nr));
  for (int64_t k = nl - 1; k >= 0; --k) R.push_back(center - s * (double)k);
  for (int64_t k = 0; k < nr; ++k) R.push_back(center + s + s * (double)k);
  const int64_t c0 = nl - M / 2;  // find(R == center) = nl (1-based)
  const int64_t qinit = c0 - (int64_t)M * (int64_t)std::floor((double)c0 / M);
  if (qinit > (int64_t)R.size()) return {};
  return std::vector<double>(R.begin() + qinit, R.end());
}

int rectify_run(const void* d_raw, int dtype, int64_t total, int64_t fstride, int64_t cstride, int64_t row0, int64_t col0,
                int64_t h, int64_t w, double xc, double yc, int M, double dx, int64_t out_h, int64_t out_w,
                int64_t f0, int64_t fstep, int navg, int64_t flast, int64_t n_out, float* d_out, bool normalize,
                cudaStream_t st) {
  std::vector<double> xq = rectify_axis_query(xc, -dx / M, (double)w + 0.9, M, dx);
  std::vector<double> yq = rectify_axis_query(yc, -dx / M, (double)h + 0.9, M, dx);
  const int64_t kh = M * ((int64_t)yq.size() / M), kw = M * ((int64_t)xq.size() / M);
  if (kh != out_h || kw != out_w)
    return fail(MLF_ERR_INVALID, "After raw patch read and rectification, the shape is different from what was "
                                 "expected. (" + std::to_string(kh) + " x " + std::to_string(kw) + " vs " +
                                 std::to_string(out_h) + " x " + std::to_string(out_w) + ")");
  // per-row / per-column cell (0-based, clamped to [0, n-2]) and weight inside the cell
  std::vector<int> iy(out_h), ix(out_w);
  std::vector<float> wy(out_h), wx(out_w);
  for (int64_t r = 0; r < out_h; ++r) {
    const double c = std::min(std::max(std::floor(yq[r]), 1.0), (double)(h - 1));
    iy[r] = (int)c - 1;
    wy[r] = (float)(yq[r] - c);
  }
  for (int64_t c = 0; c < out_w; ++c) {
    const double cc = std::min(std::max(std::floor(xq[c]), 1.0), (double)(w - 1));
    ix[c] = (int)cc - 1;
    wx[c] = (float)(xq[c] - cc);
  }
  DevBuf tabs;
  const size_t tb = sizeof(int) * (out_h + out_w) + sizeof(float) * (out_h + out_w);
  MLF_TRY(tabs.alloc(tb, "rectification tables"));
  char* base = static_cast<char*>(tabs.p);
  int* d_iy = reinterpret_cast<int*>(base);
  int* d_ix = d_iy + out_h;
  float* d_wy = reinterpret_cast<float*>(d_ix + out_w);
  float* d_wx = d_wy + out_h;
  MLF_CUDA(cudaMemcpyAsync(d_iy, iy.data(), sizeof(int) * out_h, cudaMemcpyHostToDevice, st));
  MLF_CUDA(cudaMemcpyAsync(d_ix, ix.data(), sizeof(int) * out_w, cudaMemcpyHostToDevice, st));
  MLF_CUDA(cudaMemcpyAsync(d_wy, wy.data(), sizeof(float) * out_h, cudaMemcpyHostToDevice, st));
  MLF_CUDA(cudaMemcpyAsync(d_wx, wx.data(), sizeof(float) * out_w, cudaMemcpyHostToDevice, st));
  const int64_t P = out_h * out_w;
  int dev = 0, nsm = 0;
  MLF_CUDA(cudaGetDevice(&dev));
  MLF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // rows per block: of 96, 128 and 160 (the whole image's warps below 96) the one that covers
  // out_h with the fewest idle lanes, the larger on a tie.  Shorter runs of rows write partial
  // sectors at both ends too often (1065 rows: 3.76 ms with 64, 3.13 with 128, 3.15 with 160),
  // longer ones leave too few blocks on an SM (3.30 with 224, 3.68 with 288).
  int rows = out_h <= 96 ? (int)((out_h + 31) / 32 * 32) : 96;
  for (int w = rows + 32; out_h > 96 && w <= RR_MAX_ROWS; w += 32)
    if ((out_h + w - 1) / w * w <= (out_h + rows - 1) / rows * rows) rows = w;
  // largest raw tile of a block (rows and columns of the four-neighbour footprint)
  int maxr = 0, maxc = 0;
  for (int64_t r0 = 0; r0 < out_h; r0 += rows)
    maxr = std::max(maxr, iy[std::min<int64_t>(r0 + rows, out_h) - 1] + 2 - iy[r0]);
  for (int64_t c0 = 0; c0 < out_w; c0 += RR_COLS)
    maxc = std::max(maxc, ix[std::min<int64_t>(c0 + RR_COLS, out_w) - 1] + 2 - ix[c0]);
  const int es = dtype == MLF_DTYPE_U16 ? 2 : 4, vec = 16 / es;
  const int slot = ((maxr + 2 * vec - 2) / vec) * vec;
  const size_t smem = 2 * (size_t)RR_SF * maxc * slot * es;  // two stage buffers
  const int64_t gx = (out_h + rows - 1) / rows, gy = (out_w + RR_COLS - 1) / RR_COLS;
  const int64_t stages = (n_out + RR_SF - 1) / RR_SF;
  // the gather takes averaged frames, raw buffers off the 16-byte grid, pitches whose tiles
  // would leave fewer than two blocks on an SM, and 32-bit frames from pitch 1.1 on, whose large tiles
  // leave few warps on an SM (1000 x 1000 x 200, pitch 1.2: 774 us against 1127 staged; 1.1: 827 against
  // 961; at 1.02 941 against 1090, but there the staged kernel's rounding is kept; 0.8: 1276 against 1030)
  const int64_t hx = (out_h + RC_ROWS - 1) / RC_ROWS, hy = (out_w + RC_COLS - 1) / RC_COLS;  // the gather's blocks
  const bool aligned = reinterpret_cast<uintptr_t>(d_raw) % 16 == 0;
  const bool staged = navg == 1 && aligned && smem <= 112 * 1024 && hy <= 65535 &&
                      !(dtype == MLF_DTYPE_F32 && dx >= 1.1 * M);
  // calls that the 128 x 4 tiles of 16 frames took were limited to 65535 such stages: still refused,
  // whichever kernel takes them now
  if (navg == 1 && aligned && hy <= 65535 && n_out > (int64_t)16 * 65535) {
    int rows4 = 0, cols4 = 0;
    for (int64_t r0 = 0; r0 < out_h; r0 += 128)
      rows4 = std::max(rows4, iy[std::min<int64_t>(r0 + 128, out_h) - 1] + 2 - iy[r0]);
    for (int64_t c0 = 0; c0 < out_w; c0 += 4)
      cols4 = std::max(cols4, ix[std::min<int64_t>(c0 + 4, out_w) - 1] + 2 - ix[c0]);
    if (cols4 <= 8 && 32 * (size_t)cols4 * ((rows4 + 2 * vec - 2) / vec * vec) * es <= 112 * 1024)
      return fail(MLF_ERR_UNSUPPORTED, "mlf_rectify_frames: more than 1048560 output frames");
  }
  DevBuf part;
  if (staged) {
    RectifyRows A{};
    A.total = total; A.fstride = fstride; A.cstride = cstride; A.row0 = row0; A.col0 = col0;
    A.iy = d_iy; A.wy = d_wy; A.ix = d_ix; A.wx = d_wx;
    A.oh = (int)out_h; A.ow = (int)out_w;
    A.f0 = f0; A.fstep = fstep; A.n_out = n_out; A.slot = slot; A.maxc = maxc;
    const bool same = (fstep * fstride) % vec == 0;  // frames share their 16-byte alignment
    // enough z-slices for about sixteen waves of resident blocks (a short last wave), each
    // walking its stages with the next one in flight
    const int64_t gz = std::max<int64_t>(1, std::min<int64_t>({stages, (16 * 10 * (int64_t)nsm + gx * gy - 1) / (gx * gy), 65535}));
    const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)gz), block(rows, 2);
    if (!normalize) {
      MLF_TRY(launch_rows<RR_PLAIN>(dtype, d_raw, A, same, grid, block, smem, d_out, st));
    } else {
      const int64_t nb = gx * gy * gz;
      MLF_TRY(part.alloc(sizeof(float) * (nb + 2), "rectification max partials"));
      A.mx = part.as<float>();
      A.best = part.as<int>() + 1;
      A.max_part = part.as<float>() + 2;
      MLF_CUDA(cudaMemsetAsync(A.best, 0x80, sizeof(int), st));  // below any value's key but the lowest
      MLF_TRY(launch_rows<RR_MAX>(dtype, d_raw, A, same, grid, block, smem, d_out, st));
      k_rc_max<<<1, 1024, 0, st>>>(A.max_part, nb, part.as<float>());
      MLF_LAUNCHED();
      MLF_TRY(launch_rows<RR_DIV>(dtype, d_raw, A, same, grid, block, smem, d_out, st));
    }
  } else {
    const int64_t per_block = (int64_t)RC_FCH * RC_NCH;
    const int64_t hz = (n_out + per_block - 1) / per_block;
    if (hz > 65535 || hy > 65535)
      return fail(MLF_ERR_UNSUPPORTED, "mlf_rectify_frames: too many output frames or columns for one launch");
    const dim3 grid((unsigned)hx, (unsigned)hy, (unsigned)hz), block(RC_ROWS, RC_COLS);
    float* max_part = nullptr;
    if (normalize) {
      MLF_TRY(part.alloc(sizeof(float) * (hx * hy * hz + 1), "rectification max partials"));
      max_part = part.as<float>() + 1;
    }
    auto gather = [&](auto kernel, auto* src) {
      kernel<<<grid, block, 0, st>>>(src, fstride, cstride, row0, col0, d_iy, d_wy, (int)out_h, d_ix, d_wx, (int)out_w,
                                     f0, fstep, navg, flast, n_out, d_out, max_part);
    };
    if (dtype == MLF_DTYPE_U16)
      gather(navg > 1 ? k_rectify<uint16_t, true> : k_rectify<uint16_t, false>, static_cast<const uint16_t*>(d_raw));
    else
      gather(navg > 1 ? k_rectify<float, true> : k_rectify<float, false>, static_cast<const float*>(d_raw));
    MLF_LAUNCHED();
    if (normalize) {
      const int64_t n = P * n_out;
      k_rc_max<<<1, 1024, 0, st>>>(max_part, hx * hy * hz, part.as<float>());
      const bool v4 = n % 4 == 0 && reinterpret_cast<uintptr_t>(d_out) % 16 == 0;
      const int64_t want = ((v4 ? n / 4 : n) + 255) / 256;
      const unsigned nb = (unsigned)std::min<int64_t>(want, 64 * (int64_t)nsm);
      if (v4)
        k_rc_scale<true><<<nb, 256, 0, st>>>(d_out, n, part.as<float>());
      else
        k_rc_scale<false><<<nb, 256, 0, st>>>(d_out, n, part.as<float>());
      MLF_LAUNCHED();
    }
  }
  MLF_CUDA(cudaStreamSynchronize(st));  // the tables and partials are released on return
  return MLF_OK;
}

}  // namespace mlf
