// Summary image of a sensor movie: the input LFIMG of the reconstruction.  Follows
// src/module/summary_image_generation_module.m:43-133 with src/rank_1_factorization.m:32-45
// and src/compute_std_image.m:22-26.  The movie is P pixels x T frames, column-major (one
// frame = P contiguous floats), as the reference's sensor_movie.
//
//   rank-1 background (both modes; mathematically s = Y t / M, t normalised):
//     t = colsum(Y);  repeat bg_iter times { t = t / |t|;  s = Y t / M;  t = s' Y }
//   The reference normalises s between iterations; that scale cancels in the next t, so it
//   is not applied (s stays below sqrt(T) in magnitude).  M = max(Y).
//   'pixelwise':  y = Y / M;  z = y - movmean(y, w1);  m = movmean(z, w2);  x = m.^poly;
//                 img = sqrt(sum(x.^2)/T - mean(x)^2)
//   'global':     y = Y / M;  img = sqrt((sum(y.^2) - s.^2)/T - B.^2 + 2 B s C - s.^2 C^2),
//                 B = mean(y), C = mean(t) (compute_std_image as written)
//   summary = img / max(img).
//
// Passes over the movie (HBM-bound streams): a first column pass (t = colsum, and the max), then
// one pass per iteration but the last that forms s and the next t together (k_si_power), and a
// last row pass that also computes the image: bg_iter = 5 reads the movie 6 times.  Movies that
// k_si_power does not take (few frames, more than 2048, off the 16-byte grid) need a row and a
// column pass per iteration, 2 * bg_iter reads.
//
// Column passes: one block per 4 frames x pixel split; each float4 of s is loaded once for
// the 4 frames; partial sums per split are reduced in a fixed order (deterministic).  Row
// passes: one thread per pixel (per 4 pixels in the plain row pass), frames streamed with a
// register prefetch of the next group of frames.  The moving means run as sliding window
// sums over ring buffers in shared memory (one ring column per thread, conflict-free); the
// window-1 sum carries a TwoSum compensation term so that its error does not grow with T.
#include <cooperative_groups.h>

#include "mlf_internal.h"

namespace mlf {

namespace {

constexpr int SI_COL_THREADS = 512;
constexpr int SI_FPB = 4;           // frames per column-pass block
constexpr int SI_ROW_THREADS = 256;
constexpr int SI_ROW_U = 8;         // float4 frames prefetched per plain row-pass group
constexpr int SI_PIX_U = 32;        // frames prefetched per pixelwise group
constexpr int SI_RED_THREADS = 1024;

// scal[]: 0 M, 1 1/M, 2 max(img)
enum { SC_M = 0, SC_INVM = 1, SC_IMGMAX = 2, SC_N = 3 };

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

template <class T>
__device__ __forceinline__ T block_sum(T v, T* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  T r = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += sh[i];
  return r;  // valid in thread 0
}

__device__ __forceinline__ float block_max(float v, float* sh) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = -INFINITY;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r = fmaxf(r, sh[i]);
  return r;  // valid in thread 0
}

// t_part[ps*T + j] = sum_{p in split ps} w[p] * Y[p, j] (w = 1 when null), for the
// SI_FPB frames of block x; WITH_MAX: max_part[block] = max of Y over the block's elements.
// VEC: P % 4 == 0, Y and w 16-byte aligned, chunk % 4 == 0.
template <bool VEC, bool WITH_MAX>
__global__ void __launch_bounds__(SI_COL_THREADS)
k_si_coldot(const float* __restrict__ Y, int64_t P, int64_t T, const float* __restrict__ w, int64_t chunk,
            float* __restrict__ t_part, float* __restrict__ max_part) {
  __shared__ float sh[32];
  const int64_t j0 = (int64_t)blockIdx.x * SI_FPB;
  const int nf = (int)(T - j0 < SI_FPB ? T - j0 : SI_FPB);
  const int64_t p0 = (int64_t)blockIdx.y * chunk, p1 = P < p0 + chunk ? P : p0 + chunk;
  float acc[SI_FPB];
#pragma unroll
  for (int f = 0; f < SI_FPB; ++f) acc[f] = 0.f;
  float m = -INFINITY;
  if (VEC) {
    for (int64_t p = p0 + 4 * (int64_t)threadIdx.x; p < p1; p += 4 * SI_COL_THREADS) {
      const float4 wv = w ? __ldg(reinterpret_cast<const float4*>(w + p)) : make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
      for (int f = 0; f < SI_FPB; ++f) {
        if (f < nf) {
          const float4 y = __ldcs(reinterpret_cast<const float4*>(Y + (j0 + f) * P + p));
          acc[f] = fmaf(wv.x, y.x, fmaf(wv.y, y.y, fmaf(wv.z, y.z, fmaf(wv.w, y.w, acc[f]))));
          if (WITH_MAX) m = fmaxf(m, fmaxf(fmaxf(y.x, y.y), fmaxf(y.z, y.w)));
        }
      }
    }
  } else {
    for (int64_t p = p0 + threadIdx.x; p < p1; p += SI_COL_THREADS) {
      const float wv = w ? __ldg(w + p) : 1.f;
#pragma unroll
      for (int f = 0; f < SI_FPB; ++f) {
        if (f < nf) {
          const float y = __ldcs(Y + (j0 + f) * P + p);
          acc[f] = fmaf(wv, y, acc[f]);
          if (WITH_MAX) m = fmaxf(m, y);
        }
      }
    }
  }
#pragma unroll
  for (int f = 0; f < SI_FPB; ++f) {
    const float r = block_sum(acc[f], sh);
    if (threadIdx.x == 0 && f < nf) t_part[(int64_t)blockIdx.y * T + j0 + f] = r;
  }
  if (WITH_MAX) {
    const float r = block_max(m, sh);
    if (threadIdx.x == 0) max_part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = r;
  }
}

// One block: t = sum over splits of t_part (fixed order), t /= |t| (FP64 norm);
// nmax > 0: M = max(max_part[0..nmax)).
// Bound: latency of the one block, and FP64, of which an SM does two operations a cycle: so four
// warps take the FP64 sum (32 warps' shuffles alone cost 2 x 1.3 us) and the division by the
// norm is one reciprocal.
__global__ void __launch_bounds__(SI_RED_THREADS)
k_si_tnorm(const float* __restrict__ t_part, int ps, int64_t T, const float* __restrict__ max_part, int64_t nmax,
           float* __restrict__ t, float* __restrict__ scal) {
  constexpr int NS = 128;  // threads of the FP64 sum
  __shared__ double shd[NS / 32];
  __shared__ float shf[32];
  const int tid = threadIdx.x;
  for (int64_t j = tid; j < T; j += SI_RED_THREADS) {
    // 16 splits' loads in flight, added pairwise; their sums with compensation (up to 152 splits: one
    // chain of additions put 2.3e-7 into t at 165 x 165 x 140, where a few long splits had 7e-8)
    float v = 0.f, l = 0.f;
    for (int s0 = 0; s0 < ps; s0 += 16) {
      float x[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) x[u] = s0 + u < ps ? t_part[(int64_t)(s0 + u) * T + j] : 0.f;
#pragma unroll
      for (int st = 8; st > 0; st >>= 1)
#pragma unroll
        for (int u = 0; u < st; ++u) x[u] += x[u + st];
      float s, e;
      two_sum(v, x[0], s, e);
      v = s;
      l += e;
    }
    t[j] = isfinite(v) ? v + l : v;  // two_sum leaves NaN in l beside an infinite sum
  }
  __syncthreads();
  if (tid < NS) {
    double ss = 0.0;
    for (int64_t j = tid; j < T; j += NS) {
      const double v = t[j];
      ss += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_down_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) shd[tid >> 5] = ss;
  }
  __shared__ double rn;
  __syncthreads();
  if (tid == 0) rn = 1.0 / sqrt((shd[0] + shd[1]) + (shd[2] + shd[3]));
  __syncthreads();
  const double rnrm = rn;
  for (int64_t j = tid; j < T; j += SI_RED_THREADS) t[j] = (float)((double)t[j] * rnrm);
  if (nmax > 0) {
    float m = -INFINITY;
    for (int64_t i = tid; i < nmax; i += SI_RED_THREADS) m = fmaxf(m, max_part[i]);
    m = block_max(m, shf);
    if (tid == 0) {
      scal[SC_M] = m;
      scal[SC_INVM] = 1.f / m;
    }
  }
}

// s[p] = sum_j Y[p, j] t[j] / M, four pixels per thread (P % 4 == 0, Y 16-byte aligned).
__global__ void __launch_bounds__(SI_ROW_THREADS)
k_si_rowdot4(const float* __restrict__ Y, int64_t P, int64_t T, const float* __restrict__ t,
             const float* __restrict__ scal, float* __restrict__ s) {
  const int64_t p = 4 * ((int64_t)blockIdx.x * SI_ROW_THREADS + threadIdx.x);
  if (p >= P) return;
  const float* y = Y + p;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  int64_t j = 0;
  for (; j + SI_ROW_U <= T; j += SI_ROW_U) {
    float4 v[SI_ROW_U];
#pragma unroll
    for (int u = 0; u < SI_ROW_U; ++u) v[u] = __ldcs(reinterpret_cast<const float4*>(y + (j + u) * P));
#pragma unroll
    for (int u = 0; u < SI_ROW_U; u += 2) {
      const float t0 = __ldg(t + j + u), t1 = __ldg(t + j + u + 1);
      a.x = fmaf(v[u].x, t0, a.x); a.y = fmaf(v[u].y, t0, a.y);
      a.z = fmaf(v[u].z, t0, a.z); a.w = fmaf(v[u].w, t0, a.w);
      b.x = fmaf(v[u + 1].x, t1, b.x); b.y = fmaf(v[u + 1].y, t1, b.y);
      b.z = fmaf(v[u + 1].z, t1, b.z); b.w = fmaf(v[u + 1].w, t1, b.w);
    }
  }
  for (; j < T; ++j) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(y + j * P));
    const float tj = __ldg(t + j);
    a.x = fmaf(v.x, tj, a.x); a.y = fmaf(v.y, tj, a.y);
    a.z = fmaf(v.z, tj, a.z); a.w = fmaf(v.w, tj, a.w);
  }
  const float im = scal[SC_INVM];
  *reinterpret_cast<float4*>(s + p) = make_float4((a.x + b.x) * im, (a.y + b.y) * im, (a.z + b.z) * im, (a.w + b.w) * im);
}

// The same, one pixel per thread (any P or alignment).
__global__ void __launch_bounds__(SI_ROW_THREADS)
k_si_rowdot1(const float* __restrict__ Y, int64_t P, int64_t T, const float* __restrict__ t,
             const float* __restrict__ scal, float* __restrict__ s) {
  const int64_t p = (int64_t)blockIdx.x * SI_ROW_THREADS + threadIdx.x;
  if (p >= P) return;
  const float* y = Y + p;
  float a = 0.f, b = 0.f;
  int64_t j = 0;
  for (; j + 2 * SI_ROW_U <= T; j += 2 * SI_ROW_U) {
    float v[2 * SI_ROW_U];
#pragma unroll
    for (int u = 0; u < 2 * SI_ROW_U; ++u) v[u] = __ldcs(y + (j + u) * P);
#pragma unroll
    for (int u = 0; u < 2 * SI_ROW_U; u += 2) {
      a = fmaf(v[u], __ldg(t + j + u), a);
      b = fmaf(v[u + 1], __ldg(t + j + u + 1), b);
    }
  }
  for (; j < T; ++j) a = fmaf(__ldcs(y + j * P), __ldg(t + j), a);
  s[p] = (a + b) * scal[SC_INVM];
}

// One power iteration in one read of the movie: s = Y t / M and t_part = Y' s, t_part summed over
// clusters by k_si_tnorm.  A cluster of up to 8 CTAs splits the frames (rows per CTA <= SP_ROWS)
// and walks blocks of PB pixels.  Per block a CTA takes its rows x PB tile from shared memory into
// registers (32 values per thread), forms its part of s, adds the parts of the cluster's CTAs
// through distributed shared memory, and multiplies the same registers by s into its frames' t,
// accumulated in registers over all its blocks.
//
// Bound: HBM, at the rate that 256-byte pieces of rows a frame apart give (4.1 TB/s with 2000
// frames of 4 MB, 4.9 with 500 frames of 0.8 MB).  The two-pass form reads the movie once for s and
// once for t, at 6.4 and 5.7 TB/s; this reads it once: 1.97 ms against 1.26 + 1.41 at
// 1005 x 1005 x 2000, 0.83 against 1.36 with 1000 frames, 85 us against 66 + 86 at 465 x 450 x 500.
// With fewer than 128 frames a block's fixed latency, about 1 us, outweighs what it reads (power_fit).
// With more than 8 x 256 frames (32-pixel pieces: 4.3 against 4.0 ms at 1005 x 1005 x 3000) the two
// passes stay.  The tile of the block in work is in registers, so all three 68 KB stages are in
// flight.  The threads that publish s copy nothing: the release of a cluster barrier waits for the
// thread's own outstanding accesses.
//
// Layout: row r holds the 16-byte vectors that cover its PB pixels (PB + 4 floats); pixel p is at
// o + p with o = (frame * P) mod 4.  The rows of a thread are a multiple of 4 apart, so its o is
// one value.  Y is 16-byte aligned; bytes past the movie's end are zero-filled, not read.
constexpr int SP_THREADS = 512, SP_STAGES = 3;
constexpr int SP_PB = 64, SP_RT = 32;              // pixels per block, rows per thread
constexpr int SP_ROWS = SP_RT * SP_THREADS / SP_PB;  // 256 frames per CTA at most
constexpr int SP_MAX_CLUSTER = 8;

__device__ __forceinline__ void si_cp_async16(float* smem, const float* gmem, int src_bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(src_bytes) : "memory");
}

__global__ void __launch_bounds__(SP_THREADS, 1)
k_si_power(const float* __restrict__ Y, int64_t P, int64_t T, int rows, const float* __restrict__ t,
           const float* __restrict__ scal, float* __restrict__ t_part) {
  namespace cg = cooperative_groups;
  constexpr int PB = SP_PB, NT = SP_THREADS;
  constexpr int G = NT / PB;  // thread (pixel pa, group ga) owns rows ga, ga + G, ...
  constexpr int SLOT = PB + 4, NV = SLOT / 4;
  static_assert(G % 4 == 0, "a thread's rows must share their alignment");
  extern __shared__ __align__(16) float tiles[];  // [SP_STAGES][rows][SLOT]
  __shared__ __align__(16) float ts[G][SP_RT];    // t of row ga + G k at [ga][k], 0 past the last frame
  __shared__ float red[G][PB], sbuf[2][PB], stot[PB];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x;
  const int64_t j0 = (int64_t)rank * rows;
  const int nr = (int)max((int64_t)0, min((int64_t)rows, T - j0));  // frames of this CTA
  const int64_t total = P * T, blocks = (P + PB - 1) / PB;
  const int64_t first = blockIdx.x / C, ncl = gridDim.x / C;  // the host launches at most `blocks` clusters
  const int n = (int)((blocks - first + ncl - 1) / ncl);      // blocks of this cluster
  const int stage_floats = rows * SLOT;

  // Vector e of a stage (row e / NV) goes to floats 4e; threads PB.. copy e = le, le + NL, ...
  constexpr int NL = NT - PB, RV = (SP_ROWS * NV + NL - 1) / NL;
  const int le = tid - PB;
  const int64_t base = (j0 * P) & ~(int64_t)3;
  uint32_t rel[RV];  // first element of each vector for pixel 0, from `base` (rows * P < 2^32: host)
#pragma unroll
  for (int k = 0; k < RV; ++k) {
    const int e = max(le, 0) + NL * k, r = e / NV;
    rel[k] = (uint32_t)((((j0 + r) * P) & ~(int64_t)3) - base) + 4 * (e - r * NV);
  }
  auto load = [&](int i) {
    if (i < n && le >= 0) {
      float* dst = tiles + (i % SP_STAGES) * stage_floats + 4 * le;
      const int64_t p0 = (first + i * ncl) * PB;
      const float* src = Y + base + p0;
      if (p0 + PB + 4 <= P) {
#pragma unroll
        for (int k = 0; k < RV; ++k)
          if (le + NL * k < nr * NV) si_cp_async16(dst + 4 * NL * k, src + rel[k], 16);
      } else {  // the movie may end inside the last vectors of its last frame
        for (int e = le; e < nr * NV; e += NL) {
          const int r = e / NV;
          const int64_t at = (((j0 + r) * P) & ~(int64_t)3) + 4 * (e - r * NV) + p0, avail = total - at;
          const int bytes = avail >= 4 ? 16 : (avail > 0 ? 4 * (int)avail : 0);
          si_cp_async16(dst + 4 * (e - le), bytes > 0 ? Y + at : Y, bytes);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (int i = 0; i < SP_STAGES; ++i) load(i);
  for (int e = tid; e < G * SP_RT; e += NT) {
    const int row = e / SP_RT + G * (e % SP_RT);
    ts[e / SP_RT][e % SP_RT] = row < nr ? __ldg(t + j0 + row) : 0.f;
  }
  const int pa = tid % PB, ga = tid / PB;
  const int oa = (int)(((j0 + ga) * P) & 3);
  const int nk = ga < nr ? (nr - ga + G - 1) / G : 0;  // rows of this thread
  const float invM = scal[SC_INVM];
  float acc[SP_RT];
#pragma unroll
  for (int k = 0; k < SP_RT; ++k) acc[k] = 0.f;

  for (int i = 0; i < n; ++i) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SP_STAGES - 1) : "memory");
    __syncthreads();  // block i staged by every thread; red, sbuf and stot of block i - 1 are read
    const float* src = tiles + (i % SP_STAGES) * stage_floats + ga * SLOT + oa + pa;
    float y[SP_RT], a = 0.f, b = 0.f;
#pragma unroll
    for (int k = 0; k < SP_RT; ++k) y[k] = k < nk ? src[G * k * SLOT] : 0.f;
#pragma unroll
    for (int k = 0; k < SP_RT; k += 4) {
      const float4 tk = *reinterpret_cast<const float4*>(&ts[ga][k]);
      a = fmaf(y[k], tk.x, a);
      b = fmaf(y[k + 1], tk.y, b);
      a = fmaf(y[k + 2], tk.z, a);
      b = fmaf(y[k + 3], tk.w, b);
    }
    red[ga][pa] = a + b;
    __syncthreads();  // red complete; the stage is in registers
    if (tid < PB) {
      float v = 0.f;
#pragma unroll
      for (int g = 0; g < G; ++g) v += red[g][tid];
      sbuf[i & 1][tid] = v;
    }
    if (C > 1) {
      if (tid < PB)  // whole warps
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
      else
        asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
    }
    load(i + SP_STAGES);
    if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    if (tid < PB) {
      // sbuf[i & 1] is written again for block i + 2, after the barrier of block i + 1, at which
      // every CTA has read it
      float v = sbuf[i & 1][tid];  // one CTA: this thread's own value
      if (C > 1) {
        float part[SP_MAX_CLUSTER];
#pragma unroll
        for (int r = 0; r < SP_MAX_CLUSTER; ++r) part[r] = r < C ? *cl.map_shared_rank(&sbuf[i & 1][tid], r) : 0.f;
        v = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
      }
      stot[tid] = v * invM;
    }
    __syncthreads();
    if ((first + i * ncl) * PB + pa < P) {  // pixels past the last one contribute nothing
      const float s = stot[pa];
#pragma unroll
      for (int k = 0; k < SP_RT; ++k) acc[k] = fmaf(y[k], s, acc[k]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // t of row ga + G k: the sums of the group's two warps
  float* out = t_part + (blockIdx.x / C) * T + j0;
  constexpr int HW = PB / 32;
  static_assert(G * SP_RT * HW == G * PB, "the warp sums take red's place");
  float* wsum = &red[0][0];  // [G][SP_RT][HW]
#pragma unroll
  for (int k = 0; k < SP_RT; ++k) {
    float v = acc[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) wsum[(ga * SP_RT + k) * HW + pa / 32] = v;
  }
  __syncthreads();
  for (int e = tid; e < G * SP_RT; e += NT) {
    const int row = e / SP_RT + G * (e % SP_RT);
    float v = wsum[e * HW];
#pragma unroll
    for (int h = 1; h < HW; ++h) v += wsum[e * HW + h];
    if (row < nr) out[row] = v;
  }
  if (C > 1) cl.sync();  // no CTA leaves while its shared memory is read
}

template <int POLY>
__device__ __forceinline__ float powi(float m, int poly) {
  if (POLY >= 0) {
    if (POLY == 0) return 1.f;
    float x = m;
#pragma unroll
    for (int q = 1; q < POLY; ++q) x *= m;
    return x;
  }
  float x = 1.f;
  for (int q = 0; q < poly; ++q) x *= m;
  return x;
}

// Last pass, 'pixelwise': s (as k_si_rowdot1) and the detrended std image of each pixel.
// Shared memory: ring1[R1][blockDim] (last raw values), ring2[R2][blockDim] (last z values),
// R = min(window, T).  Unified step k = 0 .. T-1+a1+a2: Y[k] enters window 1 (k < T),
// Y[k-w1] leaves it; z[i1] (i1 = k - a1) enters window 2, z[i1-w2] leaves it; the mean of
// window 2 around i2 = i1 - a2 gives x[i2].  Window of element i: [i-b, i+a] clipped to
// [0, T-1], b = floor(w/2), a = w-1-b (MATLAB movmean / smoothdata 'movmean').  The rings
// hold raw movie values; 1/M is applied to the window-2 mean (the detrend is linear).
// Steps k in [max(w1, a1 + w2), T) have full windows on both sides and every add and drop:
// they run a branch-free form (R1 = w1, R2 = w2 there, so drop slot = write slot) that adds
// (new - dropped) to the window-1 sum with one TwoSum.  POLY >= 0 fixes the power at compile
// time; -1 takes it from `poly`.
template <int POLY>
__global__ void __launch_bounds__(128)
k_si_pixelwise(const float* __restrict__ Y, int64_t P, int T, const float* __restrict__ t,
               const float* __restrict__ scal, int w1, int w2, int R1, int R2, int poly,
               float* __restrict__ s_out, float* __restrict__ img, float* __restrict__ img_max_part) {
  extern __shared__ float ring[];
  __shared__ float sh[32];
  const int nt = blockDim.x;
  float* ring1 = ring + threadIdx.x;
  float* ring2 = ring + (int64_t)R1 * nt + threadIdx.x;
  const int64_t p = (int64_t)blockIdx.x * nt + threadIdx.x;
  float v_img = -INFINITY;
  if (p < P) {
    const float invM = scal[SC_INVM];
    const int b1 = w1 / 2, a1 = w1 - 1 - b1, b2 = w2 / 2, a2 = w2 - 1 - b2;
    const float rw1 = 1.f / (float)w1, rw2i = invM / (float)w2;
    const int R1n = R1 * nt, R2n = R2 * nt;
    const float* y = Y + p;
    float S1 = 0.f, L1 = 0.f, S2 = 0.f, sx = 0.f, sxx = 0.f, sa = 0.f, sb = 0.f;
    // ring offsets (slot * nt): in1 = k % R1, dr1 = (k - w1) % R1, c1 = (k - a1) % R1,
    //                           in2 = i1 % R2, dr2 = (i1 - w2) % R2
    int in1 = 0, dr1 = 0, c1 = 0, in2 = 0, dr2 = 0;
    auto adv = [](int& o, int nt_, int Rn) {
      o += nt_;
      if (o == Rn) o = 0;
    };
    const int K = T + a1 + a2;
    auto step = [&](int k, float raw) {
      // window 1
      if (k < T) {
        if (k >= w1) {  // R1 == w1 here: the dropped value sits in the slot being written
          float s, e;
          two_sum(S1, -ring1[in1], s, e);
          S1 = s;
          L1 += e;
        }
        ring1[in1] = raw;
        float s, e;
        two_sum(S1, raw, s, e);
        S1 = s;
        L1 += e;
        adv(in1, nt, R1n);
      } else if (k >= w1 && k - w1 < T) {
        float s, e;
        two_sum(S1, -ring1[dr1], s, e);
        S1 = s;
        L1 += e;
      }
      if (k >= w1) adv(dr1, nt, R1n);
      const int i1 = k - a1;
      if (i1 < 0) return;
      // z[i1], window 2
      if (i1 < T) {
        const int cnt = min(i1 + a1, T - 1) - max(i1 - b1, 0) + 1;
        const float rc = cnt == w1 ? rw1 : 1.f / (float)cnt;
        const float z = fmaf(-(S1 + L1), rc, ring1[c1]);
        adv(c1, nt, R1n);
        float zd = 0.f;
        if (i1 >= w2) zd = ring2[in2];  // R2 == w2 here
        ring2[in2] = z;
        S2 += z - zd;
        adv(in2, nt, R2n);
      } else if (i1 >= w2 && i1 - w2 < T) {
        S2 -= ring2[dr2];
      }
      if (i1 >= w2) adv(dr2, nt, R2n);
      const int i2 = i1 - a2;
      if (i2 < 0 || i2 >= T) return;
      const int cnt = min(i2 + a2, T - 1) - max(i2 - b2, 0) + 1;
      const float m = S2 * (cnt == w2 ? rw2i : invM / (float)cnt);
      const float x = powi<POLY>(m, poly);
      sx += x;
      sxx = fmaf(x, x, sxx);
    };
    const int k_bulk = max(w1, a1 + w2);
    float cur[SI_PIX_U];
#pragma unroll
    for (int u = 0; u < SI_PIX_U; ++u) cur[u] = u < T ? __ldcs(y + (int64_t)u * P) : 0.f;
    int k = 0;
    for (; k < T; k += SI_PIX_U) {
      float nxt[SI_PIX_U];
      if (k + 2 * SI_PIX_U <= T) {
#pragma unroll
        for (int u = 0; u < SI_PIX_U; ++u) nxt[u] = __ldcs(y + (int64_t)(k + SI_PIX_U + u) * P);
      } else {
#pragma unroll
        for (int u = 0; u < SI_PIX_U; ++u) {
          const int kk = k + SI_PIX_U + u;
          nxt[u] = kk < T ? __ldcs(y + (int64_t)kk * P) : 0.f;
        }
      }
      if (k >= k_bulk && k + SI_PIX_U <= T) {
        // bulk: both windows full, every add and drop present
        float4 tq[SI_PIX_U / 4];
#pragma unroll
        for (int q = 0; q < SI_PIX_U / 4; ++q) tq[q] = __ldg(reinterpret_cast<const float4*>(t + k) + q);
#pragma unroll
        for (int u = 0; u < SI_PIX_U; ++u) {
          const float raw = cur[u];
          const float4 tv = tq[u / 4];
          const float tj = (u & 3) == 0 ? tv.x : (u & 3) == 1 ? tv.y : (u & 3) == 2 ? tv.z : tv.w;
          if (u & 1)
            sb = fmaf(raw, tj, sb);
          else
            sa = fmaf(raw, tj, sa);
          const float d = ring1[in1];
          ring1[in1] = raw;
          float s1, e1;
          two_sum(S1, raw - d, s1, e1);  // (raw - d) rounds relative to the values, not to S1
          S1 = s1;
          L1 += e1;
          adv(in1, nt, R1n);
          const float z = fmaf(-(S1 + L1), rw1, ring1[c1]);
          adv(c1, nt, R1n);
          const float zd = ring2[in2];
          ring2[in2] = z;
          S2 += z - zd;
          adv(in2, nt, R2n);
          const float x = powi<POLY>(S2 * rw2i, poly);
          sx += x;
          sxx = fmaf(x, x, sxx);
        }
        dr1 = in1;  // R1 == w1, R2 == w2: the drop slots follow the write slots
        dr2 = in2;
      } else {
#pragma unroll
        for (int u = 0; u < SI_PIX_U; ++u) {
          const int kk = k + u;
          if (kk < T) {
            const float tj = __ldg(t + kk);
            if (u & 1)
              sb = fmaf(cur[u], tj, sb);
            else
              sa = fmaf(cur[u], tj, sa);
            step(kk, cur[u]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < SI_PIX_U; ++u) cur[u] = nxt[u];
    }
    for (k = T; k < K; ++k) step(k, 0.f);
    s_out[p] = (sa + sb) * invM;
    const float mx = sx / (float)T;
    const float v = sxx / (float)T - mx * mx;
    v_img = sqrtf(fmaxf(v, 0.f));
    img[p] = v_img;
  }
  const float r = block_max(v_img, sh);
  if (threadIdx.x == 0) img_max_part[blockIdx.x] = r;
}

// 1 / |t| and the mean of the FP32 t, for k_si_global (one block; in each of its blocks the FP64 sums
// took a third of its 133 us at 1005 x 1005 x 16).
__global__ void __launch_bounds__(SI_ROW_THREADS) k_si_tstat(const float* __restrict__ t, int64_t T, double* __restrict__ tn) {
  __shared__ double shd[32];
  double n2 = 0.0, m = 0.0;
  for (int64_t j = threadIdx.x; j < T; j += SI_ROW_THREADS) {
    const double v = __ldg(t + j);
    n2 += v * v;
    m += v;
  }
  n2 = block_sum(n2, shd);
  m = block_sum(m, shd);
  if (threadIdx.x == 0) {
    tn[0] = 1.0 / sqrt(n2);
    tn[1] = m / (double)T;
  }
}

// Last pass, 'global': s and compute_std_image(Y/M, s, t) as written in the reference.  The
// expansion cancels terms of the size of mean(y)^2 against each other, so sum(y^2), sum(y)
// and s carry TwoSum compensation (s also the exact product error) and the formula runs in
// FP64 per pixel.  There s and mean(t) are divided by the norm of the FP32 t, which its rounding leaves
// 2^-25 / sqrt(T) off one: s^2 / T is a thousand times the variance left, so that error alone put up to
// 3e-6 into the image at 140 frames.
__global__ void __launch_bounds__(SI_ROW_THREADS)
k_si_global(const float* __restrict__ Y, int64_t P, int64_t T, const float* __restrict__ t,
            const float* __restrict__ scal, const double* __restrict__ tn, float* __restrict__ s_out,
            float* __restrict__ img, float* __restrict__ img_max_part) {
  __shared__ float sh[32];
  const int64_t p = (int64_t)blockIdx.x * SI_ROW_THREADS + threadIdx.x;
  float v_img = -INFINITY;
  if (p < P) {
    const float invM = scal[SC_INVM];
    const float* y = Y + p;
    float S = 0.f, LS = 0.f, A = 0.f, LA = 0.f, B = 0.f, LB = 0.f;
    auto acc = [&](float raw, float tj) {
      const float yv = raw * invM;
      const float pr = yv * tj;
      const float ep = fmaf(yv, tj, -pr);
      float s, e;
      two_sum(S, pr, s, e);
      S = s;
      LS += e + ep;
      const float sq = yv * yv;
      const float eq = fmaf(yv, yv, -sq);
      two_sum(A, sq, s, e);
      A = s;
      LA += e + eq;
      two_sum(B, yv, s, e);
      B = s;
      LB += e;
    };
    int64_t j = 0;
    for (; j + 2 * SI_ROW_U <= T; j += 2 * SI_ROW_U) {
      float v[2 * SI_ROW_U];
#pragma unroll
      for (int u = 0; u < 2 * SI_ROW_U; ++u) v[u] = __ldcs(y + (j + u) * P);
#pragma unroll
      for (int u = 0; u < 2 * SI_ROW_U; ++u) acc(v[u], __ldg(t + j + u));
    }
    for (; j < T; ++j) acc(__ldcs(y + j * P), __ldg(t + j));
    const double sd = (double)S + (double)LS;  // Y/M already applied: s = (Y/M) t
    s_out[p] = (float)sd;
    const double Tn = (double)T, su = sd * tn[0], C = tn[1] * tn[0];  // of the unit t
    const double Ad = (double)A + (double)LA, Bm = ((double)B + (double)LB) / Tn;
    const double v = (Ad - su * su) / Tn - Bm * Bm + 2.0 * Bm * su * C - su * su * C * C;
    v_img = (float)sqrt(fmax(v, 0.0));
    img[p] = v_img;
  }
  const float r = block_max(v_img, sh);
  if (threadIdx.x == 0) img_max_part[blockIdx.x] = r;
}

__global__ void __launch_bounds__(SI_RED_THREADS)
k_si_imgmax(const float* __restrict__ part, int64_t n, float* __restrict__ scal) {
  __shared__ float sh[32];
  float m = -INFINITY;
  for (int64_t i = threadIdx.x; i < n; i += SI_RED_THREADS) m = fmaxf(m, part[i]);
  m = block_max(m, sh);
  if (threadIdx.x == 0) scal[SC_IMGMAX] = m;
}

__global__ void k_si_scale(float* __restrict__ img, int64_t P, const float* __restrict__ scal) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < P) img[p] = img[p] / scal[SC_IMGMAX];
}

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace

// Threads per block of the pixelwise pass (128, or fewer for long windows) so that the rings
// fit the device's shared memory; 0 if even 32 do not fit.
int summary_block(int64_t T, int w1, int w2, size_t smem_max, size_t* smem) {
  const int64_t per = 4 * (std::min<int64_t>(w1, T) + std::min<int64_t>(w2, T));
  for (int nt = 128; nt >= 32; nt /= 2)
    if ((size_t)(per * nt) <= smem_max) {
      *smem = (size_t)(per * nt);
      return nt;
    }
  return 0;
}

namespace {
// One power iteration in one pass (k_si_power): CTAs per cluster, frames per CTA and clusters;
// clusters = 0 where it does not apply (a movie off the 16-byte grid, more than 2048 frames) or the two
// passes are faster: below 128 frames, except movies of at most three blocks per cluster, for which two
// launches cost more than the blocks, and movies of 96 frames and more far beyond the L2, whose second
// read would come from HBM.  One pass against two, all of summary_image: 1005 x 1005 px, 16 frames 955 / 608 us, 64
// 1267 / 1161, 96 (388 MB) 1560 / 1587, 128 1731 / 1886; 700 x 700, 32 700 / 504, 96 (188 MB) 969 / 937,
// 128 1064 / 1090; 465 x 450, 16 495 / 414, 96 623 / 579, 160 707 / 736; 165 x 165 (three blocks), 8 393 /
// 405, 96 423 / 429.
struct PowerPlan {
  int cluster = 1, rows = 0, clusters = 0;
};
size_t power_smem(int64_t rows) { return sizeof(float) * SP_STAGES * (size_t)rows * (SP_PB + 4); }
int power_fit(PowerPlan* pp, int64_t P, int64_t T) {
  // clusters of 1, 2, 4, 5 and 8: eight CTAs for 1025 to 1280 frames are little more than half full, and their
  // blocks take as long (1005 x 1005 x 1100: 8.85 ms, two passes 8.11, five CTAs 6.27).  Three and six
  // are faster than four and eight too (x 520 3.47 and 3.99 ms), but leave t further off FP64 (330 x 300 x
  // 560 4.4e-8 and 4.0e-8, 300 x 165 x 1400 4.7e-8 and 4.1e-8; five 4.5e-8 and 4.3e-8 at 165 x 165 x 1100,
  // 4.7e-8 and 4.9e-8 at 450 x 420 x 1200, the two passes before 5e-8 to 7e-8)
  int c = 1;
  for (int size : {1, 2, 4, 5, SP_MAX_CLUSTER})
    if (cdiv(T, c) > SP_ROWS) c = size;
  if (cdiv(T, c) > SP_ROWS || cdiv(T, c) * P >= ((int64_t)1 << 32)) return MLF_OK;
  MLF_TRY(allow_max_dyn_smem((const void*)k_si_power));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)c;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)c);
  cfg.blockDim = dim3(SP_THREADS);
  cfg.dynamicSmemBytes = power_smem(cdiv(T, c));
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int nc = 0;
  MLF_CUDA(cudaOccupancyMaxActiveClusters(&nc, k_si_power, &cfg));
  if (nc < 1) return MLF_OK;
  if (T < 128 && !(T >= 96 && 4 * P * T >= 230000000) && cdiv(P, SP_PB) > 3 * (int64_t)nc) return MLF_OK;
  pp->cluster = c;
  pp->rows = (int)cdiv(T, c);
  pp->clusters = (int)std::min<int64_t>(nc, cdiv(P, SP_PB));
  return MLF_OK;
}
int power_launch(const PowerPlan& pp, const float* Y, int64_t P, int64_t T, const float* t, const float* scal,
                 float* t_part, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)pp.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(pp.cluster * pp.clusters));
  cfg.blockDim = dim3(SP_THREADS);
  cfg.dynamicSmemBytes = power_smem(pp.rows);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  MLF_CUDA(cudaLaunchKernelEx(&cfg, k_si_power, Y, P, T, pp.rows, t, scal, t_part));
  return MLF_OK;
}
}  // namespace

namespace {
// CUDA events around each pass when pass times are wanted (none otherwise)
struct PassClock {
  std::vector<cudaEvent_t> ev;
  bool on;
  explicit PassClock(bool want) : on(want) {}
  ~PassClock() {
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
  }
  int mark(cudaStream_t st) {
    if (!on) return MLF_OK;
    cudaEvent_t e;
    MLF_CUDA(cudaEventCreate(&e));
    ev.push_back(e);
    MLF_CUDA(cudaEventRecord(e, st));
    return MLF_OK;
  }
  float ms(size_t i) const {
    float v = 0.f;
    cudaEventElapsedTime(&v, ev[i], ev[i + 1]);
    return v;
  }
};
}  // namespace

int summary_run(const float* dY, int64_t P, int64_t T, int mode, int bg_iter, int w1, int w2, int poly,
                float* d_img, float* d_s, float* d_t, double* pass_ms, cudaStream_t st) {
  PassClock clk(pass_ms != nullptr);
  // a window of 2T or more covers the whole series for every element: same result as 2T
  w1 = (int)std::min<int64_t>(w1, 2 * T);
  w2 = (int)std::min<int64_t>(w2, 2 * T);
  int dev = 0, optin = 0;
  MLF_CUDA(cudaGetDevice(&dev));
  MLF_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  size_t smem = 0;
  const int nt = mode == MLF_DETREND_PIXELWISE ? summary_block(T, w1, w2, (size_t)optin - 256, &smem) : 128;
  if (nt == 0)
    return fail(MLF_ERR_UNSUPPORTED, "mlf_summary_image: moving-mean windows of " + std::to_string(w1) + " and " +
                                         std::to_string(w2) + " frames exceed the shared-memory rings");
  const bool vec = P % 4 == 0 && reinterpret_cast<uintptr_t>(dY) % 16 == 0;
  const int64_t ngrp = cdiv(T, SI_FPB);
  // pixel splits: about 16 column blocks per SM in total, splits of >= 16K pixels
  int64_t ps = std::max<int64_t>(1, std::min<int64_t>(cdiv(2432, ngrp), P / 16384));
  int64_t chunk = (cdiv(P, ps) + 3) / 4 * 4;
  ps = cdiv(P, chunk);
  PowerPlan pp;
  if (bg_iter > 1 && reinterpret_cast<uintptr_t>(dY) % 16 == 0) {
    MLF_TRY(power_fit(&pp, P, T));
  }
  const int64_t nrow = cdiv(P, nt);
  // one allocation for the scratch (each costs a call and, at its release, a device
  // synchronisation), every part 16-byte aligned
  const int64_t parts[7] = {T + 4, std::max<int64_t>(ps, pp.clusters) * T, ps * ngrp, SC_N,
                            std::max(nrow, cdiv(P, SI_ROW_THREADS)), P, 4};
  int64_t off[8] = {0};
  for (int k = 0; k < 7; ++k) off[k + 1] = off[k] + (parts[k] + 3) / 4 * 4;
  DevBuf scratch;
  MLF_TRY(scratch.alloc(sizeof(float) * off[7], "summary: scratch"));
  float* const tb = scratch.as<float>();
  float* const tpart = tb + off[1];
  float* const maxpart = tb + off[2];
  float* const sc = tb + off[3];
  float* const imgpart = tb + off[4];
  float* const s_tmp = tb + off[5];
  double* const tn = reinterpret_cast<double*>(tb + off[6]);
  const dim3 cgrid((unsigned)ngrp, (unsigned)ps);
  MLF_TRY(clk.mark(st));
  for (int it = 0; it < bg_iter; ++it) {
    if (it == 0) {
      if (vec)
        k_si_coldot<true, true><<<cgrid, SI_COL_THREADS, 0, st>>>(dY, P, T, nullptr, chunk, tpart,
                                                                  maxpart);
      else
        k_si_coldot<false, true><<<cgrid, SI_COL_THREADS, 0, st>>>(dY, P, T, nullptr, chunk, tpart,
                                                                   maxpart);
    } else if (pp.clusters == 0) {
      if (vec)
        k_si_coldot<true, false><<<cgrid, SI_COL_THREADS, 0, st>>>(dY, P, T, s_tmp, chunk, tpart, nullptr);
      else
        k_si_coldot<false, false><<<cgrid, SI_COL_THREADS, 0, st>>>(dY, P, T, s_tmp, chunk, tpart, nullptr);
    }
    MLF_LAUNCHED();
    k_si_tnorm<<<1, SI_RED_THREADS, 0, st>>>(tpart, it > 0 && pp.clusters ? pp.clusters : (int)ps, T, maxpart,
                                             it == 0 ? ps * ngrp : 0, tb, sc);
    MLF_LAUNCHED();
    MLF_TRY(clk.mark(st));
    if (it + 1 < bg_iter) {
      if (pp.clusters)  // this iteration's s and the next one's t
        MLF_TRY(power_launch(pp, dY, P, T, tb, sc, tpart, st));
      else if (vec)
        k_si_rowdot4<<<(unsigned)cdiv(P / 4, SI_ROW_THREADS), SI_ROW_THREADS, 0, st>>>(dY, P, T, tb, sc, s_tmp);
      else
        k_si_rowdot1<<<(unsigned)cdiv(P, SI_ROW_THREADS), SI_ROW_THREADS, 0, st>>>(dY, P, T, tb, sc, s_tmp);
      MLF_LAUNCHED();
      MLF_TRY(clk.mark(st));
    }
  }
  int64_t nparts;
  if (mode == MLF_DETREND_PIXELWISE) {
    const int R1 = (int)std::min<int64_t>(w1, T), R2 = (int)std::min<int64_t>(w2, T);
    auto kp = poly == 1 ? k_si_pixelwise<1> : poly == 2 ? k_si_pixelwise<2> : poly == 3 ? k_si_pixelwise<3>
                                                                                      : k_si_pixelwise<-1>;
    MLF_TRY(allow_max_dyn_smem((const void*)kp));
    kp<<<(unsigned)nrow, nt, smem, st>>>(dY, P, (int)T, tb, sc, w1, w2, R1, R2, poly, d_s, d_img, imgpart);
    nparts = nrow;
  } else {
    nparts = cdiv(P, SI_ROW_THREADS);
    k_si_tstat<<<1, SI_ROW_THREADS, 0, st>>>(tb, T, tn);
    MLF_LAUNCHED();
    k_si_global<<<(unsigned)nparts, SI_ROW_THREADS, 0, st>>>(dY, P, T, tb, sc, tn, d_s, d_img, imgpart);
  }
  MLF_LAUNCHED();
  MLF_TRY(clk.mark(st));
  k_si_imgmax<<<1, SI_RED_THREADS, 0, st>>>(imgpart, nparts, sc);
  k_si_scale<<<(unsigned)cdiv(P, 256), 256, 0, st>>>(d_img, P, sc);
  MLF_LAUNCHED();
  MLF_TRY(clk.mark(st));
  MLF_CUDA(cudaMemcpyAsync(d_t, tb, sizeof(float) * T, cudaMemcpyDeviceToDevice, st));
  MLF_CUDA(cudaStreamSynchronize(st));  // the scratch above is released on return
  if (pass_ms) {
    // marks: start, then per iteration: after column pass (+ t normalisation), after row pass
    // (all but the last iteration); after the last pass; after the finalisation
    double col0 = 0, col = 0, row = 0;
    size_t m = 0;
    for (int it = 0; it < bg_iter; ++it) {
      (it == 0 ? col0 : col) += clk.ms(m++);
      if (it + 1 < bg_iter) row += clk.ms(m++);
    }
    pass_ms[0] = col0;
    pass_ms[1] = bg_iter > 1 ? col / (bg_iter - 1) : 0.0;
    pass_ms[2] = bg_iter > 1 ? row / (bg_iter - 1) : 0.0;
    pass_ms[3] = clk.ms(m++);
    pass_ms[4] = clk.ms(m);
  }
  return MLF_OK;
}

}  // namespace mlf
