// Position-variant light-field correlation with the semantics of the reference MEX
// (src/cuda/mex_lfm_convolution_vec.cu:43-266):
//
//   out[i][y][x] = sum_{ky,kx < kw} in[i][y+ky-kw/2][x+kx-kw/2] * K[(y%nn)*nn + x%nn][ky][kx]
//
// (x is MATLAB dims[0], the fast axis; kernel slot (x%nn, y%nn) is taken from the bitmap
// origin), zero outside the bitmap.  The reference clips the tap window at the edges
// (:55-78); for odd kw that is exactly zero padding.  For even kw its clip
// (bitmap_end = x + kw/2 + 1) never reaches the last input column / row, so those are
// treated as zero here too.
//
// Direct kernel (k_conv_vec_lanes).  The outputs of one row phase b = y % 15 share one set of
// 15 kernels (one per x phase).  A thread owns SEG consecutive outputs x = 15 i + a of a segment of
// 15 -- all its x phases a, or one half of them (a = 0..7 or 8..14, a CTA's threads the same half) --
// in RPT rows y = b + 15 j of one slice; the (slice, row group, segment) triples of a phase are the
// lanes of its CTAs, so warps are full whatever the sizes (narrow images: further warps that only
// stage).  Per kernel row ky a CTA stages the input
// rows its lanes read and its kernels' row ky ([kx][a], padded to 16 or 8) in shared memory with
// zero-filling cp.async, double buffered so that row ky + 1 loads while row ky is computed.  Along kx
// the thread slides a window of inputs per row in registers (one new shared load per step and row)
// and reads the step's taps as broadcast 16-byte loads.  Whole segments: kw is padded to a multiple
// of 15 with zero taps so that the 15-step rotation of the window needs no tail.  Every output adds its products in the
// reference's order -- kernel rows in order, each row left to right, one FP32 FMA chain
// (mex_lfm_convolution_vec.cu:147-251) -- and the products it adds beyond the reference's
// clipped window multiply zero-filled inputs, which adds exactly 0 for finite kernels; so
// the output equals the reference kernel's bit for bit (tests/test_gpu_ref_mex.py).
//
// Bound: small calls have fewer warps than the chip has schedulers, and a lone warp spends 2.5 cycles
// per instruction, so there one row and half a segment per thread give twice the warps for the same
// instructions per FMA; where the SMs are full, the shared-memory pipe, which returns a step's taps to
// every warp (two wavefronts per broadcast 16-byte load): two rows of a whole segment share four.
// The columns that a row has off the image are zeroed once, so staging copies what the image has and
// needs no test per element.  Half segments against one row of a whole segment: 253 x 198 x 4, kw 136
// 571 -> 483 us, 33 x 200 x 1, kw 241 1486 -> 765, 40 x 35 x 2, kw 21 54 -> 38; two rows of a whole
// segment: 396 x 380 x 9, kw 151 2.07 ms, 376 x 376 x 77, kw 241 33.9 ms (37 TFLOP/s).
#include <algorithm>
#include <climits>
#include <cmath>

#include "mlf_internal.h"

namespace mlf {

namespace {

constexpr int CV_NN = 15;           // kernels per axis (the reference's num_kernels)
constexpr int CV_HALF = 8;           // x phases of the first half of a segment (the second has 7)
constexpr int CV_RING = 2 * CV_HALF; // half segments: inputs of a row held in registers
constexpr int CV_TAHEAD = 2;         // ... kernel columns whose taps are
constexpr int CV_MAX_THREADS = 384;  // 12 warps of up to 168 registers
constexpr int CV_MAX_ROWS = 512;    // staged rows per CTA

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

struct ConvArgs {
  const float* in;   // W x H x n slices (x fastest)
  const float* K;    // kw x kw x 15 x 15 (kx fastest; kernel (a, b) at kw*kw*(a + 15 b))
  float* out;
  int W, H, kw, hk, Wv, Hv;  // Wv, Hv: columns / rows that can contribute (even kw: W-1, H-1)
  int kwp;                   // kernel columns walked: kw, or with whole segments the next multiple of 15 (zero taps)
  int SX, tilesX;            // segments per group and groups along x
  int width, pitch, gstride; // staged row: width = 15 SX + kwp - 1 floats, pitch apart; a group's RPT rows gstride
  int cta_lanes;             // lanes of a CTA, one per thread; further threads stage and compute nothing
  int max_groups;            // groups that they can touch
  int64_t n;                 // slices
};

// Lane l of phase b: group l / SX = (slice * nP + row group) * tilesX + x tile, segment l % SX.
// SEG 15: blockIdx.y is the phase; SEG CV_HALF: 2 * phase + half.
template <int RPT, int SEG>
__global__ void __launch_bounds__(CV_MAX_THREADS) k_conv_vec_lanes(ConvArgs A) {
  constexpr bool HALF = SEG != CV_NN;
  constexpr int TP = HALF ? CV_HALF : 16;     // floats per kernel column of the staged taps
  extern __shared__ __align__(16) float sm[];
  __shared__ int row_y[CV_MAX_ROWS];          // staged row: image row at ky = 0 (INT_MIN / 2: none)
  __shared__ int64_t row_src[CV_MAX_ROWS];    // ... its offset, at the tile's first column
  __shared__ short2 row_col[CV_MAX_ROWS];     // ... staged columns [x, y) that the image has
  const int b = HALF ? blockIdx.y >> 1 : blockIdx.y;        // row phase
  const int a0 = HALF ? (blockIdx.y & 1) * CV_HALF : 0;     // first x phase
  const int na = HALF && a0 ? CV_NN - CV_HALF : SEG;        // x phases
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int nJ = b < A.H ? (A.H - b + CV_NN - 1) / CV_NN : 0;  // rows of this phase
  const int nP = (nJ + RPT - 1) / RPT;
  const int64_t lanes = A.n * nP * A.tilesX * A.SX;
  const int64_t l0 = (int64_t)blockIdx.x * A.cta_lanes;
  if (l0 >= lanes) return;  // CTA-uniform
  const int64_t lN = lanes < l0 + A.cta_lanes ? lanes : l0 + A.cta_lanes;
  const int64_t g0 = l0 / A.SX;
  const int ng = (int)((lN - 1) / A.SX - g0) + 1;  // <= max_groups
  auto group = [&](int64_t g, int& jp, int& xt) {  // -> slice
    xt = (int)(g % A.tilesX);
    const int64_t q = g / A.tilesX;
    jp = (int)(q % nP);
    return q / nP;
  };
  for (int rr = tid; rr < ng * RPT; rr += nthr) {
    int jp, xt;
    const int64_t slice = group(g0 + rr / RPT, jp, xt);
    const int j = jp * RPT + rr % RPT;
    const int y0 = b + CV_NN * j - A.hk;
    row_y[rr] = j < nJ ? y0 : INT_MIN / 2;
    const int c0 = CV_NN * A.SX * xt + a0 - A.hk;
    const int ca = min(max(-c0, 0), A.width), cb = max(min(A.Wv - c0, A.width), ca);
    row_col[rr] = make_short2((short)ca, (short)cb);
    row_src[rr] = slice * (int64_t)A.W * A.H + (int64_t)y0 * A.W + c0;
  }
  // this thread's lane
  const int64_t lane_id = l0 + tid;
  const bool active = tid < A.cta_lanes && lane_id < lanes;
  const int64_t g = active ? lane_id / A.SX : g0;
  const int il = active ? (int)(lane_id - g * A.SX) : 0;
  int jp, xt;
  const int64_t slice = group(g, jp, xt);
  const int x_seg = CV_NN * (xt * A.SX + il) + a0;
  const int rowbuf = A.max_groups * A.gstride;
  float* const rows0 = sm + 2 * TP * A.kwp;  // taps of buffer s at sm + TP kwp s, rows at rows0 + rowbuf s
  const int64_t kplane = (int64_t)A.kw * A.kw;
  const float* kb = A.K + kplane * CV_NN * b;  // kernels (a, b), a = 0..14

  // Kernel row ky into buffer s, then commit.  Columns off the image stay as zeroed below; a row
  // off the image is zeroed where the buffer may hold another one.
  const int warp = tid >> 5, lane = tid & 31, nwarps = nthr >> 5;
  auto stage = [&](int ky, int s) {
    float* tb = sm + s * TP * A.kwp;
    const int ta = tid & (TP - 1);
    if (ta < na) {
      const float* src = kb + kplane * (a0 + ta) + (int64_t)A.kw * ky;
#pragma unroll 4
      for (int kx = tid / TP; kx < A.kw; kx += nthr / TP) cp_async4(tb + TP * kx + ta, src + kx);
    }
    float* rb = rows0 + s * rowbuf;
    for (int rr = warp; rr < ng * RPT; rr += nwarps) {
      const int y = row_y[rr] + ky;
      const short2 cc = row_col[rr];
      float* dst = rb + (rr / RPT) * A.gstride + (rr % RPT) * A.pitch;
      if (y >= 0 && y < A.Hv) {
        const float* src = A.in + row_src[rr] + (int64_t)ky * A.W;
#pragma unroll 4
        for (int c = cc.x + lane; c < cc.y; c += 32) cp_async4(dst + c, src + c);
      } else {
        for (int c = cc.x + lane; c < cc.y; c += 32) dst[c] = 0.f;
      }
    }
    cp_async_commit();
  };
  // the padding taps are zero in both buffers; nothing writes them again
  if (HALF) {  // the eighth phase of the second half
    if (a0)
      for (int e = tid; e < 2 * A.kwp; e += nthr) sm[TP * e + TP - 1] = 0.f;
  } else {
    for (int e = tid; e < 2 * TP * (A.kwp - A.kw); e += nthr) {
      const int s = e / (TP * (A.kwp - A.kw)), k = e - s * TP * (A.kwp - A.kw);
      sm[s * TP * A.kwp + TP * A.kw + k] = 0.f;
    }
  }
  for (int e = tid; e < 2 * rowbuf; e += nthr) rows0[e] = 0.f;
  __syncthreads();  // the row table; the zeroed buffers

  float acc[RPT][SEG];
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int a = 0; a < SEG; ++a) acc[r][a] = 0.f;
  stage(0, 0);
  cp_async_wait0();
  __syncthreads();
  for (int ky = 0; ky < A.kw; ++ky) {
    const int sel = ky & 1;
    if (ky + 1 < A.kw) stage(ky + 1, sel ^ 1);
    if (active) {
      const float* rowp = rows0 + sel * rowbuf + (int)(g - g0) * A.gstride + CV_NN * il;
      const float* tp = sm + sel * TP * A.kwp;
      const float4* t4 = reinterpret_cast<const float4*>(tp);
      if constexpr (HALF) {
        // Rings of registers: slot k % 16 of the window holds the row's value at column k, slot
        // k % CV_TAHEAD of the taps those of kernel column k.  A slot is loaded again as soon as it is
        // used; the loads past the last column (other data of this CTA's shared memory) are not used.
        float w[RPT][CV_RING];
        float4 tq[CV_TAHEAD][2];
#pragma unroll
        for (int k = 0; k < CV_TAHEAD; ++k)
#pragma unroll
          for (int q = 0; q < 2; ++q) tq[k][q] = t4[2 * k + q];
#pragma unroll
        for (int k = 0; k < CV_RING; ++k)
#pragma unroll
          for (int r = 0; r < RPT; ++r) w[r][k] = rowp[r * A.pitch + k];
        auto column = [&](int kx0, int m) {
          const float4 u = tq[m % CV_TAHEAD][0], v = tq[m % CV_TAHEAD][1];
          const float t[CV_HALF] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
          for (int a = 0; a < SEG; ++a)
#pragma unroll
            for (int r = 0; r < RPT; ++r) acc[r][a] = fmaf(w[r][(m + a) % CV_RING], t[a], acc[r][a]);
#pragma unroll
          for (int q = 0; q < 2; ++q) tq[m % CV_TAHEAD][q] = t4[2 * (kx0 + m + CV_TAHEAD) + q];
#pragma unroll
          for (int r = 0; r < RPT; ++r) w[r][m] = rowp[r * A.pitch + kx0 + m + CV_RING];
        };
        int kx0 = 0;
#pragma unroll 1
        for (; kx0 + CV_RING <= A.kwp; kx0 += CV_RING) {
#pragma unroll
          for (int m = 0; m < CV_RING; ++m) column(kx0, m);
        }
#pragma unroll
        for (int m = 0; m < CV_RING - 1; ++m) {  // the remaining columns
          if (kx0 + m >= A.kwp) break;
          column(kx0, m);
        }
      } else {
        float w[RPT][CV_NN];  // w[r][(m + a) % 15] holds row r at kx0 + m + a
#pragma unroll
        for (int r = 0; r < RPT; ++r)
#pragma unroll
          for (int a = 0; a < CV_NN - 1; ++a) w[r][a] = rowp[r * A.pitch + a];
        float4 tc[4];  // taps of the step in work; the next step's load during it
#pragma unroll
        for (int q = 0; q < 4; ++q) tc[q] = t4[q];
#pragma unroll
        for (int r = 0; r < RPT; ++r) w[r][CV_NN - 1] = rowp[r * A.pitch + CV_NN - 1];
#pragma unroll 1
        for (int kx0 = 0; kx0 < A.kwp; kx0 += CV_NN) {
#pragma unroll
          for (int m = 0; m < CV_NN; ++m) {
            float4 tn[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) tn[q] = t4[4 * (kx0 + m + 1) + q];  // past the last step: not used
            float wn[RPT];
#pragma unroll
            for (int r = 0; r < RPT; ++r) wn[r] = rowp[r * A.pitch + kx0 + m + CV_NN];
            const float t[16] = {tc[0].x, tc[0].y, tc[0].z, tc[0].w, tc[1].x, tc[1].y, tc[1].z, tc[1].w,
                                 tc[2].x, tc[2].y, tc[2].z, tc[2].w, tc[3].x, tc[3].y, tc[3].z, tc[3].w};
#pragma unroll
            for (int a = 0; a < CV_NN; ++a)
#pragma unroll
              for (int r = 0; r < RPT; ++r) acc[r][a] = fmaf(w[r][(m + a) % CV_NN], t[a], acc[r][a]);
#pragma unroll
            for (int q = 0; q < 4; ++q) tc[q] = tn[q];
#pragma unroll
            for (int r = 0; r < RPT; ++r) w[r][m] = wn[r];
          }
        }
      }
    }
    cp_async_wait0();
    __syncthreads();
  }
  if (!active) return;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int j = jp * RPT + r;
    if (j >= nJ) continue;
    float* o = A.out + slice * (int64_t)A.W * A.H + (int64_t)(b + CV_NN * j) * A.W;
#pragma unroll
    for (int a = 0; a < SEG; ++a)
      if (a < na && x_seg + a < A.W) o[x_seg + a] = acc[r][a];
  }
}

// ---- tensor-core route: the correlation above (kernel slot from the OUTPUT pixel's phase)
// equals the full light-field forward projection (PSF slice from the SOURCE pixel's phase,
// forwardProjectGPU.m) of the re-indexed kernel
//   H'[d][psi] = K[c - d + hk][(psi - (c - d)) mod 15]   per axis, c = (K0-1)/2, hk = kw/2,
// embedded in K0 = 15 + 30 m >= kw + 14 so that every tap lies inside the phase-space crop.
__global__ void k_mex_reindex(const float* __restrict__ K, int kw, int K0, int nn, float* __restrict__ Hp) {
  const int c = (K0 - 1) / 2, hk = kw / 2;
  const int64_t total = (int64_t)K0 * K0 * nn * nn;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int dx = (int)(e % K0);
    const int dy = (int)((e / K0) % K0);
    const int px = (int)((e / ((int64_t)K0 * K0)) % nn);
    const int py = (int)(e / ((int64_t)K0 * K0 * nn));
    const int kx = c - dx + hk, ky = c - dy + hk;
    float v = 0.f;
    if (kx >= 0 && kx < kw && ky >= 0 && ky < kw) {
      const int fx = ((px - (c - dx)) % nn + nn) % nn, fy = ((py - (c - dy)) % nn + nn) % nn;
      v = K[(int64_t)kx + (int64_t)kw * (ky + (int64_t)kw * (fx + (int64_t)nn * fy))];
    }
    Hp[e] = v;
  }
}

// slices of the bitmap -> zero-padded Wp x Hq slices; for even kw the reference never reads
// the last input row / column, so they are zeroed
__global__ void k_mex_pad(const float* __restrict__ bm, int64_t W, int64_t H, int64_t n, int64_t Wp, int64_t Hq,
                          int zero_last, float* __restrict__ dst) {
  const int64_t total = Wp * Hq * n;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = e % Wp, y = (e / Wp) % Hq, i = e / (Wp * Hq);
    float v = 0.f;
    if (x < W && y < H && !(zero_last && (x == W - 1 || y == H - 1))) v = bm[x + W * (y + H * i)];
    dst[e] = v;
  }
}

// dst += src zero-padded to Wp x Hq (one slice; last row / column dropped for even kw)
__global__ void k_mex_pad_add(const float* __restrict__ src, int64_t W, int64_t H, int64_t Wp, int64_t Hq,
                              int zero_last, float* __restrict__ dst) {
  const int64_t total = W * H;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = e % W, y = e / W;
    if (zero_last && (x == W - 1 || y == H - 1)) continue;
    dst[x + Wp * y] += src[e];
  }
}

__global__ void k_mex_crop(const float* __restrict__ src, int64_t Wp, int64_t Hq, int64_t W, int64_t H, int64_t n,
                           float* __restrict__ out) {
  const int64_t total = W * H * n;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = e % W, y = (e / W) % H, i = e / (W * H);
    out[e] = src[x + Wp * (y + Hq * i)];
  }
}

}  // namespace

int launch_mex_reindex(const float* K, int kw, int K0, int nn, float* Hp, cudaStream_t st) {
  k_mex_reindex<<<2048, 256, 0, st>>>(K, kw, K0, nn, Hp);
  MLF_LAUNCHED();
  return MLF_OK;
}
int launch_mex_pad(const float* bm, int64_t W, int64_t H, int64_t n, int64_t Wp, int64_t Hq, bool zero_last,
                   float* dst, cudaStream_t st) {
  k_mex_pad<<<2048, 256, 0, st>>>(bm, W, H, n, Wp, Hq, zero_last ? 1 : 0, dst);
  MLF_LAUNCHED();
  return MLF_OK;
}
int launch_mex_pad_add(const float* src, int64_t W, int64_t H, int64_t Wp, int64_t Hq, bool zero_last, float* dst,
                       cudaStream_t st) {
  k_mex_pad_add<<<512, 256, 0, st>>>(src, W, H, Wp, Hq, zero_last ? 1 : 0, dst);
  MLF_LAUNCHED();
  return MLF_OK;
}
int launch_mex_crop(const float* src, int64_t Wp, int64_t Hq, int64_t W, int64_t H, int64_t n, float* out,
                    cudaStream_t st) {
  k_mex_crop<<<2048, 256, 0, st>>>(src, Wp, Hq, W, H, n, out);
  MLF_LAUNCHED();
  return MLF_OK;
}

namespace {

struct ConvVariant {
  int rpt, halves, regs;
  double lone, each;
  const void* kernel;
};
constexpr int CV_VARIANTS = 2;
const ConvVariant* conv_variants() {
  static const ConvVariant v[CV_VARIANTS] = {{1, 2, 80, 26, 5.7, (const void*)k_conv_vec_lanes<1, CV_HALF>},
                                             {2, 1, 112, 84, 14.5, (const void*)k_conv_vec_lanes<2, CV_NN>}};
  return v;
}

// The sizes of a call, less its pointers.
ConvArgs conv_sizes(int64_t W, int64_t H, int64_t n, int64_t kw) {
  ConvArgs a{};
  a.W = (int)W;
  a.H = (int)H;
  a.n = n;
  a.kw = (int)kw;
  a.hk = (int)(kw / 2);
  a.Wv = (kw % 2 == 0) ? a.W - 1 : a.W;  // even kw: the reference's clip never reaches the last column / row
  a.Hv = (kw % 2 == 0) ? a.H - 1 : a.H;
  const int nI = (a.W + CV_NN - 1) / CV_NN;
  a.tilesX = (nI + 31) / 32;  // at most 32 segments of a row per group, evenly
  a.SX = (nI + a.tilesX - 1) / a.tilesX;
  return a;
}
int64_t conv_lanes(const ConvArgs& a, int rpt) {
  const int nJ = (a.H + CV_NN - 1) / CV_NN;
  return a.n * ((nJ + rpt - 1) / rpt) * (int64_t)a.tilesX * a.SX;
}

// Shared memory and group geometry of CTAs of `lanes` lanes; 0: they do not fit.
size_t conv_fit(const ConvVariant& v, int lanes, size_t budget, ConvArgs& c) {
  c.cta_lanes = lanes;
  c.kwp = v.halves == 2 ? c.kw : (c.kw + CV_NN - 1) / CV_NN * CV_NN;
  c.width = c.pitch = CV_NN * c.SX + c.kwp - 1;
  c.gstride = v.rpt * c.pitch;  // the next group's segments on the banks that follow (15 SX apart)
  while (c.gstride % 32 != (CV_NN * c.SX) % 32) ++c.gstride;
  c.max_groups = (int)std::min<int64_t>((lanes + c.SX - 2) / c.SX + 1, (conv_lanes(c, v.rpt) + c.SX - 1) / c.SX);
  // the rings read ahead, a few floats past their rows and taps: the last row's are past its group
  // where the stride has no padding
  constexpr size_t over = 64;
  const size_t bytes = sizeof(float) * (2 * (v.halves == 2 ? CV_HALF : 16) * (size_t)c.kwp +
                                        2 * (size_t)c.max_groups * c.gstride + over);
  return bytes <= budget && c.max_groups * v.rpt <= CV_MAX_ROWS ? bytes : (size_t)0;
}

struct ConvPlan {
  int variant = -1, warps = 0, lanes = 0;
  size_t smem = 0;
};
// Rows per thread, whole or half segments, and warps per CTA: those with the fewest cycles per
// kernel column.  A step takes `lone` cycles while the SM has at most one warp per scheduler, and
// `each` cycles of the SM per warp beyond that (measured).  One row of half a segment where that
// leaves few warps on an SM (253 x 198 x 4, kw 136: 483 us against 830 with two rows of a whole
// segment, 571 with one; 300 x 300 x 30, kw 40: 498 against 414), two rows of a whole segment where
// the SMs are full (376 x 376 x 20, kw 241: 9.6 ms against 13.7), and the CTA size that leaves the
// shortest last wave.  Two rows of half a segment lose to one or the other everywhere (400 x 400 x 1,
// kw 200: 904 us against 884; 376 x 376 x 20: 11.0 ms).
// only: that variant alone (-1: any).
ConvPlan conv_plan(const ConvArgs& a, int nsm, int optin, int smem_sm, int only) {
  const size_t budget = (size_t)optin - 12 * 1024;  // the row table is static
  ConvPlan p;
  double best = 0;
  for (int i = 0; i < CV_VARIANTS; ++i) {
    if (only >= 0 && i != only) continue;
    const ConvVariant& v = conv_variants()[i];
    const int64_t wp = (conv_lanes(a, v.rpt) + 31) / 32;  // warps per phase (and half)
    for (int k = 1; k <= CV_MAX_THREADS / 32; ++k) {
      ConvArgs c = a;
      const size_t bytes = conv_fit(v, 32 * k, budget, c);
      if (!bytes) continue;
      const int64_t per_sm = std::max<int64_t>(1, std::min<int64_t>(smem_sm / (int64_t)(bytes + 10 * 1024), 65536 / (v.regs * 32 * k)));
      const int64_t ctas = CV_NN * v.halves * ((wp + k - 1) / k);
      const int64_t waves = (ctas + nsm * per_sm - 1) / (nsm * per_sm);
      const int64_t on_sm = std::min<int64_t>(per_sm, (ctas + nsm - 1) / nsm);
      // the busiest of four schedulers; each CTA stages taps and rows of its own, shared by its
      // warps (idle ones too: 40 x 35 x 2, kw 21 has 18 lanes per phase and takes 48 us with two
      // warps, 38 with six), whose barriers cost more the more there are
      const int64_t w = k * on_sm <= 4 ? 4 : (k * on_sm + 3) / 4 * 4;
      const double stage = 8.0 * (0.5 / v.halves + (double)(c.max_groups * v.rpt) * c.width / (32.0 * a.kw)) / k;
      const double cyc = (double)waves * (std::max(v.lone, v.each * (double)w) + (stage + 2.0) * (double)on_sm + 0.35 * k);
      if (p.variant < 0 || cyc < best) {
        best = cyc;
        p = ConvPlan{i, k, 32 * k, bytes};
      }
    }
  }
  // A warp of lanes on a narrow image has 32 / SX rows of its own to stage, one after the other, per
  // kernel row.  Where all CTAs still run at once, warps without lanes share them: 31 x 31 x 60, kw 15
  // 85 -> 66 us, 45 x 45 x 60, kw 25 114 -> 81, 62 x 62 x 40, kw 15 79 -> 72 with 64 lanes, 31 x 31 x 30,
  // kw 21 101 -> 68 with eight warps; not in two waves (39 x 344 x 17, kw 220: 1622 -> 1942) nor on wider
  // images (253 x 198 x 4, kw 136, 17 segments: 509 -> 578; 100 x 100 x 60, kw 15, 7 segments: 104 -> 109).
  if (p.variant >= 0 && conv_variants()[p.variant].halves == 2 && a.SX <= 6 && conv_lanes(a, 1) > 32) {
    const ConvVariant& v = conv_variants()[p.variant];
    const int64_t lanes = conv_lanes(a, 1);
    const bool few = CV_NN * 2 * ((lanes + 31) / 32) <= 2 * (int64_t)nsm;  // at most two warps of lanes per SM
    const int shapes[3][2] = {{32, 8}, {32, 4}, {64, 4}};  // lanes, warps
    for (int i = few ? 0 : 1; i < 3; ++i) {
      ConvArgs c = a;
      const size_t bytes = conv_fit(v, shapes[i][0], budget, c);
      if (!bytes) continue;
      const int64_t per_sm = std::min<int64_t>(smem_sm / (int64_t)(bytes + 10 * 1024), 65536 / (v.regs * 32 * shapes[i][1]));
      if (CV_NN * 2 * ((lanes + shapes[i][0] - 1) / shapes[i][0]) > nsm * per_sm) continue;
      p = ConvPlan{p.variant, shapes[i][1], shapes[i][0], bytes};
      break;
    }
  }
  return p;
}

}  // namespace

int conv_plan_probe(int64_t W, int64_t H, int64_t n, int64_t kw, int nsm, int optin, int smem_sm, int variant,
                    int64_t out[10]) {
  ConvArgs a = conv_sizes(W, H, n, kw);
  const ConvPlan p = conv_plan(a, nsm, optin, smem_sm, variant);
  if (p.variant < 0) return fail(MLF_ERR_UNSUPPORTED, "direct MEX projector: kernel row does not fit in shared memory");
  const ConvVariant& v = conv_variants()[p.variant];
  conv_fit(v, p.lanes, (size_t)optin, a);
  const int64_t o[10] = {p.variant, p.warps, (int64_t)p.smem, a.kwp, a.SX, a.pitch, a.gstride, a.max_groups,
                         conv_lanes(a, v.rpt), p.lanes};
  std::copy(o, o + 10, out);
  return MLF_OK;
}

int conv_vec_run(const float* d_bitmap, int64_t W, int64_t H, int64_t n, const float* d_kernels,
                 int64_t kw, int nnum, float* d_out, cudaStream_t st) {
  if (nnum != CV_NN) return fail(MLF_ERR_INVALID, "direct MEX projector: the kernel grid must be 15 x 15");
  if (W > (1 << 24) || H > (1 << 24) || W * H > ((int64_t)1 << 31))
    return fail(MLF_ERR_UNSUPPORTED, "direct MEX projector: slice larger than 2^31 pixels");
  int dev = 0, optin = 0, nsm = 0, smem_sm = 0;
  MLF_CUDA(cudaGetDevice(&dev));
  MLF_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  MLF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  MLF_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  ConvArgs a = conv_sizes(W, H, n, kw);
  a.in = d_bitmap;
  a.K = d_kernels;
  a.out = d_out;
  const ConvPlan p = conv_plan(a, nsm, optin, smem_sm, -1);
  if (p.variant < 0) return fail(MLF_ERR_UNSUPPORTED, "direct MEX projector: kernel row does not fit in shared memory");
  const ConvVariant& v = conv_variants()[p.variant];
  conv_fit(v, p.lanes, (size_t)optin, a);
  const int threads = 32 * p.warps;
  const int64_t ctas = (conv_lanes(a, v.rpt) + p.lanes - 1) / p.lanes;
  if (ctas > INT32_MAX) return fail(MLF_ERR_UNSUPPORTED, "direct MEX projector: too many slices");
  MLF_TRY(allow_max_dyn_smem(v.kernel));
  void* args[] = {&a};
  MLF_CUDA(cudaLaunchKernel(v.kernel, dim3((unsigned)ctas, CV_NN * v.halves), dim3(threads), args, p.smem, st));
  MLF_LAUNCHED();
  return MLF_OK;
}

}  // namespace mlf
