// xb_cmv.cu — the cmv stage (src/bach.cpp:172-268, src/cmvUtil.cpp):
// Gaussian-basis convolutions of every current substamp (W), the per-stamp
// Gram matrix Q and the projection B.
//
// Plain mode keeps the reference's precision choices: the Y pass
// accumulates in FP32 over FP64 products (cl_kern/cmv.cl:70-106), the X pass
// in FP64 (:108-135), Q and B are FP64 dot products in the reference's
// summation order (createQ :195-215 ascending pixel index, createB :217-248
// column-major).  Basis functions sharing a bit-identical Y filter share one
// Y pass.

#include <algorithm>

#include "xb_device.cuh"
#include "xb_internal.h"

namespace xb {

namespace {

constexpr int FILL_THREADS = 256;

// (x - (w * 0.5f)) / (w * 0.5f) evaluated in float (cl_kern/cmv.cl:180).
__device__ __forceinline__ double floatNorm(int x, int w) {
  float hw = (float)w * 0.5f;
  float r = ((float)x - hw) / hw;
  return (double)r;
}
__device__ __forceinline__ double ipow(double x, int n) {
  double r = 1.0;
  for(int i = 0; i < n; i++) r *= x;
  return r;
}

// Y then X pass for one (stamp, Y-filter group).  The window and the Y outputs
// are held as doubles (exact), so that a tap is one product and one sum, the
// Y accumulator's rounding to float on its bits: bound by FP64, which issues
// one warp instruction per 19 cycles per SM, conversions included (with a
// conversion of the window, one of the accumulator to float and one back per
// Y tap, and one of the Y output per X tap, 256 stamps took 3.15 ms; now
// 2.37 ms).
template <class T>
__global__ void __launch_bounds__(FILL_THREADS)
    k_fill_w(const T* __restrict__ img, int w, int h, const int* __restrict__ list,
             const int* __restrict__ count, const int* __restrict__ cur,
             const int2* __restrict__ ssxy, int maxSS, const double* __restrict__ fX,
             const double* __restrict__ fY, const int* __restrict__ gStart,
             const int* __restrict__ gMembers, int hSS, int hK, int wRows,
             double* __restrict__ W) {
  extern __shared__ double fill_s[];
  const int s = list[blockIdx.x], gi = blockIdx.y, tid = threadIdx.x;
  const int fK = 2 * hK + 1, fSS = 2 * hSS + 1, wCols = fSS * fSS;
  const int xHalf = hSS + hK, tw = 2 * xHalf + 1, th = fSS;
  const int m0 = gStart[gi], m1 = gStart[gi + 1];
  double* Ws = W + (size_t)s * wRows * wCols;
  const bool live = cur[s] < count[s];
  if(!live) {
    for(int m = m0; m < m1; m++) {
      const int n = gMembers[m];
      for(int p = tid; p < wCols; p += FILL_THREADS) Ws[(size_t)n * wCols + p] = 0.0;
    }
    return;
  }
  const int2 c = ssxy[(size_t)s * maxSS + cur[s]];
  double* win = fill_s;                        // tw x tw, rows y, cols x
  double* tmp = win + tw * tw;                 // th x tw
  double* fy = tmp + th * tw;
  double* fx = fy + fK;
  const int n0 = gMembers[m0];
  // reversed, so that a tap and its filter value run in the same direction
  for(int i = tid; i < fK; i += FILL_THREADS) fy[i] = fY[(size_t)n0 * fK + fK - 1 - i];
  // input window: x in [ssx - xHalf, ssx + xHalf], y in [ssy - xHalf, ssy + xHalf]
  for(int i = tid; i < tw * tw; i += FILL_THREADS) {
    int lx = i % tw, ly = i / tw;
    // substamp centres keep hSS+hK from the frame edge (the border mask of
    // maskInput); the clamp only guards the address
    int gx = min(max(c.x - xHalf + lx, 0), w - 1);
    int gy = min(max(c.y - xHalf + ly, 0), h - 1);
    win[i] = (double)(float)img[(size_t)gx + (size_t)gy * w];
  }
  __syncthreads();
  // Y pass (cmv.cl:70-106): v accumulates in float, products in double
  for(int p = tid; p < th * tw; p += FILL_THREADS) {
    const int row = p / tw, col = p % tw;
    const double* wc = win + row * tw + col;
    double v = 0.0;
#pragma unroll 7
    for(int y = 0; y < fK; y++) v = roundToFloat(v + wc[y * tw] * fy[y]);
    tmp[p] = v;
  }
  __syncthreads();
  for(int m = m0; m < m1; m++) {
    const int n = gMembers[m];
    for(int i = tid; i < fK; i += FILL_THREADS) fx[i] = fX[(size_t)n * fK + fK - 1 - i];
    __syncthreads();
    // X pass (cmv.cl:108-135)
    for(int p = tid; p < wCols; p += FILL_THREADS) {
      const int row = p / fSS, ii = p % fSS;
      const double* tr = tmp + row * tw + ii;
      double w0 = 0.0;
#pragma unroll 7
      for(int x = 0; x < fK; x++) w0 += tr[x] * fx[x];
      Ws[(size_t)n * wCols + p] = w0;
    }
    __syncthreads();
  }
}

// convStampOdd (cmv.cl:137-154) and convStampBg (:156-193), one row of W per
// CTA (one CTA per stamp, row after row, took 44 us for its dependent loads).
__global__ void __launch_bounds__(FILL_THREADS)
    k_fill_finish(const int* __restrict__ list, const int* __restrict__ count,
                  const int* __restrict__ cur, const int2* __restrict__ ssxy, int maxSS,
                  const int* __restrict__ kx, const int* __restrict__ ky, int nPSF,
                  const int2* __restrict__ bgXY, int nBG, int hSS, int w, int h,
                  int wRows, double* __restrict__ W) {
  const int s = list[blockIdx.x], n = 1 + blockIdx.y, tid = threadIdx.x;
  const int fSS = 2 * hSS + 1, wCols = fSS * fSS;
  double* Ws = W + (size_t)s * wRows * wCols;
  if(n < nPSF) {
    if(kx[n] % 2 != 0 || ky[n] % 2 != 0) return;
#pragma unroll 4
    for(int p = tid; p < wCols; p += FILL_THREADS) Ws[(size_t)n * wCols + p] -= Ws[p];
    return;
  }
  const int b = n - nPSF;
  const bool live = cur[s] < count[s];
  int2 c = make_int2(0, 0);
  if(live) c = ssxy[(size_t)s * maxSS + cur[s]];
  for(int p = tid; p < wCols; p += FILL_THREADS) {
    double a = 0.0;
    if(live) {
      int x = c.x - hSS + p % fSS, y = c.y - hSS + p / fSS;
      double xf = floatNorm(x, w), yf = floatNorm(y, h);
      a = ipow(xf, bgXY[b].x) * ipow(yf, bgXY[b].y);
    }
    Ws[(size_t)(nPSF + b) * wCols + p] = a;
  }
}

// createQ (cmv.cl:195-215) and createB (:217-248).  A CTA of NT threads owns NT
// entries of a stamp's lower triangle, row after row, each accumulated over the
// pixels in ascending order by one thread while the rows of W it needs stream
// through two shared-memory tiles; the last CTA of a stamp (blockIdx.y) makes
// B and the zeros of Q.  A product and a sum per entry and pixel, so bound by
// FP64 (19 cycles per warp instruction and SM) where the list fills the GPU and
// by one entry's chain of 961 sums (62 cycles each) where it does not: 64
// threads per CTA then spread a stamp over 21 SMs.  One CTA per stamp took
// 1.62 ms for 256 stamps and 0.80 ms for a single one; now 1.37 and 0.09 ms.
constexpr int GQ_KT = 32;
constexpr int GQ_MAXENT = 2048;  // entries of the triangle (host check)
template <class T, int NT>
__global__ void __launch_bounds__(NT)
    k_gram_qb(const T* __restrict__ other, const T* __restrict__ conv, int w, int h,
              const int* __restrict__ list,
              const int* __restrict__ count, const int* __restrict__ cur,
              const int2* __restrict__ ssxy, int maxSS, int hSS, int wRows, int qCount,
              const double* __restrict__ W, double* __restrict__ Q, double* __restrict__ B,
              double invGain, double rn2x2, double* __restrict__ omega) {
  extern __shared__ double gq_s[];
  const int s = list[blockIdx.x], tid = threadIdx.x;
  const int fSS = 2 * hSS + 1, wCols = fSS * fSS;
  const int R = qCount - 1;                 // W rows 0..R-1 enter Q
  const int nEnt = R * (R + 1) / 2;
  const double* Ws = W + (size_t)s * wRows * wCols;
  double* Qs = Q + (size_t)s * qCount * qCount;
  double* Bs = B + (size_t)s * qCount;
  double* om = gq_s;                                // fSS * fSS pixel weights (weighted fit)
  double* tile = om + (omega ? wCols : 0);          // 2 x (rows x (GQ_KT + 1)), or the image values
  const bool live = cur[s] < count[s];
  const int2 c = live ? ssxy[(size_t)s * maxSS + cur[s]] : make_int2(0, 0);
  if(omega) {
    // weights of the current substamp's pixels (exhausted stamps: zero)
    for(int i = tid; i < wCols; i += NT) {
      double v = 0.0;
      if(live) {
        const int gx = min(max(i % fSS - hSS + c.x, 0), w - 1);
        const int gy = min(max(i / fSS - hSS + c.y, 0), h - 1);
        const size_t id = (size_t)gx + (size_t)gy * w;
        v = fitWeight((double)conv[id], (double)other[id], invGain, rn2x2);
      }
      om[i] = v;
      if(blockIdx.y == 0) omega[(size_t)s * wCols + i] = v;
    }
  }
  if(blockIdx.y == gridDim.y - 1) {
    // zeros of the Q buffer: row 0, column 0 and above the diagonal
    for(int i = tid; i < qCount * qCount; i += NT)
      if(i % qCount > i / qCount || i % qCount == 0) Qs[i] = 0.0;
    // B: W[i-1] . other image, x outer / y inner (column-major)
    double* sub = tile;
    if(live)
      for(int i = tid; i < wCols; i += NT) {
        int x = i % fSS - hSS, y = i / fSS - hSS;
        int gx = min(max(x + c.x, 0), w - 1), gy = min(max(y + c.y, 0), h - 1);
        sub[i] = (double)other[(size_t)gx + (size_t)gy * w];
      }
    __syncthreads();
    for(int i = tid; i < qCount; i += NT) {
      double p0 = 0.0;
      if(live && i > 0) {
        const double* wr = Ws + (size_t)(i - 1) * wCols;
        for(int x = 0; x < fSS; x++) {
          const double* wx = wr + x;
          const double* sx = sub + x;
          const double* ox = om + x;
#pragma unroll 8
          for(int y = 0; y < fSS; y++)
            p0 += omega ? wx[(size_t)fSS * y] * (sx[fSS * y] * ox[fSS * y])
                        : wx[(size_t)fSS * y] * sx[fSS * y];
        }
      }
      Bs[i] = p0;
    }
    return;
  }
  // idx -> (i, j), i >= j, row-major lower triangle
  auto rowOf = [](int idx) {
    int i = (int)((sqrtf(8.f * (float)idx + 1.f) - 1.f) * 0.5f);
    while((i + 1) * (i + 2) / 2 <= idx) i++;
    while(i * (i + 1) / 2 > idx) i--;
    return i;
  };
  const int idx = blockIdx.y * NT + tid;
  const int rows = rowOf(min((int)(blockIdx.y + 1) * NT, nEnt) - 1) + 1;  // rows of W needed
  const int ei = idx < nEnt ? rowOf(idx) : 0, ej = idx < nEnt ? idx - ei * (ei + 1) / 2 : 0;
  const int tileLen = rows * (GQ_KT + 1), nT = (wCols + GQ_KT - 1) / GQ_KT;
  auto load = [&](int t) {
    const int k = t * GQ_KT + (tid & 31);
    double* dst = tile + (t & 1) * tileLen + (tid & 31);
    if(k < wCols)
      for(int r = tid >> 5; r < rows; r += NT / 32)
        cpAsync8(dst + r * (GQ_KT + 1), Ws + (size_t)r * wCols + k);
    cpAsyncCommit();
  };
  load(0);
  double q = 0.0;
  for(int t = 0; t < nT; t++) {
    if(t + 1 < nT) {
      load(t + 1);
      cpAsyncWaitGroup<1>();
    } else {
      cpAsyncWaitGroup<0>();
    }
    __syncthreads();
    const double* a = tile + (t & 1) * tileLen + ei * (GQ_KT + 1);
    const double* b = tile + (t & 1) * tileLen + ej * (GQ_KT + 1);
    const int kt = min(GQ_KT, wCols - t * GQ_KT);
    if(omega) {
      const double* o = om + t * GQ_KT;
#pragma unroll 4
      for(int kk = 0; kk < kt; kk++) q += a[kk] * (b[kk] * o[kk]);
    } else if(kt == GQ_KT) {
#pragma unroll 8
      for(int kk = 0; kk < GQ_KT; kk++) q += a[kk] * b[kk];
    } else {
      for(int kk = 0; kk < kt; kk++) q += a[kk] * b[kk];
    }
    __syncthreads();
  }
  if(idx < nEnt) Qs[(size_t)(ei + 1) * qCount + (ej + 1)] = q;
}

// ------------------------------------------------------- per-stamp dots ---
// The W dot products the global matrix needs (cd.cl:199-261,
// cdkscUtil.cpp:363-392) and the background projections of both RHS forms:
//   dots[s][0 .. nC1*nBG)            W[i1] . W[bg]       (i1 = 1..nC1)
//   dots[s][nC1*nBG + ib]            W[0]  . W[bg ib]
//   dots[s][.. + nBG + ib*nBG + jb]  W[bg ib] . W[bg jb]  (jb <= ib)
//   dots[s][.. + nBG*nBG + ib]       W[bg ib] . O, row-major, FP64 (cd.cl:331-339)
//   dots[s][.. + nBG + ib]           W[bg ib] . float(O), column-major
//                                    (cdkscUtil.cpp:459-469)
// Every dot runs in ascending pixel order (or the stated order) per thread.
// Made when a stamp is filled: they change only with its substamp, so a refit
// makes those of the refilled stamps only.
// A CTA owns DOT_THREADS products of a stamp, whose rows of W stream through
// two shared-memory tiles, the last CTA of a stamp (blockIdx.y) the background
// projections: 961 chained sums of 62 cycles, so spreading a stamp over CTAs is
// what shortens it (one CTA per stamp, the projections after the products and
// from dependent global loads, took 0.46 ms for 256 stamps; now 0.27 ms, 0.09 ms for one stamp).
constexpr int DOT_THREADS = 64, DOT_KT = 32;
struct DotPair {
  int ra, rb, oi;  // rows of W and output index; ra < 0: none
};
__device__ __forceinline__ DotPair dotPair(int pi, int nC1, int nPSF, int nBG) {
  const int nKB = nC1 * nBG;
  if(pi < nKB) return {1 + pi / nBG, nPSF + pi % nBG, pi};
  if(pi < nKB + nBG) return {0, nPSF + (pi - nKB), pi};
  const int e = pi - nKB - nBG, ib = e / nBG, jb = e % nBG;
  if(ib < nBG && jb <= ib) return {nPSF + ib, nPSF + jb, nKB + nBG + ib * nBG + jb};
  return {-1, -1, -1};
}
template <class T>
__global__ void __launch_bounds__(DOT_THREADS)
    k_stamp_dots(const int* __restrict__ list, const int* __restrict__ count,
                 const int* __restrict__ cur, const int2* __restrict__ ssxy, int maxSS,
                 const double* __restrict__ W, int wRows, int hSS, int nPSF, int nBG,
                 const T* __restrict__ O, int w, int h, double* __restrict__ dots, int stride,
                 int rowsAt, const double* __restrict__ omega) {
  extern __shared__ double dot_s[];
  const int s = list[blockIdx.x], tid = threadIdx.x;
  const int fSS = 2 * hSS + 1, wCols = fSS * fSS, nC1 = nPSF - 1;
  const double* Ws = W + (size_t)s * wRows * wCols;
  double* out = dots + (size_t)s * stride;
  const int nKB = nC1 * nBG, nPairs = nKB + nBG + nBG * nBG;
  double* om = dot_s;                         // wCols pixel weights (weighted fit)
  double* tile = om + (omega ? wCols : 0);    // 2 x rows x (DOT_KT+1), or the image values
  if(omega)
    for(int i = tid; i < wCols; i += DOT_THREADS) om[i] = omega[(size_t)s * wCols + i];
  if(blockIdx.y == gridDim.y - 1) {
    // background projections on the other image, as many background rows at a
    // time as `rowsAt` says fit behind the image values (and those as floats)
    const bool live = cur[s] < count[s];
    double* sub = tile;
    double* subF = sub + wCols;
    double* bg = subF + wCols;
    if(live) {
      const int2 c = ssxy[(size_t)s * maxSS + cur[s]];
      for(int i = tid; i < wCols; i += DOT_THREADS) {
        int x = i % fSS - hSS, y = i / fSS - hSS;
        int gx = min(max(x + c.x, 0), w - 1), gy = min(max(y + c.y, 0), h - 1);
        sub[i] = (double)O[(size_t)gx + (size_t)gy * w];
        subF[i] = (double)(float)sub[i];
      }
    }
    for(int b0 = 0; b0 < nBG; b0 += rowsAt) {
      const int nb = min(rowsAt, nBG - b0);
      __syncthreads();
#pragma unroll 8
      for(int i = tid; i < nb * wCols; i += DOT_THREADS) bg[i] = Ws[(size_t)(nPSF + b0) * wCols + i];
      __syncthreads();
      // lanes 0..nb-1 row-major, the next nb column-major
      for(int e = tid; e < 2 * nb; e += DOT_THREADS) {
        const bool byCol = e >= nb;
        const double* wb = bg + (size_t)(e % nb) * wCols;
        const double* o = byCol ? subF : sub;
        double q = 0.0;
        if(live)
          for(int a = 0; a < fSS; a++) {
            const int k0 = byCol ? a : a * fSS, dk = byCol ? fSS : 1;
#pragma unroll 8
            for(int i = 0; i < fSS; i++) {
              const int k = k0 + i * dk;
              q += omega ? wb[k] * (o[k] * om[k]) : wb[k] * o[k];
            }
          }
        out[nPairs + (byCol ? nBG : 0) + b0 + e % nb] = q;
      }
    }
    return;
  }
  // rows of this CTA's products: the background rows, row 0 and, while it has
  // products of kernel rows, those from rLo on
  const int p0 = blockIdx.y * DOT_THREADS, pi = p0 + tid;
  const int rLo = min(1 + p0 / nBG, nC1 + 1), rHi = min(1 + (p0 + DOT_THREADS - 1) / nBG, nC1);
  const int rows = 1 + nBG + max(rHi - rLo + 1, 0);
  auto rowAt = [&](int slot) { return slot == 0 ? 0 : slot <= nBG ? nPSF + slot - 1 : rLo + slot - 1 - nBG; };
  auto slotOf = [&](int r) { return r == 0 ? 0 : r >= nPSF ? 1 + r - nPSF : 1 + nBG + r - rLo; };
  const DotPair dp = pi < nPairs ? dotPair(pi, nC1, nPSF, nBG) : DotPair{-1, -1, -1};
  const int sa = dp.ra < 0 ? 0 : slotOf(dp.ra), sb = dp.ra < 0 ? 0 : slotOf(dp.rb);
  const int tileLen = rows * (DOT_KT + 1), nT = (wCols + DOT_KT - 1) / DOT_KT;
  auto load = [&](int kt) {
    const int k = kt * DOT_KT + (tid & 31);
    double* dst = tile + (kt & 1) * tileLen + (tid & 31);
    if(k < wCols)
      for(int r = tid >> 5; r < rows; r += DOT_THREADS / 32)
        cpAsync8(dst + r * (DOT_KT + 1), Ws + (size_t)rowAt(r) * wCols + k);
    cpAsyncCommit();
  };
  load(0);
  double acc = 0.0;
  for(int kt = 0; kt < nT; kt++) {
    if(kt + 1 < nT) {
      load(kt + 1);
      cpAsyncWaitGroup<1>();
    } else {
      cpAsyncWaitGroup<0>();
    }
    __syncthreads();
    const double* a = tile + (kt & 1) * tileLen + sa * (DOT_KT + 1);
    const double* b = tile + (kt & 1) * tileLen + sb * (DOT_KT + 1);
    const int len = min(DOT_KT, wCols - kt * DOT_KT);
    if(omega) {
      const double* o = om + kt * DOT_KT;
#pragma unroll 4
      for(int kk = 0; kk < len; kk++) acc += a[kk] * (b[kk] * o[kk]);
    } else if(len == DOT_KT) {
#pragma unroll 8
      for(int kk = 0; kk < DOT_KT; kk++) acc += a[kk] * b[kk];
    } else {
      for(int kk = 0; kk < len; kk++) acc += a[kk] * b[kk];
    }
    __syncthreads();
  }
  if(dp.ra >= 0) out[dp.oi] = acc;
}

}  // namespace

// Refill W, Q and B of the listed stamps of set `si`, convolving image
// `imgConv` and projecting on the other image (fillStamps,
// src/cmvUtil.cpp:37-187).
void fillStamps(xb_ctx* c, int si, const int* dList, int nList, int imgConv, const int* liveN) {
  if(nList <= 0) return;
  if(mixedMode(c)) {
    fillStampsMixed(c, si, dList, nList, imgConv, liveN);
    return;
  }
  if(liveN) throw XbError{XB_ERR_STATE, "device-counted fills are a mixed-mode path"};
  const Geo& g = c->g;
  StampSetDev& S = c->set[si];
  const int nGroups = (int)c->basis.yGroupStart.size() - 1;
  const int tw = 2 * (g.hSS + g.hK) + 1, th = g.fSS;
  const size_t smemFill = ((size_t)tw * tw + (size_t)th * tw + 2 * g.fK) * sizeof(double);
  dim3 grid(nList, nGroups);
  double* W = (double*)S.W;
  XB_CUDA(allowMaxDynamicSmem((const void*)k_fill_w<double>, c->device));
  XB_CUDA(allowMaxDynamicSmem((const void*)k_fill_w<float>, c->device));
  { KT_SCOPE(c, "fill_w");
  if(c->imgIsF64)
    k_fill_w<double><<<grid, FILL_THREADS, smemFill, c->stream>>>(
        (const double*)c->img[imgConv], c->w, c->h, dList, S.count, S.cur, S.ssxy, g.maxSS, c->dFX,
        c->dFY, c->dYGroupStart, c->dYGroupMembers, g.hSS, g.hK, g.wRows, W);
  else
    k_fill_w<float><<<grid, FILL_THREADS, smemFill, c->stream>>>(
        (const float*)c->img[imgConv], c->w, c->h, dList, S.count, S.cur, S.ssxy, g.maxSS, c->dFX,
        c->dFY, c->dYGroupStart, c->dYGroupMembers, g.hSS, g.hK, g.wRows, W);
  XB_LAUNCHED(c);
  }
  int2* bgXY = buf<int2>(c, "bgXY", g.nBG);
  { KT_SCOPE(c, "fill_finish");
  k_fill_finish<<<dim3(nList, g.nPSF - 1 + g.nBG), FILL_THREADS, 0, c->stream>>>(dList, S.count, S.cur, S.ssxy, g.maxSS,
                                                       c->dKx, c->dKy, g.nPSF, bgXY, g.nBG,
                                                       g.hSS, c->w, c->h, g.wRows, W);
  XB_LAUNCHED(c);
  }
  const double invGain = noiseInvGain(c->p), rn2x2 = noiseRn2x2(c->p);
  double* omega = c->p.fitWeighted ? S.omega : nullptr;
  const int other = 1 - imgConv;
  const size_t smemGram = (std::max((size_t)2 * (g.qCount - 1) * (GQ_KT + 1), (size_t)g.wCols) +
                           (omega ? (size_t)g.wCols : 0)) * sizeof(double);
  const int nEnt = (g.qCount - 1) * g.qCount / 2;
  // 128 entries per CTA where the list fills the SMs, else 64: of 50 rows, 64 and
  // 128 entries take 148 and 151 us for 20 stamps, 204 and 219 for 36, 269 and 290
  // for 47, 416 and 361 for 60, 412 and 403 for 70, 452 and 477 for 83, 580 and 574
  // for 106, 726 and 651 for 122; the line is at 61 stamps
  auto gram = [&](auto* img, auto kernel, int nt) {
    XB_CUDA(allowMaxDynamicSmem((const void*)kernel, c->device));
    kernel<<<dim3(nList, (nEnt + nt - 1) / nt + 1), nt, smemGram, c->stream>>>(
        img, (decltype(img))c->img[imgConv], c->w, c->h, dList, S.count, S.cur, S.ssxy, g.maxSS,
        g.hSS, g.wRows, g.qCount, W, S.Q, S.B, invGain, rn2x2, omega);
  };
  const bool wide = (long long)nList * nEnt > 2ll * 256 * c->smCount;
  { KT_SCOPE(c, "gram_qb");
  if(c->imgIsF64) {
    if(wide) gram((const double*)c->img[other], k_gram_qb<double, 128>, 128);
    else gram((const double*)c->img[other], k_gram_qb<double, 64>, 64);
  } else {
    if(wide) gram((const float*)c->img[other], k_gram_qb<float, 128>, 128);
    else gram((const float*)c->img[other], k_gram_qb<float, 64>, 64);
  }
  XB_LAUNCHED(c);
  }
  const int nPairs = g.nComp1 * g.nBG + g.nBG + g.nBG * g.nBG;
  const int maxRows = 1 + g.nBG + std::min(g.nComp1, DOT_THREADS / g.nBG + 2);
  // background rows staged at a time: all of them, or what 96 KB hold
  const int rowsAt = std::max(1, std::min(g.nBG, (int)((96 << 10) / (g.wCols * sizeof(double)))));
  const size_t smemDots = (std::max((size_t)2 * maxRows * (DOT_KT + 1), (size_t)(2 + rowsAt) * g.wCols) +
                           (omega ? (size_t)g.wCols : 0)) * sizeof(double);
  auto dots = [&](auto* img, auto kernel) {
    XB_CUDA(allowMaxDynamicSmem((const void*)kernel, c->device));
    kernel<<<dim3(nList, (nPairs + DOT_THREADS - 1) / DOT_THREADS + 1), DOT_THREADS, smemDots,
             c->stream>>>(dList, S.count, S.cur, S.ssxy, g.maxSS, W, g.wRows, g.hSS, g.nPSF, g.nBG,
                          img, c->w, c->h, S.dots, plainDotStride(g), rowsAt, omega);
  };
  { KT_SCOPE(c, "stamp_dots");
  if(c->imgIsF64) dots((const double*)c->img[other], k_stamp_dots<double>);
  else dots((const float*)c->img[other], k_stamp_dots<float>);
  XB_LAUNCHED(c);
  }
}

void stageCmv(xb_ctx* c) {
  const Geo& g = c->g;
  if((g.qCount - 1) * (g.qCount) / 2 > GQ_MAXENT)
    throw XbError{XB_ERR_UNSUPPORTED, "too many basis functions for the Gram kernel"};
  // basis tables (host-built once per context) and background exponents
  std::vector<int2> bg(g.nBG);
  for(int b = 0; b < g.nBG; b++) bg[b] = make_int2(c->basis.bgX[b], c->basis.bgY[b]);
  toDevice(c, buf<int2>(c, "bgXY", g.nBG), bg);
  for(int si = 0; si < 2; si++) {
    StampSetDev& S = c->set[si];
    const std::string sfx = std::to_string(si);
    if(mixedMode(c)) {
      S.Wf = buf<float>(c, "Wf" + sfx, (size_t)std::max(S.n, 1) * g.wRows * mixedLd(g));
      S.Wlo = buf<float>(c, "Wlo" + sfx, (size_t)std::max(S.n, 1) * g.wRows * mixedLd(g));
      S.dots = buf<double>(c, "dots" + sfx, (size_t)std::max(S.n, 1) * mixedDotStride(g));
    } else {
      S.W = buf<double>(c, "W" + sfx, (size_t)std::max(S.n, 1) * g.wRows * g.wCols);
      S.dots = buf<double>(c, "dots" + sfx, (size_t)std::max(S.n, 1) * plainDotStride(g));
      S.omega = c->p.fitWeighted ? buf<double>(c, "omega" + sfx, (size_t)std::max(S.n, 1) * g.wCols)
                                 : nullptr;
    }
    S.Q = buf<double>(c, "Q" + sfx, (size_t)std::max(S.n, 1) * g.qCount * g.qCount);
    S.B = buf<double>(c, "B" + sfx, (size_t)std::max(S.n, 1) * g.bCount);
    std::vector<int> all(S.n);
    for(int s = 0; s < S.n; s++) all[s] = s;
    int* dList = buf<int>(c, "fillList" + sfx, std::max(S.n, 1));
    toDevice(c, dList, all);
    fillStamps(c, si, dList, S.n, si, S.dN);
  }
  if(c->trace) {
    for(int si = 0; si < 2; si++) {
      const StampSetDev& S = c->set[si];
      const std::string sfx = std::to_string(si);
      c->put("Q" + sfx, toHost(c, S.Q, (size_t)S.n * g.qCount * g.qCount));
      c->put("B" + sfx, toHost(c, S.B, (size_t)S.n * g.bCount));
      if(mixedMode(c)) {
        c->put("Wf" + sfx, toHost(c, S.Wf, (size_t)S.n * g.wRows * mixedLd(g)));
        c->put("Wlo" + sfx, toHost(c, S.Wlo, (size_t)S.n * g.wRows * mixedLd(g)));
      }
      else
        c->put("W" + sfx, toHost(c, (const double*)S.W, (size_t)S.n * g.wRows * g.wCols));
    }
  }
}

}  // namespace xb
