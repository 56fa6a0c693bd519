// xb_fit.cu — cd and ksc: per-stamp test fits, convolution-direction merit,
// global normal matrix, global LU solve, per-stamp chi^2 and the
// reject/refill loop (src/cdkscUtil.cpp, src/bachUtil.cpp:288-541,
// cl_kern/cd.cl, cl_kern/ksc.cl, cl_kern/bach.cl:1-127).
//
// Plain mode reproduces the reference's FP64 operation order, so kernel sums,
// merits, chi^2 and therefore the test-stamp and rejection sets are
// bit-identical to the CPU oracle.  Atomic-order compactions of the
// reference (genCdTestStamps, removeBadSigs, checkBadSubStamps) keep
// ascending stamp order.

#include <cooperative_groups.h>

#include <algorithm>
#include <climits>

#include "xb_device.cuh"
#include "xb_internal.h"

namespace cg = cooperative_groups;

namespace xb {

namespace {

// ----------------------------------------------------------- LU helpers ---
// NR lubksb (bach.cl:89-127 / bachUtil.cpp:386-411) by one warp: lanes form
// the products, lane 0 runs each row's subtraction chain in the reference's
// order.  a is row-major with leading dimension ld, 1-based.
__device__ void warpLubksb(const double* a, int ld, int n, const int* idx, double* b,
                           double* prod) {
  const int lane = threadIdx.x & 31;
  int ii = 0;
  for(int i = 1; i <= n; i++) {
    const int ip = idx[i];
    double sum = b[ip];
    __syncwarp();
    if(lane == 0) b[ip] = b[i];
    __syncwarp();
    if(ii != 0) {
      for(int j = ii + lane; j < i; j += 32) prod[j] = a[(size_t)i * ld + j] * b[j];
      __syncwarp();
      if(lane == 0)
        for(int j = ii; j < i; j++) sum -= prod[j];
      sum = __shfl_sync(0xffffffffu, sum, 0);
    } else if(sum != 0.0) {
      ii = i;
    }
    if(lane == 0) b[i] = sum;
    __syncwarp();
  }
  for(int i = n; i >= 1; i--) {
    double sum = b[i];
    for(int j = i + 1 + lane; j <= n; j += 32) prod[j] = a[(size_t)i * ld + j] * b[j];
    __syncwarp();
    if(lane == 0) {
      for(int j = i + 1; j <= n; j++) sum -= prod[j];
      b[i] = sum / a[(size_t)i * ld + i];
    }
    __syncwarp();
  }
}

// Pivot reduction: larger value wins, ties go to the larger row (the
// sequential `dum >= big` rule), NaN never wins.
__device__ __forceinline__ void pivotCombine(double& v, int& i, double ov, int oi) {
  if(oi >= 0 && (i < 0 || ov > v || (ov == v && oi > i))) {
    v = ov;
    i = oi;
  }
}

// Both stamp sets of cd in one launch (grid dimension y, or x of a one-CTA
// kernel): n bounds a set's kept stamps, liveN, when set, counts them on the
// device.
struct CdSets {
  const double* Q[2];
  const double* B[2];
  int n[2];
  const int* liveN[2];
  double* ks[2];
  int* testIdx[2];
};

// ------------------------------------------------------ per-stamp test fit --
// createTestVec/createTestMat (cd.cl:15-44), GPU ludcmp (bach.cl:1-87, no
// zero-row check) and lubksb, saveKernelSums (cd.cl:46-52).  The Crout
// elimination of the reference is run right-looking: every entry receives
// the same products in the same order, so the factors are identical.
constexpr int LU_THREADS = 128;
__global__ void __launch_bounds__(LU_THREADS)
    k_stamp_test_fit(const __grid_constant__ CdSets sets, int qc) {
  extern __shared__ double lu_s[];
  const int set = blockIdx.y;
  const int* liveN = sets.liveN[set];
  if((int)blockIdx.x >= sets.n[set] || (liveN && (int)blockIdx.x >= *liveN)) return;
  const double* __restrict__ Q = sets.Q[set];
  const double* __restrict__ B = sets.B[set];
  double* __restrict__ kernelSums = sets.ks[set];
  const int s = blockIdx.x, tid = threadIdx.x, n = qc - 1;
  double* a = lu_s;                 // qc * qc
  double* b = a + qc * qc;          // qc
  double* vv = b + qc;              // qc
  double* prod = vv + qc;           // qc
  int* idx = (int*)(prod + qc);     // qc
  __shared__ double rv[LU_THREADS / 32];
  __shared__ int ri[LU_THREADS / 32];
  __shared__ int sMaxI;
  const double* Qs = Q + (size_t)s * qc * qc;
  for(int k = tid; k < qc * qc; k += LU_THREADS) {
    int i = k / qc, j = k % qc;
    a[k] = (i > 0 && j > 0) ? Qs[(size_t)max(i, j) * qc + min(i, j)] : 0.0;
  }
  for(int i = tid; i < qc; i += LU_THREADS) {
    b[i] = i > 0 ? B[(size_t)s * qc + i] : 0.0;
    idx[i] = 0;
  }
  __syncthreads();
  for(int i = tid; i < qc; i += LU_THREADS) {
    double big = 0.0;
    if(i > 0)
      for(int j = 1; j <= n; j++) {
        double t = fabs(a[i * qc + j]);
        if(t > big) big = t;
      }
    vv[i] = i > 0 ? 1.0 / big : 0.0;
  }
  if(tid == 0) sMaxI = 0;
  __syncthreads();
  for(int j = 1; j <= n; j++) {
    double bv = 0.0;
    int bi = -1;
    for(int i = j + tid; i <= n; i += LU_THREADS) {
      double dum = vv[i] * fabs(a[i * qc + j]);
      if(dum >= 0.0) pivotCombine(bv, bi, dum, i);
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {
      double ov = __shfl_down_sync(0xffffffffu, bv, o);
      int oi = __shfl_down_sync(0xffffffffu, bi, o);
      pivotCombine(bv, bi, ov, oi);
    }
    if((tid & 31) == 0) {
      rv[tid >> 5] = bv;
      ri[tid >> 5] = bi;
    }
    __syncthreads();
    if(tid == 0) {
      double v = rv[0];
      int i0 = ri[0];
      for(int w = 1; w < LU_THREADS / 32; w++) pivotCombine(v, i0, rv[w], ri[w]);
      if(i0 >= 0) sMaxI = i0;
      idx[j] = sMaxI;
    }
    __syncthreads();
    const int p = sMaxI;
    if(p != j) {
      for(int k = 1 + tid; k <= n; k += LU_THREADS) {
        double t = a[p * qc + k];
        a[p * qc + k] = a[j * qc + k];
        a[j * qc + k] = t;
      }
      __syncthreads();
      if(tid == 0) vv[p] = vv[j];
    }
    __syncthreads();
    if(tid == 0 && a[j * qc + j] == 0.0) a[j * qc + j] = 1.0e-20;
    __syncthreads();
    if(j != n) {
      const double dum = 1.0 / a[j * qc + j];
      for(int i = j + 1 + tid; i <= n; i += LU_THREADS) a[i * qc + j] *= dum;
    }
    __syncthreads();
    const int m = n - j;
    for(int e = tid; e < m * m; e += LU_THREADS) {
      int i = j + 1 + e / m, k = j + 1 + e % m;
      a[i * qc + k] -= a[i * qc + j] * a[j * qc + k];
    }
    __syncthreads();
  }
  if(tid < 32) warpLubksb(a, qc, n, idx, b, prod);
  __syncthreads();
  if(tid == 0) kernelSums[s] = b[1];
}

// ------------------------------------------- per-stamp test fit, mixed ----
// The mixed path only needs each stamp's kernel sum (the first unknown of
// its test system; cd.cl:46-52) for the sigma clip of cd, and its Q, B already
// differ from the plain ones at the 1e-11 level, so it solves the symmetric
// positive definite test system (createTestMat / createTestVec, cd.cl:15-44)
// by LDL^T without pivoting, one warp per stamp, instead of the reference's
// LU with partial pivoting.  The kernel-sum unknown is ordered last and the
// right-hand side rides along as an extra column of the elimination, so after
// it the kernel sum is that column's last entry over the last pivot (with L D
// L^T x = b and z = L^-1 b, the last row of L^T x = D^-1 z is x_n = z_n / d_n):
// no back substitution.  A zero pivot becomes 1e-20, as in the reference's LU.
// Warps (stamps) per CTA: 4 (variant 0), 2 or 8; identical results.
//
// Bound by FP64, one warp instruction per 19 cycles and SM.  A lane per row
// spent 1700 of them on the 640 warp instructions' worth of entries, and
// waited for each entry's loads; so the entries of the trailing triangle (and
// of the right-hand side) go to the lanes one by one, from a table in the order
// of falling columns, of which every step takes a prefix, four per lane at a
// time.  Both sets of 256 stamps of 49 unknowns in one launch: 82 us (two
// launches of a row per lane: 371).
constexpr int TF_MAXN = 127;  // the table's fields hold 7 bits of row and column
inline size_t tfEntries(int n) { return (size_t)(n - 1) * n / 2 + (n - 1); }
inline size_t tfSmemBytes(int n, int warps) {
  return ((size_t)(n + 1) * (n | 1) + n) * warps * sizeof(double) + tfEntries(n) * sizeof(unsigned);
}
template <int TF_WARPS>
__global__ void __launch_bounds__(TF_WARPS * 32)
    k_stamp_test_fit_ldl(const __grid_constant__ CdSets sets, int qc) {
  extern __shared__ double tf_s[];
  const int set = blockIdx.y, nStamps = sets.n[set];
  const int* liveN = sets.liveN[set];
  const double* __restrict__ Q = sets.Q[set];
  const double* __restrict__ B = sets.B[set];
  double* __restrict__ kernelSums = sets.ks[set];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s = blockIdx.x * TF_WARPS + warp;
  const int nLive = liveN ? min(nStamps, *liveN) : nStamps;
  if((int)blockIdx.x * TF_WARPS >= nLive) return;
  const int n = qc - 1, ld = n | 1;  // unknowns; row stride (row n = the RHS)
  const int perWarp = (n + 1) * ld + n;
  double* a = tf_s + (size_t)warp * perWarp;
  double* l = a + (n + 1) * ld;
  unsigned* tab = (unsigned*)(tf_s + (size_t)TF_WARPS * perWarp);  // dst << 14 | i << 7 | j
  for(int j = 1 + threadIdx.x; j < n; j += TF_WARPS * 32) {
    const int m = n - 1 - j;
    unsigned* t = tab + m * (m + 1) / 2 + m;
    *t++ = (unsigned)(n * ld + j) << 14 | j << 7 | n;
    for(int i = j; i < n; i++) *t++ = (unsigned)(i * ld + j) << 14 | i << 7 | j;
  }
  __syncthreads();
  if(s >= nLive) return;  // whole warps only; no block barrier from here on
  const double* Qs = Q + (size_t)s * qc * qc;
  // unknown order: 2, 3, ..., n, then 1 (the kernel sum)
  auto unk = [&](int p) { return p < n - 1 ? p + 2 : 1; };
  for(int q = lane; q < n; q += 32) {
    const int t = unk(q);
#pragma unroll 8
    for(int p = 0; p < n; p++) {
      const int u = unk(p);
      a[p * ld + q] = Qs[(size_t)max(u, t) * qc + min(u, t)];
    }
    a[n * ld + q] = B[(size_t)s * qc + t];
  }
  __syncwarp();
  for(int k = 0; k < n - 1; k++) {
    double d = a[k * ld + k];
    if(d == 0.0) d = 1.0e-20;
    const double rd = 1.0 / d;
    for(int i = k + 1 + lane; i < n; i += 32) l[i] = a[i * ld + k] * rd;
    __syncwarp();
    const int m = n - 1 - k, cnt = m * (m + 1) / 2 + m;
    for(int e = lane; e < cnt; e += 128) {
      double c[4], x[4], y[4];
      unsigned t[4];
#pragma unroll
      for(int v = 0; v < 4; v++) t[v] = tab[min(e + 32 * v, cnt - 1)];
#pragma unroll
      for(int v = 0; v < 4; v++) {
        c[v] = a[t[v] >> 14];
        x[v] = l[t[v] >> 7 & 127];
        y[v] = a[(t[v] & 127) * ld + k];
      }
#pragma unroll
      for(int v = 0; v < 4; v++)
        if(e + 32 * v < cnt) a[t[v] >> 14] = fma(-x[v], y[v], c[v]);
    }
    __syncwarp();
  }
  if(lane == 0) {
    double d = a[(n - 1) * ld + n - 1];
    if(d == 0.0) d = 1.0e-20;
    kernelSums[s] = a[n * ld + n - 1] / d;
  }
}

// ------------------------------------------------------------ cd select ---
// sigmaClip of the kernel sums (10 iterations, cdkscUtil.cpp:74-76) and
// genCdTestStamps (cd.cl:54-94) in ascending order.
__global__ void __launch_bounds__(256)
    k_cd_select(const __grid_constant__ CdSets sets, int nMax, double alpha, double sigKernFit,
                uint8_t* flags, double* cs, double* cs2, int* __restrict__ nTest,
                double* __restrict__ stats) {
  const int set = blockIdx.x, n = sets.liveN[set] ? *sets.liveN[set] : sets.n[set];
  const double* __restrict__ ks = sets.ks[set];
  int* __restrict__ testIdx = sets.testIdx[set];
  flags += (size_t)set * nMax;
  cs += (size_t)set * nMax;
  cs2 += (size_t)set * nMax;
  nTest += set;
  stats += 2 * set;
  __shared__ double sMean, sStd;
  __shared__ int sh[4];
  __shared__ int warpTot[8];
  __shared__ int sTotal;
  blockSigmaClip(ks, n, 10, alpha, flags, cs, cs2, &sMean, &sStd, sh);
  const double m = sMean, sd = sStd;
  int done = 0;
  for(int base = 0; base < n; base += 256) {
    int s = base + threadIdx.x;
    int keep = (s < n && fabs((ks[s] - m) / sd) < sigKernFit) ? 1 : 0;
    int pos = blockScanExcl(keep, warpTot, &sTotal) + done;
    if(keep) testIdx[pos] = s;
    done += sTotal;
    __syncthreads();
  }
  if(threadIdx.x == 0) {
    *nTest = done;
    stats[0] = m;
    stats[1] = sd;
  }
}

// ---------------------------------------------------- spatial weights -----
// createMatrixWeights (cd.cl:152-180) = the weight loop of CPU createMatrix
// (cdkscUtil.cpp:331-342), as the table of products the matrix entries use:
// pw[t][a][b] = w_a w_b over the nC2 weights and, at index nC2, a one; and the
// listed stamps, exhausted ones with bit 31 set.
__global__ void __launch_bounds__(128)
    k_weights(const int* __restrict__ list, const int* __restrict__ count,
              const int* __restrict__ cur, const int2* __restrict__ ssxy, int maxSS,
              const int2* __restrict__ kp, int nC2, int w, int h, double* __restrict__ pw,
              int* __restrict__ stamps) {
  extern __shared__ double wt_s[];
  const int t = blockIdx.x, s = list[t], tid = threadIdx.x, n1 = nC2 + 1;
  if(tid == 0) stamps[t] = cur[s] < count[s] ? s : s | INT_MIN;
  for(int k = tid; k < n1; k += 128) {
    double a = k == nC2 ? 1.0 : 0.0;
    if(k < nC2 && cur[s] < count[s]) {
      int2 c = ssxy[(size_t)s * maxSS + cur[s]];
      a = ipowD(floatNormD(c.x, w), kp[k].x) * ipowD(floatNormD(c.y, h), kp[k].y);
    }
    wt_s[k] = a;
  }
  __syncthreads();
  for(int e = tid; e < n1 * n1; e += 128)
    pw[(size_t)t * n1 * n1 + e] = wt_s[e / n1] * wt_s[e % n1];
}

// ------------------------------------------------------ global matrix ------
// Lower triangle of createMatrix (cd.cl:182-295 == cdkscUtil.cpp:307-402),
// each entry summed over the listed stamps in order, then mirrored, and
// createScProd: kernel terms and the constant term are common to both RHS
// forms, the background terms come from the stamps' dots (bgBase selects the form).
// Every term is a table weight (a product of two spatial weights, of which one
// or both may be the one) times one number of the stamp; multiplying by one is
// exact, so all entries run the same loop, eight stamps' loads ahead of its two
// FP64 instructions (a chain of dependent loads per stamp took 340 us for 256
// stamps and 190 us for the right-hand side; now 138 us for both).
__global__ void __launch_bounds__(256)
    k_build_system(const int* __restrict__ stamps, int nList, const double* __restrict__ Q,
                   const double* __restrict__ B, int qc, const double* __restrict__ pw,
                   const double* __restrict__ dots, int stride, int bgBase, int nC1, int nC2,
                   int nBG, int matSize, int nSol, double* __restrict__ M,
                   double* __restrict__ res) {
  const int ld = matSize + 1, nComp = nC1 * nC2, n1 = nC2 + 1, one = nC2;
  const long long nTri = (long long)matSize * (matSize + 1) / 2;
  for(long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nTri + nSol;
      e += (long long)gridDim.x * blockDim.x) {
    const double* base;  // the stamp's number: base[stamp * stampStride]
    size_t stampStride = stride;
    int wa = one, wb = one, row = 0, col = 0;
    const bool rhs = e >= nTri;
    if(!rhs) {
      // e -> (r, c) with 1 <= c <= r <= matSize
      int r = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
      while((long long)(r + 1) * (r + 2) / 2 <= e) r++;
      while((long long)r * (r + 1) / 2 > e) r--;
      row = r + 1;
      col = (int)(e - (long long)r * (r + 1) / 2) + 1;
      const int ib = row - (nComp + 2);
      if(ib >= 0) {
        if(col > nComp + 1) {
          base = dots + nC1 * nBG + nBG + ib * nBG + (col - (nComp + 2));
        } else if(col == 1) {
          base = dots + nC1 * nBG + ib;
        } else {
          base = dots + ((col - 2) / nC2) * nBG + ib;
          wa = (col - 2) % nC2;
        }
      } else {
        stampStride = (size_t)qc * qc;
        int qi = 1, qj = 1;
        if(row >= 2) {
          qi = (row - 2) / nC2 + 2;
          wa = (row - 2) % nC2;
        }
        if(col >= 2) {
          qj = (col - 2) / nC2 + 2;
          wb = (col - 2) % nC2;
        }
        base = Q + (size_t)qi * qc + qj;
      }
    } else {
      const int id = (int)(e - nTri);
      base = nullptr;
      if(id == 1) {
        base = B + 1;
        stampStride = qc;
      } else if(id >= 2 && id < nComp + 2) {
        base = B + (id - 2) / nC2 + 2;
        stampStride = qc;
        wa = (id - 2) % nC2;
      } else if(id >= nComp + 2 && id < nComp + 2 + nBG) {
        base = dots + bgBase + (id - (nComp + 2));
      }
      if(!base) {
        res[id] = 0.0;
        continue;
      }
    }
    const double* pwe = pw + wa * n1 + wb;
    const size_t pwS = (size_t)n1 * n1;
    double m0 = 0.0;
    int t = 0;
    for(; t + 8 <= nList; t += 8) {
      double v[8], f[8];
#pragma unroll
      for(int u = 0; u < 8; u++) {
        const int s = stamps[t + u];
        v[u] = base[(size_t)(s & INT_MAX) * stampStride];
        f[u] = pwe[(t + u) * pwS];
        if(rhs && s < 0) v[u] = f[u] = 0.0;  // createScProd skips exhausted stamps
      }
#pragma unroll
      for(int u = 0; u < 8; u++) m0 += f[u] * v[u];
    }
    for(; t < nList; t++) {
      const int s = stamps[t];
      if(rhs && s < 0) continue;
      m0 += pwe[t * pwS] * base[(size_t)(s & INT_MAX) * stampStride];
    }
    if(rhs) {
      res[e - nTri] = m0;
    } else {
      M[(size_t)row * ld + col] = m0;
      M[(size_t)col * ld + row] = m0;
    }
  }
  // row 0 / column 0 stay zero
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < ld; i += gridDim.x * blockDim.x) {
    M[i] = 0.0;
    M[(size_t)i * ld] = 0.0;
  }
}

// ------------------------------------------------------ global LU ---------
// CPU ludcmp and the forward half of lubksb (bachUtil.cpp:319-411) on the
// matSize^2 system, distributed over a thread-block cluster: CTA r owns the
// columns j with (j-1) % CL == r in shared memory, the right-hand side being
// column n + 1.  Right-looking elimination gives every entry the same products
// in the same order as the reference's Crout loops, and the right-hand side's
// column the ones of its forward substitution (the rows a leading zero of b
// skips there only subtract zeros here).
//
// Step j: every CTA copies the scaled column j and its pivot row from the
// owner, swaps the pivot rows of its columns and updates them.  The owner of
// column j + 1 updates that column first, finds its pivot and publishes it
// before its other columns, so that chain (two products, the pivot search, a
// reciprocal, one exchange) runs while the others update.  The pivot search
// compares the bits of the nonnegative scaled values: an FP64 compare takes
// as long as a product (62 cycles).  Bound by that chain and by FP64 (a
// product and a subtraction per entry, one warp instruction per 19 cycles per
// SM): 0.77 ms at n = 292 on 16 CTAs; 8 CTAs with the search between the
// exchange and the update took 2.0 ms.
constexpr int GLU_T = 512;
inline size_t gluDoubles(int n, int CL) {
  const size_t ld = n + 1;
  return (size_t)((n + CL) / CL) * ld + 4 * ld + 4;
}

// Larger (value, row) of nonnegative values by their bits; row < 0 never wins.
struct PivotKey {
  long long v;
  int i;
};
__device__ __forceinline__ void pivotMax(PivotKey& a, const PivotKey& b) {
  if(b.v > a.v || (b.v == a.v && b.i > a.i)) a = b;
}
__device__ __forceinline__ PivotKey pivotWarpMax(PivotKey k) {
#pragma unroll
  for(int o = 16; o > 0; o >>= 1) {
    PivotKey b;
    b.v = __shfl_xor_sync(0xffffffffu, k.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, k.i, o);
    pivotMax(k, b);
  }
  return k;
}

template <int CL>
__global__ void __launch_bounds__(GLU_T)
    k_global_lu(double* __restrict__ M, int n, double* __restrict__ b, int* __restrict__ singular) {
  extern __shared__ double glu_s[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int ld = n + 1;
  const int ncol = (n + CL) / CL;               // local columns of the n + 1 (some may be past it)
  double* col = glu_s;                          // ncol * ld (column-major)
  double* vv = col + (size_t)ncol * ld;         // ld
  double* bc = vv + ld;                         // 2 x ld: published columns; entry 0 the pivot row
  double* L = bc + 2 * ld;                      // ld
  __shared__ PivotKey wk[GLU_T / 32];
  __shared__ double sRecip;
  __shared__ int sSing;
  // row scaling (CPU form: a zero row aborts before the elimination)
  if(tid == 0) sSing = 0;
  __syncthreads();
  for(int i = 1 + warp; i <= n; i += GLU_T / 32) {
    long long big = 0;
    for(int j = 1 + lane; j <= n; j += 32) {
      const double t = fabs(M[(size_t)i * ld + j]);
      const long long tb = __double_as_longlong(t);
      if(tb <= 0x7FF0000000000000ll && tb > big) big = tb;  // a NaN is never larger
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {
      const long long t = __shfl_xor_sync(0xffffffffu, big, o);
      if(t > big) big = t;
    }
    if(lane == 0) {
      if(big == 0) sSing = 1;
      vv[i] = 1.0 / __longlong_as_double(big);
    }
  }
  __syncthreads();
  if(sSing) {
    if(rank == 0 && tid == 0) *singular = 1;
    cluster.sync();
    return;
  }
  for(int lc = 0; lc < ncol; lc++) {
    const int j = lc * CL + rank + 1;
    for(int i = tid; i <= n; i += GLU_T)
      col[(size_t)lc * ld + i] = i == 0 || j > n + 1 ? 0.0 : j <= n ? M[(size_t)i * ld + j] : b[i];
  }
  __syncthreads();
  cluster.sync();

  int lastPivot = 0;
  // Pivot of column j (owned here, updated through step j - 1), its scaling
  // and its publication.
  auto publish = [&](int j) {
    double* c = col + (size_t)((j - 1) / CL) * ld;
    double* my = bc + (j & 1) * ld;
    PivotKey k = {-1, -1};
    for(int i = j + tid; i <= n; i += GLU_T) {
      const double v = vv[i] * fabs(c[i]);
      const long long vb = __double_as_longlong(v);
      if(vb >= 0 && vb <= 0x7FF0000000000000ll) pivotMax(k, PivotKey{vb, i});
    }
    k = pivotWarpMax(k);
    if(lane == 0) wk[warp] = k;
    __syncthreads();
    k = wk[lane & (GLU_T / 32 - 1)];
    k = pivotWarpMax(k);
    const int p = k.i >= 0 ? k.i : lastPivot;
    double cj = c[j], d = c[p];
    if(d == 0.0) d = 1.0e-20;
    if(warp == 0) {
      const double r = 1.0 / d;
      if(lane == 0) sRecip = r;
    }
    __syncthreads();
    const double r = sRecip;
    for(int i = j + 1 + tid; i <= n; i += GLU_T) {
      const double l = (i == p ? cj : c[i]) * r;
      c[i] = l;
      my[i] = l;
    }
    if(tid == 0) {
      c[j] = d;
      my[0] = (double)p;
    }
  };
  if(rank == 0) publish(1);
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  for(int j = 1; j <= n; j++) {
    const int owner = (j - 1) % CL, lcj = (j - 1) / CL;
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    const double* src = cluster.map_shared_rank(bc + (j & 1) * ld, owner);
    const int p = (int)src[0];
    lastPivot = p;
    for(int i = j + 1 + tid; i <= n; i += GLU_T) L[i] = src[i];
    const bool ahead = j < n && j % CL == rank;  // this CTA owns column j + 1
    if(!ahead) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if(p != j) {
      for(int lc = tid; lc < ncol; lc += GLU_T) {
        if(rank == owner && lc == lcj) continue;  // swapped by its publication
        double* c = col + (size_t)lc * ld;
        const double t = c[p];
        c[p] = c[j];
        c[j] = t;
      }
      if(tid == 0) vv[p] = vv[j];
    }
    __syncthreads();
    const int lcStart = (j - rank + CL - 1) / CL;  // first lc with lc*CL + rank + 1 > j
    int lcA = lcStart;
    if(ahead) {
      double* c = col + (size_t)lcStart * ld;
      const double cj = c[j];
      for(int i = j + 1 + tid; i <= n; i += GLU_T) c[i] -= L[i] * cj;
      __syncthreads();
      publish(j + 1);
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      lcA++;
    }
    // the other local columns k > j, flattened over (column, row)
    const int lcEnd = min(ncol, (n - rank) / CL + 1);  // columns past n + 1 do not exist
    const int m = n - j, tot = (lcEnd - lcA) * m;
    const float im = 1.f / (float)max(m, 1);
    for(int e = tid; e < tot; e += GLU_T) {
      int q = (int)((float)e * im);
      q -= q * m > e;
      q += (q + 1) * m <= e;
      double* c = col + (size_t)(lcA + q) * ld;
      const int i = j + 1 + e - q * m;
      c[i] -= L[i] * c[j];
    }
    __syncthreads();
  }
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  for(int lc = 0; lc < ncol; lc++) {
    const int j = lc * CL + rank + 1;
    const double* c = col + (size_t)lc * ld;
    if(j <= n)
      for(int i = 1 + tid; i <= j; i += GLU_T) M[(size_t)i * ld + j] = c[i];  // U
    else if(j == n + 1)
      for(int i = 1 + tid; i <= n; i += GLU_T) b[i] = c[i];  // L^-1 P b
  }
  cluster.sync();  // no CTA leaves while another may still read its columns
}

// x / y for the correctly rounded r = 1 / y.  A q within one ulp of the
// quotient has an exact remainder x - q y (one FMA), and RN(q + (x - q y) r) is
// then the correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34,
// 1990).  RN(x r) can be 1.5 ulp off, so one such step brings q there and a
// second one rounds.  Exponents that could over- or underflow take the
// division.
__device__ __forceinline__ double quotient(double x, double y, double r) {
  const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7FF);
  const int ey = (int)((__double_as_longlong(y) >> 52) & 0x7FF);
  if(ex < 400 || ex > 1600 || ey < 700 || ey > 1350) return x / y;
  double q = x * r;
  q = fma(fma(-q, y, x), r, q);
  return fma(fma(-q, y, x), r, q);
}

// Back half of lubksb (bachUtil.cpp:399-409): U x = y, b <- x.  Warp 0 runs each
// row's chain `sum -= a[i][j] * b[j]` in the reference's order and roundings
// while warps 1 and 2 form the next row's products a[i'][j] * b[j] of the b[j]
// already final; the one product that needs the row just finished is formed by
// warp 0.  One barrier per row.  The n^2/2 subtractions of the chains are one
// dependent sequence (every row starts from the unknown before it), 62 cycles
// each: 1.67 ms at n = 292, of which 1.3 ms the chain alone (half of the
// 3.43 ms that one lane took for both halves; warp steps on the integer grid of
// the running sum, as in the stamp statistics, took 3.1 ms: these sums of mixed
// signs leave a binade every two or three terms).
//
// With *singular set (a zero row) the matrix is as built and the reference
// runs lubksb on it with the pivot indices it has, zeros: lane 0 does the same.
constexpr int LUB_THREADS = 96;
constexpr int LUB_PAD = 16;  // terms past n that the chain may read
__global__ void __launch_bounds__(LUB_THREADS)
    k_global_backsub(const double* __restrict__ M, int n, const int* __restrict__ singular,
                     double* __restrict__ b) {
  extern __shared__ double sol_s[];
  const int len = n + LUB_PAD;
  double* bs = sol_s;        // len
  double* pA = bs + len;     // len: products of the current row, zeros past n
  double* pB = pA + len;     // len: products of the next row
  double* dg = pB + len;     // len: diagonal
  double* rd = dg + len;     // len: its reciprocals
  double* sup = rd + len;    // len: entries right of the diagonal
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ld = n + 1;
  for(int i = tid; i <= n; i += LUB_THREADS) {
    bs[i] = b[i];
    dg[i] = i > 0 ? M[(size_t)i * ld + i] : 1.0;
    sup[i] = i > 0 && i < n ? M[(size_t)i * ld + i + 1] : 0.0;
  }
  __syncthreads();
  if(*singular) {
    if(tid == 0) {
      int ii = 0;
      for(int i = 1; i <= n; i++) {
        double sum = bs[0];
        bs[0] = bs[i];
        if(ii != 0)
          for(int j = ii; j < i; j++) sum -= M[(size_t)i * ld + j] * bs[j];
        else if(sum != 0.0)
          ii = i;
        bs[i] = sum;
      }
      for(int i = n; i >= 1; i--) {
        double sum = bs[i];
        for(int j = i + 1; j <= n; j++) sum -= M[(size_t)i * ld + j] * bs[j];
        bs[i] = sum / dg[i];
      }
    }
    __syncthreads();
    for(int i = tid; i <= n; i += LUB_THREADS) b[i] = bs[i];
    return;
  }
  for(int i = tid; i <= n; i += LUB_THREADS) rd[i] = 1.0 / dg[i];
  for(int i = tid; i < len; i += LUB_THREADS) pA[i] = pB[i] = 0.0;
  __syncthreads();
  double* cur = pA;
  double* nxt = pB;
  double x = 0.0;  // warp 0: the row before
  for(int i = n; i >= 1; i--) {
    if(warp == 0) {
      double s = bs[i];
      if(i < n) {
        // terms in fours, the next four loaded meanwhile; subtracting the
        // zeros past n leaves the sum as it is
        const double* c = cur + i + 2;
        double a0 = c[0], a1 = c[1], a2 = c[2], a3 = c[3];
        s -= sup[i] * x;
#pragma unroll 2
        for(int m = n - i - 1; m > 0; m -= 4) {
          c += 4;
          const double b0 = c[0], b1 = c[1], b2 = c[2], b3 = c[3];
          s -= a0;
          s -= a1;
          s -= a2;
          s -= a3;
          a0 = b0;
          a1 = b1;
          a2 = b2;
          a3 = b3;
        }
      }
      x = quotient(s, dg[i], rd[i]);
      if(lane == 0) bs[i] = x;
    } else if(i > 1) {  // row i - 1, columns past i
      const double* row = M + (size_t)(i - 1) * ld;
      constexpr int W = LUB_THREADS - 32;
      int j = i + 1 + tid - 32;
      for(; j + 3 * W <= n; j += 4 * W) {
        double a[4];
#pragma unroll
        for(int u = 0; u < 4; u++) a[u] = row[j + u * W];
#pragma unroll
        for(int u = 0; u < 4; u++) nxt[j + u * W] = a[u] * bs[j + u * W];
      }
      for(; j <= n; j += W) nxt[j] = row[j] * bs[j];
    }
    __syncthreads();
    double* t = cur;
    cur = nxt;
    nxt = t;
  }
  for(int i = tid; i <= n; i += LUB_THREADS) b[i] = bs[i];
}

// ----------------------------------------------------- kernel sums --------
// makeKernelCoeffs + makeKernel + sumKernel (cd.cl:354-442): kernel image at
// (x, y) and its sum; tree=1 sums in 32-wide groups like sumKernel, tree=0
// sequentially like the CPU makeKernel (bachUtil.cpp:532-538).
// One tap per thread, the terms' loads ahead of the ordered sums; the groups of
// the tree sum run side by side (two rounds of taps from dependent loads and
// one lane's serial sum took 40 us; now 23 to 37).
constexpr int KS_THREADS = 512;
__global__ void __launch_bounds__(KS_THREADS)
    k_kernel_sum(const double* __restrict__ sol, const double* __restrict__ vec,
                             int nPSF, int kOrder, int fK, double xf, double yf, int tree,
                             double* __restrict__ out) {
  __shared__ double coeff[MAX_NPSF];
  __shared__ double kern[MAX_FK * MAX_FK + 16];
  __shared__ double part[64];
  const int tid = threadIdx.x, nk = fK * fK;
  const int nC2 = (kOrder + 1) * (kOrder + 2) / 2;
  for(int i = tid; i < nPSF; i += KS_THREADS) {
    double c = 0.0;
    if(i == 0) {
      c = sol[1];
    } else {
      const double* p = sol + 2 + (size_t)(i - 1) * nC2;
      double aX = 1.0;
      for(int x = 0; x <= kOrder; x++) {
        double aY = 1.0;
#pragma unroll 4
        for(int y = 0; y <= kOrder - x; y++) {
          c += *p++ * aX * aY;
          aY *= yf;
        }
        aX *= xf;
      }
    }
    coeff[i] = c;
  }
  __syncthreads();
  for(int p = tid; p < nk; p += KS_THREADS) {
    double k0 = 0.0;
    int q = 0;
    for(; q + 8 <= nPSF; q += 8) {
      double v[8];
#pragma unroll
      for(int u = 0; u < 8; u++) v[u] = vec[(size_t)(q + u) * nk + p];
#pragma unroll
      for(int u = 0; u < 8; u++) k0 += coeff[q + u] * v[u];
    }
    for(; q < nPSF; q++) k0 += coeff[q] * vec[(size_t)q * nk + p];
    kern[p] = k0;
  }
  if(tid < 16) kern[nk + tid] = 0.0;
  __syncthreads();
  if(!tree) {
    if(tid == 0) {
      double s = 0.0;
      for(int p = 0; p < nk; p += 8) {  // the zeros past nk leave the sum as it is
        double v[8];
#pragma unroll
        for(int u = 0; u < 8; u++) v[u] = kern[p + u];
#pragma unroll
        for(int u = 0; u < 8; u++) s += v[u];
      }
      *out = s;
    }
    return;
  }
  for(int count = nk; count > 1;) {
    const int groups = (count + 31) / 32;
    if(tid < groups) {
      double a = 0.0;
      const int lc = min(32, count - tid * 32);
#pragma unroll 8
      for(int l = 0; l < lc; l++) a += kern[tid * 32 + l];
      part[tid] = a;
    }
    __syncthreads();
    if(tid < groups) kern[tid] = part[tid];
    __syncthreads();
    count = groups;
  }
  if(tid == 0) *out = kern[0];
}

// --------------------------------------------------------------- chi^2 ----
// calcSigs (cdkscUtil.cpp:477-583): calcSigBg + getBackground (cd.cl:444-487),
// makeModel (:489-531, FP32 model), calcSig (:533-598) and reduceSig
// (:600-655), one CTA per listed stamp.
constexpr int SIG_THREADS = 256;
template <class T>
__global__ void __launch_bounds__(SIG_THREADS)
    k_sigs(const int* __restrict__ list, const int* __restrict__ count,
           const int* __restrict__ cur, const int2* __restrict__ ssxy, int maxSS,
           const double* __restrict__ W, int wRows, int hSS, int nPSF, int kOrder, int bgOrder,
           int nComp, const double* __restrict__ sol, const T* __restrict__ tImg,
           const T* __restrict__ sImg, uint16_t* __restrict__ mask, int w, int h,
           double invGain, double rn2x2, double* __restrict__ sig) {
  extern __shared__ double sig_s[];
  const int t = blockIdx.x, s = list[t], tid = threadIdx.x;
  const int fSS = 2 * hSS + 1, pix = fSS * fSS, reduceCount = (pix + 31) / 32;
  double* coeff = sig_s;                        // nPSF
  double* term = coeff + nPSF;                  // reduceCount*32
  double* part = term + reduceCount * 32;       // reduceCount
  int* cnt = (int*)(part + reduceCount);        // reduceCount*32
  int* pcnt = cnt + reduceCount * 32;           // reduceCount
  __shared__ double sBg;
  const bool live = cur[s] < count[s];
  int2 c = make_int2(0, 0);
  if(live) c = ssxy[(size_t)s * maxSS + cur[s]];
  const double* Ws = W + (size_t)s * wRows * pix;
  if(live) {
    const double xf = (c.x - w * 0.5) / (w * 0.5), yf = (c.y - h * 0.5) / (h * 0.5);
    const int nC2 = (kOrder + 1) * (kOrder + 2) / 2;
    for(int i = 1 + tid; i < nPSF; i += SIG_THREADS) {
      int k = 2 + (i - 1) * nC2;
      double cc = 0.0, ax = 1.0;
      for(int x = 0; x <= kOrder; x++) {
        double ay = 1.0;
        for(int y = 0; y <= kOrder - x; y++) {
          cc += sol[k++] * ax * ay;
          ay *= yf;
        }
        ax *= xf;
      }
      coeff[i] = cc;
    }
    if(tid == 0) {
      // getBackground with the double normalisation of cd.cl:446-447
      const double bxf = (c.x - 0.5 * w) / (0.5 * w), byf = (c.y - 0.5 * h) / (0.5 * h);
      double bg = 0.0, ax = 1.0;
      int k = nComp + 2;
      for(int i = 0; i <= bgOrder; i++) {
        double ay = 1.0;
        for(int j = 0; j <= bgOrder - i; j++) {
          bg += sol[k++] * ax * ay;
          ay *= byf;
        }
        ax *= bxf;
      }
      sBg = bg;
    }
  }
  __syncthreads();
  const double bg = sBg, sol1 = sol[1];
  for(int gi = tid; gi < reduceCount * 32; gi += SIG_THREADS) {
    const int gx = gi % fSS, gy = gi / fSS;
    double s0 = 0.0;
    int ok = 0;
    if(live && gy < fSS) {
      const int j = gx + gy * fSS;
      // the model accumulates in float (cd.cl:489-531)
      double m0 = roundToFloat(sol1 * Ws[j]);
#pragma unroll 8
      for(int i = 1; i < nPSF; i++) m0 = roundToFloat(m0 + coeff[i] * Ws[(size_t)i * pix + j]);
      const int ax = gx - fSS / 2 + c.x, ay = gy - fSS / 2 + c.y;
      const size_t ai = (size_t)min(max(ax, 0), w - 1) + (size_t)min(max(ay, 0), h - 1) * w;
      const double tD = m0, sD = (double)sImg[ai];
      const double diff = tD - sD + bg;
      if((mask[ai] & BAD_INPUT) == 0 && fabs(sD) > 1e-10) {
        if(isnan(tD) || isnan(sD)) {
          maskOr(mask, ai, NAN_PIXEL);
        } else {
          ok = 1;
          s0 = diff * diff / ((fabs((double)tImg[ai]) + fabs(sD)) * invGain + rn2x2);
        }
      }
    }
    term[gi] = s0;
    cnt[gi] = ok;
  }
  __syncthreads();
  for(int g = tid; g < reduceCount; g += SIG_THREADS) {
    double a = 0.0;
    int k = 0;
    for(int l = 0; l < 32; l++) {
      a += term[g * 32 + l];
      k += cnt[g * 32 + l];
    }
    part[g] = a;
    pcnt[g] = k;
  }
  __syncthreads();
  if(tid == 0) {
    int count_ = reduceCount;
    double result = 0.0;
    bool first = true;
    while(count_ > 1 || first) {
      const int next = (count_ + 31) / 32;
      for(int g = 0; g < next; g++) {
        double a = 0.0;
        int k = 0;
        const int lc = min(32, count_ - g * 32);
        for(int l = 0; l < lc; l++) {
          a += part[g * 32 + l];
          k += pcnt[g * 32 + l];
        }
        if(next == 1) {
          if(k == 0) a = -1.0;
          else {
            a /= k;
            if(a >= 1e10) a = -1.0;
          }
          result = a;
        }
        part[g] = a;
        pcnt[g] = k;
      }
      count_ = next;
      first = false;
    }
    sig[t] = result;
  }
}

// ------------------------------------------------------- cd merit ----------
// removeBadSigs (cd.cl:657-695, ascending order) + sigmaClip (10 iterations)
// + merit = mean / kernelMean, or 666 when nothing survives
// (cdkscUtil.cpp:234-265).
__global__ void __launch_bounds__(256)
    k_cd_merit(const double* __restrict__ sig, int n, const int* __restrict__ liveN,
               const double* __restrict__ kernelMean, double alpha, double* clean, uint8_t* flags,
               double* cs, double* cs2, double* __restrict__ merit) {
  if(liveN) n = *liveN;
  __shared__ int warpTot[8];
  __shared__ int sTotal;
  __shared__ double sMean, sStd;
  __shared__ int sh[4];
  int done = 0;
  for(int base = 0; base < n; base += 256) {
    int i = base + threadIdx.x;
    int keep = (i < n && sig[i] >= 0.0) ? 1 : 0;
    int pos = blockScanExcl(keep, warpTot, &sTotal) + done;
    if(keep) clean[pos] = sig[i];
    done += sTotal;
    __syncthreads();
  }
  if(done == 0) {
    if(threadIdx.x == 0) *merit = 666;
    return;
  }
  blockSigmaClip(clean, done, 10, alpha, flags, cs, cs2, &sMean, &sStd, sh);
  if(threadIdx.x == 0) *merit = sMean / *kernelMean;
}

// ---------------------------------------------------------- ksc check -----
// checkFitSolution (cdkscUtil.cpp:686-770): checkBadSubStamps (ksc.cl:1-49,
// ascending chi^2 list), sigmaClip (10 iterations),
// checkBadSubStampsFromSigmaClip (ksc.cl:51-72) on the stale chi^2 with the
// advanced indices.  The two refills of the reference are merged into one
// list: a stamp advanced in the first pass has chi^2 = -1, which the second
// pass can never reject, and a refill depends only on the new index.
__global__ void __launch_bounds__(256)
    k_ksc_check(const double* __restrict__ sig, int n, const int* __restrict__ liveN,
                const int* __restrict__ count, int* __restrict__ cur, double alpha,
                double sigKernFit, double* chi2, uint8_t* flags, double* cs, double* cs2,
                int* __restrict__ refill,
                int* __restrict__ out /* [0]=nRefill [1]=nPass1 [2]=nPass2 */,
                int* __restrict__ passOf) {
  if(liveN) n = *liveN;
  __shared__ int warpTot[8];
  __shared__ int sTotal;
  __shared__ double sMean, sStd;
  __shared__ int sh[4];
  int done = 0;
  for(int base = 0; base < n; base += 256) {
    int s = base + threadIdx.x;
    int keep = 0;
    if(s < n) {
      passOf[s] = -1;
      if(cur[s] < count[s]) {
        if(sig[s] == -1.0) {
          cur[s] = cur[s] + 1;
          passOf[s] = 0;
        } else {
          keep = 1;
        }
      }
    }
    int pos = blockScanExcl(keep, warpTot, &sTotal) + done;
    if(keep) chi2[pos] = sig[s];
    done += sTotal;
    __syncthreads();
  }
  blockSigmaClip(chi2, done, 10, alpha, flags, cs, cs2, &sMean, &sStd, sh);
  const double m = sMean, sd = sStd;
  int nRef = 0, n1 = 0, n2 = 0;
  for(int base = 0; base < n; base += 256) {
    int s = base + threadIdx.x;
    int inv = 0;
    if(s < n) {
      if(passOf[s] == 0) {
        inv = 1;
        n1++;
      } else if(cur[s] < count[s] && (sig[s] - m) > sigKernFit * sd) {
        cur[s] = cur[s] + 1;
        passOf[s] = 1;
        inv = 1;
        n2++;
      }
    }
    int pos = blockScanExcl(inv, warpTot, &sTotal) + nRef;
    if(inv) refill[pos] = s;
    nRef += sTotal;
    __syncthreads();
  }
  atomicAdd(&out[1], n1);
  atomicAdd(&out[2], n2);
  if(threadIdx.x == 0) out[0] = nRef;
}

__global__ void k_zero_ints(int* p, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i < n) p[i] = 0;
}

}  // namespace

// ========================================================= host side ======

struct FitBuffers {
  int* list;
  double* wts;
  int stride;
  double* M;
  double* rhs;
  int* piv;
  int* singular;
  double* sig;
  double* scratchD;   // clip data copies
  uint8_t* flags;
  double* cs;
  double* cs2;
};

static FitBuffers fitBuffers(xb_ctx* c, int nMax) {
  const Geo& g = c->g;
  FitBuffers f{};
  const int ld = g.matSize + 1;
  f.list = buf<int>(c, laneName(c, "fit_list", "fit_list_side"), std::max(nMax, 1));
  f.wts = buf<double>(c, laneName(c, "fit_wts", "fit_wts_side"), mixedMode(c) ? 1 : (size_t)std::max(nMax, 1) * (g.nComp2 + 1) * (g.nComp2 + 1));
  f.stride = plainDotStride(g);
  f.M = buf<double>(c, laneName(c, "fit_M", "fit_M_side"), (size_t)ld * ld);
  f.rhs = buf<double>(c, laneName(c, "fit_rhs", "fit_rhs_side"), std::max(g.nSol, ld));
  f.piv = buf<int>(c, laneName(c, "fit_piv", "fit_piv_side"), ld);
  f.singular = buf<int>(c, laneName(c, "fit_singular", "fit_singular_side"), 1);
  f.sig = buf<double>(c, laneName(c, "fit_sig", "fit_sig_side"), std::max(nMax, 1));
  f.scratchD = buf<double>(c, laneName(c, "fit_clipdata", "fit_clipdata_side"), std::max(nMax, 1));
  f.flags = buf<uint8_t>(c, laneName(c, "fit_flags", "fit_flags_side"), 2 * std::max(nMax, 1));  // cd clips both sets at once
  f.cs = buf<double>(c, laneName(c, "fit_cs", "fit_cs_side"), 2 * std::max(nMax, 1));
  f.cs2 = buf<double>(c, laneName(c, "fit_cs2", "fit_cs2_side"), 2 * std::max(nMax, 1));
  return f;
}

static int2* kernelPowers(xb_ctx* c) {
  const Geo& g = c->g;
  std::vector<int2> kp(g.nComp2);
  for(int k = 0; k < g.nComp2; k++) kp[k] = make_int2(c->basis.kpX[k], c->basis.kpY[k]);
  int2* d = buf<int2>(c, laneName(c, "kernelPowers", "kernelPowers_side"), g.nComp2);
  toDevice(c, d, kp);
  return d;
}

// matrix + RHS + LU + solve for the stamps list[0..nList) of set si, with
// the other image `other`; cpuRhs selects the ksc RHS form.  liveN, when
// set, holds the live length of the list on the device (nList bounds it).
static void solveGlobal(xb_ctx* c, int si, const FitBuffers& f, const int* list, int nList,
                        const int* liveN, int other, bool cpuRhs, double* dSol) {
  const Geo& g = c->g;
  StampSetDev& S = c->set[si];
  const bool mixed = mixedMode(c);
  const int bgBase = g.nComp1 * g.nBG + g.nBG + g.nBG * g.nBG + (cpuRhs ? g.nBG : 0);
  if(mixed) {  // forms its spatial weights itself; its dots are filled by the Gram kernel
    buildSystemMixed(c, si, list, nList, bgBase, f.M, dSol, liveN);
  } else {
    // xb_cd and xb_ksc take at most this many products per stamp; xb_cmv, whose
    // results can be read by themselves, has no such bound
    constexpr int MAX_PRODUCTS = 1024;
    if(nList > 0 && g.nComp1 * g.nBG + g.nBG + g.nBG * g.nBG > MAX_PRODUCTS)
      throw XbError{XB_ERR_UNSUPPORTED, "too many basis and background terms for the plain fit"};
    const int2* kp = kernelPowers(c);
    const int n1 = g.nComp2 + 1;
    { KT_SCOPE(c, "weights");
    k_weights<<<nList, 128, n1 * sizeof(double), c->stream>>>(
        list, S.count, S.cur, S.ssxy, g.maxSS, kp, g.nComp2, c->w, c->h, f.wts, f.list);
    XB_LAUNCHED(c);
    }
    const long long nEnt = (long long)g.matSize * (g.matSize + 1) / 2 + g.nSol;
    { KT_SCOPE(c, "build_matrix");
    k_build_system<<<(int)std::min<long long>((nEnt + 255) / 256, c->smCount * 8), 256,
                     0, c->stream>>>(f.list, nList, S.Q, S.B, g.qCount, f.wts, S.dots, f.stride,
                                     bgBase, g.nComp1, g.nComp2, g.nBG, g.matSize, g.nSol, f.M,
                                     dSol);
    XB_LAUNCHED(c);
    }
  }
  if(c->trace) {
    const int ld = g.matSize + 1;
    std::string key = cpuRhs ? "ksc_matrix" : ("cd_matrix" + std::to_string(si));
    if(!cpuRhs || !c->arrays.count("ksc_matrix0"))
      c->put(cpuRhs ? "ksc_matrix0" : key, toHost(c, f.M, (size_t)ld * ld));
  }
  // LU on a thread-block cluster
  const int n = g.matSize;
  k_zero_ints<<<1, 32, 0, c->stream>>>(f.singular, 1);
  XB_LAUNCHED(c);
  if(mixed) {
    globalSolveMixed(c, f.M, n, dSol, f.piv, f.singular);
    return;
  }
  // 16 CTAs where the device allows that cluster, else 8 (the same products
  // in the same order either way)
  auto launchLu = [&](auto kernel, int CL) -> cudaError_t {
    cudaError_t e = allowMaxDynamicSmem((const void*)kernel, c->device);
    if(e == cudaSuccess && CL > 8)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if(e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CL);
    cfg.blockDim = dim3(GLU_T);
    cfg.dynamicSmemBytes = gluDoubles(n, CL) * sizeof(double);
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, f.M, n, dSol, f.singular);
  };
  { KT_SCOPE(c, "global_lu");
  if(launchLu(k_global_lu<16>, 16) != cudaSuccess) {
    cudaGetLastError();
    XB_CUDA(launchLu(k_global_lu<8>, 8));
  }
  XB_LAUNCHED(c);
  }
  { KT_SCOPE(c, "global_lubksb");
  k_global_backsub<<<1, LUB_THREADS, (size_t)(6 * (n + LUB_PAD)) * sizeof(double), c->stream>>>(
      f.M, n, f.singular, dSol);
  XB_LAUNCHED(c);
  }
}

static void computeSigs(xb_ctx* c, int si, const int* dList, int nList, const double* dSol,
                        int convImg, double* dSig, const int* liveN = nullptr) {
  if(nList <= 0) return;
  if(mixedMode(c)) {
    sigsMixed(c, si, dList, nList, dSol, convImg, dSig, liveN);
    return;
  }
  const Geo& g = c->g;
  StampSetDev& S = c->set[si];
  const int pix = g.wCols, rc = (pix + 31) / 32;
  const size_t smem = ((size_t)g.nPSF + rc * 32 + rc) * sizeof(double) + (size_t)(rc * 32 + rc) * sizeof(int);
  const int other = 1 - convImg;
  { KT_SCOPE(c, "sigs");
  if(c->imgIsF64)
    k_sigs<double><<<nList, SIG_THREADS, smem, c->stream>>>(
        dList, S.count, S.cur, S.ssxy, g.maxSS, (const double*)S.W, g.wRows, g.hSS, g.nPSF,
        c->p.kernelOrder, c->p.backgroundOrder, g.nComp, dSol, (const double*)c->img[convImg],
        (const double*)c->img[other], c->mask, c->w, c->h, noiseInvGain(c->p),
        noiseRn2x2(c->p), dSig);
  else
    k_sigs<float><<<nList, SIG_THREADS, smem, c->stream>>>(
        dList, S.count, S.cur, S.ssxy, g.maxSS, (const double*)S.W, g.wRows, g.hSS, g.nPSF,
        c->p.kernelOrder, c->p.backgroundOrder, g.nComp, dSol, (const float*)c->img[convImg],
        (const float*)c->img[other], c->mask, c->w, c->h, noiseInvGain(c->p),
        noiseRn2x2(c->p), dSig);
  XB_LAUNCHED(c);
  }
}

void kernelSumLaunch(xb_ctx* c, const double* dSol, double xf, double yf, int tree, double* dOut) {
  { KT_SCOPE(c, "kernel_sum");
  k_kernel_sum<<<1, KS_THREADS, 0, c->stream>>>(dSol, c->dVec, c->g.nPSF, c->p.kernelOrder, c->g.fK, xf, yf,
                                         tree, dOut);
  XB_LAUNCHED(c);
  }
}

// The mixed path's per-stamp test fits (k_stamp_test_fit_ldl), with the
// tuned number of warps (stamps) per CTA among those whose factors fit in
// shared memory (8 warps of a 61-row system do not); systems too large for
// two warps take the one-CTA-per-stamp LU of the plain path.
static void testFitLdl(xb_ctx* c, const CdSets& sets, int qc) {
  int optin = 0;
  XB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const int n = std::max(sets.n[0], sets.n[1]);
  if(qc - 1 > TF_MAXN || tfSmemBytes(qc - 1, 2) > (size_t)optin) {
    const size_t smemLU = ((size_t)qc * qc + 3 * qc) * sizeof(double) + qc * sizeof(int);
    if(smemLU > (size_t)optin) throw XbError{XB_ERR_UNSUPPORTED, "test fit: system too large"};
    XB_CUDA(allowMaxDynamicSmem((const void*)k_stamp_test_fit, c->device));
    k_stamp_test_fit<<<dim3(n, 2), LU_THREADS, smemLU, c->stream>>>(sets, qc);
    XB_LAUNCHED(c);
    return;
  }
  // variants: 0 = 4 warps, 1 = 2 warps, 2 = 8 warps
  const int nVar = tfSmemBytes(qc - 1, 8) <= (size_t)optin ? 3 : 2;
  auto launch = [&](int v) {
    if(v == 0 && tfSmemBytes(qc - 1, 4) > (size_t)optin) v = 1;
    const int W = v == 1 ? 2 : (v == 2 ? 8 : 4);
    const size_t smem = tfSmemBytes(qc - 1, W);
    const dim3 grid((n + W - 1) / W, 2);
    if(W == 2) k_stamp_test_fit_ldl<2><<<grid, 64, smem, c->stream>>>(sets, qc);
    else if(W == 8) k_stamp_test_fit_ldl<8><<<grid, 256, smem, c->stream>>>(sets, qc);
    else k_stamp_test_fit_ldl<4><<<grid, 128, smem, c->stream>>>(sets, qc);
    XB_LAUNCHED(c);
  };
  XB_CUDA(allowMaxDynamicSmem((const void*)k_stamp_test_fit_ldl<2>, c->device));
  XB_CUDA(allowMaxDynamicSmem((const void*)k_stamp_test_fit_ldl<4>, c->device));
  XB_CUDA(allowMaxDynamicSmem((const void*)k_stamp_test_fit_ldl<8>, c->device));
  launch(tunedVariant(c, "stamp_test_fit_ldl", (long long)qc, nVar, launch));
}

// Test fits, clipping and test lists of both sets (cdkscUtil.cpp:44-120); live:
// the kept counts are on the device (frame graphs).
static void cdTestStamps(xb_ctx* c, const FitBuffers& f, int nMax, double* const ks[2],
                         int* const testIdx[2], int* nTest, double* stats, bool live) {
  CdSets sets{};
  for(int si = 0; si < 2; si++) {
    const StampSetDev& S = c->set[si];
    sets.Q[si] = S.Q;
    sets.B[si] = S.B;
    sets.n[si] = S.n;
    sets.liveN[si] = live ? S.dN : nullptr;
    sets.ks[si] = ks[si];
    sets.testIdx[si] = testIdx[si];
  }
  const int qc = c->g.qCount, n = std::max(sets.n[0], sets.n[1]);
  if(n > 0) {
    KT_SCOPE(c, "stamp_test_fit");
    if(mixedMode(c)) {
      testFitLdl(c, sets, qc);
    } else {
      const size_t smemLU = ((size_t)qc * qc + 3 * qc) * sizeof(double) + qc * sizeof(int);
      XB_CUDA(allowMaxDynamicSmem((const void*)k_stamp_test_fit, c->device));
      k_stamp_test_fit<<<dim3(n, 2), LU_THREADS, smemLU, c->stream>>>(sets, qc);
      XB_LAUNCHED(c);
    }
  }
  KT_SCOPE(c, "cd_select");
  k_cd_select<<<2, 256, 0, c->stream>>>(sets, nMax, c->p.sigClipAlpha, c->p.sigKernFit, f.flags,
                                        f.cs, f.cs2, nTest, stats);
  XB_LAUNCHED(c);
}

// What the fits of both sets read and one of them would fill in first.
static void cdTables(xb_ctx* c) {
  if(!mixedMode(c)) return;
  mixedTables(c);
  deviceStatus(c);
}

// The two sets' global test fits are chains of small kernels on a few SMs each
// (the mixed solve takes 16), so they run side by side: one fit's time less
// (0.4 ms of a 2048 x 2048 mixed frame's 5.2, 3.5 ms of a plain 437 x 611 one's
// 16.9).
void stageCd(xb_ctx* c) {
  const Geo& g = c->g;
  const int nMax = std::max(std::max(c->set[0].n, c->set[1].n), 1);
  FitBuffers f = fitBuffers(c, nMax);
  double* ks[2] = {buf<double>(c, "cd_ks0", nMax), buf<double>(c, "cd_ks1", nMax)};
  int* testIdx[2] = {buf<int>(c, "cd_test0", nMax), buf<int>(c, "cd_test1", nMax)};
  int* nTest = buf<int>(c, "cd_ntest", 2);
  double* stats = buf<double>(c, "cd_stats", 4);
  double* dSolCd = buf<double>(c, "cd_sol", 2 * (size_t)std::max(g.nSol, g.matSize + 1));
  double* kMean = buf<double>(c, "cd_kmean", 2);
  double* merit = buf<double>(c, "cd_merit", 2);
  cdTestStamps(c, f, nMax, ks, testIdx, nTest, stats, false);
  std::vector<int> hT = toHost(c, nTest, 2);
  const int solStride = std::max(g.nSol, g.matSize + 1);
  FitBuffers fb[2] = {f, f};
  auto fit = [&](int si) {  // the global test fit of set si up to its merit
    double* sol = dSolCd + (size_t)si * solStride;
    solveGlobal(c, si, fb[si], testIdx[si], hT[si], nullptr, 1 - si, false, sol);
    kernelSumLaunch(c, sol, (0 - 0.5 * c->w) / (0.5 * c->w), (0 - 0.5 * c->h) / (0.5 * c->h), 1,
                    kMean + si);
    computeSigs(c, si, testIdx[si], hT[si], sol, si, fb[si].sig);
    KT_SCOPE(c, "cd_merit");
    k_cd_merit<<<1, 256, 0, c->stream>>>(fb[si].sig, hT[si], nullptr, kMean + si,
                                         c->p.sigClipAlpha, fb[si].scratchD, fb[si].flags, fb[si].cs,
                                         fb[si].cs2, merit + si);
    XB_LAUNCHED(c);
  };
  if(hT[0] > 0 && hT[1] > 0) {
    cdTables(c);
    SideWork side(c);
    side.enter();
    fb[1] = fitBuffers(c, nMax);
    fit(1);
    side.leave();
    fit(0);
    side.join();
  } else {
    for(int si = 0; si < 2; si++)
      if(hT[si] > 0) fit(si);
  }
  for(int si = 0; si < 2; si++) {
    if(c->trace) c->put("kernel_sums" + std::to_string(si), toHost(c, ks[si], c->set[si].n));
    c->merit[si] = hT[si] > 0 ? toHost(c, merit + si, 1)[0] : 666;
    if(c->trace && hT[si] > 0) {
      const std::string sfx = std::to_string(si);
      c->put("cd_test" + sfx, toHost(c, testIdx[si], hT[si]));
      c->put("cd_solution" + sfx, toHost(c, dSolCd + (size_t)si * solStride, g.nSol));
      c->put("cd_sig" + sfx, toHost(c, fb[si].sig, hT[si]));
      c->scalars["cd_kernel_mean" + sfx] = toHost(c, kMean + si, 1)[0];
    }
  }
  if(mixedMode(c)) checkSolveTimeout(c);
  c->convTemplate = c->merit[1] > c->merit[0] ? 1 : 0;
  c->chosen = c->convTemplate ? 0 : 1;
  c->scalars["merit0"] = c->merit[0];
  c->scalars["merit1"] = c->merit[1];
  c->scalars["convTemplate"] = c->convTemplate;
}

void stageKsc(xb_ctx* c) {
  const Geo& g = c->g;
  const int si = c->chosen;
  StampSetDev& S = c->set[si];
  const int n = S.n;
  FitBuffers f = fitBuffers(c, std::max(n, 1));
  std::vector<int> all(std::max(n, 1));
  for(int s = 0; s < n; s++) all[s] = s;
  int* allList = buf<int>(c, "ksc_all", std::max(n, 1));
  toDevice(c, allList, all);
  int* refill = buf<int>(c, "ksc_refill", std::max(n, 1));
  int* passOf = buf<int>(c, "ksc_passof", std::max(n, 1));
  int* outs = buf<int>(c, "ksc_out", 4);
  double* chi2 = buf<double>(c, "ksc_chi2", std::max(n, 1));
  c->dSol = buf<double>(c, "solution", std::max(g.nSol, g.matSize + 1));
  std::vector<int> rejects;
  int iteration = 0;
  long long refills = 0;  // substamps replaced over the loop
  bool check;
  do {
    solveGlobal(c, si, f, allList, n, nullptr, 1 - si, true, c->dSol);
    computeSigs(c, si, allList, n, c->dSol, si, f.sig);
    k_zero_ints<<<1, 32, 0, c->stream>>>(outs, 4);
    XB_LAUNCHED(c);
    { KT_SCOPE(c, "ksc_check");
    k_ksc_check<<<1, 256, 0, c->stream>>>(f.sig, n, nullptr, S.count, S.cur, c->p.sigClipAlpha,
                                          c->p.sigKernFit, chi2, f.flags, f.cs, f.cs2, refill,
                                          outs, passOf);
    XB_LAUNCHED(c);
    }
    std::vector<int> o = toHost(c, outs, 3);
    const int nRefill = o[0];
    refills += nRefill;
    check = nRefill > 0;
    if(c->trace && nRefill > 0) {
      std::vector<int> po = toHost(c, passOf, n);
      for(int pass = 0; pass < 2; pass++)
        for(int s = 0; s < n; s++)
          if(po[s] == pass) rejects.insert(rejects.end(), {iteration, pass, s});
    }
    if(nRefill > 0) fillStamps(c, si, refill, nRefill, si);
    if(c->trace && !check) c->put("ksc_sig_last", toHost(c, f.sig, n));
    iteration++;
    if(iteration > 4 * std::max(n, 1) * g.maxSS + 8)
      throw XbError{XB_ERR_STATE, "ksc did not converge"};  // cannot happen: indices only grow
  } while(check);
  c->kscIterations = iteration;
  c->hSol = toHost(c, c->dSol, g.nSol);
  c->singular = toHost(c, f.singular, 1)[0];
  if(mixedMode(c)) checkSolveTimeout(c);
  c->scalars["ksc_iterations"] = iteration;
  c->scalars["ksc_refills"] = (double)refills;
  c->scalars["singular"] = c->singular;
  if(c->trace) {
    c->put("ksc_rejects", rejects);
    c->put("cur", toHost(c, S.cur, n));
    c->put("solution", c->hSol);
  }
}

// cd as a frame graph captures it: the kept counts and the test-list
// lengths stay on the device (S.n is the stamp-grid bound, S.dN the count);
// each set's global test fit runs in a conditional node when its list is not
// empty, and its merit is 666 otherwise (cdkscUtil.cpp:234-265).
void stageCdGraph(xb_ctx* c, long long lCd[2]) {
  const Geo& g = c->g;
  const int nMax = std::max(std::max(c->set[0].n, c->set[1].n), 1);
  FitBuffers f = fitBuffers(c, nMax);
  double* ks[2] = {buf<double>(c, "cd_ks0", nMax), buf<double>(c, "cd_ks1", nMax)};
  int* testIdx[2] = {buf<int>(c, "cd_test0", nMax), buf<int>(c, "cd_test1", nMax)};
  int* nTest = buf<int>(c, "cd_ntest", 2);
  double* stats = buf<double>(c, "cd_stats", 4);
  double* dSolCd = buf<double>(c, "cd_sol", 2 * (size_t)std::max(g.nSol, g.matSize + 1));
  double* kMean = buf<double>(c, "cd_kmean", 2);
  double* merit = buf<double>(c, "cd_merit", 2);
  cdTestStamps(c, f, nMax, ks, testIdx, nTest, stats, true);
  const int solStride = std::max(g.nSol, g.matSize + 1);
  FitBuffers fb[2] = {f, f};
  auto fit = [&](int si) {
    double* sol = dSolCd + (size_t)si * solStride;
    const int bound = c->set[si].n;
    graphSetDouble(c, merit + si, 666.0);
    lCd[si] = graphIfPositive(c, nTest + si, 1, [&] {
      solveGlobal(c, si, fb[si], testIdx[si], bound, nTest + si, 1 - si, false, sol);
      kernelSumLaunch(c, sol, (0 - 0.5 * c->w) / (0.5 * c->w), (0 - 0.5 * c->h) / (0.5 * c->h), 1,
                      kMean + si);
      computeSigs(c, si, testIdx[si], bound, sol, si, fb[si].sig, nTest + si);
      k_cd_merit<<<1, 256, 0, c->stream>>>(fb[si].sig, bound, nTest + si, kMean + si,
                                           c->p.sigClipAlpha, fb[si].scratchD, fb[si].flags,
                                           fb[si].cs, fb[si].cs2, merit + si);
      XB_LAUNCHED(c);
    });
  };
  cdTables(c);
  SideWork side(c);
  side.enter();
  fb[1] = fitBuffers(c, nMax);
  fit(1);
  side.leave();
  fit(0);
  side.join();
}

// ksc as a frame graph captures it: the reject-and-refit loop is a WHILE
// node; each pass solves, checks, refills the rejected stamps (count on the
// device) and continues while refills were made.
long long stageKscGraph(xb_ctx* c) {
  const Geo& g = c->g;
  const int si = c->chosen;
  StampSetDev& S = c->set[si];
  const int n = std::max(S.n, 1);  // bound; the kept count is *S.dN
  FitBuffers f = fitBuffers(c, n);
  std::vector<int> all(n);
  for(int s = 0; s < n; s++) all[s] = s;
  int* allList = buf<int>(c, "ksc_all", n);
  toDevice(c, allList, all);
  int* refill = buf<int>(c, "ksc_refill", n);
  int* passOf = buf<int>(c, "ksc_passof", n);
  int* outs = buf<int>(c, "ksc_out", 4);
  double* chi2 = buf<double>(c, "ksc_chi2", n);
  c->dSol = buf<double>(c, "solution", std::max(g.nSol, g.matSize + 1));
  k_zero_ints<<<1, 32, 0, c->stream>>>(graphRec(c) + 2, 3);  // iterations, overflow, refills
  XB_LAUNCHED(c);
  const int limit = 4 * n * g.maxSS + 8;
  return graphWhile(c, [&](cudaGraphConditionalHandle h) {
    solveGlobal(c, si, f, allList, n, S.dN, 1 - si, true, c->dSol);
    computeSigs(c, si, allList, n, c->dSol, si, f.sig, S.dN);
    k_zero_ints<<<1, 32, 0, c->stream>>>(outs, 4);
    XB_LAUNCHED(c);
    k_ksc_check<<<1, 256, 0, c->stream>>>(f.sig, n, S.dN, S.count, S.cur, c->p.sigClipAlpha,
                                          c->p.sigKernFit, chi2, f.flags, f.cs, f.cs2, refill,
                                          outs, passOf);
    XB_LAUNCHED(c);
    fillStamps(c, si, refill, n, si, outs);
    graphKscContinue(c, h, outs, limit);
  });
}

}  // namespace xb
