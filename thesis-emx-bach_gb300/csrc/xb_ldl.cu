// xb_ldl.cu — the global normal system of the mixed path: LDL^T factorisation
// and a refined solve on one thread-block cluster.
//
// The global matrix built by createMatrix (src/cdkscUtil.cpp:307-402) is a
// sum of Gram blocks weighted by outer products of the spatial terms, so it
// is symmetric positive semi-definite; the reference solves it with the
// Numerical-Recipes LU with implicit row scaling (src/bachUtil.cpp:319-411).
// The mixed path factors it as L D L^T instead (half the arithmetic, no
// pivot search); a non-positive or non-finite pivot raises a flag and the
// pivoted LU of xb_mixed.cu redoes the system, so singular systems end exactly
// as in the reference.  One step of iterative refinement (FP64 residual of the
// original matrix, corrected with the same factors) follows, which brings the
// rounding of the factorisation back to the accuracy of the residual; the
// correction is added once.

#include <cooperative_groups.h>

#include <atomic>

#include "xb_internal.h"

namespace cg = cooperative_groups;

namespace xb {

namespace {

// Factorisation and refined solve in one cluster launch (below).  Rows are
// dealt cyclically: row i (0-based) lives in CTA i % CL, packed to its lower
// part, so that every panel of 16 columns has its diagonal rows spread evenly
// over the cluster and the trailing work stays balanced.
constexpr int LS_THREADS = 512;
constexpr int LS_BG = 4;          // warps that update while a panel is factored
constexpr int LS_P = 16;          // panel width
constexpr int LS_OWN = 64;         // own rows of a panel step: eight warps of eight
constexpr int LS_SB = LS_P + 2;   // row stride of the exchanged 16-vectors
constexpr int LS_TC = LS_P + 1;   // row stride of the factored diagonal block's columns

struct LsLayout {
  int nP, nPad;        // panels, padded order
  int nr;              // rows per CTA (the right-hand side is one more row of CTA 0)
  size_t rows, y, vec, small;  // doubles of each part of shared memory
  __host__ __device__ size_t doubles() const { return rows + y + vec + small; }
};
__host__ __device__ inline LsLayout lsLayout(int n, int CL) {
  LsLayout l;
  l.nP = (n + LS_P - 1) / LS_P;
  l.nPad = l.nP * LS_P;
  l.nr = l.nPad / CL;  // CL is 8 or 16
  l.rows = (size_t)CL * l.nr * (l.nr + 1) / 2 + l.nPad;
  l.y = (size_t)l.nP * LS_P * LS_P;
  l.vec = (size_t)(5 + LS_P / CL) * l.nPad;
  // kept factors of diagonal blocks, the rows' right-hand sides
  l.small = (size_t)((l.nP + CL - 1) / CL) * LS_P * LS_P + ((l.nr + 1) & ~1);
  return l;
}

// x > 0 and finite by its bits (an FP64 compare costs as much as a product)
__device__ __forceinline__ bool positiveFinite(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b < 0x7FF0000000000000ll;
}

__device__ __forceinline__ void clusterArrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void clusterWait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Barrier 1 over the first warps of a phase (count threads).
__device__ __forceinline__ void barSome(int count) {
  asm volatile("bar.sync 1, %0;" ::"r"(count) : "memory");
}

// M x = rhs by L D L^T and one step of iterative refinement with the FP64
// residual of M, rhs <- x, on one cluster; status[0] bit 0 and rhs untouched
// when a pivot is not positive and finite (the pivoted LU solves it then).
//
// Per panel of 16 columns: every CTA holds the panel's updated diagonal
// block, gathered by remote shared-memory stores, and factors it redundantly
// together with the panel columns of its own rows (four threads per row, four
// columns each in registers; one barrier per column).  A pivot's reciprocal is
// the 20-bit estimate x0 (PTX rcp.approx.ftz.f64) times 1 + e + e^2 with
// e = 1 - d x0, the truncated series of 1/(1 - e): its error is e^3 < 2^-60.
// (A conversion to or from FP32 takes as long as an FP64 product here.)  The
// unscaled panel columns Y = L D go through global memory (each CTA writes its
// rows, reads all): pushing them into 15 CTAs' shared memory took 4.2k cycles
// per panel, the store, barrier and L2 reads ~3.5k.  Then the next panel's
// diagonal rows are updated first and sent, the other rows of its columns
// while that exchange runs, and the rest by LS_BG warps under the next panel's
// factorisation and by all under the exchange after it.  The right-hand side
// rides along as one more row, which is the forward substitution.
//
// The triangular passes exchange one 16-vector per panel: a pass applies the
// inverse of the panel's diagonal block to it and every CTA updates its own
// part.  Partial sums are kept per residue of the row modulo 16, so 8- and
// 16-CTA clusters give the same bits.  No wait depends on anything but the
// hardware cluster barrier.
//
// Bound by FP64: one warp instruction per 19 cycles per SM (62 in a chain), so
// the n^3/6 products alone take 74 us on 16 SMs at n = 292 and the chains of
// the n pivots ~65 us.  Alone on a GB300: 309 us at n = 292 and 1.01 ms at
// n = 587; a column-by-column factorisation followed by block inverses, two
// one-CTA triangular solves and a residual kernel took 640 us and 2.0 ms.
template <int CL>
__global__ void __launch_bounds__(LS_THREADS)
    k_ldl_factor_solve(const double* __restrict__ M, double* __restrict__ rhs, int n,
                       double* __restrict__ Yg, int* __restrict__ status) {
  extern __shared__ __align__(16) double ls_s[];
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int G = LS_P / CL;  // rows of a panel per CTA
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const LsLayout lay = lsLayout(n, CL);
  const int nP = lay.nP, nPad = lay.nPad, nr = lay.nr, ld = n + 1;
  double* A = ls_s;                          // own rows, packed
  double* Y = A + lay.rows;                  // [16][nPad]; later the inverses [nP][16][16]
  double* wv = Y + lay.y;                    // nPad
  double* xg = wv + nPad;                    // nPad
  double* x1 = xg + nPad;                    // nPad
  double* dinv = x1 + nPad;                  // nPad
  double* yv = dinv + nPad;                  // nPad
  double* sPart = yv + nPad;                 // G x nPad
  double* keep = sPart + (size_t)G * nPad;   // slots x 16 x 16: L of diagonal blocks kept here
  double* accv = keep + (size_t)((nP + CL - 1) / CL) * LS_P * LS_P;  // nr: the rows' right-hand sides
  __shared__ __align__(16) double Tg[LS_P * LS_P];      // gathered diagonal block
  __shared__ __align__(16) double Tc[LS_P * LS_TC];     // its column q at step q
  __shared__ __align__(16) double Rq[LS_P];             // reciprocal pivots of the panel
  __shared__ __align__(16) double SB[2 * LS_P * LS_SB]; // exchanged partial sums
  __shared__ __align__(16) double FB[2 * LS_P];         // exchanged right-hand sides
  __shared__ __align__(16) double tv[2 * LS_P];         // own values to send
  __shared__ int sFlag, sNext, sPanel;
  auto rowPtr = [&](int lr) { return A + (size_t)CL * lr * (lr + 1) / 2; };
  double* rhsRow = rowPtr(nr);  // CTA 0

  // own rows (lower part; identity past n) and the right-hand side
  for(int lr = warp; lr < nr; lr += LS_THREADS / 32) {
    const int i = lr * CL + rank;
    double* a = rowPtr(lr);
    for(int j = lane; j < (lr + 1) * CL; j += 32)
      a[j] = (i < n && j <= i) ? M[(size_t)(i + 1) * ld + j + 1] : (i == j ? 1.0 : 0.0);
  }
  if(rank == 0)
    for(int j = tid; j < nPad; j += LS_THREADS) rhsRow[j] = j < n ? rhs[j + 1] : 0.0;
  if(tid == 0) sFlag = sNext = sPanel = 0;
  cluster.sync();  // every CTA runs: its shared memory may be written

  // The G rows of 16 values in `rows` to row g * CL + rank of `dst` (row
  // stride ldd) in every CTA, one 16-byte store per thread.
  auto push = [&](const double* rows, double* dst, int ldd) {
    if(tid >= 128 * CL / 16 * G) return;
    const int k = tid & 7, d = (tid >> 3) % CL, g = (tid >> 3) / CL;
    ((double2*)(cluster.map_shared_rank(dst, d) + (size_t)(g * CL + rank) * ldd))[k] =
        ((const double2*)(rows + g * LS_P))[k];
  };
  // Diagonal rows of panel p, the columns of panel p - 1 applied: group g of
  // 64 threads has row p*16 + g*CL + rank, four threads per column, which
  // split the 16 products.
  auto diagRows = [&](int p) {
    if(tid < 64 * G) {
      const int g = tid >> 6, c = (tid >> 2) & 15, part = tid & 3;
      const int lr = p * G + g, i = lr * CL + rank, j = p * LS_P + c;
      double* a = rowPtr(lr);
      double s = 0.0;
      if(p > 0 && j <= i) {
        const double* l = a + (p - 1) * LS_P + 4 * part;
        const double* y = Y + (size_t)4 * part * nPad + j;
#pragma unroll
        for(int q = 0; q < 4; q++) s = fma(l[q], y[(size_t)q * nPad], s);
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if(part == 0) tv[g * LS_P + c] = j <= i ? a[j] - s : 0.0;
    }
    if(tid < 128) {
      barSome(128);
      push(tv, Tg, LS_P);
    }
  };

  // Columns of panel p applied to one entry of an own row.
  auto update = [&](double* a, int p, int j) {
    double v = a[j];
    const double* l = a + p * LS_P;
    const double* y = Y + j;
#pragma unroll
    for(int q = 0; q < LS_P; q++) v = fma(-l[q], y[(size_t)q * nPad], v);
    a[j] = v;
  };
  // What is left of a panel's trailing update, the columns past the next
  // panel, flattened over (row, column); warps take 32 entries at a time.
  struct Rest {
    int p, lrA, nRow, c0, nTri, tot, j0;
    float b;
    __device__ void set(int p_, int rank, int nr, int nPad) {
      p = p_;
      lrA = (p + 2) * G;
      j0 = (p + 2) * LS_P;
      nRow = nr - lrA;
      c0 = lrA * CL + rank - j0 + 1;  // columns of the first row
      nTri = nRow > 0 ? nRow * c0 + CL * (nRow * (nRow - 1) / 2) : 0;
      tot = p < 0 ? 0 : nTri + (rank == 0 ? nPad - j0 : 0);
      b = (float)c0 - 0.5f * CL;
    }
  } rest;
  rest.set(-1, rank, nr, nPad);
  auto restStep = [&]() -> bool {
    int e = 0;
    if(lane == 0) e = atomicAdd(&sNext, 32);
    e = __shfl_sync(0xffffffffu, e, 0);
    if(e >= rest.tot) return false;
    e += lane;
    if(e < rest.nTri) {
      int t = (int)((sqrtf(rest.b * rest.b + 2.f * CL * (float)e) - rest.b) * (1.f / CL));
      t = max(0, min(t, rest.nRow - 1));
      while(t > 0 && t * rest.c0 + CL * (t * (t - 1) / 2) > e) t--;
      while(t + 1 < rest.nRow && (t + 1) * rest.c0 + CL * ((t + 1) * t / 2) <= e) t++;
      update(rowPtr(rest.lrA + t), rest.p, rest.j0 + e - (t * rest.c0 + CL * (t * (t - 1) / 2)));
    } else if(e < rest.tot) {
      update(rhsRow, rest.p, rest.j0 + e - rest.nTri);
    }
    __syncwarp();
    return true;
  };

  diagRows(0);
  clusterArrive();
  clusterWait();
  for(int p = 0; p < nP; p++) {
    const int K = p * LS_P;
    // ---- the panel: diagonal block (warps 0, 1) and own rows below it
    // (warps 2, 3, 6, 7, ...: the other two schedulers)
    const int lr0 = (p + 1) * G;                          // first own row below the panel
    const int nOwn = nr - lr0 + (rank == 0 ? 1 : 0);      // CTA 0: the right-hand side too
    const int nOwnW = (nOwn + 7) >> 3, nBar = 32 * (3 + nOwnW);
    const bool isT = warp < 2, isR = warp == 4;  // the block; its pivots' reciprocals
    const int ow = (warp >> 2) * 2 + (warp & 1);          // own-row warp index
    __syncthreads();  // the panel's columns are up to date
    if(isT || isR || ((warp & 2) && ow < nOwnW)) {
      const int u = lane & 3;
      const int t = isT ? tid >> 2 : ow * 8 + (lane >> 2);
      const bool live = isT || (!isR && t < nOwn);
      double* a = isT ? nullptr : (lr0 + t < nr ? rowPtr(lr0 + t) : rhsRow) + K;
      double z[4], l[4];
#pragma unroll
      for(int m = 0; m < 4; m++) {
        const int c = 4 * m + u;
        l[m] = 0.0;
        z[m] = isT ? (c <= t ? Tg[t * LS_P + c] : 0.0) : (live ? a[c] : 0.0);
      }
      if(isT && u == 0) Tc[t] = z[0];
      double dl = 0.0, dc[4];  // the block's updates of a step that its chain does not wait for
#pragma unroll
      for(int m = 0; m < 4; m++) dc[m] = 0.0;
#pragma unroll
      for(int q = 0; q < LS_P; q++) {
        barSome(nBar);
        if(isT) {
          if(q > 7 && warp == 0) continue;  // its rows 0..7 are done
          const double* tc = Tc + q * LS_TC;
          const double d = tc[q];
          double x0;
          asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x0) : "d"(d));
          if(q > 0) {  // step q - 1 of the columns beyond q
#pragma unroll
            for(int m = (q >> 2) + 1; m < 4; m++) z[m] = fma(-dl, dc[m], z[m]);
          }
          const double zq = __shfl_sync(0xffffffffu, z[q >> 2], (lane & ~3) | (q & 3));
          const double e = fma(-d, x0, 1.0), v = zq * x0;
          const double lq = fma(v, fma(e, e, e), v);
          if(u == (q & 3)) l[q >> 2] = lq;
          if(q + 1 < LS_P) {
            const int m0 = (q + 1) >> 2;
#pragma unroll
            for(int m = m0; m < 4; m++) dc[m] = tc[4 * m + u];
            if(4 * m0 + u > q) z[m0] = fma(-lq, dc[m0], z[m0]);
            if(u == ((q + 1) & 3)) Tc[(q + 1) * LS_TC + t] = z[m0];
            dl = lq;
          }
        } else if(isR) {
          // the pivot's reciprocal, its check and its copy
          const double d = Tc[q * LS_TC + q];
          double x0;
          asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x0) : "d"(d));
          const double e = fma(-d, x0, 1.0);
          double r = fma(x0, fma(e, e, e), x0);
          if(!positiveFinite(d) || !positiveFinite(r)) {
            if(lane == 0) sFlag = 1;
            r = 0.0;
          }
          if(lane == 0) {
            Rq[q] = r;
            dinv[K + q] = r;
          }
        } else if(q > 0) {
          // own rows run one step behind: the reciprocal of step q - 1 was
          // stored before this step's barrier
          const double* tp = Tc + (q - 1) * LS_TC;
          const double zp = __shfl_sync(0xffffffffu, z[(q - 1) >> 2], (lane & ~3) | ((q - 1) & 3));
          const double lp = zp * Rq[q - 1];
#pragma unroll
          for(int m = q >> 2; m < 4; m++) {
            const int c = 4 * m + u;
            if(c >= q) z[m] = fma(-lp, tp[c], z[m]);
          }
          if(u == ((q - 1) & 3)) l[(q - 1) >> 2] = lp;
        }
      }
      barSome(nBar);
      if(isT) {
        if(p % CL == rank) {
          double* kp = keep + (size_t)(p / CL) * LS_P * LS_P + t * LS_P;
#pragma unroll
          for(int m = 0; m < 4; m++) kp[4 * m + u] = 4 * m + u < t ? l[m] : 0.0;
        }
      } else if(!isR) {
        const double zp = __shfl_sync(0xffffffffu, z[3], lane | 3);
        if(u == 3) l[3] = zp * Rq[LS_P - 1];
        if(live) {
          const int i = (lr0 + t) * CL + rank;
#pragma unroll
          for(int m = 0; m < 4; m++) {
            a[4 * m + u] = l[m];
            if(lr0 + t < nr) Yg[(size_t)(4 * m + u) * nPad + i] = z[m];
          }
        }
      }
    }
    // the other warps: LS_BG of them work on the panel before's update
    // meanwhile, the rest wait
    else if(warp >= LS_THREADS / 32 - LS_BG) {
      while(*(volatile int*)&sPanel <= p && restStep()) {
      }
    }
    if(isR && lane == 0) *(volatile int*)&sPanel = p + 1;
    __syncthreads();
    if(p + 1 == nP) break;
    clusterArrive();
    while(restStep()) {
    }
    __syncthreads();  // Y of the panel before is read
    clusterWait();
    // ---- all rows' Y of this panel into shared memory
    {
      const int j0 = K + LS_P, half = (nPad - j0) / 2, tot = LS_P * half;
      for(int e = tid; e < tot; e += LS_THREADS) {
        const int q = e / half, j = j0 + 2 * (e - q * half);
        *(double2*)(Y + (size_t)q * nPad + j) = __ldcg((const double2*)(Yg + (size_t)q * nPad + j));
      }
    }
    __syncthreads();
    diagRows(p + 1);
    clusterArrive();
    // ---- the next panel's columns of the other own rows
    {
      const int lrA = (p + 2) * G, nRow = nr - lrA + (rank == 0 ? 1 : 0);
      for(int e = tid; e < nRow * LS_P; e += LS_THREADS) {
        const int lr = lrA + (e >> 4);
        update(lr < nr ? rowPtr(lr) : rhsRow, p, K + LS_P + (e & 15));
      }
    }
    rest.set(p + 2 < nP ? p : -1, rank, nr, nPad);
    if(tid == 0) sNext = 0;
    clusterWait();
  }
  __syncthreads();
  if(sFlag) {  // the same in every CTA: the block was factored from the same bits
    if(rank == 0 && tid == 0) atomicOr(status, 1);
    cluster.sync();  // remote stores into this CTA are done
    return;
  }

  // ---- inverses of the unit lower diagonal blocks: CTA p % CL inverts block
  // p by recursive doubling (a 2m block [[A, 0], [C, B]] has the inverse's
  // lower left -B^-1 (C A^-1)), then all CTAs get all of them
  {
    const int slot = tid >> 7, h = tid & 127, nSlot = (nP - rank + CL - 1) / CL;
    for(int s0 = 0; s0 < (nP + CL - 1) / CL; s0 += 4) {
      const bool on = s0 + slot < nSlot;
      double* X = keep + (size_t)(s0 + slot) * LS_P * LS_P;
      if(on && h < LS_P) X[h * LS_P + h] = 1.0;
      __syncthreads();
#pragma unroll
      for(int m = 1; m < LS_P; m *= 2) {
        const int cnt = (LS_P / (2 * m)) * m * m;  // 8, 16, 32, 64
        const int pr = h / (m * m), r = (h / m) % m, cc = h % m, o = pr * 2 * m;
        double acc = 0.0;
        if(on && h < cnt)
          for(int k = cc; k < m; k++)
            acc = fma(X[(o + m + r) * LS_P + o + k], X[(o + k) * LS_P + o + cc], acc);
        __syncthreads();
        if(on && h < cnt) X[(o + m + r) * LS_P + o + cc] = acc;
        __syncthreads();
        acc = 0.0;
        if(on && h < cnt)
          for(int k = 0; k <= r; k++)
            acc = fma(X[(o + m + r) * LS_P + o + m + k], X[(o + m + k) * LS_P + o + cc], acc);
        __syncthreads();
        if(on && h < cnt) X[(o + m + r) * LS_P + o + cc] = -acc;
        __syncthreads();
      }
    }
    for(int e = tid; e < nSlot * 128; e += LS_THREADS)
      __stcg((double2*)(Yg + (size_t)((e >> 7) * CL + rank) * 256) + (e & 127),
             ((const double2*)(keep + (size_t)(e >> 7) * 256))[e & 127]);
    if(rank == 0)  // D^-1 L^-1 rhs: the right-hand side's scaled row
      for(int k = tid; k < nPad; k += LS_THREADS) __stcg(Yg + (size_t)LS_P * nPad + k, rhsRow[k]);
    cluster.sync();
    for(int e = tid; e < nP * 128; e += LS_THREADS) ((double2*)Y)[e] = __ldcg((const double2*)Yg + e);
    for(int k = tid; k < nPad; k += LS_THREADS) wv[k] = __ldcg(Yg + (size_t)LS_P * nPad + k);
    __syncthreads();
  }
  const double* Li = Y;

  // A 16 x 16 product in 128 threads (warps 0-3): out[c] = sum_k m(c, k) v[k],
  // eight threads per c with two terms each.
  auto block16 = [&](auto mat, const double* v) -> double {
    const int c = tid >> 3, k = tid & 7;
    double s = mat(c, k) * v[k];
    s = fma(mat(c, k + 8), v[k + 8], s);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
  };

  // L^T x = wv into xg, panels from the bottom.
  auto backward = [&]() {
    for(int k = tid; k < G * nPad; k += LS_THREADS) sPart[k] = 0.0;
    __syncthreads();
    for(int p = nP - 1; p >= 0; p--) {
      const int K = p * LS_P;
      double* sb = SB + (p & 1) * LS_P * LS_SB;
      // this panel's partial sums, the panel below applied, to every CTA
      if(tid < 128) {
        if(tid < LS_P * G) {
          const int g = tid >> 4, c = tid & 15;
          double v = sPart[g * nPad + K + c];
          if(p + 1 < nP) {
            const int lr = (p + 1) * G + g;
            v = fma(rowPtr(lr)[K + c], xg[lr * CL + rank], v);
          }
          tv[tid] = v;
        }
        barSome(128);
        push(tv, sb, LS_SB);
      }
      clusterArrive();
      if(p + 1 < nP)
        for(int k = tid; k < G * K; k += LS_THREADS) {  // the panels further up
          const int g = G == 1 ? 0 : k / K, j = G == 1 ? k : k - g * K;
          const int lr = (p + 1) * G + g;
          sPart[g * nPad + j] = fma(rowPtr(lr)[j], xg[lr * CL + rank], sPart[g * nPad + j]);
        }
      clusterWait();
      if(tid < 128) {
        const int c = tid >> 3, k = tid & 7;
        double s = sb[k * LS_SB + c] + sb[(k + 8) * LS_SB + c];
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if(k == 0) tv[c] = wv[K + c] - s;
        barSome(128);
        const double* L = Li + (size_t)p * 256;
        const double x = block16([&](int cc, int kk) { return L[kk * LS_P + cc]; }, tv);
        if(k == 0) xg[K + c] = x;
      }
      __syncthreads();
    }
  };
  // L y = (own parts in accv) and wv <- D^-1 y, panels from the top.
  auto forward = [&]() {
    for(int p = 0; p < nP; p++) {
      const int K = p * LS_P;
      double* fb = FB + (p & 1) * LS_P;
      if(tid < CL * G) {
        const int g = tid / CL, d = tid % CL;
        cluster.map_shared_rank(fb, d)[g * CL + rank] = accv[p * G + g];
      }
      clusterArrive();
      clusterWait();
      if(tid < 128) {
        const double* L = Li + (size_t)p * 256;
        const double y = block16([&](int cc, int kk) { return L[cc * LS_P + kk]; }, fb);
        if((tid & 7) == 0) {
          yv[K + (tid >> 3)] = y;
          wv[K + (tid >> 3)] = y * dinv[K + (tid >> 3)];
        }
      }
      __syncthreads();
      // own rows below the panel, eight threads per row
      const int lr0 = (p + 1) * G;
      for(int r0 = lr0; r0 < nr; r0 += LS_THREADS / 8) {
        const int lr = r0 + (tid >> 3), k = tid & 7;
        double s = 0.0;
        if(lr < nr) {
          const double* l = rowPtr(lr) + K;
          s = l[k] * yv[K + k];
          s = fma(l[k + 8], yv[K + k + 8], s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if(lr < nr && k == 0) accv[lr] -= s;
      }
      __syncthreads();
    }
  };

  backward();
  for(int k = tid; k < nPad; k += LS_THREADS) x1[k] = xg[k];
  __syncthreads();
  // residual of the own rows against M, one warp per row
  for(int lr = warp; lr < nr; lr += LS_THREADS / 32) {
    const int i = lr * CL + rank;
    double s = 0.0;
    if(i < n) {
      const double* row = M + (size_t)(i + 1) * ld + 1;
      constexpr int RU = 10;
      for(int j0 = lane; j0 < n; j0 += 32 * RU) {
        double av[RU];
#pragma unroll
        for(int u = 0; u < RU; u++) av[u] = j0 + 32 * u < n ? row[j0 + 32 * u] : 0.0;
#pragma unroll
        for(int u = 0; u < RU; u++)
          if(j0 + 32 * u < n) s = fma(av[u], x1[j0 + 32 * u], s);
      }
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if(lane == 0) accv[lr] = i < n ? rhs[i + 1] - s : 0.0;
  }
  __syncthreads();
  forward();
  backward();
  cluster.sync();  // every CTA has read rhs, and no remote store is pending
  if(rank == 0)
    for(int k = tid; k < n; k += LS_THREADS) rhs[k + 1] = x1[k] + xg[k];
}

template <class Kern, class... Args>
cudaError_t launchCluster(xb_ctx* c, Kern kernel, int CL, int threads, size_t smem,
                          Args... args) {
  cudaError_t e =
      allowMaxDynamicSmem((const void*)kernel, c->device);
  if(e != cudaSuccess) return e;
  if(CL > 8) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if(e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

int* deviceStatus(xb_ctx* c) {
  const bool fresh = c->pool.find("ldl_status") == c->pool.end();
  int* status = buf<int>(c, "ldl_status", 3);
  if(fresh) {
    const int zero[3] = {0, 0, 0};
    if(c->capturing) uploadNow(c, status, zero, sizeof(zero));
    else XB_CUDA(cudaMemsetAsync(status, 0, 3 * sizeof(int), c->stream));
  }
  return status;
}

void globalSolveMixed(xb_ctx* c, const double* M, int n, double* rhs, int* piv, int* singular) {
  const int ld = n + 1;
  int* status = deviceStatus(c) + (c->lane ? 2 : 0);
  XB_CUDA(cudaMemsetAsync(status, 0, sizeof(int), c->stream));
  // 16-CTA clusters where the device allows them and the context asks for
  // them, else 8 (the same bits)
  static std::atomic<int> clusterSize{0};
  {
    KT_SCOPE(c, "global_ldl");
    double* Yg = buf<double>(c, laneName(c, "ldl_y", "ldl_y_side"), (size_t)(LS_P + 1) * lsLayout(n, 16).nPad);
    auto launch = [&](auto kernel, int CL) -> cudaError_t {
      const LsLayout lay = lsLayout(n, CL);
      if(lay.nr + 1 > LS_OWN) return cudaErrorInvalidConfiguration;
      return launchCluster(c, kernel, CL, LS_THREADS, lay.doubles() * sizeof(double), M, rhs, n, Yg,
                           status);
    };
    cudaError_t e = cudaErrorUnknown;
    if(clusterSize.load() != 8 && c->ldlCluster == 16) {
      e = launch(k_ldl_factor_solve<16>, 16);
      if(e == cudaSuccess) clusterSize = 16;
      else cudaGetLastError();
    }
    if(e != cudaSuccess) {
      XB_CUDA(launch(k_ldl_factor_solve<8>, 8));
      if(c->ldlCluster == 16) clusterSize = 8;
    }
    XB_LAUNCHED(c);
  }
  luFallbackSolve(c, M, buf<double>(c, laneName(c, "ldl_F", "ldl_F_side"), (size_t)ld * ld), n, rhs, piv, singular, status);
}

void checkSolveTimeout(xb_ctx* c) {
  auto it = c->pool.find("ldl_status");
  if(it == c->pool.end()) return;
  int st[2] = {0, 0};
  XB_CUDA(cudaMemcpyAsync(st, it->second.p, sizeof(st), cudaMemcpyDeviceToHost, c->stream));
  XB_CUDA(cudaStreamSynchronize(c->stream));
  if(st[1]) {
    XB_CUDA(cudaMemsetAsync((int*)it->second.p + 1, 0, sizeof(int), c->stream));
    throw XbError{XB_ERR_DEVICE_TIMEOUT, "a bounded device-side wait ran out of time"};
  }
}

}  // namespace xb
