// xb_sss.cu — the sss stage: stamp grid, per-stamp statistics, substamp
// search, empty-stamp compaction and the low-threshold retry
// (src/bach.cpp:44-170, src/sssUtil.cpp, src/bachUtil.cpp:130-280,
// cl_kern/sss.cl).
//
// Every quantity that decides a stamp or substamp is computed in the
// reference's operation order (no contraction: the library is built with
// -fmad=false), so the stamp and substamp sets are bit-identical to the CPU
// oracle.  Where the reference compacts with atomics (maskStamp,
// sss.cl:157-188) the order is the ascending pixel index.

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "xb_device.cuh"
#include "xb_internal.h"
#include "xb_osum.cuh"

namespace xb {

namespace {

constexpr int NSAMPLES = 100, PADDED = 128;

__device__ __forceinline__ int satFloorToInt(double v) {
  double f = floor(v);
  if(f != f) return 0;
  if(f >= 2147483647.0) return INT_MAX;
  if(f <= -2147483648.0) return INT_MIN;
  return (int)f;
}

// Numerical Recipes ran1 (cl_kern/sss.cl:52-79): three LCGs with a
// 97-entry shuffle table; 64-bit integer state, exact.
struct Ran1 {
  long long ix1, ix2, ix3;
  int idum, iff;
  __host__ __device__ constexpr void init(int seed) {
    idum = seed;
    iff = 0;
    ix1 = ix2 = ix3 = 0;
  }
  __host__ __device__ constexpr double next(double* r) {
    const long long M1 = 259200, IA1 = 7141, IC1 = 54773;
    const long long M2 = 134456, IA2 = 8121, IC2 = 28411;
    const long long M3 = 243000, IA3 = 4561, IC3 = 51349;
    const double RM1 = 1.0 / 259200, RM2 = 1.0 / 134456;
    if(idum < 0 || iff == 0) {
      iff = 1;
      ix1 = (IC1 - idum) % M1;
      ix1 = (IA1 * ix1 + IC1) % M1;
      ix2 = ix1 % M2;
      ix1 = (IA1 * ix1 + IC1) % M1;
      ix3 = ix1 % M3;
      for(int j = 1; j <= 97; j++) {
        ix1 = (IA1 * ix1 + IC1) % M1;
        ix2 = (IA2 * ix2 + IC2) % M2;
        r[j] = ((double)ix1 + (double)ix2 * RM2) * RM1;
      }
      idum = 1;
    }
    ix1 = (IA1 * ix1 + IC1) % M1;
    ix2 = (IA2 * ix2 + IC2) % M2;
    ix3 = (IA3 * ix3 + IC3) % M3;
    int j = 1 + (int)((97 * ix3) / M3);
    double t = r[j];
    r[j] = ((double)ix1 + (double)ix2 * RM2) * RM1;
    return t;
  }
};

// ------------------------------------------------------- stamp statistics --
// One CTA per stamp: sampleStamp + pad + sortSamples (sss.cl:81-150),
// maskStamp (:157-188), sigmaClip with maxIter 3 (bachUtil.cpp:255-266,
// bach.cl:129-184) and createHistogram (sss.cl:190-324).
//
// Every stamp seeds ran1 with -666, so all stamps draw the same sequence:
// with `draws` (that sequence, precomputed on the host; without it, the
// sequence's first 1024 numbers from a constant table) the 32 candidates of a
// sampling round are formed in parallel; beyond the table one lane runs ran1.
// The clip test |v - m| * inv > alpha is monotone in v on each side of m, so
// each clip round first finds the exact thresholds v_lo < m < v_hi where it
// turns true (a 32-ary search of one warp over the ordered doubles) and then
// compares pixels against them.  The histogram bin floor((v - lbv) / bs) of
// an FP32 pixel comes from an FP32 estimate whose error is bounded per pass;
// only pixels within that bound of a bin edge redo it in FP64.  All decisions
// and sums are those of the reference's order.

// A stamp's slice of the good-pixel scratch: fSW^2 rounded up to a multiple of
// 1024 elements.
__host__ __device__ __forceinline__ size_t statsSlice(int fSW) {
  return ((size_t)fSW * fSW + 1023) & ~(size_t)1023;
}
// Order-preserving map of doubles (no NaN) to 64-bit keys and back.
__device__ __forceinline__ unsigned long long dKey(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double keyD(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
  return __longlong_as_double((long long)b);
}
__device__ __forceinline__ bool clipOut(double v, double m, double inv, double alpha) {
  return fabs(v - m) * inv > alpha;
}

// One warp: the key of the first double (walking away from m, upwards when
// up, downwards otherwise) at which clipOut turns true; `none` when it never
// does.  clipOut is false at m and monotone along the walk.  sd = 1/inv up to
// rounding: the edge is usually among the doubles around m +- alpha sd, which
// the lanes test first.
__device__ unsigned long long clipEdge(double m, double inv, double sd, double alpha, bool up,
                                       bool* none) {
  const int lane = threadIdx.x & 31;
  const unsigned long long kEnd = dKey(up ? INFINITY : -INFINITY);
  unsigned long long lo = dKey(m), hi = kEnd;  // clipOut(lo) false, clipOut(hi) true
  *none = !clipOut(up ? INFINITY : -INFINITY, m, inv, alpha);
  if(*none) return kEnd;
  {
    const unsigned long long k0 = dKey(up ? m + alpha * sd : m - alpha * sd);
    const unsigned long long k = up ? k0 - 16 + lane : k0 + 16 - lane;
    const bool valid = up ? k > lo && k <= hi : k < lo && k >= hi;
    const bool p = valid && clipOut(keyD(k), m, inv, alpha);
    const unsigned bal = __ballot_sync(0xffffffffu, p);
    if(__all_sync(0xffffffffu, valid) && !(bal & 1u) && bal)
      return __shfl_sync(0xffffffffu, k, __ffs(bal) - 1);
  }
  for(int guard = 0; guard < 40; guard++) {
    const unsigned long long span = up ? hi - lo : lo - hi;
    if(span <= 1) break;
    unsigned long long step = span / 33;
    if(step == 0) step = 1;
    const unsigned long long off = (unsigned long long)(lane + 1) * step;
    const bool valid = off < span;
    const unsigned long long k = up ? lo + off : lo - off;
    const bool p = valid && clipOut(keyD(k), m, inv, alpha);
    const unsigned bal = __ballot_sync(0xffffffffu, p);
    const unsigned vmask = __ballot_sync(0xffffffffu, valid);
    if(bal) {
      const int j = __ffs(bal) - 1;
      const unsigned long long kj = __shfl_sync(0xffffffffu, k, j);
      const unsigned long long kprev = __shfl_sync(0xffffffffu, k, j > 0 ? j - 1 : 0);
      hi = kj;
      if(j > 0) lo = kprev;
    } else {
      const int jl = 31 - __clz(vmask);
      lo = __shfl_sync(0xffffffffu, k, jl);
    }
  }
  return hi;
}

// The first draws of ran1(-666), for callers without a table of their own
// (the serial generator takes 110 us for a stamp's usual 256 draws).
constexpr int RAN1_DRAWS = 1024;
struct Ran1Table {
  double v[RAN1_DRAWS];
};
constexpr Ran1Table ran1Table() {
  Ran1Table t{};
  Ran1 rng{};
  double r[98] = {};
  rng.init(-666);
  for(int i = 0; i < RAN1_DRAWS; i++) t.v[i] = rng.next(r);
  return t;
}
__device__ const Ran1Table kRan1 = ran1Table();

// An FP32 good pixel (positive, not NaN, normal or infinite) in FP64, on its
// bits: conversions run on the FP64 unit.
__device__ __forceinline__ double widenGood(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b >> 3) + ((b >= 0x7F800000u ? 1792u : 896u) << 20)), (int)(b << 29));
}
__device__ __forceinline__ double widenGood(double v) { return v; }

// Shared memory of a stamp's chunks: sums, live bits, changed list and (SM)
// the good pixels, 33 words per chunk so that a chunk per lane reads without
// bank conflicts.
constexpr int ST_CHUNKS_SMEM = 1280;  // chunk sums of the other form kept in shared memory
inline size_t statsSmemBytes(int maxChunks, bool sm) {
  if(!sm) return maxChunks <= ST_CHUNKS_SMEM ? (size_t)maxChunks * 16 : 0;
  return (size_t)maxChunks * (16 + 4 + 2) + 4 + (size_t)maxChunks * 33 * 4;
}

// One CTA per stamp: NW warps for the pixels and one that draws and sorts the
// samples meanwhile (they are needed for the histogram only).
//
// SM: the good pixels (FP32) stay in shared memory; else they go to the scratch
// slice.  Bound by FP64, one warp instruction per 19 cycles
// and SM, and by its serial chains: a pixel's part of a chunk's sum of squares
// is one FP64 instruction (an FP32 pixel's square is exact in FP64, so the
// fused multiply-add rounds as the sum does); the plain sums are exact whenever
// the pixels' total fits 53 bits of their common quantum, and then they are
// integers and need no order; only chunks that lost a pixel are summed again.
// Both images, 256 stamps of 107 px: 206 us, 400 of 183 px: 529 us (the
// good pixels and a byte flag each in global memory, four FP64 instructions per
// pixel, the samples first: 662 and 1909 us).
template <class T, bool SM, int NW>
__global__ void __launch_bounds__(NW * 32 + 32, sizeof(T) == 8 ? 2 : 3)
    k_stamp_stats(const T* __restrict__ img, uint16_t* __restrict__ mask,
                  const int4* __restrict__ geom, int w, int h, int fSW,
                  T* __restrict__ good, uint8_t* __restrict__ clip,
                  double* __restrict__ chunkBuf, int maxChunks,
                  double sigClipAlpha, double iqRange, double* __restrict__ skyOut,
                  double* __restrict__ fwhmOut, const double* __restrict__ draws) {
  const int s = blockIdx.x;
  const int4 gm = geom[s];  // cx, cy, sx, sy
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int NT = NW * 32;  // threads on the pixels
  static_assert(F32 || !SM, "the pixels in shared memory are floats");
  // A stamp must have the form of the reference's grid (createStampBounds,
  // cl_kern/sss.cl:19-40): its origin inside the image and its size the full
  // stamp width clipped by the image edge.  Its histogram is then taken over
  // the good pixels of the clipped fSW^2 window (phase D), which are exactly
  // the stamp's pixels.  The grid that xb_sss builds always has this form;
  // geometry passed in from outside (xb_stamp_stats_noalloc) that does not
  // gets NaN statistics and no pixel of it is read (the test is uniform over
  // the CTA, before any barrier).
  if(gm.x < 0 || gm.y < 0 || gm.x >= w || gm.y >= h || gm.z != min(fSW, w - gm.x) ||
     gm.w != min(fSW, h - gm.y)) {
    if(tid == 0) {
      skyOut[s] = __longlong_as_double(0x7ff8000000000000ll);
      fwhmOut[s] = __longlong_as_double(0x7ff8000000000000ll);
    }
    return;
  }
  extern __shared__ __align__(16) unsigned char st_s[];
  __shared__ double samples[PADDED];
  __shared__ double rtab[98];
  __shared__ int cand[32];
  __shared__ int sCount;
  __shared__ int warpGood[2][NW];
  __shared__ unsigned sKMin, sKMax;
  __shared__ unsigned long long sTot;  // exact sum of the unclipped pixels, in quanta
  __shared__ double sMean, sStd, sInv, sSum, sSum2;
  __shared__ int sPrev, sCurr, sClip, sDone, sChanged, sNan;
  __shared__ int bins[256];
  __shared__ int hC[257];         // prefix sums of the bin counts
  __shared__ long long hCE[257];  // and of index * count
  __shared__ double hLower, hUpper, hSky, hBinSize, hLowerBinVal;
  __shared__ int hState;  // 0 continue, 1 stop (setFwhm), 2 stop (no fwhm)
  __shared__ double tLo, tHi;          // clip thresholds of the current round
  __shared__ float fLo, fHi;           // the same, rounded outward to float
  __shared__ int tNoLo, tNoHi, tDirect;
  __shared__ float bLbv, bInv, bDelta;  // FP32 bin estimate of the current pass
  __shared__ int bExact;
  __shared__ double bRec;
  auto pixSync = [] { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); };

  // ---- phase A: random sampling (the last warp) ----
  if(warp == NW) {
    Ran1 rng;
    if(lane == 0) rng.init(-666);
    const int numPix = gm.z * gm.w;
    const double* dr = draws ? draws : kRan1.v;
    const int nDr = draws ? numPix : min(numPix, RAN1_DRAWS / 2);  // candidates with draws
    // the candidates of the first PRE rounds (32 each) are read together
    constexpr int PRE = 4;
    double preV[PRE];
    bool preOk[PRE];
#pragma unroll
    for(int r = 0; r < PRE; r++) {
      preV[r] = 0.0;
      preOk[r] = false;
      if(r * 32 + lane < numPix) {
        const int rx = (int)floor(dr[2 * (r * 32 + lane)] * (int)gm.z);
        const int ry = (int)floor(dr[2 * (r * 32 + lane) + 1] * (int)gm.w);
        const size_t idx = (size_t)(rx + gm.x) + (size_t)(ry + gm.y) * w;
        preV[r] = (double)img[idx];
        preOk[r] = !(mask[idx] > 0 || fabs(preV[r]) <= 1e-10);
      }
    }
    int cnt = 0, iter = 0, drawn = 0;  // drawn: candidates the generator has passed
    while(cnt < NSAMPLES && iter < numPix) {
      const int b = min(32, numPix - iter);
      const int round = iter / 32;
      bool ok = false;
      double v = 0.0;
      if(round < PRE) {
        v = round == 0 ? preV[0] : round == 1 ? preV[1] : round == 2 ? preV[2] : preV[3];
        ok = round == 0 ? preOk[0] : round == 1 ? preOk[1] : round == 2 ? preOk[2] : preOk[3];
      } else {
        size_t idx = 0;
        if(iter + b <= nDr) {
          if(lane < b) {
            const int rx = (int)floor(dr[2 * (iter + lane)] * (int)gm.z);
            const int ry = (int)floor(dr[2 * (iter + lane) + 1] * (int)gm.w);
            idx = (size_t)(rx + gm.x) + (size_t)(ry + gm.y) * w;
          }
        } else {
          // beyond the table: one lane runs the generator
          if(lane == 0) {
            for(; drawn < iter; drawn++) {
              rng.next(rtab);
              rng.next(rtab);
            }
            for(int k = 0; k < b; k++) {
              const int rx = (int)floor(rng.next(rtab) * (int)gm.z);
              const int ry = (int)floor(rng.next(rtab) * (int)gm.w);
              cand[k] = rx | ry << 16;
            }
            drawn = iter + b;
          }
          __syncwarp();
          if(lane < b)
            idx = (size_t)((cand[lane] & 0xFFFF) + gm.x) + (size_t)((cand[lane] >> 16) + gm.y) * w;
        }
        if(lane < b) {
          v = (double)img[idx];
          ok = !(mask[idx] > 0 || fabs(v) <= 1e-10);
        }
      }
      unsigned bal = __ballot_sync(0xffffffffu, ok);
      int pos = cnt + __popc(bal & ((1u << lane) - 1u));
      if(ok && pos < NSAMPLES) samples[pos] = v;
      cnt = min(NSAMPLES, cnt + __popc(bal));
      iter += b;
      __syncwarp();
    }
    if(lane == 0) sCount = cnt;
    __syncwarp();
    for(int i = lane; i < PADDED; i += 32)
      if(i >= cnt) samples[i] = i < NSAMPLES ? 0.0 : INFINITY;
    __syncwarp();
    // bitonic network of the 28 host-launched sortSamples passes
    for(int k = 2; k <= PADDED; k <<= 1)
      for(int j = k >> 1; j > 0; j >>= 1) {
        for(int i = lane; i < PADDED; i += 32) {
          int ixj = i ^ j;
          if(ixj > i) {
            double a = samples[i], c = samples[ixj];
            if((i & k) == 0 && a > c) {
              samples[i] = c;
              samples[ixj] = a;
            } else if((i & k) != 0 && a < c) {
              samples[i] = c;
              samples[ixj] = a;
            }
          }
        }
        __syncwarp();
      }
    __syncthreads();  // meets the pixel warps before phase D
    return;
  }

  // ---- phase B: ordered compaction of good pixels (maskStamp) ----
  // The stamp's pixels go through in ascending order, NT * BB at a time: each
  // warp takes 32 * BB consecutive ones, ballots order them inside the warp
  // and the warps' counts order the warps.  The good pixels are kept as read
  // (FP32 pixels stay FP32).
  // A scratch slice holds them in order; a chunk pass, one chunk per thread, reads
  // its 32 in 16-byte loads, whose lines the L1 keeps for the following ones.
  T* gd = good + (size_t)s * statsSlice(fSW);
  const bool chunksInSmem = SM || maxChunks <= ST_CHUNKS_SMEM;
  double* cS = chunksInSmem ? (double*)st_s : chunkBuf + (size_t)s * 2 * maxChunks;
  double* cS2 = cS + maxChunks;
  unsigned* cm = SM ? (unsigned*)(cS2 + maxChunks)  // a chunk's unclipped pixels
                    : (unsigned*)(clip + (size_t)s * statsSlice(fSW));
  float* list = (float*)(cm + maxChunks);                                   // SM only
  uint16_t* changed = (uint16_t*)(list + (size_t)33 * maxChunks);            // SM only
  const int nPixS = fSW * fSW;
  const unsigned magic = fSW > 1 ? 0xFFFFFFFFu / (unsigned)fSW + 1u : 0u;
  // v <= 1e-10 of the reference: for an FP32 pixel the same test as f <= fTiny,
  // the largest float not above 1e-10
  const float fTiny = __double2float_rd(1e-10);
  auto tiny = [&](T v) -> bool {
    if(F32) return (float)v <= fTiny;
    return (double)v <= 1e-10;
  };
  auto pixelAt = [&](int idxS, size_t* id) -> bool {
    // idxS / fSW: the rounded-up reciprocal gives it or one more
    int y = fSW > 1 ? (int)__umulhi((unsigned)idxS, magic) : idxS;
    if(y * fSW > idxS) y--;
    const int x = idxS - y * fSW;
    *id = (size_t)(x + gm.x) + (size_t)(y + gm.y) * w;
    return idxS < nPixS && x < gm.z && y < gm.w;
  };
  if(tid == 0) {
    sKMin = 0xFFFFFFFFu;
    sKMax = 0u;
    sTot = 0ull;
    sNan = 0;
  }
  constexpr int BB = 8;
  int nGood = 0;
  unsigned kMin = 0xFFFFFFFFu, kMax = 0u;
  bool sawNan = false;
  {
    T px[BB], pn[BB];
    uint16_t mk[BB], mn[BB];
    auto fetch = [&](int base, T* v, uint16_t* m) {
#pragma unroll
      for(int u = 0; u < BB; u++) {
        size_t id;
        const bool in = pixelAt(base + (warp * BB + u) * 32 + lane, &id);
        v[u] = in ? img[id] : T(0);
        m[u] = in ? mask[id] : (uint16_t)1;
      }
    };
    fetch(0, px, mk);
    for(int base = 0, buf = 0; base < nPixS; base += NT * BB, buf ^= 1) {
      if(base + NT * BB < nPixS) fetch(base + NT * BB, pn, mn);
      unsigned bal[BB];
      int cnt = 0;
#pragma unroll
      for(int u = 0; u < BB; u++) {
        const bool cand_ = mk[u] == 0 && !tiny(px[u]);
        const bool g = cand_ && !isnan(px[u]);
        sawNan |= cand_ && !g;
        bal[u] = __ballot_sync(0xffffffffu, g);
        cnt += __popc(bal[u]);
      }
      if(lane == 0) warpGood[buf][warp] = cnt;
      pixSync();
      const int wg = lane < NW ? warpGood[buf][lane] : 0;
      int pos = nGood + __reduce_add_sync(0xffffffffu, lane < warp ? wg : 0);
      nGood += __reduce_add_sync(0xffffffffu, wg);
#pragma unroll
      for(int u = 0; u < BB; u++) {
        if(bal[u] >> lane & 1u) {
          const int q = pos + __popc(bal[u] & ((1u << lane) - 1u));
          if constexpr(SM) list[q + (q >> 5)] = px[u];
          else gd[q] = px[u];
          if constexpr(F32) {
            const unsigned b = __float_as_uint(px[u]);
            kMin = min(kMin, b);
            kMax = max(kMax, b);
          }
        }
        pos += __popc(bal[u]);
      }
#pragma unroll
      for(int u = 0; u < BB; u++) {
        px[u] = pn[u];
        mk[u] = mn[u];
      }
    }
  }
  if(F32) {
    kMin = __reduce_min_sync(0xffffffffu, kMin);
    kMax = __reduce_max_sync(0xffffffffu, kMax);
    if(lane == 0) {
      atomicMin(&sKMin, kMin);
      atomicMax(&sKMax, kMax);
    }
  }
  if(sawNan) sNan = 1;
  pixSync();

  // ---- phase C: sigma clip, maxIter 3 (bachUtil.cpp:34-128) ----
  if(tid == 0) {
    sPrev = nGood;
    sCurr = 0;
    sDone = 0;
    sMean = 0.0;
    sStd = 1e10;
    if(nGood == 0) sDone = 1;
  }
  const int nChunks = (nGood + 31) / 32;
  auto pixel = [&](int c, int l) -> T {
    if constexpr(SM) return list[c * 33 + l];
    else return gd[c * 32 + l];
  };
  // 16 pixels of a chunk from l on (what lies past the list is garbage)
  auto pixels16 = [&](int c, int l, T (&v)[16]) {
    if constexpr(SM) {
#pragma unroll
      for(int k = 0; k < 16; k++) v[k] = list[c * 33 + l + k];
    } else if constexpr(F32) {
#pragma unroll
      for(int k = 0; k < 4; k++) {
        const float4 q = ((const float4*)(gd + c * 32 + l))[k];
        v[4 * k] = q.x;
        v[4 * k + 1] = q.y;
        v[4 * k + 2] = q.z;
        v[4 * k + 3] = q.w;
      }
    } else {
#pragma unroll
      for(int k = 0; k < 8; k++) {
        const double2 q = ((const double2*)(gd + c * 32 + l))[k];
        v[2 * k] = q.x;
        v[2 * k + 1] = q.y;
      }
    }
  };
  // exact clip thresholds for (m, inv) into tLo/tHi (warp 0; all pixel threads call)
  // (warp 0 searches the upper edge, warp 1 the lower one)
  auto thresholds = [&](double m, double inv, double sd) {
    if(warp < 2) {
      const bool direct = !isfinite(m) || isnan(inv);
      if(!direct) {
        bool none;
        const unsigned long long k = clipEdge(m, inv, sd, sigClipAlpha, warp == 0, &none);
        if(lane == 0) {
          const double t = keyD(k);
          if(warp == 0) {
            tHi = t;
            fHi = __double2float_ru(t);  // f >= tHi  <=>  f >= fHi for a float f
            tNoHi = none;
          } else {
            tLo = t;
            fLo = __double2float_rd(t);
            tNoLo = none;
          }
        }
      }
      if(warp == 0 && lane == 0) tDirect = direct;
    }
    pixSync();
  };
  // A pixel against the thresholds (no FP64 operation for FP32 pixels); an
  // absent threshold is NaN, which no pixel passes.
  struct Clip {
    bool direct;
    T lo, hi;
  };
  auto clipNow = [&]() -> Clip {
    const T nan_ = (T)__int_as_float(0x7fffffff);
    if(F32) return {tDirect != 0, tNoLo ? nan_ : (T)fLo, tNoHi ? nan_ : (T)fHi};
    return {tDirect != 0, tNoLo ? nan_ : (T)tLo, tNoHi ? nan_ : (T)tHi};
  };
  // The plain sums as integers: each FP32 good pixel is a multiple of 2^(eMin -
  // 150), eMin the smallest exponent field; while the total stays below 2^53
  // quanta every partial sum of the reference's order is exact.  (Bits beyond
  // 62 of a total are excluded first.)
  const int eMin = (int)(sKMin >> 23), eMax = (int)(sKMax >> 23);
  bool exact = F32 && nGood > 0 && eMin > 0 && eMax < 255 &&
               24 + eMax - eMin + (32 - __clz(nGood)) <= 62;
  auto quanta = [&](float f) -> long long {
    const unsigned b = __float_as_uint(f);
    return (long long)((unsigned long long)((b & 0x7FFFFFu) | 0x800000u) << ((int)(b >> 23) - eMin));
  };
  // Sums of a chunk's unclipped pixels (bits of m) in order, 16 loads issued
  // at a time: squares always, the pixels themselves as the mode says.
  enum { SQUARES, WITH_TOTAL, WITH_SUM };
  long long tot = 0;
  auto chunkSums = [&](int c, unsigned m, auto mode) {
    double a = 0.0, a2 = 0.0;
#pragma unroll
    for(int h0 = 0; h0 < 32; h0 += 16) {
      T v[16];
      pixels16(c, h0, v);
#pragma unroll
      for(int l = 0; l < 16; l++) {
        const bool on = m >> (h0 + l) & 1u;
        const double d = on ? widenGood(v[l]) : 0.0;
        if constexpr(F32) {
          a2 = fma(d, d, a2);
          if constexpr(mode == WITH_TOTAL) tot += on ? quanta(v[l]) : 0ll;
        } else {
          a2 += d * d;
        }
        if constexpr(mode == WITH_SUM) a += d;
      }
    }
    if constexpr(mode == WITH_SUM) cS[c] = a;
    cS2[c] = a2;
  };
  using Squares = std::integral_constant<int, SQUARES>;
  using Total = std::integral_constant<int, WITH_TOTAL>;
  using Sum = std::integral_constant<int, WITH_SUM>;
  auto addTotal = [&](long long t) {  // into sTot, by all pixel threads
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if(lane == 0 && t) atomicAdd(&sTot, (unsigned long long)t);
  };
  auto allOf = [&](int c) -> unsigned {
    const int lc = nGood - c * 32;
    return lc >= 32 ? 0xFFFFFFFFu : (1u << lc) - 1u;
  };
  for(int c = tid; c < nChunks; c += NT) {
    cm[c] = allOf(c);
    if(exact) chunkSums(c, allOf(c), Total());
    else chunkSums(c, allOf(c), Sum());
  }
  if(exact) {
    addTotal(tot);
    pixSync();
    if(sTot >= 1ull << 53) {
      exact = false;
      for(int c = tid; c < nChunks; c += NT) chunkSums(c, allOf(c), Sum());
    }
  }
  pixSync();
  for(int it = 0; it < 3; it++) {
    if(sDone || sCurr == sPrev) break;
    if(sPrev <= 1) {
      if(tid == 0) {
        sMean = 0.0;
        sStd = 1e10;
      }
      break;
    }
    pixSync();
    // the two sequential chunk sums (the reference's serial FP64 loops, bit
    // for bit) on two warps
    if(warp == 0) {
      const double sum2 = osum::warpOrderedSum<2>(cS2, nChunks);
      if(lane == 0) {
        sSum2 = sum2;
        sCurr = sPrev;
      }
    } else if(warp == 1 && !exact) {
      const double sum = osum::warpOrderedSum<2>(cS, nChunks);
      if(lane == 0) sSum = sum;
    }
    pixSync();
    if(tid == 0) {
      const double sum = exact ? (double)(long long)sTot *
                                     __longlong_as_double((long long)(eMin - 150 + 1023) << 52)
                               : sSum;
      const double sum2 = sSum2;
      double n = (double)sCurr;
      double m = sum / n;
      double sd = sqrt((sum2 - n * m * m) / (double)(sCurr - 1));
      sMean = m;
      sStd = sd;
      sInv = 1.0 / sd;
      sClip = 0;
      sChanged = 0;
    }
    pixSync();
    const double m = sMean, inv = sInv;
    thresholds(m, inv, sStd);
    const Clip k = clipNow();
    int myClip = 0;
    tot = 0;
    for(int c = tid; c < nChunks; c += NT) {
      // a chunk none of whose pixels is clipped in this round keeps its sums
      // (the same terms in the same order)
      const unsigned live = cm[c];
      unsigned out = 0;
#pragma unroll
      for(int h0 = 0; h0 < 32; h0 += 16) {
        T v[16];
        pixels16(c, h0, v);
        if(k.direct) {
#pragma unroll
          for(int l = 0; l < 16; l++)
            if(clipOut((double)v[l], m, inv, sigClipAlpha)) out |= 1u << (h0 + l);
        } else {
#pragma unroll
          for(int l = 0; l < 16; l++)
            if(v[l] >= k.hi || v[l] <= k.lo) out |= 1u << (h0 + l);
        }
      }
      out &= live;
      if(out) {
        cm[c] = live & ~out;
        myClip += __popc(out);
        if constexpr(F32)
          if(exact)
            for(unsigned o = out; o; o &= o - 1) tot -= quanta(pixel(c, __ffs(o) - 1));
        if constexpr(SM) {
          changed[atomicAdd(&sChanged, 1)] = (uint16_t)c;
        } else {
          if(exact) chunkSums(c, live & ~out, Squares());
          else chunkSums(c, live & ~out, Sum());
        }
      }
    }
    myClip = __reduce_add_sync(0xffffffffu, myClip);
    if(lane == 0 && myClip) atomicAdd(&sClip, myClip);
    if(exact) addTotal(tot);
    pixSync();
    if(tid == 0) sPrev = sCurr - sClip;
    if constexpr(SM)
      for(int i = tid; i < sChanged; i += NT) {
        const int c = changed[i];
        if(exact) chunkSums(c, cm[c], Squares());
        else chunkSums(c, cm[c], Sum());
      }
    pixSync();
  }
  pixSync();
  const double mean = sMean, invStd = 1.0 / sStd;
  thresholds(mean, invStd, sStd);
  const Clip clipEnd = clipNow();
  __syncthreads();  // the samples are sorted
  // NaN pixels get their mask bits now that the samples have been taken
  if(sNan)
    for(int i = tid; i < nPixS; i += NT) {
      size_t id;
      if(pixelAt(i, &id) && mask[id] == 0 && isnan(img[id])) mask[id] |= NAN_PIXEL | BAD_INPUT;
    }

  // ---- phase D: histogram sky / robust sigma (sss.cl:190-324) ----
  if(tid == 0) {
    int sc = sCount;
    double upS = samples[(int)(0.9 * sc)];
    double midS = samples[(int)(0.5 * sc)];
    hBinSize = (upS - midS) / (double)NSAMPLES;
    hLowerBinVal = midS - (128.0 * hBinSize);
    hLower = hUpper = hSky = 0.0;
    hState = 0;
  }
  pixSync();
  for(int attempts = 0;; attempts++) {
    if(attempts >= 5) {
      if(tid == 0) hState = 2;
      break;
    }
    for(int i = tid; i < 256; i += NT) bins[i] = 0;
    if(tid == 0) {
      // FP32 estimate q' of q = (v - lbv) / bs: |q' - q| <= delta for |q| <= 512
      // (lbv and 1/bs rounded to float, one FP32 rounding each in the
      // subtraction and the product; the FP64 q itself is within 2^-51 |q|)
      const double lbv = hLowerBinVal, bs = hBinSize;
      const double delta = fabs(lbv) / bs * 0x1p-23 + 512.0 * 0x1p-21;
      const bool ok = F32 && bs > 0.0 && isfinite(bs) && isfinite(lbv) && delta < 0.125;
      bExact = ok ? 0 : 1;
      bLbv = (float)lbv;
      bRec = 1.0 / bs;
      bInv = (float)bRec;
      bDelta = (float)delta;
    }
    pixSync();
    const double lbv = hLowerBinVal, bs = hBinSize;
    const bool exactAll = bExact != 0;
    const float fl = bLbv, fi = bInv, half = 0.5f - bDelta;
    const double rbs = bRec;
    // the pixels of createHistogram (mask 0, above 1e-10, not clipped) are
    // the good list of phase B (the kernel changes no other mask bit of the
    // stamp) less the final clip
    constexpr int HB = 8;  // list entries loaded ahead per thread
    for(int base0 = 0; base0 < nGood; base0 += NT * HB) {
      T pvs[HB];
      bool in[HB];
#pragma unroll
      for(int u = 0; u < HB; u++) {
        const int k = base0 + u * NT + tid;
        in[u] = k < nGood;
        if constexpr(SM) pvs[u] = in[u] ? list[k + (k >> 5)] : 0.f;
        else pvs[u] = in[u] ? gd[k] : T(0);
      }
      unsigned rest = 0;  // entries whose bin the FP32 estimate leaves open
#pragma unroll
      for(int u = 0; u < HB; u++) {
        const T pv = pvs[u];
        const bool out = clipEnd.direct ? clipOut((double)pv, mean, invStd, sigClipAlpha)
                                        : pv >= clipEnd.hi || pv <= clipEnd.lo;
        const float q = fminf(fmaxf(((float)pv - fl) * fi, -50.f), 300.f);
        const float f0 = floorf(q), fr = q - f0;
        const bool open = exactAll || (fabsf(fr - 0.5f) >= half && q > -50.f && q < 300.f);
        if(in[u] && !out) {
          if(open) rest |= 1u << u;
          else atomicAdd(&bins[min(max((int)f0 + 1, 0), 255)], 1);
        }
      }
      if(__any_sync(0xffffffffu, rest))
#pragma unroll
        for(int u = 0; u < HB; u++)
          if(rest >> u & 1u) {
            // floor of the quotient from the reciprocal, whose product is within
            // 2^-40 of it below 2^10; at a bin's edge the division decides
            const double v = (double)pvs[u], q = (v - lbv) * rbs, f0 = floor(q);
            int index;
            if(fabs(q) < 1024.0 && fabs(q - f0 - 0.5) < 0.5 - 0x1p-40) {
              index = (int)f0 + 1;
            } else {
              index = satFloorToInt((v - lbv) / bs);
              index = index == INT_MAX ? INT_MAX : index + 1;
            }
            atomicAdd(&bins[min(max(index, 0), 255)], 1);
          }
    }
    pixSync();
    if(warp == 0) {
      const double binSize = hBinSize, lowerBinVal = hLowerBinVal;
      // The reference walks the bins serially (createHistogram,
      // sss.cl:190-324); every quantity it forms is a prefix sum of the
      // counts, so one warp scans the 256 bins once and finds each walk's
      // stopping point by binary search, all of them side by side.
      // The running sums of bin counts (sumBins, sumExpect) are FP64 in the
      // reference but hold integers below 2^53, so they are integers here;
      // S < x for an integer S and a double x is S < ceil(x).
      int c8[8], tc = 0;
      long long e8[8], te = 0;
#pragma unroll
      for(int k = 0; k < 8; k++) {
        const int i = 8 * lane + k;
        tc += bins[i];
        te += (long long)i * bins[i];
        c8[k] = tc;
        e8[k] = te;
      }
      int pc = tc;
      long long pe = te;  // inclusive scan of the lane totals
#pragma unroll
      for(int o = 1; o < 32; o <<= 1) {
        const int uc = __shfl_up_sync(0xffffffffu, pc, o);
        const long long ue = __shfl_up_sync(0xffffffffu, pe, o);
        if(lane >= o) {
          pc += uc;
          pe += ue;
        }
      }
      const int ok = __shfl_sync(0xffffffffu, pc, 31);
      if(ok == 0 || binSize == 0.0) {
        if(lane == 0) hState = 2;
      } else {
#pragma unroll
        for(int k = 0; k < 8; k++) {  // hC[i] = sum of bins[0..i), hCE[i] = sum of j * bins[j]
          hC[8 * lane + k + 1] = pc - tc + c8[k];
          hCE[8 * lane + k + 1] = pe - te + e8[k];
        }
        if(lane == 0) hC[0] = hCE[0] = 0;
        __syncwarp();
        const int tenth = (int)((ok + 9u) / 10u);  // ceil of the FP64 quotient
        // first i in [lo, hi] with hC[i] >= target, hi when none
        auto firstAtLeast = [&](int lo, int hi, unsigned target) {
          while(lo < hi) {
            const int mid = (lo + hi) >> 1;
            if((unsigned)hC[mid] >= target) hi = mid;
            else lo = mid + 1;
          }
          return lo;
        };
        // Densest run of bins holding a tenth of the pixels: the serial
        // window for lower index L ends at U(L) = the first U in [L+1, 255]
        // with hC[U] - hC[L] >= tenth (255 when none; U(L) never decreases,
        // so this is where the two-pointer walk stands), and the walk visits
        // L = 1, 2, ... while the previous window ended below 255, that is
        // while a bin count up to 254 had reached its target.  The
        // reference compares the FP64 quotients S / (U - L); both are integer
        // over integer (sums of counts < 2^31, widths 1..254), and two
        // different such fractions differ by more than 2^-47 relative, so
        // their correctly rounded quotients compare like the fractions:
        // S / D > S' / D'  <=>  S * D' > S' * D, exact in 64-bit integers.
        // The walk keeps the first L of the largest density (strict >), from
        // maxDens = 0.
        int lo[8], hi[8];
        unsigned goal[8];  // counts stay below 2^31
#pragma unroll
        for(int k = 0; k < 8; k++) {
          goal[k] = (unsigned)hC[1 + lane + 32 * k] + tenth;
          lo[k] = 2 + lane + 32 * k;
          hi[k] = 255;
        }
#pragma unroll
        for(int step = 0; step < 8; step++)
#pragma unroll
          for(int k = 0; k < 8; k++) {
            const int mid = (lo[k] + hi[k]) >> 1;
            if(lo[k] < hi[k]) {
              if((unsigned)hC[mid] >= goal[k]) hi[k] = mid;
              else lo[k] = mid + 1;
            }
          }
        long long bN = 0, bD = 1;
        int bL = -1;
#pragma unroll
        for(int k = 0; k < 8; k++) {
          const int L = 1 + lane + 32 * k;
          if(L > 254 || (L > 1 && (unsigned)hC[254] < (unsigned)hC[L - 1] + tenth)) continue;
          const int U = lo[k];
          const long long S = hC[U] - hC[L], D = U - L;
          if(S * bD > bN * D) {
            bN = S;
            bD = D;
            bL = L;
          }
        }
#pragma unroll
        for(int o = 16; o > 0; o >>= 1) {
          const long long oN = __shfl_xor_sync(0xffffffffu, bN, o);
          const long long oD = __shfl_xor_sync(0xffffffffu, bD, o);
          const int oL = __shfl_xor_sync(0xffffffffu, bL, o);
          const long long lhs = oN * bD, rhs = bN * oD;
          if(oL >= 0 && (bL < 0 || lhs > rhs || (lhs == rhs && oL < bL))) {
            bN = oN;
            bD = oD;
            bL = oL;
          }
        }
        // Lane 0: the mode's walk from maxIndex adds bins while below a tenth.
        // Lanes 1 and 2: the quartile walks from bin 0 (hC[256] = ok bounds
        // both, and the upper one ends no earlier than the lower one); a quarter
        // of a count is exact in FP64, so its ceiling is the integer one.
        const int maxIndex = bL < 0 ? 0 : bL;
        const double part = ok * (lane == 2 ? 0.75 : 0.25);
        const int iEnd = lane == 0 ? firstAtLeast(maxIndex + 1, 255, (unsigned)hC[maxIndex] + tenth)
                                   : firstAtLeast(0, 256, (unsigned)(((lane == 2 ? 3ll : 1ll) * ok + 3) / 4));
        const double num = lane == 0 ? (double)(hCE[iEnd] - hCE[maxIndex]) : (double)hC[iEnd] - part;
        const int den = lane == 0 ? hC[iEnd] - hC[maxIndex] : bins[max(iEnd, 1) - 1];
        const double quot = num / (double)den;
        const double value = lane == 0 ? quot + 0.5 : iEnd - quot;
        const double lower = __shfl_sync(0xffffffffu, value, 1);
        const double upper = __shfl_sync(0xffffffffu, value, 2);
        if(lane == 0) {
          const double skyEst = lowerBinVal + binSize * (value - 1.0);
          hSky = skyEst;
          hLower = lower;
          hUpper = upper;
          if(lower < 1.0 || upper > 255.0) {
            hLowerBinVal = lowerBinVal - 128.0 * binSize;
            hBinSize = binSize * 2;
          } else if(upper - lower < 40.0) {
            hBinSize = binSize / 3.0;
            hLowerBinVal = skyEst - 128.0 * hBinSize;
          } else {
            hState = 1;
          }
        }
      }
    }
    pixSync();
    if(hState != 0) break;
  }
  if(tid == 0) {
    fwhmOut[s] = hState == 1 ? hBinSize * (hUpper - hLower) / iqRange : 0.0;
    skyOut[s] = hSky;
  }
}

// Launches the statistics of n stamps.  FP32 stamps of which three fit on an SM
// keep their pixels in shared memory (up to about 119 px on a side); larger ones
// and FP64 images use the scratch, also three CTAs to an SM, which overlap each
// other's serial chains (an image's 390 stamps of 132 px in shared memory, two to an
// SM, 190 us, in the scratch 147; 400 of 183 px, one of 16 warps to an SM, 372
// and 264).  The limit of a block, 227 KB, stands in for an SM's 228 KB.
template <class T>
cudaError_t launchStampStats(const T* img, uint16_t* mask, const int4* geom, int n, int w, int h,
                             int fSW, T* good, uint8_t* clip, double* chunkBuf, double alpha,
                             double iqRange, double* sky, double* fwhm, const double* draws,
                             int device, cudaStream_t stream) {
  const int maxChunks = (int)(((long long)fSW * fSW + 31) / 32);
  int optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if(e != cudaSuccess) return e;
  auto go = [&](auto kernel, int threads, size_t smem) -> cudaError_t {
    if(smem > 32 * 1024) {
      const cudaError_t a = allowMaxDynamicSmem((const void*)kernel, device);
      if(a != cudaSuccess) return a;
    }
    kernel<<<n, threads, smem, stream>>>(img, mask, geom, w, h, fSW, good, clip, chunkBuf, maxChunks,
                                         alpha, iqRange, sky, fwhm, draws);
    return cudaSuccess;
  };
  if constexpr(sizeof(T) == 4) {
    const size_t smem = statsSmemBytes(maxChunks, true), fixed = 8192;  // static and reserved
    if(3 * (smem + fixed) <= (size_t)optin) return go(k_stamp_stats<T, true, 8>, 288, smem);
  }
  return go(k_stamp_stats<T, false, 8>, 288, statsSmemBytes(maxChunks, false));
}

// Mask access shared by the substamp search: volatile 16-bit loads (other
// CTAs of the same launch may set SKIP bits nearby) and a 16-bit OR done as a
// 32-bit atomic on the containing word (the mask buffer has 2 spare entries).
__device__ __forceinline__ uint16_t ldMask(const uint16_t* m, size_t i) {
  return *((volatile const uint16_t*)m + i);
}
__device__ __forceinline__ void orMask(uint16_t* m, size_t i, uint16_t bits) {
  uintptr_t a = (uintptr_t)(m + i);
  unsigned* w32 = (unsigned*)(a & ~(uintptr_t)3);
  unsigned sh = (a & 2) ? 16u : 0u;
  atomicOr(w32, (unsigned)bits << sh);
}

// ---------------------------------------------------------- substamp search --
// One CTA per (stamp, image): findSubStamps (cl_kern/sss.cl:381-505).  The
// reference scans the stamp in raster order, testing each pixel.  Between two
// accepted substamps the mask does not change, so for every pixel of the stamp window
// the reference's local-maximum search (sss.cl:427-459) and window check
// (checkSStamp, :326-361) are tabulated once per mask state:
//   * a separable sliding-window argmax over the qualifying pixels (largest
//     value, ties to the first pixel in raster order: row pass keeps the
//     smallest x, column pass the smallest y), keys compared as the bit
//     patterns of positive doubles;
//   * separable window ORs of "bad", "above kernel-fit threshold" and "above
//     threshold but not positive".
// Each pass then looks for the first candidate in raster order whose window
// passes, in parallel; the scan before it changes nothing, and after an
// acceptance the maps are rebuilt and the scan resumes at the next pixel.
// The accepted substamp's value is the sequential sum of sss.cl:354-357; for
// FP32 input every summand is a float, all partial sums are exact in FP64
// whenever sum|v| < 2^52 * (quantum of the smallest |v|), which is checked,
// and then a parallel sum is the same number.  The reference's writes of the
// bad-pixel bit for pixels above threshHigh (sss.cl:349-352, :417-420,
// :445-448) are unreachable: such pixels carry BAD_INPUT from maskInput
// (ini.cl:29), which every badMask contains, and that test comes first.
constexpr int FM_THREADS = 256;
enum : uint8_t { FL_PRED = 1, FL_NONPOS = 2, FL_KFQ = 4, FL_VPOS = 8 };
enum : uint8_t { OK_BAD = 1, OK_PRED = 2, OK_NONPOS = 4 };


// Bad map and keys of the whole stamp from the mask (the search's start).
template <class T>
__device__ void fmInit(const T* img, const uint16_t* mask, int w, int cx, int cy, int n,
                       uint16_t badMask, const uint8_t* flags, uint8_t* bad,
                       unsigned long long* key) {
  const int N = n * n, tid = threadIdx.x;
  for(int p = tid; p < N; p += FM_THREADS) {
    const int lx = p % n, ly = p / n;
    const size_t a = (size_t)(cx + lx) + (size_t)(cy + ly) * w;
    const uint8_t b = (ldMask(mask, a) & badMask) ? 1 : 0;
    bad[p] = b;
    const uint8_t f = flags[p];
    key[p] = (!b && (f & FL_KFQ) && (f & FL_VPOS))
                 ? (unsigned long long)__double_as_longlong((double)img[a]) : 0ull;
  }
  __syncthreads();
}

// Window maps over the columns [x0, x1] of the rows [k0, k1] (row maps) and
// [r0, r1] (column maps), by block scans (van Herk / Gil-Werman): split the
// line into blocks of the window width W, scan each forwards (prefix) and
// backwards (suffix); the window [a, b] is then suffix(a) with prefix(b) when
// they lie in different blocks, prefix(b) when a starts its block, suffix(a)
// otherwise (b is then the line's end).  Ties keep the smaller index: the
// prefix updates on a larger key, the suffix on a larger or equal one, and
// prefix(b) wins only with a larger key.  16-bit indices for stamps up to 2048
// pixels wide.
__device__ void fmMaps(int n, int sx, int sy, int hSS, const uint8_t* flags, const uint8_t* bad,
                       const unsigned long long* key, unsigned short* hx, uint8_t* rowf, int* arg,
                       uint8_t* okw, unsigned short* tPA, unsigned short* tSA, uint8_t* tPO,
                       uint8_t* tSO, int x0, int x1, int k0, int k1, int r0, int r1) {
  const int tid = threadIdx.x, W = 2 * hSS + 1;
  constexpr unsigned short NONE = 0xFFFF;
  auto orAt = [&](int p) -> uint8_t {
    const uint8_t fl = flags[p];
    return (bad[p] ? OK_BAD : 0) | ((fl & FL_PRED) ? OK_PRED : 0) | ((fl & FL_NONPOS) ? OK_NONPOS : 0);
  };
  const int kw = x1 - x0 + 1;
  {
    const int ba = max(x0 - hSS, 0) / W, bb = min(x1 + hSS, n - 1) / W;
    const int nr = k1 - k0 + 1, nTask = nr * (bb - ba + 1);
    for(int t = tid; t < 2 * nTask; t += FM_THREADS) {
      const bool suffix = t >= nTask;
      const int tt = suffix ? t - nTask : t;
      const int ly = k0 + tt % nr, blk = ba + tt / nr;
      const size_t row = (size_t)ly * n;
      const int b0 = blk * W, b1 = min(b0 + W - 1, n - 1);
      unsigned long long bk = 0;
      unsigned short bi = NONE;
      uint8_t o = 0;
      if(!suffix) {
        for(int x = b0; x <= b1; x++) {
          const unsigned long long k = key[row + x];
          if(k > bk) {
            bk = k;
            bi = (unsigned short)x;
          }
          if(x < sx) o |= orAt((int)(row + x));
          tPA[row + x] = bi;
          tPO[row + x] = o;
        }
      } else {
        for(int x = b1; x >= b0; x--) {
          const unsigned long long k = key[row + x];
          if(k != 0 && k >= bk) {
            bk = k;
            bi = (unsigned short)x;
          }
          if(x < sx) o |= orAt((int)(row + x));
          tSA[row + x] = bi;
          tSO[row + x] = o;
        }
      }
    }
  }
  __syncthreads();
  for(int i = tid; i < (k1 - k0 + 1) * kw; i += FM_THREADS) {
    const int ly = k0 + i / kw, lx = x0 + i % kw;
    const size_t row = (size_t)ly * n;
    const int a = max(lx - hSS, 0), b = min(lx + hSS, n - 1);
    unsigned short h;
    uint8_t o;
    if(a / W != b / W) {
      const unsigned short L = tSA[row + a], R = tPA[row + b];
      h = L == NONE ? R : R == NONE ? L : (key[row + R] > key[row + L] ? R : L);
      o = tSO[row + a] | tPO[row + b];
    } else if(a % W == 0) {
      h = tPA[row + b];
      o = tPO[row + b];
    } else {
      h = tSA[row + a];
      o = tSO[row + a];
    }
    hx[row + lx] = h;
    rowf[row + lx] = o;
  }
  __syncthreads();
  {
    auto candKey = [&](int y, int lx) -> unsigned long long {
      const unsigned short xx = hx[(size_t)y * n + lx];
      return xx == NONE ? 0ull : key[(size_t)y * n + xx];
    };
    const int ba = max(r0 - hSS, 0) / W, bb = min(r1 + hSS, n - 1) / W;
    const int nTask = kw * (bb - ba + 1);
    for(int t = tid; t < 2 * nTask; t += FM_THREADS) {
      const bool suffix = t >= nTask;
      const int tt = suffix ? t - nTask : t;
      const int lx = x0 + tt % kw, blk = ba + tt / kw;
      const int b0 = blk * W, b1 = min(b0 + W - 1, n - 1);
      unsigned long long bk = 0;
      unsigned short bi = NONE;
      uint8_t o = 0;
      if(!suffix) {
        for(int y = b0; y <= b1; y++) {
          const unsigned long long k = candKey(y, lx);
          if(k > bk) {
            bk = k;
            bi = (unsigned short)y;
          }
          if(y < sy) o |= rowf[(size_t)y * n + lx];
          tPA[(size_t)y * n + lx] = bi;
          tPO[(size_t)y * n + lx] = o;
        }
      } else {
        for(int y = b1; y >= b0; y--) {
          const unsigned long long k = candKey(y, lx);
          if(k != 0 && k >= bk) {
            bk = k;
            bi = (unsigned short)y;
          }
          if(y < sy) o |= rowf[(size_t)y * n + lx];
          tSA[(size_t)y * n + lx] = bi;
          tSO[(size_t)y * n + lx] = o;
        }
      }
    }
    __syncthreads();
    for(int i = tid; i < (r1 - r0 + 1) * kw; i += FM_THREADS) {
      const int ly = r0 + i / kw, lx = x0 + i % kw;
      const int a = max(ly - hSS, 0), b = min(ly + hSS, n - 1);
      unsigned short yb;
      uint8_t o;
      if(a / W != b / W) {
        const unsigned short L = tSA[(size_t)a * n + lx], R = tPA[(size_t)b * n + lx];
        yb = L == NONE ? R : R == NONE ? L : (candKey(R, lx) > candKey(L, lx) ? R : L);
        o = tSO[(size_t)a * n + lx] | tPO[(size_t)b * n + lx];
      } else if(a % W == 0) {
        yb = tPA[(size_t)b * n + lx];
        o = tPO[(size_t)b * n + lx];
      } else {
        yb = tSA[(size_t)a * n + lx];
        o = tSO[(size_t)a * n + lx];
      }
      arg[(size_t)ly * n + lx] = yb == NONE ? -1 : yb * n + hx[(size_t)yb * n + lx];
      okw[(size_t)ly * n + lx] = o;
    }
  }
  __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(FM_THREADS)
    k_find_substamps_maps(const T* __restrict__ img0, const T* __restrict__ img1,
                          uint16_t* __restrict__ mask, const int4* __restrict__ geom,
                          const double* __restrict__ sky0, const double* __restrict__ fwhm0,
                          const double* __restrict__ sky1, const double* __restrict__ fwhm1,
                          int2* __restrict__ xy0, double* __restrict__ val0, int* __restrict__ cnt0,
                          int2* __restrict__ xy1, double* __restrict__ val1, int* __restrict__ cnt1,
                          int w, int fSW, int hSS, int maxSS, double tH, double tKF,
                          unsigned char* __restrict__ scratch, size_t perCta, int floatInput) {
  const int s = blockIdx.x, im = blockIdx.y, tid = threadIdx.x;
  const T* img = im == 0 ? img0 : img1;
  const double sky = im == 0 ? sky0[s] : sky1[s];
  const double fwhm = im == 0 ? fwhm0[s] : fwhm1[s];
  int2* xyOut = (im == 0 ? xy0 : xy1) + (size_t)s * maxSS;
  double* valOut = (im == 0 ? val0 : val1) + (size_t)s * maxSS;
  const uint16_t badMask =
      (uint16_t)((MASK_ALL & ~OK_CONV) & ~(im == 0 ? (BAD_PIXEL_S | SKIP_S) : (BAD_PIXEL_T | SKIP_T)));
  const uint16_t skipMask = im == 0 ? SKIP_T : SKIP_S;
  const int4 gm = geom[s];
  const int cx = gm.x, cy = gm.y, sx = gm.z, sy = gm.w, n = fSW, N = n * n;
  const double invFwhm = 1.0 / fwhm;
  unsigned char* base = scratch + (size_t)(im * gridDim.x + s) * perCta;
  unsigned long long* key = (unsigned long long*)base;  // N
  int* arg = (int*)(key + N);                           // N
  unsigned short* hx = (unsigned short*)(arg + N);      // N
  uint8_t* flags = (uint8_t*)(hx + N);                  // N
  uint8_t* bad = flags + N;                             // N
  uint8_t* rowf = bad + N;                              // N
  uint8_t* okw = rowf + N;                              // N
  unsigned short* tPA = (unsigned short*)(okw + N);     // N (block scans of fmMaps)
  unsigned short* tSA = tPA + N;                        // N
  uint8_t* tPO = (uint8_t*)(tSA + N);                   // N
  uint8_t* tSO = tPO + N;                               // N
  __shared__ int2 locXY[MAX_MAXSS];
  __shared__ double locVal[MAX_MAXSS];
  __shared__ int sBest;
  __shared__ double rA[FM_THREADS / 32], rB[FM_THREADS / 32];
  __shared__ double sSum;
  // static flags: checkSStamp predicate, kernel-fit qualification, v > 0
  for(int p = tid; p < N; p += FM_THREADS) {
    const double v = (double)img[(size_t)(cx + p % n) + (size_t)(cy + p / n) * w];
    uint8_t f = 0;
    const bool pr = (v - sky) / fwhm > tKF;
    if(pr) f |= FL_PRED;
    if(pr && !(v > 0.0)) f |= FL_NONPOS;
    if(!((v - sky) * invFwhm < tKF)) f |= FL_KFQ;
    if(v > 0.0) f |= FL_VPOS;
    flags[p] = f;
  }
  __syncthreads();
  fmInit(img, mask, w, cx, cy, n, badMask, flags, bad, key);
  fmMaps(n, sx, sy, hSS, flags, bad, key, hx, rowf, arg, okw, tPA, tSA, tPO, tSO, 0, n - 1, 0,
         n - 1, 0, n - 1);
  const double floorV = sky + tKF * fwhm;
  double dfrac = 0.9;
  int cnt = 0, passes = 0;
  while(cnt < maxSS && passes < 256) {
    passes++;
    const double alt = sky + (tH - sky) * dfrac;
    const double lim = floorV < alt ? alt : floorV;  // OpenCL max()
    int start = 0;
    while(cnt < maxSS && start < N) {
      // first candidate >= start whose window passes (or needs the exact sum)
      int mine = INT_MAX;
      for(int p0 = start; p0 < N && mine == INT_MAX; p0 += 4 * FM_THREADS) {
        for(int k = 0; k < 4; k++) {
          const int p = p0 + k * FM_THREADS + tid;
          if(p >= N || p >= mine) break;
          if(bad[p] || !(flags[p] & FL_KFQ)) continue;
          const double v = (double)img[(size_t)(cx + p % n) + (size_t)(cy + p / n) * w];
          if(!(v > lim)) continue;
          const int m = arg[p] >= 0 ? arg[p] : p;
          const uint8_t o = okw[m];
          if(!(o & OK_BAD) && (o & OK_PRED)) {
            mine = p;
            break;
          }
        }
        mine = __reduce_min_sync(0xffffffffu, mine);
        if(tid == 0) sBest = INT_MAX;
        __syncthreads();
        if((tid & 31) == 0 && mine != INT_MAX) atomicMin(&sBest, mine);
        __syncthreads();
        mine = sBest;
        __syncthreads();
      }
      if(mine == INT_MAX) break;
      const int p = mine, m = arg[p] >= 0 ? arg[p] : p;
      const int mx = cx + m % n, my = cy + m / n;
      const int u0 = max(mx - hSS, cx), v0 = max(my - hSS, cy);
      const int u1 = min(mx + hSS, cx + sx - 1), v1 = min(my + hSS, cy + sy - 1);
      const int uw = u1 - u0 + 1, un = uw * (v1 - v0 + 1);
      // value of the substamp: sum of the thresholded pixels in raster order
      double part = 0.0, amin = INFINITY;
      for(int i = tid; i < un; i += FM_THREADS) {
        const int lx = u0 + i % uw - cx, ly = v0 + i / uw - cy;
        if(flags[ly * n + lx] & FL_PRED) {
          const double v = (double)img[(size_t)(cx + lx) + (size_t)(cy + ly) * w];
          part += v;
          amin = fmin(amin, fabs(v));
        }
      }
#pragma unroll
      for(int o = 16; o > 0; o >>= 1) {
        part += __shfl_down_sync(0xffffffffu, part, o);
        amin = fmin(amin, __shfl_down_sync(0xffffffffu, amin, o));
      }
      if((tid & 31) == 0) {
        rA[tid >> 5] = part;
        rB[tid >> 5] = amin;
      }
      __syncthreads();
      if(tid == 0) {
        double t = 0.0, mn = INFINITY;
        for(int i = 0; i < FM_THREADS / 32; i++) {
          t += rA[i];
          mn = fmin(mn, rB[i]);
        }
        int exact = 0;
        if(floatInput && !(okw[m] & OK_NONPOS) && mn > 0.0 && mn < INFINITY) {
          int e;
          frexp(mn, &e);                           // mn in [2^(e-1), 2^e)
          const double quantum = ldexp(1.0, e - 1 - 23);
          exact = t < ldexp(quantum, 52) ? 1 : 0;  // t = sum|v| here (all v > 0)
        }
        if(!exact) {
          t = 0.0;
          for(int yy = v0; yy <= v1; yy++)
            for(int xx = u0; xx <= u1; xx++)
              if(flags[(yy - cy) * n + (xx - cx)] & FL_PRED) t += (double)img[(size_t)xx + (size_t)yy * w];
        }
        sSum = t;
      }
      __syncthreads();
      const double ret = sSum;
      start = p + 1;
      if(ret == 0.0) continue;
      if(tid == 0) {
        locXY[cnt] = make_int2(mx, my);
        locVal[cnt] = ret;
      }
      cnt++;
      // the window turns bad (its skip bit is part of this image's bad mask,
      // and no other CTA touches this image's bits of the stamp): keys inside
      // it vanish, and only maps within hSS of it can change
      for(int i = tid; i < un; i += FM_THREADS) {
        const int gx = u0 + i % uw, gy = v0 + i / uw;
        orMask(mask, (size_t)gx + (size_t)gy * w, skipMask);
        const size_t q = (size_t)(gx - cx) + (size_t)(gy - cy) * n;
        bad[q] = 1;
        key[q] = 0ull;
      }
      __syncthreads();
      if(cnt < maxSS) {
        const int a0 = u0 - cx, a1 = u1 - cx, b0 = v0 - cy, b1 = v1 - cy;
        fmMaps(n, sx, sy, hSS, flags, bad, key, hx, rowf, arg, okw, tPA, tSA, tPO, tSO,
               max(a0 - hSS, 0), min(a1 + hSS, n - 1), b0, b1, max(b0 - hSS, 0),
               min(b1 + hSS, n - 1));
      }
    }
    if(cnt >= maxSS || lim == floorV) break;
    dfrac -= 0.2;
  }
  __syncthreads();
  if(tid == 0) {
    for(int i = 1; i < cnt; i++)
      for(int j = i; j > 0 && locVal[j - 1] < locVal[j]; j--) {
        int2 t = locXY[j - 1];
        locXY[j - 1] = locXY[j];
        locXY[j] = t;
        double tv = locVal[j - 1];
        locVal[j - 1] = locVal[j];
        locVal[j] = tv;
      }
    for(int i = 0; i < maxSS; i++) {
      xyOut[i] = i < cnt ? locXY[i] : make_int2(INT_MAX, INT_MAX);
      valOut[i] = i < cnt ? locVal[i] : -INFINITY;
    }
    (im == 0 ? cnt0 : cnt1)[s] = min(cnt, maxSS / 2);
  }
}

// ------------------------------------------- substamp search in shared memory --
// The decisions of k_find_substamps_maps for FP32 images, with the stamp in
// shared memory at 6.4 bytes per pixel (pixel, flags, row winner, two bit
// maps), so that stamps up to 190 px fit and two 107-px ones share an SM:
//   * a candidate's window maximum (the largest key, ties to the first in
//     raster order) is found when the scan reaches the candidate, by one thread
//     from the window rows' winners (hx, the maximum over the 2 hSS + 1 columns
//     around the candidate's);
//   * the window conditions "holds a bad pixel" and "holds a pixel above the
//     stamp's threshold" are bit maps dilated by the window, so a lookup each;
//     an acceptance turns its window bad, which ORs one rectangle into the
//     first and can change hx only in the window's rows within hSS of it in x.
// Keys are the float bit patterns (ordered like the doubles of the reference
// for positive values); the two static predicates (v - sky) / fwhm > tKF and
// !((v - sky) * (1/fwhm) < tKF), monotone in v, become compares against their
// exact thresholds, found once per stamp by a warp search over the ordered
// doubles; so does the pass threshold v > lim.
// A pass lists its candidates in raster order, 2048 at a time (512 in the largest
// stamps); a thread takes one, and the first that passes is the next substamp.
// Two-dimensional maps of the winners and conditions by block scans, rebuilt
// around every acceptance (15 bytes per pixel, one CTA per SM, stamps above
// 123 px from global memory), took 0.55 ms for 2 x 256 stamps of 107 px and
// 3.77 ms for 2 x 400 of 183; these forms with a warp per candidate, a load at a
// time and the thresholds searched over all doubles 0.38 and 0.88 ms; now 0.20
// and 0.53 ms.
constexpr int FS_T = 512;
constexpr uint8_t FS_BAD = 0x80;  // in the flags byte
constexpr int FS_MAXN = 255;      // row winners are bytes, 0xFF none
constexpr int FS_SEG = 8;         // columns per task of the row winners
constexpr int FS_LIST = 2048;     // candidates listed at a time, FS_T where more do not fit

// One warp: smallest key in (lo, hi] at which pred turns true, given
// pred(lo) false and pred(hi) true (pred monotone between them).
// The key is usually among the doubles around `guess`, which the lanes test
// first.
template <class P>
__device__ unsigned long long warpFirstTrue(unsigned long long lo, unsigned long long hi,
                                            double guess, P pred) {
  const int lane = threadIdx.x & 31;
  if(isfinite(guess)) {
    const unsigned long long k = dKey(guess) - 16 + lane;
    const bool valid = k > lo && k <= hi;
    const unsigned bal = __ballot_sync(0xffffffffu, valid && pred(keyD(k)));
    if(__all_sync(0xffffffffu, valid) && !(bal & 1u) && bal)
      return __shfl_sync(0xffffffffu, k, __ffs(bal) - 1);
  }
  for(int guard = 0; guard < 40; guard++) {
    const unsigned long long span = hi - lo;
    if(span <= 1) break;
    unsigned long long step = span / 33;
    if(step == 0) step = 1;
    const unsigned long long off = (unsigned long long)(lane + 1) * step;
    const bool valid = off < span;
    const unsigned long long k = lo + off;
    const bool t = valid && pred(keyD(k));
    const unsigned bal = __ballot_sync(0xffffffffu, t);
    const unsigned vmask = __ballot_sync(0xffffffffu, valid);
    if(bal) {
      const int j = __ffs(bal) - 1;
      const unsigned long long kj = __shfl_sync(0xffffffffu, k, j);
      const unsigned long long kp = __shfl_sync(0xffffffffu, k, j > 0 ? j - 1 : 0);
      hi = kj;
      if(j > 0) lo = kp;
    } else {
      lo = __shfl_sync(0xffffffffu, k, 31 - __clz(vmask));
    }
  }
  return hi;
}

inline int fsWords(int n) { return (n + 31) / 32; }
size_t fsSmemBytes(int n) {
  return (((size_t)n * n * 6 + 3) & ~(size_t)3) + (size_t)3 * n * fsWords(n) * 4;
}

// Dilation of bit rows by r columns each way, in place, one thread per row
// (at most 8 words, r < 64).
__device__ void dilateRow(uint32_t* row, int nw, int r) {
  uint32_t up[8], dn[8];
#pragma unroll
  for(int j = 0; j < 8; j++) up[j] = dn[j] = j < nw ? row[j] : 0u;
  for(int len = 1; len < r + 1;) {
    const int sh = min(min(len, r + 1 - len), 31);
#pragma unroll
    for(int j = 7; j >= 0; j--) up[j] |= (up[j] << sh) | (j > 0 ? up[j - 1] >> (32 - sh) : 0u);
#pragma unroll
    for(int j = 0; j < 8; j++) dn[j] |= (dn[j] >> sh) | (j < 7 ? dn[j + 1] << (32 - sh) : 0u);
    len += sh;
  }
#pragma unroll
  for(int j = 0; j < 8; j++)
    if(j < nw) row[j] = up[j] | dn[j];
}

__global__ void __launch_bounds__(FS_T, 2)
    k_find_substamps_sm(const float* __restrict__ img0, const float* __restrict__ img1,
                        uint16_t* __restrict__ mask, const int4* __restrict__ geom,
                        const double* __restrict__ sky0, const double* __restrict__ fwhm0,
                        const double* __restrict__ sky1, const double* __restrict__ fwhm1,
                        int2* __restrict__ xy0, double* __restrict__ val0, int* __restrict__ cnt0,
                        int2* __restrict__ xy1, double* __restrict__ val1, int* __restrict__ cnt1,
                        int w, int fSW, int hSS, int maxSS, double tH, double tKF, int cap) {
  extern __shared__ __align__(16) unsigned char fs_s[];
  const int s = blockIdx.x, im = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = FS_T / 32;
  const float* img = im == 0 ? img0 : img1;
  const double sky = im == 0 ? sky0[s] : sky1[s];
  const double fwhm = im == 0 ? fwhm0[s] : fwhm1[s];
  int2* xyOut = (im == 0 ? xy0 : xy1) + (size_t)s * maxSS;
  double* valOut = (im == 0 ? val0 : val1) + (size_t)s * maxSS;
  const uint16_t badMask =
      (uint16_t)((MASK_ALL & ~OK_CONV) & ~(im == 0 ? (BAD_PIXEL_S | SKIP_S) : (BAD_PIXEL_T | SKIP_T)));
  const uint16_t skipMask = im == 0 ? SKIP_T : SKIP_S;
  const int4 gm = geom[s];
  const int cx = gm.x, cy = gm.y, sx = gm.z, sy = gm.w, n = fSW, N = n * n, nw = (n + 31) / 32;
  const double invFwhm = 1.0 / fwhm;
  float* V = (float*)fs_s;                 // N pixel values
  uint8_t* F = (uint8_t*)(V + N);          // N flags
  uint8_t* hx = F + N;                     // N row winners (0xFF: none)
  uint32_t* dBad = (uint32_t*)(fs_s + (((size_t)N * 6 + 3) & ~(size_t)3));  // n x nw bit rows
  uint32_t* dTmp = dBad + n * nw;
  uint32_t* dPred = dTmp + n * nw;
  uint16_t* list = (uint16_t*)(dPred + n * nw);  // cap candidates
  __shared__ int2 locXY[MAX_MAXSS];
  __shared__ double locVal[MAX_MAXSS];
  __shared__ int sBest[2], sM, sTotal, sScan[NW];
  __shared__ double rA[NW];
  __shared__ unsigned rB[NW];
  __shared__ double sSum;
  __shared__ float sfP, sfK, sfLim;
  __shared__ int sDirect;

  // warps 2.. load the stamp while warps 0 and 1 search the exact
  // thresholds of the two static predicates; the window conditions cover
  // the pixels inside the frame (x < sx, y < sy)
  if(warp >= 2) {
    // whole rows (at most eight words) ahead of their tests
    for(int ly = warp - 2; ly < n; ly += NW - 2) {
      float v[8];
      uint16_t mk[8];
      const size_t row = (size_t)cx + (size_t)(cy + ly) * w;
#pragma unroll
      for(int j = 0; j < 8; j++) {
        const int lx = 32 * j + lane;
        v[j] = lx < n ? img[row + lx] : 0.f;
        mk[j] = lx < n ? ldMask(mask, row + lx) : (uint16_t)0;
      }
#pragma unroll
      for(int j = 0; j < 8; j++) {
        if(j >= nw) break;
        const int lx = 32 * j + lane;
        const bool b = (mk[j] & badMask) != 0;
        if(lx < n) {
          V[ly * n + lx] = v[j];
          F[ly * n + lx] = b ? FS_BAD : 0;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, b && lx < sx && ly < sy);
        if(lane == 0) dTmp[ly * nw + j] = m;
      }
    }
  }
  if(warp < 2) {
    auto pr = [&](double v) { return (v - sky) / fwhm > tKF; };
    auto kq = [&](double v) { return !((v - sky) * invFwhm < tKF); };
    const bool direct = !(fwhm > 0.0 && isfinite(fwhm) && isfinite(sky) && isfinite(invFwhm) &&
                          pr(INFINITY) && !pr(-INFINITY) && kq(INFINITY) && !kq(-INFINITY));
    if(!direct) {
      const unsigned long long kLo = dKey(-INFINITY), kHi = dKey(INFINITY);
      if(warp == 0) {
        const unsigned long long kP = warpFirstTrue(kLo, kHi, sky + tKF * fwhm, pr);
        if(lane == 0) sfP = __double2float_ru(keyD(kP));  // pr(v) <=> v >= sfP for a float v
      } else {
        const unsigned long long kK = warpFirstTrue(kLo, kHi, sky + tKF * fwhm, kq);
        if(lane == 0) sfK = __double2float_ru(keyD(kK));
      }
    }
    if(warp == 0 && lane == 0) sDirect = direct;
  }
  __syncthreads();
  const bool direct = sDirect != 0;
  const float fP = sfP, fK = sfK;
  for(int ly = warp; ly < n; ly += NW)
    for(int j = 0; j < nw; j++) {
      const int lx = 32 * j + lane;
      bool pr = false;
      if(lx < n) {
        const int p = ly * n + lx;
        const float f = V[p];
        bool kq;
        if(direct) {
          pr = ((double)f - sky) / fwhm > tKF;
          kq = !(((double)f - sky) * invFwhm < tKF);
        } else {
          pr = f >= fP;
          kq = isnan(f) || f >= fK;
        }
        const bool vpos = f > 0.f;
        uint8_t fl = F[p];
        if(pr) fl |= FL_PRED;
        if(pr && !vpos) fl |= FL_NONPOS;
        if(kq) fl |= FL_KFQ;
        if(vpos) fl |= FL_VPOS;
        F[p] = fl;
      }
      const uint32_t m = __ballot_sync(0xffffffffu, pr && lx < sx && ly < sy);
      if(lane == 0) dPred[ly * nw + j] = m;
    }
  __syncthreads();
  // window conditions: rows, then columns (bad: dTmp -> dBad, pred: dPred ->
  // dTmp, which is the final map)
  if(tid < n) dilateRow(dTmp + tid * nw, nw, hSS);
  else if(tid - 256 >= 0 && tid - 256 < n) dilateRow(dPred + (tid - 256) * nw, nw, hSS);
  __syncthreads();
  auto dilateColumns = [&](const uint32_t* src, uint32_t* dst) {
    for(int e = tid; e < n * nw; e += FS_T) {
      const int y = e / nw, j = e - y * nw;
      uint32_t o = 0;
      for(int yy = max(y - hSS, 0); yy <= min(y + hSS, n - 1); yy++) o |= src[yy * nw + j];
      dst[e] = o;
    }
    __syncthreads();
  };
  dilateColumns(dTmp, dBad);
  dilateColumns(dPred, dTmp);
  const uint32_t* dOk = dTmp;
  uint32_t* cands = dPred;  // free from here on
  auto bitAt = [&](const uint32_t* d, int y, int x) { return (d[y * nw + (x >> 5)] >> (x & 31)) & 1u; };

  // A key is the float bit pattern of a qualifying pixel (0: none).
  auto keyAt = [&](int p) -> uint32_t {
    const uint8_t fl = F[p];
    return (fl & (FS_BAD | FL_KFQ | FL_VPOS)) == (FL_KFQ | FL_VPOS) ? __float_as_uint(V[p]) : 0u;
  };
  // Row winners of the columns [x0, x1] of the rows [k0, k1], FS_SEG columns
  // per task: their windows share the middle, so each is the best of a suffix
  // of the columns left of it, the middle, and a prefix of those right of it
  // (ties keep the smaller column).  Neighbouring lanes take neighbouring rows.
  auto rowWinners = [&](int x0, int x1, int k0, int k1) {
    const int s0 = x0 / FS_SEG, s1 = x1 / FS_SEG, nr = k1 - k0 + 1;
    for(int t = tid; t < nr * (s1 - s0 + 1); t += FS_T) {
      const int q = t / nr, xs = (s0 + q) * FS_SEG, row = (k0 + t - q * nr) * n;
      if(hSS < FS_SEG / 2) {  // windows without a shared middle
        for(int i = 0; i < FS_SEG && xs + i < n; i++) {
          uint32_t bk = 0;
          int bi = 0xFF;
          for(int x = max(xs + i - hSS, 0); x <= min(xs + i + hSS, n - 1); x++) {
            const uint32_t k = keyAt(row + x);
            if(k > bk) {
              bk = k;
              bi = x;
            }
          }
          hx[row + xs + i] = (uint8_t)bi;
        }
        continue;
      }
      uint32_t lk[FS_SEG - 1], mk = 0, bk = 0;
      int li[FS_SEG - 1], mi = 0xFF, bi = 0xFF;
#pragma unroll
      for(int i = FS_SEG - 2; i >= 0; i--) {
        const int x = xs - hSS + i;
        const uint32_t k = x >= 0 && x < n ? keyAt(row + x) : 0u;
        if(k != 0 && k >= bk) {
          bk = k;
          bi = x;
        }
        lk[i] = bk;
        li[i] = bi;
      }
      for(int x = max(xs - hSS + FS_SEG - 1, 0); x <= min(xs + hSS, n - 1); x++) {
        const uint32_t k = keyAt(row + x);
        if(k > mk) {
          mk = k;
          mi = x;
        }
      }
      uint32_t rk = 0;
      int ri = 0xFF;
#pragma unroll
      for(int i = 0; i < FS_SEG; i++) {
        uint32_t k = i < FS_SEG - 1 ? lk[i < FS_SEG - 1 ? i : 0] : 0u;
        int o = i < FS_SEG - 1 ? li[i < FS_SEG - 1 ? i : 0] : 0xFF;
        if(mk > k) {
          k = mk;
          o = mi;
        }
        if(i > 0) {
          const int x = xs + hSS + i;
          const uint32_t kx = x < n ? keyAt(row + x) : 0u;
          if(kx > rk) {
            rk = kx;
            ri = x;
          }
        }
        if(rk > k) o = ri;
        if(xs + i < n) hx[row + xs + i] = (uint8_t)o;
      }
    }
    __syncthreads();
  };
  rowWinners(0, n - 1, 0, n - 1);
  // The pixel a candidate stands for: its window's first largest key, or
  // itself where the window has none.
  auto windowMax = [&](int p, int ly, int lx) -> int {
    const int y1 = min(ly + hSS, n - 1);
    uint32_t bk = 0;
    int m = p;
    for(int y = max(ly - hSS, 0); y <= y1; y += 8) {
      int q[8];
      uint32_t k[8];
#pragma unroll
      for(int u = 0; u < 8; u++) q[u] = y + u <= y1 ? hx[(y + u) * n + lx] : 0xFF;
#pragma unroll
      for(int u = 0; u < 8; u++) {
        k[u] = 0;
        if(q[u] != 0xFF) {
          q[u] += (y + u) * n;
          k[u] = __float_as_uint(V[q[u]]);
        }
      }
#pragma unroll
      for(int u = 0; u < 8; u++)
        if(k[u] > bk) {
          bk = k[u];
          m = q[u];
        }
    }
    return m;
  };
  const double floorV = sky + tKF * fwhm;
  double dfrac = 0.9;
  int cnt = 0, passes = 0;
  while(cnt < maxSS && passes < 256) {
    passes++;
    const double alt = sky + (tH - sky) * dfrac;
    const double lim = floorV < alt ? alt : floorV;  // OpenCL max()
    if(tid == 0) sfLim = __double2float_rd(lim);    // v > lim <=> v > sfLim for a float v
    __syncthreads();
    const float fLim = sfLim;
    // this pass's candidates: bits, then lists in raster order
    for(int ly = warp; ly < n; ly += NW) {
      uint8_t f[8];
      float v[8];
#pragma unroll
      for(int j = 0; j < 8; j++) {
        const int lx = 32 * j + lane, p = ly * n + lx;
        f[j] = lx < n ? F[p] : (uint8_t)0;
        v[j] = lx < n ? V[p] : 0.f;
      }
#pragma unroll
      for(int j = 0; j < 8; j++) {
        if(j >= nw) break;
        const uint32_t c = __ballot_sync(0xffffffffu, (f[j] & (FS_BAD | FL_KFQ)) == FL_KFQ && v[j] > fLim);
        if(lane == 0) cands[ly * nw + j] = c;
      }
    }
    if(tid < 2) sBest[tid] = INT_MAX;
    __syncthreads();
    int from = 0, at = 0, nList = 0, turn = 0;  // list of the candidates from `from` on
    while(cnt < maxSS) {
      int mine = INT_MAX;  // index in the list
      while(mine == INT_MAX) {
        if(at >= nList) {
          if(from >= N) break;
          const int ys = from / n, xs = from - ys * n, e0 = ys * nw + (xs >> 5);
          nList = 0;
          for(int eb = e0; eb < n * nw && nList < cap; eb += FS_T) {
            const int e = eb + tid, y = e / nw;
            unsigned c = e < n * nw ? cands[e] : 0u;
            if(e == e0) c &= 0xFFFFFFFFu << (xs & 31);
            int k = nList + blockScanExcl(__popc(c), sScan, &sTotal);
            for(; c && k < cap; c &= c - 1, k++)
              list[k] = (uint16_t)(y * n + 32 * (e - y * nw) + __ffs(c) - 1);
            nList += sTotal;
            __syncthreads();
          }
          // a full list, also one that filled exactly, goes on behind its last
          // candidate: words may be left that no step has looked at
          from = N;
          if(nList >= cap) {
            nList = cap;
            from = list[cap - 1] + 1;
          }
          at = 0;
          if(nList == 0) break;
        }
        // a candidate per thread
        const int k = at + tid;
        int m = 0;
        if(k < nList) {
          const int pc = list[k], ly = pc / n;
          if(!(F[pc] & FS_BAD)) {  // not in an accepted window since
            m = windowMax(pc, ly, pc - ly * n);
            const int my = m / n, mx = m - my * n;
            if(!bitAt(dBad, my, mx) && bitAt(dOk, my, mx)) mine = k;
          }
        }
        const int own = mine, best = __reduce_min_sync(0xffffffffu, mine);
        if(lane == 0 && best != INT_MAX) atomicMin(&sBest[turn], best);
        __syncthreads();
        mine = sBest[turn];
        if(own != INT_MAX && own == mine) sM = m;
        if(tid == 0) sBest[turn ^ 1] = INT_MAX;
        __syncthreads();
        turn ^= 1;
        at = mine == INT_MAX ? at + FS_T : mine + 1;
      }
      if(mine == INT_MAX) break;
      const int m = sM;
      const int mx = cx + m % n, my = cy + m / n;
      const int u0 = max(mx - hSS, cx), v0 = max(my - hSS, cy);
      const int u1 = min(mx + hSS, cx + sx - 1), v1 = min(my + hSS, cy + sy - 1);
      const int uw = u1 - u0 + 1, un = uw * (v1 - v0 + 1);
      // value of the substamp: the reference's serial FP64 sum of the
      // thresholded pixels in raster order.  When they are all positive and
      // the sum of their magnitudes stays below 2^52 quanta of the smallest
      // (every pixel is a multiple of that quantum), no partial sum rounds in
      // any order; otherwise warp 0 forms the serial sum bit for bit (osum;
      // a pixel below the threshold adds +0.0, which changes nothing).
      double part = 0.0;
      unsigned amin = 0x7F800000u;  // bits of the smallest magnitude
      bool nonpos = false;
      for(int i = tid; i < un; i += FS_T) {
        const int q = (v0 + i / uw - cy) * n + (u0 + i % uw - cx);
        const uint8_t fl = F[q];
        if(fl & FL_PRED) {
          part += (double)V[q];
          amin = min(amin, __float_as_uint(V[q]) & 0x7FFFFFFFu);
          nonpos |= (fl & FL_NONPOS) != 0;
        }
      }
#pragma unroll
      for(int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      amin = __reduce_min_sync(0xffffffffu, amin);
      if(lane == 0) {
        rA[warp] = part;
        rB[warp] = amin;
      }
      nonpos = __syncthreads_or(nonpos);
      if(warp == 0) {
        double t = lane < NW ? rA[lane] : 0.0;
#pragma unroll
        for(int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        const unsigned mn = __reduce_min_sync(0xffffffffu, lane < NW ? rB[lane] : 0x7F800000u);
        // smallest in [2^(e-127), 2^(e-126)), so every pixel is a multiple of
        // 2^(e-150), and the sum must stay below 2^(e-98)
        const int e = (int)(mn >> 23);
        const bool exact = !nonpos && e > 0 && e < 255 &&
                           __double_as_longlong(t) < (long long)(e - 98 + 1023) << 52;
        if(!exact)
          t = osum::warpOrderedSumOf(un, [&](int i) {
            const int q = (v0 + i / uw - cy) * n + (u0 + i % uw - cx);
            return (F[q] & FL_PRED) ? V[q] : 0.f;
          });
        if(lane == 0) sSum = t;
      }
      __syncthreads();
      const double ret = sSum;
      if(ret == 0.0) continue;
      if(tid == 0) {
        locXY[cnt] = make_int2(mx, my);
        locVal[cnt] = ret;
      }
      cnt++;
      // the window turns bad (skipMask is part of badMask)
      for(int i = tid; i < un; i += FS_T) {
        const int gx = u0 + i % uw, gy = v0 + i / uw;
        orMask(mask, (size_t)gx + (size_t)gy * w, skipMask);
        F[(gy - cy) * n + (gx - cx)] |= FS_BAD;
      }
      if(cnt < maxSS) {
        const int a0 = max(u0 - cx - hSS, 0), a1 = min(u1 - cx + hSS, n - 1);
        const int b0 = max(v0 - cy - hSS, 0), b1 = min(v1 - cy + hSS, n - 1);
        for(int e = tid; e < (b1 - b0 + 1) * nw; e += FS_T) {
          const int y = b0 + e / nw, j = e % nw;
          const int l = max(a0 - 32 * j, 0), h = min(a1 - 32 * j, 31);  // bits l..h of word j
          if(l <= h) dBad[y * nw + j] |= (0xFFFFFFFFu >> (31 - h)) & (0xFFFFFFFFu << l);
        }
        __syncthreads();
        rowWinners(a0, a1, v0 - cy, v1 - cy);
      }
    }
    if(cnt >= maxSS || lim == floorV) break;
    dfrac -= 0.2;
  }
  __syncthreads();
  if(tid == 0) {
    for(int i = 1; i < cnt; i++)
      for(int j = i; j > 0 && locVal[j - 1] < locVal[j]; j--) {
        int2 t = locXY[j - 1];
        locXY[j - 1] = locXY[j];
        locXY[j] = t;
        double tv = locVal[j - 1];
        locVal[j - 1] = locVal[j];
        locVal[j] = tv;
      }
    for(int i = 0; i < maxSS; i++) {
      xyOut[i] = i < cnt ? locXY[i] : make_int2(INT_MAX, INT_MAX);
      valOut[i] = i < cnt ? locVal[i] : -INFINITY;
    }
    (im == 0 ? cnt0 : cnt1)[s] = min(cnt, maxSS / 2);
  }
}

// removeEmptyStamps (src/sssUtil.cpp:106-197, sss.cl:543-571): keep stamps
// with at least one substamp in ascending original order.  One CTA per image.
__global__ void __launch_bounds__(256)
    k_compact_stamps(const int* __restrict__ cntAll, const int2* __restrict__ xyAll,
                     const double* __restrict__ valAll, int nAll, int maxSS,
                     int* __restrict__ orig, int* __restrict__ count, int* __restrict__ cur,
                     int2* __restrict__ xy, double* __restrict__ val, int* __restrict__ nOut) {
  __shared__ int warpTot[8];
  __shared__ int sTotal;
  int done = 0;
  for(int base = 0; base < nAll; base += 256) {
    int s = base + threadIdx.x;
    int keep = (s < nAll && cntAll[s] > 0) ? 1 : 0;
    int pos = blockScanExcl(keep, warpTot, &sTotal) + done;
    if(keep) {
      orig[pos] = s;
      count[pos] = cntAll[s];
      cur[pos] = 0;
      for(int k = 0; k < maxSS; k++) {
        bool live = k < cntAll[s];
        xy[(size_t)pos * maxSS + k] = live ? xyAll[(size_t)s * maxSS + k] : make_int2(INT_MAX, INT_MAX);
        val[(size_t)pos * maxSS + k] = live ? valAll[(size_t)s * maxSS + k] : -INFINITY;
      }
    }
    done += sTotal;
    __syncthreads();
  }
  if(threadIdx.x == 0) *nOut = done;
}

// createStampBounds (sss.cl:19-38) on the device, for frame graphs: the
// same integer expressions as the host table of stageSss.
__global__ void k_stamp_geom(int4* __restrict__ geom, int nAll, int stampsx, int stampsy, int w,
                             int h, int fSW) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if(id >= nAll) return;
  const int sxI = id % stampsx, syI = id / stampsx;
  const int startX = sxI * w / stampsx, startY = syI * h / stampsy;
  const int stopX = min(startX + fSW, w), stopY = min(startY + fSW, h);
  geom[id] = make_int4(startX, startY, stopX - startX, stopY - startY);
}

__global__ void k_reset_skip(uint16_t* mask, long long n) {
  for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += (long long)gridDim.x * blockDim.x)
    mask[i] &= (uint16_t)~(SKIP_S | SKIP_T);
}

}  // namespace

// The ran1 sequence of seed -666 (the seed of every stamp, sss.cl:81-116),
// n draws, generated once per context and size.
static const double* ran1Draws(xb_ctx* c, int n) {
  const std::string key = "ran1_draws";
  auto it = c->pool.find(key);
  const bool have = it != c->pool.end() && it->second.bytes >= (size_t)n * sizeof(double) &&
                    c->scalars.count("ran1_draws_n") && c->scalars["ran1_draws_n"] >= n;
  double* d = buf<double>(c, key, n);
  if(!have) {
    std::vector<double> h(n);
    Ran1 rng;
    double r[98];
    rng.init(-666);
    for(int i = 0; i < n; i++) h[i] = rng.next(r);
    toDevice(c, d, h);
    c->scalars["ran1_draws_n"] = n;
  }
  return d;
}

static void sssPass(xb_ctx* c, int* nKept) {
  const Geo& g = c->g;
  const int fSW = c->fStampWidth, nAll = c->nAll;
  double* chunkBuf = c->dWork;  // sized by stageSss
  const double* draws = ran1Draws(c, 2 * fSW * fSW);
  for(int im = 0; im < 2; im++) {
    { KT_SCOPE(c, "stamp_stats");
    auto stats = [&](auto* img, auto* good) {
      XB_CUDA(launchStampStats(img, c->mask, c->geomAll, nAll, c->w, c->h, fSW, good, c->clipScratch,
                               chunkBuf, c->p.sigClipAlpha, c->p.iqRange, c->skyAll[im],
                               c->fwhmAll[im], draws, c->device, c->stream));
    };
    if(c->imgIsF64) stats((const double*)c->img[im], c->goodScratch);
    else stats((const float*)c->img[im], reinterpret_cast<float*>(c->goodScratch));
    XB_LAUNCHED(c);
    }
  }
  dim3 grid(nAll, 2);
  { KT_SCOPE(c, "find_substamps");
  const size_t perCta = ((size_t)fSW * fSW * 24 + 255) / 256 * 256;
  const size_t fsSmem = fsSmemBytes(fSW);
  // stamps that fit in shared memory with byte row winners, of FP32 images;
  // else maps in global memory
  int optin = 0;
  XB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const bool inShared = !c->imgIsF64 && fSW <= FS_MAXN && fsSmem + 2 * FS_T + 1024 <= (size_t)optin;
  const int cap = fsSmem + 2 * FS_LIST + 1024 <= (size_t)optin ? FS_LIST : FS_T;
  // global-memory maps only for the kernel that uses them
  unsigned char* scratch =
      inShared ? nullptr : buf<unsigned char>(c, "fm_scratch", (size_t)2 * nAll * perCta);
  if(inShared) {
    XB_CUDA(allowMaxDynamicSmem((const void*)k_find_substamps_sm, c->device));
    k_find_substamps_sm<<<grid, FS_T, fsSmem + 2 * cap, c->stream>>>(
        (const float*)c->img[0], (const float*)c->img[1], c->mask, c->geomAll, c->skyAll[0],
        c->fwhmAll[0], c->skyAll[1], c->fwhmAll[1], c->ssxyAll[0], c->ssvalAll[0], c->cntAll[0],
        c->ssxyAll[1], c->ssvalAll[1], c->cntAll[1], c->w, fSW, g.hSS, g.maxSS, c->p.threshHigh,
        c->p.threshKernFit, cap);
  } else if(c->imgIsF64)
    k_find_substamps_maps<double><<<grid, FM_THREADS, 0, c->stream>>>(
        (const double*)c->img[0], (const double*)c->img[1], c->mask, c->geomAll,
        c->skyAll[0], c->fwhmAll[0], c->skyAll[1], c->fwhmAll[1], c->ssxyAll[0],
        c->ssvalAll[0], c->cntAll[0], c->ssxyAll[1], c->ssvalAll[1], c->cntAll[1], c->w,
        fSW, g.hSS, g.maxSS, c->p.threshHigh, c->p.threshKernFit, scratch, perCta, 0);
  else
    k_find_substamps_maps<float><<<grid, FM_THREADS, 0, c->stream>>>(
        (const float*)c->img[0], (const float*)c->img[1], c->mask, c->geomAll,
        c->skyAll[0], c->fwhmAll[0], c->skyAll[1], c->fwhmAll[1], c->ssxyAll[0],
        c->ssvalAll[0], c->cntAll[0], c->ssxyAll[1], c->ssvalAll[1], c->cntAll[1], c->w,
        fSW, g.hSS, g.maxSS, c->p.threshHigh, c->p.threshKernFit, scratch, perCta, 1);
  XB_LAUNCHED(c);
  }
  for(int im = 0; im < 2; im++) {
    StampSetDev& S = c->set[im];
    { KT_SCOPE(c, "compact_stamps");
    k_compact_stamps<<<1, 256, 0, c->stream>>>(c->cntAll[im], c->ssxyAll[im], c->ssvalAll[im],
                                               nAll, g.maxSS, S.orig, S.count, S.cur, S.ssxy,
                                               S.ssval, c->dIWork + im);
    XB_LAUNCHED(c);
    }
  }
  if(c->capturing) return;  // frame graphs keep the counts on the device
  std::vector<int> n = toHost(c, c->dIWork, 2);
  nKept[0] = n[0];
  nKept[1] = n[1];
}

void stageSss(xb_ctx* c) {
  const Geo& g = c->g;
  const int w = c->w, h = c->h;
  // stamp width rule of src/bach.cpp:51-66
  c->stampsx = c->p.stampsx;
  c->stampsy = c->p.stampsy;
  int fSW = std::min(w / c->stampsx, h / c->stampsy);
  fSW -= g.fK;
  fSW -= fSW % 2 == 0 ? 1 : 0;
  if(fSW < g.fSS) {
    fSW = g.fSS + g.fK;
    fSW -= fSW % 2 == 0 ? 1 : 0;
    c->stampsx = w / fSW;
    c->stampsy = h / fSW;
  }
  c->fStampWidth = fSW;
  if(c->stampsx <= 0 || c->stampsy <= 0) throw XbError{XB_ERR_ARG, "image too small for one stamp"};
  if(fSW > 2048) throw XbError{XB_ERR_UNSUPPORTED, "stamp width above 2048"};
  if(g.maxSS > MAX_MAXSS || g.fSS > MAX_FSS)
    throw XbError{XB_ERR_UNSUPPORTED, "substamp parameters above this build's limits"};
  const int nAll = c->stampsx * c->stampsy;
  c->nAll = nAll;
  // createStampBounds (sss.cl:19-38)
  std::vector<int4> geom(nAll);
  for(int id = 0; id < nAll; id++) {
    int sxI = id % c->stampsx, syI = id / c->stampsx;
    int startX = sxI * w / c->stampsx, startY = syI * h / c->stampsy;
    int stopX = std::min(startX + fSW, w), stopY = std::min(startY + fSW, h);
    geom[id] = make_int4(startX, startY, stopX - startX, stopY - startY);
    if((stopX - startX) * (stopY - startY) < NSAMPLES)  // bachUtil.cpp:145-155
      throw XbError{XB_ERR_STAMP_TOO_SMALL, "Not enough pixels in a stamp"};
  }
  // buffers for this grid
  c->geomAll = buf<int4>(c, "geomAll", nAll);
  for(int im = 0; im < 2; im++) {
    const std::string sfx = std::to_string(im);
    c->skyAll[im] = buf<double>(c, "skyAll" + sfx, nAll);
    c->fwhmAll[im] = buf<double>(c, "fwhmAll" + sfx, nAll);
    c->cntAll[im] = buf<int>(c, "cntAll" + sfx, nAll);
    c->ssxyAll[im] = buf<int2>(c, "ssxyAll" + sfx, (size_t)nAll * g.maxSS);
    c->ssvalAll[im] = buf<double>(c, "ssvalAll" + sfx, (size_t)nAll * g.maxSS);
    StampSetDev& S = c->set[im];
    S.orig = buf<int>(c, "orig" + sfx, nAll);
    S.count = buf<int>(c, "count" + sfx, nAll);
    S.cur = buf<int>(c, "cur" + sfx, nAll);
    S.ssxy = buf<int2>(c, "ssxy" + sfx, (size_t)nAll * g.maxSS);
    S.ssval = buf<double>(c, "ssval" + sfx, (size_t)nAll * g.maxSS);
  }
  c->goodScratch = buf<double>(c, "goodScratch", (size_t)nAll * statsSlice(fSW));
  c->clipScratch = buf<uint8_t>(c, "clipScratch", (size_t)nAll * statsSlice(fSW));
  const size_t chunkDoubles = (size_t)nAll * 2 * ((fSW * fSW + 31) / 32);
  c->dWork = buf<double>(c, "chunkScratch", chunkDoubles);
  c->dIWork = buf<int>(c, "iwork", 64);
  int nKept[2];
  if(c->capturing) {
    // frame graph: the grid is computed on the device (the upload would be a
    // per-shape constant), the retry is a conditional node on the counts
    k_stamp_geom<<<(nAll + 255) / 256, 256, 0, c->stream>>>(c->geomAll, nAll, c->stampsx,
                                                            c->stampsy, w, h, fSW);
    XB_LAUNCHED(c);
    sssPass(c, nKept);
    graphSssRetry(c, c->dIWork, nAll, [&] {
      const long long n = (long long)w * h;
      k_reset_skip<<<std::min<long long>((n + 255) / 256, c->smCount * 8), 256, 0, c->stream>>>(
          c->mask, n);
      XB_LAUNCHED(c);
      sssPass(c, nKept);
    });
    for(int im = 0; im < 2; im++) {
      c->set[im].n = nAll;  // bound; the kept count is dIWork[im]
      c->set[im].dN = c->dIWork + im;
    }
    if(c->rank && c->rankW) rankSubstamps(c);  // learned order, on the device
    c->scalars["stampsx"] = c->stampsx;
    c->scalars["stampsy"] = c->stampsy;
    c->scalars["fStampWidth"] = c->fStampWidth;
    return;
  }
  c->set[0].dN = c->set[1].dN = nullptr;
  toDevice(c, c->geomAll, geom);
  sssPass(c, nKept);
  const int oldCount = nAll;
  const double fT = (double)nKept[0] / oldCount, fS = (double)nKept[1] / oldCount;
  c->sssRetry = 0;
  if(fT < 0.1 || fS < 0.1) {
    // bach.cpp:142-161: halve threshLow (unused by sss), clear the SKIP bits,
    // recompute everything with the current mask
    c->sssRetry = 1;
    const long long n = (long long)w * h;
    k_reset_skip<<<std::min<long long>((n + 255) / 256, c->smCount * 8), 256, 0, c->stream>>>(c->mask, n);
    XB_LAUNCHED(c);
    sssPass(c, nKept);
  }
  c->set[0].n = nKept[0];
  c->set[1].n = nKept[1];
  c->scalars["nstamps0"] = nKept[0];
  c->scalars["nstamps1"] = nKept[1];
  if(nKept[0] == 0 && nKept[1] == 0) throw XbError{XB_ERR_NO_SUBSTAMPS, "No substamps found"};
  if(c->rank && c->rankW) rankSubstamps(c);  // learned order of each stamp's substamps
  if(c->trace) {
    for(int im = 0; im < 2; im++) {
      const std::string sfx = std::to_string(im);
      c->put("sky" + sfx, toHost(c, c->skyAll[im], nAll));
      c->put("fwhm" + sfx, toHost(c, c->fwhmAll[im], nAll));
      c->put("ss_count_all" + sfx, toHost(c, c->cntAll[im], nAll));
      c->put("ss_xy_all" + sfx, toHost(c, c->ssxyAll[im], (size_t)nAll * g.maxSS));
      c->put("ss_val_all" + sfx, toHost(c, c->ssvalAll[im], (size_t)nAll * g.maxSS));
      const StampSetDev& S = c->set[im];
      c->put("stamp_index" + sfx, toHost(c, S.orig, S.n));
      c->put("ss_count" + sfx, toHost(c, S.count, S.n));
      c->put("ss_xy" + sfx, toHost(c, S.ssxy, (size_t)S.n * g.maxSS));
      c->put("ss_val" + sfx, toHost(c, S.ssval, (size_t)S.n * g.maxSS));
      c->scalars["nstamps" + sfx] = S.n;
    }
    c->put("mask_sss", toHost(c, c->mask, (size_t)w * h));
  }
  c->scalars["stampsx"] = c->stampsx;
  c->scalars["stampsy"] = c->stampsy;
  c->scalars["fStampWidth"] = c->fStampWidth;
  c->scalars["sss_retry"] = c->sssRetry;
}

}  // namespace xb

// ---------------------------------------------------------------------------
// Per-stamp statistics without any allocation.
//
// Some callers cannot allocate device memory: code that runs while another
// allocator (a framework's caching pool, a service's preallocated arena)
// owns the device and must not be bypassed, or code that must not let a
// cudaMalloc/cudaFree implicitly synchronise the device in the middle of
// its own work.  For them the stamp statistics of the sss stage (sky level
// and robust sigma per stamp, the same kernel xb_sss runs) are available
// with all scratch memory taken from a fixed device array that is part of the
// library image: every GPU that loads the library holds these 32 MiB until
// the process exits.  The caller passes the image, the mask, the stamp
// geometry and the two output arrays, all in device memory.

#include <cstring>
#include <mutex>

namespace {

constexpr size_t kStatsScratchBytes = size_t(32) << 20;  // 32 MiB
constexpr int kMaxDevices = 64;
static __device__ __align__(256) unsigned char g_statsScratch[kStatsScratchBytes];

std::mutex g_statsScratchMutex;
void* g_statsScratchAddr[kMaxDevices] = {};

size_t alignUp(size_t v) { return (v + 255) & ~size_t(255); }

int noallocFail(char* err, size_t errCap, int code, const char* msg) {
  if(err && errCap) {
    std::strncpy(err, msg, errCap - 1);
    err[errCap - 1] = '\0';
  }
  return code;
}

}  // namespace

extern "C" int xb_stamp_stats_noalloc(const float* dImg, uint16_t* dMask, int w, int h,
                                      const int* dGeom, int nStamps, int fStampWidth,
                                      double sigClipAlpha, double iqRange, double* dSky,
                                      double* dFwhm, void* stream, char* err, size_t errCap) {
  if(!dImg || !dMask || !dGeom || !dSky || !dFwhm || w <= 0 || h <= 0 || nStamps <= 0 ||
     fStampWidth <= 0)
    return noallocFail(err, errCap, XB_ERR_ARG, "null pointer or non-positive size");
  if(((uintptr_t)dGeom & 15u) != 0)
    return noallocFail(err, errCap, XB_ERR_ARG, "stamp geometry must be 16-byte aligned");
  // scratch carve-up: good pixels (FP64), clip flags (bytes), chunk sums
  const size_t pix = (size_t)fStampWidth * fStampWidth;
  const int maxChunks = (int)((pix + 31) / 32);
  if(pix > (size_t)1 << 26)
    return noallocFail(err, errCap, XB_ERR_UNSUPPORTED, "stamps beyond 8192 px on a side");
  const size_t slice = xb::statsSlice(fStampWidth);
  const size_t goodBytes = alignUp((size_t)nStamps * slice * sizeof(double));
  const size_t clipBytes = alignUp((size_t)nStamps * slice);
  const size_t chunkBytes = alignUp((size_t)nStamps * 2 * maxChunks * sizeof(double));
  if(goodBytes + clipBytes + chunkBytes > kStatsScratchBytes)
    return noallocFail(err, errCap, XB_ERR_UNSUPPORTED,
                       "stamps need more than the 32 MiB scratch: nStamps * (9 * P + 16 * "
                       "ceil(fStampWidth^2 / 32)) bytes must fit, P = fStampWidth^2 rounded up "
                       "to a multiple of 1024");
  // An error left pending by the caller's own work is reported as such and
  // left in place (not cleared), so it is not mistaken for this call's.
  const cudaError_t pending = cudaPeekAtLastError();
  if(pending != cudaSuccess)
    return noallocFail(err, errCap, XB_ERR_CUDA, "a CUDA error was already pending; nothing launched");
  int dev = -1;
  if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return noallocFail(err, errCap, XB_ERR_CUDA, "no usable current CUDA device");
  void* base = nullptr;
  {
    // The array's device address is looked up once per device, with that
    // device current; host code must not use the symbol itself as an address.
    // The cached address belongs to the device's current context: after a
    // cudaDeviceReset the module is reloaded elsewhere, so the entry point
    // must not be used across a reset.
    std::lock_guard<std::mutex> lock(g_statsScratchMutex);
    if(!g_statsScratchAddr[dev]) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_statsScratch);
      if(e != cudaSuccess || !p)
        return noallocFail(err, errCap, XB_ERR_CUDA, cudaGetErrorString(e));
      g_statsScratchAddr[dev] = p;
    }
    base = g_statsScratchAddr[dev];
  }
  unsigned char* b = static_cast<unsigned char*>(base);
  double* good = reinterpret_cast<double*>(b);
  uint8_t* clip = b + goodBytes;
  double* chunks = reinterpret_cast<double*>(b + goodBytes + clipBytes);
  // Nothing needs clearing: within one launch every scratch byte the kernel
  // reads is written first (clip flags and good pixels during the
  // compaction, chunk sums before they are summed).
  cudaError_t e = xb::launchStampStats(
      dImg, dMask, reinterpret_cast<const int4*>(dGeom), nStamps, w, h, fStampWidth,
      reinterpret_cast<float*>(good), clip, chunks, sigClipAlpha, iqRange, dSky, dFwhm,
      (const double*)nullptr, dev, (cudaStream_t)stream);
  if(e != cudaSuccess) cudaGetLastError();  // not left pending for the caller
  if(e != cudaSuccess) return noallocFail(err, errCap, XB_ERR_CUDA, cudaGetErrorString(e));
  // no error was pending before the launch, so any error now is the launch's
  e = cudaGetLastError();
  if(e != cudaSuccess) return noallocFail(err, errCap, XB_ERR_CUDA, cudaGetErrorString(e));
  return XB_OK;
}

namespace xb {
namespace {
__global__ void k_ordered_sum(const double* __restrict__ c, int n, double* __restrict__ out) {
  const double s = osum::warpOrderedSum<2>(c, n);
  if(threadIdx.x == 0) *out = s;
}
__global__ void k_ordered_sum_f32(const float* __restrict__ c, int n, double* __restrict__ out) {
  const double s = osum::warpOrderedSumOf(n, [c](int i) { return c[i]; });
  if(threadIdx.x == 0) *out = s;
}
}  // namespace
}  // namespace xb

extern "C" double xb_ordered_sum_host(const double* c, int n) {
  return (c == nullptr || n <= 0) ? 0.0 : xb::osum::orderedSumHost(c, n);
}

extern "C" int xb_ordered_sum_device(const double* dC, int n, double* dOut, void* stream) {
  if(dOut == nullptr || n < 0 || (n > 0 && dC == nullptr)) return XB_ERR_ARG;
  xb::k_ordered_sum<<<1, 32, 0, (cudaStream_t)stream>>>(dC, n, dOut);
  return cudaGetLastError() == cudaSuccess ? XB_OK : XB_ERR_CUDA;
}

extern "C" int xb_ordered_sum_device_f32(const float* dC, int n, double* dOut, void* stream) {
  if(dOut == nullptr || n < 0 || (n > 0 && dC == nullptr)) return XB_ERR_ARG;
  xb::k_ordered_sum_f32<<<1, 32, 0, (cudaStream_t)stream>>>(dC, n, dOut);
  return cudaGetLastError() == cudaSuccess ? XB_OK : XB_ERR_CUDA;
}
