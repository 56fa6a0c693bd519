// xb_device.cuh — device helpers shared by the stage kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace xb {

// Block-wide exclusive scan of one int per thread; *total receives the sum.
// Every thread of the block must call it.
__device__ __forceinline__ int blockScanExcl(int v, int* warpTot, int* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for(int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if(lane >= o) x += y;
  }
  if(lane == 31) warpTot[wid] = x;
  __syncthreads();
  if(threadIdx.x == 0) {
    int s = 0;
    for(int i = 0; i < (int)(blockDim.x >> 5); i++) {
      int t = warpTot[i];
      warpTot[i] = s;
      s += t;
    }
    *total = s;
  }
  __syncthreads();
  int r = warpTot[wid] + x - v;
  __syncthreads();
  return r;
}

// (x - (w * 0.5f)) / (w * 0.5f) evaluated in float, as cl_kern/cmv.cl:180 and
// cl_kern/cd.cl:170 write it (an int times a float literal is float).
__device__ __forceinline__ double floatNormD(int x, int w) {
  float hw = (float)w * 0.5f;
  float r = ((float)x - hw) / hw;
  return (double)r;
}

// OpenCL pown(x, n) as the repeated product 1*x*x*...
__device__ __forceinline__ double ipowD(double x, int n) {
  double r = 1.0;
  for(int i = 0; i < n; i++) r *= x;
  return r;
}

// (double)(float)t without the two conversions (each takes an FP64 issue slot
// here): round the bits to 24 significant ones, ties to even.  Values whose
// float is subnormal, zero, infinite or NaN, or could overflow, convert.
__device__ __forceinline__ double roundToFloat(double t) {
  const long long b = __double_as_longlong(t);
  const unsigned e = (unsigned)(b >> 52) & 0x7FFu;
  if(e - 897u >= 253u) return (double)(float)t;  // below 2^-126 or from 2^127 up
  return __longlong_as_double((b + 0x0FFFFFFFll + ((b >> 29) & 1)) & ~0x1FFFFFFFll);
}

// Copies of 4, 8 or 16 bytes to shared memory that complete asynchronously, in
// groups.
__device__ __forceinline__ void cpAsync4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpAsync8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpAsync16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWaitGroup() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// OR `bits` into the 16-bit mask entry i with a 32-bit atomic on its
// aligned word (the mask buffer carries two spare entries at the end).
__device__ __forceinline__ void maskOr(uint16_t* m, size_t i, uint16_t bits) {
  uintptr_t a = (uintptr_t)(m + i);
  unsigned* w32 = (unsigned*)(a & ~(uintptr_t)3);
  unsigned sh = (a & 2) ? 16u : 0u;
  atomicOr(w32, (unsigned)bits << sh);
}

// sigmaClip of src/bachUtil.cpp:34-128 for one CTA: data[0..n) in global
// memory, sums in 32-element chunks (sequential inside a chunk,
// cl_kern/bach.cl:135-170) added sequentially (bachUtil.cpp:103-104).  Up to
// SC_CAP values stay in shared memory, their squares beside them: one warp sums
// the chunks, one their squares, a lane per chunk, and two threads add the
// chunks; bound by those chains (with every operand from global memory and one
// thread for both sums a check of 256 stamps took 20 us, now 15).  More values:
// clipped flags in `flags` (n bytes), chunk sums in cs/cs2.  The result
// is written to *outMean / *outStd (shared) by thread 0; all threads must
// call it.
constexpr int SC_CAP = 1024, SC_PER = 4;
__device__ inline void blockSigmaClip(const double* data, int n, int maxIter, double alpha,
                                      uint8_t* flags, double* cs, double* cs2,
                                      double* outMean, double* outStd, int* sh) {
  // sh[0] = prev, sh[1] = curr, sh[2] = clip, sh[3] = stop
  const int tid = threadIdx.x, nt = blockDim.x;
  __shared__ double sInv;
  if(n > SC_CAP || nt * SC_PER < SC_CAP)
    for(int k = tid; k < n; k += nt) flags[k] = 0;
  if(tid == 0) {
    sh[0] = n;
    sh[1] = 0;
    sh[3] = 0;
    *outMean = 0.0;
    *outStd = 1e10;
    if(n == 0) sh[3] = 1;
  }
  __syncthreads();
  const int nChunks = (n + 31) / 32;
  if(n <= SC_CAP && nt * SC_PER >= SC_CAP) {
    // value k at k + k / 32: a lane's chunk meets no bank conflicts
    __shared__ double sv[SC_CAP + SC_CAP / 32], sq[SC_CAP + SC_CAP / 32];
    __shared__ double sc[2][SC_CAP / 32], sSums[2];
    const int lane = tid & 31, warp = tid >> 5;
    double d[SC_PER];
    unsigned live = 0;
#pragma unroll
    for(int u = 0; u < SC_PER; u++) {
      const int k = tid + u * nt;
      d[u] = 0.0;
      if(k < n) {
        d[u] = data[k];
        live |= 1u << u;
        sv[k + (k >> 5)] = d[u];
        sq[k + (k >> 5)] = d[u] * d[u];
      }
    }
    for(int it = 0; it < maxIter; it++) {
      if(sh[3] || sh[1] == sh[0]) break;
      if(sh[0] <= 1) {
        __syncthreads();
        if(tid == 0) {
          *outMean = 0.0;
          *outStd = 1e10;
        }
        break;
      }
      __syncthreads();
      if(tid == 0) sh[1] = sh[0];
      if(warp < 2 && lane < nChunks) {
        const double* v = (warp ? sq : sv) + 33 * lane;
        const int lc = min(32, n - 32 * lane);
        double a = 0.0;
#pragma unroll 8
        for(int l = 0; l < lc; l++) a += v[l];
        sc[warp][lane] = a;
      }
      __syncthreads();
      if(warp < 2 && lane == 0) {
        double a = 0.0;
#pragma unroll 4
        for(int c = 0; c < nChunks; c++) a += sc[warp][c];
        sSums[warp] = a;
      }
      __syncthreads();
      if(tid == 0) {
        const double nn = (double)sh[1];
        const double m = sSums[0] / nn;
        const double sd = sqrt((sSums[1] - nn * m * m) / (double)(sh[1] - 1));
        *outMean = m;
        *outStd = sd;
        sInv = 1.0 / sd;
        sh[2] = 0;
      }
      __syncthreads();
      const double m = *outMean, inv = sInv;
      int myClip = 0;
#pragma unroll
      for(int u = 0; u < SC_PER; u++)
        if((live >> u & 1u) && fabs(d[u] - m) * inv > alpha) {
          const int k = tid + u * nt;
          live &= ~(1u << u);
          sv[k + (k >> 5)] = sq[k + (k >> 5)] = 0.0;
          myClip++;
        }
      if(myClip) atomicAdd(&sh[2], myClip);
      __syncthreads();
      if(tid == 0) sh[0] = sh[1] - sh[2];
      __syncthreads();
    }
    __syncthreads();
    return;
  }
  for(int it = 0; it < maxIter; it++) {
    if(sh[3] || sh[1] == sh[0]) break;
    if(sh[0] <= 1) {
      __syncthreads();
      if(tid == 0) {
        *outMean = 0.0;
        *outStd = 1e10;
      }
      break;
    }
    __syncthreads();
    if(tid == 0) sh[1] = sh[0];
    for(int c = tid; c < nChunks; c += nt) {
      double a = 0.0, a2 = 0.0;
      int lc = min(32, n - c * 32);
      for(int l = 0; l < lc; l++) {
        int k = c * 32 + l;
        double d = flags[k] == 0 ? data[k] : 0.0;
        a += d;
        a2 += d * d;
      }
      cs[c] = a;
      cs2[c] = a2;
    }
    __syncthreads();
    if(tid == 0) {
      double sum = 0.0, sum2 = 0.0;
      for(int c = 0; c < nChunks; c++) {
        sum += cs[c];
        sum2 += cs2[c];
      }
      double nn = (double)sh[1];
      double m = sum / nn;
      double sd = sqrt((sum2 - nn * m * m) / (double)(sh[1] - 1));
      *outMean = m;
      *outStd = sd;
      sInv = 1.0 / sd;
      sh[2] = 0;
    }
    __syncthreads();
    const double m = *outMean, inv = sInv;
    int myClip = 0;
    for(int k = tid; k < n; k += nt)
      if(flags[k] == 0 && fabs(data[k] - m) * inv > alpha) {
        flags[k] = 1;
        myClip++;
      }
    if(myClip) atomicAdd(&sh[2], myClip);
    __syncthreads();
    if(tid == 0) sh[0] = sh[1] - sh[2];
    __syncthreads();
  }
  __syncthreads();
}

}  // namespace xb
