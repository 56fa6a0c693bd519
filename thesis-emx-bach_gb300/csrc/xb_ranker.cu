// xb_ranker.cu — learned substamp ranking (no counterpart in the reference).
//
// The reference tries each stamp's substamps in order of brightness
// (sss.cl:363-379) and replaces a substamp only after the global fit has
// rejected it (ksc.cl:1-72, cdkscUtil.cpp:686-802), one refit per round of
// rejections.  A small network scores every candidate substamp from
//   * 16 statistics of the template/science windows around it, and
//   * the 2 x 31 x 31 window pair itself (sky-subtracted, peak-normalised),
// and the candidates of each stamp are reordered by score before cmv, so the
// ones the fit would reject are tried last.  The ksc sigma-clip check still
// runs on every pick; the network only changes the order.
//
// Network (2161 parameters, row-major in the order below), computed with
// BF16 weights and FP32 activations and accumulation: the training kernels
// take FP32 master weights (Adam updates those) and round each to BF16 as it
// is loaded, the inference copy in a context is stored as BF16, so both
// evaluate the same BF16-weight network:
//   conv1 2->8, 5x5, stride 2   (31 -> 14), ReLU
//   conv2 8->8, 3x3, stride 2   (14 -> 6),  ReLU
//   conv3 8->8, 3x3, stride 1   (6 -> 4),   ReLU, mean over the 4x4 map -> 8
//   mlp   16->32,                ReLU
//   head  [pool 8, mlp 32] -> 1 logit (accept probability = sigmoid)
// Training: binary cross-entropy with per-sample weights; one CTA computes
// the forward pass, the loss and the gradient of one sample; the gradients
// are summed over the batch in a fixed order (deterministic) and Adam updates
// the parameters.  Everything runs on the GPU from the C ABI.

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>

#include "xb_device.cuh"
#include "xb_internal.h"

namespace xb {

namespace {

constexpr int RK_T = 128;  // threads per candidate (features)
constexpr int RK_WIN = 31, RK_HWIN = 15, RK_NS = 16, RK_C = 8, RK_H = 32;
constexpr int RK_S1 = 14, RK_S2 = 6, RK_S3 = 4;
constexpr int RK_PIX = 2 * RK_WIN * RK_WIN;
constexpr int O_C1W = 0, O_C1B = O_C1W + RK_C * 2 * 25, O_C2W = O_C1B + RK_C,
              O_C2B = O_C2W + RK_C * RK_C * 9, O_C3W = O_C2B + RK_C,
              O_C3B = O_C3W + RK_C * RK_C * 9, O_M1W = O_C3B + RK_C,
              O_M1B = O_M1W + RK_H * RK_NS, O_HW = O_M1B + RK_H, O_HB = O_HW + RK_C + RK_H,
              RK_NP = O_HB + 1;
static_assert(RK_NP == 2161, "parameter layout");

// A weight as the network uses it: the FP32 master rounded to BF16 (nearest,
// ties to even), or a stored BF16 weight, as a float.
__device__ __forceinline__ float rkWeight(const float* W, int q) {
  return __bfloat162float(__float2bfloat16_rn(W[q]));
}
__device__ __forceinline__ float rkWeight(const __nv_bfloat16* W, int q) { return __bfloat162float(W[q]); }

// ------------------------------------------------------------------ forward --
// Two warps per sample.  The 109k multiply-adds of a sample are bound by the
// FP32 pipe only where each value read from shared memory feeds several of
// them: conv1 keeps 7 outputs of a row x 4 channels per lane (140 FMAs per 17
// window values and 5 broadcast float4 of weights), conv2 6 outputs of one
// channel, conv3 2.  Every output is summed in the order bias, input channel,
// row, column, so the logits are those of one thread per output (whose two
// shared reads per FMA took 101 us for 2000 samples on a GB300; this form takes
// 27 us).  24 warps per SM hide the latencies of the short layers; one warp
// per sample with all 8 channels had half of them and took 53 us.
constexpr int RF_SAMPLES = 4;           // samples per CTA
constexpr int RF_T = 64 * RF_SAMPLES;
constexpr int RF_LD = 35;               // window row: columns 0..16, then 14..30, and a pad
constexpr int RF_IN = RK_WIN * RF_LD;   // one image of the pair
constexpr int RF_A2 = RK_C * RK_S2 * RK_S2, RF_A3 = RK_C * RK_S3 * RK_S3;
constexpr int RF_A1 = RK_C * RK_S1 * RK_S1;
constexpr int RF_BUF = 2 * RF_IN + RF_A1 + 2;  // floats per sample
static_assert(RF_BUF % 4 == 0, "16-byte rows");
// weights with the output channel innermost
constexpr int RW_1 = 0, RW_2 = RW_1 + 400, RW_3 = RW_2 + 576, RW_M = RW_3 + 576,
              RW_B1 = RW_M + RK_H * RK_NS, RW_B2 = RW_B1 + 8, RW_B3 = RW_B2 + 8,
              RW_BM = RW_B3 + 8, RW_H = RW_BM + RK_H, RW_HB = RW_H + RK_C + RK_H, RW_N = RW_HB + 4;
constexpr size_t RF_SMEM = (size_t)(RW_N + RF_SAMPLES * RF_BUF) * sizeof(float);

__device__ __forceinline__ int rwIndex(int q) {
  if(q < O_C1B) return RW_1 + (q % 50) * 8 + q / 50;
  if(q < O_C2W) return RW_B1 + q - O_C1B;
  if(q < O_C2B) return RW_2 + ((q - O_C2W) % 72) * 8 + (q - O_C2W) / 72;
  if(q < O_C3W) return RW_B2 + q - O_C2B;
  if(q < O_C3B) return RW_3 + ((q - O_C3W) % 72) * 8 + (q - O_C3W) / 72;
  if(q < O_M1W) return RW_B3 + q - O_C3B;
  if(q < O_M1B) return RW_M + ((q - O_M1W) % RK_NS) * RK_H + (q - O_M1W) / RK_NS;
  if(q < O_HW) return RW_BM + q - O_M1B;
  return RW_H + q - O_HW;  // head weights, then its bias
}

// Barrier of the two warps of sample slot s.
__device__ __forceinline__ void pairSync(int s) {
  asm volatile("bar.sync %0, 64;" ::"r"(s + 1) : "memory");
}

// Logit of one sample by the two warps (half 0 and 1) of slot s; the lanes of
// half 0 return it.
__device__ float rfSample(const float* __restrict__ Wt, const float* __restrict__ stats,
                          const float* __restrict__ pix, float* __restrict__ buf, int s, int half) {
  const int lane = threadIdx.x & 31;
  float* in = buf;
  float* a1 = buf + 2 * RF_IN;
  float* a2 = buf;                // over the window, which is spent after conv1
  float* a3 = buf + RF_A2;
  float* hid = a3 + RF_A3;
  pairSync(s);  // the sample before is done
  if(lane < RK_WIN) {
    const float* src = pix + half * RK_WIN * RK_WIN + lane;
    float* dst = in + half * RF_IN + lane;
#pragma unroll 4
    for(int r = 0; r < RK_WIN; r++) {  // four-byte copies: any alignment of the caller's array
      if(lane < 17) cpAsync4(dst + r * RF_LD, src + r * RK_WIN);
      if(lane >= 14) cpAsync4(dst + r * RF_LD + 3, src + r * RK_WIN);
    }
  }
  const float st = lane < RK_NS ? stats[lane] : 0.f;
  cpAsyncCommit();
  cpAsyncWaitGroup<0>();
  pairSync(s);
  if(lane < 2 * RK_S1) {
    const int y = lane >> 1, h = lane & 1;
    float acc[7][4];
#pragma unroll
    for(int c = 0; c < 4; c++)
#pragma unroll
      for(int k = 0; k < 7; k++) acc[k][c] = Wt[RW_B1 + 4 * half + c];
#pragma unroll 1
    for(int r = 0; r < 10; r++) {
      const int ci = r / 5, ky = r - 5 * ci;
      const float* row = in + ci * RF_IN + (2 * y + ky) * RF_LD + 17 * h;
      float x[17];
#pragma unroll
      for(int k = 0; k < 17; k++) x[k] = row[k];
      const float4* w4 = (const float4*)(Wt + RW_1 + r * 40) + half;
#pragma unroll
      for(int kx = 0; kx < 5; kx++) {
        const float4 wv = w4[2 * kx];
        const float w[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for(int k = 0; k < 7; k++)
#pragma unroll
          for(int c = 0; c < 4; c++) acc[k][c] = fmaf(w[c], x[2 * k + kx], acc[k][c]);
      }
    }
#pragma unroll
    for(int c = 0; c < 4; c++)
#pragma unroll
      for(int k = 0; k < 7; k++)
        a1[((4 * half + c) * RK_S1 + y) * RK_S1 + 7 * h + k] = fmaxf(acc[k][c], 0.f);
  }
  pairSync(s);
  if(lane < 4 * RK_S2) {
    const int y = lane >> 2, c = 4 * half + (lane & 3);
    float acc[RK_S2];
#pragma unroll
    for(int k = 0; k < RK_S2; k++) acc[k] = Wt[RW_B2 + c];
#pragma unroll 2
    for(int r = 0; r < 24; r++) {
      const int ci = r / 3, ky = r - 3 * ci;
      const float* row = a1 + (ci * RK_S1 + 2 * y + ky) * RK_S1;
      float x[13];
#pragma unroll
      for(int k = 0; k < 13; k++) x[k] = row[k];
#pragma unroll
      for(int kx = 0; kx < 3; kx++) {
        const float w = Wt[RW_2 + (r * 3 + kx) * 8 + c];
#pragma unroll
        for(int k = 0; k < RK_S2; k++) acc[k] = fmaf(w, x[2 * k + kx], acc[k]);
      }
    }
#pragma unroll
    for(int k = 0; k < RK_S2; k++) a2[(c * RK_S2 + y) * RK_S2 + k] = fmaxf(acc[k], 0.f);
  }
  pairSync(s);
  {
    const int y = lane >> 3, c = lane & 7, x0 = 2 * half;
    float v0 = Wt[RW_B3 + c], v1 = v0;
#pragma unroll 3
    for(int r = 0; r < 24; r++) {
      const int ci = r / 3, ky = r - 3 * ci;
      const float* row = a2 + (ci * RK_S2 + y + ky) * RK_S2 + x0;
      float x[4];
#pragma unroll
      for(int k = 0; k < 4; k++) x[k] = row[k];
#pragma unroll
      for(int kx = 0; kx < 3; kx++) {
        const float w = Wt[RW_3 + (r * 3 + kx) * 8 + c];
        v0 = fmaf(w, x[kx], v0);
        v1 = fmaf(w, x[1 + kx], v1);
      }
    }
    a3[(c * RK_S3 + y) * RK_S3 + x0] = fmaxf(v0, 0.f);
    a3[(c * RK_S3 + y) * RK_S3 + x0 + 1] = fmaxf(v1, 0.f);
  }
  if(half) {
    float v = Wt[RW_BM + lane];
#pragma unroll
    for(int i = 0; i < RK_NS; i++)
      v = fmaf(Wt[RW_M + i * RK_H + lane], __shfl_sync(0xffffffffu, st, i), v);
    hid[RK_C + lane] = fmaxf(v, 0.f);
  }
  pairSync(s);
  float z = 0.f;
  if(!half) {
    if(lane < RK_C) {
      float v = 0.f;
#pragma unroll
      for(int p = 0; p < RK_S3 * RK_S3; p++) v += a3[lane * RK_S3 * RK_S3 + p];
      hid[lane] = v * (1.f / (RK_S3 * RK_S3));
    }
    __syncwarp();
    z = Wt[RW_HB];
#pragma unroll
    for(int i = 0; i < RK_C + RK_H; i++) z = fmaf(Wt[RW_H + i], hid[i], z);
  }
  return z;
}

// slots (optional): the candidate slots of the stamps, maxSS per stamp; a
// slot that is empty, past nRank in its stamp or in a stamp past *liveN
// gets no score (k_rank_order reads none for it).
template <class WT>
__global__ void __launch_bounds__(RF_T, 3)
    k_rank_forward(const WT* __restrict__ W, const float* __restrict__ stats,
                   const float* __restrict__ pix, int n, float* __restrict__ logit,
                   const int2* __restrict__ slots = nullptr, int maxSS = 1, int nRank = 1,
                   const int* __restrict__ liveN = nullptr) {
  extern __shared__ __align__(16) float rf_s[];
#pragma unroll 4
  for(int q = threadIdx.x; q < RK_NP; q += RF_T) rf_s[rwIndex(q)] = rkWeight(W, q);
  __syncthreads();
  const int s = threadIdx.x >> 6, half = (threadIdx.x >> 5) & 1;
  float* buf = rf_s + RW_N + s * RF_BUF;
  for(int i = blockIdx.x * RF_SAMPLES + s; i < n; i += gridDim.x * RF_SAMPLES) {
    if(slots && ((liveN && i / maxSS >= *liveN) || i % maxSS >= nRank || slots[i].x == INT_MAX))
      continue;  // uniform over the two warps
    const float z = rfSample(rf_s, stats + (size_t)i * RK_NS, pix + (size_t)i * RK_PIX, buf, s, half);
    if((threadIdx.x & 63) == 0) logit[i] = z;
  }
}

// ----------------------------------------------------------------- gradient --
// One CTA of eight warps per sample: forward, loss and the gradient of every
// parameter (loss = sw * BCE(sigmoid(z), y)) into the sample's row of gPer.
// A warp owns one output channel; a lane keeps a row segment of outputs, or
// the three or five weights of one kernel row, in registers, so that a row
// read from shared memory feeds several products (one thread per output or
// weight, two shared reads per product, took 123 us for 512 samples on a GB300;
// this form takes 44 us).  The gradients at the pre-activations of conv2
// and conv3 are stored with a border of zeros, which the gathers of the layer
// below read in the place of bounds checks.
constexpr int RG_T = 256;
constexpr int RG_LD = 33;             // window rows
constexpr int RG_P = 8;               // rows of the padded gradient maps
struct RkSample {
  float in[2 * RK_WIN * RG_LD];
  float a1[RK_C * RK_S1 * RK_S1];     // post-ReLU activations
  float a2[RK_C * RK_S2 * RK_S2];
  float a3[RK_C * RK_S3 * RK_S3];
  float st[RK_NS];
  float hid[RK_C + RK_H];
  float dh[RK_C + RK_H];
  float z;
  float d3[RK_C * RG_P * RG_P];       // (y, x) at [y + 2][x + 2]
  float d2[RK_C * RG_P * RG_P];       // (y, x) at [y + 1][x + 1]
  float d1[RK_C * RK_S1 * RK_S1];
};

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for(int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ void rgForward(const float* __restrict__ W, RkSample& A) {
  const int tid = threadIdx.x, lane = tid & 31, c = tid >> 5;
  if(lane < 2 * RK_S1) {
    const int y = lane >> 1, h = lane & 1;
    float acc[7];
#pragma unroll
    for(int k = 0; k < 7; k++) acc[k] = W[O_C1B + c];
#pragma unroll 2
    for(int r = 0; r < 10; r++) {
      const int ci = r / 5, ky = r - 5 * ci;
      const float* row = A.in + (ci * RK_WIN + 2 * y + ky) * RG_LD + 14 * h;
      const float* w = W + O_C1W + (c * 2 + ci) * 25 + ky * 5;
      float x[17];
#pragma unroll
      for(int k = 0; k < 17; k++) x[k] = row[k];
#pragma unroll
      for(int kx = 0; kx < 5; kx++)
#pragma unroll
        for(int k = 0; k < 7; k++) acc[k] = fmaf(w[kx], x[2 * k + kx], acc[k]);
    }
#pragma unroll
    for(int k = 0; k < 7; k++) A.a1[(c * RK_S1 + y) * RK_S1 + 7 * h + k] = fmaxf(acc[k], 0.f);
  }
  __syncthreads();
  if(lane < 3 * RK_S2) {
    const int y = lane / 3, x0 = 2 * (lane % 3);
    float v0 = W[O_C2B + c], v1 = v0;
#pragma unroll 4
    for(int r = 0; r < 24; r++) {
      const int ci = r / 3, ky = r - 3 * ci;
      const float* row = A.a1 + (ci * RK_S1 + 2 * y + ky) * RK_S1 + 2 * x0;
      const float* w = W + O_C2W + (c * RK_C + ci) * 9 + ky * 3;
      float x[5];
#pragma unroll
      for(int k = 0; k < 5; k++) x[k] = row[k];
#pragma unroll
      for(int kx = 0; kx < 3; kx++) {
        v0 = fmaf(w[kx], x[kx], v0);
        v1 = fmaf(w[kx], x[2 + kx], v1);
      }
    }
    A.a2[(c * RK_S2 + y) * RK_S2 + x0] = fmaxf(v0, 0.f);
    A.a2[(c * RK_S2 + y) * RK_S2 + x0 + 1] = fmaxf(v1, 0.f);
  }
  __syncthreads();
  {
    const int y = (lane >> 2) & 3, x = lane & 3, half = lane >> 4;
    float v = half ? 0.f : W[O_C3B + c];
#pragma unroll
    for(int q = 0; q < 4; q++) {
      const int ci = 4 * half + q;
      const float* w = W + O_C3W + (c * RK_C + ci) * 9;
#pragma unroll
      for(int k = 0; k < 9; k++)
        v = fmaf(w[k], A.a2[(ci * RK_S2 + y + k / 3) * RK_S2 + x + k % 3], v);
    }
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    v = fmaxf(v, 0.f);
    if(!half) A.a3[c * 16 + lane] = v;
    v = half ? 0.f : v;
    v = warpSum(v);
    if(lane == 0) A.hid[c] = v * (1.f / (RK_S3 * RK_S3));
  }
  if(c == 0) {
    float v = W[O_M1B + lane];
#pragma unroll
    for(int i = 0; i < RK_NS; i++) v = fmaf(W[O_M1W + lane * RK_NS + i], A.st[i], v);
    A.hid[RK_C + lane] = fmaxf(v, 0.f);
  }
  __syncthreads();
  if(c == 0) {
    float v = W[O_HW + lane] * A.hid[lane];
    if(lane < RK_C) v = fmaf(W[O_HW + 32 + lane], A.hid[32 + lane], v);
    v = warpSum(v);
    if(lane == 0) A.z = v + W[O_HB];
  }
  __syncthreads();
}

__device__ void rgBackward(const float* __restrict__ W, RkSample& A, float dz,
                           float* __restrict__ g) {
  const int tid = threadIdx.x, lane = tid & 31, c = tid >> 5;
  if(tid < RK_C + RK_H) {
    g[O_HW + tid] = dz * A.hid[tid];
    A.dh[tid] = dz * W[O_HW + tid];
  }
  if(tid == RK_C + RK_H) g[O_HB] = dz;
  __syncthreads();
  for(int q = tid; q < RK_H * RK_NS; q += RG_T) {
    const int j = q / RK_NS;
    g[O_M1W + q] = A.hid[RK_C + j] > 0.f ? A.dh[RK_C + j] * A.st[q % RK_NS] : 0.f;
  }
  if(tid < RK_H) g[O_M1B + tid] = A.hid[RK_C + tid] > 0.f ? A.dh[RK_C + tid] : 0.f;
  // pool -> conv3 pre-activation
  float v3 = 0.f;
  if(lane < 16) {
    v3 = A.a3[c * 16 + lane] > 0.f ? A.dh[c] * (1.f / (RK_S3 * RK_S3)) : 0.f;
    A.d3[(c * RG_P + 2 + (lane >> 2)) * RG_P + 2 + (lane & 3)] = v3;
  }
  v3 = warpSum(v3);
  if(lane == 0) g[O_C3B + c] = v3;
  __syncthreads();
  // conv3 weights: lane = (input channel, kernel row)
  if(lane < 24) {
    const int ci = lane / 3, ky = lane % 3;
    float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for(int y = 0; y < RK_S3; y++) {
      const float* d = A.d3 + (c * RG_P + 2 + y) * RG_P + 2;
      const float* row = A.a2 + (ci * RK_S2 + y + ky) * RK_S2;
      float x[6];
#pragma unroll
      for(int k = 0; k < 6; k++) x[k] = row[k];
#pragma unroll
      for(int k = 0; k < RK_S3; k++) {
        const float dv = d[k];
#pragma unroll
        for(int kx = 0; kx < 3; kx++) acc[kx] = fmaf(dv, x[k + kx], acc[kx]);
      }
    }
#pragma unroll
    for(int kx = 0; kx < 3; kx++) g[O_C3W + (c * RK_C + ci) * 9 + ky * 3 + kx] = acc[kx];
  }
  // conv2 pre-activation
  for(int o = tid; o < RK_C * RK_S2 * RK_S2; o += RG_T) {
    const int ci = o / (RK_S2 * RK_S2), yy = (o / RK_S2) % RK_S2, xx = o % RK_S2;
    float v = 0.f;
    if(A.a2[o] > 0.f)
#pragma unroll 2
      for(int cc = 0; cc < RK_C; cc++) {
        const float* w = W + O_C3W + (cc * RK_C + ci) * 9;
        const float* d = A.d3 + (cc * RG_P + 2 + yy) * RG_P + 2 + xx;
#pragma unroll
        for(int k = 0; k < 9; k++) v = fmaf(d[-(k / 3) * RG_P - k % 3], w[k], v);
      }
    A.d2[(ci * RG_P + 1 + yy) * RG_P + 1 + xx] = v;
  }
  __syncthreads();
  // conv2 weights and bias
  {
    float v = A.d2[(c * RG_P + 1 + lane / RK_S2) * RG_P + 1 + lane % RK_S2];
    if(lane < 4) v += A.d2[(c * RG_P + 6) * RG_P + 3 + lane];
    v = warpSum(v);
    if(lane == 0) g[O_C2B + c] = v;
  }
  if(lane < 24) {
    const int ci = lane / 3, ky = lane % 3;
    float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll 2
    for(int y = 0; y < RK_S2; y++) {
      const float* d = A.d2 + (c * RG_P + 1 + y) * RG_P + 1;
      const float* row = A.a1 + (ci * RK_S1 + 2 * y + ky) * RK_S1;
      float x[13];
#pragma unroll
      for(int k = 0; k < 13; k++) x[k] = row[k];
#pragma unroll
      for(int k = 0; k < RK_S2; k++) {
        const float dv = d[k];
#pragma unroll
        for(int kx = 0; kx < 3; kx++) acc[kx] = fmaf(dv, x[2 * k + kx], acc[kx]);
      }
    }
#pragma unroll
    for(int kx = 0; kx < 3; kx++) g[O_C2W + (c * RK_C + ci) * 9 + ky * 3 + kx] = acc[kx];
  }
  // conv1 pre-activation, 2 x 2 outputs per thread: with stride 2 an even row
  // (column) takes kernel rows 0 and 2, an odd one row 1
  for(int o = tid; o < RK_C * 49; o += RG_T) {
    const int ci = o / 49, by = (o / 7) % 7, bx = o % 7;
    float v00 = 0.f, v01 = 0.f, v10 = 0.f, v11 = 0.f;
#pragma unroll 2
    for(int cc = 0; cc < RK_C; cc++) {
      const float* d = A.d2 + (cc * RG_P + 1 + by) * RG_P + 1 + bx;
      const float* w = W + O_C2W + (cc * RK_C + ci) * 9;
      const float a = d[0], up = d[-RG_P], le = d[-1], ul = d[-RG_P - 1];
      v00 = fmaf(a, w[0], fmaf(up, w[6], fmaf(le, w[2], fmaf(ul, w[8], v00))));
      v01 = fmaf(a, w[1], fmaf(up, w[7], v01));
      v10 = fmaf(a, w[3], fmaf(le, w[5], v10));
      v11 = fmaf(a, w[4], v11);
    }
    const int e = (ci * RK_S1 + 2 * by) * RK_S1 + 2 * bx;
    A.d1[e] = A.a1[e] > 0.f ? v00 : 0.f;
    A.d1[e + 1] = A.a1[e + 1] > 0.f ? v01 : 0.f;
    A.d1[e + RK_S1] = A.a1[e + RK_S1] > 0.f ? v10 : 0.f;
    A.d1[e + RK_S1 + 1] = A.a1[e + RK_S1 + 1] > 0.f ? v11 : 0.f;
  }
  __syncthreads();
  // conv1 weights and bias: lane = (input channel, kernel row, third of the
  // output rows), summed over the thirds at the end
  {
    float v = 0.f;
    for(int p = lane; p < RK_S1 * RK_S1; p += 32) v += A.d1[c * RK_S1 * RK_S1 + p];
    v = warpSum(v);
    if(lane == 0) g[O_C1B + c] = v;
    const int part = lane % 3, ck = lane / 3, ci = ck / 5, ky = ck % 5;
    float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if(lane < 30)
#pragma unroll 1
      for(int y = 5 * part; y < min(5 * part + 5, RK_S1); y++) {
        const float* d = A.d1 + (c * RK_S1 + y) * RK_S1;
        const float* row = A.in + (ci * RK_WIN + 2 * y + ky) * RG_LD;
        float x[RK_WIN];
#pragma unroll
        for(int k = 0; k < RK_WIN; k++) x[k] = row[k];
#pragma unroll
        for(int k = 0; k < RK_S1; k++) {
          const float dv = d[k];
#pragma unroll
          for(int kx = 0; kx < 5; kx++) acc[kx] = fmaf(dv, x[2 * k + kx], acc[kx]);
        }
      }
#pragma unroll
    for(int kx = 0; kx < 5; kx++) {
      const float s1 = __shfl_down_sync(0xffffffffu, acc[kx], 1);
      const float s2 = __shfl_down_sync(0xffffffffu, acc[kx], 2);
      if(lane < 30 && part == 0) g[O_C1W + (c * 2 + ci) * 25 + ky * 5 + kx] = acc[kx] + s1 + s2;
    }
  }
}

__global__ void __launch_bounds__(RG_T, 4)
    k_rank_grad(const float* __restrict__ W, const float* __restrict__ stats,
                const float* __restrict__ pix, const float* __restrict__ label,
                const float* __restrict__ sweight, int n, float* __restrict__ gPer,
                float* __restrict__ loss) {
  __shared__ float Ws[RK_NP];
  __shared__ RkSample A;
  const int tid = threadIdx.x;
#pragma unroll 9
  for(int q = tid; q < RK_NP; q += RG_T) Ws[q] = rkWeight(W, q);
  for(int q = tid; q < RK_C * RG_P * RG_P; q += RG_T) A.d3[q] = A.d2[q] = 0.f;
  for(int i = blockIdx.x; i < n; i += gridDim.x) {
    __syncthreads();
#pragma unroll 8
    for(int q = tid; q < RK_PIX; q += RG_T) {
      const int r = q / RK_WIN;
      A.in[r * RG_LD + q - r * RK_WIN] = pix[(size_t)i * RK_PIX + q];
    }
    if(tid < RK_NS) A.st[tid] = stats[(size_t)i * RK_NS + tid];
    __syncthreads();
    rgForward(Ws, A);
    const float z = A.z, y = label[i], sw = sweight ? sweight[i] : 1.f;
    if(tid == 0)  // sw * BCE with logits, stable form
      loss[i] = sw * (fmaxf(z, 0.f) - z * y + log1pf(expf(-fabsf(z))));
    rgBackward(Ws, A, sw * (1.f / (1.f + expf(-z)) - y), gPer + (size_t)i * RK_NP);
  }
}

// g[p] = (sum over the samples of gPer[s][p]) * scale: 32 parameters per CTA,
// warp w sums the samples w, w + 16, ... in order and the 16 partial sums are
// added in order (one thread per parameter over all samples was bound by the
// latency of its loads: 22 us for 512 samples against 4.1 us).
constexpr int RR_W = 16;
__global__ void __launch_bounds__(32 * RR_W)
    k_rank_reduce(const float* __restrict__ gPer, int n, float scale, float* __restrict__ g) {
  __shared__ float part[RR_W][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
  float v = 0.f;
  if(p < RK_NP) {
    int s = warp;
    for(; s + 7 * RR_W < n; s += 8 * RR_W) {
      float x[8];
#pragma unroll
      for(int k = 0; k < 8; k++) x[k] = gPer[(size_t)(s + k * RR_W) * RK_NP + p];
#pragma unroll
      for(int k = 0; k < 8; k++) v += x[k];
    }
    for(; s < n; s += RR_W) v += gPer[(size_t)s * RK_NP + p];
  }
  part[warp][lane] = v;
  __syncthreads();
  if(warp == 0 && p < RK_NP) {
    v = 0.f;
#pragma unroll
    for(int k = 0; k < RR_W; k++) v += part[k][lane];
    g[p] = v * scale;
  }
}

__global__ void k_rank_adam(float* __restrict__ W, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if(p >= RK_NP) return;
  const float gp = g[p];
  const float mp = b1 * m[p] + (1.f - b1) * gp;
  const float vp = b2 * v[p] + (1.f - b2) * gp * gp;
  m[p] = mp;
  v[p] = vp;
  W[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

// ---------------------------------------------------------------- features --
// One CTA per candidate (stamp s of the set, slot k): the 16 statistics and
// the normalised window pair.  T = the template, S = the science image.
template <class T>
__global__ void __launch_bounds__(RK_T)
    k_rank_features(const T* __restrict__ imT, const T* __restrict__ imS,
                    const uint16_t* __restrict__ mask, int w, int h, const int* __restrict__ orig,
                    const int2* __restrict__ ssxy, int maxSS, const int2* __restrict__ cand,
                    int nCand, const int* __restrict__ liveN,
                    const double* __restrict__ skyT, const double* __restrict__ sigT,
                    const double* __restrict__ skyS, const double* __restrict__ sigS,
                    float threshHigh, float* __restrict__ stats, float* __restrict__ pix) {
  __shared__ float wt[RK_WIN * RK_WIN], ws[RK_WIN * RK_WIN];
  __shared__ float red[16][RK_T / 32];
  __shared__ float sh[16];
  const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if(i >= nCand) return;
  // candidates from the list, or (no list) slot i % maxSS of stamp i / maxSS,
  // whose features are zero when the slot is empty or the stamp not kept
  int s, k;
  if(cand) {
    s = cand[i].x;
    k = cand[i].y;
  } else {
    s = i / maxSS;
    k = i % maxSS;
    if((liveN && s >= *liveN) || ssxy[(size_t)s * maxSS + k].x == INT_MAX) {
      for(int q = tid; q < RK_NS; q += RK_T) stats[(size_t)i * RK_NS + q] = 0.f;
      for(int q = tid; q < RK_PIX; q += RK_T) pix[(size_t)i * RK_PIX + q] = 0.f;
      return;
    }
  }
  const int o = orig[s];
  const int2 c = ssxy[(size_t)s * maxSS + k];
  int nValid = 0;
  for(int q = 0; q < maxSS; q++) nValid += ssxy[(size_t)s * maxSS + q].x != INT_MAX;
  const float bT = (float)skyT[o], bS = (float)skyS[o];
  const float gT = fmaxf((float)sigT[o], 1e-3f), gS = fmaxf((float)sigS[o], 1e-3f);
  float acc[16];
  for(int q = 0; q < 16; q++) acc[q] = 0.f;
  float mxT = -INFINITY, mxS = -INFINITY, rawMax = -INFINITY;
  for(int p = tid; p < RK_WIN * RK_WIN; p += RK_T) {
    const int dx = p % RK_WIN - RK_HWIN, dy = p / RK_WIN - RK_HWIN;
    const int gx = min(max(c.x + dx, 0), w - 1), gy = min(max(c.y + dy, 0), h - 1);
    const size_t gi = (size_t)gx + (size_t)gy * w;
    const float vT = (float)imT[gi], vS = (float)imS[gi];
    rawMax = fmaxf(rawMax, fmaxf(vT, vS));
    const float a = vT - bT, b = vS - bS;
    wt[p] = a;
    ws[p] = b;
    mxT = fmaxf(mxT, a);
    mxS = fmaxf(mxS, b);
    const float ap = fmaxf(a, 0.f), bp = fmaxf(b, 0.f), r2 = (float)(dx * dx + dy * dy);
    acc[0] += a;                     // flux T
    acc[1] += b;                     // flux S
    acc[2] += (mask[gi] & (BAD_INPUT | BAD_PIXEL_T | BAD_PIXEL_S | NAN_PIXEL)) ? 1.f : 0.f;
    acc[3] += ap;
    acc[4] += ap * r2;
    acc[5] += ap * dx;
    acc[6] += ap * dy;
    acc[7] += bp;
    acc[8] += bp * r2;
    acc[9] += bp * dx;
    acc[10] += bp * dy;
    acc[11] += a * b;
    acc[12] += a * a;
    acc[13] += b * b;
    acc[14] += (a > 20.f * gT) ? 1.f : 0.f;
  }
  // block reductions: sums 0..14 and the T peak into red[]; the S peak and
  // the raw maximum into mx2[]
  for(int q = 0; q < 15; q++) {
    float v = acc[q];
#pragma unroll
    for(int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if(lane == 0) red[q][warp] = v;
  }
  float m3[3] = {mxT, mxS, rawMax};
  for(int q = 0; q < 3; q++) {
#pragma unroll
    for(int off = 16; off > 0; off >>= 1) m3[q] = fmaxf(m3[q], __shfl_xor_sync(0xffffffffu, m3[q], off));
  }
  __shared__ float mx2[2][RK_T / 32];
  if(lane == 0) {
    red[15][warp] = m3[0];
    mx2[0][warp] = m3[1];
    mx2[1][warp] = m3[2];
  }
  __syncthreads();
  if(tid < 16) {
    float v = tid == 15 ? -INFINITY : 0.f;
    for(int q = 0; q < RK_T / 32; q++) v = tid == 15 ? fmaxf(v, red[15][q]) : v + red[tid][q];
    sh[tid] = v;
  }
  __syncthreads();
  float pS = -INFINITY, rmax = -INFINITY;
  for(int q = 0; q < RK_T / 32; q++) {
    pS = fmaxf(pS, mx2[0][q]);
    rmax = fmaxf(rmax, mx2[1][q]);
  }
  const float pT = sh[15];
  // sharpness: largest excess of a pixel over its 4-neighbour mean (cosmic rays)
  float sharp = 0.f;
  for(int p = tid; p < RK_WIN * RK_WIN; p += RK_T) {
    const int x = p % RK_WIN, y = p / RK_WIN;
    if(x == 0 || y == 0 || x == RK_WIN - 1 || y == RK_WIN - 1) continue;
    const float nT = 0.25f * (wt[p - 1] + wt[p + 1] + wt[p - RK_WIN] + wt[p + RK_WIN]);
    const float nS = 0.25f * (ws[p - 1] + ws[p + 1] + ws[p - RK_WIN] + ws[p + RK_WIN]);
    sharp = fmaxf(sharp, fmaxf((wt[p] - nT) / (fabsf(pT) + gT), (ws[p] - nS) / (fabsf(pS) + gS)));
  }
#pragma unroll
  for(int off = 16; off > 0; off >>= 1) sharp = fmaxf(sharp, __shfl_xor_sync(0xffffffffu, sharp, off));
  __shared__ float shp[RK_T / 32];
  if(lane == 0) shp[warp] = sharp;
  // normalised window pair
  const float nT = 1.f / (fmaxf(pT, 0.f) + gT), nS = 1.f / (fmaxf(pS, 0.f) + gS);
  for(int p = tid; p < RK_WIN * RK_WIN; p += RK_T) {
    pix[(size_t)i * RK_PIX + p] = fminf(fmaxf(wt[p] * nT, -1.f), 2.f);
    pix[(size_t)i * RK_PIX + RK_WIN * RK_WIN + p] = fminf(fmaxf(ws[p] * nS, -1.f), 2.f);
  }
  __syncthreads();
  if(tid == 0) {
    float shv = 0.f;
    for(int q = 0; q < RK_T / 32; q++) shv = fmaxf(shv, shp[q]);
    const float fT = sh[0], fS = sh[1], npx = (float)(RK_WIN * RK_WIN);
    const float momT = sh[4] / fmaxf(sh[3], 1e-20f), momS = sh[8] / fmaxf(sh[7], 1e-20f);
    float* f = stats + (size_t)i * RK_NS;
    f[0] = asinhf(pT / gT) * 0.125f;
    f[1] = asinhf(pS / gS) * 0.125f;
    f[2] = asinhf(fT / (gT * RK_WIN)) * 0.125f;
    f[3] = asinhf(fS / (gS * RK_WIN)) * 0.125f;
    f[4] = sh[2] / npx;
    f[5] = logf((momS + 1.f) / (momT + 1.f));
    f[6] = sh[5] / fmaxf(sh[3], 1e-20f) / RK_HWIN;
    f[7] = sh[6] / fmaxf(sh[3], 1e-20f) / RK_HWIN;
    f[8] = sh[9] / fmaxf(sh[7], 1e-20f) / RK_HWIN;
    f[9] = sh[10] / fmaxf(sh[7], 1e-20f) / RK_HWIN;
    f[10] = sh[11] / sqrtf(fmaxf(sh[12] * sh[13], 1e-30f));
    f[11] = (fS - fT) / (fabsf(fS) + fabsf(fT) + npx * (gT + gS));
    f[12] = (float)k / maxSS;
    f[13] = (float)nValid / maxSS;
    f[14] = rmax / threshHigh;
    f[15] = fminf(shv, 4.f);
  }
}

// The learned order of each kept stamp's candidates (one thread per stamp):
// the valid slots (a prefix of the stamp's maxSS slots) are reordered by
// their scores z, policy 1 moving those below zTau behind the others (each
// group in the reference's order), policy 2 sorting all by descending score
// (ties in the reference's order).
// Reorders the first nRank candidates of every stamp by score (the others
// keep their places after them).
__global__ void k_rank_order(int2* __restrict__ ssxy, double* __restrict__ ssval,
                             const float* __restrict__ z, int nBound,
                             const int* __restrict__ liveN, int maxSS, int nRank, int policy,
                             float zTau) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = liveN ? min(*liveN, nBound) : nBound;
  if(s >= n) return;
  int2 xy[MAX_MAXSS];
  double v[MAX_MAXSS];
  float sc[MAX_MAXSS];
  int order[MAX_MAXSS];
  int cnt = 0;
  for(int k = 0; k < maxSS; k++) {
    xy[k] = ssxy[(size_t)s * maxSS + k];
    v[k] = ssval[(size_t)s * maxSS + k];
    if(xy[k].x != INT_MAX && k < nRank) {
      sc[cnt] = z[(size_t)s * maxSS + k];
      order[cnt++] = k;
    }
  }
  if(policy == 2) {
    for(int a = 1; a < cnt; a++)  // stable insertion sort, descending
      for(int b = a; b > 0 && sc[b - 1] < sc[b]; b--) {
        const float t = sc[b - 1];
        sc[b - 1] = sc[b];
        sc[b] = t;
        const int u = order[b - 1];
        order[b - 1] = order[b];
        order[b] = u;
      }
  } else {
    int tmp[MAX_MAXSS], m = 0;
    for(int a = 0; a < cnt; a++)
      if(sc[a] >= zTau) tmp[m++] = order[a];
    for(int a = 0; a < cnt; a++)
      if(!(sc[a] >= zTau)) tmp[m++] = order[a];
    for(int a = 0; a < cnt; a++) order[a] = tmp[a];
  }
  for(int r = 0; r < cnt; r++) {
    ssxy[(size_t)s * maxSS + r] = xy[order[r]];
    ssval[(size_t)s * maxSS + r] = v[order[r]];
  }
}

}  // namespace

constexpr int kRankParams = RK_NP;

// Candidate list (stamp, slot) of set si: every valid substamp slot.
static int rankCandidates(xb_ctx* c, int si, std::vector<int2>& cand) {
  const Geo& g = c->g;
  StampSetDev& S = c->set[si];
  cand.clear();
  if(S.n <= 0) return 0;
  std::vector<int2> xy = toHost(c, S.ssxy, (size_t)S.n * g.maxSS);
  for(int s = 0; s < S.n; s++)
    for(int k = 0; k < g.maxSS; k++)
      if(xy[(size_t)s * g.maxSS + k].x != INT_MAX) cand.push_back(make_int2(s, k));
  return (int)cand.size();
}

// Features of every candidate of set si into device buffers (stats, pix).
static void rankFeatures(xb_ctx* c, int si, const std::vector<int2>& cand, float* dStats,
                         float* dPix) {
  const Geo& g = c->g;
  StampSetDev& S = c->set[si];
  const int n = (int)cand.size();
  if(n == 0) return;
  int2* dCand = buf<int2>(c, "rank_cand", n);
  toDevice(c, dCand, cand);
  if(c->imgIsF64)
    k_rank_features<double><<<n, RK_T, 0, c->stream>>>(
        (const double*)c->img[0], (const double*)c->img[1], c->mask, c->w, c->h, S.orig, S.ssxy,
        g.maxSS, dCand, n, nullptr, c->skyAll[0], c->fwhmAll[0], c->skyAll[1], c->fwhmAll[1],
        (float)c->p.threshHigh, dStats, dPix);
  else
    k_rank_features<float><<<n, RK_T, 0, c->stream>>>(
        (const float*)c->img[0], (const float*)c->img[1], c->mask, c->w, c->h, S.orig, S.ssxy,
        g.maxSS, dCand, n, nullptr, c->skyAll[0], c->fwhmAll[0], c->skyAll[1], c->fwhmAll[1],
        (float)c->p.threshHigh, dStats, dPix);
  XB_LAUNCHED(c);
}

// Reorders the valid substamp slots of every stamp of both sets; counts are
// unchanged.  Called after sss when a ranker is loaded and the "rank" option
// is on.  rank = 1: candidates whose accept probability is below the
// threshold (option "rank_tau", in thousandths) move behind the others, each
// group keeping the reference's order; rank = 2: all by descending score.
// Everything runs on the device (features of every slot, scores, the
// per-stamp reorder), so a frame graph captures it; S.dN, when set, holds the
// kept count and S.n bounds it.
void rankSubstamps(xb_ctx* c) {
  const float tau = c->rankTau / 1000.f;
  const float zTau = logf(tau / (1.f - tau));  // logit of the threshold
  const Geo& g = c->g;
  for(int si = 0; si < 2; si++) {
    StampSetDev& S = c->set[si];
    if(S.n <= 0) continue;
    const int n = S.n * g.maxSS;
    float* dStats = buf<float>(c, "rank_stats", (size_t)n * RK_NS);
    float* dPix = buf<float>(c, "rank_pix", (size_t)n * RK_PIX);
    float* dLogit = buf<float>(c, "rank_logit", n);
    const int nRank = c->rankCandidates > 0 ? std::min(c->rankCandidates, g.maxSS) : g.maxSS;
    if(c->imgIsF64)
      k_rank_features<double><<<n, RK_T, 0, c->stream>>>(
          (const double*)c->img[0], (const double*)c->img[1], c->mask, c->w, c->h, S.orig,
          S.ssxy, g.maxSS, nullptr, n, S.dN, c->skyAll[0], c->fwhmAll[0], c->skyAll[1],
          c->fwhmAll[1], (float)c->p.threshHigh, dStats, dPix);
    else
      k_rank_features<float><<<n, RK_T, 0, c->stream>>>(
          (const float*)c->img[0], (const float*)c->img[1], c->mask, c->w, c->h, S.orig,
          S.ssxy, g.maxSS, nullptr, n, S.dN, c->skyAll[0], c->fwhmAll[0], c->skyAll[1],
          c->fwhmAll[1], (float)c->p.threshHigh, dStats, dPix);
    XB_LAUNCHED(c);
    {
      KT_SCOPE(c, "rank_score");
      XB_CUDA(allowMaxDynamicSmem((const void*)k_rank_forward<__nv_bfloat16>, c->device));
      k_rank_forward<__nv_bfloat16>
          <<<std::min((n + RF_SAMPLES - 1) / RF_SAMPLES, c->smCount * 3), RF_T, RF_SMEM,
             c->stream>>>((const __nv_bfloat16*)c->rankW, dStats, dPix, n, dLogit, S.ssxy, g.maxSS,
                          nRank, S.dN);
      XB_LAUNCHED(c);
    }
    k_rank_order<<<(S.n + 127) / 128, 128, 0, c->stream>>>(S.ssxy, S.ssval, dLogit, S.n, S.dN,
                                                           g.maxSS, nRank, c->rank, zTau);
    XB_LAUNCHED(c);
  }
}

}  // namespace xb

using namespace xb;

namespace {
template <class F>
int rkGuard(xb_ctx* c, F&& f) {
  try {
    f();
    return XB_OK;
  } catch(const CudaError& e) {
    if(c) c->lastError = std::string(e.where) + ": " + cudaGetErrorString(e.code);
    return XB_ERR_CUDA;
  } catch(const XbError& e) {
    if(c) c->lastError = e.msg;
    return e.code;
  }
}
cudaError_t rkLaunched() { return cudaGetLastError(); }
}  // namespace

extern "C" {

int xb_ranker_param_count(void) { return kRankParams; }

int xb_ranker_set(xb_ctx* c, const float* weights, int n) {
  if(!c) return XB_ERR_ARG;
  return rkGuard(c, [&] {
    if(n != kRankParams || !weights) throw XbError{XB_ERR_ARG, "ranker weights: wrong count"};
    XB_CUDA(cudaSetDevice(c->device));
    // stored as BF16 (nearest, ties to even), the weights the network computes with
    std::vector<uint16_t> wb(kRankParams);
    for(int q = 0; q < kRankParams; q++) {
      uint32_t u;
      memcpy(&u, &weights[q], 4);
      if((u & 0x7F800000u) == 0x7F800000u && (u & 0x7FFFFFu)) wb[q] = (uint16_t)((u >> 16) | 0x40u);
      else wb[q] = (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
    }
    c->rankW = buf<uint16_t>(c, "rank_weights", kRankParams);
    XB_CUDA(cudaMemcpyAsync(c->rankW, wb.data(), sizeof(uint16_t) * kRankParams,
                            cudaMemcpyHostToDevice, c->stream));
    XB_CUDA(cudaStreamSynchronize(c->stream));
  });
}

int xb_ranker_features(xb_ctx* c, int set, float* stats, float* pix, int* stamp, int* slot,
                       int cap, int* nOut) {
  if(!c || set < 0 || set > 1 || !nOut) return XB_ERR_ARG;
  return rkGuard(c, [&] {
    XB_CUDA(cudaSetDevice(c->device));
    if(c->stage < 2) throw XbError{XB_ERR_STATE, "ranker features need sss first"};
    std::vector<int2> cand;
    const int n = rankCandidates(c, set, cand);
    *nOut = n;
    if(!stats && !pix && !stamp && !slot) return;
    if(n > cap) throw XbError{XB_ERR_ARG, "ranker features: capacity too small"};
    float* dStats = buf<float>(c, "rank_stats", (size_t)std::max(n, 1) * RK_NS);
    float* dPix = buf<float>(c, "rank_pix", (size_t)std::max(n, 1) * RK_PIX);
    rankFeatures(c, set, cand, dStats, dPix);
    if(stats)
      XB_CUDA(cudaMemcpyAsync(stats, dStats, sizeof(float) * n * RK_NS, cudaMemcpyDeviceToHost,
                              c->stream));
    if(pix)
      XB_CUDA(cudaMemcpyAsync(pix, dPix, sizeof(float) * (size_t)n * RK_PIX,
                              cudaMemcpyDeviceToHost, c->stream));
    XB_CUDA(cudaStreamSynchronize(c->stream));
    for(int i = 0; i < n; i++) {
      if(stamp) stamp[i] = cand[i].x;
      if(slot) slot[i] = cand[i].y;
    }
  });
}

int xb_ranker_forward(const float* dW, const float* dStats, const float* dPix, int n,
                      float* dLogit, void* stream) {
  if(n < 0 || (n > 0 && (!dW || !dStats || !dPix || !dLogit))) return XB_ERR_ARG;
  if(n == 0) return XB_OK;
  int device = 0, sms = 0;
  if(cudaGetDevice(&device) != cudaSuccess ||
     cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
     allowMaxDynamicSmem((const void*)k_rank_forward<float>, device) != cudaSuccess)
    return XB_ERR_CUDA;
  k_rank_forward<float><<<std::min((n + RF_SAMPLES - 1) / RF_SAMPLES, sms * 3), RF_T, RF_SMEM,
                          (cudaStream_t)stream>>>(dW, dStats, dPix, n, dLogit);
  return rkLaunched() == cudaSuccess ? XB_OK : XB_ERR_CUDA;
}

int xb_ranker_grad(const float* dW, const float* dStats, const float* dPix, const float* dLabel,
                   const float* dWeight, int n, float* dGradPerSample, float* dGrad,
                   float* dLoss, void* stream) {
  if(n <= 0 || !dW || !dStats || !dPix || !dLabel || !dGradPerSample || !dGrad || !dLoss)
    return XB_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  k_rank_grad<<<std::min(n, 4096), RG_T, 0, st>>>(dW, dStats, dPix, dLabel, dWeight, n,
                                                  dGradPerSample, dLoss);
  if(rkLaunched() != cudaSuccess) return XB_ERR_CUDA;
  k_rank_reduce<<<(RK_NP + 31) / 32, 32 * RR_W, 0, st>>>(dGradPerSample, n, 1.f / n, dGrad);
  return rkLaunched() == cudaSuccess ? XB_OK : XB_ERR_CUDA;
}

int xb_ranker_adam(float* dW, const float* dGrad, float* dM, float* dV, int step, float lr,
                   void* stream) {
  if(!dW || !dGrad || !dM || !dV || step < 1) return XB_ERR_ARG;
  const float b1 = 0.9f, b2 = 0.999f;
  k_rank_adam<<<(RK_NP + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
      dW, dGrad, dM, dV, lr, b1, b2, 1e-8f, 1.f - powf(b1, (float)step), 1.f - powf(b2, (float)step));
  return rkLaunched() == cudaSuccess ? XB_OK : XB_ERR_CUDA;
}

}  // extern "C"
