// xb_ctx.cu — context lifetime, basis tables and the init stage.
//
// init (src/bach.cpp:14-42): the images are uploaded once and the mask is
// built by two streaming kernels, maskInput (cl_kern/ini.cl:15-35) and
// spreadMask (cl_kern/ini.cl:37-67).

#include <algorithm>
#include <cmath>
#include <cstring>

#include <mutex>
#include <set>
#include <utility>

#include "xb_internal.h"

namespace xb {

Geo makeGeo(const xb_params& p) {
  Geo g{};
  g.hSS = p.hSStampWidth;
  g.fSS = 2 * g.hSS + 1;
  g.hK = p.hKernelWidth;
  g.fK = 2 * g.hK + 1;
  g.nPSF = xb_params_npsf(&p);
  g.nComp1 = g.nPSF - 1;
  g.nComp2 = triNum(p.kernelOrder + 1);
  g.nComp = g.nComp1 * g.nComp2;
  g.nBG = triNum(p.backgroundOrder + 1);
  g.matSize = g.nComp + g.nBG + 1;
  g.nSol = g.nPSF * g.nComp2 + g.nBG + 1;
  g.wRows = g.nPSF + g.nBG;
  g.wCols = g.fSS * g.fSS;
  g.qCount = g.nPSF + 2;
  g.bCount = g.nPSF + 2;
  g.maxSS = 2 * p.maxKSStamps;
  return g;
}

// pown(x, n) of the OpenCL kernels, evaluated as 1*x*x*... (the form the
// host loops of src/cdkscUtil.cpp:334-342 use).
static double ipowHost(double x, int n) {
  double r = 1.0;
  for(int i = 0; i < n; i++) r *= x;
  return r;
}

Basis buildBasis(const xb_params& p, const Geo& g) {
  Basis b;
  const int fK = g.fK, hK = g.hK;
  // enumeration order of src/bach.cpp:181-188: Gaussian, x degree, y degree
  for(int gs = 0; gs < p.nGauss; gs++)
    for(int x = 0; x <= p.dg[gs]; x++)
      for(int y = 0; y <= p.dg[gs] - x; y++) {
        b.gauss.push_back(gs);
        b.kx.push_back(x);
        b.ky.push_back(y);
      }
  const int nPSF = (int)b.kx.size();
  b.fX.assign((size_t)nPSF * fK, 0.0);
  b.fY.assign((size_t)nPSF * fK, 0.0);
  for(int n = 0; n < nPSF; n++) {
    const double bw = (double)p.bg[b.gauss[n]];  // float width, as the reference
    double sx = 0.0, sy = 0.0;
    for(int i = 0; i < fK; i++) {
      const double x = (double)(i - hK);
      const double qe = std::exp(-x * x * bw);
      const double fx = qe * ipowHost(x, b.kx[n]);
      const double fy = qe * ipowHost(x, b.ky[n]);
      b.fX[(size_t)n * fK + i] = fx;
      b.fY[(size_t)n * fK + i] = fy;
      sx += fx;
      sy += fy;
    }
    if(b.kx[n] % 2 == 0 && b.ky[n] % 2 == 0) {  // normalise even/even filters
      const double ix = 1.0 / sx, iy = 1.0 / sy;
      for(int i = 0; i < fK; i++) {
        b.fX[(size_t)n * fK + i] *= ix;
        b.fY[(size_t)n * fK + i] *= iy;
      }
    }
  }
  b.vec.assign((size_t)nPSF * fK * fK, 0.0);
  for(int n = 0; n < nPSF; n++)
    for(int v = 0; v < fK; v++)
      for(int u = 0; u < fK; u++) {
        double vv = b.fX[(size_t)n * fK + u] * b.fY[(size_t)n * fK + v];
        if(b.kx[n] % 2 == 0 && b.ky[n] % 2 == 0 && n > 0) vv -= b.fX[u] * b.fY[v];
        b.vec[(size_t)n * fK * fK + (size_t)v * fK + u] = vv;
      }
  for(int x = 0; x <= p.backgroundOrder; x++)
    for(int y = 0; y <= p.backgroundOrder - x; y++) {
      b.bgX.push_back(x);
      b.bgY.push_back(y);
    }
  for(int i = 0; i <= p.kernelOrder; i++)
    for(int j = 0; j <= p.kernelOrder - i; j++) {
      b.kpX.push_back(i);
      b.kpY.push_back(j);
    }
  // Group basis functions whose Y filters are bit-identical: the Y pass of
  // the substamp convolution (cl_kern/cmv.cl:70-106) depends only on the Y
  // filter, so one pass serves the whole group with identical results.
  std::vector<int> groupOf(nPSF, -1);
  std::vector<std::vector<int>> groups;
  for(int n = 0; n < nPSF; n++) {
    for(size_t gi = 0; gi < groups.size(); gi++) {
      int m = groups[gi][0];
      if(memcmp(&b.fY[(size_t)m * fK], &b.fY[(size_t)n * fK], sizeof(double) * fK) == 0) {
        groupOf[n] = (int)gi;
        groups[gi].push_back(n);
        break;
      }
    }
    if(groupOf[n] < 0) {
      groupOf[n] = (int)groups.size();
      groups.push_back({n});
    }
  }
  b.yGroupStart.push_back(0);
  for(auto& gr : groups) {
    for(int n : gr) b.yGroupMembers.push_back(n);
    b.yGroupStart.push_back((int)b.yGroupMembers.size());
  }
  return b;
}

cudaError_t allowMaxDynamicSmem(const void* func, int device) {
  // once per (function, device): the attribute outlives the call
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  {
    std::lock_guard<std::mutex> l(mu);
    if(done.count({func, device})) return cudaSuccess;
  }
  int optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if(e != cudaSuccess) return e;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, func);
  if(e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           optin - (int)fa.sharedSizeBytes);
  if(e == cudaSuccess) {
    std::lock_guard<std::mutex> l(mu);
    done.insert({func, device});
  }
  return e;
}

void* poolGet(xb_ctx* c, const char* name, size_t bytes) {
  DevBuf& b = c->pool[name];
  if(b.bytes >= bytes) return b.p;
  if(b.p) {
    if(c->keepBuffers) {
      // a captured frame graph may still address it: freed with the context
      c->retired.push_back(b.p);
    } else {
      XB_CUDA(cudaStreamSynchronize(c->stream));
      cudaFree(b.p);
    }
    b.p = nullptr;
    b.bytes = 0;
  }
  void* p = nullptr;
  if(cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();
    throw XbError{XB_ERR_NOMEM, std::string("cudaMalloc failed for ") + name};
  }
  b.p = p;
  b.bytes = bytes;
  return p;
}

SideWork::SideWork(xb_ctx* c) : c_(c), main_(c->stream) {
  if(!c->sideStream) XB_CUDA(cudaStreamCreateWithFlags(&c->sideStream, cudaStreamNonBlocking));
  if(!c->sideFork) XB_CUDA(cudaEventCreateWithFlags(&c->sideFork, cudaEventDisableTiming));
  if(!c->sideJoin) XB_CUDA(cudaEventCreateWithFlags(&c->sideJoin, cudaEventDisableTiming));
  XB_CUDA(cudaEventRecord(c->sideFork, main_));
}
void SideWork::enter() {
  XB_CUDA(cudaStreamWaitEvent(c_->sideStream, c_->sideFork, 0));
  c_->stream = c_->sideStream;
  c_->lane = 1;
  in_ = used_ = true;
}
void SideWork::leave() {
  c_->stream = main_;
  c_->lane = 0;
  in_ = false;
}
void SideWork::join() {
  if(in_) leave();
  if(used_ && !joined_) {
    joined_ = true;
    XB_CUDA(cudaEventRecord(c_->sideJoin, c_->sideStream));
    XB_CUDA(cudaStreamWaitEvent(main_, c_->sideJoin, 0));
  }
}
SideWork::~SideWork() {
  if(in_) leave();
  if(used_ && !joined_) {  // an error on the way: the main stream still waits
    cudaEventRecord(c_->sideJoin, c_->sideStream);
    cudaStreamWaitEvent(main_, c_->sideJoin, 0);
  }
}

cudaEvent_t ktEvent(xb_ctx* c) {
  if(!c->kt.pool.empty()) {
    cudaEvent_t e = c->kt.pool.back();
    c->kt.pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  XB_CUDA(cudaEventCreate(&e));
  return e;
}

void ktCollect(xb_ctx* c) {
  if(c->kt.pending.empty()) return;
  XB_CUDA(cudaStreamSynchronize(c->stream));
  for(auto& o : c->kt.pending) {
    float ms = 0.f;
    XB_CUDA(cudaEventElapsedTime(&ms, o.a, o.b));
    auto& t = c->kt.total[o.name];
    t.first += ms;
    t.second += 1;
    c->kt.pool.push_back(o.a);
    c->kt.pool.push_back(o.b);
  }
  c->kt.pending.clear();
}

// ---------------------------------------------------------------- kernels --

// maskInput (cl_kern/ini.cl:15-35) and the caller's input mask; a warp takes 256
// pixels of a row, 32 neighbours at a time, and a ballot of each 32 is a word of
// the BAD_INPUT bit rows.  Bound by HBM: both images in, the mask out.  FP32
// pixels are compared with the thresholds rounded outward to float (t >= tH is
// t >= the smallest float not below tH), without an FP64 operation.
// 4096 x 4096: 43 us of 24 at the measured copy rate (FP64 comparisons and a
// division per pixel: 192).
template <class T>
__global__ void __launch_bounds__(256)
    k_mask_input(const T* __restrict__ tImg, const T* __restrict__ sImg,
                 const uint8_t* __restrict__ in, uint16_t* __restrict__ mask,
                 unsigned* __restrict__ badBits, int wpr, int w, int h, int border, double tH,
                 double tL) {
  const int lane = threadIdx.x & 31, x0 = blockIdx.x * 256;
  const T hi = sizeof(T) == 4 ? (T)__double2float_ru(tH) : (T)tH;
  const T lo = sizeof(T) == 4 ? (T)__double2float_rd(tL) : (T)tL;
  for(int y = blockIdx.y * 8 + (threadIdx.x >> 5); y < h; y += gridDim.y * 8) {
    const size_t row = (size_t)y * w;
    const bool yEdge = y < border || y >= h - border;
    T t[8], s[8];
    uint8_t im[8];
#pragma unroll
    for(int k = 0; k < 8; k++) {
      const int x = x0 + 32 * k + lane;
      t[k] = x < w ? tImg[row + x] : T(0);
      s[k] = x < w ? sImg[row + x] : T(0);
      im[k] = in && x < w ? in[row + x] : (uint8_t)0;
    }
#pragma unroll
    for(int k = 0; k < 8; k++) {
      const int x = x0 + 32 * k + lane;
      uint16_t m = 0;
      if(t[k] == T(0) || s[k] == T(0)) m |= BAD_INPUT | BAD_PIX_VAL;
      if(t[k] >= hi || s[k] >= hi) m |= BAD_INPUT | SAT_PIXEL;
      if(t[k] <= lo || s[k] <= lo) m |= BAD_INPUT | LOW_PIXEL;
      if(yEdge || x < border || x >= w - border) m |= BAD_PIXEL_S | BAD_PIXEL_T;
      if(im[k]) m |= INPUT_MASK | BAD_INPUT;
      const unsigned bad = __ballot_sync(0xffffffffu, x < w && (m & BAD_INPUT));
      if(x < w) mask[row + x] = m;
      if(lane == 0 && x0 + 32 * k < w) badBits[(size_t)y * wpr + (x0 >> 5) + k] = bad;
    }
  }
}

// spreadMask (cl_kern/ini.cl:37-67): OK_CONV on every pixel without
// BAD_INPUT that has a BAD_INPUT pixel within +-r (clipped to the frame).  A
// lane takes a word of 32 pixels: the rows within r are ORed word by word, the
// word's own bits are widened by shifts, and of a word further left (right)
// only the last (first) bit matters.  Where words have pixels to mark, the warp
// does so word by word.  4096 x 4096: 30 us (a byte per pixel of a tile and
// its halo from the mask: 110).
__global__ void __launch_bounds__(256)
    k_spread_mask(const unsigned* __restrict__ badBits, int wpr, uint16_t* __restrict__ mask, int w,
                  int h, int r) {
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * 256 + threadIdx.x;  // word of the row
  const int reach = (r + 31) / 32;
  for(int y = blockIdx.y; y < h; y += gridDim.y) {
    unsigned out = 0;
    if(k < wpr) {
      const int ya = max(y - r, 0), yb = min(y + r, h - 1);
      auto column = [&](int word) {  // the bits of a word within r rows
        unsigned v = 0;
        if(word >= 0 && word < wpr)
#pragma unroll 4
          for(int yy = ya; yy <= yb; yy++) v |= badBits[(size_t)yy * wpr + word];
        return v;
      };
      unsigned v = column(k);
      for(int left = r; left > 0 && v;) {  // v | v shifted by 1..r either way
        const int step = min(left, 31);
        unsigned a = v;
        for(int done = 0; done < step;) {
          const int sh = min(done + 1, step - done);
          a |= a << sh | a >> sh;
          done += sh;
        }
        v = a;
        left -= step;
      }
      out = v;
      for(int d = 1; d <= reach; d++) {
        const unsigned a = column(k - d), b = column(k + d);
        if(a) {  // its last bit p reaches the bits up to p + r - 32 d
          const int n = 31 - __clz(a) + r - 32 * d + 1;
          if(n > 0) out |= n >= 32 ? 0xFFFFFFFFu : (1u << n) - 1u;
        }
        if(b) {  // its first bit p reaches the bits from 32 d + p - r
          const int n = 32 * d + __ffs(b) - 1 - r;
          if(n < 32) out |= n <= 0 ? 0xFFFFFFFFu : ~((1u << n) - 1u);
        }
      }
      out &= ~badBits[(size_t)y * wpr + k];
      if(32 * k + 32 > w) out &= (1u << (w - 32 * k)) - 1u;
    }
    for(unsigned any = __ballot_sync(0xffffffffu, out != 0); any; any &= any - 1) {
      const int l = __ffs(any) - 1;
      const unsigned o = __shfl_sync(0xffffffffu, out, l);
      const size_t at = (size_t)y * w + 32 * (size_t)(k - lane + l) + lane;
      if(o >> lane & 1u) mask[at] |= OK_CONV;
    }
  }
}

void stageInitMask(xb_ctx* c) {
  const int border = c->p.hSStampWidth + c->p.hKernelWidth;
  if(c->inputMask && (c->inputMaskW != c->w || c->inputMaskH != c->h))
    throw XbError{XB_ERR_SIZE_MISMATCH, "input mask and frame differ in size"};
  const int wpr = (c->w + 31) / 32;
  unsigned* bad = buf<unsigned>(c, "bad_bits", (size_t)wpr * c->h);
  { KT_SCOPE(c, "mask_input");
  const dim3 grid((c->w + 255) / 256, std::min((c->h + 7) / 8, 65535));
  auto launch = [&](auto* t, auto* s) {
    k_mask_input<<<grid, 256, 0, c->stream>>>(t, s, c->inputMask, c->mask, bad, wpr, c->w, c->h,
                                              border, c->p.threshHigh, c->p.threshLow);
  };
  if(c->imgIsF64) launch((const double*)c->img[0], (const double*)c->img[1]);
  else launch((const float*)c->img[0], (const float*)c->img[1]);
  XB_LAUNCHED(c);
  }
  const int spreadWidth = (int)(c->p.hKernelWidth * c->p.inSpreadMaskFactor);
  const int r = spreadWidth / 2;
  if(r > 0) {
    // spreads of more than 78 pixels are refused, by the interface: the kernel has no
    // bound of its own (a byte per pixel of a 64 x 16 tile with its halo, and of the
    // halo's rows, within 48 KB)
    if((64ll + 2 * r) * (16 + 2 * r) + (16ll + 2 * r) * 64 > 48 * 1024)
      throw XbError{XB_ERR_CUDA, "input mask spread too wide"};
    KT_SCOPE(c, "spread_mask");
    k_spread_mask<<<dim3((wpr + 255) / 256, std::min(c->h, 65535)), 256, 0, c->stream>>>(bad, wpr, c->mask, c->w,
                                                                         c->h, r);
    XB_LAUNCHED(c);
  }
}

}  // namespace xb
