// SSIM / MS-SSIM of two device planes without allocating any device memory
// (rg_ssim_plane_device_noalloc in include/ragdoll_cuda.h).
//
// Who needs this: callers that are not allowed to call cudaMalloc / cudaFree at the time they
// measure quality -- a frame loop with a fixed memory budget whose device memory is already
// reserved by another allocator (a framework's caching pool), or a latency-critical loop where
// an allocation would synchronise the device and stall the other streams. They pass the two
// planes and a two-double output buffer that they own; the working memory (the 2x2-decimated
// pyramid and the per-row sums) lives in one file-scope __device__ array instead.
//
// That array is shared by every call on a device and keeps the last call's contents; nothing in
// it has to start at zero (every byte read is written first by the same call). Calls that
// overlap on the GPU (on different streams, or on different host threads) race on it and must
// be serialised by the caller. Its size bounds the planes: width and height 8..4096 and at most
// 1920 x 1088 samples.
//
// The arithmetic is that of the allocating path (ssim_rows.cuh), and the 5-scale product of
// crates/ragdoll-pix/src/metrics.rs:154, here evaluated on the device.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "../../include/ragdoll_cuda.h"

namespace rg {
void set_last_error(const char* msg);
}

namespace {

constexpr long kNaMaxPixels = 1920L * 1088L;
constexpr int kNaMaxDim = 4096;
// pyramid rows are padded to whole words: up to 3 bytes each, 2 x (2048 + 1024 + 512 + 256) rows
constexpr size_t kNaPyrBytes =
    2 * (kNaMaxPixels / 4 + kNaMaxPixels / 16 + kNaMaxPixels / 64 + kNaMaxPixels / 256) + 2 * 3 * (kNaMaxDim / 2) * 2 + 4096;
constexpr size_t kNaRowFloats = 2 * (kNaMaxDim / 4) + 64;
constexpr size_t kNaScratchBytes = kNaPyrBytes + kNaRowFloats * sizeof(float) + 16 * sizeof(double);

// The working memory of every call on this device: pyramid planes, then row sums, then the five
// per-scale SSIM values.
__device__ __align__(256) uint8_t g_noalloc_scratch[kNaScratchBytes];

#include "ssim_rows.cuh"

template <bool kPyramid>
__global__ void __launch_bounds__(kRowThreads) na_rows_kernel(const __grid_constant__ SsimPair p) {
  ssim_pass<kPyramid, kFlatStrip, kFlatChunk>(p);
}
// A warp per scale (its sum, then its factor of the product), and the product in the scales' order.
__global__ void __launch_bounds__(160) na_finish_kernel(const __grid_constant__ SsimPair p) {
  __shared__ float stage[5][128];
  __shared__ double factor[5];
  const double w5[5] = {0.0448, 0.2856, 0.3001, 0.2363, 0.1333};
  const int warp = threadIdx.x >> 5;
  if (warp < p.levels) {
    const double s = ssim_total(p.lv[warp], stage[warp]);
    if ((threadIdx.x & 31) == 0) {
      const double c = fmin(1.0, fmax(0.0, s));
      double wsum = 0.0;
      for (int l = 0; l < p.levels; l++) wsum += w5[l];
      factor[warp] = pow(fmax(c, 1e-9), w5[warp] / wsum);
      if (warp == 0) {
        p.out[0] = s;
        // one scale, or level 0 within 1e-12 of one: level 0 itself
        if (fabs(1.0 - c) < 1e-12 || p.levels == 1) factor[0] = -c;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (p.levels == 1 || signbit(factor[0])) {
    p.out[1] = -factor[0];
    return;
  }
  double prod = 1.0;
  for (int l = 0; l < p.levels; l++) prod *= factor[l];
  p.out[1] = fmin(1.0, fmax(0.0, prod));
}

int na_fail(int code, const char* fmt, ...) {
  char buf[384];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  rg::set_last_error(buf);
  return code;
}

// Device address of g_noalloc_scratch per device, found once per device with that device
// current. In host code the array's name is only a stand-in for the symbol, never an address.
std::mutex na_mu;
uint8_t* na_scratch_ptr[64] = {nullptr};

int na_setup(int dev, uint8_t** out) {
  std::lock_guard<std::mutex> lock(na_mu);
  if (dev < 0 || dev >= 64) return na_fail(RG_ERR_INVALID, "rg_ssim_plane_device_noalloc: device %d out of range", dev);
  if (!na_scratch_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return na_fail(RG_ERR_CUDA, "rg_ssim_plane_device_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    na_scratch_ptr[dev] = (uint8_t*)p;
  }
  *out = na_scratch_ptr[dev];
  return RG_OK;
}

}  // namespace

extern "C" int rg_ssim_plane_device_noalloc(const uint8_t* dev_a, size_t stride_a, const uint8_t* dev_b,
                                            size_t stride_b, int32_t width, int32_t height, double* dev_out,
                                            void* cuda_stream) {
  if (!dev_a || !dev_b || !dev_out) return na_fail(RG_ERR_INVALID, "rg_ssim_plane_device_noalloc: null pointer");
  if (width < 8 || height < 8)
    return na_fail(RG_ERR_INVALID, "rg_ssim_plane_device_noalloc: %dx%d is smaller than one 8x8 window", width, height);
  if (width > kNaMaxDim || height > kNaMaxDim || (long)width * height > kNaMaxPixels)
    return na_fail(RG_ERR_INVALID,
                   "rg_ssim_plane_device_noalloc: %dx%d exceeds the fixed working memory (width and height <= %d, "
                   "at most %ld samples); use rg_ssim_plane",
                   width, height, kNaMaxDim, kNaMaxPixels);
  if (stride_a < (size_t)width || stride_b < (size_t)width)
    return na_fail(RG_ERR_INVALID, "rg_ssim_plane_device_noalloc: stride smaller than width");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return na_fail(RG_ERR_CUDA, "rg_ssim_plane_device_noalloc: %s", cudaGetErrorString(e));
  uint8_t* scratch = nullptr;
  int r = na_setup(dev, &scratch);
  if (r) return r;
  cudaStream_t st = (cudaStream_t)cuda_stream;

  // pyramid levels while the next one is at least 8x8 (ms_ssim_plane_u8)
  SsimPair p{};
  p.out = dev_out;
  float* rows = (float*)(scratch + kNaPyrBytes);
  size_t rofs = 0, pofs = 0;
  int strips = 0;
  long sa = (long)stride_a, sb = (long)stride_b;
  const uint8_t *a = dev_a, *b = dev_b;
  for (int w = width, h = height; p.levels < 5 && w >= 8 && h >= 8; w >>= 1, h >>= 1) {
    if (p.levels) {
      sa = sb = (w + 3) & ~3;
      a = scratch + pofs;
      b = a + sa * h;
      pofs += 2 * (size_t)sa * h;
      strips += ssim_strips(h, false, kFlatStrip);
    }
    p.lv[p.levels++] = SsimLevel{a, b, sa, sb, w, h, rows + rofs};
    rofs += (size_t)(h / 4) + 1;
  }
  na_rows_kernel<true><<<ssim_strips(height, p.levels > 1, kFlatStrip), kRowThreads, 0, st>>>(p);
  if (strips) na_rows_kernel<false><<<strips, kRowThreads, 0, st>>>(p);
  na_finish_kernel<<<1, 160, 0, st>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return na_fail(RG_ERR_CUDA, "rg_ssim_plane_device_noalloc: launch failed: %s", cudaGetErrorString(e));
  return RG_OK;
}
