// SSIM / MS-SSIM / PSNR of 8-bit planes on the device (FFmpeg vf_ssim 4x4-sum reuse), with the
// reference's floating-point order reproduced exactly (ssim_rows.cuh).
//
// VMAF-Lite (crates/ragdoll-pix/src/metrics.rs:218 vmaf_lite_plane_u8): per non-overlapping 4x4
// block the local SSIM term and the VIF information terms in f64 (the same expressions, no fused
// multiply-add); one block per block row sums its terms, rows are added in order, and the host
// forms the score. The reference adds all blocks in one raster-order sum; the row-wise sum here
// differs from it only in rounding (about 1e-13 of the score).
#include <cmath>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ssim_kernels.h"

namespace rg {

namespace {

#include "ssim_rows.cuh"

template <bool kPyramid, int kStrip, int kChunk>
__global__ void __launch_bounds__(kRowThreads) ssim_rows_kernel(const SsimPair* __restrict__ pairs) {
  ssim_pass<kPyramid, kStrip, kChunk>(pairs[blockIdx.y]);
}
// A warp per (pair, level).
__global__ void __launch_bounds__(32) ssim_finish_kernel(const SsimPair* __restrict__ pairs) {
  __shared__ float stage[128];
  const SsimPair& p = pairs[blockIdx.y];
  if ((int)blockIdx.x >= p.levels) return;
  const double s = ssim_total(p.lv[blockIdx.x], stage);
  if (threadIdx.x == 0) p.out[blockIdx.x] = s;
}

// Squared error of each job's planes.
__global__ void sse_kernel(const SseJob* __restrict__ jobs) {
  const SseJob& j = jobs[blockIdx.y];
  unsigned long long acc = 0;
  long n = (long)j.width * j.height;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    long y = i / j.width, x = i - y * j.width;
    int d = (int)j.a[y * j.stride_a + x] - (int)j.b[y * j.stride_b + x];
    acc += (unsigned long long)(d * d);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(j.sse, acc);
}

// One 4-row strip of 4x4 blocks of job blockIdx.y: its three f64 sums into rows[3 * by ..].
__global__ void vmaf_rows_kernel(const VmafJob* __restrict__ jobs) {
  const VmafJob& j = jobs[blockIdx.y];
  const int bw = j.width >> 2, bh = j.height >> 2, by = blockIdx.x;
  if (by >= bh) return;
  const double kSigmaNsq = 2.0 * 256.0, kEps = 1.0e-10, kGainLimit = 100.0, c1 = 26.0, c2 = 234.0;
  double num = 0.0, den = 0.0, ssim = 0.0;
  for (int bx = threadIdx.x; bx < bw; bx += blockDim.x) {
    int s1 = 0, s2 = 0, ss = 0, s12 = 0;
#pragma unroll
    for (int dy = 0; dy < 4; dy++) {
      const uint8_t* pa = j.a + (long)(by * 4 + dy) * j.stride_a + bx * 4;
      const uint8_t* pb = j.b + (long)(by * 4 + dy) * j.stride_b + bx * 4;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        int va = pa[k], vb = pb[k];
        s1 += va; s2 += vb; ss += va * va + vb * vb; s12 += va * vb;
      }
    }
    const double mean_sq_sum = (double)(s1 * s1 + s2 * s2);
    const double total_var = (double)max(ss * 16 - s1 * s1 - s2 * s2, 0);
    const double covar = (double)(s12 * 16 - s1 * s2);
    const double blk = ((2.0 * (double)s1 * (double)s2 + c1) * (2.0 * covar + c2)) / ((mean_sq_sum + c1) * (total_var + c2));
    ssim += fmin(1.0, fmax(0.0, blk));
    double err_var = (double)max(ss - 2 * s12, 0) * 16.0 - (double)((s1 - s2) * (s1 - s2));
    err_var = fmax(err_var, 0.0);
    const double sigma1_sq = fmax((total_var - err_var) * 0.5, fmax(covar, 0.0));
    const double sigma2_sq = fmax(total_var - sigma1_sq, 0.0);
    const double sigma12 = fmax(covar, 0.0);
    double g, sv_sq;
    if (sigma1_sq < kEps) {
      g = 0.0;
      sv_sq = sigma2_sq;
    } else if (sigma2_sq < kEps) {
      g = 0.0;
      sv_sq = 0.0;
    } else {
      const double g_raw = sigma12 / (sigma1_sq + kEps);
      if (g_raw < 0.0) {
        g = 0.0;
        sv_sq = sigma2_sq;
      } else {
        g = fmin(g_raw, kGainLimit);
        sv_sq = fmax(sigma2_sq - g_raw * sigma12, kEps);
      }
    }
    sv_sq = fmax(sv_sq, kEps);
    g = fmin(g, kGainLimit);
    num += log2(1.0 + (g * g * sigma1_sq) / (sv_sq + kSigmaNsq));
    den += log2(1.0 + sigma1_sq / kSigmaNsq);
  }
  __shared__ double part[3][32];
  for (int o = 16; o > 0; o >>= 1) {
    num += __shfl_xor_sync(0xffffffffu, num, o);
    den += __shfl_xor_sync(0xffffffffu, den, o);
    ssim += __shfl_xor_sync(0xffffffffu, ssim, o);
  }
  const int warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  if ((threadIdx.x & 31) == 0) {
    part[0][warp] = num;
    part[1][warp] = den;
    part[2][warp] = ssim;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double acc = 0.0;
    for (int w = 0; w < nwarps; w++) acc += part[threadIdx.x][w];
    j.rows[3 * by + threadIdx.x] = acc;
  }
}

// Rows of each job added in order; also |a - prev| over the plane when prev is given.
__global__ void vmaf_finish_kernel(const VmafJob* __restrict__ jobs, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const VmafJob& j = jobs[i];
  double acc[3] = {0.0, 0.0, 0.0};
  for (int by = 0; by < (j.height >> 2); by++)
    for (int k = 0; k < 3; k++) acc[k] += j.rows[3 * by + k];
  for (int k = 0; k < 3; k++) j.out[k] = acc[k];
}

__global__ void sad_kernel(const VmafJob* __restrict__ jobs) {
  const VmafJob& j = jobs[blockIdx.y];
  if (!j.prev || !j.sad) return;
  unsigned long long acc = 0;
  long n = (long)j.width * j.height;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    long y = i / j.width, x = i - y * j.width;
    acc += (unsigned long long)abs((int)j.a[y * j.stride_a + x] - (int)j.prev[y * j.stride_prev + x]);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(j.sad, acc);
}

}  // namespace

void launch_vmaf(const VmafJob* d_jobs, int n_jobs, int max_height, cudaStream_t st) {
  dim3 grid(std::max(max_height >> 2, 1), n_jobs);
  vmaf_rows_kernel<<<grid, 128, 0, st>>>(d_jobs);
  vmaf_finish_kernel<<<(n_jobs + 63) / 64, 64, 0, st>>>(d_jobs, n_jobs);
  sad_kernel<<<dim3(64, n_jobs), 256, 0, st>>>(d_jobs);
}

double vmaf_lite_score(double info_num, double info_den, double ssim_sum, long blocks, bool have_prev,
                       unsigned long long sad, long pixels) {
  if (blocks <= 0) return 100.0;
  const double mean_ssim = ssim_sum / (double)blocks;
  if (std::fabs(1.0 - mean_ssim) < 1e-9) return 100.0;
  const double vif = info_den <= 1e-9 ? mean_ssim : std::fmin(1.0, std::fmax(0.0, info_num / info_den));
  double boost = 0.0;
  if (have_prev) boost = std::fmin((double)sad / (double)pixels / 255.0 * 0.08, 0.05);
  const double raw = (0.65 * std::pow(mean_ssim, 0.85) + 0.35 * vif + boost) * 100.0;
  return std::fmin(100.0, std::fmax(0.0, raw));
}

size_t ssim_pair_bytes() { return sizeof(SsimPair); }

void ssim_pair_fill(void* pair, const uint8_t* a, long sa, const uint8_t* b, long sb, int w, int h, bool ms, float* rows,
                    double* out, uint8_t* pyr, SsimSizes& used) {
  SsimPair& p = *(SsimPair*)pair;
  used = SsimSizes{0, 0, 0};
  p.out = out;
  p.levels = 0;
  for (int l = 0; l < 5; l++) {
    if (l) {
      w >>= 1;
      h >>= 1;
      if (!ms || w < 8 || h < 8) break;
      sa = sb = (w + 3) & ~3;  // rows of whole words
      a = pyr ? pyr + used.pyramid : nullptr;
      b = pyr ? a + sa * h : nullptr;
      used.pyramid += 2 * (size_t)sa * h;
    }
    p.lv[l] = SsimLevel{a, b, sa, sb, w, h, rows ? rows + used.rows : nullptr};
    used.rows += h / 4 + 1;
    p.levels++;
  }
  used.levels = p.levels;
}

// 60 pairs of 1080p, every scale, with the call around it: 2.64 ms with a decimation launch per level,
// byte loads, an allocation per array and a squared-error pass nobody read; 0.27 ms so. The planes are
// 249 MB, 0.04 ms of HBM.
template <int kStrip, int kChunk>
static void launch_rows(const SsimPair* p, int n, int h, bool pyramid, cudaStream_t st) {
  if (const int s = ssim_strips(h, pyramid, kStrip)) ssim_rows_kernel<true, kStrip, kChunk><<<dim3(s, n), kRowThreads, 0, st>>>(p);
  int s = 0;
  if (pyramid)
    for (int l = 1; l < 5 && (h >>= 1) >= 8; l++) s += ssim_strips(h, false, kStrip);
  if (s) ssim_rows_kernel<false, kStrip, kChunk><<<dim3(s, n), kRowThreads, 0, st>>>(p);
}

void launch_ssim(const void* d_pairs, int n, int max_height, bool pyramid, int sms, cudaStream_t st) {
  const SsimPair* p = (const SsimPair*)d_pairs;
  // two blocks an SM of the tall kind: about as many as hide each other's loads
  if (n * ssim_strips(max_height, pyramid, kTallStrip) >= 2 * sms) launch_rows<kTallStrip, kTallChunk>(p, n, max_height, pyramid, st);
  else launch_rows<kFlatStrip, kFlatChunk>(p, n, max_height, pyramid, st);
  ssim_finish_kernel<<<dim3(pyramid ? 5 : 1, n), 32, 0, st>>>(p);
}

void launch_sse(const SseJob* d_jobs, int n_jobs, cudaStream_t st) {
  dim3 grid(64, n_jobs);
  sse_kernel<<<grid, 256, 0, st>>>(d_jobs);
}

}  // namespace rg
