// Device SSIM / MS-SSIM / PSNR jobs (ssim_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace rg {

// One plane pair's squared error, added to *sse (device, zeroed).
struct SseJob {
  const uint8_t* a;
  const uint8_t* b;
  long stride_a, stride_b;
  int width, height;
  unsigned long long* sse;
};

// What a plane pair's SSIM (ms: and its pyramid's) needs: floats of row sums, bytes of pyramid planes,
// and its scales.
struct SsimSizes {
  size_t rows, pyramid;
  int levels;
};
// Host descriptor of a pair (ssim_pair_bytes() bytes at `pair`) over device scratch rows / pyr (pyr
// 4-byte aligned; both may be null to get the sizes alone) and the device doubles out[levels].
size_t ssim_pair_bytes();
void ssim_pair_fill(void* pair, const uint8_t* a, long sa, const uint8_t* b, long sb, int w, int h, bool ms, float* rows,
                    double* out, uint8_t* pyr, SsimSizes& used);
// SSIM of every scale of n pairs into their out (pyramid: some have more than one scale) on a device of `sms` SMs.
void launch_ssim(const void* d_pairs, int n, int max_height, bool pyramid, int sms, cudaStream_t st);
void launch_sse(const SseJob* d_jobs, int n_jobs, cudaStream_t st);

// VMAF-Lite of one plane pair (ref a, distorted b; prev: the previous reference frame or null).
// rows: device scratch of 3 * (height / 4) doubles; out: device {info_num, info_den, ssim_sum};
// sad: optional accumulator of |a - prev| over the plane.
struct VmafJob {
  const uint8_t* a;
  const uint8_t* b;
  const uint8_t* prev;
  long stride_a, stride_b, stride_prev;
  int width, height;
  double* rows;
  double* out;
  unsigned long long* sad;
};

void launch_vmaf(const VmafJob* d_jobs, int n_jobs, int max_height, cudaStream_t st);
// The score from the sums (crates/ragdoll-pix/src/metrics.rs:301-324); host code.
double vmaf_lite_score(double info_num, double info_den, double ssim_sum, long blocks, bool have_prev,
                       unsigned long long sad, long pixels);

}  // namespace rg
