// The learned form's candidate network (no counterpart in the reference): a small CNN that reads
// each macroblock of a picture with a 4-sample border (24x24 luma of the picture, and the same
// window of the previous picture, as two channels) and predicts the partition types, the intra
// 4x4 modes and an offset of the integer search's centre that the learned analysis form tries.
//
//   x (2 x 24 x 24, (sample - 128) / 64)
//   conv 3x3 2 -> 32, ReLU (22 x 22); conv 3x3 32 -> 32, ReLU (20 x 20); conv 3x3 32 -> 32, ReLU (18 x 18)
//   g   = mean of the 18 x 18 map (32);   f_b = mean of 4x4 block b's 4 x 4 area of the map (32)
//   partition logits = Wp g + bp (4);  search offset = Wm g + bm (2, in units of 16 quarter samples)
//   intra 4x4 logits of block b = Wi f_b + bi (9)
//
// Inference (cnn_infer_kernel): BF16 implicit-GEMM convolutions on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory), two CTAs per SM, each a strip of two macroblocks
// per step: every activation map of the strip is stored with one row stride, so the 3x3 taps of a
// 128-position tile are the same K-major operand shifted by whole rows of 16 bytes, and each tap is
// one descriptor of the map -- no im2col copy. The epilogue adds the bias, applies the ReLU and
// stores the next layer's BF16 operand over its input; the heads run on the CUDA cores and write
// the hints. While one CTA's epilogue runs, the other's MMAs can.
// Training: the same network in f32 on the CUDA cores -- forward, the losses, the
// backward pass and Adam -- on per-macroblock crops.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/ragdoll_cuda.h"

namespace rg {
void set_last_error(const char* msg);
}

namespace {

constexpr int C = 32;
// parameter offsets (f32, the order of rg_net_params)
constexpr int kW1 = 0, kB1 = kW1 + C * 2 * 9, kW2 = kB1 + C, kB2 = kW2 + C * C * 9, kW3 = kB2 + C,
              kB3 = kW3 + C * C * 9, kWp = kB3 + C, kBp = kWp + 4 * C, kWm = kBp + 4, kBm = kWm + 2 * C,
              kWi = kBm + 2, kBi = kWi + 9 * C, kParams = kBi + 9;
constexpr int kLogits = 4 + 2 + 16 * 9;  // per macroblock: partition, offset, intra 4x4

__device__ __forceinline__ float pix_norm(uint8_t v) { return ((float)v - 128.0f) * (1.0f / 64.0f); }

// ---------------------------------------------------------------------------------------------
// Inference on the tensor cores. Two CTAs per SM, each a strip of two macroblocks at a time; one
// activation buffer per CTA holds every map of its strip in turn (the input in plane 0, then each
// layer's output over its input, tile by tile: a tile's MMAs read its positions and the next tile's, so
// tile t is stored once the MMAs of tiles t - 1 and t have completed).
constexpr int kStripMbs = 2;
constexpr int kThreads = 256;  // 8 warps; warps w and w + 4 share TMEM lanes 32 (w % 4)..; a ninth issues the MMAs
constexpr int kCtasPerSm = 2;
constexpr int kRow = 16 * kStripMbs + 8;  // row stride (positions) of every map of a strip: 40
constexpr int kTiles1 = (22 * kRow + 127) / 128, kTiles2 = (20 * kRow + 127) / 128, kTiles3 = (18 * kRow + 127) / 128;
constexpr int kTap = 2 * kRow + 2;  // reach of the last tap
constexpr int kPosBuf = ((kTiles1 * 128 + kTap > kTiles2 * 128 + kTap ? kTiles1 * 128 + kTap : kTiles2 * 128 + kTap) +
                         kThreads - 1) / kThreads * kThreads;  // positions of the buffer
static_assert(kPosBuf >= kTiles1 * 128 + kTap + 1 && kPosBuf >= kTiles3 * 128 + kTap,
              "tap reach (conv1's last pair one position further) and outputs fit the buffer");
static_assert(kPosBuf >= 24 * kRow, "the input map fits plane 0");
static_assert(kTap < 128 && kTiles2 == kTiles1 && kTiles3 <= kTiles1, "a tile reads its positions and the next tile's; layers 0 and 1 store every tile");
static_assert(kTiles1 * 32 <= 256, "accumulators of one layer fit the CTA's 256 tensor-memory columns");
static_assert(kStripMbs * 4 <= kThreads / 32, "pooling: a warp per (macroblock, 8-channel plane)");
// shared memory (bytes): the buffer (4 planes of 8 channels) | B operands | the rest
constexpr int kPlane = kPosBuf * 16;
constexpr int kOffBuf = 0, kOffB = kOffBuf + 4 * kPlane;
constexpr int kB1Mmas = 5, kBMmas = 18;  // conv1: taps paired; conv2/3: 9 taps x 2 channel halves
constexpr int kOffB2 = kOffB + kB1Mmas * 1024, kOffB3 = kOffB2 + kBMmas * 1024, kOffMisc = kOffB3 + kBMmas * 1024;
constexpr int kHeadPitch = C + 1;  // the heads' weights and the pooled maps: rows in different banks
struct InferMisc {
  alignas(16) float bias[3][C];
  float head[15][kHeadPitch];    // weights, then the bias: partition (4), offset (2), intra 4x4 (9)
  float pool[kStripMbs][17][kHeadPitch];  // per macroblock: the 18 x 18 mean, then the 16 block means
  float logit[kStripMbs * 16 * 9 + kStripMbs * 6];
  alignas(8) uint64_t mbar[kTiles1], ready[kTiles1];  // per tile: its MMAs have completed; its map is stored
  uint32_t tmem;
  int strip;
};
constexpr int kSmemInfer = kOffMisc + (int)sizeof(InferMisc);
static_assert(kSmemInfer <= 233472 / kCtasPerSm - 1024, "two CTAs' shared memory fit an SM");

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Shared-memory matrix descriptor, K-major without swizzle: 8-row core matrices of 16-byte rows,
// sbo between 8-row groups, lbo between the two 8-element halves of K (sm100 version 1).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}
// kind::f16 instruction descriptor: BF16 A and B (K-major), F32 accumulator, M = 128, N = 32.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(32 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void umma_commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
               : "memory");
}
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Waits for the mbarrier's phase `parity` to complete; false after ~4 M polls (the error path).
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity) {
  uint32_t a = smem_u32(mbar);
  for (int i = 0; i < (1 << 22); i++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\tselp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// 32 consecutive columns of this thread's lane (one accumulator tile).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// The pictures one launch reads, and where the hints go.
struct InferJob {
  const uint8_t* cur;   // luma of the picture (display size)
  const uint8_t* prev;  // luma of the previous picture (the picture itself for an IDR picture)
  rg_mb_hint* hints;    // mb_w * mb_h hints
  float* logits;        // mb_w * mb_h * kLogits, or null
};
struct InferParams {
  const InferJob* jobs;
  int n_jobs, width, height, stride, mb_w, mb_h, strips_per_row;
  const __nv_bfloat16* bops;  // B operands of the three layers in their shared-memory layout
  const float* params;        // f32 parameters (biases and heads)
  int* counter;               // strip ticket
  int* error;                 // set when a wait on the tensor cores gives up
  int part_k, i4_k;           // hint policy: candidates kept at most,
  float part_margin, i4_margin;  // and only those within this logit margin of the best
};

// The candidates of n logits as a bit mask: the best, then the next ones in logit order (the lower
// index on ties) up to k in all, each only while its logit is at least the best's minus `margin`.
template <int N>
__device__ __forceinline__ uint32_t topk_mask(const float (&l)[N], int k, float margin) {
  uint32_t m = 0;
  float top = 0.0f;
#pragma unroll
  for (int r = 0; r < N; r++) {
    if (r >= k) break;
    int best = -1;
    float bv = 0.0f;
#pragma unroll
    for (int i = 0; i < N; i++)  // constant indices: the logits stay in registers
      if (!((m >> i) & 1) && (best < 0 || l[i] > bv)) {
        best = i;
        bv = l[i];
      }
    if (r == 0) top = bv;
    else if (bv < top - margin) break;
    m |= 1u << best;
  }
  return m;
}

__global__ void __launch_bounds__(kThreads + 32, kCtasPerSm) cnn_infer_kernel(InferParams ip) {
  extern __shared__ __align__(1024) uint8_t smem[];
  InferMisc& ms = *reinterpret_cast<InferMisc*>(smem + kOffMisc);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* buf = smem + kOffBuf;
  // B operands, biases and heads once per CTA
  for (int i = tid; i < (kB1Mmas + 2 * kBMmas) * 1024 / 16; i += kThreads)
    ((uint4*)(smem + kOffB))[i] = ((const uint4*)ip.bops)[i];
  for (int i = tid; i < 3 * C; i += kThreads) ms.bias[i / C][i % C] = ip.params[(i / C == 0 ? kB1 : (i / C == 1 ? kB2 : kB3)) + i % C];
  for (int i = tid; i < 15 * kHeadPitch; i += kThreads) {
    const int o = i / kHeadPitch, c = i - o * kHeadPitch;
    const int w = o < 4 ? kWp + o * C : (o < 6 ? kWm + (o - 4) * C : kWi + (o - 6) * C), b = o < 4 ? kBp + o : (o < 6 ? kBm + o - 4 : kBi + o - 6);
    ms.head[o][c] = ip.params[c < C ? w + c : b];
  }
  if (tid == 0) {
#pragma unroll
    for (int t = 0; t < kTiles1; t++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&ms.mbar[t])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&ms.ready[t])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&ms.tmem)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = ms.tmem;
  const uint32_t sBuf = smem_u32(buf), sB1 = smem_u32(smem + kOffB), sB2 = smem_u32(smem + kOffB2),
                 sB3 = smem_u32(smem + kOffB3);
  uint32_t phase = 0;
  bool ok = true;
  const int total = ip.n_jobs * ip.mb_h * ip.strips_per_row;
  // The input map of a strip (plane 0 of the buffer): position r * kRow + c is sample (x0 - 4 + c,
  // y0 - 4 + r), clamped to the picture; 16 bytes each, the two channels and six zero channels. A
  // strip's bytes are loaded into registers while the previous strip's MMAs run.
  constexpr int kPer = kPosBuf / kThreads;
  uint8_t ca[kPer], pa[kPer];
  auto load_input = [&](int st) {
    const int job = st / (ip.mb_h * ip.strips_per_row), rem = st % (ip.mb_h * ip.strips_per_row);
    const int y0 = (rem / ip.strips_per_row) * 16 - 4, x0 = (rem % ip.strips_per_row) * kStripMbs * 16 - 4;
    const InferJob jb = ip.jobs[job];
#pragma unroll
    for (int k = 0; k < kPer; k++) {  // all of this thread's loads in flight together
      const int p = tid + kThreads * k;
      const int r = p / kRow, c = p - r * kRow;
      const int yy = min(max(y0 + r, 0), ip.height - 1), xx = min(max(x0 + c, 0), ip.width - 1);
      const size_t o = (size_t)yy * ip.stride + xx;
      ca[k] = p < 24 * kRow ? jb.cur[o] : 128;
      pa[k] = p < 24 * kRow ? jb.prev[o] : 128;
    }
  };
  if (tid == 0) ms.strip = atomicAdd(ip.counter, 1);
  __syncthreads();
  int strip = ms.strip;
  __syncthreads();  // every thread has it before the next one is written
  if (strip < total && warp < 8) load_input(strip);
  // shared-memory descriptors: conv1's five tap pairs on plane 0, the two channel halves of the
  // buffer for conv2 and conv3, the B operands; a tile / tap adds its offset in 16-byte units
  const uint64_t bufd0 = umma_desc(sBuf, kPlane, 128), bufd1 = umma_desc(sBuf + 2 * kPlane, kPlane, 128);
  const uint64_t b1d = umma_desc(sB1, 512, 128), b2d = umma_desc(sB2, 512, 128), b3d = umma_desc(sB3, 512, 128);
  // The loaded bytes into the input map, and the ticket of the strip after (read behind the barrier).
  auto store_input = [&]() {
    if (warp < 8)
#pragma unroll
      for (int k = 0; k < kPer; k++) {
        __nv_bfloat162 two = __floats2bfloat162_rn(pix_norm(ca[k]), pix_norm(pa[k]));
        ((uint4*)buf)[tid + kThreads * k] = make_uint4(*(uint32_t*)&two, 0u, 0u, 0u);
      }
    if (tid == 0) ms.strip = atomicAdd(ip.counter, 1);
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
  };
  // Logits and hints of strip st from its pooled map (warps 0 .. 7, beside the next strip's first MMAs).
  auto finish = [&](int st) {
    const int job = st / (ip.mb_h * ip.strips_per_row), rem = st % (ip.mb_h * ip.strips_per_row);
    const int mby = rem / ip.strips_per_row, mbx0 = (rem % ip.strips_per_row) * kStripMbs;
    const InferJob jb = ip.jobs[job];
    // logits, one a thread at a time: of (block, intra 4x4 mode), then of (macroblock, partition or offset)
    constexpr int kBlockLogits = kStripMbs * 16 * 9;
    for (int i = tid; i < kBlockLogits + kStripMbs * 6; i += kThreads) {
      const bool block = i < kBlockLogits;
      const int n = block ? i / 9 : (i - kBlockLogits) / 6, o = block ? 6 + i - n * 9 : i - kBlockLogits - n * 6;
      const float* f = block ? ms.pool[n >> 4][1 + (n & 15)] : ms.pool[n][0];
      const float* W = ms.head[o];
      float s = W[C];
#pragma unroll
      for (int c = 0; c < C; c++) s += W[c] * f[c];
      ms.logit[i] = s;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");  // warps 0 .. 7
    // heads and hints: threads 0 .. 16 kStripMbs - 1 the intra 4x4 heads of (macroblock tid / 16,
    // block tid % 16), the next kStripMbs threads the partition and offset heads of their macroblock
    if (tid < 16 * kStripMbs + kStripMbs) {
      const bool blockhead = tid < 16 * kStripMbs;
      const int j = blockhead ? tid / 16 : tid - 16 * kStripMbs, mbx = mbx0 + j;
      if (mbx < ip.mb_w) {
        const int m = mby * ip.mb_w + mbx;
        float* lg = jb.logits ? jb.logits + (size_t)m * kLogits : nullptr;
        if (blockhead) {
          const int b = tid % 16;
          float li[9];
#pragma unroll
          for (int o = 0; o < 9; o++) li[o] = ms.logit[tid * 9 + o];
          // 4x4 block b in raster order; the hint holds decoding order
          const int bx = b & 3, by = b >> 2;
          const int dec = ((by >> 1) << 3) | ((bx >> 1) << 2) | ((by & 1) << 1) | (bx & 1);
          jb.hints[m].i4_mask[dec] = (uint16_t)topk_mask(li, ip.i4_k, ip.i4_margin);
          if (lg)
            for (int o = 0; o < 9; o++) lg[6 + b * 9 + o] = li[o];
        } else {
          const float* l = &ms.logit[kBlockLogits + 6 * j];
          const float lp[4] = {l[0], l[1], l[2], l[3]}, lm[2] = {l[4], l[5]};
          rg_mb_hint& hh = jb.hints[m];
          hh.part_mask = (uint8_t)topk_mask(lp, ip.part_k, ip.part_margin);
          hh.flags = 0;  // the coarse motion pass, when on, follows
          hh.mv_coarse[0] = hh.mv_coarse[1] = 0;
          for (int o = 0; o < 2; o++) hh.mv_off[o] = (int8_t)max(-127, min(127, __float2int_rn(16.0f * lm[o])));
          if (lg) {
            for (int o = 0; o < 4; o++) lg[o] = lp[o];
            lg[4] = lm[0];
            lg[5] = lm[1];
          }
        }
      }
    }
  };
  if (strip < total) store_input();
  int pooled = -1;  // the strip whose hints are still to be written
  while (strip < total && ok) {
    const int next = ms.strip;
    // The ninth warp issues the MMAs of all three layers, tile by tile; each tile completes on its own
    // barrier, and its epilogue, which stores the tile's positions 128 t .. 128 t + 127 over the layer's
    // input, runs while other tiles' MMAs do. A tile reads the positions of tiles t and t + 1 of its input:
    // its MMAs start once both are stored, and tile t is stored once tiles t - 1 and t have completed. The
    // MMAs bound the kernel: 269 a strip, each 46 cycles (M = 128, N = 32: 16 of the tensor pipe; measured
    // alone, whatever the layout of A). Layers one after the other for the whole strip left the tensor
    // cores 67 cycles a MMA: 2.39 ms for eight 1080p pictures with the coarse pass, 2.15 so, and 2.12 with a strip's logits
    // beside the next strip's first MMAs.
    if (warp == 8) {
      if (lane == 0) {
#pragma unroll 1
        for (int t = 0; t < kTiles1; t++) {
#pragma unroll
          for (int k = 0; k < kB1Mmas; k++) {
            // taps 2k and 2k + 1 (tap 9: a zero-weight partner one position on) as the two
            // 8-element halves of K, LBO their distance
            const int ta = 2 * k, tb = 2 * k + 1;
            const int oa = (ta / 3) * kRow + ta % 3, ob = tb < 9 ? (tb / 3) * kRow + tb % 3 : oa + 1;
            const uint64_t a = umma_desc(sBuf + (uint32_t)((t * 128 + oa) * 16), (uint32_t)((ob - oa) * 16), 128);
            umma_bf16(tmem + (uint32_t)(t * 32), a, b1d + (uint64_t)(k * 64), k > 0);
          }
          umma_commit(&ms.mbar[t]);
        }
#pragma unroll 1
        for (int layer = 1; layer < 3; layer++) {
          const int tiles = layer == 1 ? kTiles2 : kTiles3, before = layer == 1 ? kTiles1 : kTiles2;
          const uint64_t bd = layer == 1 ? b2d : b3d;
          if (ok) ok = mbar_wait(&ms.ready[0], (uint32_t)(layer - 1));
#pragma unroll 1
          for (int t = 0; t < kTiles1; t++) {
            if (ok && t + 1 < before) ok = mbar_wait(&ms.ready[t + 1], (uint32_t)(layer - 1));
            if (!ok) break;
            fence_after_sync();
            if (t < tiles) {
              const uint32_t d = tmem + (uint32_t)(t * 32);
#pragma unroll
              for (int tap = 0; tap < 9; tap++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                  const uint64_t off = (uint64_t)(t * 128 + (tap / 3) * kRow + tap % 3);
                  umma_bf16(d, (h ? bufd1 : bufd0) + off, bd + (uint64_t)((tap * 2 + h) * 64), tap > 0 || h > 0);
                }
            }
            umma_commit(&ms.mbar[t]);  // (also without a tile: every barrier's phase turns every layer)
          }
        }
      }
      phase ^= 1;  // three layers
      __syncwarp();
    } else {
      if (next < total) load_input(next);  // the next strip's bytes, in flight while the tensor cores work
      if (pooled >= 0) finish(pooled);
    }
    for (int layer = 0; layer < 3 && warp < 8; layer++, phase ^= 1) {
      const int tiles = layer == 0 ? kTiles1 : (layer == 1 ? kTiles2 : kTiles3);
      // epilogue: warp w reads rows 32 (w % 4) .. + 31 of tiles w / 4, + 2, ..; bias, ReLU, BF16 into the
      // buffer's four planes
      const int wl = warp & 3;
#pragma unroll 1
      for (int t = warp >> 2; t < kTiles1; t += 2) {
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&ms.mbar[max(t - 1, 0)], phase) && mbar_wait(&ms.mbar[t], phase));
        if (!ok || t >= tiles) continue;
        fence_after_sync();
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(wl * 32) << 16) + (uint32_t)(t * 32), v);
        const int p = t * 128 + wl * 32 + lane;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint32_t w[4];
          const float4 b0 = *(const float4*)&ms.bias[layer][8 * q], b1 = *(const float4*)&ms.bias[layer][8 * q + 4];
          const float bs[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float a = fmaxf(v[8 * q + 2 * k] + bs[2 * k], 0.0f);
            const float b = fmaxf(v[8 * q + 2 * k + 1] + bs[2 * k + 1], 0.0f);
            __nv_bfloat162 two = __floats2bfloat162_rn(a, b);
            w[k] = *(uint32_t*)&two;
          }
          *(uint4*)(buf + q * kPlane + p * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (layer < 2) {  // the tile's map to the MMAs of the next layer
          fence_async_smem();
          fence_before_sync();
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&ms.ready[t])) : "memory");
        }
      }
    }
    // a wait that gave up is made uniform before anyone acts on it (this also completes conv3's map)
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok && tid == 0) atomicExch(ip.error, 1);
    if (!ok) break;
    // pooling of the conv3 map (map column 16 j + i is sample x 16 (mbx0 + j) - 1 + i): warp w
    // takes macroblock j = w / 4 and 8-channel plane q = w % 4; lane l < 16 sums map column l + 1
    // down the 18 rows (16-byte reads), lanes 16 and 17 the border columns 0 and 17; block sums
    // over the four lanes of a block column, the 18 x 18 sum over the warp
    if (warp < kStripMbs * 4) {
      const int j = warp >> 2, q = warp & 3;
      const int col = lane < 16 ? lane + 1 : (lane == 16 ? 0 : 17);
      float tot[8], blk[4][8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        tot[k] = 0.0f;
#pragma unroll
        for (int b = 0; b < 4; b++) blk[b][k] = 0.0f;
      }
      if (lane < 18) {
        const uint8_t* colp = buf + q * kPlane + (16 * j + col) * 16;
#pragma unroll
        for (int r = 0; r < 18; r++) {
          const uint4 v = *(const uint4*)(colp + r * kRow * 16);
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float2 f = __bfloat1622float2(*(const __nv_bfloat162*)&w[k]);
            tot[2 * k] += f.x;
            tot[2 * k + 1] += f.y;
            if (r >= 1 && r <= 16 && lane < 16) {
              blk[(r - 1) >> 2][2 * k] += f.x;
              blk[(r - 1) >> 2][2 * k + 1] += f.y;
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 8; k++) {
#pragma unroll
        for (int b = 0; b < 4; b++) {
          blk[b][k] += __shfl_xor_sync(0xffffffffu, blk[b][k], 1);
          blk[b][k] += __shfl_xor_sync(0xffffffffu, blk[b][k], 2);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) tot[k] += __shfl_xor_sync(0xffffffffu, tot[k], o);
      }
      if (lane < 16 && (lane & 3) == 0)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
          for (int k = 0; k < 8; k++) ms.pool[j][1 + b * 4 + (lane >> 2)][8 * q + k] = blk[b][k] * (1.0f / 16.0f);
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < 8; k++) ms.pool[j][0][8 * q + k] = tot[k] * (1.0f / 324.0f);
    }
    __syncthreads();
    if (next < total) store_input();  // over the map that has been pooled
    pooled = strip;
    strip = next;
  }
  if (ok && pooled >= 0 && warp < 8) finish(pooled);
  fence_before_sync();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem));
}

// ---------------------------------------------------------------------------------------------
// Coarse motion (rg_net_set_coarse_range): a warp per macroblock, eight neighbours of a row per block. The
// decimated picture's sample (x, y) is the rounded mean of the four samples (2x + i, 2y + j), coordinates
// clamped to the picture; the macroblock's 8 x 8 decimated block is compared with the decimated
// previous picture at every displacement of +-r (SAD), the least (SAD, |dx| + |dy|, raster index)
// wins. Bound by instructions: the eight windows of a block overlap and are decimated once, by words
// where they lie inside the picture, and a lane slides down a column of displacements, so that a row of
// the window is read once for eight of them. Eight 1080p pictures at r = 16: 0.77 ms with a window per
// macroblock and a vector at a time, 0.20 ms so (the launch alone).
constexpr int kCoarseMaxR = 32;
constexpr int kCoarseMbs = 8;                                             // macroblocks (warps) of a block
constexpr int kCoarseRow = 8 * kCoarseMbs + 2 * kCoarseMaxR + 4;          // window row stride (bytes), an odd number of words
constexpr int kCoarseRows = (2 * kCoarseMaxR + 8) / 8 * 8 + 8;            // rows the bands of eight displacements read
constexpr int kCoarseBlkRow = 8 * kCoarseMbs;
struct CoarseParams {
  const InferJob* jobs;
  int n_jobs, width, height, stride, mb_w, mb_h, r;
};
__device__ __forceinline__ uint32_t dec_sample(const uint8_t* p, int stride, int w, int h, int x, int y) {
  const int x0 = min(max(2 * x, 0), w - 1), x1 = min(max(2 * x + 1, 0), w - 1);
  const int y0 = min(max(2 * y, 0), h - 1), y1 = min(max(2 * y + 1, 0), h - 1);
  const uint8_t* r0 = p + (size_t)y0 * stride;
  const uint8_t* r1 = p + (size_t)y1 * stride;
  return ((uint32_t)r0[x0] + r0[x1] + r1[x0] + r1[x1] + 2u) >> 2;
}
// Decimated samples (x, y) .. (x + 3, y), packed.
__device__ __forceinline__ uint32_t dec_quad(const uint8_t* p, int stride, int w, int h, int x, int y) {
  const uint8_t* q = p + (long)(2 * y) * stride + 2 * x;
  if (x >= 0 && 2 * x + 8 <= w && y >= 0 && 2 * y + 2 <= h && (((uintptr_t)q | (uintptr_t)stride) & 3) == 0) {
    auto mean = [](uint32_t a, uint32_t b) {  // two samples, 16 bits apart
      const uint32_t t = (a & 0x00ff00ffu) + ((a >> 8) & 0x00ff00ffu) + (b & 0x00ff00ffu) + ((b >> 8) & 0x00ff00ffu);
      return ((t + 0x00020002u) >> 2) & 0x00ff00ffu;
    };
    const uint32_t *a = (const uint32_t*)q, *b = (const uint32_t*)(q + stride);
    const uint32_t a0 = __ldg(a), a1 = __ldg(a + 1), b0 = __ldg(b), b1 = __ldg(b + 1);
    return __byte_perm(mean(a0, b0), mean(a1, b1), 0x6420);
  }
  uint32_t v = 0;
  for (int k = 0; k < 4; k++) v |= dec_sample(p, stride, w, h, x + k, y) << (8 * k);
  return v;
}
__global__ void __launch_bounds__(32 * kCoarseMbs) coarse_motion_kernel(CoarseParams cp) {
  __shared__ __align__(16) uint8_t win[kCoarseRows * kCoarseRow];
  __shared__ __align__(16) uint8_t blk[8 * kCoarseBlkRow];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_row = (cp.mb_w + kCoarseMbs - 1) / kCoarseMbs;
  const int row = blockIdx.x / per_row, job = row / cp.mb_h, mby = row - job * cp.mb_h;
  const int mbx0 = (blockIdx.x - row * per_row) * kCoarseMbs;
  const InferJob jb = cp.jobs[job];
  if (jb.cur == jb.prev) return;  // an IDR picture: no previous picture
  const int R = cp.r, nw = 2 * R + 1, bx = 8 * mbx0, by = 8 * mby;  // the first block's decimated origin
  const int quads = (8 * kCoarseMbs + 2 * R + 3) >> 2;
#pragma unroll 2
  for (int i = tid; i < (8 + 2 * R) * quads; i += 32 * kCoarseMbs) {
    const int y = i / quads, x = i - y * quads;
    *(uint32_t*)&win[y * kCoarseRow + 4 * x] = dec_quad(jb.prev, cp.stride, cp.width, cp.height, bx - R + 4 * x, by - R + y);
  }
  for (int i = tid; i < 8 * kCoarseBlkRow / 4; i += 32 * kCoarseMbs) {
    const int y = i / (kCoarseBlkRow / 4), x = i - y * (kCoarseBlkRow / 4);
    ((uint32_t*)blk)[i] = dec_quad(jb.cur, cp.stride, cp.width, cp.height, bx + 4 * x, by + y);
  }
  __syncthreads();
  if (mbx0 + warp >= cp.mb_w) return;
  uint2 b[8];
#pragma unroll
  for (int r = 0; r < 8; r++) b[r] = *(const uint2*)&blk[r * kCoarseBlkRow + 8 * warp];
  uint64_t best = ~0ull;
  // Columns of displacements 32 at a time; up to four left over (2 r + 1 leaves one) a displacement a lane.
  const int rem = nw & 31, cols = rem <= 4 ? rem : 0, slide = nw - cols;
#pragma unroll 1
  for (int d0 = 0; d0 < slide; d0 += 32) {
    const int dxi = min(d0 + lane, slide - 1), at = 8 * warp + dxi;
    const uint32_t sh = (uint32_t)(at & 3) * 8u, ax = (uint32_t)abs(dxi - R);
    const uint32_t* p = (const uint32_t*)&win[at & ~3];
    uint32_t key = ~0u;  // SAD (14 bits), distance (7), row (7)
#pragma unroll 1
    for (int y0 = 0; y0 < nw; y0 += 8) {
      uint32_t acc[8];
#pragma unroll
      for (int d = 0; d < 8; d++) acc[d] = 0;
#pragma unroll
      for (int i = 0; i < 15; i++) {  // window row y0 + i pairs with block row i - d of displacement row y0 + d
        const uint32_t w0 = p[0], w1 = p[1], w2 = p[2];
        p += kCoarseRow / 4;
        const uint32_t u = __funnelshift_r(w0, w1, sh), v = __funnelshift_r(w1, w2, sh);
#pragma unroll
        for (int d = 0; d < 8; d++)
          if (i - d >= 0 && i - d < 8) acc[d] = __vsadu4(u, b[(i - d) & 7].x) + __vsadu4(v, b[(i - d) & 7].y) + acc[d];
      }
      p -= 7 * (kCoarseRow / 4);
#pragma unroll
      for (int d = 0; d < 8; d++) {
        const int y = y0 + d;
        const uint32_t k = (acc[d] << 14) | ((ax + (uint32_t)abs(y - R)) << 7) | (uint32_t)y;
        key = min(key, y < nw ? k : ~0u);
      }
    }
    best = min(best, ((uint64_t)(key >> 14) << 32) | ((uint64_t)((key >> 7) & 127u) << 16) | (uint64_t)((key & 127u) * (uint32_t)nw + (uint32_t)dxi));
  }
#pragma unroll 1
  for (int i = lane; i < cols * nw; i += 32) {
    const int y = i / cols, dxi = slide + i - y * cols, at = 8 * warp + dxi;
    const uint32_t sh = (uint32_t)(at & 3) * 8u;
    const uint32_t* p = (const uint32_t*)&win[y * kCoarseRow + (at & ~3)];
    uint32_t sad = 0;
#pragma unroll
    for (int r = 0; r < 8; r++, p += kCoarseRow / 4)
      sad = __vsadu4(__funnelshift_r(p[0], p[1], sh), b[r].x) + __vsadu4(__funnelshift_r(p[1], p[2], sh), b[r].y) + sad;
    best = min(best, ((uint64_t)sad << 32) | ((uint64_t)(uint32_t)(abs(dxi - R) + abs(y - R)) << 16) | (uint64_t)(uint32_t)(y * nw + dxi));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = min(best, (uint64_t)__shfl_xor_sync(0xffffffffu, (unsigned long long)best, o));
  if (lane == 0) {
    const int p = (int)(best & 0xffffu), dyi = p / nw, dxi = p - dyi * nw;
    rg_mb_hint& h = jb.hints[mby * cp.mb_w + mbx0 + warp];
    h.mv_coarse[0] = (int16_t)(8 * (dxi - R));
    h.mv_coarse[1] = (int16_t)(8 * (dyi - R));
    h.flags |= 1;
  }
}

// ---------------------------------------------------------------------------------------------
// Training on the CUDA cores (f32), per-macroblock crops: 2 x 24 x 24 bytes per sample.
// Maps: A1 [N][32][22][22], A2 [N][32][20][20], A3 [N][32][18][18] (after the ReLU).
// The pass is about 22 M multiply-adds a sample; its kernels are bound by the FMA pipes and keep a
// register tile per thread, so that a shared-memory load feeds about ten of them. A batch of 256:
// 6.1 ms with a position or a weight per thread (the weight gradients in 32 blocks), 0.5 ms as below.
constexpr int kIn = 2 * 24 * 24, kA1 = C * 22 * 22, kA2 = C * 20 * 20, kA3 = C * 18 * 18;
constexpr int kW = C * C * 9;                  // weights of a 32 -> 32 layer
constexpr int kHeadParams = kParams - kWp;
// Transposed weights (train_prep_kernel): [ci][tap][co] for the forward passes, [co][8 - tap][ci] for the
// input gradients -- the layout a convolution block loads.
constexpr int kT1 = 0, kT2 = kT1 + 2 * 9 * C, kT3 = kT2 + kW, kTb3 = kT3 + kW, kTb2 = kTb3 + kW, kTrans = kTb2 + kW;

// The transposed weights; the last block counts the labels and writes 1 / count of each loss (0 for
// none) to scales: partition, intra 4x4, offset.
__global__ void train_prep_kernel(const float* __restrict__ P, float* __restrict__ T, const int* __restrict__ part,
                                  const int* __restrict__ i4, const int* __restrict__ mvv, int n, float* __restrict__ scales) {
  if (blockIdx.x + 1 < gridDim.x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kTrans) return;
    if (i < kT2) {
      const int ci = i / (9 * C), t = (i / C) % 9, co = i % C;
      T[i] = P[kW1 + (co * 2 + ci) * 9 + t];
    } else {
      const int l = (i - kT2) / kW, k = (i - kT2) % kW, a = k / (9 * C), t = (k / C) % 9, b = k % C;
      // forward: a = ci, b = co; input gradient: a = co, b = ci, taps reversed
      T[i] = l < 2 ? P[(l == 0 ? kW2 : kW3) + (b * C + a) * 9 + t] : P[(l == 2 ? kW3 : kW2) + (a * C + b) * 9 + 8 - t];
    }
    return;
  }
  __shared__ int cnt[3];
  if (threadIdx.x < 3) cnt[threadIdx.x] = 0;
  __syncthreads();
  int np = 0, ni = 0, nm = 0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) { np += part[k] >= 0; nm += mvv[k] != 0; }
  for (int k = threadIdx.x; k < n * 16; k += blockDim.x) ni += i4[k] >= 0;
  np = __reduce_add_sync(0xffffffffu, np);
  ni = __reduce_add_sync(0xffffffffu, ni);
  nm = __reduce_add_sync(0xffffffffu, nm);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&cnt[0], np);
    atomicAdd(&cnt[1], ni);
    atomicAdd(&cnt[2], nm);
  }
  __syncthreads();
  if (threadIdx.x < 3) scales[threadIdx.x] = cnt[threadIdx.x] ? 1.0f / (float)cnt[threadIdx.x] : 0.0f;
}

// A 3x3 convolution of one sample per block (blockIdx.y: a part of its output channels, for batches
// that do not fill the GPU): kHin x kHin input of kCin channels in shared memory, 16 channels at a
// time (two blocks an SM). A thread computes 4 positions of a row x 8 channels: per input channel
// three rows of six samples and 72 weights (the same for the whole warp, but at group borders) for 288
// multiply-adds. kU8: the input are crops (bytes, normalised); kBwd: the input is an output
// gradient, surrounded by zeros (the full correlation with the reversed taps is the input's
// gradient), and the result is masked by the ReLU of the map `act`; otherwise bias and ReLU.
constexpr int kConvChunk = 16;
template <int kHin>
struct ConvShape {
  static constexpr int hout = kHin - 2, groups = (hout + 3) / 4, row = (4 * groups + 2 + 3) / 4 * 4;
  static constexpr int threads = hout * groups;  // of one group of 8 channels
};
template <int kHin, int kCin, bool kU8, bool kBwd>
__global__ void __launch_bounds__(kHin == 24 ? 544 : 416, kHin == 24 ? 1 : 2)
    conv_kernel(const void* __restrict__ in, const float* __restrict__ wt, const float* __restrict__ bias,
                const float* __restrict__ act, float* __restrict__ out, int cgs) {
  using S = ConvShape<kHin>;
  constexpr int kCh = kCin < kConvChunk ? kCin : kConvChunk, kMap = kHin * S::row, npos = S::hout * S::hout;
  extern __shared__ float4 sh4[];
  float* w = (float*)sh4;           // [kCh][9][32]
  float* x = w + kCh * 9 * C;       // [kCh][kHin][row]
  const int n = blockIdx.x, tid = threadIdx.x;
  const int cg = tid / S::threads, pos = tid - cg * S::threads, y = pos / S::groups, x0 = (pos - y * S::groups) * 4;
  const bool on = cg < cgs;
  const int co = (blockIdx.y * cgs + (on ? cg : 0)) * 8;
  float acc[8][4];
#pragma unroll
  for (int o = 0; o < 8; o++)
#pragma unroll
    for (int k = 0; k < 4; k++) acc[o][k] = 0.0f;
  for (int c0 = 0; c0 < kCin; c0 += kCh) {
    if (c0) __syncthreads();
    for (int i = tid; i < kCh * 9 * C / 4; i += blockDim.x) ((float4*)w)[i] = ((const float4*)(wt + c0 * 9 * C))[i];
    for (int i = tid; i < kCh * kMap; i += blockDim.x) {
      const int ci = i / kMap, r = (i - ci * kMap) / S::row, c = i - ci * kMap - r * S::row;
      float v = 0.0f;
      if constexpr (kBwd) {  // the gradient map is kHin - 4 wide
        constexpr int h = kHin - 4;
        if (r >= 2 && r < kHin - 2 && c >= 2 && c < kHin - 2) v = ((const float*)in)[((size_t)n * kCin + c0 + ci) * h * h + (r - 2) * h + c - 2];
      } else if (c < kHin) {
        const size_t at = ((size_t)n * kCin + c0 + ci) * kHin * kHin + r * kHin + c;
        v = kU8 ? pix_norm(((const uint8_t*)in)[at]) : ((const float*)in)[at];
      }
      x[i] = v;
    }
    __syncthreads();
    if (on) {
#pragma unroll 1
      for (int ci = 0; ci < kCh; ci++) {
        const float* xp = x + ci * kMap + y * S::row + x0;
        const float* wp = w + ci * 9 * C + co;
#pragma unroll
        for (int r = 0; r < 3; r++) {
          const float4 a = *(const float4*)(xp + r * S::row);
          const float2 b = *(const float2*)(xp + r * S::row + 4);
          const float v[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
#pragma unroll
          for (int t = 0; t < 3; t++) {
            const float4 w0 = *(const float4*)(wp + (r * 3 + t) * C), w1 = *(const float4*)(wp + (r * 3 + t) * C + 4);
            const float q[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int o = 0; o < 8; o++)
#pragma unroll
              for (int k = 0; k < 4; k++) acc[o][k] = fmaf(q[o], v[t + k], acc[o][k]);
          }
        }
      }
    }
  }
  if (!on) return;
#pragma unroll
  for (int o = 0; o < 8; o++) {
    const size_t base = ((size_t)n * C + co + o) * npos + y * S::hout + x0;
    const float bo = kBwd ? 0.0f : bias[co + o];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (x0 + k < S::hout) out[base + k] = kBwd ? (act[base + k] > 0.0f ? acc[o][k] : 0.0f) : fmaxf(acc[o][k] + bo, 0.0f);
  }
}
template <int kHin, int kCin>
constexpr int conv_smem() {
  return ((kCin < kConvChunk ? kCin : kConvChunk) * (9 * C + kHin * ConvShape<kHin>::row)) * 4;
}

// Heads, losses and their gradient (a block per sample): labels part [N] (-1 none), i4 [N][16] (raster
// 4x4 blocks, -1 none), mv [N][2] with mvv [N] (0 none); scales: train_prep_kernel's. Writes the logits
// (optional), the sample's part of the loss and of the head parameters' gradients (loss_part [N],
// head_part [N][kHeadParams]) and dA3 (the gradient at the conv3 map, masked by its ReLU).
constexpr int kHeadThreads = 256, kHeadRow = 325;
__global__ void __launch_bounds__(kHeadThreads) heads_kernel(const float* __restrict__ A3, const float* __restrict__ P, const int* __restrict__ part,
                             const int* __restrict__ i4, const float* __restrict__ mv, const int* __restrict__ mvv,
                             const float* __restrict__ scales, float mv_weight, float* __restrict__ logits,
                             float* __restrict__ head_part, float* __restrict__ dA3, float* __restrict__ loss_part) {
  extern __shared__ float4 sh4[];
  float* a = (float*)sh4;  // [32][kHeadRow]
  __shared__ float H[kHeadParams], f[17][C], rows[8][C], lg[kLogits], dl[kLogits], dg[C], df[16][C], lsum[18];
  const int n = blockIdx.x, t = threadIdx.x, c = t & 31, q = t >> 5;
  const float* src = A3 + (size_t)n * kA3;
  for (int i = t; i < kA3; i += kHeadThreads) a[(i / 324) * kHeadRow + i % 324] = src[i];
  for (int i = t; i < kHeadParams; i += kHeadThreads) H[i] = P[kWp + i];
  for (int i = t; i < kLogits; i += kHeadThreads) dl[i] = 0.0f;
  if (t < 18) lsum[t] = 0.0f;
  __syncthreads();
  // pooling: warp q sums blocks 2q and 2q + 1, and the rows q, q + 8, q + 16 of the whole map
  const float* m = a + c * kHeadRow;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int b = 2 * q + k;
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i++) s += m[((b >> 2) * 4 + 1 + (i >> 2)) * 18 + (b & 3) * 4 + 1 + (i & 3)];
    f[1 + b][c] = s / 16.0f;
  }
  float s = 0.0f;
  for (int r = q; r < 18; r += 8)
#pragma unroll
    for (int i = 0; i < 18; i++) s += m[r * 18 + i];
  rows[q][c] = s;
  __syncthreads();
  if (t < C) {
    float all = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k++) all += rows[k][t];
    f[0][t] = all / 324.0f;
  }
  __syncthreads();
  if (t < kLogits) {  // partition 4, offset 2, intra 4x4 9 per block
    const int b = t < 6 ? 0 : 1 + (t - 6) / 9, o = t < 4 ? t : (t < 6 ? t - 4 : (t - 6) % 9);
    const int wo = t < 4 ? 0 : (t < 6 ? kWm - kWp : kWi - kWp), bo = t < 4 ? kBp - kWp : (t < 6 ? kBm - kWp : kBi - kWp);
    float v = H[bo + o];
#pragma unroll
    for (int k = 0; k < C; k++) v += H[wo + o * C + k] * f[b][k];
    lg[t] = v;
    if (logits) logits[(size_t)n * kLogits + t] = v;
  }
  __syncthreads();
  const float sp = scales[0], si = scales[1], sm = scales[2];
  if (t == 0 && part[n] >= 0) {
    const float mx = fmaxf(fmaxf(lg[0], lg[1]), fmaxf(lg[2], lg[3]));
    float se = 0.0f;
    for (int o = 0; o < 4; o++) se += expf(lg[o] - mx);
    for (int o = 0; o < 4; o++) dl[o] = sp * (expf(lg[o] - mx) / se - (o == part[n] ? 1.0f : 0.0f));
    lsum[16] = sp * (logf(se) + mx - lg[part[n]]);
  }
  if (t == 32 && mvv[n]) {  // Huber (delta 1) on the offset in units of 16 quarter samples
    float L = 0.0f;
    for (int o = 0; o < 2; o++) {
      const float d = lg[4 + o] - mv[2 * n + o], ad = fabsf(d);
      L += sm * mv_weight * (ad <= 1.0f ? 0.5f * d * d : ad - 0.5f);
      dl[4 + o] = sm * mv_weight * (ad <= 1.0f ? d : (d > 0 ? 1.0f : -1.0f));
    }
    lsum[17] = L;
  }
  if (t >= 64 && t < 80) {
    const int b = t - 64, lab = i4[n * 16 + b];
    if (lab >= 0) {
      const float* li = lg + 6 + b * 9;
      float mx = li[0], se = 0.0f;
      for (int o = 1; o < 9; o++) mx = fmaxf(mx, li[o]);
      for (int o = 0; o < 9; o++) se += expf(li[o] - mx);
      for (int o = 0; o < 9; o++) dl[6 + b * 9 + o] = si * (expf(li[o] - mx) / se - (o == lab ? 1.0f : 0.0f));
      lsum[b] = si * (logf(se) + mx - li[lab]);
    }
  }
  __syncthreads();
  if (t == 0) {
    float L = 0.0f;
    for (int k = 0; k < 18; k++) L += lsum[k];
    loss_part[n] = L;
  }
  // this sample's part of the head parameters' gradients
  for (int e = t; e < kHeadParams; e += kHeadThreads) {
    const int p = kWp + e;
    float g = 0.0f;
    if (p < kBp) g = dl[e / C] * f[0][e % C];
    else if (p < kWm) g = dl[p - kBp];
    else if (p < kBm) g = dl[4 + (p - kWm) / C] * f[0][(p - kWm) % C];
    else if (p < kWi) g = dl[4 + p - kBm];
    else if (p < kBi)
      for (int b = 0; b < 16; b++) g += dl[6 + b * 9 + (p - kWi) / C] * f[1 + b][(p - kWi) % C];
    else
      for (int b = 0; b < 16; b++) g += dl[6 + b * 9 + p - kBi];
    head_part[(size_t)n * kHeadParams + e] = g;
  }
  // the gradient at the pooled features
  if (t < C) {
    float g = 0.0f;
    for (int o = 0; o < 4; o++) g += H[o * C + t] * dl[o];
    for (int o = 0; o < 2; o++) g += H[kWm - kWp + o * C + t] * dl[4 + o];
    dg[t] = g / 324.0f;
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int b = 2 * q + k;
    float g = 0.0f;
    for (int o = 0; o < 9; o++) g += H[kWi - kWp + o * C + c] * dl[6 + b * 9 + o];
    df[b][c] = g / 16.0f;
  }
  __syncthreads();
  // dA3 = pooled gradients spread over the map, masked by the ReLU
  float* d = dA3 + (size_t)n * kA3;
  for (int i = t; i < kA3; i += kHeadThreads) {
    const int ch = i / 324, p = i % 324, r = p / 18, x = p % 18;
    float v = dg[ch];
    if (r >= 1 && r <= 16 && x >= 1 && x <= 16) v += df[((r - 1) >> 2) * 4 + ((x - 1) >> 2)][ch];
    d[i] = a[ch * kHeadRow + p] > 0.0f ? v : 0.0f;
  }
}

// Weight gradients of a 32 -> 32 layer, dW[co][ci][t] = sum over samples, positions of dout[co][p]
// in[ci][p + t]: a block takes `per` samples one after the other, a thread 4 output channels x 9
// taps of one input channel (its lane) over half of the rows: per 4 positions of a row three rows of
// six samples and 4 x 4 gradients (the same for the whole warp) for 144 multiply-adds. Channel maps are
// 20 banks apart (mod 32), which spreads the lanes' 16-byte loads over all banks. Partial sums, a row of
// kWgRow per (block, half), added up by train_reduce_kernel; the bias gradients behind the weights of
// half 0.
constexpr int kWgRow = kW + C, kWgThreads = 512;
template <int kHin>
struct WgShape {
  static constexpr int hout = kHin - 2, row = 24, map = kHin * row + (kHin * row % 32 == 16 ? 4 : 20), drow = 20, dmap = hout * drow;
  static_assert(map % 32 == 20 || map % 32 == 12 || map % 32 == 4, "the lanes' maps fall into different banks");
  static constexpr int smem = C * (map + dmap) * 4;
};
template <int kHin>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_kernel(const float* __restrict__ dout, const float* __restrict__ in, int n_samples,
                                                              int per, float* __restrict__ part) {
  using S = WgShape<kHin>;
  constexpr int hout = S::hout;
  extern __shared__ float4 sh4[];
  float* x = (float*)sh4;        // [32][map]: rows of 24
  float* d = x + C * S::map;     // [32][hout][20], columns past hout zero
  const int tid = threadIdx.x, lane = tid & 31, cg = (tid >> 5) & 7, half = tid >> 8;
  const int y0 = half ? hout / 2 : 0, y1 = half ? hout : hout / 2;
  float acc[4][9];
#pragma unroll
  for (int o = 0; o < 4; o++)
#pragma unroll
    for (int t = 0; t < 9; t++) acc[o][t] = 0.0f;
  float bsum = 0.0f;
  for (int s = 0; s < per; s++) {
    const int n = blockIdx.x * per + s;
    if (n >= n_samples) break;
    __syncthreads();
    for (int i = tid; i < C * kHin * kHin; i += kWgThreads) {
      const int ci = i / (kHin * kHin), p = i - ci * kHin * kHin, r = p / kHin;
      x[ci * S::map + r * S::row + p - r * kHin] = in[(size_t)n * C * kHin * kHin + i];
    }
    for (int i = tid; i < C * S::dmap; i += kWgThreads) {
      const int r = i / S::drow, c = i - r * S::drow;
      d[i] = c < hout ? dout[((size_t)n * C * hout + r) * hout + c] : 0.0f;
    }
    if (kHin < 24)  // the columns past the map, multiplied with zero gradients
      for (int i = tid; i < C * kHin * (24 - kHin); i += kWgThreads) {
        const int r = i / (24 - kHin);
        x[(r / kHin) * S::map + (r % kHin) * S::row + kHin + i % (24 - kHin)] = 0.0f;
      }
    __syncthreads();
    const float* xc = x + lane * S::map;
    const float* dc = d + cg * 4 * S::dmap;
#pragma unroll 1
    for (int y = y0; y < y1; y++)
#pragma unroll 1
      for (int g = 0; g < 5; g++) {
        float4 dv[4];
#pragma unroll
        for (int o = 0; o < 4; o++) dv[o] = *(const float4*)(dc + o * S::dmap + y * S::drow + 4 * g);
#pragma unroll
        for (int r = 0; r < 3; r++) {
          const float4 a = *(const float4*)(xc + (y + r) * S::row + 4 * g);
          const float2 b = *(const float2*)(xc + (y + r) * S::row + 4 * g + 4);
          const float v[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
#pragma unroll
          for (int t = 0; t < 3; t++)
#pragma unroll
            for (int o = 0; o < 4; o++) {
              acc[o][r * 3 + t] = fmaf(dv[o].x, v[t], acc[o][r * 3 + t]);
              acc[o][r * 3 + t] = fmaf(dv[o].y, v[t + 1], acc[o][r * 3 + t]);
              acc[o][r * 3 + t] = fmaf(dv[o].z, v[t + 2], acc[o][r * 3 + t]);
              acc[o][r * 3 + t] = fmaf(dv[o].w, v[t + 3], acc[o][r * 3 + t]);
            }
        }
      }
    // bias: sixteen threads a channel
    for (int i = tid & 15; i < S::dmap; i += 16) bsum += d[(tid >> 4) * S::dmap + i];
  }
  float* row = part + ((size_t)blockIdx.x * 2 + half) * kWgRow;
#pragma unroll
  for (int o = 0; o < 4; o++)
#pragma unroll
    for (int t = 0; t < 9; t++) row[((cg * 4 + o) * C + lane) * 9 + t] = acc[o][t];
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) bsum += __shfl_xor_sync(0xffffffffu, bsum, o);
  float* row0 = part + (size_t)blockIdx.x * 2 * kWgRow;
  if ((tid & 15) == 0) {
    row0[kW + (tid >> 4)] = bsum;
    row0[kWgRow + kW + (tid >> 4)] = 0.0f;
  }
}
// The first layer's: warp = (4 output channels, input channel), lane = row of the map, its sums over
// the row's positions, then over the lanes. A row of kWg1Row per block: the weights, then the biases.
constexpr int kWg1Row = 2 * 9 * C + C, kWg1D = 23, kWg1X = 25;
constexpr int kWg1Smem = (C * 22 * kWg1D + 2 * 24 * kWg1X) * 4;
__global__ void __launch_bounds__(kWgThreads, 1) wgrad1_kernel(const float* __restrict__ dout, const uint8_t* __restrict__ crops, int n_samples,
                                                               int per, float* __restrict__ part) {
  extern __shared__ float4 sh4[];
  float* d = (float*)sh4;          // [32][22][23]
  float* x = d + C * 22 * kWg1D;   // [2][24][25]
  const int tid = threadIdx.x, lane = tid & 31, cg = (tid >> 5) & 7, ci = tid >> 8;
  float acc[4][9], bacc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int o = 0; o < 4; o++)
#pragma unroll
    for (int t = 0; t < 9; t++) acc[o][t] = 0.0f;
  for (int s = 0; s < per; s++) {
    const int n = blockIdx.x * per + s;
    if (n >= n_samples) break;
    __syncthreads();
    for (int i = tid; i < kA1; i += kWgThreads) d[(i / 22) * kWg1D + i % 22] = dout[(size_t)n * kA1 + i];
    for (int i = tid; i < kIn; i += kWgThreads) x[(i / 24) * kWg1X + i % 24] = pix_norm(crops[(size_t)n * kIn + i]);
    __syncthreads();
    if (lane < 22) {
      const float* xr = x + (ci * 24 + lane) * kWg1X;
      const float* dr = d + (cg * 4 * 22 + lane) * kWg1D;
#pragma unroll 2
      for (int p = 0; p < 22; p++) {
        float v[9];
#pragma unroll
        for (int t = 0; t < 9; t++) v[t] = xr[(t / 3) * kWg1X + p + t % 3];
#pragma unroll
        for (int o = 0; o < 4; o++) {
          const float g = dr[o * 22 * kWg1D + p];
          bacc[o] += g;
#pragma unroll
          for (int t = 0; t < 9; t++) acc[o][t] = fmaf(g, v[t], acc[o][t]);
        }
      }
    }
  }
  float* row = part + (size_t)blockIdx.x * kWg1Row;
#pragma unroll
  for (int o = 0; o < 4; o++) {
#pragma unroll
    for (int t = 0; t < 9; t++) {
      float v = acc[o][t];
#pragma unroll
      for (int k = 16; k > 0; k >>= 1) v += __shfl_xor_sync(0xffffffffu, v, k);
      if (lane == 0) row[((cg * 4 + o) * 2 + ci) * 9 + t] = v;
    }
    float v = bacc[o];
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) v += __shfl_xor_sync(0xffffffffu, v, k);
    if (lane == 0 && ci == 0) row[2 * 9 * C + cg * 4 + o] = v;
  }
}
// The gradients: parameter e's partial sums over the blocks (or samples) that made them; the last one
// is the loss. 32 parameters a block, eight strided parts of the rows each.
struct TrainParts {
  const float *w1, *w2, *w3, *head, *loss;
  int n1, n2, n;  // rows of w1, of w2 and w3, of head and loss
};
__global__ void __launch_bounds__(256) train_reduce_kernel(TrainParts tp, float* __restrict__ G, float* __restrict__ loss) {
  __shared__ float red[8][32];
  const int e = blockIdx.x * 32 + (threadIdx.x & 31), q = threadIdx.x >> 5;
  const float* p = nullptr;
  int rows = 0, stride = 0;
  if (e < kW2) { p = tp.w1 + e; rows = tp.n1; stride = kWg1Row; }
  else if (e < kW3) { p = tp.w2 + e - kW2; rows = tp.n2; stride = kWgRow; }
  else if (e < kWp) { p = tp.w3 + e - kW3; rows = tp.n2; stride = kWgRow; }
  else if (e < kParams) { p = tp.head + e - kWp; rows = tp.n; stride = kHeadParams; }
  else if (e == kParams) { p = tp.loss; rows = tp.n; stride = 1; }
  float s = 0.0f;
#pragma unroll 4
  for (int r = q; r < rows; r += 8) s += p[(size_t)r * stride];
  red[q][threadIdx.x & 31] = s;
  __syncthreads();
  if (q == 0) {
    s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k++) s += red[k][threadIdx.x];
    if (e < kParams) G[e] = s;
    else if (e == kParams) *loss = s;
  }
}
static_assert(kW2 - kW1 == kWg1Row && kW3 - kW2 == kWgRow && kWp - kW3 == kWgRow && kW1 == 0, "partial rows in the parameters' order");

__global__ void adam_kernel(float* P, const float* G, float* m, float* v, int n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = G[i];
  m[i] = b1 * m[i] + (1.0f - b1) * g;
  v[i] = b2 * v[i] + (1.0f - b2) * g * g;
  P[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
}

// Crops of the training set: sample k is macroblock (mbx, mby) of picture pics[k] (cur and prev
// luma, display size, stride), 2 x 24 x 24 bytes, coordinates clamped to the picture.
struct CropSrc {
  const uint8_t* cur;
  const uint8_t* prev;
  int mbx, mby;
};
__global__ void crops_kernel(const CropSrc* __restrict__ src, int n, int width, int height, int stride,
                             uint8_t* __restrict__ out) {
  const int k = blockIdx.x;
  if (k >= n) return;
  const CropSrc s = src[k];
  for (int i = threadIdx.x; i < kIn; i += blockDim.x) {
    const int ch = i / 576, r = (i % 576) / 24, c = i % 24;
    const int y = min(max(s.mby * 16 - 4 + r, 0), height - 1), x = min(max(s.mbx * 16 - 4 + c, 0), width - 1);
    out[(size_t)k * kIn + i] = (ch ? s.prev : s.cur)[(size_t)y * stride + x];
  }
}

}  // namespace

// ---------------------------------------------------------------------------------------------
struct rg_net {
  int device = 0;
  float* P = nullptr;      // parameters (f32)
  float* G = nullptr;      // gradients
  float* M = nullptr;      // Adam moments
  float* V = nullptr;
  int step = 0;
  __nv_bfloat16* bops = nullptr;  // inference B operands (from P)
  bool bops_stale = true;
  int* counter = nullptr;  // [0] strip ticket, [1] error word
  // training scratch
  float *a1 = nullptr, *a2 = nullptr, *a3 = nullptr, *d3 = nullptr, *d2 = nullptr, *d1 = nullptr, *loss = nullptr;
  float *trans = nullptr, *parts = nullptr;  // transposed weights and scales; partial sums of the gradients
  int cap = 0;
  InferJob* jobs = nullptr;
  int jobs_cap = 0;
  int part_k = 3, i4_k = 3;  // hint policy (rg_net_set_hint_policy)
  float part_margin = INFINITY, i4_margin = INFINITY;
  int coarse_range = 32;      // rg_net_set_coarse_range
};

namespace {
int nfail(int code, const char* msg) {
  rg::set_last_error(msg);
  return code;
}
#define NCK(expr)                                                    \
  do {                                                               \
    cudaError_t e_ = (expr);                                         \
    if (e_ != cudaSuccess) return nfail(RG_ERR_CUDA, cudaGetErrorString(e_)); \
  } while (0)

// The B operands of the three layers in the shared-memory order the inference kernel loads: per
// MMA 1 KB -- two 8-element halves of K (512 bytes apart), 32 rows of N (output channels) of 16 bytes.
void pack_bops(const std::vector<float>& p, std::vector<__nv_bfloat16>& out) {
  out.assign((size_t)(kB1Mmas + 2 * kBMmas) * 512, __float2bfloat16(0.0f));
  auto put = [&](int mma, int n, int k, float v) { out[(size_t)mma * 512 + (k >> 3) * 256 + n * 8 + (k & 7)] = __float2bfloat16(v); };
  const int pairs[kB1Mmas][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {8, 9}};
  for (int m = 0; m < kB1Mmas; m++)
    for (int n = 0; n < C; n++)
      for (int h = 0; h < 2; h++) {
        int t = pairs[m][h];
        if (t > 8) continue;
        for (int ci = 0; ci < 2; ci++) put(m, n, 8 * h + ci, p[kW1 + (n * 2 + ci) * 9 + t]);
      }
  for (int layer = 0; layer < 2; layer++) {
    const int woff = layer == 0 ? kW2 : kW3, base = kB1Mmas + layer * kBMmas;
    for (int t = 0; t < 9; t++)
      for (int h = 0; h < 2; h++)
        for (int n = 0; n < C; n++)
          for (int k = 0; k < 16; k++) put(base + t * 2 + h, n, k, p[woff + (n * C + 16 * h + k) * 9 + t]);
  }
}
int ensure_bops(rg_net* net) {
  if (!net->bops_stale) return RG_OK;
  std::vector<float> p(kParams);
  NCK(cudaMemcpy(p.data(), net->P, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
  std::vector<__nv_bfloat16> b;
  pack_bops(p, b);
  NCK(cudaMemcpy(net->bops, b.data(), b.size() * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice));
  net->bops_stale = false;
  return RG_OK;
}
// Samples of one block of the weight-gradient kernels: the batch spread over the SMs.
int wgrad_per(int n, int sms) { return (n + sms - 1) / sms; }
// Floats of the partial sums of batches of up to n samples: a row per block of the weight-gradient kernels (one
// an SM at most, whatever the batch), and one per sample of the heads.
size_t parts_floats(int n, int sms) {
  return (size_t)(n < sms ? n : sms) * (kWg1Row + 2 * 2 * kWgRow) + (size_t)n * (kHeadParams + 1);
}
int ensure_train(rg_net* net, int n, int sms) {
  if (n <= net->cap) return RG_OK;
  cudaFree(net->a1); cudaFree(net->a2); cudaFree(net->a3); cudaFree(net->d3); cudaFree(net->d2); cudaFree(net->d1);
  cudaFree(net->parts);
  net->a1 = net->a2 = net->a3 = net->d3 = net->d2 = net->d1 = net->parts = nullptr;
  net->cap = 0;
  size_t f = sizeof(float);
  if ((!net->trans && cudaMalloc((void**)&net->trans, f * (kTrans + 4)) != cudaSuccess) ||
      cudaMalloc((void**)&net->parts, f * parts_floats(n, sms)) != cudaSuccess ||
      cudaMalloc((void**)&net->a1, f * n * kA1) != cudaSuccess || cudaMalloc((void**)&net->a2, f * n * kA2) != cudaSuccess ||
      cudaMalloc((void**)&net->a3, f * n * kA3) != cudaSuccess || cudaMalloc((void**)&net->d3, f * n * kA3) != cudaSuccess ||
      cudaMalloc((void**)&net->d2, f * n * kA2) != cudaSuccess || cudaMalloc((void**)&net->d1, f * n * kA1) != cudaSuccess)
    return nfail(RG_ERR_OOM, "rg_net: training scratch allocation failed");
  net->cap = n;
  return RG_OK;
}
// One convolution layer of a training pass: a block per sample, its output channels over four blocks
// when the samples alone do not fill the GPU.
template <int kHin, int kCin, bool kU8, bool kBwd>
void launch_conv(int n, int sms, const void* in, const float* wt, const float* bias, const float* act, float* out) {
  constexpr int smem = conv_smem<kHin, kCin>();
  cudaFuncSetAttribute(conv_kernel<kHin, kCin, kU8, kBwd>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int split = n >= sms ? 1 : (2 * n >= sms ? 2 : 4), cgs = 4 / split;
  const int threads = (cgs * ConvShape<kHin>::threads + 31) / 32 * 32;
  conv_kernel<kHin, kCin, kU8, kBwd><<<dim3(n, split), threads, smem>>>(in, wt, bias, act, out, cgs);
}
template <int kHin>
void launch_wgrad(int n, int per, const float* dout, const float* in, float* part) {
  constexpr int smem = WgShape<kHin>::smem;
  cudaFuncSetAttribute(wgrad_kernel<kHin>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  wgrad_kernel<kHin><<<(n + per - 1) / per, kWgThreads, smem>>>(dout, in, n, per, part);
}
}  // namespace

extern "C" {

int32_t rg_net_param_count(void) { return kParams; }

rg_net* rg_net_create(int32_t device, uint64_t seed) {
  if (cudaSetDevice(device) != cudaSuccess) { nfail(RG_ERR_CUDA, "rg_net_create: cudaSetDevice failed"); return nullptr; }
  auto* net = new rg_net();
  net->device = device;
  size_t pb = sizeof(float) * kParams;
  if (cudaMalloc((void**)&net->P, pb) != cudaSuccess || cudaMalloc((void**)&net->G, pb) != cudaSuccess ||
      cudaMalloc((void**)&net->M, pb) != cudaSuccess || cudaMalloc((void**)&net->V, pb) != cudaSuccess ||
      cudaMalloc((void**)&net->bops, (size_t)(kB1Mmas + 2 * kBMmas) * 1024) != cudaSuccess ||
      cudaMalloc((void**)&net->counter, 2 * sizeof(int)) != cudaSuccess ||
      cudaMalloc((void**)&net->loss, sizeof(float)) != cudaSuccess) {
    nfail(RG_ERR_OOM, "rg_net_create: allocation failed");
    rg_net_destroy(net);
    return nullptr;
  }
  // He-uniform initialisation from a 64-bit LCG (heads a tenth of that)
  std::vector<float> p(kParams, 0.0f);
  uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
  auto uni = [&]() {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    return (float)((s >> 40) & 0xFFFFFF) / 16777216.0f * 2.0f - 1.0f;
  };
  auto fill = [&](int off, int n, float lim) { for (int i = 0; i < n; i++) p[off + i] = lim * uni(); };
  fill(kW1, C * 2 * 9, std::sqrt(6.0f / 18.0f));
  fill(kW2, C * C * 9, std::sqrt(6.0f / 288.0f));
  fill(kW3, C * C * 9, std::sqrt(6.0f / 288.0f));
  fill(kWp, 4 * C, 0.1f * std::sqrt(6.0f / 32.0f));
  fill(kWm, 2 * C, 0.1f * std::sqrt(6.0f / 32.0f));
  fill(kWi, 9 * C, 0.1f * std::sqrt(6.0f / 32.0f));
  if (rg_net_set_params(net, p.data(), kParams) != RG_OK) {
    rg_net_destroy(net);
    return nullptr;
  }
  return net;
}

void rg_net_destroy(rg_net* net) {
  if (!net) return;
  cudaFree(net->P); cudaFree(net->G); cudaFree(net->M); cudaFree(net->V); cudaFree(net->bops); cudaFree(net->counter);
  cudaFree(net->a1); cudaFree(net->a2); cudaFree(net->a3); cudaFree(net->d3); cudaFree(net->d2); cudaFree(net->d1);
  cudaFree(net->loss); cudaFree(net->jobs); cudaFree(net->trans); cudaFree(net->parts);
  delete net;
}

int rg_net_set_params(rg_net* net, const float* params, int32_t count) {
  if (!net || !params || count != kParams) return nfail(RG_ERR_INVALID, "rg_net_set_params: bad arguments");
  NCK(cudaSetDevice(net->device));
  NCK(cudaMemcpy(net->P, params, sizeof(float) * kParams, cudaMemcpyHostToDevice));
  NCK(cudaMemset(net->M, 0, sizeof(float) * kParams));
  NCK(cudaMemset(net->V, 0, sizeof(float) * kParams));
  net->step = 0;
  net->bops_stale = true;
  return RG_OK;
}

int rg_net_get_params(const rg_net* net, float* params, int32_t count) {
  if (!net || !params || count != kParams) return nfail(RG_ERR_INVALID, "rg_net_get_params: bad arguments");
  NCK(cudaMemcpy(params, net->P, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
  return RG_OK;
}

int rg_net_crops(rg_net* net, const uint8_t* const* cur, const uint8_t* const* prev, const int32_t* mb_xy, int32_t n,
                 int32_t width, int32_t height, size_t stride, uint8_t* dev_out, void* stream) {
  if (!net || !cur || !prev || !mb_xy || !dev_out || n < 0) return nfail(RG_ERR_INVALID, "rg_net_crops: bad arguments");
  if (!n) return RG_OK;
  std::vector<CropSrc> h(n);
  for (int k = 0; k < n; k++) h[k] = CropSrc{cur[k], prev[k], mb_xy[2 * k], mb_xy[2 * k + 1]};
  CropSrc* d = nullptr;
  NCK(cudaMalloc((void**)&d, sizeof(CropSrc) * n));
  cudaStream_t st = (cudaStream_t)stream;
  NCK(cudaMemcpyAsync(d, h.data(), sizeof(CropSrc) * n, cudaMemcpyHostToDevice, st));
  crops_kernel<<<n, 256, 0, st>>>(d, n, width, height, (int)stride, dev_out);
  NCK(cudaGetLastError());
  NCK(cudaStreamSynchronize(st));
  cudaFree(d);
  return RG_OK;
}

int rg_net_forward_backward(rg_net* net, const uint8_t* dev_crops, int32_t n, const int32_t* dev_part,
                            const int32_t* dev_i4, const float* dev_mv, const int32_t* dev_mvv, float mv_weight,
                            float* dev_logits, float* loss_out, float* grads_out) {
  if (!net || !dev_crops || n < 1 || !dev_part || !dev_i4 || !dev_mv || !dev_mvv)
    return nfail(RG_ERR_INVALID, "rg_net_forward_backward: bad arguments");
  NCK(cudaSetDevice(net->device));
  int sms = 0;
  NCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device));
  int r = ensure_train(net, n, sms);
  if (r) return r;
  const float* P = net->P;
  float *T = net->trans, *scales = T + kTrans;
  // the labels' counts normalise each loss
  train_prep_kernel<<<(kTrans + 255) / 256 + 1, 256>>>(P, T, dev_part, dev_i4, dev_mvv, n, scales);
  launch_conv<24, 2, true, false>(n, sms, dev_crops, T + kT1, P + kB1, nullptr, net->a1);
  launch_conv<22, C, false, false>(n, sms, net->a1, T + kT2, P + kB2, nullptr, net->a2);
  launch_conv<20, C, false, false>(n, sms, net->a2, T + kT3, P + kB3, nullptr, net->a3);
  const int per = wgrad_per(n, sms), nb = (n + per - 1) / per;
  float* w1 = net->parts;
  float* w2 = w1 + (size_t)nb * kWg1Row;
  float* w3 = w2 + (size_t)nb * 2 * kWgRow;
  float* head = w3 + (size_t)nb * 2 * kWgRow;
  float* loss = head + (size_t)n * kHeadParams;
  constexpr int hs = C * kHeadRow * 4;
  cudaFuncSetAttribute(heads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, hs);
  heads_kernel<<<n, kHeadThreads, hs>>>(net->a3, P, dev_part, dev_i4, dev_mv, dev_mvv, scales, mv_weight, dev_logits, head,
                                        net->d3, loss);
  launch_conv<22, C, false, true>(n, sms, net->d3, T + kTb3, nullptr, net->a2, net->d2);
  launch_conv<24, C, false, true>(n, sms, net->d2, T + kTb2, nullptr, net->a1, net->d1);
  launch_wgrad<20>(n, per, net->d3, net->a2, w3);
  launch_wgrad<22>(n, per, net->d2, net->a1, w2);
  cudaFuncSetAttribute(wgrad1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWg1Smem);
  wgrad1_kernel<<<nb, kWgThreads, kWg1Smem>>>(net->d1, dev_crops, n, per, w1);
  train_reduce_kernel<<<(kParams + 1 + 31) / 32, 256>>>(TrainParts{w1, w2, w3, head, loss, nb, 2 * nb, n}, net->G, net->loss);
  NCK(cudaGetLastError());
  NCK(cudaDeviceSynchronize());
  if (loss_out) NCK(cudaMemcpy(loss_out, net->loss, sizeof(float), cudaMemcpyDeviceToHost));
  if (grads_out) NCK(cudaMemcpy(grads_out, net->G, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
  return RG_OK;
}

int rg_net_adam_step(rg_net* net, float lr) {
  if (!net || !(lr > 0.0f)) return nfail(RG_ERR_INVALID, "rg_net_adam_step: bad arguments");
  net->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - std::pow(b1, (float)net->step), c2 = 1.0f - std::pow(b2, (float)net->step);
  adam_kernel<<<(kParams + 255) / 256, 256>>>(net->P, net->G, net->M, net->V, kParams, lr, b1, b2, 1e-8f, c1, c2);
  NCK(cudaGetLastError());
  net->bops_stale = true;
  return RG_OK;
}

int rg_net_predict_hints(rg_net* net, const uint8_t* const* dev_cur, const uint8_t* const* dev_prev, int32_t n_pictures,
                         int32_t width, int32_t height, size_t stride, rg_mb_hint* const* dev_hints,
                         float* const* dev_logits, void* stream) {
  if (!net || !dev_cur || !dev_prev || !dev_hints || n_pictures < 1 || width < 1 || height < 1 || stride < (size_t)width)
    return nfail(RG_ERR_INVALID, "rg_net_predict_hints: bad arguments");
  NCK(cudaSetDevice(net->device));
  int r = ensure_bops(net);
  if (r) return r;
  if (n_pictures > net->jobs_cap) {
    cudaFree(net->jobs);
    if (cudaMalloc((void**)&net->jobs, sizeof(InferJob) * n_pictures) != cudaSuccess) {
      net->jobs_cap = 0;
      return nfail(RG_ERR_OOM, "rg_net_predict_hints: job list allocation failed");
    }
    net->jobs_cap = n_pictures;
  }
  std::vector<InferJob> h(n_pictures);
  for (int k = 0; k < n_pictures; k++)
    h[k] = InferJob{dev_cur[k], dev_prev[k], dev_hints[k], dev_logits ? dev_logits[k] : nullptr};
  cudaStream_t st = (cudaStream_t)stream;
  NCK(cudaMemcpyAsync(net->jobs, h.data(), sizeof(InferJob) * n_pictures, cudaMemcpyHostToDevice, st));
  NCK(cudaMemsetAsync(net->counter, 0, 2 * sizeof(int), st));
  InferParams ip;
  ip.jobs = net->jobs;
  ip.n_jobs = n_pictures;
  ip.width = width;
  ip.height = height;
  ip.stride = (int)stride;
  ip.mb_w = (width + 15) / 16;
  ip.mb_h = (height + 15) / 16;
  ip.strips_per_row = (ip.mb_w + kStripMbs - 1) / kStripMbs;
  ip.bops = net->bops;
  ip.params = net->P;
  ip.counter = net->counter;
  ip.error = net->counter + 1;
  ip.part_k = net->part_k;
  ip.i4_k = net->i4_k;
  ip.part_margin = net->part_margin;
  ip.i4_margin = net->i4_margin;
  NCK(cudaFuncSetAttribute(cnn_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemInfer));
  NCK(cudaFuncSetAttribute(cnn_infer_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, net->device);
  const int strips = n_pictures * ip.mb_h * ip.strips_per_row;
  const int ctas = kCtasPerSm * sms < strips ? kCtasPerSm * sms : strips;
  cnn_infer_kernel<<<ctas, kThreads + 32, kSmemInfer, st>>>(ip);
  NCK(cudaGetLastError());
  if (net->coarse_range > 0) {
    CoarseParams cp{net->jobs, n_pictures, width, height, (int)stride, ip.mb_w, ip.mb_h, net->coarse_range / 2};
    const unsigned blocks = (unsigned)n_pictures * ip.mb_h * ((ip.mb_w + kCoarseMbs - 1) / kCoarseMbs);
    coarse_motion_kernel<<<blocks, 32 * kCoarseMbs, 0, st>>>(cp);
    NCK(cudaGetLastError());
  }
  return RG_OK;
}

int rg_net_set_coarse_range(rg_net* net, int32_t range) {
  if (!net || range < 0 || range > 2 * kCoarseMaxR || (range & 1)) return nfail(RG_ERR_INVALID, "rg_net_set_coarse_range: bad arguments");
  net->coarse_range = range;
  return RG_OK;
}

int rg_net_set_hint_policy(rg_net* net, int32_t part_k, float part_margin, int32_t i4_k, float i4_margin) {
  if (!net || part_k < 1 || part_k > 4 || i4_k < 1 || i4_k > 9 || !(part_margin >= 0.0f) || !(i4_margin >= 0.0f))
    return nfail(RG_ERR_INVALID, "rg_net_set_hint_policy: bad arguments");
  net->part_k = part_k;
  net->part_margin = part_margin;
  net->i4_k = i4_k;
  net->i4_margin = i4_margin;
  return RG_OK;
}

int rg_net_check(rg_net* net, void* stream) {
  if (!net) return nfail(RG_ERR_INVALID, "rg_net_check: null network");
  int e[2] = {0, 0};
  NCK(cudaMemcpyAsync(e, net->counter, sizeof e, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  NCK(cudaStreamSynchronize((cudaStream_t)stream));
  if (e[1]) return nfail(RG_ERR_TIMEOUT, "rg_net_predict_hints: a wait on the tensor cores gave up");
  return RG_OK;
}

}  // extern "C"
