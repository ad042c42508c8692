// B200 (sm_100a) macroblock engine: one warp analyses, reconstructs or deblocks one macroblock.
//
// A picture is processed as a 2:1 wavefront over anti-diagonals d = mb_x + 2 mb_y: every
// macroblock of diagonal d depends only on macroblocks of smaller diagonals (left, top, top-left
// and top-right neighbours: unfiltered reconstruction for intra edges, motion for the median
// predictor), so one launch per diagonal reproduces the reference's raster-order decisions
// exactly. Deblocking of diagonal d runs in the launch of analysis diagonal d + 3: by then every
// macroblock that reads its unfiltered pixels (right, below, below-left, below-right neighbours)
// has been analysed, and the two touch disjoint samples. Streams (independent GOPs) sit side by
// side in blockIdx.y.
//
// Arithmetic follows ragdoll's Balanced encoder (crates/ragdoll-codec/src/h264/enc.rs) and the
// scalar kernels it calls (crates/ragdoll-simd/src/*.rs); citations are given per function.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "h264_consts.h"

namespace rg {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr uint32_t UMAX = 0xffffffffu;

__constant__ uint16_t c_lambda[52];
__constant__ uint8_t c_dec4[16];
__constant__ uint8_t c_dec8[64];
__constant__ uint8_t c_scan4[16];
__constant__ uint8_t c_scan8[64];
__constant__ uint16_t c_mf4[6][3];
__constant__ uint8_t c_dq4[6][3];
__constant__ uint16_t c_mf8[6][6];
__constant__ uint8_t c_dq8[6][6];
__constant__ uint8_t c_cqp[52];
__constant__ uint8_t c_alpha[52];
__constant__ uint8_t c_beta[52];
__constant__ uint8_t c_tc0[52][3];

// ---------------------------------------------------------------------------------------------
// Shared memory of one macroblock warp.
// Block stride (words) of the 8x8 intermediates: 8 banks apart, so the four blocks' rows and columns
// fall into different banks.
constexpr int kT8Block = 72;
struct __align__(16) Smem {
  uint8_t src_y[256];
  uint8_t src_u[64];
  uint8_t src_v[64];
  uint8_t pred_y[256];
  uint8_t pred_u[64];
  uint8_t pred_v[64];
  uint8_t tmp_y[256];       // plane prediction / I4x4 reconstruction
  alignas(16) uint8_t win[23 * 24];  // integer samples of a half-sample window (rows -2.., cols -2..)
  // The half-sample planes live until the sub-pel search ends; the 8x8 transform's intermediates
  // are needed only after it (the residual), so they share the space.
  union alignas(16) {
    struct {
      uint8_t hph[18 * 20];  // b samples (horizontal half)
      uint8_t hpv[18 * 20];  // h samples (vertical half)
      uint8_t hpj[18 * 20];  // j samples (centre)
      int16_t hr[23 * 18];   // unrounded horizontal 6-tap sums
    };
    int32_t t8[4 * kT8Block];  // 8x8 transform intermediates, block b at [kT8Block b]
  };
  alignas(16) int16_t coef[256];  // luma 4x4 levels: block b (decoding order) at [16 b], raster
  alignas(16) int16_t coef8[256]; // luma 8x8 levels: block b at [64 b], zig-zag order
  alignas(16) uint8_t zz8[64];    // zig-zag index of row y, column x of an 8x8 block at [8 x + y] (init_tables)
  alignas(16) int16_t ccoef[128]; // chroma levels: block (plane * 4 + b) at [16 *], raster
  alignas(16) int16_t cdc[8];
  int16_t ldc[16];          // I16x16 DC levels, raster
  int16_t ldcr[16];         // I16x16 DC reconstruction, raster
  uint8_t top[24];          // luma row above the macroblock (x0 .. x0 + 23)
  uint8_t left[16];
  uint8_t ctop[2][8];
  uint8_t cleft[2][8];
  alignas(16) StreamDev sd;       // the picture worked on (load_desc) and its stream's size (load_params)
  alignas(16) FrameParams fp;
  int db_row, seen_db;            // last acquired progress db_prev[db_row] of the reference picture
  int reach_y, reach_x;           // 1 + the largest reach waited for beyond zero motion, in macroblocks
  alignas(16) uint8_t i4m[16];    // Intra4x4PredMode of this macroblock (decoding order)
  uint8_t i4q[16];          // edge samples of the current 4x4 block (i4_edge_index)
};
static_assert(offsetof(Smem, coef) % 4 == 0 && offsetof(Smem, ccoef) % 4 == 0, "level arrays cleared by words");
static_assert(offsetof(rg_mb_out, luma) % 4 == 0 && offsetof(rg_mb_out, chroma_dc) % 4 == 0 &&
                  offsetof(rg_mb_out, chroma_ac) % 4 == 0 && sizeof(rg_mb_out) % 4 == 0,
              "record levels written by words");
static_assert(offsetof(Smem, coef) % 8 == 0 && offsetof(Smem, ccoef) % 8 == 0 && offsetof(Smem, coef8) % 8 == 0 &&
                  offsetof(Smem, t8) % 16 == 0 && offsetof(Smem, zz8) % 8 == 0 && offsetof(Smem, i4m) % 4 == 0 &&
                  offsetof(Smem, src_u) % 8 == 0 && offsetof(Smem, pred_u) % 8 == 0,
              "rows of levels, intermediates and samples move as vectors");
static_assert(offsetof(Smem, pred_y) % 8 == 0 && offsetof(Smem, tmp_y) % 8 == 0, "16x16 predictions written 8 bytes per lane");

// Every kernel of this file runs one warp per block, and its shared memory has this one name: the
// functions below address it directly (shared-memory loads at constant offsets) instead of through
// a reference, which a call turns into a generic address -- a 64-bit pointer in registers and loads
// that resolve their memory space as they run.
__shared__ Smem sm;
__device__ __forceinline__ uint8_t* sm_at(int off) { return (uint8_t*)&sm + off; }

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ MbInfo ld_info(const MbInfo* p) {
  int4 v = *(const int4*)p;
  MbInfo m;
  *(int4*)&m = v;
  return m;
}
__device__ __forceinline__ uint32_t wsum(uint32_t v) { return __reduce_add_sync(FULL, v); }
__device__ __forceinline__ uint32_t wor(uint32_t v) { return __reduce_or_sync(FULL, v); }
__device__ __forceinline__ int clip255(int v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }
__device__ __forceinline__ int16_t clamp_i16(int v) { return (int16_t)(v < -32768 ? -32768 : (v > 32767 ? 32767 : v)); }

// Column and row of 4x4 block b in decoding order (enc.rs:522 blk_xy).
__device__ __forceinline__ int blk_x(int b) { return (b & 1) + ((b >> 1) & 2); }
__device__ __forceinline__ int blk_y(int b) { return ((b >> 1) & 1) + ((b >> 2) & 2); }
// Position class of raster coefficient i in a 4x4 block (h264.rs:1204).
__device__ __forceinline__ int pos4(int i) {
  int r = i >> 2, c = i & 3;
  if (((r | c) & 1) == 0) return 0;
  return ((r & c) & 1) ? 1 : 2;
}
__device__ __forceinline__ int chroma_qp(int qp) { return c_cqp[qp < 0 ? 0 : (qp > 51 ? 51 : qp)]; }
// Bits of se(v) (enc.rs:546).
__device__ __forceinline__ uint32_t se_bits(int d) {
  uint32_t v = (uint32_t)(d < 0 ? -d : d) * 2u - (d > 0 ? 1u : 0u);
  return 2u * (32u - (uint32_t)__clz(v + 1u)) - 1u;
}
__device__ __forceinline__ uint32_t mvd_cost(int d, uint32_t lambda) {
  uint32_t c = lambda * se_bits(d);
  return (d >= -4096 && d <= 4096) ? (c & 0xFFFFu) : c;
}

// Reconstructed pictures and macroblock state are produced by other warps of the same launch in
// the pipelined mode. They are read with plain (weak, coherent-path) loads -- never the
// non-coherent read-only path -- and only after an ld.acquire that observed the producer's
// release, which the memory model makes sufficient for the loads to see the produced values.
// Plain loads also let the compiler issue independent loads back to back.
__device__ __forceinline__ uint32_t ldw32(const void* p) { return *(const uint32_t*)p; }
__device__ __forceinline__ uint8_t ldcg_u8(const uint8_t* p) { return *p; }
__device__ __forceinline__ uint32_t ldcg_u32(const uint8_t* p) { return ldw32(p); }
__device__ __forceinline__ uint2 ldg8(const uint8_t* p) {
  uintptr_t a = (uintptr_t)p;
  const uint32_t* b = (const uint32_t*)(a & ~(uintptr_t)3);
  uint32_t sh = (uint32_t)(a & 3) * 8u;
  uint32_t w0 = b[0], w1 = b[1], w2 = b[2];
  return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}
__device__ __forceinline__ uint32_t vsad8(uint2 a, uint2 b) { return __vsadu4(a.x, b.x) + __vsadu4(a.y, b.y); }

// ---------------------------------------------------------------------------------------------
// Per-lane transforms (crates/ragdoll-simd/src/fixed.rs:104,192,322; h264_idct.rs:225)
__device__ __forceinline__ void fdct4(const int* d, int* o) {
  int t[16];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    int s03 = d[r * 4] + d[r * 4 + 3], s12 = d[r * 4 + 1] + d[r * 4 + 2];
    int d03 = d[r * 4] - d[r * 4 + 3], d12 = d[r * 4 + 1] - d[r * 4 + 2];
    t[r * 4] = s03 + s12; t[r * 4 + 1] = 2 * d03 + d12; t[r * 4 + 2] = s03 - s12; t[r * 4 + 3] = d03 - 2 * d12;
  }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    int s03 = t[c] + t[c + 12], s12 = t[c + 4] + t[c + 8], d03 = t[c] - t[c + 12], d12 = t[c + 4] - t[c + 8];
    o[c] = (int16_t)(s03 + s12); o[c + 4] = (int16_t)(2 * d03 + d12);
    o[c + 8] = (int16_t)(s03 - s12); o[c + 12] = (int16_t)(d03 - 2 * d12);
  }
}
__device__ __forceinline__ void idct4(const int* c, int* o) {
  int t[16];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    int e0 = c[r * 4] + c[r * 4 + 2], e1 = c[r * 4] - c[r * 4 + 2];
    int e2 = (c[r * 4 + 1] >> 1) - c[r * 4 + 3], e3 = c[r * 4 + 1] + (c[r * 4 + 3] >> 1);
    t[r * 4] = e0 + e3; t[r * 4 + 1] = e1 + e2; t[r * 4 + 2] = e1 - e2; t[r * 4 + 3] = e0 - e3;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    int e0 = t[k] + t[k + 8], e1 = t[k] - t[k + 8];
    int e2 = (t[k + 4] >> 1) - t[k + 12], e3 = t[k + 4] + (t[k + 12] >> 1);
    o[k] = (int16_t)((e0 + e3 + 32) >> 6); o[k + 4] = (int16_t)((e1 + e2 + 32) >> 6);
    o[k + 8] = (int16_t)((e1 - e2 + 32) >> 6); o[k + 12] = (int16_t)((e0 - e3 + 32) >> 6);
  }
}
// One row / column of the 8x8 forward transform (fixed.rs:392).
__device__ __forceinline__ void fdct8_1d(const int* a, int* o) {
  int a0 = a[0] + a[7], a1 = a[1] + a[6], a2 = a[2] + a[5], a3 = a[3] + a[4];
  int a4 = a[0] - a[7], a5 = a[1] - a[6], a6 = a[2] - a[5], a7 = a[3] - a[4];
  int b0 = a0 + a3, b1 = a1 + a2, b2 = a0 - a3, b3 = a1 - a2;
  int b4 = a5 + a6 + ((a4 >> 1) + a4), b5 = a4 - a7 - ((a6 >> 1) + a6);
  int b6 = a4 + a7 - ((a5 >> 1) + a5), b7 = a5 - a6 + ((a7 >> 1) + a7);
  o[0] = b0 + b1; o[1] = b4 + (b7 >> 2); o[2] = b2 + (b3 >> 1); o[3] = b5 + (b6 >> 2);
  o[4] = b0 - b1; o[5] = b6 - (b5 >> 2); o[6] = (b2 >> 1) - b3; o[7] = (b4 >> 2) - b7;
}
// The 1-D inverse 8x8 transform in wrapping 32-bit arithmetic (h264_idct.rs:225).
__device__ __forceinline__ void idct8_1d(const int* d, int* o) {
  unsigned a0 = (unsigned)d[0] + (unsigned)d[4];
  unsigned a1 = (unsigned)d[5] - (unsigned)d[3] - (unsigned)d[7] - (unsigned)(d[7] >> 1);
  unsigned a2 = (unsigned)d[0] - (unsigned)d[4];
  unsigned a3 = (unsigned)d[1] + (unsigned)d[7] - (unsigned)d[3] - (unsigned)(d[3] >> 1);
  unsigned a4 = (unsigned)(d[2] >> 1) - (unsigned)d[6];
  unsigned a5 = (unsigned)d[7] - (unsigned)d[1] + (unsigned)d[5] + (unsigned)(d[5] >> 1);
  unsigned a6 = (unsigned)d[2] + (unsigned)(d[6] >> 1);
  unsigned a7 = (unsigned)d[3] + (unsigned)d[5] + (unsigned)d[1] + (unsigned)(d[1] >> 1);
  unsigned b0 = a0 + a6, b1 = a1 + (unsigned)((int)a7 >> 2), b2 = a2 + a4, b3 = a3 + (unsigned)((int)a5 >> 2);
  unsigned b4 = a2 - a4, b5 = (unsigned)((int)a3 >> 2) - a5, b6 = a0 - a6, b7 = a7 - (unsigned)((int)a1 >> 2);
  o[0] = (int)(b0 + b7); o[1] = (int)(b2 + b5); o[2] = (int)(b4 + b3); o[3] = (int)(b6 + b1);
  o[4] = (int)(b6 - b1); o[5] = (int)(b4 - b3); o[6] = (int)(b2 - b5); o[7] = (int)(b0 - b7);
}
// One pass of the 4x4 forward core transform along the axis whose lanes are `step` apart in a
// 16-lane group (i = position along it): [1 1 1 1; 2 1 -1 -2; 1 -1 -1 1; 1 -2 2 -1].
__device__ __forceinline__ int fwd4_pass(int v, int step, int i) {
  int b = __shfl_xor_sync(FULL, v, 3 * step);
  int s = v + b, dd = v - b;
  int ps = __shfl_xor_sync(FULL, s, step), pd = __shfl_xor_sync(FULL, dd, step);
  return i == 0 ? s + ps : (i == 1 ? 2 * pd + dd : (i == 2 ? ps - s : 2 * pd - dd));
}
// One pass of the inverse core transform (fixed.rs:192): e0 = c0 + c2, e1 = c0 - c2,
// e2 = (c1 >> 1) - c3, e3 = c1 + (c3 >> 1); out = e0 + e3, e1 + e2, e1 - e2, e0 - e3.
__device__ __forceinline__ int inv4_pass(int v, int step, int i) {
  int b = __shfl_xor_sync(FULL, v, 2 * step);
  int ea, eb;
  if (i == 0) { ea = v + b; eb = v - b; }
  else if (i == 2) { ea = b + v; eb = b - v; }
  else if (i == 1) { ea = (v >> 1) - b; eb = v + (b >> 1); }
  else { ea = (b >> 1) - v; eb = b + (v >> 1); }
  int pa = __shfl_xor_sync(FULL, ea, step), pb = __shfl_xor_sync(FULL, eb, step);
  return i == 0 ? ea + pb : (i == 1 ? pb + ea : (i == 2 ? eb - pa : pa - eb));
}

// ---------------------------------------------------------------------------------------------
// Half-sample window (h264_enc.rs:747 hpel_window, :803 hpel_window_centre): integer origin
// (ox, oy); plane coordinate (r, c) is the sample at (ox + c, oy + r).
__device__ __noinline__ void stage_window(const uint8_t* ref, int stride, int ox, int oy) {
  int lane = lane_id();
  // 23 rows x 6 words: five words per lane, all loads issued before the first use
  uint32_t lo[5], hi[5], sh[5];
#pragma unroll
  for (int r = 0; r < 5; r++) {
    int q = min(lane + 32 * r, 23 * 6 - 1);
    int k = q / 6, w = q - 6 * (q / 6);
    uintptr_t a = (uintptr_t)(ref + (long)(oy - 2 + k) * stride + (ox - 2) + 4 * w);
    const uint32_t* b = (const uint32_t*)(a & ~(uintptr_t)3);
    sh[r] = (uint32_t)(a & 3) * 8u;
    lo[r] = b[0];
    hi[r] = b[1];
  }
#pragma unroll
  for (int r = 0; r < 5; r++) {
    int q = lane + 32 * r;
    if (q < 23 * 6) {
      int k = q / 6, w = q - 6 * (q / 6);
      *(uint32_t*)&sm.win[k * 24 + 4 * w] = __funnelshift_r(lo[r], hi[r], sh[r]);
    }
  }
  __syncwarp();
}
// need: bit 0 b plane (h), bit 1 h plane (v), bit 2 j plane (c)
__device__ __noinline__ void build_hpel(int need) {
  int lane = lane_id();
  if (need & 5) {
    for (int i = lane; i < 23 * 18; i += 32) {
      int k = i / 18, c = i - k * 18;
      const uint8_t* w = &sm.win[k * 24 + c];
      sm.hr[i] = (int16_t)(w[0] - 5 * w[1] + 20 * w[2] + 20 * w[3] - 5 * w[4] + w[5]);
    }
  }
  __syncwarp();
  for (int i = lane; i < 18 * 18; i += 32) {
    int r = i / 18, c = i - r * 18;
    if (need & 1) sm.hph[r * 20 + c] = (uint8_t)clip255((sm.hr[(r + 2) * 18 + c] + 16) >> 5);
    if (need & 2) {
      const uint8_t* w = &sm.win[r * 24 + c + 2];
      int v = w[0] - 5 * w[24] + 20 * w[48] + 20 * w[72] - 5 * w[96] + w[120];
      sm.hpv[r * 20 + c] = (uint8_t)clip255((v + 16) >> 5);
    }
    if (need & 4) {
      const int16_t* t = &sm.hr[r * 18 + c];
      int j = t[0] - 5 * t[18] + 20 * t[36] + 20 * t[54] - 5 * t[72] + t[90];
      sm.hpj[r * 20 + c] = (uint8_t)clip255((j + 512) >> 10);
    }
  }
  __syncwarp();
}
// Planes a vector with fractional part (fx, fy) reads (window_src, enc.rs:1395).
__device__ __forceinline__ int planes_needed(int fx, int fy) {
  if ((fx | fy) == 0) return 0;
  if (fy == 0) return 1;
  if (fx == 0) return 2;
  if (fx == 2 && fy == 2) return 4;
  if (fx == 2) return 5;
  if (fy == 2) return 6;
  return 3;
}
// Quarter-sample prediction of the 16x16 block whose integer position is (wx, wy) in window
// coordinates: one window plane, or the rounded average of two (window_src, enc.rs:1395; equal
// to h264_luma_mc_scalar, h264_mc.rs:148, by enc.rs:4030). Returns the two source rows' bases.
// (byte offsets in Smem).
struct QSrc {
  int a, b, sa, sb, avg;
};
__device__ __noinline__ QSrc qpel_src(int wx, int wy, int fx, int fy) {
  const int G = (int)offsetof(Smem, win) + (wy + 2) * 24 + wx + 2;
  const int B = (int)offsetof(Smem, hph) + wy * 20 + wx;
  const int V = (int)offsetof(Smem, hpv) + wy * 20 + wx;
  const int J = (int)offsetof(Smem, hpj) + wy * 20 + wx;
  switch (fx | (fy << 2)) {
    case 0: return {G, G, 24, 24, 0};
    case 1: return {G, B, 24, 20, 1};
    case 2: return {B, B, 20, 20, 0};
    case 3: return {B, G + 1, 20, 24, 1};
    case 4: return {G, V, 24, 20, 1};
    case 5: return {B, V, 20, 20, 1};
    case 6: return {B, J, 20, 20, 1};
    case 7: return {B, V + 1, 20, 20, 1};
    case 8: return {V, V, 20, 20, 0};
    case 9: return {V, J, 20, 20, 1};
    case 10: return {J, J, 20, 20, 0};
    case 11: return {J, V + 1, 20, 20, 1};
    case 12: return {V, G + 24, 20, 24, 1};
    case 13: return {V, B + 20, 20, 20, 1};
    case 14: return {J, B + 20, 20, 20, 1};
    default: return {V + 1, B + 20, 20, 20, 1};
  }
}
// 8 bytes of shared memory at any alignment (rows of the window planes are 4-byte aligned).
__device__ __forceinline__ uint2 lds8(const uint8_t* p) {
  uintptr_t a = (uintptr_t)p;
  const uint32_t* b = (const uint32_t*)(a & ~(uintptr_t)3);
  uint32_t sh = (uint32_t)(a & 3) * 8u;
  uint32_t w0 = b[0], w1 = b[1], w2 = b[2];
  return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}
// This lane's 8 prediction samples (row lane/2, columns 8 (lane&1) ..) packed in two words.
__device__ __forceinline__ uint2 qpel8(const QSrc& q) {
  int lane = lane_id(), i = lane >> 1, j0 = (lane & 1) * 8;
  uint2 a = lds8(sm_at(q.a + i * q.sa + j0));
  if (!q.avg) return a;
  uint2 b = lds8(sm_at(q.b + i * q.sb + j0));
  return make_uint2(__vavgu4(a.x, b.x), __vavgu4(a.y, b.y));
}
// Cost of a full-pel position (mx, my): the warp's SAD of the 16x16 block (this lane's 8 source
// samples sv against its 8 reference samples r) plus lambda * bits of the vector difference to
// the predictor (enc.rs:1207 cost). Shared by the candidates and the diamond steps.
__device__ __noinline__ uint32_t fullpel_cost(uint2 sv, uint2 r, int mx, int my, int mvp0, int mvp1, uint32_t lambda) {
  return wsum(vsad8(sv, r)) + mvd_cost(mx * 4 - mvp0, lambda) + mvd_cost(my * 4 - mvp1, lambda);
}
// This lane's SAD against the quarter-sample prediction at window position (wx, wy), phase
// (fx, fy): shared by the candidates of the sub-pel search.
__device__ __noinline__ uint32_t qpel_sad(uint2 sv, int wx, int wy, int fx, int fy) {
  return vsad8(sv, qpel8(qpel_src(wx, wy, fx, fy)));
}
__device__ __forceinline__ uint2 src8() {
  int lane = lane_id();
  return *(const uint2*)&sm.src_y[(lane >> 1) * 16 + (lane & 1) * 8];
}
// Prediction of the 16x16 block displaced by mv into pred_y (enc.rs:1058 mc_luma).
__device__ __noinline__ void mc_luma16(const uint8_t* ref, int stride, int x0, int y0, int mvx, int mvy) {
  int ix = x0 + (mvx >> 2), iy = y0 + (mvy >> 2), fx = mvx & 3, fy = mvy & 3;
  int lane = lane_id();
  if ((fx | fy) == 0) {
    uint2 v = ldg8(ref + (long)(iy + (lane >> 1)) * stride + ix + (lane & 1) * 8);
    *(uint2*)&sm.pred_y[(lane >> 1) * 16 + (lane & 1) * 8] = v;
    __syncwarp();
    return;
  }
  stage_window(ref, stride, ix, iy);
  build_hpel(planes_needed(fx, fy));
  uint2 v = qpel8(qpel_src(0, 0, fx, fy));
  *(uint2*)&sm.pred_y[(lane >> 1) * 16 + (lane & 1) * 8] = v;
  __syncwarp();
}
// Chroma prediction of both planes (h264_enc.rs:1279 chroma_mc_8x8_x2_scalar; enc.rs:1082).
__device__ __noinline__ void mc_chroma8(const uint8_t* ru, const uint8_t* rv, int stride, int mbx, int mby, int mvx, int mvy) {
  int lane = lane_id();
  int cx = mbx * 8 + (mvx >> 3), cy = mby * 8 + (mvy >> 3), fx = mvx & 7, fy = mvy & 7;
  int wa = (8 - fx) * (8 - fy), wb = fx * (8 - fy), wc = (8 - fx) * fy, wd = fx * fy;
  int plane = lane >> 4, idx = (lane & 15) * 4, r = idx >> 3, c0 = idx & 7;
  const uint8_t* src = (plane ? rv : ru) + (long)(cy + r) * stride + cx + c0;
  uint8_t* out = (plane ? sm.pred_v : sm.pred_u) + r * 8 + c0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    int a = ldcg_u8(src + k), b = ldcg_u8(src + k + 1), cc = ldcg_u8(src + stride + k), d = ldcg_u8(src + stride + k + 1);
    out[k] = (uint8_t)((wa * a + wb * b + wc * cc + wd * d + 32) >> 6);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// Quantisation helpers (enc.rs:1703-1779, h264_enc.rs:408)
__device__ __forceinline__ void quant4_params(int qp, bool intra, uint32_t& shift, uint32_t& bias) {
  shift = 15 + qp / 6;
  bias = (1u << shift) / (intra ? 3u : 6u);
}
// Level of coefficient c. Every transform here is of 8-bit differences: |c| is at most 64 * 255 and
// the scales at most 20972, so the product and the bias fit 32 bits and the level 16.
__device__ __forceinline__ int quant_level(int c, uint32_t mf, uint32_t bias, uint32_t shift) {
  uint32_t a = (uint32_t)(c < 0 ? -c : c);
  int l = (int)((a * mf + bias) >> shift);
  return c < 0 ? -l : l;
}

// ---- 4x4 blocks, two lanes each -----------------------------------------------------------------
// A macroblock's 4x4 transforms are done all at once: lane 2 b + h holds half of block b, the pixel
// rows (0, 3) when h = 0 and (1, 2) when h = 1 -- the pairs the core transform's first butterfly
// adds -- and after the forward transform the coefficient rows (0, 2) or (1, 3), the pairs the
// inverse starts from. Rows are transformed in registers, and a column pass needs four words of the
// partner lane (four independent shuffles). A macroblock is one chain of instructions of one warp, so
// what counts is the chain's length: one lane per coefficient and two blocks a step was eight steps
// of two passes of three dependent shuffles, 7.2 k cycles for the luma quantisation even on a nearly
// idle SM. With this split (and the record written by words) a 720p stream's launch of 30 pictures
// went from 21.6 to 17.6 ms, 1080p 8 x 15 from 54.6 to 50.7 ms.
struct Half4 {
  int a[4], b[4];  // its first and second row
};
// The lane's two rows (r0 = the first's index) of samples at byte offset `off` in Smem.
__device__ __forceinline__ uint2 half_rows(int off, int stride, int h) {
  return make_uint2(*(const uint32_t*)sm_at(off + h * stride), *(const uint32_t*)sm_at(off + (3 - h) * stride));
}
__device__ __forceinline__ Half4 half_diff(uint2 s, uint2 p) {
  Half4 d;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    d.a[k] = (int)((s.x >> (8 * k)) & 255u) - (int)((p.x >> (8 * k)) & 255u);
    d.b[k] = (int)((s.y >> (8 * k)) & 255u) - (int)((p.y >> (8 * k)) & 255u);
  }
  return d;
}
// Forward core transform (fixed.rs:104).
__device__ __forceinline__ void half_fwd(Half4& v, int h) {
  auto row = [](int (&r)[4]) {
    int s03 = r[0] + r[3], s12 = r[1] + r[2], d03 = r[0] - r[3], d12 = r[1] - r[2];
    r[0] = s03 + s12; r[1] = 2 * d03 + d12; r[2] = s03 - s12; r[3] = d03 - 2 * d12;
  };
  row(v.a);
  row(v.b);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // h = 0: sum s03 and difference d03 of rows 0 and 3; h = 1: s12 and d12 of rows 1 and 2
    int s = v.a[k] + v.b[k], d = v.a[k] - v.b[k];
    int o = __shfl_xor_sync(FULL, h ? s : d, 1);
    int x = h ? o : s, y = h ? d : o;   // s03, s12 or d03, d12
    v.a[k] = (x << h) + y;              // row 0: s03 + s12, row 1: 2 d03 + d12
    v.b[k] = x - (y << h);              // row 2: s03 - s12, row 3: d03 - 2 d12
  }
}
// Inverse core transform with its rounding (fixed.rs:192): coefficient rows in, residual rows out.
__device__ __forceinline__ void half_inv(Half4& v, int h) {
  auto row = [](int (&r)[4]) {
    int e0 = r[0] + r[2], e1 = r[0] - r[2], e2 = (r[1] >> 1) - r[3], e3 = r[1] + (r[3] >> 1);
    r[0] = e0 + e3; r[1] = e1 + e2; r[2] = e1 - e2; r[3] = e0 - e3;
  };
  row(v.a);
  row(v.b);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // h = 0 (rows 0, 2): e0, e1; h = 1 (rows 1, 3): e2, e3
    int p = h ? (v.a[k] >> 1) - v.b[k] : v.a[k] + v.b[k];
    int q = h ? v.a[k] + (v.b[k] >> 1) : v.a[k] - v.b[k];
    int o = __shfl_xor_sync(FULL, q, 1);
    int x = h ? o : p, y = h ? p : o;  // h = 0: e0, e3 -> rows 0, 3; h = 1: e1, e2 -> rows 1, 2
    v.a[k] = (x + y + 32) >> 6;
    v.b[k] = (x - y + 32) >> 6;
  }
}
// This half's share of the block's SATD (metrics.rs:705): a column's four Hadamard outputs are
// |x + y| and |x - y| of each lane's (x, y), and |x + y| + |x - y| = 2 max(|x|, |y|), so the sums
// below are the halved ones.
__device__ __forceinline__ uint32_t half_satd(Half4 v, int h) {
  auto row = [](int (&r)[4]) {
    int s03 = r[0] + r[3], s12 = r[1] + r[2], d03 = r[0] - r[3], d12 = r[1] - r[2];
    r[0] = s03 + s12; r[1] = d03 + d12; r[2] = s03 - s12; r[3] = d03 - d12;
  };
  row(v.a);
  row(v.b);
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    int s = v.a[k] + v.b[k], d = v.a[k] - v.b[k];
    int o = __shfl_xor_sync(FULL, h ? s : d, 1);
    sum += (uint32_t)max(abs(h ? d : s), abs(o));
  }
  return sum;
}
// The per-lane scales of the half's even and odd columns (position classes 0, 2 / 2, 1).
__device__ __forceinline__ void half_scales(uint32_t c0, uint32_t c1, uint32_t c2, int h, uint32_t& even, uint32_t& odd) {
  even = h ? c2 : c0;
  odd = h ? c1 : c2;
}
// The half's zig-zag indices: rows 0 and 2, or rows 1 and 3, of the frame scan (Table 8-12).
__device__ __forceinline__ uint32_t half_zigzag_bit(int row, int k, int h) {
  constexpr uint32_t z[2][2][4] = {{{0, 1, 5, 6}, {3, 8, 11, 13}}, {{2, 4, 7, 12}, {9, 10, 14, 15}}};
  return h ? 1u << z[1][row][k] : 1u << z[0][row][k];
}
// Quantises the half. Returns, alike in both lanes, the block's nonzero levels by zig-zag index
// (bits 0..15, indices >= first) and in bit 16 whether one of them is above 1.
__device__ __forceinline__ uint32_t half_quant(Half4& v, int h, int first, uint32_t mf_even, uint32_t mf_odd, uint32_t bias,
                                               uint32_t shift) {
  uint32_t mask = 0, big = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t mf = (k & 1) ? mf_odd : mf_even;
    const uint32_t la = ((uint32_t)abs(v.a[k]) * mf + bias) >> shift, lb = ((uint32_t)abs(v.b[k]) * mf + bias) >> shift;
    const bool dc = k == 0 && first && !h;
    if (la && !dc) mask |= half_zigzag_bit(0, k, h);
    if (lb) mask |= half_zigzag_bit(1, k, h);
    big |= (dc ? 0u : la) | lb;
    v.a[k] = v.a[k] < 0 ? -(int)la : (int)la;
    v.b[k] = v.b[k] < 0 ? -(int)lb : (int)lb;
  }
  mask |= big > 1u ? 0x10000u : 0u;
  return mask | __shfl_xor_sync(FULL, mask, 1);
}
// Decimation score (enc.rs:559, without its |level| > 1 rule) of a block's nonzero zig-zag
// positions: 3 / 2 / 1 / 0 for a zero run of 0 / 1-2 / 3-5 / longer below each -- the positions with
// another one (or the start, index first - 1) at most 1, 3 and 6 below, counted.
__device__ __forceinline__ uint32_t score4(uint32_t m, int first) {
  m &= 0xffffu;
  const uint32_t w1 = (first ? m | 1u : m) << 1, w3 = w1 | (w1 << 1) | (w1 << 2), w6 = w3 | (w3 << 3);
  const uint32_t u = first ? 0u : 0x3fu;  // the start, one below index 0
  return __popc(m & (w1 | (u & 1u))) + __popc(m & (w3 | (u & 7u))) + __popc(m & (w6 | u));
}
__device__ __forceinline__ uint2 pack_half(const int (&r)[4]) {
  return make_uint2(__byte_perm((uint32_t)r[0], (uint32_t)r[1], 0x5410), __byte_perm((uint32_t)r[2], (uint32_t)r[3], 0x5410));
}
__device__ __forceinline__ void unpack_half(uint2 w, int (&r)[4]) {
  r[0] = (int16_t)(w.x & 0xffffu); r[1] = (int)w.x >> 16;
  r[2] = (int16_t)(w.y & 0xffffu); r[3] = (int)w.y >> 16;
}
// Four clipped samples p + r, packed.
__device__ __forceinline__ uint32_t add_clip4(uint32_t p, const int (&r)[4]) {
  uint32_t w = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) w |= (uint32_t)clip255((int)((p >> (8 * k)) & 255u) + r[k]) << (8 * k);
  return w;
}
// Byte offset of 4x4 luma block b (decoding order) in a 16x16 plane, and of chroma block b (plane b
// / 4) in the two 8x8 planes u, v (v right behind u).
__device__ __forceinline__ int blk_off16(int b) { return blk_y(b) * 64 + blk_x(b) * 4; }
__device__ __forceinline__ int blk_off8(int b) { return (b >> 2) * 64 + ((b & 3) >> 1) * 32 + (b & 1) * 4; }
static_assert(offsetof(Smem, src_v) == offsetof(Smem, src_u) + 64 && offsetof(Smem, pred_v) == offsetof(Smem, pred_u) + 64,
              "the chroma planes lie back to back");
// The even bits of w (one per lane pair) as 16 bits.
__device__ __forceinline__ uint32_t even_bits(uint32_t w) {
  w &= 0x55555555u;
  w = (w | (w >> 1)) & 0x33333333u;
  w = (w | (w >> 2)) & 0x0f0f0f0fu;
  w = (w | (w >> 4)) & 0x00ff00ffu;
  return (w | (w >> 8)) & 0xffffu;
}

// SATD (metrics.rs:705, halved) of the macroblock's source against the 16x16 plane at byte offset `at`.
__device__ __noinline__ uint32_t satd16(int at) {
  const int lane = lane_id(), h = lane & 1, off = blk_off16(lane >> 1);
  return wsum(half_satd(half_diff(half_rows((int)offsetof(Smem, src_y) + off, 16, h), half_rows(at + off, 16, h)), h));
}
// Forward transform and inter quantisation of the macroblock's luma residual, one block per lane pair.
__device__ __forceinline__ uint32_t luma4x4_levels(int qp, Half4& v) {
  const int lane = lane_id(), b = lane >> 1, h = lane & 1, off = blk_off16(b);
  uint32_t shift, bias, even, odd;
  quant4_params(qp, false, shift, bias);
  const int rem = qp % 6;
  half_scales(c_mf4[rem][0], c_mf4[rem][1], c_mf4[rem][2], h, even, odd);
  v = half_diff(half_rows((int)offsetof(Smem, src_y) + off, 16, h), half_rows((int)offsetof(Smem, pred_y) + off, 16, h));
  half_fwd(v, h);
  return half_quant(v, h, 0, even, odd, bias, shift);
}

// Luma 4x4 residual of pred_y, quantised (inter) and decimated into sm.coef
// (enc.rs:1810 quant_luma_4x4_inter).
struct Luma4 {
  uint32_t cbp, nnz, nz16;  // coded block pattern, nonzero levels kept, blocks holding levels (bit b)
};
__device__ __noinline__ Luma4 luma4x4_inter(int qp) {
  const int lane = lane_id(), b = lane >> 1, h = lane & 1;
  Half4 v;
  const uint32_t m = luma4x4_levels(qp, v);
  // the 8x8 group's any, |level| > 1 and score sums over its four blocks (lanes 8 g .. 8 g + 7)
  uint32_t g = score4(m, 0) | ((m >> 16) << 12) | ((m & 0xffffu) ? 1u << 16 : 0u);
  g += __shfl_xor_sync(FULL, g, 2);
  g += __shfl_xor_sync(FULL, g, 4);
  const bool any = (g >> 16) != 0, big = ((g >> 12) & 15u) != 0;
  const uint32_t sc = g & 0xfffu;
  const uint32_t keep = __ballot_sync(FULL, any && (big || sc >= 4));
  const uint32_t total = wsum((lane & 7) == 0 && any ? (big ? 9u : sc) : 0u);
  uint32_t cbp = (keep & 1u) | ((keep >> 7) & 2u) | ((keep >> 14) & 4u) | ((keep >> 21) & 8u);
  if (total < 6) cbp = 0;
  const bool coded = (cbp >> (lane >> 3)) & 1u;  // levels of dropped groups are cleared
  uint2 ra = pack_half(v.a), rb = pack_half(v.b);
  if (!coded) ra = rb = make_uint2(0u, 0u);
  *(uint2*)&sm.coef[b * 16 + h * 4] = ra;
  *(uint2*)&sm.coef[b * 16 + h * 4 + 8] = rb;
  Luma4 r;
  r.cbp = cbp;
  r.nz16 = even_bits(__ballot_sync(FULL, coded && (m & 0xffffu)));
  r.nnz = wsum(h == 0 && coded ? __popc(m & 0xffffu) : 0u);
  __syncwarp();
  return r;
}

// Zig-zag index of (row y, column x) of an 8x8 block (frame scan, Table 8-13): diagonal s = x + y,
// walked up-right on even s and down-left on odd s.
__device__ __forceinline__ int zigzag8(int y, int x) {
  int s = x + y;
  if (s < 8) return s * (s + 1) / 2 + ((s & 1) ? y : x);
  return 64 - (16 - s) * (15 - s) / 2 + ((s & 1) ? 7 - x : 7 - y);
}
// The tables a warp keeps in its shared memory, once per kernel.
__device__ __forceinline__ void init_tables() {
  for (int i = lane_id(); i < 64; i += 32) sm.zz8[i] = (uint8_t)zigzag8(i & 7, i >> 3);
  __syncwarp();
}
// The scales of row (or column) q of an 8x8 block by the other coordinate's low two bits: position
// classes (h264.rs:1343) {0, 3, 4, 3}, {3, 1, 5, 1}, {4, 5, 2, 5}, {3, 1, 5, 1}.
struct Scale8 {
  int m0, m1, m2;  // index 0, odd, 2
  __device__ __forceinline__ int at(int k) const { return (k & 1) ? m1 : ((k & 2) ? m2 : m0); }
};
template <typename T>
__device__ __forceinline__ Scale8 scale8(const T* c, int q) {
  const int k0 = c[0], k1 = c[1], k2 = c[2], k3 = c[3], k4 = c[4], k5 = c[5];
  const bool odd = q & 1, two = (q & 3) == 2;
  return {odd ? k3 : (two ? k4 : k0), odd ? k1 : (two ? k5 : k3), odd ? k5 : (two ? k2 : k4)};
}
// Eight words of a block's row (contiguous) to and from shared memory.
__device__ __forceinline__ void t8_store_row(int at, const int (&r)[8]) {
  *(int4*)&sm.t8[at] = make_int4(r[0], r[1], r[2], r[3]);
  *(int4*)&sm.t8[at + 4] = make_int4(r[4], r[5], r[6], r[7]);
}

// Luma 8x8 residual of pred_y, quantised (inter) and decimated into sm.coef8
// (enc.rs:2041 quant_luma_8x8_inter). Lanes 8b..8b+7 own block b: row q in registers for the first
// pass, column q (through shared memory) for the second. The decimation score of a block comes from
// the bitmask of its nonzero zig-zag positions (weights 3 / 2 / 1 / 0 for zero runs of 0-3 / 4-11 /
// 12-23 / longer below each, enc.rs:559 with the 8x8 table), counted as in score4. Returns cbp |
// nonzero levels << 4.
__device__ __noinline__ uint32_t luma8x8_inter(int qp) {
  const int lane = lane_id(), b = lane >> 3, q = lane & 7;
  const int off = ((b >> 1) * 8 + q) * 16 + (b & 1) * 8;
  const uint32_t shift = 16 + qp / 6, bias = (1u << shift) / 6u;
  int d[8], o[8];
  {
    const uint2 s = *(const uint2*)&sm.src_y[off], p = *(const uint2*)&sm.pred_y[off];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      d[k] = (int)((s.x >> (8 * k)) & 255u) - (int)((p.x >> (8 * k)) & 255u);
      d[k + 4] = (int)((s.y >> (8 * k)) & 255u) - (int)((p.y >> (8 * k)) & 255u);
    }
  }
  fdct8_1d(d, o);
  t8_store_row(b * kT8Block + q * 8, o);
  __syncwarp();
#pragma unroll
  for (int y = 0; y < 8; y++) d[y] = sm.t8[b * kT8Block + y * 8 + q];
  fdct8_1d(d, o);
  const Scale8 mf = scale8(c_mf8[qp % 6], q);
  const uint2 zz = *(const uint2*)&sm.zz8[q * 8];
  uint32_t lo = 0, hi = 0, big = 0;
#pragma unroll
  for (int y = 0; y < 8; y++) {
    const uint32_t l = ((uint32_t)abs(o[y]) * (uint32_t)mf.at(y) + bias) >> shift;
    const uint32_t z = ((y < 4 ? zz.x : zz.y) >> (8 * (y & 3))) & 255u, bit = l ? 1u << (z & 31u) : 0u;
    if (z & 32u) hi |= bit; else lo |= bit;
    big |= l;
    o[y] = o[y] < 0 ? -(int)l : (int)l;
  }
#pragma unroll
  for (int k = 1; k < 8; k <<= 1) {
    lo |= __shfl_xor_sync(FULL, lo, k);
    hi |= __shfl_xor_sync(FULL, hi, k);
  }
  const bool anybig = ((__ballot_sync(FULL, big > 1u) >> (8 * b)) & 0xffu) != 0;
  const unsigned long long m = ((unsigned long long)hi << 32) | lo;
  const unsigned long long s1 = m << 1, s2 = s1 | (s1 << 1), s4 = s2 | (s2 << 2), s8 = s4 | (s4 << 4),
                           s12 = s8 | (s4 << 8), s24 = s12 | (s12 << 12);
  uint32_t score = __popcll(m & (s4 | 0xfull)) + __popcll(m & (s12 | 0xfffull)) + __popcll(m & (s24 | 0xffffffull));
  if (anybig) score = 9u;
  const uint32_t keep = __ballot_sync(FULL, score >= 4);
  const uint32_t total = wsum(q == 0 ? score : 0u);
  uint32_t cbp = (keep & 1u) | ((keep >> 7) & 2u) | ((keep >> 14) & 4u) | ((keep >> 21) & 8u);
  if (total < 6) cbp = 0;
  const bool coded = (cbp >> b) & 1u;
#pragma unroll
  for (int y = 0; y < 8; y++) {
    const uint32_t z = ((y < 4 ? zz.x : zz.y) >> (8 * (y & 3))) & 255u;
    sm.coef8[b * 64 + z] = (int16_t)(coded ? o[y] : 0);
  }
  __syncwarp();
  return cbp | (wsum(q == 0 && coded ? (uint32_t)__popcll(m) : 0u) << 4);
}

// Chroma residual of pred_u/pred_v (enc.rs:1899 quant_chroma): lane pair b < 8 owns block b
// (plane = b / 4); the other lanes repeat them. Levels into sm.ccoef (raster), DC levels into sm.cdc.
// Returns, in every lane and per plane: AC present, AC decimation score, and any DC level.
struct ChromaAc {
  uint32_t w;  // byte p: the score of plane p (at most 4 x 45); bits 16, 17: AC present; bit 18: DC present
  __device__ __forceinline__ bool any(int p) const { return (w >> (16 + p)) & 1u; }
  __device__ __forceinline__ uint32_t score(int p) const { return (w >> (8 * p)) & 255u; }
  __device__ __forceinline__ bool dc() const { return (w >> 18) & 1u; }
};
__device__ __noinline__ ChromaAc chroma_quant(int qpc, bool intra) {
  const int lane = lane_id(), h = lane & 1, b = (lane >> 1) & 7, off = blk_off8(b);
  uint32_t shift, bias, even, odd;
  quant4_params(qpc, intra, shift, bias);
  const int rem = qpc % 6;
  const uint32_t mf0 = c_mf4[rem][0];
  half_scales(mf0, c_mf4[rem][1], c_mf4[rem][2], h, even, odd);
  Half4 v = half_diff(half_rows((int)offsetof(Smem, src_u) + off, 8, h), half_rows((int)offsetof(Smem, pred_u) + off, 8, h));
  half_fwd(v, h);
  // 2x2 DC transform + quantisation (enc.rs:1938 quant_chroma_dc; f = 2^qbits / 3 always); block b & 3
  // of the plane ends with output b & 3
  int dc = v.a[0];
  {
    int o = __shfl_xor_sync(FULL, dc, 2);
    dc = (b & 1) ? o - dc : dc + o;
    o = __shfl_xor_sync(FULL, dc, 4);
    dc = (b & 2) ? o - dc : dc + o;
    const int qbits = 16 + qpc / 6, f = (1 << qbits) / 3;
    const int l = (abs(dc) * (int)mf0 + f) >> qbits;
    dc = dc < 0 ? -l : l;
  }
  const uint32_t m = half_quant(v, h, 1, even, odd, bias, shift);
  if (lane < 16) {
    *(uint2*)&sm.ccoef[b * 16 + h * 4] = pack_half(v.a);
    *(uint2*)&sm.ccoef[b * 16 + h * 4 + 8] = pack_half(v.b);
    if (!h) sm.cdc[b] = (int16_t)dc;
  }
  const bool dcany = __ballot_sync(FULL, !h && dc != 0) != 0;
  // a plane's score (9 for a block with a level above 1) and AC count over its four blocks
  uint32_t g = ((m >> 16) ? 9u : score4(m, 1)) | ((m & 0xffffu) ? 1u << 16 : 0u);
  g += __shfl_xor_sync(FULL, g, 2);
  g += __shfl_xor_sync(FULL, g, 4);
  const uint32_t u = __shfl_sync(FULL, g, 0), w = __shfl_sync(FULL, g, 8);
  __syncwarp();
  return ChromaAc{(u & 0xffu) | ((w & 0xffu) << 8) | ((u >> 16) ? 1u << 16 : 0u) | ((w >> 16) ? 1u << 17 : 0u) |
                  (dcany ? 1u << 18 : 0u)};
}

// Adds the dequantised chroma residual to pred_u / pred_v (enc.rs:1992 recon_chroma): the DC of
// each block from the 2x2 inverse (h264.rs:1674 dequantize_idct_chroma_dc2x2), its AC dequantised
// when cbpc == 2, then the inverse core transform. Two lanes per block as in chroma_quant.
__device__ __noinline__ void chroma_recon(int qpc, int cbpc) {
  if (cbpc == 0) return;
  const int lane = lane_id(), h = lane & 1, b = (lane >> 1) & 7, bb = b & 3, off = blk_off8(b) + (int)offsetof(Smem, pred_u);
  const int rem = qpc % 6, qdiv = qpc / 6, qmul = (c_dq4[rem][0] * 16) << (qdiv + 2);
  uint32_t even, odd;
  half_scales(c_dq4[rem][0], c_dq4[rem][1], c_dq4[rem][2], h, even, odd);
  int lv[4];
  unpack_half(*(const uint2*)&sm.cdc[b & 4], lv);
  const int e = lv[0] - lv[1], apb = lv[0] + lv[1], cmd = lv[2] - lv[3], cpd = lv[2] + lv[3];
  const int dcv = bb == 0 ? apb + cpd : (bb == 1 ? e + cmd : (bb == 2 ? apb - cpd : e - cmd));
  Half4 v;
  unpack_half(*(const uint2*)&sm.ccoef[b * 16 + h * 4], v.a);
  unpack_half(*(const uint2*)&sm.ccoef[b * 16 + h * 4 + 8], v.b);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int dq = (int)((k & 1) ? odd : even) << qdiv;
    v.a[k] = cbpc >= 2 ? (int)clamp_i16(v.a[k] * dq) : 0;
    v.b[k] = cbpc >= 2 ? (int)clamp_i16(v.b[k] * dq) : 0;
  }
  if (!h) v.a[0] = (int16_t)((dcv * qmul) >> 7);
  half_inv(v, h);
  const uint2 p = half_rows(off, 8, h);
  if (lane < 16) {
    *(uint32_t*)sm_at(off + h * 8) = add_clip4(p.x, v.a);
    *(uint32_t*)sm_at(off + (3 - h) * 8) = add_clip4(p.y, v.b);
  }
  __syncwarp();
}

// Raster position of each 4x4 zig-zag index, 4 bits per index (frame scan, Table 8-12).
constexpr unsigned long long kScan4Packed = 0xfeb7adc963258410ull;

// Adds the dequantised 8x8 residual of the coded blocks of sm.coef8 to pred_y (enc.rs:2013
// recon_8x8: dequantize_block8x8, h264.rs:1403, then h264_idct8_add, h264_idct.rs:207).
// Lanes 8b..8b+7 own block b: row q, then column q. Blocks that are not coded add zero.
__device__ __noinline__ void recon_luma8x8(int qp, int cbp) {
  const int lane = lane_id(), b = lane >> 3, q = lane & 7;
  const bool coded = (cbp >> b) & 1;
  const int qdiv = qp / 6;
  const Scale8 dq = scale8(c_dq8[qp % 6], q);
  int d[8], o[8];
#pragma unroll
  for (int x = 0; x < 8; x++) {
    const int l = coded ? sm.coef8[b * 64 + sm.zz8[x * 8 + q]] : 0, v = dq.at(x);
    const int dv = qdiv >= 2 ? l * (v << (qdiv - 2)) : ((l * v + (1 << (1 - qdiv))) >> (2 - qdiv));
    d[x] = clamp_i16(dv);
  }
  idct8_1d(d, o);
  t8_store_row(b * kT8Block + q * 8, o);
  __syncwarp();
#pragma unroll
  for (int y = 0; y < 8; y++) d[y] = sm.t8[b * kT8Block + y * 8 + q];
  idct8_1d(d, o);
  uint8_t* px = &sm.pred_y[(b >> 1) * 128 + (b & 1) * 8 + q];
#pragma unroll
  for (int y = 0; y < 8; y++) {
    const int v = (int)((unsigned)o[y] + 32u) >> 6;
    px[y * 16] = (uint8_t)clip255((int)((unsigned)px[y * 16] + (unsigned)v));
  }
  __syncwarp();
}

// Adds the dequantised luma 4x4 residual of sm.coef to pred_y (enc.rs:1978 recon_luma_4x4; blocks
// without levels add zero), two lanes per block.
__device__ __noinline__ void recon_luma4x4(int qp) {
  const int lane = lane_id(), b = lane >> 1, h = lane & 1, off = blk_off16(b) + (int)offsetof(Smem, pred_y);
  const int rem = qp % 6, qdiv = qp / 6;
  uint32_t even, odd;
  half_scales(c_dq4[rem][0], c_dq4[rem][1], c_dq4[rem][2], h, even, odd);
  Half4 v;
  unpack_half(*(const uint2*)&sm.coef[b * 16 + h * 4], v.a);
  unpack_half(*(const uint2*)&sm.coef[b * 16 + h * 4 + 8], v.b);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int dq = (int)((k & 1) ? odd : even) << qdiv;
    v.a[k] = clamp_i16(v.a[k] * dq);
    v.b[k] = clamp_i16(v.b[k] * dq);
  }
  half_inv(v, h);
  const uint2 p = half_rows(off, 16, h);
  *(uint32_t*)sm_at(off + h * 16) = add_clip4(p.x, v.a);
  *(uint32_t*)sm_at(off + (3 - h) * 16) = add_clip4(p.y, v.b);
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// Intra prediction (h264.rs:1715 predict_intra_16x16_scalar, :1967 chroma; enc.rs:1561,1586)
// Plane-mode parameters; called by the whole warp: lanes 0..7 take the terms of H
// ((q + 1) (top[8 + q] - top[6 - q])), lanes 8..15 those of V down the left column.
__device__ void plane16_params(bool ht, bool hl, int tl, int& pa, int& pb, int& pc) {
  int lane = lane_id(), q = lane & 7;
  int term = 0;
  if (lane < 16) {
    bool top = lane < 8, av = top ? ht : hl;
    const uint8_t* e = top ? sm.top : sm.left;
    int e8 = av ? e[8 + q] : 128, ep = q == 7 ? tl : (av ? e[6 - q] : 128);
    term = (q + 1) * (e8 - ep);
  }
  int H = (int)wsum(lane < 8 ? (uint32_t)term : 0u), V = (int)wsum(lane >= 8 ? (uint32_t)term : 0u);
  int t15 = ht ? sm.top[15] : 128, l15 = hl ? sm.left[15] : 128;
  pa = 16 * (t15 + l15);
  pb = (5 * H + 32) >> 6;
  pc = (5 * V + 32) >> 6;
}
// DC of the 16x16 prediction; called by the whole warp: lane q < 16 adds top[q], lane 16 + q
// left[q] (both sums below 2^16, one reduction).
__device__ __forceinline__ int dc16(bool ht, bool hl) {
  int lane = lane_id();
  uint32_t v = lane < 16 ? (ht ? (uint32_t)sm.top[lane] : 0u) : (hl ? (uint32_t)sm.left[lane - 16] << 16 : 0u);
  uint32_t both = wsum(v), st = both & 0xffffu, sl = both >> 16;
  if (ht && hl) return (int)((st + sl + 16) >> 5);
  if (ht) return (int)((st + 8) >> 4);
  if (hl) return (int)((sl + 8) >> 4);
  return 128;
}
__device__ __noinline__ void pred16_into(int mode, int dst, bool ht, bool hl, int tl) {
  int lane = lane_id();
  int y = lane >> 1, x0 = (lane & 1) * 8;
  uint8_t* o = sm_at(dst + y * 16 + x0);  // this lane's 8 samples (8-byte aligned)
  if (mode == 3) {
    int pa, pb, pc;
    plane16_params(ht, hl, tl, pa, pb, pc);
    uint32_t w[2] = {0u, 0u};
#pragma unroll
    for (int k = 0; k < 8; k++)
      w[k >> 2] |= (uint32_t)clip255((pa + pb * (x0 + k - 7) + pc * (y - 7) + 16) >> 5) << (8 * (k & 3));
    *(uint2*)o = make_uint2(w[0], w[1]);
  } else {
    uint2 v;
    if (mode == 0) {
      v = ht ? lds8(&sm.top[x0]) : make_uint2(0x80808080u, 0x80808080u);
    } else {
      uint32_t b = mode == 1 ? (hl ? sm.left[y] : 128u) : (uint32_t)dc16(ht, hl);
      v = make_uint2(b * 0x01010101u, b * 0x01010101u);
    }
    *(uint2*)o = v;
  }
  __syncwarp();
}
// Intra 16x16 analysis (enc.rs:1637 analyse_i16_edges): SATD per mode; the best mode and its cost.
struct I16Fit {
  int mode;
  uint32_t cost;
};
__device__ __noinline__ I16Fit analyse_i16(bool ht, bool hl, int tl) {
  int lane = lane_id();
  int dc = dc16(ht, hl);
  uint32_t sv = 0, sh = 0, sd = 0;
  if (lane < 16) {
    int bx = lane & 3, by = lane >> 2;
    // hadamard4x4_16x4_scalar of the source block, out[4 v + h]
    int rows[4][4];
#pragma unroll
    for (int y = 0; y < 4; y++) {
      const uint8_t* s = &sm.src_y[(by * 4 + y) * 16 + bx * 4];
      int s01 = s[0] + s[1], d01 = s[0] - s[1], s23 = s[2] + s[3], d23 = s[2] - s[3];
      rows[y][0] = s01 + s23; rows[y][1] = s01 - s23; rows[y][2] = d01 + d23; rows[y][3] = d01 - d23;
    }
    int tv[4], th[4];
    {
      const uint8_t* t = &sm.top[bx * 4];
      int e0 = ht ? t[0] : 0, e1 = ht ? t[1] : 0, e2 = ht ? t[2] : 0, e3 = ht ? t[3] : 0;
      int s01 = e0 + e1, d01 = e0 - e1, s23 = e2 + e3, d23 = e2 - e3;
      tv[0] = 4 * (s01 + s23); tv[1] = 4 * (s01 - s23); tv[2] = 4 * (d01 + d23); tv[3] = 4 * (d01 - d23);
      const uint8_t* l = &sm.left[by * 4];
      e0 = hl ? l[0] : 0; e1 = hl ? l[1] : 0; e2 = hl ? l[2] : 0; e3 = hl ? l[3] : 0;
      s01 = e0 + e1; d01 = e0 - e1; s23 = e2 + e3; d23 = e2 - e3;
      th[0] = 4 * (s01 + s23); th[1] = 4 * (s01 - s23); th[2] = 4 * (d01 + d23); th[3] = 4 * (d01 - d23);
    }
#pragma unroll
    for (int h = 0; h < 4; h++) {
      int c0 = rows[0][h], c1 = rows[1][h], c2 = rows[2][h], c3 = rows[3][h];
      int s01 = c0 + c1, d01 = c0 - c1, s23 = c2 + c3, d23 = c2 - c3;
      int col[4] = {s01 + s23, s01 - s23, d01 + d23, d01 - d23};
#pragma unroll
      for (int v = 0; v < 4; v++) {
        int c = col[v], k = 4 * v + h;
        int pv = v == 0 ? tv[h] : 0, ph = h == 0 ? th[v] : 0, pd = k == 0 ? 16 * dc : 0;
        sv += abs(c - pv); sh += abs(c - ph); sd += abs(c - pd);
      }
    }
  }
  sv = wsum(sv) >> 1; sh = wsum(sh) >> 1; sd = wsum(sd) >> 1;
  uint32_t best = sd;
  int mode = 2;
  if (ht && sv < best) { best = sv; mode = 0; }
  if (hl && sh < best) { best = sh; mode = 1; }
  if (ht && hl) {
    pred16_into(3, (int)offsetof(Smem, tmp_y), ht, hl, tl);
    const uint32_t s = satd16((int)offsetof(Smem, tmp_y));
    if (s < best) { best = s; mode = 3; }
  }
  return I16Fit{mode, best};
}
// Chroma intra prediction sample of mode for plane p at (x, y).
__device__ __forceinline__ int predc_sample(int mode, int p, bool ht, bool hl, int tl, int x, int y,
                                            const int* dcv, int pa, int pb, int pc) {
  switch (mode) {
    case 0: return dcv[(y >> 2) * 2 + (x >> 2)];
    case 1: return hl ? sm.cleft[p][y] : 128;
    case 2: return ht ? sm.ctop[p][x] : 128;
    default: return clip255((pa + pb * (x - 3) + pc * (y - 3) + 16) >> 5);
  }
}
// DC and plane parameters of plane p's chroma prediction; called by the whole warp with p =
// lane / 16. In each half-warp lanes 0..7 hold top[0..7], lanes 8..15 left[0..7] (DC sums of four
// by two butterflies), then lanes 0..3 the terms of H, lanes 4..7 those of V.
__device__ void chroma_pred_params(int p, bool ht, bool hl, int tl, int* dcv, int& pa, int& pb, int& pc) {
  const uint8_t* t = sm.ctop[p];
  const uint8_t* l = sm.cleft[p];
  int lane = lane_id(), j = lane & 15, base = lane & 16;
  int e = j < 8 ? (ht ? t[j] : 0) : (hl ? l[j - 8] : 0);
  e += __shfl_xor_sync(FULL, e, 1);
  e += __shfl_xor_sync(FULL, e, 2);
  int st0 = __shfl_sync(FULL, e, base), st1 = __shfl_sync(FULL, e, base + 4);
  int sl0 = __shfl_sync(FULL, e, base + 8), sl1 = __shfl_sync(FULL, e, base + 12);
  if (ht && hl) {
    dcv[0] = (st0 + sl0 + 4) >> 3; dcv[1] = (st1 + 2) >> 2; dcv[2] = (sl1 + 2) >> 2; dcv[3] = (st1 + sl1 + 4) >> 3;
  } else if (ht) {
    dcv[0] = dcv[2] = (st0 + 2) >> 2; dcv[1] = dcv[3] = (st1 + 2) >> 2;
  } else if (hl) {
    dcv[0] = dcv[1] = (sl0 + 2) >> 2; dcv[2] = dcv[3] = (sl1 + 2) >> 2;
  } else {
    dcv[0] = dcv[1] = dcv[2] = dcv[3] = 128;
  }
  int q = j & 3;
  bool top = j < 4, av = top ? ht : hl;
  const uint8_t* ed = top ? t : l;
  int e4 = av ? ed[4 + q] : 128, ep = q == 3 ? tl : (av ? ed[2 - q] : 128);
  int term = j < 8 ? (q + 1) * (e4 - ep) : 0;
  term += __shfl_xor_sync(FULL, term, 1);
  term += __shfl_xor_sync(FULL, term, 2);
  int H = __shfl_sync(FULL, term, base), V = __shfl_sync(FULL, term, base + 4);
  pa = 16 * ((ht ? t[7] : 128) + (hl ? l[7] : 128));
  pb = (17 * H + 16) >> 5;
  pc = (17 * V + 16) >> 5;
}
// The sample diagonally above-left of the macroblock in each plane (128 when absent).
struct Corner {
  int y, u, v;
};
// Intra chroma mode by SAD (enc.rs:1526 analyse_chroma_intra); best prediction into pred_u/v.
__device__ __noinline__ int analyse_chroma(bool ht, bool hl, Corner k0) {
  int lane = lane_id();
  int plane = lane >> 4, idx = (lane & 15) * 4, y = idx >> 3, x0 = idx & 7;
  const int plane_tl = plane ? k0.v : k0.u;
  int dcv[4], pa, pb, pc;
  chroma_pred_params(plane, ht, hl, plane_tl, dcv, pa, pb, pc);
  const uint8_t* s = (plane ? sm.src_v : sm.src_u) + y * 8 + x0;
  uint32_t best = UMAX;
  int bm = 0;
  for (int mode = 0; mode < 4; mode++) {
    bool ok = mode == 1 ? hl : (mode == 2 ? ht : (mode == 3 ? (ht && hl) : true));
    if (!ok) continue;
    uint32_t sad = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) sad += abs((int)s[k] - predc_sample(mode, plane, ht, hl, plane_tl, x0 + k, y, dcv, pa, pb, pc));
    uint32_t cost = wsum(sad) + (mode == 0 ? 0u : 8u);
    if (cost < best) { best = cost; bm = mode; }
  }
  uint8_t* out = (plane ? sm.pred_v : sm.pred_u) + y * 8 + x0;
#pragma unroll
  for (int k = 0; k < 4; k++) out[k] = (uint8_t)predc_sample(bm, plane, ht, hl, plane_tl, x0 + k, y, dcv, pa, pb, pc);
  __syncwarp();
  return bm;
}

// Intra 4x4 prediction of mode m (h264_dsp.rs:799 predict_intra_4x4_u8_scalar) into out[16].
// Intra 4x4 prediction (h264.rs:3223 predict_4x4, the nine modes of H.264 8.3.1.2) in closed
// form. The block's edge samples are gathered into Q[16]:
//   Q[0] = Q[1] = l3, Q[2] = l2, Q[3] = l1, Q[4] = l0, Q[5] = top-left, Q[6..13] = t0..t7,
//   Q[14] = t7, Q[15] = the DC value,
// so that every predicted sample of every mode is Q[i], avg2(Q[i], Q[i+1]) or avg3(Q[i], Q[i+1],
// Q[i+2]) with i a function of (mode, x, y) -- e.g. diagonal down-right is avg3 at 4 + x - y,
// horizontal-up at z = x + 2y is avg2 at 3 - z/2 (z even), avg3 at 2 - z/2 (z odd) and l3 past z = 5.
// Returns kind (0 copy, 1 avg2, 2 avg3) << 8 | i.
__host__ __device__ __forceinline__ int i4_tap(int m, int x, int y) {
  switch (m) {
    case 0: return 6 + x;
    case 1: return 4 - y;
    case 2: return 15;
    case 3: return 0x200 | (6 + x + y);
    case 4: return 0x200 | (4 + x - y);
    case 5: {
      int z = 2 * x - y;
      return z < 0 ? 0x200 | (5 + z) : ((z & 1) ? 0x200 | (4 + x - (y >> 1)) : 0x100 | (5 + x - (y >> 1)));
    }
    case 6: {
      int z = 2 * y - x;
      return z < 0 ? 0x200 | (3 - z) : ((z & 1) ? 0x200 | (3 - (z >> 1)) : 0x100 | (4 - (z >> 1)));
    }
    case 7: return ((y & 1) ? 0x200 : 0x100) | (6 + x + (y >> 1));
    default: {
      int z = x + 2 * y;
      return z > 5 ? 1 : ((z & 1) ? 0x200 | (2 - (z >> 1)) : 0x100 | (3 - (z >> 1)));
    }
  }
}
// The taps of every (mode, sample) for the nine-prediction loop: i | min(i + 1, 15) << 4 |
// min(i + 2, 15) << 8 | kind << 12, at [16 m + 4 y + x] (filled from i4_tap by upload_tables).
__device__ uint16_t g_i4tap[9 * 16];
// ---------------------------------------------------------------------------------------------
// A macroblock; its picture's descriptor and parameters are in shared memory (sm.sd, sm.fp): the
// acquire of every wait drops the SM's L1, so read through global memory each use of them was an
// L2 access.
struct Ctx {
  int mbx, mby, mb;
};
__device__ __forceinline__ void load_desc(const StreamDev* p) {
  constexpr int n = (int)(sizeof(StreamDev) / 8);
  static_assert(n <= 32, "a word a lane");
  const int lane = lane_id();
  uint2 a = make_uint2(0u, 0u);
  if (lane < n) a = ((const uint2*)p)[lane];
  __syncwarp();
  if (lane < n) ((uint2*)&sm.sd)[lane] = a;
  __syncwarp();
}
__device__ __forceinline__ void load_params(const FrameParams& fp) {
  constexpr int n = (int)(sizeof(FrameParams) / 4);
  static_assert(n <= 32, "a word a lane");
  const int lane = lane_id();
  __syncwarp();
  if (lane < n) ((int*)&sm.fp)[lane] = ((const int*)&fp)[lane];
  __syncwarp();
}

// Loads the source macroblock, replicating the last row / column past the picture edges
// (enc.rs:400 MbSrc::load, h264.rs:3660 extract_mb_planes).
__device__ __noinline__ void load_source(const Ctx c) {
  const FrameParams& fp = sm.fp;
  int lane = lane_id();
  int W = fp.width, H = fp.height, cw = (W + 1) >> 1, ch = (H + 1) >> 1;
  int y = min(c.mby * 16 + (lane >> 1), H - 1);
  const uint8_t* row = sm.sd.src_y + (long)y * fp.src_stride_y;
  int x0 = c.mbx * 16 + (lane & 1) * 8;
#pragma unroll
  for (int k = 0; k < 8; k++) sm.src_y[(lane >> 1) * 16 + (lane & 1) * 8 + k] = __ldg(row + min(x0 + k, W - 1));
  int plane = lane >> 4, idx = (lane & 15) * 4, r = idx >> 3, c0 = idx & 7;
  int cy = min(c.mby * 8 + r, ch - 1);
  const uint8_t* crow = (plane ? sm.sd.src_v : sm.sd.src_u) + (long)cy * fp.src_stride_uv;
  uint8_t* dst = (plane ? sm.src_v : sm.src_u) + r * 8 + c0;
#pragma unroll
  for (int k = 0; k < 4; k++) dst[k] = __ldg(crow + min(c.mbx * 8 + c0 + k, cw - 1));
  __syncwarp();
}
// Intra edges from the unfiltered reconstruction of this picture (enc.rs:1459-1521) into shared
// memory; returns the samples at the corner.
__device__ __noinline__ Corner load_edges(const Ctx c, bool want_topright) {
  const FrameParams& fp = sm.fp;
  int lane = lane_id();
  const uint8_t* Y = sm.sd.cur_y;
  int x0 = c.mbx * 16, y0 = c.mby * 16;
  bool ht = c.mby > 0, hl = c.mbx > 0;
  if (ht && lane < 24) {
    bool ok = lane < 16 || (want_topright && c.mbx + 1 < fp.mb_w);
    sm.top[lane] = ok ? ldcg_u8(Y + (long)(y0 - 1) * fp.stride_y + x0 + lane) : 0;
  }
  if (hl && lane < 16) sm.left[lane] = ldcg_u8(Y + (long)(y0 + lane) * fp.stride_y + x0 - 1);
  int cx0 = c.mbx * 8, cy0 = c.mby * 8;
  if (lane < 16) {
    int p = lane >> 3, k = lane & 7;
    const uint8_t* P = p ? sm.sd.cur_v : sm.sd.cur_u;
    if (ht) sm.ctop[p][k] = ldcg_u8(P + (long)(cy0 - 1) * fp.stride_c + cx0 + k);
    if (hl) sm.cleft[p][k] = ldcg_u8(P + (long)(cy0 + k) * fp.stride_c + cx0 - 1);
  }
  Corner k;
  k.y = (ht && hl) ? ldcg_u8(Y + (long)(y0 - 1) * fp.stride_y + x0 - 1) : 128;
  k.u = (ht && hl) ? ldcg_u8(sm.sd.cur_u + (long)(cy0 - 1) * fp.stride_c + cx0 - 1) : 128;
  k.v = (ht && hl) ? ldcg_u8(sm.sd.cur_v + (long)(cy0 - 1) * fp.stride_c + cx0 - 1) : 128;
  __syncwarp();
  return k;
}

// Stores the reconstruction of pred_y/u/v (or tmp_y for luma: its byte offset in Smem) into the current picture.
__device__ __noinline__ void store_recon(const Ctx c, int ly) {
  const FrameParams& fp = sm.fp;
  int lane = lane_id();
  int y = lane >> 1, x = (lane & 1) * 8;
  uint2 v = *(const uint2*)sm_at(ly + y * 16 + x);
  *(uint2*)(sm.sd.cur_y + (long)(c.mby * 16 + y) * fp.stride_y + c.mbx * 16 + x) = v;
  if (sm.sd.unf_y) {
    int cw = fp.mb_w * 16;
    *(uint2*)(sm.sd.unf_y + (long)(c.mby * 16 + y) * cw + c.mbx * 16 + x) = v;
  }
  if (lane < 16) {
    int p = lane >> 3, r = lane & 7;
    uint2 cv = *(const uint2*)&(p ? sm.pred_v : sm.pred_u)[r * 8];
    uint8_t* P = p ? sm.sd.cur_v : sm.sd.cur_u;
    *(uint2*)(P + (long)(c.mby * 8 + r) * fp.stride_c + c.mbx * 8) = cv;
    uint8_t* U = p ? sm.sd.unf_v : sm.sd.unf_u;
    if (U) *(uint2*)(U + (long)(c.mby * 8 + r) * (fp.mb_w * 8) + c.mbx * 8) = cv;
  }
}

// The record is written by 32-bit words, a word per lane and store (it is 8-byte aligned at best, so
// no wider): words 0..8 the head, 9..136 the luma levels, 137..144 the Intra16x16 DC levels, 145..148
// and 149..212 the chroma levels.
constexpr int kWordLuma = offsetof(rg_mb_out, luma) / 4, kWordLumaDc = offsetof(rg_mb_out, luma_dc) / 4,
              kWordChromaDc = offsetof(rg_mb_out, chroma_dc) / 4, kWordChromaAc = offsetof(rg_mb_out, chroma_ac) / 4,
              kWordParts = offsetof(rg_mb_out, part_mv) / 4;
static_assert(kWordLuma == 9 && offsetof(rg_mb_out, mv) == 8 && offsetof(rg_mb_out, mvd) == 12 &&
                  offsetof(rg_mb_out, i4_modes) == 16 && offsetof(rg_mb_out, nz_mask) == 32,
              "the head's words");
__device__ __forceinline__ uint32_t pack16(int lo, int hi) { return __byte_perm((uint32_t)lo, (uint32_t)hi, 0x5410); }
// The chroma levels of the record (zig-zag): word w of the AC levels holds slots 2 (w & 7), 2 (w & 7)
// + 1 of block w / 8 (plane * 4 + block); slot 0 (the DC position) stays 0.
__device__ __noinline__ void record_chroma(rg_mb_out* rec, int cbpc) {
  const int lane = lane_id(), i = (lane & 7) * 2;
  const int r0 = (int)((kScan4Packed >> (4 * i)) & 15), r1 = (int)((kScan4Packed >> (4 * i + 4)) & 15);
  uint32_t* w = (uint32_t*)rec;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int blk = (lane >> 3) + 4 * k;
    const uint32_t v = pack16(i ? sm.ccoef[blk * 16 + r0] : 0, sm.ccoef[blk * 16 + r1]);
    w[kWordChromaAc + lane + 32 * k] = cbpc >= 2 ? v : 0u;
  }
  if (lane < 4) w[kWordChromaDc + lane] = cbpc >= 1 ? ((const uint32_t*)sm.cdc)[lane] : 0u;
}
// The 4x4 luma levels of the record in zig-zag order: word w holds levels 2 (w & 7), 2 (w & 7) + 1 of
// block w / 8.
__device__ __noinline__ void record_luma4x4(rg_mb_out* rec) {
  const int lane = lane_id(), i = (lane & 7) * 2;
  const int r0 = (int)((kScan4Packed >> (4 * i)) & 15), r1 = (int)((kScan4Packed >> (4 * i + 4)) & 15);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int16_t* c = &sm.coef[((lane >> 3) + 4 * k) * 16];
    ((uint32_t*)rec)[kWordLuma + lane + 32 * k] = pack16(c[r0], c[r1]);
  }
}
// The head's words. i4: the modes of sm.i4m, otherwise all DC (2).
__device__ __noinline__ void record_header(rg_mb_out* rec, int type, int i16_mode, int cmode, int cbp, int t8, int qp, int mvx, int mvy,
                              int mvdx, int mvdy, uint32_t nz, bool i4) {
  const int lane = lane_id();
  uint32_t v = i4 ? ((const uint32_t*)sm.i4m)[lane & 3] : 0x02020202u;  // words 4..7
  v = lane == 0 ? (uint32_t)(type | (i16_mode << 8) | (cmode << 16) | (cbp << 24)) : v;
  v = lane == 1 ? (uint32_t)(t8 | (qp << 8)) : v;
  v = lane == 2 ? pack16(mvx, mvy) : v;
  v = lane == 3 ? pack16(mvdx, mvdy) : v;
  v = lane == 8 ? nz : v;
  if (lane < 9) ((uint32_t*)rec)[lane] = v;
}
// What later macroblocks and the deblocking filter read of this one (lane 0 stores it).
__device__ __forceinline__ void write_info(const Ctx c, int flags, int cbpl, int mvx, int mvy, int ref, uint32_t nz, bool i4) {
  if (lane_id() != 0) return;
  uint32_t bottom = 0x2222u, right = 0x2222u;
  if (i4) {  // bottom row blocks 10, 11, 14, 15 and right column blocks 5, 7, 13, 15 (decoding order)
    bottom = sm.i4m[10] | (sm.i4m[11] << 4) | (sm.i4m[14] << 8) | (sm.i4m[15] << 12);
    right = sm.i4m[5] | (sm.i4m[7] << 4) | (sm.i4m[13] << 8) | (sm.i4m[15] << 12);
  }
  static_assert(offsetof(MbInfo, ref) == 4 && offsetof(MbInfo, qp) == 7 && offsetof(MbInfo, i4_bottom) == 10 &&
                    offsetof(MbInfo, i4_right) == 12, "MbInfo packed by words");
  *(uint4*)(sm.sd.info + c.mb) = make_uint4(pack16(mvx, mvy), (uint32_t)(ref & 255) | (flags << 8) | (cbpl << 16) | (sm.sd.qp << 24),
                                            nz | (bottom << 16), right);
}

// I16x16 coding and reconstruction (enc.rs:3587 code_i16) with prediction mode `mode`.
__device__ __noinline__ void code_i16(const Ctx c, int mode, bool ht, bool hl, Corner k0) {
  int lane = lane_id();
  int qp = sm.sd.qp, qpc = sm.sd.qpc;
  pred16_into(mode, (int)offsetof(Smem, pred_y), ht, hl, k0.y);
  int cmode = analyse_chroma(ht, hl, k0);
  uint32_t shift, bias;
  quant4_params(qp, true, shift, bias);
  uint32_t my_ac = 0, my_nz = 0;
  int lv[16];
  if (lane < 16) {
    int bx = blk_x(lane), by = blk_y(lane);
    int d[16], cc[16];
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
      for (int x = 0; x < 4; x++) {
        int o = (by * 4 + y) * 16 + bx * 4 + x;
        d[y * 4 + x] = (int)sm.src_y[o] - (int)sm.pred_y[o];
      }
    fdct4(d, cc);
    sm.ldc[by * 4 + bx] = (int16_t)cc[0];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      lv[i] = quant_level(cc[i], c_mf4[qp % 6][pos4(i)], bias, shift);
      if (lv[i]) my_nz = 1;
    }
  }
  // a group with any level drops its DC slots; AC presence counts only slots 1..15
  uint32_t gnz = my_nz | __shfl_xor_sync(FULL, my_nz, 1);
  gnz |= __shfl_xor_sync(FULL, gnz, 2);
  if (lane < 16) {
    if (gnz) lv[0] = 0;
    else {
#pragma unroll
      for (int i = 0; i < 16; i++) lv[i] = 0;
    }
#pragma unroll
    for (int i = 1; i < 16; i++) if (lv[i]) my_ac = 1;
#pragma unroll
    for (int i = 0; i < 16; i++) sm.coef[lane * 16 + i] = (int16_t)lv[i];
  }
  __syncwarp();
  int cbpl = wor(my_ac) ? 15 : 0;
  // luma DC: Hadamard (>> 1) + quantisation (enc.rs:1960), then inverse (h264.rs:1645)
  if (lane == 0) {
    int t[16], had[16];
    for (int r = 0; r < 4; r++) {
      int b0 = sm.ldc[r * 4], b1 = sm.ldc[r * 4 + 1], b2 = sm.ldc[r * 4 + 2], b3 = sm.ldc[r * 4 + 3];
      int s03 = b0 + b3, s12 = b1 + b2, d03 = b0 - b3, d12 = b1 - b2;
      t[r * 4] = s03 + s12; t[r * 4 + 1] = d03 + d12; t[r * 4 + 2] = s03 - s12; t[r * 4 + 3] = d03 - d12;
    }
    for (int k = 0; k < 4; k++) {
      int s03 = t[k] + t[k + 12], s12 = t[k + 4] + t[k + 8], d03 = t[k] - t[k + 12], d12 = t[k + 4] - t[k + 8];
      had[k] = (int16_t)((s03 + s12) >> 1); had[k + 4] = (int16_t)((d03 + d12) >> 1);
      had[k + 8] = (int16_t)((s03 - s12) >> 1); had[k + 12] = (int16_t)((d03 - d12) >> 1);
    }
    int qbits = 16 + qp / 6, mf = c_mf4[qp % 6][0], f = (1 << qbits) / 3;
    int lvl[16];
    for (int i = 0; i < 16; i++) {
      int a = had[i] < 0 ? -had[i] : had[i];
      int l = (a * mf + f) >> qbits;
      lvl[i] = had[i] < 0 ? -l : l;
      sm.ldc[i] = (int16_t)lvl[i];
    }
    int qmul = (c_dq4[qp % 6][0] * 16) << (qp / 6 + 2);
    int tt[16];
    for (int i = 0; i < 4; i++) {
      int z0 = lvl[4 * i] + lvl[4 * i + 1], z1 = lvl[4 * i] - lvl[4 * i + 1];
      int z2 = lvl[4 * i + 2] - lvl[4 * i + 3], z3 = lvl[4 * i + 2] + lvl[4 * i + 3];
      tt[4 * i] = z0 + z3; tt[4 * i + 1] = z0 - z3; tt[4 * i + 2] = z1 - z2; tt[4 * i + 3] = z1 + z2;
    }
    for (int i = 0; i < 4; i++) {
      int z0 = tt[i] + tt[8 + i], z1 = tt[i] - tt[8 + i], z2 = tt[4 + i] - tt[12 + i], z3 = tt[4 + i] + tt[12 + i];
      sm.ldcr[i] = (int16_t)(((z0 + z3) * qmul + 128) >> 8);
      sm.ldcr[4 + i] = (int16_t)(((z1 + z2) * qmul + 128) >> 8);
      sm.ldcr[8 + i] = (int16_t)(((z1 - z2) * qmul + 128) >> 8);
      sm.ldcr[12 + i] = (int16_t)(((z0 - z3) * qmul + 128) >> 8);
    }
  }
  const ChromaAc ac = chroma_quant(qpc, true);
  int cbpc = (ac.any(0) || ac.any(1)) ? 2 : (ac.dc() ? 1 : 0);
  __syncwarp();
  // record
  rg_mb_out* rec = sm.sd.rec + c.mb;
  record_luma4x4(rec);
  if (lane < 16) rec->luma_dc[lane] = sm.ldc[(kScan4Packed >> (4 * lane)) & 15];
  const uint32_t nzm = __ballot_sync(FULL, lane < 16 && cbpl && my_ac);
  record_chroma(rec, cbpc);
  record_header(rec, RG_MB_I16X16, mode, cmode, cbpl | (cbpc << 4), 0, qp, 0, 0, 0, 0, nzm, false);
  // reconstruction
  if (lane < 16) {
    int bx = blk_x(lane), by = blk_y(lane);
    int blk[16], res[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      int v = sm.coef[lane * 16 + i];
      blk[i] = cbpl ? clamp_i16(v * ((int)c_dq4[qp % 6][pos4(i)] << (qp / 6))) : v;
    }
    blk[0] = sm.ldcr[by * 4 + bx];
    idct4(blk, res);
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
      for (int x = 0; x < 4; x++) {
        int o = (by * 4 + y) * 16 + bx * 4 + x;
        sm.pred_y[o] = (uint8_t)clip255(sm.pred_y[o] + res[y * 4 + x]);
      }
  }
  __syncwarp();
  chroma_recon(qpc, cbpc);
  store_recon(c, (int)offsetof(Smem, pred_y));
  write_info(c, kFlagIntra, cbpl, 0, 0, -1, nzm, false);
}

// I4x4 analysis (enc.rs:3336 analyse_i4): sixteen blocks in decoding order, each choosing among
// the available modes by SATD + lambda * (1 if the predicted mode else 4), then quantising and
// reconstructing before the next block. Per block the warp gathers the edge samples (lane k ->
// Q[k]), builds all nine predictions (lane -> pixel, the two half-warps taking even / odd modes),
// costs the modes (lane -> mode), and transforms the chosen residual with shuffles (lane ->
// coefficient). Returns the luma coded block pattern with the blocks
// holding levels in bits 4.. (bit 4 + b: block b), or -1 as soon as the running cost reaches `budget`.
// kMask: only the modes of masks[b] (bit m: Intra4x4PredMode m) that are available at block b are
// tried -- DC alone when none is (the learned form); the plain form tries every available mode.
template <bool kMask>
__device__ __noinline__ int analyse_i4(const Ctx c, uint32_t budget, bool ht_mb, bool hl_mb, int tl_mb,
                                        const uint16_t* masks) {
  const FrameParams& fp = sm.fp;
  int lane = lane_id();
  int p = lane & 15, xl = p & 3, yl = p >> 2;
  int qp = sm.sd.qp;
  uint32_t lambda = c_lambda[qp];
  uint32_t shift, bias;
  quant4_params(qp, true, shift, bias);
  uint32_t mf = c_mf4[qp % 6][pos4(p)];
  int dqs = (int)c_dq4[qp % 6][pos4(p)] << (qp / 6);
  uint32_t total = lambda * 24;
  int cbpl = 0;
  const MbInfo* info = sm.sd.info;
  uint32_t lmodes = hl_mb ? ld_info(&info[c.mb - 1]).i4_right : 0x2222u;
  uint32_t tmodes = ht_mb ? ld_info(&info[c.mb - fp.mb_w]).i4_bottom : 0x2222u;
  // this lane's taps for its predictions (modes lane / 16 + 2 k, sample p): the same for every block
  uint32_t taps[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    int m = (lane >> 4) + 2 * k;
    taps[k] = m < 9 ? __ldg(&g_i4tap[m * 16 + p]) : 0u;
  }
  for (int b = 0; b < 16; b++) {
    int bx = blk_x(b), by = blk_y(b), px = bx * 4, py = by * 4;
    bool ht = by > 0 || ht_mb, hl = bx > 0 || hl_mb;
    bool tr = !(b == 3 || b == 7 || b == 11 || b == 13 || b == 15) && (b != 5 || c.mbx + 1 < fp.mb_w);
    // edge samples (unavailable ones 128; top-right replicated from t3 when unavailable)
    int q = 128;
    if (p <= 4) {
      int j = p <= 1 ? 3 : 4 - p;
      if (hl) q = bx > 0 ? sm.tmp_y[(py + j) * 16 + px - 1] : sm.left[py + j];
    } else if (p == 5) {
      if (ht && hl)
        q = (by > 0 && bx > 0) ? sm.tmp_y[(py - 1) * 16 + px - 1]
                               : (by > 0 ? sm.left[py - 1] : (bx > 0 ? sm.top[px - 1] : tl_mb));
    } else if (p <= 14) {
      int i = min(p - 6, 7);
      if (i >= 4 && !tr) i = 3;
      if (ht) q = by > 0 ? sm.tmp_y[(py - 1) * 16 + px + i] : sm.top[px + i];
    }
    uint32_t sums = wsum(lane < 16 ? ((p >= 6 && p <= 9) ? (uint32_t)q : 0u) + ((p >= 1 && p <= 4) ? (uint32_t)q << 16 : 0u) : 0u);
    int st = (int)(sums & 0xffff), sl = (int)(sums >> 16);
    int dc = ht && hl ? (st + sl + 4) >> 3 : (ht ? (st + 2) >> 2 : (hl ? (sl + 2) >> 2 : 128));
    if (lane < 16) sm.i4q[p] = (uint8_t)(p == 15 ? dc : q);
    // predicted mode (h264.rs:3283)
    int gx = c.mbx * 4 + bx, gy = c.mby * 4 + by;
    int pm;
    if (gx == 0 || gy == 0) pm = 2;
    else {
      int ml = bx > 0 ? sm.i4m[(((by >> 1) << 3) | (((bx - 1) >> 1) << 2) | ((by & 1) << 1) | ((bx - 1) & 1))]
                      : (int)((lmodes >> (4 * by)) & 15);
      int mt = by > 0 ? sm.i4m[((((by - 1) >> 1) << 3) | ((bx >> 1) << 2) | (((by - 1) & 1) << 1) | (bx & 1))]
                      : (int)((tmodes >> (4 * bx)) & 15);
      pm = min(ml, mt);
    }
    __syncwarp();
    // nine predictions and their SATDs: half-warp h takes modes h, h + 2, ... (k = 0..4), lane p
    // sample p; the 4x4 Hadamard of the difference (metrics.rs:705) by four shuffle butterflies,
    // both halves' sums of magnitudes in one reduction (each below 2^16). Every lane ends with
    // the same key, the least cost first and the lower mode on a tie.
    int srcp = sm.src_y[(py + yl) * 16 + px + xl];
    int pv[5];
    uint32_t key = UMAX;
    uint32_t allow = 0x1ffu;
    if constexpr (kMask) {
      uint32_t avail = 0x4u | (ht ? 0x89u : 0u) | (hl ? 0x102u : 0u) | (ht && hl ? 0x70u : 0u);
      allow = masks[b] & avail;
      if (!allow) allow = 0x4u;
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {
      if constexpr (kMask) {
        if (!((allow >> (2 * k)) & 3u)) { pv[k] = 0; continue; }  // neither mode of this step is tried
      }
      uint32_t tp = taps[k], kind = tp >> 12;
      int a0 = sm.i4q[tp & 15], a1 = sm.i4q[(tp >> 4) & 15], a2 = sm.i4q[(tp >> 8) & 15];
      int v = kind == 0 ? a0 : (kind == 1 ? (a0 + a1 + 1) >> 1 : (a0 + 2 * a1 + a2 + 2) >> 2);
      pv[k] = v;
      int d = srcp - v;
#pragma unroll
      for (int b = 1; b < 16; b <<= 1) {
        int o = __shfl_xor_sync(FULL, d, b);
        d = (lane & b) ? o - d : d + o;
      }
      uint32_t sums = __reduce_add_sync(FULL, (uint32_t)(d < 0 ? -d : d) << (16 * (lane >> 4)));
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int m = 2 * k + h;
        if (m > 8) continue;
        bool av = (m == 0 || m == 3 || m == 7) ? ht : ((m == 1 || m == 8) ? hl : (m == 2 ? true : (ht && hl)));
        if constexpr (kMask) av = av && ((allow >> m) & 1u);
        uint32_t cost = (((sums >> (16 * h)) & 0xffffu) >> 1) + lambda * (m == pm ? 1u : 4u);
        if (av) key = min(key, (cost << 4) | (uint32_t)m);
      }
    }
    int bm = (int)(key & 15);
    total += key >> 4;
    if (total >= budget) return -1;
    if (lane == 0) sm.i4m[b] = (uint8_t)bm;
    // residual transform and quantisation, lane p -> coefficient p (raster); the chosen mode's
    // sample p is in lane 16 (bm & 1) + p
    int kb = bm >> 1, mine = pv[0];
#pragma unroll
    for (int k = 1; k < 5; k++)
      if (kb == k) mine = pv[k];
    int pred = __shfl_sync(FULL, mine, (bm & 1) * 16 + p);
    int acc = fwd4_pass(fwd4_pass(srcp - pred, 1, xl), 4, yl);
    acc = (int16_t)acc;
    uint32_t aa = (uint32_t)(acc < 0 ? -acc : acc);
    int l = (int)((aa * mf + bias) >> shift);
    int lvl = acc < 0 ? -l : l;
    if (lane < 16) sm.coef[b * 16 + p] = (int16_t)lvl;
    bool nz = __ballot_sync(FULL, lane < 16 && lvl != 0) != 0;
    if (nz) cbpl |= (1 << (b >> 2)) | (16 << b);
    // inverse transform (rows then columns) and reconstruction
    int rec = pred;
    if (nz) {
      int dq = clamp_i16(lvl * dqs);
      int r = (int16_t)((inv4_pass(inv4_pass(dq, 1, xl), 4, yl) + 32) >> 6);
      rec = clip255(pred + r);
    }
    if (lane < 16) sm.tmp_y[(py + yl) * 16 + px + xl] = (uint8_t)rec;
    __syncwarp();
  }
  return cbpl;
}

// `luma`: what analyse_i4 returned.
__device__ __noinline__ void code_i4(const Ctx c, int luma, bool ht, bool hl, Corner k0) {
  int lane = lane_id();
  int qpc = sm.sd.qpc;
  const int cbpl = luma & 15;
  const uint32_t nzm = (uint32_t)luma >> 4;
  int cmode = analyse_chroma(ht, hl, k0);
  const ChromaAc ac = chroma_quant(qpc, true);
  int cbpc = (ac.any(0) || ac.any(1)) ? 2 : (ac.dc() ? 1 : 0);
  rg_mb_out* rec = sm.sd.rec + c.mb;
  record_luma4x4(rec);
  if (lane < 8) ((uint32_t*)rec)[kWordLumaDc + lane] = 0u;
  record_chroma(rec, cbpc);
  record_header(rec, RG_MB_I4X4, 0, cmode, cbpl | (cbpc << 4), 0, sm.sd.qp, 0, 0, 0, 0, nzm, true);
  chroma_recon(qpc, cbpc);
  store_recon(c, (int)offsetof(Smem, tmp_y));
  write_info(c, kFlagIntra, cbpl, 0, 0, -1, nzm, true);
}

// One macroblock of an I slice (enc.rs:3311 code_intra).
__device__ __noinline__ void analyse_intra_mb(const Ctx c) {
  const Corner k0 = load_edges(c, true);
  bool ht = c.mby > 0, hl = c.mbx > 0;
  uint32_t lambda = c_lambda[sm.sd.qp];
  const I16Fit fit16 = analyse_i16(ht, hl, k0.y);
  if (fit16.cost > 40 * lambda) {
    const int cbpl = analyse_i4<false>(c, fit16.cost + lambda * 4, ht, hl, k0.y, nullptr);
    if (cbpl >= 0) {
      code_i4(c, cbpl, ht, hl, k0);
      return;
    }
  }
  code_i16(c, fit16.mode, ht, hl, k0);
}

// Codes P_Skip with vector mv; prediction already in pred_y / pred_u / pred_v.
__device__ __noinline__ void code_skip(const Ctx c, int mvx, int mvy) {
  const int lane = lane_id();
  rg_mb_out* rec = sm.sd.rec + c.mb;
#pragma unroll
  for (int k = 0; k < 7; k++)
    if (kWordLuma + lane + 32 * k < kWordParts) ((uint32_t*)rec)[kWordLuma + lane + 32 * k] = 0u;
  record_header(rec, RG_MB_P_SKIP, 0, 0, 0, 0, sm.sd.qp, mvx, mvy, 0, 0, 0, false);
  write_info(c, kFlagSkip, 0, mvx, mvy, 0, 0, false);
  store_recon(c, (int)offsetof(Smem, pred_y));
}

// Probe of the skip residual (enc.rs:2163 probe_skip_luma): no level above 1 and a total
// decimation score below 6.
__device__ __noinline__ bool probe_skip_luma(int qp) {
  Half4 v;
  const uint32_t m = luma4x4_levels(qp, v);
  const uint32_t score = (lane_id() & 1) ? 0u : score4(m, 0);
  return wsum(score | ((m >> 16) << 16)) < 6;
}

// The residual of an inter macroblock whose prediction lies in pred_y / pred_u / pred_v
// (enc.rs:3158-3190), its record (code_inter, enc.rs:3196) and its reconstruction. can_skip: nothing
// coded makes it P_Skip with vector (mvx, mvy). Returns whether it did.
__device__ __noinline__ bool code_inter(const Ctx c, int type, bool can_skip, int mvx, int mvy, int mvdx, int mvdy) {
  const int lane = lane_id(), qp = sm.sd.qp, qpc = sm.sd.qpc;
  const Luma4 l4 = luma4x4_inter(qp);
  uint32_t cbpl = l4.cbp;
  bool use8 = false;
  if (sm.fp.t8x8 && l4.cbp) {
    const uint32_t r8 = luma8x8_inter(qp);
    if ((r8 >> 4) <= l4.nnz) { use8 = true; cbpl = r8 & 15u; }
  }
  const ChromaAc ac = chroma_quant(qpc, false);
  // drop a plane's AC levels when nearly empty (enc.rs:2095)
  const bool drop_u = ac.any(0) && ac.score(0) < 7, drop_v = ac.any(1) && ac.score(1) < 7;
  if ((lane & 16) ? drop_v : drop_u) *(uint2*)&sm.ccoef[lane * 4] = make_uint2(0u, 0u);
  __syncwarp();
  const bool acu = ac.any(0) && !drop_u, acv = ac.any(1) && !drop_v;
  const int cbpc = (acu || acv) ? 2 : (ac.dc() ? 1 : 0);
  if (cbpl == 0 && cbpc == 0 && can_skip) {
    code_skip(c, mvx, mvy);
    return true;
  }
  rg_mb_out* rec = sm.sd.rec + c.mb;
  const bool t8flag = use8 && cbpl != 0;
  uint32_t nzm = l4.nz16;
  if (use8) {
#pragma unroll
    for (int k = 0; k < 4; k++) ((uint32_t*)rec)[kWordLuma + lane + 32 * k] = ((const uint32_t*)sm.coef8)[lane + 32 * k];
    nzm = (cbpl & 1u ? 0xfu : 0u) | (cbpl & 2u ? 0xf0u : 0u) | (cbpl & 4u ? 0xf00u : 0u) | (cbpl & 8u ? 0xf000u : 0u);
  } else {
    record_luma4x4(rec);
  }
  if (lane < 8) ((uint32_t*)rec)[kWordLumaDc + lane] = 0u;
  record_chroma(rec, cbpc);
  record_header(rec, type, 0, 0, (int)cbpl | (cbpc << 4), t8flag, qp, mvx, mvy, mvdx, mvdy, nzm, false);
  write_info(c, t8flag ? kFlagT8 : 0, (int)cbpl, mvx, mvy, 0, nzm, false);
  if (cbpl) {
    if (use8) recon_luma8x8(qp, (int)cbpl);
    else recon_luma4x4(qp);
  }
  chroma_recon(qpc, cbpc);
  store_recon(c, (int)offsetof(Smem, pred_y));
  return false;
}

// ---------------------------------------------------------------------------------------------
// Pipelined mode synchronisation: monotonic progress counters, published with a release store
// after a fence, awaited with an acquire load. Every wait has a time limit; when it runs out
// the kernel records RG_ERR_TIMEOUT and all warps leave.
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int atom_add_acq_rel(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void st_release_sys(int* p, int v) {
  asm volatile("st.release.sys.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits until every lane's counter has reached its need (p null: the lane waits for nothing). The
// counters a macroblock depends on are taken by different lanes at once: one round trip, and one
// drop of the SM's L1 by the acquires, instead of one per counter. `seen` is the lane's last acquired
// value: no load when it covers `need` already (the acquire that returned it orders every later load
// of this warp). The first check and the final one are acquire loads; in between the lanes poll with
// relaxed loads (which leave the L1 alone) and sleep 32 ns doubling to 512 ns. False on timeout
// (recorded in *error) or when another warp failed.
__device__ __noinline__ bool wait_all(const int* p, int need, int& seen, int* error, unsigned long long timeout_ns) {
  bool ok = !p || seen >= need;
  if (__all_sync(FULL, ok)) return true;
  unsigned long long t0 = 0;
  unsigned int sleep = 32;
  while (true) {
    if (!ok) seen = ld_acquire(p);
    ok = !p || seen >= need;
    if (__all_sync(FULL, ok)) {
      __syncwarp();  // every lane's later loads follow the acquires
      return true;
    }
    if (!t0) t0 = global_ns();
    while (true) {  // until no lane is behind
      const bool behind = !ok && ld_relaxed(p) < need;
      const bool fail = lane_id() == 0 && ld_relaxed(error);
      const bool late = lane_id() == 0 && global_ns() - t0 > timeout_ns;
      const uint32_t b = __ballot_sync(FULL, behind);
      if (!b) break;
      if (__any_sync(FULL, fail)) return false;
      if (__any_sync(FULL, late)) {
        if (lane_id() == 0) atomicCAS(error, 0, 1);
        return false;
      }
      __nanosleep(sleep);
      sleep = min(sleep * 2, 512u);
    }
  }
}
// Publishes v after this warp's global writes: the warp barrier orders every lane's writes before lane
// 0's release store, which is cumulative over them.
__device__ __forceinline__ void publish(int* p, int v) {
  __syncwarp();
  if (lane_id() == 0) st_release(p, v);
}
// What a P macroblock of the pipelined mode waits for in its reference picture (kernel constants and
// addresses; the state is in shared memory).
struct PipeWait {
  const int* db_prev;    // deblocking progress per row of the reference picture (padding included); null: no wait
  int* error;
  unsigned long long timeout_ns;
};
// Waits until the reference picture is final over the macroblocks left of and above (xx, rr),
// clamped to the picture: rows above the last are final where the row below is deblocked; the last
// row where its right neighbour is.
__device__ __noinline__ bool wait_reference(const Ctx c, const PipeWait pw, int xb, int rb) {
  const FrameParams& fp = sm.fp;
  const int rr = min(max(rb, 0), fp.mb_h - 1), xx = min(max(xb, 0), fp.mb_w - 1);
  const int row = rr < fp.mb_h - 1 ? rr + 1 : rr, need = rr < fp.mb_h - 1 ? xx + 1 : min(xx + 2, fp.mb_w);
  int seen = row == sm.db_row ? sm.seen_db : 0;
  // zero motion reaches (mbx + 2, mby + 2); the host sizes the picture lag from the maximum
  const int ry = max(sm.reach_y, max(rr - c.mby - 2, 0) + 1), rx = max(sm.reach_x, max(xx - c.mbx - 2, 0) + 1);
  const bool ok = wait_all(lane_id() == 0 ? pw.db_prev + row : nullptr, need, seen, pw.error, pw.timeout_ns);
  __syncwarp();
  if (lane_id() == 0) {
    sm.reach_y = ry;
    sm.reach_x = rx;
    sm.db_row = row;
    sm.seen_db = seen;
  }
  __syncwarp();
  return ok;
}

// One macroblock of a P slice (enc.rs:3011 code_p_mb). In the pipelined mode (pw.db_prev) it first
// waits for the reference frame to be final over every sample its search can read; when a wait
// gives up it returns false and writes nothing.
__device__ __noinline__ bool analyse_p_mb(const Ctx c, const PipeWait pw) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  int lane = lane_id();
  int mbx = c.mbx, mby = c.mby, mb_w = fp.mb_w;
  int x0 = mbx * 16, y0 = mby * 16;
  int qp = sm.sd.qp;
  uint32_t lambda = c_lambda[qp];
  int cw = fp.mb_w * 16, chh = fp.mb_h * 16;
  // MvBounds (enc.rs:1105)
  int bmin0 = -4 * (x0 + 28), bmin1 = max(-4 * (y0 + 28), -2048);
  int bmax0 = 4 * (cw - 16 - x0 + 28), bmax1 = min(4 * (chh - 16 - y0 + 28), 2044);
  // neighbours (this picture)
  const MbInfo* info = sd.info;
  int lref = -2, tref = -2, dref = -2;
  int a0 = 0, a1 = 0, b0 = 0, b1 = 0, c0 = 0, c1 = 0;
  if (mbx > 0) { MbInfo n = ld_info(&info[c.mb - 1]); lref = n.ref; a0 = n.mv[0]; a1 = n.mv[1]; }
  if (mby > 0) { MbInfo n = ld_info(&info[c.mb - mb_w]); tref = n.ref; b0 = n.mv[0]; b1 = n.mv[1]; }
  if (mby > 0 && mbx + 1 < mb_w) { MbInfo n = ld_info(&info[c.mb - mb_w + 1]); dref = n.ref; c0 = n.mv[0]; c1 = n.mv[1]; }
  else if (mby > 0 && mbx > 0) { MbInfo n = ld_info(&info[c.mb - mb_w - 1]); dref = n.ref; c0 = n.mv[0]; c1 = n.mv[1]; }
  // pred_motion_partition (h264.rs:3577), 16x16, ref 0
  int mvp0, mvp1;
  {
    auto med = [](int x, int y, int z) { return min(max(x, y), max(min(x, y), z)); };
    int m = (lref == 0) + (tref == 0) + (dref == 0);
    if (m > 1) { mvp0 = med(a0, b0, c0); mvp1 = med(a1, b1, c1); }
    else if (m == 1) {
      if (lref == 0) { mvp0 = a0; mvp1 = a1; }
      else if (tref == 0) { mvp0 = b0; mvp1 = b1; }
      else { mvp0 = c0; mvp1 = c1; }
    } else if (tref == -2 && dref == -2 && lref != -2) { mvp0 = a0; mvp1 = a1; }
    else { mvp0 = med(a0, b0, c0); mvp1 = med(a1, b1, c1); }
  }
  int ps0 = mvp0, ps1 = mvp1;
  if (mbx == 0 || mby == 0 || (lref == 0 && a0 == 0 && a1 == 0) || (tref == 0 && b0 == 0 && b1 == 0)) { ps0 = 0; ps1 = 0; }
  load_source(c);
  int qpc = sm.sd.qpc;
  // co-located vector of the previous picture: a search candidate (enc.rs:3094)
  MbInfo prevmb = ld_info(&sd.prev_info[c.mb]);
  if (pw.db_prev) {
    // The right- and bottom-most reference sample this macroblock can read: the full-pel
    // candidates, a diamond of at most 16 steps around the best, the half-sample window
    // (-3..+20) and 8-byte loads. Everything above and to the left of it (padding included) is
    // final once the macroblock holding it is.
    int cx[5] = {mvp0, 0, a0, b0, prevmb.mv[0]}, cy[5] = {mvp1, 0, a1, b1, prevmb.mv[1]};
    int hi0 = -(1 << 20), hi1 = -(1 << 20);
    int imn0 = (bmin0 + 3) >> 2, imn1 = (bmin1 + 3) >> 2, imx0 = bmax0 >> 2, imx1 = bmax1 >> 2;
#pragma unroll
    for (int k = 0; k < 5; k++) {
      hi0 = max(hi0, min(max((cx[k] + 2) >> 2, imn0), imx0));
      hi1 = max(hi1, min(max((cy[k] + 2) >> 2, imn1), imx1));
    }
    if (!wait_reference(c, pw, (x0 + hi0 + 44) >> 4, (y0 + hi1 + 40) >> 4)) return false;
  }

  // 1. skip probe (enc.rs:2906 try_p_skip)
  if (ps0 >= bmin0 && ps0 <= bmax0 && ps1 >= bmin1 && ps1 <= bmax1) {
    mc_luma16(sd.ref_y, fp.stride_y, x0, y0, ps0, ps1);
    uint2 s = src8(), p = *(const uint2*)&sm.pred_y[(lane >> 1) * 16 + (lane & 1) * 8];
    uint32_t sad = wsum(vsad8(s, p));
    if (sad < sm.sd.sb_probe) {
      bool lz = sad <= sm.sd.sb_luma;
      if (!lz) {
        uint32_t ssd = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          int d0 = (int)((s.x >> (8 * k)) & 255) - (int)((p.x >> (8 * k)) & 255);
          int d1 = (int)((s.y >> (8 * k)) & 255) - (int)((p.y >> (8 * k)) & 255);
          ssd += d0 * d0 + d1 * d1;
        }
        lz = wsum(ssd) <= sm.sd.sb_luma_ssd;
      }
      if (!lz) lz = probe_skip_luma(qp);
      if (lz) {
        mc_chroma8(sd.ref_u, sd.ref_v, fp.stride_c, mbx, mby, ps0, ps1);
        // per plane SAD / SSD bounds (lanes 0..15 U, 16..31 V, 4 samples each)
        int plane = lane >> 4, idx = (lane & 15) * 4;
        const uint8_t* ss = (plane ? sm.src_v : sm.src_u) + idx;
        const uint8_t* pp = (plane ? sm.pred_v : sm.pred_u) + idx;
        uint32_t sadp = 0, ssdp = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) { int d = (int)ss[k] - (int)pp[k]; sadp += abs(d); ssdp += d * d; }
        uint32_t sad_u = wsum(plane == 0 ? sadp : 0), sad_v = wsum(plane == 1 ? sadp : 0);
        uint32_t ssd_u = wsum(plane == 0 ? ssdp : 0), ssd_v = wsum(plane == 1 ? ssdp : 0);
        bool zu = sad_u <= sm.sd.sb_chroma || ssd_u <= sm.sd.sb_chroma_ssd;
        bool zv = sad_v <= sm.sd.sb_chroma || ssd_v <= sm.sd.sb_chroma_ssd;
        bool cz = zu && zv;
        if (!cz) {
          const ChromaAc ac = chroma_quant(qpc, false);
          cz = !ac.dc() && ac.score(0) < 7 && ac.score(1) < 7;
        }
        if (cz) {
          code_skip(c, ps0, ps1);
          return true;
        }
      }
    }
  }

  // 2. motion search (enc.rs:3084-3117)
  const uint8_t* ref = sd.ref_y;
  int stride = fp.stride_y;
  // candidates in order: predictor, zero, left (if any), top (if any), co-located of the previous
  // picture -- five fixed slots, the left / top ones skipped when absent
  int imin0 = (bmin0 + 3) >> 2, imin1 = (bmin1 + 3) >> 2, imax0 = bmax0 >> 2, imax1 = bmax1 >> 2;
  uint2 sv = src8();
  const uint8_t* base = ref + (long)(y0 + (lane >> 1)) * stride + x0 + (lane & 1) * 8;
  int best0 = 0, best1 = 0;
  uint32_t best_cost = UMAX;
  // clamped full-pel candidates, their samples loaded together, then costed in order (a
  // repeated position is skipped)
  int cmx[5], cmy[5];
  bool cval[5];
  uint2 cref[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    int vx = k == 0 ? mvp0 : k == 1 ? 0 : k == 2 ? a0 : k == 3 ? b0 : prevmb.mv[0];
    int vy = k == 0 ? mvp1 : k == 1 ? 0 : k == 2 ? a1 : k == 3 ? b1 : prevmb.mv[1];
    cval[k] = k == 2 ? mbx > 0 : (k == 3 ? mby > 0 : true);
    cmx[k] = min(max((vx + 2) >> 2, imin0), imax0);
    cmy[k] = min(max((vy + 2) >> 2, imin1), imax1);
    cref[k] = ldg8(base + (long)cmy[k] * stride + cmx[k]);
  }
#pragma unroll
  for (int k = 0; k < 5; k++) {
    bool use = cval[k];  // absent, or at the position of an earlier candidate: skipped
#pragma unroll
    for (int j = 0; j < k; j++) use &= !(cval[j] && cmx[j] == cmx[k] && cmy[j] == cmy[k]);
    if (!use) continue;  // uniform across the warp
    uint32_t cost = fullpel_cost(sv, cref[k], cmx[k], cmy[k], mvp0, mvp1, lambda);
    if (cost < best_cost) { best_cost = cost; best0 = cmx[k]; best1 = cmy[k]; }
  }
  // diamond (enc.rs:1207-1272): up, left, right, down around the best, first strict minimum
  // wins; each step's four loads are issued together
#pragma unroll 1
  for (int it = 0; it < 16; it++) {
    const uint8_t* cp = base + (long)best1 * stride + best0;
    uint2 r[4];
    bool in[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      int dx = k == 1 ? -1 : (k == 2 ? 1 : 0), dy = k == 0 ? -1 : (k == 3 ? 1 : 0);
      int px = best0 + dx, py = best1 + dy;
      in[k] = px >= imin0 && px <= imax0 && py >= imin1 && py <= imax1;
      r[k] = in[k] ? ldg8(cp + dy * stride + dx) : make_uint2(0u, 0u);
    }
    int nb0 = best0, nb1 = best1;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      int dx = k == 1 ? -1 : (k == 2 ? 1 : 0), dy = k == 0 ? -1 : (k == 3 ? 1 : 0);
      if (!in[k]) continue;  // uniform across the warp
      uint32_t cost = fullpel_cost(sv, r[k], best0 + dx, best1 + dy, mvp0, mvp1, lambda);
      if (cost < best_cost) {
        best_cost = cost;
        nb0 = best0 + dx;
        nb1 = best1 + dy;
      }
    }
    if (nb0 == best0 && nb1 == best1) break;
    best0 = nb0;
    best1 = nb1;
  }
  int mv0, mv1;
  {
    int fm0 = best0 * 4, fm1 = best1 * 4;
    uint32_t full_mvc = mvd_cost(fm0 - mvp0, lambda) + mvd_cost(fm1 - mvp1, lambda);
    if (best_cost - full_mvc <= sm.sd.sb_luma) {
      mv0 = fm0; mv1 = fm1;
      uint2 v = ldg8(base + (long)best1 * stride + best0);
      *(uint2*)&sm.pred_y[(lane >> 1) * 16 + (lane & 1) * 8] = v;
      __syncwarp();
    } else {
      // sub-pel refinement over a half-sample window around the full-pel best (enc.rs:1283)
      int bxp = x0 + best0, byp = y0 + best1;
      stage_window(ref, stride, bxp - 1, byp - 1);
      build_hpel(7);
      int q0 = fm0, q1 = fm1;
      uint32_t bc = best_cost;
#pragma unroll 1
      for (int si = 0; si < 2; si++) {
        int st = si == 0 ? 2 : 1, iters = si == 0 ? 1 : 2;
#pragma unroll 1
        for (int it = 0; it < iters; it++) {
          int f0 = q0, f1 = q1;
          int dd[4][2] = {{0, -st}, {-st, 0}, {st, 0}, {0, st}};
          uint32_t cc[4];
#pragma unroll
          for (int k = 0; k < 4; k++) {
            int cx = f0 + dd[k][0], cy = f1 + dd[k][1];
            bool ok = abs(cx - fm0) <= 3 && abs(cy - fm1) <= 3 && cx >= bmin0 && cx <= bmax0 && cy >= bmin1 && cy <= bmax1;
            uint32_t s = ok ? qpel_sad(sv, (cx >> 2) - best0 + 1, (cy >> 2) - best1 + 1, cx & 3, cy & 3) : 0u;
            s = wsum(s);
            cc[k] = ok ? s + mvd_cost(cx - mvp0, lambda) + mvd_cost(cy - mvp1, lambda) : UMAX;
          }
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (cc[k] < bc) { bc = cc[k]; q0 = f0 + dd[k][0]; q1 = f1 + dd[k][1]; }
          if (q0 == f0 && q1 == f1) break;
        }
      }
      mv0 = q0; mv1 = q1;
      uint2 v = qpel8(qpel_src((q0 >> 2) - best0 + 1, (q1 >> 2) - best1 + 1, q0 & 3, q1 & 3));
      *(uint2*)&sm.pred_y[(lane >> 1) * 16 + (lane & 1) * 8] = v;
      __syncwarp();
    }
  }

  // 3. intra 16x16 when the inter prediction is poor (enc.rs:3121-3156)
  const uint32_t inter_satd = satd16((int)offsetof(Smem, pred_y));
  uint32_t inter_cost = inter_satd + lambda * (se_bits(mv0 - mvp0) + se_bits(mv1 - mvp1) + 1);
  if (inter_satd > 24 * lambda) {
    const Corner k0 = load_edges(c, false);
    bool ht = mby > 0, hl = mbx > 0;
    const I16Fit fit16 = analyse_i16(ht, hl, k0.y);
    if (fit16.cost + lambda * 8 < inter_cost) {
      code_i16(c, fit16.mode, ht, hl, k0);
      return true;
    }
  }

  // 4. P_L0_16x16 residual, record and reconstruction
  mc_chroma8(sd.ref_u, sd.ref_v, fp.stride_c, mbx, mby, mv0, mv1);
  code_inter(c, RG_MB_P_L0_16X16, mv0 == ps0 && mv1 == ps1, mv0, mv1, mv0 - mvp0, mv1 - mvp1);
  return true;
}

// ---------------------------------------------------------------------------------------------
// The full-search and learned forms' analysis (neither exists in the reference).
#include "search_form.cuh"

// ---------------------------------------------------------------------------------------------
// Deblocking of one macroblock (enc.rs:3776 deblock, h264_deblock.rs:71,187): vertical edges
// then horizontal ones, on a shared-memory tile with 4 samples of the left / top neighbours.
struct EdgeParams {
  int alpha, beta, tc0[4];
  bool strong, on;
};
__device__ __forceinline__ EdgeParams edge_params(int qp, const int* bs) {
  EdgeParams e;
  int ia = qp < 0 ? 0 : (qp > 51 ? 51 : qp);
  e.alpha = c_alpha[ia];
  e.beta = c_beta[ia];
  e.on = e.alpha != 0 && e.beta != 0;
  for (int k = 0; k < 4; k++) {
    int b = bs[k] > 4 ? 4 : bs[k];
    e.tc0[k] = b == 0 ? -1 : (b == 4 ? 0 : c_tc0[ia][b - 1]);
  }
  e.strong = bs[0] == 4;
  return e;
}
__device__ __forceinline__ void luma_line(uint8_t* o, int xs, const EdgeParams& e, int tc0) {
  if (!e.strong && tc0 < 0) return;
  int p0 = o[-xs], q0 = o[0], p1 = o[-2 * xs], q1 = o[xs];
  if (abs(p0 - q0) >= e.alpha || abs(p1 - p0) >= e.beta || abs(q1 - q0) >= e.beta) return;
  int p2 = o[-3 * xs], q2 = o[2 * xs];
  bool ap = abs(p2 - p0) < e.beta, aq = abs(q2 - q0) < e.beta;
  if (!e.strong) {
    int tc = tc0 + ap + aq;
    int d = min(max((((q0 - p0) << 2) + (p1 - q1) + 4) >> 3, -tc), tc);
    o[-xs] = (uint8_t)clip255(p0 + d);
    o[0] = (uint8_t)clip255(q0 - d);
    if (ap) o[-2 * xs] = (uint8_t)(p1 + min(max((p2 + ((p0 + q0 + 1) >> 1) - (p1 << 1)) >> 1, -tc0), tc0));
    if (aq) o[xs] = (uint8_t)(q1 + min(max((q2 + ((p0 + q0 + 1) >> 1) - (q1 << 1)) >> 1, -tc0), tc0));
  } else {
    int p3 = o[-4 * xs], q3 = o[3 * xs];
    bool small = abs(p0 - q0) < ((e.alpha >> 2) + 2);
    if (ap && small) {
      o[-xs] = (uint8_t)((p2 + 2 * p1 + 2 * p0 + 2 * q0 + q1 + 4) >> 3);
      o[-2 * xs] = (uint8_t)((p2 + p1 + p0 + q0 + 2) >> 2);
      o[-3 * xs] = (uint8_t)((2 * p3 + 3 * p2 + p1 + p0 + q0 + 4) >> 3);
    } else {
      o[-xs] = (uint8_t)((2 * p1 + p0 + q1 + 2) >> 2);
    }
    if (aq && small) {
      o[0] = (uint8_t)((p1 + 2 * p0 + 2 * q0 + 2 * q1 + q2 + 4) >> 3);
      o[xs] = (uint8_t)((p0 + q0 + q1 + q2 + 2) >> 2);
      o[2 * xs] = (uint8_t)((2 * q3 + 3 * q2 + q1 + q0 + p0 + 4) >> 3);
    } else {
      o[0] = (uint8_t)((2 * q1 + q0 + p1 + 2) >> 2);
    }
  }
}
__device__ __forceinline__ void chroma_line(uint8_t* o, int xs, const EdgeParams& e, int tc0) {
  if (!e.strong && tc0 < 0) return;
  int p1 = o[-2 * xs], p0 = o[-xs], q0 = o[0], q1 = o[xs];
  if (abs(p0 - q0) >= e.alpha || abs(p1 - p0) >= e.beta || abs(q1 - q0) >= e.beta) return;
  if (e.strong) {
    o[-xs] = (uint8_t)((2 * p1 + p0 + q1 + 2) >> 2);
    o[0] = (uint8_t)((2 * q1 + q0 + p1 + 2) >> 2);
  } else {
    int tc = tc0 + 1;
    int d = min(max((((q0 - p0) << 2) + (p1 - q1) + 4) >> 3, -tc), tc);
    o[-xs] = (uint8_t)clip255(p0 + d);
    o[0] = (uint8_t)clip255(q0 - d);
  }
}
__device__ __forceinline__ int nz_at(uint16_t nz, int bx, int by) {
  int b = ((by >> 1) << 3) | ((bx >> 1) << 2) | ((by & 1) << 1) | (bx & 1);
  return (nz >> b) & 1;
}
// Boundary strengths of edge e in direction dir (0 vertical); returns false to skip the edge.
// kMv4 (search forms): the motion term compares the quadrant vectors on either side of each
// 4-sample segment (qm: this macroblock's, pm4: the neighbour's across edge 0), so the internal
// edge between partitions gets strength 1 where their vectors differ by 4 quarter samples.
template <bool kMv4>
__device__ bool edge_bs(const MbInfo& q, const MbInfo* p, int dir, int e, int* bs, const MbMv4* qm, const MbMv4* pm4) {
  bool qi = q.flags & kFlagIntra;
  bool pi = p ? (p->flags & kFlagIntra) : qi;
  if (qi || pi) {
    for (int k = 0; k < 4; k++) bs[k] = e == 0 ? 4 : 3;
    return true;
  }
  int coded[4];
  for (int k = 0; k < 4; k++) {
    if (dir == 0) coded[k] = nz_at(q.nz16, e, k) | (e == 0 ? nz_at(p->nz16, 3, k) : nz_at(q.nz16, e - 1, k));
    else coded[k] = nz_at(q.nz16, k, e) | (e == 0 ? nz_at(p->nz16, k, 3) : nz_at(q.nz16, k, e - 1));
  }
  if constexpr (!kMv4) {
    bool motion = false;
    if (e == 0) motion = q.ref != p->ref || abs(q.mv[0] - p->mv[0]) >= 4 || abs(q.mv[1] - p->mv[1]) >= 4;
    if (!coded[0] && !coded[1] && !coded[2] && !coded[3] && !motion) return false;
    for (int k = 0; k < 4; k++) bs[k] = coded[k] ? 2 : (motion ? 1 : 0);
    return true;
  } else {
    bool any = false;
    for (int k = 0; k < 4; k++) {
      int qq = dir == 0 ? (k >> 1) * 2 + (e >> 1) : (e >> 1) * 2 + (k >> 1);
      int pq = e == 0 ? (dir == 0 ? (k >> 1) * 2 + 1 : 2 + (k >> 1))
                      : (dir == 0 ? (k >> 1) * 2 + ((e - 1) >> 1) : ((e - 1) >> 1) * 2 + (k >> 1));
      const MbMv4* pmm = e == 0 ? pm4 : qm;
      bool motion = (e == 0 && q.ref != p->ref) || abs(qm->mv[qq][0] - pmm->mv[pq][0]) >= 4 ||
                    abs(qm->mv[qq][1] - pmm->mv[pq][1]) >= 4;
      bs[k] = coded[k] ? 2 : (motion ? 1 : 0);
      any |= bs[k] != 0;
    }
    return any;
  }
}
// Whether a search-form macroblock's quadrants share one vector.
__device__ __forceinline__ bool one_vector(const MbMv4& m) {
  const uint32_t* w = (const uint32_t*)&m;
  return w[0] == w[1] && w[0] == w[2] && w[0] == w[3];
}

template <bool kMv4>
__device__ __noinline__ void deblock_mb(int mbx, int mby) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  int lane = lane_id();
  int m = mby * fp.mb_w + mbx;
  MbInfo q = ld_info(&sd.info[m]);
  MbInfo lf, tp;
  bool hasl = mbx > 0, hast = mby > 0;
  if (hasl) lf = ld_info(&sd.info[m - 1]);
  if (hast) tp = ld_info(&sd.info[m - fp.mb_w]);
  auto quiet = [](const MbInfo& i) { return !(i.flags & kFlagIntra) && i.cbp_luma == 0; };
  MbMv4 qm, lm, tm;
  bool split = false;
  if constexpr (kMv4) {
    qm = sd.mv4[m];
    if (hasl) lm = sd.mv4[m - 1];
    if (hast) tm = sd.mv4[m - fp.mb_w];
    split = !one_vector(qm);
    const uint32_t qv = *(const uint32_t*)&qm;
    if (quiet(q) && !split && (!hasl || (quiet(lf) && one_vector(lm) && *(const uint32_t*)&lm == qv)) &&
        (!hast || (quiet(tp) && one_vector(tm) && *(const uint32_t*)&tm == qv)))
      return;
  } else {
    if (quiet(q) && (!hasl || (quiet(lf) && lf.mv[0] == q.mv[0] && lf.mv[1] == q.mv[1])) &&
        (!hast || (quiet(tp) && tp.mv[0] == q.mv[0] && tp.mv[1] == q.mv[1])))
      return;
  }
  // tiles: luma 20x20 at (x0-4, y0-4) stride 20 in win; chroma 12x12 each in hph / hpv
  uint8_t* ty = sm.win;
  auto tc = [](int p) { return sm.hph + p * (int)(offsetof(Smem, hpv) - offsetof(Smem, hph)); };
  const int x0 = mbx * 16, y0 = mby * 16, cx0 = mbx * 8, cy0 = mby * 8;
  for (int w = lane; w < 100; w += 32) {  // 20 rows x 5 words
    int r = w / 5, k = w % 5;
    if ((r < 4 && !hast) || (k == 0 && !hasl)) continue;
    *(uint32_t*)&ty[r * 20 + 4 * k] = ldcg_u32(sd.cur_y + (long)(y0 - 4 + r) * fp.stride_y + x0 - 4 + 4 * k);
  }
  for (int w = lane; w < 72; w += 32) {  // 2 planes x 12 rows x 3 words
    int p = w / 36, rem = w % 36, r = rem / 3, k = rem % 3;
    if ((r < 4 && !hast) || (k == 0 && !hasl)) continue;
    const uint8_t* P = p ? sd.cur_v : sd.cur_u;
    *(uint32_t*)&tc(p)[r * 12 + 4 * k] = ldcg_u32(P + (long)(cy0 - 4 + r) * fp.stride_c + cx0 - 4 + 4 * k);
  }
  __syncwarp();
  bool intra = q.flags & kFlagIntra;
  bool internal = intra || q.cbp_luma != 0 || split;
  bool skip_odd = q.flags & kFlagT8;
  int qpq = q.qp, qpcq = chroma_qp(qpq);
  for (int dir = 0; dir < 2; dir++) {
    for (int e = 0; e < 4; e++) {
      const MbInfo* pm;
      if (e == 0) {
        if (dir == 0 ? !hasl : !hast) continue;
        pm = dir == 0 ? &lf : &tp;
      } else {
        if (!internal || ((e & 1) && skip_odd)) continue;
        pm = nullptr;
      }
      int bs[4];
      if (!edge_bs<kMv4>(q, pm ? pm : &q, dir, e, bs, &qm, dir == 0 ? &lm : &tm)) continue;
      int qpl, qpc;
      if (!pm) { qpl = qpq; qpc = qpcq; }
      else { qpl = (qpq + pm->qp + 1) >> 1; qpc = (qpcq + chroma_qp(pm->qp) + 1) >> 1; }
      EdgeParams el = edge_params(qpl, bs);
      if (lane < 16 && el.on) {
        if (dir == 0) luma_line(&ty[(4 + lane) * 20 + 4 + e * 4], 1, el, el.tc0[lane >> 2]);
        else luma_line(&ty[(4 + e * 4) * 20 + 4 + lane], 20, el, el.tc0[lane >> 2]);
      }
      if (!(e & 1) && lane >= 16) {
        EdgeParams ec = edge_params(qpc, bs);
        if (ec.on) {
          int j = lane - 16, p = j >> 3, k = j & 7;
          if (dir == 0) chroma_line(&tc(p)[(4 + k) * 12 + 4 + e * 2], 1, ec, ec.tc0[k >> 1]);
          else chroma_line(&tc(p)[(4 + e * 2) * 12 + 4 + k], 12, ec, ec.tc0[k >> 1]);
        }
      }
      __syncwarp();
    }
  }
  // write back the samples this macroblock filters (rows 0..15 x cols -4..15, rows -4..-1 x cols 0..15)
  for (int w = lane; w < 100; w += 32) {
    int r = w / 5, k = w % 5;
    if (r < 4 && k == 0) continue;
    if ((r < 4 && !hast) || (k == 0 && !hasl)) continue;
    *(uint32_t*)(sd.cur_y + (long)(y0 - 4 + r) * fp.stride_y + x0 - 4 + 4 * k) = *(const uint32_t*)&ty[r * 20 + 4 * k];
  }
  for (int w = lane; w < 72; w += 32) {
    int p = w / 36, rem = w % 36, r = rem / 3, k = rem % 3;
    if (r < 4 && k == 0) continue;
    if ((r < 4 && !hast) || (k == 0 && !hasl)) continue;
    uint8_t* P = p ? sd.cur_v : sd.cur_u;
    *(uint32_t*)(P + (long)(cy0 - 4 + r) * fp.stride_c + cx0 - 4 + 4 * k) = *(const uint32_t*)&tc(p)[r * 12 + 4 * k];
  }
}

// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int diag_first(const FrameParams& fp, int d) {
  int a = d - fp.mb_w + 1;
  return a > 0 ? (a + 1) >> 1 : 0;
}
__device__ __forceinline__ int diag_len(const FrameParams& fp, int d) {
  if (d < 0) return 0;
  int lo = diag_first(fp, d), hi = min(fp.mb_h - 1, d >> 1);
  return hi >= lo ? hi - lo + 1 : 0;
}

template <int kForm>
__global__ void __launch_bounds__(32) wavefront_step_kernel(const __grid_constant__ FrameParams fp, const StreamDev* __restrict__ streams, int step) {
  init_tables();
  load_params(fp);
  load_desc(streams + blockIdx.y);
  const StreamDev& sd = sm.sd;
  int na = diag_len(fp, step);
  int nd = fp.deblock ? diag_len(fp, step - 3) : 0;
  int k = blockIdx.x;
  if (k < na) {
    int mby = diag_first(fp, step) + k, mbx = step - 2 * mby;
    Ctx c{mbx, mby, mby * fp.mb_w + mbx};
    const PipeWait none{nullptr, nullptr, 0};
    if (sd.kind == RG_FRAME_IDR) {
      load_source(c);
      if constexpr (kForm != 0) analyse_intra_mb_search(c);
      else analyse_intra_mb(c);
    } else {
      if constexpr (kForm != 0) analyse_p_mb_search(c, none);
      else analyse_p_mb(c, none);
    }
  } else if (k - na < nd) {
    int d = step - 3;
    int mby = diag_first(fp, d) + (k - na), mbx = d - 2 * mby;
    deblock_mb<kForm != 0>(mbx, mby);
  }
}

// Border extension (enc.rs:165 extend_borders) of the padding that takes its values from
// macroblock (a, b), once that macroblock is final: the left / right padding of its rows when it
// is the first / last of its row, and the padding above / below its columns when it is in the
// first / last row -- corners included, which come from the corner macroblocks. Applied to every
// macroblock of the picture this writes every padding sample exactly once, so a picture's
// padding is complete wherever the macroblocks it copies are final. One warp, 4-byte stores.
__device__ __noinline__ void extend_mb(int a, int b) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  int lane = lane_id();
  bool left = a == 0, right = a == fp.mb_w - 1, top = b == 0, bottom = b == fp.mb_h - 1;
  if (!(left || right || top || bottom)) return;
  for (int plane = 0; plane < 3; plane++) {
    uint8_t* P = plane == 0 ? sd.cur_y : (plane == 1 ? sd.cur_u : sd.cur_v);
    int bw = plane ? 8 : 16;
    int w = fp.mb_w * bw, h = fp.mb_h * bw;
    int pad = plane ? kPadC : kPadY, stride = plane ? fp.stride_c : fp.stride_y;
    int lw = pad / 4;
    // columns owned by this macroblock, in 4-byte words relative to the padded row start
    int c_lo = left ? 0 : (pad + a * bw) / 4;
    int c_hi = right ? stride / 4 : (pad + (a + 1) * bw) / 4;
    // rows owned: its own rows, plus the padding above / below the picture
    int r_lo = top ? -pad : b * bw, r_hi = bottom ? h + pad : (b + 1) * bw;
    int ncol = c_hi - c_lo, n = (r_hi - r_lo) * ncol;
    for (int i = lane; i < n; i += 32) {
      int yy = r_lo + i / ncol, cw = c_lo + i % ncol;
      int xw = cw * 4 - pad;  // first picture column of this word
      bool in_rows = yy >= 0 && yy < h;
      if (in_rows && cw >= lw && cw < lw + w / 4) continue;  // picture sample: no copy
      int sy = min(max(yy, 0), h - 1);
      const uint8_t* srow = P + (long)sy * stride;
      uint32_t v;
      if (xw < 0) v = ldcg_u8(srow) * 0x01010101u;
      else if (xw >= w) v = ldcg_u8(srow + w - 1) * 0x01010101u;
      else v = ldcg_u32(srow + xw);
      *(uint32_t*)(P + (long)yy * stride + xw) = v;
    }
  }
}

// Persistent pipelined mode: F pictures of every stream in one launch. The work is cut into
// segments of `seg` consecutive macroblocks of one row -- analysis segments and deblocking
// segments -- listed by the host in the order they are expected to become ready (pipeline_task_
// list) and handed out by an atomic ticket. A warp only holds one short segment, so the resident
// warps cover the work that is about to be ready rather than whole rows far from it, and every
// wait is normally for a segment of a smaller ticket. Picture f+1 of a stream starts as soon as
// the part of picture f its search can reach is deblocked and border-extended.
struct PipeParams {
  int* ticket;
  int* error;
  int* ana;    // analysed macroblocks per row, descriptor d's rows from ana + d.rows_base
  int* db;     // deblocked macroblocks per row (the same layout); a macroblock's deblocking also
               // extends the padding of the macroblocks it makes final
  const int2* tasks;  // {descriptor, row << 16 | first macroblock << 1 | deblock}
  int n_tasks;
  int qbeg[3], qend[3];  // queue q = tasks[qbeg[q], qend[q]): 0 analysis, 1 deblocking, 2 IDR analysis
  int deblock_sms;    // SMs whose warps take queue 1 first
  int intra_sms;      // the next SMs, whose warps take queue 2 first
  int role_by_sm;     // 0: by block index instead (a grid too small to reach every SM)
  int seg;
  unsigned long long timeout_ns;
  int* rows_done;     // [descriptor] rows of a picture fully analysed
  int* ready;         // [descriptor] in mapped host memory (or null): seq once a picture's records are final
  int seq;
  int* host_err;      // mapped host memory: the error word as the launch ends (no copy to wait for)
  int* reach;         // [2] 1 + the largest reach of a reference wait beyond zero motion (rows, columns)
  // compact records (cwords null: none): row r of the launch (rows like ana) has a slot of crow
  // words at cwords + r * crow in mapped host memory and its size in bytes (or -1) at cbytes[r]
  uint32_t* cwords;
  int crow;
  int* cbytes;
};
__device__ __forceinline__ unsigned sm_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}

// Counts a picture's fully analysed row; the warp completing its last row tells the host that the
// picture's records are final. Each row's records were ordered before its count by the release
// chain of the row's segments; the acq_rel count gathers all rows, and the system-scope release
// store orders them before the flag the host polls.
__device__ __noinline__ void picture_row_done(int* rows_done, int* ready, int seq, int H) {
  if (lane_id() == 0) {
    int before = atom_add_acq_rel(rows_done, 1);
    if (before == H - 1) st_release_sys(ready, seq);
  }
  __syncwarp();
}

static_assert(sizeof(rg_mb_out) == 4 * kRecordWords, "a record is kRecordWords words");
// Staging of compact records in the warp's shared memory (the front of its Smem, which no task reads
// before writing it): kStageWords words, flushed to host memory in 16-byte stores.
constexpr int kStageWords = 512;
static_assert(offsetof(Smem, coef) >= 4 * kStageWords && offsetof(Smem, zz8) > offsetof(Smem, coef) &&
                  offsetof(Smem, sd) > offsetof(Smem, coef),
              "the staging buffer ends before what a warp keeps between macroblocks");
static_assert(kStageWords >= 2 * (kCompactMaskWords + kRecordWords), "a flush leaves room for a whole record");

// Writes the first n (a multiple of 4) staged words to dst + at (16-byte aligned) while they fit
// the slot of cap words (a multiple of 4), then moves the rest (< 4 words) to the front.
__device__ __noinline__ void flush_stage(uint32_t* stage, int n, int rest, uint32_t* dst, long long at, int cap) {
  const int lane = lane_id();
  __syncwarp();
  const uint4* s4 = reinterpret_cast<const uint4*>(stage);
  uint4* d4 = reinterpret_cast<uint4*>(dst + at);
  for (int c = lane; c < n / 4; c += 32)
    if (at + 4 * c + 4 <= cap) d4[c] = s4[c];
  __syncwarp();
  uint32_t v = lane < rest ? stage[n + lane] : 0u;
  __syncwarp();
  if (lane < rest) stage[lane] = v;
  __syncwarp();
}

// Compact records of row y, written by the warp that deblocked the row's last segment (after it
// published its progress) into the row's own slot (no row waits for another). A record's compact form is kCompactMaskWords mask words (bit j of
// mask word i: record word 32 i + j is nonzero), then its nonzero words in increasing order:
// zero-filling rebuilds the record exactly. The row's records are final: the deblocking warp
// acquired the row's analysis progress up to its end; they are read through L2. The
// words are gathered in shared memory and leave in whole 16-byte stores (word-sized stores to
// host memory made the row ~10x slower). Words past the slot are not written, and the row's size
// is then -1 (the host copies the picture's full records instead). The size is written before the
// row is counted towards the picture's flag. (Scalar arguments: a reference to the kernel's
// parameters would copy them to local memory.)
__device__ __noinline__ void compact_row(const rg_mb_out* rec, uint32_t* dst, int cap, int* bytes, int Wm,
                                         uint32_t* stage) {
  const int lane = lane_id();
  long long done = 0;  // words flushed (a multiple of 4)
  int sp = 0;          // words staged
  const uint32_t* src = reinterpret_cast<const uint32_t*>(rec);
  const unsigned below = (1u << lane) - 1u;
  for (int m0 = 0; m0 < Wm; m0 += 4) {
    // four records in flight, then their words into the stage
    uint32_t w[4][kCompactMaskWords];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int i = 0; i < kCompactMaskWords; i++) {
        const int j = lane + 32 * i;
        w[k][i] = (m0 + k < Wm && j < kRecordWords) ? __ldcg(src + (size_t)(m0 + k) * kRecordWords + j) : 0u;
      }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (m0 + k >= Wm) break;
      if (sp + kCompactMaskWords + kRecordWords > kStageWords) {
        const int n = sp & ~3;
        flush_stage(stage, n, sp - n, dst, done, cap);
        done += n;
        sp -= n;
      }
      uint32_t mask = 0;
      int at = sp + kCompactMaskWords;
#pragma unroll
      for (int i = 0; i < kCompactMaskWords; i++) {
        const unsigned b = __ballot_sync(FULL, w[k][i] != 0u);
        if (lane == i) mask = b;
        if (w[k][i] != 0u) stage[at + __popc(b & below)] = w[k][i];
        at += __popc(b);
      }
      if (lane < kCompactMaskWords) stage[sp + lane] = mask;
      sp = at;
    }
  }
  // the tail, padded to whole 16-byte stores (the padding stays inside the slot: cap is a
  // multiple of 4 and the row's words, when they fit, are at most cap)
  const long long total = done + sp;
  flush_stage(stage, (sp + 3) & ~3, 0, dst, done, cap);
  if (lane == 0) *bytes = total <= cap ? (int)(total * 4) : -1;
  // the row's words and size reach host memory before the row is counted towards the flag
  __threadfence_system();
  __syncwarp();
}

// At least 16 warps per SM: up to 128 registers a thread, so nothing spills (4.5 % faster than 20,
// which held it to 96 registers with spills).
template <int kForm>
__global__ void __launch_bounds__(32, 16) pipeline_kernel(const __grid_constant__ FrameGroups fg, const StreamDev* __restrict__ sds, PipeParams pp) {
  const int lane = lane_id();
  // Warps on the first deblock_sms SMs take deblocking segments first, on the next intra_sms SMs
  // segments of IDR pictures (the critical path of a GOP), and the others the remaining analysis
  // (each SM then runs a smaller code footprint); a warp whose queue is empty takes from the next.
  int role = 0;
  if (pp.role_by_sm) {
    int id = (int)sm_id();
    role = id < pp.deblock_sms ? 1 : (id < pp.deblock_sms + pp.intra_sms ? 2 : 0);
  } else {
    int k = blockIdx.x % 9;
    role = k == 0 ? 1 : (k == 1 ? 2 : 0);
  }
  init_tables();
  bool empty[3] = {pp.qbeg[0] >= pp.qend[0], pp.qbeg[1] >= pp.qend[1], pp.qbeg[2] >= pp.qend[2]};
  if (lane == 0) sm.reach_y = sm.reach_x = 0;  // this warp's, published once as it exits
  int group = -1;                              // whose parameters sm.fp holds
  while (true) {
    int t = -1;
    if (lane == 0) {
      for (int k = 0; k < 3 && t < 0; k++) {
        int q = role + k >= 3 ? role + k - 3 : role + k;
        if (empty[q]) continue;
        int v = pp.qbeg[q] + atomicAdd(pp.ticket + (q ? q + 1 : 0), 1);
        if (v < pp.qend[q]) t = v; else empty[q] = true;
      }
    }
    t = __shfl_sync(FULL, t, 0);
    if (t < 0) break;
    if (__shfl_sync(FULL, lane == 0 ? ld_relaxed(pp.error) : 0, 0)) break;
    int2 task = __ldg(pp.tasks + t);
    int ps = task.x;
    load_desc(sds + ps);
    const StreamDev& sd = sm.sd;
    if (sd.group != group) {  // the descriptor's picture size
      group = sd.group;
      load_params(fg.g[group]);
    }
    const int H = sm.fp.mb_h, Wm = sm.fp.mb_w;
    const int y = task.y >> 16, x0 = (task.y >> 1) & 0x7fff, x1 = min(x0 + pp.seg, Wm);
    const bool ana = (task.y & 1) == 0;
    int* ana_rows = pp.ana + sd.rows_base;
    int* db_rows = pp.db + sd.rows_base;
    bool failed = false;
    int seen = 0;  // of this lane's counter (wait_all)
    if (ana) {
      const bool has_prev = sd.prev_rows >= 0 && sd.kind == RG_FRAME_P;
      const PipeWait pw{has_prev ? pp.db + sd.prev_rows : nullptr, pp.error, pp.timeout_ns};
      if (lane == 0) sm.db_row = -1;
      // lane 0: the previous segment of this row; lane 1: the row above two macroblocks ahead; lane 2
      // (plain form): the co-located macroblock of the previous picture, whose vector is a candidate
      const int* flag = lane == 0 && x0 > 0 ? ana_rows + y : nullptr;
      if (lane == 1 && y > 0) flag = ana_rows + y - 1;
      if (kForm == 0 && lane == 2 && has_prev) flag = pp.ana + sd.prev_rows + y;
      for (int x = x0; x < x1; x++) {
        if (!wait_all(flag, lane == 0 ? x0 : (lane == 1 ? min(x + 2, Wm) : x + 1), seen, pp.error, pp.timeout_ns)) {
          failed = true;
          break;
        }
        Ctx c{x, y, y * Wm + x};
        if (sd.kind == RG_FRAME_IDR) {
          load_source(c);
          if constexpr (kForm != 0) analyse_intra_mb_search(c);
          else analyse_intra_mb(c);
        } else {
          if constexpr (kForm != 0) failed = !analyse_p_mb_search(c, pw);
          else failed = !analyse_p_mb(c, pw);
          if (failed) break;
        }
        publish(ana_rows + y, x + 1);
      }
      // (with compact records, the row is counted once its deblocking warp has compacted it)
      int* const rdy = sd.ready ? sd.ready : (pp.ready ? pp.ready + ps : nullptr);
      if (!failed && x1 == Wm && rdy && !pp.cwords) picture_row_done(pp.rows_done + ps, rdy, pp.seq, H);
    } else {
      // lane 0: the analysis of this row one macroblock further; lane 1: of the row below; lane 2: the
      // deblocking of the row above one further; lane 3: the previous segment of this row
      const int* flag = lane == 0 ? ana_rows + y : nullptr;
      if (lane == 1 && y + 1 < H) flag = ana_rows + y + 1;
      if (lane == 2 && y > 0) flag = db_rows + y - 1;
      if (lane == 3 && x0 > 0) flag = db_rows + y;
      for (int x = x0; x < x1; x++) {
        if (!wait_all(flag, lane == 3 ? x0 : min(x + (lane == 1 ? 1 : 2), Wm), seen, pp.error, pp.timeout_ns)) {
          failed = true;
          break;
        }
        deblock_mb<kForm != 0>(x, y);
        // Macroblock (x, y - 1) is final now: (x + 1, y - 1) was deblocked before this one. In
        // the last row, so is (x - 1, y), and the last macroblock is final after its own pass.
        __syncwarp();
        if (y >= 1) extend_mb(x, y - 1);
        if (y == H - 1) {
          if (x >= 1) extend_mb(x - 1, y);
          if (x == Wm - 1) extend_mb(x, y);
        }
        publish(db_rows + y, x + 1);
      }
      // Compact records of the row, by the warp that deblocked its last segment: on the deblocking
      // SMs and after the row's deblocking progress was published, so neither the analysis
      // wavefront nor the deblocking chain waits for it (done at the end of the row's analysis it
      // slowed the launch ~5 %). Its wait for the analysis of the row up to its end ordered every
      // record of the row before it.
      if (!failed && x1 == Wm && pp.cwords) {
        const long long r = (long long)sd.rows_base + y;
        compact_row(sd.rec + (size_t)y * Wm, pp.cwords + r * pp.crow, pp.crow, pp.cbytes + r, Wm,
                    reinterpret_cast<uint32_t*>(&sm));
        int* const rdy = sd.ready ? sd.ready : (pp.ready ? pp.ready + ps : nullptr);
        if (rdy) picture_row_done(pp.rows_done + ps, rdy, pp.seq, H);
      }
    }
    if (failed) break;
  }
  if (lane == 0 && sm.reach_y) {
    atomicMax(pp.reach, sm.reach_y);
    atomicMax(pp.reach + 1, sm.reach_x);
  }
}

// The launch's error word (and the reach its reference waits saw) into mapped host memory, queued
// after the launch (a kernel, not a copy: a device-to-host copy waiting for a launch would stall
// later copies of the context).
__global__ void error_to_host_kernel(const int* error, const int* reach, int* host_err, int* host_reach) {
  if (host_reach) {
    host_reach[0] = reach[0];
    host_reach[1] = reach[1];
  }
  st_release_sys(host_err, *error);
}

// Border extension (enc.rs:165 extend_borders): every padding sample takes the value of the
// nearest picture sample. One thread per 16-byte chunk of a padded row.
__global__ void extend_borders_kernel(FrameParams fp, const StreamDev* __restrict__ streams) {
  const StreamDev& sd = streams[blockIdx.z / 3];
  int plane = blockIdx.z % 3;
  int w = plane ? fp.mb_w * 8 : fp.mb_w * 16, h = plane ? fp.mb_h * 8 : fp.mb_h * 16;
  int pad = plane ? kPadC : kPadY, stride = plane ? fp.stride_c : fp.stride_y;
  uint8_t* P = plane == 0 ? sd.cur_y : (plane == 1 ? sd.cur_u : sd.cur_v);
  int chunks = stride / 16;
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  int rows = h + 2 * pad;
  if (idx >= rows * chunks) return;
  int ry = idx / chunks, cx = (idx % chunks) * 16;  // padded coordinates
  int y = ry - pad;
  int xs = cx - pad;
  bool row_inside = y >= 0 && y < h;
  if (row_inside && xs >= 0 && xs + 16 <= w) return;  // all interior
  int sy = min(max(y, 0), h - 1);
  const uint8_t* srow = P + (long)sy * stride;
  uint8_t* drow = P + (long)y * stride;
  for (int k = 0; k < 16; k++) {
    int x = xs + k;
    if (row_inside && x >= 0 && x < w) continue;
    drow[x] = srow[min(max(x, 0), w - 1)];
  }
}

}  // namespace

void upload_tables() {
  using namespace tables;
  cudaMemcpyToSymbol(c_lambda, kLambda, sizeof(kLambda));
  cudaMemcpyToSymbol(c_dec4, kDecimate4, sizeof(kDecimate4));
  uint8_t d8[64] = {0};
  for (int i = 0; i < 24; i++) d8[i] = kDecimate8[i];
  cudaMemcpyToSymbol(c_dec8, d8, sizeof(d8));
  cudaMemcpyToSymbol(c_scan4, kScan4, sizeof(kScan4));
  cudaMemcpyToSymbol(c_scan8, kScan8, sizeof(kScan8));
  cudaMemcpyToSymbol(c_mf4, kMf4, sizeof(kMf4));
  cudaMemcpyToSymbol(c_dq4, kDq4, sizeof(kDq4));
  cudaMemcpyToSymbol(c_mf8, kMf8, sizeof(kMf8));
  cudaMemcpyToSymbol(c_dq8, kDq8, sizeof(kDq8));
  cudaMemcpyToSymbol(c_cqp, kChromaQp, sizeof(kChromaQp));
  cudaMemcpyToSymbol(c_alpha, kAlpha, sizeof(kAlpha));
  cudaMemcpyToSymbol(c_beta, kBeta, sizeof(kBeta));
  cudaMemcpyToSymbol(c_tc0, kTc0, sizeof(kTc0));
  uint16_t taps[9 * 16];
  for (int m = 0; m < 9; m++)
    for (int q = 0; q < 16; q++) {
      int t = i4_tap(m, q & 3, q >> 2), i = t & 0xff;
      taps[m * 16 + q] = (uint16_t)(i | (i + 1 < 15 ? i + 1 : 15) << 4 | (i + 2 < 15 ? i + 2 : 15) << 8 | (t >> 8) << 12);
    }
  cudaMemcpyToSymbol(g_i4tap, taps, sizeof(taps));
}

int wavefront_steps(const FrameParams& fp) {
  int diags = (fp.mb_w - 1) + 2 * (fp.mb_h - 1) + 1;
  return diags + (fp.deblock ? 3 : 0);
}

static int max_diag_len(const FrameParams& fp) {
  int best = 0;
  int diags = (fp.mb_w - 1) + 2 * (fp.mb_h - 1) + 1;
  for (int d = 0; d < diags; d++) {
    int a = d - fp.mb_w + 1;
    int lo = a > 0 ? (a + 1) >> 1 : 0, hi = fp.mb_h - 1 < (d >> 1) ? fp.mb_h - 1 : (d >> 1);
    if (hi - lo + 1 > best) best = hi - lo + 1;
  }
  return best;
}

void launch_wavefront_step(const FrameParams& fp, const StreamDev* d_streams, int step, cudaStream_t st, int form) {
  dim3 grid(2 * max_diag_len(fp), fp.n_streams);
  if (form) wavefront_step_kernel<1><<<grid, 32, 0, st>>>(fp, d_streams, step);
  else wavefront_step_kernel<0><<<grid, 32, 0, st>>>(fp, d_streams, step);
}

int pipeline_sms(int device) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

// Resident warps of the pipelined mode: sixteen per SM (fewer when they do not fit). More warps
// overlap more of each other's waits, until the SM's front end saturates and every macroblock on
// the critical path slows (measured on B200, 1080p 8 x 15 pictures, launch time: 7 per SM
// 62.9 ms, 8 61.0, 10 59.1, 12 57.4, 14 56.0, 16 55.8, 18 56.2, 20-21 56.3).
int pipeline_grid(int device, int form) {
  int per_sm = 0;
  if (form) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pipeline_kernel<1>, 32, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pipeline_kernel<0>, 32, 0);
  return (per_sm < 16 ? per_sm : 16) * pipeline_sms(device);
}

// Work list of the pipelined mode, written to `tasks` (pipeline_task_count entries): every
// analysis and deblocking segment of every picture and stream, ordered by a key of the
// macroblock-time it can start -- a = max(seg, 2) per row, 1 per column, lag per picture:
//   analysis of row y from column x0:    a * y + x0 + lag * f
//   deblocking of row y from column x0:  a * (y + 1) + x0 + 1 + lag * f
// and, at equal keys, by picture, role (analysis first), stream and row. Every macroblock of a
// segment depends only on segments of a smaller key or of an equal key earlier in that order
// (the row above two macroblocks ahead lies in a segment of key <= a * (y - 1) + x0 + seg; the
// deblocking of (x, y) needs the analysis of (x + 1, y) and (x, y + 1) and the deblocking of
// (x + 1, y - 1)), so warps taking tickets in order never wait for an untaken segment of the same
// picture. The wait for the reference picture depends on the motion vectors: a search whose
// window reaches r macroblocks beyond the co-located ones (r = 0 for zero motion) waits for a
// smaller key when lag >= a * (4 + r) + seg + r + 3. lag <= 0 takes r = 4 (about 64 samples).
size_t pipeline_task_count(const FrameParams& fp, int frames, int seg) {
  size_t segs = (size_t)(fp.mb_w + seg - 1) / seg;
  return 2 * (size_t)frames * fp.n_streams * fp.mb_h * segs;
}

size_t pipeline_task_list(const FrameParams& fp, int frames, int lag, int seg, bool split, const int32_t* kinds,
                          int2* tasks, int qbeg[3], int qend[3], uint32_t* keys) {
  int S = fp.n_streams, H = fp.mb_h, W = fp.mb_w;
  int segs = (W + seg - 1) / seg, a = seg > 2 ? seg : 2;
  if (lag <= 0) lag = a * 8 + seg + 7;
  auto key = [&](int f, int role, int y, int k) {
    return (size_t)a * (y + role) + (size_t)k * seg + role + (size_t)lag * f;
  };
  // queue of a segment: deblocking (1) when split, analysis of an IDR picture (2) when kinds are
  // given, else 0; each queue occupies its own range of keys, so each is in key order
  auto queue = [&](int f, int s, int role) {
    if (role) return split ? 1 : 0;
    return kinds && kinds[f * S + s] == RG_FRAME_IDR ? 2 : 0;
  };
  size_t n_keys1 = key(frames - 1, 1, H - 1, segs - 1) + 1, n_keys = 3 * n_keys1;
  auto slot = [&](int f, int s, int role, int y, int k) { return key(f, role, y, k) + queue(f, s, role) * n_keys1; };
  std::vector<size_t> start(n_keys + 1, 0);
  for (int f = 0; f < frames; f++)
    for (int role = 0; role < 2; role++)
      for (int s = 0; s < S; s++)
        for (int y = 0; y < H; y++)
          for (int k = 0; k < segs; k++) start[slot(f, s, role, y, k) + 1]++;
  for (size_t i = 0; i < n_keys; i++) start[i + 1] += start[i];
  for (int q = 0; q < 3; q++) {
    qbeg[q] = (int)start[q * n_keys1];
    qend[q] = (int)start[(q + 1) * n_keys1];
  }
  // placed in (picture, role, stream, row, segment) order within a key: a stable counting sort
  for (int f = 0; f < frames; f++)
    for (int role = 0; role < 2; role++)
      for (int s = 0; s < S; s++)
        for (int y = 0; y < H; y++)
          for (int k = 0; k < segs; k++) {
            size_t at = start[slot(f, s, role, y, k)]++;
            tasks[at] = make_int2(f * S + s, (y << 16) | ((k * seg) << 1) | role);
            if (keys) keys[at] = (uint32_t)key(f, role, y, k);
          }
  return pipeline_task_count(fp, frames, seg);
}

void launch_pipeline(const FrameGroups& fg, const StreamDev* d_streams, int n_desc, int total_rows, int* counters,
                     const int2* d_tasks, size_t n_tasks, const int qbeg[3], const int qend[3], int deblock_sms,
                     int intra_sms, int sms, int seg, int grid, unsigned long long timeout_ns, int* ready, int seq,
                     int* host_err, int* host_reach, cudaStream_t st, int form, const CompactOut* co) {
  PipeParams pp;
  pp.ticket = counters;
  pp.error = counters + 1;
  pp.ana = counters + 4;
  pp.db = pp.ana + total_rows;
  pp.tasks = d_tasks;
  pp.n_tasks = (int)n_tasks;
  for (int q = 0; q < 3; q++) {
    pp.qbeg[q] = qbeg[q];
    pp.qend[q] = qend[q];
  }
  pp.deblock_sms = deblock_sms;
  pp.intra_sms = intra_sms;
  pp.role_by_sm = grid >= sms;
  pp.seg = seg;
  pp.timeout_ns = timeout_ns;
  pp.rows_done = pp.db + total_rows;
  pp.ready = ready;
  pp.seq = seq;
  pp.host_err = host_err;
  pp.reach = pp.rows_done + n_desc;
  pp.cwords = co ? co->words : nullptr;
  pp.crow = co ? co->row_words : 0;
  pp.cbytes = co ? co->row_bytes : nullptr;
  int g = grid < pp.n_tasks ? grid : pp.n_tasks;
  if (form) pipeline_kernel<1><<<g, 32, 0, st>>>(fg, d_streams, pp);
  else pipeline_kernel<0><<<g, 32, 0, st>>>(fg, d_streams, pp);
  if (host_err) error_to_host_kernel<<<1, 1, 0, st>>>(pp.error, pp.reach, host_err, host_reach);
}

void launch_error_to_host(const int* counters, int n_desc, int total_rows, int* host_err, int* host_reach,
                          cudaStream_t st) {
  const int* reach = counters + 4 + 2 * (size_t)total_rows + n_desc;
  error_to_host_kernel<<<1, 1, 0, st>>>(counters + 1, reach, host_err, host_reach);
}

size_t pipeline_counter_ints(int total_rows, int n_desc) { return 4 + 2 * (size_t)total_rows + n_desc + 2; }

size_t pipeline_counter_ints(const FrameParams& fp, int frames) {
  return pipeline_counter_ints(frames * fp.n_streams * fp.mb_h, frames * fp.n_streams);
}

void launch_extend_borders(const FrameParams& fp, const StreamDev* d_streams, cudaStream_t st) {
  int rows = fp.mb_h * 16 + 2 * kPadY;
  int chunks = fp.stride_y / 16;
  int threads = 256;
  dim3 grid((rows * chunks + threads - 1) / threads, 1, 3 * fp.n_streams);
  extend_borders_kernel<<<grid, threads, 0, st>>>(fp, d_streams);
}

}  // namespace rg
