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

// Everything the analysis needs of one QP, in the form its lanes use it (upload_tables); a warp keeps
// its picture's luma and chroma entries in shared memory (load_desc).
struct QTab {
  uint32_t mf[2][2];   // quantiser scales of a 4x4 half (quant_half): [coefficient rows h, h + 2][column parity]
  int32_t dq[2][2];    // dequantiser scales alike, shifted by qp / 6
  uint32_t bias[2];    // inter, intra
  uint32_t shift;
  int32_t dc_mf, dc_dq;  // DC transforms: quantiser scale, dequantiser scale
  uint32_t lambda;
  uint32_t mf8[3][3];  // 8x8: [column 0, odd, 2 of four][row 0, odd, 2 of four]
  int32_t dq8[3][3];
  uint32_t bias8;
  int32_t rnd8, sh8;   // dequantised level = (level * dq8 + rnd8) >> sh8
};
__device__ QTab g_qtab[52];
constexpr int kQTabWords = (int)(sizeof(QTab) / 4), kQTabWords4 = (int)(offsetof(QTab, mf8) / 4);  // all, and chroma's
__constant__ uint8_t c_cqp[52];
// Deblocking thresholds by QP: {alpha | beta << 8, tC0 of strengths 1..3 a byte each}.
__constant__ uint2 c_deblock[52];

// ---------------------------------------------------------------------------------------------
// Shared memory of one macroblock warp.
// Block stride (words) of the 8x8 intermediates: 8 banks apart, so the four blocks' rows and columns
// fall into different banks.
constexpr int kT8Block = 72;
// A plane of the interpolation window: 23 rows of 24 samples.
constexpr int kWinPlane = 23 * 24 + 8;
struct __align__(16) Smem {
  uint8_t src_y[256];
  uint8_t src_u[64];
  uint8_t src_v[64];
  uint8_t pred_y[256];
  uint8_t pred_u[64];
  uint8_t pred_v[64];
  uint8_t tmp_y[256];       // plane prediction / I4x4 reconstruction
  // Samples around an integer position of the reference (ensure_window): plane 0 the integer samples
  // (23 rows of 24 from two rows / columns above-left of one sample above-left of the position), and
  // on the same grid b (between a sample and its right neighbour), h (and the one below) and j (the
  // four); rows and columns 2..19 of those hold values.
  alignas(16) uint8_t win[kWinPlane];
  // The half-sample planes live until the prediction is made; the 8x8 transform's intermediates are
  // needed only after it (the residual), so they share the space.
  union alignas(16) {
    struct {
      uint8_t hp[3][kWinPlane];     // b, h, j
      alignas(8) int16_t hr[23 * 20];  // unrounded horizontal 6-tap sums, columns 0..19
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
  alignas(4) uint8_t top[24];  // luma row above the macroblock (x0 .. x0 + 23)
  alignas(4) uint8_t left[16];
  alignas(4) uint8_t ctop[2][8];
  uint8_t cleft[2][8];
  alignas(16) StreamDev sd;       // the picture worked on (load_desc) and its stream's size (load_params)
  alignas(16) FrameParams fp;
  alignas(16) QTab qt[2];         // the picture's luma and chroma QP
  int qt_qp;                      // the luma QP they are of
  uint32_t qpt[16];               // quarter-sample phases: the two planes averaged (init_tables)
  alignas(16) uint32_t dbmv[12];  // deblocking, search forms: quadrant vectors of the macroblock, its left and top neighbours
  int win_x, win_y, win_have;     // ensure_window: the position held (kNoWin: none), its planes built (bits 0..2)
  int recon_seen;                 // this macroblock's neighbours are reconstructed (wait_recon)
  int db_row, seen_db;            // last acquired progress db_prev[db_row] of the reference picture
  int reach_y, reach_x;           // 1 + the largest reach waited for beyond zero motion, in macroblocks
  alignas(16) uint8_t i4m[16];    // Intra4x4PredMode of this macroblock (decoding order)
  uint8_t i4e[48];          // the current 4x4 block's edge samples Q, their avg2 and their avg3 (i4_tap)
};
static_assert(offsetof(Smem, coef) % 4 == 0 && offsetof(Smem, ccoef) % 4 == 0, "level arrays cleared by words");
static_assert(offsetof(rg_mb_out, luma) % 4 == 0 && offsetof(rg_mb_out, chroma_dc) % 4 == 0 &&
                  offsetof(rg_mb_out, chroma_ac) % 4 == 0 && sizeof(rg_mb_out) % 4 == 0,
              "record levels written by words");
static_assert(offsetof(Smem, coef) % 8 == 0 && offsetof(Smem, ccoef) % 8 == 0 && offsetof(Smem, coef8) % 8 == 0 &&
                  offsetof(Smem, t8) % 16 == 0 && offsetof(Smem, zz8) % 8 == 0 && offsetof(Smem, i4m) % 4 == 0 &&
                  offsetof(Smem, src_u) % 8 == 0 && offsetof(Smem, pred_u) % 8 == 0,
              "rows of levels, intermediates and samples move as vectors");
static_assert(20 * 24 <= kWinPlane && 24 * 12 <= kWinPlane, "the deblocking tiles fit the window's planes");
static_assert(offsetof(Smem, pred_y) % 8 == 0 && offsetof(Smem, tmp_y) % 8 == 0, "16x16 predictions written 8 bytes per lane");

// The warps of a block each work on a macroblock of their own; sm is the calling warp's shared memory.
// The functions below address it directly (shared-memory loads from one offset) instead of through a
// reference, which a call turns into a generic address -- a 64-bit pointer in registers and loads
// that resolve their memory space as they run.
// Blocks are 32 x warps threads.
extern __shared__ __align__(16) uint8_t smw[];
#define sm (((Smem*)smw)[threadIdx.y])
__device__ __forceinline__ uint8_t* sm_at(int off) { return (uint8_t*)&sm + off; }

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t pack16(int lo, int hi) { return __byte_perm((uint32_t)lo, (uint32_t)hi, 0x5410); }
__device__ __forceinline__ uint32_t wsum(uint32_t v) { return __reduce_add_sync(FULL, v); }
__device__ __forceinline__ int clip255(int v) { return v < 0 ? 0 : (v > 255 ? 255 : v); }
__device__ __forceinline__ int16_t clamp_i16(int v) { return (int16_t)(v < -32768 ? -32768 : (v > 32767 ? 32767 : v)); }

// Column and row of 4x4 block b in decoding order (enc.rs:522 blk_xy).
__device__ __forceinline__ int blk_x(int b) { return (b & 1) + ((b >> 1) & 2); }
__device__ __forceinline__ int blk_y(int b) { return ((b >> 1) & 1) + ((b >> 2) & 2); }
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
// Per-lane 8-point transforms (crates/ragdoll-simd/src/fixed.rs:392; h264_idct.rs:225)
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
// ---------------------------------------------------------------------------------------------
// Half-sample window (h264_enc.rs:747 hpel_window, :803 hpel_window_centre) around the integer
// position (px, py) of a 16x16 block: quarter-sample vectors up to 3 away from it. Window row y,
// column x is the sample at (px - 3 + x, py - 3 + y); the block itself starts at (3, 3).
constexpr int kNoWin = 1 << 20;
__device__ __forceinline__ void stage_window(int px, int py) {
  const int lane = lane_id(), stride = sm.fp.stride_y;
  const uint8_t* ref = sm.sd.ref_y + (long)(py - 3) * stride + px - 3;
  const uint32_t sh = (uint32_t)((uintptr_t)ref & 3) * 8u;  // rows are 64-byte multiples apart
  ref = (const uint8_t*)((uintptr_t)ref & ~(uintptr_t)3);
  // 23 rows x 6 words: five words per lane, all loads issued before the first use
  uint32_t lo[5], hi[5];
#pragma unroll
  for (int r = 0; r < 5; r++) {
    const int q = min(lane + 32 * r, 23 * 6 - 1), k = q / 6, w = q - 6 * k;
    const uint32_t* b = (const uint32_t*)(ref + k * stride + 4 * w);
    lo[r] = b[0];
    hi[r] = b[1];
  }
#pragma unroll
  for (int r = 0; r < 5; r++) {
    const int q = lane + 32 * r;
    if (q < 23 * 6) *(uint32_t*)&sm.win[4 * q] = __funnelshift_r(lo[r], hi[r], sh);
  }
}
__device__ __forceinline__ int dp4a_us(uint32_t a, int b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ int dp2a_ss(uint32_t a, int b, int c) {
  int d;
  asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
constexpr int taps4(int t0, int t1, int t2, int t3) {
  return (t0 & 255) | ((t1 & 255) << 8) | ((t2 & 255) << 16) | (int)((unsigned)(t3 & 255) << 24);
}
__device__ __forceinline__ uint32_t pack_clip(int a, int b, int c, int d) {
  return (uint32_t)clip255(a) | ((uint32_t)clip255(b) << 8) | ((uint32_t)clip255(c) << 16) | ((uint32_t)clip255(d) << 24);
}
// The 6-tap filter (1, -5, 20, 20, -5, 1) along rows: four outputs of an item from three words by
// byte dot products; the unrounded sums for j, and plane b of rows 2..19.
__device__ __forceinline__ void build_b() {
#pragma unroll 1
  for (int i = lane_id(); i < 23 * 5; i += 32) {
    const int y = i / 5, k = i - 5 * y;
    const uint32_t* w = (const uint32_t*)&sm.win[y * 24 + 4 * k];
    const uint32_t w0 = w[-1], w1 = w[0], w2 = w[1];  // (word -1 of item 0: columns 0, 1, never read)
    const int h0 = dp4a_us(w0, taps4(0, 0, 1, -5), dp4a_us(w1, taps4(20, 20, -5, 1), 0));
    const int h1 = dp4a_us(w0, taps4(0, 0, 0, 1), dp4a_us(w1, taps4(-5, 20, 20, -5), dp4a_us(w2, taps4(1, 0, 0, 0), 0)));
    const int h2 = dp4a_us(w1, taps4(1, -5, 20, 20), dp4a_us(w2, taps4(-5, 1, 0, 0), 0));
    const int h3 = dp4a_us(w1, taps4(0, 1, -5, 20), dp4a_us(w2, taps4(20, -5, 1, 0), 0));
    *(uint2*)&sm.hr[y * 20 + 4 * k] = make_uint2(pack16(h0, h1), pack16(h2, h3));
    if (y >= 2 && y < 20)
      *(uint32_t*)&sm.hp[0][y * 24 + 4 * k] = pack_clip((h0 + 16) >> 5, (h1 + 16) >> 5, (h2 + 16) >> 5, (h3 + 16) >> 5);
  }
}
// Down the columns: lane = (word column, three rows); two samples per word in 16-bit halves, biased by
// 80 << 5 so that no half goes negative.
__device__ __forceinline__ void build_h() {
  const int lane = lane_id(), seg = lane / 5, k = lane - 5 * seg;
  if (seg > 5) return;
  const uint8_t* w = &sm.win[3 * seg * 24 + 4 * k];
  uint32_t e[8], o[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const uint32_t v = *(const uint32_t*)(w + r * 24);
    e[r] = v & 0x00ff00ffu;
    o[r] = (v >> 8) & 0x00ff00ffu;
  }
  auto tap = [](const uint32_t* a) {
    const uint32_t v = (a[0] + a[5]) + 20u * (a[2] + a[3]) + 0x0a100a10u - 5u * (a[1] + a[4]);
    return __vminu2(__vmaxu2((v >> 5) & 0x07ff07ffu, 0x00500050u), 0x014f014fu) - 0x00500050u;
  };
#pragma unroll
  for (int r = 0; r < 3; r++) *(uint32_t*)&sm.hp[1][(3 * seg + 2 + r) * 24 + 4 * k] = tap(e + r) | (tap(o + r) << 8);
}
// j: the filter down the unrounded row sums, the same split, by 16-bit dot products of vertical pairs.
__device__ __forceinline__ void build_j() {
  const int lane = lane_id(), seg = lane / 5, k = lane - 5 * seg;
  if (seg > 5) return;
  uint32_t r[3] = {0u, 0u, 0u};
#pragma unroll 1
  for (int half = 0; half < 2; half++) {  // two columns
    uint32_t v[8];
#pragma unroll
    for (int y = 0; y < 8; y++) v[y] = *(const uint32_t*)&sm.hr[(3 * seg + y) * 20 + 4 * k + 2 * half];
    int j[3][2];
#pragma unroll
    for (int x = 0; x < 2; x++) {
      uint32_t w[7];
#pragma unroll
      for (int y = 0; y < 7; y++) w[y] = __byte_perm(v[y], v[y + 1], x ? 0x7632 : 0x5410);
#pragma unroll
      for (int y = 0; y < 3; y++)
        j[y][x] = dp2a_ss(w[y], taps4(1, -5, 0, 0), dp2a_ss(w[y + 2], taps4(20, 20, 0, 0), dp2a_ss(w[y + 4], taps4(-5, 1, 0, 0), 512))) >> 10;
    }
#pragma unroll
    for (int y = 0; y < 3; y++)
      r[y] = (r[y] >> 16) | ((uint32_t)clip255(j[y][0]) << 16) | ((uint32_t)clip255(j[y][1]) << 24);
  }
#pragma unroll
  for (int y = 0; y < 3; y++) *(uint32_t*)&sm.hp[2][(3 * seg + 2 + y) * 24 + 4 * k] = r[y];
}
// Makes the window around (px, py) hold its integer samples and the planes of `need` (bit 0 b, bit 1
// h, bit 2 j); what is there already is kept.
__device__ __noinline__ void ensure_window(int px, int py, int need) {
  int have = sm.win_have;
  if (sm.win_x != px || sm.win_y != py) {
    __syncwarp();
    stage_window(px, py);
    have = 0;
  }
  __syncwarp();
  const int miss = need & ~have;
  if ((miss & 5) && !(have & 1)) { build_b(); have |= 1; }
  if (miss & 2) { build_h(); have |= 2; }
  if (miss & 4) {
    __syncwarp();
    build_j();
    have |= 4;
  }
  if (lane_id() == 0) {
    sm.win_x = px;
    sm.win_y = py;
    sm.win_have = have;
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
// Quarter-sample prediction (window_src, enc.rs:1395; equal to h264_luma_mc_scalar, h264_mc.rs:148, by
// enc.rs:4030): phase fx | fy << 2 is the rounded average of two planes at fixed offsets, the same one
// twice where it is a plane itself. The offsets, in bytes from sm.win, packed in sm.qpt.
constexpr uint32_t qpel_entry(int phase) {
  constexpr uint32_t P = kWinPlane, B = (uint32_t)(offsetof(Smem, hp) - offsetof(Smem, win)), V = B + P, J = V + P;
  constexpr uint32_t a[16] = {0, 0, B, B, 0, B, B, B, V, V, J, J, V, V, J, V + 1};
  constexpr uint32_t b[16] = {0, B, B, 1, V, V, J, V + 1, V, J, J, V + 1, 24, B + 24, B + 24, B + 24};
  return a[phase] | (b[phase] << 16);
}
// 8 bytes of shared memory at any alignment.
__device__ __forceinline__ uint2 lds8(const uint8_t* p) {
  uintptr_t a = (uintptr_t)p;
  const uint32_t* b = (const uint32_t*)(a & ~(uintptr_t)3);
  uint32_t sh = (uint32_t)(a & 3) * 8u;
  uint32_t w0 = b[0], w1 = b[1], w2 = b[2];
  return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}
// Offset in a plane of the sample a quarter-sample vector (dx, dy) from the window's position points
// at, for the block's sample (0, 0).
__device__ __forceinline__ int qpel_pos(int dx, int dy) { return ((dy >> 2) + 3) * 24 + (dx >> 2) + 3; }
// This lane's 8 prediction samples (row lane / 2, columns 8 (lane & 1) ..) for the vector (dx, dy) from
// the window's position.
__device__ __noinline__ uint2 qpel8(int dx, int dy) {
  const int lane = lane_id(), at = qpel_pos(dx, dy) + (lane >> 1) * 24 + (lane & 1) * 8;
  const uint32_t e = sm.qpt[(dx & 3) | ((dy & 3) << 2)];
  const uint2 a = lds8(&sm.win[0] + at + (e & 0xffffu)), b = lds8(&sm.win[0] + at + (e >> 16));
  return make_uint2(__vavgu4(a.x, b.x), __vavgu4(a.y, b.y));
}
// The cheapest of the four neighbours of (x, y) at distance st (quarter samples) inside the bounds:
// up, left, right, down, the first on ties. s01, s23: this lane's share of their SADs, two to a word
// (a 16x16 SAD fits 16 bits). Lane k costs neighbour k. Returns cost << 2 | k, all ones when none is
// inside. exact_bits: vector bits by vec_cost's rule, without mvd_cost's 16-bit wrap.
struct Box {
  int lo0, hi0, lo1, hi1;
};
__device__ __noinline__ uint32_t best4(uint32_t s01, uint32_t s23, int x, int y, int st, Box b, int mvp0, int mvp1, uint32_t lambda,
                                       bool exact_bits) {
  s01 = wsum(s01);
  s23 = wsum(s23);
  const int k = lane_id() & 3;
  x += k == 1 ? -st : (k == 2 ? st : 0);
  y += k == 0 ? -st : (k == 3 ? st : 0);
  const uint32_t sad = ((k & 2 ? s23 : s01) >> (16 * (k & 1))) & 0xffffu;
  const uint32_t cost = sad + (exact_bits ? lambda * (se_bits(x - mvp0) + se_bits(y - mvp1))
                                          : mvd_cost(x - mvp0, lambda) + mvd_cost(y - mvp1, lambda));
  const bool ok = x >= b.lo0 && x <= b.hi0 && y >= b.lo1 && y <= b.hi1;
  return __reduce_min_sync(FULL, ok ? (cost << 2) | (uint32_t)k : UMAX);
}
__device__ __forceinline__ uint2 src8() {
  int lane = lane_id();
  return *(const uint2*)&sm.src_y[(lane >> 1) * 16 + (lane & 1) * 8];
}
// Prediction of the 16x16 block at (x0, y0) displaced by mv into pred_y (enc.rs:1058 mc_luma). A
// fractional vector leaves its window behind for the sub-pel search, which often starts there.
__device__ __noinline__ void mc_luma16(int x0, int y0, int mvx, int mvy) {
  const int ix = x0 + (mvx >> 2), iy = y0 + (mvy >> 2), fx = mvx & 3, fy = mvy & 3, lane = lane_id();
  uint2 v;
  if ((fx | fy) == 0) {
    v = ldg8(sm.sd.ref_y + (long)(iy + (lane >> 1)) * sm.fp.stride_y + ix + (lane & 1) * 8);
  } else {
    ensure_window(ix, iy, planes_needed(fx, fy));
    v = qpel8(fx, fy);
  }
  *(uint2*)&sm.pred_y[(lane >> 1) * 16 + (lane & 1) * 8] = v;
  __syncwarp();
}
// Four chroma samples (the bilinear 1/8-sample filter), the first at src for phase (0, 0): weights of the
// samples (0, 0), (1, 0), (0, 1), (1, 1) a byte each, a dot product a sample.
__device__ __forceinline__ uint32_t chroma4(const uint8_t* src, int stride, int fx, int fy) {
  const uint32_t w = (uint32_t)((8 - fx) * (8 - fy) | (fx * (8 - fy)) << 8 | ((8 - fx) * fy) << 16 | (fx * fy) << 24);
  const uint2 a = ldg8(src), b = ldg8(src + stride);
  uint32_t v = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t ra = __funnelshift_r(a.x, a.y, 8 * k), rb = __funnelshift_r(b.x, b.y, 8 * k);
    v |= (__dp4a(__byte_perm(ra, rb, 0x5410), w, 32u) >> 6) << (8 * k);
  }
  return v;
}
// Chroma prediction of both planes (h264_enc.rs:1279 chroma_mc_8x8_x2_scalar; enc.rs:1082).
__device__ __noinline__ void mc_chroma8(const uint8_t* ru, const uint8_t* rv, int stride, int mbx, int mby, int mvx, int mvy) {
  int lane = lane_id();
  int cx = mbx * 8 + (mvx >> 3), cy = mby * 8 + (mvy >> 3), fx = mvx & 7, fy = mvy & 7;
  const int plane = lane >> 4, idx = (lane & 15) * 4, r = idx >> 3, c0 = idx & 7;
  *(uint32_t*)((plane ? sm.pred_v : sm.pred_u) + r * 8 + c0) = chroma4((plane ? rv : ru) + (long)(cy + r) * stride + cx + c0, stride, fx, fy);
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// Quantisation helpers (enc.rs:1703-1779, h264_enc.rs:408)
// (Every transform here is of 8-bit differences: |coefficient| is at most 64 * 255 and the scales at
// most 20972, so a product and the bias fit 32 bits, and a level 16.)

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
// A helper is one copy of code for luma and chroma, inter and intra: the warps of an SM run different
// phases of their macroblocks, and what they fetch is the kernel's scarcest resource (the code of a P
// macroblock is several times the instruction cache).
struct Half4 {
  int a[4], b[4];  // its first and second row
};
// Rows of samples at byte offset `off` in Smem: the lane's two.
__device__ __forceinline__ uint2 half_rows(int off, int stride, int h) {
  return make_uint2(*(const uint32_t*)sm_at(off + h * stride), *(const uint32_t*)sm_at(off + (3 - h) * stride));
}
// The column pass of the forward transform and of the Hadamard transform: differences of the lane's
// rows of s and p, columns 0, 2 and 1, 3 packed as hi * 65536 + lo (sums, differences and small
// multiples of such pairs are the pairs of the results), then the butterfly with the partner lane.
// m = 1 + h for the core transform, 1 for Hadamard.
__device__ __forceinline__ void half_columns(uint2 s, uint2 p, int h, int m, int (&a)[4], int (&b)[4]) {
  const int ae = (int)(s.x & 0x00ff00ffu) - (int)(p.x & 0x00ff00ffu), be = (int)(s.y & 0x00ff00ffu) - (int)(p.y & 0x00ff00ffu);
  const int ao = (int)__byte_perm(s.x, 0u, 0x4341) - (int)__byte_perm(p.x, 0u, 0x4341),
            bo = (int)__byte_perm(s.y, 0u, 0x4341) - (int)__byte_perm(p.y, 0u, 0x4341);
  // h = 0: sum s03 and difference d03 of rows 0 and 3; h = 1: s12 and d12 of rows 1 and 2
  auto exchange = [&](int r0, int r1, int& x, int& y) {
    const int sum = r0 + r1, dif = r0 - r1, o = __shfl_xor_sync(FULL, h ? sum : dif, 1);
    const int u = h ? o : sum, v = h ? dif : o;  // s03, s12 or d03, d12
    x = u * m + v;  // row 0: s03 + s12, row 1: 2 d03 + d12
    y = u - v * m;  // row 2: s03 - s12, row 3: d03 - 2 d12
  };
  int xe, ye, xo, yo;
  exchange(ae, be, xe, ye);
  exchange(ao, bo, xo, yo);
  a[0] = (int16_t)xe; a[2] = (xe + 0x8000) >> 16; a[1] = (int16_t)xo; a[3] = (xo + 0x8000) >> 16;
  b[0] = (int16_t)ye; b[2] = (ye + 0x8000) >> 16; b[1] = (int16_t)yo; b[3] = (yo + 0x8000) >> 16;
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
__device__ __forceinline__ uint2 pack_half(const int (&r)[4]) {
  return make_uint2(pack16(r[0], r[1]), pack16(r[2], r[3]));
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

// SATD (metrics.rs:705, halved) of the macroblock's source against the 16x16 plane at byte offset
// `at`: half the sum of the magnitudes of every block's Hadamard coefficients.
__device__ __noinline__ uint32_t satd16(int at) {
  const int lane = lane_id(), h = lane & 1, off = blk_off16(lane >> 1);
  int a[4], b[4];
  half_columns(half_rows((int)offsetof(Smem, src_y) + off, 16, h), half_rows(at + off, 16, h), h, 1, a, b);
  // |x + y| + |x - y| = 2 max(|x|, |y|): the last butterfly and the halving in one
  auto row = [](const int (&r)[4]) {
    const int s03 = r[0] + r[3], s12 = r[1] + r[2], d03 = r[0] - r[3], d12 = r[1] - r[2];
    return (uint32_t)(max(abs(s03), abs(s12)) + max(abs(d03), abs(d12)));
  };
  return wsum(row(a) + row(b));
}
// Forward transform (fixed.rs:104) and quantisation (enc.rs:1703-1779) of the lane's half of the block
// at byte offsets src and pred of Smem. mask, alike in both lanes: the block's nonzero levels by
// zig-zag index (bits 0..15, the DC of a chroma block left out) and in bit 16 whether one of them is above 1. ra, rb:
// the levels of its two coefficient rows; dc: the block's DC coefficient before quantisation (h = 0).
struct HalfLevels {
  uint2 ra, rb;
  uint32_t mask;
  int dc;
};
__device__ __noinline__ HalfLevels quant_half(int src, int pred, int stride, int chroma, bool intra) {
  const int first = chroma;  // a chroma block's DC is coded apart
  const int h = lane_id() & 1;
  const QTab& qt = sm.qt[chroma];
  const uint32_t shift = qt.shift, bias = qt.bias[intra], mf[2] = {qt.mf[h][0], qt.mf[h][1]};
  Half4 v;
  half_columns(half_rows(src, stride, h), half_rows(pred, stride, h), h, 1 + h, v.a, v.b);
  auto row = [](int (&r)[4]) {
    const int s03 = r[0] + r[3], s12 = r[1] + r[2], d03 = r[0] - r[3], d12 = r[1] - r[2];
    r[0] = s03 + s12; r[1] = 2 * d03 + d12; r[2] = s03 - s12; r[3] = d03 - 2 * d12;
  };
  row(v.a);
  row(v.b);
  HalfLevels q;
  q.dc = v.a[0];
  // zig-zag indices (Table 8-12) of rows 0 and 2, or 1 and 3, four bits each
  uint32_t zz = h ? 0xfea9c742u : 0xdb836510u, mask = 0, big = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    int& c = k < 4 ? v.a[k & 3] : v.b[k & 3];
    const uint32_t l = ((uint32_t)abs(c) * mf[k & 1] + bias) >> shift;
    if (l) mask |= 1u << ((zz >> (4 * k)) & 15u);
    big |= k == 0 && first && !h ? 0u : l;
    c = c < 0 ? -(int)l : (int)l;
  }
  mask &= first ? 0xfffeu : 0xffffu;
  mask |= big > 1u ? 0x10000u : 0u;
  q.mask = mask | __shfl_xor_sync(FULL, mask, 1);
  q.ra = pack_half(v.a);
  q.rb = pack_half(v.b);
  return q;
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
// quant_half of the macroblock's luma: lane pair b owns block b.
__device__ __forceinline__ HalfLevels quant_luma(bool intra) {
  const int off = blk_off16(lane_id() >> 1);
  return quant_half((int)offsetof(Smem, src_y) + off, (int)offsetof(Smem, pred_y) + off, 16, 0, intra);
}

// Luma 4x4 residual of pred_y, quantised (inter) and decimated into sm.coef
// (enc.rs:1810 quant_luma_4x4_inter).
struct Luma4 {
  uint32_t cbp, nnz, nz16;  // coded block pattern, nonzero levels kept, blocks holding levels (bit b)
};
__device__ __noinline__ Luma4 luma4x4_inter() {
  const int lane = lane_id(), b = lane >> 1, h = lane & 1;
  HalfLevels q = quant_luma(false);
  const uint32_t m = q.mask;
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
  if (!coded) q.ra = q.rb = make_uint2(0u, 0u);
  *(uint2*)&sm.coef[b * 16 + h * 4] = q.ra;
  *(uint2*)&sm.coef[b * 16 + h * 4 + 8] = q.rb;
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
#pragma unroll
  for (int k = 0; k < 16; k++)
    if (lane_id() == k) sm.qpt[k] = qpel_entry(k);
  if (lane_id() == 0) sm.qt_qp = -1;
  __syncwarp();
}
// Row of the 8x8 scale tables (QTab::mf8, dq8) for coordinate k: position classes (h264.rs:1343)
// {0, 3, 4, 3}, {3, 1, 5, 1}, {4, 5, 2, 5}, {3, 1, 5, 1} by the low two bits of row and column.
__device__ __forceinline__ int class8(int k) { return (k & 1) ? 1 : (k & 2); }
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
__device__ __noinline__ uint32_t luma8x8_inter() {
  const int lane = lane_id(), b = lane >> 3, q = lane & 7;
  const int off = ((b >> 1) * 8 + q) * 16 + (b & 1) * 8;
  const QTab& qt = sm.qt[0];
  const uint32_t shift = qt.shift + 1, bias = qt.bias8;
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
  const uint32_t* mf = qt.mf8[class8(q)];
  const uint2 zz = *(const uint2*)&sm.zz8[q * 8];
  uint32_t lo = 0, hi = 0, big = 0;
#pragma unroll
  for (int y = 0; y < 8; y++) {
    const uint32_t l = ((uint32_t)abs(o[y]) * mf[class8(y)] + bias) >> shift;
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

// |Level| of a DC transform's coefficient (enc.rs:1938, :1960: one bit more, f = 2^qbits / 3).
__device__ __forceinline__ int quant_dc(int a, const QTab& q) {
  const uint32_t qbits = q.shift + 1;
  return (int)(((uint32_t)a * (uint32_t)q.dc_mf + (1u << qbits) / 3u) >> qbits);
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
__device__ __noinline__ ChromaAc chroma_quant(bool intra) {
  const int lane = lane_id(), h = lane & 1, b = (lane >> 1) & 7, off = blk_off8(b);
  const HalfLevels q = quant_half((int)offsetof(Smem, src_u) + off, (int)offsetof(Smem, pred_u) + off, 8, 1, intra);
  const uint32_t m = q.mask;
  // 2x2 DC transform + quantisation (enc.rs:1938 quant_chroma_dc; f = 2^qbits / 3 always); block b & 3
  // of the plane ends with output b & 3
  int dc = q.dc;
  {
    int o = __shfl_xor_sync(FULL, dc, 2);
    dc = (b & 1) ? o - dc : dc + o;
    o = __shfl_xor_sync(FULL, dc, 4);
    dc = (b & 2) ? o - dc : dc + o;
    const int l = quant_dc(abs(dc), sm.qt[1]);
    dc = dc < 0 ? -l : l;
  }
  if (lane < 16) {
    *(uint2*)&sm.ccoef[b * 16 + h * 4] = q.ra;
    *(uint2*)&sm.ccoef[b * 16 + h * 4 + 8] = q.rb;
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

// Adds the dequantised residual (levels of coefficient rows h, h + 2 in ra, rb; has_dc: the DC
// coefficient given, dequantised, instead) of the lane's half of a block to the samples at byte offset
// `off` of Smem; lanes not `on` leave them.
__device__ __noinline__ void recon_half(uint2 ra, uint2 rb, int chroma, bool has_dc, int dc, int off, int stride, bool on) {
  const int h = lane_id() & 1, dq[2] = {sm.qt[chroma].dq[h][0], sm.qt[chroma].dq[h][1]};
  Half4 v;
  unpack_half(ra, v.a);
  unpack_half(rb, v.b);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v.a[k] = clamp_i16(v.a[k] * dq[k & 1]);
    v.b[k] = clamp_i16(v.b[k] * dq[k & 1]);
  }
  if (has_dc && !h) v.a[0] = dc;
  half_inv(v, h);
  const uint2 p = half_rows(off, stride, h);
  if (on) {
    *(uint32_t*)sm_at(off + h * stride) = add_clip4(p.x, v.a);
    *(uint32_t*)sm_at(off + (3 - h) * stride) = add_clip4(p.y, v.b);
  }
  __syncwarp();
}
// The lane's rows of block b of sm.coef / sm.ccoef.
__device__ __forceinline__ uint2 level_row(const int16_t* c, int b, int row) { return *(const uint2*)&c[b * 16 + row * 4]; }

// Adds the dequantised chroma residual to pred_u / pred_v (enc.rs:1992 recon_chroma): the DC of
// each block from the 2x2 inverse (h264.rs:1674 dequantize_idct_chroma_dc2x2), its AC dequantised
// when cbpc == 2, then the inverse core transform. Two lanes per block as in chroma_quant.
__device__ __noinline__ void chroma_recon(int cbpc) {
  if (cbpc == 0) return;
  const int lane = lane_id(), h = lane & 1, b = (lane >> 1) & 7, bb = b & 3;
  int lv[4];
  unpack_half(*(const uint2*)&sm.cdc[b & 4], lv);
  const int e = lv[0] - lv[1], apb = lv[0] + lv[1], cmd = lv[2] - lv[3], cpd = lv[2] + lv[3];
  const int dcv = bb == 0 ? apb + cpd : (bb == 1 ? e + cmd : (bb == 2 ? apb - cpd : e - cmd));
  uint2 ra = level_row(sm.ccoef, b, h), rb = level_row(sm.ccoef, b, h + 2);
  if (cbpc < 2) ra = rb = make_uint2(0u, 0u);
  recon_half(ra, rb, 1, true, (int16_t)((dcv * sm.qt[1].dc_dq) >> 7), blk_off8(b) + (int)offsetof(Smem, pred_u), 8, lane < 16);
}

// Raster position of each 4x4 zig-zag index, 4 bits per index (frame scan, Table 8-12).
constexpr unsigned long long kScan4Packed = 0xfeb7adc963258410ull;

// Adds the dequantised 8x8 residual of the coded blocks of sm.coef8 to pred_y (enc.rs:2013
// recon_8x8: dequantize_block8x8, h264.rs:1403, then h264_idct8_add, h264_idct.rs:207).
// Lanes 8b..8b+7 own block b: row q, then column q. Blocks that are not coded add zero.
__device__ __noinline__ void recon_luma8x8(int cbp) {
  const int lane = lane_id(), b = lane >> 3, q = lane & 7;
  const bool coded = (cbp >> b) & 1;
  const int* dq = sm.qt[0].dq8[class8(q)];
  const int rnd = sm.qt[0].rnd8, sh = sm.qt[0].sh8;
  int d[8], o[8];
#pragma unroll
  for (int x = 0; x < 8; x++) {
    const int l = coded ? sm.coef8[b * 64 + sm.zz8[x * 8 + q]] : 0;
    d[x] = clamp_i16((l * dq[class8(x)] + rnd) >> sh);
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
__device__ __forceinline__ void recon_luma4x4() {
  const int lane = lane_id(), b = lane >> 1, h = lane & 1;
  recon_half(level_row(sm.coef, b, h), level_row(sm.coef, b, h + 2), 0, false, 0, blk_off16(b) + (int)offsetof(Smem, pred_y), 16, true);
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
// Four samples of a plane prediction, (v + k step) >> 5 clipped.
__device__ __forceinline__ uint32_t plane4(int v, int step) {
  return pack_clip(v >> 5, (v + step) >> 5, (v + 2 * step) >> 5, (v + 3 * step) >> 5);
}
__device__ __noinline__ void pred16_into(int mode, int dst, bool ht, bool hl, int tl) {
  int lane = lane_id();
  int y = lane >> 1, x0 = (lane & 1) * 8;
  uint8_t* o = sm_at(dst + y * 16 + x0);  // this lane's 8 samples (8-byte aligned)
  if (mode == 3) {
    int pa, pb, pc;
    plane16_params(ht, hl, tl, pa, pb, pc);
    const int v = pa + pb * (x0 - 7) + pc * (y - 7) + 16;
    *(uint2*)o = make_uint2(plane4(v, pb), plane4(v + 4 * pb, pb));
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
// Intra 16x16 analysis (enc.rs:1637 analyse_i16_edges): SATD per mode; the best mode and its cost. The
// vertical, horizontal and DC predictions have one nonzero row, column or coefficient of each
// block's Hadamard transform, so their SATDs are the source's with those terms replaced.
struct I16Fit {
  int mode;
  uint32_t cost;
};
__device__ __noinline__ I16Fit analyse_i16(bool ht, bool hl, int tl) {
  const int lane = lane_id(), h = lane & 1, b = lane >> 1, off = blk_off16(b);
  const int dc = 16 * dc16(ht, hl);
  int a[4], c[4];  // coefficient rows: h = 0: all rows' sum, s03 - s12; h = 1: d03 + d12, d03 - d12
  half_columns(half_rows((int)offsetof(Smem, src_y) + off, 16, h), make_uint2(0u, 0u), h, 1, a, c);
  auto row = [](int (&r)[4]) {
    const int s03 = r[0] + r[3], s12 = r[1] + r[2], d03 = r[0] - r[3], d12 = r[1] - r[2];
    r[0] = s03 + s12; r[1] = d03 + d12; r[2] = s03 - s12; r[3] = d03 - d12;
  };
  row(a);
  row(c);
  int top[4], left[4];
  const uint32_t tw = ht ? *(const uint32_t*)&sm.top[blk_x(b) * 4] : 0u, lw = hl ? *(const uint32_t*)&sm.left[blk_y(b) * 4] : 0u;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    top[k] = (int)((tw >> (8 * k)) & 255u) * 4;
    left[k] = (int)((lw >> (8 * k)) & 255u) * 4;
  }
  row(top);
  row(left);
  uint32_t all = 0, row0 = 0, row0v = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    all += (uint32_t)(abs(a[k]) + abs(c[k]));
    row0 += (uint32_t)abs(a[k]);
    row0v += (uint32_t)abs(a[k] - top[k]);
  }
  const uint32_t col0 = (uint32_t)(abs(a[0]) + abs(c[0])), col0h = (uint32_t)(abs(a[0] - left[h]) + abs(c[0] - left[h + 2]));
  const uint32_t sv = wsum(h ? all : all - row0 + row0v) >> 1, sh = wsum(all - col0 + col0h) >> 1,
                 sd = wsum(h ? all : all - (uint32_t)abs(a[0]) + (uint32_t)abs(a[0] - dc)) >> 1;
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
  const int lane = lane_id(), plane = lane >> 4, idx = (lane & 15) * 4, y = idx >> 3, x0 = idx & 7;
  int dcv[4], pa, pb, pc;
  chroma_pred_params(plane, ht, hl, plane ? k0.v : k0.u, dcv, pa, pb, pc);
  // this lane's four samples of every mode: DC, horizontal, vertical, plane
  const int dc = (y & 4) ? (x0 ? dcv[3] : dcv[2]) : (x0 ? dcv[1] : dcv[0]);
  const uint32_t w0 = (uint32_t)dc * 0x01010101u, w1 = hl ? sm.cleft[plane][y] * 0x01010101u : 0x80808080u,
                 w2 = ht ? *(const uint32_t*)&sm.ctop[plane][x0] : 0x80808080u,
                 w3 = plane4(pa + pb * (x0 - 3) + pc * (y - 3) + 16, pb);
  const uint32_t src = *(const uint32_t*)&sm.src_u[lane * 4];
  // the SADs of two modes per reduction (each below 2^16)
  const uint32_t s01 = wsum(__vsadu4(src, w0) | (__vsadu4(src, w1) << 16)), s23 = wsum(__vsadu4(src, w2) | (__vsadu4(src, w3) << 16));
  uint32_t best = s01 & 0xffffu, w = w0;
  int bm = 0;
  auto take = [&](int m, bool ok, uint32_t sad, uint32_t v) {
    if (ok && sad + 8u < best) { best = sad + 8u; bm = m; w = v; }
  };
  take(1, hl, s01 >> 16, w1);
  take(2, ht, s23 & 0xffffu, w2);
  take(3, ht && hl, s23 >> 16, w3);
  *(uint32_t*)&sm.pred_u[lane * 4] = w;
  __syncwarp();
  return bm;
}

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
// The taps of half h of mode m (its rows as in Half4) at [2 m + h], a byte 16 kind + i per sample:
// offsets into sm.i4e, the edge samples, their avg2 and their avg3 (filled by upload_tables).
__device__ uint2 g_i4tap[18];
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
  if (sm.sd.qp != sm.qt_qp) {  // another QP than the last picture's (init_tables: none)
    const uint32_t* l = (const uint32_t*)&g_qtab[sm.sd.qp];
    const uint32_t* ch = (const uint32_t*)&g_qtab[sm.sd.qpc];
    const uint32_t w0 = l[lane], w1 = lane + 32 < kQTabWords ? l[lane + 32] : 0u, w2 = lane < kQTabWords4 ? ch[lane] : 0u;
    __syncwarp();
    ((uint32_t*)&sm.qt[0])[lane] = w0;
    if (lane + 32 < kQTabWords) ((uint32_t*)&sm.qt[0])[lane + 32] = w1;
    if (lane < kQTabWords4) ((uint32_t*)&sm.qt[1])[lane] = w2;
    if (lane == 0) sm.qt_qp = sm.sd.qp;
    __syncwarp();
  }
}
static_assert(kQTabWords > 32 && kQTabWords <= 64 && kQTabWords4 <= 32, "a luma entry is two words a lane, a chroma one less");
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
  const int lane = lane_id(), W = fp.width, H = fp.height, cw = (W + 1) >> 1, ch = (H + 1) >> 1;
  const int y = min(c.mby * 16 + (lane >> 1), H - 1), x0 = c.mbx * 16 + (lane & 1) * 8;
  const uint8_t* row = sm.sd.src_y + (long)y * fp.src_stride_y + x0;
  const int idx = (lane & 15) * 4, cy = min(c.mby * 8 + (idx >> 3), ch - 1), cx0 = c.mbx * 8 + (idx & 7);
  const uint8_t* crow = ((lane & 16) ? sm.sd.src_v : sm.sd.src_u) + (long)cy * fp.src_stride_uv + cx0;
  // inside the picture's width and aligned: a vector per lane (an 8-byte and a 4-byte load instead of
  // twelve of a byte)
  const bool fast = c.mbx * 16 + 16 <= W && (((uintptr_t)row & 7) | ((uintptr_t)crow & 3)) == 0;
  if (__all_sync(FULL, fast)) {
    const uint2 v = __ldg((const uint2*)row);
    const uint32_t w = __ldg((const uint32_t*)crow);
    *(uint2*)&sm.src_y[lane * 8] = v;
    *(uint32_t*)&sm.src_u[lane * 4] = w;
  } else {
#pragma unroll 4
    for (int k = 0; k < 8; k++) sm.src_y[lane * 8 + k] = __ldg(row + min(k, W - 1 - x0));
#pragma unroll 4
    for (int k = 0; k < 4; k++) sm.src_u[lane * 4 + k] = __ldg(crow + min(k, cw - 1 - cx0));
  }
  __syncwarp();
}
// Intra edges from the unfiltered reconstruction of this picture (enc.rs:1459-1521) into shared
// memory; returns the samples at the corner.
__device__ __noinline__ Corner load_edges(const Ctx c, bool want_topright) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  const int lane = lane_id(), x0 = c.mbx * 16, y0 = c.mby * 16;
  const bool ht = c.mby > 0, hl = c.mbx > 0;
  // two loads a lane, both in flight together: a word of the rows above -- lanes 0..5 luma (the last two
  // its top-right neighbour's), 6 / 7 U, 8 / 9 V, 10..12 the words that end in the corners -- and a
  // sample of the columns to the left -- lanes 0..15 luma, 16..23 U, 24..31 V. (Byte by byte, plane by
  // plane: 4 round trips to L2, 4 k cycles.)
  const int tp = lane < 6 ? 0 : (lane < 10 ? 1 + ((lane - 6) >> 1) : lane - 10), lp = lane < 16 ? 0 : (lane < 24 ? 1 : 2);
  auto plane = [&](int p) -> const uint8_t* { return p == 0 ? sd.cur_y : (p == 1 ? sd.cur_u : sd.cur_v); };
  const bool corner = lane >= 10;
  const bool tl = ht && lane < 13 && (corner ? hl : (lane < 4 || lane >= 6 || (want_topright && c.mbx + 1 < fp.mb_w)));
  const int tx = corner ? -4 : 4 * (lane < 6 ? lane : (lane - 6) & 1);
  uint32_t t = 0, l = 0;
  if (tl) t = __ldcg((const uint32_t*)(plane(tp) + (long)((tp ? y0 >> 1 : y0) - 1) * (tp ? fp.stride_c : fp.stride_y) + (tp ? x0 >> 1 : x0) + tx));
  if (hl)
    l = __ldcg(plane(lp) + (long)(lp ? (y0 >> 1) + (lane & 7) : y0 + lane) * (lp ? fp.stride_c : fp.stride_y) + (lp ? x0 >> 1 : x0) - 1);
  if (ht) {
    if (lane < 6) *(uint32_t*)&sm.top[4 * lane] = t;
    else if (lane < 10) *(uint32_t*)&sm.ctop[tp - 1][tx] = t;
  }
  if (hl) {
    if (lane < 16) sm.left[lane] = (uint8_t)l;
    else sm.cleft[lp - 1][lane & 7] = (uint8_t)l;
  }
  Corner k;
  k.y = ht && hl ? (int)(__shfl_sync(FULL, t, 10) >> 24) : 128;
  k.u = ht && hl ? (int)(__shfl_sync(FULL, t, 11) >> 24) : 128;
  k.v = ht && hl ? (int)(__shfl_sync(FULL, t, 12) >> 24) : 128;
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

// The 4x4 Hadamard transform of sixteen values, lane i < 16 holding entry i (row-major; the upper
// half-warp repeats it): outputs in the rows / columns order ++++, ++--, +--+, +-+- of both the
// forward (enc.rs:1960) and the inverse (h264.rs:1645) luma DC transform.
__device__ __noinline__ int hadamard16(int v) {
  const int lane = lane_id();
#pragma unroll
  for (int k = 1; k < 16; k <<= 1) {
    const int o = __shfl_xor_sync(FULL, v, k);
    v = (lane & k) ? o - v : v + o;
  }
  // natural order (bit 0: +-+-, bit 1: ++--) to the order above: 0, 2, 3, 1
  const int x = lane & 3, y = (lane >> 2) & 3;
  return __shfl_sync(FULL, v, (((0x1320 >> (4 * y)) & 3) << 2) | ((0x1320 >> (4 * x)) & 3));
}
// I16x16 coding and reconstruction (enc.rs:3587 code_i16) with prediction mode `mode`.
__device__ __noinline__ void code_i16(const Ctx c, int mode, bool ht, bool hl, Corner k0) {
  const int lane = lane_id(), b = lane >> 1, h = lane & 1;
  const int qp = sm.sd.qp;
  pred16_into(mode, (int)offsetof(Smem, pred_y), ht, hl, k0.y);
  const int cmode = analyse_chroma(ht, hl, k0);
  HalfLevels q = quant_luma(true);
  const int raster = blk_y(b) * 4 + blk_x(b);
  if (!h) {
    sm.ldc[raster] = (int16_t)q.dc;
    q.ra.x &= 0xffff0000u;  // the DC is coded apart
  }
  // without an AC level the macroblock codes none (cbp 0)
  const bool ac = (q.mask & 0xfffeu) != 0;
  const uint32_t nz = even_bits(__ballot_sync(FULL, ac));
  const int cbpl = nz ? 15 : 0;
  const uint32_t nzm = cbpl ? nz : 0u;
  *(uint2*)&sm.coef[b * 16 + h * 4] = q.ra;
  *(uint2*)&sm.coef[b * 16 + h * 4 + 8] = q.rb;
  __syncwarp();
  // luma DC: Hadamard (>> 1) + quantisation (enc.rs:1960), then the inverse (h264.rs:1645)
  const int had = hadamard16(sm.ldc[lane & 15]) >> 1;
  const int l = quant_dc(abs(had), sm.qt[0]), level = had < 0 ? -l : l;
  const int dcr = (hadamard16(level) * sm.qt[0].dc_dq + 128) >> 8;
  __syncwarp();
  if (lane < 16) {
    sm.ldc[lane] = (int16_t)level;
    sm.ldcr[lane] = (int16_t)dcr;
  }
  const ChromaAc ca = chroma_quant(true);
  const int cbpc = (ca.any(0) || ca.any(1)) ? 2 : (ca.dc() ? 1 : 0);
  __syncwarp();
  rg_mb_out* rec = sm.sd.rec + c.mb;
  record_luma4x4(rec);
  if (lane < 16) rec->luma_dc[lane] = sm.ldc[(kScan4Packed >> (4 * lane)) & 15];
  record_chroma(rec, cbpc);
  record_header(rec, RG_MB_I16X16, mode, cmode, cbpl | (cbpc << 4), 0, qp, 0, 0, 0, 0, nzm, false);
  recon_half(q.ra, q.rb, 0, true, sm.ldcr[raster], blk_off16(b) + (int)offsetof(Smem, pred_y), 16, true);
  chroma_recon(cbpc);
  store_recon(c, (int)offsetof(Smem, pred_y));
  write_info(c, kFlagIntra, cbpl, 0, 0, -1, nzm, false);
}

// I4x4 analysis (enc.rs:3336 analyse_i4): sixteen blocks in decoding order, each choosing among
// the available modes by SATD + lambda * (1 if the predicted mode else 4), then quantising and
// reconstructing before the next block: a serial chain, and the head of every GOP. Lane 2 m + h takes
// half of the block under mode m (Half4): all nine modes are predicted, costed, transformed,
// quantised and reconstructed side by side, the residual's chain beside the cost's, and the winner's
// two lanes store theirs (one mode per step and the residual after the choice: 3.4 k cycles a block
// on an idle SM). The macroblock and its edges form one tile (sm.win: sample (x, y) at 24 (y + 1) + 4 + x,
// unavailable samples 128). `masks`: lane b's mask of the modes tried in block b (the learned form's
// hints; bit m: Intra4x4PredMode m) -- those of them available, DC alone when none is. Returns the
// luma coded block pattern with the blocks holding levels in bits 4.. (bit 4 + b: block b), or -1 as
// soon as the running cost reaches `budget`.
__device__ __noinline__ int analyse_i4(const Ctx c, uint32_t budget, bool ht_mb, bool hl_mb, int tl_mb, uint32_t masks) {
  const int lane = lane_id(), h = lane & 1, m = lane >> 1, p = lane & 15;
  const QTab& qt = sm.qt[0];
  const uint32_t lambda = qt.lambda, shift = qt.shift, bias = qt.bias[1], mf[2] = {qt.mf[h][0], qt.mf[h][1]};
  const int dq[2] = {qt.dq[h][0], qt.dq[h][1]};
  const MbInfo* info = sm.sd.info;
  const uint32_t lmodes = hl_mb ? info[c.mb - 1].i4_right : 0x2222u, tmodes = ht_mb ? info[c.mb - sm.fp.mb_w].i4_bottom : 0x2222u;
  const uint2 taps = __ldg(&g_i4tap[min(lane, 17)]);
  // the tile's edges: the row above from its corner to the top-right neighbour's first four samples,
  // the column to the left
  if (lane < 20) sm.win[4 + lane] = ht_mb ? sm.top[lane] : 128;
  if (lane < 16) sm.win[24 * (lane + 1) + 3] = hl_mb ? sm.left[lane] : 128;
  if (lane == 20) sm.win[3] = (uint8_t)tl_mb;
  // this lane's edge sample relative to the block (lanes 0..14: Q[p]), and where t4.. are unavailable
  const int eoff = p <= 4 ? 24 * (p <= 1 ? 3 : 4 - p) - 1 : (p == 5 ? -25 : min(p - 6, 7) - 24), eoff3 = p >= 10 ? -21 : eoff;
  uint32_t total = lambda * 24;
  int luma = 0;
  __syncwarp();
#pragma unroll 1
  for (int b = 0; b < 16; b++) {
    const int bx = blk_x(b), by = blk_y(b), px = bx * 4, py = by * 4;
    const bool ht = by > 0 || ht_mb, hl = bx > 0 || hl_mb;
    const bool tr = !((0xa888 >> b) & 1) && (b != 5 || c.mbx + 1 < sm.fp.mb_w);  // blocks 3, 7, 11, 13, 15 have none
    uint8_t* tile = &sm.win[24 * (py + 1) + 4 + px];
    const int q = tile[tr ? eoff : eoff3];
    const uint32_t sums = wsum(lane >= 6 && lane <= 9 ? (uint32_t)q : (lane >= 1 && lane <= 4 ? (uint32_t)q << 16 : 0u));
    const int st = (int)(sums & 0xffffu), sl = (int)(sums >> 16);
    const int dc = ht && hl ? (st + sl + 4) >> 3 : (ht ? (st + 2) >> 2 : (hl ? (sl + 2) >> 2 : 128));
    const int q1 = __shfl_down_sync(FULL, q, 1), q2 = __shfl_down_sync(FULL, q, 2);
    if (lane < 16) {
      sm.i4e[p] = (uint8_t)(p == 15 ? dc : q);
      sm.i4e[16 + p] = (uint8_t)((q + q1 + 1) >> 1);
      sm.i4e[32 + p] = (uint8_t)((q + 2 * q1 + q2 + 2) >> 2);
    }
    // predicted mode (h264.rs:3283)
    int pm = 2;
    if ((c.mbx | bx) && (c.mby | by)) {
      const int ml = bx > 0 ? sm.i4m[((by >> 1) << 3) | (((bx - 1) >> 1) << 2) | ((by & 1) << 1) | ((bx - 1) & 1)]
                            : (int)((lmodes >> (4 * by)) & 15);
      const int mt = by > 0 ? sm.i4m[(((by - 1) >> 1) << 3) | ((bx >> 1) << 2) | (((by - 1) & 1) << 1) | (bx & 1)]
                            : (int)((tmodes >> (4 * bx)) & 15);
      pm = min(ml, mt);
    }
    const uint32_t avail = 0x4u | (ht ? 0x89u : 0u) | (hl ? 0x102u : 0u) | (ht && hl ? 0x70u : 0u);
    uint32_t allow = __shfl_sync(FULL, masks, b) & avail;
    if (!allow) allow = 0x4u;
    __syncwarp();
    // this lane's two predicted rows and their residual's columns; the butterflies of the Hadamard and
    // of the core transform share the exchange (half_columns)
    uint2 pr, sr = half_rows((int)offsetof(Smem, src_y) + py * 16 + px, 16, h);
    {
      uint32_t w[2] = {0u, 0u};
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint32_t tp = ((k < 4 ? taps.x : taps.y) >> (8 * (k & 3))) & 255u;
        w[k >> 2] |= (uint32_t)sm.i4e[tp] << (8 * (k & 3));
      }
      pr = make_uint2(w[0], w[1]);
    }
    Half4 v;
    uint32_t cost;
    {
      int u[2], w[2];
#pragma unroll
      for (int o = 0; o < 2; o++) {
        auto cols = [&](uint32_t r) { return (int)(o ? __byte_perm(r, 0u, 0x4341) : r & 0x00ff00ffu); };
        const int r0 = cols(sr.x) - cols(pr.x), r1 = cols(sr.y) - cols(pr.y), sum = r0 + r1, dif = r0 - r1;
        const int x = __shfl_xor_sync(FULL, h ? sum : dif, 1);
        u[o] = h ? x : sum;
        w[o] = h ? dif : x;
      }
      auto satd_row = [](int e, int o) {
        const int r0 = (int16_t)e, r2 = (e + 0x8000) >> 16, r1 = (int16_t)o, r3 = (o + 0x8000) >> 16;
        const int s03 = r0 + r3, s12 = r1 + r2, d03 = r0 - r3, d12 = r1 - r2;
        return (uint32_t)(max(abs(s03), abs(s12)) + max(abs(d03), abs(d12)));
      };
      cost = satd_row(u[0] + w[0], u[1] + w[1]) + satd_row(u[0] - w[0], u[1] - w[1]);
      auto fwd_row = [](int e, int o, int (&r)[4]) {
        const int r0 = (int16_t)e, r2 = (e + 0x8000) >> 16, r1 = (int16_t)o, r3 = (o + 0x8000) >> 16;
        const int s03 = r0 + r3, s12 = r1 + r2, d03 = r0 - r3, d12 = r1 - r2;
        r[0] = s03 + s12; r[1] = 2 * d03 + d12; r[2] = s03 - s12; r[3] = d03 - 2 * d12;
      };
      const int k = 1 + h;
      fwd_row(u[0] * k + w[0], u[1] * k + w[1], v.a);
      fwd_row(u[0] - w[0] * k, u[1] - w[1] * k, v.b);
    }
    cost += __shfl_xor_sync(FULL, cost, 1);
    cost += lambda * (m == pm ? 1u : 4u);
    const uint32_t key = __reduce_min_sync(FULL, m < 9 && ((allow >> m) & 1u) ? (cost << 4) | (uint32_t)m : UMAX);
    const int bm = (int)(key & 15u);
    total += key >> 4;
    if (total >= budget) return -1;
    // residual of every mode
    uint32_t any = 0;
    Half4 r;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      int& x = k < 4 ? v.a[k & 3] : v.b[k & 3];
      const uint32_t l = ((uint32_t)abs(x) * mf[k & 1] + bias) >> shift;
      any |= l;
      x = x < 0 ? -(int)l : (int)l;
      (k < 4 ? r.a[k & 3] : r.b[k & 3]) = clamp_i16(x * dq[k & 1]);
    }
    half_inv(r, h);
    const uint32_t nz = __ballot_sync(FULL, any != 0);
    if (m == bm) {
      *(uint2*)&sm.coef[b * 16 + h * 4] = pack_half(v.a);
      *(uint2*)&sm.coef[b * 16 + h * 4 + 8] = pack_half(v.b);
      *(uint32_t*)(tile + 24 * h) = add_clip4(pr.x, r.a);
      *(uint32_t*)(tile + 24 * (3 - h)) = add_clip4(pr.y, r.b);
      if (!h) sm.i4m[b] = (uint8_t)bm;
    }
    if ((nz >> (2 * bm)) & 3u) luma |= (1 << (b >> 2)) | (16 << b);
    __syncwarp();
  }
  const uint32_t* t = (const uint32_t*)&sm.win[24 * ((lane >> 1) + 1) + 4 + (lane & 1) * 8];
  *(uint2*)&sm.tmp_y[lane * 8] = make_uint2(t[0], t[1]);
  __syncwarp();
  return luma;
}

// `luma`: what analyse_i4 returned.
__device__ __noinline__ void code_i4(const Ctx c, int luma, bool ht, bool hl, Corner k0) {
  int lane = lane_id();
  const int cbpl = luma & 15;
  const uint32_t nzm = (uint32_t)luma >> 4;
  int cmode = analyse_chroma(ht, hl, k0);
  const ChromaAc ac = chroma_quant(true);
  int cbpc = (ac.any(0) || ac.any(1)) ? 2 : (ac.dc() ? 1 : 0);
  rg_mb_out* rec = sm.sd.rec + c.mb;
  record_luma4x4(rec);
  if (lane < 8) ((uint32_t*)rec)[kWordLumaDc + lane] = 0u;
  record_chroma(rec, cbpc);
  record_header(rec, RG_MB_I4X4, 0, cmode, cbpl | (cbpc << 4), 0, sm.sd.qp, 0, 0, 0, 0, nzm, true);
  chroma_recon(cbpc);
  store_recon(c, (int)offsetof(Smem, tmp_y));
  write_info(c, kFlagIntra, cbpl, 0, 0, -1, nzm, true);
}

// One macroblock of an I slice (enc.rs:3311 code_intra).
__device__ __noinline__ void analyse_intra_mb(const Ctx c) {
  const Corner k0 = load_edges(c, true);
  bool ht = c.mby > 0, hl = c.mbx > 0;
  uint32_t lambda = sm.qt[0].lambda;
  const I16Fit fit16 = analyse_i16(ht, hl, k0.y);
  if (fit16.cost > 40 * lambda) {
    const int cbpl = analyse_i4(c, fit16.cost + lambda * 4, ht, hl, k0.y, 0x1ffu);
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
__device__ __noinline__ bool probe_skip_luma() {
  const uint32_t m = quant_luma(false).mask;
  const uint32_t score = (lane_id() & 1) ? 0u : score4(m, 0);
  return wsum(score | ((m >> 16) << 16)) < 6;
}

// The residual of an inter macroblock whose prediction lies in pred_y / pred_u / pred_v
// (enc.rs:3158-3190), its record (code_inter, enc.rs:3196) and its reconstruction. can_skip: nothing
// coded makes it P_Skip with vector (mvx, mvy). Returns whether it did.
__device__ __noinline__ bool code_inter(const Ctx c, int type, bool can_skip, int mvx, int mvy, int mvdx, int mvdy) {
  const int lane = lane_id(), qp = sm.sd.qp;
  const Luma4 l4 = luma4x4_inter();
  uint32_t cbpl = l4.cbp;
  bool use8 = false;
  if (sm.fp.t8x8 && l4.cbp) {
    const uint32_t r8 = luma8x8_inter();
    if ((r8 >> 4) <= l4.nnz) { use8 = true; cbpl = r8 & 15u; }
  }
  const ChromaAc ac = chroma_quant(false);
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
    if (use8) recon_luma8x8((int)cbpl);
    else recon_luma4x4();
  }
  chroma_recon(cbpc);
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
// kHelp: the warp holds nothing but its segment, and takes part in its block's searches meanwhile.
__device__ void help_searches(unsigned* board);
template <bool kHelp = false>
__device__ __noinline__ bool wait_all(const int* p, int need, int& seen, int* error, unsigned long long timeout_ns, unsigned* board = nullptr) {
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
      if (kHelp && __shfl_sync(FULL, *(volatile unsigned*)board, 0)) {
        help_searches(board);
        t0 = global_ns();  // (the time limit is of waiting)
        continue;
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
  const int* ana;        // analysis progress per row of this picture, where macroblocks start before their
                         // neighbours are reconstructed; null: those are
  int* error;
  unsigned long long timeout_ns;
  unsigned* board;       // search forms: the block's open searches (help_searches); null: nobody helps
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

// A launch of few pictures is one chain of macroblocks, each waiting for its neighbours. What the next one
// needs first is only their vectors: its own reconstructed neighbours it reads after its motion search.
// So there a macroblock publishes its decision before its residual is coded, and one starts on its
// neighbours' decisions and waits for their reconstruction before the intra check. One 720p stream, 30
// pictures: 11.86 -> 10.2 ms.
//
// A macroblock's decision (vector and ref) for the neighbours that wait for it alone (StreamDev.dec): one
// 64-bit word that is its own flag, so neither side needs a fence.
__device__ __forceinline__ void decide(const Ctx c, int mv0, int mv1, int ref) {
  if (lane_id() == 0)
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(sm.sd.dec + c.mb), "l"((unsigned long long)(0x100u | (ref & 255)) << 32 | pack16(mv0, mv1)) : "memory");
}
// Waits until every lane's decision (p null: none) is there and returns it in w. False as wait_all.
__device__ __noinline__ bool wait_decided(const uint2* p, uint2& w, int* error, unsigned long long timeout_ns) {
  unsigned long long t0 = 0;
  bool ok = !p;
  while (true) {
    const int failed = lane_id() == 0 ? ld_relaxed(error) : 0;  // (in flight beside the decisions)
    if (!ok) {
      unsigned long long v;
      asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
      ok = (v >> 40) & 1u;
      w = make_uint2((uint32_t)v, (uint32_t)(v >> 32));
    }
    if (__all_sync(FULL, ok)) return true;
    if (!t0) t0 = global_ns();
    const bool late = lane_id() == 0 && global_ns() - t0 > timeout_ns;
    if (__any_sync(FULL, failed)) return false;
    if (__any_sync(FULL, late)) {
      if (lane_id() == 0) atomicCAS(error, 0, 1);
      return false;
    }
    __nanosleep(100);
  }
}
// Waits until the left and top neighbours (and the top-right one) are reconstructed, where the
// macroblock started before they were.
__device__ __noinline__ bool wait_recon(const Ctx c, const PipeWait pw) {
  if (sm.recon_seen) return true;
  const int* flag = lane_id() == 0 && c.mbx > 0 ? pw.ana + c.mby : nullptr;
  if (lane_id() == 1 && c.mby > 0) flag = pw.ana + c.mby - 1;
  int seen = -1;
  const bool ok = wait_all(flag, lane_id() == 0 ? c.mbx : min(c.mbx + 2, sm.fp.mb_w), seen, pw.error, pw.timeout_ns);
  if (lane_id() == 0) sm.recon_seen = 1;
  __syncwarp();
  return ok;
}

struct Bounds {
  int min0, min1, max0, max1;  // quarter samples (MvBounds, enc.rs:1105)
};
__device__ __forceinline__ bool in_bounds(const Bounds& b, int x, int y) {
  return x >= b.min0 && x <= b.max0 && y >= b.min1 && y <= b.max1;
}
__device__ __forceinline__ Bounds mv_bounds(int x0, int y0) {
  const int cw = sm.fp.mb_w * 16, ch = sm.fp.mb_h * 16;
  return {-4 * (x0 + 28), max(-4 * (y0 + 28), -2048), 4 * (cw - 16 - x0 + 28), min(4 * (ch - 16 - y0 + 28), 2044)};
}
__device__ __forceinline__ int lo16(int w) { return (int16_t)(w & 0xffff); }

// P_Skip probe (enc.rs:2906 try_p_skip) at skip vector (ps0, ps1): true when the macroblock is coded as
// P_Skip (prediction left in pred_y / pred_u / pred_v).
__device__ __noinline__ bool skip_probe(const Ctx c, int ps0, int ps1) {
  const StreamDev& sd = sm.sd;
  const int lane = lane_id();
  mc_luma16(c.mbx * 16, c.mby * 16, ps0, ps1);
  {
    const uint2 s = src8(), p = *(const uint2*)&sm.pred_y[lane * 8];
    const uint32_t dx = __vabsdiffu4(s.x, p.x), dy = __vabsdiffu4(s.y, p.y);
    const uint32_t sad = wsum(__dp4a(dx, 0x01010101u, __dp4a(dy, 0x01010101u, 0u)));
    if (sad >= sd.sb_probe) return false;
    if (sad > sd.sb_luma && wsum(__dp4a(dx, dx, __dp4a(dy, dy, 0u))) > sd.sb_luma_ssd && !probe_skip_luma()) return false;
  }
  mc_chroma8(sd.ref_u, sd.ref_v, sm.fp.stride_c, c.mbx, c.mby, ps0, ps1);
  // per plane SAD / SSD bounds (lanes 0..15 U, 16..31 V, 4 samples each)
  const uint32_t d = __vabsdiffu4(*(const uint32_t*)&sm.src_u[lane * 4], *(const uint32_t*)&sm.pred_u[lane * 4]);
  const uint32_t sad = __dp4a(d, 0x01010101u, 0u), ssd = __dp4a(d, d, 0u);
  const bool v = lane & 16;
  const uint32_t sads = wsum(v ? sad << 16 : sad), ssd_u = wsum(v ? 0u : ssd), ssd_v = wsum(v ? ssd : 0u);
  if (((sads & 0xffffu) <= sd.sb_chroma || ssd_u <= sd.sb_chroma_ssd) && ((sads >> 16) <= sd.sb_chroma || ssd_v <= sd.sb_chroma_ssd))
    return true;
  const ChromaAc ac = chroma_quant(false);
  return !ac.dc() && ac.score(0) < 7 && ac.score(1) < 7;
}

// This lane's SADs of the source (sv) against the predictions of the vectors (dx0, dy0) and (dx1, dy1)
// from the window's position, two to a word.
__device__ __forceinline__ uint32_t qpel_sad2(uint2 sv, int dx0, int dy0, int dx1, int dy1) {
  const uint32_t a = vsad8(sv, qpel8(dx0, dy0));
  return a | (vsad8(sv, qpel8(dx1, dy1)) << 16);
}

// One macroblock of a P slice (enc.rs:3011 code_p_mb). In the pipelined mode (pw.db_prev) it first
// waits for the reference frame to be final over every sample its search can read; when a wait
// gives up it returns false and writes nothing.
// kEarly: it starts on its neighbours' decisions, and publishes its own before the residual.
template <bool kEarly>
__device__ __noinline__ bool analyse_p_mb(const Ctx c, const PipeWait pw) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  const int lane = lane_id(), mbx = c.mbx, mby = c.mby, x0 = mbx * 16, y0 = mby * 16;
  const uint32_t lambda = sm.qt[0].lambda;
  const Bounds bd = mv_bounds(x0, y0);
  // neighbours (this picture) and the co-located macroblock of the previous one, a lane each: left,
  // top, top-right (top-left where that is absent), co-located; ref -2 when absent
  int nb = -1;
  if (lane == 0 && mbx > 0) nb = c.mb - 1;
  if (lane == 1 && mby > 0) nb = c.mb - fp.mb_w;
  if (lane == 2 && mby > 0 && fp.mb_w > 1) nb = c.mb - fp.mb_w + (mbx + 1 < fp.mb_w ? 1 : -1);
  if (lane == 3) nb = c.mb;
  uint2 nw = make_uint2(0u, 0xfeu);
  load_source(c);
  // While the neighbours decide: what zero motion reads of the reference picture, which is waited for
  // in any case, and its lines into the L1.
  if (kEarly && pw.db_prev) {
    if (!wait_reference(c, pw, (x0 + 44) >> 4, (y0 + 40) >> 4)) return false;
    if (lane < 26) {
      const uint8_t* p = sd.ref_y + (long)(y0 - 5 + lane) * fp.stride_y + x0 - 8;
      asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
      if (((uintptr_t)p ^ (uintptr_t)(p + 31)) & 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 31));
    }
  }
  const uint2* const dec = !kEarly ? nullptr : (lane == 3 ? sd.prev_dec : sd.dec);
  if (kEarly && !wait_decided(nb >= 0 && dec ? dec + nb : nullptr, nw, pw.error, pw.timeout_ns)) return false;
  if (nb >= 0 && !dec) nw = *(const uint2*)&(lane == 3 ? sd.prev_info : sd.info)[nb];
  const int va = __shfl_sync(FULL, (int)nw.x, 0), vb = __shfl_sync(FULL, (int)nw.x, 1), vc = __shfl_sync(FULL, (int)nw.x, 2),
            vp = __shfl_sync(FULL, (int)nw.x, 3);
  const int ref = (int8_t)(nw.y & 255u);
  const uint32_t inter = __ballot_sync(FULL, ref == 0) & 7u, absent = __ballot_sync(FULL, ref == -2) & 7u;
  // pred_motion_partition (h264.rs:3577), 16x16, ref 0: the only inter neighbour, the left one when
  // it is the only one there is, else the median
  int mvp;
  {
    auto med = [](int x, int y, int z) { return min(max(x, y), max(min(x, y), z)); };
    mvp = (int)pack16(med(lo16(va), lo16(vb), lo16(vc)), med(va >> 16, vb >> 16, vc >> 16));
    if (inter == 1u || (inter == 0u && absent == 6u)) mvp = va;
    if (inter == 2u) mvp = vb;
    if (inter == 4u) mvp = vc;
  }
  const int ps = mbx == 0 || mby == 0 || ((inter & 1u) && va == 0) || ((inter & 2u) && vb == 0) ? 0 : mvp;
  const int mvp0 = lo16(mvp), mvp1 = mvp >> 16, ps0 = lo16(ps), ps1 = ps >> 16;
  // Full-pel candidates (enc.rs:3084-3105): predictor, zero, left (if any), top (if any) and the
  // co-located vector of the previous picture, rounded and clamped; lane k holds candidate k.
  const int imin0 = (bd.min0 + 3) >> 2, imin1 = (bd.min1 + 3) >> 2, imax0 = bd.max0 >> 2, imax1 = bd.max1 >> 2;
  int cx, cy;
  {
    const int v = lane == 1 ? 0 : (lane == 2 ? va : (lane == 3 ? vb : (lane == 4 ? vp : mvp)));
    cx = min(max((lo16(v) + 2) >> 2, imin0), imax0);
    cy = min(max(((v >> 16) + 2) >> 2, imin1), imax1);
  }
  if (pw.db_prev) {
    // The right- and bottom-most reference sample this macroblock can read: the full-pel
    // candidates, a diamond of at most 16 steps around the best, the half-sample window
    // (-3..+20) and 8-byte loads. Everything above and to the left of it (padding included) is
    // final once the macroblock holding it is.
    const int hi0 = __reduce_max_sync(FULL, cx), hi1 = __reduce_max_sync(FULL, cy);
    if (!wait_reference(c, pw, (x0 + hi0 + 44) >> 4, (y0 + hi1 + 40) >> 4)) return false;
  }
  if (lane == 0) sm.win_x = kNoWin;  // the last macroblock's window
  __syncwarp();

  // 1. skip probe
  if (in_bounds(bd, ps0, ps1) && skip_probe(c, ps0, ps1)) {
    if (kEarly) decide(c, ps0, ps1, 0);
    code_skip(c, ps0, ps1);
    return true;
  }

  // 2. motion search (enc.rs:3084-3117): the first of the cheapest candidates
  const int stride = fp.stride_y;
  const uint2 sv = src8();
  const uint8_t* base = sd.ref_y + (long)(y0 + (lane >> 1)) * stride + x0 + (lane & 1) * 8;
  int best0, best1;
  uint32_t best_cost;
  {
    const int at = cy * stride + cx;
    uint2 r[5];
#pragma unroll
    for (int k = 0; k < 5; k++) r[k] = ldg8(base + __shfl_sync(FULL, at, k));
    const uint32_t s01 = wsum(vsad8(sv, r[0]) | (vsad8(sv, r[1]) << 16)), s23 = wsum(vsad8(sv, r[2]) | (vsad8(sv, r[3]) << 16)),
                   s4 = wsum(vsad8(sv, r[4]));
    const uint32_t w = lane < 2 ? s01 : (lane < 4 ? s23 : s4);
    const uint32_t cost = ((w >> (16 * (lane & 1))) & 0xffffu) + mvd_cost(cx * 4 - mvp0, lambda) + mvd_cost(cy * 4 - mvp1, lambda);
    const bool use = lane < 5 && (lane != 2 || mbx > 0) && (lane != 3 || mby > 0);
    const uint32_t key = __reduce_min_sync(FULL, use ? (cost << 3) | (uint32_t)lane : UMAX);
    best_cost = key >> 3;
    best0 = __shfl_sync(FULL, cx, (int)(key & 7u));
    best1 = __shfl_sync(FULL, cy, (int)(key & 7u));
  }
  // diamond (enc.rs:1207-1272): up, left, right, down around the best, first strict minimum
  // wins; each step's four loads are issued together (a neighbour past the bounds is still inside
  // the padded picture, and not counted)
  const Box ibox{4 * imin0, 4 * imax0, 4 * imin1, 4 * imax1};
#pragma unroll 1
  for (int it = 0; it < 16; it++) {
    const uint8_t* cp = base + best1 * stride + best0;
    const uint2 u = ldg8(cp - stride), l = ldg8(cp - 1), r = ldg8(cp + 1), d = ldg8(cp + stride);
    const uint32_t key = best4(vsad8(sv, u) | (vsad8(sv, l) << 16), vsad8(sv, r) | (vsad8(sv, d) << 16), 4 * best0, 4 * best1, 4, ibox,
                               mvp0, mvp1, lambda, false);
    if ((key >> 2) >= best_cost) break;
    best_cost = key >> 2;
    const int k = (int)(key & 3u);
    best0 += k == 1 ? -1 : (k == 2 ? 1 : 0);
    best1 += k == 0 ? -1 : (k == 3 ? 1 : 0);
  }
  int mv0 = best0 * 4, mv1 = best1 * 4;
  {
    uint2 v = ldg8(base + best1 * stride + best0);
    if (wsum(vsad8(sv, v)) > sd.sb_luma) {
      // sub-pel refinement over a half-sample window around the full-pel best (enc.rs:1283): a
      // half-sample diamond step, then up to two quarter-sample ones. The steps from the full-pel
      // position itself never read plane j.
      ensure_window(x0 + best0, y0 + best1, 3);
      const Box box{max(bd.min0, mv0 - 3), min(bd.max0, mv0 + 3), max(bd.min1, mv1 - 3), min(bd.max1, mv1 + 3)};
      int q0 = 0, q1 = 0;  // from the full-pel best
#pragma unroll 1
      for (int it = 0; it < 3; it++) {
        const int st = it == 0 ? 2 : 1;
        if (it == 1 && (q0 | q1)) ensure_window(x0 + best0, y0 + best1, 7);
        const uint32_t s01 = qpel_sad2(sv, q0, q1 - st, q0 - st, q1), s23 = qpel_sad2(sv, q0 + st, q1, q0, q1 + st);
        const uint32_t key = best4(s01, s23, mv0 + q0, mv1 + q1, st, box, mvp0, mvp1, lambda, false);
        if ((key >> 2) < best_cost) {
          best_cost = key >> 2;
          const int k = (int)(key & 3u);
          q0 += k == 1 ? -st : (k == 2 ? st : 0);
          q1 += k == 0 ? -st : (k == 3 ? st : 0);
        } else if (it) {
          break;
        }
      }
      v = qpel8(q0, q1);
      mv0 += q0;
      mv1 += q1;
    }
    *(uint2*)&sm.pred_y[lane * 8] = v;
    __syncwarp();
  }

  // 3. intra 16x16 when the inter prediction is poor (enc.rs:3121-3156)
  const uint32_t inter_satd = satd16((int)offsetof(Smem, pred_y));
  if (inter_satd > 24 * lambda) {
    if (kEarly && !wait_recon(c, pw)) return false;
    const Corner k0 = load_edges(c, false);
    const bool ht = mby > 0, hl = mbx > 0;
    const I16Fit fit16 = analyse_i16(ht, hl, k0.y);
    if (fit16.cost + lambda * 8 < inter_satd + lambda * (se_bits(mv0 - mvp0) + se_bits(mv1 - mvp1) + 1)) {
      if (kEarly) decide(c, 0, 0, -1);
      code_i16(c, fit16.mode, ht, hl, k0);
      return true;
    }
  }

  // 4. P_L0_16x16 residual, record and reconstruction
  if (kEarly) decide(c, mv0, mv1, 0);
  mc_chroma8(sd.ref_u, sd.ref_v, fp.stride_c, mbx, mby, mv0, mv1);
  code_inter(c, RG_MB_P_L0_16X16, mv0 == ps0 && mv1 == ps1, mv0, mv1, mv0 - mvp0, mv1 - mvp1);
  return true;
}

// ---------------------------------------------------------------------------------------------
// The full-search and learned forms' analysis (neither exists in the reference).
#include "search_form.cuh"

// ---------------------------------------------------------------------------------------------
// Deblocking of one macroblock (enc.rs:3776 deblock, h264_deblock.rs:71,187): vertical edges, then
// horizontal ones, on tiles in shared memory with 4 samples of the left / top neighbours. Lanes 0..15
// own a luma line across the edges (row, then column), lanes 16..31 a chroma line of either plane;
// a lane's edges in one direction follow one another without a barrier, and one rolled copy of the
// filter serves every edge, both directions, luma and chroma, both strengths. (Every lane computing
// every edge's parameters, the filters unrolled: 12.2 k cycles a macroblock on an idle SM.)
constexpr int kDbY = 24, kDbC = 12;       // tile strides: luma rows from x = -4 at byte 4, chroma rows from x = -4
constexpr int kDbPlane = 12 * kDbC;       // a chroma tile
// nz16 (decoding order) as a raster mask: bit 4 y + x.
__device__ __forceinline__ uint32_t raster_nz(uint32_t nz) {
  const uint32_t t = (nz ^ (nz >> 2)) & 0x0c0cu;
  return (nz ^ t ^ (t << 2)) & 0xffffu;
}
__device__ __forceinline__ bool far_mv(uint32_t a, uint32_t b) {
  return abs(lo16((int)a) - lo16((int)b)) >= 4 || abs(((int)a >> 16) - ((int)b >> 16)) >= 4;
}
// kMv4 (search forms): the motion term of the strengths compares the quadrant vectors on either side of
// each 4-sample segment, so the internal edge between partitions gets strength 1 where their vectors
// differ by 4 quarter samples.
template <bool kMv4>
__device__ __noinline__ void deblock_mb(int mbx, int mby) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  const int lane = lane_id(), m = mby * fp.mb_w + mbx;
  const bool hasl = mbx > 0, hast = mby > 0;
  // the macroblocks' state: words mv, ref | flags << 8 | cbp << 16 | qp << 24, nz | ..
  const uint4 q = *(const uint4*)&sd.info[m];
  const uint4 l = hasl ? *(const uint4*)&sd.info[m - 1] : q, t = hast ? *(const uint4*)&sd.info[m - fp.mb_w] : q;
  // the tiles: lane = luma row (20 from y = -4), and chroma row (12 of either plane from y = -4)
  uint8_t* gy = sd.cur_y + (long)(mby * 16 - 4 + lane) * fp.stride_y + mbx * 16;
  const int cp = lane >= 12, cr = lane - 12 * cp;
  uint8_t* gc = (cp ? sd.cur_v : sd.cur_u) + (long)(mby * 8 - 4 + cr) * fp.stride_c + mbx * 8;
  const bool ly = lane < 20 && (lane >= 4 || hast), lc = lane < 24 && (cr >= 4 || hast);
  const bool ly4 = ly && lane >= 4 && hasl, lc4 = lc && cr >= 4 && hasl;  // with the left neighbour's samples
  uint4 wy = make_uint4(0u, 0u, 0u, 0u);
  uint2 wc = make_uint2(0u, 0u);
  uint32_t wy4 = 0, wc4 = 0;
  if (ly) wy = *(const uint4*)gy;
  if (ly4) wy4 = *(const uint32_t*)(gy - 4);
  if (lc) wc = *(const uint2*)gc;
  if (lc4) wc4 = *(const uint32_t*)(gc - 4);
  auto intra = [](const uint4& i) { return (i.y >> 8) & kFlagIntra; };
  auto quiet = [](const uint4& i) { return ((i.y >> 8) & kFlagIntra) == 0 && ((i.y >> 16) & 255u) == 0; };
  bool split = false;
  if constexpr (kMv4) {
    const uint4 qm = *(const uint4*)&sd.mv4[m];
    const uint4 lm = hasl ? *(const uint4*)&sd.mv4[m - 1] : qm, tm = hast ? *(const uint4*)&sd.mv4[m - fp.mb_w] : qm;
    auto same = [&](const uint4& v) { return v.x == qm.x && v.y == qm.x && v.z == qm.x && v.w == qm.x; };
    split = !same(qm);
    if (quiet(q) && !split && quiet(l) && same(lm) && quiet(t) && same(tm)) return;
    __syncwarp();
    if (lane < 3) *(uint4*)&sm.dbmv[4 * lane] = lane == 0 ? qm : (lane == 1 ? lm : tm);
  } else {
    if (quiet(q) && quiet(l) && l.x == q.x && quiet(t) && t.x == q.x) return;
  }
  uint8_t* const ty = sm.win;
  uint8_t* const tc = sm.hp[0];
  if (ly) {
    *(uint32_t*)&ty[lane * kDbY + 4] = wy4;
    *(uint2*)&ty[lane * kDbY + 8] = make_uint2(wy.x, wy.y);
    *(uint2*)&ty[lane * kDbY + 16] = make_uint2(wy.z, wy.w);
  }
  if (lc) {
    uint32_t* r = (uint32_t*)&tc[lane * kDbC];
    r[0] = wc4;
    r[1] = wc.x;
    r[2] = wc.y;
  }
  __syncwarp();
  // this lane's line: luma line lane, or line lane & 7 of chroma plane (lane >> 3) & 1; segment k of four
  const bool luma = lane < 16;
  const int line = luma ? lane : lane & 7, k = luma ? lane >> 2 : line >> 1;
  const int xy = luma ? kDbY : kDbC;  // row stride of its tile
  uint8_t* const origin = luma ? ty + 4 * kDbY + 8 : tc + ((lane >> 3) & 1) * kDbPlane + 4 * kDbC + 4;
  const int qp = (int)(q.y >> 24), qpc = chroma_qp(qp);
  auto thresholds = [&](const uint4& p) {  // of an edge between q and p
    const int pq = (int)(p.y >> 24);
    return c_deblock[luma ? (qp + pq + 1) >> 1 : (qpc + chroma_qp(pq) + 1) >> 1];
  };
  const uint2 th_in = thresholds(q);
  const uint32_t qz = raster_nz(q.z);
  const bool internal = intra(q) || ((q.y >> 16) & 255u) != 0 || split;
  const int step = !internal ? 4 : (((q.y >> 8) & kFlagT8) ? 2 : 1);
#pragma unroll 1
  for (int dir = 0; dir < 2; dir++) {
    const uint4& p = dir ? t : l;
    const bool has = dir ? hast : hasl;
    const uint2 th_p = thresholds(p);
    const uint32_t pz = raster_nz(p.z);
    const int along = dir ? 1 : xy, xs = dir ? xy : 1;
    uint8_t* const base = origin + line * along;
#pragma unroll 1
    for (int e = has ? 0 : step; e < 4; e += step) {
      const bool edge = e == 0;  // between macroblocks
      int bs;
      if (intra(q) || (edge && intra(p))) {
        bs = edge ? 4 : 3;
      } else {
        const int qb = dir ? 4 * e + k : 4 * k + e;  // the block on either side
        const uint32_t coded = (qz >> qb) | (edge ? pz >> (dir ? 12 + k : 4 * k + 3) : qz >> (dir ? qb - 4 : qb - 1));
        bool motion;
        if constexpr (kMv4) {
          const int qq = dir ? (e >> 1) * 2 + (k >> 1) : (k >> 1) * 2 + (e >> 1), e1 = (e - 1) >> 1;
          const int pq = edge ? (dir ? 8 + 2 + (k >> 1) : 4 + (k >> 1) * 2 + 1) : (dir ? e1 * 2 + (k >> 1) : (k >> 1) * 2 + e1);
          motion = (edge && ((q.y ^ p.y) & 255u)) || far_mv(sm.dbmv[qq], sm.dbmv[pq]);
        } else {
          motion = edge && (((q.y ^ p.y) & 255u) || far_mv(q.x, p.x));
        }
        bs = (coded & 1u) ? 2 : (motion ? 1 : 0);
      }
      if (!luma && (e & 1)) bs = 0;
      if (bs) {
        const uint2 th = edge ? th_p : th_in;
        const int alpha = (int)(th.x & 255u), beta = (int)(th.x >> 8);
        uint8_t* const o = base + (luma ? 4 * e : 2 * e) * xs;
        const int p0 = o[-xs], q0 = o[0], p1 = o[-2 * xs], q1 = o[xs], p2 = o[-3 * xs], q2 = o[2 * xs];
        if (abs(p0 - q0) < alpha && abs(p1 - p0) < beta && abs(q1 - q0) < beta) {
          const bool ap = luma && abs(p2 - p0) < beta, aq = luma && abs(q2 - q0) < beta;
          if (bs < 4) {
            const int tc0 = (int)((th.y >> (8 * (bs - 1))) & 255u), tcc = tc0 + (luma ? (int)ap + (int)aq : 1);
            const int d = min(max((((q0 - p0) << 2) + (p1 - q1) + 4) >> 3, -tcc), tcc), a = (p0 + q0 + 1) >> 1;
            o[-xs] = (uint8_t)clip255(p0 + d);
            o[0] = (uint8_t)clip255(q0 - d);
            if (ap) o[-2 * xs] = (uint8_t)(p1 + min(max((p2 + a - (p1 << 1)) >> 1, -tc0), tc0));
            if (aq) o[xs] = (uint8_t)(q1 + min(max((q2 + a - (q1 << 1)) >> 1, -tc0), tc0));
          } else {
            const bool small = abs(p0 - q0) < ((alpha >> 2) + 2);
            const int p3 = o[-4 * xs], q3 = o[3 * xs];
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
      }
      __syncwarp();
    }
    __syncwarp();
  }
  // write back the samples this macroblock filters (rows 0..15 x cols -4..15, rows -4..-1 x cols 0..15)
  if (ly) {
    const uint2 a = *(const uint2*)&ty[lane * kDbY + 8], b = *(const uint2*)&ty[lane * kDbY + 16];
    *(uint4*)gy = make_uint4(a.x, a.y, b.x, b.y);
    if (ly4) *(uint32_t*)(gy - 4) = *(const uint32_t*)&ty[lane * kDbY + 4];
  }
  if (lc) {
    const uint32_t* r = (const uint32_t*)&tc[lane * kDbC];
    *(uint2*)gc = make_uint2(r[1], r[2]);
    if (lc4) *(uint32_t*)(gc - 4) = r[0];
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
      else analyse_p_mb<false>(c, none);
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
  int grid;           // warps that take segments
  int meet_ns;        // limit of a meeting of a block's warps (meet), 0: they do not wait for each other
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

// Sixteen warps per SM, one block: up to 128 registers a thread, so nothing spills.
constexpr int kBlockWarps = 16;

// The warps of an SM run the same code on different macroblocks, and the code is several times the
// SM's instruction cache: with every warp somewhere else in it, the cache that the SMs of a group
// share behind theirs was busy all the time (0.44 lines a cycle), and a macroblock took three times as
// long as on an idle SM. So the warps of a block (one block an SM) start their macroblocks together:
// most of what one of them fetches is then still there for the other fifteen. A warp that has finished
// its segment waits here until the others have finished theirs, for at most `limit` ns (a long
// macroblock's time): one that waits for another SM's macroblock holds nobody for long, and no wait
// of the schedule depends on a meeting. 1080p 8 x 15 launch: 34.9 ms without, 24.1 with 30 us, 21.5 with
// 60, 21.2 with 120; learned 1080p 8 x 8 (macroblocks three times as long) 53 with 100 us, 44.6 with 400 and
// with 1 ms. round: the arrivals that complete this warp's round.
constexpr int kMeetNs = 120000, kMeetNsSearch = 400000;
__device__ __forceinline__ void meet(int* arrived, int round, int limit) {
  if (lane_id() == 0) {
    int n = atomicAdd(arrived, 1) + 1;
    if (n < round && limit) {
      const unsigned long long t0 = global_ns();
      do {
        __nanosleep(200);
        n = *(volatile int*)arrived;
      } while (n < round && global_ns() - t0 < limit);
    }
  }
  __syncwarp();
}

template <int kForm, bool kEarly>
__global__ void __launch_bounds__(32 * kBlockWarps, 1) pipeline_kernel(const __grid_constant__ FrameGroups fg, const StreamDev* __restrict__ sds, PipeParams pp) {
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
  uint32_t empty = (pp.qbeg[0] >= pp.qend[0] ? 1u : 0u) | (pp.qbeg[1] >= pp.qend[1] ? 2u : 0u) | (pp.qbeg[2] >= pp.qend[2] ? 4u : 0u);
  __shared__ unsigned board;  // search forms: warps whose search others may take part in
  __shared__ int arrived;  // warps that have finished a segment, all rounds together
  int round = 0;
  if (threadIdx.y == 0 && lane == 0) {
    arrived = 0;
    board = 0;
  }
  if constexpr (kForm != 0)
    if (lane == 0) {
      ss.job.ticket = kNoJob;
      ss.job.failed = false;
    }
  if (lane == 0) sm.reach_y = sm.reach_x = 0;  // this warp's, published once as it exits
  int group = -1;                              // whose parameters sm.fp holds
  __syncthreads();
  bool failed = (int)(blockIdx.x * blockDim.y + threadIdx.y) >= pp.grid;  // a warp past the grid takes nothing
  while (!failed) {
    int t = -1;
    if (lane == 0) {
      for (int k = 0; k < 3 && t < 0; k++) {
        const int q = role + k >= 3 ? role + k - 3 : role + k;
        if ((empty >> q) & 1u) continue;
        const int v = pp.qbeg[q] + atomicAdd(pp.ticket + (q ? q + 1 : 0), 1);
        if (v < pp.qend[q]) t = v; else empty |= 1u << q;
      }
    }
    t = __shfl_sync(FULL, t, 0);
    if (t < 0) break;
    const int2 task = __ldg(pp.tasks + t);
    if (__shfl_sync(FULL, ld_relaxed(pp.error), 0)) break;  // (both loads in flight together)
    const int ps = task.x;
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
    int seen = 0;  // of this lane's counter (wait_all)
    if (ana) {
      const bool has_prev = sd.prev_rows >= 0 && sd.kind == RG_FRAME_P;
      const bool early = kEarly && sd.kind == RG_FRAME_P;
      const PipeWait pw{has_prev ? pp.db + sd.prev_rows : nullptr, early ? ana_rows : nullptr, pp.error, pp.timeout_ns, kForm != 0 ? &board : nullptr};
      if (lane == 0) sm.db_row = -1;
      // lane 0: the previous segment of this row; lane 1: the row above two macroblocks ahead; lane 2
      // (plain form): the co-located macroblock of the previous picture, whose vector is a candidate
      // (early: analyse_p_mb waits for their decisions instead)
      const int* flag = lane == 0 && x0 > 0 ? ana_rows + y : nullptr;
      if (lane == 1 && y > 0) flag = ana_rows + y - 1;
      if (kForm == 0 && lane == 2 && has_prev) flag = pp.ana + sd.prev_rows + y;
      if (early) flag = nullptr;
      for (int x = x0; x < x1; x++) {
        if (!wait_all<kForm != 0>(flag, lane == 0 ? x0 : (lane == 1 ? min(x + 2, Wm) : x + 1), seen, pp.error, pp.timeout_ns, &board)) {
          failed = true;
          break;
        }
        Ctx c{x, y, y * Wm + x};
        if (sd.kind == RG_FRAME_IDR) {
          load_source(c);
          if constexpr (kForm != 0) analyse_intra_mb_search(c);
          else analyse_intra_mb(c);
          if constexpr (kEarly) decide(c, 0, 0, -1);
        } else {
          if (kEarly && lane == 0) sm.recon_seen = 0;
          if constexpr (kForm != 0) failed = !analyse_p_mb_search(c, pw);
          else failed = !analyse_p_mb<kEarly>(c, pw) || (kEarly && !wait_recon(c, pw));  // (the row's progress counts the left one)
          if (failed) break;
          if constexpr (kForm != 0)
            if (*(volatile bool*)&ss.job.failed) {  // (nothing of it is published)
              failed = true;
              break;
            }
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
        if (!wait_all<kForm != 0>(flag, lane == 3 ? x0 : min(x + (lane == 1 ? 1 : 2), Wm), seen, pp.error, pp.timeout_ns, &board)) {
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
      // the last row's last macroblock comes after every other of the picture
      if (!failed && y == H - 1 && x1 == Wm && sd.done && lane == 0) st_release_sys(sd.done, pp.seq);
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
    round += blockDim.y;
    meet(&arrived, round, ana ? pp.meet_ns : 0);  // (the deblocking code fits the cache by itself)
  }
  // whoever is left need not wait for this warp any more
  if (lane == 0) atomicAdd(&arrived, 1 << 26);
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
  QTab qt[52];
  for (int qp = 0; qp < 52; qp++) {
    QTab& t = qt[qp];
    const int rem = qp % 6, d = qp / 6;
    const uint16_t* m = kMf4[rem];
    const uint8_t* k = kDq4[rem];
    t.mf[0][0] = m[0]; t.mf[0][1] = t.mf[1][0] = m[2]; t.mf[1][1] = m[1];
    t.dq[0][0] = k[0] << d; t.dq[0][1] = t.dq[1][0] = k[2] << d; t.dq[1][1] = k[1] << d;
    t.shift = 15 + d;
    t.bias[0] = (1u << t.shift) / 6u;
    t.bias[1] = (1u << t.shift) / 3u;
    t.dc_mf = m[0];
    t.dc_dq = (k[0] * 16) << (d + 2);
    t.lambda = kLambda[qp];
    const int cls[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
    for (int x = 0; x < 3; x++)
      for (int y = 0; y < 3; y++) {
        t.mf8[x][y] = kMf8[rem][cls[x][y]];
        t.dq8[x][y] = kDq8[rem][cls[x][y]] << (d >= 2 ? d - 2 : 0);
      }
    t.bias8 = (1u << (16 + d)) / 6u;
    t.rnd8 = d >= 2 ? 0 : 1 << (1 - d);
    t.sh8 = d >= 2 ? 0 : 2 - d;
  }
  cudaMemcpyToSymbol(g_qtab, qt, sizeof(qt));
  cudaMemcpyToSymbol(c_cqp, kChromaQp, sizeof(kChromaQp));
  uint2 db[52];
  for (int qp = 0; qp < 52; qp++)
    db[qp] = make_uint2(kAlpha[qp] | (kBeta[qp] << 8), kTc0[qp][0] | (kTc0[qp][1] << 8) | (kTc0[qp][2] << 16));
  cudaMemcpyToSymbol(c_deblock, db, sizeof(db));
  uint2 taps[18];
  for (int m = 0; m < 9; m++)
    for (int h = 0; h < 2; h++) {
      uint32_t w[2] = {0u, 0u};
      for (int r = 0; r < 2; r++)
        for (int x = 0; x < 4; x++) {
          const int v = i4_tap(m, x, r ? 3 - h : h);
          w[r] |= (uint32_t)((v >> 8) * 16 + (v & 255)) << (8 * x);
        }
      taps[2 * m + h] = make_uint2(w[0], w[1]);
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

// Shared memory of a warp of the analysis kernels.
static size_t warp_smem(int form) { return sizeof(Smem) + (form ? sizeof(SearchSmem) : 0); }

void launch_wavefront_step(const FrameParams& fp, const StreamDev* d_streams, int step, cudaStream_t st, int form) {
  dim3 grid(2 * max_diag_len(fp), fp.n_streams);
  if (form) wavefront_step_kernel<1><<<grid, 32, warp_smem(1), st>>>(fp, d_streams, step);
  else wavefront_step_kernel<0><<<grid, 32, warp_smem(0), st>>>(fp, d_streams, step);
}

int pipeline_sms(int device) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

// Resident warps of the pipelined mode: a block of sixteen on every SM (launch time of 1080p 8 x 15
// pictures by the warps an SM, before they met: 6 45.1 ms, 8 40.8, 10 38.7, 12 36.9, 14 35.6, 16 34.9).
int pipeline_grid(int device) { return kBlockWarps * pipeline_sms(device); }

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

int pipeline_key_span(const FrameParams& fp, int frames, int lag, int seg) {
  const int a = seg > 2 ? seg : 2;
  return a * fp.mb_h + fp.mb_w + lag * (frames - 1);
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

// Meetings pay where there is work for enough warps, and cost a little where the launch is one chain of
// macroblocks and they wait anyway. The measure is the segments ready side by side (both roles: all of them
// over the span of their keys) for each warp; launch times apart -> meeting, 2368 warps (in the plain form a
// launch whose warps stay apart also starts macroblocks early, so both sides differ by that too):
//   plain (720p, 1080p, 360p High, 2 to 15 pictures): 0.05 7.2 -> 9.1 ms, 0.10 8.8 -> 9.8, 0.127 8.13 -> 8.03,
//     0.14 10.9 -> 10.5, 0.19 13.1 -> 11.5, 0.24 14.6 -> 12.0, 0.38 18.8 -> 13.8;
//   learned (360p to 4K): 0.06 15.4 -> 15.6, 0.10 12.0 -> 12.2, 0.12 18.5 -> 17.9, 0.18 22.9 -> 20.6, 0.30 46.5 -> 38.6;
//   IDR pictures alone: 0.12 3.7 -> 3.9, 0.18 3.90 -> 3.98, 0.215 12.1 -> 12.3, 0.233 4.14 -> 4.08, 0.36 4.7 -> 4.3;
//   single pictures, IDR and P side by side: 0.054 3.52 -> 3.59, 0.072 2.10 -> 1.90, 0.08 11.7 -> 11.1, 0.107 13.5 -> 11.6;
//   full search (its searches are shared by the warps that wait instead): 0.06 22.1 -> 23.3, 0.24 34.2 -> 38.9,
//     0.37 99 -> 108, 0.44 92.6 -> 88.7, 0.48 56.2 -> 51.9.
// So the lines lie at 1/8, at 2/9 for IDR pictures alone, at 1/14 for single pictures of both kinds (the code
// of both is then fetched all along) and at 2/5 for the full search.
PictureMix picture_mix(const int32_t* kinds, int streams, int frames) {
  const int n = streams * frames;
  int idr = 0;
  for (int i = 0; i < n; i++) idr += kinds[i] == RG_FRAME_IDR;
  return idr == n ? PictureMix::kIdr : (frames == 1 && idr ? PictureMix::kSingles : PictureMix::kGops);
}
bool pipeline_meets(size_t n_tasks, int grid, int key_span, int form, PictureMix mix) {
  const size_t ready = n_tasks / 2, warps = (size_t)grid * (size_t)key_span;
  if (form == RG_FORM_FULLSEARCH) return 5 * ready >= 2 * warps;
  if (mix == PictureMix::kIdr) return 9 * ready >= 2 * warps;
  return (mix == PictureMix::kSingles ? 14 : 8) * ready >= warps;
}

void launch_pipeline(const FrameGroups& fg, const StreamDev* d_streams, int n_desc, int total_rows, int* counters,
                     const int2* d_tasks, size_t n_tasks, bool meet, const int qbeg[3], const int qend[3], int deblock_sms,
                     int intra_sms, int sms, int seg, int grid, unsigned long long timeout_ns, int* ready, int seq,
                     int* host_err, int* host_reach, cudaStream_t st, int form, const CompactOut* co, bool early) {
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
  pp.meet_ns = meet ? (form ? kMeetNsSearch : kMeetNs) : 0;
  // spread over the SMs, then up to a block's warps on each
  pp.grid = grid < pp.n_tasks ? grid : pp.n_tasks;
  int warps = (pp.grid + sms - 1) / sms;
  if (warps > kBlockWarps) warps = kBlockWarps;
  const int g = (pp.grid + warps - 1) / warps;
  pp.role_by_sm = g >= sms;
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
  const dim3 block(32, warps);
  const size_t smem = warps * warp_smem(form);
  const auto kernel = form ? pipeline_kernel<1, false> : (early ? pipeline_kernel<0, true> : pipeline_kernel<0, false>);
  // (a whole block's, whatever this launch takes: contexts of other threads launch the same kernel)
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kBlockWarps * warp_smem(form)));
  kernel<<<g, block, smem, st>>>(fg, d_streams, pp);
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
