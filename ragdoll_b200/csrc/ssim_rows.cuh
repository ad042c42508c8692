// SSIM rows and the 2x2 pyramid of plane pairs (included by ssim_kernels.cu and ssim_noalloc.cu, each
// inside its own namespace; compiled without fused multiply-add). The reference's arithmetic:
//   crates/ragdoll-simd/src/metrics.rs:417  ssim_end1_8bit: integer sums, two f32 products, one
//                                           f32 division
//   crates/ragdoll-simd/src/metrics.rs:667  row_ssim: sequential f32 sum over the windows of a row
//   crates/ragdoll-simd/src/metrics.rs:675  total: f64 sum of the rows in order
//   crates/ragdoll-pix/src/metrics.rs:87    decimate_2x2_u8: (a + b + c + d + 2) >> 2
// Two launches measure a pair at every scale: one reads the full planes once, writes the SSIM of its
// window rows and all four pyramid levels; the other measures the levels. Bound by the planes' bytes
// for many pairs, by the chain load - window values - ordered sums of one strip for few.

constexpr int kSsimC1 = 416;
constexpr int kSsimC2 = 235963;
constexpr int kRowThreads = 256;
// A block has kStrip window rows (kStrip + 1 rows of 4x4 blocks) and walks them kChunk windows at a
// time. Many pairs: strips of 16 rows, each row of blocks read 1.06 times. Few pairs leave most SMs
// without a strip, so that one strip's latency is the launch: strips of 4 rows, 256 windows at a time
// (640x360, every scale: 39.9 us a call with tall strips, 24.6 with flat ones).
constexpr int kTallStrip = 16, kTallChunk = 64, kFlatStrip = 4, kFlatChunk = 256;

// One scale of a plane pair: rows receives an f32 per window row.
struct SsimLevel {
  const uint8_t* a;
  const uint8_t* b;
  long sa, sb;
  int w, h;
  float* rows;
};
// A plane pair: levels 1 .. levels - 1 are pyramid planes written by the pass over level 0 (their
// strides are multiples of 4, their bases 4-byte aligned). out: the f64 SSIM of every level.
struct SsimPair {
  SsimLevel lv[5];
  int levels;
  double* out;
};

__device__ __forceinline__ float ssim_end1(int s1, int s2, int ss, int s12) {
  int vars = ss * 64 - s1 * s1 - s2 * s2;
  int covar = s12 * 64 - s1 * s2;
  float num = __fmul_rn(__int2float_rn(2 * s1 * s2 + kSsimC1), __int2float_rn(2 * covar + kSsimC2));
  float den = __fmul_rn(__int2float_rn(s1 * s1 + s2 * s2 + kSsimC1), __int2float_rn(vars + kSsimC2));
  return __fdiv_rn(num, den);
}

// Strips of a plane of height h: its window rows, and with the pyramid its rows of 4x4 blocks.
__host__ __device__ __forceinline__ int ssim_strips(int h, bool pyramid, int strip) {
  const int rows = pyramid ? (h + 3) / 4 : (h >> 2) - 1;
  return rows > 0 ? (rows + strip - 1) / strip : 0;
}

template <int kStrip, int kChunk>
struct RowsSmem {
  int4 sums[(kStrip + 1) * (kChunk + 1)];  // per 4x4 block: sum a, sum b, sum a a + b b, sum a b
  float vals[kStrip * (kChunk + 1)];       // the chunk's window values
  uint8_t p2[2][kStrip][kChunk];           // the chunk's second pyramid level (a sample per block)
  uint8_t p3[2][kStrip / 2][kChunk / 2];
};

// Four samples at p; past the plane's width (n of them inside) zeros.
__device__ __forceinline__ uint32_t load4(const uint8_t* p, bool aligned, int n) {
  if (aligned && n >= 4) return __ldg((const uint32_t*)p);
  uint32_t v = 0;
  for (int k = 0; k < 4 && k < n; k++) v |= (uint32_t)__ldg(p + k) << (8 * k);
  return v;
}
// Rounded 2x2 means of two rows of four samples: two samples, 16 bits apart.
__device__ __forceinline__ uint32_t mean2x2(uint32_t r0, uint32_t r1) {
  const uint32_t s = (r0 & 0x00ff00ffu) + ((r0 >> 8) & 0x00ff00ffu) + (r1 & 0x00ff00ffu) + ((r1 >> 8) & 0x00ff00ffu);
  return ((s + 0x00020002u) >> 2) & 0x00ff00ffu;
}

// The window rows kStrip * strip .. of one scale. A block walks its strip in chunks of kChunk windows:
// the 4x4 blocks' sums (byte dot products, shared by the four windows around each), the window
// values, and a lane per row adding them up in order. kPyramid: the same words also give the
// strip's samples of the four coarser levels.
template <bool kPyramid, int kStrip, int kChunk>
__device__ void ssim_strip(const SsimPair& pair, int level, int strip, RowsSmem<kStrip, kChunk>& sh) {
  const SsimLevel& lv = pair.lv[level];
  const int tid = threadIdx.x, w = lv.w, h = lv.h, bw = w >> 2, bh = h >> 2;
  const int nrows = bh >= 2 && bw >= 2 ? bh - 1 : 0, nwin = bw - 1, r0 = strip * kStrip;
  const bool al_a = (((uintptr_t)lv.a | (uintptr_t)lv.sa) & 3) == 0, al_b = (((uintptr_t)lv.b | (uintptr_t)lv.sb) & 3) == 0;
  const int levels = kPyramid ? pair.levels : 1;
  const int cols = levels > 1 ? (w + 3) >> 2 : nwin;  // of blocks with pyramid samples, or of windows
  float row = 0.0f;  // lanes 0 .. kStrip - 1 of the first warp: the rows' running sums
  for (int c0 = 0; c0 < cols; c0 += kChunk) {
    // the 4x4 blocks
    for (int i = tid; i < (kStrip + 1) * (kChunk + 1); i += kRowThreads) {
      const int br = i / (kChunk + 1), bx = i - br * (kChunk + 1), R = r0 + br, X = c0 + bx;
      const bool full = R < bh && X < bw;
      const bool pyr = kPyramid && levels > 1 && br < kStrip && bx < kChunk && R * 4 < h && X * 4 < w;
      if (!full && !pyr) continue;
      uint32_t a[4], b[4];
      const uint8_t* pa = lv.a + (long)R * 4 * lv.sa + X * 4;
      const uint8_t* pb = lv.b + (long)R * 4 * lv.sb + X * 4;
#pragma unroll
      for (int y = 0; y < 4; y++) {
        const int n = R * 4 + y < h ? w - X * 4 : 0;
        a[y] = load4(pa + y * lv.sa, al_a, n);
        b[y] = load4(pb + y * lv.sb, al_b, n);
      }
      if (full) {
        uint32_t s1 = 0, s2 = 0, ss = 0, s12 = 0;
#pragma unroll
        for (int y = 0; y < 4; y++) {
          s1 = __dp4a(a[y], 0x01010101u, s1);
          s2 = __dp4a(b[y], 0x01010101u, s2);
          ss = __dp4a(a[y], a[y], __dp4a(b[y], b[y], ss));
          s12 = __dp4a(a[y], b[y], s12);
        }
        sh.sums[i] = make_int4((int)s1, (int)s2, (int)ss, (int)s12);
      }
      if constexpr (kPyramid) {
        if (pyr) {
#pragma unroll
          for (int p = 0; p < 2; p++) {
            const uint32_t* v = p ? b : a;
            const uint32_t m[2] = {mean2x2(v[0], v[1]), mean2x2(v[2], v[3])};
            const SsimLevel& l1 = pair.lv[1];
            uint8_t* d1 = (uint8_t*)(p ? l1.b : l1.a);
            const long s1 = p ? l1.sb : l1.sa;
#pragma unroll
            for (int y = 0; y < 2; y++)
              if (R * 2 + y < l1.h) {
                uint8_t* q = d1 + (long)(R * 2 + y) * s1 + X * 2;
                if (X * 2 + 1 < l1.w) *(uint16_t*)q = (uint16_t)((m[y] & 0xffu) | (m[y] >> 8));
                else if (X * 2 < l1.w) *q = (uint8_t)m[y];
              }
            const uint32_t t = m[0] + m[1];
            const uint8_t v2 = (uint8_t)(((t & 0xffffu) + (t >> 16) + 2u) >> 2);
            sh.p2[p][br][bx] = v2;
            if (levels > 2 && full) {
              const SsimLevel& l2 = pair.lv[2];
              ((uint8_t*)(p ? l2.b : l2.a))[(long)R * (p ? l2.sb : l2.sa) + X] = v2;
            }
          }
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < kStrip * kChunk; i += kRowThreads) {
      const int r = i / kChunk, k = i - r * kChunk;
      if (r0 + r >= nrows || c0 + k >= nwin) continue;
      const int4* s = &sh.sums[r * (kChunk + 1) + k];
      const int4 a0 = s[0], a1 = s[1], b0 = s[kChunk + 1], b1 = s[kChunk + 2];
      sh.vals[r * (kChunk + 1) + k] =
          ssim_end1(a0.x + a1.x + b0.x + b1.x, a0.y + a1.y + b0.y + b1.y, a0.z + a1.z + b0.z + b1.z, a0.w + a1.w + b0.w + b1.w);
    }
    if (kPyramid && levels > 3)
      for (int i = tid; i < 2 * (kStrip / 2) * (kChunk / 2); i += kRowThreads) {
        const int p = i / ((kStrip / 2) * (kChunk / 2)), r = (i / (kChunk / 2)) % (kStrip / 2), k = i % (kChunk / 2);
        const uint8_t* q = &sh.p2[p][2 * r][2 * k];
        const uint8_t v = (uint8_t)((q[0] + q[1] + q[kChunk] + q[kChunk + 1] + 2) >> 2);
        const SsimLevel& l = pair.lv[3];
        const int y = r0 / 2 + r, x = c0 / 2 + k;
        sh.p3[p][r][k] = v;
        if (y < l.h && x < l.w) ((uint8_t*)(p ? l.b : l.a))[(long)y * (p ? l.sb : l.sa) + x] = v;
      }
    __syncthreads();
    if (kPyramid && levels > 4) {
      const int i = tid - 128;  // the upper warps
      if (i >= 0 && i < 2 * (kStrip / 4) * (kChunk / 4)) {
        const int p = i / ((kStrip / 4) * (kChunk / 4)), r = (i / (kChunk / 4)) % (kStrip / 4), k = i % (kChunk / 4);
        const uint8_t* q = &sh.p3[p][2 * r][2 * k];
        const SsimLevel& l = pair.lv[4];
        const int y = r0 / 4 + r, x = c0 / 4 + k;
        if (y < l.h && x < l.w)
          ((uint8_t*)(p ? l.b : l.a))[(long)y * (p ? l.sb : l.sa) + x] = (uint8_t)((q[0] + q[1] + q[kChunk / 2] + q[kChunk / 2 + 1] + 2) >> 2);
      }
    }
    if (tid < kStrip && r0 + tid < nrows) {
      const float* v = &sh.vals[tid * (kChunk + 1)];
      const int n = min(kChunk, nwin - c0);
#pragma unroll 8
      for (int k = 0; k < n; k++) row = __fadd_rn(row, v[k]);
    }
  }
  if (tid < kStrip && r0 + tid < nrows) lv.rows[r0 + tid] = row;
}

// Level 0 and the pyramid (blockIdx.x a strip), or levels 1 .. (their strips one level after the other).
template <bool kPyramid, int kStrip, int kChunk>
__device__ __forceinline__ void ssim_pass(const SsimPair& p) {
  __shared__ RowsSmem<kStrip, kChunk> sh;
  int strip = blockIdx.x;
  for (int l = kPyramid ? 0 : 1; l < (kPyramid ? 1 : p.levels); l++) {
    const int n = ssim_strips(p.lv[l].h, kPyramid && p.levels > 1, kStrip);
    if (strip < n) {
      ssim_strip<kPyramid>(p, l, strip, sh);
      return;
    }
    strip -= n;
  }
}

// The f64 SSIM of one scale from its rows, in order; of a plane without a full window pair, the one
// 8x8 window at the origin. Every thread of a warp calls it; lane 0 holds the result.
__device__ double ssim_total(const SsimLevel& l, float* stage) {  // stage: 128 floats of shared memory
  const int lane = threadIdx.x & 31, bw = l.w >> 2, bh = l.h >> 2;
  double total = 0.0;
  if (bw < 2 || bh < 2) {
    if (lane == 0) {
      int s1 = 0, s2 = 0, ss = 0, s12 = 0;
      for (int y = 0; y < 8; y++)
        for (int x = 0; x < 8; x++) {
          int va = l.a[(long)y * l.sa + x], vb = l.b[(long)y * l.sb + x];
          s1 += va; s2 += vb; ss += va * va + vb * vb; s12 += va * vb;
        }
      total = (double)ssim_end1(s1, s2, ss, s12);
    }
    return total;
  }
  for (int r = 0; r < bh - 1; r += 128) {
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (r + 32 * k + lane < bh - 1) stage[32 * k + lane] = l.rows[r + 32 * k + lane];
    __syncwarp();
    if (lane == 0) {
      const int n = min(128, bh - 1 - r);
#pragma unroll 8
      for (int k = 0; k < n; k++) total = __dadd_rn(total, (double)stage[k]);
    }
  }
  return __ddiv_rn(total, (double)((bw - 1) * (bh - 1)));
}
