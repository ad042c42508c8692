// Search forms of the macroblock engine (included by engine_kernels.cu inside its anonymous
// namespace; uses its helpers). Neither form exists in the reference: they are the exhaustive
// "full search" the learned form is trained on and judged against, and the learned form itself.
//
// P macroblock (analyse_p_mb_search):
//   1. the P_Skip probe of the plain form (enc.rs:2906 try_p_skip) with the skip vector of the
//      quadrant grid;
//   2. integer search: the SAD of each 8x8 quadrant at every integer vector of a window, and for
//      each of the nine partition parts (16x16; 16x8 top, bottom; 8x16 left, right; four 8x8) the
//      vector of least SAD + lambda * (bits(4 vx - mvp.x) + bits(4 vy - mvp.y)) against the 16x16
//      predictor, first in raster order on ties. Full search: the window is +-search_range around
//      the 16x16 predictor. Learned: +-2 around a centre chosen among seven integer candidates --
//      predictor plus the hinted offset, predictor, the hint's coarse vector (when it has one), the
//      left, top and top-right (top-left where that is absent) neighbours' vectors, zero -- by the
//      16x16 SAD + lambda * vector bits, first in that order on ties; while the 16x16 part's best lies on that window's edge (and not on
//      the vector bounds) the window is centred on it again, up to `walk` times, and then the full
//      window is searched;
//   3. for every partition type tried (all four; learned: the hinted ones), each part in coding
//      order from its integer best: half-sample step (centre, then 8 neighbours at distance 2,
//      quarter units) and quarter-sample step (8 neighbours at distance 1), costs (SATD >> 1) +
//      lambda * vector bits against the part's own predictor (H.264 8.4.1.3, directional for 16x8
//      and 8x16), least cost first in candidate order; learned: the SAD diamonds of
//      refine_part_sad instead;
//   4. the type of least total cost, the stream's type bits (per partition type) * lambda added,
//      first on ties;
//   5. intra 16x16 check, residual, late skip and reconstruction exactly as the plain form.
// IDR macroblock: the plain form's analysis; learned: intra 4x4 blocks try only their hinted modes
// (those of them available at the block, DC when none is).

constexpr int kBandRows = 8;               // integer vectors per band row
constexpr int kUnitBands = 1;  // (2: full search 8 x 3 720p 24.8 ms against 23.7)
constexpr int kBandBytes = (kUnitBands + 2) * kBandRows * (2 * kMaxSearchRange + 24);  // the rows of a unit
constexpr int kLearnedRange = 2;           // learned form: integer window around the seed
constexpr int kCentreCands = 7;            // learned form: candidates of the window's centre


// The quadrants around and in the current macroblock that motion prediction reads, by index 4 (row + 1) +
// column + 1 (columns -1 .. 2, rows -1 .. 1): D B0 B1 C / A0 0 1 - / A1 2 3 -. ref -2 not available (or not
// yet decided), -1 intra, 0 inter; mv packed, 0 unless inter.
struct NbMv {
  uint32_t mv;
  int ref;
  __device__ __forceinline__ int x() const { return lo16((int)mv); }
  __device__ __forceinline__ int y() const { return (int)mv >> 16; }
};
struct IntBest {
  int x[9], y[9];
  uint32_t c[9];
};
// The whole groups of an integer search, in units of kUnitBands bands: what a warp of the block needs to do one.
struct SearchJob {
  const uint8_t* ref;
  int stride, x0, y0, xlo, xt, ylo, yhi, nwx, mvp0, mvp1;
  uint32_t lambda;
  uint32_t ticket;   // next unit | units << 16; kNoJob while there is none
  int done;          // units finished
  bool failed;       // the wait for them gave up: the launch fails, and this warp leaves with its macroblock
  uint32_t key[9];   // the least so far
};
constexpr uint32_t kNoJob = 0x8000u;  // (a ticket past any unit)
struct SearchSmem {
  uint8_t band[kBandBytes];
  SearchJob job;
  IntBest ib;
  alignas(8) NbMv nb[12];
  int qmv[4][2];
  uint32_t pmvd[4];    // the chosen type's parts' vector differences
  int ccx[8], ccy[8];  // the learned form's centre candidates (ok: cok)
  bool cok[8];
};
// Behind every warp's Smem.
static_assert(sizeof(Smem) % 16 == 0, "SearchSmem follows aligned");
#define ss (((SearchSmem*)(smw + blockDim.y * sizeof(Smem)))[threadIdx.y])
// The neighbours into ss.nb, all loads in flight together: lanes 0..3 the refs of the left, top,
// top-right and top-left macroblocks, lanes 4..9 the vectors A0, A1, B0, B1, C, D.
__device__ __forceinline__ uint32_t load_nb(const Ctx c) {
  const StreamDev& sd = sm.sd;
  const int lane = lane_id(), mb_w = sm.fp.mb_w;
  const int k = lane < 4 ? lane : (lane < 8 ? (lane - 4) >> 1 : lane - 6);  // which macroblock
  const bool have = k == 0 ? c.mbx > 0 : (c.mby > 0 && (k == 1 || (k == 2 ? c.mbx + 1 < mb_w : c.mbx > 0)));
  const int mb = c.mb + (k == 0 ? -1 : (k == 1 ? 0 : (k == 2 ? 1 : -1)) - mb_w);
  uint32_t w = lane < 4 ? 0xfeu : 0u;
  if (lane < 10 && have) {
    const int quad = lane == 4 ? 1 : (lane == 6 || lane == 8 ? 2 : 3);
    w = lane < 4 ? ((const uint32_t*)&sd.info[mb])[1] : ((const uint32_t*)&sd.mv4[mb])[quad];
  }
  return w;
}
__device__ __forceinline__ void store_nb(uint32_t w) {
  const int lane = lane_id();
  const int ref = (int8_t)(w & 255u);
  const int r = __shfl_sync(FULL, ref, lane < 8 ? max(lane - 4, 0) >> 1 : min(lane - 6, 3));  // the vector's macroblock
  if (lane >= 4 && lane < 10) ss.nb[(int)((0x032184u >> (4 * (lane - 4))) & 15u)] = NbMv{r == 0 ? w : 0u, r};
  if (lane == 10 || lane == 11) ss.nb[lane == 10 ? 7 : 11] = NbMv{0u, -2};
  __syncwarp();
}
// Partition parts 0..8 in coding order: 16x16 | 16x8 top, bottom | 8x16 left, right | 8x8. Their neighbours A,
// B, C, D as indices into ss.nb (4 bits each, A lowest), then the quadrants covered (bits 16..19), the
// directional rule (bits 20..21: 1 B, 2 A, 3 C), and x / 8, y / 8, width 8, height 8 (bits 24..27).
__device__ __constant__ uint32_t c_part[9] = {
    0x00000314u | 15u << 16,
    0x00000314u | 3u << 16 | 1u << 20 | 8u << 24, 0x00004758u | 12u << 16 | 2u << 20 | (2u | 8u) << 24,
    0x00000214u | 5u << 16 | 2u << 20 | 4u << 24, 0x00001325u | 10u << 16 | 3u << 20 | (1u | 4u) << 24,
    0x00000214u | 1u << 16 | 12u << 24, 0x00001325u | 2u << 16 | (1u | 12u) << 24,
    0x00004658u | 4u << 16 | (2u | 12u) << 24, 0x00005769u | 8u << 16 | 15u << 24};
__device__ __forceinline__ int type_first(int t) { return (0x5310 >> (4 * t)) & 15; }
__device__ __forceinline__ int type_parts(int t) { return (0x4221 >> (4 * t)) & 15; }
// Motion vector predictor of a part (H.264 8.4.1.3), packed.
__device__ __noinline__ uint32_t mv_pred(uint32_t part) {
  const NbMv A = ss.nb[part & 15u], B = ss.nb[(part >> 4) & 15u], D = ss.nb[(part >> 12) & 15u];
  NbMv C = ss.nb[(part >> 8) & 15u];
  if (C.ref == -2) C = D;
  const int dir = (int)((part >> 20) & 3u);
  if (dir == 1 && B.ref == 0) return B.mv;
  if (dir == 2 && A.ref == 0) return A.mv;
  if (dir == 3 && C.ref == 0) return C.mv;
  if (B.ref == -2 && C.ref == -2 && A.ref != -2) return A.mv;
  if ((A.ref == 0) + (B.ref == 0) + (C.ref == 0) == 1) return A.ref == 0 ? A.mv : (B.ref == 0 ? B.mv : C.mv);
  auto med = [](int x, int y, int z) { return min(max(x, y), max(min(x, y), z)); };
  return pack16(med(A.x(), B.x(), C.x()), med(A.y(), B.y(), C.y()));
}
// A refined part: its cost and quarter-sample vector.
struct PartFit {
  uint32_t cost;
  int x, y;
};

__device__ __forceinline__ uint32_t vec_cost(int dx, int dy, uint32_t lambda) {
  return lambda * (se_bits(dx) + se_bits(dy));
}

// ---------------------------------------------------------------------------------------------
// Integer search over [xlo, xhi] x [ylo, yhi]. Lanes take columns xlo + lane + 32 j; the reference
// rows of 8 vector rows (a band) are staged in shared memory, and each lane slides its column's 16 x 16
// comparison down the band, a reference row at a time against the source rows it pairs
// with. Up to four columns past the last whole group (a window of 2 R + 1 vectors has one) go a vector
// to a lane instead of a group of their own. Costs and raster indices share a word (cost <= 65280 +
// 91 * 66 < 2^17, index < 129^2 < 2^15), so the first least one is a minimum. ss.ib: the nine parts'
// results. (A group for the odd column, a compare of cost and index, source and reference by single
// words: 284 k cycles a macroblock at range 32.)
__device__ __forceinline__ uint32_t lds4u(const uint8_t* p) {
  uintptr_t a = (uintptr_t)p;
  const uint32_t* b = (const uint32_t*)(a & ~(uintptr_t)3);
  return __funnelshift_r(b[0], b[1], (uint32_t)(a & 3) * 8u);
}
constexpr int kKeyBits = 15;  // of the raster index
static_assert((2 * kMaxSearchRange + 1) * (2 * kMaxSearchRange + 1) <= 1 << kKeyBits, "raster index");
constexpr int kPitch = 36;    // bytes of a staged row of stage_rows: consecutive rows in different banks
// The 32 bytes from column xs (a multiple of 4) of n picture rows from row y into the band.
__device__ __forceinline__ void stage_rows(int xs, int y, int n) {
  const int lane = lane_id(), k = lane & 7;
  const uint8_t* p = sm.sd.ref_y + (long)y * sm.fp.stride_y + xs + 4 * k;
  __syncwarp();
#pragma unroll 6
  for (int r = lane >> 3; r < n; r += 4) *(uint32_t*)(ss.band + r * kPitch + 4 * k) = ldw32(p + (long)r * sm.fp.stride_y);
  __syncwarp();
}
// Keys of the nine parts (minimum kept) at the vector whose quadrant SADs are q; mci: its vector cost
// and index.
__device__ __forceinline__ void part_keys(uint32_t (&key)[9], uint32_t q0, uint32_t q1, uint32_t q2, uint32_t q3, uint32_t mci) {
  const uint32_t t = q0 + q1, b = q2 + q3;
  const uint32_t part[9] = {t + b, t, b, q0 + q2, q1 + q3, q0, q1, q2, q3};
#pragma unroll
  for (int k = 0; k < 9; k++) key[k] = min(key[k], (part[k] << kKeyBits) + mci);
}
// The same for a lane's own vector over the rows of stage_rows: its 16 x 16 block starts at byte `at`.
__device__ __noinline__ uint4 quad_sads(int at) {
  const uint32_t* p = (const uint32_t*)(ss.band + (at & ~3));
  const uint32_t sh = (uint32_t)(at & 3) * 8u;
  uint32_t q[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll 4
    for (int r = 8 * h; r < 8 * h + 8; r++) {
      const uint4 s = *(const uint4*)&sm.src_y[r * 16];
      const uint32_t* w = p + r * (kPitch / 4);
      const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
      q[2 * h] = __vsadu4(__funnelshift_r(w0, w1, sh), s.x) + __vsadu4(__funnelshift_r(w1, w2, sh), s.y) + q[2 * h];
      q[2 * h + 1] = __vsadu4(__funnelshift_r(w2, w3, sh), s.z) + __vsadu4(__funnelshift_r(w3, w4, sh), s.w) + q[2 * h + 1];
    }
  return make_uint4(q[0], q[1], q[2], q[3]);
}
// Unit u (kUnitBands bands) of warp `owner`'s search, over this warp's band; the least keys into the job's.
__device__ __noinline__ void search_unit(int owner, int u) {
  SearchSmem& os = ((SearchSmem*)(smw + blockDim.y * sizeof(Smem)))[owner];
  const SearchJob& jb = os.job;
  const uint8_t* const src = ((const Smem*)smw)[owner].src_y;
  const int lane = lane_id(), yhi = jb.yhi, nwx = jb.nwx, ylo = jb.ylo + kUnitBands * kBandRows * u;
  const uint32_t lambda = jb.lambda;
  uint32_t key[9];
#pragma unroll
  for (int k = 0; k < 9; k++) key[k] = UMAX;
  const int xs = (jb.x0 + jb.xlo) & ~3;              // picture column of band column 0
  const int wpr = (jb.x0 + jb.xt + 22 - xs) >> 2;    // words of a band row
  {
    // its reference rows from y0 + ylo, in words, lane by lane
    const int dr = 32 / wpr, dk = 32 - dr * wpr, n = min((kUnitBands + 2) * kBandRows, yhi - ylo + 16);
    const uint8_t* p = jb.ref + (long)(jb.y0 + ylo) * jb.stride + xs;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ss.band);
    __syncwarp();
    int r = lane / wpr, k = lane - r * wpr;
#pragma unroll 1
    for (; r < n; r += dr) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + (uint32_t)(r * wpr + k) * 4u),
                   "l"(p + (long)r * jb.stride + 4 * k) : "memory");
      k += dk;
      if (k >= wpr) {
        k -= wpr;
        r++;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }
#pragma unroll 1
  for (int dy0 = ylo, b = 0; b < kUnitBands && dy0 <= yhi; dy0 += kBandRows, b++) {
#pragma unroll 1
    for (int d0 = jb.xlo; d0 < jb.xt; d0 += 32) {
      const int dx = d0 + lane;
      const bool act = dx < jb.xt;
      const int co = act ? jb.x0 + dx - xs : 0;
      const uint32_t sh = (uint32_t)(co & 3) * 8u;
      uint32_t top[kBandRows][2], acc[kBandRows][2] = {};
#pragma unroll 1
      for (int half = 0; half < 2; half++) {
        uint4 s[8];
#pragma unroll
        for (int r = 0; r < 8; r++) s[r] = *(const uint4*)(src + (half * 8 + r) * 16);
#pragma unroll
        for (int d = 0; d < kBandRows; d++) {
          top[d][0] = acc[d][0];
          top[d][1] = acc[d][1];
          acc[d][0] = acc[d][1] = 0;
        }
        const uint32_t* rp = (const uint32_t*)ss.band + (b + half) * kBandRows * wpr + (co >> 2);
#pragma unroll
        for (int i = 0; i < kBandRows + 7; i++) {
          // reference row half * 8 + i of the band pairs with source row r = i - d for d = 0..7
          const uint32_t w0 = rp[0], w1 = rp[1], w2 = rp[2], w3 = rp[3], w4 = rp[4];
          rp += wpr;
          const uint32_t R0 = __funnelshift_r(w0, w1, sh), R1 = __funnelshift_r(w1, w2, sh), R2 = __funnelshift_r(w2, w3, sh),
                         R3 = __funnelshift_r(w3, w4, sh);
#pragma unroll
          for (int d = 0; d < kBandRows; d++) {
            const int r = i - d;
            if (r < 0 || r > 7) continue;
            acc[d][0] = __vsadu4(R0, s[r].x) + __vsadu4(R1, s[r].y) + acc[d][0];
            acc[d][1] = __vsadu4(R2, s[r].z) + __vsadu4(R3, s[r].w) + acc[d][1];
          }
        }
      }
      const uint32_t cx = lambda * se_bits(4 * dx - jb.mvp0);
      uint32_t idx = (uint32_t)((dy0 - jb.ylo) * nwx + (dx - jb.xlo));
#pragma unroll
      for (int d = 0; d < kBandRows; d++, idx += nwx)
        if (act && dy0 + d <= yhi)
          part_keys(key, top[d][0], top[d][1], acc[d][0], acc[d][1],
                    ((cx + lambda * se_bits(4 * (dy0 + d) - jb.mvp1)) << kKeyBits) + idx);
    }
  }
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const uint32_t m = __reduce_min_sync(FULL, key[k]);
    if (lane == k) atomicMin(&os.job.key[k], m);
  }
  // the keys before the count
  __threadfence_block();
  __syncwarp();
  if (lane == 0) atomicAdd(&os.job.done, 1);
}
// Takes units of `owner`'s search until none is left.
__device__ __forceinline__ void search_units(int owner) {
  SearchJob& jb = ((SearchSmem*)(smw + blockDim.y * sizeof(Smem)))[owner].job;
  while (true) {
    uint32_t t = 0;
    if (lane_id() == 0) t = atomicAdd(&jb.ticket, 1u);
    t = __shfl_sync(FULL, t, 0);
    if ((t & 0xffffu) >= (t >> 16)) break;
    __threadfence_block();  // the job was written before its ticket
    search_unit(owner, (int)(t & 0xffffu));
  }
}
// A warp that waits for its segment meanwhile takes part in the searches open in its block (board: a bit per
// warp with one).
__device__ __noinline__ void help_searches(unsigned* board) {
  unsigned open = __shfl_sync(FULL, *(volatile unsigned*)board, 0);
  while (open) {
    search_units(__ffs(open) - 1);
    if (lane_id() == 0) atomicAnd(board, ~(open & -open));  // no unit left (a search opened since goes without help)
    open &= open - 1;
  }
}

// pw.board (or null): the block's warps that wait take part. A macroblock's search is then a few units long
// instead of nine bands: at range 32 a macroblock's search took 105 k cycles of the chain that a launch of
// few pictures is (full search 8 x 3 720p: 28.6 ms without help, 23.6 so; learned 1080p 8 x 8, whose walk
// falls back to it, 50.2 and 46.7, 4K 4 x 3 48.7 and 46.6). Sharing the partition types' refinement the same
// way gave the full search 6 % more and cost the learned form 3 %.
//
// ss.job.failed once the wait for units others took gave up: the window's first vector stands for every part's
// then, so that what follows reads what it may, and the macroblock is not published (pipeline_kernel): the warp
// leaves, as after any wait that gave up, and the job that others may still read stays as it is. (As this
// function's result it made the full search 6 % slower, read after it the learned form 0.7 %; so it is 1 and 0.1 %.)
__device__ __noinline__ void int_search(const Ctx c, int xlo, int xhi, int ylo, int yhi,
                                        int mvp0, int mvp1, uint32_t lambda, const PipeWait pw) {
  const int lane = lane_id();
  const int x0 = c.mbx * 16, y0 = c.mby * 16;
  const int nwx = xhi - xlo + 1, nwy = yhi - ylo + 1;
  uint32_t key[9];
#pragma unroll
  for (int k = 0; k < 9; k++) key[k] = UMAX;
  // a window of at most 32 vectors (the learned form's), or the columns past the last whole group: `cols`
  // columns from xt, a lane a vector, as many rows at a time as fit
  const bool small = nwx <= 8 && nwx * nwy <= 32;
  const int rem = nwx & 31, cols = small ? nwx : (rem <= 4 ? rem : 0), xt = xhi - cols + 1;
  const int units = xt > xlo ? (nwy + kUnitBands * kBandRows - 1) / (kUnitBands * kBandRows) : 0;
  if (units) {
    SearchJob& jb = ss.job;
    if (lane == 0) {
      jb.ref = sm.sd.ref_y;
      jb.stride = sm.fp.stride_y;
      jb.x0 = x0; jb.y0 = y0; jb.xlo = xlo; jb.xt = xt; jb.ylo = ylo; jb.yhi = yhi; jb.nwx = nwx;
      jb.mvp0 = mvp0; jb.mvp1 = mvp1; jb.lambda = lambda;
      jb.done = 0;
    }
    if (lane < 9) jb.key[lane] = UMAX;
    __threadfence_block();  // the job (and this warp's source) before its ticket
    __syncwarp();
    if (lane == 0) {
      atomicExch(&jb.ticket, (uint32_t)units << 16);
      if (pw.board) atomicOr(pw.board, 1u << threadIdx.y);
    }
    __syncwarp();
    search_units(threadIdx.y);
    if (lane == 0) {
      if (pw.board) atomicAnd(pw.board, ~(1u << threadIdx.y));
      atomicExch(&jb.ticket, kNoJob);
      // units others still have, each of bounded work; past the limit the launch fails as for any wait
      unsigned long long t0 = 0;
      while (*(volatile int*)&jb.done < units) {
        if (!t0) t0 = global_ns();
        else if (global_ns() - t0 > pw.timeout_ns) {
          if (pw.error) atomicCAS(pw.error, 0, 1);
          jb.failed = true;
          for (int k = 0; k < 9; k++) atomicExch(&jb.key[k], 0u);  // (below any cost: it stays)
          break;
        }
        __nanosleep(50);
      }
    }
    __threadfence_block();
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 9; k++) key[k] = ((volatile uint32_t*)jb.key)[k];
  }
  if (cols) {
    const int vrows = 32 / cols, vy = lane / cols, vx = lane - vy * cols;
    const int xs = (x0 + xt) & ~3, dx = xt + vx;
    const uint32_t cx = lambda * se_bits(4 * dx - mvp0);
#pragma unroll 1
    for (int dy0 = ylo; dy0 <= yhi; dy0 += vrows) {
      const int n = min(vrows, yhi - dy0 + 1), dy = dy0 + vy;
      stage_rows(xs, y0 + dy0, n + 15);
      const bool act = vy < n;
      const uint4 q = quad_sads(act ? vy * kPitch + (x0 + dx - xs) : 0);
      if (act)
        part_keys(key, q.x, q.y, q.z, q.w, ((cx + lambda * se_bits(4 * dy - mvp1)) << kKeyBits) + (uint32_t)((dy - ylo) * nwx + (dx - xlo)));
    }
  }
  // the least across the warp; lane k < 9 writes part k's
  uint32_t mine = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const uint32_t m = __reduce_min_sync(FULL, key[k]);
    if (lane == k) mine = m;
  }
  __syncwarp();
  if (lane < 9) {
    const int i = (int)(mine & ((1u << kKeyBits) - 1u)), y = i / nwx;
    ss.ib.c[lane] = mine >> kKeyBits;
    ss.ib.x[lane] = xlo + i - y * nwx;
    ss.ib.y[lane] = ylo + y;
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// Quarter-sample refinement of one part (px, py, pw, ph samples within the macroblock) from its
// integer best (bx, by) with predictor mvp. Candidates of one step are evaluated in parallel: slot
// = candidate * blocks + 4x4 block, each lane the SATD of one block's prediction (from the
// half-sample planes of a window around the integer best) against the source.
// Half the SATD of a 4x4 block of byte rows (an even number before the halving): columns 0, 2 and 1, 3 packed as
// hi * 65536 + lo through the column butterflies, |x + y| + |x - y| = 2 max(|x|, |y|) for the last one.
__device__ __forceinline__ uint32_t half_satd4(const uint32_t* sa, const uint32_t* pa) {
  int e[4], o[4];
#pragma unroll
  for (int y = 0; y < 4; y++) {
    e[y] = (int)(sa[y] & 0x00ff00ffu) - (int)(pa[y] & 0x00ff00ffu);
    o[y] = (int)__byte_perm(sa[y], 0u, 0x4341) - (int)__byte_perm(pa[y], 0u, 0x4341);
  }
  auto cols = [](int (&v)[4]) {
    const int s03 = v[0] + v[3], s12 = v[1] + v[2], d03 = v[0] - v[3], d12 = v[1] - v[2];
    v[0] = s03 + s12; v[1] = d03 + d12; v[2] = s03 - s12; v[3] = d03 - d12;
  };
  cols(e);
  cols(o);
  uint32_t s = 0;
#pragma unroll
  for (int y = 0; y < 4; y++) {
    const int r0 = (int16_t)e[y], r2 = (e[y] + 0x8000) >> 16, r1 = (int16_t)o[y], r3 = (o[y] + 0x8000) >> 16;
    const int s03 = r0 + r3, s12 = r1 + r2, d03 = r0 - r3, d12 = r1 - r2;
    s += (uint32_t)(max(abs(s03), abs(s12)) + max(abs(d03), abs(d12)));
  }
  return s;
}
// The 4x4 prediction at the block's sample (ox, oy) for the vector (dx, dy) from the window's position:
// four packed rows.
__device__ __forceinline__ void qpel4(int ox, int oy, int dx, int dy, uint32_t* out) {
  const uint8_t* p = &sm.win[0] + qpel_pos(dx, dy) + oy * 24 + ox;
  const uint32_t e = sm.qpt[(dx & 3) | ((dy & 3) << 2)];
#pragma unroll
  for (int r = 0; r < 4; r++) out[r] = __vavgu4(lds4u(p + r * 24 + (e & 0xffffu)), lds4u(p + r * 24 + (e >> 16)));
}
__device__ __constant__ int8_t c_hstep[8][2] = {{0, -2}, {-2, 0}, {2, 0}, {0, 2}, {-2, -2}, {2, -2}, {-2, 2}, {2, 2}};

// The half-sample planes in shared memory serve every part whose integer vector they were built
// around: the macroblock's window (ensure_window) covers every 4x4 block of the macroblock at
// quarter-sample offsets -3..3.
__device__ __forceinline__ void ensure_mb_window(const Ctx c, int bx, int by) {
  ensure_window(c.mbx * 16 + bx, c.mby * 16 + by, 7);
}

__device__ __noinline__ PartFit refine_part(const Ctx c, int px, int py, int pw, int ph, int bx,
                                            int by, int2 mvp, uint32_t lambda, Bounds bd) {
  const int lane = lane_id();
  ensure_mb_window(c, bx, by);
  const int bw4 = pw >> 2, nblk = bw4 * (ph >> 2);
  const int m0x = 4 * bx, m0y = 4 * by;
  int cx = m0x, cy = m0y;
  uint32_t best_key = UMAX;
  for (int step = 0; step < 2; step++) {
    const int ncand = step == 0 ? 9 : 8;
    const int sc = step == 0 ? 1 : 2;  // step 0: centre + distance 2; step 1: distance 1
    uint32_t key = step == 0 ? UMAX : best_key & ~15u;  // the current best keeps index 0
    for (int base = 0; base < ncand * nblk; base += 32) {
      const int slot = base + lane;
      const int cand = slot / nblk, blk = slot - cand * nblk;
      int vx = cx, vy = cy;
      if (cand < ncand) {
        if (step == 0 && cand > 0) { vx += c_hstep[cand - 1][0]; vy += c_hstep[cand - 1][1]; }
        if (step == 1) { vx += c_hstep[cand][0] / sc; vy += c_hstep[cand][1] / sc; }
      }
      const bool ok = cand < ncand && in_bounds(bd, vx, vy);
      uint32_t s = 0;
      if (ok) {
        const int ox = 4 * (blk % bw4), oy = 4 * (blk / bw4);
        uint32_t pa[4], sa[4];
        qpel4(px + ox, py + oy, vx - m0x, vy - m0y, pa);
#pragma unroll
        for (int r = 0; r < 4; r++) sa[r] = *(const uint32_t*)&sm.src_y[(py + oy + r) * 16 + px + ox];
        s = half_satd4(sa, pa);
      }
      // sum over the candidate's blocks (consecutive lanes; nblk divides 32)
      for (int o = 1; o < nblk; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
      uint32_t k = UMAX;
      if (ok && blk == 0) {
        uint32_t cost = s + vec_cost(vx - mvp.x, vy - mvp.y, lambda);
        k = (cost << 4) | (uint32_t)(step == 0 ? cand : cand + 1);
      }
      key = min(key, __reduce_min_sync(FULL, k));
    }
    // the winner's vector
    const int wi = (int)(key & 15u);
    if (step == 0) {
      if (wi > 0) { cx += c_hstep[wi - 1][0]; cy += c_hstep[wi - 1][1]; }
    } else if (wi > 0) {
      cx += c_hstep[wi - 1][0] / 2;
      cy += c_hstep[wi - 1][1] / 2;
    }
    best_key = (key & ~15u);
  }
  return PartFit{best_key >> 4, cx, cy};
}

// Learned form: refinement of one part from its integer best (bx, by), whose SAD is sad0, by SAD -- the
// half-sample diamond (up, left, right, down at distance 2, one step), then the quarter-sample diamond
// (the same at distance 1, up to two steps, each from the step's start), cost SAD + lambda * vector bits
// against the part's predictor, the first strict minimum in that order. Eight lanes a neighbour, each
// every eighth of the part's 4-sample words, and planes built when a step reads them. (The neighbours one
// after the other over the whole warp, every plane for every part: 86 k cycles for the refinement of a
// macroblock.)
__device__ __noinline__ PartFit refine_part_sad(const Ctx c, int px, int py, int pw, int ph,
                                                int bx, int by, int2 mvp, uint32_t lambda, Bounds bd, uint32_t sad0) {
  const int lane = lane_id(), k = lane >> 3, shift = pw == 16 ? 2 : 1, nw = (pw * ph) >> 2;
  const int m0x = 4 * bx, m0y = 4 * by;
  uint32_t best = sad0 + vec_cost(m0x - mvp.x, m0y - mvp.y, lambda);
  const Box box{max(bd.min0, m0x - 3), min(bd.max0, m0x + 3), max(bd.min1, m0y - 3), min(bd.max1, m0y + 3)};
  // the lane's words: rows r0, r0 + dr, .. (8 words are two rows of a 16-sample part, four of an 8-sample one)
  const int r0 = (lane & 7) >> shift, x = ((lane & 7) & ((1 << shift) - 1)) * 4, dr = 8 >> shift;
  const int at = (py + r0) * 24 + px + x;
  const uint8_t* const sp = &sm.src_y[(py + r0) * 16 + px + x];
  int q0 = 0, q1 = 0;
#pragma unroll 1
  for (int it = 0; it < 3; it++) {
    // the half-sample step reads planes b and h; so do quarter-sample steps from the integer position
    // itself; those around another read j too
    if (it < 2) ensure_window(c.mbx * 16 + bx, c.mby * 16 + by, q0 | q1 ? 7 : 3);
    const int st = it == 0 ? 2 : 1;
    const int dx = q0 + (k == 1 ? -st : (k == 2 ? st : 0)), dy = q1 + (k == 0 ? -st : (k == 3 ? st : 0));
    const uint32_t e = sm.qpt[(dx & 3) | ((dy & 3) << 2)];
    const uint8_t* const p = &sm.win[0] + qpel_pos(dx, dy) + at;
    const uint8_t *pa = p + (e & 0xffffu), *pb = p + (e >> 16), *s = sp;
    uint32_t sad = 0;
#pragma unroll 1
    for (int w = 0; w < nw; w += 16) {
#pragma unroll
      for (int u = 0; u < 2; u++)
        sad = __vsadu4(__vavgu4(lds4u(pa + u * dr * 24), lds4u(pb + u * dr * 24)), *(const uint32_t*)(s + u * dr * 16)) + sad;
      pa += 48 * dr;
      pb += 48 * dr;
      s += 32 * dr;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sad += __shfl_xor_sync(FULL, sad, o);
    const int vx = m0x + dx, vy = m0y + dy;
    const bool ok = vx >= box.lo0 && vx <= box.hi0 && vy >= box.lo1 && vy <= box.hi1;
    const uint32_t cost = sad + vec_cost(vx - mvp.x, vy - mvp.y, lambda);
    const uint32_t key = __reduce_min_sync(FULL, ok ? (cost << 2) | (uint32_t)k : UMAX);
    if ((key >> 2) < best) {
      best = key >> 2;
      const int b = (int)(key & 3u);
      q0 += b == 1 ? -st : (b == 2 ? st : 0);
      q1 += b == 0 ? -st : (b == 3 ? st : 0);
    } else if (it) {
      break;
    }
  }
  return PartFit{best, m0x + q0, m0y + q1};
}

// The luma prediction of a part at quarter-sample vector mv (within 3 quarter samples of 4 (bx, by),
// the integer vector its refinement started from) into pred_y.
__device__ __noinline__ void predict_part(const Ctx c, int px, int py, int pw, int ph, int bx,
                                          int by, int mvx, int mvy) {
  const int lane = lane_id();
  ensure_mb_window(c, bx, by);
  const int dx = mvx - 4 * bx, dy = mvy - 4 * by, shift = pw == 16 ? 2 : 1, nw = (pw * ph) >> 2;
  const uint32_t e = sm.qpt[(dx & 3) | ((dy & 3) << 2)];
  const uint8_t* p = &sm.win[0] + qpel_pos(dx, dy) + py * 24 + px;
  for (int w = lane; w < nw; w += 32) {
    const int r = w >> shift, x = (w - (r << shift)) * 4;
    const uint8_t* q = p + r * 24 + x;
    *(uint32_t*)&sm.pred_y[(py + r) * 16 + px + x] = __vavgu4(lds4u(q + (e & 0xffffu)), lds4u(q + (e >> 16)));
  }
  __syncwarp();
}
// Chroma prediction of both planes with each 8x8 luma quadrant's own vector (4x4 chroma blocks;
// the bilinear 1/8-sample filter of chroma_mc_8x8_x2, h264_enc.rs:1279, per sample).
__device__ __noinline__ void mc_chroma_q(const Ctx c) {
  const FrameParams& fp = sm.fp;
  const StreamDev& sd = sm.sd;
  const int lane = lane_id();
  const int plane = lane >> 4, idx = (lane & 15) * 4, r = idx >> 3, c0 = idx & 7;
  const int q = (r >> 2) * 2 + (c0 >> 2);
  const int mvx = ss.qmv[q][0], mvy = ss.qmv[q][1];
  const int cx = c.mbx * 8 + c0 + (mvx >> 3), cy = c.mby * 8 + r + (mvy >> 3), fx = mvx & 7, fy = mvy & 7;
  *(uint32_t*)((plane ? sm.pred_v : sm.pred_u) + r * 8 + c0) =
      chroma4((plane ? sd.ref_v : sd.ref_u) + (long)cy * fp.stride_c + cx, fp.stride_c, fx, fy);
  __syncwarp();
}

// Search-form side state of a coded macroblock: the record's partition fields and the quadrant
// vectors later macroblocks and the deblocking filter read (lane 0 writes). parts: the quadrants'
// vectors ss.qmv and the partitions' differences ss.pmvd; otherwise (mvx, mvy) everywhere and no
// differences.
__device__ __noinline__ void search_tail(const Ctx c, int ptype, bool parts, int mvx, int mvy) {
  if (lane_id() != 0) return;
  rg_mb_out* rec = sm.sd.rec + c.mb;
  MbMv4 m;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    m.mv[q][0] = (int16_t)(parts ? ss.qmv[q][0] : mvx);
    m.mv[q][1] = (int16_t)(parts ? ss.qmv[q][1] : mvy);
    rec->part_mv[q][0] = m.mv[q][0];
    rec->part_mv[q][1] = m.mv[q][1];
    rec->part_mvd[q][0] = (int16_t)(parts ? ss.pmvd[q] & 0xffffu : 0u);
    rec->part_mvd[q][1] = (int16_t)(parts ? ss.pmvd[q] >> 16 : 0u);
  }
  rec->part_type = (uint8_t)ptype;
  rec->reserved2[0] = rec->reserved2[1] = rec->reserved2[2] = 0;
  sm.sd.mv4[c.mb] = m;
}

// Reach of a search window for the pipelined mode's wait on the reference picture: every
// sample the integer search (band staging), the refinement windows and the final prediction can
// read lies above row (y0 + yhi + 28) and left of column (x0 + xhi + 36); everything above and
// to the left of the macroblock holding that sample is final once it is.
__device__ __forceinline__ bool wait_window(const Ctx c, const PipeWait& pw, int xhi, int yhi) {
  return !pw.db_prev || wait_reference(c, pw, (c.mbx * 16 + xhi + 36) >> 4, (c.mby * 16 + yhi + 28) >> 4);
}

// Learned form: the centre of the first +-2 window among the integer candidates of ss.ccx / ccy (cok false:
// absent) -- the first of least 16x16 SAD + lambda * vector bits against the 16x16 predictor.
__device__ __noinline__ int2 learned_centre(const Ctx c, int mvp0, int mvp1, uint32_t lambda) {
  const int* cx = ss.ccx;
  const int* cy = ss.ccy;
  const bool* ok = ss.cok;
  constexpr int n = kCentreCands;
  int bx, by;
  const int lane = lane_id();
  const int stride = sm.fp.stride_y;
  const uint8_t* base = sm.sd.ref_y + (long)(c.mby * 16 + (lane >> 1)) * stride + c.mbx * 16 + (lane & 1) * 8;
  const uint2 sv = src8();
  uint2 r[kCentreCands];
#pragma unroll
  for (int k = 0; k < kCentreCands; k++) r[k] = k < n && ok[k] ? ldg8(base + (long)cy[k] * stride + cx[k]) : make_uint2(0u, 0u);
  // two SADs to a word (each fits 16 bits); lane k costs candidate k
  uint32_t sad = 0;
#pragma unroll
  for (int k = 0; k < kCentreCands; k += 2) {
    const uint32_t w = wsum(vsad8(sv, r[k]) | (k + 1 < kCentreCands ? vsad8(sv, r[min(k + 1, kCentreCands - 1)]) << 16 : 0u));
    if ((lane >> 1) == (k >> 1)) sad = (w >> (16 * (lane & 1))) & 0xffffu;
  }
  const int k = min(lane, kCentreCands - 1);
  const uint32_t cost = sad + mvd_cost(cx[k] * 4 - mvp0, lambda) + mvd_cost(cy[k] * 4 - mvp1, lambda);
  const uint32_t key = __reduce_min_sync(FULL, lane < n && ok[k] ? (cost << 3) | (uint32_t)lane : UMAX);
  const int b = key == UMAX ? 0 : (int)(key & 7u);
  bx = cx[b];
  by = cy[b];
  return make_int2(bx, by);
}

// One macroblock of a P slice in the search forms (see the head of this file); false when a wait for
// the reference picture gave up (for shared search units: ss.job.failed).
__device__ __noinline__ bool analyse_p_mb_search(const Ctx c, const PipeWait pw) {
  const StreamDev& sd = sm.sd;
  const int lane = lane_id();
  const int mbx = c.mbx, mby = c.mby;
  const int x0 = mbx * 16, y0 = mby * 16;
  const uint32_t lambda = sm.qt[0].lambda;
  const Bounds bd = mv_bounds(x0, y0);
  const int imin0 = (bd.min0 + 3) >> 2, imin1 = (bd.min1 + 3) >> 2, imax0 = bd.max0 >> 2, imax1 = bd.max1 >> 2;
  __syncwarp();
  const uint32_t nw = load_nb(c);
  load_source(c);
  store_nb(nw);
  const uint32_t p16 = mv_pred(c_part[0]);
  const int mvp16[2] = {lo16((int)p16), (int)p16 >> 16};
  int ps0 = mvp16[0], ps1 = mvp16[1];
  const NbMv nbA = ss.nb[4], nbB = ss.nb[1];
  if (mbx == 0 || mby == 0 || (nbA.ref == 0 && nbA.mv == 0) || (nbB.ref == 0 && nbB.mv == 0)) ps0 = ps1 = 0;
  const rg_mb_hint* hint = sd.hint ? sd.hint + c.mb : nullptr;
  // integer window: full search, or the learned seed's small window
  const int R = sd.search_range;
  int fcx = min(max((mvp16[0] + 2) >> 2, imin0), imax0), fcy = min(max((mvp16[1] + 2) >> 2, imin1), imax1);
  int xlo = max(fcx - R, imin0), xhi = min(fcx + R, imax0), ylo = max(fcy - R, imin1), yhi = min(fcy + R, imax1);
  int part_mask = 15;
  // learned: the candidates of the first window's centre (integer, clamped to the bounds)
  int* ccx = ss.ccx;  // warp-uniform, in shared memory
  int* ccy = ss.ccy;
  bool* cok = ss.cok;
  if (hint) {
    const NbMv A = nbA, B = nbB, C = ss.nb[3].ref == -2 ? ss.nb[0] : ss.nb[3];
    const int vx[kCentreCands] = {mvp16[0] + hint->mv_off[0], mvp16[0], hint->mv_coarse[0], A.x(), B.x(), C.x(), 0};
    const int vy[kCentreCands] = {mvp16[1] + hint->mv_off[1], mvp16[1], hint->mv_coarse[1], A.y(), B.y(), C.y(), 0};
    const bool use[kCentreCands] = {true, true, (hint->flags & 1) != 0, A.ref == 0, B.ref == 0, C.ref == 0, true};
    xhi = -(1 << 20);
    yhi = -(1 << 20);
#pragma unroll
    for (int k = 0; k < kCentreCands; k++) {
      ccx[k] = min(max((vx[k] + 2) >> 2, imin0), imax0);
      ccy[k] = min(max((vy[k] + 2) >> 2, imin1), imax1);
      cok[k] = use[k];
      if (use[k]) {
        xhi = max(xhi, min(ccx[k] + kLearnedRange, imax0));
        yhi = max(yhi, min(ccy[k] + kLearnedRange, imax1));
      }
    }
    part_mask = hint->part_mask & 15;
    if (!part_mask) part_mask = 1;
  }
  // the reference region of the skip probe and the search window (learned: every candidate's)
  if (!wait_window(c, pw, max(xhi, (max(ps0, 0) + 3) >> 2), max(yhi, (max(ps1, 0) + 3) >> 2))) return false;
  if (lane == 0) sm.win_x = kNoWin;  // the last macroblock's window
  __syncwarp();
  // 1. skip probe
  if (in_bounds(bd, ps0, ps1) && skip_probe(c, ps0, ps1)) {
    code_skip(c, ps0, ps1);
    search_tail(c, 255, false, ps0, ps1);
    return true;
  }
  // 2. integer search
  if (hint) {
    const int2 lc = learned_centre(c, mvp16[0], mvp16[1], lambda);
    const int lcx = lc.x, lcy = lc.y;
    xlo = max(lcx - kLearnedRange, imin0);
    xhi = min(lcx + kLearnedRange, imax0);
    ylo = max(lcy - kLearnedRange, imin1);
    yhi = min(lcy + kLearnedRange, imax1);
  }
  IntBest& ib = ss.ib;  // warp-uniform: once per warp in shared memory
  int_search(c, xlo, xhi, ylo, yhi, mvp16[0], mvp16[1], lambda, pw);
  if (hint) {
    bool edge = (ib.x[0] == xlo && xlo > imin0) || (ib.x[0] == xhi && xhi < imax0) ||
                (ib.y[0] == ylo && ylo > imin1) || (ib.y[0] == yhi && yhi < imax1);
    for (int it = 0; edge && it < sd.walk; it++) {  // centre the window on its best again
      const int cx = ib.x[0], cy = ib.y[0];
      xlo = max(cx - kLearnedRange, imin0);
      xhi = min(cx + kLearnedRange, imax0);
      ylo = max(cy - kLearnedRange, imin1);
      yhi = min(cy + kLearnedRange, imax1);
      if (!wait_window(c, pw, xhi, yhi)) return false;
      int_search(c, xlo, xhi, ylo, yhi, mvp16[0], mvp16[1], lambda, pw);
      edge = (ib.x[0] == xlo && xlo > imin0) || (ib.x[0] == xhi && xhi < imax0) ||
             (ib.y[0] == ylo && ylo > imin1) || (ib.y[0] == yhi && yhi < imax1);
    }
    if (edge) {  // the walk did not reach the minimum: full search
      xlo = max(fcx - R, imin0); xhi = min(fcx + R, imax0);
      ylo = max(fcy - R, imin1); yhi = min(fcy + R, imax1);
      if (!wait_window(c, pw, xhi, yhi)) return false;
      int_search(c, xlo, xhi, ylo, yhi, mvp16[0], mvp16[1], lambda, pw);
    }
  }
  // 3-4. refinement of every tried type, the least total cost wins
  int best_t = -1;
  uint32_t best_j = UMAX;
  // lane k < 4: part k's vector and difference of the current and of the best type; their quadrants' vectors
  uint32_t mv_k = 0, mvd_k = 0, quad = 0, best_mv = 0, best_mvd = 0, best_quad = 0;
#pragma unroll 1
  for (int t = 0; t < 4; t++) {
    if (!((part_mask >> t) & 1)) continue;
    __syncwarp();
    const int own = 5 + (lane & 1) + 2 * (lane & 2);  // quadrant lane's place in ss.nb
    if (lane < 4) ss.nb[own] = NbMv{0u, -2};
    __syncwarp();
    uint32_t J = lambda * (uint32_t)sd.type_bits[t];
    const int first = type_first(t), np = type_parts(t);
    mvd_k = 0;
#pragma unroll 1
    for (int k = 0; k < np; k++) {
      const uint32_t part = c_part[first + k];
      const uint32_t mvp = mv_pred(part);
      const int bx = ss.ib.x[first + k], by = ss.ib.y[first + k];
      const int2 mp = make_int2(lo16((int)mvp), (int)mvp >> 16);
      const int px = (part >> 21) & 8u, py = (part >> 22) & 8u, pw = (part >> 26) & 1u ? 8 : 16, ph = (part >> 27) & 1u ? 8 : 16;
      const PartFit fit = hint ? refine_part_sad(c, px, py, pw, ph, bx, by, mp, lambda, bd,
                                                 ss.ib.c[first + k] - vec_cost(4 * bx - mvp16[0], 4 * by - mvp16[1], lambda))
                               : refine_part(c, px, py, pw, ph, bx, by, mp, lambda, bd);
      J += fit.cost;
      const uint32_t mv = pack16(fit.x, fit.y);
      if (lane == k) {
        mv_k = mv;
        mvd_k = pack16(fit.x - mp.x, fit.y - mp.y);
      }
      __syncwarp();
      if (lane < 4 && ((part >> (16 + lane)) & 1u)) {
        ss.nb[own] = NbMv{mv, 0};
        quad = mv;
      }
      __syncwarp();
    }
    if (J < best_j) {
      best_j = J;
      best_t = t;
      best_mv = mv_k;
      best_mvd = mvd_k;
      best_quad = quad;
    }
  }
  // quadrant vectors of the chosen type and its prediction
  if (lane < 4) {
    ss.qmv[lane][0] = lo16((int)best_quad);
    ss.qmv[lane][1] = (int)best_quad >> 16;
    ss.pmvd[lane] = best_mvd;
  }
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < type_parts(best_t); k++) {
    const int i = type_first(best_t) + k;
    const uint32_t part = c_part[i], mv = __shfl_sync(FULL, best_mv, k);
    predict_part(c, (part >> 21) & 8u, (part >> 22) & 8u, (part >> 26) & 1u ? 8 : 16, (part >> 27) & 1u ? 8 : 16, ss.ib.x[i], ss.ib.y[i],
                 lo16((int)mv), (int)mv >> 16);
  }
  // 5. intra 16x16 when the inter prediction is poor (the plain form's rule, enc.rs:3121-3156)
  const uint32_t inter_satd = satd16((int)offsetof(Smem, pred_y));
  if (inter_satd > 24 * lambda) {
    const Corner k0 = load_edges(c, false);
    bool ht = mby > 0, hl = mbx > 0;
    const I16Fit fit16 = analyse_i16(ht, hl, k0.y);
    if (fit16.cost + lambda * 8 < best_j) {
      code_i16(c, fit16.mode, ht, hl, k0);
      search_tail(c, best_t, false, 0, 0);
      return true;
    }
  }
  // residual, late skip (a 16x16 macroblock at the skip vector), record and reconstruction
  mc_chroma_q(c);
  const int type = best_t == 0 ? RG_MB_P_L0_16X16 : (best_t == 1 ? RG_MB_P_L0_16X8 : (best_t == 2 ? RG_MB_P_L0_8X16 : RG_MB_P_8X8));
  const uint32_t mv = __shfl_sync(FULL, best_mv, 0), mvd = __shfl_sync(FULL, best_mvd, 0);
  const bool skipped = code_inter(c, type, best_t == 0 && mv == pack16(ps0, ps1), lo16((int)mv), (int)mv >> 16, lo16((int)mvd),
                                  (int)mvd >> 16);
  search_tail(c, best_t, !skipped, ps0, ps1);
  return true;
}

// One macroblock of an I slice in the search forms: the plain analysis (enc.rs:3311 code_intra),
// intra 4x4 blocks restricted to the hinted modes in the learned form.
__device__ __noinline__ void analyse_intra_mb_search(const Ctx c) {
  const Corner k0 = load_edges(c, true);
  bool ht = c.mby > 0, hl = c.mbx > 0;
  uint32_t lambda = sm.qt[0].lambda;
  const I16Fit fit16 = analyse_i16(ht, hl, k0.y);
  if (fit16.cost > 40 * lambda) {
    const rg_mb_hint* hint = sm.sd.hint;
    const uint32_t masks = hint ? hint[c.mb].i4_mask[lane_id() & 15] : 0x1ffu;
    const int cbpl = analyse_i4(c, fit16.cost + lambda * 4, ht, hl, k0.y, masks);
    if (cbpl >= 0) {
      code_i4(c, cbpl, ht, hl, k0);
      search_tail(c, 255, false, 0, 0);
      return;
    }
  }
  code_i16(c, fit16.mode, ht, hl, k0);
  search_tail(c, 255, false, 0, 0);
}
