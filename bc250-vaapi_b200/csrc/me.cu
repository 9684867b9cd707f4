// me.cu - plain full-search block motion estimation, one CTA per 16x16 MB.
//
// Reference stage: A1/shaders/motion_estimation.comp (zero-MV early-out
// :312-331, lambda cost :363, half/quarter-pel refine :388-459 with the
// 6-tap interpolation of :154-215). The reference searches a diamond; the
// plain form here is exhaustive over [-R,R]^2 with a raster tie-break (the
// CPU oracle states the exact rule) and keeps the reference's refine.
//
// B200 layout: the (2R+24)^2 reference window (search range plus the 6-tap
// reach of the refine) is staged once in shared memory, by one 2-D TMA load
// (cp.async.bulk.tensor, no multicast) of a box that starts on the 16-byte
// boundary 12 bytes left of the window when the window lies inside the
// reference plane, by clamped word loads into the same layout at the picture
// edges and in batched steps. The search is exhaustive by elimination:
//   1. a lower bound of every candidate's cost, thread t owning column
//      dx = t - R: the SAD is at least the sum over the four 8x8 blocks of
//      |difference of the blocks' sample sums| (successive elimination, Li and
//      Salari 1995), formed from running 8-row sums of the column's samples
//      (dp4a on masked words, sad.u32);
//   2. an upper bound: the exact costs of the zero vector, of each column's
//      candidate of smallest bound and of the column dx = +R;
//   3. the exact SADs of every run of eight candidates of a column whose bound
//      does not exceed it, listed and searched a run per thread: each window
//      row's 16 bytes (one funnel shift per word off 5 aligned shared loads)
//      feed the runs' candidates that use it (vabsdiff4 with add).
// A candidate is dropped only when its bound exceeds a cost another candidate
// has, so the winner and the raster tie-break are the exhaustive search's.
//
// What bounds it: the integer ALU (vabsdiff4, funnel shifts, sad at 64 lanes
// per clock and SM) and the issue slots; a 1080p window set is 4 MB of DRAM.
// Scoring every candidate in an 80-row sweep took 244 us for a 1080p frame at
// R = 32 (ALU pipe 81 %, a fifth of it on rows outside the range) and 123 at
// R = 16 with a scalar refine; now, on textured video with 10 % uniform noise,
// 146 and 70 (30 and 50 % of the runs survive), 90 and 49 on smooth video
// (2 %); on uniform noise, where every run survives, 243 and 83.
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "b200enc_internal.h"
#include "me_common.cuh"
#include "umma.cuh"

namespace b200enc {

constexpr int kMeUnit = 8;  // candidates of a column searched (or ruled out) together

template <int R>
struct MeShared {
  static constexpr int WP = 2 * R + 24;                   // window side in pels
  static constexpr int WW = WP / 4;                       // 32-bit words of a window row
  static constexpr int OFF = 3;                           // window column 0 sits 12 bytes into a staged row
  static constexpr int BW = (4 * OFF + WP + 15) / 16 * 16;  // staged row: the TMA box width in bytes
  static constexpr int WS = BW / 4;                       // 32-bit words per staged row
  alignas(128) uint32_t win[WP * WS];
  alignas(16) uint32_t cur[64];
  uint32_t red[8];
  uint16_t ubound[2 * R * (2 * R / kMeUnit)];  // half (rounded down) of each unit's smallest bound
  uint32_t nlist;                          // units to search exactly
  uint16_t list[2 * R * (2 * R / kMeUnit)];
  uint64_t bar;  // TMA completion
  RefineSimd rf;
};
static_assert(MeShared<16>::BW == 80 && MeShared<32>::BW == 112, "box widths");

// Where a CTA's macroblocks come from (MODE): 0 one CTA per MB of one frame;
// 1 a persistent grid over a list of that frame's MBs; 2 a persistent grid
// over every P macroblock of a batch; 3 over a list of compact batch P
// indices (the learned form's fallback in a batch). The search itself is
// the same in all four.
enum : int { kMeGrid = 0, kMeList = 1, kMeBatch = 2, kMeBatchList = 3 };

// Error word of launches given no scratch word (b200enc_me_wait_errors).
__device__ uint32_t g_me_wait_err;

// CTAs of one SM the kernel is compiled for: 30 warps of 64 registers (20
// warps of 96, all of the current macroblock in registers: 152 us for the
// 1080p frame that takes 149 at 30, before the smaller refine).
template <int R>
constexpr int kMeCtas = R == 32 ? 15 : 30;

// Threads per macroblock. One per column of the search area (SEG = 1) does the
// least work, and is what a picture that fills the chip takes; with few macroblocks
// the chip idles while each is a serial chain, so SEG threads share a column: each
// bounds its part of the rows (two fills of the rings more), and staging and the
// exact costs have SEG times the threads. The line lies where both take the same
// time (us, SEG = 1 / wide): at +-16 99 macroblocks 17.6 / 8.1, 396 17.9 / 11.3, 690
// 20.1 / 14.5, 1,200 22.1 / 22.0, 1,900 27.6 / 30.0; at +-32 99 21.3 / 13.0, 690
// 28.2 / 23.6, 2,304 55.2 / 53.1, 3,600 72.2 / 76.1: 8 and 16 macroblocks per SM. A
// list's length is known on the device only: a learned search leaves a tenth of a
// frame, beside the re-scoring of the rest (fallback alone / pair: 98 of 1,200
// macroblocks 18.5 / 9.7 us, 583 of 8,160 pair 36.8 / 33.0, 898 of 14,400 56.6 / 53.3,
// 2,215 of 32,400 108.9 / 112.0), so its line is 100 per SM. Batches, whose lists hold
// whole frames without history, keep SEG = 1 (eight mixed streams 4.02 ms, not 4.10).
template <int R>
constexpr int kMeSeg = R == 16 ? 4 : 2;
constexpr int kMeWideList = 100;

template <int R, int MODE, int SEG>
__global__ void __launch_bounds__(2 * R * SEG, kMeCtas<R> / SEG) me_full_search_kernel(const uint8_t* __restrict__ cur_, int cur_pitch_,
                                                               const uint8_t* __restrict__ ref_, int ref_pitch_,
                                                               Geo g_, int lambda_, int zero_thresh_,
                                                               MV* __restrict__ out_, const int* __restrict__ mb_list,
                                                               const int* __restrict__ mb_count, int flags,
                                                               BatchTab bt, const __grid_constant__ CUtensorMap tmap,
                                                               int use_tma, uint32_t* err) {
  constexpr int NT = 2 * R * SEG, COLS = 2 * R;
  using S = MeShared<R>;
  constexpr int WP = S::WP, WW = S::WW, WS = S::WS, OFF = S::OFF, SIDE = 2 * R + 1;
  constexpr uint64_t kWaitNs = 2000000000ull;
  __shared__ S sh;
  // The refine, the corner candidate and a last partial round of units run on
  // the first logical warp; every other CTA swaps its warps, so that this work
  // does not always fall to the same two of an SM's four schedulers.
  const int tid = NT > 32 ? (int)(threadIdx.x ^ (((blockIdx.x + blockIdx.y) & 1u) << 5)) : (int)threadIdx.x;
  // the map describes this launch's single reference plane; batched steps
  // read one plane per stream and stage with loads
  const bool tma_ok = (MODE == kMeGrid || MODE == kMeList) && use_tma;
  uint32_t phase = 0;
  if (tma_ok) {
    if (tid == 0) {
      mbar_init(&sh.bar, 1);
      fence_async_smem();
    }
    __syncthreads();
  }
  const int n_items = MODE == kMeGrid ? 1 : (MODE == kMeBatch ? bt.p_mbs.total() : *mb_count);
  for (int item = MODE == kMeGrid ? 0 : (int)blockIdx.x; item < n_items; item += MODE == kMeGrid ? 1 : (int)gridDim.x) {
  int mbx = blockIdx.x, mby = blockIdx.y;
  const uint8_t* cur = cur_;
  const uint8_t* ref = ref_;
  int cur_pitch = cur_pitch_, ref_pitch = ref_pitch_, lambda = lambda_, zero_thresh = zero_thresh_;
  Geo g = g_;
  MV* o;
  if (MODE == kMeList) {
    const int mb = mb_list[item];
    mby = mb / g.mbw;
    mbx = mb - mby * g.mbw;
  }
  if (MODE == kMeBatch || MODE == kMeBatchList) {
    const int ci = MODE == kMeBatch ? item : mb_list[item];
    const int k = bt.p_mbs.find(ci);
    const BatchStream& st = bt.p_mbs.stream(k);
    const int local = ci - bt.p_mbs.prefix[k];
    g = st.g;
    mby = local / g.mbw;
    mbx = local - mby * g.mbw;
    cur = st.cur_y;
    cur_pitch = st.cur_pitch;
    ref = st.ref_y;
    ref_pitch = st.rec_pitch;
    lambda = st.lambda;
    zero_thresh = st.zero_thresh;
    o = bt.mvc + ci;
  } else {
    o = out_ + (size_t)mby * g.mbw + mbx;
  }
  if (MODE != kMeGrid) {
    if (tma_ok) fence_async_smem();  // this thread's accesses of the window precede the next TMA write
    __syncthreads();                 // the previous item's shared memory is no longer read
  }
  if ((MODE == kMeBatch || MODE == kMeBatchList) && mby >= g.mbh) continue;  // padding of the compact index
  const int X = mbx * 16, Y = mby * 16;
  const int ox = X - R - 4, oy = Y - R - 4;  // window origin (multiple of 4)

  // ---- stage the reference window and the current MB --------------------
  // A window inside the plane needs no clamping: one TMA box of WP rows of
  // BW bytes from column ox - 12 (a multiple of 16: ox = X - R - 4 with X a
  // multiple of 16 and R 16 or 32); the bytes either side of the window in
  // the box are never read.
  const bool tma = tma_ok && ox >= 0 && ox + WP <= g.RW && oy >= 0 && oy + WP <= g.RH;
  if (tma) {
    if (tid == 0) {
      mbar_arrive_expect_tx(&sh.bar, (uint32_t)(S::BW * WP));
      tma_load_2d(sh.win, &tmap, ox - 4 * OFF, oy, &sh.bar);
    }
  } else {
    for (int i = tid; i < WP * WW; i += NT) {
      const int row = i / WW, w = i - row * WW;
      const int gy = clampi(oy + row, 0, g.RH - 1);
      sh.win[row * WS + OFF + w] = load_word_clamped(ref + (size_t)gy * ref_pitch, ox + 4 * w, g.RW);
    }
  }
  for (int i = tid; i < 64; i += NT) {
    const int r = i >> 2, w = i & 3;
    const uint8_t* cp = cur + (size_t)clampi(Y + r, 0, g.H - 1) * cur_pitch;
    const int gx = X + 4 * w;
    uint32_t v;
    if (gx + 3 < g.W) {
      v = __ldg(reinterpret_cast<const uint32_t*>(cp + gx));
    } else {
      v = (uint32_t)__ldg(cp + min(gx, g.W - 1)) | ((uint32_t)__ldg(cp + min(gx + 1, g.W - 1)) << 8) |
          ((uint32_t)__ldg(cp + min(gx + 2, g.W - 1)) << 16) | ((uint32_t)__ldg(cp + min(gx + 3, g.W - 1)) << 24);
    }
    sh.cur[i] = v;
  }
  bool waited = true;
  if (tma) {
    waited = mbar_wait(&sh.bar, phase, kWaitNs);
    phase ^= 1u;
  }
  if (__syncthreads_or(!waited)) {
    // the window never arrived: report, give the copy one more bounded
    // wait, leave this CTA's remaining macroblocks unwritten
    if (tid == 0) {
      uint32_t* e = err ? err : &g_me_wait_err;
      if (atomicCAS(e, 0u, kErrWaitTimeout) == 0u && err) atomicExch(err + 1, (uint32_t)(mby * g.mbw + mbx));
      *o = MV{0, 0, 0xffffffffu, 0u};
      mbar_wait(&sh.bar, phase ^ 1u, kWaitNs);
    }
    return;
  }

  // ---- zero-MV check (motion_estimation.comp:312-331) --------------------
  uint32_t z = 0;
  for (int i = tid; i < 64; i += NT) {
    const int r = i >> 2, w = i & 3;
    z = sad4_acc(sh.cur[i], sh.win[(R + 4 + r) * WS + OFF + (R + 4) / 4 + w], z);
  }
  const uint32_t sad0 = block_sum<NT>(z, sh.red);
  if (zero_thresh >= 0 && sad0 <= (uint32_t)zero_thresh) {
    if (tid == 0) *o = MV{0, 0, sad0, (flags & B200ENC_ME_LOG_INTEGER) ? me_log_word(0, 0, true) : 0u};
    continue;
  }

  // ---- integer full search ------------------------------------------------
  // 1. Lower bounds of every candidate's cost, a column per thread: the SAD of
  // a 16x16 block is at least the sum over its four 8x8 blocks of the
  // difference of their sample sums. Each window row gives the column's two
  // 8-sample sums (packed in halves of a word), a ring keeps the last eight.
  const int lam = lambda;
  const int col = tid & (COLS - 1), seg = tid / COLS;  // this thread's column and share of its rows
  const uint32_t lam_dx = (uint32_t)lam * (uint32_t)abs(col - R);
  const uint32_t* wcol = sh.win + 4 * WS + OFF + ((col + 4) >> 2);  // window row 0 of this thread's column
  const int wsh = ((col + 4) & 3) * 8;
  constexpr int NU = 2 * R / kMeUnit / SEG;  // units (runs of kMeUnit candidates) of a column per thread
  const int u0 = seg * NU;
  uint32_t lkey, ckey = 0xffffffffu;   // smallest (bound << 14 | raster index) of the last row, of the column
  {
    uint32_t c00, c01, c10, c11;  // the current macroblock's 8x8 sums
    {
      const uint32_t w0 = sh.cur[2 * lane_id()], w1 = sh.cur[2 * lane_id() + 1];  // a lane per half row
      uint32_t s8 = __dp4a(w1, 0x01010101u, __dp4a(w0, 0x01010101u, 0u));
#pragma unroll
      for (int o = 2; o < 16; o <<= 1) s8 += __shfl_xor_sync(0xffffffffu, s8, o);
      c00 = __shfl_sync(0xffffffffu, s8, 0);
      c01 = __shfl_sync(0xffffffffu, s8, 1);
      c10 = __shfl_sync(0xffffffffu, s8, 16);
      c11 = __shfl_sync(0xffffffffu, s8, 17);
    }
    // Rings over the last eight rows: row sums, sums of the eight rows ending
    // at a row, of the column's left and right eight samples. Candidate cy
    // covers window rows cy .. cy + 15 of the column: its upper sums ended at
    // row cy + 7, its lower ones end at cy + 15. The first two passes (rows
    // -1 .. 14) only fill the rings.
    uint32_t hl[8], hr[8], vl[8], vr[8], rl = 0, rr = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) hl[k] = hr[k] = vl[k] = vr[k] = 0;
    // An unaligned run of eight bytes is the sum of three words' masked bytes.
    const uint32_t m0 = 0x01010101u << wsh, m2 = wsh ? 0x01010101u >> (32 - wsh) : 0u;
    auto bound = [&](int k, int cy) -> uint32_t {  // k = cy & 7, a constant
      const uint32_t* rp = wcol + (cy + 15) * WS;
      const uint32_t w0 = rp[0], w1 = rp[1], w2 = rp[2], w3 = rp[3], w4 = rp[4];
      const uint32_t nl = __dp4a(w2, m2, __dp4a(w1, 0x01010101u, __dp4a(w0, m0, 0u)));
      const uint32_t nr = __dp4a(w4, m2, __dp4a(w3, 0x01010101u, __dp4a(w2, m0, 0u)));
      rl += nl - hl[k];
      rr += nr - hr[k];
      hl[k] = nl;
      hr[k] = nr;
      uint32_t lb = lam_dx + (uint32_t)(lam * abs(cy - R));
      lb = __usad(rr, c11, __usad(rl, c10, __usad(vr[k], c01, __usad(vl[k], c00, lb))));
      vl[k] = rl;
      vr[k] = rr;
      return (lb << 14) | (uint32_t)(cy * SIDE + col);
    };
#pragma unroll 1
    for (int u = u0 - 2; u < u0 + NU; ++u) {
      uint32_t m = 0xffffffffu;
#pragma unroll
      for (int k = 0; k < kMeUnit; ++k) m = min(m, bound(k & 7, u * kMeUnit + k));
      if (u >= u0) {
        sh.ubound[u * COLS + col] = (uint16_t)(m >> 15);
        ckey = min(ckey, m);
      }
    }
    lkey = seg == SEG - 1 ? bound(0, 2 * R) : 0xffffffffu;
    ckey = min(ckey, lkey);
  }

  // 2. An upper bound: the exact costs of the zero vector, of each thread's
  // candidate of smallest bound and of the column dx = +R (aligned words).
  auto key_of = [&](uint32_t sad, int cx, int cy) -> uint32_t {
    return ((sad + (uint32_t)(lam * (abs(cx - R) + abs(cy - R)))) << 14) | (uint32_t)(cy * SIDE + cx);
  };
  auto exact = [&](int cx, int cy) -> uint32_t {
    const uint32_t* rp = sh.win + (4 + cy) * WS + OFF + ((cx + 4) >> 2);
    const int xs = ((cx + 4) & 3) * 8;
    uint32_t s = 0;
#pragma unroll 2
    for (int r = 0; r < 16; ++r, rp += WS) {
      const uint4 c = reinterpret_cast<const uint4*>(sh.cur)[r];
      const uint32_t w0 = rp[0], w1 = rp[1], w2 = rp[2], w3 = rp[3], w4 = rp[4];
      s = sad4_acc(__funnelshift_r(w0, w1, xs), c.x, s);
      s = sad4_acc(__funnelshift_r(w1, w2, xs), c.y, s);
      s = sad4_acc(__funnelshift_r(w2, w3, xs), c.z, s);
      s = sad4_acc(__funnelshift_r(w3, w4, xs), c.w, s);
    }
    return key_of(s, cx, cy);
  };
  uint32_t best = key_of(sad0, R, R);
#pragma unroll 1
  for (int j = 0; j < (seg == SEG / 2 ? 2 : 1); ++j)
    best = min(best, j ? exact(2 * R, col) : exact(col, (int)(ckey & 0x3fffu) / SIDE));
  if (tid < 32) {  // the corner (+R, +R): a row per lane
    const uint32_t* rp = sh.win + (4 + 2 * R + (tid & 15)) * WS + OFF + (2 * R + 4) / 4;
    const uint4 c = reinterpret_cast<const uint4*>(sh.cur)[tid & 15];
    uint32_t s = sad4_acc(rp[3], c.w, sad4_acc(rp[2], c.z, sad4_acc(rp[1], c.y, sad4_acc(rp[0], c.x, 0u))));
    s = __reduce_add_sync(0xffffffffu, tid < 16 ? s : 0u);
    best = min(best, key_of(s, 2 * R, 2 * R));
  }
  best = block_min<NT>(best, sh.red);

  // 3. The units whose bound does not exceed it, listed unit row by unit row
  // (neighbouring columns stay neighbours: their window words are in
  // different banks), and their exact costs, one unit per thread: kMeUnit
  // candidates share the window rows they have in common.
  const uint32_t ub = best >> 14;
  {
    uint32_t alive[NU], total = 0;
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      alive[u] = __ballot_sync(0xffffffffu, 2u * sh.ubound[(u0 + u) * COLS + col] <= ub);
      total += (uint32_t)__popc(alive[u]);
    }
    const int lane = lane_id();
    uint32_t base = 0;
    if (NT > 32) {
      if (tid == 0) sh.nlist = 0;
      __syncthreads();
      if (lane == 0 && total) base = atomicAdd(&sh.nlist, total);
      base = __shfl_sync(0xffffffffu, base, 0);
    } else if (lane == 0) {
      sh.nlist = total;
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      if ((alive[u] >> lane) & 1u) sh.list[base + __popc(alive[u] & ((1u << lane) - 1u))] = (uint16_t)((u0 + u) * COLS + col);
      base += (uint32_t)__popc(alive[u]);
    }
    if ((lkey >> 14) <= ub) best = min(best, exact(col, 2 * R));
    if (NT > 32) __syncthreads();
    else __syncwarp();
  }
  const int n_units = (int)sh.nlist;
#pragma unroll 1
  for (int i = tid; i < n_units; i += NT) {
    const int e = sh.list[i], cx = e & (COLS - 1), cy0 = (e / COLS) * kMeUnit;
    const uint32_t* up = sh.win + (4 + cy0) * WS + OFF + ((cx + 4) >> 2);
    const int us = ((cx + 4) & 3) * 8;
    uint32_t acc[kMeUnit];
#pragma unroll
    for (int c = 0; c < kMeUnit; ++c) acc[c] = 0;
    // the macroblock's upper, then its lower eight rows: 32 registers of
    // current samples instead of 64, which lets twice the CTAs share an SM
#pragma unroll 1
    for (int hb = 0; hb < 2; ++hb, up += 8 * WS) {
      uint32_t cw[8][4];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const uint4 c = reinterpret_cast<const uint4*>(sh.cur)[8 * hb + r];
        cw[r][0] = c.x;
        cw[r][1] = c.y;
        cw[r][2] = c.z;
        cw[r][3] = c.w;
      }
#pragma unroll
      for (int k = 0; k < kMeUnit + 7; ++k) {
        const uint32_t* rp = up + k * WS;
        const uint32_t w0 = rp[0], w1 = rp[1], w2 = rp[2], w3 = rp[3], w4 = rp[4];
        const uint32_t r0 = __funnelshift_r(w0, w1, us), r1 = __funnelshift_r(w1, w2, us);
        const uint32_t r2 = __funnelshift_r(w2, w3, us), r3 = __funnelshift_r(w3, w4, us);
#pragma unroll
        for (int c = 0; c < kMeUnit; ++c) {
          const int r = k - c;
          if (r < 0 || r > 7) continue;
          acc[c] =
              sad4_acc(r3, cw[r][3], sad4_acc(r2, cw[r][2], sad4_acc(r1, cw[r][1], sad4_acc(r0, cw[r][0], acc[c]))));
        }
      }
    }
#pragma unroll
    for (int c = 0; c < kMeUnit; ++c) best = min(best, key_of(acc[c], cx, cy0 + c));
  }
  best = block_min<NT>(best, sh.red);
  const int idx = (int)(best & 0x3fffu);
  const int mx = idx % SIDE - R, my = idx / SIDE - R;
  const uint32_t int_sad = (best >> 14) - (uint32_t)lambda * (uint32_t)(abs(mx) + abs(my));

  // ---- half/quarter-pel refine around the winner (one warp) ---------------
  if (tid < 32) {
    int qx, qy;
    const uint32_t bsad =
        qpel_refine_warp_simd(sh.rf, reinterpret_cast<const uint8_t*>(sh.win) + 4 * OFF, S::BW, my + R + 4, mx + R + 4,
                              sh.cur, int_sad, &qx, &qy);
    if (tid == 0)
      *o = MV{4 * mx + qx, 4 * my + qy, bsad, (flags & B200ENC_ME_LOG_INTEGER) ? me_log_word(mx, my, false) : 0u};
  }
  }
}

}  // namespace b200enc

using namespace b200enc;

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Tensor map of a reference luma plane (RW x RH bytes, `pitch` apart) whose
// box is one search window of range R: MeShared<R>::BW bytes by WP rows.
// False when TMA cannot describe the plane (base or pitch not 16-byte
// aligned, a plane smaller than the box), the plane is not device memory
// (page-locked or managed host memory is staged with loads), or staging by
// TMA is tuned off; the kernel then stages every window with loads.
template <int R>
bool window_map(CUtensorMap* m, const uint8_t* ref, int pitch, int RW, int RH) {
  using S = MeShared<R>;
  memset(m, 0, sizeof(*m));
  if (b200enc_tuned(B200ENC_TUNE_ME_STAGE) == 1) return false;
  if ((reinterpret_cast<uintptr_t>(ref) & 15) || (pitch & 15) || RW < S::BW || RH < S::WP) return false;
  cudaPointerAttributes pa;
  if (cudaPointerGetAttributes(&pa, ref) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (pa.type != cudaMemoryTypeDevice) return false;
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)RW, (cuuint64_t)RH};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch};
  const cuuint32_t box[2] = {(cuuint32_t)S::BW, (cuuint32_t)S::WP};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(ref), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int R>
void launch_frame(dim3 grid, bool list, const uint8_t* cur_y, int cur_pitch, const uint8_t* ref_y, int ref_pitch,
                  const Geo& g, int lambda, int zero_thresh, MV* out, const int* mb_list, const int* mb_count,
                  int flags, int capacity, int sms, uint32_t* err, cudaStream_t st) {
  CUtensorMap map;
  const int use_tma = window_map<R>(&map, ref_y, ref_pitch, g.RW, g.RH) ? 1 : 0;
  const BatchTab none{};
  auto launch = [&](auto k, int threads) {
    k<<<grid, threads, 0, st>>>(cur_y, cur_pitch, ref_y, ref_pitch, g, lambda, zero_thresh, out, mb_list, mb_count, flags, none,
                                map, use_tma, err);
  };
  constexpr int kSeg = kMeSeg<R>;
  if (list) {
    if (capacity <= kMeWideList * sms)
      launch(me_full_search_kernel<R, kMeList, kSeg>, 2 * R * kSeg);
    else
      launch(me_full_search_kernel<R, kMeList, 1>, 2 * R);
  } else {
    if (g.mbw * g.mbh <= (R == 16 ? 8 : 16) * sms)
      launch(me_full_search_kernel<R, kMeGrid, kSeg>, 2 * R * kSeg);
    else
      launch(me_full_search_kernel<R, kMeGrid, 1>, 2 * R);
  }
}

}  // namespace

// b200enc_me_full_search_ex with the error word of a wavefront scratch
// region: a window copy that never completes sets err[0] (kErrWaitTimeout)
// and err[1] (the macroblock). err == nullptr: the library's own word, read
// by b200enc_me_wait_errors.
int b200enc_me_full_search_err(const uint8_t* cur_y, int cur_pitch, const uint8_t* ref_y, int ref_pitch, int W,
                               int H, int RW, int RH, int range, int lambda, int zero_thresh, void* mv_out,
                               const int* mb_list, const int* mb_count, int list_capacity, int flags, uint32_t* err,
                               cudaStream_t st) {
  if (!cur_y || !ref_y || !mv_out || W <= 0 || H <= 0 || RW <= 0 || RH <= 0) return -1;
  if ((cur_pitch & 3) || (ref_pitch & 3) || (((uintptr_t)cur_y) & 3) || (((uintptr_t)ref_y) & 3)) return -1;
  if (lambda < 0 || lambda > 1023) return -1;
  if ((mb_list == nullptr) != (mb_count == nullptr)) return -1;
  Geo g{W, H, RW, RH, (W + 15) / 16, (H + 15) / 16};
  if (mb_list && (list_capacity <= 0 || list_capacity > g.mbw * g.mbh)) return -1;
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // list mode: a persistent grid of up to 16 CTAs per SM (or the tuned
  // count) walks the list
  const int per_sm = b200enc_tuned(B200ENC_TUNE_FALLBACK_CTAS_PER_SM) > 0 ? b200enc_tuned(B200ENC_TUNE_FALLBACK_CTAS_PER_SM) : 16;
  dim3 grid = mb_list ? dim3(std::min(list_capacity, per_sm * sms)) : dim3(g.mbw, g.mbh);
  const bool list = mb_list != nullptr;
  switch (range) {
    case 16:
      launch_frame<16>(grid, list, cur_y, cur_pitch, ref_y, ref_pitch, g, lambda, zero_thresh, (MV*)mv_out, mb_list,
                       mb_count, flags, list_capacity, sms, err, st);
      break;
    case 32:
      launch_frame<32>(grid, list, cur_y, cur_pitch, ref_y, ref_pitch, g, lambda, zero_thresh, (MV*)mv_out, mb_list,
                       mb_count, flags, list_capacity, sms, err, st);
      break;
    default:
      return -1;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int b200enc_me_full_search_ex(const uint8_t* cur_y, int cur_pitch, const uint8_t* ref_y, int ref_pitch,
                                         int W, int H, int RW, int RH, int range, int lambda, int zero_thresh,
                                         void* mv_out, const int* mb_list, const int* mb_count, int list_capacity,
                                         int flags, void* stream) {
  return b200enc_me_full_search_err(cur_y, cur_pitch, ref_y, ref_pitch, W, H, RW, RH, range, lambda, zero_thresh,
                                    mv_out, mb_list, mb_count, list_capacity, flags, nullptr, (cudaStream_t)stream);
}

extern "C" int b200enc_me_full_search(const uint8_t* cur_y, int cur_pitch, const uint8_t* ref_y, int ref_pitch,
                                      int W, int H, int RW, int RH, int range, int lambda, int zero_thresh,
                                      void* mv_out, void* stream) {
  return b200enc_me_full_search_ex(cur_y, cur_pitch, ref_y, ref_pitch, W, H, RW, RH, range, lambda, zero_thresh,
                                   mv_out, nullptr, nullptr, 0, 0, stream);
}

extern "C" int b200enc_me_wait_errors(int clear) {
  uint32_t v = 0;
  if (cudaMemcpyFromSymbol(&v, g_me_wait_err, 4) != cudaSuccess) return -1;
  if (clear && v) {
    const uint32_t zero = 0;
    if (cudaMemcpyToSymbol(g_me_wait_err, &zero, 4) != cudaSuccess) return -1;
  }
  return (int)v;
}

// Batched full search: every P macroblock of a batch (list == nullptr: a
// persistent grid of `ctas` CTAs over the compact P index), or the compact
// indices of a list (the learned form's fallback). MVs go to bt.mvc.
int b200enc_me_batch_launch(const BatchTab& bt, int range, const int* list, const int* count, int ctas,
                            cudaStream_t st) {
  if (ctas <= 0) return -1;
  CUtensorMap none;
  memset(&none, 0, sizeof(none));
  switch (range) {
    case 16:
      if (list)
        me_full_search_kernel<16, kMeBatchList, 1><<<ctas, 32, 0, st>>>(nullptr, 0, nullptr, 0, Geo{}, 0, 0, nullptr,
                                                                     list, count, 0, bt, none, 0, nullptr);
      else
        me_full_search_kernel<16, kMeBatch, 1><<<ctas, 32, 0, st>>>(nullptr, 0, nullptr, 0, Geo{}, 0, 0, nullptr, nullptr,
                                                                 nullptr, 0, bt, none, 0, nullptr);
      break;
    case 32:
      if (list)
        me_full_search_kernel<32, kMeBatchList, 1><<<ctas, 64, 0, st>>>(nullptr, 0, nullptr, 0, Geo{}, 0, 0, nullptr,
                                                                     list, count, 0, bt, none, 0, nullptr);
      else
        me_full_search_kernel<32, kMeBatch, 1><<<ctas, 64, 0, st>>>(nullptr, 0, nullptr, 0, Geo{}, 0, 0, nullptr, nullptr,
                                                                 nullptr, 0, bt, none, 0, nullptr);
      break;
    default:
      return -1;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
