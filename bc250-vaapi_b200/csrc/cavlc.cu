// cavlc.cu - CAVLC slice data (H.264 clause 7.3.4 / 9.2) on the GPU.
//
// The reference's host encoder entropy-codes a picture's slices after the
// GPU stages (A1/src/encoder_h264.c:3128-3290 for CAVLC): I slices code every
// macroblock as I16x16 (encode_mb_i16x16, :1120), P slices skip the
// macroblocks that qualify (:3236-3255) and code the others as mb_skip_run +
// P_L0_16x16 (encode_mb_p16x16, :1248). Nothing in that loop is sequential
// except two things: each block's nC is the neighbours' TotalCoeff, and each
// coded macroblock is preceded by the run of skipped macroblocks before it.
// Both are known up front: TotalCoeff is the number of nonzero levels the
// block codes (the staged nz masks), and the skip decision depends only on the
// macroblock's own levels and the vectors around it. So the slice data is
// built in three launches over the picture's staged outputs (levels, DC, nz
// masks, modes, vectors), all in device memory:
//   1. cavlc_mb_kernel: per macroblock (a warp, a lane per block), the skip
//      decision, coded block pattern and nC, then its header and residual bits
//      into a private region of the scratch;
//   2. cavlc_slice_kernel: per slice (one CTA), the skip runs and every
//      macroblock's bit offset (two block-wide scans), the slice's length;
//   3. cavlc_gather_kernel: each output word collects the bits that fall into
//      it (slice header, skip runs, macroblocks, trailing bits) and is stored
//      as stream bytes.
// The output is each slice's RBSP (header + slice data + trailing bits), ready
// for emulation prevention and a NAL header, bit for bit the reference's.
//
// What bounds it: instruction issue in the serial symbol loop of the densest
// block of each macroblock, and, below 640x480, the launches themselves. The
// macroblock kernel keeps one copy of each writer (37 KB of code; with the
// writers inlined at every call it was 152 KB, most of it fetched cold), and
// the gather replaced clearing the words, atomics into them and a byte swap.
// Before (five launches and a clear) and now, us: a 176x144 P picture 41 and
// 19, 640x480 39 and 23, a 1280x720 I picture at QP 20 81 and 33 (its 360 KB
// to mapped host memory take 7 at the bus's rate), a 1080p P picture at QP 22
// 44 and 32.
#include <algorithm>

#include "b200enc_internal.h"
#include "cavlc_core.h"
#include "common.cuh"
#include "t8x8.cuh"

namespace b200enc {

using namespace b200cavlc;

constexpr int kCavlcMbWords = 640;  // 2560 bytes of bits per macroblock at most (the reference's CAVLC allowance)
constexpr int kCavlcMaxSlices = 16;
constexpr int kCavlcScanThreads = 1024;
constexpr uint32_t kCavlcOver = 0xffffffffu;
constexpr uint32_t kCavlcNoRun = 0xffffffffu;

// The code tables as words of (length << 8 | code), in device memory (not
// __constant__: lanes index them at different positions, which the constant
// cache would serialise).
struct CavlcTabs {
  uint16_t ct[5][68];    // coeff_token: [nC class, 4 chroma DC][TotalCoeff * 4 + TrailingOnes]
  uint16_t tz[15][16];   // total_zeros: [TotalCoeff - 1][total_zeros]
  uint16_t cdtz[3][4];   // of chroma DC
  uint16_t run[7][16];   // run_before: [min(zerosLeft, 7) - 1][run_before]
};
constexpr CavlcTabs make_cavlc_tabs() {
  constexpr uint8_t ctl[5][68] = B200_CAVLC_COEFF_TOKEN_LEN, ctc[5][68] = B200_CAVLC_COEFF_TOKEN_CODE;
  constexpr uint8_t tzl[15][16] = B200_CAVLC_TOTAL_ZEROS_LEN, tzc[15][16] = B200_CAVLC_TOTAL_ZEROS_CODE;
  constexpr uint8_t cdl[3][4] = B200_CAVLC_CDC_TOTAL_ZEROS_LEN, cdc[3][4] = B200_CAVLC_CDC_TOTAL_ZEROS_CODE;
  constexpr uint8_t rl[7][16] = B200_CAVLC_RUN_LEN, rc[7][16] = B200_CAVLC_RUN_CODE;
  CavlcTabs t{};
  for (int i = 0; i < 5; ++i)
    for (int j = 0; j < 68; ++j) t.ct[i][j] = (uint16_t)(ctl[i][j] << 8 | ctc[i][j]);
  for (int i = 0; i < 15; ++i)
    for (int j = 0; j < 16; ++j) t.tz[i][j] = (uint16_t)(tzl[i][j] << 8 | tzc[i][j]);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 4; ++j) t.cdtz[i][j] = (uint16_t)(cdl[i][j] << 8 | cdc[i][j]);
  for (int i = 0; i < 7; ++i)
    for (int j = 0; j < 16; ++j) t.run[i][j] = (uint16_t)(rl[i][j] << 8 | rc[i][j]);
  return t;
}
static __device__ const CavlcTabs d_cavlc = make_cavlc_tabs();
static __device__ const uint8_t d_cbp_code[48] = B200_CAVLC_INTER_CBP_CODE;

// spec luma block index (8x8 quadrants, then 4x4 within) -> block column / row
__device__ __forceinline__ int blk_x4(int k) { return (k & 1) | ((k >> 1) & 2); }
__device__ __forceinline__ int blk_y4(int k) { return ((k >> 1) & 1) | ((k >> 2) & 2); }
__device__ __forceinline__ int spec_blk(int y4, int x4) { return ((y4 >> 1) << 3) | ((x4 >> 1) << 2) | ((y4 & 1) << 1) | (x4 & 1); }

// Per-slice header bits (MSB first) of a launch, passed by value.
struct CavlcHdr {
  uint32_t bits[kCavlcMaxSlices][4];
  int len[kCavlcMaxSlices];
};

// A frame's motion field and status words for the host, stored by the macroblock
// kernel on its way (mv null: none; s1 null: no such word, 0).
struct CavlcStage {
  MV* mv;
  const uint32_t *s0, *s1;
  uint32_t* status;
};

struct CavlcArgs {
  CavlcStage stage;
  int mbw, mbh, qp, is_intra, ns, quality;
  int t8;  // P macroblocks code their luma with the 8x8 transform (levels in 8x8 raster order)
  const uint8_t* t8f;  // NULL, or per macroblock: 0 = this one codes 4x4 blocks after all
  const int16_t* levels;
  const int32_t* dc;
  const uint32_t* nz;
  const uint32_t* pred_mode;
  const MV* mv;
  // scratch
  uint32_t* nbits;   // [mbs] bits of the macroblock (header + residual, no skip run); 0: skipped,
                     // kCavlcOver: they outgrew its region
  uint32_t* words;   // [mbs][kCavlcMbWords]
  uint4* place;      // [mbs] bit offset of the macroblock (of its skip run, if coded) in its slice; its bits;
                     // the skip run before a coded macroblock (kCavlcNoRun: none, I slices); unused
  uint32_t* next;    // [mbs] the coded macroblock after a coded one, and after a slice's first if that is
                     // skipped (all ones: none); others unused
  uint32_t* sl;      // [kCavlcMaxSlices * 4] per slice: total bits, trailing run, did not fit, end of the data
  // output
  uint8_t* out;
  uint32_t slice_cap;  // bytes per slice region (multiple of 4)
  uint32_t* out_bytes; // [ns]
  uint8_t* out_copy;   // where the stream bytes go (out itself, or e.g. mapped page-locked host memory)
};

__device__ __forceinline__ uint32_t slice_start(uint32_t s, uint32_t total, uint32_t ns) {
  return (uint32_t)(((uint64_t)s * total) / ns);
}

// Neighbour macroblock (dx, dy) of (mbx, mby) inside the picture and the
// slice that starts at `start` (encoder_h264.c:948-958).
__device__ __forceinline__ bool nb_ok(int mbx, int mby, int dx, int dy, int mbw, uint32_t start, int* nb) {
  const int x = mbx + dx, y = mby + dy;
  if (x < 0 || y < 0 || x >= mbw) return false;
  *nb = y * mbw + x;
  return (uint32_t)*nb >= start;
}

__device__ __forceinline__ int median3(int a, int b, int c) {
  return a + b + c - min(a, min(b, c)) - max(a, max(b, c));
}

// 8.4.1.3 median predictor as the reference derives it (encoder_h264.c:974-1000).
__device__ void mv_pred(const MV* mv, int mbx, int mby, int mbw, uint32_t start, int* px, int* py) {
  int na, nbb, nc;
  const bool a = nb_ok(mbx, mby, -1, 0, mbw, start, &na);
  const bool b = nb_ok(mbx, mby, 0, -1, mbw, start, &nbb);
  bool c = nb_ok(mbx, mby, 1, -1, mbw, start, &nc);
  if (!c) c = nb_ok(mbx, mby, -1, -1, mbw, start, &nc);
  if (!b && !c && a) {
    *px = mv[na].mvx;
    *py = mv[na].mvy;
    return;
  }
  const int ax = a ? mv[na].mvx : 0, ay = a ? mv[na].mvy : 0;
  const int bx = b ? mv[nbb].mvx : 0, by = b ? mv[nbb].mvy : 0;
  const int cx = c ? mv[nc].mvx : 0, cy = c ? mv[nc].mvy : 0;
  *px = median3(ax, bx, cx);
  *py = median3(ay, by, cy);
}

// 8.4.1.1 P_Skip predictor (encoder_h264.c:1036-1051): zero when the left or
// upper neighbour is missing or has a zero vector.
__device__ void skip_pred(const MV* mv, int mbx, int mby, int mbw, uint32_t start, int* px, int* py) {
  int na, nbb;
  const bool a = nb_ok(mbx, mby, -1, 0, mbw, start, &na);
  const bool b = nb_ok(mbx, mby, 0, -1, mbw, start, &nbb);
  if (!a || !b || (mv[na].mvx == 0 && mv[na].mvy == 0) || (mv[nbb].mvx == 0 && mv[nbb].mvy == 0)) {
    *px = 0;
    *py = 0;
    return;
  }
  mv_pred(mv, mbx, mby, mbw, start, px, py);
}

// Prediction modes the decoder can form at the slice and picture edges
// (h264_sanitize_i16_mode / _chroma_mode, encoder_h264.c:919-946).
__device__ __forceinline__ int sanitize_i16(int m, bool top, bool left) {
  if (!top && !left) return 2;                              // DC
  if (!top && (m == 0 || m == 3)) return left ? 1 : 2;      // vertical, plane -> horizontal or DC
  if (!left && (m == 1 || m == 3)) return top ? 0 : 2;      // horizontal, plane -> vertical or DC
  return m;
}
__device__ __forceinline__ int sanitize_chroma(int m, bool top, bool left) {
  if (!top && !left) return 0;                              // DC
  if (!top && (m == 2 || m == 3)) return left ? 1 : 0;      // vertical, plane -> horizontal or DC
  if (!left && (m == 1 || m == 3)) return top ? 2 : 0;      // horizontal, plane -> vertical or DC
  return m;
}

// ---- 1. per macroblock: skip, coded block pattern, header and residual bits ----
// One warp per macroblock; each lane writes one syntax element group into its
// own bit buffer, in the order the reference writes them: lane 0 the header,
// 1 the I16x16 luma DC block, 2..17 the luma blocks (spec order), 18 and 19 the
// chroma DC blocks, 20..27 the chroma AC blocks (Cb then Cr). A warp scan of
// the lanes' lengths places them; the lanes OR their words into the warp's
// shared copy of the macroblock's region, which is then stored.
constexpr int kCavlcLaneWords = 25;  // a block: at most 16 levels of 36 bits, token and runs < 24 words; odd
                                     // stride: the lanes' words lie in different banks
constexpr int kCavlcMbWarps = 4;

struct CavlcWarp {
  alignas(16) int16_t lev[24 * 16];
  int16_t dcl[16];   // quantised luma DC, raster positions
  int16_t cdl[8];    // quantised chroma DC (Cb, Cr)
  uint32_t lane[28 * kCavlcLaneWords];
  uint32_t out[kCavlcMbWords];
};

// MSB-first bit writer: `acc` ends in the nb < 32 pending bits.
struct BitW {
  uint64_t acc;
  uint32_t* w;
  uint32_t nb, pos;
  __device__ __forceinline__ void put(uint32_t n, uint32_t v) {  // n <= 32 bits, v < 2^n
    acc = (acc << n) | v;
    nb += n;
    pos += n;
    if (nb >= 32u) {
      nb -= 32u;
      *w++ = (uint32_t)(acc >> nb);
    }
  }
};

// Raster mask of a 4x4 block's nonzero levels -> frame zig-zag scan positions
// (scan position i holds raster position i + d; positions grouped by d), and
// the raster position of scan position i.
__device__ __forceinline__ uint32_t zigzag_mask(uint32_t m) {
  return (m & 0xc003u) | ((m >> 2) & 0x0004u) | ((m >> 5) & 0x0008u) | ((m >> 1) & 0x0110u) | ((m << 3) & 0x0060u) |
         ((m << 1) & 0x0880u) | ((m >> 3) & 0x0600u) | ((m << 5) & 0x1000u) | ((m << 2) & 0x2000u);
}
__device__ __forceinline__ int zigzag_pos(int i) { return (int)((0xFEB7ADC963258410ull >> (4 * i)) & 15u); }

// P_Skip (encoder_h264.c:3236-3255): no luma level, a zero chroma DC Hadamard
// (every raw term zero) and no chroma AC level, the vector on the skip
// predictor; quality levels from 5 up also accept two tiny DC words.
__device__ __forceinline__ bool p_skip(const CavlcArgs& a, int mb, int mbx, int mby, uint32_t start, bool luma,
                                       bool cdc_raw, bool cac) {
  if (luma) return false;
  bool zc = !cdc_raw && !cac;
  if (a.quality >= 5 && !zc && abs(a.dc[mb * 2 + 0]) <= 1 && abs(a.dc[mb * 2 + 1]) <= 1) zc = true;
  if (!zc) return false;
  int px, py;
  skip_pred(a.mv, mbx, mby, a.mbw, start, &px, &py);
  return a.mv[mb].mvx == px && a.mv[mb].mvy == py;
}

__global__ void __launch_bounds__(32 * kCavlcMbWarps) cavlc_mb_kernel(CavlcArgs a) {
  pdl_wait();
  __shared__ CavlcWarp shw[kCavlcMbWarps];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int mb = blockIdx.x * kCavlcMbWarps + wi;
  const int mbs = a.mbw * a.mbh;
  if (mb >= mbs) return;
  if (lane == 0) a.next[mb] = 0xffffffffu;
  if (a.stage.mv && lane < 4) {
    reinterpret_cast<uint32_t*>(a.stage.mv + mb)[lane] = reinterpret_cast<const uint32_t*>(a.mv + mb)[lane];
    if (mb == 0 && lane < 2) a.stage.status[lane] = lane == 0 ? *a.stage.s0 : (a.stage.s1 ? *a.stage.s1 : 0u);
  }
  CavlcWarp& sh = shw[wi];
  const int mbx = mb % a.mbw, mby = mb / a.mbw;
  const uint32_t start = slice_start(slice_of(mb, mbs, a.ns), mbs, a.ns);
  const bool intra = a.is_intra != 0;
  int nl, nt;
  const bool left = nb_ok(mbx, mby, -1, 0, a.mbw, start, &nl), top = nb_ok(mbx, mby, 0, -1, a.mbw, start, &nt);

  // lanes 2..17: luma block k (spec order), 20..27: chroma block k
  const bool lu = lane >= 2 && lane < 18, ch = lane >= 20 && lane < 28;
  const int k = lu ? lane - 2 : (lane & 3);
  const int x4 = blk_x4(k), y4 = blk_y4(k);
  const int blk = lu ? y4 * 4 + x4 : (ch ? lane - 4 : 0);  // staged block (raster luma, chroma from 16)
  uint32_t zo = 0, zl = 0, zt = 0;
  if (lu || ch) {
    zo = __ldg(a.nz + (size_t)mb * 24 + blk);
    if (left) zl = __ldg(a.nz + (size_t)nl * 24 + blk);
    if (top) zt = __ldg(a.nz + (size_t)nt * 24 + blk);
  }
  const uint32_t used = ch || intra ? 0xfffeu : 0xffffu;  // levels the block codes (position 0 goes by the DC blocks)
  zo &= used;
  zl &= used;
  zt &= used;
  // raw DC terms: luma on the luma lanes, chroma on the chroma lanes
  const int dcv = lu || ch ? __ldg(a.dc + (size_t)mb * 24 + blk) : 0;
  // chroma DC: 2x2 Hadamard output of the lane, quantised (encoder_h264.c:791-797)
  int cq;
  {
    const int g = lane & ~3;
    const int c0 = __shfl_sync(full, dcv, g), c1 = __shfl_sync(full, dcv, g + 1);
    const int c2 = __shfl_sync(full, dcv, g + 2), c3 = __shfl_sync(full, dcv, g + 3);
    const int s1 = (lane & 1) ? -1 : 1, s2 = (lane & 2) ? -1 : 1;
    cq = quantize_dc(c0 + s1 * c1 + s2 * c2 + s1 * s2 * c3, make_qp(chroma_qp(a.qp), intra));
  }
  const uint32_t bz = __ballot_sync(full, zo != 0u);
  const uint32_t blu = (bz >> 2) & 0xffffu;  // luma blocks with levels, spec order
  const bool cac = (bz >> 20) != 0u;
  const bool cdc_raw = (__ballot_sync(full, ch && dcv != 0) != 0u);
  const bool cdc = (__ballot_sync(full, ch && cq != 0) != 0u);
  if (!intra && p_skip(a, mb, mbx, mby, start, blu != 0u, cdc_raw, cac)) {  // its run is counted by the slice pass
    if (lane == 0) a.nbits[mb] = 0;
    return;
  }
  // TotalCoeff of the lane's block and its neighbours. A skipped neighbour has
  // none: no levels either, but for the quality rule's chroma AC.
  int tl = __popc(zl), tt = __popc(zt);
  const int tc_own = __popc(zo);
  if (!intra && a.quality >= 5) {
    auto nb_skip = [&](bool ok, int n, int nx, int ny, uint32_t z) -> bool {
      const uint32_t b = __ballot_sync(full, z != 0u);
      const int d = ok && ch ? a.dc[(size_t)n * 24 + blk] : 0;
      const bool raw = __ballot_sync(full, d != 0) != 0u;
      return ok && p_skip(a, n, nx, ny, start, (b & 0x3fffcu) != 0u, raw, (b >> 20) != 0u);
    };
    if (nb_skip(left, nl, mbx - 1, mby, zl)) tl = 0;
    if (nb_skip(top, nt, mbx, mby - 1, zt)) tt = 0;
  }
  // nC (encoder_h264.c:800-841): the neighbours inside the macroblock are other lanes
  int nc;
  {
    const int sl_in = lu ? 2 + spec_blk(y4, (x4 + 3) & 3) : lane ^ 1, st_in = lu ? 2 + spec_blk((y4 + 3) & 3, x4) : lane ^ 2;
    const int o_l = __shfl_sync(full, tc_own, sl_in), o_t = __shfl_sync(full, tc_own, st_in);
    const int n_l = __shfl_sync(full, tl, sl_in), n_t = __shfl_sync(full, tt, st_in);
    const int xx = lu ? x4 : (lane & 1), yy = lu ? y4 : (lane & 2);
    const int na = xx ? o_l : (left ? n_l : -1), nb = yy ? o_t : (top ? n_t : -1);
    nc = na >= 0 && nb >= 0 ? (na + nb + 1) >> 1 : (na >= 0 ? na : (nb >= 0 ? nb : 0));
  }
  // coded block pattern: the 8x8 quadrants with levels (any luma AC in an I16x16)
  uint32_t cbp_l = 0;
  if (intra) cbp_l = blu ? 1u : 0u;
  else cbp_l = (blu & 0xfu ? 1u : 0u) | (blu & 0xf0u ? 2u : 0u) | (blu & 0xf00u ? 4u : 0u) | (blu & 0xf000u ? 8u : 0u);
  const int cbp_c = cac ? 2 : (cdc ? 1 : 0);
  const bool use8 = a.t8 && !intra && (!a.t8f || a.t8f[mb]);

  // ---- the levels, and the DC blocks, to shared memory ----------------------
  {
    const int16_t* lv = a.levels + (size_t)mb * 384;
    if (((reinterpret_cast<uintptr_t>(lv)) & 15) == 0) {
      const uint4* src = reinterpret_cast<const uint4*>(lv);
      uint4* dst = reinterpret_cast<uint4*>(sh.lev);
      dst[lane] = __ldg(src + lane);
      if (lane < 16) dst[32 + lane] = __ldg(src + 32 + lane);
    } else {
#pragma unroll 1
      for (int i = lane; i < 384; i += 32) sh.lev[i] = __ldg(lv + i);
    }
    if (ch) sh.cdl[lane - 20] = (int16_t)cq;
  }
  uint32_t m = 0;          // nonzero levels in scan order
  int vlc = 0, maxc = 16;  // nC class (4: chroma DC), levels the block may have
  bool active = false;
  const int16_t* src = sh.lev;  // level of scan position i: src[pos(i)]
  if (intra) {
    // Luma DC of an I16x16 macroblock: 2-D Hadamard of the 16 raw terms
    // (rows + + + +, + + - -, + - - +, + - + -), (sum + 1) >> 1, quantised
    // (h264_intra16_luma_dc_transform, encoder_h264.c:711-789); lane 4r + c
    // forms frequency (r, c), first along rows, then down columns.
    const int r = (lane >> 2) & 3, c = lane & 3;
    auto sgn = [](int h, int i) -> int { return ((h == 1 ? 0xc : (h == 2 ? 0x6 : (h == 3 ? 0xa : 0))) >> i) & 1 ? -1 : 1; };
    int t = 0, v = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) t += sgn(c, j) * __shfl_sync(full, dcv, 2 + spec_blk(r, j));
#pragma unroll
    for (int i = 0; i < 4; ++i) v += sgn(r, i) * __shfl_sync(full, t, 4 * i + c);
    const int l = quantize_dc((v + 1) >> 1, make_qp(a.qp, true));
    if (lane < 16) sh.dcl[lane] = (int16_t)l;
    const uint32_t md = __ballot_sync(full, lane < 16 && (int16_t)l != 0);
    const int nc0 = __shfl_sync(full, nc, 2);
    if (lane == 1) {
      active = true;
      m = zigzag_mask(md);
      vlc = nc0;
      src = sh.dcl;
    }
  }
  const uint32_t mc = __ballot_sync(full, ch && cq != 0) >> 20;  // chroma DC levels: Cb 0..3, Cr 4..7
  bool raw_scan = false;  // positions are 8x8 scan positions (use8) or the levels are in scan order already (chroma DC)
  if (lu) {
    active = intra ? cbp_l != 0u : ((cbp_l >> (k >> 2)) & 1u) != 0u;
    vlc = nc;
    if (use8) {
      m = zo;
      src = sh.lev + 64 * (k >> 2);
      raw_scan = true;
    } else {
      m = zigzag_mask(zo);
      src = sh.lev + 16 * blk;
    }
  } else if (lane == 18 || lane == 19) {
    active = cbp_c >= 1;
    m = (mc >> (4 * (lane - 18))) & 15u;
    src = sh.cdl + 4 * (lane - 18);
    maxc = 4;
  } else if (ch) {
    active = cbp_c == 2;
    m = zigzag_mask(zo);
    vlc = nc;
    src = sh.lev + 16 * blk;
  }
  vlc = maxc == 4 ? 4 : (vlc < 2 ? 0 : (vlc < 4 ? 1 : (vlc < 8 ? 2 : 3)));
  const int first = (lu && intra) || ch ? 1 : 0;  // AC blocks: scan positions 1..15
  m >>= first;
  if (first) maxc = 15;
  __syncwarp();
  const bool cd = maxc == 4;
  auto level = [&](int i) -> int {
    const int pos = cd ? i : (raw_scan ? (int)kZigzag8[4 * i + (k & 3)] : zigzag_pos(i + first));
    return src[pos];
  };

  BitW b;
  b.acc = 0;
  b.w = sh.lane + (lane < 28 ? lane : 27) * kCavlcLaneWords;
  b.nb = b.pos = 0;
  if (lane == 0) {
    // macroblock header (clause 7.3.5): ue(v) values, one bit of
    // transform_size_8x8_flag after the coded block pattern, mb_qp_delta 0
    int px = 0, py = 0;
    uint32_t v[4] = {0u, 0u, 0u, 0u};
    int n;
    if (intra) {
      const uint32_t pm = a.pred_mode[mb];
      v[0] = (uint32_t)(1 + sanitize_i16((int)(pm & 3u), top, left) + 4 * cbp_c) + 12u * cbp_l;
      v[1] = (uint32_t)sanitize_chroma((int)((pm >> 2) & 3u), top, left);
      n = 3;  // v[2] = 0: mb_qp_delta
    } else {
      mv_pred(a.mv, mbx, mby, a.mbw, start, &px, &py);
      const int dx = a.mv[mb].mvx - px, dy = a.mv[mb].mvy - py;
      v[1] = dx > 0 ? 2u * (uint32_t)dx - 1u : 2u * (0u - (uint32_t)dx);
      v[2] = dy > 0 ? 2u * (uint32_t)dy - 1u : 2u * (0u - (uint32_t)dy);
      v[3] = d_cbp_code[cbp_l | ((uint32_t)cbp_c << 4)];
      n = 4;
    }
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const uint32_t c = (i == 0 ? v[0] : (i == 1 ? v[1] : (i == 2 ? v[2] : v[3]))) + 1u;
      const uint32_t l = 31u - (uint32_t)__clz((int)c);
      b.put(l, 0u);
      b.put(l + 1u, c);
    }
    if (!intra) {
      if (a.t8 && cbp_l) b.put(1u, use8 ? 1u : 0u);
      if (cbp_l || cbp_c) b.put(1u, 1u);
    }
  } else if (active) {
    // ---- a residual block (clause 9.2): coeff_token and trailing-one signs,
    //      levels from the highest frequency down, total_zeros, run_before -----
    const int tc = __popc(m);
    uint32_t rest = m, signs = 0, t1 = 0;
#pragma unroll 1
    while (t1 < 3u && rest) {  // trailing ones
      const int i = 31 - __clz((int)rest), v = level(i);
      if (v != 1 && v != -1) break;
      signs = (signs << 1) | (v < 0 ? 1u : 0u);
      ++t1;
      rest ^= 1u << i;
    }
    {
      const uint32_t e = d_cavlc.ct[vlc][tc * 4 + (int)t1];
      b.put((e >> 8) + t1, ((e & 0xffu) << t1) | signs);
    }
    int sl = (tc > 10 && t1 < 3u) ? 1 : 0;
    int sub = t1 < 3u ? 2 : 0;  // the first level after fewer than three trailing ones is not +-1
#pragma unroll 1
    while (rest) {
      const int i = 31 - __clz((int)rest), v = level(i);
      rest ^= 1u << i;
      // level_prefix / level_suffix (9.2.2.1) with the reference's escape
      // arithmetic for level_prefix >= 15 (cavlc.c:429-480)
      const int code = (v > 0 ? 2 * v - 2 : -2 * v - 1) - sub;
      sub = 0;
      uint32_t zeros, ss, suf;
      const int prefix = code >> sl;
      if (sl == 0 && code >= 14 && code < 30) {
        zeros = 14u;
        ss = 4u;
        suf = (uint32_t)(code - 14);
      } else if (prefix < (sl == 0 ? 14 : 15)) {
        zeros = (uint32_t)prefix;
        ss = (uint32_t)sl;
        suf = (uint32_t)(code & ((1 << sl) - 1));
      } else {
        const uint32_t total = (uint32_t)(sl == 0 ? code + 4066 : code - (15 << sl) + 4096);
        ss = 31u - (uint32_t)__clz((int)total);
        zeros = ss + 3u;
        suf = total - (1u << ss);
      }
      uint32_t n = zeros + 1u + ss;
      if (n > 32u) {  // at most 36 bits, the first ones zeros
        b.put(n - 32u, 0u);
        n = 32u;
      }
      b.put(n, (1u << ss) | suf);
      if (sl == 0) sl = 1;
      if (abs(v) > (3 << (sl - 1)) && sl < 6) ++sl;
    }
    if (tc) {
      int i = 31 - __clz((int)m), zleft = i + 1 - tc;
      if (tc < maxc) {
        const uint32_t e = cd ? d_cavlc.cdtz[tc - 1][zleft] : d_cavlc.tz[tc - 1][zleft];
        b.put(e >> 8, e & 0xffu);
      }
      rest = m ^ (1u << i);
#pragma unroll 1
      while (rest && zleft > 0) {
        const int j = 31 - __clz((int)rest), r = i - j - 1;
        const uint32_t e = d_cavlc.run[zleft <= 6 ? zleft - 1 : 6][r];
        b.put(e >> 8, e & 0xffu);
        rest ^= 1u << j;
        zleft -= r;
        i = j;
      }
    }
  }
  if (b.nb) *b.w = (uint32_t)(b.acc << (32u - b.nb));

  // ---- place the lanes' bits one after another -------------------------------
  __syncwarp();
  const uint32_t len = b.pos;
  uint32_t off = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(full, off, o);
    if (lane >= o) off += y;
  }
  const uint32_t total = __shfl_sync(full, off, 31);
  off -= len;
  if (total > 32u * kCavlcMbWords) {
    if (lane == 0) a.nbits[mb] = kCavlcOver;
    return;
  }
  const uint32_t nw = (total + 31u) >> 5;
  for (uint32_t i = lane; i < nw; i += 32) sh.out[i] = 0u;
  __syncwarp();
  {
    const uint32_t* w = sh.lane + (lane < 28 ? lane : 27) * kCavlcLaneWords;
    uint32_t* d = sh.out + (off >> 5);
    const uint32_t s = off & 31u;
#pragma unroll 1
    for (uint32_t i = 0; 32u * i < len; ++i) {  // the last word's unused low bits are zero
      const uint32_t v = w[i];
      atomicOr(d + i, v >> s);
      if (s && (v << (32u - s))) atomicOr(d + i + 1, v << (32u - s));
    }
  }
  __syncwarp();
  uint32_t* dst = a.words + (size_t)mb * kCavlcMbWords;
  for (uint32_t i = lane; i < nw; i += 32) dst[i] = sh.out[i];
  if (lane == 0) a.nbits[mb] = total;
}

// ---- 2. per slice: skip runs, offsets, length --------------------------------------
// A chunk of consecutive macroblocks seen from the run of skipped macroblocks:
// `has` a coded one, R = the skips after its last coded macroblock (or all
// of its macroblocks when none is coded). Chunks compose left to right.
struct RunState {
  uint32_t has, r;
};
__device__ __forceinline__ RunState run_then(RunState a, RunState b) {
  return b.has ? b : RunState{a.has, a.r + b.r};
}

// Exclusive block-wide scans over kCavlcScanThreads threads (32 warps).
__device__ RunState scan_run(RunState v, RunState* sh, RunState* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  RunState x = v;
  for (int o = 1; o < 32; o <<= 1) {
    RunState y{__shfl_up_sync(0xffffffffu, x.has, o), __shfl_up_sync(0xffffffffu, x.r, o)};
    if (lane >= o) x = run_then(y, x);
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    RunState t = sh[lane];
    for (int o = 1; o < 32; o <<= 1) {
      RunState y{__shfl_up_sync(0xffffffffu, t.has, o), __shfl_up_sync(0xffffffffu, t.r, o)};
      if (lane >= o) t = run_then(y, t);
    }
    sh[lane] = t;  // inclusive over warps
  }
  __syncthreads();
  RunState before = w > 0 ? sh[w - 1] : RunState{0u, 0u};
  RunState xin{__shfl_up_sync(0xffffffffu, x.has, 1), __shfl_up_sync(0xffffffffu, x.r, 1)};
  if (lane > 0) before = run_then(before, xin);
  *total = sh[31];
  __syncthreads();
  return before;
}

__device__ uint32_t scan_sum(uint32_t v, uint32_t* sh, uint32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    uint32_t t = sh[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    sh[lane] = t;
  }
  __syncthreads();
  const uint32_t r = (w > 0 ? sh[w - 1] : 0u) + x - v;
  *total = sh[31];
  __syncthreads();
  return r;
}

__device__ __forceinline__ uint32_t ue_len(uint32_t v) { return 2u * (31u - (uint32_t)__clz((int)(v + 1u))) + 1u; }

__global__ void __launch_bounds__(kCavlcScanThreads) cavlc_slice_kernel(CavlcArgs a, CavlcHdr h) {
  pdl_wait();
  __shared__ RunState shr[32];
  __shared__ uint32_t shs[32];
  const int s = blockIdx.x, t = threadIdx.x;
  const uint32_t mbs = (uint32_t)(a.mbw * a.mbh);
  const uint32_t m0 = slice_start(s, mbs, a.ns), m1 = slice_start(s + 1, mbs, a.ns);
  const uint32_t per = (m1 - m0 + kCavlcScanThreads - 1) / kCavlcScanThreads;
  const uint32_t i0 = min(m1, m0 + t * per), i1 = min(m1, i0 + per);
  // this thread's chunk: leading skips, skips after its last coded
  // macroblock, the bits of its coded macroblocks but the first one's run
  // (I slices have no mb_skip_run: every macroblock is coded, runs are 0 bits)
  const bool runs = !a.is_intra;
  uint32_t lead = 0, tail = 0, inner = 0, has = 0;
  for (uint32_t mb = i0; mb < i1; ++mb) {
    const uint32_t n = a.nbits[mb];
    if (n == 0u) {
      if (has) ++tail;
      else ++lead;
    } else {
      inner += (has && runs ? ue_len(tail) : 0u) + n;
      tail = 0;
      has = 1;
    }
  }
  // a macroblock of any slice that outgrew its region fails the picture
  bool over = false;
  for (uint32_t mb = t; mb < mbs; mb += kCavlcScanThreads) over |= a.nbits[mb] == kCavlcOver;
  over = __syncthreads_or(over);
  RunState all;
  const RunState in = scan_run(RunState{has, has ? tail : lead}, shr, &all);
  const uint32_t mine = has ? (runs ? ue_len(in.r + lead) : 0u) + inner : 0u;
  uint32_t data = 0;
  const uint32_t base = (uint32_t)h.len[s] + scan_sum(mine, shs, &data);
  const uint32_t trail = all.r;  // skips after the slice's last coded macroblock
  const uint32_t bits = (uint32_t)h.len[s] + data + (trail ? ue_len(trail) : 0u) + 1u;
  const uint32_t bytes = (bits + 7u) >> 3;
  const bool fits = bytes <= a.slice_cap && !over;
  // offsets of the macroblocks, runs of the coded ones
  uint32_t pos = base, run = in.r;
  for (uint32_t mb = i0; mb < i1; ++mb) {
    const uint32_t n = a.nbits[mb];
    a.place[mb] = make_uint4(pos, n, runs ? run : kCavlcNoRun, 0u);
    if (n == 0u) {
      ++run;
    } else {
      // the coded macroblock before this one, or the slice's skipped first
      if (mb > m0) a.next[mb - m0 > run ? mb - 1u - run : m0] = mb;
      pos += (runs ? ue_len(run) : 0u) + n;
      run = 0;
    }
  }
  if (t == 0) {
    a.sl[4 * s + 0] = bits;
    a.sl[4 * s + 1] = trail;
    a.sl[4 * s + 2] = fits ? 0u : 1u;
    a.sl[4 * s + 3] = (uint32_t)h.len[s] + data;
    a.out_bytes[s] = fits ? bytes : 0xffffffffu;
  }
}

// ---- 3. every output word's bits -------------------------------------------------
// A thread per 32-bit word of the slice: it finds the macroblock its first bit
// falls into and collects the pieces that overlap the word, so no word is
// cleared, shared or swapped afterwards. A warp's 32 words are found together:
// a 32-way search over the offsets (three dependent loads for a 1080p frame
// where a binary search takes thirteen) down to the first word's macroblock,
// then the 32 macroblocks from there on in registers.
__global__ void __launch_bounds__(256) cavlc_gather_kernel(CavlcArgs a, CavlcHdr h) {
  pdl_wait();
  const int s = blockIdx.y;
  if (a.sl[4 * s + 2]) return;  // the slice did not fit
  const uint32_t bits = a.sl[4 * s + 0], trail = a.sl[4 * s + 1], end = a.sl[4 * s + 3];
  const uint32_t nw = (((bits + 7u) >> 3) + 3u) >> 2, hl = (uint32_t)h.len[s];
  const uint32_t mbs = (uint32_t)(a.mbw * a.mbh);
  const uint32_t m0 = slice_start(s, mbs, a.ns), m1 = slice_start(s + 1, mbs, a.ns);
  uint32_t* dst = reinterpret_cast<uint32_t*>(a.out_copy + (size_t)s * a.slice_cap);
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t k0 = blockIdx.x * blockDim.x + threadIdx.x - lane; k0 < nw; k0 += gridDim.x * blockDim.x) {
    const uint32_t k = k0 + lane, p = 32u * k, p0 = 32u * k0;
    // the last macroblock that starts at or before p0 (the first one, if none does)
    uint32_t lo = m0, cnt = m1 - m0;
    while (cnt > 1u) {
      const uint32_t step = (cnt + 31u) >> 5, i = lo + lane * step;
      const uint32_t le = __ballot_sync(0xffffffffu, lane * step < cnt && a.place[i].x <= p0);
      const uint32_t j = le ? 31u - (uint32_t)__clz((int)le) : 0u;
      cnt = min(step, cnt - j * step);
      lo += j * step;
    }
    const uint32_t o = lo + lane < m1 ? a.place[lo + lane].x : 0xffffffffu;
    uint32_t mb0 = 0;
#pragma unroll
    for (uint32_t st = 16u; st > 0u; st >>= 1) {
      const uint32_t t = __shfl_sync(0xffffffffu, o, (int)(mb0 + st));
      if (t <= p) mb0 += st;
    }
    const bool beyond = mb0 == 31u;  // words reaching past the 32 macroblocks (few bits each)
    mb0 += lo;
    if (k >= nw) continue;
    uint32_t w = 0;
    // n <= 32 bits v at stream position at (overlapping this word or not)
    auto add = [&](uint32_t at, uint32_t n, uint32_t v) {
      const uint32_t lft = n < 32u ? (n ? v << (32u - n) : 0u) : v;  // left-aligned
      const int d = (int)(at - p);
      if (d >= 0 && d < 32) w |= lft >> d;
      else if (d < 0 && d > -32) w |= lft << -d;
    };
    if (p < hl) w |= h.bits[s][k] & (hl - p < 32u ? ~(0xffffffffu >> (hl - p)) : 0xffffffffu);
    if (p + 32u > hl && p < end) {
      if (beyond) {
        uint32_t hi = m1 - 1u;
        while (mb0 < hi) {
          const uint32_t mid = (mb0 + hi + 1u) >> 1;
          if (a.place[mid].x <= p) mb0 = mid;
          else hi = mid - 1u;
        }
      }
      // From coded macroblock to coded macroblock: a still picture is a few of
      // them between skip runs of thousands (a 1080p one 274 us, walking every
      // macroblock). Only a slice's beginning lies at a skipped one.
      uint32_t mb = mb0;
      uint4 pl = a.place[mb];
      if (pl.y == 0u) {
        mb = a.next[m0];
        if (mb < m1) pl = a.place[mb];
      }
      uint32_t nx = mb < m1 ? a.next[mb] : 0xffffffffu;
      while (mb < m1 && pl.x < p + 32u) {
        uint4 pn = pl;
        uint32_t nn = 0xffffffffu;
        if (nx < m1) {  // in flight while this one's words are read
          pn = a.place[nx];
          nn = a.next[nx];
        }
        uint32_t at = pl.x;
        const uint32_t n = pl.y, run = pl.z;
        if (run != kCavlcNoRun) {  // mb_skip_run (P slices): the last l + 1 bits of its 2l + 1
          const uint32_t l = 31u - (uint32_t)__clz((int)(run + 1u));
          add(at + l, l + 1u, run + 1u);
          at += 2u * l + 1u;
        }
        // the macroblock's words that overlap [p, p + 32): at most two
        const uint32_t* mw = a.words + (size_t)mb * kCavlcMbWords;
        const uint32_t f = p > at ? (p - at) >> 5 : 0u;
#pragma unroll
        for (uint32_t i = 0; i < 2u; ++i)
          if (32u * (f + i) < n) add(at + 32u * (f + i), 32u, mw[f + i]);  // unused low bits are zero
        mb = nx;
        pl = pn;
        nx = nn;
      }
    }
    if (p + 32u > end) {  // trailing skips, rbsp_stop_one_bit; alignment zeros
      uint32_t at = end;
      if (trail) {
        const uint32_t l = 31u - (uint32_t)__clz((int)(trail + 1u));
        add(at + l, l + 1u, trail + 1u);
        at += 2u * l + 1u;
      }
      add(at, 1u, 1u);
    }
    dst[k] = __byte_perm(w, 0u, 0x0123);
  }
}

}  // namespace b200enc

using namespace b200enc;

namespace {

struct CavlcLayout {
  size_t nbits, next, words, place, sl, bytes;
};

size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

CavlcLayout cavlc_layout(int mbw, int mbh) {
  const size_t mbs = (size_t)mbw * mbh;
  CavlcLayout l;
  l.sl = 0;
  l.nbits = l.sl + up256(kCavlcMaxSlices * 16);
  l.next = l.nbits + up256(mbs * 4);
  l.place = l.next + up256(mbs * 4);
  l.words = l.place + up256(mbs * 16);
  l.bytes = l.words + mbs * kCavlcMbWords * 4;
  return l;
}

}  // namespace

extern "C" size_t b200enc_cavlc_scratch_bytes(int mbw, int mbh) {
  if (mbw <= 0 || mbh <= 0) return 0;
  return cavlc_layout(mbw, mbh).bytes;
}

static int cavlc_launch(const b200enc_cavlc_t* p, const CavlcStage& stage, cudaStream_t st) {
  if (!p || p->mbw <= 0 || p->mbh <= 0 || p->qp < 0 || p->qp > 51 || p->num_slices < 1 ||
      p->num_slices > kCavlcMaxSlices || p->num_slices > p->mbw * p->mbh)
    return -1;
  if (!p->levels || !p->dc || !p->nz || !p->mv || (p->is_intra && !p->pred_mode) || !p->out || !p->out_bytes ||
      !p->scratch)
    return -1;
  if ((p->slice_cap & 3) || p->slice_cap < 4 || (((uintptr_t)p->out) & 3) || (((uintptr_t)p->out_copy) & 3) ||
      (((uintptr_t)p->scratch) & 255))
    return -1;
  const CavlcLayout L = cavlc_layout(p->mbw, p->mbh);
  if (p->scratch_bytes < L.bytes) return -1;
  CavlcHdr h{};
  for (int s = 0; s < p->num_slices; ++s) {
    const int n = p->header_bits ? p->header_bits[s] : 0;
    if (n < 0 || n > 128 || (n > 0 && !p->header)) return -1;
    h.len[s] = n;
    for (int k = 0; k < 4; ++k) {
      uint32_t w = 0;
      for (int j = 0; j < 4; ++j) w = (w << 8) | (n > 0 ? p->header[16 * s + 4 * k + j] : 0u);
      h.bits[s][k] = w;
    }
  }
  uint8_t* sc = static_cast<uint8_t*>(p->scratch);
  CavlcArgs a;
  a.stage = stage;
  a.mbw = p->mbw;
  a.mbh = p->mbh;
  a.qp = p->qp;
  a.is_intra = p->is_intra ? 1 : 0;
  a.ns = p->num_slices;
  a.quality = p->quality_level;
  a.t8 = p->transform8x8 ? 1 : 0;
  a.t8f = p->t8_flags;
  a.levels = p->levels;
  a.dc = p->dc;
  a.nz = p->nz;
  a.pred_mode = p->pred_mode;
  a.mv = static_cast<const MV*>(p->mv);
  a.nbits = reinterpret_cast<uint32_t*>(sc + L.nbits);
  a.next = reinterpret_cast<uint32_t*>(sc + L.next);
  a.words = reinterpret_cast<uint32_t*>(sc + L.words);
  a.place = reinterpret_cast<uint4*>(sc + L.place);
  a.sl = reinterpret_cast<uint32_t*>(sc + L.sl);
  a.out = p->out;
  a.slice_cap = (uint32_t)std::min<size_t>(p->slice_cap, 0xfffffffcu);
  a.out_bytes = p->out_bytes;
  a.out_copy = p->out_copy ? p->out_copy : p->out;
  const int mbs = p->mbw * p->mbh;
  launch_early(cavlc_mb_kernel, (mbs + kCavlcMbWarps - 1) / kCavlcMbWarps, 32 * kCavlcMbWarps, 0, st, a);
  launch_early(cavlc_slice_kernel, p->num_slices, kCavlcScanThreads, 0, st, a, h);
  // words per slice are known on the device only: a CTA of 256 words per 16
  // macroblocks (the share of a dense one), walking the rest in strides
  const int ctas = std::max(1, std::min(128, mbs / p->num_slices / 16));
  launch_early(cavlc_gather_kernel, dim3(ctas, p->num_slices), 256, 0, st, a, h);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int b200enc_cavlc_slices(const b200enc_cavlc_t* p, void* stream) {
  return cavlc_launch(p, CavlcStage{}, static_cast<cudaStream_t>(stream));
}

int cavlc_slices_and_stage(const b200enc_cavlc_t* p, void* mv_host, const uint32_t* s0, const uint32_t* s1,
                           uint32_t* status_host, cudaStream_t st) {
  return cavlc_launch(p, CavlcStage{static_cast<MV*>(mv_host), s0, s1, status_host}, st);
}
