// pframe.cu - fused P-macroblock chain: motion-compensated prediction,
// residual, forward 4x4, AC quant + nonzero masks, chroma DC Hadamard,
// dequant, inverse 4x4 and reconstruction, three warps per MB.
//
// Reference stages, which run as five separate dispatches with int32
// residual/pred/coeff buffers round-tripping through memory:
//   A1/shaders/residual_predict.comp:417-434, :576-635 (luma qpel MC, chroma
//   eighth-pel MC), dct_transform.comp:75-98, quantize.comp:189-225,
//   reconstruct.comp:318-442.
// Here nothing but the frame planes, the MV and the staged outputs touch HBM.
// Lane r of a quad owns row r of one 4x4 block from its source samples to its
// reconstruction: it predicts the row's four samples at once (packed bytes and
// 16-bit pairs), and the transposes between rows and columns (residual, levels,
// prediction, reconstruction) are quad shuffles. Shared memory holds only the
// reference patch, there is one barrier, and levels and samples are stored from
// registers. Bound by instructions issued: a 2160p picture (32,400 MBs) with
// vectors at every quarter sample 58.5 us, whole samples 51.5; a sample per lane
// with byte reads of the patch, and every step through shared memory, 88 and 71.
#include <type_traits>

#include "b200enc_internal.h"
#include "common.cuh"
#include "t8x8.cuh"

namespace b200enc {

// Reference rows staged as 16-byte units. The luma patch row r holds reference
// row iy0-2+r from column lxa (16-aligned) on; the patch origin (ix0-2, iy0-2)
// is at byte lo of row 0. The chroma patch (NV12 pairs) starts at byte cxa
// (16-aligned); chroma sample (ixc, iyc) is at byte co of row 0. 48-byte luma
// rows: the eight rows and four words a warp reads at once are in 32 banks.
struct PPatch {
  alignas(16) uint8_t lp[21][48];
  alignas(16) uint8_t cp[9][48];
};
// What the 8x8 luma transform shares between the lanes of a macroblock.
struct PShared8 : PPatch {
  int16_t pred[16][16];            // luma prediction per block, raster within block
  int16_t res[16][16];             // luma residual
  alignas(16) int16_t lev[16][16];  // luma levels
  alignas(16) uint8_t ry[16][16];  // reconstructed luma
  int32_t t8[4][65];               // the four blocks between their row and column passes
  int32_t cost[3];                 // 4x4 (two warps' halves) and 8x8 Hadamard costs of the luma residual
};

// Bytes o .. o + 3 of a shared row.
__device__ __forceinline__ uint32_t bytes4(const uint8_t* row, int o) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(row + (o & ~3));
  return __funnelshift_r(w[0], w[1], (o & 3) * 8);
}
// Horizontal 6-tap sums of four neighbouring samples: bytes o .. o + 8 of a row.
__device__ __forceinline__ void tap6_row(const uint8_t* row, int o, int (&t)[4]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(row + (o & ~3));
  const int sh = (o & 3) * 8;
  const uint32_t a = __funnelshift_r(w[0], w[1], sh), b = __funnelshift_r(w[1], w[2], sh), c = w[2] >> sh;
  constexpr uint32_t ta = 0x1414fb01u, tb = 0x000001fbu;  // 1 -5 20 20, -5 1
#pragma unroll
  for (int j = 0; j < 4; ++j)
    t[j] = dot4(j ? __funnelshift_r(a, b, 8 * j) : a, ta, dot4(j ? __funnelshift_r(b, c, 8 * j) : b, tb, 0));
}

// Four luma quarter-pel samples (residual_predict.comp:263-298) of row y from
// column x, whose integer anchors are patch row y + 2, bytes lo + x + 2 on. A
// phase is one of, or the rounded average of two of: the nearest whole sample G,
// the horizontal half sample B of the nearer row, the vertical one H of the
// nearer column, and the centre J. The phase is the macroblock's: no divergence.
__device__ __forceinline__ uint32_t mc_luma4(const uint8_t (*lp)[48], int lo, int x, int y, int fx, int fy) {
  const int o = lo + x, right = fx == 3 ? 1 : 0, down = fy == 3 ? 1 : 0;
  const bool g = (fx == 0 && fy != 2) || (fy == 0 && fx != 2), b = fx != 0 && fy != 2 && (fy != 0 || fx != 0),
             h = fy != 0 && fx != 2, j = (fx == 2 && fy != 0) || (fy == 2 && fx != 0);
  uint32_t v = 0;
  bool have = false;
  auto add = [&](uint32_t s) {
    v = have ? avg4(v, s) : s;
    have = true;
  };
  if (g) add(bytes4(lp[y + 2 + down], o + 2 + right));
  if (b) {
    int t[4];
    tap6_row(lp[y + 2 + down], o, t);
    add(clip4((t[0] + 16) >> 5, (t[1] + 16) >> 5, (t[2] + 16) >> 5, (t[3] + 16) >> 5));
  }
  if (h) {
    uint32_t lo2[6], hi2[6];  // two columns to a register: a column's sum is under 16 bits
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const uint32_t w = bytes4(lp[y + k], o + 2 + right);
      lo2[k] = __byte_perm(w, 0, 0x4140);
      hi2[k] = __byte_perm(w, 0, 0x4342);
    }
    const uint32_t p = (lo2[2] + lo2[3]) * 20u - (lo2[1] + lo2[4]) * 5u + (lo2[0] + lo2[5]) + 0x00100010u;
    const uint32_t q = (hi2[2] + hi2[3]) * 20u - (hi2[1] + hi2[4]) * 5u + (hi2[0] + hi2[5]) + 0x00100010u;
    add(clip4((int16_t)p >> 5, (int)(p + 0x8000u) >> 21, (int16_t)q >> 5, (int)(q + 0x8000u) >> 21));
  }
  if (j) {
    int s[4] = {512, 512, 512, 512};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      constexpr int tap[6] = {1, -5, 20, 20, -5, 1};
      int t[4];
      tap6_row(lp[y + k], o, t);
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] += tap[k] * t[i];
    }
    add(clip4(s[0] >> 10, s[1] >> 10, s[2] >> 10, s[3] >> 10));
  }
  return v;
}

// Four bytes of NV12 chroma (two sample pairs) at bytes o .. of patch row y,
// bilinear at eighth samples: the weights sum to 64, so a sum is under 16 bits.
__device__ __forceinline__ uint32_t mc_chroma4(const uint8_t (*cp)[48], int o, int y, int fx, int fy) {
  const uint32_t wa = (8 - fx) * (8 - fy), wb = fx * (8 - fy), wc = (8 - fx) * fy, wd = fx * fy;
  const uint32_t a = bytes4(cp[y], o), b = bytes4(cp[y], o + 2), c = bytes4(cp[y + 1], o), d = bytes4(cp[y + 1], o + 2);
  constexpr uint32_t m = 0x00ff00ffu;
  const uint32_t even = (a & m) * wa + (b & m) * wb + (c & m) * wc + (d & m) * wd + 0x00200020u;
  const uint32_t odd = (a >> 8 & m) * wa + (b >> 8 & m) * wb + (c >> 8 & m) * wc + (d >> 8 & m) * wd + 0x00200020u;
  return (even >> 6 & m) | (odd >> 6 & m) << 8;
}

// 4x4 transposes across a quad (lane r's row r to lane r's column r) of bytes,
// and of 16-bit values held as two pairs.
__device__ __forceinline__ uint32_t quad_transpose_bytes(uint32_t w, int r) {
  w = __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 2), (r & 2) ? 0x3276 : 0x5410);
  return __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 1), (r & 1) ? 0x3715 : 0x6240);
}
__device__ __forceinline__ uint2 quad_transpose_pairs(uint2 w, int r) {
  const bool hi = (r & 2) != 0, odd = (r & 1) != 0;
  uint32_t o = __shfl_xor_sync(0xffffffffu, hi ? w.x : w.y, 2);
  if (hi) w.x = o; else w.y = o;
  o = __shfl_xor_sync(0xffffffffu, __byte_perm(w.x, w.y, odd ? 0x5410 : 0x7632), 1);
  // even: (own low, other's low) of each pair; odd: (other's high, own high)
  return make_uint2(__byte_perm(w.x, o, odd ? 0x3254 : 0x5410), __byte_perm(w.y, o, odd ? 0x3276 : 0x7610));
}

// Forward 4x4 (dct_transform.comp:75-98) of the residual src - pred, lane r
// holding its row r: column r of the coefficients. Both butterflies are integer
// dot products, the first of the samples themselves (its outputs are under 12
// bits), which leaves the busiest pipe (permutes, selects, adds) alone.
__device__ __forceinline__ void quad_forward_bytes(uint32_t src, uint32_t pred, int r, int (&c)[4]) {
  const int t0 = dot4(src, 0x01010101u, dot4(pred, 0xffffffffu, 0)), t1 = dot4(src, 0xfeff0102u, dot4(pred, 0x0201fffeu, 0));
  const int t2 = dot4(src, 0x01ffff01u, dot4(pred, 0xff0101ffu, 0)), t3 = dot4(src, 0xff02fe01u, dot4(pred, 0x01fe02ffu, 0));
  const uint2 w = quad_transpose_pairs(make_uint2(__byte_perm(t0, t1, 0x5410), __byte_perm(t2, t3, 0x5410)), r);
  c[0] = __dp2a_lo((int)w.x, 0x0101, __dp2a_lo((int)w.y, 0x0101, 0));
  c[1] = __dp2a_lo((int)w.x, 0x0102, __dp2a_lo((int)w.y, 0xfeff, 0));
  c[2] = __dp2a_lo((int)w.x, 0xff01, __dp2a_lo((int)w.y, 0x01ff, 0));
  c[3] = __dp2a_lo((int)w.x, 0xfe01, __dp2a_lo((int)w.y, 0xff02, 0));
}

// make_qp of every QP, and chroma_qp: constants of the whole grid, read instead of
// computed by every thread (a tenth of the kernel's instructions).
struct QpTable {
  QP q[52];
  uint8_t chroma[52];
};
constexpr QpTable qp_table() {
  constexpr int mf[6][3] = {{13107, 5243, 8066}, {11916, 4660, 7490}, {10082, 4194, 6554},
                            {9362, 3647, 5825},  {8192, 3355, 5243},  {7282, 2893, 4559}};
  constexpr int v[6][3] = {{10, 16, 13}, {11, 18, 14}, {13, 20, 16}, {14, 23, 18}, {16, 25, 20}, {18, 29, 23}};
  constexpr uint8_t c[22] = {29, 30, 31, 32, 32, 33, 34, 34, 35, 35, 36, 36, 37, 37, 37, 38, 38, 38, 39, 39, 39, 39};
  QpTable t{};
  for (int i = 0; i < 52; ++i) {
    const int per = i / 6, rem = i % 6;
    t.q[i] = QP{per,       rem,       15 + per,  (1 << (15 + per)) / 6, mf[rem][0],
                mf[rem][1], mf[rem][2], v[rem][0], v[rem][1],             v[rem][2]};
    t.chroma[i] = i < 30 ? (uint8_t)i : c[i - 30];
  }
  return t;
}
__constant__ QpTable kQpInter = qp_table();

// Four source bytes of a row at byte gx, clamped as stage16_clamped's.
__device__ __forceinline__ uint32_t source4(const uint8_t* row, int gx, int lim, bool vec, bool pair) {
  if (vec && gx + 4 <= lim) return __ldg(reinterpret_cast<const uint32_t*>(row + gx));
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int b = gx + j;
    w |= (uint32_t)__ldg(row + (pair ? 2 * min(b >> 1, (lim >> 1) - 1) + (b & 1) : min(b, lim - 1))) << (8 * j);
  }
  return w;
}

// Stages sixteen bytes of a row, `gx` 16-aligned, into `dst` (shared,
// 16-aligned): one vector load where the bytes lie inside [0, lim) of a row
// whose base is 16-byte aligned (`vec`), else byte loads of the clamped
// columns. `pair` selects NV12 chroma clamping: byte b of the row is
// component b&1 of sample clamp(b>>1, 0, lim/2-1).
__device__ __forceinline__ void stage16_clamped(uint8_t* dst, const uint8_t* row, int gx, int lim, bool vec,
                                                bool pair) {
  if (vec && gx >= 0 && gx + 16 <= lim) {
    *reinterpret_cast<uint4*>(dst) = __ldg(reinterpret_cast<const uint4*>(row + gx));
    return;
  }
#pragma unroll 1
  for (int j = 0; j < 16; ++j) {
    const int b = gx + j;
    const int c = pair ? 2 * clampi(b >> 1, 0, (lim >> 1) - 1) + (b & 1) : clampi(b, 0, lim - 1);
    dst[j] = __ldg(row + c);
  }
}

// One CTA holds blockDim.y macroblocks of a row (the autotuner's tile
// shape: 1, 2 or 4), 96 threads (three warps) each; a macroblock's shared
// state is its slice of the dynamic shared memory. T8: the 8x8 luma transform
// may be used (t8 = 1: everywhere, 2: chosen per macroblock). BATCH: one CTA per P
// macroblock of a batch (compact index blockIdx.x), which finds its stream,
// takes its vector from the batch's compact field and stores it into the
// stream's own field.
template <bool BATCH, bool T8>
__global__ void __launch_bounds__(384, 3) p_mb_kernel(const uint8_t* __restrict__ cur_y_, const uint8_t* __restrict__ cur_uv_,
                                                  int cur_pitch_, const uint8_t* __restrict__ ref_y_,
                                                  const uint8_t* __restrict__ ref_uv_, int ref_pitch_, Geo g_, int qp_,
                                                  const MV* __restrict__ mvs, int16_t* __restrict__ levels_,
                                                  int32_t* __restrict__ dc_, uint32_t* __restrict__ nzm_,
                                                  uint32_t* __restrict__ pred_mode_, uint8_t* __restrict__ rec_y_,
                                                  uint8_t* __restrict__ rec_uv_, int rec_pitch_, BatchTab bt,
                                                  int t8 = 0, uint8_t* __restrict__ t8_flags = nullptr) {
  pdl_wait();
  extern __shared__ __align__(16) uint8_t p_smem[];
  using Shared = typename std::conditional<T8, PShared8, PPatch>::type;
  Shared& s = reinterpret_cast<Shared*>(p_smem)[threadIdx.y];
  const int tid = threadIdx.x;
  const uint8_t *cur_y = cur_y_, *cur_uv = cur_uv_, *ref_y = ref_y_, *ref_uv = ref_uv_;
  int cur_pitch = cur_pitch_, ref_pitch = ref_pitch_, qp = qp_, rec_pitch = rec_pitch_;
  Geo g = g_;
  int16_t* levels = levels_;
  int32_t* dc = dc_;
  uint32_t *nzm = nzm_, *pred_mode = pred_mode_;
  uint8_t *rec_y = rec_y_, *rec_uv = rec_uv_;
  bool active;
  int mbx, mby, mb;
  MV mv;
  if (BATCH) {
    const int ci = blockIdx.x;
    const int k = bt.p_mbs.find(ci);
    const BatchStream& st = bt.p_mbs.stream(k);
    mb = ci - bt.p_mbs.prefix[k];
    g = st.g;
    if (mb >= g.mbw * g.mbh) return;  // padding of the compact index (uniform over the CTA)
    mby = mb / g.mbw;
    mbx = mb - mby * g.mbw;
    active = true;
    cur_y = st.cur_y;
    cur_uv = st.cur_uv;
    cur_pitch = st.cur_pitch;
    ref_y = st.ref_y;
    ref_uv = st.ref_uv;
    ref_pitch = rec_pitch = st.rec_pitch;
    qp = st.qp;
    levels = st.levels;
    dc = st.dc;
    nzm = st.nz;
    pred_mode = st.pred_mode;
    rec_y = st.rec_y;
    rec_uv = st.rec_uv;
    mv = bt.mvc[ci];
    if (tid == 0) st.mv[mb] = mv;
  } else {
    // a tile reaching past the right edge computes a copy of the last
    // macroblock and stores nothing
    const int mbx_t = blockIdx.x * blockDim.y + threadIdx.y;
    active = mbx_t < g.mbw;
    mbx = active ? mbx_t : g.mbw - 1;
    mby = blockIdx.y;
    mb = mby * g.mbw + mbx;
    mv = mvs[mb];
  }
  const int X = mbx * 16, Y = mby * 16, Xc = X >> 1, Yc = Y >> 1;
  const int ix0 = X + (mv.mvx >> 2), iy0 = Y + (mv.mvy >> 2), fx = mv.mvx & 3, fy = mv.mvy & 3;
  const int ixc = Xc + (mv.mvx >> 3), iyc = Yc + (mv.mvy >> 3), fxc = mv.mvx & 7, fyc = mv.mvy & 7;
  const int cmx = g.RW / 2 - 1, cmy = g.RH / 2 - 1;

  // ---- stage reference patches (16-byte units) ---------------------------
  // Units: 0..62 luma patch (21 rows x 3), 63..80 chroma patch (9 x 2). Reads
  // clamp to (RW, RH) for the reference and (W, H) for the source, per sample,
  // as the byte-wise reference stages do; the vector path is taken where no
  // clamp applies.
  const int lxa = (ix0 - 2) & ~15, lo = (ix0 - 2) - lxa;
  const int cxa = (2 * ixc) & ~15, co = 2 * ixc - cxa;
  const bool rvec = ((ref_pitch & 15) == 0) && ((reinterpret_cast<uintptr_t>(ref_y) & 15) == 0) &&
                    ((reinterpret_cast<uintptr_t>(ref_uv) & 15) == 0);
  const bool cvec = ((cur_pitch & 3) == 0) && ((reinterpret_cast<uintptr_t>(cur_y) & 3) == 0) &&
                    ((reinterpret_cast<uintptr_t>(cur_uv) & 3) == 0);
  if (tid < 63) {
    const int r = tid / 3, q = tid - 3 * r;
    const uint8_t* row = ref_y + (size_t)clampi(iy0 - 2 + r, 0, g.RH - 1) * ref_pitch;
    stage16_clamped(&s.lp[r][16 * q], row, lxa + 16 * q, g.RW, rvec, false);
  } else if (tid < 81) {
    const int r = (tid - 63) >> 1, q = (tid - 63) & 1;
    const uint8_t* row = ref_uv + (size_t)clampi(iyc + r, 0, cmy) * ref_pitch;
    stage16_clamped(&s.cp[r][16 * q], row, cxa + 16 * q, 2 * (g.RW / 2), rvec, true);
  }

  // Quad (b, r) owns row r of block b: luma blocks in raster order (warps 0 and
  // 1), then 2x2 of Cb and of Cr (warp 2). Chroma words are loaded, predicted and
  // stored as NV12 (lanes 16 apart hold the two halves of eight bytes) and
  // separated into planes by a shuffle in between.
  const int b = tid >> 2, r = tid & 3;
  const bool luma = b < 16;  // the same in a warp
  const int pl = (b - 16) >> 2, sub = b & 3;
  const int bx = b & 3, x0 = luma ? 4 * bx : 8 * (sub & 1) + 4 * pl;          // byte of the MB's row
  const int y0 = luma ? 4 * (b >> 2) + r : 4 * (sub >> 1) + r;
  uint32_t src = luma ? source4(cur_y + (size_t)min(Y + y0, g.H - 1) * cur_pitch, X + x0, g.W, cvec, false)
                      : source4(cur_uv + (size_t)min(Yc + y0, g.H / 2 - 1) * cur_pitch, 2 * Xc + x0, 2 * (g.W / 2), cvec, true);
  auto planes = [&](uint32_t w) -> uint32_t {  // NV12 halves to one plane's four samples
    const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 16);
    return pl ? __byte_perm(w, o, 0x3175) : __byte_perm(w, o, 0x6420);
  };
  __syncthreads();

  // ---- prediction + residual --------------------------------------------
  uint32_t pred;
  if (luma) {
    pred = mc_luma4(s.lp, lo, x0, y0, fx, fy);
  } else {
    pred = planes(mc_chroma4(s.cp, co + x0, y0, fxc, fyc));
    src = planes(src);
  }
  // ---- 4x4 or 8x8 luma transform (t8 = 2: chosen per macroblock) --------
  // The residual's cost under each size, on the scale of a SAD: 4x4 blocks
  // (sum |H4 R H4|) / 2 - quads of warps 0-1, row r of block b, the column
  // pass across the quad by shuffles - and 8x8 blocks (sum |H8 R H8| + 2) / 4
  // - warp 2, eight lanes per block, transposed through s.t8. H4 and H8 are
  // unnormalised Walsh-Hadamard matrices; any row order gives the same sums.
  bool use8 = false;
  if constexpr (T8) {
    if (luma) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pv = (int)(pred >> (8 * i) & 0xffu);
        s.res[b][4 * r + i] = (int16_t)((int)(src >> (8 * i) & 0xffu) - pv);
        s.pred[b][4 * r + i] = (int16_t)pv;
      }
    }
    __syncthreads();
    use8 = t8 == 1;
    if (t8 == 2) {
      if (tid < 64) {
        const int bb = tid >> 2, rr = tid & 3;
        int h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = s.res[bb][4 * rr + i];
        const int a0 = h[0] + h[1], a1 = h[0] - h[1], a2 = h[2] + h[3], a3 = h[2] - h[3];
        h[0] = a0 + a2;
        h[1] = a1 + a3;
        h[2] = a0 - a2;
        h[3] = a1 - a3;
        int sum = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int o1 = __shfl_xor_sync(0xffffffffu, h[i], 1);
          const int u = (rr & 1) ? o1 - h[i] : h[i] + o1;
          const int o2 = __shfl_xor_sync(0xffffffffu, u, 2);
          const int w = (rr & 2) ? o2 - u : u + o2;
          sum += abs(w);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        int c = rr == 0 ? sum >> 1 : 0;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if ((tid & 31) == 0) s.cost[tid >> 5] = c;
      } else {
        const int ln = tid - 64, qq = ln >> 3, kk = ln & 7, ox = 8 * (qq & 1), oy = 8 * (qq >> 1);
        int v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int xx = ox + c, yy = oy + kk;
          v[c] = s.res[(yy >> 2) * 4 + (xx >> 2)][(yy & 3) * 4 + (xx & 3)];
        }
        had8(v);
#pragma unroll
        for (int c = 0; c < 8; ++c) s.t8[qq][8 * kk + c] = v[c];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = s.t8[qq][8 * i + kk];
        had8(v);
        int sum = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += abs(v[i]);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        int c = kk == 0 ? (sum + 2) >> 2 : 0;
        c += __shfl_xor_sync(0xffffffffu, c, 8);
        c += __shfl_xor_sync(0xffffffffu, c, 16);
        if (ln == 0) s.cost[2] = c;
      }
      __syncthreads();
      use8 = s.cost[2] < s.cost[0] + s.cost[1];
    }
  }

  // ---- forward + quant ----------------------------------------------------
  // (with the 8x8 luma transform, warp 0 codes the four 8x8 luma blocks
  // instead and warp 1 has no luma block; chroma is the same). Position class
  // of coefficient (i, r), and of (r, i): two per lane, by the parity of i.
  const QP q = kQpInter.q[luma ? qp : kQpInter.chroma[qp]];
  const int mf_even = (r & 1) ? q.mf2 : q.mf0, mf_odd = (r & 1) ? q.mf1 : q.mf2;
  const int v_even = (r & 1) ? q.v2 : q.v0, v_odd = (r & 1) ? q.v1 : q.v2;
  const bool quad = !(T8 && use8 && luma);  // the same in a warp
  if (quad) {
    int x[4];
    quad_forward_bytes(src, pred, r, x);  // x[i] = coef[i][r]
    const int c0 = x[0];
    uint32_t nz = 0;
    int l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int a = (abs(x[i]) * ((i & 1) ? mf_odd : mf_even) + q.f) >> q.f_shift;
      l[i] = x[i] < 0 ? -a : a;  // under 3,673: 36 * 255 * 13107 >> 15
      nz |= (a != 0 ? 1u : 0u) << (4 * i + r);
    }
    nz |= __shfl_xor_sync(0xffffffffu, nz, 1);
    nz |= __shfl_xor_sync(0xffffffffu, nz, 2);
    if (r == 0 && active) {
      nzm[(size_t)mb * 24 + b] = nz;
      dc[(size_t)mb * 24 + b] = c0;
    }
    const uint2 row = quad_transpose_pairs(make_uint2(__byte_perm(l[0], l[1], 0x5410), __byte_perm(l[2], l[3], 0x5410)), r);
    if (active) reinterpret_cast<uint2*>(levels + (size_t)mb * 384)[4 * b + r] = row;

    // ---- dequant + inverse + recon ----------------------------------------
    // (level * 16 V << per) >> 4, rounded (reconstruct.comp): the sixteen makes
    // the division exact and the rounding empty for every per
    int d[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      d[i] = ((int)(int16_t)((i < 2 ? row.x : row.y) >> (16 * (i & 1))) * ((i & 1) ? v_odd : v_even)) << q.per;
    if (!luma) {
      // chroma DC Hadamard + quant + inverse + dequant (reconstruct.comp:393-414):
      // lane r quantizes the plane's coefficient r, lane 0 of a quad takes its
      // block's value
      const int plane0 = tid & 16;
      const int k0 = __shfl_sync(0xffffffffu, c0, plane0), k1 = __shfl_sync(0xffffffffu, c0, plane0 + 4);
      const int k2 = __shfl_sync(0xffffffffu, c0, plane0 + 8), k3 = __shfl_sync(0xffffffffu, c0, plane0 + 12);
      auto hadamard = [](int a, int b, int c, int d, int k) {
        return a + ((k & 1) ? -b : b) + ((k & 2) ? -c : c) + ((k == 1 || k == 2) ? -d : d);
      };
      const int lr = quantize_dc(hadamard(k0, k1, k2, k3, r), q);
      const int lane0 = tid & 28;
      const int l0 = __shfl_sync(0xffffffffu, lr, lane0), l1 = __shfl_sync(0xffffffffu, lr, lane0 + 1);
      const int l2 = __shfl_sync(0xffffffffu, lr, lane0 + 2), l3 = __shfl_sync(0xffffffffu, lr, lane0 + 3);
      if (r == 0) d[0] = dequant_dc_chroma(hadamard(l0, l1, l2, l3, sub), q);
    }
    if (r == 0) d[0] += 32;
    quad_inverse(d, r);  // d[i] = res[i][r]
    const uint32_t pc = quad_transpose_bytes(pred, r);
    // sample i of the column, plus its residual
    uint32_t rec = clip4(dot4(pc, 0x00000001u, d[0]), dot4(pc, 0x00000100u, d[1]), dot4(pc, 0x00010000u, d[2]),
                         dot4(pc, 0x01000000u, d[3]));
    rec = quad_transpose_bytes(rec, r);
    if (luma) {
      const int gy = Y + y0, gx = X + x0;
      if (active && gy < g.RH) {
        uint8_t* dst = rec_y + (size_t)gy * rec_pitch + gx;
        if (gx + 4 <= g.RW) {
          *reinterpret_cast<uint32_t*>(dst) = rec;
        } else {
          for (int c = 0; c < 4 && gx + c < g.RW; ++c) dst[c] = (uint8_t)(rec >> (8 * c));
        }
      }
    } else {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, rec, 16);  // back to NV12 halves
      rec = pl ? __byte_perm(o, rec, 0x7362) : __byte_perm(rec, o, 0x5140);
      const int gy = Yc + y0, gc = Xc + (x0 >> 1);
      if (active && gy <= cmy) {
        uint8_t* dst = rec_uv + (size_t)gy * rec_pitch + 2 * gc;
        if (gc + 1 <= cmx) {
          *reinterpret_cast<uint32_t*>(dst) = rec;
        } else if (gc <= cmx) {
          dst[0] = (uint8_t)rec;
          dst[1] = (uint8_t)(rec >> 8);
        }
      }
    }
  }

  // 8x8 luma (warp 0): block q8 = tid >> 3 (raster of the four), thread k8
  // owns its row k8, then its column k8. Levels in raster order at
  // lev[0..255] (block q8 at 64 * q8); the nz word of 4x4 block 4 * q8 + i
  // (spec order) holds the nonzero mask of the 16 levels CAVLC codes as that
  // block: 8x8 scan positions i, i + 4, ... (7.3.5.3.2).
  if constexpr (T8) {
    if (use8 && tid < 32) {
      const int q8 = tid >> 3, k8 = tid & 7, qx = 8 * (q8 & 1), qy = 8 * (q8 >> 1);
      const int per8 = qp / 6, rem8 = qp - 6 * per8;
      auto res_at = [&](int xx, int yy) { return (int)s.res[(yy >> 2) * 4 + (xx >> 2)][(yy & 3) * 4 + (xx & 3)]; };
      int v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = res_at(qx + c, qy + k8);
      fwd8(v);
#pragma unroll
      for (int c = 0; c < 8; ++c) s.t8[q8][8 * k8 + c] = v[c];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = s.t8[q8][8 * i + k8];
      fwd8(v);
      const int sh = 16 + per8;
      const long long f = (1ll << sh) / 6;  // inter rounding
      uint32_t m[4] = {0u, 0u, 0u, 0u};
      int16_t* lev8 = &s.lev[0][0] + 64 * q8;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int l = quant8(v[i], i, k8, rem8, sh, f);
        lev8[8 * i + k8] = (int16_t)clampi(l, -32768, 32767);
        const int z = kZigzag8Inv[8 * i + k8];
        m[z & 3] |= (l != 0 ? 1u : 0u) << (z >> 2);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        m[j] |= __shfl_xor_sync(0xffffffffu, m[j], 1);
        m[j] |= __shfl_xor_sync(0xffffffffu, m[j], 2);
        m[j] |= __shfl_xor_sync(0xffffffffu, m[j], 4);
      }
      if (k8 == 0 && active) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // spec block 4 * q8 + i -> raster: quadrant origin (qx / 4, qy / 4) + (i & 1, i >> 1)
          const int rb = (qy / 4 + (i >> 1)) * 4 + qx / 4 + (i & 1);
          nzm[(size_t)mb * 24 + rb] = m[i];
          dc[(size_t)mb * 24 + rb] = 0;
        }
      }
      __syncwarp();
      // scaling + inverse (8.5.13) onto the prediction
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = scale8(lev8[8 * k8 + c], k8, c, per8, rem8);
      inv8(v);
#pragma unroll
      for (int c = 0; c < 8; ++c) s.t8[q8][8 * k8 + c] = v[c];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = s.t8[q8][8 * i + k8];
      inv8(v);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int yy = qy + i, xx = qx + k8;
        s.ry[yy][xx] = (uint8_t)clip1(s.pred[(yy >> 2) * 4 + (xx >> 2)][(yy & 3) * 4 + (xx & 3)] + ((v[i] + 32) >> 6));
      }
      __syncwarp();
      if (active) {
        reinterpret_cast<uint4*>(levels + (size_t)mb * 384)[tid] = reinterpret_cast<const uint4*>(&s.lev[0][0])[tid];
        const int gy = Y + tid;
        if (tid < 16 && gy < g.RH) {
          uint8_t* dst = rec_y + (size_t)gy * rec_pitch + X;
          if (X + 16 <= g.RW) {
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(s.ry[tid]);
          } else {
            for (int c = 0; c < 16 && X + c < g.RW; ++c) dst[c] = s.ry[tid][c];
          }
        }
      }
    }
  }
  if (tid == 0 && active) {
    pred_mode[mb] = 2u;  // residual_predict.comp:422
    if (t8_flags) t8_flags[mb] = use8 ? 1u : 0u;
  }
}

}  // namespace b200enc

using namespace b200enc;

extern "C" int b200enc_p_frame_t8(const uint8_t* cur_y, const uint8_t* cur_uv, int cur_pitch, const uint8_t* ref_y,
                                  const uint8_t* ref_uv, int ref_pitch, int W, int H, int RW, int RH, int qp,
                                  const void* mv, int16_t* levels, int32_t* dc, uint32_t* nz, uint32_t* pred_mode,
                                  uint8_t* rec_y, uint8_t* rec_uv, int rec_pitch, int t8, uint8_t* t8_flags,
                                  void* stream);

extern "C" int b200enc_p_frame(const uint8_t* cur_y, const uint8_t* cur_uv, int cur_pitch, const uint8_t* ref_y,
                               const uint8_t* ref_uv, int ref_pitch, int W, int H, int RW, int RH, int qp,
                               const void* mv, int16_t* levels, int32_t* dc, uint32_t* nz, uint32_t* pred_mode,
                               uint8_t* rec_y, uint8_t* rec_uv, int rec_pitch, void* stream) {
  return b200enc_p_frame_t8(cur_y, cur_uv, cur_pitch, ref_y, ref_uv, ref_pitch, W, H, RW, RH, qp, mv, levels, dc,
                            nz, pred_mode, rec_y, rec_uv, rec_pitch, 0, nullptr, stream);
}

extern "C" int b200enc_p_frame_t8(const uint8_t* cur_y, const uint8_t* cur_uv, int cur_pitch, const uint8_t* ref_y,
                                  const uint8_t* ref_uv, int ref_pitch, int W, int H, int RW, int RH, int qp,
                                  const void* mv, int16_t* levels, int32_t* dc, uint32_t* nz, uint32_t* pred_mode,
                                  uint8_t* rec_y, uint8_t* rec_uv, int rec_pitch, int t8, uint8_t* t8_flags,
                                  void* stream) {
  if (t8 < 0 || t8 > 2) return -1;
  if (!cur_y || !cur_uv || !ref_y || !ref_uv || !mv || !levels || !dc || !nz || !pred_mode || !rec_y || !rec_uv)
    return -1;
  if (qp < 0 || qp > 51 || W <= 0 || H <= 0 || RW <= 1 || RH <= 1) return -1;
  if ((rec_pitch & 15) || (((uintptr_t)rec_y) & 15) || (((uintptr_t)rec_uv) & 15) || (((uintptr_t)levels) & 15))
    return -1;
  if ((ref_pitch & 1) || (((uintptr_t)ref_uv) & 1)) return -1;
  Geo g{W, H, RW, RH, (W + 15) / 16, (H + 15) / 16};
  const int T = b200enc_tuned(B200ENC_TUNE_PCHAIN_MBS_PER_CTA) > 0 ? b200enc_tuned(B200ENC_TUNE_PCHAIN_MBS_PER_CTA) : 1;
  const dim3 grid((g.mbw + T - 1) / T, g.mbh), block(96, T);
  const cudaStream_t st = (cudaStream_t)stream;
  if (t8 != 0) {
    launch_early(p_mb_kernel<false, true>, grid, block, T * sizeof(PShared8), st, cur_y, cur_uv, cur_pitch, ref_y, ref_uv,
                 ref_pitch, g, qp, (const MV*)mv, levels, dc, nz, pred_mode, rec_y, rec_uv, rec_pitch, BatchTab{}, t8,
                 t8_flags);
  } else {
    launch_early(p_mb_kernel<false, false>, grid, block, T * sizeof(PPatch), st, cur_y, cur_uv, cur_pitch, ref_y, ref_uv,
                 ref_pitch, g, qp, (const MV*)mv, levels, dc, nz, pred_mode, rec_y, rec_uv, rec_pitch, BatchTab{}, 0,
                 t8_flags);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// The P chain of every P macroblock of a batch (n = the compact P count).
int b200enc_p_frame_batch_launch(const BatchTab& bt, int n, cudaStream_t st) {
  if (n <= 0) return 0;
  p_mb_kernel<true, false><<<n, dim3(96, 1), sizeof(PPatch), st>>>(nullptr, nullptr, 0, nullptr, nullptr, 0, Geo{}, 0,
                                                             nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                             nullptr, 0, bt);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
