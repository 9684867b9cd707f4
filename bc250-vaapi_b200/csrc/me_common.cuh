// me_common.cuh - pieces shared by the full-search and learned-proposal
// motion estimators: byte-SIMD SAD, block reductions, and the half/quarter-pel
// refine of A1/shaders/motion_estimation.comp (:154-215 interpolation,
// :388-459 refine order), run on an integer winner whose neighbourhood the
// caller has staged in shared memory.
#pragma once
#include "common.cuh"

namespace b200enc {

__device__ __forceinline__ uint32_t sad4_acc(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

__device__ __forceinline__ int lane_id() { return (int)(threadIdx.x & 31); }

template <int NT>
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (NT == 32) return v;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < NT / 32; ++i) s += red[i];
  return s;
}

template <int NT>
__device__ __forceinline__ uint32_t block_min(uint32_t v, uint32_t* red) {
  v = __reduce_min_sync(0xffffffffu, v);
  if (NT == 32) return v;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t m = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < NT / 32; ++i) m = min(m, red[i]);
  return m;
}

// The log word a search writes into MV.pad under B200ENC_ME_LOG_INTEGER:
// bit 31 set, bit 30 = zero-MV early-out, bits 8-15 = integer winner dy +
// 128, bits 0-7 = dx + 128.
__device__ __forceinline__ uint32_t me_log_word(int mx, int my, bool early) {
  return 0x80000000u | (early ? 0x40000000u : 0u) | ((uint32_t)(my + 128) << 8) | (uint32_t)(mx + 128);
}

// Candidate offsets in quarter pels, motion_estimation.comp:395-398, :435-438.
__constant__ int8_t kHalfOff[8][2] = {{2, 0}, {-2, 0}, {0, 2}, {0, -2}, {2, 2}, {2, -2}, {-2, 2}, {-2, -2}};
__constant__ int8_t kQtrOff[8][2] = {{1, 0}, {-1, 0}, {0, 1}, {0, -1}, {1, 1}, {1, -1}, {-1, 1}, {-1, -1}};

// One 32-bit word of a reference row (4 pels from gx), with the column
// clamped to [0, RW-1] per pel when the word leaves the plane.
__device__ __forceinline__ uint32_t load_word_clamped(const uint8_t* row, int gx, int RW) {
  if (gx >= 0 && gx + 3 < RW) return __ldg(reinterpret_cast<const uint32_t*>(row + gx));
  return (uint32_t)__ldg(row + clampi(gx, 0, RW - 1)) | ((uint32_t)__ldg(row + clampi(gx + 1, 0, RW - 1)) << 8) |
         ((uint32_t)__ldg(row + clampi(gx + 2, 0, RW - 1)) << 16) |
         ((uint32_t)__ldg(row + clampi(gx + 3, 0, RW - 1)) << 24);
}

// ---------------------------------------------------------------------------
// Half- then quarter-pel refine around an integer winner (strict improvement
// only, offsets tried in table order), one warp, on byte-SIMD words: the
// half-pel planes are bytes (their values are clipped to 0..255), every
// quarter-pel sample is either a plane value or the rounded byte average
// (a + b + 1) >> 1 of two, which vavgu4 forms for 4 pels at once, and
// vabsdiff4 accumulates the SAD. Instructions bound it (one warp per
// macroblock, no reuse between macroblocks): the planes take one pass of
// packed 16-bit arithmetic instead of eleven passes of a sample per lane, the
// positions one loop instead of sixteen unrolled bodies. Re-scoring a 640x480
// frame: 13.8 -> 11.1 us; the fallback search of a few macroblocks: 31 -> 17.
struct RefineSimd {
  alignas(4) uint8_t pl[3][18][20];  // b, h, j at [ry+1][rx+1], ry, rx in -1..16
};

// The operands of each quarter-pel phase (fy*4+fx), motion_estimation.comp:
// 197-213: plane (0 G, 1 b, 2 h, 3 j) and extra shifts sx, sy of each; the
// sample is the rounded average of both, which is the operand itself where a
// phase has one (listed twice). Bits: plane a 0-1, sx a 2, sy a 3, plane b
// 4-5, sx b 6, sy b 7.
#define B200ENC_QOP(pa, xa, ya, pb, xb, yb) \
  (uint8_t)((pa) | ((xa) << 2) | ((ya) << 3) | ((pb) << 4) | ((xb) << 6) | ((yb) << 7))
__constant__ uint8_t kQpelOp[16] = {
    B200ENC_QOP(0, 0, 0, 0, 0, 0), B200ENC_QOP(0, 0, 0, 1, 0, 0), B200ENC_QOP(1, 0, 0, 1, 0, 0),
    B200ENC_QOP(1, 0, 0, 0, 1, 0), B200ENC_QOP(0, 0, 0, 2, 0, 0), B200ENC_QOP(1, 0, 0, 2, 0, 0),
    B200ENC_QOP(1, 0, 0, 3, 0, 0), B200ENC_QOP(1, 0, 0, 2, 1, 0), B200ENC_QOP(2, 0, 0, 2, 0, 0),
    B200ENC_QOP(2, 0, 0, 3, 0, 0), B200ENC_QOP(3, 0, 0, 3, 0, 0), B200ENC_QOP(3, 0, 0, 2, 1, 0),
    B200ENC_QOP(2, 0, 0, 0, 0, 1), B200ENC_QOP(2, 0, 0, 1, 0, 1), B200ENC_QOP(3, 0, 0, 1, 0, 1),
    B200ENC_QOP(2, 1, 0, 1, 0, 1)};
#undef B200ENC_QOP

// Two samples in the 16-bit halves of a word (each 0 .. 65535; sums and
// multiples stay below 65536 per half, differences are biased to stay
// non-negative, so plain 32-bit arithmetic never carries across).
//
// The 6-tap sum a - 5b + 20c + 20d - 5e + f of byte samples, plus kTapBias
// (2560 = 80 * 32 > 2550): 10 .. 13270.
constexpr uint32_t kTapBias = 2560u;
__device__ __forceinline__ uint32_t tap6_pair(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f) {
  return (c + d) * 20u + (a + f + kTapBias * 0x10001u) - (b + e) * 5u;
}
// clip1((tap + 16) >> 5) of both halves of a biased sum.
__device__ __forceinline__ uint32_t tap_round_pair(uint32_t t) {
  const uint32_t v = ((t + 0x00100010u) >> 5) & 0x07ff07ffu;  // + 80
  uint32_t lo, hi;
  asm("max.u16x2 %0, %1, %2;" : "=r"(lo) : "r"(v), "r"(0x00500050u));
  asm("min.u16x2 %0, %1, %2;" : "=r"(hi) : "r"(lo), "r"(0x014f014fu));
  return hi - 0x00500050u;
}

// Half-pel planes b, h, j (motion_estimation.comp:154-215) of the 18 x 18
// positions around the winner: lane = (group of three rows, four columns);
// the lane reads the eight reference rows its rows reach (nine bytes each)
// and keeps their horizontal sums in registers, so nothing but the planes is
// written. g: 4-aligned rows, gstride bytes apart; the winner's top-left pel
// is at row g_r0, byte g_c0.
__device__ __forceinline__ void refine_planes(RefineSimd& rf, const uint8_t* g, int gstride, int g_r0, int g_c0,
                                              int lane) {
  if (lane < 30) {
    const int grp = lane / 5, q = lane - 5 * grp;
    const int bo = g_c0 + 4 * q - 3, sh = (bo & 3) * 8;  // byte of column rx - 2, rx = 4q - 1
    const uint8_t* rows = g + (g_r0 + 3 * grp - 3) * gstride + (bo & ~3);
    uint32_t t01[8], t23[8], g01[8], g23[8];  // horizontal sums (biased) and samples, rows 3 grp - 3 .. + 4
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(rows + r * gstride);
      const uint32_t a0 = wp[0], a1 = wp[1], a2 = wp[2];
      const uint32_t lo = __funnelshift_r(a0, a1, sh), hi = __funnelshift_r(a1, a2, sh), up = a2 >> sh;  // e0.., e4.., e8
      constexpr uint32_t ta = 0x1414fb01u, tb = 0x000001fbu;  // 1 -5 20 20, -5 1
      const int t0 = dot4(lo, ta, dot4(hi, tb, (int)kTapBias));
      const int t1 = dot4(__funnelshift_r(lo, hi, 8), ta, dot4(__funnelshift_r(hi, up, 8), tb, (int)kTapBias));
      const int t2 = dot4(__funnelshift_r(lo, hi, 16), ta, dot4(hi >> 16, tb, (int)kTapBias));
      const int t3 = dot4(__funnelshift_r(lo, hi, 24), ta, dot4(__funnelshift_r(hi, up, 24), tb, (int)kTapBias));
      t01[r] = __byte_perm(t0, t1, 0x5410);
      t23[r] = __byte_perm(t2, t3, 0x5410);
      g01[r] = __byte_perm(lo, 0, 0x4342);
      g23[r] = __byte_perm(hi, 0, 0x4140);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // plane row 3 grp + k (ry = that - 1): reference rows k .. k + 5 of the eight
      uint32_t* bp = reinterpret_cast<uint32_t*>(&rf.pl[0][3 * grp + k][4 * q]);
      uint32_t* hp = reinterpret_cast<uint32_t*>(&rf.pl[1][3 * grp + k][4 * q]);
      uint32_t* jp = reinterpret_cast<uint32_t*>(&rf.pl[2][3 * grp + k][4 * q]);
      *bp = __byte_perm(tap_round_pair(t01[k + 2]), tap_round_pair(t23[k + 2]), 0x6420);
      *hp = __byte_perm(tap_round_pair(tap6_pair(g01[k], g01[k + 1], g01[k + 2], g01[k + 3], g01[k + 4], g01[k + 5])),
                        tap_round_pair(tap6_pair(g23[k], g23[k + 1], g23[k + 2], g23[k + 3], g23[k + 4], g23[k + 5])),
                        0x6420);
      // the taps' weights sum to 32, so the bias of the sums comes out as 32 * kTapBias
      int v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {  // a column's sums two rows to a word, three integer dot products
        const uint32_t* t = c < 2 ? t01 : t23;
        auto rows2 = [&](int i) -> int { return (int)__byte_perm(t[k + i], t[k + i + 1], (c & 1) ? 0x7632 : 0x5410); };
        v[c] = __dp2a_lo(rows2(0), 0xfb01, __dp2a_lo(rows2(2), 0x1414, __dp2a_lo(rows2(4), 0x01fb, 512 - 32 * (int)kTapBias))) >> 10;
      }
      *jp = clip4(v[0], v[1], v[2], v[3]);
    }
  }
}

// g: 4-aligned rows of the reference, gstride bytes apart; the integer
// winner's top-left pel is at row g_r0, byte g_c0 (rows g_r0-3 .. g_r0+19
// and bytes g_c0-3 .. g_c0+19+8 must be readable). cur: the 64 words of the
// current MB. Every lane of the warp returns the same result.
__device__ __forceinline__ uint32_t qpel_refine_warp_simd(RefineSimd& rf, const uint8_t* g, int gstride, int g_r0,
                                                          int g_c0, const uint32_t* cur, uint32_t int_sad,
                                                          int* qx_out, int* qy_out) {
  const int lane = threadIdx.x & 31;
  refine_planes(rf, g, gstride, g_r0, g_c0, lane);
  __syncwarp();

  // Each stage's eight positions at once: lane L scores four rows of position
  // L >> 2 (rows (L & 3), + 4, ...), two shuffles finish the sums and one
  // redux min over (SAD << 3 | position) picks the earliest smallest. Both
  // stages run the same few instructions: the code of the eight positions
  // written out (three times the instructions, most of them fetched cold by a
  // launch of a few macroblocks) was the slower form.
  const int pos = lane >> 2;
  uint32_t bsad = int_sad;
  int bx = 0, by = 0;
#pragma unroll 1
  for (int stage = 0; stage < 2; ++stage) {
    const int ox = bx + (stage ? kQtrOff[pos][0] : kHalfOff[pos][0]);
    const int oy = by + (stage ? kQtrOff[pos][1] : kHalfOff[pos][1]);
    const uint32_t op = kQpelOp[(oy & 3) * 4 + (ox & 3)];
    // the first row of an operand: address of its word, bit shift, row pitch
    auto operand = [&](uint32_t o, const uint32_t*& p, int& sh, int& pitch) {
      const int rx = (ox >> 2) + (int)((o >> 2) & 1u), ry = (oy >> 2) + (int)((o >> 3) & 1u) + (lane & 3);
      const int pl = (int)(o & 3u);
      pitch = pl ? 20 : gstride;
      const int c = pl ? rx + 1 : g_c0 + rx;
      const uint8_t* base = pl ? &rf.pl[0][0][0] + (pl - 1) * 360 + (ry + 1) * 20 : g + (g_r0 + ry) * gstride;
      p = reinterpret_cast<const uint32_t*>(base + (c & ~3));
      sh = (c & 3) * 8;
    };
    const uint32_t *pa, *pb;
    int sa, sb, ia, ib;
    operand(op, pa, sa, ia);
    operand(op >> 4, pb, sb, ib);
    uint32_t sad = 0;
    // every fourth row: word steps of 4 pitches / 4 bytes; the half positions
    // are samples of one plane, not averages of two
#pragma unroll 1
    for (int r = 0; r < 4; ++r, pa += ia, pb += ib) {
      const uint4 c = *reinterpret_cast<const uint4*>(cur + 4 * ((lane & 3) + 4 * r));
      const uint32_t a0 = pa[0], a1 = pa[1], a2 = pa[2], a3 = pa[3], a4 = pa[4];
      uint32_t v0 = __funnelshift_r(a0, a1, sa), v1 = __funnelshift_r(a1, a2, sa);
      uint32_t v2 = __funnelshift_r(a2, a3, sa), v3 = __funnelshift_r(a3, a4, sa);
      if (stage) {
        const uint32_t b0 = pb[0], b1 = pb[1], b2 = pb[2], b3 = pb[3], b4 = pb[4];
        v0 = avg4(v0, __funnelshift_r(b0, b1, sb));
        v1 = avg4(v1, __funnelshift_r(b1, b2, sb));
        v2 = avg4(v2, __funnelshift_r(b2, b3, sb));
        v3 = avg4(v3, __funnelshift_r(b3, b4, sb));
      }
      sad = sad4_acc(v0, c.x, sad);
      sad = sad4_acc(v1, c.y, sad);
      sad = sad4_acc(v2, c.z, sad);
      sad = sad4_acc(v3, c.w, sad);
    }
    sad += __shfl_xor_sync(0xffffffffu, sad, 1);
    sad += __shfl_xor_sync(0xffffffffu, sad, 2);
    const uint32_t m = __reduce_min_sync(0xffffffffu, (sad << 3) | (uint32_t)pos);
    if ((m >> 3) < bsad) {
      bsad = m >> 3;
      bx += stage ? kQtrOff[m & 7][0] : kHalfOff[m & 7][0];
      by += stage ? kQtrOff[m & 7][1] : kHalfOff[m & 7][1];
    }
  }
  *qx_out = bx;
  *qy_out = by;
  return bsad;
}

}  // namespace b200enc
