// deblock_tile.cuh - the filtering of one deblocking tile in seven phases of
// independent lines (H.264 clause 8.7, raster order reproduced exactly).
//
// Raster-order deblocking looks like a wavefront (vertical then horizontal
// edges of a macroblock, macroblocks left to right, top to bottom), but its
// dependencies are short. Write e0..e3 for the edges of a direction (e0 the
// macroblock edge), 0..15 for the samples across them. A normal filter (every
// internal edge) changes p1 p0 q0 q1 and reads p2..q2, and the q1 it leaves
// depends on p1 p0 q0 q1 q2 alone. So the sample e2 hands on to e3 (sample 9)
// and e3 itself follow from samples 6..14, which e0 and e1 do not change:
// samples 9..15 of a line are final for a direction without e0, e1 or the
// rest of e2. That cuts the chains from macroblock to macroblock:
//
//   1   vertical   sample 9 of e2, then e3   every row
//   2   horizontal sample 9 of e2, then e3   columns 9..15
//   3   vertical   e0 e1 e2                  rows 9..15
//   4   horizontal e0 e1 e2                  columns 9..15
//   5   vertical   e0 e1 e2                  rows 0..8
//   6   horizontal sample 9 of e2, then e3   columns 0..8
//   7   horizontal e0 e1 e2                  columns 0..8
//
// Each phase's lines are independent of each other over the whole tile, and
// every sample reaches each filter in its raster-order state: the left
// macroblock's columns 12..15 have passed its horizontal edges (2 and 4)
// before the vertical e0 reads them (3 and 5); the rows 12..15 above have
// passed their own horizontal edges (2, 6) and the next macroblock's vertical
// e0 (3) before the horizontal e0 reads them (4, 7). The second visit of e2
// takes the two q samples phases 1, 2 and 6 may have changed from a saved
// copy. Chroma (edges e0 and e2, filters that change p0 q0 and read p1..q1)
// runs in the same phases: 1 vertical e2; 2 horizontal e2, columns 2..7;
// 3 vertical e0, rows 2..7; 4 horizontal e0, columns 2..7; 5 vertical e0,
// rows 0..1; 6 horizontal e2, columns 0..1; 7 horizontal e0, columns 0..1.
//
// The margin a tile needs is what those phases read: 10 luma rows above, 7
// below, 12 columns left (9..15 filtered), 4 right; 2 chroma rows above and
// below, 2 columns left and right. A macroblock of the margin runs only the
// edges whose results reach the tile (of the rows above only 13..15 do in
// columns 0..8, and row 13's value, e3's q1, follows from rows 10..14).
//
// The functions take one line each and hold no CUDA intrinsics, so the CPU
// test drives the same code (tests/test_deblock_phases.py).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define DT_FN __host__ __device__ __forceinline__
#else
#define DT_FN static inline
#endif

namespace b200enc {

DT_FN int dt_abs(int v) { return v < 0 ? -v : v; }
DT_FN int dt_clamp(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Filter thresholds of one picture (uniform QP): luma and chroma alpha/beta
// and tC0 for bS 1..3.
struct DbQ {
  int al, be, alc, bec, tcl1, tcl2, tcl3, tcc1, tcc2, tcc3, is_intra;
};

DT_FN int tc0_for(int bs, int t1, int t2, int t3) { return bs == 1 ? t1 : (bs == 2 ? t2 : t3); }

// Line filters (clause 8.7.2.3 / 8.7.2.4) on samples held in registers. They
// are branch-free: every lane evaluates the whole filter and keeps the result
// by selection, so lanes whose edges differ in bS or in the sample tests never
// split the warp, and the dependent chain per edge stays short. A line with
// bS 0 or a failed sample test is left as it is.
//
// This encoder's boundary strengths are 4 on the macroblock edges of intra
// pictures, 3 on their internal edges and 0-2 in P pictures, so the strong
// filter is taken on a uniform condition (intra picture, macroblock edge) and
// the normal filter elsewhere.
DT_FN void luma_normal(int p2, int& p1, int& p0, int& q0, int& q1, int q2, int bs, int alpha, int beta, int tc0) {
  const int dqp = q0 - p0;
  const bool f = (bs != 0) & (dt_abs(dqp) < alpha) & (dt_abs(p1 - p0) < beta) & (dt_abs(q1 - q0) < beta);
  const bool ap = dt_abs(p2 - p0) < beta, aq = dt_abs(q2 - q0) < beta;
  const int tc = tc0 + (int)ap + (int)aq;
  const int delta = dt_clamp((dqp * 4 + (p1 - q1) + 4) >> 3, -tc, tc);
  const int avg = (p0 + q0 + 1) >> 1;
  const int np1 = p1 + dt_clamp((p2 + avg - (p1 << 1)) >> 1, -tc0, tc0);
  const int nq1 = q1 + dt_clamp((q2 + avg - (q1 << 1)) >> 1, -tc0, tc0);
  const int np0 = dt_clamp(p0 + delta, 0, 255), nq0 = dt_clamp(q0 - delta, 0, 255);
  p1 = (f & ap) ? np1 : p1;
  q1 = (f & aq) ? nq1 : q1;
  p0 = f ? np0 : p0;
  q0 = f ? nq0 : q0;
}

// The q1 a normal filter leaves (it depends on neither p2 nor on what the
// edge before changes).
DT_FN int luma_normal_q1(int p1, int p0, int q0, int q1, int q2, int bs, int alpha, int beta, int tc0) {
  const bool f = (bs != 0) & (dt_abs(q0 - p0) < alpha) & (dt_abs(p1 - p0) < beta) & (dt_abs(q1 - q0) < beta) &
                 (dt_abs(q2 - q0) < beta);
  const int nq1 = q1 + dt_clamp((q2 + ((p0 + q0 + 1) >> 1) - (q1 << 1)) >> 1, -tc0, tc0);
  return f ? nq1 : q1;
}

DT_FN void luma_strong(int p3, int& p2, int& p1, int& p0, int& q0, int& q1, int& q2, int q3, int bs, int alpha,
                       int beta) {
  const int d0 = dt_abs(p0 - q0);
  const bool f = (bs != 0) & (d0 < alpha) & (dt_abs(p1 - p0) < beta) & (dt_abs(q1 - q0) < beta);
  const bool small = d0 < ((alpha >> 2) + 2);
  const bool sp = f & small & (dt_abs(p2 - p0) < beta), sq = f & small & (dt_abs(q2 - q0) < beta);
  const int a0 = (p2 + 2 * p1 + 2 * p0 + 2 * q0 + q1 + 4) >> 3;
  const int a1 = (p2 + p1 + p0 + q0 + 2) >> 2;
  const int a2 = (2 * p3 + 3 * p2 + p1 + p0 + q0 + 4) >> 3;
  const int aw = (2 * p1 + p0 + q1 + 2) >> 2;
  const int b0 = (q2 + 2 * q1 + 2 * q0 + 2 * p0 + p1 + 4) >> 3;
  const int b1 = (q2 + q1 + q0 + p0 + 2) >> 2;
  const int b2 = (2 * q3 + 3 * q2 + q1 + q0 + p0 + 4) >> 3;
  const int bw = (2 * q1 + q0 + p1 + 2) >> 2;
  p0 = sp ? a0 : (f ? aw : p0);
  p1 = sp ? a1 : p1;
  p2 = sp ? a2 : p2;
  q0 = sq ? b0 : (f ? bw : q0);
  q1 = sq ? b1 : q1;
  q2 = sq ? b2 : q2;
}

DT_FN void chroma_normal(int p1, int& p0, int& q0, int q1, int bs, int alpha, int beta, int tc0) {
  const int dqp = q0 - p0;
  const bool f = (bs != 0) & (dt_abs(dqp) < alpha) & (dt_abs(p1 - p0) < beta) & (dt_abs(q1 - q0) < beta);
  const int tc = tc0 + 1;
  const int delta = dt_clamp((dqp * 4 + (p1 - q1) + 4) >> 3, -tc, tc);
  const int np0 = dt_clamp(p0 + delta, 0, 255), nq0 = dt_clamp(q0 - delta, 0, 255);
  p0 = f ? np0 : p0;
  q0 = f ? nq0 : q0;
}

DT_FN void chroma_strong(int p1, int& p0, int& q0, int q1, int bs, int alpha, int beta) {
  const bool f = (bs != 0) & (dt_abs(p0 - q0) < alpha) & (dt_abs(p1 - p0) < beta) & (dt_abs(q1 - q0) < beta);
  const int np0 = (2 * p1 + p0 + q1 + 2) >> 2, nq0 = (2 * q1 + q0 + p1 + 2) >> 2;
  p0 = f ? np0 : p0;
  q0 = f ? nq0 : q0;
}

// A tile in (shared) memory: TW x TH macroblocks in local macroblock
// positions 1..TW, 1..TH, its margin in column 0 / TW+1 and row 0 / TH+1
// where L, R, T, B say there is one. Luma sample (x, y) of the tile is at
// ly[(10 + y) * sp + 16 + x], chroma byte b of row y at cy[(2 + y) * sp + 16 + b].
constexpr int kDtTop = 10, kDtBottom = 7, kDtTopC = 2, kDtBottomC = 2;

struct DtTile {
  uint8_t *ly, *cy;
  int sp;             // row pitch of both, bytes: 16 * (TW + 1) + 4, an odd word count
  const uint8_t* bs;  // [TH + 2][TW + 2] macroblocks x 32 strengths ([dir][edge][segment])
  uint8_t* save;      // [TH + 2][TW + 2] x 64: e2's q1 q2 of 16 rows (vertical), of 16 columns (horizontal)
  int stride;         // macroblocks per row of bs and save
  int TW, TH;         // the tile's size (a tile at the picture's edge may be smaller)
  int L, R, T, B;     // 1 where the margin exists
};

DT_FN uint32_t dt_word(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }
DT_FN void dt_set_word(uint8_t* p, int a, int b, int c, int d) {
  *reinterpret_cast<uint32_t*>(p) = (uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)c << 16) | ((uint32_t)d << 24);
}
DT_FN int dt_byte(uint32_t w, int k) { return (int)((w >> (8 * k)) & 255u); }

// ---- luma lines ------------------------------------------------------------
// Phase 1: sample row r of macroblock (mx, my); p = its first sample.
DT_FN void dt_luma_v_tail(uint8_t* p, const uint8_t* bs, uint8_t* save, int r, const DbQ& q) {
  const int seg = r >> 2, b2 = bs[8 + seg], b3 = bs[12 + seg];
  const uint32_t w1 = dt_word(p + 4), w2 = dt_word(p + 8), w3 = dt_word(p + 12);
  const int x6 = dt_byte(w1, 2), x7 = dt_byte(w1, 3);
  int x8 = dt_byte(w2, 0), x9 = dt_byte(w2, 1), x10 = dt_byte(w2, 2), x11 = dt_byte(w2, 3);
  int x12 = dt_byte(w3, 0), x13 = dt_byte(w3, 1);
  *reinterpret_cast<uint16_t*>(save + 2 * r) = (uint16_t)(x9 | (x10 << 8));
  if ((b2 | b3) == 0) return;
  x9 = luma_normal_q1(x6, x7, x8, x9, x10, b2, q.al, q.be, tc0_for(b2, q.tcl1, q.tcl2, q.tcl3));
  luma_normal(x9, x10, x11, x12, x13, dt_byte(w3, 2), b3, q.al, q.be, tc0_for(b3, q.tcl1, q.tcl2, q.tcl3));
  dt_set_word(p + 8, x8, x9, x10, x11);
  dt_set_word(p + 12, x12, x13, dt_byte(w3, 2), dt_byte(w3, 3));
}

// Phases 3 and 5: e0, e1, e2 of a row; edges = how many of them (1: e0 only).
DT_FN void dt_luma_v_head(uint8_t* p, const uint8_t* bs, const uint8_t* save, int r, int edges, const DbQ& q) {
  const int seg = r >> 2, b0 = bs[seg], b1 = bs[4 + seg], b2 = bs[8 + seg];
  if ((edges == 1 ? b0 : (b0 | b1 | b2)) == 0) return;
  const uint32_t wl = dt_word(p - 4), w0 = dt_word(p);
  int l1 = dt_byte(wl, 1), l2 = dt_byte(wl, 2), l3 = dt_byte(wl, 3);
  int x0 = dt_byte(w0, 0), x1 = dt_byte(w0, 1), x2 = dt_byte(w0, 2), x3 = dt_byte(w0, 3);
  if (q.is_intra) luma_strong(dt_byte(wl, 0), l1, l2, l3, x0, x1, x2, x3, b0, q.al, q.be);
  else luma_normal(l1, l2, l3, x0, x1, x2, b0, q.al, q.be, tc0_for(b0, q.tcl1, q.tcl2, q.tcl3));
  dt_set_word(p - 4, dt_byte(wl, 0), l1, l2, l3);
  if (edges > 1) {
    const uint32_t w1 = dt_word(p + 4);
    int x4 = dt_byte(w1, 0), x5 = dt_byte(w1, 1), x6 = dt_byte(w1, 2), x7 = dt_byte(w1, 3);
    luma_normal(x1, x2, x3, x4, x5, x6, b1, q.al, q.be, tc0_for(b1, q.tcl1, q.tcl2, q.tcl3));
    const int s = *reinterpret_cast<const uint16_t*>(save + 2 * r);
    int x8 = p[8], x9 = s & 255;
    luma_normal(x5, x6, x7, x8, x9, s >> 8, b2, q.al, q.be, tc0_for(b2, q.tcl1, q.tcl2, q.tcl3));
    dt_set_word(p + 4, x4, x5, x6, x7);
    p[8] = (uint8_t)x8;
  }
  dt_set_word(p, x0, x1, x2, x3);
}

// Phases 2 and 6: sample column c of a macroblock; p = its row 0 (rows 6..14
// are read), save = the macroblock's horizontal half.
DT_FN void dt_luma_h_tail(uint8_t* p, int sp, const uint8_t* bs, uint8_t* save, int c, const DbQ& q) {
  const int seg = c >> 2, b2 = bs[16 + 8 + seg], b3 = bs[16 + 12 + seg];
  int x9 = p[9 * sp], x10 = p[10 * sp];
  *reinterpret_cast<uint16_t*>(save + 2 * c) = (uint16_t)(x9 | (x10 << 8));
  if ((b2 | b3) == 0) return;
  const int x6 = p[6 * sp], x7 = p[7 * sp], x8 = p[8 * sp], x14 = p[14 * sp];
  int x11 = p[11 * sp], x12 = p[12 * sp], x13 = p[13 * sp];
  x9 = luma_normal_q1(x6, x7, x8, x9, x10, b2, q.al, q.be, tc0_for(b2, q.tcl1, q.tcl2, q.tcl3));
  luma_normal(x9, x10, x11, x12, x13, x14, b3, q.al, q.be, tc0_for(b3, q.tcl1, q.tcl2, q.tcl3));
  p[9 * sp] = (uint8_t)x9;
  p[10 * sp] = (uint8_t)x10;
  p[11 * sp] = (uint8_t)x11;
  p[12 * sp] = (uint8_t)x12;
  p[13 * sp] = (uint8_t)x13;
}

// Phase 6 in the margin above the tile: e3's q1 (row 13).
DT_FN void dt_luma_h_row13(uint8_t* p, int sp, const uint8_t* bs, int c, const DbQ& q) {
  const int b3 = bs[16 + 12 + (c >> 2)];
  if (b3 == 0) return;
  p[13 * sp] = (uint8_t)luma_normal_q1(p[10 * sp], p[11 * sp], p[12 * sp], p[13 * sp], p[14 * sp], b3, q.al, q.be,
                                       tc0_for(b3, q.tcl1, q.tcl2, q.tcl3));
}

// Phases 4 and 7: e0, e1, e2 of a column; edges = 1, 2 or 3 of them.
DT_FN void dt_luma_h_head(uint8_t* p, int sp, const uint8_t* bs, const uint8_t* save, int c, int edges, const DbQ& q) {
  const int seg = c >> 2, b0 = bs[16 + seg], b1 = bs[16 + 4 + seg], b2 = bs[16 + 8 + seg];
  if ((edges == 1 ? b0 : (edges == 2 ? (b0 | b1) : (b0 | b1 | b2))) == 0) return;
  const int t0 = p[-4 * sp];
  int t1 = p[-3 * sp], t2 = p[-2 * sp], t3 = p[-1 * sp];
  int x0 = p[0], x1 = p[sp], x2 = p[2 * sp], x3 = p[3 * sp];
  if (b0) {
    if (q.is_intra) {
      luma_strong(t0, t1, t2, t3, x0, x1, x2, x3, b0, q.al, q.be);
      p[-3 * sp] = (uint8_t)t1;
    } else {
      luma_normal(t1, t2, t3, x0, x1, x2, b0, q.al, q.be, tc0_for(b0, q.tcl1, q.tcl2, q.tcl3));
    }
    p[-2 * sp] = (uint8_t)t2;
    p[-1 * sp] = (uint8_t)t3;
  }
  if (edges > 1) {
    int x4 = p[4 * sp], x5 = p[5 * sp], x6 = p[6 * sp];
    luma_normal(x1, x2, x3, x4, x5, x6, b1, q.al, q.be, tc0_for(b1, q.tcl1, q.tcl2, q.tcl3));
    p[3 * sp] = (uint8_t)x3;
    p[4 * sp] = (uint8_t)x4;
    p[5 * sp] = (uint8_t)x5;
    if (edges > 2) {
      const int s = *reinterpret_cast<const uint16_t*>(save + 2 * c);
      int x7 = p[7 * sp], x8 = p[8 * sp], x9 = s & 255;
      luma_normal(x5, x6, x7, x8, x9, s >> 8, b2, q.al, q.be, tc0_for(b2, q.tcl1, q.tcl2, q.tcl3));
      p[6 * sp] = (uint8_t)x6;
      p[7 * sp] = (uint8_t)x7;
      p[8 * sp] = (uint8_t)x8;
    }
  }
  p[0] = (uint8_t)x0;
  p[sp] = (uint8_t)x1;
  p[2 * sp] = (uint8_t)x2;
}

// ---- chroma lines ------------------------------------------------------------
// One edge of one line: p = the sample at q0, st = bytes between samples
// across the edge, b its strength, e0 = a macroblock edge.
DT_FN void dt_chroma(uint8_t* p, int st, int b, bool e0, const DbQ& q) {
  if (b == 0) return;
  const int p1 = p[-2 * st], q1 = p[st];
  int p0 = p[-st], q0 = p[0];
  if (q.is_intra && e0) chroma_strong(p1, p0, q0, q1, b, q.alc, q.bec);
  else chroma_normal(p1, p0, q0, q1, b, q.alc, q.bec, tc0_for(b, q.tcc1, q.tcc2, q.tcc3));
  p[-st] = (uint8_t)p0;
  p[0] = (uint8_t)q0;
}

// ---- phases --------------------------------------------------------------------
// Lines of a phase: dt_luma_lines(t, phase) luma ones, then
// dt_chroma_lines(t, phase) chroma ones; dt_luma_line / dt_chroma_line run
// line i. Neighbouring i are neighbouring rows (vertical edges) or columns
// (horizontal edges).
DT_FN int dt_luma_lines(const DtTile& t, int phase) {
  const int nx = t.TW + t.L;  // macroblock columns of the lines that reach into the left margin
  switch (phase) {
    case 1: return (kDtTop * t.T + 16 * t.TH + kDtBottom * t.B) * nx;
    case 2: return (t.TH + t.T) * 7 * nx;
    case 3: return 7 * (t.TH + t.T) * (t.TW + t.R);
    case 4: return (t.TH + t.B) * 7 * nx;
    case 5: return (9 * t.TH + 3 * t.B) * (t.TW + t.R);
    case 6: return (t.TH + t.T) * 9 * t.TW;
    default: return (t.TH + t.B) * 9 * t.TW;
  }
}

DT_FN void dt_luma_line(const DtTile& t, int phase, int i, const DbQ& q) {
  int mx, my, k;
  if (phase == 1 || phase == 3 || phase == 5) {
    // vertical edges: i = (column of macroblocks, row)
    const int rows = phase == 1 ? kDtTop * t.T + 16 * t.TH + kDtBottom * t.B
                                : (phase == 3 ? 7 * (t.TH + t.T) : 9 * t.TH + 3 * t.B);
    mx = i / rows;
    const int rr = i - mx * rows;
    if (phase == 1) {
      const int r = rr + 16 - kDtTop * t.T;  // row 16 is the tile's first
      mx += 1 - t.L;
      my = r >> 4;
      k = r & 15;
    } else if (phase == 3) {
      mx += 1;
      my = rr / 7;
      k = 9 + rr - 7 * my;
      my += 1 - t.T;
    } else {
      mx += 1;
      my = rr / 9;
      k = rr - 9 * my;
      my += 1;
    }
  } else if (phase == 2 || phase == 4) {
    const int cols = 7 * (t.TW + t.L);
    my = i / cols;
    const int cc = i - my * cols;
    mx = cc / 7;
    k = 9 + cc - 7 * mx;
    mx += 1 - t.L;
    my += phase == 2 ? 1 - t.T : 1;
  } else {
    const int cols = 9 * t.TW;
    my = i / cols;
    const int cc = i - my * cols;
    mx = cc / 9;
    k = cc - 9 * mx;
    mx += 1;
    my += phase == 6 ? 1 - t.T : 1;
  }
  const int mb = my * t.stride + mx;
  const uint8_t* bs = t.bs + 32 * mb;
  uint8_t* save = t.save + 64 * mb;
  uint8_t* p = t.ly + (kDtTop + 16 * (my - 1)) * t.sp + 16 * mx;  // the macroblock's first sample
  if (phase == 1) dt_luma_v_tail(p + k * t.sp, bs, save, k, q);
  else if (phase == 3 || phase == 5) dt_luma_v_head(p + k * t.sp, bs, save, k, mx > t.TW ? 1 : 3, q);
  else if (phase == 6 && my == 0) dt_luma_h_row13(p + k, t.sp, bs, k, q);
  else if (phase == 2 || phase == 6) dt_luma_h_tail(p + k, t.sp, bs, save + 32, k, q);
  else dt_luma_h_head(p + k, t.sp, bs, save + 32, k, my > t.TH ? (phase == 4 ? 2 : 1) : 3, q);
}

DT_FN int dt_chroma_lines(const DtTile& t, int phase) {
  const int nx = t.TW + t.L;
  switch (phase) {
    case 1: return 2 * (kDtTopC * t.T + 8 * t.TH + kDtBottomC * t.B) * t.TW;
    case 2: return t.TH * 12 * nx;
    case 3: return 2 * (2 * t.T + 6 * t.TH) * (t.TW + t.R);
    case 4: return (t.TH + t.B) * 12 * nx;
    case 5: return 2 * 2 * (t.TH + t.B) * (t.TW + t.R);
    case 6: return t.TH * 4 * t.TW;
    default: return (t.TH + t.B) * 4 * t.TW;
  }
}

DT_FN void dt_chroma_line(const DtTile& t, int phase, int i, const DbQ& q) {
  int mx, my, k, pl;
  if (phase == 1 || phase == 3 || phase == 5) {
    // vertical edges: i = (column of macroblocks, plane, row)
    const int rows = phase == 1 ? kDtTopC * t.T + 8 * t.TH + kDtBottomC * t.B
                                : (phase == 3 ? 2 * t.T + 6 * t.TH : 2 * (t.TH + t.B));
    const int j = i / rows;
    const int rr = i - j * rows;
    mx = 1 + (j >> 1);
    pl = j & 1;
    if (phase == 1) {
      const int r8 = rr + 8 - kDtTopC * t.T;
      my = r8 >> 3;
      k = r8 & 7;
    } else if (phase == 3) {
      const int r6 = rr + 6 - 2 * t.T;  // the macroblock above: its rows 6 and 7
      my = r6 / 6;
      k = 2 + r6 - 6 * my;
    } else {
      my = 1 + (rr >> 1);
      k = rr & 1;
    }
    const uint8_t* bs = t.bs + 32 * (my * t.stride + mx) + (phase == 1 ? 8 : 0);
    uint8_t* p = t.cy + (kDtTopC + 8 * (my - 1) + k) * t.sp + 16 * mx + pl + (phase == 1 ? 8 : 0);
    dt_chroma(p, 2, bs[k >> 1], phase != 1, q);
    return;
  }
  if (phase == 2 || phase == 4) {
    const int cols = 12 * (t.TW + t.L);  // bytes 4..15 of each macroblock: columns 2..7 of both planes
    my = i / cols;
    const int cc = i - my * cols;
    mx = cc / 12;
    k = 4 + cc - 12 * mx;
    mx += 1 - t.L;
  } else {
    const int cols = 4 * t.TW;
    my = i / cols;
    const int cc = i - my * cols;
    mx = 1 + (cc >> 2);
    k = cc & 3;
  }
  my += 1;
  const bool e2 = phase == 2 || phase == 6;
  const uint8_t* bs = t.bs + 32 * (my * t.stride + mx) + 16 + (e2 ? 8 : 0);
  uint8_t* p = t.cy + (kDtTopC + 8 * (my - 1) + (e2 ? 4 : 0)) * t.sp + 16 * mx + k;
  dt_chroma(p, t.sp, bs[k >> 2], !e2, q);
}

// ---- boundary strengths --------------------------------------------------------
// The four strengths (one byte a segment) of edge e in direction dir (0
// vertical edges, 1 horizontal). mq, mp: the 16 blocks with coefficients of
// the macroblock and of the neighbour across e0 (bit b = raster block b, the
// blocks of an 8x8 transform all set when any of its levels is nonzero);
// mvd: their vectors differ by 4 or more quarter samples; edge0: e0 lies
// inside the picture; t8: 8x8 transform (no odd luma edge; chroma reads the
// even ones).
DT_FN uint32_t dt_strengths(int dir, int e, uint32_t mq, uint32_t mp, bool mvd, bool edge0, bool intra, bool t8) {
  if (e == 0 && !edge0) return 0u;
  if ((e & 1) && t8) return 0u;
  if (intra) return e == 0 ? 0x04040404u : 0x03030303u;
  uint32_t w = 0;
  for (int k = 0; k < 4; ++k) {
    const int bq = dir == 0 ? k * 4 + e : e * 4 + k;
    uint32_t c = (mq >> bq) & 1u;
    if (e == 0) c |= (mp >> (dir == 0 ? k * 4 + 3 : 12 + k)) & 1u;
    else c |= (mq >> (dir == 0 ? bq - 1 : bq - 4)) & 1u;
    w |= (c ? 2u : (e == 0 && mvd ? 1u : 0u)) << (8 * k);
  }
  return w;
}

// Block mask of a macroblock with the 8x8 transform: a block counts when any
// block of its 8x8 quadrant does.
DT_FN uint32_t dt_mask_t8(uint32_t m) {
  const uint32_t h = (m | (m >> 1)) & 0x5555u;        // pairs, at even columns
  const uint32_t v = (h | (h >> 4)) & 0x0505u;        // quadrants, at their first block
  return v * 0x33u;                                   // spread: +1, +4, +5
}

}  // namespace b200enc
