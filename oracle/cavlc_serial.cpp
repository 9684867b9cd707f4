// cavlc_serial.cpp - CAVLC slice data written the plain way, one syntax
// element after another (H.264 clauses 7.3.4, 9.1, 9.2; the reference's
// A1/src/encoder_h264.c:800-1051, 1120-1340, 3128-3290 and src/cavlc.c:75-801).
// TEST INFRASTRUCTURE ONLY: the GPU coder (csrc/cavlc.cu) is compared with it
// where the reference's own sources are not built. It shares the code tables
// (csrc/cavlc_core.h, the standard's) and nothing else with the GPU coder; its
// block and header writers equal the reference's byte for byte.
#include <cstdlib>
#include <cstring>
#include <vector>

#include "cavlc_core.h"

#define TAB(x) h_##x

namespace {
using namespace b200cavlc;

// ---- bit writer ----------------------------------------------------------------
// MSB first into 32-bit words (word k holds stream bits 32k .. 32k+31, the
// first in bit 31). `cur` holds the nf < 32 pending bits, right-aligned.
struct BitW {
  uint32_t* w;
  uint32_t cap_words, nw, cur, pos;
  int nf;
  bool over;
};

static void bw_init(BitW& b, uint32_t* words, uint32_t cap_words) {
  b.w = words;
  b.cap_words = cap_words;
  b.nw = 0;
  b.cur = 0;
  b.pos = 0;
  b.nf = 0;
  b.over = false;
}

// n <= 32 bits of v (its low n bits).
static void put(BitW& b, int n, uint32_t v) {
  if (n <= 0) return;
  if (n < 32) v &= (1u << n) - 1u;
  const uint64_t t = ((uint64_t)b.cur << n) | v;
  int nf = b.nf + n;
  if (nf >= 32) {
    nf -= 32;
    if (b.nw < b.cap_words) b.w[b.nw] = (uint32_t)(t >> nf);
    else b.over = true;
    ++b.nw;
    b.cur = nf ? (uint32_t)(t & ((1ull << nf) - 1ull)) : 0u;
  } else {
    b.cur = (uint32_t)t;
  }
  b.nf = nf;
  b.pos += (uint32_t)n;
}

static void put_zeros(BitW& b, int n) {
  while (n > 32) {
    put(b, 32, 0u);
    n -= 32;
  }
  put(b, n, 0u);
}

// The pending bits as the last (partial) word; call once at the end.
static void bw_flush(BitW& b) {
  if (b.nf > 0) {
    if (b.nw < b.cap_words) b.w[b.nw] = b.cur << (32 - b.nf);
    else b.over = true;
    ++b.nw;
    b.cur = 0;
    b.nf = 0;
  }
}

static int ilog2(uint32_t v) {  // floor(log2(v)), v > 0
  int r = 0;
  while (v >>= 1) ++r;
  return r;
}

// Exp-Golomb ue(v) (clause 9.1): floor(log2(v + 1)) zeros, then v + 1.
static void put_ue(BitW& b, uint32_t v) {
  const uint64_t c = (uint64_t)v + 1u;
  const int l = c >> 32 ? 32 : ilog2((uint32_t)c);
  put_zeros(b, l);
  if (l + 1 > 32) {
    put(b, 1, (uint32_t)(c >> 32));
    put(b, 32, (uint32_t)c);
  } else {
    put(b, l + 1, (uint32_t)c);
  }
}
static int ue_bits(uint32_t v) { return 2 * ilog2(v + 1u) + 1; }

static void put_se(BitW& b, int v) { put_ue(b, v > 0 ? (uint32_t)(2 * v - 1) : (uint32_t)(-2 * (int64_t)v)); }

// ---- residual block (clause 9.2) -------------------------------------------------
// One level (level_prefix / level_suffix, 9.2.2.1) with the reference's
// escape arithmetic for level_prefix >= 15 (cavlc.c:429-480); returns the
// next suffixLength.
static int put_level(BitW& b, int level, bool first, bool t1_lt3, int sl) {
  int code = level > 0 ? 2 * level - 2 : -2 * level - 1;
  if (first && t1_lt3) code -= 2;
  if (sl == 0) {
    if (code < 14) {
      put_zeros(b, code);
      put(b, 1, 1u);
    } else if (code < 30) {
      put_zeros(b, 14);
      put(b, 1, 1u);
      put(b, 4, (uint32_t)(code - 14));
    } else {
      const uint32_t total = (uint32_t)code + 4066u;
      const int ss = ilog2(total);
      put_zeros(b, ss + 3);
      put(b, 1, 1u);
      put(b, ss, total - (1u << ss));
    }
  } else {
    const int prefix = code >> sl;
    if (prefix < 15) {
      put_zeros(b, prefix);
      put(b, 1, 1u);
      put(b, sl, (uint32_t)(code & ((1 << sl) - 1)));
    } else {
      const uint32_t total = (uint32_t)(code - (15 << sl)) + 4096u;
      const int ss = ilog2(total);
      put_zeros(b, ss + 3);
      put(b, 1, 1u);
      put(b, ss, total - (1u << ss));
    }
  }
  const int a = level < 0 ? -level : level;
  if (sl == 0) sl = 1;
  if (a > (3 << (sl - 1)) && sl < 6) ++sl;
  return sl;
}

// A residual block of max_coeff coefficients in scan order: coeff_token,
// trailing-one signs, levels, total_zeros, run_before. vlc: the nC class
// (0..3) or 4 for chroma DC (nC = -1). Returns TotalCoeff.
static int put_block(BitW& b, const int* sc, int max_coeff, int vlc) {
  uint32_t mask = 0;
  for (int i = 0; i < max_coeff; ++i)
    if (sc[i] != 0) mask |= 1u << i;
  if (!mask) {
    put(b, TAB(ct_len)[vlc][0], TAB(ct_code)[vlc][0]);
    return 0;
  }
  // from the highest frequency down: trailing ones (at most 3, consecutive
  // from the top), the other levels, the zero runs between coefficients
  int tc = 0, t1 = 0, signs = 0, tz = 0, prev = -1;
  int lev[16], run[16];
  for (uint32_t m = mask; m;) {
    const int i = ilog2(m);
    m &= ~(1u << i);
    if (prev >= 0) {
      run[tc - 1] = prev - i - 1;
      tz += prev - i - 1;
    }
    const int v = sc[i];
    if (tc < 3 && (v == 1 || v == -1) && t1 == tc) {
      ++t1;
      signs = (signs << 1) | (v < 0 ? 1 : 0);
    } else {
      lev[tc - t1] = v;
    }
    ++tc;
    prev = i;
  }
  tz += prev;
  const int ti = tc * 4 + t1;
  const int cl = TAB(ct_len)[vlc][ti];
  if (cl > 0) put(b, cl, TAB(ct_code)[vlc][ti]);
  else put_ue(b, (uint32_t)tc);
  if (t1 > 0) put(b, t1, (uint32_t)signs);
  int sl = (tc > 10 && t1 < 3) ? 1 : 0;
  for (int i = 0; i < tc - t1; ++i) sl = put_level(b, lev[i], i == 0, t1 < 3, sl);
  if (tc < max_coeff) {
    if (vlc == 4) {
      if (tz < 4) put(b, TAB(cdtz_len)[tc - 1][tz], TAB(cdtz_code)[tc - 1][tz]);
      else put_ue(b, (uint32_t)tz);
    } else {
      const int l = (tc - 1 < 15 && tz < 16) ? TAB(tz_len)[tc - 1][tz] : 0;
      if (l > 0) put(b, l, TAB(tz_code)[tc - 1][tz]);
      else put_ue(b, (uint32_t)tz);
    }
  }
  int zl = tz;
  for (int i = 1; i < tc && zl > 0; ++i) {
    const int r = run[i - 1];
    const int zi = zl <= 6 ? zl - 1 : 6;
    const int l = r < 16 ? TAB(run_len)[zi][r] : 0;
    if (l > 0) put(b, l, TAB(run_code)[zi][r]);
    else put_ue(b, (uint32_t)r);
    zl -= r;
  }
  return tc;
}

static int nc_class(int nc) { return nc < 2 ? 0 : (nc < 4 ? 1 : (nc < 8 ? 2 : 3)); }

// A 4x4 block stored in raster positions, zig-zag scanned: all 16
// coefficients (ac = false) or positions 1..15 (ac = true).
static int put_4x4(BitW& b, const int16_t* blk, bool ac, int nc) {
  int sc[16];
  const int n = ac ? 15 : 16;
  for (int i = 0; i < n; ++i) sc[i] = blk[TAB(zigzag)[i + (ac ? 1 : 0)]];
  return put_block(b, sc, n, nc_class(nc));
}

// Macroblock headers (clause 7.3.5): I16x16 with mb_type 1 + mode +
// 4 * cbp_chroma + 12 * (cbp_luma != 0), intra_chroma_pred_mode and
// mb_qp_delta 0; P_L0_16x16 with its vector difference, the inter
// coded_block_pattern codeNum and mb_qp_delta 0 when cbp != 0.
static void put_i16_header(BitW& b, int mode, int chroma_mode, int cbp_chroma, int cbp_luma_flag) {
  put_ue(b, (uint32_t)(1 + mode + 4 * cbp_chroma + 12 * cbp_luma_flag));
  put_ue(b, (uint32_t)chroma_mode);
  put_se(b, 0);
}
// t8: the macroblock's luma uses the 8x8 transform (transform_size_8x8_flag,
// present when the luma pattern is nonzero, 7.3.5).
// t8_mode: the picture parameter set has transform_8x8_mode_flag, so every
// macroblock with a coded luma block carries transform_size_8x8_flag (t8,
// 7.3.5: 0 for a macroblock coded with 4x4 transforms).
static void put_p16_header(BitW& b, int mvd_x, int mvd_y, int cbp, int t8_mode = 0, int t8 = 0) {
  put_ue(b, 0u);
  put_se(b, mvd_x);
  put_se(b, mvd_y);
  put_ue(b, TAB(cbp_code)[cbp]);
  if (t8_mode && (cbp & 15)) put(b, 1, t8 ? 1u : 0u);
  if (cbp > 0) put_se(b, 0);
}


const int8_t X4[16] = {0, 1, 0, 1, 2, 3, 2, 3, 0, 1, 0, 1, 2, 3, 2, 3};
const int8_t Y4[16] = {0, 0, 1, 1, 0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 3, 3};
int spec(int y4, int x4) { return ((y4 >> 1) << 3) | ((x4 >> 1) << 2) | ((y4 & 1) << 1) | (x4 & 1); }
int min3(int a, int b, int c) { return a < b ? (a < c ? a : c) : (b < c ? b : c); }
int max3(int a, int b, int c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }

const int LS[6] = {160, 176, 208, 224, 256, 288};  // 16 * V(rem, 0)
int chroma_qp(int q) {
  static const int t[22] = {29, 30, 31, 32, 32, 33, 34, 34, 35, 35, 36, 36, 37, 37, 37, 38, 38, 38, 39, 39, 39, 39};
  return q < 30 ? q : t[q - 30];
}
int quant_dc(int v, int qp) {  // encoder_h264.c:653-709
  const int per = qp / 6, ls = LS[qp % 6], a = v < 0 ? -v : v;
  int num, den;
  if (per >= 5) { num = a; den = ls << (per - 5); }
  else { num = a << (5 - per); den = ls; }
  const int l = (num + den / 2) / den;
  return v < 0 ? -l : l;
}

struct Pic {
  int mbw, mbh, qp, intra, ns, quality, t8;
  const int16_t* levels;
  const int32_t* dc;
  const uint32_t* nz;
  const uint32_t* pm;
  const int32_t* mv;  // [mbs][4]
  const uint8_t* t8f;
};

bool nb(const Pic& p, int x, int y, int dx, int dy, int start, int* n) {
  if (x + dx < 0 || y + dy < 0 || x + dx >= p.mbw) return false;
  *n = (y + dy) * p.mbw + x + dx;
  return *n >= start;
}
void pred(const Pic& p, int x, int y, int start, int* px, int* py) {
  int na, nbb, nc;
  const bool a = nb(p, x, y, -1, 0, start, &na), b = nb(p, x, y, 0, -1, start, &nbb);
  bool c = nb(p, x, y, 1, -1, start, &nc);
  if (!c) c = nb(p, x, y, -1, -1, start, &nc);
  if (a && !b && !c) { *px = p.mv[4 * na]; *py = p.mv[4 * na + 1]; return; }
  int v[2];
  for (int k = 0; k < 2; ++k) {
    const int va = a ? p.mv[4 * na + k] : 0, vb = b ? p.mv[4 * nbb + k] : 0, vc = c ? p.mv[4 * nc + k] : 0;
    v[k] = va + vb + vc - min3(va, vb, vc) - max3(va, vb, vc);
  }
  *px = v[0]; *py = v[1];
}
void cdc(const int32_t* d, int o[4]) {
  o[0] = d[0] + d[1] + d[2] + d[3]; o[1] = d[0] - d[1] + d[2] - d[3];
  o[2] = d[0] + d[1] - d[2] - d[3]; o[3] = d[0] - d[1] - d[2] + d[3];
}
int pop(uint32_t v) { return __builtin_popcount(v); }

struct Mb { int skip, cbp_l, cbp_c; uint8_t tc[24]; };

Mb info(const Pic& p, int mb, int start) {
  Mb m{};
  const uint32_t* z = p.nz + 24 * (size_t)mb;
  const int32_t* d = p.dc + 24 * (size_t)mb;
  const int x = mb % p.mbw, y = mb / p.mbw, qc = chroma_qp(p.qp);
  int c[8];
  cdc(d + 16, c); cdc(d + 20, c + 4);
  bool raw = false, cq = false, cac = false, zl = true;
  for (int k = 0; k < 8; ++k) { raw |= c[k] != 0; cq |= quant_dc(c[k], qc) != 0; }
  for (int k = 16; k < 24; ++k) cac |= (z[k] & 0xfffe) != 0;
  m.cbp_c = cac ? 2 : cq;
  if (p.intra) {
    for (int k = 0; k < 16; ++k) m.cbp_l |= (z[k] & 0xfffe) != 0;
    for (int b = 0; b < 16; ++b) m.tc[b] = m.cbp_l ? pop(z[Y4[b] * 4 + X4[b]] & 0xfffe) : 0;
  } else {
    for (int k = 0; k < 16; ++k) zl &= (z[k] & 0xffff) == 0;
    bool zc = !raw && !cac;
    if (p.quality >= 5 && zl && !zc && abs(p.dc[mb * 2]) <= 1 && abs(p.dc[mb * 2 + 1]) <= 1) zc = true;
    int px = 0, py = 0, na, nbb;
    const bool a = nb(p, x, y, -1, 0, start, &na), b = nb(p, x, y, 0, -1, start, &nbb);
    if (a && b && (p.mv[4 * na] || p.mv[4 * na + 1]) && (p.mv[4 * nbb] || p.mv[4 * nbb + 1])) pred(p, x, y, start, &px, &py);
    if (zl && zc && p.mv[4 * mb] == px && p.mv[4 * mb + 1] == py) { m.skip = 1; m.cbp_c = 0; return m; }
    for (int b2 = 0; b2 < 16; ++b2)
      if (z[Y4[b2] * 4 + X4[b2]] & 0xffff) m.cbp_l |= 1 << (b2 >> 2);
    for (int b2 = 0; b2 < 16; ++b2) m.tc[b2] = pop(z[Y4[b2] * 4 + X4[b2]] & 0xffff);
  }
  for (int k = 0; k < 8; ++k) m.tc[16 + k] = m.cbp_c == 2 ? pop(z[16 + k] & 0xfffe) : 0;
  return m;
}
int nc_of(int a, int b) { return a >= 0 && b >= 0 ? (a + b + 1) >> 1 : (a >= 0 ? a : (b >= 0 ? b : 0)); }

void block16(BitW& w, const int16_t* lv, const uint8_t* scan, int first, int step, int n, int nc) {
  int sc[16];
  for (int i = 0; i < n; ++i) sc[i] = lv[scan[first + step * i]];
  put_block(w, sc, n, nc_class(nc));
}

}  // namespace

// zz8: the 8x8 frame zig-zag scan (raster positions). Slices back to back in
// out, their byte counts in bytes; header: [ns][16], header_bits: [ns].
extern "C" void orc_cavlc_slices(int mbw, int mbh, int qp, int intra, int ns, int quality, int t8, const int16_t* levels,
                                 const int32_t* dc, const uint32_t* nz, const uint32_t* pm, const int32_t* mv,
                                 const uint8_t* t8f, const uint8_t* zz8, const uint8_t* header, const int* header_bits,
                                 uint8_t* out, int64_t* bytes) {
  const Pic p{mbw, mbh, qp, intra, ns, quality, t8, levels, dc, nz, pm, mv, t8f};
  const int mbs = mbw * mbh;
  std::vector<uint32_t> words((size_t)mbs * 800 + 64);
  int64_t at = 0;
  for (int s = 0; s < ns; ++s) {
    const int m0 = (int)((int64_t)s * mbs / ns), m1 = (int)((int64_t)(s + 1) * mbs / ns);
    BitW w;
    bw_init(w, words.data(), (uint32_t)words.size());
    for (int k = 0; k < header_bits[s]; ++k) put(w, 1, (header[16 * s + (k >> 3)] >> (7 - (k & 7))) & 1u);
    std::vector<Mb> mi((size_t)mbs);
    for (int mb = m0; mb < m1; ++mb) mi[mb] = info(p, mb, m0);
    uint32_t run = 0;
    for (int mb = m0; mb < m1; ++mb) {
      const Mb& m = mi[mb];
      if (m.skip) { ++run; continue; }
      const int x = mb % mbw, y = mb / mbw;
      int nl, nt;
      const bool left = nb(p, x, y, -1, 0, m0, &nl), top = nb(p, x, y, 0, -1, m0, &nt);
      const int16_t* lv = levels + (size_t)mb * 384;
      const int32_t* d = dc + (size_t)mb * 24;
      const bool use8 = t8 && !intra && (!t8f || t8f[mb]);
      auto luma_nc = [&](int b) {
        const int a4 = X4[b], b4 = Y4[b];
        const int na = a4 ? m.tc[spec(b4, a4 - 1)] : (left ? mi[nl].tc[spec(b4, 3)] : -1);
        const int nt4 = b4 ? m.tc[spec(b4 - 1, a4)] : (top ? mi[nt].tc[spec(3, a4)] : -1);
        return nc_of(na, nt4);
      };
      if (!intra) {
        put_ue(w, run);
        run = 0;
        int px, py;
        pred(p, x, y, m0, &px, &py);
        put_p16_header(w, mv[4 * mb] - px, mv[4 * mb + 1] - py, m.cbp_l | (m.cbp_c << 4), t8, use8);
      } else {
        int md = pm[mb] & 3, cm = (pm[mb] >> 2) & 3;
        if (!top && !left) md = 2, cm = 0;
        else if (!top) md = (md == 0 || md == 3) ? 1 : md, cm = (cm == 2 || cm == 3) ? 1 : cm;
        else if (!left) md = (md == 1 || md == 3) ? 0 : md, cm = (cm == 1 || cm == 3) ? 2 : cm;
        put_i16_header(w, md, cm, m.cbp_c, m.cbp_l);
        // luma DC: 2-D Hadamard (rows h: ++++ ++-- +--+ +-+-), (sum + 1) >> 1, quantised
        static const int H[4][4] = {{1, 1, 1, 1}, {1, 1, -1, -1}, {1, -1, -1, 1}, {1, -1, 1, -1}};
        int16_t q[16];
        for (int r = 0; r < 4; ++r)
          for (int c = 0; c < 4; ++c) {
            int sum = 0;
            for (int i = 0; i < 4; ++i)
              for (int j = 0; j < 4; ++j) sum += H[r][i] * H[c][j] * d[4 * i + j];
            q[4 * r + c] = (int16_t)quant_dc((sum + 1) >> 1, qp);
          }
        block16(w, q, h_zigzag, 0, 1, 16, luma_nc(0));
      }
      for (int b = 0; b < 16; ++b) {
        if (!(intra ? m.cbp_l : (m.cbp_l >> (b >> 2)) & 1)) continue;
        if (use8) block16(w, lv + 64 * (b >> 2), zz8, b & 3, 4, 16, luma_nc(b));
        else block16(w, lv + 16 * (Y4[b] * 4 + X4[b]), h_zigzag, intra, 1, intra ? 15 : 16, luma_nc(b));
      }
      if (m.cbp_c >= 1)
        for (int pl = 0; pl < 2; ++pl) {
          int c[4];
          cdc(d + 16 + 4 * pl, c);
          for (int k = 0; k < 4; ++k) c[k] = quant_dc(c[k], chroma_qp(qp));
          put_block(w, c, 4, 4);
        }
      if (m.cbp_c == 2)
        for (int b = 0; b < 8; ++b) {
          const int o = 16 + (b & 4), k = b & 3, x2 = k & 1, y2 = k >> 1;
          const int na = x2 ? m.tc[o + 2 * y2] : (left ? mi[nl].tc[o + 2 * y2 + 1] : -1);
          const int nt2 = y2 ? m.tc[o + x2] : (top ? mi[nt].tc[o + 2 + x2] : -1);
          block16(w, lv + 16 * (16 + b), h_zigzag, 1, 1, 15, nc_of(na, nt2));
        }
    }
    if (run) put_ue(w, run);
    put(w, 1, 1u);
    bw_flush(w);
    bytes[s] = (w.pos + 7) >> 3;
    for (int64_t k = 0; k < bytes[s]; ++k) out[at + k] = (uint8_t)(words[k >> 2] >> (24 - 8 * (k & 3)));
    at += bytes[s];
  }
}
