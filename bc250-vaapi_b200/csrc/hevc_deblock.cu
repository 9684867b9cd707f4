// hevc_deblock.cu - HEVC deblocking (H.265 clause 8.7.2) of one 4:2:0
// picture, in place, in two launches.
//
// Reproduces the deblocking stages of the reference decoder's loop filter
// (approach1-compute-encoder/src/hevc_filter.c:449-490 over
// hevc_filter_template.c:48-420): every vertical edge of the picture first,
// then every horizontal edge over the vertically filtered picture; luma on
// the 8x8 edge grid with the strong/weak decision of the first and last
// line of each 4-line segment, chroma on the 16-luma-sample grid where the
// boundary strength is 2; per-slice beta/tC offsets and switches, tile and
// slice boundaries, lossless (no-filter) blocks, QpY averaged across the
// edge, 8- and 10-bit samples.
//
// Two launches, as the clause orders it: all vertical edges, then all
// horizontal edges. Inside a pass the edges are independent: they sit on
// the 8-sample grid and a luma filter reads 4 and writes 3 samples either
// side (chroma: 8 chroma samples apart, reads 2, writes 1), so no edge reads
// or writes a sample another edge of the same pass writes: filtered in place in
// global memory, no tiles, no halos. (A single launch over tiles with halos
// would need the neighbours' samples as the vertical pass left them, which
// an in-place neighbour may already have overwritten.)
//
// A warp takes 32 4-line segments along a row. First each lane decides one of
// them (slice and tile rules, QP, boundary strength from the motion and cbf
// maps); then, eight segments at a time and only where one of the eight is
// filtered, four lanes filter a segment's lines, the decision and the first and
// last line's figures coming by shuffles. Bound by instructions issued and the
// latency of the maps' chained reads. A picture that does not fill the chip with
// such warps pays their four rounds one after another, so there (kHdbFew) a warp
// takes eight segments, each of a segment's four lanes decides for itself and has its
// samples on the way meanwhile. Several pictures of each size in turn, 8 / 10 bits, us,
// with eight segments a warp and with 32: 1280x720 9.6 and 17.8, 1920x1080 16.2 / 17.5 and
// 20.3 / 22.4, 2560x1440 22.7 / 24.1 and 22.5 / 24.8, 3840x2160 42.5 / 45.2 and 36.9 / 40.1.
// (Eight segments a warp without early launches, a load per sample: 13.9, 18.4 / 20.5,
// 24.8 / 26.7, 41.4 / 45.1.)
#include <cstddef>
#include <type_traits>

#include "b200enc_internal.h"
#include "common.cuh"

// The layouts the Python bindings mirror (b200enc/__init__.py).
static_assert(sizeof(b200enc_hevc_mvf_t) == 20, "mvf record");
static_assert(sizeof(b200enc_hevc_slice_filter_t) == 8, "slice filter record");
static_assert(sizeof(b200enc_hevc_deblock_t) == 168 && offsetof(b200enc_hevc_deblock_t, edges) == 64 &&
                  offsetof(b200enc_hevc_deblock_t, qp_y) == 104 && offsetof(b200enc_hevc_deblock_t, tile_of_ctb) == 144,
              "parameter block");

namespace b200enc {

// Table 8-12 (beta' by Q = 0..51, tC' by Q = 0..53) and Table 8-10 (QpC for
// qPi = 30..43), as clause 8.7.2.5.3 / 8.7.2.5.5 and 8.6.1 give them.
__constant__ uint8_t kHdbBeta[52] = {0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  0,  6,  7,
                                     8,  9,  10, 11, 12, 13, 14, 15, 16, 17, 18, 20, 22, 24, 26, 28, 30, 32,
                                     34, 36, 38, 40, 42, 44, 46, 48, 50, 52, 54, 56, 58, 60, 62, 64};
__constant__ uint8_t kHdbTc[54] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1,  1,  1,  1,  1,  1,  1,  1,  1,
                                   2, 2, 2, 2, 3, 3, 3, 3, 4, 4, 4, 5, 5, 6, 6, 7, 8, 9, 10, 11, 13, 14, 16, 18, 20, 22, 24};
__constant__ uint8_t kHdbQpC[14] = {29, 30, 31, 32, 33, 33, 34, 34, 35, 35, 36, 36, 37, 37};

constexpr int kHdbThreads = 256;
// Segments of one direction up to which a warp takes eight instead of 32: the two
// forms take the same time at 2560x1440 (115,200).
constexpr int kHdbFew = 110000;

__device__ __forceinline__ int hdb_clip(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// What one edge cell asks once for both its segments (hevc_filter_template.c
// :266-296): tile and slice boundaries, the q-side slice's settings, the
// lossless sides, the averaged QpY and beta.
struct HdbEdge {
  bool on, keep_p, keep_q;
  int qp, beta, tc_offset;
};

__device__ __forceinline__ int hdb_ctb(const b200enc_hevc_deblock_t& p, int x, int y, int ctb_w) {
  return (y >> p.log2_ctb) * ctb_w + (x >> p.log2_ctb);
}

__device__ __forceinline__ HdbEdge hdb_edge(const b200enc_hevc_deblock_t& p, int x, int y, bool vertical, int ctb_w) {
  // Every map read is issued before any of them is looked at (one round
  // trip instead of a chain); only the slice settings wait for the slice id.
  const int xp = vertical ? x - 1 : x, yp = vertical ? y : y - 1;
  const int cq = hdb_ctb(p, x, y, ctb_w), cp = hdb_ctb(p, xp, yp, ctb_w);
  const int l = p.log2_min_cb, mcw = p.width >> l;
  const int bq = (y >> l) * mcw + (x >> l), bp = (yp >> l) * mcw + (xp >> l);
  const int tq = p.tile_of_ctb ? __ldg(p.tile_of_ctb + cq) : 0, tp = p.tile_of_ctb ? __ldg(p.tile_of_ctb + cp) : 0;
  const int sq = p.slice_of_ctb ? __ldg(p.slice_of_ctb + cq) : 0, sp = p.slice_of_ctb ? __ldg(p.slice_of_ctb + cp) : 0;
  const bool nq = p.no_filter && __ldg(p.no_filter + bq) != 0, np = p.no_filter && __ldg(p.no_filter + bp) != 0;
  const int qq = __ldg(p.qp_y + bq), qp = __ldg(p.qp_y + bp);
  HdbEdge r;
  r.on = false;
  if (!p.loop_filter_across_tiles && tp != tq) return r;
  if (sq < 0 || !p.slice_filter || sq >= p.n_slice_filter) return r;
  const b200enc_hevc_slice_filter_t f = p.slice_filter[sq];
  if (f.disabled) return r;
  if (!f.across_slices && sp != sq) return r;
  r.keep_p = np;
  r.keep_q = nq;
  if (np && nq) return r;
  r.qp = (qq + qp + 1) >> 1;
  r.beta = (int)kHdbBeta[hdb_clip(r.qp + f.beta_offset, 0, 51)] << (p.bit_depth_luma - 8);
  r.tc_offset = f.tc_offset;
  r.on = true;
  return r;
}

// One prediction unit's motion in registers (the list index is a run-time
// value, so the arrays are selected from rather than indexed).
struct HdbMv {
  int x[2], y[2], poc[2], flag;
};

__device__ __forceinline__ HdbMv hdb_mv(const b200enc_hevc_mvf_t* m) {
  // 20-byte entries are 4-byte aligned only: five word loads
  const int* w = reinterpret_cast<const int*>(m);
  const int m0 = __ldg(w), m1 = __ldg(w + 1);  // mv[0][x, y], mv[1][x, y]
  HdbMv r;
  r.x[0] = (int16_t)(m0 & 0xffff);
  r.y[0] = (int16_t)(m0 >> 16);
  r.x[1] = (int16_t)(m1 & 0xffff);
  r.y[1] = (int16_t)(m1 >> 16);
  r.poc[0] = __ldg(w + 2);
  r.poc[1] = __ldg(w + 3);
  r.flag = __ldg(w + 4) & 0xff;
  return r;
}

__device__ __forceinline__ bool hdb_differ(const HdbMv& a, int la, const HdbMv& b, int lb) {
  const int ax = la ? a.x[1] : a.x[0], ay = la ? a.y[1] : a.y[0];
  const int bx = lb ? b.x[1] : b.x[0], by = lb ? b.y[1] : b.y[0];
  return abs(ax - bx) >= 4 || abs(ay - by) >= 4;
}

// Boundary strength of one segment, clause 8.7.2.4
// (hevc_filter_template.c:207-259).
__device__ int hdb_strength(const b200enc_hevc_deblock_t& p, int xp, int yp, int xq, int yq, bool transform_edge) {
  if (!p.mvf) return 2;
  const int ip = (yp >> 2) * p.min_pu_width + (xp >> 2), iq = (yq >> 2) * p.min_pu_width + (xq >> 2);
  const HdbMv P = hdb_mv(p.mvf + ip), Q = hdb_mv(p.mvf + iq);
  if (!P.flag || !Q.flag) return 2;
  if (transform_edge && p.cbf && (__ldg(p.cbf + ip) || __ldg(p.cbf + iq))) return 1;
  const int np = P.flag == 3 ? 2 : 1, nq = Q.flag == 3 ? 2 : 1;
  if (np != nq) return 1;
  if (np == 1) {
    const int lp = (P.flag & 1) ? 0 : 1, lq = (Q.flag & 1) ? 0 : 1;
    if ((lp ? P.poc[1] : P.poc[0]) != (lq ? Q.poc[1] : Q.poc[0])) return 1;
    return hdb_differ(P, lp, Q, lq) ? 1 : 0;
  }
  const bool same = P.poc[0] == Q.poc[0] && P.poc[1] == Q.poc[1];
  const bool crossed = P.poc[0] == Q.poc[1] && P.poc[1] == Q.poc[0];
  if (!same && !crossed) return 1;
  if (P.poc[0] != P.poc[1]) {
    if (same) return (hdb_differ(P, 0, Q, 0) || hdb_differ(P, 1, Q, 1)) ? 1 : 0;
    return (hdb_differ(P, 0, Q, 1) || hdb_differ(P, 1, Q, 0)) ? 1 : 0;
  }
  const bool straight = !(hdb_differ(P, 0, Q, 0) || hdb_differ(P, 1, Q, 1));
  const bool swapped = !(hdb_differ(P, 0, Q, 1) || hdb_differ(P, 1, Q, 0));
  return (straight || swapped) ? 0 : 1;
}

// One line of a 4-line luma segment across an edge. `q` points at its q0 and `fw`
// steps from p to q. VEC: the line lies along a row of aligned samples, and its
// eight are read and written as two words (the outer two, which no edge of the
// pass changes, with their own values).
template <typename T, bool VEC>
struct HdbLine {
  using Half = typename std::conditional<sizeof(T) == 1, uint32_t, uint2>::type;  // four samples
  int p3 = 0, p2 = 0, p1 = 0, p0 = 0, q0 = 0, q1 = 0, q2 = 0, q3 = 0;
  __device__ __forceinline__ void load(const T* q, int fw) {
    if (VEC) {
      alignas(8) T v[8];
      *reinterpret_cast<Half*>(v) = *reinterpret_cast<const Half*>(q - 4);
      *reinterpret_cast<Half*>(v + 4) = *reinterpret_cast<const Half*>(q);
      p3 = v[0], p2 = v[1], p1 = v[2], p0 = v[3], q0 = v[4], q1 = v[5], q2 = v[6], q3 = v[7];
    } else {
      p3 = q[-4 * fw];
      p2 = q[-3 * fw];
      p1 = q[-2 * fw];
      p0 = q[-fw];
      q0 = q[0];
      q1 = q[fw];
      q2 = q[2 * fw];
      q3 = q[3 * fw];
    }
  }
};

// Filters a loaded line (clauses 8.7.2.5.3, 8.7.2.5.6, 8.7.2.5.7;
// hevc_filter_template.c:48-140). The four lanes 4k..4k+3 of a warp hold a
// segment's four lines; the decisions read lines 0 and 3 only, so those lanes'
// figures are shuffled to the other two. Every lane of the warp calls it (the
// shuffles); `act` says that the segment is filtered.
template <typename T, bool VEC>
__device__ __forceinline__ void hdb_luma_filter(const HdbLine<T, VEC>& s, T* q, int fw, bool act, int beta, int tc,
                                                bool keep_p, bool keep_q, int maxv) {
  using Half = typename HdbLine<T, VEC>::Half;
  const int p3 = s.p3, p2 = s.p2, p1 = s.p1, p0 = s.p0, q0 = s.q0, q1 = s.q1, q2 = s.q2, q3 = s.q3;
  const int dp = abs(p2 - 2 * p1 + p0), dq = abs(q2 - 2 * q1 + q0);
  const int flat = abs(p3 - p0) + abs(q0 - q3), step = abs(p0 - q0);
  const int l0 = (threadIdx.x & 31) & ~3, l3 = l0 + 3;
  const int dp0 = __shfl_sync(0xffffffffu, dp, l0), dp3 = __shfl_sync(0xffffffffu, dp, l3);
  const int dq0 = __shfl_sync(0xffffffffu, dq, l0), dq3 = __shfl_sync(0xffffffffu, dq, l3);
  const int fl0 = __shfl_sync(0xffffffffu, flat, l0), fl3 = __shfl_sync(0xffffffffu, flat, l3);
  const int st0 = __shfl_sync(0xffffffffu, step, l0), st3 = __shfl_sync(0xffffffffu, step, l3);
  if (!act) return;
  const int dpq0 = dp0 + dq0, dpq3 = dp3 + dq3;
  if (dpq0 + dpq3 >= beta) return;
  const int thr = (5 * tc + 1) >> 1;
  const bool strong = 2 * dpq0 < (beta >> 2) && fl0 < (beta >> 3) && st0 < thr && 2 * dpq3 < (beta >> 2) &&
                      fl3 < (beta >> 3) && st3 < thr;
  int o[6] = {p2, p1, p0, q0, q1, q2};
  bool wp = !keep_p, wq = !keep_q, outer = true;  // outer: p2 and q2 change too (in the strong filter)
  if (strong) {
    o[0] = hdb_clip((2 * p3 + 3 * p2 + p1 + p0 + q0 + 4) >> 3, p2 - 2 * tc, p2 + 2 * tc);
    o[1] = hdb_clip((p2 + p1 + p0 + q0 + 2) >> 2, p1 - 2 * tc, p1 + 2 * tc);
    o[2] = hdb_clip((p2 + 2 * p1 + 2 * p0 + 2 * q0 + q1 + 4) >> 3, p0 - 2 * tc, p0 + 2 * tc);
    o[3] = hdb_clip((p1 + 2 * p0 + 2 * q0 + 2 * q1 + q2 + 4) >> 3, q0 - 2 * tc, q0 + 2 * tc);
    o[4] = hdb_clip((p0 + q0 + q1 + q2 + 2) >> 2, q1 - 2 * tc, q1 + 2 * tc);
    o[5] = hdb_clip((p0 + q0 + q1 + 3 * q2 + 2 * q3 + 4) >> 3, q2 - 2 * tc, q2 + 2 * tc);
  } else {
    int delta = (9 * (q0 - p0) - 3 * (q1 - p1) + 8) >> 4;
    if (abs(delta) >= tc * 10) return;
    delta = hdb_clip(delta, -tc, tc);
    const int side = (beta + (beta >> 1)) >> 3;
    outer = false;
    o[2] = hdb_clip(p0 + delta, 0, maxv);
    o[3] = hdb_clip(q0 - delta, 0, maxv);
    if (dp0 + dp3 < side)
      o[1] = hdb_clip(p1 + hdb_clip((((p2 + p0 + 1) >> 1) - p1 + delta) >> 1, -(tc >> 1), tc >> 1), 0, maxv);
    if (dq0 + dq3 < side)
      o[4] = hdb_clip(q1 + hdb_clip((((q2 + q0 + 1) >> 1) - q1 - delta) >> 1, -(tc >> 1), tc >> 1), 0, maxv);
  }
  if (VEC) {
    alignas(8) T v[8] = {(T)p3, (T)o[0], (T)o[1], (T)o[2], (T)o[3], (T)o[4], (T)o[5], (T)q3};
    if (wp) *reinterpret_cast<Half*>(q - 4) = *reinterpret_cast<const Half*>(v);
    if (wq) *reinterpret_cast<Half*>(q) = *reinterpret_cast<const Half*>(v + 4);
    return;
  }
  if (wp) {
    if (outer) q[-3 * fw] = (T)o[0];
    q[-2 * fw] = (T)o[1];
    q[-fw] = (T)o[2];
  }
  if (wq) {
    q[0] = (T)o[3];
    q[fw] = (T)o[4];
    if (outer) q[2 * fw] = (T)o[5];
  }
}

// One line of a chroma segment (clause 8.7.2.5.5; hevc_filter_template.c
// :149-162): no decision, so nothing crosses lanes.
template <typename T>
__device__ __forceinline__ void hdb_chroma_line(T* q, int fw, int tc, bool keep_p, bool keep_q, int maxv) {
  const int p1 = q[-2 * fw], p0 = q[-fw], q0 = q[0], q1 = q[fw];
  const int delta = hdb_clip((((q0 - p0) * 4) + p1 - q1 + 4) >> 3, -tc, tc);
  if (!keep_p) q[-fw] = (T)hdb_clip(p0 + delta, 0, maxv);
  if (!keep_q) q[0] = (T)hdb_clip(q0 - delta, 0, maxv);
}

// tC of one chroma plane, hevc_filter_template.c:176-181 and :322-329.
__device__ __forceinline__ int hdb_tc_chroma(const b200enc_hevc_deblock_t& p, const HdbEdge& ed, int plane) {
  const int qpi = hdb_clip(ed.qp + (plane == 0 ? p.cb_qp_offset : p.cr_qp_offset), 0, 57);
  const int qpc = qpi < 30 ? qpi : (qpi > 43 ? qpi - 6 : (int)kHdbQpC[qpi - 30]);
  return (int)kHdbTc[hdb_clip(qpc + 2 + ed.tc_offset, 0, 53)] << (p.bit_depth_chroma - 8);
}

// What a segment's lines need (x, y its first sample): strength, kept sides, tC and
// beta in `luma`, 0 where it is not filtered, and the chroma planes' tC. Chroma goes
// with the first segment of a cell on the 16-sample grid, one chroma line per lane
// (hevc_filter_template.c:298-335).
struct HdbSegment {
  uint32_t luma = 0, chroma = 0;
};
template <bool VERT>
__device__ __forceinline__ HdbSegment hdb_decide(const b200enc_hevc_deblock_t& p, int x, int y) {
  HdbSegment s;
  const int e = __ldg(p.edges + (size_t)(y >> 3) * p.edges_stride + (x >> 3));
  const int ctb_w = (p.width + (1 << p.log2_ctb) - 1) >> p.log2_ctb;
  const HdbEdge ed = hdb_edge(p, VERT ? x : x & ~7, VERT ? y & ~7 : y, VERT, ctb_w);
  const int b = hdb_strength(p, VERT ? x - 1 : x, VERT ? y : y - 1, x, y, (e & (VERT ? 4 : 8)) != 0);
  const int bs = ((e & (VERT ? 1 : 2)) && ed.on) ? b : 0;
  if (bs) {
    const int tc = (int)kHdbTc[hdb_clip(ed.qp + 2 * (bs - 1) + ed.tc_offset, 0, 53)] << (p.bit_depth_luma - 8);
    s.luma = bs | (ed.keep_p ? 4u : 0u) | (ed.keep_q ? 8u : 0u) | (uint32_t)tc << 4 | (uint32_t)ed.beta << 11;
    if (bs == 2 && !((VERT ? x : y) & 15) && !((VERT ? y : x) & 7))
      s.chroma = (uint32_t)hdb_tc_chroma(p, ed, 0) | (uint32_t)hdb_tc_chroma(p, ed, 1) << 8;
  }
  return s;
}

// One direction's edges: 4-row segments of vertical ones (VERT; a cell column
// each) or 4-column segments of horizontal ones (a cell row each). ROUNDS: how many
// times eight segments a warp takes; with one round every lane decides for itself,
// its samples on the way meanwhile. VEC: see HdbLine.
// Five CTAs per SM (48 registers; with 58 the 10-bit horizontal pass loses a fifth
// of its warps).
template <typename T, bool VERT, bool VEC, int ROUNDS>
__global__ void __launch_bounds__(kHdbThreads, 5) hevc_deblock_kernel(const __grid_constant__ b200enc_hevc_deblock_t p) {
  pdl_wait();
  const int per_row = VERT ? p.width >> 3 : p.width >> 2, rows = VERT ? p.height >> 2 : p.height >> 3;
  const int lane = threadIdx.x & 31, line = lane & 3;
  const int maxv = (int)(sizeof(T) == 1 ? 255 : 1023), fw = VERT ? 1 : p.stride[0];
  T* Y = reinterpret_cast<T*>(p.plane[0]);
  // ---- this lane's segment (of the warp's 8 x ROUNDS)
  const int at = blockIdx.x * kHdbThreads + threadIdx.x, sid = ROUNDS == 1 ? at >> 2 : at;
  const int row = sid / per_row, col = sid - row * per_row;
  const bool inside = row < rows && (VERT ? col > 0 : row > 0);  // an edge of the picture's inside
  const int x = VERT ? col << 3 : col << 2, y = VERT ? row << 2 : row << 3;
  HdbSegment mine;
  HdbLine<T, VEC> s;
  if (ROUNDS == 1 && inside) s.load(Y + (size_t)(VERT ? y + line : y) * p.stride[0] + (VERT ? x : x + line), fw);
  if (inside) mine = hdb_decide<VERT>(p, x, y);
  // ---- the warp's segments, eight at a time and a line per lane, where one of the
  //      eight is filtered
  const uint32_t active = __ballot_sync(0xffffffffu, mine.luma != 0);
#pragma unroll 1
  for (int first = 0; first < (ROUNDS == 1 ? 1 : 32); first += 8) {
    if (ROUNDS == 1 ? !active : !(active >> first & 0xffu)) continue;
    uint32_t lw = mine.luma, cw = mine.chroma;
    int sx = x, sy = y;
    if (ROUNDS > 1) {
      const int from = first + (lane >> 2);
      lw = __shfl_sync(0xffffffffu, lw, from);
      cw = __shfl_sync(0xffffffffu, cw, from);
      sx = __shfl_sync(0xffffffffu, sx, from);
      sy = __shfl_sync(0xffffffffu, sy, from);
    }
    const bool keep_p = lw & 4u, keep_q = lw & 8u;
    T* q = Y + (size_t)(VERT ? sy + line : sy) * p.stride[0] + (VERT ? sx : sx + line);
    if (ROUNDS > 1) {
      s = HdbLine<T, VEC>();
      if (lw) s.load(q, fw);
    }
    hdb_luma_filter<T, VEC>(s, q, fw, lw != 0, (int)(lw >> 11), (int)(lw >> 4 & 127u), keep_p, keep_q, maxv);
    if (!cw) continue;
    const int cx = VERT ? sx >> 1 : (sx >> 1) + line, cy = VERT ? (sy >> 1) + line : sy >> 1;
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
      const int tcc = (int)(cw >> (8 * pl) & 255u);
      if (!tcc) continue;
      T* C = reinterpret_cast<T*>(p.plane[1 + pl]);
      hdb_chroma_line<T>(C + (size_t)cy * p.stride[1 + pl] + cx, VERT ? 1 : p.stride[1 + pl], tcc, keep_p, keep_q, maxv);
    }
  }
}

template <typename T, int ROUNDS>
static void hdb_launch(const b200enc_hevc_deblock_t& q, cudaStream_t st) {
  // segments, and warps of 8 ROUNDS of them
  const int nv = (q.width >> 3) * (q.height >> 2), nh = (q.width >> 2) * (q.height >> 3);
  constexpr int kBlock = kHdbThreads / 32 * 8 * ROUNDS;
  const unsigned gv = (nv + kBlock - 1) / kBlock, gh = (nh + kBlock - 1) / kBlock;
  // four samples before and behind an edge start at a multiple of four of the row
  const bool vec = (reinterpret_cast<uintptr_t>(q.plane[0]) | (uintptr_t)q.stride[0] * sizeof(T)) % (4 * sizeof(T)) == 0;
  if (vec)
    launch_early(hevc_deblock_kernel<T, true, true, ROUNDS>, gv, kHdbThreads, 0, st, q);
  else
    launch_early(hevc_deblock_kernel<T, true, false, ROUNDS>, gv, kHdbThreads, 0, st, q);
  launch_early(hevc_deblock_kernel<T, false, false, ROUNDS>, gh, kHdbThreads, 0, st, q);
}

}  // namespace b200enc

using namespace b200enc;

extern "C" int b200enc_hevc_deblock(const b200enc_hevc_deblock_t* p, void* stream) {
  if (!p) return -1;
  const b200enc_hevc_deblock_t& q = *p;
  if (q.bit_depth_luma != 8 && q.bit_depth_luma != 10) return -1;
  if (q.bit_depth_chroma < 8 || q.bit_depth_chroma > q.bit_depth_luma) return -1;
  if (q.width <= 0 || q.height <= 0 || (q.width & 7) || (q.height & 7)) return -1;
  if (q.log2_ctb < 4 || q.log2_ctb > 6 || q.log2_min_cb < 3 || q.log2_min_cb > q.log2_ctb) return -1;
  if ((q.width & ((1 << q.log2_min_cb) - 1)) || (q.height & ((1 << q.log2_min_cb) - 1))) return -1;
  if (!q.plane[0] || !q.plane[1] || !q.plane[2] || !q.edges || !q.qp_y) return -1;
  if (q.stride[0] < q.width || q.stride[1] < q.width / 2 || q.stride[2] < q.width / 2) return -1;
  if (q.edges_stride < q.width / 8) return -1;
  if ((q.mvf || q.cbf) && q.min_pu_width < q.width / 4) return -1;
  if (((uintptr_t)q.mvf & 3) || ((uintptr_t)q.slice_filter & 3)) return -1;
  if (q.slice_filter && q.n_slice_filter <= 0) return -1;
  const cudaStream_t st = (cudaStream_t)stream;
  const bool few = (q.width >> 3) * (q.height >> 2) <= kHdbFew;
  if (q.bit_depth_luma == 8)
    few ? hdb_launch<uint8_t, 1>(q, st) : hdb_launch<uint8_t, 4>(q, st);
  else
    few ? hdb_launch<uint16_t, 1>(q, st) : hdb_launch<uint16_t, 4>(q, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
