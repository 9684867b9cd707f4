// hevc.cu - HEVC encoder primitives the reference's host RD loop calls per
// block, as batched GPU kernels:
//   H1  half-sample planes of the previous reconstruction for the motion
//       search (approach1-compute-encoder/src/hevc_enc_template.c:312-400,
//       build_hpel / hpel_pass): the whole-sample plane and the H, V and HV
//       planes of the 8-tap filter -1 4 -11 40 40 -11 4 -1, with a margin;
//   H2  8x8 CU motion search on those planes (search_sad :463, motion_search
//       :958);
//   H3  4x4 intra luma mode choice (hevc_intra_template.c:177);
//   H1-H3 at 8 bits and at 10 (Main10): the reference builds its template
//       twice (encoder_h265.c:1220-1227, hevc_intra.c), changing only the
//       sample type, the clip value, the no-neighbour fill and the search
//       SAD's scaling to eight-bit units;
//   H4  forward transform + quantisation of 4x4 (DCT-II or DST-VII) and 8x8
//       (DCT-II) residual blocks at 8 or 10 bits (hevc_intra.c:468, :565, :720);
//   H5  dequantisation + inverse transform of the same blocks
//       (hevc_intra.c:484, :586, :761).
// Arithmetic is the reference's compiled (SSE2) path: both transform passes
// round, shift and saturate to int16 exactly where its packs instructions
// do; the quantiser divides by levelScale through the same reciprocal
// multiply, which is exact over the reachable range.
#include <algorithm>
#include <type_traits>

#include "b200enc_internal.h"
#include "common.cuh"

namespace b200enc {

// H.265 transform matrices and levelScale (standard constants; the decoder
// uses the same values).
__constant__ int16_t kHDct4[4][4] = {{64, 64, 64, 64}, {83, 36, -36, -83}, {64, -64, -64, 64}, {36, -83, 83, -36}};
__constant__ int16_t kHDst4[4][4] = {{29, 55, 74, 84}, {74, 74, 0, -74}, {84, -29, -74, 55}, {55, -84, 74, -29}};
__constant__ int kHLevelScale[6] = {40, 45, 51, 57, 64, 72};

__device__ __forceinline__ int sat16(int v) { return v > 32767 ? 32767 : (v < -32768 ? -32768 : v); }

// Quantiser parameters of one QP: level = ((|x| << shift) + offset) >> p,
// then * m >> 32 (division by levelScale), capped at 32767, sign restored.
struct HQuant {
  int shift, p;
  uint32_t offset, m;
};

__device__ __forceinline__ HQuant hquant(int q, int shift, int round_q12) {
  HQuant h;
  h.shift = shift;
  h.p = q / 6 + 4;
  const uint32_t d = (uint32_t)kHLevelScale[q % 6];
  h.offset = (uint32_t)((((uint64_t)d << h.p) * (uint64_t)round_q12) / 12u);
  h.m = (uint32_t)((((uint64_t)1 << 32) + d - 1) / d);
  return h;
}

__device__ __forceinline__ int16_t hquant_level(int x, const HQuant& h) {
  const uint32_t mag = (uint32_t)(x < 0 ? -x : x);
  const uint32_t t = ((mag << h.shift) + h.offset) >> h.p;
  uint32_t l = (uint32_t)(((uint64_t)t * h.m) >> 32);
  if (l > 32767u) l = 32767u;
  return (int16_t)(x < 0 ? -(int)l : (int)l);
}

// Dequantisation, flat scaling list (8.6.3): level * levelScale << (q/6+4),
// rounded and shifted down by bd_shift, saturated to int16.
__device__ __forceinline__ int hdequant(int c, int q, int bd_shift) {
  const int a = q / 6 + 4, ls = kHLevelScale[q % 6];
  const int prod = c * ls;
  int v;
  if (a >= bd_shift) v = (int)((uint32_t)prod << (a - bd_shift));
  else v = (prod + (1 << (bd_shift - a - 1))) >> (bd_shift - a);
  return sat16(v);
}

// ---- 4x4 -------------------------------------------------------------------
__global__ void hevc_tq4_kernel(const int16_t* __restrict__ res, int16_t* __restrict__ out, int n, int q, int use_dst,
                                int round_q12, int s1, int qshift) {
  pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  const int16_t(*M)[4] = use_dst ? kHDst4 : kHDct4;
  int x[16];
  const int4* src = reinterpret_cast<const int4*>(res + (size_t)b * 16);
  const int4 v0 = src[0], v1 = src[1];
  const int w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    x[2 * i] = (int)(int16_t)(w[i] & 0xffff);
    x[2 * i + 1] = (int)(int16_t)((uint32_t)w[i] >> 16);
  }
  // an all-zero block gives all-zero levels whatever the rounding offset
  // (with a full-step offset the quantiser alone would give 1s)
  if (!(v0.x | v0.y | v0.z | v0.w | v1.x | v1.y | v1.z | v1.w)) {
    int4* dst = reinterpret_cast<int4*>(out + (size_t)b * 16);
    dst[0] = dst[1] = make_int4(0, 0, 0, 0);
    return;
  }
  int t[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      int s = 0;
#pragma unroll
      for (int r = 0; r < 4; ++r) s += M[i][r] * x[r * 4 + c];
      t[i][c] = sat16((s + (1 << (s1 - 1))) >> s1);
    }
  const HQuant h = hquant(q, qshift, round_q12);
  __align__(16) int16_t o[16];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int s = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) s += M[j][c] * t[i][c];
      o[i * 4 + j] = hquant_level(sat16((s + 128) >> 8), h);
    }
  int4* dst = reinterpret_cast<int4*>(out + (size_t)b * 16);
  dst[0] = *reinterpret_cast<const int4*>(&o[0]);
  dst[1] = *reinterpret_cast<const int4*>(&o[8]);
}

__global__ void hevc_dqit4_kernel(const int16_t* __restrict__ coeff, int16_t* __restrict__ out, int n, int q,
                                  int use_dst, int bd_shift, int s2) {
  pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  const int16_t(*M)[4] = use_dst ? kHDst4 : kHDct4;
  const int4* src = reinterpret_cast<const int4*>(coeff + (size_t)b * 16);
  const int4 v0 = src[0], v1 = src[1];
  const int w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
  int d[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    d[2 * i] = hdequant((int)(int16_t)(w[i] & 0xffff), q, bd_shift);
    d[2 * i + 1] = hdequant((int)(int16_t)((uint32_t)w[i] >> 16), q, bd_shift);
  }
  int g[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      int s = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) s += M[k][r] * d[k * 4 + c];
      g[r][c] = sat16((s + 64) >> 7);
    }
  __align__(16) int16_t o[16];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      int s = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) s += M[k][c] * g[r][k];
      o[r * 4 + c] = (int16_t)sat16((s + (1 << (s2 - 1))) >> s2);
    }
  int4* dst = reinterpret_cast<int4*>(out + (size_t)b * 16);
  dst[0] = *reinterpret_cast<const int4*>(&o[0]);
  dst[1] = *reinterpret_cast<const int4*>(&o[8]);
}

// ---- 8x8 -------------------------------------------------------------------
// Eight lanes per block: lane r loads row r (16 bytes; a warp's four blocks lie
// together), the column pass follows a transpose across the lanes and the row pass
// another, both as integer dot products of value pairs (the matrix fits in bytes).
// 32,400 blocks 5.4 us, inverse 3.6; a thread per block, 128 bytes apart, 7.6 and
// 6.9 (8.3 MB moved, 1.3 us).
//
// Entry (i, k) of the 8-point matrix: the standard's integer for
// cos(i (2k + 1) pi / 16), which takes eight values and their negatives.
__host__ __device__ constexpr int hdct8(int i, int k) {
  const int turn = i * (2 * k + 1) % 32, half = turn > 16 ? 32 - turn : turn, a = half > 8 ? 16 - half : half;
  const int c = a == 0 ? 64 : a == 1 ? 89 : a == 2 ? 83 : a == 3 ? 75 : a == 4 ? 64 : a == 5 ? 50 : a == 6 ? 36 : a == 7 ? 18 : 0;
  return half > 8 ? -c : c;
}
__device__ __forceinline__ uint32_t pack_sat16(int lo, int hi) {
  uint32_t d;
  asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(d) : "r"(hi), "r"(lo));
  return d;
}
// 8x8 transpose of 16-bit values over eight lanes: row r in, column r out, both
// as pairs (0, 1), (2, 3), ...
__device__ __forceinline__ void transpose8(uint32_t (&w)[4], int r) {
  const bool odd = r & 1, b1 = r & 2, b2 = r & 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {  // two rows' values of one column to a word
    const uint32_t o = __shfl_xor_sync(0xffffffffu, w[k], 1);
    w[k] = __byte_perm(w[k], o, odd ? 0x3276 : 0x5410);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {  // a 4x4 transpose of those words over the row pairs
    const uint32_t o = __shfl_xor_sync(0xffffffffu, b2 ? w[k] : w[k + 2], 4);
    (b2 ? w[k] : w[k + 2]) = o;
  }
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const uint32_t o = __shfl_xor_sync(0xffffffffu, b1 ? w[k] : w[k + 1], 2);
    (b1 ? w[k] : w[k + 1]) = o;
  }
}
// One pass over a lane's eight values: o[i] = (sum_k M[i][k] v[k] + round) >> shift,
// M the matrix (FWD) or its transpose.
template <bool FWD>
__device__ __forceinline__ void dct8_pass(const uint32_t (&w)[4], int round, int shift, int (&o)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int s = round;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c0 = FWD ? hdct8(i, 2 * k) : hdct8(2 * k, i);
      const int c1 = FWD ? hdct8(i, 2 * k + 1) : hdct8(2 * k + 1, i);
      s = __dp2a_lo((int)w[k], (c0 & 0xff) | (c1 & 0xff) << 8, s);
    }
    o[i] = s >> shift;
  }
}

__global__ void __launch_bounds__(256) hevc_tq8_kernel(const int16_t* __restrict__ res, int16_t* __restrict__ out,
                                                       int n, int q, int round_q12, int s1, int qshift) {
  pdl_wait();
  const long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // of all blocks
  const int r = threadIdx.x & 7;
  const bool in = row < (long long)n * 8;
  const uint4 v = in ? __ldg(reinterpret_cast<const uint4*>(res) + row) : make_uint4(0u, 0u, 0u, 0u);
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
  // as for 4x4: an all-zero block gives all-zero levels
  const uint32_t any = __ballot_sync(0xffffffffu, (v.x | v.y | v.z | v.w) != 0u) >> (threadIdx.x & 24) & 0xffu;
  int o[8];
  transpose8(w, r);
  dct8_pass<true>(w, 1 << (s1 - 1), s1, o);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = pack_sat16(o[2 * k], o[2 * k + 1]);
  transpose8(w, r);
  dct8_pass<true>(w, 256, 9, o);
  const HQuant h = hquant(q, qshift, round_q12);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    w[k] = any ? (uint32_t)(uint16_t)hquant_level(sat16(o[2 * k]), h) | (uint32_t)(uint16_t)hquant_level(sat16(o[2 * k + 1]), h) << 16
               : 0u;
  if (in) reinterpret_cast<uint4*>(out)[row] = make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(256) hevc_dqit8_kernel(const int16_t* __restrict__ coeff, int16_t* __restrict__ out,
                                                         int n, int q, int bd_shift, int s2) {
  pdl_wait();
  const long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = threadIdx.x & 7;
  const bool in = row < (long long)n * 8;
  const uint4 v = in ? __ldg(reinterpret_cast<const uint4*>(coeff) + row) : make_uint4(0u, 0u, 0u, 0u);
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    w[k] = pack_sat16(hdequant((int)(int16_t)(w[k] & 0xffffu), q, bd_shift), hdequant((int)w[k] >> 16, q, bd_shift));
  int o[8];
  transpose8(w, r);
  dct8_pass<false>(w, 64, 7, o);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = pack_sat16(o[2 * k], o[2 * k + 1]);
  transpose8(w, r);
  dct8_pass<false>(w, 1 << (s2 - 1), s2, o);
  if (in)
    reinterpret_cast<uint4*>(out)[row] =
        make_uint4(pack_sat16(o[0], o[1]), pack_sat16(o[2], o[3]), pack_sat16(o[4], o[5]), pack_sat16(o[6], o[7]));
}

// ---- half-sample planes ----------------------------------------------------
// Plane coordinates (r, c) are picture coordinates + margin; every reference
// read is clamped to the picture (the reference's edge extension). With
// Y(k) = clampY(r - M - 3 + k) and X(k) = clampX(c - M - 3 + k):
//   I  = ref[clampY(r - M)][clampX(c - M)]
//   H  = clip((sum_k tap[k] * ref[clampY(r - M)][X(k)] + 32) >> 6)
//   V  = clip((sum_k tap[k] * ref[Y(k)][clampX(c - M)] + 32) >> 6)
//   HV = clip((sum_k tap[k] * T(Y(k)) + 2048) >> 12),  T(y) = sum_j tap[j] * ref[y][X(j)]
// A block makes a tile of 128 columns x 32 rows, a thread 4 columns x 8 rows of
// it: the clamped samples are staged once, four at a time, in shared memory, and
// each thread walks 15 of its rows with the last eight rows' column samples and
// horizontal sums in registers. Horizontal sums are integer dot products (dp4a,
// dp2a), vertical ones of 8-bit samples two columns to a register (a column's sum
// is under 16 bits). Bound by instructions issued until the planes' four writes
// per sample are what is left: 1080p at 8 bits 8.6 us, a thread per sample with
// the sums staged in shared memory 17.5 (10.6 MB moved, 1.6 us).
constexpr int kHpTileW = 128, kHpTileH = 32, kHpRows = 8;

__device__ __forceinline__ int dot2(uint32_t samples, uint32_t taps, int acc) {
  int d;
  asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(samples), "r"(taps), "r"(acc));
  return d;
}
template <class T>
__device__ __forceinline__ T filter8(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7) {
  return (a3 + a4) * 40 - (a2 + a5) * 11 + (a1 + a6) * 4 - (a0 + a7);
}

// Four samples; P: the sample type (uint8_t at 8 bits, uint16_t at 10).
template <typename P>
struct Quad;
template <>
struct Quad<uint8_t> {
  uint32_t w;
  __device__ __forceinline__ void load(const uint8_t* p) {  // any alignment; only words holding the samples are read
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
    const uint32_t off = (uint32_t)a & 3u;
    w = __funnelshift_r(__ldg(q), __ldg(q + (off ? 1 : 0)), off * 8);
  }
  __device__ __forceinline__ void set(int a, int b, int c, int d) { w = a | b << 8 | c << 16 | d << 24; }
  __device__ __forceinline__ void store(uint8_t* p) const { *reinterpret_cast<uint32_t*>(p) = w; }
  __device__ __forceinline__ uint8_t at(int i) const { return (uint8_t)(w >> (8 * i)); }
  // horizontal sums of this quad's samples, given the quads on either side
  __device__ __forceinline__ void sums(const Quad& l, const Quad& r, int (&t)[4]) const {
    constexpr uint32_t ta = 0x28f504ffu, tb = 0xff04f528u;  // -1 4 -11 40, 40 -11 4 -1
#pragma unroll
    for (int j = 0; j < 4; ++j)
      t[j] = dot4(j == 3 ? w : __funnelshift_r(l.w, w, 8 * (j + 1)), ta,
                  dot4(j == 3 ? r.w : __funnelshift_r(w, r.w, 8 * (j + 1)), tb, 0));
  }
};
template <>
struct Quad<uint16_t> {
  uint2 w;
  __device__ __forceinline__ void load(const uint16_t* p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
    const uint32_t off = (uint32_t)a & 3u, mid = __ldg(q + 1);
    w.x = __funnelshift_r(__ldg(q), mid, off * 8);
    w.y = __funnelshift_r(mid, __ldg(q + (off ? 2 : 1)), off * 8);
  }
  __device__ __forceinline__ void set(int a, int b, int c, int d) { w = make_uint2(a | b << 16, c | d << 16); }
  __device__ __forceinline__ void store(uint16_t* p) const { *reinterpret_cast<uint2*>(p) = w; }
  __device__ __forceinline__ uint16_t at(int i) const { return (uint16_t)((i < 2 ? w.x : w.y) >> (16 * (i & 1))); }
  __device__ __forceinline__ void sums(const Quad& l, const Quad& r, int (&t)[4]) const {
    const uint32_t e[6] = {l.w.x, l.w.y, w.x, w.y, r.w.x, r.w.y};  // pairs from even samples on
    constexpr uint32_t tap[4] = {0x04ffu, 0x28f5u, 0xf528u, 0xff04u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      t[j] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {  // samples j + 1 + 2k of the twelve, and the next
        const int i = (j + 1) / 2 + k;
        t[j] = dot2((j & 1) ? e[i] : __funnelshift_r(e[i], e[i + 1 < 6 ? i + 1 : i], 16), tap[k], t[j]);
      }
    }
  }
};

// maxv: the largest sample value, (1 << BitDepth) - 1 (hevc_enc_template.c:23-25);
// vec: planes and their pitch aligned for four-sample stores.
template <typename P>
__global__ void __launch_bounds__(128) hevc_hpel_kernel(const P* __restrict__ ref, int pitch, int w, int h, int M,
                                                        P* __restrict__ pI, P* __restrict__ pH, P* __restrict__ pV,
                                                        P* __restrict__ pHV, int opitch, int rows, int cols, int maxv,
                                                        int vec) {
  pdl_wait();
  constexpr int kQuads = kHpTileW / 4 + 2;
  __shared__ Quad<P> src[kHpTileH + 7][kQuads];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c0 = blockIdx.x * kHpTileW, r0 = blockIdx.y * kHpTileH;
  // source rows r0-M-3 .. r0-M+kHpTileH+3, columns c0-M-4 .. c0-M+kHpTileW+3
  for (int i = threadIdx.x; i < (kHpTileH + 7) * kQuads; i += 128) {
    const int sr = i / kQuads, sc = i - sr * kQuads;
    const P* row = ref + (size_t)clampi(r0 - M - 3 + sr, 0, h - 1) * pitch;
    const int x = c0 - M - 4 + 4 * sc;
    Quad<P> q;
    if (x >= 0 && x + 3 < w)
      q.load(row + x);
    else
      q.set(row[clampi(x, 0, w - 1)], row[clampi(x + 1, 0, w - 1)], row[clampi(x + 2, 0, w - 1)],
            row[clampi(x + 3, 0, w - 1)]);
    src[sr][sc] = q;
  }
  __syncthreads();
  const int c = c0 + 4 * tx, r1 = r0 + ty * kHpRows;
  if (c >= cols || r1 >= rows) return;
  const bool whole = vec && c + 3 < cols;
  auto put = [&](P* plane, int r, const Quad<P>& q) {
    P* p = plane + (size_t)r * opitch + c;
    if (whole) {
      q.store(p);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < cols) p[j] = q.at(j);
    }
  };
  auto clip = [&](const int (&v)[4], int round, int shift) {
    Quad<P> q;
    q.set(clampi((v[0] + round) >> shift, 0, maxv), clampi((v[1] + round) >> shift, 0, maxv),
          clampi((v[2] + round) >> shift, 0, maxv), clampi((v[3] + round) >> shift, 0, maxv));
    return q;
  };
  int t[kHpRows][4];     // horizontal sums of the last eight rows
  Quad<P> s[kHpRows];    // and their samples
#pragma unroll
  for (int k = 0; k < kHpRows + 7; ++k) {
    const Quad<P>* q = &src[ty * kHpRows + k][tx];
    s[k % 8] = q[1];
    q[1].sums(q[0], q[2], t[k % 8]);
    if (k < 7) continue;
    const int r = r1 + k - 7;  // rows k - 7 .. k around it; its own is k - 4
    if (r >= rows) return;
    put(pI, r, s[(k - 4) % 8]);
    put(pH, r, clip(t[(k - 4) % 8], 32, 6));
    int v[4];
    if constexpr (sizeof(P) == 1) {
#pragma unroll
      for (int p = 0; p < 2; ++p) {  // columns 2p and 2p + 1
        uint32_t a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = __byte_perm(s[(k - 7 + i) % 8].w, 0, p ? 0x4342 : 0x4140);
        const uint32_t f = filter8(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
        v[2 * p] = (int16_t)f;
        v[2 * p + 1] = (int)(f + 0x8000u) >> 16;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[j] = filter8<int>(s[(k - 7) % 8].at(j), s[(k - 6) % 8].at(j), s[(k - 5) % 8].at(j), s[(k - 4) % 8].at(j),
                            s[(k - 3) % 8].at(j), s[(k - 2) % 8].at(j), s[(k - 1) % 8].at(j), s[k % 8].at(j));
    }
    put(pV, r, clip(v, 32, 6));
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = filter8(t[(k - 7) % 8][j], t[(k - 6) % 8][j], t[(k - 5) % 8][j], t[(k - 4) % 8][j], t[(k - 3) % 8][j],
                     t[(k - 2) % 8][j], t[(k - 1) % 8][j], t[k % 8][j]);
    put(pHV, r, clip(v, 2048, 12));
  }
}

// ---- 8x8 CU motion search -------------------------------------------------
// Half a warp per CU job, the reference's walk (hevc_enc_template.c:958-1043).
// The walk compares its candidates against a fixed centre per step, in order,
// strictly; so the lowest cost with the lowest candidate number is the same
// choice, and four candidates are scored at a time: each of the four lanes of a
// candidate holds two rows of the CU (read once) and scores them with packed
// arithmetic, a step of the walk being one such pass, and each refinement two.
// A job is a chain of about ten dependent passes of loads and shuffles, so the
// kernel is bound by their latency and the instructions issued, not by bytes;
// with two jobs in a warp each instruction serves both. 32,400 CUs of a 1080p
// picture at 8 bits: 45 us; one job per warp, a row per lane, 75; one candidate
// at a time, two samples per lane, 185.
// Strides in samples. sad_shift brings a SAD back to eight-bit units (0 at
// eight bits, 2 at ten: hevc_enc_template.c:484).
template <typename P>
struct HevcSearch {
  const P* src;
  int src_pitch, w, h, M, qpel;
  const P* plane[4];
  int ppitch, sad_shift;
};

__device__ __forceinline__ int hevc_mvd_bits(int d) {
  const unsigned a = (unsigned)(d < 0 ? -d : d);
  if (a == 0) return 1;
  if (a == 1) return 3;
  return 3 + 2 * (31 - __clz((int)((a - 2) / 2 + 1))) + 2;
}

// Eight samples from any address: the aligned words that hold them (none other
// is read), shifted together.
template <typename P>
struct HevcRow {
  static constexpr int kWords = 2 * (int)sizeof(P);
  uint32_t w[kWords];
  __device__ __forceinline__ void load(const P* p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
    const uint32_t off = (uint32_t)a & 3u;
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = __ldg(q + i);
    const uint32_t last = __ldg(q + (off ? kWords : kWords - 1));
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = __funnelshift_r(w[i], i + 1 < kWords ? w[i + 1 < kWords ? i + 1 : i] : last, off * 8);
  }
  // rounded average of each sample with o's
  __device__ __forceinline__ void average(const HevcRow& o) {
    constexpr uint32_t m = sizeof(P) == 1 ? 0x7f7f7f7fu : 0x7fff7fffu;
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = (w[i] | o.w[i]) - (((w[i] ^ o.w[i]) >> 1) & m);
  }
  __device__ __forceinline__ uint32_t sad(const HevcRow& o) const {
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      if (sizeof(P) == 1) {
        s += __vsadu4(w[i], o.w[i]);
      } else {
        s = __dp2a_lo(__vmaxu2(w[i], o.w[i]) - __vminu2(w[i], o.w[i]), 0x0101u, s);
      }
    }
    return s;
  }
};

// SAD of the CU (rows `row` and row + 4 in `cu`) against the search planes at
// absolute quarter-sample position (qx, qy), the same for the four lanes of a
// candidate (search_sad, hevc_enc_template.c:463): positions are clamped to the
// planes' margin; even/even reads one half-grid block, a position odd in x, y or
// both averages (rounded) the two blocks beside it. ODD false: the caller's
// positions are all even.
template <typename P, bool ODD>
__device__ __forceinline__ uint32_t hevc_search_sad(const HevcSearch<P>& S, const HevcRow<P> (&cu)[2], int qx, int qy,
                                                    int row) {
  const int lo = -(S.M - 2) * 4;
  const int hx = (S.w - 8 + S.M - 2) * 4, hy = (S.h - 8 + S.M - 2) * 4;
  qx = qx < lo ? lo : (qx > hx ? hx : qx);
  qy = qy < lo ? lo : (qy > hy ? hy : qy);
  auto at = [&](int bqx, int bqy) -> const P* {
    const int ph = ((bqx & 2) ? 1 : 0) + ((bqy & 2) ? 2 : 0);
    return S.plane[ph] + ((size_t)((bqy >> 2) + S.M + row) * S.ppitch + ((bqx >> 2) + S.M));
  };
  const size_t down = (size_t)4 * S.ppitch;
  HevcRow<P> a[2];
  if (ODD) {
    const int ox = qx & 1, oy = qy & 1;
    HevcRow<P> b[2];  // even/even: the block itself twice, whose average it is
    const P *pa = at(qx - ox, qy - oy), *pb = at(qx + ox, qy + oy);
    a[0].load(pa);
    a[1].load(pa + down);
    b[0].load(pb);
    b[1].load(pb + down);
    a[0].average(b[0]);
    a[1].average(b[1]);
  } else {
    const P* pa = at(qx, qy);
    a[0].load(pa);
    a[1].load(pa + down);
  }
  uint32_t sad = a[0].sad(cu[0]) + a[1].sad(cu[1]);
  sad += __shfl_xor_sync(0xffffffffu, sad, 1);
  sad += __shfl_xor_sync(0xffffffffu, sad, 2);
  return sad >> S.sad_shift;
}

template <typename P>
__global__ void __launch_bounds__(128) hevc_me_kernel(const __grid_constant__ HevcSearch<P> S,
                                                      const b200enc_hevc_me_job_t* __restrict__ jobs, int n,
                                                      b200enc_hevc_me_result_t* __restrict__ out) {
  pdl_wait();
  const int lane = threadIdx.x & 31, first = lane & 16, cand = (lane >> 2) & 3, row = lane & 3;
  const int j = blockIdx.x * 8 + (threadIdx.x >> 4);
  if (j - (first >> 4) >= n) return;  // neither half has a job
  const b200enc_hevc_me_job_t& job = jobs[min(j, n - 1)];
  int cu_x = job.cu_x, cu_y = job.cu_y;
  const bool bad = cu_x < 0 || cu_y < 0 || cu_x > S.w - 8 || cu_y > S.h - 8;  // not a CU of this picture
  if (bad) cu_x = cu_y = 0;  // searched with the other half's, then answered as invalid
  HevcRow<P> cu[2];
  cu[0].load(S.src + (size_t)(cu_y + row) * S.src_pitch + cu_x);
  cu[1].load(S.src + (size_t)(cu_y + row + 4) * S.src_pitch + cu_x);
  const int min_dx = -cu_x - 8, max_dx = S.w - cu_x, min_dy = -cu_y - 8, max_dy = S.h - cu_y;
  const int range = 64, qx0 = cu_x * 4, qy0 = cu_y * 4;
  const long long lambda = job.lambda_q8;
  // this lane's share of the vector bits: one component against one predictor
  const bool is_y = lane & 1;
  const int pred = is_y ? job.mvp[(lane >> 1) & 1].y : job.mvp[(lane >> 1) & 1].x;
  constexpr long long kNone = 0x7fffffffffffffffll;
  long long best = kNone;
  uint32_t best_sad = 0;

  // Scores four candidates per half, this lane's at (qx, qy) relative to its CU;
  // returns the number of the one that beats the half's `best` (updated), or -1.
  // Costs are far under 2^60, so the candidate number fits below them.
  auto pass = [&](auto odd, int qx, int qy, bool valid) -> int {
    const uint32_t sd = hevc_search_sad<P, decltype(odd)::value>(S, cu, qx0 + qx, qy0 + qy, row);
    int bits = hevc_mvd_bits((is_y ? qy : qx) - pred);
    bits += __shfl_xor_sync(0xffffffffu, bits, 1);
    bits = min(bits, __shfl_xor_sync(0xffffffffu, bits, 2));
    const long long c = (long long)sd * 256 + lambda * bits;
    long long key = valid && c < best ? c * 4 + cand : kNone;
#pragma unroll
    for (int o = 4; o < 16; o <<= 1) {
      const long long k = __shfl_xor_sync(0xffffffffu, key, o);
      key = k < key ? k : key;
    }
    const int k = (int)(key & 3);
    const uint32_t ks = __shfl_sync(0xffffffffu, sd, first + k * 4);
    if (key == kNone) return -1;
    best = key >> 2;
    best_sad = ks;
    return k;
  };
  using Even = std::false_type;
  using Odd = std::true_type;

  // start points, each distinct one once (a repeat cannot beat its first)
  int bx = 0, by = 0;
  {
    const int i = lane & 15, ns = min(max(job.n_starts, 0), 16);
    int dx = 0, dy = 0;
    if (i < ns) {  // within +-8192: the limits lie on both sides of 0
      dx = min(max((job.starts[i].x + 2) >> 2, min_dx), max_dx);
      dy = min(max((job.starts[i].y + 2) >> 2, min_dy), max_dy);
    }
    const uint32_t key = i < ns ? (uint32_t)(dy + 8192) << 15 | (uint32_t)(dx + 8192) : 1u << 30 | i;
    const uint32_t same = __match_any_sync(0xffffffffu, key | (uint32_t)first << 27);
    uint32_t todo = __ballot_sync(0xffffffffu, i < ns && (same & ((1u << lane) - 1u)) == 0u) >> first & 0xffffu;
    while (__any_sync(0xffffffffu, todo != 0)) {
      uint32_t t = todo;  // this candidate's start: the cand-th of those left, or the last
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (q < cand && (t & (t - 1))) t &= t - 1;
      const int from = first + (t ? __ffs(t) - 1 : 0);
      const int gx = __shfl_sync(0xffffffffu, dx, from), gy = __shfl_sync(0xffffffffu, dy, from);
      const int k = pass(Even{}, gx * 4, gy * 4, cand < __popc(todo));
      const int kx = __shfl_sync(0xffffffffu, gx, first + (k & 3) * 4), ky = __shfl_sync(0xffffffffu, gy, first + (k & 3) * 4);
      if (k >= 0) bx = kx, by = ky;
#pragma unroll
      for (int q = 0; q < 4; ++q) todo &= todo - 1;
    }
  }
  const int cx0 = bx, cy0 = by;
  const int ddx = cand == 0 ? -1 : (cand == 1 ? 1 : 0), ddy = cand == 2 ? -1 : (cand == 3 ? 1 : 0);
  int back = -1;
  bool walking = true;
  for (int step = 0; step < 32 && __any_sync(0xffffffffu, walking); ++step) {
    const int dx = bx + ddx, dy = by + ddy;
    const bool valid = walking && cand != back && dx >= min_dx && dx <= max_dx && dy >= min_dy && dy <= max_dy &&
                       dx >= cx0 - range && dx <= cx0 + range && dy >= cy0 - range && dy <= cy0 + range;
    const int k = pass(Even{}, dx * 4, dy * 4, valid);
    walking = k >= 0;
    if (walking) {
      bx += k == 0 ? -1 : (k == 1 ? 1 : 0);
      by += k == 2 ? -1 : (k == 3 ? 1 : 0);
      back = k ^ 1;
    }
  }
  int mx = bx * 4, my = by * 4;
  // the eight neighbours in raster order, four above and left, four right and below
  auto refine = [&](auto odd, int st) {
    const int c0x = mx, c0y = my;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      auto off_x = [&](int k) { return half == 0 ? (k == 3 ? -1 : k - 1) : (k == 0 ? 1 : k - 2); };
      auto off_y = [&](int k) { return half == 0 ? (k == 3 ? 0 : -1) : (k == 0 ? 0 : 1); };
      const int k = pass(odd, c0x + off_x(cand) * st, c0y + off_y(cand) * st, true);
      if (k >= 0) {
        mx = c0x + off_x(k) * st;
        my = c0y + off_y(k) * st;
      }
    }
  };
  refine(Even{}, 2);
  if (S.qpel) refine(Odd{}, 1);
  int bits = hevc_mvd_bits((is_y ? my : mx) - pred);
  bits += __shfl_xor_sync(0xffffffffu, bits, 1);
  const int b1 = __shfl_sync(0xffffffffu, bits, first + 2);
  if (lane == first && j < n) {
    b200enc_hevc_me_result_t r{};
    if (bad) {
      r.sad = 0xffffffffu;
      r.cost_q8 = -1;
    } else {
      r.mv.x = (int16_t)mx;
      r.mv.y = (int16_t)my;
      r.mvp_idx = b1 < bits ? 1 : 0;
      r.cost_q8 = best;
      r.sad = best_sad;
    }
    out[j] = r;
  }
}

// ---- intra 4x4 luma mode choice ----------------------------------------------
// hevc_intra_template.c:20-260 (gather_neighbors, predict_from_refs,
// hevc_choose_luma_mode) with hevc_intra.c's z-scan availability: a
// neighbour is available iff it is inside the picture, at or below the
// slice's first row, and earlier in the encoder's fixed coding order (CTU
// 16x16 raster, CU 8x8 z-order, PU 4x4 z-order).
__device__ __forceinline__ long long hz_rank(int x, int y, int width) {
  const int width_ctu = (width + 15) >> 4;
  const int rx = x & 15, ry = y & 15;
  long long rank = ((long long)(y >> 4) * width_ctu + (x >> 4)) * 4 + ((ry >> 3) * 2 + (rx >> 3));
  return rank * 4 + (((ry & 7) >> 2) * 2 + ((rx & 7) >> 2));
}
__device__ __forceinline__ bool hz_avail(int nx, int ny, int width, int height, int y_min, long long cur) {
  if (nx < 0 || ny < y_min || nx >= width || ny >= height) return false;
  return hz_rank(nx, ny, width) < cur;
}

constexpr int kHModePlanar = 0, kHModeDc = 1, kHModeHor = 10, kHModeVer = 26;

__device__ __forceinline__ void hpredict(const int* left, const int* top, int corner, int mode, int maxv, int* pred) {
  if (mode == kHModePlanar) {
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int x = 0; x < 4; ++x)
        pred[y * 4 + x] = ((3 - x) * left[y] + (x + 1) * top[4] + (3 - y) * top[x] + (y + 1) * left[4] + 4) >> 3;
  } else if (mode == kHModeDc) {
    const int dc = (left[0] + left[1] + left[2] + left[3] + top[0] + top[1] + top[2] + top[3] + 4) >> 3;
#pragma unroll
    for (int i = 0; i < 16; ++i) pred[i] = dc;
    pred[0] = (left[0] + 2 * dc + top[0] + 2) >> 2;
#pragma unroll
    for (int x = 1; x < 4; ++x) pred[x] = (top[x] + 3 * dc + 2) >> 2;
#pragma unroll
    for (int y = 1; y < 4; ++y) pred[y * 4] = (left[y] + 3 * dc + 2) >> 2;
  } else if (mode == kHModeHor) {
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int x = 0; x < 4; ++x) pred[y * 4 + x] = left[y];
#pragma unroll
    for (int x = 0; x < 4; ++x) pred[x] = clampi(left[0] + ((top[x] - corner) >> 1), 0, maxv);
  } else {
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int x = 0; x < 4; ++x) pred[y * 4 + x] = top[x];
#pragma unroll
    for (int y = 0; y < 4; ++y) pred[y * 4] = clampi(top[0] + ((left[y] - corner) >> 1), 0, maxv);
  }
}

// P: the sample type; bd the bit depth (8 or 10). Pitches in samples.
template <typename P>
__global__ void hevc_intra4_kernel(const P* __restrict__ src, int src_pitch, const P* __restrict__ rec,
                                   int rec_pitch, int width, int height, const int* __restrict__ jobs, int n,
                                   int* __restrict__ modes, P* __restrict__ preds, int bd) {
  pdl_wait();
  const int maxv = (1 << bd) - 1;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int x0 = jobs[3 * j], y0 = jobs[3 * j + 1], y_min = jobs[3 * j + 2];
  if (x0 < 0 || y0 < 0 || x0 + 4 > width || y0 + 4 > height || (x0 & 3) || (y0 & 3)) {
    modes[j] = -1;  // not a 4x4 PU of this picture
    return;
  }
  const long long cur = hz_rank(x0, y0, width);
  const bool a_left = hz_avail(x0 - 1, y0, width, height, y_min, cur);
  const bool a_top = hz_avail(x0, y0 - 1, width, height, y_min, cur);
  const bool a_corner = hz_avail(x0 - 1, y0 - 1, width, height, y_min, cur);
  const bool a_tr = hz_avail(x0 + 4, y0 - 1, width, height, y_min, cur);
  // the substitution scan over p[-1][3..0], p[-1][-1], p[0..4][-1]
  int sv[10];
  bool sa[10];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sa[i] = a_left;
    sv[i] = a_left ? rec[(size_t)(y0 + 3 - i) * rec_pitch + x0 - 1] : 0;
  }
  sa[4] = a_corner;
  sv[4] = a_corner ? rec[(size_t)(y0 - 1) * rec_pitch + x0 - 1] : 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sa[5 + i] = a_top;
    sv[5 + i] = a_top ? rec[(size_t)(y0 - 1) * rec_pitch + x0 + i] : 0;
  }
  sa[9] = a_tr;
  sv[9] = a_tr ? rec[(size_t)(y0 - 1) * rec_pitch + x0 + 4] : 0;
  int first = -1;
#pragma unroll
  for (int i = 9; i >= 0; --i)
    if (sa[i]) first = i;
  if (first < 0) {
#pragma unroll
    for (int i = 0; i < 10; ++i) sv[i] = 1 << (bd - 1);  // 128 at eight bits, 512 at ten
  } else {
    const int f = sv[first];
#pragma unroll
    for (int i = 0; i < 10; ++i)
      if (i < first) sv[i] = f;
#pragma unroll
    for (int i = 1; i < 10; ++i)
      if (i > first && !sa[i]) sv[i] = sv[i - 1];
  }
  int left[5], top[5];
  left[3] = sv[0]; left[2] = sv[1]; left[1] = sv[2]; left[0] = sv[3];
  const int corner = sv[4];
  top[0] = sv[5]; top[1] = sv[6]; top[2] = sv[7]; top[3] = sv[8]; top[4] = sv[9];
  left[4] = hz_avail(x0 - 1, y0 + 4, width, height, y_min, cur) ? rec[(size_t)(y0 + 4) * rec_pitch + x0 - 1]
                                                                : left[3];
  int s[16];
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int x = 0; x < 4; ++x) s[y * 4 + x] = src[(size_t)(y0 + y) * src_pitch + x0 + x];
  const int order[4] = {kHModePlanar, kHModeDc, kHModeHor, kHModeVer};
  int best_mode = -1, best_sad = 0;
  int best_pred[16];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    int pr[16];
    hpredict(left, top, corner, order[m], maxv, pr);
    int sad = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) sad += abs(s[i] - pr[i]);
    if (m == 0 || sad < best_sad) {
      best_sad = sad;
      best_mode = order[m];
#pragma unroll
      for (int i = 0; i < 16; ++i) best_pred[i] = pr[i];
    }
  }
  modes[j] = best_mode;
  if (sizeof(P) == 1) {
    uint32_t w4[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      w4[r] = (uint32_t)best_pred[4 * r] | ((uint32_t)best_pred[4 * r + 1] << 8) |
              ((uint32_t)best_pred[4 * r + 2] << 16) | ((uint32_t)best_pred[4 * r + 3] << 24);
    *reinterpret_cast<uint4*>(preds + (size_t)j * 16) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
  } else {
    uint32_t w8[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) w8[k] = (uint32_t)best_pred[2 * k] | ((uint32_t)best_pred[2 * k + 1] << 16);
    uint4* o = reinterpret_cast<uint4*>(preds + (size_t)j * 16);
    o[0] = make_uint4(w8[0], w8[1], w8[2], w8[3]);
    o[1] = make_uint4(w8[4], w8[5], w8[6], w8[7]);
  }
}

bool aligned16(const void* p) { return (((uintptr_t)p) & 15) == 0; }
int hclamp(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Whether four samples of every plane row can be stored at once.
template <typename P>
static int quad_aligned(const P* a, const P* b, const P* c, const P* d, int pitch) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
                        reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(d) | (uintptr_t)pitch * sizeof(P);
  return all % (4 * sizeof(P)) == 0;
}

}  // namespace b200enc

using namespace b200enc;

extern "C" {

int b200enc_hevc_transform_quant_4x4(const int16_t* residual, int16_t* coeff, int n, int qp, int use_dst,
                                     int round_q12, int bit_depth, void* stream) {
  if (!residual || !coeff || n < 0 || (bit_depth != 8 && bit_depth != 10)) return -1;
  if (!aligned16(residual) || !aligned16(coeff) || round_q12 < 0 || round_q12 > 12) return -1;
  if (n == 0) return 0;
  const int q = bit_depth == 8 ? hclamp(qp, 0, 51) : hclamp(qp, 0, 63);
  launch_early(hevc_tq4_kernel, (n + 255) / 256, 256, 0, (cudaStream_t)stream, residual, coeff, n, q, use_dst ? 1 : 0,
               round_q12, bit_depth == 8 ? 1 : 3, bit_depth == 8 ? 5 : 7);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_dequant_itransform_4x4(const int16_t* coeff, int16_t* residual, int n, int qp, int use_dst,
                                        int bit_depth, void* stream) {
  if (!residual || !coeff || n < 0 || (bit_depth != 8 && bit_depth != 10)) return -1;
  if (!aligned16(residual) || !aligned16(coeff)) return -1;
  // the reference clamps the 10-bit Qp' but takes the 8-bit QP as given
  if (bit_depth == 8 && (qp < 0 || qp > 51)) return -1;
  if (n == 0) return 0;
  const int q = bit_depth == 8 ? qp : hclamp(qp, 0, 63);
  launch_early(hevc_dqit4_kernel, (n + 255) / 256, 256, 0, (cudaStream_t)stream, coeff, residual, n, q, use_dst ? 1 : 0,
               bit_depth == 8 ? 5 : 7, bit_depth == 8 ? 12 : 10);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_transform_quant_8x8(const int16_t* residual, int16_t* coeff, int n, int qp, int bit_depth,
                                     int round_q12, void* stream) {
  if (!residual || !coeff || n < 0 || (bit_depth != 8 && bit_depth != 10)) return -1;
  if (!aligned16(residual) || !aligned16(coeff) || round_q12 < 0 || round_q12 > 12) return -1;
  if (n == 0) return 0;
  launch_early(hevc_tq8_kernel, (unsigned)((n + 31ll) / 32), 256, 0, (cudaStream_t)stream, residual, coeff, n, hclamp(qp, 0, 63),
               round_q12, 3 + bit_depth - 9, bit_depth - 2);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_dequant_itransform_8x8(const int16_t* coeff, int16_t* residual, int n, int qp, int bit_depth,
                                        void* stream) {
  if (!residual || !coeff || n < 0 || (bit_depth != 8 && bit_depth != 10)) return -1;
  if (!aligned16(residual) || !aligned16(coeff)) return -1;
  if (n == 0) return 0;
  launch_early(hevc_dqit8_kernel, (unsigned)((n + 31ll) / 32), 256, 0, (cudaStream_t)stream, coeff, residual, n, hclamp(qp, 0, 63),
               bit_depth - 2, 20 - bit_depth);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_build_hpel(const uint8_t* recon, int pitch, int w, int h, int margin, uint8_t* plane_i,
                            uint8_t* plane_h, uint8_t* plane_v, uint8_t* plane_hv, int plane_pitch, void* stream) {
  if (!recon || !plane_i || !plane_h || !plane_v || !plane_hv || w <= 0 || h <= 0) return -1;
  if (margin < 0 || margin > 256 || pitch < w) return -1;
  const int rows = h + 2 * margin, cols = w + 2 * margin;
  if (plane_pitch < cols) return -1;
  dim3 grid((cols + kHpTileW - 1) / kHpTileW, (rows + kHpTileH - 1) / kHpTileH);
  launch_early(hevc_hpel_kernel<uint8_t>, grid, 128, 0, (cudaStream_t)stream, recon, pitch, w, h, margin, plane_i,
               plane_h, plane_v, plane_hv, plane_pitch, rows, cols, 255, quad_aligned(plane_i, plane_h, plane_v,
               plane_hv, plane_pitch));
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_build_hpel_10(const uint16_t* recon, int pitch, int w, int h, int margin, uint16_t* plane_i,
                               uint16_t* plane_h, uint16_t* plane_v, uint16_t* plane_hv, int plane_pitch,
                               void* stream) {
  if (!recon || !plane_i || !plane_h || !plane_v || !plane_hv || w <= 0 || h <= 0) return -1;
  if (margin < 0 || margin > 256 || pitch < w) return -1;
  const int rows = h + 2 * margin, cols = w + 2 * margin;
  if (plane_pitch < cols) return -1;
  dim3 grid((cols + kHpTileW - 1) / kHpTileW, (rows + kHpTileH - 1) / kHpTileH);
  launch_early(hevc_hpel_kernel<uint16_t>, grid, 128, 0, (cudaStream_t)stream, recon, pitch, w, h, margin, plane_i,
               plane_h, plane_v, plane_hv, plane_pitch, rows, cols, 1023, quad_aligned(plane_i, plane_h, plane_v,
               plane_hv, plane_pitch));
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_motion_search(const uint8_t* src_y, int src_pitch, int w, int h, const uint8_t* plane_i,
                               const uint8_t* plane_h, const uint8_t* plane_v, const uint8_t* plane_hv, int plane_pitch,
                               int margin, int qpel, const b200enc_hevc_me_job_t* jobs, int n,
                               b200enc_hevc_me_result_t* results, void* stream) {
  if (!src_y || !plane_i || !plane_h || !plane_v || !plane_hv || !jobs || !results || n < 0) return -1;
  if (w < 8 || h < 8 || margin < 10 || plane_pitch < w + 2 * margin || src_pitch < w) return -1;
  if (n == 0) return 0;
  HevcSearch<uint8_t> S{src_y, src_pitch, w, h, margin, qpel ? 1 : 0, {plane_i, plane_h, plane_v, plane_hv},
                        plane_pitch, 0};
  launch_early(hevc_me_kernel<uint8_t>, (unsigned)(n / 8 + 1), 128, 0, (cudaStream_t)stream, S, jobs, n, results);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_motion_search_10(const uint16_t* src_y, int src_pitch, int w, int h, const uint16_t* plane_i,
                                  const uint16_t* plane_h, const uint16_t* plane_v, const uint16_t* plane_hv,
                                  int plane_pitch, int margin, int qpel, const b200enc_hevc_me_job_t* jobs, int n,
                                  b200enc_hevc_me_result_t* results, void* stream) {
  if (!src_y || !plane_i || !plane_h || !plane_v || !plane_hv || !jobs || !results || n < 0) return -1;
  if (w < 8 || h < 8 || margin < 10 || plane_pitch < w + 2 * margin || src_pitch < w) return -1;
  if (n == 0) return 0;
  HevcSearch<uint16_t> S{src_y, src_pitch, w, h, margin, qpel ? 1 : 0, {plane_i, plane_h, plane_v, plane_hv},
                         plane_pitch, 2};
  launch_early(hevc_me_kernel<uint16_t>, (unsigned)(n / 8 + 1), 128, 0, (cudaStream_t)stream, S, jobs, n, results);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_choose_luma_mode(const uint8_t* src_y, int src_pitch, const uint8_t* recon_y, int recon_pitch,
                                  int width, int height, const int* jobs, int n, int* modes, uint8_t* preds,
                                  void* stream) {
  if (!src_y || !recon_y || !jobs || !modes || !preds || n < 0 || width < 4 || height < 4) return -1;
  if (!aligned16(preds) || src_pitch < width || recon_pitch < width) return -1;
  if (n == 0) return 0;
  launch_early(hevc_intra4_kernel<uint8_t>, (n + 127) / 128, 128, 0, (cudaStream_t)stream, src_y, src_pitch, recon_y,
               recon_pitch, width, height, jobs, n, modes, preds, 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int b200enc_hevc_choose_luma_mode_10(const uint16_t* src_y, int src_pitch, const uint16_t* recon_y, int recon_pitch,
                                     int width, int height, const int* jobs, int n, int* modes, uint16_t* preds,
                                     void* stream) {
  if (!src_y || !recon_y || !jobs || !modes || !preds || n < 0 || width < 4 || height < 4) return -1;
  if (!aligned16(preds) || src_pitch < width || recon_pitch < width) return -1;
  if (n == 0) return 0;
  launch_early(hevc_intra4_kernel<uint16_t>, (n + 127) / 128, 128, 0, (cudaStream_t)stream, src_y, src_pitch, recon_y,
               recon_pitch, width, height, jobs, n, modes, preds, 10);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// The same planes from and to host memory, for a host encoder that keeps its
// reconstruction and search planes in host buffers (the reference's
// hevc_encoder_t: prev_recon_y, hpel[4], hpel_stride). Each calling thread
// keeps its own device workspace and stream, grown to the largest picture
// it has seen; the call returns when the four planes are in `planes`.
namespace {
struct HpelWork {
  cudaStream_t st = nullptr;
  void* buf = nullptr;
  size_t bytes = 0;
  ~HpelWork() {
    if (buf) cudaFree(buf);
    if (st) cudaStreamDestroy(st);
  }
};
thread_local HpelWork t_hpel;
}  // namespace

int b200enc_hevc_build_hpel_host(const void* recon, int w, int h, int bit_depth, int margin, void* const planes[4],
                                 int plane_stride) {
  if (!recon || !planes || w <= 0 || h <= 0 || (bit_depth != 8 && bit_depth != 10)) return -1;
  if (margin < 0 || margin > 256 || plane_stride < w + 2 * margin) return -1;
  for (int i = 0; i < 4; ++i)
    if (!planes[i]) return -1;
  const size_t bps = bit_depth == 8 ? 1 : 2;
  const int rows = h + 2 * margin;
  const size_t rec_bytes = (size_t)w * h * bps, plane_bytes = (size_t)plane_stride * rows * bps;
  const size_t need = ((rec_bytes + 255) & ~(size_t)255) + 4 * ((plane_bytes + 255) & ~(size_t)255);
  HpelWork& wk = t_hpel;
  if (!wk.st && cudaStreamCreateWithFlags(&wk.st, cudaStreamNonBlocking) != cudaSuccess) return -1;
  if (wk.bytes < need) {
    if (wk.buf) cudaFree(wk.buf);
    wk.buf = nullptr;
    wk.bytes = 0;
    if (cudaMalloc(&wk.buf, need) != cudaSuccess) return -1;
    wk.bytes = need;
  }
  uint8_t* d = static_cast<uint8_t*>(wk.buf);
  uint8_t* drec = d;
  uint8_t* dp[4];
  for (int i = 0; i < 4; ++i) dp[i] = d + ((rec_bytes + 255) & ~(size_t)255) + i * ((plane_bytes + 255) & ~(size_t)255);
  if (cudaMemcpyAsync(drec, recon, rec_bytes, cudaMemcpyHostToDevice, wk.st) != cudaSuccess) return -1;
  const int rc = bit_depth == 8
                     ? b200enc_hevc_build_hpel(drec, w, w, h, margin, dp[0], dp[1], dp[2], dp[3], plane_stride, wk.st)
                     : b200enc_hevc_build_hpel_10(reinterpret_cast<const uint16_t*>(drec), w, w, h, margin,
                                                  reinterpret_cast<uint16_t*>(dp[0]),
                                                  reinterpret_cast<uint16_t*>(dp[1]),
                                                  reinterpret_cast<uint16_t*>(dp[2]),
                                                  reinterpret_cast<uint16_t*>(dp[3]), plane_stride, wk.st);
  if (rc != 0) return -1;
  for (int i = 0; i < 4; ++i)
    if (cudaMemcpyAsync(planes[i], dp[i], plane_bytes, cudaMemcpyDeviceToHost, wk.st) != cudaSuccess) return -1;
  return cudaStreamSynchronize(wk.st) == cudaSuccess ? 0 : -1;
}

int b200enc_pin_host(void* ptr, size_t bytes) {
  if (!ptr || bytes == 0) return -1;
  if (cudaHostRegister(ptr, bytes, cudaHostRegisterDefault) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return 0;
}

int b200enc_unpin_host(void* ptr) {
  if (!ptr) return -1;
  if (cudaHostUnregister(ptr) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return 0;
}

}  // extern "C"
