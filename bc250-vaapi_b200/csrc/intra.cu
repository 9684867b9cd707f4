// intra.cu - I-frame intra wavefront as ONE persistent kernel.
//
// Reference: A1/shaders/intra_wavefront.comp:398-756, dispatched once per
// anti-diagonal with a barrier between dispatches (A1/src/gpu_compute.c:
// 3238-3249: 187 dispatches for a 1080p frame). An I16x16 macroblock needs
// only its left, top and top-left neighbours' reconstruction, and only inside
// its slice; luma and chroma (always DC-predicted) need nothing of each other.
//
// The frame's time is the dependent chain: mbw macroblocks along a row plus a
// macroblock and a handoff for each of mbh rows. So:
//   * a plane's row is one warp, free of barriers: a lane
//     pair holds a 4x4 block (rows 0 and 3, rows 1 and 2, so that every
//     butterfly of the transforms is one exchange per column), predictions,
//     sums and the DC Hadamards are shuffles and redux; a macroblock's AC
//     inverse runs while its DC terms are still in the Hadamard (they are
//     added last: the inverse transform carries a DC unchanged to all samples);
//   * a CTA owns kIRows consecutive rows of luma or of chroma, a warp to each
//     of the SM's schedulers (a row is bound by its own ~550 instructions per
//     macroblock as much as by their latency: luma and chroma rows sharing
//     the schedulers ran 1.14 us a macroblock), taken by ticket (only running
//     CTAs take tickets, so no wait can deadlock whatever the grid size). It
//     hands bottom lines from row to row through shared memory: a ring of 32
//     macroblocks per row and a progress word;
//   * a loader warp brings the lines above the CTA's first row from memory as
//     the CTA above publishes them, a publisher warp stores, fences and
//     publishes those below its last row; no row warp fences or touches a
//     global flag;
//   * a macroblock whose top neighbour is in another slice waits for nothing,
//     so slices that start a row run side by side. One that starts inside a row
//     does not: the row's warp reaches it after the end of the slice before, whose
//     rows it has waited for (1280x720 in four slices of 11.25 rows 167 us, in one
//     171; 1920x1080 in four of 17 rows 190, in one 253).
// Waits are bounded: on timeout a warp records the error in the scratch and
// the CTA leaves; every waiter gives up as soon as it sees a recorded error.
//
// A row walks at ~1 us a macroblock (its warp's instructions and shuffles), a
// group's handoff through memory adds ~2.8 us every fourth row. A row per CTA
// of three compute warps meeting at seven barriers per macroblock (3.3 us),
// every row handing over through memory, took, in us: 1920x1080 586 (one
// slice) and 688 (four), 1280x720 384 and 454, 640x480 222 and 257, 176x144 67
// and 75; now 253 and 190, 171 and 167, 96 and 80, 29 and 29.
#include "b200enc_internal.h"
#include "common.cuh"

namespace b200enc {

constexpr int kIRows = 4;   // macroblock rows per CTA, one warp each (an SM has four schedulers)
constexpr int kIRing = 32;  // macroblocks of a line kept in shared memory
constexpr int kIWarps = kIRows + 2;

struct IShared {
  // bottom lines: [0] the row above the CTA's first, [r + 1] its row r (luma, or NV12 pairs)
  alignas(16) uint8_t line[kIRows + 1][kIRing * 16];
  int prog[kIRows + 1];  // macroblocks of each line written
  int published;         // of the last row's line
  int ticket;
  int abort_flag;
};

__device__ __forceinline__ int shared_acquire(const int& w) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];"
               : "=r"(v)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&w)))
               : "memory");
  return v;
}
__device__ __forceinline__ void shared_release(int& w, int v) {
  asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(&w))),
               "r"(v)
               : "memory");
}

// Four samples -> a word, clipped to 0..255.
__device__ __forceinline__ uint32_t pack_clip(int x0, int x1, int x2, int x3) {
  uint32_t hi, d;
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(x3), "r"(x2), "r"(0u));
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(x1), "r"(x0), "r"(hi));
  return d;
}
__device__ __forceinline__ int byte_of(uint32_t w, int k) { return (int)((w >> (8 * k)) & 255u); }
__device__ __forceinline__ uint32_t sad4(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Quantiser of one lane's half block: coefficient rows (0, 2) (h = 0) or
// (1, 3) (h = 1); even and odd columns differ in their position class.
struct HalfQ {
  int mfe, mfo, ve, vo;      // MF and 16 V of the even and odd columns
  int f, f_shift;            // AC rounding
  int dq_add, dq_l, dq_r;    // dequantisation: (level * 16 V + add) << l >> r
  int ls, per;               // DC level scale
  uint32_t ls_inv;           // ceil(2^32 / ls): exact quotients below 2^32 / 288
  int dc_add, dc_l, dc_r;    // DC quantisation: ((|v| << l) + add) >> r, then / ls
};
__device__ __forceinline__ HalfQ half_q(int qp, int h) {
  const QP q = make_qp(qp, true);
  HalfQ r;
  r.mfe = h ? q.mf2 : q.mf0;
  r.mfo = h ? q.mf1 : q.mf2;
  r.ve = 16 * (h ? q.v2 : q.v0);
  r.vo = 16 * (h ? q.v1 : q.v2);
  r.f = q.f;
  r.f_shift = q.f_shift;
  r.dq_add = q.per >= 4 ? 0 : 1 << (3 - q.per);
  r.dq_l = q.per >= 4 ? q.per - 4 : 0;
  r.dq_r = q.per >= 4 ? 0 : 4 - q.per;
  r.per = q.per;
  r.ls = dc_ls(q.rem);
  r.ls_inv = 0xffffffffu / (uint32_t)r.ls + 1u;
  r.dc_l = q.per >= 5 ? 0 : 5 - q.per;
  r.dc_r = q.per >= 5 ? q.per - 5 : 0;
  r.dc_add = q.per >= 5 ? (r.ls << (q.per - 5)) >> 1 : r.ls >> 1;
  return r;
}
// quantize_dc (A1/src/encoder_h264.c:653-709): (num + den / 2) / den with den
// = ls << (per - 5), or num shifted left instead. floor((n >> k) / ls) is
// floor(n / (ls << k)), and the quotient by ls is exact by the reciprocal (n <
// 2^21: |v| < 2^16).
__device__ __forceinline__ int half_quant_dc(int v, const HalfQ& q) {
  const uint32_t n = (((uint32_t)abs(v) << q.dc_l) + (uint32_t)q.dc_add) >> q.dc_r;
  const int l = (int)__umulhi(n, q.ls_inv);
  return v < 0 ? -l : l;
}

// A 4x4 block on a lane pair. a, b: the residual's (or prediction error's)
// rows 0 and 3 (h = 0) or 1 and 2 (h = 1); on return a, b: coefficient rows 0
// and 2, or 1 and 3 (columns first; the forward transform is exact, so the
// order is free).
__device__ __forceinline__ void half_forward(int (&a)[4], int (&b)[4], int h) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int u = a[i] + b[i], w = a[i] - b[i];  // h = 0: a0, a3; h = 1: a1, a2
    const int o = __shfl_xor_sync(0xffffffffu, h ? u : w, 1);
    a[i] = h ? 2 * o + w : u + o;
    b[i] = h ? o - 2 * w : u - o;
  }
  fwd4(a[0], a[1], a[2], a[3]);
  fwd4(b[0], b[1], b[2], b[3]);
}
// Inverse of dequantised coefficient rows (0, 2) or (1, 3): rows first
// (reconstruct.comp:162-177), then columns; sample rows (0, 3) or (1, 2)
// before the final (+ 32) >> 6.
__device__ __forceinline__ void half_inverse_columns(int (&a)[4], int (&b)[4], int h) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int z0 = h ? (a[i] >> 1) - b[i] : a[i] + b[i];   // h = 0: z0; h = 1: z2
    const int z1 = h ? a[i] + (b[i] >> 1) : a[i] - b[i];   // h = 0: z1; h = 1: z3
    const int o = __shfl_xor_sync(0xffffffffu, z1, 1);     // z3 to h = 0, z1 to h = 1
    const int p = h ? o : z0, q = h ? z0 : o;
    a[i] = p + q;
    b[i] = p - q;
  }
}
__device__ __forceinline__ void half_inverse(int (&a)[4], int (&b)[4], int h) {
  inv4(a[0], a[1], a[2], a[3]);
  inv4(b[0], b[1], b[2], b[3]);
  half_inverse_columns(a, b, h);
}

// AC levels of the lane's eight coefficients (position 0 of a block belongs to
// the DC path), their nonzero bits in raster positions, and the dequantised
// values in place.
__device__ __forceinline__ uint32_t half_quant(int (&a)[4], int (&b)[4], int h, const HalfQ& q, uint2& la, uint2& lb) {
  uint32_t nz = 0;
  int l[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = i < 4 ? a[i & 3] : b[i & 3];
    const int m = (i & 1) ? q.mfo : q.mfe;
    int v = (abs(c) * m + q.f) >> q.f_shift;
    if (i == 0) v = h ? v : 0;
    nz |= (v != 0 ? 1u : 0u) << (i < 4 ? i : i + 4);  // rows f and f + 2
    l[i] = c < 0 ? -v : v;
  }
  la = make_uint2((uint32_t)(uint16_t)l[0] | ((uint32_t)l[1] << 16), (uint32_t)(uint16_t)l[2] | ((uint32_t)l[3] << 16));
  lb = make_uint2((uint32_t)(uint16_t)l[4] | ((uint32_t)l[5] << 16), (uint32_t)(uint16_t)l[6] | ((uint32_t)l[7] << 16));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int d = ((l[i] * ((i & 1) ? q.vo : q.ve) + q.dq_add) << q.dq_l) >> q.dq_r;
    if (i < 4) a[i] = d;
    else b[i - 4] = d;
  }
  return h ? nz << 4 : nz;
}

// Tickets: word 0 of the scratch counts luma rows, kIRows at a time, word 3
// chroma rows; CTAs start on luma or chroma by their parity and go over to the
// other plane when theirs is done. BATCH: bt.ticket[0] and [1] count the row
// groups of every stream of a batch that codes an I frame (bt.i_rows counts
// each stream's groups of kIRows rows); a group waits on its own stream's
// progress words (that stream's scratch). Tickets are taken in order and a
// group only waits on an earlier group of its stream and plane, so every wait
// is on a group some running CTA owns.
template <bool BATCH>
__global__ void __launch_bounds__(32 * kIWarps, 1)
    i_frame_kernel(const uint8_t* __restrict__ cur_y_, const uint8_t* __restrict__ cur_uv_, int cur_pitch_, Geo g_, int qp_,
                   int num_slices_, int16_t* __restrict__ levels_, int32_t* __restrict__ dc_, uint32_t* __restrict__ nzm_,
                   uint32_t* __restrict__ pred_mode_, MV* __restrict__ mvs_, uint8_t* rec_y_, uint8_t* rec_uv_,
                   int rec_pitch_, uint32_t* scratch_, uint32_t max_wait, int flags_, BatchTab bt) {
  __shared__ IShared s;
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  bool is_luma = (blockIdx.x & 1) == 0;

  for (int planes = 0; planes < 2;) {
    if (tid == 0) {
      s.ticket = (int)(BATCH ? atomicAdd(bt.ticket + (is_luma ? 0 : 1), 1u)
                             : atomicAdd(scratch_ + (is_luma ? 0 : 3), (uint32_t)kIRows));
      s.abort_flag = 0;
      s.published = 0;
    }
    if (tid <= kIRows) s.prog[tid] = 0;
    __syncthreads();
    const uint8_t *cur_y = cur_y_, *cur_uv = cur_uv_;
    int cur_pitch = cur_pitch_, qp = qp_, num_slices = num_slices_, rec_pitch = rec_pitch_, flags = flags_;
    Geo g = g_;
    int16_t* levels = levels_;
    int32_t* dc = dc_;
    uint32_t *nzm = nzm_, *pred_mode = pred_mode_, *scratch = scratch_;
    MV* mvs = mvs_;
    uint8_t *rec_y = rec_y_, *rec_uv = rec_uv_;
    int row0;
    if (BATCH) {
      const int grp = s.ticket;
      if (grp >= bt.i_rows.total()) {
        is_luma = !is_luma;
        ++planes;
        __syncthreads();  // the ticket has been read
        continue;
      }
      const int k = bt.i_rows.find(grp);
      const BatchStream& st = bt.i_rows.stream(k);
      row0 = (grp - bt.i_rows.prefix[k]) * kIRows;
      g = st.g;
      cur_y = st.cur_y;
      cur_uv = st.cur_uv;
      cur_pitch = st.cur_pitch;
      qp = st.qp;
      num_slices = st.num_slices;
      flags = st.intra_flags;
      levels = st.levels;
      dc = st.dc;
      nzm = st.nz;
      pred_mode = st.pred_mode;
      mvs = st.mv;
      rec_y = st.rec_y;
      rec_uv = st.rec_uv;
      rec_pitch = st.rec_pitch;
      scratch = st.scr_intra;
    } else {
      row0 = s.ticket;
      if (row0 >= g.mbh) {
        is_luma = !is_luma;
        ++planes;
        __syncthreads();
        continue;
      }
    }
    const int rows = min(kIRows, g.mbh - row0);
    const Scratch sc{scratch};
    uint32_t* const flags_of = sc.progress(0) + (is_luma ? 0 : g.mbh);  // the plane's row progress words
    const uint32_t total = (uint32_t)(g.mbw * g.mbh);
    const uint64_t budget = (uint64_t)max_wait * 1000u;  // max_wait in microseconds
    auto vload = [](const int& w) { return *reinterpret_cast<const volatile int*>(&w); };
    // Bounded wait of a whole warp until a shared word has reached `need`:
    // false (on every lane) when the wait gave up (error recorded) or another
    // one did.
    auto wait_shared = [&](const int& w, int need, uint32_t where) -> bool {
      if (__all_sync(full, shared_acquire(w) >= need)) return true;
      const uint64_t t0 = global_ns();
      for (uint32_t it = 0;; ++it) {
        if (__all_sync(full, shared_acquire(w) >= need)) return true;
        bool stop = vload(s.abort_flag) != 0;
        if ((it & 63) == 63 && global_ns() - t0 > budget) {
          if (lane == 0 && atomicCAS(sc.err(), 0u, kErrWaitTimeout) == 0u) atomicExch(sc.err_detail(), where);
          stop = true;
        }
        if (__any_sync(full, stop)) {
          if (lane == 0) *reinterpret_cast<volatile int*>(&s.abort_flag) = 1;
          return false;
        }
      }
    };
    const int rmx = g.RW - 1, rmy = g.RH - 1, cmx = g.RW / 2 - 1, cmy = g.RH / 2 - 1;
    const bool corner_check = (flags & B200ENC_INTRA_CORNER_CHECK) != 0;
    auto slice_first = [&](uint32_t sl) { return (uint32_t)(((uint64_t)sl * total) / (uint32_t)num_slices); };

    if (wid < kIRows) {
      const int r = wid;
      const int mby = row0 + r;
      if (r < rows) {
        // the slice of the row's next macroblock: [ss, se)
        uint32_t sl = slice_of((uint32_t)(mby * g.mbw), total, (uint32_t)num_slices);
        uint32_t ss = slice_first(sl), se = slice_first(sl + 1);
        const int h = lane & 1;
        const bool src_vec = ((cur_pitch & 3) == 0) && ((reinterpret_cast<uintptr_t>(cur_y) & 3) == 0) &&
                             ((reinterpret_cast<uintptr_t>(cur_uv) & 3) == 0);
        const int& prog_in = s.prog[r];
        int& prog_out = s.prog[r + 1];
        // who reads this row's line: the next row, or the publisher (none below the picture's last row)
        const bool has_reader = mby + 1 < g.mbh;
        const int& prog_reader = r + 1 < rows ? s.prog[r + 2] : s.published;
        const uint8_t* line_in = s.line[r];
        uint8_t* line_out = s.line[r + 1];
        // The row's per-macroblock frame: slice bookkeeping, `before` (what
        // needs nothing from above), the waits, `body` (up to the line the
        // next row reads), the handoff, then `store` (all global accesses: the
        // release waits for those in flight, so they follow it and have a
        // macroblock's time to finish).
        auto walk = [&](auto&& before, auto&& body, auto&& store) {
          for (int mbx = 0; mbx < g.mbw; ++mbx) {
            const uint32_t mb = (uint32_t)(mby * g.mbw + mbx);
            while (mb >= se) {  // (slices of no macroblock are passed over)
              ++sl;
              ss = se;
              se = slice_first(sl + 1);
            }
            const bool top_av = mby > 0 && mb - (uint32_t)g.mbw >= ss;
            const bool left_av = mbx > 0 && mb - 1u >= ss;
            // Plane also predicts from the top-left sample; with the corner
            // check it needs the top-left macroblock in this slice as well
            // (the reference shader checks only top and left)
            const bool plane_av = top_av && left_av && (!corner_check || mb - (uint32_t)g.mbw - 1u >= ss);
            // without it the corner may come from above a macroblock of another slice
            const bool need = top_av || (!corner_check && mby > 0 && mbx + 1 < g.mbw && mb + 1u - (uint32_t)g.mbw >= (mb + 1u >= se ? se : ss));
            before(mbx, left_av);
            if (need && !wait_shared(prog_in, mbx + 1, mb)) return;
            // ring space for the next eight macroblocks' lines: macroblock m
            // replaces m - kIRing
            if ((mbx & 7) == 0 && has_reader && mbx + 8 > kIRing && !wait_shared(prog_reader, mbx + 8 - kIRing, mb)) return;
            body(mbx, top_av, left_av, plane_av, need);
            __syncwarp();
            if (lane == 31) shared_release(prog_out, mbx + 1);
            store(mbx, (int)mb);
          }
        };

        if (is_luma) {
          const int b = lane >> 1, bx = b & 3, by = b >> 2;
          const int ra = 4 * by + (h ? 1 : 0), rb = 4 * by + (h ? 2 : 3);  // the lane's sample rows
          const HalfQ q = half_q(qp, h);
          const int Y = mby * 16;
          const uint8_t* pa_row = cur_y + (size_t)clampi(Y + ra, 0, g.H - 1) * cur_pitch;
          const uint8_t* pb_row = cur_y + (size_t)clampi(Y + rb, 0, g.H - 1) * cur_pitch;
          uint32_t sa, sb, na = 0, nb = 0;  // this and the next macroblock's source
          auto src_word = [&](const uint8_t* rp, int gx) -> uint32_t {
            if (src_vec && gx + 4 <= g.W) return __ldg(reinterpret_cast<const uint32_t*>(rp + gx));
            uint32_t w = 0;
            for (int k = 0; k < 4; ++k) w |= (uint32_t)__ldg(rp + clampi(gx + k, 0, g.W - 1)) << (8 * k);
            return w;
          };
          sa = src_word(pa_row, 4 * bx);
          sb = src_word(pb_row, 4 * bx);
          if (g.mbw > 1) {
            na = src_word(pa_row, 16 + 4 * bx);
            nb = src_word(pb_row, 16 + 4 * bx);
          }
          uint8_t* out_a = rec_y + (size_t)(Y + ra) * rec_pitch + 4 * bx;
          uint8_t* out_b = rec_y + (size_t)(Y + rb) * rec_pitch + 4 * bx;
          const size_t mb0 = (size_t)mby * g.mbw;
          uint2* lv_out = reinterpret_cast<uint2*>(levels + mb0 * 384 + b * 16) + h;
          uint32_t* nz_out = nzm + mb0 * 24 + b;
          int32_t* dc_out = dc + mb0 * 24 + b;
          uint2 lva_, lvb_;
          uint32_t nz_;
          int raw_, mode_;
          const bool clamp_l = Y + 15 > rmy;  // rows past the clamp limit read its last row
          // lane and register (0: rows 0 and 1 of a block, 1: rows 2 and 3) holding the left sample of a row
          auto left_lane = [&](int row) { const int c = clampi(rmy - Y, 0, row), k = c & 3; return (((c >> 2) * 4 + 3) << 1) | ((k == 1 || k == 2) ? 1 : 0); };
          auto left_reg = [&](int row) { return (clampi(rmy - Y, 0, row) & 3) >> 1; };
          const int lla = left_lane(ra), llb = left_lane(rb), lra = left_reg(ra), lrb = left_reg(rb);
          const int l15_lane = left_lane(15), l15_reg = left_reg(15);
          uint32_t reca = 0x80808080u, recb = 0x80808080u;
          int prev_t15 = 128;
          const uint32_t wt = 0x04030201u + 0x04040404u * (uint32_t)bx;  // x + 1 of the lane's four columns
          int la, lb, l15;
          uint32_t ls;
          auto before = [&](int mbx, bool) {
            // left: this warp's own previous macroblock
            uint32_t va = __shfl_sync(full, reca, lla), vb = __shfl_sync(full, recb, llb);
            if (clamp_l) {
              const uint32_t va1 = __shfl_sync(full, recb, lla), vb0 = __shfl_sync(full, reca, llb);
              va = lra ? va1 : va;
              vb = lrb ? vb : vb0;
            }
            const uint32_t l15w = __shfl_sync(full, l15_reg ? recb : reca, l15_lane);
            la = (int)(va >> 24);  // 128 at the picture's edge: reca and recb start as 0x80s
            lb = (int)(vb >> 24);
            l15 = (int)(l15w >> 24);
            ls = __reduce_add_sync(full, bx == 0 ? (((uint32_t)(la * (ra + 1) + lb * (rb + 1))) << 16) + (uint32_t)(la + lb) : 0u);
          };
          auto body = [&](int mbx, bool top_av, bool left_av, bool plane_av, bool need) {
            const int X = mbx * 16;
            // ---- the line above, its sums --------------------------------------
            uint32_t tw = 0x80808080u;
            const int corner = mby > 0 && mbx > 0 ? prev_t15 : 128;
            prev_t15 = 128;
            if (need) {
              const uint8_t* lp = line_in + (mbx & (kIRing - 1)) * 16;
              tw = *reinterpret_cast<const uint32_t*>(lp + 4 * bx);
              // (the line's own last byte: the clamp applies to what this macroblock reads, not to the corner)
              prev_t15 = (int)lp[15];
              if (X + 15 > rmx) {  // columns past the clamp limit read its last one
                tw = 0;
                for (int k = 0; k < 4; ++k) tw |= (uint32_t)lp[clampi(rmx - X, 0, 4 * bx + k)] << (8 * k);
              }
            }
            const int t15 = (int)(__shfl_sync(full, tw, 6) >> 24);
            const uint32_t ts = __reduce_add_sync(full, lane < 8 && !h ? (__dp4a(tw, wt, 0u) << 16) + __dp4a(tw, 0x01010101u, 0u) : 0u);
            const int st = (int)(ts & 0xffffu), sl_ = (int)(ls & 0xffffu);
            // ---- the I16x16 candidates (intra_wavefront.comp:454-476) --------
            int dcv = 128;
            if (top_av && left_av) dcv = (st + sl_ + 16) >> 5;
            else if (top_av) dcv = (st + 8) >> 4;
            else if (left_av) dcv = (sl_ + 8) >> 4;
            const uint32_t dcw = (uint32_t)dcv * 0x01010101u;
            const uint32_t ha = (uint32_t)la * 0x01010101u, hb = (uint32_t)lb * 0x01010101u;
            // sum of (x - 7) T[x] - 8 corner, of (y - 7) L[y] - 8 corner
            const int hs = (int)(ts >> 16) - 8 * st - 8 * corner, vs = (int)(ls >> 16) - 8 * sl_ - 8 * corner;
            const int pb = (5 * hs + 32) >> 6, pc = (5 * vs + 32) >> 6, pa = 16 * (l15 + t15);
            const int ba = pa + pb * (4 * bx - 7) + pc * (ra - 7) + 16, bb = ba + pc * (rb - ra);
            const uint32_t pla = pack_clip(ba >> 5, (ba + pb) >> 5, (ba + 2 * pb) >> 5, (ba + 3 * pb) >> 5);
            const uint32_t plb = pack_clip(bb >> 5, (bb + pb) >> 5, (bb + 2 * pb) >> 5, (bb + 3 * pb) >> 5);
            // two 16-bit sums to a redux: a SAD is at most 65280
            const uint32_t s01 = __reduce_add_sync(full, sad4(sa, dcw, sad4(sb, dcw, 0u)) + (sad4(sa, tw, sad4(sb, tw, 0u)) << 16));
            const uint32_t s23 = __reduce_add_sync(full, sad4(sa, ha, sad4(sb, hb, 0u)) + (sad4(sa, pla, sad4(sb, plb, 0u)) << 16));
            uint32_t best = s01 & 0xffffu;
            int mode = 2;
            uint32_t pwa = dcw, pwb = dcw;
            if (top_av && (s01 >> 16) < best) { best = s01 >> 16; mode = 0; pwa = pwb = tw; }
            if (left_av && (s23 & 0xffffu) < best) { best = s23 & 0xffffu; mode = 1; pwa = ha; pwb = hb; }
            if (plane_av && (s23 >> 16) < best) { mode = 3; pwa = pla; pwb = plb; }
            // ---- residual, transform, levels ------------------------------------
            int xa[4], xb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              xa[i] = byte_of(sa, i) - byte_of(pwa, i);
              xb[i] = byte_of(sb, i) - byte_of(pwb, i);
            }
            half_forward(xa, xb, h);
            const int raw = xa[0];  // h = 0: the block's DC term
            // The luma DC transform (A1/src/encoder_h264.c:711-730), out[i][k] =
            // sum_ab h_k(a) h_i(b) in[a][b] with h the Walsh rows in sequency
            // order: natural butterflies over the block bits of the lane leave
            // it permuted, and the inverse's butterflies on that order come out
            // at the blocks' own lanes (h is symmetric). Integer sums: exact in
            // any order.
            int v = raw;
#pragma unroll
            for (int m = 2; m <= 16; m <<= 1) {
              const int o = __shfl_xor_sync(full, v, m);
              v = (lane & m) ? o - v : v + o;
            }
            // (the AC half of the block fills the shuffles' latency)
            v = half_quant_dc((v + 1) >> 1, q);
            int o1 = __shfl_xor_sync(full, v, 2);
            uint2 lva, lvb;
            const uint32_t nz = half_quant(xa, xb, h, q, lva, lvb);
            v = (lane & 2) ? o1 - v : v + o1;
            o1 = __shfl_xor_sync(full, v, 4);
            inv4(xa[0], xa[1], xa[2], xa[3]);
            v = (lane & 4) ? o1 - v : v + o1;
            o1 = __shfl_xor_sync(full, v, 8);
            inv4(xb[0], xb[1], xb[2], xb[3]);
            v = (lane & 8) ? o1 - v : v + o1;
            o1 = __shfl_xor_sync(full, v, 16);
            half_inverse_columns(xa, xb, h);
            v = (lane & 16) ? o1 - v : v + o1;
            v = q.per >= 6 ? (v * q.ls) << (q.per - 6) : (v * q.ls + (1 << (5 - q.per))) >> (6 - q.per);
            v = __shfl_sync(full, v, lane & ~1) + 32;
            reca = pack_clip(byte_of(pwa, 0) + ((xa[0] + v) >> 6), byte_of(pwa, 1) + ((xa[1] + v) >> 6),
                             byte_of(pwa, 2) + ((xa[2] + v) >> 6), byte_of(pwa, 3) + ((xa[3] + v) >> 6));
            recb = pack_clip(byte_of(pwb, 0) + ((xb[0] + v) >> 6), byte_of(pwb, 1) + ((xb[1] + v) >> 6),
                             byte_of(pwb, 2) + ((xb[2] + v) >> 6), byte_of(pwb, 3) + ((xb[3] + v) >> 6));
            if (by == 3 && !h) *reinterpret_cast<uint32_t*>(line_out + (mbx & (kIRing - 1)) * 16 + 4 * bx) = recb;
            raw_ = raw;
            nz_ = nz;
            lva_ = lva;
            lvb_ = lvb;
            mode_ = mode;
          };
          auto store = [&](int mbx, int mb) {
            const int X = mbx * 16;
            sa = na;
            sb = nb;
            if (mbx + 2 < g.mbw) {
              na = src_word(pa_row, X + 32 + 4 * bx);
              nb = src_word(pb_row, X + 32 + 4 * bx);
            }
            nz_ |= __shfl_xor_sync(full, nz_, 1);
            lv_out[0] = lva_;  // coefficient rows h and h + 2 (four levels to a uint2)
            lv_out[2] = lvb_;
            lv_out += 96;
            if (!h) {
              nz_out[0] = nz_;
              dc_out[0] = raw_;
            }
            nz_out += 24;
            dc_out += 24;
            if (X + 16 <= g.RW) {
              if (Y + ra <= rmy) *reinterpret_cast<uint32_t*>(out_a) = reca;
              if (Y + rb <= rmy) *reinterpret_cast<uint32_t*>(out_b) = recb;
            } else {
              for (int k = 0; k < 4 && X + 4 * bx + k < g.RW; ++k) {
                if (Y + ra <= rmy) out_a[k] = (uint8_t)byte_of(reca, k);
                if (Y + rb <= rmy) out_b[k] = (uint8_t)byte_of(recb, k);
              }
            }
            out_a += 16;
            out_b += 16;
            if (lane == 0) {
              pred_mode[mb] = (uint32_t)mode_;  // chroma mode bits 2-3 = 0 (DC)
              mvs[mb] = MV{0, 0, 0u, 0u};
            }
          };
          walk(before, body, store);
        } else {
          // chroma: lanes 0..15 hold the eight blocks (Cb 0..3, Cr 4..7); the
          // other lanes shadow them and store nothing
          const int b = (lane >> 1) & 7, pl = b >> 2, bx = b & 1, by = (b >> 1) & 1;
          const bool act = lane < 16;
          const int ra = 4 * by + (h ? 1 : 0), rb = 4 * by + (h ? 2 : 3);
          const HalfQ q = half_q(chroma_qp(qp), h);
          const int Yc = mby * 8;
          const uint8_t* pa_row = cur_uv + (size_t)clampi(Yc + ra, 0, g.H / 2 - 1) * cur_pitch;
          const uint8_t* pb_row = cur_uv + (size_t)clampi(Yc + rb, 0, g.H / 2 - 1) * cur_pitch;
          const uint32_t pick = pl ? 0x7531u : 0x6420u;
          uint32_t sa, sb, na = 0, nb = 0;
          auto src_word = [&](const uint8_t* rp, int px) -> uint32_t {  // four samples of the plane from pair px
            if (src_vec && px + 4 <= g.W / 2)
              return __byte_perm(__ldg(reinterpret_cast<const uint32_t*>(rp + 2 * px)),
                                 __ldg(reinterpret_cast<const uint32_t*>(rp + 2 * px + 4)), pick);
            uint32_t w = 0;
            for (int k = 0; k < 4; ++k) w |= (uint32_t)__ldg(rp + 2 * clampi(px + k, 0, g.W / 2 - 1) + pl) << (8 * k);
            return w;
          };
          sa = src_word(pa_row, 4 * bx);
          sb = src_word(pb_row, 4 * bx);
          if (g.mbw > 1) {
            na = src_word(pa_row, 8 + 4 * bx);
            nb = src_word(pb_row, 8 + 4 * bx);
          }
          const bool clamp_l = Yc + 7 > cmy;
          auto left_lane = [&](int row) { const int c = clampi(cmy - Yc, 0, row), k = c & 3; return ((pl * 4 + (c >> 2) * 2 + 1) << 1) | ((k == 1 || k == 2) ? 1 : 0); };
          auto left_reg = [&](int row) { return (clampi(cmy - Yc, 0, row) & 3) >> 1; };
          const int lla = left_lane(ra), llb = left_lane(rb), lra = left_reg(ra), lrb = left_reg(rb);
          uint32_t reca = 0x80808080u, recb = 0x80808080u;
          uint2 lva, lvb, px;
          uint32_t nz = 0;
          int raw = 0;
          const int row = pl ? rb : ra;  // of the NV12 half row the lane stores
          int l;
          auto before = [&](int, bool) {
            // left: rows 4 by .. 4 by + 3 of the plane, two to a lane
            if (clamp_l) {
              const uint32_t a0 = __shfl_sync(full, reca, lla), a1 = __shfl_sync(full, recb, lla);
              const uint32_t b0 = __shfl_sync(full, reca, llb), b1 = __shfl_sync(full, recb, llb);
              l = (int)((lra ? a1 : a0) >> 24) + (int)((lrb ? b1 : b0) >> 24);
              l += __shfl_xor_sync(full, l, 1);
            } else {
              l = (int)(reca >> 24) + (int)(recb >> 24);
              l += __shfl_xor_sync(full, l, 1);
              l = __shfl_sync(full, l, lane | 2);  // the right-hand block's
            }
          };
          auto body = [&](int mbx, bool top_av, bool left_av, bool, bool need) {
            const int Xc = mbx * 8;
            int tsum = 0;
            if (need) {
              const uint8_t* lp = line_in + (mbx & (kIRing - 1)) * 16;
              uint32_t tw = __byte_perm(*reinterpret_cast<const uint32_t*>(lp + 8 * bx),
                                        *reinterpret_cast<const uint32_t*>(lp + 8 * bx + 4), pick);
              if (Xc + 7 > cmx) {
                tw = 0;
                for (int k = 0; k < 4; ++k) tw |= (uint32_t)lp[2 * clampi(cmx - Xc, 0, 4 * bx + k) + pl] << (8 * k);
              }
              tsum = (int)__dp4a(tw, 0x01010101u, 0u);
            }
            // DC predictors (intra_wavefront.comp:612-641): corner blocks from
            // both sides, the others from their own side first
            int pv;
            if (bx == by) pv = (top_av && left_av) ? (tsum + l + 4) >> 3 : (top_av ? (tsum + 2) >> 2 : (left_av ? (l + 2) >> 2 : 128));
            else if (bx) pv = top_av ? (tsum + 2) >> 2 : (left_av ? (l + 2) >> 2 : 128);
            else pv = left_av ? (l + 2) >> 2 : (top_av ? (tsum + 2) >> 2 : 128);
            int xa[4], xb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              xa[i] = byte_of(sa, i) - pv;
              xb[i] = byte_of(sb, i) - pv;
            }
            half_forward(xa, xb, h);
            raw = xa[0];
            int v = raw;  // 2x2 Hadamard over the plane's blocks, quantised, and back
#pragma unroll
            for (int m = 2; m <= 4; m <<= 1) {
              const int o = __shfl_xor_sync(full, v, m);
              v = (lane & m) ? o - v : v + o;
            }
            nz = half_quant(xa, xb, h, q, lva, lvb);
            v = half_quant_dc(v, q);
            half_inverse(xa, xb, h);
#pragma unroll
            for (int m = 2; m <= 4; m <<= 1) {
              const int o = __shfl_xor_sync(full, v, m);
              v = (lane & m) ? o - v : v + o;
            }
            v = q.per >= 5 ? (v * q.ls) << (q.per - 5) : (v * q.ls) >> (5 - q.per);
            v = __shfl_sync(full, v, lane & ~1) + 32;
            reca = pack_clip(pv + ((xa[0] + v) >> 6), pv + ((xa[1] + v) >> 6), pv + ((xa[2] + v) >> 6), pv + ((xa[3] + v) >> 6));
            recb = pack_clip(pv + ((xb[0] + v) >> 6), pv + ((xb[1] + v) >> 6), pv + ((xb[2] + v) >> 6), pv + ((xb[3] + v) >> 6));
            // NV12 rows: the Cb lane stores row ra, the Cr lane row rb
            const uint32_t o = __shfl_xor_sync(full, pl ? reca : recb, 8);
            const uint32_t cb = pl ? o : reca, cr = pl ? recb : o;
            px = make_uint2(__byte_perm(cb, cr, 0x5140), __byte_perm(cb, cr, 0x7362));
            if (act && row == 7) *reinterpret_cast<uint2*>(line_out + (mbx & (kIRing - 1)) * 16 + 8 * bx) = px;
          };
          auto store = [&](int mbx, int mb) {
            const int Xc = mbx * 8;
            sa = na;
            sb = nb;
            if (mbx + 2 < g.mbw) {
              na = src_word(pa_row, Xc + 16 + 4 * bx);
              nb = src_word(pb_row, Xc + 16 + 4 * bx);
            }
            nz |= __shfl_xor_sync(full, nz, 1);
            if (act) {
              uint2* lv = reinterpret_cast<uint2*>(levels + (size_t)mb * 384 + (16 + b) * 16);
              lv[h] = lva;
              lv[h + 2] = lvb;
              if (!h) {
                nzm[(size_t)mb * 24 + 16 + b] = nz;
                dc[(size_t)mb * 24 + 16 + b] = raw;
              }
              if (Yc + row <= cmy) {
                uint8_t* dst = rec_uv + (size_t)(Yc + row) * rec_pitch + 2 * (Xc + 4 * bx);
                if (Xc + 8 <= cmx + 1) *reinterpret_cast<uint2*>(dst) = px;
                else
                  for (int k = 0; k < 4 && Xc + 4 * bx + k <= cmx; ++k) {
                    const uint32_t w = k < 2 ? px.x : px.y;
                    dst[2 * k] = (uint8_t)byte_of(w, 2 * (k & 1));
                    dst[2 * k + 1] = (uint8_t)byte_of(w, 2 * (k & 1) + 1);
                  }
              }
            }
          };
          walk(before, body, store);
        }
      }
    } else if (wid == kIRows) {
      // ---- loader warp: the lines above the first row, as far as the CTA
      //      above has published them and a macroblock needs them ---------------
      if (row0 > 0) {
        const uint32_t* flag = flags_of + row0 - 1;
        const uint8_t* src = is_luma ? rec_y + (size_t)min(row0 * 16 - 1, rmy) * rec_pitch
                                     : rec_uv + (size_t)min(row0 * 8 - 1, cmy) * rec_pitch;
        int m = 0, seen = 0, chunk = -1;
        unsigned needs = 0;  // of the chunk's 32 macroblocks
        uint64_t t0 = global_ns();
        uint32_t it = 0;
        while (m < g.mbw) {
          if ((m >> 5) != chunk) {
            chunk = m >> 5;
            const int x = 32 * chunk + lane;
            bool need = false;
            if (x < g.mbw) {
              const uint32_t mb = (uint32_t)(row0 * g.mbw + x);
              need = mb - (uint32_t)g.mbw >= slice_first(slice_of(mb, total, (uint32_t)num_slices));
              if (!need && !corner_check && x + 1 < g.mbw)
                need = mb + 1u - (uint32_t)g.mbw >= slice_first(slice_of(mb + 1u, total, (uint32_t)num_slices));
            }
            needs = __ballot_sync(full, need);
          }
          // macroblocks of the chunk from m on that need no line or have one,
          // as far as the ring has space (line x replaces line x - kIRing)
          const int x = 32 * chunk + lane;
          const bool need = (needs >> lane) & 1u;
          const unsigned stop_at = __ballot_sync(full, x >= m && (x >= g.mbw || (need && x >= seen)));
          int n = (stop_at ? 32 * chunk + __ffs((int)stop_at) - 1 : 32 * chunk + 32) - m;
          n = min(n, __shfl_sync(full, shared_acquire(s.prog[1]), 0) + kIRing - m);
          // their lines and the next progress word in one round trip
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          const bool take = n > 0 && x >= m && x < m + n && need && 16 * x < rec_pitch;
          if (take) v = __ldcg(reinterpret_cast<const uint4*>(src + 16 * x));
          int now = (int)load_acquire(flag);
          if (n > 0) {
            if (take) *reinterpret_cast<uint4*>(s.line[0] + (x & (kIRing - 1)) * 16) = v;
            __syncwarp();
            m += n;
            if (lane == 0) shared_release(s.prog[0], m);
            t0 = global_ns();
          } else if ((++it & 15) == 0) {
            bool stop = load_acquire(sc.err()) != 0u || vload(s.abort_flag) != 0;
            if (!stop && global_ns() - t0 > budget) {
              if (lane == 0 && atomicCAS(sc.err(), 0u, kErrWaitTimeout) == 0u)
                atomicExch(sc.err_detail(), (uint32_t)(row0 * g.mbw + m));
              stop = true;
            }
            if (__any_sync(full, stop)) {
              if (lane == 0) *reinterpret_cast<volatile int*>(&s.abort_flag) = 1;
              break;
            }
          }
          seen = __shfl_sync(full, now, 0);
          __syncwarp();  // orders lane 0's acquire before every lane's loads
        }
      }
    } else {
      // ---- publisher warp: the last row's line to memory, fence, progress -------
      if (row0 + rows < g.mbh) {
        uint8_t* dst = is_luma ? rec_y + (size_t)((row0 + rows) * 16 - 1) * rec_pitch
                               : rec_uv + (size_t)((row0 + rows) * 8 - 1) * rec_pitch;
        // bytes of the row to store; none of a row past the clamp limit (a macroblock
        // wholly outside the limits is coded, as before, but not kept)
        const bool kept = is_luma ? (row0 + rows) * 16 - 1 <= rmy : (row0 + rows) * 8 - 1 <= cmy;
        const int limit = kept ? (is_luma ? g.RW : 2 * (cmx + 1)) : 0;
        int done = 0;
        while (done < g.mbw) {
          if (!wait_shared(s.prog[rows], done + 1, (uint32_t)((row0 + rows - 1) * g.mbw + done))) break;
          int avail = min(shared_acquire(s.prog[rows]), done + 32);
          avail = __shfl_sync(full, avail, 0);
          __syncwarp();  // orders lane 0's acquire before every lane's reads
          const int x = done + lane;
          if (x < avail) {
            const int slot = (x & (kIRing - 1)) * 16;
            if (16 * x + 16 <= limit) *reinterpret_cast<uint4*>(dst + 16 * x) = *reinterpret_cast<const uint4*>(s.line[rows] + slot);
            else
              for (int k = 0; k < 16 && 16 * x + k < limit; ++k) dst[16 * x + k] = s.line[rows][slot + k];
          }
          __threadfence();
          __syncwarp();
          done = avail;
          if (lane == 0) {
            store_release(flags_of + row0 + rows - 1, (uint32_t)done);
            shared_release(s.published, done);
          }
        }
      }
    }
    __syncthreads();  // the group's end: every warp
    if (s.abort_flag) return;
  }
}

}  // namespace b200enc

using namespace b200enc;

extern "C" size_t b200enc_wavefront_scratch_bytes(int mbh) { return scratch_words(mbh < 1 ? 1 : mbh) * sizeof(uint32_t); }

extern "C" int b200enc_wavefront_status(const void* scratch, void* stream) {
  if (!scratch) return -1;
  uint32_t e = 0;
  if (cudaMemcpyAsync(&e, (const uint32_t*)scratch + 1, sizeof(e), cudaMemcpyDeviceToHost, (cudaStream_t)stream) !=
      cudaSuccess)
    return -1;
  if (cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess) return -1;
  return e == 0 ? 0 : 1;
}

// Time budget of one progress wait before a wavefront CTA gives up.
static constexpr uint32_t kMaxWaitUs = 2000000u;  // 2 s

extern "C" int b200enc_i_frame_launch(const uint8_t* cur_y, const uint8_t* cur_uv, int cur_pitch, int W, int H,
                                      int RW, int RH, int qp, int num_slices, int16_t* levels, int32_t* dc,
                                      uint32_t* nz, uint32_t* pred_mode, void* mv, uint8_t* rec_y, uint8_t* rec_uv,
                                      int rec_pitch, uint32_t* scratch, int ctas, uint32_t max_wait, int flags,
                                      void* stream) {
  Geo g{W, H, RW, RH, (W + 15) / 16, (H + 15) / 16};
  const int groups = b200enc_i_frame_groups(g.mbh);
  if (ctas <= 0) ctas = b200enc_tuned(B200ENC_TUNE_INTRA_CTAS);
  if (ctas <= 0 || ctas > 2 * groups) ctas = 2 * groups;  // luma and chroma
  i_frame_kernel<false><<<ctas, 32 * kIWarps, 0, (cudaStream_t)stream>>>(
      cur_y, cur_uv, cur_pitch, g, qp, num_slices, levels, dc, nz, pred_mode, (MV*)mv, rec_y, rec_uv, rec_pitch, scratch,
      max_wait, flags, BatchTab{});
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Row groups (a CTA's rows) of a picture of mbh macroblock rows.
int b200enc_i_frame_groups(int mbh) { return (mbh + kIRows - 1) / kIRows; }

// The intra wavefront of every I-frame stream of a batch: `ctas` persistent
// CTAs over the row groups of bt.i_rows (each stream's scratch and both
// tickets of bt.ticket zeroed by the caller).
int b200enc_i_frame_batch_launch(const BatchTab& bt, int ctas, uint32_t max_wait, cudaStream_t st) {
  if (ctas <= 0) return 0;
  i_frame_kernel<true><<<2 * ctas, 32 * kIWarps, 0, st>>>(nullptr, nullptr, 0, Geo{}, 0, 1, nullptr, nullptr, nullptr, nullptr,
                                            nullptr, nullptr, nullptr, 0, nullptr, max_wait, 0, bt);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int b200enc_i_frame(const uint8_t* cur_y, const uint8_t* cur_uv, int cur_pitch, int W, int H, int RW,
                               int RH, int qp, int num_slices, int16_t* levels, int32_t* dc, uint32_t* nz,
                               uint32_t* pred_mode, void* mv, uint8_t* rec_y, uint8_t* rec_uv, int rec_pitch,
                               void* scratch, size_t scratch_bytes, int ctas, int flags, void* stream) {
  if (!cur_y || !cur_uv || !levels || !dc || !nz || !pred_mode || !mv || !rec_y || !rec_uv || !scratch) return -1;
  if (qp < 0 || qp > 51 || W <= 0 || H <= 0 || RW <= 1 || RH <= 1 || num_slices < 1) return -1;
  if ((rec_pitch & 15) || (((uintptr_t)rec_y) & 15) || (((uintptr_t)rec_uv) & 15) || (((uintptr_t)levels) & 15))
    return -1;
  const int mbh = (H + 15) / 16;
  if (scratch_bytes < b200enc_wavefront_scratch_bytes(mbh)) return -1;
  if (cudaMemsetAsync(scratch, 0, b200enc_wavefront_scratch_bytes(mbh), (cudaStream_t)stream) != cudaSuccess) return -1;
  return b200enc_i_frame_launch(cur_y, cur_uv, cur_pitch, W, H, RW, RH, qp, num_slices, levels, dc, nz, pred_mode, mv,
                                rec_y, rec_uv, rec_pitch, (uint32_t*)scratch, ctas, kMaxWaitUs, flags, stream);
}
