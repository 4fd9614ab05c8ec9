// sat_kernel_wd.cuh -- the warp-specialized tile loop for 1-byte and 4-byte inputs with 4-byte sums
// (configuration 5 for those pairs; 4-byte inputs also have 128-row tiles there, config5_kernel in satgb_api.cu).
//
// A tile's data flow is that of sat_kernel_ws.cuh with direct stores.  What bounds that kernel for 8-bit
// pixels is not memory (u8 -> u32 8192^2: 99.7 us, floor 49.5): with its stores left out it is as
// slow, since its compute warps add pixel by pixel, and a tile's carries have one tile period to arrive
// in, while an SM stores 25 bytes a cycle at most, the 64 KB of a tile's results are 1.4 us of
// that, and the look-backs' loads queue behind them.  Three things differ here (82.7 us at 8192^2, 30.9 at
// 4096^2 for 33.5; 70.4 with look-backs that find everything published, 57.9 without stores on top).
//
// Arithmetic.  A tile's own sums of 8-bit pixels are small integers, so the compute warps work
// on the packed words: a row's four pixels a lane are added with one dp4a, column sums
// and the lanes' row totals go two to a register in 16 bits (128 columns of 255 are
// 32,640), a warp reduction is one instruction for two rows, and each output's row prefix is
// one dp4a on top of its base.  Signed pixels are biased by 128 where sums are packed.
// Wider inputs: the sums need the rows' totals only (nine exchanges for eight rows), and the lanes'
// row prefixes are scanned, eight rows side by side, when the tile's results are due.
//
// Depth.  Stages are small beside shared memory, so the sums of tile k+D-1 are taken before the results of
// tile k are stored (D sets of the shared vectors), and carries have D-1 tile periods.  1-byte
// inputs: D = 4, 16 KB stages (8192^2: depth 3 88.7 us, 4 82.7, 5 and 6 82.6 to 82.8).  4-byte inputs: tiles
// of 96 rows, four 48 KB stages, D = 3 (f32 8192^2: 113; 64 rows and D = 4 123, 128 rows and
// D = 2 125; sat_kernel_ws.cuh 116.5; i32 125 -> 113.4; 95 to 98 with look-backs that find
// everything published, 82 without stores on top, floor 79).
//
// Roles.  Publishing waits for no other tile: the compute warps publish the rows' sums as they take
// them, the summing warps the columns', and the resolving warps, which walk row j's and column j's
// look-back side by side, are warps of their own; the corner's look-back has another.  With one group
// of warps that published, walked the rows and walked the columns in turn, a tile that waited
// held back the aggregates of the next (u8 101 us at depth 2).
//
// Packed rows off 16-byte boundaries come through a map of row groups (SKEW): u8 8191^2 135 us with a
// copy to padded rows before the launch, 120 so; f32 8191^2 191 read with plain loads by the compute
// warps, 143 so, 4095^2 53 and 46.9, 2999 x 3001 34.5 and 28.
#pragma once
#include "sat_kernel_ws.cuh"

namespace satgb {

// SKEW: images whose packed rows are off 16-byte boundaries come through a map of row groups (kInSkew), with
// others beside them; the launches of aligned images alone leave that out (with it they took 3 to 6 % more).
template <class TIn, class TOut, class A, bool SKEW>
struct TileShapeWD {
  static constexpr bool PACKED = sizeof(TIn) == 1;
  static constexpr int CPT = 4, RPW = 8, NWC = PACKED ? 16 : 12;
  static constexpr int TW = 128, TH = NWC * RPW;
  // sets of the shared vectors: the tile in output and D - 1 whose sums are out
  static constexpr int D = PACKED ? 4 : 3;
  static constexpr int NPW = TW / 32, NVW = 4, NRW = TH / 32; // summing, resolving warps (and of them, with rows)
  // Rows off 16-byte boundaries come with the 16 bytes that cover their shift.
  static constexpr int SKEW_W = TW + 16 / (int)sizeof(TIn);
  static constexpr int STAGE_ELEMS = TH * (SKEW ? SKEW_W : TW);
  static constexpr int STAGE_BYTES = STAGE_ELEMS * (int)sizeof(TIn);
  static constexpr int STATIC_BYTES =
      D * (NWC * TW + TH + 2 * TW + TH + NWC + NRW + 4) * (int)sizeof(A) + 640;
  static constexpr int S = Stages<STAGE_BYTES, STATIC_BYTES, 1>::value;
  static constexpr int DYN_SMEM = S * STAGE_BYTES;
  static constexpr int THREADS = (NWC + NPW + NVW + 2) * 32;
  // named barriers, one a set: partials in, sums in, carries in; the resolving warps' own
  static constexpr int AGG0 = 1, SUM0 = 1 + D, CAR0 = 1 + 2 * D, ROWS = 1 + 3 * D;
  static_assert(ROWS < 16, "named barriers");
  static_assert(sizeof(A) == 4 && sizeof(TOut) == 4, "4-byte sums");
};

// Sends tile `tp` of an image whose packed rows are off 16-byte boundaries to stage `st`, in the
// 2^skew loads of its tensor map: rows r, r + 2^skew, ... of the tile share their shift and are one box, each
// box's rows after the last box's, from the 16-byte boundary at or before their first pixel.
template <class SH, class TIn>
__device__ __forceinline__ void issue_skewed(const ImageDesc* D, const TilePlan& tp, TIn* stage, uint32_t bar) {
  constexpr int CHUNK = 16 / (int)sizeof(TIn); // columns in 16 bytes
  mbar_arrive_expect_tx(bar, (uint32_t)SH::STAGE_BYTES);
  const int n = (int)D->skew, boxes = 1 << n;
  const int pitch = (int)D->in_pitch, y = (tp.ty * SH::TH) >> n;
  for (int q = 0; q < boxes; ++q)
    tma_load_3d(smem_u32(stage + q * ((SH::TH >> n) * SH::SKEW_W)), &D->tmap_in,
                (q * pitch + tp.tx * SH::TW) & ~(CHUNK - 1), y, 0, bar);
}
// where row `row` of such a tile starts in its stage (elements)
template <class SH, class TIn>
__device__ __forceinline__ uint32_t skewed_row(const ImageView& D, int row) {
  constexpr int CHUNK = 16 / (int)sizeof(TIn);
  const int q = row & ((1 << D.skew) - 1);
  return (uint32_t)(q * ((SH::TH >> D.skew) * SH::SKEW_W) + (row >> D.skew) * SH::SKEW_W +
                    ((q * (int)D.in_pitch) & (CHUNK - 1)));
}
// A warp's rows of such a tile, N = its skew: the words of the lane's four pixels, from the two aligned words that
// hold them.  (`pitch` in bytes: rows r, r + 2^N have the same shift.)
template <class SH, int N>
__device__ __forceinline__ void skewed_words(const void* stage, int warp, int lane, uint32_t pitch,
                                             uint32_t (&w)[SH::RPW]) {
  constexpr int BOX = (SH::TH >> N) * SH::SKEW_W, R = 1 << N;
  const int q0 = (warp * SH::RPW) & (R - 1);
  const char* base = static_cast<const char*>(stage) + q0 * BOX + ((warp * SH::RPW) >> N) * SH::SKEW_W + lane * 4;
#pragma unroll
  for (int r = 0; r < SH::RPW; ++r) {
    const uint32_t shift = (uint32_t)(q0 + (r & (R - 1))) * pitch; // mod 16
    const uint32_t* p =
        reinterpret_cast<const uint32_t*>(base + (r & (R - 1)) * BOX + (r >> N) * SH::SKEW_W + (shift & 12u));
    w[r] = __funnelshift_r(p[0], p[1], shift * 8u); // by the low five bits
  }
}

// The same for 4-byte inputs: from the two aligned 16-byte groups that hold the lane's four columns.
template <class SH, class TIn, int N>
__device__ __forceinline__ void skewed_segs(const TIn* stage, int warp, int lane, uint32_t pitch,
                                            RowSeg<TIn, SH::CPT> (&x)[SH::RPW]) {
  constexpr int BOX = (SH::TH >> N) * SH::SKEW_W, R = 1 << N;
  static_assert(SH::RPW % R == 0, "a warp's first row has no shift");
  const TIn* base = stage + ((warp * SH::RPW) >> N) * SH::SKEW_W + lane * 4;
#pragma unroll
  for (int r = 0; r < SH::RPW; ++r) {
    const uint32_t m = (uint32_t)(r & (R - 1)) * pitch; // mod 4
    const TIn* p = base + (r & (R - 1)) * BOX + (r >> N) * SH::SKEW_W;
    if (r & (R - 1)) {
      RowSeg<TIn, 4> lo, hi;
      lo.u.v = *reinterpret_cast<const typename RowSeg<TIn, 4>::V*>(p);
      hi.u.v = *reinterpret_cast<const typename RowSeg<TIn, 4>::V*>(p + 4);
      TIn a[5]; // from column m & 2
      a[0] = (m & 2u) ? lo.u.e[2] : lo.u.e[0];
      a[1] = (m & 2u) ? lo.u.e[3] : lo.u.e[1];
      a[2] = (m & 2u) ? hi.u.e[0] : lo.u.e[2];
      a[3] = (m & 2u) ? hi.u.e[1] : lo.u.e[3];
      a[4] = (m & 2u) ? hi.u.e[2] : hi.u.e[0];
#pragma unroll
      for (int c = 0; c < 4; ++c) x[r].u.e[c] = (m & 1u) ? a[c + 1] : a[c];
    } else {
      x[r].u.v = *reinterpret_cast<const typename RowSeg<TIn, 4>::V*>(p);
    }
  }
}

// The lanes' eight row partials -> the total of row (lane >> 2): every step hands half of the rows to the
// lane across, so eight rows take nine exchanges.
template <class A>
__device__ __forceinline__ A row_totals(const A (&v)[8], int lane) {
  using AR = Ar<A>;
  A h[4], q[2];
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = AR::add(b4 ? v[4 + i] : v[i], __shfl_xor_sync(0xffffffffu, b4 ? v[i] : v[4 + i], 16));
#pragma unroll
  for (int i = 0; i < 2; ++i) q[i] = AR::add(b3 ? h[2 + i] : h[i], __shfl_xor_sync(0xffffffffu, b3 ? h[i] : h[2 + i], 8));
  A t = AR::add(b2 ? q[1] : q[0], __shfl_xor_sync(0xffffffffu, b2 ? q[0] : q[1], 4));
  t = AR::add(t, __shfl_xor_sync(0xffffffffu, t, 2));
  return AR::add(t, __shfl_xor_sync(0xffffffffu, t, 1));
}

// The sum of a word's four pixels picked by the mask's bytes (0 or 1), plus c.
template <class TIn>
__device__ __forceinline__ uint32_t pixel_sum(uint32_t w, uint32_t mask, uint32_t c) {
  if constexpr (sizeof(TIn) == 1 && TIn(-1) < TIn(0)) return (uint32_t)__dp4a((int)w, (int)mask, (int)c);
  else return __dp4a(w, mask, c);
}

// A small integer (|v| < 2^22) as the accumulator.
template <class A>
__device__ __forceinline__ A small_int(uint32_t v) {
  if constexpr (sizeof(A) == 4 && A(0.5f) != A(0)) return __uint_as_float(0x4B400000u + v) - 12582912.0f; // exact
  else return v;
}

template <class TIn, class TOut, class A, bool REV, bool SKEW>
__global__ void __launch_bounds__(TileShapeWD<TIn, TOut, A, SKEW>::THREADS, 1)
    sat_tile_kernel_wd(const __grid_constant__ SatParams P) {
  using SH = TileShapeWD<TIn, TOut, A, SKEW>;
  constexpr int CPT = SH::CPT, RPW = SH::RPW, NWC = SH::NWC;
  constexpr int TW = SH::TW, TH = SH::TH, S = SH::S;
  constexpr int NPW = SH::NPW, NVW = SH::NVW, NRW = SH::NRW;
  constexpr int WSUM = NWC, WRES = NWC + NPW, WCOR = WRES + NVW, WSTORE = WCOR + 1; // first warp of each role
  constexpr int NAGG = (NWC + NPW) * 32;     // compute + summing warps
  constexpr int NSUM = (NPW + NVW) * 32;     // summing + resolving warps
  constexpr int NCAR = (NWC + NVW + 1) * 32; // compute + resolving + corner warps
  constexpr bool SIGNED = TIn(-1) < TIn(0);
  constexpr uint32_t kBias = SIGNED ? 128u : 0u;
  constexpr bool PACKED = SH::PACKED;
  static_assert(S > SH::D, "stages for the tile in output, those whose sums are out and one loading");
  static_assert(NRW <= NVW && NPW == NVW, "a resolving thread has one column and a row at most");
  constexpr int K = Ar<A>::K;
  using AR = Ar<A>;
  using C = CornerAcc<A>;

  extern __shared__ __align__(128) unsigned char dsmem[];
  TIn* stages = reinterpret_cast<TIn*>(dsmem);

  __shared__ A s_colp[SH::D][NWC][TW];   // column partials a warp (by slot), then their exclusive prefix over the warps
  __shared__ A s_rowagg[SH::D][TH];      // row totals
  __shared__ A s_colagg[SH::D][TW];      // column sums (by slot)
  __shared__ A s_colabove[SH::D][TW];    // column look-back results (by slot)
  __shared__ A s_rowleft[SH::D][TH];     // row look-back results
  __shared__ A s_rlprev[SH::D][NWC];     // per compute warp: sum of rowleft over the rows before it (scan order)
  __shared__ A s_rwt[SH::D][NRW];        // resolving warps: sum of rowleft over each warp's 32 rows
  __shared__ A s_corner[SH::D], s_u[SH::D];
  __shared__ int s_uready[SH::D];  // k + 1 once tile k's u is in s_u
  __shared__ long long s_tile[S];    // spatial tile index per stage (-1: no more tiles)
  __shared__ int s_img[S];
  __shared__ int s_tx[S], s_ty[S], s_pl[S];
  __shared__ __align__(8) unsigned long long s_full[S];
  __shared__ __align__(8) unsigned long long s_done[S]; // the stage has been read and may be refilled

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const uint32_t epoch = ld_relaxed_u32(&P.ws->epoch);
  const uint32_t tagA = make_tag(epoch, kStateAgg);
  const uint32_t tagI = make_tag(epoch, kStateInc);

  if (tid < SH::D) s_uready[tid] = 0;
  clear_stages(tid, s_tile, s_img, s_tx, s_ty, s_pl);
  if (warp == WSTORE && lane == 0) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&s_full[s]), 1);
      mbar_init(smem_u32(&s_done[s]), NWC);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == WSTORE && lane == 0) {
    // ---- producer thread: fills the stages, then refills each once the output phase of its
    //      tile has read it; a ticket is fetched a tile ahead ---------------------------
    auto issue = [&](const TilePlan& tp, int st) {
      const ImageDesc* D = (P.n_images == 1 || tp.t < 0) ? &P.img0 : &P.images[tp.img];
      if (SKEW && tp.t >= 0 && (D->flags & kInSkew)) {
        s_tile[st] = tp.t;
        s_img[st] = tp.img;
        s_tx[st] = tp.tx;
        s_ty[st] = tp.ty;
        s_pl[st] = tp.pl;
        issue_skewed<SH>(D, tp, stages + st * SH::STAGE_ELEMS, smem_u32(&s_full[st]));
      } else {
        issue_tile<TIn, TW, TH, TH * TW * (int)sizeof(TIn)>(P, tp, st, stages + st * SH::STAGE_ELEMS, s_tile, s_img, s_tx, s_ty, s_pl, s_full);
      }
    };
    bool producing = true;
    for (int s = 0; s < S && producing; ++s) {
      const TilePlan tp = plan_tile<REV>(P, atomicAdd(&P.ws->ticket, 1ull));
      issue(tp, s);
      producing = tp.t >= 0;
    }
    unsigned long long pending = producing ? atomicAdd(&P.ws->ticket, 1ull) : 0ull;
    for (int k = 0; producing; ++k) {
      const TilePlan next = plan_tile<REV>(P, pending);
      if (next.t >= 0) pending = atomicAdd(&P.ws->ticket, 1ull);
      const int st = k % S;
      mbar_wait_bounded(smem_u32(&s_done[st]), (k / S) & 1, P, -1);
      issue(next, st);
      producing = next.t >= 0;
    }
  }

  if (warp < NWC) {
    // ---- compute warps ----------------------------------------------------------
    // The warp's rows of a tile, a word of four pixels a lane.
    auto rows_in = [&](const ImageView& D, const TIn* stage, int nvalid, uint32_t (&w)[RPW]) {
      if (!SKEW || !(D.flags & kInSkew)) {
        const TIn* sb = stage + (warp * RPW) * TW + lane * CPT;
#pragma unroll
        for (int r = 0; r < RPW; ++r) w[r] = *reinterpret_cast<const uint32_t*>(sb + r * TW);
        return;
      }
      const uint32_t pitch = (uint32_t)D.in_pitch;
      switch (D.skew) {
        case 1: skewed_words<SH, 1>(stage, warp, lane, pitch, w); break;
        case 2: skewed_words<SH, 2>(stage, warp, lane, pitch, w); break;
        case 3: skewed_words<SH, 3>(stage, warp, lane, pitch, w); break;
        default: skewed_words<SH, 4>(stage, warp, lane, pitch, w); break;
      }
      // past the image's right edge the stage has the next rows' pixels
      const uint32_t keep = nvalid >= CPT ? 0xffffffffu : (1u << (8 * nvalid)) - 1u;
#pragma unroll
      for (int r = 0; r < RPW; ++r) w[r] &= keep;
    };

    // ... and segments of four columns of wider inputs, their sums a row, and those sums' exclusive prefix
    // over the lanes.
    auto segs_in = [&](const ImageView& D, const TIn* stage, int nvalid, RowSeg<TIn, CPT> (&x)[RPW]) {
      if (!SKEW || !(D.flags & kInSkew)) {
        const TIn* sb = stage + (warp * RPW) * TW + lane * CPT;
#pragma unroll
        for (int r = 0; r < RPW; ++r) x[r].u.v = *reinterpret_cast<const typename RowSeg<TIn, CPT>::V*>(sb + r * TW);
        return;
      }
      if constexpr (!PACKED) {
        const uint32_t pitch = (uint32_t)D.in_pitch;
        if (D.skew == 1) skewed_segs<SH, TIn, 1>(stage, warp, lane, pitch, x);
        else skewed_segs<SH, TIn, 2>(stage, warp, lane, pitch, x);
        if (nvalid < CPT) // past the image's right edge the stage has the next rows' elements
#pragma unroll
          for (int r = 0; r < RPW; ++r)
#pragma unroll
            for (int c = 0; c < CPT; ++c)
              if (c >= nvalid) x[r].u.e[c] = TIn(0);
      }
    };
    auto rows_of = [&](const RowSeg<TIn, CPT> (&x)[RPW], A (&rowp)[RPW]) {
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        rowp[r] = Cvt<A, TIn>::in(x[r].u.e[0]);
#pragma unroll
        for (int c = 1; c < CPT; ++c) rowp[r] = AddIn<A, TIn>::add(rowp[r], x[r].u.e[c]);
      }
    };
    auto lane_prefix = [&](const A (&rowp)[RPW], A (&E)[RPW]) {
      // eight rows' scans side by side: a step's latency is shared, and nothing goes through shared memory
      A incl[RPW];
#pragma unroll
      for (int r = 0; r < RPW; ++r) incl[r] = rowp[r];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const bool in = REV ? (lane + d < 32) : (lane >= d);
        A o[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) o[r] = REV ? AR::shfl_down(incl[r], d) : AR::shfl_up(incl[r], d);
#pragma unroll
        for (int r = 0; r < RPW; ++r)
          if (in) incl[r] = AR::add(o[r], incl[r]);
      }
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        E[r] = REV ? AR::shfl_down(incl[r], 1) : AR::shfl_up(incl[r], 1);
        if (lane == (REV ? 31 : 0)) E[r] = AR::zero();
      }
    };

    // The sums of tile kk: false when the tickets ran out (the summing warps still get their
    // AGG arrival, to see the end).
    auto sums = [&](int kk) -> bool {
      const int st = kk % S, kb = kk % SH::D;
      mbar_wait_bounded(smem_u32(&s_full[st]), (kk / S) & 1, P, -1);
      const bool have = s_tile[st] >= 0;
      if (have) {
        const ImageView D = image_view(P, s_img[st]);
        const long long x0 = (long long)s_tx[st] * TW, y0 = (long long)s_ty[st] * TH;
        const long long xt = x0 + (long long)lane * CPT;
        const long long rem = D.width - xt;
        const int nvalid = rem <= 0 ? 0 : (rem >= CPT ? CPT : (int)rem);
        TIn* stage = stages + st * SH::STAGE_ELEMS;
        TIn* sb = stage + (warp * RPW) * TW + lane * CPT;
        const bool tma = D.flags & kInTma;
        if (SKEW && (D.flags & kInSkew)) {
          // the rows after the last whole row of the map (they arrived as zeros)
          const long long mapped = (D.height >> D.skew) << D.skew;
          if (y0 + (warp + 1) * RPW > mapped && y0 + warp * RPW < D.height) {
            for (int r = 0; r < RPW; ++r) {
              const long long y = y0 + warp * RPW + r;
              if (y < mapped || y >= D.height) continue;
              TIn* at = stage + skewed_row<SH, TIn>(D, warp * RPW + r) + lane * CPT;
#pragma unroll
              for (int c = 0; c < CPT; ++c)
                if (c < nvalid) at[c] = static_cast<const TIn*>(D.in)[y * D.in_pitch + xt + c];
            }
            __syncwarp();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // before TMA refills the stage
          }
        } else if (!tma || (nvalid > 0 && xt + nvalid > D.tma_in_w)) {
          // no TMA for this image, or columns past the map (they arrived as zeros)
          const TIn* gin = static_cast<const TIn*>(D.in) + (long long)s_pl[st] * D.in_plane +
                           (y0 + warp * RPW) * D.in_pitch + xt;
          const long long rows = D.height - (y0 + warp * RPW);
          const int c0 = tma ? (int)(D.tma_in_w - xt > 0 ? D.tma_in_w - xt : 0) : 0;
          stage_fill<TIn, CPT, RPW, TW>(sb, gin, D.in_pitch, rows < 0 ? 0 : (rows > RPW ? RPW : (int)rows), nvalid,
                                        c0, (D.flags & kInVec) != 0);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // before TMA refills the stage
        }
        A sum;           // total of the lane's row ...
        int row;         // ... which is this one of the warp's
        bool mine;       // (one lane a row)
        if constexpr (PACKED) {
          uint32_t in[RPW];
          rows_in(D, stage, nvalid, in);
          uint32_t even = 0, odd = 0; // columns 0, 2 and 1, 3 over the rows, 16 bits each
          uint32_t t[RPW / 2];        // the lane's row totals, rows 2i and 2i + 1
#pragma unroll
          for (int r = 0; r < RPW; ++r) {
            const uint32_t b = SIGNED ? in[r] ^ 0x80808080u : in[r];
            even += b & 0x00ff00ffu;
            odd += (b >> 8) & 0x00ff00ffu;
            const uint32_t s = __dp4a(b, 0x01010101u, 0u);
            if (r & 1) t[r / 2] += s << 16;
            else t[r / 2] = s;
          }
          s_colp[kb][warp][0 * 32 + lane] = small_int<A>((even & 0xffffu) - RPW * kBias);
          s_colp[kb][warp][1 * 32 + lane] = small_int<A>((odd & 0xffffu) - RPW * kBias);
          s_colp[kb][warp][2 * 32 + lane] = small_int<A>((even >> 16) - RPW * kBias);
          s_colp[kb][warp][3 * 32 + lane] = small_int<A>((odd >> 16) - RPW * kBias);
          uint32_t total = 0;
#pragma unroll
          for (int i = 0; i < RPW / 2; ++i) {
            const uint32_t s = __reduce_add_sync(0xffffffffu, t[i]);
            if (lane >> 1 == i) total = lane & 1 ? s >> 16 : s & 0xffffu;
          }
          sum = small_int<A>(total - TW * kBias);
          row = lane;
          mine = lane < RPW;
        } else {
          RowSeg<TIn, CPT> x[RPW];
          segs_in(D, stage, nvalid, x);
          A colp[CPT], rowp[RPW];
#pragma unroll
          for (int c = 0; c < CPT; ++c) colp[c] = Cvt<A, TIn>::in(x[0].u.e[c]);
#pragma unroll
          for (int r = 1; r < RPW; ++r)
#pragma unroll
            for (int c = 0; c < CPT; ++c) colp[c] = AddIn<A, TIn>::add(colp[c], x[r].u.e[c]);
          rows_of(x, rowp);
          sum = row_totals<A>(rowp, lane);
          row = lane >> 2;
          mine = (lane & 3) == 0;
#pragma unroll
          for (int c = 0; c < CPT; ++c) s_colp[kb][warp][c * 32 + lane] = colp[c];
        }
        if (mine) {
          const int y = warp * RPW + row, lx = REV ? D.ntx - 1 - s_tx[st] : s_tx[st];
          s_rowagg[kb][y] = sum;
          if (lx < D.ntx - 1 && s_tile[st] != P.stall_tile)
            publish<A>(P.row_words + ((unsigned long long)s_tile[st] * TH + y) * K, sum, tagA);
        }
      }
      named_arrive(SH::AGG0 + kb, NAGG);
      return have;
    };

    // ahead[i]: tile k + i exists
    bool ahead[SH::D];
    ahead[0] = sums(0);
#pragma unroll
    for (int i = 1; i < SH::D - 1; ++i) ahead[i] = ahead[i - 1] && sums(i);
    for (int k = 0; ahead[0]; ++k) {
      ahead[SH::D - 1] = ahead[SH::D - 2] && sums(k + SH::D - 1);
      const int st = k % S, kb = k % SH::D;

      // ---- output phase of tile k: the row scans of wider inputs before its carries are in -------------
      if constexpr (PACKED) named_sync(SH::CAR0 + kb, NCAR); // tile k's carries are in
      const ImageView D = image_view(P, s_img[st]);
      const uint32_t flags = D.flags;
      const long long x0 = (long long)s_tx[st] * TW, y0 = (long long)s_ty[st] * TH;
      const long long xt = x0 + (long long)lane * CPT;
      const long long rem = D.width - xt;
      const int nvalid = rem <= 0 ? 0 : (rem >= CPT ? CPT : (int)rem);
      uint32_t w[RPW];
      RowSeg<TIn, CPT> x[PACKED ? 1 : RPW];
      if constexpr (PACKED) rows_in(D, stages + st * SH::STAGE_ELEMS, nvalid, w);
      else segs_in(D, stages + st * SH::STAGE_ELEMS, nvalid, x);
      TOut* out = static_cast<TOut*>(D.out) + (long long)s_pl[st] * D.out_plane + (y0 + warp * RPW) * D.out_pitch + xt;
      const long long left = D.height - (y0 + warp * RPW);
      const int rows = left < 0 ? 0 : (left > RPW ? RPW : (int)left);
      // the lanes' exclusive row prefixes: packed pixels two rows a register, inclusive scans less the lane's
      // own total
      uint32_t ex[PACKED ? RPW / 2 : 1], own[PACKED ? RPW / 2 : 1];
      A E[PACKED ? 1 : RPW];
      if constexpr (PACKED) {
#pragma unroll
        for (int i = 0; i < RPW / 2; ++i) {
          const uint32_t lo = __dp4a(SIGNED ? w[2 * i] ^ 0x80808080u : w[2 * i], 0x01010101u, 0u);
          const uint32_t hi = __dp4a(SIGNED ? w[2 * i + 1] ^ 0x80808080u : w[2 * i + 1], 0x01010101u, 0u);
          own[i] = ex[i] = lo + (hi << 16);
        }
      } else {
        A rowp[RPW];
        rows_of(x, rowp);
        lane_prefix(rowp, E);
      }
      if constexpr (!PACKED) named_sync(SH::CAR0 + kb, NCAR);
      __syncwarp();
      // the stage goes back to the producer: read here, and every role is done with its tile's descriptor
      if (lane == 0) mbar_arrive(smem_u32(&s_done[st]));
      A top[CPT], cp[CPT];
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        const int c = REV ? CPT - 1 - i : i;
        cp[c] = AR::add(s_colabove[kb][c * 32 + lane], s_colp[kb][warp][c * 32 + lane]);
        if (i) cp[c] = AR::add(cp[REV ? c + 1 : c - 1], cp[c]);
      }
      A incl = cp[REV ? 0 : CPT - 1];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const A o = REV ? AR::shfl_down(incl, d) : AR::shfl_up(incl, d);
        const bool in = REV ? (lane + d < 32) : (lane >= d);
        if constexpr (PACKED) {
          uint32_t e[RPW / 2];
#pragma unroll
          for (int i = 0; i < RPW / 2; ++i)
            e[i] = REV ? __shfl_down_sync(0xffffffffu, ex[i], d) : __shfl_up_sync(0xffffffffu, ex[i], d);
          if (in) {
#pragma unroll
            for (int i = 0; i < RPW / 2; ++i) ex[i] += e[i];
          }
        }
        if (in) incl = AR::add(o, incl);
      }
      {
        A e = REV ? AR::shfl_down(incl, 1) : AR::shfl_up(incl, 1);
        if (lane == (REV ? 31 : 0)) e = AR::zero();
        const A base = AR::add(AR::add(s_corner[kb], s_rlprev[kb][warp]), e);
#pragma unroll
        for (int c = 0; c < CPT; ++c) top[c] = AR::add(base, cp[c]);
      }
      const bool vout = (flags & kOutVec) && nvalid == CPT;
      const uint32_t unbias = (uint32_t)(REV ? 31 - lane : lane) * (4u * kBias);
#pragma unroll
      for (int i = 0; i < RPW; ++i) {
        const int r = REV ? RPW - 1 - i : i;
        TOut o[CPT];
        if constexpr (PACKED) {
          const uint32_t pair = ex[r / 2] - own[r / 2]; // no borrow between the halves: each total is in its sum
          const uint32_t e = (r & 1 ? pair >> 16 : pair & 0xffffu) - unbias;
          const A rl = s_rowleft[kb][warp * RPW + r];
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            const uint32_t mask = REV ? 0x01010101u << (8 * c) : 0x01010101u >> (8 * (CPT - 1 - c));
            A run;
            if constexpr (A(0.5f) != A(0))
              run = AR::add(rl, __uint_as_float(pixel_sum<TIn>(w[r], mask, e + 0x4B400000u)) - 12582912.0f);
            else run = pixel_sum<TIn>(w[r], mask, e + rl);
            top[c] = AR::add(top[c], run);
            o[c] = OutCvt<TOut, A>::out(top[c]);
          }
        } else {
          A run = AR::add(E[r], s_rowleft[kb][warp * RPW + r]);
#pragma unroll
          for (int ii = 0; ii < CPT; ++ii) {
            const int c = REV ? CPT - 1 - ii : ii;
            run = AddIn<A, TIn>::add(run, x[r].u.e[c]);
            top[c] = AR::add(top[c], run);
            o[c] = OutCvt<TOut, A>::out(top[c]);
          }
        }
        if (r < rows && nvalid > 0) store_seg<TOut, CPT>(out + r * D.out_pitch, vout, nvalid, o);
      }
#pragma unroll
      for (int i = 0; i + 1 < SH::D; ++i) ahead[i] = ahead[i + 1];
    }
  }

  if (warp >= WSUM && warp < WRES) {
    // ---- summing warps: one column (slot) per thread; they wait for no other tile ------------------
    const int j = tid - WSUM * 32;
    for (int k = 0;; ++k) {
      const int st = k % S;
      mbar_wait_bounded(smem_u32(&s_full[st]), (k / S) & 1, P, -1);
      const long long t = s_tile[st];
      named_sync(SH::AGG0 + k % SH::D, NAGG); // tile k's partials are in (or there is no tile k)
      if (t < 0) break;
      const int kb = k % SH::D;
      const ImageView D = image_view(P, s_img[st]);
      const int ly = REV ? D.nty - 1 - s_ty[st] : s_ty[st];
      // the column's partials of every compute warp: all loads first, then the
      // exclusive prefix over the warps (scan order) and the column sum
      A v[NWC];
#pragma unroll
      for (int w = 0; w < NWC; ++w) v[w] = s_colp[kb][w][j];
      A run = AR::zero();
#pragma unroll
      for (int i = 0; i < NWC; ++i) {
        const int w = REV ? NWC - 1 - i : i;
        s_colp[kb][w][j] = run;
        run = AR::add(run, v[w]);
      }
      s_colagg[kb][j] = run;
      if (ly < D.nty - 1 && t != P.stall_tile)
        publish<A>(P.col_words + ((unsigned long long)t * TW + j) * K, run, tagA);
      named_arrive(SH::SUM0 + kb, NSUM);
    }
  }

  if (warp >= WRES && warp < WCOR) {
    // ---- resolving warps: row j and column (slot) j per thread -------------------------
    const int j = tid - WRES * 32;
    const int rw = warp - WRES;
    const bool has_row = rw < NRW;
    constexpr int D1 = REV ? 1 : -1; // towards the tiles before
    for (int k = 0;; ++k) {
      const int st = k % S;
      mbar_wait_bounded(smem_u32(&s_full[st]), (k / S) & 1, P, -1);
      const long long t = s_tile[st];
      if (t < 0) break;
      const int kb = k % SH::D;
      const ImageView D = image_view(P, s_img[st]);
      const int ntx = D.ntx, nty = D.nty;
      const int lx = REV ? ntx - 1 - s_tx[st] : s_tx[st], ly = REV ? nty - 1 - s_ty[st] : s_ty[st];
      const bool live = t != P.stall_tile;
      unsigned long long* rbase = P.row_words + ((unsigned long long)t * TH + j) * K;
      unsigned long long* cbase = P.col_words + ((unsigned long long)t * TW + j) * K;
      const long long rstep = D1 * (long long)TH * K, cstep = D1 * (long long)ntx * TW * K;
      EarlyWin<A> wr, wc;
      early_read<A>(wr, rbase, rstep, has_row ? lx : 0);
      early_read<A>(wc, cbase, cstep, ly);
      named_sync(SH::SUM0 + kb, NSUM); // tile k's own sums are in
      // the row's and the column's look-back side by side: every round walks both windows as far as they
      // reach and reads again what is still open
      A left = AR::zero(), above = AR::zero();
      int ri = 0, ci = 0; // predecessors accounted for
      bool rdone = lx == 0 || !has_row, cdone = ly == 0;
      if (rdone && has_row && lx < ntx - 1 && live) publish<A>(rbase, s_rowagg[kb][j], tagI);
      if (cdone && ly < nty - 1 && live) publish<A>(cbase, s_colagg[kb][j], tagI);
      unsigned long long t0 = 0;
      for (uint32_t round = 0; !(rdone && cdone); ++round) {
        bool moved = false;
        if (!rdone) {
#pragma unroll
          for (int q = 0; q < EarlyWin<A>::W; ++q) {
            A val;
            const uint32_t state = rdone ? 0u : decode_word<A>(wr.w[q], tagA, tagI, val);
            if (!state) break;
            left = AR::add(val, left);
            ++ri;
            moved = true;
            rdone = state == kStateInc || ri >= lx;
          }
          if (rdone && lx < ntx - 1 && live) publish<A>(rbase, AR::add(left, s_rowagg[kb][j]), tagI);
        }
        if (!cdone) {
#pragma unroll
          for (int q = 0; q < EarlyWin<A>::W; ++q) {
            A val;
            const uint32_t state = cdone ? 0u : decode_word<A>(wc.w[q], tagA, tagI, val);
            if (!state) break;
            above = AR::add(val, above);
            ++ci;
            moved = true;
            cdone = state == kStateInc || ci >= ly;
          }
          if (cdone && ly < nty - 1 && live) publish<A>(cbase, AR::add(above, s_colagg[kb][j]), tagI);
        }
        if (rdone && cdone) break;
        if (!moved) {
          if (t0 == 0) t0 = global_timer_ns();
          __nanosleep(64);
          if ((round & 15u) == 15u &&
              ((long long)(global_timer_ns() - t0) > P.wait_limit_ns || ld_relaxed_u32(&P.ws->error) != 0u)) {
            record_error(P, t);
            break;
          }
        }
        if (!rdone) early_read<A>(wr, rbase, rstep, lx, ri);
        if (!cdone) early_read<A>(wc, cbase, cstep, ly, ci);
      }
      s_colabove[kb][j] = above;
      if (has_row) {
        s_rowleft[kb][j] = left;
        // inclusive scan of rowleft over the tile's rows, in scan order: within
        // the warp, then across the warps
        A incl = left;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const A o = REV ? AR::shfl_down(incl, d) : AR::shfl_up(incl, d);
          if (REV ? (lane + d < 32) : (lane >= d)) incl = AR::add(o, incl);
        }
        if (lane == (REV ? 0 : 31)) s_rwt[kb][rw] = incl;
        named_sync(SH::ROWS, NRW * 32);
        A before = AR::zero();
#pragma unroll
        for (int i = 0; i < NRW; ++i) {
          const int w = REV ? NRW - 1 - i : i;
          if (REV ? (w > rw) : (w < rw)) before = AR::add(before, s_rwt[kb][w]);
        }
        incl = AR::add(before, incl);
        // rowleft summed over the rows before compute warp w (scan order)
        if (!REV && (j + 1) % RPW == 0 && j + 1 < TH) s_rlprev[kb][(j + 1) / RPW] = incl;
        if (REV && j % RPW == 0 && j > 0) s_rlprev[kb][j / RPW - 1] = incl;
        if (j == (REV ? TH - 1 : 0)) s_rlprev[kb][REV ? NWC - 1 : 0] = AR::zero();
        if (j == (REV ? 0 : TH - 1)) {
          vstore(&s_u[kb], incl); // u
          if (live && ly < nty - 1)
            publish<C>(P.corner_words + (unsigned long long)t * Ar<C>::K, (C)incl, tagA);
          __threadfence_block();
          vstore(&s_uready[kb], k + 1);
        }
      }
      __syncwarp();
      named_arrive(SH::CAR0 + kb, NCAR);
    }
  }

  if (warp == WCOR) {
    // ---- corner warp: lane 0 ----------------------------------------------------------
    constexpr int D1 = REV ? 1 : -1;
    for (int k = 0;; ++k) {
      const int st = k % S;
      mbar_wait_bounded(smem_u32(&s_full[st]), (k / S) & 1, P, -1);
      const long long t = s_tile[st];
      if (t < 0) break;
      const int kb = k % SH::D;
      const ImageView D = image_view(P, s_img[st]);
      const int nty = D.nty, ly = REV ? nty - 1 - s_ty[st] : s_ty[st];
      unsigned long long* base = P.corner_words + (unsigned long long)t * Ar<C>::K;
      if (lane == 0) {
        const long long step = D1 * (long long)D.ntx * Ar<C>::K;
        EarlyWin<C> w[1];
        early_read<C>(w[0], base, step, ly);
        C corner[1];
        resolve_n<C, 1>(w, base, 0, step, ly, tagA, tagI, P, t, corner);
        // u of tile k: the resolving warps have it after every compute warp took tile k's sums, and so is done
        // with the set's last tile (nothing else keeps this warp from running ahead of them)
        CtaWait wait;
        while (vload(&s_uready[kb]) != k + 1 && wait.again(P, t)) {
        }
        __threadfence_block();
        s_corner[kb] = (A)corner[0];
        if (t != P.stall_tile && ly < nty - 1) publish<C>(base, Ar<C>::add(corner[0], (C)vload(&s_u[kb])), tagI);
      }
      __syncwarp();
      named_arrive(SH::CAR0 + kb, NCAR);
    }
  }

  // ---- end of launch: the last CTA resets the ticket and advances the epoch --
  __syncthreads();
  if (tid == 0) finish_launch(P, epoch);
}

}  // namespace satgb
