// scan_cols.cu -- the column-only scan of images wide enough to give every SM columns of its own
// (satgb_scan_cols; the reference's IncrementScanY, integralImage/IncrementScanY.cu:10-126).
//
// A column's sums depend on that column alone, so a CTA takes a strip of 32 columns from the first row to
// the last and no sum ever crosses CTAs: no status words, no look-back, no order of tiles.  Blocks of NW x R
// rows go through registers: a warp sums its R rows (a lane a column, rows of the strip 32 coalesced
// elements at any alignment), the warps' sums meet in shared memory, and each warp runs down its rows from the
// sum of everything above.  The next block's loads are in flight meanwhile (two blocks ahead f32 4096^2 was 26.6 us
// for 28.5, but 4600 x 3000 30.3 for 25.9: 64 registers a thread were short).
//
// What bounds it: a block's time on one SM, whose stores (25 bytes a cycle at most) and whose
// scan over the warps follow one another (1.1 us a block of 256 rows of 4-byte results, half of it the
// stores); f64 results the FP64 adds, 7 us (9 from narrower inputs).  Memory only where every SM has a strip.  With 16
// warps of 16 rows and each warp adding up the ones before it a block took 2 us, and f32 errors doubled; an f32
// column's sum over the blocks is a two-sum pair (mean relative error at 8192 rows 7.9e-8 -> 4.6e-8).
// us in a graph, look-back over tiles and strips: f32 256 x 256 8.0 and 3.1, 1024^2 10.1 and 6.2, 4096 x 2048 18.1 and
// 11.1, 4096^2 33.6 and 28.7, packed 3001 x 3003 33.4 and 17.6, 8191^2 221 and 129; f64 4096^2 177 and 116.  On
// buffers used in turn 4096^2 is 32.0: of the same two, 134 MB, L2 keeps a part.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "sat_types.cuh"
#include "satgb.h"

namespace satgb {
satgb_status api_fail(satgb_status st, const char* msg);
satgb_status api_cuda_fail(cudaError_t e, const char* what);
void api_count_launch();

namespace {

constexpr int kColWarps = 32; // one a column of the strip, for the scan over the warps
constexpr int kColRows = 8;   // rows a warp takes of a block

// The sum of all blocks above.  f32: a two-sum pair, as the chain down the image is long.
template <class A>
struct Carry {
  A s = Ar<A>::zero();
  __device__ __forceinline__ A below(A x) const { return Ar<A>::add(s, x); }
  __device__ __forceinline__ void add(A x) { s = Ar<A>::add(s, x); }
};
template <>
struct Carry<float> {
  float s = 0.f, e = 0.f;
  __device__ __forceinline__ float below(float x) const {
    const float y = e + x;
    return s + (y == y ? y : x); // past the finite numbers the error term is a NaN, the sum need not be
  }
  __device__ __forceinline__ void add(float x) {
    float err;
    s = two_sum(s, x, err);
    e += err;
  }
};

template <class T>
__device__ __forceinline__ T* next_row(T* p, long long pitch) {
  asm volatile("" : "+l"(p));
  return p + pitch;
}

template <class TIn, class TOut, class A>
__global__ void __launch_bounds__(kColWarps * 32, 1)
    scan_cols_strip_kernel(const TIn* in, long long in_pitch, TOut* out, long long out_pitch, long long width,
                           long long height) {
  constexpr int R = kColRows, NW = kColWarps, BLOCK = NW * R;
  using AR = Ar<A>;
  __shared__ A s_sum[NW][33]; // a warp's sums by column, then the sums of the warps above (and of all blocks above)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Lanes past the last column compute and store that column too, the same bits to the same place, so that all lanes go one
  // way (with lanes that did nothing the last strip's CTA went two, took half as long again, and the launch with it).
  const long long mine = (long long)blockIdx.x * 32 + lane, col = mine < width ? mine : width - 1;
  const long long n_blocks = (height + BLOCK - 1) / BLOCK, full = height / BLOCK;
  const TIn* gin = in + (long long)warp * R * in_pitch + col; // the warp's rows of the next block to load
  TOut* gout = out + (long long)warp * R * out_pitch + col;   // ... to store

  // A row after the other from one pointer: the pitch's multiples, which the compiler would otherwise keep
  // through the loop, take the registers that the rows need.
  auto load = [&](TIn (&v)[R], long long b) {
    const TIn* p = gin;
    if (b < full) {
#pragma unroll
      for (int r = 0; r < R; ++r, p = next_row(p, in_pitch)) v[r] = __ldcs(p);
    } else {
      const long long y = b * BLOCK + warp * R;
#pragma unroll
      for (int r = 0; r < R; ++r, p = next_row(p, in_pitch)) v[r] = y + r < height ? __ldcs(p) : TIn(0);
    }
    gin += BLOCK * in_pitch;
  };
  Carry<A> carry; // of column `warp`
  auto step = [&](const TIn (&v)[R], long long b) {
    A sum = Cvt<A, TIn>::in(v[0]);
#pragma unroll
    for (int r = 1; r < R; ++r) sum = AddIn<A, TIn>::add(sum, v[r]);
    s_sum[warp][lane] = sum;
    __syncthreads();
    {
      A incl = s_sum[lane][warp]; // column `warp`, the sums of warp `lane`
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const A o = AR::shfl_up(incl, d);
        if (lane >= d) incl = AR::add(o, incl);
      }
      A ex = AR::shfl_up(incl, 1);
      if (lane == 0) ex = AR::zero();
      s_sum[lane][warp] = carry.below(ex);
      carry.add(AR::shfl(incl, 31));
    }
    __syncthreads();
    A above = s_sum[warp][lane];
    TOut* p = gout;
    if (b < full) {
#pragma unroll
      for (int r = 0; r < R; ++r, p = next_row(p, out_pitch)) {
        above = AddIn<A, TIn>::add(above, v[r]);
        __stcs(p, OutCvt<TOut, A>::out(above));
      }
    } else {
      const long long y = b * BLOCK + warp * R;
#pragma unroll
      for (int r = 0; r < R; ++r, p = next_row(p, out_pitch)) {
        above = AddIn<A, TIn>::add(above, v[r]);
        if (y + r < height) __stcs(p, OutCvt<TOut, A>::out(above));
      }
    }
    gout += BLOCK * out_pitch;
  };

  TIn v0[R], v1[R];
  load(v0, 0);
  for (long long b = 0; b < n_blocks; b += 2) {
    load(v1, b + 1);
    step(v0, b);
    if (b + 1 >= n_blocks) break;
    load(v0, b + 2);
    step(v1, b + 1);
  }
}

template <class TIn, class TOut, class A>
cudaError_t launch_cols(const void* in, int64_t in_pitch, void* out, int64_t out_pitch, int64_t width, int64_t height,
                        cudaStream_t s) {
  scan_cols_strip_kernel<TIn, TOut, A><<<(unsigned)((width + 31) / 32), kColWarps * 32, 0, s>>>(
      static_cast<const TIn*>(in), in_pitch, static_cast<TOut*>(out), out_pitch, width, height);
  return cudaGetLastError();
}

}  // namespace

// Strips or tiles with look-back (sat_kernel.cuh), whichever two lines through the measured times say is faster (64
// to 20000 columns by 64 to 8192 rows of every type, packed and padded, both ways forced: 0.2 % above the faster
// one in the mean).  Tiles: a start and a rate in bytes in and out.  Strips: a start, and for each wave of strips over the
// SMs another and a time a block of rows, longer where 32 results lie across 128-byte lines; no faster than 4.6
// TB/s, 3.6 across lines.  Few strips or many rows are the tiles': f32 1024 x 8192 (w x h) 19 us by tiles, 36 by strips,
// 8192^2 99 and 120; the strips': f32 1024 x 1000 9.9 and 6.2, 3000 x 2000 15.7 and 10.5, 4096^2 33.3 and 29.1, packed
// 8191^2 220 and 143, f64 4096^2 177 and 116.
struct ColsLine {
  double tile_start, tile_rate; // us, TB/s
  double start, wave, block;    // us: strips, a wave of them, a block of rows
};

// f32 sums of f32 rows on 16-byte boundaries also take strips where the older of those lines had them (3 us and 1.4 a block and wave
// against 8 us and 5.3 TB/s): strips' two-sum pairs halve the error, and a result gets no worse.  That costs up to a fifth at
// widths past the last wave's (10500 x 2000 40 us by tiles, 48 by strips; 6500 x 2000 26.5 and 26.9).
bool scan_cols_by_strips(const void* in, int64_t in_pitch, size_t in_sz, const void* out, int64_t out_pitch,
                         size_t out_sz, int64_t width, int64_t height, bool f32, int sms) {
  const int64_t strips = (width + 31) / 32;
  if (strips >= (1LL << 31) || sms < 1) return false;
  const bool tma = (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0 && ((size_t)in_pitch * in_sz) % 16 == 0 &&
                   ((size_t)out_pitch * out_sz) % 16 == 0;
  const bool lines = (uintptr_t)out % 128 == 0 && ((size_t)out_pitch * out_sz) % 128 == 0;
  ColsLine c;
  if (out_sz == 4 && in_sz == 1) c = {tma ? 10.8 : 13.0, tma ? 4.8 : 2.9, 0.4, 1.1, lines ? 1.42 : 1.52};
  else if (out_sz == 4) c = {tma ? 10.0 : 11.0, tma ? 6.0 : 3.0, 0.6, 1.1, lines ? 1.25 : 1.3};
  else if (in_sz == 1) c = {tma ? 11.9 : 12.4, tma ? 0.61 : 0.60, 1.1, 1.1, 8.9};
  else if (in_sz == 4) c = {tma ? 11.7 : 12.4, tma ? 0.81 : 0.64, 1.1, 1.1, 8.9};
  else c = {tma ? 10.2 : 10.9, tma ? 1.52 : 1.16, 1.0, 1.1, 6.9};
  const double blocks = (double)((height + kColWarps * kColRows - 1) / (kColWarps * kColRows));
  const double waves = (double)((strips + sms - 1) / sms);
  const double mb = (double)width * (double)height * (double)(in_sz + out_sz) * 1e-6; // a us at 1 TB/s
  const double by_strips = c.start + std::max(waves * (c.wave + blocks * c.block), mb / (lines ? 4.6 : 3.6));
  return by_strips < c.tile_start + mb / c.tile_rate ||
         (f32 && tma && 3.0 + std::max(blocks * waves * 1.4, mb / 4.7) < 8.0 + mb / 5.3);
}

satgb_status scan_cols_strips(int in_t, int out_t, const void* d_in, int64_t in_pitch, void* d_out, int64_t out_pitch,
                              int64_t width, int64_t height, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
#define SG_C(IT, OT, TIN, TOUT, A) \
  if (in_t == IT && out_t == OT) e = launch_cols<TIN, TOUT, A>(d_in, in_pitch, d_out, out_pitch, width, height, s); else
  SG_C(SATGB_U8, SATGB_U32, uint8_t, uint32_t, uint32_t)
  SG_C(SATGB_U8, SATGB_F32, uint8_t, float, float)
  SG_C(SATGB_U8, SATGB_F64, uint8_t, double, double)
  SG_C(SATGB_I8, SATGB_I32, int8_t, int32_t, uint32_t)
  SG_C(SATGB_I8, SATGB_F32, int8_t, float, float)
  SG_C(SATGB_I8, SATGB_F64, int8_t, double, double)
  SG_C(SATGB_I32, SATGB_I32, int32_t, int32_t, uint32_t)
  SG_C(SATGB_I32, SATGB_F64, int32_t, double, double)
  SG_C(SATGB_U32, SATGB_U32, uint32_t, uint32_t, uint32_t)
  SG_C(SATGB_F32, SATGB_F32, float, float, float)
  SG_C(SATGB_F32, SATGB_F64, float, double, double)
  SG_C(SATGB_F64, SATGB_F64, double, double, double)
  return api_fail(SATGB_ERR_UNSUPPORTED_TYPES, "scan_cols: type pair not offered");
#undef SG_C
  if (e != cudaSuccess) return api_cuda_fail(e, "scan_cols_strip_kernel launch");
  api_count_launch();
  return SATGB_OK;
}

}  // namespace satgb
