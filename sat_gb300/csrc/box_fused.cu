// box_fused.cu -- box means of up to four radii straight from the image, and
// their gradient with respect to the image, one launch each, no SAT in memory.
//
// A box mean is a window sum times 1 / area, and the gradient of all the means
// with respect to the image is the sum over radii of the window sums of
// h = g / area (the clipped window relation is symmetric: i lies in the window
// of j exactly when j lies in the window of i).  A window sum is taken in two
// steps, columns first:
//
//   V_k(y, x) = V_k(y - 1, x) + v(y + r_k, x) - v(y - r_k - 1, x)   in registers
//   p_k(y, x) = sum_{i <= x} V_k(y, i)                              one warp scan a row
//   window    = p_k(y, x + r_k) - p_k(y, x - r_k - 1)               through shared memory
//
// Every sum starts inside the strip, so its rounding errors are those of sums of
// a few hundred elements instead of those of a whole plane's SAT.  An infinity or
// NaN stays in the sums that pass it, to the end of the strip and of the block, so
// each kernel runs the way its SAT does, the gradient from the last row and column
// back: what it spoils the way through the SAT spoils too.
//
// A block owns a strip of sy rows of kW = 256 prefix columns, of which tx (host:
// columns) are output columns and the rest the windows' reach to both sides, and has one
// warp a radius; a lane owns 8 adjacent prefix columns.  The rows from the first
// that leaves to the last that enters wait in a ring in shared memory, filled by
// asynchronous copies a batch of rows ahead, so that every element is read from
// memory once a strip: reading the leaving rows from global memory again instead
// spilled L2 (64 x 3 x 1024^2, radii 3, 7, 15: 1.16 GB read for 0.72 GB, 1290 us).
// The outputs of a row are taken 32 adjacent columns at a time.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "box_args.h"

namespace satgb {
satgb_status api_fail(satgb_status st, const char* msg);
satgb_status api_cuda_fail(cudaError_t e, const char* what);
void api_count_launch();
}  // namespace satgb

using satgb::BoxArgs;

namespace {

constexpr int kW = 256; // prefix columns of a block
constexpr int kG = 7;   // most groups of 32 output columns
// Rows in shared memory are plain.  A lane's 8 elements are two 16-byte chunks, 32
// bytes from the next lane's: it takes the second one first where lane / 4 is odd, so
// that the eight lanes of a wavefront touch all the banks.  "First" and "second"
// below are in that order.
__device__ __forceinline__ bool second_first(int lane) { return lane & 4; }

// Strips of tx output columns and sy output rows, copies `ahead` (1 or 2) batches ahead.
struct Shape {
  int tx, sy, ahead;
};

// Two f32 values in one 64-bit register pair and the packed arithmetic on them.
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack(F2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// v += the value D lanes below (REV: above), where there is one
template <bool REV, int D>
__device__ __forceinline__ void add_across(float& v) {
  if constexpr (REV)
    asm("{\n\t.reg .pred p;\n\t.reg .f32 t;\n\tshfl.sync.down.b32 t|p, %0, %1, 31, 0xffffffff;\n\t@p add.rn.f32 %0, %0, t;\n\t}"
        : "+f"(v)
        : "n"(D));
  else
    asm("{\n\t.reg .pred p;\n\t.reg .f32 t;\n\tshfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n\t@p add.rn.f32 %0, %0, t;\n\t}"
        : "+f"(v)
        : "n"(D));
}

__device__ __forceinline__ float clipped_inv(int i, int r, int n, float inv_full) {
  if (i - r >= 0 && i + r <= n - 1) return inv_full;
  return __frcp_rn((float)(min(n - 1, i + r) - max(0, i - r) + 1));
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(live ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(live ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits for the thread's copies but for its last n groups (n <= 2).
__device__ __forceinline__ void copies_wait_ahead(int n) {
  if (n == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
  else if (n == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 2;" ::: "memory");
}

// Starts the copies of one row's kW elements from column xs (a multiple of 4) into a ring row, NT threads
// taking part; zeros outside the plane.  `base` stands for a source that is not read.
template <bool VEC, int NT>
__device__ __forceinline__ void copy_row(float* dst, const float* row, const float* base, int xs, int W, bool live,
                                         int t) {
  constexpr int E = VEC ? 4 : 1; // elements of a copy
#pragma unroll
  for (int i = 0; i < kW / E; i += NT) {
    const int c = (i + t) * E;
    if (kW / E % NT != 0 && i + t >= kW / E) break;
    const bool ok = live && xs + c >= 0 && xs + c + E <= W;
    if constexpr (VEC) copy16(dst + c, ok ? row + xs + c : base, ok);
    else copy4(dst + c, ok ? row + xs + c : base, ok);
  }
}

// A lane's 8 elements of a ring row; `row` points at the lane's first chunk, `d` is the way to its second.
__device__ __forceinline__ void ring_read(F2 (&v)[4], const float* row, int d) {
  const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(row);
  const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + d);
  v[0] = s.x;
  v[1] = s.y;
  v[2] = t.x;
  v[3] = t.y;
}

// The prefix sums of D rows whose elements the warp holds, 8 adjacent ones a lane, into shared memory rows
// `pitch` apart; REV: for each column the sum of those after it.  The rows go side by side: a row alone is one long
// chain of shuffles.
template <int D, bool REV = false>
__device__ __forceinline__ void prefix_rows(const F2 (&u)[D][4], float* dst, int pitch, int d, int lane) {
  float a[D], b[D], incl[D]; // the chunks' sums
#pragma unroll
  for (int i = 0; i < D; ++i) {
    float ax, ay, bx, by;
    unpack(add2(u[i][0], u[i][1]), ax, ay);
    unpack(add2(u[i][2], u[i][3]), bx, by);
    a[i] = ax + ay;
    b[i] = bx + by;
    incl[i] = a[i] + b[i];
  }
#pragma unroll
  for (int i = 0; i < D; ++i) add_across<REV, 1>(incl[i]);
#pragma unroll
  for (int i = 0; i < D; ++i) add_across<REV, 2>(incl[i]);
#pragma unroll
  for (int i = 0; i < D; ++i) add_across<REV, 4>(incl[i]);
#pragma unroll
  for (int i = 0; i < D; ++i) add_across<REV, 8>(incl[i]);
#pragma unroll
  for (int i = 0; i < D; ++i) add_across<REV, 16>(incl[i]);
#pragma unroll
  for (int i = 0; i < D; ++i) {
    float ex = REV ? __shfl_down_sync(0xffffffffu, incl[i], 1) : __shfl_up_sync(0xffffffffu, incl[i], 1);
    if (lane == (REV ? 31 : 0)) ex = 0.f;
    float v[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) unpack(u[i][q], v[2 * q], v[2 * q + 1]);
    if constexpr (REV) {
      // sums of the columns after: each chunk's last column has what comes after the chunk
      float ra = d < 0 ? ex : ex + b[i], rb = d < 0 ? ex + a[i] : ex;
#pragma unroll
      for (int q = 3; q >= 0; --q) {
        const float na = v[q] + ra, nb = v[q + 4] + rb;
        v[q] = ra;
        v[q + 4] = rb;
        ra = na;
        rb = nb;
      }
    } else {
      v[0] += d < 0 ? ex + b[i] : ex;
      v[4] += d < 0 ? ex : ex + a[i];
#pragma unroll
      for (int q = 1; q < 4; ++q) {
        v[q] += v[q - 1];
        v[q + 4] += v[q + 3];
      }
    }
    *reinterpret_cast<float4*>(dst + i * pitch) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(dst + i * pitch + d) = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// The warp's number, in a register the compiler knows to be the same in all lanes.
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

// ---------------------------------------------------------------------------
// Box means: the ring of image rows serves every radius' warp, and the warps meet
// once a batch of kDMeans rows, whose scans go side by side kPMeans at a time; copies
// run sh.ahead batches ahead.  64 x 3 x 1024^2, radii 3, 7, 15, us by (kDMeans, kPMeans):
// (2, 2) 765, (4, 2) 780, (2, 1) 790, (4, 1) 792, (8, 1) 846; through the SAT 1210.
// The shared-memory pipe bounds it (67 % of its wavefronts busy: per output and radius
// two ring reads, one prefix written and two read), then its own latency at 13 warps an SM (issue slots 50 % busy).
constexpr int kDMeans = 2, kPMeans = 2;

// The outputs of D rows (of the first `rows` of them): G groups of 32 columns and, in lanes below `rest`,
// one more.
template <int G, int D>
__device__ __forceinline__ void put_means(float* out, int64_t pitch, const float* rd, const float* ld,
                                          const float (&ix)[kG], bool rest, int rows) {
#pragma unroll
  for (int i = 0; i < D; ++i) {
    if (i < rows) {
#pragma unroll
      for (int c = 0; c < G; ++c) __stcs(out + c * 32, (rd[i * kW + c * 32] - ld[i * kW + c * 32]) * ix[c]);
      if (G < kG && rest) __stcs(out + G * 32, (rd[i * kW + G * 32] - ld[i * kW + G * 32]) * ix[G < kG ? G : 0]);
    }
    out += pitch;
  }
}

template <int NR, bool VEC>
__global__ void __launch_bounds__(NR * 32) box_means_kernel(const __grid_constant__ BoxArgs a, Shape sh) {
  constexpr int D = kDMeans, P = kPMeans, NT = NR * 32;
  extern __shared__ __align__(16) float smem[];
  float* ring = smem + P * NR * kW;
  const int W = (int)a.w, H = (int)a.h, R = a.rmax;
  const int lane = threadIdx.x & 31, k = warp_id();
  const int X0 = blockIdx.x * sh.tx, y0 = blockIdx.y * sh.sy, y1 = min(H, y0 + sh.sy);
  const int xs = (X0 - R - 1) & ~3;
  const int r = a.r[k];
  const float inv = a.inv_full[k];
  const int wrap = (2 * R + 1 + (1 + sh.ahead) * D) * kW; // the ring
  const float* src = a.sat + (int64_t)blockIdx.z * a.sat_plane;
  int jn = y0 - R - 1; // the row copied next, ...
  int jslot = 0;       // ... its ring offset
  auto copy = [&](int n) {
    if (jn < y1 + R) {
      for (int i = 0; i < n; ++i, ++jn) {
        copy_row<VEC, NT>(ring + jslot, src + (int64_t)jn * a.sat_pitch, src, xs, W, jn >= 0 && jn < min(H, y1 + R),
                          threadIdx.x);
        jslot += kW;
        if (jslot == wrap) jslot = 0;
      }
    }
    copies_commit();
  };
  copy(2 * R + 1);
  for (int i = 0; i < sh.ahead; ++i) copy(D);
  const int d = second_first(lane) ? -4 : 4, first = lane * 8 + (second_first(lane) ? 4 : 0);
  float* row = smem + k * (P * kW);
  float* wr = row + first;
  const float* rd = row + lane + X0 - xs + r;
  const float* ld = row + lane + X0 - xs - r - 1;
  const float* mine = ring + first;
  const int n = min(sh.tx, W - X0), ng = n >> 5; // output columns, whole groups of 32
  const bool rest = lane < (n & 31);
  float ix[kG];
#pragma unroll
  for (int c = 0; c < kG; ++c) ix[c] = clipped_inv(min(X0 + c * 32 + lane, W - 1), r, W, inv);
  float* out = a.box[k] + (int64_t)blockIdx.z * a.box_plane + (int64_t)y0 * a.box_pitch + X0 + lane;

  F2 V[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) V[i] = 0ull;
  int sout = (R - r) * kW, sin = (R + r + 1) * kW; // ring offsets of the rows that leave and enter next
  copies_wait_ahead(sh.ahead);
  __syncthreads();
  for (int s = sout; s < sin; s += kW) { // the window of row y0 - 1
    F2 e[4];
    ring_read(e, mine + s, d);
#pragma unroll
    for (int i = 0; i < 4; ++i) V[i] = add2(V[i], e[i]);
  }
#pragma unroll 1
  for (int yb = y0; yb < y1; yb += D) {
    copies_wait_ahead(sh.ahead - 1);
    __syncthreads(); // the batch's rows have arrived, and the rows that left before it are free
    copy(D);
#pragma unroll 1
    for (int y = yb; y < min(yb + D, y1); y += P) {
      F2 u[P][4];
#pragma unroll
      for (int i = 0; i < P; ++i) {
        F2 e[4], l[4];
        ring_read(e, mine + sin, d);
        ring_read(l, mine + sout, d);
#pragma unroll
        for (int q = 0; q < 4; ++q) V[q] = fma2(f2(-1.f, -1.f), l[q], add2(V[q], e[q]));
        sin += kW;
        if (sin == wrap) sin = 0;
        sout += kW;
        if (sout == wrap) sout = 0;
        const float iy = clipped_inv(min(y + i, H - 1), r, H, inv);
#pragma unroll
        for (int q = 0; q < 4; ++q) u[i][q] = mul2(V[q], f2(iy, iy));
      }
      __syncwarp(); // the warp's last prefix rows have been read
      prefix_rows<P>(u, wr, kW, d, lane);
      __syncwarp();
      const int rows = min(P, y1 - y);
#define SG_PUT(G) put_means<G, P>(out, a.box_pitch, rd, ld, ix, rest, rows)
      switch (ng) {
        case 0: SG_PUT(0); break;
        case 1: SG_PUT(1); break;
        case 2: SG_PUT(2); break;
        case 3: SG_PUT(3); break;
        case 4: SG_PUT(4); break;
        case 5: SG_PUT(5); break;
        case 6: SG_PUT(6); break;
        default: SG_PUT(7); break;
      }
#undef SG_PUT
      out += P * a.box_pitch;
    }
  }
}

// ---------------------------------------------------------------------------
// The gradient: every radius has its own gradient plane and ring; the radii's
// window sums meet in shared memory, a batch at a time, and the warps share the
// outputs, one group of 32 columns of a row after the other.  The launch hands the planes over upside down
// (flipped), so rows here go from the last one up.  64 x 3 x 1024^2, radii
// 3, 7, 15: 1004 us (dL/dSAT and its reverse SAT: 1320; with rows counted down here instead 1020), bound by
// latency at 8.4 warps an SM (the rings leave room for three blocks; issue slots 41 % busy).
constexpr int kDGrad = 2;

// Blocks an SM, for the compiler's sake: the sums turned round cost four radii off 16-byte boundaries 5 %, half of it with the
// limit of 128 registers spoken out (us: 8 x 3 x 701 x 901, radii 5, 11, 21, 31 255 and 247).  Fewer radii and more registers go with no
// limit given or lose (150 registers: 4096 x 32^2, radii 1, 2 63 and 69, though 64 x 3 x 1024^2 of three radii 1014 and 983).
constexpr int grad_blocks(int nr) { return nr == 4 ? 4 : 0; }

template <int NR, bool VEC>
__global__ void __launch_bounds__(NR * 32, grad_blocks(NR)) box_grad_kernel(const __grid_constant__ BoxArgs a, Shape sh) {
  constexpr int D = kDGrad;
  constexpr int T = (D * kG + NR - 1) / NR; // most outputs of a warp in a batch
  extern __shared__ __align__(16) float smem[];
  const int W = (int)a.w, H = (int)a.h, R = a.rmax;
  const int lane = threadIdx.x & 31, k = warp_id();
  const int X0 = blockIdx.x * sh.tx, y0 = blockIdx.y * sh.sy, y1 = min(H, y0 + sh.sy);
  // The sums run from the last column back: the block's last columns are the last ones that its outputs need, so that
  // no others enter (tx + 2 R + 1 <= 253, or 255 where R + 1 is a multiple of 4: the first needed one is there too).
  const int xs = (X0 + sh.tx + R - kW + 3) & ~3;
  const int r = a.r[k];
  const float inv = a.inv_full[k];
  float* ring = smem + D * NR * kW;
#pragma unroll
  for (int i = 0; i < NR - 1; ++i)
    if (i < k) ring += (2 * a.r[i] + 1 + (1 + sh.ahead) * D) * kW;
  const int wrap = (2 * r + 1 + (1 + sh.ahead) * D) * kW;
  const float* src = a.box[k] + (int64_t)blockIdx.z * a.box_plane;
  int jn = y0 - r - 1, jslot = 0;
  auto copy = [&](int n) {
    if (jn < y1 + r) {
      for (int i = 0; i < n; ++i, ++jn) {
        copy_row<VEC, 32>(ring + jslot, src + (int64_t)jn * a.box_pitch, src, xs, W, jn >= 0 && jn < min(H, y1 + r), lane);
        jslot += kW;
        if (jslot == wrap) jslot = 0;
      }
    }
    copies_commit();
  };
  copy(2 * r + 1);
  for (int i = 0; i < sh.ahead; ++i) copy(D);
  const int d = second_first(lane) ? -4 : 4, first = lane * 8 + (second_first(lane) ? 4 : 0);
  float* wr = smem + k * kW + first; // rows of a batch one after the other, the radii side by side
  const float* mine = ring + first;
  const float *rd[NR], *ld[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    rd[i] = smem + i * kW + lane + X0 - xs + a.r[i];
    ld[i] = smem + i * kW + lane + X0 - xs - a.r[i] - 1;
  }
  // the lane's columns' reciprocal window widths, in the order it holds them
  F2 ix[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int x = xs + first + (i < 2 ? 2 * i : d + 2 * i - 4);
    ix[i] = f2(clipped_inv(min(max(x, 0), W - 1), r, W, inv), clipped_inv(min(max(x + 1, 0), W - 1), r, W, inv));
  }
  // the warp's outputs of a batch: group c of row i, dealt out in equal runs
  const int n = min(sh.tx, W - X0), ng = (n + 31) >> 5;
  const int share = (D * ng + NR - 1) / NR, t0 = k * share, nt = min(share, D * ng - t0);
  int ps[T], pi[T]; // the group's place in the prefix rows; its row (H: not to be stored)
  int64_t po[T];    // its place in the output
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int i = (t0 + t) / ng, c = (t0 + t) - i * ng;
    pi[t] = t < nt && c * 32 + lane < n ? i : H;
    ps[t] = t < nt ? i * (NR * kW) + c * 32 : 0;
    po[t] = c * 32 + i * a.sat_pitch;
  }
  float* out = a.sat + (int64_t)blockIdx.z * a.sat_plane + (int64_t)y0 * a.sat_pitch + X0 + lane;

  F2 V[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) V[i] = 0ull;
  int sout = 0, sin = (2 * r + 1) * kW;
  copies_wait_ahead(sh.ahead);
  __syncthreads();
  for (int i = 0; i <= 2 * r; ++i) { // the window of row y0 - 1
    F2 e[4];
    ring_read(e, mine + i * kW, d);
    const float f = clipped_inv(min(max(y0 - r - 1 + i, 0), H - 1), r, H, inv);
#pragma unroll
    for (int q = 0; q < 4; ++q) V[q] = fma2(f2(f, f), e[q], V[q]);
  }
#pragma unroll 1
  for (int yb = y0; yb < y1; yb += D) {
    copies_wait_ahead(sh.ahead - 1);
    __syncthreads(); // the last batch's prefix rows have been read; this batch's rows have arrived
    copy(D);
    const bool yinner = yb - 2 * r - 1 >= 0 && yb + D - 1 + 2 * r <= H - 1;
    F2 u[D][4];
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const int y = yb + i;
      F2 e[4], l[4];
      ring_read(e, mine + sin, d);
      ring_read(l, mine + sout, d);
      float fe = inv, fl = inv;
      if (!yinner) {
        fe = clipped_inv(min(max(y + r, 0), H - 1), r, H, inv);
        fl = clipped_inv(min(max(y - r - 1, 0), H - 1), r, H, inv);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) V[q] = fma2(f2(-fl, -fl), l[q], fma2(f2(fe, fe), e[q], V[q]));
      sin += kW;
      if (sin == wrap) sin = 0;
      sout += kW;
      if (sout == wrap) sout = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) u[i][q] = mul2(V[q], ix[q]);
    }
    prefix_rows<D, true>(u, wr, NR * kW, d, lane);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < T; ++t) {
      if (t >= nt) break;
      float s = ld[0][ps[t]] - rd[0][ps[t]];
#pragma unroll
      for (int q = 1; q < NR; ++q) s += ld[q][ps[t]] - rd[q][ps[t]];
      if (yb + pi[t] < y1) __stcs(out + po[t], s);
    }
    out += D * a.sat_pitch;
  }
}

int device_sms() {
  static std::atomic<int> sms[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  int n = sms[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
    sms[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

constexpr int kMaxSmem = 232448; // a block's limit
constexpr int kMaxRadius = 64;    // (96 output columns a block are left)

// Shared memory of a block: the prefix rows and the rings.
int64_t means_smem(const BoxArgs& a, int ahead) {
  return (int64_t)(kPMeans * a.nr + 2 * a.rmax + 1 + (1 + ahead) * kDMeans) * kW * 4;
}
int64_t grad_smem(const BoxArgs& a, int ahead) {
  int64_t rows = kDGrad * a.nr;
  for (int k = 0; k < a.nr; ++k) rows += 2 * a.r[k] + 1 + (1 + ahead) * kDGrad;
  return rows * kW * 4;
}
// Blocks an SM's 228 KB hold, each with 1 KB of the system's.
int resident(int64_t smem) { return (int)(233472 / (smem + 1024)); }

// A block's output columns: at most the prefix columns less the windows' reach,
// in whole groups of 32; narrower where that spreads the plane's width evenly.
int columns(const BoxArgs& a) {
  const int reach = ((a.rmax + 4) & ~3) + a.rmax;
  const int most = (kW - reach) / 32 * 32 < kG * 32 ? (kW - reach) / 32 * 32 : kG * 32;
  if (most <= 0) return 0;
  const int64_t nb = (a.w + most - 1) / most;
  return (int)(((a.w + nb - 1) / nb + 31) & ~31LL);
}

// Rows of a strip.  A block's time goes with its rows and, for the copies and sums of its
// first windows, about half the rows before them (rmax); the blocks of all strips run in
// rounds of per_sm an SM, the last one half full on average.  Measured (gradient, us by
// rows 32 / 64 / 128 / 256): 64 x 3 x 1024^2, radii 3, 7, 15 1100 / 1018 / 980 / 990;
// 8 x 3 x 700 x 900, radii 5, 11, 21, 31 279 / 254 / 264 / 289; radius 31 109 / 100 / 112.
int strip_rows(const BoxArgs& a, int tx, int per_sm) {
  const double across = (double)((a.w + tx - 1) / tx * a.planes), slots = (double)device_sms() * per_sm;
  int best = 0;
  double least = 0;
  for (int sy = 8; sy <= 128; sy <<= 1) {
    const double rounds = across * (double)((a.h + sy - 1) / sy) / slots + 0.5;
    const double t = (rounds > 1 ? rounds : 1) * (sy + a.rmax);
    if (!best || t < least) best = sy, least = t;
  }
  while ((a.h + best - 1) / best > 65535) best <<= 1;
  return best;
}

bool rows_vec(const float* base, int64_t w, int64_t pitch, int64_t plane, int64_t planes) {
  return (uintptr_t)base % 16 == 0 && w % 4 == 0 && pitch % 4 == 0 && (planes == 1 || plane % 4 == 0);
}

template <void (*KERNEL)(BoxArgs, Shape), int NT>
cudaError_t launch(const BoxArgs& a, const Shape& sh, int smem, cudaStream_t s) {
  // the dynamic shared-memory limit, raised once per kernel and device
  static std::atomic<int> raised[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !raised[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) raised[dev].store(1, std::memory_order_release);
  }
  const dim3 grid((unsigned)((a.w + sh.tx - 1) / sh.tx), (unsigned)((a.h + sh.sy - 1) / sh.sy), (unsigned)a.planes);
  KERNEL<<<grid, NT, smem, s>>>(a, sh);
  return cudaGetLastError();
}

template <bool VEC>
cudaError_t launch_means(const BoxArgs& a, const Shape& sh, int smem, cudaStream_t s) {
  switch (a.nr) {
    case 1: return launch<box_means_kernel<1, VEC>, 32>(a, sh, smem, s);
    case 2: return launch<box_means_kernel<2, VEC>, 64>(a, sh, smem, s);
    case 3: return launch<box_means_kernel<3, VEC>, 96>(a, sh, smem, s);
    default: return launch<box_means_kernel<4, VEC>, 128>(a, sh, smem, s);
  }
}

template <bool VEC>
cudaError_t launch_grad(const BoxArgs& a, const Shape& sh, int smem, cudaStream_t s) {
  switch (a.nr) {
    case 1: return launch<box_grad_kernel<1, VEC>, 32>(a, sh, smem, s);
    case 2: return launch<box_grad_kernel<2, VEC>, 64>(a, sh, smem, s);
    case 3: return launch<box_grad_kernel<3, VEC>, 96>(a, sh, smem, s);
    default: return launch<box_grad_kernel<4, VEC>, 128>(a, sh, smem, s);
  }
}

// Whether a call whose blocks stand `blocks` to an SM goes in one launch.  Few blocks leave too few warps to hide the scans'
// latency.  Measured on 8 x 3 x 700 x 900 (us, these kernels / through the SAT), by blocks an SM:
//   means     1: radius 64 366 / 90        2: radii 5, 11, 21, 31 158 / 158 (3 blocks: 109), 45, 46, 47 179 / 135
//             3: radius 31 67 / 81, radii 21, 31 87 / 107, radius 33 86 / 82
//   gradient  1: radii 21, 31 240 / 168, radii 5, 11, 21, 31 254 / 274
//             2: radii 3, 31 144 / 152     3: radius 31 95 / 108
// Over 900 sizes (16 to 2048 columns, radii 7 to 60, 1 to 150 million pixels) the SAT is the faster way within these lines too for
// planes narrower than twice the radius (16 columns, radius 23: 1.1 to 1.7 times as fast), for radii above 31, where a block
// computes 256 columns for 160 (1.1 to 1.6 in calls that fill the SMs), and for one radius of 28 to 31 below 512 columns (1.0 to 1.25).
// Those calls stay here all the same: their errors are those of a window (5e-7 of the means' norm), the SAT's 20 times as large.
bool one_launch(int nr, int blocks, bool grad) {
  return grad ? blocks >= 3 || (blocks == 2 && nr >= 2) || nr == 4 : blocks >= 3 || (blocks == 2 && nr >= 3);
}

// The same planes from their last row up: windows are symmetric, and so are their clipped lengths.
BoxArgs flipped(const BoxArgs& a) {
  BoxArgs f = a;
  f.sat += (a.h - 1) * a.sat_pitch;
  f.sat_pitch = -a.sat_pitch;
  for (int k = 0; k < a.nr; ++k) f.box[k] += (a.h - 1) * a.box_pitch;
  f.box_pitch = -a.box_pitch;
  return f;
}

}  // namespace

namespace satgb {

satgb_status box_means_fused(const BoxArgs& a, cudaStream_t s, bool only_way, bool launch, bool* done) {
  static_assert((kPMeans * SATGB_MAX_RADII + 2 * kMaxRadius + 1 + 2 * kDMeans) * kW * 4 <= kMaxSmem, "a block fits");
  *done = false;
  if (a.rmax > kMaxRadius) return SATGB_OK;
  Shape sh;
  int64_t smem = means_smem(a, sh.ahead = 1);
  const int blocks = resident(smem);
  sh.tx = columns(a);
  sh.sy = strip_rows(a, sh.tx, blocks);
  *done = only_way || one_launch(a.nr, blocks, false);
  if (!*done || !launch) return SATGB_OK;
  if (resident(means_smem(a, 2)) == blocks) smem = means_smem(a, sh.ahead = 2);
  const cudaError_t e = rows_vec(a.sat, a.w, a.sat_pitch, a.sat_plane, a.planes)
                            ? launch_means<true>(a, sh, (int)smem, s)
                            : launch_means<false>(a, sh, (int)smem, s);
  if (e != cudaSuccess) return api_cuda_fail(e, "box_means_kernel launch");
  api_count_launch();
  return SATGB_OK;
}

satgb_status box_grad_fused(const BoxArgs& a, cudaStream_t s, bool only_way, bool* done) {
  *done = false;
  Shape sh;
  int64_t smem = grad_smem(a, sh.ahead = 1);
  if (a.rmax > kMaxRadius || smem > kMaxSmem) return SATGB_OK;
  const int blocks = resident(smem);
  sh.tx = columns(a);
  sh.sy = strip_rows(a, sh.tx, blocks);
  *done = only_way || one_launch(a.nr, blocks, true);
  if (!*done) return SATGB_OK;
  if (resident(grad_smem(a, 2)) == blocks && grad_smem(a, 2) <= kMaxSmem) smem = grad_smem(a, sh.ahead = 2);
  bool vec = true;
  for (int k = 0; k < a.nr; ++k) vec = vec && rows_vec(a.box[k], a.w, a.box_pitch, a.box_plane, a.planes);
  const BoxArgs f = flipped(a);
  const cudaError_t e = vec ? launch_grad<true>(f, sh, (int)smem, s) : launch_grad<false>(f, sh, (int)smem, s);
  if (e != cudaSuccess) return api_cuda_fail(e, "box_grad_kernel launch");
  api_count_launch();
  return SATGB_OK;
}

}  // namespace satgb
