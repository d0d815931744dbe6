// Batch-union MLEM iteration kernel for the CPU-reference semantics (the
// default kernel of every accumulation mode), and the set-up passes that feed
// it.
//
// Events are sorted by image tile, then by tan in buckets, the cell of their box
// corner inside the tile and tan (strip_sort.cu), so neighbouring events in a
// chunk have nearly the same box and the same in-ellipse rows.  At set-up,
// union_batches_kernel groups each chunk's events greedily into batches of up
// to E consecutive events whose union -- per window row, from the smallest first
// column (rounded down to even) to the largest last column -- spans at most the
// rows and columns of the shape (UShape; chosen from the events' boxes), and
// writes each union row's start column and width.  An event that does not fit
// that rectangle on its own is rasterised in the reference's order instead (the
// exact path).  union_records_kernel then writes a 16-byte record per event and
// union row: the exponent's coefficients and the mask of the event's columns.
//
// The iteration kernel runs one CTA of NW warps per chunk, with the rho and
// back-projection windows of the tile in shared memory.  For a batch, union row
// r belongs to the 4 lanes (gid) of one warp, lane gl owning the pixel pairs
// 2 gl + 8 s (s < SW) of the row from its even start column: the SAME pixels for
// every event of the batch.  So rho is read once per batch, each event's K rho
// stays in registers, and the back-projection adds sum_e K_e rho inv_e to each
// owned pixel pair with one shared-memory read-modify-write per batch (not per
// event); no pixel has two writers in a batch and no atomics are issued.  A
// batch's records arrive by asynchronous copies, issued when the batch before
// the last is through with its buffer, so a batch costs one CTA barrier (the one
// that publishes the denominators, the next records and the free buffer).
//
// Bound by instruction issue.  The records used to be computed on chip for
// every batch, about 65 of its 490 instructions per warp; read from memory they
// cost 16 bytes per event and row of DRAM traffic, which the kernel otherwise
// leaves idle (2e7 events at 2 mm: at most 20 GB per iteration, 2 TB/s).  Iterations,
// computed on chip -> read: 2e7 events at 2 mm 12.39 -> 10.43 ms, 6e6 at 1 mm
// 3.99 -> 3.37 ms, 1e6 at 5 mm 0.293 -> 0.244 ms, 1e6 at 2 mm with sigma 14 / 55
// 1.49 -> 1.28 ms, 2e6 at 2 mm compensated 1.59 -> 1.37 ms.
// With the records read, the shared-memory pipe is 63 % busy; rho'' kept in
// registers from the forward sums to the back-projection instead of read and
// multiplied again there (the compiler has room for it: 123 registers): 2e7 at
// 2 mm 10.43 -> 10.0 ms, 6e6 at 1 mm 3.37 -> 3.21 ms.
//
// Accumulation modes (template argument ACC, DEN64): FP32 windows flushed with
// float atomics; compensated windows (each batch's addition followed by
// Knuth's TwoSum into a compensation window, flushed into the FP32 image and
// its FP32 compensation image); denominators in double-floats on top of that
// (lane partials over <= 8 pixels in FP32, the sums across lanes and warps as
// USum);
// fixed-point integer windows (a batch's value rounded once to 2^-22 of an
// event with a per-batch dither, flushed into the 64-bit integer image).
//
// Kernel value (src/2d/strip/gaussian_kernel.h:51-79, rewritten as in
// strip_fast.cu): along a row the exponent of K / K_ref is p + q j + c j^2 with
// c = kz pw^2.  With j counted from the union row's even start column and
// jc = j - the union row's middle column (u_centre: the further from its events
// the count starts, the more of p + q jc + c jc^2 cancels), K = 2^(p' + q' jc) * 2^(c jc^2); the second factor is the same
// for every event, row and batch, so where it stays in range (u_exponent_form) it multiplies rho when rho is read
// (rho'' = rho 2^(c jc^2)) and a pixel costs one FFMA2 per pixel pair, one ex2
// per pixel and one FMUL2; otherwise (coarse pixels, where 2^(c jc^2) would
// underflow while 2^(p' + q' jc) overflows) the full exponent is evaluated,
// one FADD2 more per pair.
//
// Chain form (where the row Gaussian spans several pixels, e.g. 2 mm or 1 mm
// pixels at sigma_z = 5 pixels: |c| = 0.058): along a row
// K' = 2^(p' + q' jc) is geometric, so a lane evaluates two ex2 per event and
// row (its first pixel pair) and steps to its next pair, 8 columns on, with one
// FMUL2 by R8 = 2^(8 q') (part of the record up to 32 columns).  Every
// K' a lane forms is a product of at most SW rounded factors, within ~1e-6
// of the direct value, and stays a normal float (u_exponent_form).
// The masked K' stay in registers; the forward sum takes K' rho'' in one FFMA2
// per pair, and the back-projection forms sum_e K'_e inv_e per pair and
// multiplies by rho'' once per batch.
//
// Pixel set: exactly the reference's (gaussian_kernel.h:131-137 in its
// rounding), from the exact per-row intervals of row_table_kernel: an event's
// row interval [lo, hi) relative to the union start becomes a column mask (bit
// j = column j of the union row), tested once per pixel.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <type_traits>

#include "strip_async.cuh"
#include "strip_device.cuh"
#include "strip_fast_common.cuh"
#include "strip_internal.h"
#include "strip_raster.cuh"

namespace jpet {
namespace {

// Shape of the batches and of the CTA that iterates them: NW warps, batches of
// up to E events whose union spans at most kRows = 8 NW RS window rows (RS row
// steps of all warps, 8 rows per warp and step, 4 lanes per row) and kCols = 8 SW
// columns (SW sweeps of 4 lanes x 2 pixels).
template <int NW_, int E_, int SW_, int RS_, int MIN_CTAS>
struct UShape {
  static constexpr int NW = NW_, E = E_, SW = SW_, RS = RS_;
  // batches of 16 events: two halves, the second only where the batch has it.
  // A batch's fixed costs (rows, sums over lanes and warps, barrier) are halved
  // where events are dense; 16 columns leave the registers for it.  1e6 events at
  // 5 mm 0.243 -> 0.222 ms per iteration; 2e4 events the same.  Batches of 4
  // instead, with 3 CTAs of 8 warps per SM: 22 % slower at 2 mm, 17 % at 5 mm.
  static constexpr int H = E > 8 ? E / 8 : 1, kHalf = E / H;
  static constexpr int kRows = 8 * NW * RS;
  static constexpr int kCols = 8 * SW;
  static constexpr int kThreads = 32 * NW;
  static constexpr int kMinCtas = MIN_CTAS;
  static constexpr int kPartials = (NW + 3) & ~3;  // warp partials of a denominator, padded
};

constexpr int kUMaxChunk = 2048;     // events per chunk (batch words keep 11 bits of offset)
constexpr int kUMaxChunkFixed = 512; // fixed point: a window pixel's integer sum stays < 2^31

// Batch word: first event (offset in the chunk) | events - 1 << 11 | union rows << 15
// | union's first window row << 22 (below 256: boxes of up to 1024 rows are
// tracked, but a batch's rows lie in the first 256 of the window).
__host__ __device__ inline uint32_t ubatch_word(int first, int cnt, int rows, int u0) {
  return static_cast<uint32_t>(first) | (static_cast<uint32_t>(cnt - 1) << 11) |
         (static_cast<uint32_t>(rows) << 15) | (static_cast<uint32_t>(u0) << 22);
}
__device__ __forceinline__ int ub_first(uint32_t w) { return static_cast<int>(w & 2047u); }
__device__ __forceinline__ int ub_cnt(uint32_t w) { return static_cast<int>((w >> 11) & 15u) + 1; }
__device__ __forceinline__ int ub_rows(uint32_t w) { return static_cast<int>((w >> 15) & 127u); }
__device__ __forceinline__ int ub_u0(uint32_t w) { return static_cast<int>(w >> 22); }

// Union row word (per batch and union row): start column in the window | width << 9.
__host__ __device__ inline uint16_t urow_word(int u, int wu) {
  return static_cast<uint16_t>(u | (wu << 9));
}

// Record of an event in a union row of its batch: p, q, and for up to 32 columns
// R8 and the column mask, else the mask's two halves.  The mask holds the 2 SW
// columns of a lane together, in the order in which the lane takes them (column
// 8 s + 2 gl + h is bit 2 s + h of lane gl's 8 bits, or 16 with two halves), so
// that a lane's tests are of a register's low bits.
__device__ __forceinline__ uint32_t u_lane_mask(uint32_t m) {
  // transpose of 4 x 4 cells of two bits
  uint32_t t = (m ^ (m >> 6)) & 0x00CC00CCu;
  m ^= t ^ (t << 6);
  t = (m ^ (m >> 12)) & 0x0000F0F0u;
  return m ^ t ^ (t << 12);
}
// Denominator sums of the FP64_DEN mode: double-floats (value h + l, |l| of the
// order of h's last bit; the partials are positive, so a sum of a few hundred
// keeps about 45 bits, of which the reciprocal takes 24).  In FP64 the 17 additions
// of a warp's batch were the bound, at 1/64 of the FP32 rate: 2e6 events at 2 mm
// 3.49 -> 1.50 ms per iteration, 1e6 at 5 mm 0.97 -> 0.33 ms, 1e6 at 2 mm with
// sigma 14 / 55 3.75 -> 1.60 ms; against an FP64 image the error is the same
// (8.6e-7 to 1.5e-5 after 1 to 10 iterations, the single-precision evaluation's).
struct __align__(8) USum {
  float h, l;
  __device__ __forceinline__ explicit USum(float v) : h(v), l(0.0f) {}
  USum() = default;
};
__device__ __forceinline__ USum u_two_sum(float a, float b) {
  USum r;
  r.h = __fadd_rn(a, b);
  const float v = __fsub_rn(r.h, a);
  r.l = __fadd_rn(__fsub_rn(a, __fsub_rn(r.h, v)), __fsub_rn(b, v));
  return r;
}
__device__ __forceinline__ USum operator+(USum a, USum b) {
  USum r = u_two_sum(a.h, b.h);
  r.l = __fadd_rn(r.l, __fadd_rn(a.l, b.l));
  return r;
}
__device__ __forceinline__ USum u_from_lane(USum v, int off) {
  USum r;
  r.h = __shfl_xor_sync(kFull, v.h, off);
  r.l = __shfl_xor_sync(kFull, v.l, off);
  return r;
}
// an overflow leaves h infinite and l not a number
__device__ __forceinline__ float u_value(USum v) {
  const float f = __fadd_rn(v.h, v.l);
  return f == f ? f : v.h;
}
// Warp sums of E values per lane, transposed as rows_transpose_sum does it.
// PLAIN: the lanes' values have no low part yet.
template <int E, bool PLAIN>
__device__ __forceinline__ USum u_warp_sum(USum (&v)[E]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = E, off = 16; off > 0; off >>= 1) {
    if (n == 1) {
      v[0] = v[0] + u_from_lane(v[0], off);
      continue;
    }
    const bool hi = (lane & off) != 0;
    n /= 2;
#pragma unroll
    for (int k = 0; k < E / 2; ++k) {
      if (k >= n) break;
      const USum send = hi ? v[k] : v[k + n], keep = hi ? v[k + n] : v[k];
      v[k] = PLAIN && off == 16 ? u_two_sum(keep.h, __shfl_xor_sync(kFull, send.h, off))
                                : keep + u_from_lane(send, off);
    }
  }
  return v[0];
}
template <int E, bool PLAIN>
__device__ __forceinline__ float u_warp_sum(float (&v)[E]) {
  return rows_transpose_sum<E>(v);
}

template <class C, class DT>
struct USmem {
  float4 rec[2][C::E][C::kRows];  // records of two batches
  uint16_t urow[2][C::kRows];     // their union row words
  __align__(16) DT den_part[2][C::E][C::kPartials];  // warp sums of the denominators
  float gfac[2 * C::kCols];          // 2^(c jc^2), jc = index - kCols (split exponent)
  float cjc[2 * C::kCols];           // c jc^2 (full exponent)
  uint32_t bw[4];  // the chunk's batch words and exact-path list: chunk_events + 4 words,
                   // the last of the allocation
};

// Exponent forms of the iteration kernel (template argument XM).
constexpr int kXFull = 0;   // p + q jc + c jc^2 per pixel
constexpr int kXSplit = 1;  // 2^(c jc^2) folded into rho''
constexpr int kXChain = 2;  // split, and K' stepped along the row by R8

// The column that a union row of width wu counts jc from: its middle, even so
// that the pairs of the jc tables stay aligned.
__device__ __forceinline__ int u_centre(int wu) { return (wu >> 1) & ~1; }

// A batch's records (zero, so no pixel, for events past its count and rows past
// its union) and union rows.  rec: the batch's first event's records.
template <class C, class DT>
__device__ __forceinline__ void u_issue_records(USmem<C, DT>& S, int buf, const float4* rec,
                                                const uint16_t* urows, int cnt, int rows) {
  constexpr int kPieces = C::E * C::kRows;
  static_assert(kPieces % C::kThreads == 0, "whole pieces per thread");
  float4* dst = &S.rec[buf][0][0];
#pragma unroll
  for (int i = 0; i < kPieces / C::kThreads; ++i) {
    const int k = i * C::kThreads + threadIdx.x;
    const bool v = k < cnt * C::kRows && k % C::kRows < rows;
    cp_async16(dst + k, rec + (v ? k : 0), v);
  }
  if (threadIdx.x < C::kRows / 8)
    cp_async16(&S.urow[buf][8 * threadIdx.x], urows + 8 * threadIdx.x, true);
  cp_async_commit();
}

// A lane's part of a record.
struct URecord {
  float p, q, r8;
  uint32_t m;  // bit 2 s + h: column 8 s + 2 gl + h inside the event's interval
};
template <class C, int XM, class DT>
__device__ __forceinline__ URecord u_record(const USmem<C, DT>& S, int buf, int j, int r_u,
                                            int gl) {
  const float4 a = S.rec[buf][j][r_u];
  if constexpr (C::SW <= 4)
    return URecord{a.x, a.y, a.z, __float_as_uint(a.w) >> (8 * gl)};
  else
    return URecord{a.x, a.y, XM == kXChain ? ex2_approx(8.0f * a.y) : 0.0f,
                   __float_as_uint(gl & 2 ? a.w : a.z) >> (16 * (gl & 1))};
}

// Forward sums of one row step with SWN active sweeps: rho'' of the owned
// pixel pairs, then every event's K rho'' (masked to its interval).
template <class C, int SWN, int RSI, bool SPLIT, class DT>
__device__ __forceinline__ void u_forward(float2 (&kr)[C::E][C::RS][C::SW], DT (&dsum)[C::H][C::kHalf],
                                          const float* w_rho, const USmem<C, DT>& S, int buf,
                                          int cnt, int base, int r_u, int jc0, int gl) {
  float2 rr[C::SW], cq[C::SW], jc2[C::SW];
#pragma unroll
  for (int s = 0; s < SWN; ++s) {
    const float2 rv = *reinterpret_cast<const float2*>(w_rho + base + 8 * s);
    if (SPLIT) {
      const float2 gv = *reinterpret_cast<const float2*>(&S.gfac[C::kCols + jc0 + 8 * s]);
      rr[s] = __fmul2_rn(rv, gv);
    } else {
      rr[s] = rv;
      cq[s] = *reinterpret_cast<const float2*>(&S.cjc[C::kCols + jc0 + 8 * s]);
    }
    const float j0 = static_cast<float>(jc0 + 8 * s);
    jc2[s] = make_float2(j0, j0 + 1.0f);
  }
#pragma unroll
  for (int j = 0; j < C::E; ++j) {
    if (j > 0 && j % 8 == 0 && cnt <= j) break;
    const URecord a = u_record<C, SPLIT ? kXSplit : kXFull>(S, buf, j, r_u, gl);
    const float2 p2 = make_float2(a.p, a.p), q2 = make_float2(a.q, a.q);
    float2 dd = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int s = 0; s < SWN; ++s) {
      const float2 e = SPLIT ? __ffma2_rn(q2, jc2[s], p2)
                             : __ffma2_rn(q2, jc2[s], __fadd2_rn(p2, cq[s]));
      float2 v = __fmul2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), rr[s]);
      v.x = (a.m & (1u << (2 * s))) ? v.x : 0.0f;
      v.y = (a.m & (2u << (2 * s))) ? v.y : 0.0f;
      kr[j][RSI][s] = v;
      dd = __fadd2_rn(dd, v);
    }
    const DT pr(dd.x + dd.y);
    DT& ds = dsum[j / C::kHalf][j % C::kHalf];
    ds = (RSI == 0) ? pr : ds + pr;
  }
}

// Forward sums of one row step in the chain form: per event two ex2 for the
// lane's first pixel pair, then one FMUL2 by R8 per further pair; the masked
// K' stay in kr and the sum takes K' rho'' with one FFMA2 per pair.
template <class C, int SWN, int RSI, class DT>
__device__ __forceinline__ void u_forward_chain(float2 (&kr)[C::E][C::RS][C::SW],
                                                DT (&dsum)[C::H][C::kHalf], float2 (&rr)[C::SW],
                                                const float* w_rho, const USmem<C, DT>& S,
                                                int buf, int cnt, int base, int r_u, int jc0,
                                                int gl) {
  const float jf = static_cast<float>(jc0);
#pragma unroll
  for (int s = 0; s < SWN; ++s) {
    const float2 rv = *reinterpret_cast<const float2*>(w_rho + base + 8 * s);
    const float2 gv = *reinterpret_cast<const float2*>(&S.gfac[C::kCols + jc0 + 8 * s]);
    rr[s] = __fmul2_rn(rv, gv);
  }
#pragma unroll
  for (int j = 0; j < C::E; ++j) {
    if (j > 0 && j % 8 == 0 && cnt <= j) break;
    const URecord a = u_record<C, kXChain>(S, buf, j, r_u, gl);
    const float e0 = fmaf(a.q, jf, a.p);
    float2 k = make_float2(ex2_approx(e0), ex2_approx(e0 + a.q));
    const float2 r8 = make_float2(a.r8, a.r8);
    float2 dd;
#pragma unroll
    for (int s = 0; s < SWN; ++s) {
      if (s > 0) k = __fmul2_rn(k, r8);
      float2 v;
      v.x = (a.m & (1u << (2 * s))) ? k.x : 0.0f;
      v.y = (a.m & (2u << (2 * s))) ? k.y : 0.0f;
      kr[j][RSI][s] = v;
      dd = (s == 0) ? __fmul2_rn(v, rr[0]) : __ffma2_rn(v, rr[s], dd);
    }
    // a lane's partial over its <= 8 pixels of the row in FP32; a USum (DEN64)
    // from the sums across lanes and warps on
    const DT pr(dd.x + dd.y);
    DT& ds = dsum[j / C::kHalf][j % C::kHalf];
    ds = (RSI == 0) ? pr : ds + pr;
  }
}

// Adds a pixel pair's batch value v (sum over the batch's events of
// K rho / den) into the back-projection window, storing only where the row
// group owns the pair (own):
//   kAccFloat        plain float addition;
//   kAccCompensated  float addition whose exact rounding error (Knuth's TwoSum)
//                    joins the compensation window;
//   kAccFixed        v rounded once to 2^-22 of an event with the batch's
//                    dither (floor(v 2^22 + U), U uniform in [0, 1): unbiased)
//                    and added to the integer window (order-independent sums;
//                    a window pixel of a chunk of <= 512 events stays < 2^31,
//                    so the fixed-point mode's chunks hold at most 512).
template <int ACC>
__device__ __forceinline__ void u_accumulate(float* w_out, float* w_comp, int idx, float2 v,
                                             bool own, float dither) {
  if (ACC == kAccFixed) {
    uint2* op = reinterpret_cast<uint2*>(w_out + idx);
    const uint2 o = *op;
    const uint32_t q0 = __float2uint_rn(fmaf(v.x, kFixedScale, dither));
    const uint32_t q1 = __float2uint_rn(fmaf(v.y, kFixedScale, dither));
    if (own) *op = make_uint2(o.x + q0, o.y + q1);
  } else {
    float2* op = reinterpret_cast<float2*>(w_out + idx);
    const float2 o = *op;
    const float2 n = __fadd2_rn(o, v);
    if (ACC == kAccCompensated) {
      float2* cp = reinterpret_cast<float2*>(w_comp + idx);
      const float2 bp = __fadd2_rn(n, make_float2(-o.x, -o.y));
      const float2 nb = __fadd2_rn(n, make_float2(-bp.x, -bp.y));
      const float2 err = __fadd2_rn(__fadd2_rn(o, make_float2(-nb.x, -nb.y)),
                                    __fadd2_rn(v, make_float2(-bp.x, -bp.y)));
      const float2 cn = __fadd2_rn(*cp, err);
      if (own) {
        *op = n;
        *cp = cn;
      }
    } else if (own) {
      *op = n;
    }
  }
}

// Back-projection of one row step in the chain form: rho'' sum_e K'_e inv_e
// per owned pixel pair (rho'' kept since the forward sums), one
// read-modify-write of the pair.
template <class C, int SWN, int RSI, int ACC>
__device__ __forceinline__ void u_back_chain(const float2 (&kr)[C::E][C::RS][C::SW],
                                             const float2 (&rr)[C::SW], float inv_l,
                                             int cnt, float* w_out, float* w_comp, int base,
                                             int wu, int gl, float dither) {
  // events outer, so that one event's 1/den is live at a time (lane j holds
  // event j's); the per-pair sums take the events in the same order as before
  float2 acc[C::SW];
#pragma unroll
  for (int j = 0; j < C::E; ++j) {
    if (j > 0 && j % 8 == 0 && cnt <= j) break;
    const float v = __shfl_sync(kFull, inv_l, j);
    const float2 i2 = make_float2(v, v);
#pragma unroll
    for (int s = 0; s < SWN; ++s)
      acc[s] = (j == 0) ? __fmul2_rn(kr[0][RSI][s], i2) : __ffma2_rn(kr[j][RSI][s], i2, acc[s]);
  }
#pragma unroll
  for (int s = 0; s < SWN; ++s) {
    // loads stay inside the windows (a row's last pair ends before the next
    // row's pitch plus the 64-float padding); the store is predicated on the
    // union row's width, the only pixels this row group owns
    const bool own = 2 * gl + 8 * s < wu;
    if (ACC == kAccFloat) {
      float2* op = reinterpret_cast<float2*>(w_out + base + 8 * s);
      const float2 nv = __ffma2_rn(acc[s], rr[s], *op);
      if (own) *op = nv;
    } else {
      u_accumulate<ACC>(w_out, w_comp, base + 8 * s, __fmul2_rn(acc[s], rr[s]),
                        own, dither);
    }
  }
}

// Back-projection of one row step: sum_e K_e rho inv_e per owned pixel pair,
// one read-modify-write of the pair (inside the union row's width).
template <class C, int SWN, int RSI, int ACC>
__device__ __forceinline__ void u_back(const float2 (&kr)[C::E][C::RS][C::SW], float inv_l,
                                       int cnt, float* w_out, float* w_comp, int base, int wu,
                                       int gl, float dither) {
  float2 acc[C::SW];
#pragma unroll
  for (int j = 0; j < C::E; ++j) {
    if (j > 0 && j % 8 == 0 && cnt <= j) break;
    const float v = __shfl_sync(kFull, inv_l, j);
    const float2 i2 = make_float2(v, v);
#pragma unroll
    for (int s = 0; s < SWN; ++s)
      acc[s] = (j == 0) ? __fmul2_rn(kr[0][RSI][s], i2) : __ffma2_rn(kr[j][RSI][s], i2, acc[s]);
  }
#pragma unroll
  for (int s = 0; s < SWN; ++s) {
    if (ACC == kAccFloat) {
      if (2 * gl + 8 * s < wu) {
        float2* op = reinterpret_cast<float2*>(w_out + base + 8 * s);
        *op = __fadd2_rn(*op, acc[s]);
      }
    } else {
      u_accumulate<ACC>(w_out, w_comp, base + 8 * s, acc[s], 2 * gl + 8 * s < wu, dither);
    }
  }
}

template <class C, int SWN, int RSI, int XM, class DT>
__device__ __forceinline__ void u_forward_x(float2 (&kr)[C::E][C::RS][C::SW], DT (&dsum)[C::H][C::kHalf],
                                            float2 (&rr)[C::RS][C::SW], const float* w_rho,
                                            const USmem<C, DT>& S, int buf, int cnt, int base,
                                            int r_u, int jc0, int gl) {
  if constexpr (SWN > 0) {
    if constexpr (XM == kXChain)
      u_forward_chain<C, SWN, RSI, DT>(kr, dsum, rr[RSI], w_rho, S, buf, cnt, base, r_u, jc0, gl);
    else
      u_forward<C, SWN, RSI, XM == kXSplit, DT>(kr, dsum, w_rho, S, buf, cnt, base, r_u, jc0, gl);
  }
}

// The code for nsw active sweeps (nsw <= N, warp-uniform: a warp maximum, so
// the shuffles inside run converged): f(integral_constant<int, nsw>).
template <int N, class F>
__device__ __forceinline__ void u_sweeps(int nsw, F&& f) {
  if constexpr (N == 0) {
    f(std::integral_constant<int, 0>{});
  } else {
    if (nsw == N)
      f(std::integral_constant<int, N>{});
    else
      u_sweeps<N - 1>(nsw, f);
  }
}

template <class C, int SWN, int RSI, int XM, int ACC>
__device__ __forceinline__ void u_back_x(const float2 (&kr)[C::E][C::RS][C::SW],
                                         const float2 (&rr)[C::RS][C::SW], float inv_l, int cnt,
                                         float* w_out, float* w_comp, int base, int wu, int gl,
                                         float dither) {
  if constexpr (SWN > 0 && XM == kXChain)
    u_back_chain<C, SWN, RSI, ACC>(kr, rr[RSI], inv_l, cnt, w_out, w_comp, base, wu, gl, dither);
  else if constexpr (SWN > 0)
    u_back<C, SWN, RSI, ACC>(kr, inv_l, cnt, w_out, w_comp, base, wu, gl, dither);
}

// Shared memory of the kernel: the rho and back-projection windows (and the
// compensation window of the compensated modes), then the batch records.
template <class C, int ACC, bool DEN64>
size_t u_smem(const Tiling& t) {
  using DT = typename std::conditional<DEN64, USum, float>::type;
  return (ACC == kAccCompensated ? 3ull : 2ull) * fast_window_floats(t) * sizeof(float) +
         sizeof(USmem<C, DT>) + static_cast<size_t>(t.chunk_events) * sizeof(uint32_t);
}

// ACC: kAccFloat (the FP32 iteration), kAccCompensated (tile windows with
// TwoSum compensation, flushed into the FP32 image and its FP32 compensation
// image), kAccFixed (integer tile windows flushed into the 64-bit fixed-point
// image); DEN64: per-event denominators reduced in double-floats.
template <class C, int XM, int ACC, bool DEN64>
__global__ void __launch_bounds__(C::kThreads, C::kMinCtas) iterate_union_kernel(
    DevGeom g, FastConst fc, Tiling t, const Chunk* __restrict__ chunks,
    const float4* __restrict__ ev_geom, const short4* __restrict__ ev_box,
    const float4* __restrict__ records, const uint16_t* __restrict__ urows,
    const uint32_t* __restrict__ batches,
    const float* __restrict__ rho, float* __restrict__ out, AuxImage aux, uint32_t seed,
    DevCounters* counters) {
  using DT = typename std::conditional<DEN64, USum, float>::type;
  constexpr int NW = C::NW, E = C::E, RS = C::RS, SW = C::SW;
  constexpr int kRowsPerStep = NW * 8;  // union rows per step of all warps
  constexpr int kWindows = ACC == kAccCompensated ? 3 : 2;
  extern __shared__ __align__(16) float smem[];
  const int pitch = fast_pitch(t);
  const int wfl = fast_window_floats(t);
  float* w_rho = smem;
  float* w_out = smem + wfl;
  float* w_comp = ACC == kAccCompensated ? smem + 2 * wfl : nullptr;
  USmem<C, DT>& S = *reinterpret_cast<USmem<C, DT>*>(smem + kWindows * wfl);

  const Chunk c = chunks[blockIdx.x];
  const int ox = c.ox & ~1, oy = c.oy;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gid = lane >> 2, gl = lane & 3;
  const int nb = c.n_batches;
  const uint32_t* bws = batches + c.start;
  auto issue = [&](int b, int buf, uint32_t w) {
    u_issue_records<C, DT>(S, buf,
                           records + static_cast<size_t>(c.rec + ub_first(w)) * C::kRows,
                           urows + static_cast<size_t>(c.start + b) * C::kRows, ub_cnt(w),
                           ub_rows(w));
  };

  if (nb > 0) issue(0, 0, bws[0]);
  if (nb > 1) issue(1, 1, bws[1]);
  for (int i = threadIdx.x; i < c.count; i += NW * 32) S.bw[i] = bws[i];
  // rho window by asynchronous copies (zero outside the image), so that its
  // loads overlap with each other and with the first batches' staging
  for (int r = warp; r < t.win_h; r += NW) {
    const int gy = oy + r;
    for (int col = lane; col < pitch; col += 32) {
      const int gx = ox + col;
      const bool in = gy < g.n_y && gx < g.n_z;
      cp_async4(&w_rho[r * pitch + col], rho + (in ? gy * g.n_z + gx : 0), in);
      w_out[r * pitch + col] = 0.0f;
      if (ACC == kAccCompensated) w_comp[r * pitch + col] = 0.0f;
    }
  }
  cp_async_commit();
  for (int i = threadIdx.x; i < 64; i += NW * 32) w_rho[t.win_h * pitch + i] = 0.0f;
  if (threadIdx.x < 2 * C::kCols) {
    const float cz = fc.kz * g.pixel_width * g.pixel_width;
    const float jc = static_cast<float>(static_cast<int>(threadIdx.x) - C::kCols);
    S.cjc[threadIdx.x] = cz * jc * jc;
    S.gfac[threadIdx.x] = ex2_approx(cz * jc * jc);
  }
  unsigned long long contrib = 0;
  cp_async_wait_all();
  __syncthreads();

  for (int b = 0; b < nb; ++b) {
    const int buf = b & 1;
    const uint32_t bw = S.bw[b];
    const int cnt = ub_cnt(bw), u0 = ub_u0(bw);
    // ---- forward: this warp's union rows of every event of the batch
    float2 kr[E][RS][SW], rr[RS][SW];  // K' (chain) or K rho''; rho'' (chain)
    DT dsum[C::H][C::kHalf];
#pragma unroll
    for (int j = 0; j < E; ++j) dsum[j / C::kHalf][j % C::kHalf] = DT(0.0f);
    int base[RS], wu[RS], nsw[RS], jc0[RS];
#pragma unroll
    for (int rs = 0; rs < RS; ++rs) {
      const int r_u = kRowsPerStep * rs + 8 * warp + gid;
      const uint32_t ur = S.urow[buf][r_u];
      const int wrow = min(u0 + r_u, t.win_h - 1);
      base[rs] = wrow * pitch + static_cast<int>(ur & 511u) + 2 * gl;
      wu[rs] = static_cast<int>(ur >> 9);
      jc0[rs] = 2 * gl - u_centre(wu[rs]);
      nsw[rs] = (__reduce_max_sync(kFull, static_cast<unsigned>(wu[rs])) + 7) >> 3;
    }
    // (RS == 1) forward sums and their transposed warp sum in one straight-line
    // block per sweep count, so that the scheduler interleaves the sum's shuffles
    // with the evaluation
    auto sums = [&]() {
#pragma unroll
      for (int h = 0; h < C::H; ++h) {
        if (h > 0 && cnt <= h * C::kHalf) break;
        const DT tot = u_warp_sum<C::kHalf, RS == 1>(dsum[h]);
        if (rows_lane_writes<C::kHalf>(lane))
          S.den_part[buf][h * C::kHalf + rows_lane_event<C::kHalf>(lane)][warp] = tot;
      }
    };
    if constexpr (RS == 1) {
      u_sweeps<SW>(nsw[0], [&](auto n) {
        u_forward_x<C, decltype(n)::value, 0, XM, DT>(kr, dsum, rr, w_rho, S, buf, cnt, base[0],
                                                      8 * warp + gid, jc0[0], gl);
        sums();
      });
    } else {
      u_sweeps<SW>(nsw[0], [&](auto n) {
        u_forward_x<C, decltype(n)::value, 0, XM, DT>(kr, dsum, rr, w_rho, S, buf, cnt, base[0],
                                                      8 * warp + gid, jc0[0], gl);
      });
      u_sweeps<SW>(nsw[RS - 1], [&](auto n) {
        u_forward_x<C, decltype(n)::value, RS - 1, XM, DT>(kr, dsum, rr, w_rho, S, buf, cnt, base[RS - 1],
                                                           kRowsPerStep + 8 * warp + gid,
                                                           jc0[RS - 1], gl);
      });
      sums();
    }
    // the barrier also publishes the next batch's records (this thread's copies,
    // issued one batch ago, are waited for first), and frees this batch's
    cp_async_wait_all();
    __syncthreads();
    if (b + 2 < nb) issue(b + 2, buf, S.bw[b + 2]);
    // ---- denominators: lane j (mod E) adds the warps' partials of event j
    float inv_l;
    {
      const int jl = lane & (E - 1);
      float den;
      if constexpr (DEN64) {
        // 32 / E lanes share an event's partials
        USum d(0.0f);
#pragma unroll
        for (int i = 0; i < NW; i += 32 / E) {
          const int w = i + lane / E;
          if (w < NW) d = i == 0 ? S.den_part[buf][jl][w] : d + S.den_part[buf][jl][w];
        }
#pragma unroll
        for (int off = E; off < 32; off *= 2) d = d + u_from_lane(d, off);
        den = u_value(d);
      } else {
        const float4* dp = reinterpret_cast<const float4*>(S.den_part[buf][jl]);
        const float4 d0 = dp[0];
        den = (d0.x + d0.y) + (d0.z + d0.w);
#pragma unroll
        for (int w = 1; w < NW / 4; ++w) {
          const float4 d1 = dp[w];
          den += (d1.x + d1.y) + (d1.z + d1.w);
        }
      }
      const bool ok = den > 0.0f;  // inv_denominator = 0 otherwise (reconstruction.h:290)
      inv_l = ok ? rcp_approx(den) : 0.0f;
      const unsigned okm = __ballot_sync(kFull, ok && lane < cnt);
      if (threadIdx.x == 0) contrib += __popc(okm);
    }
    // ---- back-projection into the owned pixel pairs (fixed-point mode: one
    // dither per batch, from the batch's position and the iteration's seed)
    float dither = 0.0f;
    if (ACC == kAccFixed) {
      const uint32_t key = hash32(static_cast<uint32_t>(c.start + b) ^ seed);
      dither = static_cast<float>(key >> 8) * 5.9604644775390625e-08f - 0.5f;
    }
#pragma unroll
    for (int rs = 0; rs < RS; ++rs) {
      // one call per row step; RSI has to be a constant
      u_sweeps<SW>(nsw[rs], [&](auto n) {
        if (rs == 0)
          u_back_x<C, decltype(n)::value, 0, XM, ACC>(kr, rr, inv_l, cnt, w_out, w_comp, base[0],
                                                       wu[0], gl, dither);
        else
          u_back_x<C, decltype(n)::value, RS - 1, XM, ACC>(kr, rr, inv_l, cnt, w_out, w_comp,
                                                            base[RS - 1], wu[RS - 1], gl,
                                                            dither);
      });
    }
  }

  // ---- events outside the batch rectangle: reference-order warp rasteriser
  __syncthreads();
  unsigned long long dummy_calls = 0, exact_path = 0;
  const int nx = c.n_exact;
  for (int k = warp; k < nx; k += NW) {
    const int ei = c.start + static_cast<int>(S.bw[c.count - 1 - k]);
    if (ACC == kAccFloat) {
      WindowAccess acc{w_rho, w_out, ox, oy, pitch};
      process_event<kCpuReference>(g, 32, ev_geom[ei], ev_box[ei], acc, nullptr, dummy_calls,
                                   contrib);
    } else {
      // the other modes' windows hold compensated or integer sums: these events
      // add into the FP32 image directly (combined with the second image after
      // the iteration)
      GlobalAccess<float> gacc{rho, out, g.n_z};
      process_event<kCpuReference>(g, 32, ev_geom[ei], ev_box[ei], gacc, nullptr, dummy_calls,
                                   contrib);
    }
    if (lane == 0) ++exact_path;
  }
  if (lane == 0 && contrib) atomicAdd(&counters->n_contributing, contrib);
  if (lane == 0 && exact_path) atomicAdd(&counters->n_exact_path, exact_path);
  __syncthreads();
  for (int r = warp; r < t.win_h; r += NW) {
    const int gy = oy + r;
    for (int col = lane; col < pitch; col += 32) {
      const int gx = ox + col;
      if (ACC == kAccFloat) {
        const float v = w_out[r * pitch + col];
        if (v != 0.0f && gy < g.n_y && gx < g.n_z) atomicAdd(&out[gy * g.n_z + gx], v);
      } else if (ACC == kAccCompensated) {
        const float v = w_out[r * pitch + col], cv = w_comp[r * pitch + col];
        if ((v != 0.0f || cv != 0.0f) && gy < g.n_y && gx < g.n_z)
          flush_compensated(out, aux.lo, gy * g.n_z + gx, v, cv);
      } else {
        const uint32_t q = reinterpret_cast<const uint32_t*>(w_out)[r * pitch + col];
        if (q != 0u && gy < g.n_y && gx < g.n_z)
          atomicAdd(&aux.q[gy * g.n_z + gx], static_cast<unsigned long long>(q));
      }
    }
  }
}


// ---- host side of one shape --------------------------------------------------------

// The exponent form: 2^(c jc^2), |jc| <= kCols / 2 + 1 in a row, may multiply rho while it
// stays a normal float with room for K' beside it (split); the chain form also
// needs every K' a lane steps through to stay one: a column of the union row is
// at most kCols + 3 sigma_z / (sqrt(2) pw) pixels from the event's row peak (the
// row's half width), where K >= 2^(c D^2) times the row's own 2^-6.5.
template <class C>
int u_exponent_form(const DevGeom& g, const FastConst& fc) {
  const float cz = -fc.kz * g.pixel_width * g.pixel_width;
  const float half = 0.5f * C::kCols + 1.0f;
  if (cz * half * half > 80.0f) return kXFull;
  const float d = C::kCols + 2.1213204f * g.sigma_z / g.pixel_width;
  return cz * d * d <= 111.0f ? kXChain : kXSplit;
}

template <class C, int ACC, bool DEN64>
cudaError_t u_prepare() {
  cudaError_t e = cudaSuccess;
  for (auto* k : {iterate_union_kernel<C, kXFull, ACC, DEN64>,
                  iterate_union_kernel<C, kXSplit, ACC, DEN64>,
                  iterate_union_kernel<C, kXChain, ACC, DEN64>})
    if (e == cudaSuccess) e = allow_shared_memory(reinterpret_cast<const void*>(k));
  return e;
}

template <class C>
struct UnionHost {
  static size_t smem(const Tiling& t, int precision) {
    switch (precision) {
      case kPrecisionCompensated: return u_smem<C, kAccCompensated, false>(t);
      case kPrecisionCompensatedDen64: return u_smem<C, kAccCompensated, true>(t);
      case kPrecisionFixed: return u_smem<C, kAccFixed, false>(t);
      default: return u_smem<C, kAccFloat, false>(t);
    }
  }
  static cudaError_t prepare(int precision) {
    switch (precision) {
      case kPrecisionCompensated: return u_prepare<C, kAccCompensated, false>();
      case kPrecisionCompensatedDen64: return u_prepare<C, kAccCompensated, true>();
      case kPrecisionFixed: return u_prepare<C, kAccFixed, false>();
      default: return u_prepare<C, kAccFloat, false>();
    }
  }
  static cudaError_t launch(const DevGeom& g, const FastConst& fc, const Tiling& t,
                            const Chunk* chunks, int32_t n_chunks, const float4* ev_geom,
                            const short4* ev_box, const float4* records, const uint16_t* urows,
                            const uint32_t* batches, const float* rho, float* out, AuxImage aux,
                            DevCounters* counters, int precision, uint32_t seed,
                            cudaStream_t s) {
    const int xm = u_exponent_form<C>(g, fc);
    const size_t bytes = smem(t, precision);
    auto go = [&](auto acc, auto den64) {
      constexpr int ACC = decltype(acc)::value;
      constexpr bool DEN64 = decltype(den64)::value;
      auto* k = xm == kXChain   ? iterate_union_kernel<C, kXChain, ACC, DEN64>
                : xm == kXSplit ? iterate_union_kernel<C, kXSplit, ACC, DEN64>
                                : iterate_union_kernel<C, kXFull, ACC, DEN64>;
      k<<<n_chunks, C::kThreads, bytes, s>>>(g, fc, t, chunks, ev_geom, ev_box, records, urows,
                                             batches, rho, out, aux, seed, counters);
      return cudaGetLastError();
    };
    using std::integral_constant;
    switch (precision) {
      case kPrecisionCompensated:
        return go(integral_constant<int, kAccCompensated>{}, std::false_type{});
      case kPrecisionCompensatedDen64:
        return go(integral_constant<int, kAccCompensated>{}, std::true_type{});
      case kPrecisionFixed: return go(integral_constant<int, kAccFixed>{}, std::false_type{});
      default: return go(integral_constant<int, kAccFloat>{}, std::false_type{});
    }
  }
  static UnionOps ops() {
    return UnionOps{C::kThreads, C::E, C::kRows, C::kCols, smem, prepare, launch};
  }
};

}  // namespace
}  // namespace jpet
