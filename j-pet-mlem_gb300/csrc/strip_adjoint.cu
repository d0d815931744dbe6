// Adjoint of the list-mode Poisson likelihood of the strip MLEM model.
//
//   L(rho, sigma) = sum_p s_p rho_p - sum_e log( sum_{p in E_e} K_e(p; sigma) rho_p )
//   dL/drho_p     = s_p - sum_e K_e(p) / den_e
//   dL/dsigma     = - sum_e ( sum_p dK_e(p)/dsigma rho_p ) / den_e
//
// K is the reference's Gaussian kernel (src/2d/strip/gaussian_kernel.h:51-79)
// with its normalisation c0 = 1/(2 pi^2) ipz sqrt(ipd) included, so that
// d log K / d ipz = 1/ipz - Pa/(2 aMa) - u^2 and
// d log K / d ipd = 1/(2 ipd) - Qa/(2 aMa) - 2 sec^2 dy^2, with aMa = Pa ipz + Qa ipd,
// Pa = 2 sec^4 (py^2 + R^2), Qa = 4 sec^2 tan^2 py^2, u = dz - dy tan.  The support
// E_e is the event's 3-sigma ellipse for the handle's sigmas (the row tables),
// held fixed while the kernel sigmas vary.  There is no reference code for this
// path.
//
// The loss has to be a smooth function of sigma to the ~1e-9 relative level for
// central differences with h = 1e-3 mm to resolve it: every sigma-dependent
// constant is rounded differently at sigma +- h, and a float rounding of, e.g.,
// ipd shifts log K of every pixel in the same direction.  So the kernel value
// uses the accurate exp2f (not the .approx form of the MLEM kernel), the row
// prefactor -log2(aMa(py)/aMa(y))/2 - 2 log2(e) ipd sec^2 dy^2 is computed to ~1e-9
// of itself and rounded to float once, the per-pixel coefficient kz = -log2(e)
// ipz is applied as a float pair (kz + kz_lo), and the event constant
// log(c0 / sqrt(aMa(y))) enters the loss in FP64.
//
// One warp per event.  The lanes set up a block of rows, 32 at a time and one each
// (the exact in-ellipse interval of the MLEM row tables, so the support is exactly
// the reference's, read from the row table where the handle has one, and the row's
// terms), then sweep the rows with 4 to 32 lanes each, two pixels a lane; the first kNllCache
// kernel values are kept for the gradient pass, which adds them with FP64
// reductions to one of a few partial images (nll_finish_kernel sums those): in
// float images, eight of them, the sum of 5e6 events of a point source was 4e-5 off
// and that of 5e5 events of 1763 pixels 2.0e-7, for 18.9 instead of 19.7 ms and
// 2.91 instead of 2.97 ms.
//
// This GPU's FP64 pipe is a sixty-fourth of its FP32 one, so FP64 is left where
// one lane's instruction serves one event: a warp takes `group` events, lane j
// prepares event j's FP64 constants before and forms its logarithm and quotients
// after; the row prefactor and the sums over lanes are double-float (pairs of
// FP32 values, Dekker 1971; the sum and product errors are Knuth's TwoSum and an
// FMA).  5e5 events of 1763 pixels (2 mm, support 14 / 55): 8.0 ms with FP64 row
// terms and per-event FP64 on one lane (FP64 pipe 70-81 % busy) and float
// atomics on windows in shared memory, 3.65 ms with all that (FP64 pipe 3 %), bound
// by instruction issue (63 % of the slots, 52 instructions a pixel in either
// pass); 2.92 ms with two pixels a lane in packed arithmetic (rows unrolled by
// 2; by 1, 3 and 4: 3.31, 3.04 and 3.00).
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "strip_device.cuh"
#include "strip_internal.h"
#include "strip_raster.cuh"

namespace jpet {
namespace {

constexpr double kNllLog2e = 1.4426950408889634;
constexpr int kNllWarps = 4;     // warps per CTA
constexpr int kNllCache = 1536;  // kernel values kept per event
constexpr int kNllRows = 96;     // rows of a block (an event's set-up is then kept for the
                                 // gradient pass)
// Rows of more than kNllWide pixels (two per lane): events of several thousand
// pixels, of which the cache would hold a few.  Their kernel keeps none and has
// larger blocks instead, and sweeps rows of any length.  2e5 events of up to 252
// rows x 85 columns (0.5 mm): 16.6 ms with the cache and a second loop past a
// row's first 64 pixels, 9.6 so (inner loop unrolled by 3; 10.4 before additions were
// spared the conversion, where by 2 took 10.5 and by 1 11.9).
constexpr int kNllWide = 64;
constexpr int kNllWideRows = 256;

// ---- double-float arithmetic: h + l, |l| <= ulp(h) / 2 ---------------------------------
struct Pair {
  float h, l;
};
__device__ __forceinline__ Pair pair_of(double v) {
  const float h = __double2float_rn(v);
  return Pair{h, __double2float_rn(v - static_cast<double>(h))};
}
__device__ __forceinline__ Pair two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), v = __fsub_rn(s, a);
  return Pair{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v))};
}
__device__ __forceinline__ Pair two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return Pair{p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {
  Pair p = two_prod(a.h, b.h);
  p.l = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l));
  return p;
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
  Pair s = two_sum(a.h, b.h);
  s.l = __fadd_rn(s.l, __fadd_rn(a.l, b.l));
  return s;
}
// Adds v, a negative normal float unless ANY, to a double.  The conversion instruction
// runs on the FP64 pipe, which one per addition kept 67 % busy (5e5 events of 1763
// pixels 3.22 ms), so the double is made of the float's bits (2.97).  Smaller values
// than normal ones are left out, as float reductions leave them.
template <bool ANY>
__device__ __forceinline__ void add_negative(double* p, float v, bool in) {
  if (ANY) {
    if (in) atomicAdd(p, static_cast<double>(v));
  } else {
    const uint32_t b = __float_as_uint(v);
    if (in && v <= -FLT_MIN)
      atomicAdd(p, __hiloint2double(static_cast<int>((b >> 3) + 0xA8000000u),
                                    static_cast<int>(b << 29)));
  }
}
// sum over the warp's lanes, in FP64
__device__ __noinline__ double warp_sum_f64(float2 v) {
  double s = static_cast<double>(v.x) + v.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
  return s;
}
// sum over the warp's lanes
__device__ __forceinline__ Pair pair_warp_sum(float2 v) {
  Pair s = two_sum(v.x, v.y);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const Pair other{__shfl_xor_sync(kFull, s.h, o), __shfl_xor_sync(kFull, s.l, o)};
    s = pair_add(s, other);
  }
  return s;
}

// -log2(1 + x) / 2 for x in [-1/4, 0.35]: log(1 + x) = 2 artanh(r), r = x / (2 + x),
// with the first term of the series in r a double-float; relative error below
// 5e-9, where the float part of the series is at most a 130th of the whole (it
// grows to 1.5e-8 at x = -0.4 and 1e-8 at 0.6; below -0.6 the series itself is short:
// 1e-6 at -0.75, 1e-3 at -0.9).  Rows of the scanners in use lie within +-0.2.
__device__ __forceinline__ Pair half_neg_log2_1p(Pair x) {
  Pair d = two_sum(2.0f, x.h);
  d.l = __fadd_rn(d.l, x.l);
  const float inv = __frcp_rn(d.h);
  const float q = __fmul_rn(x.h, inv);
  const float rem = __fadd_rn(__fmaf_rn(-q, d.h, x.h), __fmaf_rn(-q, d.l, x.l));
  Pair r{q, __fmul_rn(rem, inv)};
  const float z = q * q;
  float s = 1.0f / 19.0f;
  s = fmaf(s, z, 1.0f / 17.0f);
  s = fmaf(s, z, 1.0f / 15.0f);
  s = fmaf(s, z, 1.0f / 13.0f);
  s = fmaf(s, z, 1.0f / 11.0f);
  s = fmaf(s, z, 1.0f / 9.0f);
  s = fmaf(s, z, 1.0f / 7.0f);
  s = fmaf(s, z, 1.0f / 5.0f);
  s = fmaf(s, z, 1.0f / 3.0f);
  r.l = __fmaf_rn(__fmul_rn(q, z), s, r.l);
  // -log2(e), twice artanh and half of it
  constexpr double c = -kNllLog2e;
  constexpr float ch = static_cast<float>(c);
  constexpr float cl = static_cast<float>(c - static_cast<double>(ch));
  return pair_mul(r, Pair{ch, cl});
}

template <bool WIDE>
struct NllWarp {
  static constexpr int kRows = WIDE ? kNllWideRows : kNllRows;
  float4 row[kRows];        // prefactor exponent, d/dipz and d/dipd terms, u at column 0
  int4 at[kRows];           // pixels before the row | width << 16, image index of its first
                            // pixel, first column (float bits), unused
  float cache[WIDE ? 1 : kNllCache];  // kernel values
};

// (five CTAs per SM where the row table is read, 96 registers: for 5e5 events of 1763
// pixels 3.22 ms against 3.44 with the four of 120 registers; the kernels that compute
// the intervals would spill.  Wide rows 10.5 ms against 11.6, but the loss alone 5.9
// against 5.4.  All four measured with the conversion in add_negative)
template <bool GRAD, bool TABLE, bool WIDE>
__global__ void __launch_bounds__(32 * kNllWarps, (WIDE ? GRAD : TABLE) ? 5 : 1) nll_kernel(
    DevGeom g, NllConst k, int32_t n, int32_t group, const float4* __restrict__ ev_geom,
    const short4* __restrict__ ev_box, const uint16_t* __restrict__ table, int32_t stride,
    const float* __restrict__ rho, double* __restrict__ parts, int32_t n_parts, int64_t n_pix,
    double* __restrict__ acc, unsigned long long* skipped) {
  constexpr int kRows = NllWarp<WIDE>::kRows;
  __shared__ NllWarp<WIDE> shared[kNllWarps];
  NllWarp<WIDE>& s = shared[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int n_warps = (gridDim.x * blockDim.x) >> 5;
  double* grad = GRAD ? parts + static_cast<int64_t>(blockIdx.x % n_parts) * n_pix : nullptr;
  double loss = 0.0, gz = 0.0, gdl = 0.0;
  unsigned long long sk = 0;
  for (int64_t e0 = static_cast<int64_t>(warp) * group; e0 < n;
       e0 += static_cast<int64_t>(n_warps) * group) {
    const int cnt = static_cast<int>(e0 + group <= n ? group : n - e0);
    // lane j: event e0 + j
    float4 ev = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    short4 bx = make_short4(0, 0, 0, 0);
    Pair qq{0.0f, 0.0f}, kd{0.0f, 0.0f};
    double log_ref = 0.0;  // log(c0 / sqrt(aMa(y)))
    if (lane < cnt) {
      ev = ev_geom[e0 + lane];
      bx = ev_box[e0 + lane];
      const float y = ev.y, sec2 = ev.w * ev.w;
      const float pa_c = 2.0f * sec2 * sec2, qa_c = 4.0f * sec2 * ev.z * ev.z;
      const double ama =
          (static_cast<double>(pa_c) * (static_cast<double>(y) * y +
                                        static_cast<double>(g.radius) * g.radius)) * k.ipz_d +
          static_cast<double>(qa_c) * y * y * k.ipd_d;
      // aMa(py) / aMa(y) = 1 + qq (py - y)(py + y)
      qq = pair_of((pa_c * k.ipz_d + qa_c * k.ipd_d) / ama);
      kd = pair_of(k.kdl_d * sec2);
      log_ref = k.log_c0 - 0.5 * log(ama);
    }
    Pair den_j{0.0f, 0.0f}, dz_j{0.0f, 0.0f}, ddl_j{0.0f, 0.0f};
    for (int j = 0; j < cnt; ++j) {
      const float z = __shfl_sync(kFull, ev.x, j), y = __shfl_sync(kFull, ev.y, j);
      const float tn = __shfl_sync(kFull, ev.z, j), sec = __shfl_sync(kFull, ev.w, j);
      const int b0 = __shfl_sync(kFull, static_cast<int>(bx.x) | (static_cast<int>(bx.y) << 16), j);
      const int b1 = __shfl_sync(kFull, static_cast<int>(bx.z) | (static_cast<int>(bx.w) << 16), j);
      const int bx0 = b0 & 0xffff, by0 = b0 >> 16, bx1 = b1 & 0xffff, by1 = b1 >> 16;
      const Pair q{__shfl_sync(kFull, qq.h, j), __shfl_sync(kFull, qq.l, j)};
      const Pair kdl{__shfl_sync(kFull, kd.h, j), __shfl_sync(kFull, kd.l, j)};
      float A, B, C;
      ellipse_abc(g, tn, sec, A, B, C);
      const float sec2 = sec * sec;
      const float pa_c = 2.0f * sec2 * sec2;     // Pa = pa_c (py^2 + R^2)
      const float qa_c = 4.0f * sec2 * tn * tn;  // Qa = qa_c py^2
      const int nrows = by1 - by0;
      int n_rows = 0, total = 0, widest = 0;  // of the block last set up: rows with pixels
      auto setup = [&](int rb) {
        n_rows = total = widest = 0;
        __syncwarp();
        for (int r0 = rb; r0 < min(rb + kRows, nrows); r0 += 32) {
          int first = 0, w = 0;
          const int iy = by0 + r0 + lane;
          if (r0 + lane < nrows) {
            if (TABLE) {
              const uint32_t e = table[(e0 + j) * stride + r0 + lane];
              first = bx0 + static_cast<int>(e & 255u);
              w = static_cast<int>(e >> 8);
            } else {
              w = row_interval(g, A, B, C, z, y, tn, sec, bx0, bx1, iy, first);
            }
          }
          int off = w;  // inclusive sum of the widths
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, off, o);
            if (lane >= o) off += v;
          }
          const int sum = __shfl_sync(kFull, off, 31);
          off += total - w;
          total += sum;
          widest = max(widest, static_cast<int>(__reduce_max_sync(kFull, static_cast<unsigned>(w))));
          const unsigned rows = __ballot_sync(kFull, w > 0);
          if (w > 0) {
            const int r = n_rows + __popc(rows & ((1u << lane) - 1u));
            const float py = g.tl_y_half_h - static_cast<float>(iy) * g.pixel_height;
            const float dy = py - y;
            const float pa = pa_c * (py * py + g.radius * g.radius), qa = qa_c * py * py;
            const float ama = pa * k.ipz + qa * k.ipd;
            // x = qq dy (py + y)
            const Pair ys = two_sum(py, y);
            Pair x = two_prod(dy, ys.h);
            x.l = __fmaf_rn(dy, ys.l, x.l);
            x = pair_mul(x, q);
            Pair a = half_neg_log2_1p(x);
            if (!(x.h >= -0.25f && x.h <= 0.35f))  // beyond the series
              a = pair_of(-0.5 * kNllLog2e *
                          log1p(static_cast<double>(x.h) + static_cast<double>(x.l)));
            a = pair_add(a, pair_mul(two_prod(dy, dy), kdl));
            s.row[r] = make_float4(__fadd_rn(a.h, a.l), k.inv_ipz - 0.5f * pa / ama,
                                   k.half_inv_ipd - 0.5f * qa / ama - 2.0f * sec2 * dy * dy,
                                   g.tl_z_half_w - z - dy * tn);
            s.at[r] = make_int4(min(off, kNllCache) | (w << 16), iy * g.n_z + first,
                                __float_as_int(static_cast<float>(first)), 0);
          }
          n_rows += __popc(rows);
        }
        __syncwarp();
      };
      // f(row, its record, pixel of the row, that and the lane's other pixel as
      // floats, how far on that is, whether there are such pixels) over a block's
      // pixels: two pixels per lane, as many lanes per row as then fit the widest,
      // two rows in flight, lanes past a row's end along without a branch.  A
      // lane's pixels are a row's lanes apart, so that neighbouring lanes read
      // and add to neighbouring pixels.  Wide rows: 16 lanes each, 32 pixels at a
      // time.
      auto walk = [&](auto&& f) {
        const int sh = WIDE ? 4 : widest <= 8 ? 2 : widest <= 16 ? 3 : widest <= 32 ? 4 : 5;
        const int l = lane & ((1 << sh) - 1), on = 1 << sh;
        const float2 fl = make_float2(static_cast<float>(l), static_cast<float>(l + on));
#pragma unroll(WIDE ? 1 : 2)
        for (int r0 = 0; r0 < n_rows; r0 += 32 >> sh) {
          const int r = min(r0 + (lane >> sh), n_rows - 1);
          const int4 at = s.at[r];
          const int w = r == r0 + (lane >> sh) ? at.x >> 16 : 0;
          if constexpr (WIDE) {
#pragma unroll 3
            for (int i = 0; i < widest; i += 32) {
              const float fi = static_cast<float>(i);
              f(r, at, i + l, __fadd2_rn(fl, make_float2(fi, fi)), 16, i + l < w, i + l + 16 < w);
            }
          } else {
            f(r, at, l, fl, on, l < w, l + on < w);
          }
        }
      };
      auto value = [&](const float4 r, float2 col, float2& u) {
        u = __ffma2_rn(col, make_float2(g.pixel_width, g.pixel_width), make_float2(r.w, r.w));
        const float2 lo = __ffma2_rn(__fmul2_rn(make_float2(k.kz_lo, k.kz_lo), u), u,
                                     make_float2(r.x, r.x));
        const float2 e = __ffma2_rn(__fmul2_rn(make_float2(k.kz, k.kz), u), u, lo);
        return make_float2(exp2f(e.x), exp2f(e.y));
      };
      float2 den = make_float2(0.0f, 0.0f), dz = den, ddl = den;
      int before = 0;  // pixels of the blocks before
      for (int rb = 0; rb < nrows; rb += kRows) {
        setup(rb);
        walk([&](int r, const int4 at, int i, float2 fi, int on, bool in0, bool in1) {
          const float4 row = s.row[r];
          const float* rp = &rho[at.y + i];
          const float2 rh = make_float2(in0 ? __ldg(rp) : 0.0f, in1 ? __ldg(rp + on) : 0.0f);
          const float first = __int_as_float(at.z);
          float2 u;
          const float2 kv = value(row, __fadd2_rn(make_float2(first, first), fi), u);
          float2 kr = __fmul2_rn(kv, rh);
          kr.x = in0 ? kr.x : 0.0f;
          kr.y = in1 ? kr.y : 0.0f;
          den = __fadd2_rn(den, kr);
          dz = __ffma2_rn(kr, __ffma2_rn(make_float2(-u.x, -u.y), u, make_float2(row.y, row.y)),
                          dz);
          ddl = __ffma2_rn(kr, make_float2(row.z, row.z), ddl);
          if constexpr (GRAD && !WIDE) {
            const int c = before + (at.x & 0xffff) + i;
            if (in0 && c < kNllCache) s.cache[c] = kv.x;
            if (in1 && c + on < kNllCache) s.cache[c + on] = kv.y;
          }
        });
        before = min(before + total, kNllCache);
      }
      const Pair d = pair_warp_sum(den);
      dz = make_float2(dz.x * k.dipz_dsz, dz.y * k.dipz_dsz);
      ddl = make_float2(ddl.x * k.dipd_dsdl, ddl.y * k.dipd_dsdl);
      const Pair a = pair_warp_sum(dz), b = pair_warp_sum(ddl);
      float minus_inv;
      bool any = false;  // -K / den may be any float
      // (the sum of the three is not finite if one of them is not)
      if (fabsf(d.h) + fabsf(a.h) + fabsf(b.h) <= FLT_MAX && !(d.h > 0.0f && d.h < FLT_MIN)) {
        if (lane == j) {
          den_j = d;
          dz_j = a;
          ddl_j = b;
        }
        if (!GRAD || !(d.h > 0.0f)) continue;
        const float i0 = __frcp_rn(d.h);
        minus_inv = -fmaf(fmaf(-d.h, i0, 1.0f) - d.l * i0, i0, i0);
      } else {  // beyond what FP32 holds, or a quotient of which is: all in FP64
        const double dd = warp_sum_f64(den), ad = warp_sum_f64(dz), bd = warp_sum_f64(ddl);
        if (lane == j) {
          den_j.h = CUDART_NAN_F;  // done
          if (dd > 0.0) {
            loss -= log(dd) + log_ref;
            gz -= ad / dd;
            gdl -= bd / dd;
          } else {
            ++sk;
          }
        }
        if (!GRAD || !(dd > 0.0)) continue;
        minus_inv = -static_cast<float>(1.0 / dd);
        any = true;
      }
      auto gradient = [&](auto any_float) {
        constexpr bool ANY = decltype(any_float)::value;
        before = 0;
        for (int rb = 0; rb < nrows; rb += kRows) {
          if (nrows > kRows) setup(rb);
          walk([&](int r, const int4 at, int i, float2 fi, int on, bool in0, bool in1) {
            const int c = WIDE ? kNllCache : before + (at.x & 0xffff) + i;
            float2 kv = make_float2(0.0f, 0.0f);
            if constexpr (!WIDE)
              kv = make_float2(s.cache[min(c, kNllCache - 1)], s.cache[min(c + on, kNllCache - 1)]);
            if (in0 && c + on >= kNllCache) {  // not kept (either pixel, or none in the row)
              const float first = __int_as_float(at.z);
              float2 u;
              const float2 v = value(s.row[r], __fadd2_rn(make_float2(first, first), fi), u);
              if (c >= kNllCache) kv.x = v.x;
              kv.y = v.y;
            }
            add_negative<ANY>(&grad[at.y + i], kv.x * minus_inv, in0);
            add_negative<ANY>(&grad[at.y + i + on], kv.y * minus_inv, in1);
          });
          before = min(before + total, kNllCache);
        }
      };
      if (any)
        gradient(std::true_type{});
      else
        gradient(std::false_type{});
      __syncwarp();  // the next event's set-up overwrites the rows
    }
    if (lane < cnt) {
      const double dd = static_cast<double>(den_j.h) + static_cast<double>(den_j.l);
      if (dd > 0.0) {
        // log of the absolute denominator: K = K_ref K', K_ref = c0 / sqrt(aMa(y))
        loss -= log(dd) + log_ref;
        const double inv = 1.0 / dd;
        gz -= (static_cast<double>(dz_j.h) + static_cast<double>(dz_j.l)) * inv;
        gdl -= (static_cast<double>(ddl_j.h) + static_cast<double>(ddl_j.l)) * inv;
      } else if (den_j.h == den_j.h) {  // not done
        ++sk;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    loss += __shfl_xor_sync(kFull, loss, o);
    gz += __shfl_xor_sync(kFull, gz, o);
    gdl += __shfl_xor_sync(kFull, gdl, o);
  }
  sk = warp_sum_u64(sk);
  if (lane == 0) {
    atomicAdd(&acc[0], loss);
    atomicAdd(&acc[1], gz);
    atomicAdd(&acc[2], gdl);
    if (sk) atomicAdd(skipped, sk);
  }
}

// grad = s + the partial images; acc[0] += sum s * rho
__global__ void nll_finish_kernel(const float* __restrict__ s, const float* __restrict__ rho,
                                  const double* __restrict__ parts, int32_t n_parts,
                                  float* __restrict__ grad, double* acc, int64_t n) {
  __shared__ double part[8];
  double v = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float si = s[i];
    v += static_cast<double>(si) * rho[i];
    if (grad) {
      double t = si;
      for (int32_t p = 0; p < n_parts; ++p) t += parts[p * n + i];
      grad[i] = __double2float_rn(t);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += part[w];
    atomicAdd(&acc[0], t);
  }
}

}  // namespace

NllConst make_nll_const(double sigma_z, double sigma_dl) {
  NllConst k;
  const double ipz = 1.0 / (sigma_z * sigma_z), ipd = 1.0 / (sigma_dl * sigma_dl);
  k.ipz = static_cast<float>(ipz);
  k.ipd = static_cast<float>(ipd);
  k.kz = static_cast<float>(-kNllLog2e * ipz);
  k.kz_lo = static_cast<float>(-kNllLog2e * ipz - static_cast<double>(k.kz));
  k.ipz_d = ipz;
  k.ipd_d = ipd;
  k.kdl_d = -2.0 * kNllLog2e * ipd;
  k.inv_ipz = static_cast<float>(1.0 / ipz);
  k.half_inv_ipd = static_cast<float>(0.5 / ipd);
  k.dipz_dsz = static_cast<float>(-2.0 / (sigma_z * sigma_z * sigma_z));
  k.dipd_dsdl = static_cast<float>(-2.0 / (sigma_dl * sigma_dl * sigma_dl));
  k.log_c0 = std::log(1.0 / (2.0 * 3.14159265358979323846 * 3.14159265358979323846) * ipz *
                      std::sqrt(ipd));
  return k;
}

// Partial gradient images: where many events share a pixel, additions to one image
// wait for each other (5e6 events of a point source at 2 mm, widths 10 / 42 and 14 / 55: 35
// and 54 ms with one image, 21.5 and 35 with 4, 19.8 and 35 with 8, 19.7 and 26.7 with 16, as
// with 32); sets of fewer events do with 4, and so do their clearing and adding up.
// Together they stay in L2: 32 MB.
int nll_grad_parts(int64_t n_pix, int64_t n_events) {
  int parts = n_events >= (int64_t(1) << 20) ? 16 : 4;
  while (parts > 1 && parts * n_pix > (int64_t(1) << 22)) parts /= 2;
  return parts;
}

cudaError_t launch_nll(const DevGeom& g, const NllConst& k, int32_t n, const float4* ev_geom,
                       const short4* ev_box, const uint16_t* table, int32_t stride,
                       const float* rho, double* parts, int32_t n_parts, double* acc,
                       unsigned long long* skipped, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  // events per warp: up to 32, so that the FP64 of a lane serves an event, but
  // enough warps to fill the SMs (152 x 28)
  int group = 32;
  while (group > 2 && n / group < 2 * 152 * 28) group /= 2;
  const int64_t n_pix = static_cast<int64_t>(g.n_y) * g.n_z;
  const int warps = (n + group - 1) / group;
  const int blocks = std::min((warps + kNllWarps - 1) / kNllWarps, 152 * 7 * 4);
  auto go = [&](auto wide) {
    constexpr bool W = decltype(wide)::value;
    auto* kern = parts ? (table ? nll_kernel<true, true, W> : nll_kernel<true, false, W>)
                       : (table ? nll_kernel<false, true, W> : nll_kernel<false, false, W>);
    kern<<<blocks, 32 * kNllWarps, 0, s>>>(g, k, n, group, ev_geom, ev_box, table, stride, rho,
                                           parts, n_parts, n_pix, acc, skipped);
    return cudaGetLastError();
  };
  return row_span(g) >= kNllWide - 0.1 ? go(std::true_type{}) : go(std::false_type{});
}

cudaError_t launch_nll_finish(const float* sens, const float* rho, const double* parts,
                              int32_t n_parts, float* grad, double* acc, int64_t n,
                              cudaStream_t s) {
  nll_finish_kernel<<<152 * 4, 256, 0, s>>>(sens, rho, parts, n_parts, grad, acc, n);
  return cudaGetLastError();
}

}  // namespace jpet
