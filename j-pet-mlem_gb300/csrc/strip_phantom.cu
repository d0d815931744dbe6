// Seeded list-mode event generator for the strip scanner on the GPU (the
// phantom tool's Monte Carlo, src/2d/strip/phantom_cmd.cpp:136-444,
// src/common/phantom_monte_carlo.h:33-109).
//
// Every candidate emission has a 64-bit index; its random numbers are the
// Philox4x32-10 counter-based generator (Salmon, Moraes, Dror and Shaw,
// "Parallel random numbers: as easy as 1, 2, 3", SC 2011) at counter
// (index, draw) under the caller's 64-bit seed, so the event stream depends
// only on (regions, scanner, seed) and not on the launch shape.  A candidate:
//
//  1. picks a region with probability weight / total weight (ellipse and
//     rectangle: intensity x area, point: intensity; phantom.h:120-133,183-191);
//  2. draws a uniform point in it: ellipse r = sqrt(U), theta = 2 pi U, scaled
//     by the semi-axes and rotated (ellipse.h:83-91); rectangle uniform in
//     [x - a, x + a] x [y - b, y + b] (rectangle.h:20-51); point exact.  Unless
//     the regions are additive, a point inside an earlier-listed region is not
//     an emission (phantom.h:193-204: the reference redraws, which gives the
//     same distribution of emissions);
//  3. draws the direction angle uniform in (-phi_max, phi_max): pi/2 when
//     emissions are counted (phantom.h:213), atan(L / 2R) when detected events
//     are counted (every detected event has |tan| < L / 2R, so the accepted
//     events have the same distribution);
//  4. projects onto the strips, z_u = z + (R - y) tan, z_d = z - (R + y) tan,
//     dl = -2 y sqrt(1 + tan^2) (scanner.h:107-113), and is detected iff
//     |z_u|, |z_d| < L/2 on the exact values (scanner.h:208-213);
//  5. adds N(0, sigma_z) to z_u, z_d and N(0, sigma_dl) to dl (scanner.h:257-267,
//     Box-Muller normals), with no second acceptance test.
//
// Detected events are written in candidate order (a decision pass, a scan over
// blocks and an ordered write pass), so the output is deterministic as well.
//
// Steps 1 to 4 are FP64 arithmetic by definition, and this GPU's FP64 pipe is a
// sixty-fourth of its FP32 one.  The decision pass therefore evaluates them in
// FP32 together with a bound on its own error, and only the candidates within
// the bound of a decision (about 1e-4 of them) go through the FP64 arithmetic:
// the decisions are those of the FP64 code.  It leaves one bit per candidate,
// from which the write pass compacts each block's accepted candidates and
// evaluates those alone in FP64, all threads busy.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/jpet_strip.h"
#include "strip_device.cuh"
#include "strip_internal.h"

namespace jpet {
namespace {

struct GenRegion {
  int32_t kind;
  double x, y, a, b;
  double s, c;     // rotation
  double A, B, C;  // ellipse: A dx^2 + 2 C dx dy + B dy^2 <= 1
  double cdf;      // cumulative normalised weight
};

struct GenParams {
  double R, L, sigma_z, sigma_dl, phi_max;
  uint32_t key0, key1;
  int32_t n_regions, additive;
};

constexpr int kGenThreads = 256;
constexpr int kGenRounds = 4;  // 1024 candidates per block: small calls still spread over the SMs
constexpr int kGenPerBlock = kGenThreads * kGenRounds;
constexpr int kGenWords = kGenPerBlock / 32;
constexpr int kGenMaxBlocks = 4096;  // 4 Mi candidates per pass at most
constexpr int kGenMaxRegions = 256;

__device__ __forceinline__ void philox_round(uint32_t (&x)[4], uint32_t k0, uint32_t k1) {
  const uint32_t m0 = 0xD2511F53u, m1 = 0xCD9E8D57u;
  const uint32_t hi0 = __umulhi(m0, x[0]), lo0 = m0 * x[0];
  const uint32_t hi1 = __umulhi(m1, x[2]), lo1 = m1 * x[2];
  const uint32_t y0 = hi1 ^ x[1] ^ k0, y2 = hi0 ^ x[3] ^ k1;
  x[0] = y0;
  x[1] = lo1;
  x[2] = y2;
  x[3] = lo0;
}

// Philox4x32-10: ten rounds, the key advanced by the Weyl constants between rounds
__device__ __forceinline__ void philox(uint32_t (&x)[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    philox_round(x, k0, k1);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__device__ __forceinline__ unsigned long long warp_add(unsigned long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 53-bit uniform in [0, 1)
__device__ __forceinline__ double u53(uint32_t a, uint32_t b) {
  return (static_cast<double>(a >> 5) * 67108864.0 + static_cast<double>(b >> 6)) *
         (1.0 / 9007199254740992.0);
}

struct Candidate {
  bool emitted, detected;
  float zu, zd, dl;
  double px, py;        // emission point
  float ex_zu, ex_zd, ex_dl;  // exact (unsmeared) response
  float dir_x, dir_y;   // emission direction (sin phi, cos phi)
};

// Optional count images of the phantom tool (phantom_cmd.cpp:249-258,289-352):
// a PixelGrid with its lower-left corner at -(n_z, n_y) s / 2 + origin, pixel
// (floor((z - x0) / s), floor((y - y0) / s)), index row * n_z + column.
struct GenImages {
  int32_t* emitted;   // emission points of all emissions counted
  int32_t* detected;  // emission points of the detected events
  int32_t* naive;     // points recovered from the smeared responses
  int32_t* tan_map;   // the same, binned also by tangent
  float* exact;       // exact responses of the written events (3 floats each)
  float* events;      // their emission events (x, y, dx, dy)
  double x0, y0, s;
  int32_t n_z, n_y, tan_bins;
  // the grid in the reference's float: lower-left corner, pixel size, 2R, the
  // first tangent plane's lower edge and the plane width
  float fx0, fy0, fs, two_r, tan_left, tan_size;
};

// Naive point of a smeared response and its bins, in float without
// contraction as the reference's host code computes them:
// Response::calculate_tan_y_z (response.h:22-37), PixelGrid::pixel_at
// (pixel_grid.h:59-64), VariableVoxelSizeVoxelGrid::voxel_at (voxel_grid.h:109-118).
__device__ __forceinline__ void naive_add(const GenImages& im, float zu, float zd, float dl) {
  const float t = __fdiv_rn(__fsub_rn(zu, zd), im.two_r);
  const float y = __fmul_rn(-0.5f, __fdiv_rn(dl, __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(t, t)))));
  const float z = __fmul_rn(0.5f, __fadd_rn(__fadd_rn(zu, zd), __fmul_rn(__fmul_rn(2.0f, y), t)));
  const float col = floorf(__fdiv_rn(__fsub_rn(z, im.fx0), im.fs));
  const float row = floorf(__fdiv_rn(__fsub_rn(y, im.fy0), im.fs));
  if (!(col >= 0.0f && col < static_cast<float>(im.n_z) && row >= 0.0f &&
        row < static_cast<float>(im.n_y)))
    return;
  const int pix = static_cast<int>(row) * im.n_z + static_cast<int>(col);
  if (im.naive) atomicAdd(&im.naive[pix], 1);
  if (im.tan_map) {
    const float plane = floorf(__fdiv_rn(__fsub_rn(t, im.tan_left), im.tan_size));
    if (plane >= 0.0f && plane < static_cast<float>(im.tan_bins))
      atomicAdd(&im.tan_map[static_cast<size_t>(plane) * im.n_y * im.n_z + pix], 1);
  }
}

__device__ __forceinline__ void image_add(int32_t* img, const GenImages& im, double z, double y) {
  if (!img) return;
  const double cz = floor((z - im.x0) / im.s), cy = floor((y - im.y0) / im.s);
  if (cz >= 0.0 && cz < im.n_z && cy >= 0.0 && cy < im.n_y)
    atomicAdd(&img[static_cast<int>(cy) * im.n_z + static_cast<int>(cz)], 1);
}

__device__ Candidate gen_candidate(const GenParams& p, const GenRegion* __restrict__ regs,
                                   uint64_t index) {
  const uint32_t lo = static_cast<uint32_t>(index), hi = static_cast<uint32_t>(index >> 32);
  uint32_t r0[4] = {lo, hi, 0u, 0u};
  uint32_t r1[4] = {lo, hi, 1u, 0u};
  philox(r0, p.key0, p.key1);
  philox(r1, p.key0, p.key1);
  Candidate out{false, false, 0.f, 0.f, 0.f, 0.0, 0.0, 0.f, 0.f, 0.f, 0.f, 0.f};
  // region by cumulative weight (phantom.h:183-191: the first cdf >= u)
  const double u_reg = u53(r0[0], r0[1]);
  int k = 0;
  while (k < p.n_regions - 1 && u_reg > regs[k].cdf) ++k;
  const GenRegion& rg = regs[k];
  const double u1 = u53(r0[2], r0[3]), u2 = u53(r1[0], r1[1]);
  double px, py;
  if (rg.kind == JPET_REGION_ELLIPSE) {
    const double rr = sqrt(u1);
    double st, ct;
    sincospi(2.0 * u2, &st, &ct);
    const double ex = rg.a * rr * ct, ey = rg.b * rr * st;
    px = rg.c * ex - rg.s * ey + rg.x;
    py = rg.s * ex + rg.c * ey + rg.y;
  } else if (rg.kind == JPET_REGION_RECTANGLE) {
    px = rg.x + rg.a * (2.0 * u1 - 1.0);
    py = rg.y + rg.b * (2.0 * u2 - 1.0);
  } else {
    px = rg.x;
    py = rg.y;
  }
  if (!p.additive) {
    for (int i = 0; i < k; ++i) {
      const GenRegion& q = regs[i];
      const double dx = px - q.x, dy = py - q.y;
      bool inside;
      if (q.kind == JPET_REGION_ELLIPSE)
        inside = q.A * dx * dx + 2.0 * q.C * dx * dy + q.B * dy * dy <= 1.0;
      else if (q.kind == JPET_REGION_RECTANGLE)
        inside = fabs(dx) <= q.a && fabs(dy) <= q.b;
      else
        inside = dx == 0.0 && dy == 0.0;
      if (inside) return out;
    }
  }
  out.emitted = true;
  out.px = px;
  out.py = py;
  const double phi = p.phi_max * (2.0 * u53(r1[2], r1[3]) - 1.0);
  const double t = tan(phi);
  const double zu = px + (p.R - py) * t;
  const double zd = px - (p.R + py) * t;
  const double dl = -2.0 * py * sqrt(t * t + 1.0);
  const double half = 0.5 * p.L;
  if (!(fabs(zu) < half && fabs(zd) < half)) return out;
  out.detected = true;
  out.ex_zu = static_cast<float>(zu);
  out.ex_zd = static_cast<float>(zd);
  out.ex_dl = static_cast<float>(dl);
  {
    double sp, cp;
    sincos(phi, &sp, &cp);
    out.dir_x = static_cast<float>(sp);
    out.dir_y = static_cast<float>(cp);
  }
  // Box-Muller on two pairs of uniforms (1 - U in (0, 1]) gives the normals
  uint32_t r2[4] = {lo, hi, 2u, 0u};
  uint32_t r3[4] = {lo, hi, 3u, 0u};
  philox(r2, p.key0, p.key1);
  philox(r3, p.key0, p.key1);
  const double m0 = sqrt(-2.0 * log(1.0 - u53(r2[0], r2[1])));
  const double m1 = sqrt(-2.0 * log(1.0 - u53(r3[0], r3[1])));
  double s0, c0, s1, c1;
  sincospi(2.0 * u53(r2[2], r2[3]), &s0, &c0);
  sincospi(2.0 * u53(r3[2], r3[3]), &s1, &c1);
  out.zu = static_cast<float>(zu + p.sigma_z * m0 * c0);
  out.zd = static_cast<float>(zd + p.sigma_z * m0 * s0);
  out.dl = static_cast<float>(dl + p.sigma_dl * m1 * c1);
  return out;
}

// ---- FP64 functions of the write pass -----------------------------------------------
//
// The accepted candidates need eight uniforms, four square roots, three sines
// and cosines, a tangent and two logarithms.  On ranges as plain as these (a
// fraction of a turn, an angle below a right angle, a number in (0, 1]) the
// textbook series take about 190 FP64 operations, all within a few units in
// 1e-16, where the library's functions take about 1800 (2e6 events: 7.5 ms of
// write pass with them, 1.1 ms with these).

// 1 / x and sqrt(x): the FP32 value and two Newton steps (x > 0, normal, and
// within FP32's range).
__device__ __forceinline__ double gen_rcp(double x) {
  double y = static_cast<double>(__frcp_rn(static_cast<float>(x)));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
__device__ __forceinline__ double gen_sqrt(double x) {
  const double h = 0.5 * static_cast<double>(rsqrtf(static_cast<float>(x)));
  double r = 2.0 * h * x;
  r = fma(fma(-r, r, x), h, r);
  return fma(fma(-r, r, x), h, r);
}

// sin r and cos r for |r| <= pi / 4 + 1e-8: their Taylor series to r^15 and r^16.
__device__ __forceinline__ void gen_sincos_small(double r, double& sn, double& cs) {
  const double z = r * r;
  double a = -1.0 / 1307674368000.0;
  a = fma(a, z, 1.0 / 6227020800.0);
  a = fma(a, z, -1.0 / 39916800.0);
  a = fma(a, z, 1.0 / 362880.0);
  a = fma(a, z, -1.0 / 5040.0);
  a = fma(a, z, 1.0 / 120.0);
  a = fma(a, z, -1.0 / 6.0);
  sn = fma(a * z, r, r);
  double b = 1.0 / 20922789888000.0;
  b = fma(b, z, -1.0 / 87178291200.0);
  b = fma(b, z, 1.0 / 479001600.0);
  b = fma(b, z, -1.0 / 3628800.0);
  b = fma(b, z, 1.0 / 40320.0);
  b = fma(b, z, -1.0 / 720.0);
  b = fma(b, z, 1.0 / 24.0);
  b = fma(b, z, -0.5);
  cs = fma(b, z, 1.0);
}

// sin and cos of the turn u = u53(hi, ...): the nearest quarter turn from the
// uniform's top bits, the rest by the series.
__device__ __forceinline__ void gen_sincos_turn(uint32_t hi, double u, double& sn, double& cs) {
  const uint32_t n = (hi >> 30) + ((hi >> 29) & 1u);
  double a, b;
  gen_sincos_small(fma(4.0, u, -static_cast<double>(n)) * 1.5707963267948966, a, b);
  const double x = (n & 1u) ? b : a, y = (n & 1u) ? a : b;
  sn = (n & 2u) ? -x : x;
  cs = ((n + 1u) & 2u) ? -y : y;
}

// log x for x in (0, 1]: x = m 2^e with m in [sqrt(1/2), sqrt(2)), and log m =
// 2 artanh((m - 1) / (m + 1)) by its series to the 21st power.
__device__ __forceinline__ double gen_log(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  int e = (hi >> 20) - 1023;
  int mh = (hi & 0x000fffff) | 0x3ff00000;
  if (mh >= 0x3ff6a09e) {  // above sqrt(2)
    mh -= 0x00100000;
    ++e;
  }
  const double m = __hiloint2double(mh, lo);
  const double s = (m - 1.0) * gen_rcp(m + 1.0), z = s * s;
  double a = 1.0 / 21.0;
  a = fma(a, z, 1.0 / 19.0);
  a = fma(a, z, 1.0 / 17.0);
  a = fma(a, z, 1.0 / 15.0);
  a = fma(a, z, 1.0 / 13.0);
  a = fma(a, z, 1.0 / 11.0);
  a = fma(a, z, 1.0 / 9.0);
  a = fma(a, z, 1.0 / 7.0);
  a = fma(a, z, 1.0 / 5.0);
  a = fma(a, z, 1.0 / 3.0);
  const double s2 = 2.0 * s;
  return fma(static_cast<double>(e), 0.69314718055994530942, fma(a * z, s2, s2));
}

// gen_candidate for a candidate known to be detected.
__device__ __forceinline__ Candidate gen_detected(const GenParams& p,
                                                  const GenRegion* __restrict__ regs,
                                                  uint64_t index) {
  const uint32_t lo = static_cast<uint32_t>(index), hi = static_cast<uint32_t>(index >> 32);
  uint32_t r0[4] = {lo, hi, 0u, 0u};
  uint32_t r1[4] = {lo, hi, 1u, 0u};
  uint32_t r2[4] = {lo, hi, 2u, 0u};
  uint32_t r3[4] = {lo, hi, 3u, 0u};
  philox(r0, p.key0, p.key1);
  philox(r1, p.key0, p.key1);
  philox(r2, p.key0, p.key1);
  philox(r3, p.key0, p.key1);
  const double u_reg = u53(r0[0], r0[1]);
  int k = 0;
  while (k < p.n_regions - 1 && u_reg > regs[k].cdf) ++k;
  const GenRegion& rg = regs[k];
  const double u1 = u53(r0[2], r0[3]), u2 = u53(r1[0], r1[1]);
  double px = rg.x, py = rg.y;
  if (rg.kind == JPET_REGION_ELLIPSE) {
    double st, ct;
    gen_sincos_turn(r1[0], u2, st, ct);
    const double rr = u1 > 0.0 ? gen_sqrt(u1) : 0.0;
    const double ex = rg.a * rr * ct, ey = rg.b * rr * st;
    px = rg.c * ex - rg.s * ey + rg.x;
    py = rg.s * ex + rg.c * ey + rg.y;
  } else if (rg.kind == JPET_REGION_RECTANGLE) {
    px = rg.x + rg.a * (2.0 * u1 - 1.0);
    py = rg.y + rg.b * (2.0 * u2 - 1.0);
  }
  // the angle's sine and cosine: beyond pi / 4 those of the complement, swapped
  const double phi = p.phi_max * (2.0 * u53(r1[2], r1[3]) - 1.0);
  const double ap = fabs(phi);
  const bool steep = ap > 0.78539816339744831;
  double sp, cp;
  gen_sincos_small(steep ? (1.5707963267948966 - ap) + 6.123233995736766e-17 : ap, sp, cp);
  if (steep) {
    const double v = sp;
    sp = cp;
    cp = v;
  }
  if (phi < 0.0) sp = -sp;
  const double sec = gen_rcp(cp), t = sp * sec;
  const double zu = px + (p.R - py) * t;
  const double zd = px - (p.R + py) * t;
  const double dl = -2.0 * py * sec;
  const double x0 = 1.0 - u53(r2[0], r2[1]), x1 = 1.0 - u53(r3[0], r3[1]);
  const double l0 = -2.0 * gen_log(x0), l1 = -2.0 * gen_log(x1);
  const double m0 = l0 > 0.0 ? gen_sqrt(l0) : 0.0, m1 = l1 > 0.0 ? gen_sqrt(l1) : 0.0;
  double s0, c0, s1, c1;
  gen_sincos_turn(r2[2], u53(r2[2], r2[3]), s0, c0);
  gen_sincos_turn(r3[2], u53(r3[2], r3[3]), s1, c1);
  Candidate out{true, true, 0.f, 0.f, 0.f, px, py, 0.f, 0.f, 0.f, 0.f, 0.f};
  out.zu = static_cast<float>(zu + p.sigma_z * m0 * c0);
  out.zd = static_cast<float>(zd + p.sigma_z * m0 * s0);
  out.dl = static_cast<float>(dl + p.sigma_dl * m1 * c1);
  out.ex_zu = static_cast<float>(zu);
  out.ex_zd = static_cast<float>(zd);
  out.ex_dl = static_cast<float>(dl);
  out.dir_x = static_cast<float>(sp);
  out.dir_y = static_cast<float>(cp);
  return out;
}

// A region in FP32, for the decision pass.
struct GenRegionF {
  float x, y, a, b, s, c, A, B, C, cdf;
  int32_t kind;
};

constexpr int kGenNo = 0, kGenEmitted = 1, kGenDetected = 2, kGenUnsure = 3;

// The decision of gen_candidate (not an emission, emitted, detected) in FP32, or
// kGenUnsure where a comparison lies within the FP32 error: e counts units of
// 1e-6, about eight times the rounding of the few operations behind each value
// (the library's sinf, cosf and sincospif are within 2 units in the last place).
__device__ __forceinline__ int gen_decide(const GenParams& p, const GenRegionF* regs,
                                          uint64_t index) {
  const uint32_t lo = static_cast<uint32_t>(index), hi = static_cast<uint32_t>(index >> 32);
  uint32_t r0[4] = {lo, hi, 0u, 0u};
  uint32_t r1[4] = {lo, hi, 1u, 0u};
  philox(r0, p.key0, p.key1);
  philox(r1, p.key0, p.key1);
  constexpr float e = 1e-6f, kInv32 = 2.3283064365386963e-10f;
  const float u_reg = static_cast<float>(r0[0]) * kInv32;
  bool unsure = false;
  int k = 0;
  for (int i = 0; i < p.n_regions - 1; ++i) {
    const float d = u_reg - regs[i].cdf;
    unsure = unsure || fabsf(d) < e;
    k += d > 0.0f;
  }
  const GenRegionF rg = regs[k];
  const float u1 = static_cast<float>(r0[2]) * kInv32, u2 = static_cast<float>(r1[0]) * kInv32;
  float px, py;
  if (rg.kind == JPET_REGION_ELLIPSE) {
    const float rr = sqrtf(u1);
    float st, ct;
    sincospif(2.0f * u2, &st, &ct);
    const float ex = rg.a * rr * ct, ey = rg.b * rr * st;
    px = rg.c * ex - rg.s * ey + rg.x;
    py = rg.s * ex + rg.c * ey + rg.y;
  } else if (rg.kind == JPET_REGION_RECTANGLE) {
    px = rg.x + rg.a * (2.0f * u1 - 1.0f);
    py = rg.y + rg.b * (2.0f * u2 - 1.0f);
  } else {
    px = rg.x;
    py = rg.y;
  }
  // error of the point: the uniforms' own rounding moves sqrt(u1) near 0 by up
  // to sqrt(2^-25), which the 1e-3 of the axes next to the centre cover
  const float dp = e * (8.0f * (rg.a + rg.b) + fabsf(rg.x) + fabsf(rg.y)) +
                   (u1 < 10.0f * e ? 1e-3f * (rg.a + rg.b) : 0.0f);
  bool inside = false;
  if (!p.additive) {
    for (int i = 0; i < k; ++i) {
      const GenRegionF q = regs[i];
      const float dx = px - q.x, dy = py - q.y;
      const float ddp = dp + e * (fabsf(q.x) + fabsf(q.y));
      if (q.kind == JPET_REGION_ELLIPSE) {
        const float gx = fabsf(q.A * dx) + fabsf(q.C * dy), gy = fabsf(q.C * dx) + fabsf(q.B * dy);
        const float m = q.A * dx * dx + 2.0f * q.C * dx * dy + q.B * dy * dy;
        const float err = 4.0f * e * (gx * fabsf(dx) + gy * fabsf(dy)) +
                          2.0f * ddp * (gx + gy) + ddp * ddp * (q.A + q.B + 2.0f * fabsf(q.C));
        unsure = unsure || !(fabsf(m - 1.0f) > err);
        inside = inside || m <= 1.0f;
      } else {
        const float ax = fabsf(dx) - q.a, ay = fabsf(dy) - q.b;  // a = b = 0 for a point
        const float err = ddp + e * (q.a + q.b);
        unsure = unsure || (ax < err && ay < err && !(ax < -err && ay < -err));
        inside = inside || (ax <= 0.0f && ay <= 0.0f);
      }
    }
  }
  const float phi = static_cast<float>(p.phi_max) *
                    (2.0f * (static_cast<float>(r1[2]) * kInv32) - 1.0f);
  float sp, cp;
  sincosf(phi, &sp, &cp);
  const float t = sp / cp;
  const float R = static_cast<float>(p.R), half = static_cast<float>(0.5 * p.L);
  const float zu = px + (R - py) * t, zd = px - (R + py) * t;
  const float err = (1.0f + fabsf(t)) * (dp + 2.0f * e * (R + fabsf(px) + fabsf(py))) +
                    2.0f * e * (1.0f + t * t) * (R + fabsf(py)) + 2.0f * e * half;
  const float out = fmaxf(fabsf(zu), fabsf(zd)) - half;
  unsure = unsure || !(fabsf(out) > err);  // also where a value is not finite
  if (unsure) return kGenUnsure;
  return inside ? kGenNo : (out < 0.0f ? kGenDetected : kGenEmitted);
}

// Decision pass: per block of kGenPerBlock candidates, one bit per candidate in
// words (emitted, then detected) and the two counts.  Bound by the integer
// rounds of Philox and the region loop: 2e6 events of ten ellipses took two
// FP64 passes of 16.5 ms each over 4 Mi candidates (count 3.6, write 12.9).
__global__ void __launch_bounds__(kGenThreads)
    gen_decide_kernel(GenParams p, const GenRegion* __restrict__ regs_g, uint64_t cand0,
                      uint32_t* __restrict__ words, int2* __restrict__ block_counts) {
  __shared__ GenRegionF regs[kGenMaxRegions];
  __shared__ int s_count[2][kGenThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < p.n_regions; i += blockDim.x) {
    const GenRegion g = regs_g[i];
    GenRegionF f;
    f.x = static_cast<float>(g.x);
    f.y = static_cast<float>(g.y);
    f.a = g.kind == JPET_REGION_POINT ? 0.0f : static_cast<float>(g.a);
    f.b = g.kind == JPET_REGION_POINT ? 0.0f : static_cast<float>(g.b);
    f.s = static_cast<float>(g.s);
    f.c = static_cast<float>(g.c);
    f.A = static_cast<float>(g.A);
    f.B = static_cast<float>(g.B);
    f.C = static_cast<float>(g.C);
    f.cdf = static_cast<float>(g.cdf);
    f.kind = g.kind;
    regs[i] = f;
  }
  __syncthreads();
  int n_emit = 0, n_det = 0;
  uint32_t* w = words + static_cast<size_t>(blockIdx.x) * 2 * kGenWords;
  for (int r = 0; r < kGenRounds; ++r) {
    const int local = r * kGenThreads + threadIdx.x;
    const uint64_t idx = cand0 + static_cast<uint64_t>(blockIdx.x) * kGenPerBlock + local;
    int d = gen_decide(p, regs, idx);
    if (d == kGenUnsure) {
      const Candidate c = gen_candidate(p, regs_g, idx);
      d = c.detected ? kGenDetected : (c.emitted ? kGenEmitted : kGenNo);
    }
    __syncwarp();
    const uint32_t me = __ballot_sync(0xffffffffu, d != kGenNo);
    const uint32_t md = __ballot_sync(0xffffffffu, d == kGenDetected);
    if (lane == 0) {
      w[local >> 5] = me;
      w[kGenWords + (local >> 5)] = md;
    }
    n_emit += __popc(me);
    n_det += __popc(md);
  }
  if (lane == 0) {
    s_count[0][warp] = n_emit;
    s_count[1][warp] = n_det;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int te = 0, td = 0;
    for (int k = 0; k < kGenThreads / 32; ++k) {
      te += s_count[0][k];
      td += s_count[1][k];
    }
    block_counts[blockIdx.x] = make_int2(te, td);
  }
}

// Exclusive sums of the block counts after the earlier passes' totals, which
// move on by this pass: one CTA.
__global__ void __launch_bounds__(1024)
    gen_scan_kernel(const int2* __restrict__ counts, int blocks, longlong2* __restrict__ base,
                    longlong2* __restrict__ totals) {
  __shared__ long long s_e[32], s_d[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  longlong2 run = *totals;
  __syncthreads();
  for (int b0 = 0; b0 < blocks; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const int2 c = b < blocks ? counts[b] : make_int2(0, 0);
    long long ie = c.x, id = c.y;
    for (int o = 1; o < 32; o <<= 1) {
      const long long ve = __shfl_up_sync(0xffffffffu, ie, o), vd = __shfl_up_sync(0xffffffffu, id, o);
      if (lane >= o) {
        ie += ve;
        id += vd;
      }
    }
    if (lane == 31) {
      s_e[warp] = ie;
      s_d[warp] = id;
    }
    __syncthreads();
    long long we = 0, wd = 0, te = 0, td = 0;
    for (int k = 0; k < 32; ++k) {
      we += k < warp ? s_e[k] : 0;
      wd += k < warp ? s_d[k] : 0;
      te += s_e[k];
      td += s_d[k];
    }
    if (b < blocks) base[b] = make_longlong2(run.x + we + ie - c.x, run.y + wd + id - c.y);
    run.x += te;
    run.y += td;
    __syncthreads();
  }
  if (threadIdx.x == 0) *totals = run;
}

// Write pass: the block's accepted candidates (the detected ones; with EMITTED,
// for count images of the emissions, all emitted ones) compacted into a list,
// each evaluated once in FP64 and written at its rank.  Bound by the FP64 pipe.
template <bool EMITTED>
__global__ void __launch_bounds__(kGenThreads) gen_write_kernel(
    GenParams p, const GenRegion* __restrict__ regs_g, uint64_t cand0,
    const uint32_t* __restrict__ words, const longlong2* __restrict__ block_base, long long limit,
    int count_emissions, long long capacity, unsigned long long* taken, float* __restrict__ out,
    GenImages im) {
  __shared__ GenRegion regs[kGenMaxRegions];
  __shared__ uint32_t w_e[kGenWords], w_d[kGenWords];
  __shared__ int p_e[kGenWords], p_d[kGenWords];  // set bits before each word
  __shared__ uint16_t list[kGenPerBlock];
  static_assert(kGenWords == 32, "one word per lane");
  const int lane = threadIdx.x & 31;
  const longlong2 base = block_base[blockIdx.x];
  if ((count_emissions ? base.x : base.y) >= limit) return;  // past the last event
  for (int i = threadIdx.x; i < p.n_regions; i += blockDim.x) regs[i] = regs_g[i];
  if (threadIdx.x < 32) {
    const uint32_t* w = words + static_cast<size_t>(blockIdx.x) * 2 * kGenWords;
    const uint32_t e = w[lane], d = w[kGenWords + lane];
    int ie = __popc(e), id = __popc(d);
    for (int o = 1; o < 32; o <<= 1) {
      const int ve = __shfl_up_sync(0xffffffffu, ie, o), vd = __shfl_up_sync(0xffffffffu, id, o);
      if (lane >= o) {
        ie += ve;
        id += vd;
      }
    }
    w_e[lane] = e;
    w_d[lane] = d;
    p_e[lane] = ie - __popc(e);
    p_d[lane] = id - __popc(d);
  }
  __syncthreads();
  const uint32_t* w_l = EMITTED ? w_e : w_d;
  const int* p_l = EMITTED ? p_e : p_d;
  for (int c = threadIdx.x; c < kGenPerBlock; c += kGenThreads) {
    const uint32_t w = w_l[c >> 5], bit = 1u << (c & 31);
    if (w & bit) list[p_l[c >> 5] + __popc(w & (bit - 1u))] = static_cast<uint16_t>(c);
  }
  __syncthreads();
  const int n = p_l[kGenWords - 1] + __popc(w_l[kGenWords - 1]);
  unsigned long long n_taken = 0;
  for (int k = threadIdx.x; k < n; k += kGenThreads) {
    const int local = list[k], word = local >> 5;
    const uint32_t below = (1u << (local & 31)) - 1u;
    const long long ei = base.x + p_e[word] + __popc(w_e[word] & below);
    const long long di = base.y + p_d[word] + __popc(w_d[word] & below);
    if (!(count_emissions ? ei < limit : di < limit)) continue;
    const uint64_t index = cand0 + static_cast<uint64_t>(blockIdx.x) * kGenPerBlock + local;
    const Candidate c = EMITTED ? gen_candidate(p, regs, index) : gen_detected(p, regs, index);
    if (c.detected) {
      ++n_taken;
      if (di < capacity) {
        out[3 * di] = c.zu;
        out[3 * di + 1] = c.zd;
        out[3 * di + 2] = c.dl;
        if (im.exact) {
          im.exact[3 * di] = c.ex_zu;
          im.exact[3 * di + 1] = c.ex_zd;
          im.exact[3 * di + 2] = c.ex_dl;
        }
        if (im.events) {
          im.events[4 * di] = static_cast<float>(c.px);
          im.events[4 * di + 1] = static_cast<float>(c.py);
          im.events[4 * di + 2] = c.dir_x;
          im.events[4 * di + 3] = c.dir_y;
        }
      }
    }
    image_add(im.emitted, im, c.px, c.py);
    if (c.detected) {
      image_add(im.detected, im, c.px, c.py);
      if (im.naive || im.tan_map) naive_add(im, c.zu, c.zd, c.dl);
    }
  }
  n_taken = warp_add(n_taken);
  if (lane == 0 && n_taken) atomicAdd(taken, n_taken);
}

constexpr double kPi = 3.14159265358979323846;

}  // namespace
}  // namespace jpet

using namespace jpet;

// The phantom tool's float grids (phantom_cmd.cpp:241-253): PixelGrid with its
// lower-left corner at float(-s n / 2) + float(origin), and the tangent planes
// of VariableVoxelSizeVoxelGrid(-max_tan, bins, max_tan / bins * 2) with
// max_tan = 1.1 L / 2R.
namespace jpet {
namespace {
struct TanGrid {
  float x0, y0, s, tan_left, tan_size;
};
TanGrid tan_grid(const jpet_strip_geom& g, int bins, double origin_x, double origin_y) {
  TanGrid t;
  t.s = static_cast<float>(g.pixel_width);
  t.x0 = static_cast<float>(-g.pixel_width * g.n_z_pixels / 2) + static_cast<float>(origin_x);
  t.y0 = static_cast<float>(-g.pixel_width * g.n_y_pixels / 2) + static_cast<float>(origin_y);
  const float max_tan = 1.1f * static_cast<float>(g.scintillator_length) /
                        (2.0f * static_cast<float>(g.radius));
  t.tan_left = -max_tan;
  t.tan_size = bins > 0 ? max_tan / static_cast<float>(bins) * 2.0f : 0.0f;
  return t;
}

// One thread per voxel of the kernel map (phantom_cmd.cpp:402-430) in the
// reference's float order: tangent of the plane centre, sec, the voxel centre,
// AnalyticKernel at the kernel point, times the volume element 4 R bin_volume
// sec and the inverse sensitivity.
__global__ void __launch_bounds__(256) tan_kernel_map_kernel(DevGeom g, int32_t n_z, int32_t n_y,
                                                             int32_t bins, TanGrid tg, float kx,
                                                             float ky, float vol4r, float inv_sens,
                                                             float* __restrict__ out) {
  const size_t n = static_cast<size_t>(n_z) * n_y * bins;
  const float llcx = __fadd_rn(tg.x0, __fmul_rn(tg.s, 0.5f));
  const float llcy = __fadd_rn(tg.y0, __fmul_rn(tg.s, 0.5f));
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int x = static_cast<int>(i % n_z);
    const int y = static_cast<int>((i / n_z) % n_y);
    const int z = static_cast<int>(i / (static_cast<size_t>(n_z) * n_y));
    const float tan = __fadd_rn(__fmul_rn(__fadd_rn(static_cast<float>(z), 0.5f), tg.tan_size),
                                tg.tan_left);
    const float sec = __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(tan, tan)));
    const float cx = __fadd_rn(llcx, __fmul_rn(static_cast<float>(x), tg.s));
    const float cy = __fadd_rn(llcy, __fmul_rn(static_cast<float>(y), tg.s));
    const float k = analytic_exact(g, cy, tan, sec, __fsub_rn(kx, cx), __fsub_rn(ky, cy));
    out[i] = __fmul_rn(__fmul_rn(k, __fmul_rn(vol4r, sec)), inv_sens);
  }
}

__global__ void sensitivity_at_kernel(DevGeom g, float px, float py, float* out) {
  *out = scanner_sensitivity(g, px, py);
}
}  // namespace
}  // namespace jpet

extern "C" {

int jpet_strip_generate(const jpet_strip_geom* geom, const jpet_strip_region* regions,
                        int32_t n_regions, int64_t n, uint64_t seed, int32_t flags,
                        float* d_out_aos, int64_t capacity, int64_t* n_written,
                        const jpet_strip_gen_images* images, void* cuda_stream) {
  if (n_written) *n_written = 0;
  if (!geom || !regions || n_regions <= 0 || n_regions > kGenMaxRegions || n < 0 ||
      (n > 0 && !d_out_aos) || capacity < 0) {
    set_call_error("jpet_strip_generate: invalid argument");
    return JPET_ERR_ARGUMENT;
  }
  const bool detected = (flags & JPET_GEN_DETECTED) != 0;
  if (detected && capacity < n) {
    set_call_error("jpet_strip_generate: capacity below the requested detected events");
    return JPET_ERR_ARGUMENT;
  }
  if (!(geom->radius > 0) || !(geom->scintillator_length > 0) || !(geom->sigma_z >= 0) ||
      !(geom->sigma_dl >= 0)) {
    set_call_error("jpet_strip_generate: invalid scanner");
    return JPET_ERR_ARGUMENT;
  }
  // regions: weights, cumulative distribution (phantom.h:120-133), rotations
  std::vector<GenRegion> regs(n_regions);
  double total = 0.0;
  for (int i = 0; i < n_regions; ++i) {
    const jpet_strip_region& r = regions[i];
    GenRegion& g = regs[i];
    g.kind = r.kind;
    g.x = r.x;
    g.y = r.y;
    g.a = r.a;
    g.b = r.b;
    const double ang = r.angle_deg * kPi / 180.0;
    g.s = std::sin(ang);
    g.c = std::cos(ang);
    double w;
    if (r.kind == JPET_REGION_ELLIPSE) {
      if (!(r.a > 0) || !(r.b > 0)) {
        set_call_error("jpet_strip_generate: ellipse semi-axes must be positive");
        return JPET_ERR_ARGUMENT;
      }
      g.A = g.c * g.c / (r.a * r.a) + g.s * g.s / (r.b * r.b);
      g.B = g.s * g.s / (r.a * r.a) + g.c * g.c / (r.b * r.b);
      g.C = g.s * g.c * (1.0 / (r.a * r.a) - 1.0 / (r.b * r.b));
      w = r.intensity * kPi * r.a * r.b;
    } else if (r.kind == JPET_REGION_RECTANGLE) {
      if (!(r.a > 0) || !(r.b > 0)) {
        set_call_error("jpet_strip_generate: rectangle half sizes must be positive");
        return JPET_ERR_ARGUMENT;
      }
      g.A = g.B = g.C = 0.0;
      w = r.intensity * 4.0 * r.a * r.b;
    } else if (r.kind == JPET_REGION_POINT) {
      g.A = g.B = g.C = 0.0;
      w = r.intensity;
    } else {
      set_call_error("jpet_strip_generate: unknown region kind");
      return JPET_ERR_ARGUMENT;
    }
    if (!(w >= 0) || !std::isfinite(w)) {
      set_call_error("jpet_strip_generate: region weights must be finite and non-negative");
      return JPET_ERR_ARGUMENT;
    }
    total += w;
    g.cdf = total;
  }
  if (!(total > 0)) {
    set_call_error("jpet_strip_generate: total region weight is zero");
    return JPET_ERR_ARGUMENT;
  }
  for (auto& g : regs) g.cdf /= total;
  if (n == 0) return JPET_OK;

  GenImages im{};
  if (images && (images->tan_bins < 0 || (images->tan_bins > 0) != (images->tan_map != nullptr))) {
    set_call_error("jpet_strip_generate: tan_map needs tan_bins > 0 and the reverse");
    return JPET_ERR_ARGUMENT;
  }
  if (images && !(images->emitted || images->detected || images->naive || images->tan_map)) {
    im.exact = images->exact_responses;
    im.events = images->events;
  }
  if (images && (images->emitted || images->detected || images->naive || images->tan_map)) {
    if (geom->n_z_pixels <= 0 || geom->n_y_pixels <= 0 || !(geom->pixel_width > 0)) {
      set_call_error("jpet_strip_generate: count images need n_z, n_y and the pixel size");
      return JPET_ERR_ARGUMENT;
    }
    im.emitted = images->emitted;
    im.detected = images->detected;
    im.naive = images->naive;
    im.tan_map = images->tan_map;
    im.tan_bins = images->tan_bins;
    im.exact = images->exact_responses;
    im.events = images->events;
    im.s = geom->pixel_width;
    im.n_z = geom->n_z_pixels;
    im.n_y = geom->n_y_pixels;
    im.x0 = -im.s * im.n_z / 2.0 + images->origin_x;
    im.y0 = -im.s * im.n_y / 2.0 + images->origin_y;
    const TanGrid tg = tan_grid(*geom, im.tan_bins, images->origin_x, images->origin_y);
    im.fx0 = tg.x0;
    im.fy0 = tg.y0;
    im.fs = tg.s;
    im.two_r = 2.0f * static_cast<float>(geom->radius);
    im.tan_left = tg.tan_left;
    im.tan_size = tg.tan_size;
  }
  GenParams p;
  p.R = geom->radius;
  p.L = geom->scintillator_length;
  p.sigma_z = geom->sigma_z;
  p.sigma_dl = geom->sigma_dl;
  p.phi_max = detected ? std::atan(p.L / (2.0 * p.R)) : 0.5 * kPi;
  p.key0 = static_cast<uint32_t>(seed);
  p.key1 = static_cast<uint32_t>(seed >> 32);
  p.n_regions = n_regions;
  p.additive = (flags & JPET_GEN_ADDITIVE) ? 1 : 0;

  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  // one allocation: block bases, block counts, totals, counter, regions, bits
  const size_t o_counts = kGenMaxBlocks * sizeof(longlong2);
  const size_t o_totals = o_counts + kGenMaxBlocks * sizeof(int2);
  const size_t o_taken = o_totals + sizeof(longlong2);
  const size_t o_regs = o_taken + 16;
  const size_t o_words = (o_regs + regs.size() * sizeof(GenRegion) + 15) & ~static_cast<size_t>(15);
  unsigned char* d = nullptr;
  auto fail = [&](cudaError_t e, const char* what) {
    set_call_error(std::string("jpet_strip_generate: ") + what + ": " + cudaGetErrorString(e));
    cudaFree(d);
    return JPET_ERR_CUDA;
  };
  const long long limit = n;
  // a pass takes the candidates that the events still missing should need; the
  // first assumes that two in five count (a decision costs a fraction of an event)
  auto blocks_for = [](double candidates) {
    return static_cast<int>(std::min<double>(kGenMaxBlocks,
                                             std::max(1.0, std::ceil(candidates / kGenPerBlock))));
  };
  cudaError_t e = cudaMalloc(&d, o_words + static_cast<size_t>(kGenMaxBlocks) * 2 * kGenWords *
                                               sizeof(uint32_t));
  if (e != cudaSuccess) return fail(e, "cudaMalloc");
  auto* d_base = reinterpret_cast<longlong2*>(d);
  auto* d_counts = reinterpret_cast<int2*>(d + o_counts);
  auto* d_totals = reinterpret_cast<longlong2*>(d + o_totals);
  auto* d_taken = reinterpret_cast<unsigned long long*>(d + o_taken);
  auto* d_regs = reinterpret_cast<GenRegion*>(d + o_regs);
  auto* d_words = reinterpret_cast<uint32_t*>(d + o_words);
  e = cudaMemcpyAsync(d_regs, regs.data(), regs.size() * sizeof(GenRegion),
                      cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_totals, 0, o_regs - o_totals, s);
  if (e != cudaSuccess) return fail(e, "copy regions");
  long long have = 0;  // events (or emissions) so far
  uint64_t cand0 = 0, idle = 0;
  int blocks = blocks_for(2.5 * static_cast<double>(limit));
  while (have < limit) {
    gen_decide_kernel<<<blocks, kGenThreads, 0, s>>>(p, d_regs, cand0, d_words, d_counts);
    gen_scan_kernel<<<1, 1024, 0, s>>>(d_counts, blocks, d_base, d_totals);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(e, "decision kernel");
    if (im.emitted)
      gen_write_kernel<true><<<blocks, kGenThreads, 0, s>>>(
          p, d_regs, cand0, d_words, d_base, limit, detected ? 0 : 1, capacity, d_taken,
          d_out_aos, im);
    else
      gen_write_kernel<false><<<blocks, kGenThreads, 0, s>>>(
          p, d_regs, cand0, d_words, d_base, limit, detected ? 0 : 1, capacity, d_taken,
          d_out_aos, im);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(e, "write kernel");
    longlong2 totals;
    e = cudaMemcpyAsync(&totals, d_totals, sizeof(totals), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(e, "generation pass");
    const long long now = detected ? totals.y : totals.x;
    const uint64_t candidates = static_cast<uint64_t>(blocks) * kGenPerBlock;
    idle = now == have ? idle + candidates : 0;
    have = now;
    cand0 += candidates;
    if (have == 0 || idle > 0) {
      // 2^28 candidates in a row without one
      if (idle > 64ull * kGenMaxBlocks * kGenPerBlock) {
        set_call_error("jpet_strip_generate: the regions give no events");
        cudaFree(d);
        return JPET_ERR_ARGUMENT;
      }
      blocks = std::min(kGenMaxBlocks, 4 * blocks);
    } else {
      // the accepted share so far, with four standard deviations on top
      const double missing = static_cast<double>(limit - have);
      blocks = blocks_for((missing + 4.0 * std::sqrt(missing + 1.0)) *
                          static_cast<double>(cand0) / static_cast<double>(have));
    }
  }
  unsigned long long taken = 0;
  e = cudaMemcpyAsync(&taken, d_taken, sizeof(taken), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(e, "copy counter");
  cudaFree(d);
  if (static_cast<long long>(taken) > capacity) {
    set_call_error("jpet_strip_generate: capacity below the detected events");
    return JPET_ERR_ARGUMENT;
  }
  if (n_written) *n_written = static_cast<int64_t>(taken);
  return JPET_OK;
}

int jpet_strip_generate_host(const jpet_strip_geom* geom, const jpet_strip_region* regions,
                             int32_t n_regions, int64_t n, uint64_t seed, int32_t flags,
                             float* out_aos, int64_t capacity, int64_t* n_written,
                             const jpet_strip_gen_images* images, int32_t device) {
  if (n_written) *n_written = 0;
  if (n < 0 || capacity < 0 || (n > 0 && !out_aos)) {
    set_call_error("jpet_strip_generate_host: invalid argument");
    return JPET_ERR_ARGUMENT;
  }
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) {
    set_call_error(std::string("jpet_strip_generate_host: cudaSetDevice: ") +
                   cudaGetErrorString(e));
    return JPET_ERR_CUDA;
  }
  const int64_t cap = std::max<int64_t>(std::min(capacity, n), 1);
  float* d_out = nullptr;
  int32_t* d_img[4] = {nullptr, nullptr, nullptr, nullptr};
  int32_t* h_img[4] = {images ? images->emitted : nullptr, images ? images->detected : nullptr,
                       images ? images->naive : nullptr, images ? images->tan_map : nullptr};
  const size_t n_pix = static_cast<size_t>(std::max(geom ? geom->n_y_pixels : 0, 0)) *
                       static_cast<size_t>(std::max(geom ? geom->n_z_pixels : 0, 0));
  const size_t n_el[4] = {n_pix, n_pix, n_pix,
                          n_pix * static_cast<size_t>(images ? std::max(images->tan_bins, 0) : 0)};
  float* d_exact = nullptr;
  float* d_events = nullptr;
  auto release = [&]() {
    cudaFree(d_out);
    cudaFree(d_exact);
    cudaFree(d_events);
    for (auto* q : d_img) cudaFree(q);
  };
  e = cudaMalloc(&d_out, static_cast<size_t>(cap) * 3 * sizeof(float));
  if (e == cudaSuccess && images && images->exact_responses)
    e = cudaMalloc(&d_exact, static_cast<size_t>(cap) * 3 * sizeof(float));
  if (e == cudaSuccess && images && images->events)
    e = cudaMalloc(&d_events, static_cast<size_t>(cap) * 4 * sizeof(float));
  for (int k = 0; k < 4 && e == cudaSuccess; ++k) {
    if (!h_img[k]) continue;
    e = cudaMalloc(&d_img[k], std::max<size_t>(n_el[k], 1) * sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMemset(d_img[k], 0, n_el[k] * sizeof(int32_t));
  }
  if (e != cudaSuccess) {
    set_call_error(std::string("jpet_strip_generate_host: ") + cudaGetErrorString(e));
    release();
    return JPET_ERR_MEMORY;
  }
  jpet_strip_gen_images dim{};
  if (images) {
    dim = *images;
    dim.emitted = d_img[0];
    dim.detected = d_img[1];
    dim.naive = d_img[2];
    dim.tan_map = d_img[3];
    dim.exact_responses = d_exact;
    dim.events = d_events;
  }
  int64_t written = 0;
  int rc = jpet_strip_generate(geom, regions, n_regions, n, seed, flags, d_out, cap, &written,
                               images ? &dim : nullptr, nullptr);
  if (rc == JPET_OK) {
    e = cudaMemcpy(out_aos, d_out, static_cast<size_t>(written) * 3 * sizeof(float),
                   cudaMemcpyDeviceToHost);
    for (int k = 0; k < 4 && e == cudaSuccess; ++k)
      if (h_img[k]) e = cudaMemcpy(h_img[k], d_img[k], n_el[k] * sizeof(int32_t),
                                   cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && d_exact)
      e = cudaMemcpy(images->exact_responses, d_exact,
                     static_cast<size_t>(written) * 3 * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && d_events)
      e = cudaMemcpy(images->events, d_events, static_cast<size_t>(written) * 4 * sizeof(float),
                     cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      set_call_error(std::string("jpet_strip_generate_host: copy: ") + cudaGetErrorString(e));
      rc = JPET_ERR_CUDA;
    }
  }
  release();
  if (rc == JPET_OK && n_written) *n_written = written;
  return rc;
}

int jpet_strip_tan_kernel_map(const jpet_strip_geom* geom, int32_t tan_bins, double kernel_x,
                              double kernel_y, double origin_x, double origin_y,
                              int32_t divide_by_sensitivity, float* out, int32_t device) {
  if (!geom || !out || tan_bins <= 0 || geom->n_z_pixels <= 0 || geom->n_y_pixels <= 0 ||
      !(geom->pixel_width > 0) || !(geom->radius > 0) || !(geom->scintillator_length > 0) ||
      !(geom->sigma_z > 0) || !(geom->sigma_dl > 0)) {
    set_call_error("jpet_strip_tan_kernel_map: invalid argument");
    return JPET_ERR_ARGUMENT;
  }
  const size_t n = static_cast<size_t>(geom->n_z_pixels) * geom->n_y_pixels * tan_bins;
  cudaError_t e = cudaSetDevice(device);
  float* d_out = nullptr;
  float* d_sens = nullptr;
  if (e == cudaSuccess) e = cudaMalloc(&d_out, n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&d_sens, sizeof(float));
  const DevGeom g = make_dev_geom(*geom);
  const TanGrid tg = tan_grid(*geom, tan_bins, origin_x, origin_y);
  const float kx = static_cast<float>(kernel_x), ky = static_cast<float>(kernel_y);
  float inv_sens = 1.0f;
  if (e == cudaSuccess && divide_by_sensitivity) {
    sensitivity_at_kernel<<<1, 1>>>(g, kx, ky, d_sens);
    float sens = 0.0f;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(&sens, d_sens, sizeof(float), cudaMemcpyDeviceToHost);
    inv_sens = 1.0f / sens;
  }
  // 4 R pixel^2 dtan (phantom_cmd.cpp:409-421), float left to right
  const float vol4r = 4.0f * static_cast<float>(geom->radius) * (tg.s * tg.s * tg.tan_size);
  if (e == cudaSuccess) {
    const size_t blocks = std::min<size_t>((n + 255) / 256, 152 * 16);
    tan_kernel_map_kernel<<<static_cast<unsigned>(blocks), 256>>>(
        g, geom->n_z_pixels, geom->n_y_pixels, tan_bins, tg, kx, ky, vol4r, inv_sens, d_out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d_out, n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(d_out);
  cudaFree(d_sens);
  if (e != cudaSuccess) {
    set_call_error(std::string("jpet_strip_tan_kernel_map: ") + cudaGetErrorString(e));
    return JPET_ERR_CUDA;
  }
  return JPET_OK;
}

}  // extern "C"
