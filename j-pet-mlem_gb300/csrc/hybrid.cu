// GB300 3D hybrid list-mode MLEM (include/jpet_hybrid.h): barrel LORs in x-y,
// the strip TOF kernel along each LOR and z.
//
// Replaces PET3D::Hybrid::GPU::Reconstruction::run and its kernel
// (src/3d/hybrid/cuda/reconstruction.cu:36-187,
// src/3d/hybrid/cuda/reconstruction/warp_granularity.cuh:28-178) and moves the
// CPU set-up the reference command runs first onto the device
// (src/3d/hybrid/reconstruction.h:101-162 frame events, 218-274 weights and
// sensitivity).
//
// Device layout.  The image is held pixel-major with the planes of a pixel
// contiguous, index (x + n_columns y) pitch + z, the pitch n_planes rounded up to
// a multiple of 4, so that the voxels of one event -- a run of planes for each
// pixel info on its LOR -- are contiguous runs in memory and four planes one
// aligned 16-byte access; the reference's plane-major order (voxel_grid.h:54-56)
// is used only at the boundary (set_image / get_image).
//
// Iteration kernels: iterate_table_kernel where the handle holds the geometry's
// voxel weights (prepare_table), iterate_kernel otherwise and for events that do
// not fit it.  In both one CTA takes an event.  In iterate_kernel the threads compute the event's
// per-pixel constants of the strip kernel (the terms that do not depend on z)
// into shared memory, then walk the pixel-info x plane voxels flattened, one
// CTA-wide step of consecutive voxels at a time, so that neighbouring threads
// touch neighbouring planes of one pixel.  Each thread keeps the weights
// K(z, up) w_pixel rho of its first voxels in shared memory for the
// back-projection, which adds weight / denominator with one global float
// atomic per voxel; the denominator is reduced across the CTA.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "../../include/jpet_hybrid.h"

namespace {

thread_local std::string g_hybrid_error = "no error";

template <typename T>
struct Buf {
  T* p = nullptr;
  size_t n = 0;
  cudaError_t alloc(size_t count) {
    if (count <= n && p) return cudaSuccess;
    release();
    if (count == 0) return cudaSuccess;
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p), count * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      n = 0;
      return e;
    }
    n = count;
    return cudaSuccess;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

// Constants of the kernels: GaussianKernel's (gaussian_kernel.h:27-33) and the grid's.
struct HybConst {
  float ipz, ipd, c0;   // 1/sigma_z^2, 1/sigma_dl^2, normalisation
  float ps, z_left;     // voxel size, VoxelGrid::z_left
  float llcx, llcy;     // PixelGrid::lower_left_center
  float L2;             // length / 2 (GaussianKernel::sensitivity)
  float exp_bpq;        // -log2(e) / sigma_z^2: exponent coefficient of (dz - dy tan)^2
  int32_t n_columns, n_rows, n_planes;
  int32_t pitch;        // planes of a pixel in the device image
  int32_t n_lors;
  int64_t n_infos;
  int32_t n_planes_half;  // planes of weights (> 1: one system matrix per plane half)
  int32_t sens_depth;     // planes of the sensitivity image (1: the 2D sensitivity)
};

// Forms of the denominator loop (reconstruction.h:327-357):
constexpr int kSens2D = 0;      // one plane half, 2D sensitivity
constexpr int kMultiPlane = 1;  // weights and sensitivity of plane |iz - n_planes_half|
constexpr int kSens3D = 2;      // one plane half, sensitivity of plane |iz - depth|

// The plane of the weights / sensitivity that plane iz reads: |iz - depth|.
// The reference's index reaches depth itself for plane 0 (and for the last
// plane of an odd count), one plane past its arrays; clamped to depth - 1.
__device__ __forceinline__ int abs_plane(int iz, int depth) {
  const int a = iz > depth ? iz - depth : depth - iz;
  return a < depth ? a : depth - 1;
}

// Sizes of the iteration kernel (compile-time; -D overrides for tuning sweeps).
#ifndef JPET_HYBRID_THREADS
#define JPET_HYBRID_THREADS 128
#endif
#ifndef JPET_HYBRID_CACHE_STEPS
#define JPET_HYBRID_CACHE_STEPS 32
#endif
constexpr int kThreads = JPET_HYBRID_THREADS;     // CTA size: one event per CTA at a time
constexpr int kSteps = JPET_HYBRID_CACHE_STEPS;   // voxel weights a thread keeps for the back-projection
constexpr int kPix = 256;                         // pixel infos per chunk
constexpr int kWarpsPerCta = kThreads / 32;
// Table iteration.  1e6 events on the 384-detector ring / 5e5 on the 96-detector
// one, ms for 5 iterations: 64 x 16 32.1 / 6.4, 96 x 10 30.0 / 5.7, 128 x 8
// 30.9 / 6.2, 256 x 6 36.6 / 10.0; table entries and weights in registers instead
// of shared memory 31.0 / 7.6 (128 x 8).
constexpr int kTabThreads = 96;  // CTA size
constexpr int kTabSteps = 10;    // quads of planes a thread keeps
constexpr float kPi = 3.14159265358979323846f;

__device__ __forceinline__ int64_t lor_index(int16_t first, int16_t second) {
  return static_cast<int64_t>(static_cast<int32_t>(first) * (first + 1) / 2 + second);
}

// float -> short as the reference's x86-64 build converts (truncation to int32,
// out of range and NaN give INT32_MIN, low 16 bits kept).
__device__ __forceinline__ int16_t to_short(float v) {
  int32_t i = (v > -2147483648.0f && v < 2147483648.0f) ? __float2int_rz(v) : INT32_MIN;
  return static_cast<int16_t>(static_cast<uint32_t>(i) & 0xffffu);
}

// Pixel centre (pixel_grid.h:54-57), explicit rounding (no contraction).
__device__ __forceinline__ void pixel_center(const HybConst& c, int x, int y, float& cx,
                                             float& cy) {
  cx = __fadd_rn(c.llcx, __fmul_rn(static_cast<float>(x), c.ps));
  cy = __fadd_rn(c.llcy, __fmul_rn(static_cast<float>(y), c.ps));
}

// ---- set-up: weights, sensitivity, normalisation --------------------------------

// Reconstruction::calculate_weight (reconstruction.h:218-238): one warp per LOR.
__global__ void weights_kernel(const float4* __restrict__ seg, const float* __restrict__ widths,
                               const int2* __restrict__ pix, const uint64_t* __restrict__ ib,
                               const uint64_t* __restrict__ ie, float* __restrict__ w,
                               HybConst c, double sqrt_2pi) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int16_t* p16 = reinterpret_cast<const int16_t*>(pix);
  for (int64_t l = warp; l < c.n_lors; l += n_warps) {
    const float4 s2 = seg[3 * l + 2];  // normal_x, normal_y, length, distance_from_origin
    const float sigma_w = __fmul_rn(0.3f, widths[l]);
    const double gauss_norm_w = 1.0 / (static_cast<double>(sigma_w) * sqrt_2pi);
    const float inv_sigma2_w = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sigma_w), sigma_w));
    for (uint64_t i = ib[l] + lane; i < ie[l]; i += 32) {
      float cx, cy;
      pixel_center(c, p16[2 * i], p16[2 * i + 1], cx, cy);
      const float d = __fsub_rn(__fadd_rn(__fmul_rn(cx, s2.x), __fmul_rn(cy, s2.y)), s2.w);
      const float e = expf(__fmul_rn(__fmul_rn(-d, d), inv_sigma2_w));
      w[i] = __double2float_rn(gauss_norm_w * static_cast<double>(e));
    }
  }
}

// Sort keys of calculate_sensitivity: pixel index of every pixel info, and a
// check that every pixel lies inside the grid.
__global__ void pixel_keys_kernel(const int16_t* __restrict__ p16, int64_t n, HybConst c,
                                  int32_t* __restrict__ keys, int32_t* __restrict__ vals,
                                  int* __restrict__ bad) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int x = p16[2 * i], y = p16[2 * i + 1];
    const bool in = x >= 0 && x < c.n_columns && y >= 0 && y < c.n_rows;
    if (!in) atomicExch(bad, 1);
    keys[i] = in ? x + c.n_columns * y : 0;
    vals[i] = static_cast<int32_t>(i);
  }
}

// calculate_sensitivity (reconstruction.h:240-251): the infos of each pixel,
// in ascending info order after the stable sort, summed from zero in that
// order -- the reference's order of additions into sensitivity[pixel].
__global__ void sensitivity_sum_kernel(const int32_t* __restrict__ keys,
                                       const int32_t* __restrict__ vals, int64_t n,
                                       const float* __restrict__ w, float* __restrict__ sens) {
  for (int64_t j = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; j < n;
       j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t k = keys[j];
    if (j > 0 && keys[j - 1] == k) continue;
    float s = 0.0f;
    for (int64_t q = j; q < n && keys[q] == k; ++q) s = __fadd_rn(s, w[vals[q]]);
    sens[k] = s;
  }
}

// LOR of every pixel info (-1 for infos outside every LOR's range).
__global__ void lor_of_info_kernel(const uint64_t* __restrict__ ib, const uint64_t* __restrict__ ie,
                                   int32_t n_lors, int32_t* __restrict__ lor_of) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t l = warp; l < n_lors; l += n_warps)
    for (uint64_t i = ib[l] + lane; i < ie[l]; i += 32) lor_of[i] = static_cast<int32_t>(l);
}

// After the stable sort by pixel, two infos of one pixel and one LOR are
// adjacent: flags a LOR that lists a pixel twice.
__global__ void unique_pixels_kernel(const int32_t* __restrict__ keys,
                                     const int32_t* __restrict__ vals, int64_t n,
                                     const int32_t* __restrict__ lor_of, int* __restrict__ bad) {
  for (int64_t j = 1 + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; j < n;
       j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (keys[j] != keys[j - 1]) continue;
    const int32_t a = lor_of[vals[j]], b = lor_of[vals[j - 1]];
    if (a >= 0 && a == b) atomicExch(bad, 1);
  }
}

// normalize_geometry_weights (reconstruction.h:253-272), every plane half:
// weight (info, plane) / sensitivity (pixel, plane).
__global__ void normalize_kernel(const int16_t* __restrict__ p16, int64_t n, HybConst c,
                                 const float* __restrict__ sens, float* __restrict__ w) {
  const int64_t n_px = static_cast<int64_t>(c.n_columns) * c.n_rows;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int x = p16[2 * i], y = p16[2 * i + 1];
    for (int plane = 0; plane < c.n_planes_half; ++plane)
      w[i + n * plane] = __fdiv_rn(w[i + n * plane], sens[x + c.n_columns * y + n_px * plane]);
  }
}

__global__ void fill_kernel(float* p, int64_t n, float v) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    p[i] = v;
}

// ---- frame events -------------------------------------------------------------

__device__ __forceinline__ uint64_t lower_bound_f(const float* a, uint64_t lo, uint64_t hi,
                                                  float v) {
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo) / 2;
    if (a[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ uint64_t upper_bound_f(const float* a, uint64_t lo, uint64_t hi,
                                                  float v) {
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo) / 2;
    if (v < a[mid]) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// Reconstruction::translate_to_frame (reconstruction.h:101-147) with
// Response::calculate_tan_y_z (src/2d/strip/response.h:22-37) and
// GaussianKernel::ellipse_bb (gaussian_kernel.h:108-128), then
// bb_intersects_grid_with_positive_weight (reconstruction.h:151-162).  Every
// operation is rounded explicitly in the reference's order, so the frame event
// and its ranges are the reference's own.
__global__ void translate_kernel(const jpet_hybrid_response* __restrict__ r, int64_t n,
                                 const float4* __restrict__ seg, const int16_t* __restrict__ p16,
                                 const float* __restrict__ pos, const float* __restrict__ w,
                                 const uint64_t* __restrict__ ib, const uint64_t* __restrict__ ie,
                                 HybConst c, jpet_hybrid_frame_event* __restrict__ out,
                                 uint8_t* __restrict__ keep) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const jpet_hybrid_response q = r[i];
    jpet_hybrid_frame_event e{};
    e.lor_first = q.lor_first;
    e.lor_second = q.lor_second;
    const int64_t l = lor_index(q.lor_first, q.lor_second);
    if (q.lor_first < 0 || q.lor_second < 0 || l < 0 || l >= c.n_lors) {
      out[i] = e;
      keep[i] = 0;
      continue;
    }
    const float R = __fdiv_rn(seg[3 * l + 2].z, 2.0f);
    const float two_R = __fmul_rn(2.0f, R);
    const float t = __fdiv_rn(__fsub_rn(q.z_up, q.z_dn), two_R);
    const float y = __fmul_rn(-0.5f, __fdiv_rn(q.dl, __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(t, t)))));
    const float z = __fmul_rn(0.5f, __fadd_rn(__fadd_rn(q.z_up, q.z_dn),
                                              __fmul_rn(__fmul_rn(2.0f, y), t)));
    const float tan_sq = __fmul_rn(t, t);
    const float sec = __fsqrt_rn(__fadd_rn(1.0f, __fmul_rn(t, t)));
    const float A = __fadd_rn(__fmul_rn(__fmul_rn(__fmul_rn(4.0f, sec), sec), c.ipd),
                              __fmul_rn(__fmul_rn(2.0f, tan_sq), c.ipz));
    const float B = __fmul_rn(__fmul_rn(-4.0f, t), c.ipz);
    const float C = __fmul_rn(2.0f, c.ipz);
    const float hb = __fdiv_rn(B, 2.0f);
    const float B_2 = __fmul_rn(hb, hb);
    const float half_up = __fdiv_rn(3.0f, __fsqrt_rn(__fsub_rn(A, __fdiv_rn(B_2, C))));
    const float half_right = __fdiv_rn(3.0f, __fsqrt_rn(__fsub_rn(C, __fdiv_rn(B_2, A))));
    e.tan = t;
    e.up = y;
    e.right = z;
    e.sec = sec;
    const float z_lo = __fsub_rn(z, half_right), z_hi = __fadd_rn(z, half_right);
    const int16_t p_lo = to_short(__fdiv_rn(__fsub_rn(z_lo, c.z_left), c.ps));
    const int16_t p_hi = to_short(__fdiv_rn(__fsub_rn(z_hi, c.z_left), c.ps));
    const int16_t zero = 0;
    e.plane_begin = (zero < p_lo) ? p_lo : zero;  // std::max((S)0, plane(z_left))
    const int16_t pe = static_cast<int16_t>(p_hi + 1);
    const int16_t np = static_cast<int16_t>(c.n_planes);
    e.plane_end = (np < pe) ? np : pe;  // std::min
    const float y_up = __fadd_rn(y, half_up), y_dn = __fsub_rn(y, half_up);
    const float t_up = __fdiv_rn(__fadd_rn(y_up, R), two_R);
    const float t_dn = __fdiv_rn(__fadd_rn(y_dn, R), two_R);
    uint64_t end = upper_bound_f(pos, ib[l], ie[l], t_up) + 1;
    if (end > static_cast<uint64_t>(c.n_infos)) end = static_cast<uint64_t>(c.n_infos);
    e.pixel_info_end = end;
    e.pixel_info_begin = lower_bound_f(pos, ib[l], ie[l], t_dn);
    bool k = !(e.plane_end <= 0 || e.plane_begin >= c.n_planes);
    if (k) {
      k = false;
      for (uint64_t j = e.pixel_info_begin; j < e.pixel_info_end; ++j) {
        const int x = p16[2 * j], yy = p16[2 * j + 1];
        if (x >= 0 && x < c.n_columns && yy >= 0 && yy < c.n_rows && w[j] > 0.0f) {
          k = true;
          break;
        }
      }
    }
    out[i] = e;
    keep[i] = k ? 1 : 0;
  }
}

// Checks caller-given frame events and sums the reference's statistics
// (used_pixels, used_voxels: reconstruction.h:311-324) over them.
__global__ void event_stats_kernel(const jpet_hybrid_frame_event* __restrict__ ev, int64_t n,
                                   const uint64_t* __restrict__ ib,
                                   const uint64_t* __restrict__ ie, HybConst c,
                                   unsigned long long* __restrict__ stats, int* __restrict__ bad) {
  unsigned long long px = 0, vx = 0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const jpet_hybrid_frame_event e = ev[i];
    const int64_t l = lor_index(e.lor_first, e.lor_second);
    // the range lies within the LOR's pixel infos and the one past its end, as
    // translate_to_frame makes it; planes within the grid
    bool ok = e.lor_first >= 0 && e.lor_second >= 0 && l >= 0 && l < c.n_lors &&
              e.pixel_info_begin <= e.pixel_info_end &&
              e.pixel_info_end <= static_cast<uint64_t>(c.n_infos) &&
              (e.plane_begin >= e.plane_end || (e.plane_begin >= 0 && e.plane_end <= c.n_planes));
    if (ok && e.pixel_info_begin < e.pixel_info_end)
      ok = e.pixel_info_begin >= ib[l] && e.pixel_info_end <= ie[l] + 1;
    if (!ok) {
      atomicExch(bad, 1);
      continue;
    }
    const unsigned long long np = e.pixel_info_end - e.pixel_info_begin;
    const int planes = e.plane_end - e.plane_begin;
    px += np;
    vx += np * static_cast<unsigned long long>(planes > 0 ? planes : 0);
  }
  for (int o = 16; o > 0; o >>= 1) {
    px += __shfl_xor_sync(0xffffffffu, px, o);
    vx += __shfl_xor_sync(0xffffffffu, vx, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&stats[0], px);
    atomicAdd(&stats[1], vx);
  }
}

// ---- image layout -----------------------------------------------------------

// reference order (x + nc (y + nr z)) -> device order ((x + nc y) pitch + z); the
// planes past n_planes are zero
__global__ void to_device_layout(const float* __restrict__ in, float* __restrict__ out,
                                 int64_t n_px, int32_t np, int32_t pitch) {
  const int64_t n = n_px * pitch;
  for (int64_t j = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; j < n;
       j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t p = j / pitch, z = j - p * pitch;
    out[j] = z < np ? in[p + z * n_px] : 0.0f;
  }
}
__global__ void to_reference_layout(const float* __restrict__ in, float* __restrict__ out,
                                    int64_t n_px, int32_t np, int32_t pitch) {
  const int64_t n = n_px * np;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t z = i / n_px, p = i - z * n_px;
    out[i] = in[p * pitch + z];
  }
}

// ---- iteration ----------------------------------------------------------------

struct EvC {
  float up, right, tan, sec, R;
  float z0;  // centre of the event's first plane (voxel_grid.h:40-42)
  int32_t plane_begin;
};

// 16-byte asynchronous copy to a shared-memory address, and the wait for all of a
// thread's copies.
__device__ __forceinline__ void cp_async16(unsigned dst, const float4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// ex2.approx of the hardware; exp(x) = 2^(x log2 e).
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// rcp.approx of the hardware (relative error below 2^-23).
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// LineSegment::projection_relative_middle (line_segment.h:82-84) of a pixel
// info's centre; s1: mid_x, mid_y, direction_x, direction_y.
__device__ __forceinline__ float lor_up(const HybConst& c, float4 s1,
                                        const int16_t* __restrict__ p16, uint64_t i) {
  float cx, cy;
  pixel_center(c, p16[2 * i], p16[2 * i + 1], cx, cy);
  return __fadd_rn(__fmul_rn(__fsub_rn(cx, s1.x), s1.z), __fmul_rn(__fsub_rn(cy, s1.y), s1.w));
}

// Per-pixel terms of GaussianKernel::operator() and ::sensitivity that do not
// depend on z (gaussian_kernel.h:51-79,140-150) for pixel info i of the event.
// Forms other than kSens2D keep in pa.w the info index (kMultiPlane: its weight
// is the plane's) or the pixel weight times pi (kSens3D), and in pb.z the
// pixel index (the sensitivity is the plane's).
template <int SM>
__device__ __forceinline__ void pixel_terms(const HybConst& c, const EvC& e, float4 s1,
                                            const int16_t* __restrict__ p16,
                                            const float* __restrict__ w,
                                            const float* __restrict__ sens, uint64_t i,
                                            float4& pa, float4& pb) {
  const int x = p16[2 * i], y = p16[2 * i + 1];
  const float up = lor_up(c, s1, p16, i);
  const float dy = __fsub_rn(up, e.up);
  const float yp = __fadd_rn(dy, e.up);
  const float sec_sq = __fmul_rn(e.sec, e.sec);
  const float ap = __fmul_rn(-__fsub_rn(yp, e.R), sec_sq);
  const float aq = __fmul_rn(-__fadd_rn(yp, e.R), sec_sq);
  const float ar = __fmul_rn(__fmul_rn(__fmul_rn(-2.0f, yp), e.sec), e.tan);
  const float a_ic_a = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(ap, c.ipz), ap),
                                           __fmul_rn(__fmul_rn(aq, c.ipz), aq)),
                                 __fmul_rn(__fmul_rn(ar, c.ipd), ar));
  const float ebe = __fdiv_rn(c.c0, __fsqrt_rn(a_ic_a));
  const float br = __fmul_rn(__fmul_rn(-2.0f, dy), e.sec);
  const float brr = __fmul_rn(__fmul_rn(br, c.ipd), br);
  const int pix = x + c.n_columns * y;
  // the exponent's z-independent part -log2(e) (r ipd r) / 2 and the pixel
  // weight times pi (the frame sensitivity's 1/pi) are folded in here
  const float wv = SM == kMultiPlane ? __int_as_float(static_cast<int>(i)) : w[i] * kPi;
  const float sv = SM == kSens2D ? sens[pix] : __int_as_float(pix);
  pa = make_float4(dy, ebe, brr * (-0.5f * 1.4426950408889634f), wv);
  pb = make_float4(__frcp_rn(__fsub_rn(e.R, up)), __frcp_rn(__fadd_rn(e.R, up)), sv,
                   __int_as_float(pix * c.pitch));
}

// pixel_terms for an info of the voxel table: pa.w is the pixel's base index, the
// sensitivity (or pixel index) goes to sv.
template <int SM>
__device__ __forceinline__ float4 table_terms(const HybConst& c, const EvC& e, float2 iu,
                                              const float* __restrict__ sens, float& sv) {
  const float up = iu.x;
  const int pix = __float_as_int(iu.y);
  const float dy = __fsub_rn(up, e.up);
  const float yp = __fadd_rn(dy, e.up);
  const float sec_sq = __fmul_rn(e.sec, e.sec);
  const float ap = __fmul_rn(-__fsub_rn(yp, e.R), sec_sq);
  const float aq = __fmul_rn(-__fadd_rn(yp, e.R), sec_sq);
  const float ar = __fmul_rn(__fmul_rn(__fmul_rn(-2.0f, yp), e.sec), e.tan);
  const float a_ic_a = fmaf(__fmul_rn(ar, c.ipd), ar,
                            fmaf(__fmul_rn(aq, c.ipz), aq, __fmul_rn(__fmul_rn(ap, c.ipz), ap)));
  const float br = __fmul_rn(__fmul_rn(-2.0f, dy), e.sec);
  sv = SM == kSens2D ? sens[pix] : __int_as_float(pix);
  return make_float4(dy, c.c0 * __frsqrt_rn(a_ic_a),
                     __fmul_rn(__fmul_rn(br, c.ipd), br) * (-0.5f * 1.4426950408889634f),
                     __int_as_float(pix * c.pitch));
}

// The pixel weight (times pi) and the sensitivity a voxel of plane col uses.
template <int SM>
__device__ __forceinline__ float voxel_pixel_weight(const HybConst& c, const float4 pa, int col,
                                                    const float* __restrict__ w) {
  if (SM != kMultiPlane) return pa.w;
  const int ap = abs_plane(col, c.n_planes_half);
  return __ldg(&w[static_cast<int64_t>(ap) * c.n_infos + __float_as_int(pa.w)]) * kPi;
}
template <int SM>
__device__ __forceinline__ float voxel_sens(const HybConst& c, float sv, int col,
                                            const float* __restrict__ sens) {
  if (SM == kSens2D) return sv;
  const int ap = abs_plane(col, SM == kMultiPlane ? c.n_planes_half : c.sens_depth);
  return __ldg(&sens[static_cast<int64_t>(ap) * c.n_columns * c.n_rows + __float_as_int(sv)]);
}


// Arctangent of y / x in (-pi, pi]: reduction to r = min(|x|, |y|) / max(|x|, |y|)
// in [0, 1], atan(r) = r P(r^2) with P of degree 8 fitted by csrc/fit_atan.py
// (maximum absolute error 1e-7 on [0, 1] in float arithmetic), then the
// octant and sign reflections.  Branch-free.
__device__ __forceinline__ float atan2_poly(float y, float x) {
  const float ax = fabsf(x), ay = fabsf(y);
  const float r = fminf(ax, ay) * rcp(fmaxf(ax, ay));
  const float s = r * r;
  float p = 2.456588438e-03f;
  p = fmaf(p, s, -1.440078672e-02f);
  p = fmaf(p, s, 3.978023678e-02f);
  p = fmaf(p, s, -7.234767079e-02f);
  p = fmaf(p, s, 1.049889922e-01f);
  p = fmaf(p, s, -1.416121572e-01f);
  p = fmaf(p, s, 1.998590529e-01f);
  p = fmaf(p, s, -3.333259821e-01f);
  p = fmaf(p, s, 9.999998808e-01f);
  p *= r;
  p = (ay > ax) ? 1.57079632679489662f - p : p;
  p = (x < 0.0f) ? kPi - p : p;
  return copysignf(p, y);
}

// The frame sensitivity's angle (gaussian_kernel.h:140-150) of a pixel with
// rm = 1 / (R - up), rp = 1 / (R + up) at lp = L/2 + z, lm = L/2 - z:
// atan(a) - atan(b) as atan2(a - b, 1 + a b), the same angle for every a, b.
__device__ __forceinline__ float frame_angle(float rm, float rp, float lp, float lm) {
  const float a = fminf(lm * rm, lp * rp);
  const float b = fmaxf(-lp * rm, -lm * rp);
  return atan2_poly(a - b, fmaf(a, b, 1.0f));
}

// weight = GaussianKernel::normalized(...) * pixel weight * rho of voxel
// (pixel, plane col), reconstruction.h:327-363, with the plane's terms
// dz = z - right, lp = L/2 + z, lm = L/2 - z.  exp(-b_ic_b / 2) is
// 2^(exp_bpq (dz - dy tan)^2 + pa.z); a non-positive kernel value gives weight 0
// as in the reference (reconstruction.h:335-341).
template <int SM>
__device__ __forceinline__ float plane_weight(const HybConst& c, const EvC& e, const float4 pa,
                                              const float4 pb, float dz, float lp, float lm,
                                              int col, const float* __restrict__ rho,
                                              const float* __restrict__ w) {
  const float bpq = fmaf(-pa.x, e.tan, dz);
  const float K = pa.y * ex2(fmaf(bpq * bpq, c.exp_bpq, pa.z));
  const float ang = frame_angle(pb.x, pb.y, lp, lm);
  const float v = (K * voxel_pixel_weight<SM>(c, pa, col, w)) * rcp(ang) *
                  __ldg(&rho[__float_as_int(pb.w) + col]);
  return ang < 0.0f ? 0.0f : v;
}

// The same for the event's k-th plane, z = z0 + k pixel_size.
template <int SM>
__device__ __forceinline__ float voxel_weight(const HybConst& c, const EvC& e, const float4 pa,
                                              const float4 pb, int k,
                                              const float* __restrict__ rho,
                                              const float* __restrict__ w) {
  const float z = fmaf(static_cast<float>(k), c.ps, e.z0);
  return plane_weight<SM>(c, e, pa, pb, z - e.right, c.L2 + z, c.L2 - z, e.plane_begin + k,
                          rho, w);
}

// Advances a thread's (pixel, plane) position by one CTA-wide step of the
// flattened walk: kThreads voxels = q pixels and r planes.
__device__ __forceinline__ void walk(int& i, int& k, int q, int r, int npl) {
  k += r;
  i += q;
  if (k >= npl) {
    k -= npl;
    ++i;
  }
}

// Multiplicity of info i's voxels in the back-projection.  The reference keeps
// the kernel values in a voxel-indexed image (reconstruction.h:339,361,368)
// and back-projects every occurrence of a voxel with the value written last.
// Pixels of one LOR are distinct, so the only repeated pixel is the info one
// past the LOR's end that the range takes in (reconstruction.h:134-140): when
// it repeats the pixel of info dup, info dup contributes nothing and the last
// info twice.
__device__ __forceinline__ float multiplicity(int64_t i, int dup, int64_t last) {
  return dup < 0 ? 1.0f : (i == dup ? 0.0f : (i == last ? 2.0f : 1.0f));
}

// One CTA per event.  The pixel terms of up to kPix infos go to shared
// memory.  Thread tid takes plane tid % npl of the pixels tid / npl,
// tid / npl + G, ... (G = kThreads / npl groups), so neighbouring threads touch
// neighbouring planes of one pixel and every z-dependent term is computed once
// per event; each thread keeps its first kSteps weights in shared memory for
// the back-projection.  Events with more than kPix infos or kThreads planes are
// walked flattened, chunk by chunk, and recomputed in the back-projection.
// list: the events to take (NULL: all).
template <int SM>
__global__ void __launch_bounds__(kThreads)
    iterate_kernel(const jpet_hybrid_frame_event* __restrict__ ev,
                   const int32_t* __restrict__ list, int64_t n,
                   const float4* __restrict__ seg, const int16_t* __restrict__ p16,
                   const float* __restrict__ w, const float* __restrict__ sens,
                   const float* __restrict__ rho, float* __restrict__ out, HybConst c,
                   unsigned long long* __restrict__ n_positive) {
  __shared__ float4 pa[kPix];  // dy, element_before_exp, exponent term, pixel weight * pi
  __shared__ float4 pb[kPix];  // 1/(R - up), 1/(R + up), sensitivity, base index (int bits)
  __shared__ float cache[kSteps * kThreads];  // weights of each thread's first kSteps voxels
  __shared__ float red_den[kWarpsPerCta];
  __shared__ int red_dup[kWarpsPerCta];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t* p32 = reinterpret_cast<const uint32_t*>(p16);
  unsigned long long positive = 0;
  for (int64_t ei = blockIdx.x; ei < n; ei += gridDim.x) {
    const jpet_hybrid_frame_event fe = ev[list ? list[ei] : ei];
    const int npl = fe.plane_end - fe.plane_begin;
    const int64_t nin = static_cast<int64_t>(fe.pixel_info_end - fe.pixel_info_begin);
    if (npl <= 0 || nin <= 0) continue;
    const int64_t l = lor_index(fe.lor_first, fe.lor_second);
    const float4 s1 = seg[3 * l + 1];  // mid_x, mid_y, direction_x, direction_y
    EvC e;
    e.up = fe.up;
    e.right = fe.right;
    e.tan = fe.tan;
    e.sec = fe.sec;
    e.R = __fdiv_rn(seg[3 * l + 2].z, 2.0f);
    e.plane_begin = fe.plane_begin;
    e.z0 = __fadd_rn(__fmul_rn(__fadd_rn(static_cast<float>(fe.plane_begin), 0.5f), c.ps),
                     c.z_left);
    const uint32_t last_pixel = p32[fe.pixel_info_end - 1];
    // main path: at most kPix infos and kThreads planes; thread tid holds
    // plane k of pixel group g (G groups of npl threads)
    const bool one_chunk = nin <= kPix && npl <= kThreads;
    const int G = one_chunk ? kThreads / npl : 1;
    const int g0 = tid / npl, kk = tid - g0 * npl;
    const bool active = g0 < G;
    const int col = e.plane_begin + kk;
    const float z = fmaf(static_cast<float>(kk), c.ps, e.z0);
    const float dz = z - e.right, lp = c.L2 + z, lm = c.L2 - z;
    // fallback: the flattened walk, kThreads voxels = q pixels and r planes per step
    const int q = kThreads / npl, r = kThreads - q * npl;
    const int i0 = g0, k0 = kk;
    int dup = -1;  // info whose pixel the range's last info repeats (-1: none)
    float den = 0.0f;
    if (one_chunk) {
      const int ni = static_cast<int>(nin);
      __syncthreads();
      for (int j = tid; j < ni; j += kThreads) {
        const int64_t info = static_cast<int64_t>(fe.pixel_info_begin) + j;
        pixel_terms<SM>(c, e, s1, p16, w, sens, info, pa[j], pb[j]);
        if (j < ni - 1 && p32[info] == last_pixel) dup = j;
      }
      __syncthreads();
      // thread = (pixel group g, plane k): groups walk the pixels g, g + G, ...;
      // the first kSteps weights are kept for the back-projection
      const int nmine = active ? (ni - g0 + G - 1) / G : 0;  // pixels of this thread
      const int ncached = nmine < kSteps ? nmine : kSteps;
      const float4* a = pa + g0;
      const float4* b = pb + g0;
      float* cp = cache + tid;
      for (int t = 0; t < ncached; ++t, a += G, b += G, cp += kThreads) {
        const float4 bv = *b;
        const float v = plane_weight<SM>(c, e, *a, bv, dz, lp, lm, col, rho, w);
        den = fmaf(v, voxel_sens<SM>(c, bv.z, col, sens), den);
        *cp = v;
      }
      for (int t = ncached; t < nmine; ++t, a += G, b += G) {
        const float4 bv = *b;
        den = fmaf(plane_weight<SM>(c, e, *a, bv, dz, lp, lm, col, rho, w),
                   voxel_sens<SM>(c, bv.z, col, sens), den);
      }
    } else {
      for (int64_t cb = 0; cb < nin; cb += kPix) {
        const int cn = static_cast<int>(nin - cb < kPix ? nin - cb : kPix);
        __syncthreads();
        for (int j = tid; j < cn; j += kThreads) {
          const int64_t info = static_cast<int64_t>(fe.pixel_info_begin) + cb + j;
          pixel_terms<SM>(c, e, s1, p16, w, sens, info, pa[j], pb[j]);
          if (cb + j < nin - 1 && p32[info] == last_pixel) dup = static_cast<int>(cb + j);
        }
        __syncthreads();
        for (int i = i0, k = k0; i < cn; walk(i, k, q, r, npl))
          den = fmaf(voxel_weight<SM>(c, e, pa[i], pb[i], k, rho, w),
                     voxel_sens<SM>(c, pb[i].z, e.plane_begin + k, sens), den);
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      den += __shfl_xor_sync(0xffffffffu, den, o);
      dup = max(dup, __shfl_xor_sync(0xffffffffu, dup, o));
    }
    if (lane == 0) {
      red_den[wid] = den;
      red_dup[wid] = dup;
    }
    __syncthreads();
    den = 0.0f;
    dup = -1;
#pragma unroll
    for (int j = 0; j < kWarpsPerCta; ++j) {
      den += red_den[j];
      dup = max(dup, red_dup[j]);
    }
    if (!(den > 0.0f)) continue;
    positive += (tid == 0);
    const float inv = __frcp_rn(den);
    if (one_chunk) {
      const int ni = static_cast<int>(nin);
      const int nmine = active ? (ni - g0 + G - 1) / G : 0;
      const int ncached = nmine < kSteps ? nmine : kSteps;
      const float4* a = pa + g0;
      const float4* b = pb + g0;
      const float* cp = cache + tid;
      float* o = out + col;
      if (dup < 0) {
        int t = 0;
        for (; t < ncached; ++t, b += G, cp += kThreads) {
          const float v = *cp;
          if (v != 0.0f) atomicAdd(o + __float_as_int(b->w), v * inv);
        }
        for (a += t * G; t < nmine; ++t, a += G, b += G) {
          const float4 bv = *b;
          const float v = plane_weight<SM>(c, e, *a, bv, dz, lp, lm, col, rho, w);
          if (v != 0.0f) atomicAdd(o + __float_as_int(bv.w), v * inv);
        }
      } else {
        for (int t = 0, i = g0; t < nmine; ++t, i += G, a += G, b += G, cp += kThreads) {
          const float4 bv = *b;
          const float v =
              t < ncached ? *cp : plane_weight<SM>(c, e, *a, bv, dz, lp, lm, col, rho, w);
          const float x = v * multiplicity(i, dup, ni - 1);
          if (x != 0.0f) atomicAdd(o + __float_as_int(bv.w), x * inv);
        }
      }
    } else {
      for (int64_t cb = 0; cb < nin; cb += kPix) {
        const int cn = static_cast<int>(nin - cb < kPix ? nin - cb : kPix);
        __syncthreads();
        for (int j = tid; j < cn; j += kThreads)
          pixel_terms<SM>(c, e, s1, p16, w, sens,
                          static_cast<int64_t>(fe.pixel_info_begin) + cb + j, pa[j], pb[j]);
        __syncthreads();
        for (int i = i0, k = k0; i < cn; walk(i, k, q, r, npl)) {
          const float x = voxel_weight<SM>(c, e, pa[i], pb[i], k, rho, w) *
                          multiplicity(cb + i, dup, nin - 1);
          if (x != 0.0f) atomicAdd(&out[__float_as_int(pb[i].w) + e.plane_begin + k], x * inv);
        }
      }
    }
  }
  if (tid == 0 && positive) atomicAdd(n_positive, positive);
}


// ---- voxel weights of the geometry ---------------------------------------------

// Per (pixel info, plane): pixel weight times pi over the frame sensitivity's
// angle, the part of a voxel's weight that no event changes (0 where the angle
// is negative); per pixel info: its projection on the LOR and its pixel.  One
// warp per LOR, lanes over the planes.
template <int SM>
__global__ void voxel_table_kernel(const float4* __restrict__ seg, const int16_t* __restrict__ p16,
                                   const float* __restrict__ w, const uint64_t* __restrict__ ib,
                                   const uint64_t* __restrict__ ie, HybConst c,
                                   float* __restrict__ table, float2* __restrict__ info_up) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t l = warp; l < c.n_lors; l += n_warps) {
    if (ib[l] >= ie[l]) continue;
    const float4 s1 = seg[3 * l + 1];
    const float R = __fdiv_rn(seg[3 * l + 2].z, 2.0f);
    for (uint64_t i = ib[l]; i < ie[l]; ++i) {
      const float up = lor_up(c, s1, p16, i);
      if (lane == 0)
        info_up[i] = make_float2(up, __int_as_float(p16[2 * i] + c.n_columns * p16[2 * i + 1]));
      const float rm = __frcp_rn(__fsub_rn(R, up)), rp = __frcp_rn(__fadd_rn(R, up));
      for (int k = lane; k < c.n_planes; k += 32) {
        const float z = __fadd_rn(__fmul_rn(__fadd_rn(static_cast<float>(k), 0.5f), c.ps),
                                  c.z_left);
        const float ang = frame_angle(rm, rp, c.L2 + z, c.L2 - z);
        const float wv = SM == kMultiPlane
                             ? w[static_cast<int64_t>(abs_plane(k, c.n_planes_half)) * c.n_infos + i]
                             : w[i];
        table[static_cast<int64_t>(i) * c.pitch + k] =
            ang < 0.0f ? 0.0f : (wv * kPi) * rcp(ang);
      }
    }
  }
}

// An event of the table iteration: the frame event, its LOR's half length, and
// whether its last pixel info lies past the LOR's end.
struct TabEvent {
  float up, right, tan, sec;
  float R;
  int32_t begin, n_infos, lor;
  int32_t plane_begin, n_planes, past, pad;
};
static_assert(sizeof(TabEvent) == 3 * sizeof(float4), "three 16-byte pieces");

// Sort keys of the table iteration's event order: the first pixel info; events
// that do not fit its CTA (and those without a voxel) last, counted.
constexpr uint32_t kNotTabled = 0x80000000u;
__global__ void event_order_kernel(const jpet_hybrid_frame_event* __restrict__ ev, int32_t n,
                                   uint32_t* __restrict__ keys, int32_t* __restrict__ order,
                                   int* __restrict__ n_rest) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const jpet_hybrid_frame_event e = ev[i];
  const int npl = e.plane_end - e.plane_begin;
  const int64_t nin = static_cast<int64_t>(e.pixel_info_end - e.pixel_info_begin);
  const bool fits = npl > 0 && npl <= 4 * kTabThreads - 6 && nin > 0 && nin <= kPix;
  if (!fits) atomicAdd(n_rest, 1);
  keys[i] = fits ? static_cast<uint32_t>(e.pixel_info_begin) : kNotTabled;
  order[i] = i;
}
__global__ void tab_events_kernel(const jpet_hybrid_frame_event* __restrict__ ev,
                                  const int32_t* __restrict__ order, int32_t n,
                                  const float4* __restrict__ seg, const uint64_t* __restrict__ ie,
                                  TabEvent* __restrict__ out) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const jpet_hybrid_frame_event e = ev[order[i]];
  const int64_t l = lor_index(e.lor_first, e.lor_second);
  TabEvent t;
  t.up = e.up;
  t.right = e.right;
  t.tan = e.tan;
  t.sec = e.sec;
  t.R = __fdiv_rn(seg[3 * l + 2].z, 2.0f);
  t.begin = static_cast<int32_t>(e.pixel_info_begin);
  t.n_infos = static_cast<int32_t>(e.pixel_info_end - e.pixel_info_begin);
  t.lor = static_cast<int32_t>(l);
  t.plane_begin = e.plane_begin;
  t.n_planes = e.plane_end - e.plane_begin;
  t.past = e.pixel_info_end > ie[l];
  t.pad = 0;
  out[i] = t;
}

// Adds four values to an aligned quad of global memory that the kernel does not read.
__device__ __forceinline__ void red_add4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y),
               "f"(v.z), "f"(v.w));
}

// The iteration with the voxel table: one CTA per event, a thread takes a quad
// of planes (aligned in the image and the table) of the pixel infos g, g + G, ...
// (G groups of as many threads as the event has quads); planes outside the
// event's range get weight 0.  A thread's table entries (its first kTabSteps
// quads) arrive in its own cache slots by asynchronous copies while the CTA
// computes the event's pixel terms; a voxel then costs one ex2 and a few
// multiplications instead of an arctangent and two reciprocals, and its weight
// takes the entry's place for the back-projection, one vector reduction per
// quad.  The next event's record is loaded a whole event ahead.  Events come in
// the order of their first pixel info, so that CTAs running together read the
// same lines of the table.  An info past the LOR's end (the table holds it for
// its own LOR) is computed by the threads of its group.
//
// 1e6 events on the 384-detector ring (3112 voxels each): 10.2 ms per iteration
// with the weights computed per event (65 instructions a voxel after the table's
// loads alone replaced the arctangent); one plane per thread 8.1 ms, bound by the
// wavefronts of 4-byte accesses (80 % of the L1 data pipe); in quads 6.0 ms, 33
// instructions a voxel, bound by the reductions' way to L2 (the busiest slice's
// input 68 % busy) and the latency of the rho loads.
template <int SM>
__global__ void __launch_bounds__(kTabThreads)
    iterate_table_kernel(const TabEvent* __restrict__ ev, int32_t n,
                         const float* __restrict__ table, const float2* __restrict__ info_up,
                         const float4* __restrict__ seg, const int16_t* __restrict__ p16,
                         const float* __restrict__ w, const float* __restrict__ sens,
                         const float* __restrict__ rho, float* __restrict__ out, HybConst c,
                         unsigned long long* __restrict__ n_positive) {
  constexpr int kWarps = kTabThreads / 32;
  __shared__ float4 rec[2 * kPix];  // dy, element_before_exp, exponent term, base index (int
                                    // bits); sensitivity or pixel index (int bits), unused x 3
  __shared__ float4 past_rec[2];    // pixel_terms of the info past the LOR's end
  __shared__ float4 cache[kTabSteps * kTabThreads];
  __shared__ float red_den[kWarps];
  __shared__ int red_dup[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t* p32 = reinterpret_cast<const uint32_t*>(p16);
  const float4* evp = reinterpret_cast<const float4*>(ev);
  const unsigned slot0 = static_cast<unsigned>(__cvta_generic_to_shared(cache + tid));
  unsigned long long positive = 0;
  int32_t ei = blockIdx.x;
  if (ei >= n) return;
  float4 q0 = evp[3 * static_cast<int64_t>(ei)], q1 = evp[3 * static_cast<int64_t>(ei) + 1],
         q2 = evp[3 * static_cast<int64_t>(ei) + 2];
  for (; ei < n; ei += gridDim.x) {
    EvC e;
    e.up = q0.x;
    e.right = q0.y;
    e.tan = q0.z;
    e.sec = q0.w;
    e.R = q1.x;
    const int begin = __float_as_int(q1.y), nin = __float_as_int(q1.z);
    const int64_t l = __float_as_int(q1.w);
    e.plane_begin = __float_as_int(q2.x);
    const int npl = __float_as_int(q2.y);
    const bool past = __float_as_int(q2.z) != 0;
    {
      const int64_t nx = ei + static_cast<int32_t>(gridDim.x) < n ? ei + gridDim.x : ei;
      q0 = evp[3 * nx];
      q1 = evp[3 * nx + 1];
      q2 = evp[3 * nx + 2];
    }
    const int quad0 = e.plane_begin >> 2, Q = ((e.plane_begin + npl - 1) >> 2) - quad0 + 1;
    // (a whole number + 1/2) / Q or / G is at least 1 / 512 from a whole number:
    // these quotients are exact in FP32
    const float rq = __frcp_rn(static_cast<float>(Q));
    const int G = static_cast<int>((kTabThreads + 0.5f) * rq);
    const int g0 = static_cast<int>((static_cast<float>(tid) + 0.5f) * rq);
    const int n_tab = nin - (past ? 1 : 0);
    const bool active = g0 < G;
    const int nmt = active && n_tab > g0
                        ? static_cast<int>((static_cast<float>(n_tab - g0) - 0.5f) *
                                           __frcp_rn(static_cast<float>(G))) + 1
                        : 0;
    const int nct = nmt < kTabSteps ? nmt : kTabSteps;
    const int col = 4 * (quad0 + tid - g0 * Q);  // the thread's first plane
    const float4* tp = reinterpret_cast<const float4*>(
        table + (static_cast<int64_t>(begin) + g0) * c.pitch + col);
    const int64_t t_step = static_cast<int64_t>(G) * (c.pitch >> 2);
    {
      const float4* src = tp;
      unsigned dst = slot0;
      for (int t = 0; t < nct; ++t, src += t_step, dst += kTabThreads * sizeof(float4))
        cp_async16(dst, src);
    }
    __syncthreads();  // the last event's records have been read
    int dup = -1;     // info whose pixel the info past the LOR's end repeats (-1: none)
    for (int j = tid; j < n_tab; j += kTabThreads) {
      const float2 iu = __ldg(&info_up[begin + j]);
      float sv;
      rec[2 * j] = table_terms<SM>(c, e, iu, sens, sv);
      rec[2 * j + 1].x = sv;
      if (past && p32[begin + j] == p32[begin + n_tab]) dup = j;
    }
    e.z0 = __fadd_rn(__fmul_rn(__fadd_rn(static_cast<float>(e.plane_begin), 0.5f), c.ps), c.z_left);
    const int k0 = col - e.plane_begin;  // planes k0 .. k0 + 3 of the event
    float dz[4];
    bool in[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      dz[i] = fmaf(static_cast<float>(k0 + i), c.ps, e.z0) - e.right;
      in[i] = k0 + i >= 0 && k0 + i < npl;
    }
    if (past && tid == 0)
      pixel_terms<SM>(c, e, seg[3 * l + 1], p16, w, sens, begin + n_tab, past_rec[0], past_rec[1]);
    cp_async_wait();
    __syncthreads();
    const float* rc = rho + col;
    // weights of a quad and their contribution to the denominator
    auto quad = [&](const float4* r, const float4 W, float& den) {
      const float4 a = r[0];
      const float sv = r[1].x;
      const float4 rh = __ldg(reinterpret_cast<const float4*>(rc + __float_as_int(a.w)));
      const float ww[4] = {W.x, W.y, W.z, W.w}, rr[4] = {rh.x, rh.y, rh.z, rh.w};
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float b = fmaf(-a.x, e.tan, dz[i]);
        const float x = a.y * ex2(fmaf(b * b, c.exp_bpq, a.z)) * ww[i] * rr[i];
        v[i] = in[i] ? x : 0.0f;
        if (SM != kSens2D && in[i]) den = fmaf(v[i], voxel_sens<SM>(c, sv, col + i, sens), den);
      }
      if (SM == kSens2D) den = fmaf((v[0] + v[1]) + (v[2] + v[3]), sv, den);
      return make_float4(v[0], v[1], v[2], v[3]);
    };
    float den = 0.0f;
    {
      const float4* r = rec + 2 * g0;
      float4* s = cache + tid;
#pragma unroll 2
      for (int t = 0; t < nct; ++t, r += 2 * G, s += kTabThreads) *s = quad(r, *s, den);
      const float4* src = tp + nct * t_step;
      for (int t = nct; t < nmt; ++t, r += 2 * G, src += t_step) quad(r, __ldg(src), den);
    }
    const bool mine_past = past && active && n_tab % G == g0;
    float v_past[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (mine_past) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (!in[i]) continue;
        const float z = fmaf(static_cast<float>(k0 + i), c.ps, e.z0);
        v_past[i] = plane_weight<SM>(c, e, past_rec[0], past_rec[1], dz[i], c.L2 + z, c.L2 - z,
                                     col + i, rho, w);
        den = fmaf(v_past[i], voxel_sens<SM>(c, past_rec[1].z, col + i, sens), den);
      }
    }
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    if (past) {
      for (int o = 16; o > 0; o >>= 1) dup = max(dup, __shfl_xor_sync(0xffffffffu, dup, o));
      if (lane == 0) red_dup[wid] = dup;
    }
    if (lane == 0) red_den[wid] = den;
    __syncthreads();
    den = 0.0f;
#pragma unroll
    for (int j = 0; j < kWarps; ++j) den += red_den[j];
    if (past) {
#pragma unroll
      for (int j = 0; j < kWarps; ++j) dup = max(dup, red_dup[j]);
    }
    if (!(den > 0.0f)) continue;
    positive += (tid == 0);
    const float inv = __frcp_rn(den);
    // 1 / den overflows below 2^-128: a weight of 0 still adds nothing
    const bool plain = inv <= 3.0e38f;
    auto share = [&](float v) { return plain || v != 0.0f ? v * inv : 0.0f; };
    auto add = [&](float base, float4 v) {
      red_add4(out + col + __float_as_int(base),
               make_float4(share(v.x), share(v.y), share(v.z), share(v.w)));
    };
    const float4* r = rec + 2 * g0;
    const float4* s = cache + tid;
    const int gd = dup < 0 ? -1 : (dup - g0) % G == 0 ? (dup - g0) / G : -1;  // its step, or -1
    if (plain && dup < 0) {
#pragma unroll 2
      for (int t = 0; t < nct; ++t, r += 2 * G, s += kTabThreads) {
        const float4 v = *s;
        red_add4(out + col + __float_as_int(r[0].w),
                 make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv));
      }
    } else {
      for (int t = 0; t < nct; ++t, r += 2 * G, s += kTabThreads)
        if (t != gd) add(r[0].w, *s);
    }
    const float4* src = tp + nct * t_step;
    float unused = 0.0f;
    for (int t = nct; t < nmt; ++t, r += 2 * G, src += t_step)
      if (t != gd) add(r[0].w, quad(r, __ldg(src), unused));
    if (mine_past) {
      const float m = multiplicity(n_tab, dup, n_tab);
      add(past_rec[1].w,
          make_float4(v_past[0] * m, v_past[1] * m, v_past[2] * m, v_past[3] * m));
    }
  }
  if (tid == 0 && positive) atomicAdd(n_positive, positive);
}

}  // namespace

struct jpet_hybrid {
  jpet_hybrid_opts opts{};
  HybConst c{};
  int device = 0;
  int n_sms = 0;
  int iterate_blocks = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t own_stream = nullptr;
  std::string last_error = "no error";
  int64_t n_events = 0;
  int64_t used_pixels = 0, used_voxels = 0;
  Buf<float4> seg;           // 3 float4 per LOR (the LineSegment fields)
  Buf<float> widths, pos, w, sens, rho, out, stage;
  Buf<int2> pix_dummy;
  Buf<int16_t> pix;          // x, y per pixel info
  Buf<uint64_t> ib, ie;
  Buf<jpet_hybrid_frame_event> ev, ev_tmp;
  Buf<jpet_hybrid_response> resp;
  Buf<uint8_t> keep, temp;
  Buf<int32_t> keys, vals;
  Buf<long long> n_sel;
  Buf<unsigned long long> counters;  // [0] pixels [1] voxels [2] positive
  Buf<int> flag;
  Buf<float> table;          // voxel weights of the geometry (empty: computed per event)
  Buf<float2> info_up;       // with it: per pixel info, projection on the LOR and pixel index
  Buf<TabEvent> tab_events;  // events of the table iteration, in its order
  Buf<uint32_t> order_keys;  // event order: sort keys (input, output)
  Buf<int32_t> order;        // event order: event indices (input, output)
  int64_t n_tabled = 0;      // events of the table iteration; order[n + n_tabled ...] the rest
  double not_saved = 0.0;    // what the iterations so far would have saved (table_saves)
  bool table_refused = false, order_refused = false;  // for the held events
  bool shared_infos = false; // a pixel info lies in the ranges of several LORs: no table
  int table_blocks = 0;
};

namespace {

int fail(jpet_hybrid* h, int code, const std::string& msg) {
  if (h) h->last_error = msg;
  else g_hybrid_error = msg;
  return code;
}

int cuda_fail(jpet_hybrid* h, cudaError_t e, const char* what) {
  return fail(h, JPET_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define HYB_CUDA(h, call, what)                     \
  do {                                              \
    cudaError_t e_ = (call);                        \
    if (e_ != cudaSuccess) return cuda_fail(h, e_, what); \
  } while (0)

int grid_for(const jpet_hybrid* h, int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(h->n_sms) * 8;
  return static_cast<int>(std::max<int64_t>(1, std::min(b, cap)));
}

// Kernel constants computed as GaussianKernel's constructor computes them
// (gaussian_kernel.h:27-33: float reciprocals, the normalisation in double
// from a float square root) and the grid's as PixelGrid's (pixel_grid.h:24-30).
HybConst make_const(const jpet_hybrid_geom& g) {
  HybConst c{};
  c.ipz = 1.0f / (g.sigma_z * g.sigma_z);
  c.ipd = 1.0f / (g.sigma_dl * g.sigma_dl);
  c.c0 = static_cast<float>(1.0 / (2.0 * M_PI * M_PI) *
                            static_cast<double>(std::sqrt(c.ipz * c.ipz * c.ipd)));
  c.ps = g.pixel_size;
  c.z_left = g.z_left;
  c.llcx = g.lower_left_x + g.pixel_size / 2.0f;
  c.llcy = g.lower_left_y + g.pixel_size / 2.0f;
  c.L2 = g.length / 2.0f;
  c.exp_bpq = static_cast<float>(-1.4426950408889634 * static_cast<double>(c.ipz));
  c.n_columns = g.n_columns;
  c.n_rows = g.n_rows;
  c.n_planes = g.n_planes;
  // planes in whole quads, but for a few planes (mostly padding) and images whose
  // indices would then pass 31 bits
  const int32_t quads = (g.n_planes + 3) & ~3;
  c.pitch = g.n_planes >= 8 && static_cast<int64_t>(g.n_columns) * g.n_rows * quads <
                                   (int64_t(1) << 31)
                ? quads
                : g.n_planes;
  c.n_lors = static_cast<int32_t>((static_cast<int64_t>(g.n_detectors) + 1) * g.n_detectors / 2);
  c.n_infos = g.n_pixel_infos;
  c.n_planes_half = g.n_planes_half > 1 ? g.n_planes_half : 1;
  c.sens_depth = 1;
  return c;
}

int check_geom(const jpet_hybrid_geom* g) {
  if (!g) return fail(nullptr, JPET_ERR_ARGUMENT, "geometry is NULL");
  if (g->n_detectors < 1 || g->n_detectors > 32767)
    return fail(nullptr, JPET_ERR_ARGUMENT, "n_detectors must be in [1, 32767]");
  if (g->n_pixel_infos < 0 || g->n_pixel_infos >= (int64_t(1) << 31))
    return fail(nullptr, JPET_ERR_ARGUMENT, "n_pixel_infos must be in [0, 2^31)");
  if (g->n_columns < 1 || g->n_rows < 1 || g->n_planes < 1 || g->n_columns > 32767 ||
      g->n_rows > 32767 || g->n_planes > 32767)
    return fail(nullptr, JPET_ERR_ARGUMENT, "grid sizes must be in [1, 32767]");
  if (static_cast<int64_t>(g->n_columns) * g->n_rows * g->n_planes >= (int64_t(1) << 31))
    return fail(nullptr, JPET_ERR_ARGUMENT, "more than 2^31 - 1 voxels");
  if (!(g->pixel_size > 0) || !(g->sigma_z > 0) || !(g->sigma_dl > 0) || !(g->length > 0))
    return fail(nullptr, JPET_ERR_ARGUMENT, "pixel size, sigmas and length must be positive");
  if (!g->lor_segments || !g->lor_pixel_info_begin || !g->lor_pixel_info_end)
    return fail(nullptr, JPET_ERR_ARGUMENT, "LOR arrays are NULL");
  if (g->n_pixel_infos > 0 && (!g->pixels || !g->pixel_positions))
    return fail(nullptr, JPET_ERR_ARGUMENT, "pixel info arrays are NULL");
  if (g->n_planes_half < 0 || g->n_planes_half > g->n_planes)
    return fail(nullptr, JPET_ERR_ARGUMENT, "n_planes_half must be in [0, n_planes]");
  if (g->n_planes_half > 1 && g->n_pixel_infos * g->n_planes_half >= (int64_t(1) << 31))
    return fail(nullptr, JPET_ERR_ARGUMENT, "more than 2^31 - 1 weights");
  const int64_t n_lors = (static_cast<int64_t>(g->n_detectors) + 1) * g->n_detectors / 2;
  for (int64_t l = 0; l < n_lors; ++l) {
    if (g->lor_pixel_info_begin[l] > g->lor_pixel_info_end[l] ||
        g->lor_pixel_info_end[l] > static_cast<uint64_t>(g->n_pixel_infos))
      return fail(nullptr, JPET_ERR_ARGUMENT,
                  "LOR " + std::to_string(l) + ": pixel info range outside [0, n_pixel_infos]");
  }
  return JPET_OK;
}

// Whether a pixel info lies in the ranges of two LORs (given weights allow it): its
// voxel weights then depend on the event's LOR, which the voxel table cannot hold.
bool ranges_overlap(const jpet_hybrid_geom& g, int64_t n_lors) {
  uint64_t end = 0;
  int64_t l = 0;
  for (; l < n_lors; ++l) {  // in LOR order, as the reference's geometries have them
    if (g.lor_pixel_info_begin[l] == g.lor_pixel_info_end[l]) continue;
    if (g.lor_pixel_info_begin[l] < end) break;
    end = g.lor_pixel_info_end[l];
  }
  if (l == n_lors) return false;
  std::vector<std::pair<uint64_t, uint64_t>> r;
  for (l = 0; l < n_lors; ++l)
    if (g.lor_pixel_info_begin[l] < g.lor_pixel_info_end[l])
      r.emplace_back(g.lor_pixel_info_begin[l], g.lor_pixel_info_end[l]);
  std::sort(r.begin(), r.end());
  for (size_t k = 1; k < r.size(); ++k)
    if (r[k].first < r[k - 1].second) return true;
  return false;
}

// Stable radix sort of (pixel index, info index): the infos of each pixel in
// ascending info order.  Used to check that no LOR lists a pixel twice and, for
// the computed sensitivity, to sum each pixel's weights sequentially in that
// order (the reference's order of additions).
int sort_and_check_pixels(jpet_hybrid* h, bool sum) {
  const int64_t n = h->c.n_infos;
  const int64_t n_px = static_cast<int64_t>(h->c.n_columns) * h->c.n_rows;
  HYB_CUDA(h, cudaMemsetAsync(h->sens.p, 0, n_px * h->c.sens_depth * sizeof(float), h->stream),
           "memset");
  if (n == 0) return JPET_OK;
  Buf<int32_t> keys2, vals2, lor_of;
  struct Release {
    Buf<int32_t>* b[3];
    ~Release() {
      for (auto* x : b) x->release();
    }
  } release{{&keys2, &vals2, &lor_of}};
  HYB_CUDA(h, keys2.alloc(n), "cudaMalloc");
  HYB_CUDA(h, vals2.alloc(n), "cudaMalloc");
  HYB_CUDA(h, lor_of.alloc(n), "cudaMalloc");
  int end_bit = 1;
  while ((int64_t(1) << end_bit) < n_px) ++end_bit;
  size_t bytes = 0;
  HYB_CUDA(h, cub::DeviceRadixSort::SortPairs(nullptr, bytes, h->keys.p, keys2.p, h->vals.p,
                                              vals2.p, static_cast<int>(n), 0, end_bit,
                                              h->stream),
           "sort size");
  HYB_CUDA(h, h->temp.alloc(bytes), "cudaMalloc");
  HYB_CUDA(h, cub::DeviceRadixSort::SortPairs(h->temp.p, bytes, h->keys.p, keys2.p, h->vals.p,
                                              vals2.p, static_cast<int>(n), 0, end_bit,
                                              h->stream),
           "sort");
  HYB_CUDA(h, cudaMemsetAsync(lor_of.p, 0xff, n * sizeof(int32_t), h->stream), "memset");
  lor_of_info_kernel<<<grid_for(h, 32LL * h->c.n_lors), 256, 0, h->stream>>>(h->ib.p, h->ie.p,
                                                                           h->c.n_lors, lor_of.p);
  HYB_CUDA(h, cudaGetLastError(), "lor of info");
  HYB_CUDA(h, cudaMemsetAsync(h->flag.p, 0, sizeof(int), h->stream), "memset");
  unique_pixels_kernel<<<grid_for(h, n), 256, 0, h->stream>>>(keys2.p, vals2.p, n, lor_of.p,
                                                             h->flag.p);
  HYB_CUDA(h, cudaGetLastError(), "unique pixels");
  if (sum) {
    // one plane half after another (calculate_sensitivity sums each
    // (pixel, plane) over the infos in info order)
    for (int plane = 0; plane < h->c.n_planes_half; ++plane) {
      sensitivity_sum_kernel<<<grid_for(h, n), 256, 0, h->stream>>>(
          keys2.p, vals2.p, n, h->w.p + n * plane, h->sens.p + n_px * plane);
      HYB_CUDA(h, cudaGetLastError(), "sensitivity");
    }
  }
  int bad = 0;
  HYB_CUDA(h, cudaMemcpyAsync(&bad, h->flag.p, sizeof bad, cudaMemcpyDeviceToHost, h->stream),
           "copy");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  if (bad) return fail(h, JPET_ERR_ARGUMENT, "a LOR lists the same pixel twice");
  return JPET_OK;
}

// What the voxel table saves and costs, in microseconds.  An iteration saves about
// 1.35 ns per event and 0.88 ps per voxel: 1e6 events on the 384-detector ring (3.1e9
// voxels) 10.3 -> 6.1 ms, 5e5 on a 96-detector one (2.8e8) 2.07 -> 1.14 ms.  The table
// (4.2e9 entries, 16.9 GB, and 5.3e7) costs 3.6 ps an entry, allocation included, and
// with the first event order 0.3 ms and 2 ns an event; another set's order 0.08 ms
// and 0.15 ns an event.  So the table is made by the call that asks for enough
// iterations; calls that ask for a few at a time have to pass twice that, as they may be
// the last.  Set-up and k iterations without the table / with one made at once, ms:
// 1e6 events k = 3 31.4 / 34.2, k = 5 53.7 / 46.4; 1.7e5 k = 5 9.2 / 20.7, k = 20 35.6 /
// 36.7; on the 96-detector ring 1e5 events k = 3 1.51 / 1.55, k = 5 2.35 / 2.01, 3e4 events
// k = 5 0.90 / 1.21, k = 20 2.89 / 2.35.
double table_saves(const jpet_hybrid* h, int64_t iterations) {
  return static_cast<double>(iterations) * (1.35e-3 * static_cast<double>(h->n_events) +
                                            0.88e-6 * static_cast<double>(h->used_voxels));
}
double table_costs(const jpet_hybrid* h) {
  const double n = static_cast<double>(h->n_events);
  if (h->table.p) return 80.0 + 0.15e-3 * n;
  return 300.0 + 2e-3 * n + 3.6e-6 * static_cast<double>(h->c.n_infos * h->c.pitch);
}

// The voxel-weight table, if this handle may have it (at most a quarter of the free
// memory).
int make_table(jpet_hybrid* h) {
  const int64_t entries = h->c.n_infos * h->c.pitch;
  h->table_refused = true;
  size_t free_bytes = 0, total = 0;
  HYB_CUDA(h, cudaMemGetInfo(&free_bytes, &total), "memory info");
  if (static_cast<size_t>(entries) * sizeof(float) > free_bytes / 4) return JPET_OK;
  if (h->info_up.alloc(h->c.n_infos) != cudaSuccess || h->table.alloc(entries) != cudaSuccess) {
    cudaGetLastError();  // fragmented memory: the iterations compute the weights
    return JPET_OK;
  }
  const int blocks = h->n_sms * 8;
  if (h->c.n_planes_half > 1)
    voxel_table_kernel<kMultiPlane><<<blocks, 256, 0, h->stream>>>(
        h->seg.p, h->pix.p, h->w.p, h->ib.p, h->ie.p, h->c, h->table.p, h->info_up.p);
  else
    voxel_table_kernel<kSens2D><<<blocks, 256, 0, h->stream>>>(
        h->seg.p, h->pix.p, h->w.p, h->ib.p, h->ie.p, h->c, h->table.p, h->info_up.p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) h->table.release();
  HYB_CUDA(h, e, "voxel table");
  // the iterations may run on another stream
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  h->table_refused = false;
  return JPET_OK;
}

// The event order of the table iterations.
int order_events(jpet_hybrid* h) {
  const int64_t n = h->n_events;
  size_t bytes = 0;
  HYB_CUDA(h, cub::DeviceRadixSort::SortPairs(nullptr, bytes, h->order_keys.p, h->order_keys.p + n,
                                              h->order.p, h->order.p + n, static_cast<int>(n), 0,
                                              32, h->stream),
           "sort size");
  if (h->order_keys.alloc(2 * n) != cudaSuccess || h->order.alloc(2 * n) != cudaSuccess ||
      h->tab_events.alloc(n) != cudaSuccess || h->temp.alloc(bytes) != cudaSuccess) {
    cudaGetLastError();  // no room: the iterations compute the weights
    h->order_refused = true;
    return JPET_OK;
  }
  HYB_CUDA(h, cudaMemsetAsync(h->flag.p, 0, sizeof(int), h->stream), "memset");
  event_order_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, h->stream>>>(
      h->ev.p, static_cast<int32_t>(n), h->order_keys.p, h->order.p, h->flag.p);
  HYB_CUDA(h, cudaGetLastError(), "event order");
  HYB_CUDA(h, cub::DeviceRadixSort::SortPairs(h->temp.p, bytes, h->order_keys.p,
                                              h->order_keys.p + n, h->order.p, h->order.p + n,
                                              static_cast<int>(n), 0, 32, h->stream),
           "sort");
  int rest = 0;
  HYB_CUDA(h, cudaMemcpyAsync(&rest, h->flag.p, sizeof rest, cudaMemcpyDeviceToHost, h->stream),
           "copy");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  const int64_t tabled = n - rest;
  if (tabled > 0) {
    tab_events_kernel<<<static_cast<unsigned>((tabled + 255) / 256), 256, 0, h->stream>>>(
        h->ev.p, h->order.p + n, static_cast<int32_t>(tabled), h->seg.p, h->ie.p,
        h->tab_events.p);
    HYB_CUDA(h, cudaGetLastError(), "table events");
  }
  // the iterations may run on another stream
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  h->n_tabled = tabled;
  h->not_saved = 0.0;
  h->order_refused = tabled == 0;  // nothing to gain
  return JPET_OK;
}

// Makes the table and the event order where `asked` iterations of the held events
// pay for them (never inside a stream capture: what is there by then is used).
int prepare_table(jpet_hybrid* h, int64_t asked) {
  const int64_t n = h->n_events, entries = h->c.n_infos * h->c.pitch;
  if (n == 0 || h->n_tabled > 0 || h->order_refused || h->table_refused) return JPET_OK;
  if (h->shared_infos || entries <= 0 || (h->c.pitch & 3) != 0 || n > INT32_MAX / 2)
    return JPET_OK;
  const double cost = table_costs(h), saved = table_saves(h, asked);
  if (saved < cost && h->not_saved + saved < 2.0 * cost) return JPET_OK;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  HYB_CUDA(h, cudaStreamIsCapturing(h->stream, &capture), "capture status");
  if (capture != cudaStreamCaptureStatusNone) return JPET_OK;
  if (!h->table.p) {
    const int rc = make_table(h);
    if (rc != JPET_OK || !h->table.p) return rc;
  }
  return order_events(h);
}

int finish_events(jpet_hybrid* h, int64_t n) {
  h->n_events = n;
  h->n_tabled = 0;
  if (h->table.p) h->not_saved = 0.0;  // an event order serves one set
  h->order_refused = h->table_refused = false;
  HYB_CUDA(h, cudaMemsetAsync(h->counters.p, 0, 3 * sizeof(unsigned long long), h->stream),
           "memset");
  HYB_CUDA(h, cudaMemsetAsync(h->flag.p, 0, sizeof(int), h->stream), "memset");
  if (n > 0) {
    event_stats_kernel<<<grid_for(h, n), 256, 0, h->stream>>>(h->ev.p, n, h->ib.p, h->ie.p, h->c,
                                                              h->counters.p, h->flag.p);
    HYB_CUDA(h, cudaGetLastError(), "event check");
  }
  unsigned long long st[2];
  int bad = 0;
  HYB_CUDA(h, cudaMemcpyAsync(st, h->counters.p, sizeof st, cudaMemcpyDeviceToHost, h->stream),
           "copy");
  HYB_CUDA(h, cudaMemcpyAsync(&bad, h->flag.p, sizeof bad, cudaMemcpyDeviceToHost, h->stream),
           "copy");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  if (bad) {
    h->n_events = 0;
    return fail(h, JPET_ERR_ARGUMENT,
                "frame event with a LOR, pixel-info range or plane range outside the geometry "
                "(ranges lie within the LOR's pixel infos and the one past its end)");
  }
  h->used_pixels = static_cast<int64_t>(st[0]);
  h->used_voxels = static_cast<int64_t>(st[1]);
  return JPET_OK;
}

// n iterations; ahead: the iterations that the caller knows to follow, these included.
int iterate(jpet_hybrid* h, int n, int64_t ahead) {
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const int rc = prepare_table(h, ahead);
  if (rc != JPET_OK) return rc;
  if (h->n_tabled == 0) h->not_saved += table_saves(h, n);
  const int64_t n_vox = static_cast<int64_t>(h->c.n_columns) * h->c.n_rows * h->c.pitch;
  for (int it = 0; it < n; ++it) {
    HYB_CUDA(h, cudaMemsetAsync(h->out.p, 0, n_vox * sizeof(float), h->stream), "memset");
    HYB_CUDA(h, cudaMemsetAsync(h->counters.p + 2, 0, sizeof(unsigned long long), h->stream),
             "memset");
    if (h->n_events > 0) {
      const bool multi = h->c.n_planes_half > 1, sens3d = h->c.sens_depth > 1;
      if (h->n_tabled > 0) {
        auto* k = multi    ? iterate_table_kernel<kMultiPlane>
                  : sens3d ? iterate_table_kernel<kSens3D>
                           : iterate_table_kernel<kSens2D>;
        k<<<h->table_blocks, kTabThreads, 0, h->stream>>>(
            h->tab_events.p, static_cast<int32_t>(h->n_tabled), h->table.p, h->info_up.p, h->seg.p,
            h->pix.p, h->w.p, h->sens.p, h->rho.p, h->out.p, h->c, h->counters.p + 2);
        HYB_CUDA(h, cudaGetLastError(), "iterate");
      }
      const int64_t rest = h->n_events - h->n_tabled;
      if (rest > 0) {
        auto* k = multi    ? iterate_kernel<kMultiPlane>
                  : sens3d ? iterate_kernel<kSens3D>
                           : iterate_kernel<kSens2D>;
        k<<<h->iterate_blocks, kThreads, 0, h->stream>>>(
            h->ev.p, h->n_tabled > 0 ? h->order.p + h->n_events + h->n_tabled : nullptr, rest,
            h->seg.p, h->pix.p, h->w.p, h->sens.p, h->rho.p, h->out.p, h->c, h->counters.p + 2);
        HYB_CUDA(h, cudaGetLastError(), "iterate");
      }
    }
    std::swap(h->rho, h->out);
  }
  return JPET_OK;
}

int translate(jpet_hybrid* h, const jpet_hybrid_response* d_resp, int64_t n) {
  HYB_CUDA(h, h->ev_tmp.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  HYB_CUDA(h, h->ev.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  HYB_CUDA(h, h->keep.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  long long kept = 0;
  if (n > 0) {
    translate_kernel<<<grid_for(h, n), 256, 0, h->stream>>>(
        d_resp, n, h->seg.p, h->pix.p, h->pos.p, h->w.p, h->ib.p, h->ie.p, h->c, h->ev_tmp.p,
        h->keep.p);
    HYB_CUDA(h, cudaGetLastError(), "translate");
    size_t bytes = 0;
    HYB_CUDA(h, cub::DeviceSelect::Flagged(nullptr, bytes, h->ev_tmp.p, h->keep.p, h->ev.p,
                                           h->n_sel.p, n, h->stream),
             "select size");
    HYB_CUDA(h, h->temp.alloc(bytes), "cudaMalloc");
    HYB_CUDA(h, cub::DeviceSelect::Flagged(h->temp.p, bytes, h->ev_tmp.p, h->keep.p, h->ev.p,
                                           h->n_sel.p, n, h->stream),
             "select");
    HYB_CUDA(h, cudaMemcpyAsync(&kept, h->n_sel.p, sizeof kept, cudaMemcpyDeviceToHost,
                                h->stream),
             "copy");
    HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  }
  return finish_events(h, kept);
}

}  // namespace

extern "C" {

void jpet_hybrid_default_opts(jpet_hybrid_opts* o) {
  if (!o) return;
  std::memset(o, 0, sizeof *o);
  o->weights = JPET_HYBRID_WEIGHTS_COMPUTED;
  o->sensitivity = JPET_HYBRID_SENSITIVITY_COMPUTED;
}

const char* jpet_hybrid_last_error(const jpet_hybrid_t* h) {
  return h ? h->last_error.c_str() : g_hybrid_error.c_str();
}

int jpet_hybrid_destroy(jpet_hybrid_t* h) {
  if (!h) return JPET_OK;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  h->seg.release();
  h->widths.release();
  h->pos.release();
  h->w.release();
  h->sens.release();
  h->rho.release();
  h->out.release();
  h->stage.release();
  h->pix.release();
  h->ib.release();
  h->ie.release();
  h->ev.release();
  h->ev_tmp.release();
  h->resp.release();
  h->keep.release();
  h->temp.release();
  h->keys.release();
  h->vals.release();
  h->n_sel.release();
  h->counters.release();
  h->flag.release();
  h->table.release();
  h->info_up.release();
  h->tab_events.release();
  h->order_keys.release();
  h->order.release();
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
  delete h;
  return JPET_OK;
}

int jpet_hybrid_create(const jpet_hybrid_geom* g, const jpet_hybrid_opts* opts_in,
                       jpet_hybrid_t** out) {
  if (!out) return fail(nullptr, JPET_ERR_ARGUMENT, "out is NULL");
  *out = nullptr;
  int rc = check_geom(g);
  if (rc != JPET_OK) return rc;
  jpet_hybrid_opts opts;
  jpet_hybrid_default_opts(&opts);
  if (opts_in) opts = *opts_in;
  if (opts.weights < 0 || opts.weights > 2 || opts.sensitivity < 0 || opts.sensitivity > 3)
    return fail(nullptr, JPET_ERR_ARGUMENT, "unknown weights or sensitivity mode");
  const int planes_half = g->n_planes_half > 1 ? g->n_planes_half : 1;
  if (planes_half > 1 && opts.weights == JPET_HYBRID_WEIGHTS_COMPUTED)
    return fail(nullptr, JPET_ERR_ARGUMENT,
                "a multi-plane geometry needs given weights (one system matrix per plane half)");
  if (planes_half > 1 && opts.sensitivity == JPET_HYBRID_SENSITIVITY_GIVEN)
    return fail(nullptr, JPET_ERR_ARGUMENT,
                "a multi-plane geometry has a 3D sensitivity (JPET_HYBRID_SENSITIVITY_GIVEN_3D)");
  // planes of the sensitivity image (reconstruction.h:80-85)
  const int sens_depth = planes_half > 1 ? planes_half
                         : opts.sensitivity == JPET_HYBRID_SENSITIVITY_GIVEN_3D ? g->n_planes / 2
                                                                                : 1;
  if (sens_depth < 1)
    return fail(nullptr, JPET_ERR_ARGUMENT, "a 3D sensitivity needs at least 2 planes");
  if (opts.weights != JPET_HYBRID_WEIGHTS_COMPUTED && g->n_pixel_infos > 0 && !g->pixel_weights)
    return fail(nullptr, JPET_ERR_ARGUMENT, "given weights but pixel_weights is NULL");
  if (opts.weights == JPET_HYBRID_WEIGHTS_COMPUTED && !g->lor_widths)
    return fail(nullptr, JPET_ERR_ARGUMENT, "computed weights need lor_widths");
  if ((opts.sensitivity == JPET_HYBRID_SENSITIVITY_GIVEN ||
       opts.sensitivity == JPET_HYBRID_SENSITIVITY_GIVEN_3D) && !opts.sensitivity_map)
    return fail(nullptr, JPET_ERR_ARGUMENT, "given sensitivity but sensitivity_map is NULL");
  if (opts.block_threads != 0)
    return fail(nullptr, JPET_ERR_UNSUPPORTED, "the iteration kernel runs 128-thread CTAs");
  auto* h = new jpet_hybrid();
  h->opts = opts;
  h->device = opts.device;
  h->c = make_const(*g);
  h->c.sens_depth = sens_depth;
  auto bail = [&](int code) {
    g_hybrid_error = h->last_error;
    jpet_hybrid_destroy(h);
    return code;
  };
#define CREATE_CUDA(call, what)                               \
  do {                                                        \
    cudaError_t e_ = (call);                                  \
    if (e_ != cudaSuccess) return bail(cuda_fail(h, e_, what)); \
  } while (0)
  CREATE_CUDA(cudaSetDevice(h->device), "cudaSetDevice");
  CREATE_CUDA(cudaDeviceGetAttribute(&h->n_sms, cudaDevAttrMultiProcessorCount, h->device),
              "device attribute");
  CREATE_CUDA(cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking), "stream");
  h->stream = h->own_stream;
  int per_sm = 0;
  CREATE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, iterate_kernel<kSens2D>,
                                                            kThreads, 0),
              "occupancy");
  h->iterate_blocks = std::max(1, per_sm) * h->n_sms;
  CREATE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                  &per_sm, iterate_table_kernel<kSens2D>, kTabThreads, 0),
              "occupancy");
  h->table_blocks = std::max(1, per_sm) * h->n_sms;

  const int64_t n_lors = h->c.n_lors, n = h->c.n_infos;
  h->shared_infos = ranges_overlap(*g, n_lors);
  const int64_t n_px = static_cast<int64_t>(h->c.n_columns) * h->c.n_rows;
  const int64_t n_vox = n_px * h->c.pitch;
  CREATE_CUDA(h->seg.alloc(3 * n_lors), "cudaMalloc");
  CREATE_CUDA(h->widths.alloc(n_lors), "cudaMalloc");
  CREATE_CUDA(h->ib.alloc(n_lors), "cudaMalloc");
  CREATE_CUDA(h->ie.alloc(n_lors), "cudaMalloc");
  CREATE_CUDA(h->pix.alloc(2 * std::max<int64_t>(n, 1)), "cudaMalloc");
  CREATE_CUDA(h->pos.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  CREATE_CUDA(h->w.alloc(std::max<int64_t>(n * planes_half, 1)), "cudaMalloc");
  CREATE_CUDA(h->keys.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  CREATE_CUDA(h->vals.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  CREATE_CUDA(h->sens.alloc(n_px * sens_depth), "cudaMalloc");
  CREATE_CUDA(h->rho.alloc(n_vox), "cudaMalloc");
  CREATE_CUDA(h->out.alloc(n_vox), "cudaMalloc");
  CREATE_CUDA(h->n_sel.alloc(1), "cudaMalloc");
  CREATE_CUDA(h->counters.alloc(3), "cudaMalloc");
  CREATE_CUDA(h->flag.alloc(1), "cudaMalloc");
  cudaStream_t s = h->stream;
  static_assert(sizeof(jpet_lor_segment) == 3 * sizeof(float4), "segment layout");
  CREATE_CUDA(cudaMemcpyAsync(h->seg.p, g->lor_segments, n_lors * sizeof(jpet_lor_segment),
                              cudaMemcpyHostToDevice, s),
              "upload");
  if (g->lor_widths)
    CREATE_CUDA(cudaMemcpyAsync(h->widths.p, g->lor_widths, n_lors * sizeof(float),
                                cudaMemcpyHostToDevice, s),
                "upload");
  CREATE_CUDA(cudaMemcpyAsync(h->ib.p, g->lor_pixel_info_begin, n_lors * sizeof(uint64_t),
                              cudaMemcpyHostToDevice, s),
              "upload");
  CREATE_CUDA(cudaMemcpyAsync(h->ie.p, g->lor_pixel_info_end, n_lors * sizeof(uint64_t),
                              cudaMemcpyHostToDevice, s),
              "upload");
  if (n > 0) {
    CREATE_CUDA(cudaMemcpyAsync(h->pix.p, g->pixels, n * sizeof(jpet_pixel),
                                cudaMemcpyHostToDevice, s),
                "upload");
    CREATE_CUDA(cudaMemcpyAsync(h->pos.p, g->pixel_positions, n * sizeof(float),
                                cudaMemcpyHostToDevice, s),
                "upload");
    if (opts.weights != JPET_HYBRID_WEIGHTS_COMPUTED)
      CREATE_CUDA(cudaMemcpyAsync(h->w.p, g->pixel_weights, n * planes_half * sizeof(float),
                                  cudaMemcpyHostToDevice, s),
                  "upload");
  }
  // pixels inside the grid, and the sort keys of the sensitivity
  CREATE_CUDA(cudaMemsetAsync(h->flag.p, 0, sizeof(int), s), "memset");
  if (n > 0) {
    pixel_keys_kernel<<<grid_for(h, n), 256, 0, s>>>(h->pix.p, n, h->c, h->keys.p, h->vals.p,
                                                     h->flag.p);
    CREATE_CUDA(cudaGetLastError(), "pixel check");
  }
  int bad = 0;
  CREATE_CUDA(cudaMemcpyAsync(&bad, h->flag.p, sizeof bad, cudaMemcpyDeviceToHost, s), "copy");
  CREATE_CUDA(cudaStreamSynchronize(s), "synchronize");
  if (bad) return bail(fail(h, JPET_ERR_ARGUMENT, "a pixel info lies outside the pixel grid"));
  if (opts.weights == JPET_HYBRID_WEIGHTS_COMPUTED && n > 0) {
    weights_kernel<<<grid_for(h, 32 * n_lors), 256, 0, s>>>(
        h->seg.p, h->widths.p, reinterpret_cast<const int2*>(h->pix.p), h->ib.p, h->ie.p, h->w.p,
        h->c, std::sqrt(2 * M_PI));
    CREATE_CUDA(cudaGetLastError(), "weights");
  }
  const int rc2 = sort_and_check_pixels(h, opts.sensitivity == JPET_HYBRID_SENSITIVITY_COMPUTED);
  if (rc2 != JPET_OK) return bail(rc2);
  if (opts.sensitivity == JPET_HYBRID_SENSITIVITY_ONE) {
    fill_kernel<<<grid_for(h, n_px * sens_depth), 256, 0, s>>>(h->sens.p, n_px * sens_depth,
                                                               1.0f);
    CREATE_CUDA(cudaGetLastError(), "fill");
  } else if (opts.sensitivity == JPET_HYBRID_SENSITIVITY_GIVEN ||
             opts.sensitivity == JPET_HYBRID_SENSITIVITY_GIVEN_3D) {
    CREATE_CUDA(cudaMemcpyAsync(h->sens.p, opts.sensitivity_map,
                                n_px * sens_depth * sizeof(float), cudaMemcpyHostToDevice, s),
                "upload");
  }
  h->keys.release();
  h->vals.release();
  if (opts.weights != JPET_HYBRID_WEIGHTS_NORMALIZED && n > 0) {
    normalize_kernel<<<grid_for(h, n), 256, 0, s>>>(h->pix.p, n, h->c, h->sens.p, h->w.p);
    CREATE_CUDA(cudaGetLastError(), "normalize");
  }
  fill_kernel<<<grid_for(h, n_vox), 256, 0, s>>>(h->rho.p, n_vox, 1.0f);
  CREATE_CUDA(cudaGetLastError(), "fill");
  CREATE_CUDA(cudaStreamSynchronize(s), "synchronize");
#undef CREATE_CUDA
  *out = h;
  return JPET_OK;
}

int jpet_hybrid_set_stream(jpet_hybrid_t* h, void* stream) {
  if (!h) return fail(nullptr, JPET_ERR_ARGUMENT, "handle is NULL");
  h->stream = stream ? static_cast<cudaStream_t>(stream) : h->own_stream;
  return JPET_OK;
}

int jpet_hybrid_set_responses_device(jpet_hybrid_t* h, const jpet_hybrid_response* d, int64_t n) {
  if (!h) return fail(nullptr, JPET_ERR_ARGUMENT, "handle is NULL");
  if (n < 0 || (n > 0 && !d)) return fail(h, JPET_ERR_ARGUMENT, "bad responses");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  return translate(h, d, n);
}

int jpet_hybrid_set_responses(jpet_hybrid_t* h, const jpet_hybrid_response* r, int64_t n) {
  if (!h) return fail(nullptr, JPET_ERR_ARGUMENT, "handle is NULL");
  if (n < 0 || (n > 0 && !r)) return fail(h, JPET_ERR_ARGUMENT, "bad responses");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  HYB_CUDA(h, h->resp.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  if (n > 0)
    HYB_CUDA(h, cudaMemcpyAsync(h->resp.p, r, n * sizeof(jpet_hybrid_response),
                                cudaMemcpyHostToDevice, h->stream),
             "upload");
  return translate(h, h->resp.p, n);
}

int jpet_hybrid_set_frame_events(jpet_hybrid_t* h, const jpet_hybrid_frame_event* e, int64_t n) {
  if (!h) return fail(nullptr, JPET_ERR_ARGUMENT, "handle is NULL");
  if (n < 0 || (n > 0 && !e)) return fail(h, JPET_ERR_ARGUMENT, "bad frame events");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  HYB_CUDA(h, h->ev.alloc(std::max<int64_t>(n, 1)), "cudaMalloc");
  if (n > 0)
    HYB_CUDA(h, cudaMemcpyAsync(h->ev.p, e, n * sizeof(jpet_hybrid_frame_event),
                                cudaMemcpyHostToDevice, h->stream),
             "upload");
  return finish_events(h, n);
}

int jpet_hybrid_get_frame_events(jpet_hybrid_t* h, jpet_hybrid_frame_event* out, int64_t* n) {
  if (!h || !n) return fail(h, JPET_ERR_ARGUMENT, "NULL argument");
  *n = h->n_events;
  if (!out || h->n_events == 0) return JPET_OK;
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  HYB_CUDA(h, cudaMemcpyAsync(out, h->ev.p, h->n_events * sizeof(jpet_hybrid_frame_event),
                              cudaMemcpyDeviceToHost, h->stream),
           "download");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return JPET_OK;
}

int jpet_hybrid_set_image(jpet_hybrid_t* h, const float* rho) {
  if (!h || !rho) return fail(h, JPET_ERR_ARGUMENT, "NULL argument");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const int64_t n_px = static_cast<int64_t>(h->c.n_columns) * h->c.n_rows;
  const int64_t n_vox = n_px * h->c.n_planes;
  HYB_CUDA(h, h->stage.alloc(n_vox), "cudaMalloc");
  HYB_CUDA(h, cudaMemcpyAsync(h->stage.p, rho, n_vox * sizeof(float), cudaMemcpyHostToDevice,
                              h->stream),
           "upload");
  to_device_layout<<<grid_for(h, n_vox), 256, 0, h->stream>>>(h->stage.p, h->rho.p, n_px,
                                                              h->c.n_planes, h->c.pitch);
  HYB_CUDA(h, cudaGetLastError(), "layout");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return JPET_OK;
}

int jpet_hybrid_get_image(jpet_hybrid_t* h, float* rho) {
  if (!h || !rho) return fail(h, JPET_ERR_ARGUMENT, "NULL argument");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const int64_t n_px = static_cast<int64_t>(h->c.n_columns) * h->c.n_rows;
  const int64_t n_vox = n_px * h->c.n_planes;
  HYB_CUDA(h, h->stage.alloc(n_vox), "cudaMalloc");
  to_reference_layout<<<grid_for(h, n_vox), 256, 0, h->stream>>>(h->rho.p, h->stage.p, n_px,
                                                                 h->c.n_planes, h->c.pitch);
  HYB_CUDA(h, cudaGetLastError(), "layout");
  HYB_CUDA(h, cudaMemcpyAsync(rho, h->stage.p, n_vox * sizeof(float), cudaMemcpyDeviceToHost,
                              h->stream),
           "download");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return JPET_OK;
}

int jpet_hybrid_get_sensitivity(jpet_hybrid_t* h, float* sens) {
  if (!h || !sens) return fail(h, JPET_ERR_ARGUMENT, "NULL argument");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const int64_t n_px = static_cast<int64_t>(h->c.n_columns) * h->c.n_rows;
  HYB_CUDA(h, cudaMemcpyAsync(sens, h->sens.p, n_px * h->c.sens_depth * sizeof(float),
                              cudaMemcpyDeviceToHost, h->stream),
           "download");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return JPET_OK;
}

int jpet_hybrid_get_weights(jpet_hybrid_t* h, float* w) {
  if (!h || (!w && h->c.n_infos > 0)) return fail(h, JPET_ERR_ARGUMENT, "NULL argument");
  if (h->c.n_infos == 0) return JPET_OK;
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  HYB_CUDA(h, cudaMemcpyAsync(w, h->w.p, h->c.n_infos * h->c.n_planes_half * sizeof(float),
                              cudaMemcpyDeviceToHost, h->stream),
           "download");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return JPET_OK;
}

int jpet_hybrid_iterate(jpet_hybrid_t* h, int n) {
  if (!h) return fail(nullptr, JPET_ERR_ARGUMENT, "handle is NULL");
  if (n < 0) return fail(h, JPET_ERR_ARGUMENT, "negative iteration count");
  return iterate(h, n, n);
}

int jpet_hybrid_get_counters(jpet_hybrid_t* h, jpet_hybrid_counters* c) {
  if (!h || !c) return fail(h, JPET_ERR_ARGUMENT, "NULL argument");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  unsigned long long pos = 0;
  HYB_CUDA(h, cudaMemcpyAsync(&pos, h->counters.p + 2, sizeof pos, cudaMemcpyDeviceToHost,
                              h->stream),
           "download");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  c->used_events = h->n_events;
  c->used_pixels = h->used_pixels;
  c->used_voxels = h->used_voxels;
  c->contributing = static_cast<int64_t>(pos);
  return JPET_OK;
}

int jpet_hybrid_synchronize(jpet_hybrid_t* h) {
  if (!h) return fail(nullptr, JPET_ERR_ARGUMENT, "handle is NULL");
  HYB_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  HYB_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return JPET_OK;
}

int jpet_hybrid_run(const jpet_hybrid_geom* geom, const float* sensitivity,
                    const jpet_hybrid_frame_event* events, int64_t n_events, float* rho,
                    int n_blocks, int n_iterations_in_block, int start_iteration,
                    jpet_hybrid_output_fn output, jpet_strip_progress_fn progress, void* user,
                    int device, char* device_name, size_t device_name_len) {
  if (!rho || !sensitivity || n_blocks < 0 || n_iterations_in_block < 0)
    return fail(nullptr, JPET_ERR_ARGUMENT, "bad argument");
  jpet_hybrid_opts o;
  jpet_hybrid_default_opts(&o);
  o.device = device;
  o.weights = JPET_HYBRID_WEIGHTS_NORMALIZED;
  // a multi-plane geometry comes with its 3D sensitivity (depth n_planes_half)
  o.sensitivity = (geom && geom->n_planes_half > 1) ? JPET_HYBRID_SENSITIVITY_GIVEN_3D
                                                    : JPET_HYBRID_SENSITIVITY_GIVEN;
  o.sensitivity_map = sensitivity;
  jpet_hybrid_t* h = nullptr;
  int rc = jpet_hybrid_create(geom, &o, &h);
  if (rc != JPET_OK) return rc;
  if (device_name && device_name_len > 0) {
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) == cudaSuccess) {
      std::snprintf(device_name, device_name_len, "%s", prop.name);
    } else {
      device_name[0] = 0;
    }
  }
  auto done = [&](int code) {
    if (code != JPET_OK) g_hybrid_error = h->last_error;
    jpet_hybrid_destroy(h);
    return code;
  };
  if ((rc = jpet_hybrid_set_frame_events(h, events, n_events)) != JPET_OK) return done(rc);
  if ((rc = jpet_hybrid_set_image(h, rho)) != JPET_OK) return done(rc);
  // the reference's iteration and output schedule (cuda/reconstruction.cu:113-186)
  for (int block = 0; block < n_blocks; ++block) {
    for (int i = 0; i < n_iterations_in_block; ++i) {
      const int iteration = block * n_iterations_in_block + i;
      if (iteration < start_iteration) continue;
      if (progress) progress(iteration, 0, user);
      const int64_t all = static_cast<int64_t>(n_blocks) * n_iterations_in_block;
      if ((rc = iterate(h, 1, all - iteration)) != JPET_OK) return done(rc);
      if ((rc = jpet_hybrid_synchronize(h)) != JPET_OK) return done(rc);
      if (progress) progress(iteration, 1, user);
      if (!block && i < n_iterations_in_block - 1 &&
          (i < 5 || i == 9 || i == 14 || i == 19 || i == 29 || i == 49 || i == 99)) {
        if ((rc = jpet_hybrid_get_image(h, rho)) != JPET_OK) return done(rc);
        if (output) output(i + 1, rho, user);
      }
    }
    const int iteration = (block + 1) * n_iterations_in_block;
    if (iteration <= start_iteration) continue;
    if ((rc = jpet_hybrid_get_image(h, rho)) != JPET_OK) return done(rc);
    if (output) output(iteration, rho, user);
  }
  if (progress) progress(n_blocks * n_iterations_in_block, 0, user);
  if ((rc = jpet_hybrid_get_image(h, rho)) != JPET_OK) return done(rc);
  return done(JPET_OK);
}

}  // extern "C"
