// Set-up passes of the batch-union iteration (strip_union.cuh): the greedy
// batches of similar events, their row words and the events' records; the
// choice of the batch shape; the launches of the iteration.
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "strip_union.cuh"

namespace jpet {
namespace {

// Greedy batch formation, one warp per chunk: events in sorted order join the
// current batch while the union stays inside the shape's max_rows x max_cols and
// the batch has fewer than max_e events.  KR: window rows tracked per lane (a
// batch's rows lie in the window's first 32 KR; taller windows hold taller boxes
// than any shape takes).  Batch words go to batches[c.start ...]; events
// that fit no batch rectangle alone are listed from the end of the chunk's
// range (batches[c.start + c.count - 1 - k]).
template <int KR>
__global__ void __launch_bounds__(256) union_batches_kernel(Chunk* __restrict__ chunks,
                                                            int32_t n_chunks, int32_t max_e, int32_t max_rows,
                                                            int32_t max_cols,
                                                            const short4* __restrict__ ev_box,
                                                            const uint16_t* __restrict__ rows,
                                                            int32_t stride,
                                                            uint32_t* __restrict__ batches,
                                                            uint16_t* __restrict__ urows) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int n_warps = (gridDim.x * blockDim.x) >> 5;
  for (int ci = wid; ci < n_chunks; ci += n_warps) {
    const Chunk c = chunks[ci];
    const int ox = c.ox & ~1, oy = c.oy;
    int ulo[KR], uhi[KR];
    int u0 = INT_MAX, u1 = INT_MIN, cnt = 0, bstart = 0, nb = 0, nx = 0;
    auto reset = [&]() {
      cnt = 0;
      u0 = INT_MAX;
      u1 = INT_MIN;
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        ulo[k] = INT_MAX;
        uhi[k] = INT_MIN;
      }
    };
    auto emit = [&]() {
      if (cnt > 0) {
        if (lane == 0) batches[c.start + nb] = ubatch_word(bstart, cnt, u1 - u0, u0);
        // union row words of the batch (0: no pixel)
        uint16_t* ub = urows + static_cast<size_t>(c.start + nb) * max_rows;
        for (int r = lane; r < max_rows; r += 32) ub[r] = 0;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < KR; ++k) {
          const int r = lane + 32 * k - u0;
          if (r >= 0 && r < max_rows && ulo[k] != INT_MAX) {
            const int u = ulo[k] & ~1;
            ub[r] = urow_word(u, uhi[k] - u);
          }
        }
        ++nb;
      }
      reset();
    };
    reset();
    for (int i = 0; i < c.count; ++i) {
      const short4 b = ev_box[c.start + i];
      const int r0 = b.y - oy, n = b.w - b.y, bx = b.x - ox;
      const uint16_t* rt = rows + static_cast<size_t>(c.start + i) * stride;
      int f[KR], w[KR];
      bool alone = n <= max_rows && r0 >= 0 && r0 + n <= 32 * KR;
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        const int ri = lane + 32 * k - r0;
        const bool v = ri >= 0 && ri < n && ri < max_rows;
        const uint32_t e = v ? rt[v ? ri : 0] : 0u;
        w[k] = static_cast<int>(e >> 8);
        f[k] = bx + static_cast<int>(e & 255u);
        if (w[k] > 0 && f[k] + w[k] - (f[k] & ~1) > max_cols) alone = false;
      }
      alone = __all_sync(kFull, alone);
      if (!alone) {
        emit();  // a batch is a contiguous run of events: close the open one first
        if (lane == 0) batches[c.start + c.count - 1 - nx] = static_cast<uint32_t>(i);
        ++nx;
        continue;
      }
      // would the event join the current batch?
      bool join = cnt > 0 && cnt < max_e && max(u1, r0 + n) - min(u0, r0) <= max_rows;
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        if (w[k] > 0) {
          const int lo = min(ulo[k], f[k]), hi = max(uhi[k], f[k] + w[k]);
          if (hi - (lo & ~1) > max_cols) join = false;
        }
      }
      join = __all_sync(kFull, join);
      if (!join) {
        emit();
        bstart = i;
      }
      ++cnt;
      u0 = min(u0, r0);
      u1 = max(u1, r0 + n);
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        if (w[k] > 0) {
          ulo[k] = min(ulo[k], f[k]);
          uhi[k] = max(uhi[k], f[k] + w[k]);
        }
      }
    }
    emit();
    if (lane == 0) {
      chunks[ci].n_batches = nb;
      chunks[ci].n_exact = nx;
    }
  }
}

// Records of the events' rows (strip_union.cuh), one CTA per chunk, a warp per
// batch and its lanes along the union rows.  The arithmetic of row_coeff_kernel:
// K / K_ref = 2^(p + q jc + c jc^2) with jc counted from the union row's middle.
// Writes 16 bytes per event and row of its batch's union, once per event set:
// 1e6 events at 2 mm 0.33 ms, as much as the on-chip records cost three
// iterations, and union_batches_kernel, which no longer writes the events'
// intervals, 0.74 -> 0.51 ms.
__global__ void __launch_bounds__(256) union_records_kernel(
    DevGeom g, FastConst fc, Tiling t, const Chunk* __restrict__ chunks, int32_t max_rows,
    bool halves, const float4* __restrict__ ev_geom, const short4* __restrict__ ev_box,
    const uint16_t* __restrict__ rows, const uint32_t* __restrict__ batches,
    const uint16_t* __restrict__ urows, float4* __restrict__ records) {
  const Chunk c = chunks[blockIdx.x];
  const int lane = threadIdx.x & 31;
  const int ox = c.ox & ~1, oy = c.oy;
  for (int b = threadIdx.x >> 5; b < c.n_batches; b += blockDim.x >> 5) {
    const uint32_t bw = batches[c.start + b];
    const int first = ub_first(bw), cnt = ub_cnt(bw), n_rows = ub_rows(bw), u0 = ub_u0(bw);
    const uint16_t* ub = urows + static_cast<size_t>(c.start + b) * max_rows;
    for (int j = 0; j < cnt; ++j) {
      const float4 ev = ev_geom[c.start + first + j];
      const short4 box = ev_box[c.start + first + j];
      const uint16_t* rt = rows + static_cast<size_t>(c.start + first + j) * t.row_stride;
      float4* rec = records + static_cast<size_t>(c.rec + first + j) * max_rows;
      const float y = ev.y, tn = ev.z, sec2 = ev.w * ev.w;
      const float ky = fc.kdl * sec2;
      const float P = fc.two_r2 * sec2 * sec2 * g.ipz;
      const float Q = 2.0f * sec2 * sec2 * g.ipz + 4.0f * sec2 * tn * tn * g.ipd;
      const float lref = 0.5f * lg2_approx(fmaf(Q, y * y, P));
      const float z0 = g.tl_z_half_w - ev.x;
      for (int r = lane; r < n_rows; r += 32) {
        const uint32_t ur = ub[r];
        const int u = static_cast<int>(ur & 511u);
        const float py = g.tl_y_half_h - static_cast<float>(oy + u0 + r) * g.pixel_height;
        const float colm = static_cast<float>(ox + u + u_centre(static_cast<int>(ur >> 9)));
        const float dy = py - y;
        const float lf = lref - 0.5f * lg2_approx(fmaf(Q, py * py, P));
        const float ua = fmaf(colm, g.pixel_width, z0 - dy * tn);
        const float p = fmaf(fc.kz * ua, ua, fmaf(ky * dy, dy, lf));
        const float q = 2.0f * fc.kz * g.pixel_width * ua;
        // the event's interval of the row as a mask of the union row's columns
        const int ri = oy + u0 + r - box.y;
        const uint32_t e = ri >= 0 && ri < box.w - box.y ? rt[ri] : 0u;
        const int w = static_cast<int>(e >> 8);
        unsigned long long m = 0;
        if (w > 0)
          m = (~0ull >> (64 - w)) << (box.x - ox + static_cast<int>(e & 255u) - u);
        const uint32_t lo = u_lane_mask(static_cast<uint32_t>(m));
        float4 v = make_float4(p, q, ex2_approx(8.0f * q), __uint_as_float(lo));
        if (halves) {  // columns 32..39: two more bits for each lane
          const uint32_t hi = static_cast<uint32_t>(m >> 32);
          v.z = __uint_as_float((lo & 255u) | ((hi & 3u) << 8) | ((lo & 0xFF00u) << 8) |
                                ((hi & 0xCu) << 22));
          v.w = __uint_as_float(((lo >> 16) & 255u) | ((hi & 0x30u) << 4) |
                                ((lo >> 24) << 16) | ((hi & 0xC0u) << 18));
        }
        rec[r] = v;
      }
    }
  }
}

}  // namespace

const UnionOps& union_ops(int shape) {
  switch (shape) {
    case kUnion64x32n4: return union_ops_64x32n4();
    case kUnion32x16: return union_ops_32x16();
    case kUnion32x32: return union_ops_32x32();
    case kUnion96x40: return union_ops_96x40();
    case kUnion64x16: return union_ops_64x16();
    default: return union_ops_64x32();
  }
}

size_t union_smem_bytes(const Tiling& t, int precision) {
  return union_ops(t.union_shape).smem(t, precision);
}

cudaError_t union_prepare_kernel(const Tiling& t, int precision) {
  return union_ops(t.union_shape).prepare(precision);
}

size_t union_row_words(const Tiling& t) { return union_ops(t.union_shape).rows; }

cudaError_t launch_union_batches(const Tiling& t, Chunk* chunks, int32_t n_chunks,
                                 const short4* ev_box, const uint16_t* rows, uint32_t* batches,
                                 uint16_t* urows, cudaStream_t s) {
  if (n_chunks <= 0) return cudaSuccess;
  const UnionOps& ops = union_ops(t.union_shape);
  int blocks = (n_chunks + 7) / 8;
  if (blocks > 152 * 16) blocks = 152 * 16;
  auto* k = t.win_h <= 128 ? union_batches_kernel<4> : union_batches_kernel<8>;
  k<<<blocks, 256, 0, s>>>(chunks, n_chunks, ops.events, ops.rows, ops.cols, ev_box, rows,
                           t.row_stride, batches, urows);
  return cudaGetLastError();
}

cudaError_t launch_union_records(const DevGeom& g, const FastConst& fc, const Tiling& t,
                                 const Chunk* chunks, int32_t n_chunks, const float4* ev_geom,
                                 const short4* ev_box, const uint16_t* rows,
                                 const uint32_t* batches, const uint16_t* urows, float4* records,
                                 cudaStream_t s) {
  if (n_chunks <= 0) return cudaSuccess;
  const UnionOps& ops = union_ops(t.union_shape);
  union_records_kernel<<<n_chunks, 256, 0, s>>>(g, fc, t, chunks, ops.rows, ops.cols > 32,
                                                ev_geom, ev_box, rows, batches, urows, records);
  return cudaGetLastError();
}

cudaError_t launch_iterate_union(const DevGeom& g, const FastConst& fc, const Tiling& t,
                                 const Chunk* chunks, int32_t n_chunks, const float4* ev_geom,
                                 const short4* ev_box, const float4* records,
                                 const uint16_t* urows, const uint32_t* batches, const float* rho,
                                 float* out, AuxImage aux, DevCounters* counters, int precision,
                                 uint32_t seed, cudaStream_t s) {
  if (n_chunks <= 0) return cudaSuccess;
  if (t.chunk_events > kUMaxChunk ||
      (precision == kPrecisionFixed && t.chunk_events > kUMaxChunkFixed))
    return cudaErrorInvalidValue;
  return union_ops(t.union_shape)
      .launch(g, fc, t, chunks, n_chunks, ev_geom, ev_box, records, urows, batches, rho, out, aux,
              counters, precision, seed, s);
}

}  // namespace jpet
