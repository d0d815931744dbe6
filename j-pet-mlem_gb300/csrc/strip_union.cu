// Set-up passes of the batch-union iteration (strip_union.cuh): per-event
// constants, the greedy batches of similar events and their row words; the
// choice of the batch shape; the launches of the iteration.
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>

#include "strip_union.cuh"

namespace jpet {
namespace {

// Per-event constants of the sorted events (the arithmetic of row_coeff_kernel).
__global__ void union_events_kernel(DevGeom g, FastConst fc, Tiling t, int32_t n,
                                    const float4* __restrict__ ev_geom,
                                    const short4* __restrict__ ev_box, UEvConst* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 ev = ev_geom[i];
  const short4 b = ev_box[i];
  const float y = ev.y, tn = ev.z, sec = ev.w;
  const float sec2 = sec * sec;
  UEvConst c;
  c.y = y;
  c.tn = tn;
  c.ky = fc.kdl * sec2;
  c.P = fc.two_r2 * sec2 * sec2 * g.ipz;
  c.Q = 2.0f * sec2 * sec2 * g.ipz + 4.0f * sec2 * tn * tn * g.ipd;
  c.lref = 0.5f * lg2_approx(fmaf(c.Q, y * y, c.P));
  c.ub = g.tl_z_half_w - ev.x;
  const int oy = (b.y / t.tile_h) * t.tile_h;
  const int ox = ((b.x / t.tile_w) * t.tile_w) & ~1;
  const int rows = min(b.w - b.y, 255);
  c.box = static_cast<uint32_t>(b.y - oy) | (static_cast<uint32_t>(rows) << 8) |
          (static_cast<uint32_t>(b.x - ox) << 16);
  out[i] = c;
}

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
                                                            uint16_t* __restrict__ urows,
                                                            uint16_t* __restrict__ erows) {
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
        // union row words of the batch, and each event's intervals relative to
        // its union rows (lane: window rows lane + 32 k; the arrays start zeroed)
        uint16_t* ub = urows + static_cast<size_t>(c.start + nb) * max_rows;
#pragma unroll
        for (int k = 0; k < KR; ++k) {
          const int wr = lane + 32 * k, r = wr - u0;
          if (r >= 0 && r < max_rows && ulo[k] != INT_MAX) {
            const int u = ulo[k] & ~1;
            ub[r] = urow_word(u, uhi[k] - u);
            for (int i = bstart; i < bstart + cnt; ++i) {
              const short4 b = ev_box[c.start + i];
              const int ri = wr - (b.y - oy);
              if (ri < 0 || ri >= b.w - b.y) continue;
              const uint32_t e = rows[static_cast<size_t>(c.start + i) * stride + ri];
              const int w = static_cast<int>(e >> 8);
              if (w == 0) continue;
              const int f = (b.x - ox) + static_cast<int>(e & 255u);
              erows[static_cast<size_t>(c.start + i) * max_rows + r] =
                  static_cast<uint16_t>((f - u) | (w << 8));
            }
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

size_t union_event_bytes() { return sizeof(UEvConst); }

size_t union_smem_bytes(const Tiling& t, int precision) {
  return union_ops(t.union_shape).smem(t, precision);
}

cudaError_t union_prepare_kernel(const Tiling& t, int precision) {
  return union_ops(t.union_shape).prepare(precision);
}

size_t union_row_words(const Tiling& t) { return union_ops(t.union_shape).rows; }

cudaError_t launch_union_setup(const DevGeom& g, const FastConst& fc, const Tiling& t,
                               Chunk* chunks, int32_t n_chunks, int32_t n_events,
                               const float4* ev_geom, const short4* ev_box, const uint16_t* rows,
                               void* ev_const, uint32_t* batches, uint16_t* urows,
                               uint16_t* erows, cudaStream_t s) {
  if (n_events <= 0) return cudaSuccess;
  const UnionOps& ops = union_ops(t.union_shape);
  union_events_kernel<<<(n_events + 255) / 256, 256, 0, s>>>(
      g, fc, t, n_events, ev_geom, ev_box, static_cast<UEvConst*>(ev_const));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || n_chunks <= 0) return e;
  const size_t words = static_cast<size_t>(n_events) * ops.rows * sizeof(uint16_t);
  e = cudaMemsetAsync(urows, 0, words, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(erows, 0, words, s);
  if (e != cudaSuccess) return e;
  int blocks = (n_chunks + 7) / 8;
  if (blocks > 152 * 16) blocks = 152 * 16;
  if (t.win_h <= 128)
    union_batches_kernel<4><<<blocks, 256, 0, s>>>(chunks, n_chunks, ops.events, ops.rows,
                                                   ops.cols, ev_box, rows, t.row_stride, batches,
                                                   urows, erows);
  else
    union_batches_kernel<8><<<blocks, 256, 0, s>>>(chunks, n_chunks, ops.events, ops.rows,
                                                   ops.cols, ev_box, rows, t.row_stride, batches,
                                                   urows, erows);
  return cudaGetLastError();
}

cudaError_t launch_iterate_union(const DevGeom& g, const FastConst& fc, const Tiling& t,
                                 const Chunk* chunks, int32_t n_chunks, const float4* ev_geom,
                                 const short4* ev_box, const void* ev_const,
                                 const uint16_t* erows, const uint16_t* urows,
                                 const uint32_t* batches, const float* rho, float* out,
                                 AuxImage aux, DevCounters* counters, int precision,
                                 uint32_t seed, cudaStream_t s) {
  if (n_chunks <= 0) return cudaSuccess;
  if (t.chunk_events > kUMaxChunk ||
      (precision == kPrecisionFixed && t.chunk_events > kUMaxChunkFixed))
    return cudaErrorInvalidValue;
  return union_ops(t.union_shape)
      .launch(g, fc, t, chunks, n_chunks, ev_geom, ev_box, ev_const, erows, urows, batches, rho,
              out, aux, counters, precision, seed, s);
}

}  // namespace jpet
