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
// range (batches[c.start + c.count - 1 - k]).  The decisions are a serial chain,
// so the loads of the events to come run ahead of it; 1e6 events at 2 mm:
// 0.51 -> 0.33 ms.
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
    // Two groups of loads run ahead of the (serial) decisions: the next events'
    // row words, and the boxes of the events after those, which the row words'
    // addresses need
    constexpr int kAhead = 4;
    short4 box[kAhead], box_next[kAhead];
    uint32_t word[kAhead][KR];
    auto load_boxes = [&](int i0, short4(&bx)[kAhead]) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        bx[q] = i0 + q < c.count ? ev_box[c.start + i0 + q] : make_short4(0, 0, 0, 0);
    };
    auto load_words = [&](int i0, const short4(&bx)[kAhead]) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int r0 = bx[q].y - oy, n = min(bx[q].w - bx[q].y, max_rows);
        const uint16_t* rt = rows + static_cast<size_t>(c.start + i0 + q) * stride;
#pragma unroll
        for (int k = 0; k < KR; ++k) {
          const int ri = lane + 32 * k - r0;
          word[q][k] = ri >= 0 && ri < n ? rt[ri] : 0u;
        }
      }
    };
    load_boxes(0, box);
    load_words(0, box);
    load_boxes(kAhead, box_next);
    for (int i0 = 0; i0 < c.count; i0 += kAhead) {
      short4 cur[kAhead];
      uint32_t e[kAhead][KR];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        cur[q] = box[q];
        box[q] = box_next[q];
#pragma unroll
        for (int k = 0; k < KR; ++k) e[q][k] = word[q][k];
      }
      load_words(i0 + kAhead, box);
      load_boxes(i0 + 2 * kAhead, box_next);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (i0 + q >= c.count) break;
        const int r0 = cur[q].y - oy, n = cur[q].w - cur[q].y, bx = cur[q].x - ox;
        bool alone = n <= max_rows && r0 >= 0 && r0 + n <= 32 * KR;
        // would the event join the current batch?
        bool join = cnt > 0 && cnt < max_e && max(u1, r0 + n) - min(u0, r0) <= max_rows;
        int f[KR], w[KR];
#pragma unroll
        for (int k = 0; k < KR; ++k) {
          w[k] = static_cast<int>(e[q][k] >> 8);
          f[k] = bx + static_cast<int>(e[q][k] & 255u);
          if (w[k] > 0) {
            if (f[k] + w[k] - (f[k] & ~1) > max_cols) alone = false;
            if (max(uhi[k], f[k] + w[k]) - (min(ulo[k], f[k]) & ~1) > max_cols) join = false;
          }
        }
        alone = __all_sync(kFull, alone);
        join = __all_sync(kFull, join) && alone;
        if (!join) {
          emit();  // a batch is a contiguous run of events: close the open one first
          bstart = i0 + q;
        }
        if (!alone) {
          if (lane == 0)
            batches[c.start + c.count - 1 - nx] = static_cast<uint32_t>(i0 + q);
          ++nx;
          continue;
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
// Writes 16 bytes per event and row of its batch's union, once per event set.
// Bound by instruction issue: an event's constants are computed once (lane j for
// event j, handed on in shared memory) and what depends on the row alone is
// outside the loop over the events: 1e6 events at 2 mm 0.33 -> 0.24 ms.
struct URecordEvent {
  float y, tn, z0, ky;
  float P, Q, lref, pad;
  int32_t row0, rows, col0, table;  // box relative to the window; event's place in the row table
};

template <bool HALVES>
__global__ void __launch_bounds__(256) union_records_kernel(
    DevGeom g, FastConst fc, Tiling t, const Chunk* __restrict__ chunks, int32_t max_rows,
    const float4* __restrict__ ev_geom, const short4* __restrict__ ev_box,
    const uint16_t* __restrict__ rows, const uint32_t* __restrict__ batches,
    const uint16_t* __restrict__ urows, float4* __restrict__ records) {
  constexpr int kMaxEvents = 16;
  __shared__ __align__(16) URecordEvent events[8][kMaxEvents];
  const Chunk c = chunks[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ox = c.ox & ~1, oy = c.oy;
  for (int b = warp; b < c.n_batches; b += blockDim.x >> 5) {
    const uint32_t bw = batches[c.start + b];
    const int first = ub_first(bw), cnt = ub_cnt(bw), n_rows = ub_rows(bw), u0 = ub_u0(bw);
    if (lane < cnt) {  // lane j: the constants of event j (at most kMaxEvents in every shape)
      const float4 ev = ev_geom[c.start + first + lane];
      const short4 box = ev_box[c.start + first + lane];
      URecordEvent e;
      const float sec2 = ev.w * ev.w;
      e.y = ev.y;
      e.tn = ev.z;
      e.z0 = g.tl_z_half_w - ev.x;
      e.ky = fc.kdl * sec2;
      e.P = fc.two_r2 * sec2 * sec2 * g.ipz;
      e.Q = 2.0f * sec2 * sec2 * g.ipz + 4.0f * sec2 * ev.z * ev.z * g.ipd;
      e.lref = 0.5f * lg2_approx(fmaf(e.Q, ev.y * ev.y, e.P));
      e.pad = 0.0f;
      e.row0 = box.y - oy - u0;
      e.rows = box.w - box.y;
      e.col0 = box.x - ox;
      e.table = c.start + first + lane;
      events[warp][lane] = e;
    }
    __syncwarp();
    float4* rec = records + static_cast<size_t>(c.rec + first) * max_rows;
    for (int r = lane; r < n_rows; r += 32) {
      const uint32_t ur = urows[static_cast<size_t>(c.start + b) * max_rows + r];
      const int u = static_cast<int>(ur & 511u);
      const float py = g.tl_y_half_h - static_cast<float>(oy + u0 + r) * g.pixel_height;
      const float colm = static_cast<float>(ox + u + u_centre(static_cast<int>(ur >> 9)));
      const float py2 = py * py;
#pragma unroll 4
      for (int j = 0; j < cnt; ++j) {
        const URecordEvent e = events[warp][j];
        const float dy = py - e.y;
        const float lf = e.lref - 0.5f * lg2_approx(fmaf(e.Q, py2, e.P));
        const float ua = fmaf(colm, g.pixel_width, e.z0 - dy * e.tn);
        const float p = fmaf(fc.kz * ua, ua, fmaf(e.ky * dy, dy, lf));
        const float q = 2.0f * fc.kz * g.pixel_width * ua;
        // the event's interval of the row as a mask of the union row's columns
        const int ri = r - e.row0;
        const uint32_t iv = ri >= 0 && ri < e.rows
                                ? rows[static_cast<size_t>(e.table) * t.row_stride + ri]
                                : 0u;
        const int w = static_cast<int>(iv >> 8);
        const int shift = w > 0 ? e.col0 + static_cast<int>(iv & 255u) - u : 0;
        float4 v = make_float4(p, q, 0.0f, 0.0f);
        if constexpr (HALVES) {
          const unsigned long long m = (w > 0 ? ~0ull >> (64 - w) : 0ull) << shift;
          const uint32_t lo = u_lane_mask(static_cast<uint32_t>(m));
          const uint32_t hi = static_cast<uint32_t>(m >> 32);  // columns 32..39: two bits a lane
          v.z = __uint_as_float((lo & 255u) | ((hi & 3u) << 8) | ((lo & 0xFF00u) << 8) |
                                ((hi & 0xCu) << 22));
          v.w = __uint_as_float(((lo >> 16) & 255u) | ((hi & 0x30u) << 4) |
                                ((lo >> 24) << 16) | ((hi & 0xC0u) << 18));
        } else {
          const uint32_t m = __funnelshift_rc(0xFFFFFFFFu, 0u, static_cast<uint32_t>(32 - w));
          v.z = ex2_approx(8.0f * q);
          v.w = __uint_as_float(u_lane_mask(m << shift));
        }
        rec[static_cast<size_t>(j) * max_rows + r] = v;
      }
    }
    __syncwarp();  // the next batch's constants take this batch's place
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
  auto* k = ops.cols > 32 ? union_records_kernel<true> : union_records_kernel<false>;
  k<<<n_chunks, 256, 0, s>>>(g, fc, t, chunks, ops.rows, ev_geom, ev_box, rows, batches, urows,
                             records);
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
