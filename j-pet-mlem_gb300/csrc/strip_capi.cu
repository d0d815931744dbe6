// C ABI of the GB300 strip-PET MLEM (include/jpet_strip.h): handle management,
// device memory, event preparation and binning, and the iteration loop.
//
// Replaces GPU::Reconstruction::run (src/2d/strip/cuda/reconstruction.cu:31-113)
// and its helpers (cuda/gpu_events_soa.h:9-51, util/cuda/memory.h:51-327): every
// CUDA failure becomes a status code plus a message instead of the reference's
// abort() (util/cuda/debug.h:17-27).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "../../include/jpet_strip.h"
#include "strip_internal.h"

using namespace jpet;

namespace {

thread_local std::string g_create_error = "no error";

}  // namespace

namespace jpet {
void set_call_error(const std::string& msg) { g_create_error = msg; }
}  // namespace jpet

namespace {

template <typename T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  bool own = true;  // else a part of a block (carve)
  cudaError_t alloc(size_t count) {
    if (count <= n && p && own) return cudaSuccess;
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
    if (p && own) cudaFree(p);
    p = nullptr;
    n = 0;
    own = true;
  }
};

// Several buffers as parts of one block, so that an event set costs a few
// cudaMalloc / cudaFree calls and not twenty (65 to 250 us a pair): layout names
// the buffers and their sizes, once to add them up and once to place them.
struct Carver {
  unsigned char* base;
  size_t used;
  template <class T>
  void operator()(DevBuf<T>& b, size_t count) {
    b.release();
    if (base) {
      b.p = reinterpret_cast<T*>(base + used);
      b.n = count;
      b.own = false;
    }
    used += (count * sizeof(T) + 255) & ~static_cast<size_t>(255);
  }
};
template <class F>
cudaError_t carve(DevBuf<unsigned char>& block, F layout) {
  Carver size{nullptr, 0};
  layout(size);
  const cudaError_t e = block.alloc(size.used);
  if (e != cudaSuccess) return e;
  Carver place{block.p, 0};
  layout(place);
  return cudaSuccess;
}

}  // namespace

struct jpet_strip {
  jpet_strip_geom geom_in{};
  jpet_strip_opts opts{};
  DevGeom g{};
  Tiling tiling{};
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t own_stream = nullptr;
  std::string last_error = "no error";

  DevBuf<float> rho, out, sens_point, sens_pixel;
  DevBuf<float> out_lo;              // compensation image of the compensated modes
  DevBuf<unsigned long long> out_q;  // 64-bit fixed-point image of the FIXED mode
  DevBuf<double> out_sum;            // image sums of the exact kernel (EXACT, GPU-reference)
  DevBuf<float> raw;                 // staging for uploaded events (kept for the next upload)
  DevBuf<float4> ev_geom, sorted_geom, over_geom;
  DevBuf<short4> ev_box, sorted_box, over_box;
  DevBuf<int32_t> tile_count, hist, small;
  DevBuf<unsigned char> scratch, set_block;  // of the set-up; of the prepared events
  DevBuf<Chunk> chunks;
  DevBuf<uint16_t> row_table;
  DevBuf<float2> row_pq;     // per-row exponent coefficients of the row-owned kernel
  DevBuf<uint32_t> row_pk;   // per-row packed window offset / parity / width
  DevBuf<uint32_t> ev_pk;    // per-event packed window row / box rows / fits
  DevBuf<uint64_t> sort_keys;     // set-up sort: keys (input, output)
  DevBuf<int32_t> sort_idx;       // set-up sort: event indices (input, output)
  DevBuf<unsigned char> sort_tmp; // set-up sort: radix-sort scratch
  DevBuf<uint32_t> batches;       // batch-union kernel: batch words per chunk
  DevBuf<uint16_t> union_rows;    // batch-union kernel: union row words per batch
  DevBuf<float4> records;         // batch-union kernel: event row records
  // batch-union kernel: the chunks whose records the workspace holds at a time
  // (first, count); with one part the records are written once
  std::vector<std::pair<int32_t, int32_t>> parts;
  FastConst fc{};
  bool use_fast = false;
  bool use_union = false;
  bool counters_valid = false;
  unsigned long long table_kernel_calls = 0;
  DevBuf<unsigned long long> box_pixels;
  DevBuf<double> nll_acc;            // loss, d/dsigma_z, d/dsigma_dl
  DevBuf<double> nll_parts;          // partial gradient images
  DevBuf<DevCounters> counters;

  int64_t n_events = 0;
  int32_t n_sorted = 0;
  int32_t n_oversize = 0;
  int32_t n_chunks = 0;
  int32_t n_tiles_nonempty = 0;
  int32_t beside = 1;  // handles that iterate together (a batch's instances)
  unsigned long long total_box_pixels = 0;
  bool events_ready = false;
  int64_t iterations_done = 0;
  uint64_t generation = 0;  // event sets prepared: what a captured graph of this handle was made for

  int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    last_error = buf;
    return code;
  }
  int cuda_fail(cudaError_t e, const char* what) {
    return fail(JPET_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
  }
};

#define JPET_CUDA(h, expr, what)                 \
  do {                                           \
    cudaError_t _e = (expr);                     \
    if (_e != cudaSuccess) return (h)->cuda_fail(_e, what); \
  } while (0)

namespace {

}  // namespace

// Pixels that the longest in-ellipse row spans: it holds at most one more.
double jpet::row_span(const DevGeom& g) {
  return 2.0 * 3.0 * g.sigma_z / std::sqrt(2.0) / g.pixel_width;
}

// Scanner<float, short> constructor arithmetic (src/2d/strip/scanner.h:50-67)
// and GaussianKernel<float> constants (gaussian_kernel.h:27-33), in float.
DevGeom jpet::make_dev_geom(const jpet_strip_geom& in) {
  volatile float R = static_cast<float>(in.radius);
  volatile float L = static_cast<float>(in.scintillator_length);
  volatile float ph = static_cast<float>(in.pixel_height);
  volatile float pw = static_cast<float>(in.pixel_width);
  volatile float sz = static_cast<float>(in.sigma_z);
  volatile float sdl = static_cast<float>(in.sigma_dl);
  const int16_t n_y = static_cast<int16_t>(in.n_y_pixels);
  const int16_t n_z = static_cast<int16_t>(in.n_z_pixels);
  DevGeom g{};
  g.radius = R;
  g.half_length = L / 2;
  g.n_y = n_y;
  g.n_z = n_z;
  g.pixel_width = pw;
  g.pixel_height = ph;
  g.sigma_z = sz;
  g.sigma_dl = sdl;
  volatile float size_y = n_y * ph;
  volatile float size_z = n_z * pw;
  volatile float tl_y = 0.0f + size_y / 2;
  volatile float tl_z = 0.0f - size_z / 2;
  g.tl_y = tl_y;
  g.tl_z = tl_z;
  g.tl_y_half_h = tl_y - ph / 2;
  g.tl_z_half_w = tl_z + pw / 2;
  volatile float ipz = 1 / (sz * sz);
  volatile float ipd = 1 / (sdl * sdl);
  g.ipz = ipz;
  g.ipd = ipd;
  volatile float prod = ipz * ipz;
  prod = prod * ipd;
  g.c0 = static_cast<float>(1 / (2 * M_PI * M_PI) * std::sqrt(static_cast<float>(prod)));
  return g;
}

namespace {

int validate_geom(const jpet_strip_geom* geom, std::string& msg) {
  if (!geom) {
    msg = "geometry is NULL";
    return JPET_ERR_ARGUMENT;
  }
  if (geom->n_y_pixels <= 0 || geom->n_z_pixels <= 0 || geom->n_y_pixels > 32767 ||
      geom->n_z_pixels > 32767) {
    msg = "n_y_pixels and n_z_pixels must be in [1, 32767]";
    return JPET_ERR_ARGUMENT;
  }
  if (static_cast<int64_t>(geom->n_y_pixels) * geom->n_z_pixels > (1ll << 30)) {
    msg = "image too large";
    return JPET_ERR_ARGUMENT;
  }
  if (!(geom->pixel_height > 0) || !(geom->pixel_width > 0) || !(geom->sigma_z > 0) ||
      !(geom->sigma_dl > 0) || !(geom->radius > 0) || !(geom->scintillator_length > 0)) {
    msg = "radius, length, pixel sizes and sigmas must be positive";
    return JPET_ERR_ARGUMENT;
  }
  return JPET_OK;
}

// The widest in-ellipse row is 2 * 3 sigma_z / sqrt(2) / pixel (+ rounding).
int widest_row(const DevGeom& g) {
  const double half = 3.0 * g.sigma_z / std::sqrt(2.0) / g.pixel_width;
  return 2 * static_cast<int>(half) + 3;
}

// The batch-union kernel's batch shape for events of the given box rows (99.9 %
// of them) and widest in-ellipse row, and what a CTA of that shape can hold: the
// pixels of its windows (the largest that still let ctas_per_sm CTAs share an
// SM's shared memory) and its largest chunk.  The smallest shape that leaves the
// union of a batch a few rows and columns beyond its events' own; an explicit
// CTA size selects the 64-row shapes.  Measured per iteration: 1e6 events of 26
// rows x 11 columns (5 mm pixels) 552 us in the 64x32 shape, 294 in 32x16; 1e6
// events of 82 rows x 31 columns (2 mm, sigma 14 / 55), of which the 64x32
// shape's windows and batches take one in ten, 23.0 ms there, 1.52 ms in 96x40
// (1.64 with batches of 4 events and two CTAs per SM).  For 64x32n4 the count is
// one more than its windows and records leave room for: the chunk rule below runs
// faster with 4 than with 3 (5e5 events at 2 mm 337 and 383 us; mostly the same).
//
// Events whose rows no batch takes (40 columns from an even start) are rasterised
// one by one, and its one CTA of 12 warps per SM does that slowest: 4e5 events of
// 90 rows in the 96x40 shape / in the 64x32 one, whose windows leave them to the
// large-box kernel, at a span of 38.2 pixels 2.2 / 9.4 ms, 39.0 4.2 / 9.5,
// 39.2 14.0 / 9.5, 42.4 24.0 / 10.0.
constexpr int kUnionRows = 96;          // the tallest shape's
constexpr double kUnionSpan = 39.1;
struct UnionLimits {
  int shape, window_px, ctas_per_sm, max_chunk;
};
constexpr UnionLimits kUnionDefault{kUnion64x32, 6144, 2, 2048};
UnionLimits union_limits(const jpet_strip_opts& o, int rows, int widest, double span) {
  if (o.block_threads == 128) return UnionLimits{kUnion64x32n4, 6144, 4, 2048};
  if (o.block_threads == 256) return kUnionDefault;
  // a batch's rows are wider than its events' by a column of alignment and, at
  // the ends of the box, by the spread of slopes in half a sort bucket
  const bool narrow = widest + 1 + rows / 8 <= 16;
  if (rows <= 30 && narrow) return UnionLimits{kUnion32x16, 3328, 4, 1024};
  if (rows <= 30 && widest <= 28) return UnionLimits{kUnion32x32, 3328, 4, 1024};
  if (rows <= 64 && narrow) return UnionLimits{kUnion64x16, 4096, 2, 1024};
  if (rows <= 64 && widest <= 28) return kUnionDefault;
  return span <= kUnionSpan ? UnionLimits{kUnion96x40, 10752, 1, 1024} : kUnionDefault;
}

// JPET_PRECISION_* -> the fast kernels' accumulation mode
int precision_code(int precision) {
  return precision == JPET_PRECISION_COMPENSATED ? kPrecisionCompensated
         : precision == JPET_PRECISION_FP64_DEN  ? kPrecisionCompensatedDen64
         : precision == JPET_PRECISION_FIXED     ? kPrecisionFixed
                                                 : kPrecisionFloat;
}

// Window sizing: the largest box dimension that covers all but a tiny tail of
// the events (the tail takes the global-memory path), then the largest square
// tile whose window (tile + box) fits the shared-memory budget.
void choose_tiling(const jpet_strip_opts& o, const std::vector<int32_t>& hw,
                   const std::vector<int32_t>& hh, int64_t n_nonempty, int n_sms, int beside,
                   size_t most_smem, int n_y, int n_z, int widest, double span, double tallest,
                   Tiling& t) {
  // window pixels per array (rho, out): 12288 (~100 KiB per CTA, 2 CTAs per SM)
  // for 256-thread CTAs; 6144 (~55 KiB, 4 CTAs per SM) for the row-owned
  // kernel's 128-thread CTAs; the batch-union kernel's from its batch shape
  const bool fast = o.mode == JPET_MODE_CPU_REFERENCE &&
                    (o.variant == JPET_VARIANT_FAST || o.variant == JPET_VARIANT_ROWS);
  const bool union_k = fast && o.variant == JPET_VARIANT_FAST;
  const bool rows4 = fast && o.block_threads != 256;
  auto pct = [&](const std::vector<int32_t>& h, double keep) {
    int64_t tail = static_cast<int64_t>(std::floor((1.0 - keep) * n_nonempty));
    int64_t acc = 0;
    for (int b = kHistBins - 1; b > 0; --b) {
      acc += h[b];
      if (acc > tail) return b;
    }
    return 1;
  };
  // the box limits shrunk until at least an 8x8 tile fits the budget
  auto shrink = [](int& w, int& h, int budget) {
    while ((w + 8) * (h + 8) > budget) {
      if (w >= h) w = w * 7 / 8; else h = h * 7 / 8;
    }
  };
  int mw = std::min(255, std::max(1, pct(hw, 0.99999)));
  int mh = std::min(1024, std::max(1, pct(hh, 0.99999)));
  // batch shape of the batch-union kernel
  const int rows999 = pct(hh, 0.999);
  UnionLimits u = union_limits(o, rows999, widest, span);
  if (union_k && u.shape == kUnion96x40 && rows999 > kUnionRows) {
    // Boxes taller than any batch: one by one in the 64x32 shape's windows where
    // those hold them, else in the large-box kernel, with batches of the others
    // in the 96x40 shape.  4e5 events of up to 105 rows (2 mm, sigma 8 / 70, 62 %
    // of them taller): 14.9 ms with the tall ones in the 96x40 shape's windows,
    // 2.3 with them in the large-box kernel, 4.4 in the 64x32 shape.
    int w = mw, h = mh;
    shrink(w, h, kUnionDefault.window_px);
    if (h > kUnionRows)
      u = kUnionDefault;
    else
      mh = std::min(mh, kUnionRows);
  }
  t.union_shape = u.shape;
  const int budget_px = union_k ? u.window_px : (rows4 ? 6144 : 12288);
  shrink(mw, mh, budget_px);
  int tw = o.tile_w > 0 ? o.tile_w : 0, th = o.tile_h > 0 ? o.tile_h : 0;
  if (tw == 0 || th == 0) {
    int side = 8;
    while ((mw + 2 * side) * (mh + 2 * side) <= budget_px && side < 64) side *= 2;
    if (tw == 0) tw = side;
    if (th == 0) th = side;
  }
  tw = std::min(tw, n_z);
  th = std::min(th, n_y);
  while ((mw + tw) * (mh + th) > budget_px && (tw > 1 || th > 1)) {
    if (tw >= th && tw > 1) tw = std::max(1, tw / 2); else th = std::max(1, th / 2);
  }
  auto place = [&]() {
    t.tile_w = tw;
    t.tile_h = th;
    t.max_box_w = mw;
    t.max_box_h = mh;
    t.win_w = tw + mw;
    t.win_h = th + mh;
  };
  place();
  // The pixel budget counts a window's own columns.  A window of few columns takes
  // up to 2.7 times as much in shared memory (fast_pitch), three times over in the
  // compensated modes, so tall and narrow ones are cut until a CTA holds them; and
  // a union row's word has 9 bits for its first column.
  if (union_k) {
    t.chunk_events = u.max_chunk;
    const int prec = precision_code(o.precision);
    while (t.win_w > 511 || union_smem_bytes(t, prec) > most_smem) {
      if (t.win_w > 511)
        tw = std::max(1, tw / 2);
      else if (th > 8)
        th = th / 2;
      else
        mh = mh * 7 / 8;
      place();
    }
  }
  t.n_tiles_x = (n_z + tw - 1) / tw;
  t.n_tiles_y = (n_y + th - 1) / th;
  // events per chunk of the batch-union kernel: the largest power of two (64 to
  // 2048) that still leaves at least 4 chunks per resident CTA, or 2 below 1024.
  // Larger chunks mean fewer chunk prologues and window flushes, fewer chunks
  // leave SMs idle at the end of the launch.  Us per iteration with 16 and 4, 8
  // and 4 or 4 and 2 chunks: 2e6 events at 2 mm 1128, 1128, 1090; 3e6 1654, 1591,
  // 1577; 2e5 190, 190, 177; 1e6 at 5 mm 225, 225, 206.  With 2 and 2: 1e6 at 3 mm
  // 527 instead of 507; with 1 below 1024: 2e5 at 3 mm 160 instead of 136.  Chunks
  // of 32 events: 2e4 at 5 mm 31 instead of 25.  The fixed-point mode (whose
  // integer window sums must stay below 2^31) takes at most 512, the other
  // kernels 512.
  // Below one chunk of 64 events per SM they shrink further, to 8: each is a serial
  // chain of batches, of one or two events in sets as sparse as these (1e3 events
  // at 5 mm 39 us with 64, 28 with 32, 23 with 16, 18.5 with 8; 5e3 31, and 27 with
  // 32).  Not in the 96x40 shape, whose windows cost more (2e3 at sigma 14 / 55 33
  // and 35), and in a batch only below a handle's share of the SMs (10 iterations of
  // 100 instances of 2e3 events 6.0 ms, with short chunks 8.8).
  t.chunk_events = 512;
  if (union_k) {
    const int64_t resident = static_cast<int64_t>(u.ctas_per_sm) * std::max(n_sms, 1);
    t.chunk_events = o.precision == JPET_PRECISION_FIXED ? 512 : u.max_chunk;
    while (t.chunk_events > 64 &&
           n_nonempty / t.chunk_events < (t.chunk_events > 512 ? 4 : 2) * resident)
      t.chunk_events /= 2;
    const int least = u.shape == kUnion96x40 ? 64 : 8;
    while (t.chunk_events > least && n_nonempty / t.chunk_events < n_sms / beside)
      t.chunk_events /= 2;
  }
  t.threads = o.block_threads > 0 ? o.block_threads : (rows4 ? 128 : 256);
  // order of a tile's events: for the batch-union kernel, tan buckets of 1/4 and
  // corner cells of 2 rows x 1 column; single pixels where many events share one
  // and the rows are short (the union of 16-column batches has no column to
  // spare) or where the tallest events leave the batch no row to spare (8e5 events
  // of 63.5 rows: 2.54 slots with cells of two rows, 1.77 with one), wider cells
  // and buckets where few share a pixel.  Pixel slots of the unions per
  // evaluated pixel, against the plain row-by-row order with buckets of 1/8:
  // 6e6 events at 1 mm 2.60 -> 1.84, 2e6 at 2 mm 2.00 -> 1.72, 1e6 at 5 mm
  // 2.62 -> 2.59 (2.70 with cells of two rows), 2e4 at 5 mm 6.7 -> 3.5 (4.0 with
  // the narrow cells); the iterations follow (1 mm 4889 -> 3974 us).
  t.cell_w = t.cell_h = 1;
  t.tan_shift = 6;
  if (union_k) {
    const double per_px = static_cast<double>(n_nonempty) / (static_cast<double>(n_y) * n_z);
    const bool row_to_spare = tallest + 1.0 <= union_ops(t.union_shape).rows;
    t.cell_h = !row_to_spare || (t.union_shape == kUnion32x16 && per_px >= 6.0) ? 1
               : per_px < 2.0                                                   ? 3
                                                                                : 2;
    t.cell_w = per_px < 2.0 ? 2 : 1;
    t.tan_shift = per_px < 2.0 ? 8 : 7;
  }
  // one spare entry per event for its widest row; a multiple of 8 entries so
  // that every event's table starts on a 16-byte boundary
  t.row_stride = (mh + 1 + 7) & ~7;
  // register-cache shape of the fast kernel from the rows of 99.9% of the boxes
  // (fast_width_shape adds the widest in-ellipse row)
  t.fast_shape = rows999 <= 32 ? kShapeS : (rows999 <= 64 ? kShapeM : kShapeL);
  t.rows_shape = kRowsShape4x1x3;
}

int fast_width_shape(const DevGeom& g) {
  const int w = widest_row(g);
  return w <= 16 ? kShapeS : (w <= 24 ? kShapeM : kShapeL);
}

// Row records of the batch-union kernel for the chunks of part k.
cudaError_t write_records(jpet_strip* h, size_t k, cudaStream_t s) {
  return launch_union_records(h->g, h->fc, h->tiling, h->chunks.p + h->parts[k].first,
                              h->parts[k].second, h->sorted_geom.p, h->sorted_box.p,
                              h->row_table.p, h->batches.p, h->union_rows.p, h->records.p, s);
}

// Workspace of the row records (16 bytes per event and row of the batch shape:
// 1 KB per event with 64 rows), the parts of the chunk list that it holds at a
// time and each chunk's place in it.  Up to half of the free memory is taken
// (looked up above 1 GB only); with less than all events' records they are
// written again, part by part, in every iteration.
cudaError_t alloc_records(jpet_strip* h, std::vector<Chunk>& chunks, int64_t n_events) {
  const size_t rows = union_row_words(h->tiling), each = rows * sizeof(float4);
  const size_t least = static_cast<size_t>(h->tiling.chunk_events);
  size_t cap = static_cast<size_t>(std::max<int64_t>(n_events, 1));
  h->parts.clear();
  if (chunks.empty()) return cudaSuccess;
  if (cap * rows > h->records.n) {
    h->records.release();
    if (cap * each > (1ull << 30)) {
      size_t free_bytes = 0, total = 0;
      const cudaError_t e = cudaMemGetInfo(&free_bytes, &total);
      if (e != cudaSuccess) return e;
      cap = std::min(cap, free_bytes / 2 / each);
    }
    for (;; cap /= 2) {
      cap = std::max(cap, least);
      const cudaError_t e = h->records.alloc(cap * rows);
      if (e == cudaSuccess) break;
      if (e != cudaErrorMemoryAllocation || cap == least) return e;
      cudaGetLastError();
    }
  }
  size_t used = 0;
  for (size_t k = 0; k < chunks.size(); ++k) {
    const size_t count = static_cast<size_t>(chunks[k].count);
    if (k == 0 || used + count > cap) {
      h->parts.emplace_back(static_cast<int32_t>(k), 0);
      used = 0;
    }
    chunks[k].rec = static_cast<int32_t>(used);
    used += count;
    ++h->parts.back().second;
  }
  return cudaSuccess;
}

int prepare_events(jpet_strip* h, const float* d_zu, const float* d_zd, const float* d_dl,
                   int64_t n, int32_t stride = 1) {
  cudaStream_t s = h->stream;
  h->events_ready = false;
  ++h->generation;
  h->n_events = n;
  h->n_sorted = h->n_oversize = h->n_chunks = h->n_tiles_nonempty = 0;
  h->parts.clear();
  h->total_box_pixels = 0;
  if (n > (int64_t)INT32_MAX - 1)
    return h->fail(JPET_ERR_ARGUMENT, "at most %d events per handle", INT32_MAX - 1);
  const size_t sort_bytes = n > 0 ? sort_temp_bytes(n) : 0;
  JPET_CUDA(h, carve(h->scratch, [&](Carver& c) {
              c(h->hist, 2 * kHistBins);
              c(h->box_pixels, 1);
              c(h->small, 4);
              c(h->ev_geom, n);
              c(h->ev_box, n);
              c(h->sort_keys, 2 * static_cast<size_t>(n));
              c(h->sort_idx, 2 * static_cast<size_t>(n));
              c(h->sort_tmp, sort_bytes);
            }),
            "cudaMalloc(event set-up)");
  // the counters and histograms, placed first
  JPET_CUDA(h, cudaMemsetAsync(h->scratch.p, 0,
                               reinterpret_cast<unsigned char*>(h->ev_geom.p) - h->scratch.p, s),
            "memset");
  JPET_CUDA(h, launch_prep_events(h->g, d_zu, d_zd, d_dl, stride, n, h->ev_geom.p, h->ev_box.p,
                                  h->hist.p, h->hist.p + kHistBins, h->box_pixels.p, s),
            "prep_events launch");
  std::vector<int32_t> hist(2 * kHistBins);
  JPET_CUDA(h, cudaMemcpyAsync(hist.data(), h->hist.p, hist.size() * sizeof(int32_t),
                               cudaMemcpyDeviceToHost, s), "copy histogram");
  JPET_CUDA(h, cudaMemcpyAsync(&h->total_box_pixels, h->box_pixels.p,
                               sizeof(unsigned long long), cudaMemcpyDeviceToHost, s),
            "copy counter");
  JPET_CUDA(h, cudaStreamSynchronize(s), "prep_events");
  std::vector<int32_t> hw(hist.begin(), hist.begin() + kHistBins);
  std::vector<int32_t> hh(hist.begin() + kHistBins, hist.end());
  int64_t nonempty = 0;
  for (int b = 1; b < kHistBins; ++b) nonempty += hw[b];
  int n_sms = 0, most_smem = 0;
  JPET_CUDA(h, cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, h->device),
            "cudaDeviceGetAttribute");
  JPET_CUDA(h, cudaDeviceGetAttribute(&most_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                      h->device),
            "cudaDeviceGetAttribute");
  choose_tiling(h->opts, hw, hh, nonempty, n_sms, h->beside, static_cast<size_t>(most_smem),
                h->g.n_y, h->g.n_z, widest_row(h->g), row_span(h->g),
                3.0 * h->g.sigma_dl / h->g.pixel_height, h->tiling);
  h->tiling.fast_shape = std::max(h->tiling.fast_shape, fast_width_shape(h->g));
  {
    int64_t tail = static_cast<int64_t>(std::floor(0.001 * nonempty)), acc_h = 0;
    int rows999 = 1;
    for (int b = kHistBins - 1; b > 0; --b) {
      acc_h += hh[b];
      if (acc_h > tail) { rows999 = b; break; }
    }
    h->tiling.rows_shape = h->opts.raster_shape > 0
                               ? h->opts.raster_shape - 1
                               : rows_shape_for(rows999, widest_row(h->g) - 1);
  }
  const Tiling& t = h->tiling;
  const int32_t n_tiles = t.n_tiles_x * t.n_tiles_y;
  JPET_CUDA(h, h->tile_count.alloc(n_tiles), "cudaMalloc(tiles)");
  JPET_CUDA(h, cudaMemsetAsync(h->tile_count.p, 0, n_tiles * sizeof(int32_t), s), "memset");
  JPET_CUDA(h, launch_count_tiles(t, n, h->ev_box.p, h->tile_count.p, h->small.p, s),
            "count_tiles launch");
  std::vector<int32_t> count(n_tiles);
  int32_t n_over = 0;
  JPET_CUDA(h, cudaMemcpyAsync(count.data(), h->tile_count.p, n_tiles * sizeof(int32_t),
                               cudaMemcpyDeviceToHost, s), "copy tile counts");
  JPET_CUDA(h, cudaMemcpyAsync(&n_over, h->small.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s),
            "copy counter");
  JPET_CUDA(h, cudaStreamSynchronize(s), "count_tiles");
  // chunk list over the tiles' ranges of the sorted events (full chunks first, then the
  // partial tail chunks by decreasing size, so the longest work starts first)
  std::vector<Chunk> full, partial;
  int32_t acc = 0;
  for (int32_t k = 0; k < n_tiles; ++k) {
    const int32_t c = count[k];
    if (c > 0) ++h->n_tiles_nonempty;
    const int32_t ox = (k % t.n_tiles_x) * t.tile_w, oy = (k / t.n_tiles_x) * t.tile_h;
    for (int32_t s0 = 0; s0 < c; s0 += t.chunk_events) {
      Chunk ch{acc + s0, std::min(t.chunk_events, c - s0), ox, oy};
      (ch.count == t.chunk_events ? full : partial).push_back(ch);
    }
    acc += c;
  }
  std::stable_sort(partial.begin(), partial.end(),
                   [](const Chunk& a, const Chunk& b) { return a.count > b.count; });
  full.insert(full.end(), partial.begin(), partial.end());
  h->n_sorted = acc;
  h->n_oversize = n_over;
  h->n_chunks = static_cast<int32_t>(full.size());
  h->use_fast = h->opts.mode == JPET_MODE_CPU_REFERENCE && h->opts.variant != JPET_VARIANT_EXACT;
  h->use_union = h->use_fast && h->opts.variant == JPET_VARIANT_FAST;
  const size_t n_acc = static_cast<size_t>(acc), table = n_acc * t.row_stride;
  const bool rows_k = h->use_fast && h->opts.variant == JPET_VARIANT_ROWS;
  JPET_CUDA(h, carve(h->set_block, [&](Carver& c) {
              c(h->chunks, full.size());
              c(h->sorted_geom, n_acc);
              c(h->sorted_box, n_acc);
              c(h->over_geom, n_over);
              c(h->over_box, n_over);
              c(h->row_table, h->use_fast ? table : 0);
              c(h->batches, h->use_union ? n_acc : 0);
              c(h->union_rows, h->use_union ? n_acc * union_row_words(t) : 0);
              c(h->row_pq, rows_k ? table : 0);
              c(h->row_pk, rows_k ? table : 0);
              c(h->ev_pk, rows_k ? n_acc : 0);
            }),
            "cudaMalloc(events)");
  // the last allocation of the event set: it takes what it can get
  if (h->use_union) JPET_CUDA(h, alloc_records(h, full, acc), "cudaMalloc(row records)");
  if (n > 0) {
    // tile, then box corner inside the tile, then tan (strip_sort.cu)
    JPET_CUDA(h, sort_events(t, n, h->ev_geom.p, h->ev_box.p, h->sort_keys.p, h->sort_idx.p,
                             h->sort_tmp.p, sort_bytes, acc, n_over, h->sorted_geom.p, h->sorted_box.p,
                             h->over_geom.p, h->over_box.p, s),
              "event sort");
  }
  h->table_kernel_calls = 0;
  if (h->use_fast && acc > 0) {
    JPET_CUDA(h, cudaMemsetAsync(h->box_pixels.p, 0, sizeof(unsigned long long), s), "memset");
    JPET_CUDA(h, launch_row_tables(h->g, t, acc, h->sorted_geom.p, h->sorted_box.p,
                                   h->row_table.p, h->box_pixels.p, s),
              "row_table launch");
    JPET_CUDA(h, cudaMemcpyAsync(h->chunks.p, full.data(), full.size() * sizeof(Chunk),
                                 cudaMemcpyHostToDevice, s), "copy chunks");
    if (h->use_union) {
      JPET_CUDA(h, launch_union_batches(t, h->chunks.p, h->n_chunks, h->sorted_box.p,
                                        h->row_table.p, h->batches.p, h->union_rows.p, s),
                "batch formation launch");
      if (h->parts.size() == 1) JPET_CUDA(h, write_records(h, 0, s), "row record launch");
      JPET_CUDA(h, union_prepare_kernel(t, precision_code(h->opts.precision)),
                "batch-union kernel attributes");
    } else if (rows_k) {
      JPET_CUDA(h, launch_row_coefficients(h->g, h->fc, t, acc, h->sorted_geom.p,
                                           h->sorted_box.p, h->row_table.p, h->row_pq.p,
                                           h->row_pk.p, h->ev_pk.p, s),
                "row coefficient launch");
      JPET_CUDA(h, rows_prepare_kernel(t, precision_code(h->opts.precision)),
                "row-owned kernel attributes");
    }
    JPET_CUDA(h, cudaMemcpyAsync(&h->table_kernel_calls, h->box_pixels.p,
                                 sizeof(unsigned long long), cudaMemcpyDeviceToHost, s),
              "copy counter");
  }
  JPET_CUDA(h, cudaStreamSynchronize(s), "prepare events");
  h->scratch.release();
  h->events_ready = true;
  h->counters_valid = false;
  return JPET_OK;
}

int upload_and_prepare(jpet_strip* h, const float* zu, const float* zd, const float* dl,
                       const float* aos, int64_t n) {
  if (n < 0) return h->fail(JPET_ERR_ARGUMENT, "negative event count");
  if (n > 0 && !aos && (!zu || !zd || !dl)) return h->fail(JPET_ERR_ARGUMENT, "NULL event array");
  if (n == 0) return prepare_events(h, nullptr, nullptr, nullptr, 0);
  JPET_CUDA(h, h->raw.alloc(3 * static_cast<size_t>(n)), "cudaMalloc(events)");
  float* d_zu = h->raw.p;
  float* d_zd = h->raw.p + n;
  float* d_dl = h->raw.p + 2 * n;
  cudaStream_t s = h->stream;
  if (aos) {
    // one contiguous copy of the AoS triples; the preparation kernel reads
    // them with stride 3 (the reference transposes to SoA on the host,
    // cuda/gpu_events_soa.h:15-44)
    JPET_CUDA(h, cudaMemcpyAsync(h->raw.p, aos, 3 * static_cast<size_t>(n) * sizeof(float),
                                 cudaMemcpyHostToDevice, s),
              "copy events");
    return prepare_events(h, h->raw.p, h->raw.p + 1, h->raw.p + 2, n, 3);
  } else {
    const size_t bytes = static_cast<size_t>(n) * sizeof(float);
    JPET_CUDA(h, cudaMemcpyAsync(d_zu, zu, bytes, cudaMemcpyHostToDevice, s), "copy z_u");
    JPET_CUDA(h, cudaMemcpyAsync(d_zd, zd, bytes, cudaMemcpyHostToDevice, s), "copy z_d");
    JPET_CUDA(h, cudaMemcpyAsync(d_dl, dl, bytes, cudaMemcpyHostToDevice, s), "copy dl");
  }
  return prepare_events(h, d_zu, d_zd, d_dl, n);
}

// n iterations of the prepared events on stream s.
int iterate_on(jpet_strip* h, int n, cudaStream_t s) {
  const size_t n_pix = static_cast<size_t>(h->g.n_y) * h->g.n_z;
  const float* sens = h->sens_pixel.p;
  for (int it = 0; it < n; ++it) {
    // every variant adds into a cleared image: the exact kernel into its double one
    const bool exact = h->out_sum.p != nullptr;
    ClearList clear;
    if (exact)
      clear.add(h->out_sum.p, n_pix * sizeof(double));
    else
      clear.add(h->out.p, n_pix * sizeof(float));
    clear.add(h->counters.p, sizeof(DevCounters));
    const bool aux_img = h->opts.precision != JPET_PRECISION_FP32;
    const AuxImage aux{h->out_lo.p, h->out_q.p};
    if (h->out_lo.p) clear.add(h->out_lo.p, n_pix * sizeof(float));
    if (h->out_q.p) clear.add(h->out_q.p, n_pix * sizeof(unsigned long long));
    JPET_CUDA(h, launch_clear(clear, s), "clear image launch");
    if (h->use_fast) {
      const int prec = precision_code(h->opts.precision);
      const uint32_t seed = 0x9E3779B9u * static_cast<uint32_t>(h->iterations_done + 1);
      if (h->use_union) {
        for (size_t k = 0; k < h->parts.size(); ++k) {
          if (h->parts.size() > 1) JPET_CUDA(h, write_records(h, k, s), "row record launch");
          JPET_CUDA(h, launch_iterate_union(h->g, h->fc, h->tiling,
                                            h->chunks.p + h->parts[k].first, h->parts[k].second,
                                            h->sorted_geom.p, h->sorted_box.p, h->records.p,
                                            h->union_rows.p, h->batches.p, h->rho.p, h->out.p,
                                            aux, h->counters.p, prec, seed, s),
                    "iteration kernel launch");
        }
      } else if (h->opts.variant == JPET_VARIANT_WARP) {
        JPET_CUDA(h, launch_iterate_fast(h->g, h->fc, h->tiling, h->chunks.p, h->n_chunks,
                                         h->sorted_geom.p, h->sorted_box.p, h->row_table.p,
                                         h->rho.p, h->out.p, aux, h->counters.p, prec,
                                         seed, s),
                  "iteration kernel launch");
      } else {
        JPET_CUDA(h, launch_iterate_rows(h->g, h->fc, h->tiling, h->chunks.p, h->n_chunks,
                                         h->sorted_geom.p, h->sorted_box.p, h->ev_pk.p,
                                         h->row_pk.p, h->row_pq.p, h->rho.p, h->out.p,
                                         aux, h->counters.p, prec, seed, s),
                  "iteration kernel launch");
      }
    } else {
      JPET_CUDA(h, launch_iterate_exact(h->g, h->opts.mode, h->n_sorted, h->sorted_geom.p,
                                        h->sorted_box.p, h->rho.p, sens, h->out_sum.p,
                                        h->counters.p, s),
                "iteration kernel launch");
    }
    if (exact) {
      JPET_CUDA(h, launch_iterate_exact(h->g, h->opts.mode, h->n_oversize, h->over_geom.p,
                                        h->over_box.p, h->rho.p, sens, h->out_sum.p,
                                        h->counters.p, s),
                "large-box kernel launch");
      JPET_CUDA(h, launch_round_image(h->out_sum.p, h->out.p, n_pix, s), "image rounding launch");
    } else {
      JPET_CUDA(h, launch_iterate_exact(h->g, h->opts.mode, h->n_oversize, h->over_geom.p,
                                        h->over_box.p, h->rho.p, sens, h->out.p, h->counters.p, s),
                "large-box kernel launch");
    }
    if (aux_img)
      JPET_CUDA(h, launch_combine_aux(precision_code(h->opts.precision), aux, h->out.p, h->out.p,
                                      n_pix, s),
                "combine kernel launch");
    std::swap(h->rho, h->out);
    ++h->iterations_done;
    h->counters_valid = true;
  }
  return JPET_OK;
}

}  // namespace

// ---- access for the batch (strip_batch.cu) --------------------------------------
namespace jpet {

int handle_batch_ready(const jpet_strip* h, std::string& why) {
  if (!h->events_ready) {
    why = "events not set";
    return JPET_ERR_STATE;
  }
  if (!h->use_fast || h->opts.variant == JPET_VARIANT_WARP ||
      h->opts.precision != JPET_PRECISION_FP32) {
    why = "batched instances run the FP32 batch-union or row-owned kernel (CPU-reference mode)";
    return JPET_ERR_UNSUPPORTED;
  }
  return JPET_OK;
}

const DevGeom& handle_geom(const jpet_strip* h) { return h->g; }
const Tiling& handle_tiling(const jpet_strip* h) { return h->tiling; }
uint64_t handle_generation(const jpet_strip* h) { return h->generation; }
const float* handle_image(const jpet_strip* h) { return h->rho.p; }
// kernels of one FP32 iteration: the clear and those over the events
int handle_launches(const jpet_strip* h) {
  const int parts = static_cast<int>(h->parts.size());  // with several, their records too
  return 1 + (parts > 1 ? 2 * parts : h->n_chunks > 0 ? 1 : 0) + (h->n_oversize > 0 ? 1 : 0);
}

// Issues n iterations on the (capturing) stream and leaves the handle as it was:
// handle_batch_done counts them when the graph has run.
int handle_capture_iterations(jpet_strip* h, int n, cudaStream_t s) {
  const bool valid = h->counters_valid;
  const int64_t done = h->iterations_done;
  const float* image = h->rho.p;
  const int rc = iterate_on(h, n, s);
  if (h->rho.p != image) std::swap(h->rho, h->out);
  h->iterations_done = done;
  h->counters_valid = valid;
  return rc;
}

// After n batched iterations: the latest image is in the other buffer if n is odd.
void handle_batch_done(jpet_strip* h, int n) {
  if (n & 1) std::swap(h->rho, h->out);
  h->iterations_done += n;
  h->counters_valid = true;
}

int handle_reprepare(jpet_strip* h, int raster_shape, int block_threads, int tile,
                     const float* d_zu, const float* d_zd, const float* d_dl, int64_t n) {
  h->opts.raster_shape = raster_shape;
  h->opts.block_threads = block_threads;
  h->opts.tile_w = h->opts.tile_h = tile;
  return prepare_events(h, d_zu, d_zd, d_dl, n);
}

const char* handle_error(const jpet_strip* h) { return h->last_error.c_str(); }
void handle_set_beside(jpet_strip* h, int32_t n) { h->beside = n; }

}  // namespace jpet

extern "C" {

int jpet_strip_abi_version(void) { return JPET_STRIP_ABI_VERSION; }

void jpet_strip_default_opts(jpet_strip_opts* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
}

int jpet_strip_create(const jpet_strip_geom* geom, const jpet_strip_opts* opts,
                      jpet_strip_t** out) {
  if (!out) {
    g_create_error = "output handle pointer is NULL";
    return JPET_ERR_ARGUMENT;
  }
  *out = nullptr;
  std::string msg;
  int rc = validate_geom(geom, msg);
  if (rc != JPET_OK) {
    g_create_error = msg;
    return rc;
  }
  jpet_strip_opts o;
  jpet_strip_default_opts(&o);
  if (opts) o = *opts;
  if (o.mode != JPET_MODE_CPU_REFERENCE && o.mode != JPET_MODE_GPU_REFERENCE) {
    g_create_error = "unknown mode";
    return JPET_ERR_ARGUMENT;
  }
  if (o.variant != JPET_VARIANT_FAST && o.variant != JPET_VARIANT_EXACT &&
      o.variant != JPET_VARIANT_WARP && o.variant != JPET_VARIANT_ROWS) {
    g_create_error = "unknown kernel variant";
    return JPET_ERR_ARGUMENT;
  }
  if (o.mode == JPET_MODE_CPU_REFERENCE &&
      (o.variant == JPET_VARIANT_FAST || o.variant == JPET_VARIANT_ROWS) &&
      o.block_threads != 0 && o.block_threads != 128 && o.block_threads != 256) {
    g_create_error = "the row-owned kernel runs 128- or 256-thread CTAs";
    return JPET_ERR_ARGUMENT;
  }
  if (o.raster_shape < JPET_RASTER_AUTO || o.raster_shape > JPET_RASTER_2x1x6) {
    g_create_error = "unknown rasterisation shape";
    return JPET_ERR_ARGUMENT;
  }
  if (o.precision != JPET_PRECISION_FP32 && o.precision != JPET_PRECISION_COMPENSATED &&
      o.precision != JPET_PRECISION_FP64_DEN && o.precision != JPET_PRECISION_FIXED) {
    g_create_error = "unknown precision mode";
    return JPET_ERR_ARGUMENT;
  }
  if (o.precision != JPET_PRECISION_FP32 &&
      (o.mode != JPET_MODE_CPU_REFERENCE || o.variant == JPET_VARIANT_EXACT)) {
    g_create_error = "compensated precision modes need the fast kernel and the CPU-reference mode";
    return JPET_ERR_UNSUPPORTED;
  }
  int n_dev = 0;
  cudaError_t e = cudaGetDeviceCount(&n_dev);
  if (e != cudaSuccess || n_dev <= 0) {
    g_create_error = std::string("no CUDA device: ") + cudaGetErrorString(e);
    return JPET_ERR_CUDA;
  }
  if (o.device < 0 || o.device >= n_dev) {
    g_create_error = "device ordinal out of range";
    return JPET_ERR_ARGUMENT;
  }
  e = cudaSetDevice(o.device);
  if (e != cudaSuccess) {
    g_create_error = std::string("cudaSetDevice: ") + cudaGetErrorString(e);
    return JPET_ERR_CUDA;
  }
  jpet_strip* h = new (std::nothrow) jpet_strip();
  if (!h) {
    g_create_error = "host allocation failed";
    return JPET_ERR_MEMORY;
  }
  h->geom_in = *geom;
  h->opts = o;
  h->device = o.device;
  h->g = make_dev_geom(*geom);
  h->fc.kz = -1.4426950408889634f * h->g.ipz;
  h->fc.kdl = -2.0f * 1.4426950408889634f * h->g.ipd;
  h->fc.two_r2 = 2.0f * h->g.radius * h->g.radius;
  e = cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    g_create_error = std::string("cudaStreamCreate: ") + cudaGetErrorString(e);
    delete h;
    return JPET_ERR_CUDA;
  }
  h->stream = h->own_stream;
  const size_t n_pix = static_cast<size_t>(h->g.n_y) * h->g.n_z;
  const bool comp = o.precision == JPET_PRECISION_COMPENSATED ||
                    o.precision == JPET_PRECISION_FP64_DEN;
  const bool exact = o.mode == JPET_MODE_GPU_REFERENCE || o.variant == JPET_VARIANT_EXACT;
  if ((comp && h->out_lo.alloc(n_pix) != cudaSuccess) ||
      (exact && h->out_sum.alloc(n_pix) != cudaSuccess) ||
      (o.precision == JPET_PRECISION_FIXED && h->out_q.alloc(n_pix) != cudaSuccess) ||
      h->rho.alloc(n_pix) != cudaSuccess || h->out.alloc(n_pix) != cudaSuccess ||
      h->sens_point.alloc(n_pix) != cudaSuccess || h->sens_pixel.alloc(n_pix) != cudaSuccess ||
      h->counters.alloc(1) != cudaSuccess) {
    g_create_error = "cudaMalloc(images) failed";
    jpet_strip_destroy(h);
    return JPET_ERR_MEMORY;
  }
  if (launch_fill(h->rho.p, 1.0f, n_pix, h->stream) != cudaSuccess ||
      launch_sensitivity(h->g, 0, h->sens_point.p, h->stream) != cudaSuccess ||
      launch_sensitivity(h->g, 1, h->sens_pixel.p, h->stream) != cudaSuccess ||
      cudaMemsetAsync(h->counters.p, 0, sizeof(DevCounters), h->stream) != cudaSuccess ||
      cudaStreamSynchronize(h->stream) != cudaSuccess) {
    g_create_error = std::string("initialisation kernels failed: ") +
                     cudaGetErrorString(cudaGetLastError());
    jpet_strip_destroy(h);
    return JPET_ERR_CUDA;
  }
  *out = h;
  return JPET_OK;
}

int jpet_strip_destroy(jpet_strip_t* h) {
  if (!h) return JPET_OK;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  h->rho.release();
  h->out.release();
  h->out_lo.release();
  h->out_q.release();
  h->out_sum.release();
  h->sens_point.release();
  h->sens_pixel.release();
  h->raw.release();
  h->tile_count.release();
  h->scratch.release();
  h->set_block.release();
  h->records.release();
  h->nll_acc.release();
  h->nll_parts.release();
  h->counters.release();
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
  delete h;
  return JPET_OK;
}

const char* jpet_strip_last_error(const jpet_strip_t* h) {
  return h ? h->last_error.c_str() : g_create_error.c_str();
}

int jpet_strip_set_stream(jpet_strip_t* h, void* stream) {
  if (!h) return JPET_ERR_ARGUMENT;
  h->stream = stream ? static_cast<cudaStream_t>(stream) : h->own_stream;
  return JPET_OK;
}

int jpet_strip_set_events(jpet_strip_t* h, const float* aos, int64_t n) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (n > 0 && !aos) return h->fail(JPET_ERR_ARGUMENT, "NULL event array");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  return upload_and_prepare(h, nullptr, nullptr, nullptr, aos, n);
}

int jpet_strip_set_events_soa(jpet_strip_t* h, const float* zu, const float* zd,
                              const float* dl, int64_t n) {
  if (!h) return JPET_ERR_ARGUMENT;
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  return upload_and_prepare(h, zu, zd, dl, nullptr, n);
}

int jpet_strip_set_events_device(jpet_strip_t* h, const float* zu, const float* zd,
                                 const float* dl, int64_t n) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (n < 0) return h->fail(JPET_ERR_ARGUMENT, "negative event count");
  if (n > 0 && (!zu || !zd || !dl)) return h->fail(JPET_ERR_ARGUMENT, "NULL event array");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  return prepare_events(h, zu, zd, dl, n);
}

int jpet_strip_set_image(jpet_strip_t* h, const float* rho) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (!rho) return h->fail(JPET_ERR_ARGUMENT, "NULL image");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const size_t bytes = static_cast<size_t>(h->g.n_y) * h->g.n_z * sizeof(float);
  JPET_CUDA(h, cudaMemcpyAsync(h->rho.p, rho, bytes, cudaMemcpyHostToDevice, h->stream),
            "copy image");
  JPET_CUDA(h, cudaStreamSynchronize(h->stream), "copy image");
  h->iterations_done = 0;
  return JPET_OK;
}

int jpet_strip_set_image_device(jpet_strip_t* h, const float* d_rho) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (!d_rho) return h->fail(JPET_ERR_ARGUMENT, "NULL image");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const size_t bytes = static_cast<size_t>(h->g.n_y) * h->g.n_z * sizeof(float);
  JPET_CUDA(h, cudaMemcpyAsync(h->rho.p, d_rho, bytes, cudaMemcpyDeviceToDevice, h->stream),
            "copy image");
  h->iterations_done = 0;
  return JPET_OK;
}

int jpet_strip_iterate(jpet_strip_t* h, int n) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (n < 0) return h->fail(JPET_ERR_ARGUMENT, "negative iteration count");
  if (!h->events_ready) return h->fail(JPET_ERR_STATE, "set_events has not succeeded");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  return iterate_on(h, n, h->stream);
}

int jpet_strip_get_image(jpet_strip_t* h, float* rho) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (!rho) return h->fail(JPET_ERR_ARGUMENT, "NULL image");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const size_t bytes = static_cast<size_t>(h->g.n_y) * h->g.n_z * sizeof(float);
  JPET_CUDA(h, cudaMemcpyAsync(rho, h->rho.p, bytes, cudaMemcpyDeviceToHost, h->stream),
            "copy image");
  JPET_CUDA(h, cudaStreamSynchronize(h->stream), "iteration");
  return JPET_OK;
}

int jpet_strip_image_device(jpet_strip_t* h, const float** d_rho) {
  if (!h || !d_rho) return JPET_ERR_ARGUMENT;
  *d_rho = h->rho.p;
  return JPET_OK;
}

int jpet_strip_get_sensitivity(jpet_strip_t* h, int kind, float* out) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (!out || (kind != 0 && kind != 1)) return h->fail(JPET_ERR_ARGUMENT, "bad sensitivity kind");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  const size_t bytes = static_cast<size_t>(h->g.n_y) * h->g.n_z * sizeof(float);
  JPET_CUDA(h, cudaMemcpyAsync(out, kind == 0 ? h->sens_point.p : h->sens_pixel.p, bytes,
                               cudaMemcpyDeviceToHost, h->stream), "copy sensitivity");
  JPET_CUDA(h, cudaStreamSynchronize(h->stream), "copy sensitivity");
  return JPET_OK;
}

int jpet_strip_get_counters(jpet_strip_t* h, jpet_strip_counters* out) {
  if (!h || !out) return JPET_ERR_ARGUMENT;
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  DevCounters c{};
  JPET_CUDA(h, cudaMemcpyAsync(&c, h->counters.p, sizeof(c), cudaMemcpyDeviceToHost, h->stream),
            "copy counters");
  JPET_CUDA(h, cudaStreamSynchronize(h->stream), "copy counters");
  std::memset(out, 0, sizeof(*out));
  out->n_events = h->n_events;
  out->n_pixels = static_cast<int64_t>(h->total_box_pixels);
  out->n_kernel_calls = static_cast<int64_t>(c.n_kernel_calls) +
                        (h->use_fast && h->counters_valid
                             ? static_cast<int64_t>(h->table_kernel_calls) : 0);
  out->n_contributing = static_cast<int64_t>(c.n_contributing);
  out->n_oversize = h->n_oversize;
  out->n_tiles = h->n_tiles_nonempty;
  out->n_chunks = h->n_chunks;
  out->iterations_done = h->iterations_done;
  out->n_exact_path = static_cast<int64_t>(c.n_exact_path);
  return JPET_OK;
}

int jpet_strip_synchronize(jpet_strip_t* h) {
  if (!h) return JPET_ERR_ARGUMENT;
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  JPET_CUDA(h, cudaStreamSynchronize(h->stream), "stream");
  return JPET_OK;
}

int jpet_strip_nll_grad(jpet_strip_t* h, double sigma_z, double sigma_dl, const float* d_rho,
                        const float* d_sens, double* loss, float* d_grad_rho,
                        double* grad_sigma, int64_t* n_skipped) {
  if (!h) return JPET_ERR_ARGUMENT;
  if (!(sigma_z > 0) || !(sigma_dl > 0))
    return h->fail(JPET_ERR_ARGUMENT, "kernel sigmas must be positive");
  if (!h->events_ready) return h->fail(JPET_ERR_STATE, "set_events has not succeeded");
  if (h->opts.mode != JPET_MODE_CPU_REFERENCE)
    return h->fail(JPET_ERR_UNSUPPORTED, "the likelihood uses the Gaussian kernel (CPU-reference mode)");
  JPET_CUDA(h, cudaSetDevice(h->device), "cudaSetDevice");
  cudaStream_t s = h->stream;
  const size_t n_pix = static_cast<size_t>(h->g.n_y) * h->g.n_z;
  JPET_CUDA(h, h->nll_acc.alloc(4), "cudaMalloc(likelihood)");
  const int32_t n_parts = nll_grad_parts(static_cast<int64_t>(n_pix), h->n_events);
  if (d_grad_rho) JPET_CUDA(h, h->nll_parts.alloc(n_parts * n_pix), "cudaMalloc(gradient)");
  double* parts = d_grad_rho ? h->nll_parts.p : nullptr;
  const float* rho = d_rho ? d_rho : h->rho.p;
  const float* sens = d_sens ? d_sens : h->sens_point.p;
  JPET_CUDA(h, cudaMemsetAsync(h->nll_acc.p, 0, 4 * sizeof(double), s), "memset");
  if (parts) JPET_CUDA(h, cudaMemsetAsync(parts, 0, n_parts * n_pix * sizeof(double), s), "memset");
  const NllConst k = make_nll_const(sigma_z, sigma_dl);
  auto* skipped = reinterpret_cast<unsigned long long*>(h->nll_acc.p + 3);
  JPET_CUDA(h, launch_nll(h->g, k, h->n_sorted, h->sorted_geom.p, h->sorted_box.p,
                          h->use_fast ? h->row_table.p : nullptr, h->tiling.row_stride, rho, parts,
                          n_parts, h->nll_acc.p, skipped, s),
            "likelihood kernel launch");
  JPET_CUDA(h, launch_nll(h->g, k, h->n_oversize, h->over_geom.p, h->over_box.p, nullptr, 0, rho,
                          parts, n_parts, h->nll_acc.p, skipped, s),
            "likelihood kernel launch");
  JPET_CUDA(h, launch_nll_finish(sens, rho, parts, n_parts, d_grad_rho, h->nll_acc.p,
                                 static_cast<int64_t>(n_pix), s),
            "likelihood finish launch");
  double host[4];
  JPET_CUDA(h, cudaMemcpyAsync(host, h->nll_acc.p, sizeof(host), cudaMemcpyDeviceToHost, s),
            "copy likelihood");
  JPET_CUDA(h, cudaStreamSynchronize(s), "likelihood");
  if (loss) *loss = host[0];
  if (grad_sigma) {
    grad_sigma[0] = host[1];
    grad_sigma[1] = host[2];
  }
  unsigned long long sk;
  std::memcpy(&sk, &host[3], sizeof(sk));
  if (n_skipped) *n_skipped = static_cast<int64_t>(sk);
  return JPET_OK;
}

int jpet_strip_run(const jpet_strip_geom* geom, const jpet_strip_opts* opts,
                   const float* responses, int64_t n, float* rho, int n_blocks,
                   int n_iterations_in_block, jpet_strip_output_fn output,
                   jpet_strip_progress_fn progress, void* user, char* device_name,
                   size_t device_name_len) {
  if (!rho || n_blocks < 0 || n_iterations_in_block < 0 || (n > 0 && !responses)) {
    g_create_error = "invalid argument to jpet_strip_run";
    return JPET_ERR_ARGUMENT;
  }
  jpet_strip_t* h = nullptr;
  int rc = jpet_strip_create(geom, opts, &h);
  if (rc != JPET_OK) return rc;
  auto done = [&](int code) {
    if (code != JPET_OK) g_create_error = h->last_error;
    jpet_strip_destroy(h);
    return code;
  };
  if (device_name && device_name_len > 0) {
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, h->device) == cudaSuccess) {
      std::snprintf(device_name, device_name_len, "%s", prop.name);
    } else {
      device_name[0] = 0;
    }
  }
  const int n_z = h->g.n_z, n_y = h->g.n_y;
  std::vector<float> host(static_cast<size_t>(n_z) * n_y);
  // output(-1, sensitivity) first (cuda/reconstruction.cu:63-70)
  if (output) {
    if ((rc = jpet_strip_get_sensitivity(h, 1, host.data())) != JPET_OK) return done(rc);
    output(-1, host.data(), n_z, n_y, user);
  }
  if ((rc = jpet_strip_set_image(h, rho)) != JPET_OK) return done(rc);
  if ((rc = jpet_strip_set_events(h, responses, n)) != JPET_OK) return done(rc);
  for (int block = 0; block < n_blocks; ++block) {
    for (int i = 0; i < n_iterations_in_block; ++i) {
      const int iteration = block * n_iterations_in_block + i;
      if (progress) progress(iteration, 0, user);
      if ((rc = jpet_strip_iterate(h, 1)) != JPET_OK) return done(rc);
      if (progress) {
        if ((rc = jpet_strip_synchronize(h)) != JPET_OK) return done(rc);
        progress(iteration, 1, user);
      }
      // first 5 iterations and 10, 15, 20, 30, 50, 100 (cuda/reconstruction.cu:99-104)
      if (!block && i < n_iterations_in_block - 1 &&
          (i < 5 || i == 9 || i == 14 || i == 19 || i == 29 || i == 49 || i == 99)) {
        if ((rc = jpet_strip_get_image(h, rho)) != JPET_OK) return done(rc);
        if (output) output(i + 1, rho, n_z, n_y, user);
      }
    }
    if ((rc = jpet_strip_get_image(h, rho)) != JPET_OK) return done(rc);
    if (output) output((block + 1) * n_iterations_in_block, rho, n_z, n_y, user);
  }
  if (progress) progress(n_blocks * n_iterations_in_block, 0, user);
  return done(JPET_OK);
}

}  // extern "C"
