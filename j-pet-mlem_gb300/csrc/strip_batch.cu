// Many independent reconstructions in one graph launch (no counterpart in the
// reference, which reconstructs one event set per process).
//
// Every instance is an ordinary handle: its events are binned, sorted and
// prepared by jpet_strip_set_events*.  The batch captures one CUDA graph per
// iteration count: a parallel branch per instance (at most kMaxBranches, the
// largest instances first), each the chain of that instance's iterations, so no
// instance waits for another one's iteration and the tail of one launch overlaps
// the others' work.  A graph holds the handles' buffers; it is captured again
// when a handle's events or current image buffer are no longer those of the
// capture.  (Grouped persistent launches over all instances, one group after
// another with a barrier per iteration, took 2.96 ms per iteration of 12
// instances with 4.1e6 events where the branches take 1.80 ms.)
//
// The autotuner times candidate plans per instance on a prefix of its events with
// the single-handle iteration and keeps the fastest: two tile sides for the
// batch-union kernel (whose batch shape follows from the events), register
// shapes, CTA sizes and tile sides for the row-owned one.  Plans are cached by
// geometry, widths and event-count octave, so instances of the same kind are
// timed once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/jpet_strip.h"
#include "strip_internal.h"

namespace jpet {
int handle_batch_ready(const jpet_strip* h, std::string& why);
const DevGeom& handle_geom(const jpet_strip* h);
const Tiling& handle_tiling(const jpet_strip* h);
uint64_t handle_generation(const jpet_strip* h);
const float* handle_image(const jpet_strip* h);
int handle_launches(const jpet_strip* h);
int handle_capture_iterations(jpet_strip* h, int n, cudaStream_t s);
void handle_batch_done(jpet_strip* h, int n);
int handle_reprepare(jpet_strip* h, int raster_shape, int block_threads, int tile,
                     const float* d_zu, const float* d_zd, const float* d_dl, int64_t n);
const char* handle_error(const jpet_strip* h);
void handle_set_beside(jpet_strip* h, int32_t n);
}  // namespace jpet

using namespace jpet;

namespace {

constexpr int kMaxBranches = 64;  // concurrent instance chains of a graph
constexpr size_t kMaxGraphs = 16; // captured iteration counts and image parities kept

// What a graph was captured for: each handle's prepared events and image buffer.
using Signature = std::vector<std::pair<uint64_t, const float*>>;

struct Captured {
  int n;
  Signature sig;
  cudaGraphExec_t exec;
};

struct RawEvents {
  float* d = nullptr;  // SoA: z_u[n], z_d[n], dl[n]
  int64_t n = 0;
};

using TuneKey = std::tuple<int, int, int, int, int, int>;

__global__ void aos_to_soa_kernel(const float* __restrict__ aos, int64_t n, float* __restrict__ soa) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  soa[i] = aos[3 * i];
  soa[n + i] = aos[3 * i + 1];
  soa[2 * n + i] = aos[3 * i + 2];
}

}  // namespace

struct jpet_strip_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string last_error = "no error";
  std::vector<jpet_strip_t*> h;
  std::vector<RawEvents> raw;
  std::vector<jpet_strip_batch_plan> plan;
  bool fast = true;  // batch-union kernel (else row-owned)
  int block_threads = 0;  // CTA size asked for (plan[] reports the sizes that run)
  std::vector<Captured> graphs;
  int launches = 0;  // kernels per iteration of the last graph
  std::map<TuneKey, std::tuple<int, int, int>> tune_cache;  // shape, CTA threads, tile

  int fail(int code, const std::string& m) {
    last_error = m;
    return code;
  }
  int cuda_fail(cudaError_t e, const char* what) {
    return fail(JPET_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  }
  void drop_graphs() {
    for (auto& c : graphs) cudaGraphExecDestroy(c.exec);
    graphs.clear();
    launches = 0;
  }
};

namespace {

#define BATCH_CUDA(b, expr, what)                       \
  do {                                                  \
    cudaError_t _e = (expr);                            \
    if (_e != cudaSuccess) return (b)->cuda_fail(_e, what); \
  } while (0)

// Captures n iterations of every instance: branches of the batch's stream, the
// instances dealt to them by decreasing event count.
int capture(jpet_strip_batch* b, int n, cudaGraphExec_t* exec) {
  const int n_inst = static_cast<int>(b->h.size());
  const int n_br = std::min(n_inst, kMaxBranches);
  std::vector<int> order(n_inst);
  for (int i = 0; i < n_inst; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return b->raw[x].n > b->raw[y].n; });
  std::vector<cudaStream_t> br(n_br, nullptr);
  std::vector<cudaEvent_t> done(n_br, nullptr);
  cudaEvent_t fork = nullptr;
  cudaError_t e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
  for (int k = 0; k < n_br && e == cudaSuccess; ++k) {
    e = cudaStreamCreateWithFlags(&br[k], cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done[k], cudaEventDisableTiming);
  }
  int rc = JPET_OK;
  cudaGraph_t graph = nullptr;
  if (e == cudaSuccess) e = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    e = cudaEventRecord(fork, b->stream);
    for (int k = 0; k < n_br && e == cudaSuccess; ++k) e = cudaStreamWaitEvent(br[k], fork, 0);
    for (int i = 0; i < n_inst && e == cudaSuccess && rc == JPET_OK; ++i) {
      rc = handle_capture_iterations(b->h[order[i]], n, br[i % n_br]);
      if (rc != JPET_OK) b->fail(rc, handle_error(b->h[order[i]]));
    }
    for (int k = 0; k < n_br && e == cudaSuccess; ++k) {
      e = cudaEventRecord(done[k], br[k]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(b->stream, done[k], 0);
    }
    const cudaError_t e2 = cudaStreamEndCapture(b->stream, &graph);
    if (e == cudaSuccess) e = e2;
  }
  if (e == cudaSuccess && rc == JPET_OK) e = cudaGraphInstantiate(exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  for (int k = 0; k < n_br; ++k) {
    if (done[k]) cudaEventDestroy(done[k]);
    if (br[k]) cudaStreamDestroy(br[k]);
  }
  if (fork) cudaEventDestroy(fork);
  if (rc != JPET_OK) return rc;
  if (e != cudaSuccess) return b->cuda_fail(e, "graph capture");
  return JPET_OK;
}

}  // namespace

extern "C" {

int jpet_strip_batch_create(int32_t n, const jpet_strip_geom* geoms, const jpet_strip_opts* opts,
                            jpet_strip_batch_t** out) {
  if (!out || n <= 0 || !geoms) {
    set_call_error("jpet_strip_batch_create: invalid argument");
    return JPET_ERR_ARGUMENT;
  }
  *out = nullptr;
  jpet_strip_opts o;
  jpet_strip_default_opts(&o);
  if (opts) o = *opts;
  if (o.mode != JPET_MODE_CPU_REFERENCE ||
      (o.variant != JPET_VARIANT_FAST && o.variant != JPET_VARIANT_ROWS) ||
      o.precision != JPET_PRECISION_FP32) {
    set_call_error("jpet_strip_batch_create: batches run the FP32 batch-union or row-owned kernel "
                   "(CPU-reference mode, FAST or ROWS variant)");
    return JPET_ERR_UNSUPPORTED;
  }
  auto* b = new jpet_strip_batch();
  b->fast = o.variant == JPET_VARIANT_FAST;
  b->block_threads = o.block_threads;
  b->device = o.device;
  cudaError_t e = cudaSetDevice(o.device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    set_call_error(std::string("jpet_strip_batch_create: ") + cudaGetErrorString(e));
    delete b;
    return JPET_ERR_CUDA;
  }
  b->h.assign(n, nullptr);
  b->raw.assign(n, RawEvents{});
  b->plan.assign(n, jpet_strip_batch_plan{});
  for (int i = 0; i < n; ++i) {
    const int rc = jpet_strip_create(&geoms[i], &o, &b->h[i]);
    if (rc == JPET_OK) {
      jpet_strip_set_stream(b->h[i], b->stream);
      handle_set_beside(b->h[i], n);
    }
    if (rc != JPET_OK) {
      jpet_strip_batch_destroy(b);
      return rc;
    }
    b->plan[i].raster_shape = o.raster_shape;
    b->plan[i].block_threads = o.block_threads;
  }
  *out = b;
  return JPET_OK;
}

int jpet_strip_batch_destroy(jpet_strip_batch_t* b) {
  if (!b) return JPET_OK;
  cudaSetDevice(b->device);
  b->drop_graphs();
  for (auto* x : b->h)
    if (x) jpet_strip_destroy(x);
  for (auto& r : b->raw) cudaFree(r.d);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return JPET_OK;
}

const char* jpet_strip_batch_last_error(const jpet_strip_batch_t* b) {
  return b ? b->last_error.c_str() : "NULL batch";
}

int jpet_strip_batch_size(const jpet_strip_batch_t* b) {
  return b ? static_cast<int>(b->h.size()) : 0;
}

int jpet_strip_batch_instance(jpet_strip_batch_t* b, int32_t i, jpet_strip_t** h) {
  if (!b || !h || i < 0 || i >= static_cast<int32_t>(b->h.size())) return JPET_ERR_ARGUMENT;
  *h = b->h[i];
  return JPET_OK;
}

int jpet_strip_batch_set_events(jpet_strip_batch_t* b, int32_t i, const float* aos, int64_t n,
                                int32_t on_device) {
  if (!b) return JPET_ERR_ARGUMENT;
  if (i < 0 || i >= static_cast<int32_t>(b->h.size()) || n < 0 || (n > 0 && !aos))
    return b->fail(JPET_ERR_ARGUMENT, "jpet_strip_batch_set_events: invalid argument");
  BATCH_CUDA(b, cudaSetDevice(b->device), "cudaSetDevice");
  b->drop_graphs();
  RawEvents& r = b->raw[i];
  cudaFree(r.d);
  r.d = nullptr;
  r.n = n;
  if (n > 0) {
    // keep a device SoA copy so that the tuner can re-bin the events
    const size_t bytes = static_cast<size_t>(n) * 3 * sizeof(float);
    BATCH_CUDA(b, cudaMalloc(&r.d, bytes), "cudaMalloc(events)");
    float* staging = nullptr;
    const float* src = aos;
    if (!on_device) {
      BATCH_CUDA(b, cudaMalloc(&staging, bytes), "cudaMalloc(events)");
      cudaError_t e = cudaMemcpyAsync(staging, aos, bytes, cudaMemcpyHostToDevice, b->stream);
      if (e != cudaSuccess) {
        cudaFree(staging);
        return b->cuda_fail(e, "copy events");
      }
      src = staging;
    }
    aos_to_soa_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, b->stream>>>(src, n, r.d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    cudaFree(staging);
    if (e != cudaSuccess) return b->cuda_fail(e, "events to SoA");
  }
  const int rc = jpet_strip_set_events_device(b->h[i], r.d, r.d + n, r.d + 2 * n, n);
  if (rc != JPET_OK) return b->fail(rc, handle_error(b->h[i]));
  return JPET_OK;
}

int jpet_strip_batch_tune(jpet_strip_batch_t* b, int64_t max_tune_events) {
  if (!b) return JPET_ERR_ARGUMENT;
  BATCH_CUDA(b, cudaSetDevice(b->device), "cudaSetDevice");
  b->drop_graphs();
  if (max_tune_events <= 0) max_tune_events = 262144;
  cudaEvent_t e0, e1;
  BATCH_CUDA(b, cudaEventCreate(&e0), "event");
  BATCH_CUDA(b, cudaEventCreate(&e1), "event");
  int rc = JPET_OK;
  for (size_t i = 0; i < b->h.size() && rc == JPET_OK; ++i) {
    jpet_strip_t* h = b->h[i];
    const RawEvents& r = b->raw[i];
    {
      std::string why;
      if (handle_batch_ready(h, why) != JPET_OK) {
        rc = b->fail(JPET_ERR_STATE, "instance " + std::to_string(i) + ": " + why);
        break;
      }
    }
    const DevGeom gv = handle_geom(h);
    const int octave = r.n > 0 ? static_cast<int>(std::log2(static_cast<double>(r.n))) : 0;
    const TuneKey key{gv.n_y, gv.n_z, static_cast<int>(std::lround(gv.pixel_width * 100)),
                      static_cast<int>(std::lround(gv.sigma_z * 2)),
                      static_cast<int>(std::lround(gv.sigma_dl)), octave};
    const int64_t nt = std::min<int64_t>(r.n, max_tune_events);
    auto hit = b->tune_cache.find(key);
    int best_shape = 0, best_threads = b->fast ? b->block_threads : 128, best_tile = 0;
    double best_ms = 1e30;
    int n_cand = 0;
    if (hit != b->tune_cache.end()) {
      std::tie(best_shape, best_threads, best_tile) = hit->second;
    } else if (nt > 0) {
      // candidates: the automatic square tile of the CTA's window budget or one of
      // half its side; for the row-owned kernel also the automatic register shape
      // and the next larger one, with 4- and 8-warp CTAs
      std::vector<int> shapes, sizes{128, 256};
      if (b->fast) {
        shapes.push_back(JPET_RASTER_AUTO);
        sizes.assign(1, best_threads);
      } else {
        rc = handle_reprepare(h, JPET_RASTER_AUTO, 128, 0, r.d, r.d + r.n, r.d + 2 * r.n, nt);
        if (rc != JPET_OK) break;
        const int auto_shape = handle_tiling(h).rows_shape + 1;  // JPET_RASTER_* numbering
        shapes.push_back(auto_shape);
        if (auto_shape < JPET_RASTER_4x2x4) shapes.push_back(auto_shape + 1);
      }
      for (int shape : shapes) {
        for (int threads : sizes) {
          int auto_tile = 0;
          for (int tile_pass = 0; tile_pass < 2 && rc == JPET_OK; ++tile_pass) {
            int tile = 0;
            if (tile_pass == 1) {
              tile = auto_tile / 2;
              if (tile < 8) break;
            }
            rc = handle_reprepare(h, shape, threads, tile, r.d, r.d + r.n, r.d + 2 * r.n, nt);
            if (rc != JPET_OK) break;
            if (tile_pass == 0)
              auto_tile = std::min(handle_tiling(h).tile_w, handle_tiling(h).tile_h);
            rc = jpet_strip_iterate(h, 1);  // warm-up
            if (rc != JPET_OK) break;
            BATCH_CUDA(b, cudaEventRecord(e0, b->stream), "event");
            rc = jpet_strip_iterate(h, 3);
            if (rc != JPET_OK) break;
            BATCH_CUDA(b, cudaEventRecord(e1, b->stream), "event");
            BATCH_CUDA(b, cudaEventSynchronize(e1), "event");
            float ms = 0;
            BATCH_CUDA(b, cudaEventElapsedTime(&ms, e0, e1), "event");
            ++n_cand;
            if (ms / 3 < best_ms) {
              best_ms = ms / 3;
              best_shape = shape;
              best_threads = threads;
              best_tile = tile;
            }
          }
          if (rc != JPET_OK) break;
        }
        if (rc != JPET_OK) break;
      }
      if (rc != JPET_OK) break;
      b->tune_cache[key] = std::make_tuple(best_shape, best_threads, best_tile);
    }
    // the chosen plan on all of the instance's events, from a uniform image
    rc = handle_reprepare(h, best_shape, best_threads, best_tile, r.d, r.d + r.n, r.d + 2 * r.n,
                          r.n);
    if (rc != JPET_OK) break;
    std::vector<float> ones(static_cast<size_t>(gv.n_y) * gv.n_z, 1.0f);
    rc = jpet_strip_set_image(h, ones.data());
    if (rc != JPET_OK) break;
    // the batch-union kernel's batch shape follows from the boxes: reported as the
    // register shape that covers them and the CTA size class
    b->plan[i].raster_shape = b->fast ? handle_tiling(h).rows_shape + 1 : best_shape;
    b->plan[i].block_threads =
        b->fast ? (union_ops(handle_tiling(h).union_shape).threads > 128 ? 256 : 128)
                : best_threads;
    b->plan[i].tile = best_tile;
    b->plan[i].tuned_ms_per_iteration = best_ms < 1e30 ? best_ms : -1.0;
    b->plan[i].tuned_events = nt;
    b->plan[i].candidates = n_cand;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc != JPET_OK && b->last_error == "no error") b->last_error = "tuning failed";
  if (rc != JPET_OK) {
    for (auto* x : b->h)
      if (std::string(handle_error(x)) != "no error") {
        b->last_error = std::string("tuning: ") + handle_error(x);
        break;
      }
  }
  return rc;
}

int jpet_strip_batch_plan_of(const jpet_strip_batch_t* b, int32_t i, jpet_strip_batch_plan* p) {
  if (!b || !p || i < 0 || i >= static_cast<int32_t>(b->h.size())) return JPET_ERR_ARGUMENT;
  *p = b->plan[i];
  return JPET_OK;
}

int jpet_strip_batch_iterate(jpet_strip_batch_t* b, int32_t n) {
  if (!b) return JPET_ERR_ARGUMENT;
  if (n < 0) return b->fail(JPET_ERR_ARGUMENT, "negative iteration count");
  if (n == 0) return JPET_OK;
  BATCH_CUDA(b, cudaSetDevice(b->device), "cudaSetDevice");
  Signature sig;
  for (size_t i = 0; i < b->h.size(); ++i) {
    std::string why;
    const int rc = handle_batch_ready(b->h[i], why);
    if (rc != JPET_OK) return b->fail(rc, "instance " + std::to_string(i) + ": " + why);
    sig.emplace_back(handle_generation(b->h[i]), handle_image(b->h[i]));
  }
  // graphs of replaced event sets hold freed buffers: they go
  for (const auto& c : b->graphs) {
    bool stale = false;
    for (size_t i = 0; i < sig.size(); ++i) stale = stale || c.sig[i].first != sig[i].first;
    if (stale) {
      b->drop_graphs();
      break;
    }
  }
  auto it = std::find_if(b->graphs.begin(), b->graphs.end(),
                         [&](const Captured& c) { return c.n == n && c.sig == sig; });
  if (it == b->graphs.end()) {
    if (b->graphs.size() >= kMaxGraphs) b->drop_graphs();
    cudaGraphExec_t exec = nullptr;
    const int rc = capture(b, n, &exec);
    if (rc != JPET_OK) return rc;
    b->graphs.push_back(Captured{n, sig, exec});
    it = b->graphs.end() - 1;
  }
  b->launches = 0;
  for (auto* x : b->h) b->launches += handle_launches(x);
  BATCH_CUDA(b, cudaGraphLaunch(it->exec, b->stream), "graph launch");
  BATCH_CUDA(b, cudaStreamSynchronize(b->stream), "batched iterations");
  for (auto* x : b->h) handle_batch_done(x, n);
  return JPET_OK;
}

int jpet_strip_batch_launches_per_iteration(const jpet_strip_batch_t* b) {
  return b ? b->launches : 0;
}

}  // extern "C"
