// Host side of the batched layered-circuit launch: validation, packing,
// work order, the autotuner, graph capture and replay.

#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "batch_plan.hpp"
#include "engine.hpp"

struct qvdg_batch {
  int device = 0;
  int sms = 148;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::vector<qvdg::BatchCircuit> circuits;
  uint64_t num_matrices = 0, outputs = 0;
  uint32_t max_qubits = 0;
  void* dev = nullptr;      // circuits | gates | matrices | out
  double* matrices = nullptr;  // in dev: the complex128 matrices last given
  // Work of the chosen shape, and of the autotuner's sample: tasks | wide | queue.
  void* work = nullptr;
  void* slots = nullptr;    // states of wide circuits
  void* partials = nullptr;
  double* host_out = nullptr;  // pinned: the outputs, then the status word
  qvdg::BatchLaunch launch;    // the chosen shape, whole batch
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<uint32_t> tune_tiles, tune_threads;
  std::vector<double> tune_seconds;
  double tune_host_seconds = 0.0;
};

namespace qvdg {

namespace {

constexpr int kTileMin = 12, kTileMax = 14;
constexpr int kMaxCtasPerSm = 4;
constexpr size_t kSlotBudget = size_t(8) << 30;  // of wide circuits' states at a time

void require(bool ok, const std::string& message) {
  if (!ok) throw Error(QVDG_ERR_INVALID, message);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Whether a tile shape can run every circuit: wide circuits (n > L) run on
// tiles of min(L, 13) qubits (batch_plan.cpp), and pass B's needs two low
// qubits or more below the high ones: n <= 2 L - 3 for L = 12 and 13, and every
// n up to kBatchMaxQubits for L = 14.
bool shape_fits(uint32_t max_qubits, int L) { return max_qubits <= uint32_t(L) || max_qubits <= uint32_t(2 * L - 3); }

// Persistent CTAs for a shape: all resident CTAs (at most kMaxCtasPerSm per SM).
int ctas_for(const qvdg_batch* b, int threads, int L) {
  return b->sms * std::min(batch_kernel_occupancy(threads, L), kMaxCtasPerSm);
}

// Plans the circuits of `order` on a shape and puts their work on the device
// (an allocation of its own in *work, replacing what it held). The circuits'
// `wide` fields follow.
BatchLaunch shape(qvdg_batch* b, const BatchLaunch& base, const std::vector<uint32_t>& order, int L, int threads,
                  int ctas, size_t slots, uint64_t slot_elems, void** work) {
  const BatchWork w = plan_batch(b->circuits, order, L, ctas, std::max<size_t>(slots, 1), slot_elems);
  require(w.tasks.size() < (size_t(1) << 31), "the batch has too many tiles");
  BatchLaunch l = base;
  l.tile_qubits = L;
  l.threads = threads;
  l.ctas = ctas;
  l.count = uint32_t(w.tasks.size());
  const size_t o_tasks = 0;
  const size_t o_wide = align256(o_tasks + w.tasks.size() * sizeof(BatchTask));
  const size_t o_queue = align256(o_wide + std::max<size_t>(w.wide.size(), 1) * sizeof(BatchWide));
  const size_t queue_bytes = 256 + std::max<size_t>(w.wide.size(), 1) * sizeof(uint32_t);
  QVDG_CUDA(cudaStreamSynchronize(b->stream));
  if (*work) cudaFree(*work);
  *work = nullptr;
  QVDG_CUDA(device_malloc(work, o_queue + queue_bytes));
  char* d = static_cast<char*>(*work);
  QVDG_CUDA(cudaMemcpyAsync(d + o_tasks, w.tasks.data(), w.tasks.size() * sizeof(BatchTask), cudaMemcpyHostToDevice,
                            b->stream));
  if (!w.wide.empty())
    QVDG_CUDA(cudaMemcpyAsync(d + o_wide, w.wide.data(), w.wide.size() * sizeof(BatchWide), cudaMemcpyHostToDevice,
                              b->stream));
  for (uint32_t i : order) b->circuits[i].wide = w.wide_of[i];
  QVDG_CUDA(cudaMemcpyAsync(const_cast<BatchCircuit*>(l.circuits), b->circuits.data(),
                            b->circuits.size() * sizeof(BatchCircuit), cudaMemcpyHostToDevice, b->stream));
  // The circuits' forms are written with their records.
  launch_batch_encode(l, b->matrices, uint32_t(b->circuits.size()), b->stream);
  QVDG_CUDA(cudaStreamSynchronize(b->stream));  // the host copies go out of scope
  l.tasks = reinterpret_cast<const BatchTask*>(d + o_tasks);
  l.wide = reinterpret_cast<const BatchWide*>(d + o_wide);
  l.queue = reinterpret_cast<uint32_t*>(d + o_queue);
  l.status = reinterpret_cast<int*>(d + o_queue + 128);
  l.done = reinterpret_cast<uint32_t*>(d + o_queue + 256);
  l.queue_bytes = queue_bytes;
  return l;
}

double time_launch(qvdg_batch* b, const BatchLaunch& l) {
  launch_batch(l, b->stream);  // warm
  QVDG_CUDA(cudaEventRecord(b->ev0, b->stream));
  launch_batch(l, b->stream);
  QVDG_CUDA(cudaEventRecord(b->ev1, b->stream));
  QVDG_CUDA(cudaEventSynchronize(b->ev1));
  float ms = 0.f;
  QVDG_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
  return ms * 1e-3;
}

void release(qvdg_batch* b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->dev) cudaFree(b->dev);
  if (b->work) cudaFree(b->work);
  if (b->slots) cudaFree(b->slots);
  if (b->partials) cudaFree(b->partials);
  if (b->host_out) cudaFreeHost(b->host_out);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->stream) cudaStreamDestroy(b->stream);
}

}  // namespace

qvdg_batch* batch_create(const qvdg_layered_circuit* circuits, size_t count, const qvdg_batch_options* options) {
  require(circuits != nullptr && count > 0, "empty batch");
  require(count < (size_t(1) << 31), "too many circuits");
  uint32_t want_tile = options ? options->tile_qubits : 0, want_threads = options ? options->threads : 0;
  require(want_tile == 0 || (want_tile >= uint32_t(kTileMin) && want_tile <= uint32_t(kTileMax)),
          "tile_qubits must be 0 or 12..14");
  require(want_threads == 0 || want_threads == 128 || want_threads == 256 || want_threads == 512,
          "threads must be 0, 128, 256 or 512");
  auto* b = new qvdg_batch();
  try {
    // Validate and pack.
    b->circuits.resize(count);
    for (size_t i = 0; i < count; ++i) {
      const qvdg_layered_circuit& c = circuits[i];
      require(c.num_qubits >= 1 && c.num_qubits <= uint32_t(kBatchMaxQubits),
              "circuit " + std::to_string(i) + ": num_qubits must be 1.." + std::to_string(kBatchMaxQubits));
      require(c.entangler <= QVDG_ENTANGLE_CZ_LADDER, "circuit " + std::to_string(i) + ": unknown entangler");
      require(c.num_layers == 0 || c.gates != nullptr, "circuit " + std::to_string(i) + ": null gates");
      BatchCircuit& d = b->circuits[i];
      d.num_qubits = c.num_qubits;
      d.num_layers = c.num_layers;
      d.entangler = c.entangler;
      d.form = 0;
      d.gates = b->num_matrices;
      d.out = b->outputs;
      b->num_matrices += uint64_t(c.num_layers) * c.num_qubits;
      b->outputs += c.num_qubits;
      b->max_qubits = std::max(b->max_qubits, c.num_qubits);
    }
    if (want_tile) require(shape_fits(b->max_qubits, int(want_tile)), "tile_qubits too small for the widest circuit");
    std::vector<double> matrices(b->num_matrices * 8);
    for (size_t i = 0; i < count; ++i)
      if (circuits[i].num_layers)
        std::memcpy(matrices.data() + 8 * b->circuits[i].gates, circuits[i].gates,
                    size_t(circuits[i].num_layers) * circuits[i].num_qubits * 8 * sizeof(double));
    // Largest first: an atomic counter then hands out work longest-first.
    std::vector<uint32_t> order(count);
    std::iota(order.begin(), order.end(), 0u);
    auto cost = [&](uint32_t i) {
      const BatchCircuit& c = b->circuits[i];
      return double(uint64_t(1) << c.num_qubits) * double(c.num_layers + 1) * double(c.num_qubits);
    };
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return cost(x) > cost(y); });
    std::vector<uint32_t> sample;
    const size_t stride = count >= 64 ? 8 : 1;
    for (size_t i = 0; i < count; i += stride) sample.push_back(order[i]);

    QVDG_CUDA(cudaGetDevice(&b->device));
    QVDG_CUDA(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device));
    QVDG_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    QVDG_CUDA(cudaEventCreate(&b->ev0));
    QVDG_CUDA(cudaEventCreate(&b->ev1));
    const size_t o_circ = 0;
    const size_t o_gates = align256(o_circ + count * sizeof(BatchCircuit));
    const size_t o_mats = align256(o_gates + std::max<size_t>(b->num_matrices, 1) * kBatchGateSlots * sizeof(float2));
    const size_t o_out = align256(o_mats + std::max<size_t>(matrices.size(), 1) * sizeof(double));
    const size_t total = o_out + b->outputs * sizeof(double);
    QVDG_CUDA(device_malloc(&b->dev, total));
    char* base = static_cast<char*>(b->dev);
    b->matrices = reinterpret_cast<double*>(base + o_mats);
    if (!matrices.empty())
      QVDG_CUDA(cudaMemcpyAsync(b->matrices, matrices.data(), matrices.size() * sizeof(double),
                                cudaMemcpyHostToDevice, b->stream));
    QVDG_CUDA(cudaMallocHost(&b->host_out, (b->outputs + 1) * sizeof(double)));

    BatchLaunch whole;
    whole.circuits = reinterpret_cast<const BatchCircuit*>(base + o_circ);
    whole.gates = reinterpret_cast<const float2*>(base + o_gates);
    whole.out = reinterpret_cast<double*>(base + o_out);

    // Candidate shapes.
    struct Shape {
      int L, threads, ctas;
    };
    std::vector<Shape> shapes;
    for (int L = kTileMin; L <= kTileMax; ++L)
      for (int t : {128, 256, 512}) {
        if (want_tile && L != int(want_tile)) continue;
        if (want_threads && t != int(want_threads)) continue;
        if (!shape_fits(b->max_qubits, L)) continue;
        const int ctas = ctas_for(b, t, L);
        if (ctas > 0) shapes.push_back({L, t, ctas});
      }
    if (shapes.empty()) throw Error(QVDG_ERR_UNSUPPORTED, "no tile shape can run this batch on this device");
    // Slots for as many wide circuits as the budget holds, at least one, and
    // fewer where the device has less memory; the last pass's sums per tile.
    const uint64_t slot_elems = uint64_t(1) << b->max_qubits;
    size_t slots = 0, partials = 0;
    for (const Shape& s : shapes) {
      slots = std::max(slots, wide_count(b->circuits, order, s.L));
      partials = std::max<size_t>(partials, plan_batch(b->circuits, order, s.L, s.ctas, 1, slot_elems).partials);
    }
    if (slots) {
      slots = std::min<size_t>(slots, std::max<size_t>(1, kSlotBudget / (slot_elems * sizeof(float2))));
      while (device_malloc(&b->slots, slots * slot_elems * sizeof(float2)) != cudaSuccess) {
        cudaGetLastError();
        b->slots = nullptr;
        if (slots == 1) throw Error(QVDG_ERR_OUT_OF_MEMORY, "cannot allocate the batch's device memory");
        slots /= 2;
      }
      QVDG_CUDA(device_malloc(&b->partials, std::max<size_t>(partials, 1) * sizeof(double)));
    }
    whole.slots = static_cast<float2*>(b->slots);
    whole.partials = static_cast<double*>(b->partials);

    Shape best = shapes[0];
    if (shapes.size() > 1) {
      const auto t0 = std::chrono::steady_clock::now();
      double best_s = 1e300;
      for (const Shape& s : shapes) {
        const double sec =
            time_launch(b, shape(b, whole, sample, s.L, s.threads, s.ctas, slots, slot_elems, &b->work));
        b->tune_tiles.push_back(uint32_t(s.L));
        b->tune_threads.push_back(uint32_t(s.threads));
        b->tune_seconds.push_back(sec);
        if (sec < best_s) {
          best_s = sec;
          best = s;
        }
      }
      b->tune_host_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    b->launch = shape(b, whole, order, best.L, best.threads, best.ctas, slots, slot_elems, &b->work);

    // Capture: reset the counter, the persistent launch, results to pinned host memory.
    QVDG_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    launch_batch(b->launch, b->stream);
    QVDG_CUDA(cudaMemcpyAsync(b->host_out, b->launch.out, b->outputs * sizeof(double), cudaMemcpyDeviceToHost,
                              b->stream));
    QVDG_CUDA(cudaMemcpyAsync(b->host_out + b->outputs, b->launch.status, sizeof(int), cudaMemcpyDeviceToHost,
                              b->stream));
    QVDG_CUDA(cudaStreamEndCapture(b->stream, &b->graph));
    QVDG_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
    return b;
  } catch (...) {
    cudaStreamCaptureStatus st;
    if (b->stream && cudaStreamIsCapturing(b->stream, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(b->stream, &g);
      if (g) cudaGraphDestroy(g);
    }
    cudaGetLastError();
    release(b);
    delete b;
    throw;
  }
}

void batch_destroy(qvdg_batch* b) {
  if (!b) return;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  release(b);
  delete b;
}

void batch_set_gates(qvdg_batch* b, const double* gates, size_t num_matrices) {
  require(b != nullptr, "null batch");
  require(num_matrices == b->num_matrices, "expected " + std::to_string(b->num_matrices) + " matrices");
  require(gates != nullptr || num_matrices == 0, "null gates");
  if (num_matrices == 0) return;
  // The records and forms follow the new matrices, on the device (encoding
  // them on the host took most of a call that sets and runs a batch).
  QVDG_CUDA(cudaSetDevice(b->device));
  QVDG_CUDA(cudaMemcpyAsync(b->matrices, gates, num_matrices * 8 * sizeof(double), cudaMemcpyHostToDevice, b->stream));
  launch_batch_encode(b->launch, b->matrices, uint32_t(b->circuits.size()), b->stream);
  QVDG_CUDA(cudaStreamSynchronize(b->stream));
}

void batch_run(qvdg_batch* b, double* expect_z, size_t count, double* seconds) {
  require(b != nullptr, "null batch");
  require(expect_z != nullptr, "null output");
  require(count >= b->outputs, "output holds " + std::to_string(count) + " values, the batch has " +
                                   std::to_string(b->outputs));
  QVDG_CUDA(cudaSetDevice(b->device));
  QVDG_CUDA(cudaEventRecord(b->ev0, b->stream));
  QVDG_CUDA(cudaGraphLaunch(b->exec, b->stream));
  QVDG_CUDA(cudaEventRecord(b->ev1, b->stream));
  QVDG_CUDA(cudaEventSynchronize(b->ev1));
  QVDG_CUDA(cudaGetLastError());
  float ms = 0.f;
  QVDG_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
  int gave_up = 0;
  std::memcpy(&gave_up, b->host_out + b->outputs, sizeof(int));
  if (gave_up) throw Error(QVDG_ERR_TIMEOUT, "a task of the batch gave up waiting for the tiles it reads");
  if (seconds) *seconds = ms * 1e-3;
  std::memcpy(expect_z, b->host_out, b->outputs * sizeof(double));
}

void batch_info(const qvdg_batch* b, qvdg_batch_summary* info) {
  require(b != nullptr && info != nullptr, "null argument");
  info->tile_qubits = uint32_t(b->launch.tile_qubits);
  info->threads = uint32_t(b->launch.threads);
  info->ctas = uint32_t(b->launch.ctas);
  info->candidates = uint32_t(b->tune_seconds.size());
  info->circuits = b->circuits.size();
  info->outputs = b->outputs;
  info->tune_seconds = b->tune_host_seconds;
}

size_t batch_tuning(const qvdg_batch* b, uint32_t* tile_qubits, uint32_t* threads, double* seconds,
                    size_t capacity) {
  require(b != nullptr, "null batch");
  const size_t n = b->tune_seconds.size();
  for (size_t i = 0; i < std::min(n, capacity); ++i) {
    if (tile_qubits) tile_qubits[i] = b->tune_tiles[i];
    if (threads) threads[i] = b->tune_threads[i];
    if (seconds) seconds[i] = b->tune_seconds[i];
  }
  return n;
}

}  // namespace qvdg
