// Large copies between the device and a caller's ordinary (pageable) memory.
//
// The driver stages such a copy through its own pinned buffer with one host
// thread, about 10 GB/s, and the first touch of a fresh array's pages comes
// on top. Here a copy goes through two pinned chunks of the state: one is
// filled or emptied by the host's threads while the other crosses PCIe (a
// million uniforms in and outcomes out: about 0.3 ms less of 2.9).
// Memory that is pinned already, and small copies, go straight.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "engine.hpp"
#include "host.hpp"

namespace qvdg {

namespace {

constexpr size_t kChunk = size_t(2) << 20;   // of the two staging buffers
constexpr size_t kPiece = size_t(256) << 10;  // of one host thread at a time
constexpr size_t kDirect = size_t(1) << 20;   // copies up to this size go straight

bool staged(const void* host, size_t bytes) {
  if (bytes <= kDirect) return false;
  cudaPointerAttributes attr{};
  if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return attr.type == cudaMemoryTypeUnregistered;
}

void threaded_copy(char* dst, const char* src, size_t bytes) {
  parallel_for((bytes + kPiece - 1) / kPiece, [&](size_t i) {
    const size_t at = i * kPiece;
    std::memcpy(dst + at, src + at, std::min(kPiece, bytes - at));
  });
}

// Staging buffer k of the state, once the copies that used it are done.
char* buffer(StateImpl& s, size_t k) {
  char* base = static_cast<char*>(s.stage.get(2 * kChunk));
  if (!s.stage_event[k])
    QVDG_CUDA(cudaEventCreateWithFlags(&s.stage_event[k], cudaEventDisableTiming));
  else
    QVDG_CUDA(cudaEventSynchronize(s.stage_event[k]));
  return base + k * kChunk;
}

}  // namespace

void copy_to_host(StateImpl& s, void* dst, const void* src, size_t bytes) {
  if (!staged(dst, bytes)) {
    QVDG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s.stream));
    QVDG_CUDA(cudaStreamSynchronize(s.stream));
    return;
  }
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  auto size = [&](size_t k) { return std::min(kChunk, bytes - k * kChunk); };
  for (size_t k = 0; k <= chunks; ++k) {
    if (k < chunks) {
      char* buf = buffer(s, k & 1);
      QVDG_CUDA(cudaMemcpyAsync(buf, static_cast<const char*>(src) + k * kChunk, size(k), cudaMemcpyDeviceToHost,
                                s.stream));
      QVDG_CUDA(cudaEventRecord(s.stage_event[k & 1], s.stream));
    }
    if (k > 0) threaded_copy(static_cast<char*>(dst) + (k - 1) * kChunk, buffer(s, (k - 1) & 1), size(k - 1));
  }
}

void copy_to_device(StateImpl& s, void* dst, const void* src, size_t bytes) {
  if (!staged(src, bytes)) {
    QVDG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s.stream));
    return;
  }
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  for (size_t k = 0; k < chunks; ++k) {
    const size_t n = std::min(kChunk, bytes - k * kChunk);
    char* buf = buffer(s, k & 1);
    threaded_copy(buf, static_cast<const char*>(src) + k * kChunk, n);
    QVDG_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + k * kChunk, buf, n, cudaMemcpyHostToDevice, s.stream));
    QVDG_CUDA(cudaEventRecord(s.stage_event[k & 1], s.stream));
  }
}

}  // namespace qvdg
