// Copies between pageable host arrays and the GPU by several host threads.
//
// A pageable copy through the runtime is one thread's memcpy into the driver's
// staging buffer (10 GB/s up) or out of it into memory that is touched for
// the first time, page fault by page fault (4.4 GB/s down), against 55 GB/s
// over PCIe.  Large arrays therefore go through two pinned chunks: while one
// is on the link, a few threads copy the other (B200 host, 192^3: set_fields
// 21 -> 10 ms, get_fields into new arrays 52 -> 18 ms).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <string.h>
#include <algorithm>
#include <thread>
#include <vector>

namespace mhit {

// memcpy of `rows` rows of `bytes` bytes, `dpitch` / `spitch` bytes apart, by up
// to 8 threads (one per 2 MB); the threads end with the call.
inline void parallel_copy(void* dst, size_t dpitch, const void* src, size_t spitch, size_t bytes, size_t rows) {
  const size_t total = bytes * rows;
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t nt = std::max<size_t>(1, std::min<size_t>(std::min<size_t>(8, hw), total >> 21));
  // part t copies bytes [total*t/nt, total*(t+1)/nt) of the rows laid end to end
  auto part = [=](size_t t) {
    size_t at = total / nt * t;
    const size_t end = t + 1 == nt ? total : total / nt * (t + 1);
    while (at < end) {
      const size_t r = at / bytes, o = at - r * bytes, len = std::min(bytes - o, end - at);
      memcpy(static_cast<char*>(dst) + r * dpitch + o, static_cast<const char*>(src) + r * spitch + o, len);
      at += len;
    }
  };
  std::thread ts[8];
  size_t started = 1;
  try {
    for (; started < nt; ++started) ts[started] = std::thread(part, started);
  } catch (...) {  // no more threads: the remaining parts are copied here
  }
  part(0);
  for (size_t t = started; t < nt; ++t) part(t);
  for (size_t t = 1; t < started; ++t) ts[t].join();
}

// Two pinned chunks and their events, for one stream's host copies.
struct PinnedChunks {
  static constexpr size_t kBytes = (size_t)16 << 20;
  void* buf[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};
  // Allocated on first use; false where that is not possible (the caller then
  // copies without them).
  bool ready() {
    for (int k = 0; k < 2; ++k) {
      if (!buf[k] && cudaMallocHost(&buf[k], kBytes) != cudaSuccess) buf[k] = nullptr;
      if (!ev[k] && cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming) != cudaSuccess) ev[k] = nullptr;
      if (!buf[k] || !ev[k]) {
        cudaGetLastError();
        return false;
      }
    }
    return true;
  }
  void release() {
    for (int k = 0; k < 2; ++k) {
      if (buf[k]) cudaFreeHost(buf[k]);
      if (ev[k]) cudaEventDestroy(ev[k]);
      buf[k] = nullptr;
      ev[k] = nullptr;
    }
  }
};

// Whether an array is worth the pinned chunks: pageable, and large enough that
// their set-up (two allocations on first use) and the threads pay.
inline bool wants_chunks(const void* host, size_t bytes) {
  if (bytes < ((size_t)8 << 20)) return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace mhit
