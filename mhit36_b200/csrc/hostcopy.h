// Copies between pageable host arrays and the GPU by several host threads.
//
// A pageable copy through the runtime is one thread's memcpy into the driver's
// staging buffer (10 GB/s up) or out of it into memory that is touched for
// the first time, page fault by page fault (4.4 GB/s down), against 55 GB/s
// over PCIe.  Large arrays therefore go through pinned pieces, one per thread:
// while some are on the link, other threads copy theirs.
//
// Pinning takes about 1 ms per MB inside the first such copy of a handle, all of
// which a program that runs one simulation pays, so the pieces together are an
// eighth of a field (8 MB from 192^3, 16 at 256^3, 32 from 384^3).  B200 host,
// four FP64 fields, ms, one thread -> two 16 MB chunks copied by threads -> pieces:
//   first set_fields   192^3 21 -> 44 -> 21, 256^3 49 -> 56 -> 40, 512^3 400 -> 238 -> 146
//   a later one        192^3 21 -> 10 -> 9,  256^3 49 -> 15 -> 16, 512^3 404 -> 118 -> 92
//   get_fields (new arrays)   48 -> 18 -> 14,    112 -> 37 -> 31,       877 -> 268 -> 186
// Other choices, a later call: pieces of 1 MB at 512^3, set_fields 135; of 256
// KB at 256^3, 26; four threads at 192^3, get_fields 22; events that block
// instead of spinning at 192^3, set_fields 29.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <string.h>
#include <algorithm>
#include <atomic>
#include <thread>

namespace mhit {

// memcpy by up to 8 threads (one per 2 MB), which end with the call.
inline void parallel_copy(void* dst, const void* src, size_t total) {
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t nt = std::max<size_t>(1, std::min<size_t>(std::min<size_t>(8, hw), total >> 21));
  // part t copies bytes [total/nt*t, total/nt*(t+1))
  auto part = [=](size_t t) {
    const size_t at = total / nt * t, end = t + 1 == nt ? total : total / nt * (t + 1);
    memcpy(static_cast<char*>(dst) + at, static_cast<const char*>(src) + at, end - at);
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

// A host array of rows of `bytes` bytes, `pitch` bytes apart, addressed by the
// offset into its rows laid end to end.
struct HostRows {
  char* base;
  size_t bytes, pitch;
  void read(void* dst, size_t at, size_t len) const { each(at, len, static_cast<char*>(dst), false); }
  void write(const void* src, size_t at, size_t len) const {
    each(at, len, static_cast<char*>(const_cast<void*>(src)), true);
  }

 private:
  void each(size_t at, size_t len, char* buf, bool out) const {
    while (len) {
      const size_t r = at / bytes, o = at - r * bytes, part = std::min(bytes - o, len);
      char* const here = base + r * pitch + o;
      if (out) memcpy(here, buf, part);
      else memcpy(buf, here, part);
      buf += part;
      at += part;
      len -= part;
    }
  }
};

// The pinned pieces of one stream's host copies, one per thread, and their events.
class PinnedPieces {
 public:
  static constexpr int kThreads = 8;

  // Bytes of a piece for arrays of `total` bytes: 1, 2 or 4 MB, about 1/64.
  static size_t piece_for(size_t total) {
    size_t p = (size_t)1 << 20;
    while (p < ((size_t)4 << 20) && 2 * p <= total / 64) p *= 2;
    return p;
  }
  size_t piece() const { return piece_; }

  // Allocated on first use, for arrays of `total` bytes; false where that is
  // not possible (the caller then copies without them).
  bool ready(size_t total) {
    if (!buf_) {
      piece_ = piece_for(total);
      if (cudaMallocHost(&buf_, kThreads * piece_) != cudaSuccess) buf_ = nullptr;
    }
    bool ok = buf_ != nullptr;
    for (cudaEvent_t& e : ev_) {
      if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) e = nullptr;
      ok = ok && e;
    }
    if (!ok) cudaGetLastError();
    return ok;
  }
  void release() {
    if (buf_) cudaFreeHost(buf_);
    buf_ = nullptr;
    for (cudaEvent_t& e : ev_) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
  }

  // f(thread, buffer, event, offset, length) for every piece of `total` bytes,
  // each by whichever thread is free; a thread's buffer and event are its own.
  // Returns the first error, after which no further piece is begun.
  template <class F> cudaError_t run(int device, size_t total, const F& f) {
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
    const int nt = (int)std::min<size_t>(std::min(kThreads, hw), (total + piece_ - 1) / piece_);
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    auto work = [&](int t) {
      while (err.load() == (int)cudaSuccess) {
        const size_t at = next.fetch_add(piece_);
        if (at >= total) return;
        const cudaError_t e = f(t, static_cast<char*>(buf_) + t * piece_, ev_[t], at, std::min(piece_, total - at));
        int none = (int)cudaSuccess;
        if (e != cudaSuccess) err.compare_exchange_strong(none, (int)e);
      }
    };
    std::thread ts[kThreads];
    int started = 1;
    try {
      for (; started < nt; ++started)
        ts[started] = std::thread([&work, device, t = started] {
          if (cudaSetDevice(device) == cudaSuccess) work(t);
        });
    } catch (...) {  // no more threads: the others take its pieces
    }
    work(0);
    for (int t = 1; t < started; ++t) ts[t].join();
    return (cudaError_t)err.load();
  }

 private:
  void* buf_ = nullptr;
  size_t piece_ = 0;
  cudaEvent_t ev_[kThreads] = {};
};

// Whether an array goes through the pinned pieces: pageable, and 32 MB or more
// (192^3 in float64).  Up to there memory that was freed comes back without
// page faults, and one thread's copy is as fast: four fields of 128^3, 6 ms up
// and 4.5 down, against 7.5 and 6 by threads and 30 to 40 for a first use.
inline bool wants_pieces(const void* host, size_t bytes) {
  if (bytes < ((size_t)32 << 20)) return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace mhit
