"""Host copies by several threads (mhit36_b200/csrc/hostcopy.h) on the CPU,
against a stand-in for the few runtime calls the header makes: what a first
copy pins, which arrays take that path, and that the pieces cover an array of
rows once, whatever its size, pitch and number of threads."""
import os
import subprocess

from conftest import ROOT

RUNTIME = r"""
#pragma once
#include <stddef.h>
#include <stdlib.h>
typedef int cudaError_t;
enum { cudaSuccess = 0 };
typedef int* cudaEvent_t;
enum { cudaEventDisableTiming = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost };
struct cudaPointerAttributes { cudaMemoryType type; };
inline size_t pinned = 0;
inline bool no_pinned = false, registered = false;
inline cudaError_t cudaMallocHost(void** p, size_t b) {
  if (no_pinned) return 2;
  pinned += b;
  *p = malloc(b);
  return 0;
}
inline cudaError_t cudaFreeHost(void* p) { free(p); return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new int(0); return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
inline cudaError_t cudaSetDevice(int) { return 0; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = registered ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return 0;
}
"""

SOURCE = r"""
#include <stdio.h>
#include <vector>
#include "hostcopy.h"
using namespace mhit;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  const size_t n3 = sizeof(double) * 128 * 128 * 128, big = sizeof(double) * 192 * 192 * 192;
  double x = 0;
  CHECK(!wants_pieces(&x, n3) && wants_pieces(&x, big));
  registered = true;
  CHECK(!wants_pieces(&x, big));
  PinnedPieces pp;
  no_pinned = true;
  CHECK(!pp.ready(big));
  no_pinned = false;
  CHECK(pp.ready(big) && pp.ready(big) && pinned == PinnedPieces::kThreads * pp.piece() && pinned == 8u << 20);
  for (size_t n : {192, 256, 384, 512, 768, 1024}) {  // what a first use pins: about an eighth of a field, 32 MB at most
    const size_t total = sizeof(double) * n * n * n, all = PinnedPieces::kThreads * PinnedPieces::piece_for(total);
    CHECK(all <= total / 6 && all <= 32u << 20 && PinnedPieces::piece_for(total) % sizeof(double) == 0);
  }
  const size_t piece = pp.piece();
  for (size_t bytes : {(size_t)4096, piece / 2 + 8, piece, 3 * piece + 64})
    for (size_t rows : {1, 3, 17})
      for (size_t gap : {0, 128}) {
        const size_t total = bytes * rows, pitch = bytes + gap;
        std::vector<char> host(pitch * rows), dev(total, 0), back(pitch * rows, 7);
        for (size_t q = 0; q < host.size(); ++q) host[q] = (char)(q * 2654435761u >> 13);
        const HostRows from{host.data(), bytes, pitch}, to{back.data(), bytes, pitch};
        std::atomic<size_t> moved{0};
        CHECK(pp.run(0, total, [&](int, void* buf, cudaEvent_t, size_t at, size_t len) {
          from.read(buf, at, len);
          memcpy(dev.data() + at, buf, len);
          moved += len;
          return 0;
        }) == 0 && moved == total);
        CHECK(pp.run(0, total, [&](int, void* buf, cudaEvent_t, size_t at, size_t len) {
          memcpy(buf, dev.data() + at, len);
          to.write(buf, at, len);
          return 0;
        }) == 0);
        for (size_t r = 0; r < rows; ++r)
          for (size_t q = 0; q < pitch; ++q) {
            const char got = back[r * pitch + q];
            CHECK(got == (q < bytes ? host[r * pitch + q] : 7));
          }
      }
  std::atomic<int> calls{0};  // an error ends the copy with that error
  CHECK(pp.run(0, 1000 * piece, [&](int, void*, cudaEvent_t, size_t at, size_t) {
    ++calls;
    return at == 5 * piece ? 700 : 0;
  }) == 700 && calls < 1000);
  pp.release();
  std::vector<char> a(((size_t)9 << 20) + 5), b(a.size(), 0);  // parallel_copy, a ragged size
  for (size_t q = 0; q < a.size(); ++q) a[q] = (char)(q * 2654435761u >> 11);
  parallel_copy(b.data(), a.data(), a.size());
  CHECK(a == b);
  printf("ok\n");
  return 0;
}
"""


def test_pieces(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(tmp_path), "-I",
                    os.path.join(ROOT, "mhit36_b200", "csrc"), str(tmp_path / "t.cpp"), "-o", exe, "-pthread"],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
