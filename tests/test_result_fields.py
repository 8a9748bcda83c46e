"""The buffers of an ensemble's final fields (mhit36_b200/csrc/hostpool.h): a
request whose download fails holds none of them, so that nothing of an
earlier request's fields, which the pool's buffers still contain, can be read
through it.  Runs on the CPU: the failing copy is a function of the test."""
import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include <stdio.h>
#include "hostpool.h"
using namespace mhit;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  const size_t n = 1000;
  HostPool pool;
  auto value = [&](double v) { return [=](double* p, int f) { for (size_t q = 0; q < n; ++q) p[q] = v + f; return 0; }; };
  double* first[4];
  {
    ResultFields a;
    CHECK(!a.held() && a.fill(&pool, 4, n, 99, value(10)) == 0 && a.held() && a.count() == n);
    for (int f = 0; f < 4; ++f) {
      CHECK(a.field(f) && a.field(f)[0] == 10 + f && a.field(f)[n - 1] == 10 + f);
      first[f] = const_cast<double*>(a.field(f));
    }
  }  // released: the pool keeps the buffers and what is in them
  for (int bad = 0; bad < 4; ++bad) {
    ResultFields b;
    int reused = 0;
    const int e = b.fill(&pool, 4, n, 99, [&](double* p, int f) {
      for (double* q : first) reused += p == q;
      if (f == bad) return 7;
      for (size_t q = 0; q < n; ++q) p[q] = -1;
      return 0;
    });
    CHECK(e == 7 && !b.held() && reused == bad + 1);
    for (int f = 0; f < 4; ++f) CHECK(b.field(f) == nullptr);
    CHECK(b.fill(&pool, 3, n, 99, value(20)) == 0 && b.held());  // and the next try is whole
    for (int f = 0; f < 3; ++f) CHECK(b.field(f)[0] == 20 + f && b.field(f)[n - 1] == 20 + f);
    CHECK(b.field(3) == nullptr);
  }
  ResultFields c;  // a buffer that cannot be had
  CHECK(c.fill(&pool, 4, (size_t)1 << 57, 99, value(0)) == 99 && !c.held());
  printf("ok\n");
  return 0;
}
"""


def test_failed_download_holds_no_fields(tmp_path):
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "mhit36_b200", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe, "-pthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
