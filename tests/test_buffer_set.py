"""Buffers replaced together or not at all (csrc/buffer_set.h), which the FP64
Chebyshev tables use: compiled for the host with an allocator that fails at the
n-th call.  After a failure the set is as it was and nothing is lost; no call
after it is handed a null or a too small buffer."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include <cstdlib>
#include <map>
#include "buffer_set.h"
static std::map<void *, size_t> live;
static int left = -1;  // allocations that still succeed; -1: all do
static void *get(size_t n) {
  if (left == 0) return nullptr;
  if (left > 0) left--;
  void *p = malloc(n);
  live[p] = n;
  return p;
}
static void put(void *p) {
  assert(live.erase(p) == 1);
  free(p);
}
typedef cg::BufferSet<3> Set;
static void sound(const Set &s) {
  size_t held = 0;
  for (int q = 0; q < 3; q++) {
    held += s.buf[q] != nullptr;
    assert(s.buf[q] ? live.count(s.buf[q]) && live[s.buf[q]] >= s.cap[q] : s.cap[q] == 0);
  }
  assert(held == live.size());
}
int main() {
  const size_t sizes[4][3] = {{100, 0, 24}, {50, 300, 24}, {400, 400, 400}, {90, 10, 8}};
  for (int fail = 0; fail < 4; fail++)
    for (int first = 0; first < 4; first++) {
      Set s;
      for (int call = 0; call < 4; call++) {
        const size_t(&want)[3] = sizes[(first + call) % 4];
        const Set before = s;
        left = call == 1 || first == 0 ? fail : -1;
        const bool ok = s.reserve(want, get, put);
        left = -1;
        sound(s);
        for (int q = 0; q < 3; q++) {
          if (ok) assert(s.buf[q] && s.cap[q] >= want[q]);
          else assert(s.buf[q] == before.buf[q] && s.cap[q] == before.cap[q]);
          if (ok && before.buf[q] && before.cap[q] >= want[q]) assert(s.buf[q] == before.buf[q]);
        }
        if (!ok) assert(s.reserve(want, get, put));
        sound(s);
      }
      s.release(put);
      sound(s);
      assert(live.empty());
    }
  return 0;
}
"""


def test_buffers_replaced_together_or_not_at_all(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "comd_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
