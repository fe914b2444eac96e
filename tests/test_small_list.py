"""The one-block path on an edge list that the caller overwrites during the
call, modelled on the CPU with the descriptor that the kernel uses: the
counting pass keeps the pairs it read, and the scatter fills every slot that
was counted with an id it checked."""
from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "connectivity_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "gb_internal.cuh"
int main() {
  std::mt19937 r(1);
  const int n = 40;
  for (int m : {1, 7, 500}) {
    std::vector<int32_t> src(m), dst(m), kept(2 * m), adj(2 * m, -7);
    for (int e = 0; e < m; ++e) src[e] = (int)(r() % n), dst[e] = (int)(r() % n);
    const std::vector<int32_t> s0 = src, d0 = dst;
    gb::SmallDesc D{};
    D.n = n;
    D.m = m;
    D.src = src.data();
    D.dst = dst.data();
    D.kept = kept.data();
    std::vector<int> co(n + 1), ci(n + 1);
    for (int e = 0; e < m; ++e) {  // the counting pass
      const int32_t a = D.src[e] - D.id_base, b = D.dst[e] - D.id_base;
      D.keep(e, a, b);
      ++co[a + 1];
      ++ci[b + 1];
    }
    for (int e = 0; e < m; ++e) src[e] = dst[e] = e % 2 ? 1 << 30 : 3;  // the caller writes
    for (int v = 0; v < n; ++v) co[v + 1] += co[v], ci[v + 1] += ci[v];
    const gb::SmallDesc L = D.again();
    for (int e = 0; e < m; ++e) {  // the scatter
      const int32_t a = L.src[e] - L.id_base, b = L.dst[e] - L.id_base;
      if (a != s0[e] || b != d0[e]) return std::printf("edge %d changed\n", e), 1;
      adj[co[a]++] = b;
      adj[m + ci[b]++] = a;
    }
    for (int32_t x : adj)
      if (x < 0 || x >= n) return std::printf("slot holds %d\n", x), 1;
  }
  gb::SmallDesc D{};  // a device list is read where it is
  D.id_base = 5;
  if (D.again().id_base != 5) return 1;
  D.keep(0, 1, 2);
  return 0;
}
"""


def test_list_written_under_the_call(tmp_path):
    src, exe = tmp_path / "list.cpp", tmp_path / "list"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
