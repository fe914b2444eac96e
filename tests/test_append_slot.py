"""Slots of the contraction's and the residual's appends, modelled on the CPU
with the header that the kernels use: a counter that goes on past its array,
beyond 2^31 and 2^32 entries, never gives a slot outside it."""
from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "connectivity_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <type_traits>
#include "gb_internal.cuh"
// the counters that pass 2^31 with the edges of one graph
static_assert(std::is_same_v<std::remove_all_extents_t<decltype(gb::Ctl::con_ecnt)>, gb::append_count>);
static_assert(std::is_same_v<std::remove_all_extents_t<decltype(gb::Ctl::res_ecnt)>, gb::append_count>);
static_assert(sizeof(gb::append_count) == 8);
int main() {
  const long long caps[] = {-5, 0, 1, 31, 32, 33, 1 << 20, (1ll << 31) - 1, 1ll << 31, (1ll << 32) + 7};
  const unsigned long long at[] = {0, 1ull << 20, 1ull << 31, 1ull << 32, (1ull << 32) + (1u << 20), 1ull << 40};
  for (long long cap : caps)
    for (unsigned long long a : at)
      for (long long d = -40; d <= 40; ++d) {
        if (d < 0 && a < (unsigned long long)-d) continue;
        const gb::append_count first = a + d;
        for (unsigned k = 0; k < 256; ++k) {
          const long long s = gb::append_slot(first, k, cap);
          const bool fits = (__int128)first + k < cap;
          if (fits ? s != (long long)(first + k) : s != -1) {
            std::printf("cap %lld first %llu k %u: %lld\n", cap, first, k, s);
            return 1;
          }
        }
      }
  return 0;
}
"""


def test_slots_stay_inside(tmp_path):
    src, exe = tmp_path / "slots.cpp", tmp_path / "slots"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
