"""The buffer an advance can do without (csrc/optional_buffer.h) against an allocator that refuses."""
import os
import subprocess

from pelelm_gb300._build import CSRC

PROGRAM = r"""
#include "optional_buffer.h"
#include <cstdio>
static int made = 0, asked = 0, dropped = 0;
static size_t limit = 100;
static char mem[8];
int main() {
  pgb_host::OptionalBuffer b;
  auto get = [&](size_t n) {
    return b.ensure(n, [](size_t k) -> void* { ++asked; return k <= limit ? &mem[made++] : nullptr; },
                    [](void* old) { dropped += old != nullptr; });
  };
  if (!get(0) || asked) return 1;                              // nothing needed: nothing asked
  if (!get(50) || asked != 1 || b.p != &mem[0]) return 2;
  if (!get(30) || asked != 1) return 3;                        // fits
  if (get(200) || asked != 2) return 4;                        // refused ...
  if (b.p != &mem[0] || b.cap != 50 || dropped) return 5;      // ... and the old one stays
  if (get(200) || get(300) || asked != 2) return 6;            // not asked again at that size or above
  if (!get(50) || asked != 2) return 7;
  if (!get(90) || asked != 3 || b.p != &mem[1] || dropped != 1) return 8;  // below: still tried
  limit = 1000;
  if (get(200)) return 9;
  return 0;
}
"""


def test_a_refused_size_is_not_asked_for_again(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
