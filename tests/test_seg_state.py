"""The pointer jumping of a block of chain nodes (csrc/seg_state.h): states on a cycle never read as
states that stop, in whatever order a round updates them, and paths come to their stops."""
import os
import shutil
import subprocess

import pytest

import bruno_gb300 as bg

HARNESS = r'''
#include "seg_state.h"
#include <cstdio>
#include <vector>
using namespace bruno_seg;
/* jumping in place over n states, each round in the given order; the rounds k_seg_local runs at most */
static void jump(std::vector<uint32_t> &nx, const std::vector<int> &order) {
  for (int round = 0; round < STOP; ++round)
    for (int x : order) {
      const uint32_t w = nx[x], t = nx[w & IDX];
      if (steps(w) && steps(t)) nx[x] = join(w, t);
    }
}
int main() {
  unsigned bad_cycle = 0, bad_path = 0;
  for (int n = 2; n <= 2048; ++n) {
    std::vector<int> up(n), down(n), strided;
    for (int i = 0; i < n; ++i) { up[i] = i; down[i] = n - 1 - i; }
    for (int i = 0; i < 256; ++i) for (int x = i; x < n; x += 256) strided.push_back(x);
    for (const std::vector<int> *o : {&up, &down, &strided}) {
      std::vector<uint32_t> nx(n);
      for (int i = 0; i < n; ++i) nx[i] = (uint32_t)((i + 1) % n) | (1u << STOP);
      jump(nx, *o);
      for (uint32_t w : nx) bad_cycle += steps(w) == 0;
      for (int i = 0; i < n; ++i) nx[i] = i + 1 < n ? (uint32_t)(i + 1) | (1u << STOP) : (uint32_t)i;
      jump(nx, *o);
      for (int i = 0; i < n; ++i) bad_path += (nx[i] & IDX) != (uint32_t)(n - 1) || steps(nx[i]) != (uint32_t)(n - 1 - i);
    }
  }
  printf("%u %u\n", bad_cycle, bad_path);
}
'''


def test_cycle_states_never_stop(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "seg.cpp", tmp_path / "seg"
    src.write_text(HARNESS)
    csrc = os.path.join(os.path.dirname(bg.__file__), "csrc")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", csrc, str(src), "-o", str(exe)], check=True)
    assert subprocess.check_output([str(exe)], text=True).split() == ["0", "0"]
