"""The launchers' tables of kernel limits and resident blocks.

They answer several questions per launch, so every spectral kernel of the
library has to fit, at several launch shapes each, and a process that goes on
to new shapes must not be left asking the runtime at every launch.
"""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).parents[1] / "new_repo_b200" / "csrc"

PROGRAM = """
#include <cstdio>
#include "launch_cache.hpp"
using namespace les;
static LaunchCache<int, LIMITS_CACHE> limits;
static LaunchCache<int, RESIDENT_CACHE> resident;
static char code[1 << 20];
int main() {
  int asked = 0;
  for (int pass = 0; pass < 3; ++pass)
    for (int dev = 0; dev < 4; ++dev)
      for (int k = 0; k < SPECTRAL_KERNELS; ++k) {
        const void* kern = code + 176 * k;  // entry points of a library lie close together
        const int* l = limits.find(dev, kern, 0, 0);
        if (!l) { ++asked; limits.put(dev, kern, 0, 0, dev * 1000 + k); }
        else if (*l != dev * 1000 + k) return 1;
        for (int s = 0; s < 4; ++s) {
          const int* r = resident.find(dev, kern, 128 << (s & 1), 1024 * (40 + 16 * s));
          if (!r) { ++asked; resident.put(dev, kern, 128 << (s & 1), 1024 * (40 + 16 * s), s + k); }
          else if (*r != s + k) return 2;
        }
      }
  // ever new shapes: what was put last is there
  int late = 0;
  for (int i = 0; i < 100000; ++i) {
    const void* kern = code + 176 * (i % SPECTRAL_KERNELS);
    const size_t smem = 16 * (i / SPECTRAL_KERNELS + 100000);
    if (!resident.find(0, kern, 256, smem)) resident.put(0, kern, 256, smem, i);
    const int* r = resident.find(0, kern, 256, smem);
    if (!r || *r != i) ++late;
  }
  std::printf("%d %d", asked, late);
}
"""


def test_tables_hold_every_kernel_and_keep_taking_new_shapes(tmp_path):
    src = tmp_path / "cache.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "cache"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    kernels = int(re.search(r"SPECTRAL_KERNELS = (\d+)", (CSRC / "launch_cache.hpp").read_text()).group(1))
    # each (device, kernel) once, each (device, kernel, shape) once
    assert r.returncode == 0 and list(map(int, r.stdout.split())) == [4 * kernels * (1 + 4), 0]


def test_count_of_spectral_kernels():
    lib = CSRC.parent / "liblesgpu.so"
    if not lib.exists() or not shutil.which("nm"):
        pytest.skip("library not built")
    names = subprocess.run(["nm", "-C", str(lib)], capture_output=True, text=True, check=True).stdout
    kernels = set(re.findall(r"void (les::k_(?:xfwd|xfwd_row|xinv|ypass|yrhs)<[^>]*>)", names))
    stated = int(re.search(r"SPECTRAL_KERNELS = (\d+)", (CSRC / "launch_cache.hpp").read_text()).group(1))
    assert len(kernels) <= stated
