"""Values kept per CUDA device: kernel attributes set on one device do not hold
on another, so each device's are set on its first use, and a failure is
reported and not kept."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rtbvh_gb300", "csrc")

PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  rtbvh::PerDevice<unsigned> sizes;
  int calls = 0;
  auto find = [&](unsigned v) { return [&calls, v](unsigned* out) { ++calls; *out = v; return 0; }; };
  unsigned v = 0;
  CHECK(sizes.get(0, &v, find(16)) == 0 && v == 16 && calls == 1);
  CHECK(sizes.get(0, &v, find(99)) == 0 && v == 16 && calls == 1);
  CHECK(sizes.get(1, &v, find(8)) == 0 && v == 8 && calls == 2);  // another device: found there
  CHECK(sizes.get(70, &v, find(4)) == 0 && v == 4 && calls == 3);
  CHECK(sizes.get(0, &v, find(99)) == 0 && v == 16 && calls == 3);
  v = 5;
  CHECK(sizes.get(2, &v, [&](unsigned*) { ++calls; return 7; }) == 7 && v == 5 && calls == 4);
  CHECK(sizes.get(2, &v, find(2)) == 0 && v == 2 && calls == 5);  // tried again
  return 0;
}
"""


def test_each_device_has_its_own(tmp_path):
    src, exe = tmp_path / "per_device.cpp", tmp_path / "per_device"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_the_clustering_kernels_keep_no_process_wide_flag():
    """LOCB's attributes and cluster size go through the per-device table."""
    text = open(os.path.join(CSRC, "locb.cu")).read()
    assert "once_flag" not in text and "PerDevice<unsigned>" in text
