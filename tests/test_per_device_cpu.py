"""What the launchers look up once is kept per device and may be asked for by several threads at once.  The helper is
compiled here against a stand-in for the current device; no GPU is involved."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "host_util.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int g_dev = 0;
static std::atomic<int> g_asked{0};
int tb::host::current_device() { return g_dev; }
static int answer() {  // what one rule of a dispatch asks
  static tb::host::DeviceCache cache;
  return tb::host::per_device(cache, [] { ++g_asked; return g_dev == 5 ? 0 : 100 + g_dev; });
}
int main() {
  std::vector<std::thread> threads;
  std::atomic<int> bad{0};
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([t, &bad] {
      for (int i = 0; i < 20000; ++i) {
        g_dev = (t + i) % 4;
        if (answer() != 100 + g_dev) ++bad;
      }
    });
  for (auto& t : threads) t.join();
  const int asked = g_asked;  // at least once per device, at most once per thread and device
  g_dev = 63; bad += answer() != 163; bad += answer() != 163;
  bad += g_asked != asked + 1;
  g_dev = -1; bad += answer() != 99;   // no device, or one beyond the table: asked every time
  g_dev = 64; bad += answer() != 164;
  g_dev = 5; bad += answer() != 0; bad += answer() != 0;  // not known: asked again
  bad += g_asked != asked + 5;
  std::printf("%d %d\n", bad.load(), asked);
  return bad || asked < 4 || asked > 64;
}
"""


def test_answers_are_kept_per_device(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if cxx is None or not os.path.exists(os.path.join(cuda, "include", "cuda.h")):
        pytest.skip("needs a host compiler and the CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-I{os.path.join(ROOT, 'tybok_b200', 'csrc')}", f"-I{cuda}/include", str(src), "-o",
                    str(exe)], check=True, capture_output=True, timeout=300)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert proc.returncode == 0, proc.stdout

