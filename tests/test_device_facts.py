"""The number of SMs the launchers size their grids by is that of the current
device (moloch_device.h), compiled here against a stand-in for the CUDA
runtime: two devices of different size used in turn and from several threads,
a device above the table, and a lookup that fails and then works."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dynamical_model_gb300", "csrc")

MAIN = r"""
#include "moloch_device.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int g_dev = 0;
static std::atomic<int> g_asked{0};
static bool g_fail = false;
static const int kSms[] = {152, 148, 20};
extern "C" cudaError_t cudaGetDevice(int* d) { *d = g_dev; return cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) {
  ++g_asked;
  if (g_fail) return cudaErrorInvalidDevice;
  *v = d < 3 ? kSms[d] : 7;
  return cudaSuccess;
}
#define CHECK(x) do { if (!(x)) { std::printf("failed: %s\n", #x); return 1; } } while (0)
int main() {
  g_dev = 2; g_fail = true;
  CHECK(moloch::sm_count() == 1);
  g_fail = false;
  CHECK(moloch::sm_count() == 20);
  g_dev = 0; CHECK(moloch::sm_count() == 152);
  g_dev = 1; CHECK(moloch::sm_count() == 148);
  g_dev = 0; CHECK(moloch::sm_count() == 152);
  g_dev = 70; CHECK(moloch::sm_count() == 7);
  const int asked = g_asked;
  for (int q = 0; q < 100; ++q)
    for (g_dev = 0; g_dev < 3; ++g_dev) CHECK(moloch::sm_count() == kSms[g_dev]);
  CHECK(g_asked == asked);
  std::atomic<int> bad{0};
  std::vector<std::thread> th;
  for (int t = 0; t < 8; ++t)
    th.emplace_back([&bad, t] {
      g_dev = t % 3;
      for (int q = 0; q < 1000; ++q) if (moloch::sm_count() != kSms[t % 3]) ++bad;
    });
  for (auto& x : th) x.join();
  CHECK(bad == 0);
  return 0;
}
"""


def test_sms_of_the_current_device(tmp_path):
    inc = next((p for p in (os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),) if os.path.isdir(p)), None)
    if inc is None:
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", f"-I{inc}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
