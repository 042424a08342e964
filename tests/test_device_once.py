"""Kernel attributes (dynamic shared-memory limits) belong to one device: the
launchers' set-up (csrc/device_once.h) runs on every device that is used, and
no launcher keeps a flag for the whole process. CPU only: the two CUDA calls
are stand-ins."""
import os
import re
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "exahype_b200", "csrc")
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include "device_once.h"
#include <cstdio>
static int g_dev = 0;
static bool g_fails = false;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = g_dev; return cudaSuccess; }
int main() {
  exa::DeviceOnce once;
  int runs = 0;
  auto use = [&](int dev) {
    g_dev = dev;
    return once([&] { runs++; return g_fails ? cudaErrorInvalidValue : cudaSuccess; });
  };
  auto expect = [&](int n, const char* what) {
    if (runs != n) { std::printf("%s: %d runs, expected %d\n", what, runs, n); return 1; }
    return 0;
  };
  int bad = 0;
  use(0); use(0);
  bad += expect(1, "one device");
  use(1); use(1); use(0);
  bad += expect(2, "a second device");
  g_fails = true;
  bad += use(5) == cudaSuccess;
  g_fails = false;
  use(5); use(5);
  bad += expect(4, "after a failure");
  use(63); use(63); use(0);
  bad += expect(5, "the last bit");
  use(70); use(70);
  bad += expect(7, "a device without a bit");
  return bad;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")), reason="needs the CUDA headers")
def test_set_up_runs_once_on_every_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, "-I", CUDA, str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_no_launcher_keeps_a_flag_for_the_process():
    text = open(os.path.join(CSRC, "capi.cu")).read()
    assert not re.search(r"static\s+bool\s+\w+\s*=\s*false", text)
