"""Kernel attributes (shared-memory limit, carveout) belong to one device: a
launcher that sets them once must do so once per device, not per process."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hammerhead.jl_b200", "csrc")

SRC = r"""
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <thread>
#include <vector>
static thread_local int device = 0;
static cudaError_t fake_device(int* d) { *d = device; return cudaSuccess; }
#define cudaGetDevice fake_device
#include "hh_attr.h"
int main() {
  static hh::DeviceOnce once;
  std::atomic<int> sets[80] = {};
  auto launch = [&](int dev, cudaError_t result = cudaSuccess) {
    device = dev;
    return once([&] { ++sets[dev]; return result; });
  };
  int bad = 0;
  for (int dev : {0, 1, 5, 63, 70})  // a failure is reported and tried again
    bad += launch(dev, cudaErrorInvalidValue) != cudaErrorInvalidValue || launch(dev) != cudaSuccess || sets[dev] != 2;
  for (int dev : {0, 1, 5, 63, 70}) launch(dev);
  bad += sets[0] != 2 || sets[1] != 2 || sets[5] != 2 || sets[63] != 2 || sets[70] != 3 || sets[2] != 0;
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k) t.emplace_back([&, k] { launch(10 + k % 4); });
  for (auto& x : t) x.join();
  for (int dev = 10; dev < 14; ++dev) bad += sets[dev] < 1;
  printf("%d\n", bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(SRC)
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(cuda, "include"), str(src),
                           "-o", str(exe), "-lpthread"])
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip() == "0"


def test_no_launcher_keeps_a_process_wide_flag():
    """No function that sets a kernel attribute guards it with a static bool."""
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        for m in re.finditer(r"static (?:std::atomic<bool>|bool) \w+", text):
            body = text[m.start():m.start() + 1500].split("\n}\n")[0]
            assert "cudaFuncSetAttribute" not in body, f"{name}: {m.group(0)}"


@pytest.mark.gpu
def test_second_device(hb):
    """The default 32 px pass on a second device after the first."""
    import numpy as np
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    A, B = hb.synthetic.particle_pair((128, 128), hb.synthetic.uniform_flow(1.3, -0.6), seed=1)
    got = []
    for dev in (0, 1):
        with hb.PIVWorkspace(device=dev) as w:
            got.append(hb.run_piv(A, B, hb.PIVParameters(), workspace=w))
    np.testing.assert_array_equal(got[0].u, got[1].u)
    np.testing.assert_array_equal(got[0].v, got[1].v)
