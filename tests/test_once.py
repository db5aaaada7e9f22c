"""What happens once per device, by several threads at once (csrc/once.h, compiled for the host with a stand-in for the CUDA runtime)."""

import shutil
import subprocess
from pathlib import Path

import pytest

import layover_b200

CSRC = Path(layover_b200.__file__).parent / "csrc"

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "once.h"

thread_local int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return device < 0 ? cudaErrorNoDevice : cudaSuccess; }

int main() {
  static LbPerDeviceOnce once;
  std::atomic<int> calls{0}, early{0};
  std::atomic<bool> ready[2] = {};
  std::vector<std::thread> threads;
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([&, t] {
      device = t % 2;
      const bool ok = once.run([&] {
        ++calls;
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
        ready[device] = true;
        return true;
      });
      if (!ok || !ready[device]) ++early;      // gone on before its device was configured
    });
  for (auto& t : threads) t.join();
  if (calls != 2 || early != 0) { std::printf("calls %d, early %d\n", calls.load(), early.load()); return 1; }
  device = 2;                                   // a configuration that fails is tried again, one that succeeded is not
  int tries = 0;
  const bool first = once.run([&] { ++tries; return false; }), second = once.run([&] { ++tries; return true; }), third = once.run([&] { ++tries; return false; });
  if (first || !second || !third || tries != 2) { std::printf("tries %d\n", tries); return 2; }
  device = -1;                                  // an unknown device: every time
  for (int i = 0; i < 3; ++i) once.run([&] { ++tries; return true; });
  return tries == 5 ? 0 : 3;
}
"""


def test_once_per_device_is_done_before_anybody_goes_on(tmp_path):
    gxx = shutil.which("g++")
    include = next((p for p in (Path("/usr/local/cuda/include"),) if (p / "cuda_runtime_api.h").is_file()), None)
    if gxx is None or include is None:
        pytest.skip("no host compiler or no CUDA headers")
    source, program = tmp_path / "once.cpp", tmp_path / "once"
    source.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-pthread", f"-I{CSRC}", f"-I{include}", str(source), "-o", str(program)], check=True)
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout
