"""Attributes that a launcher sets once on a device, when several threads make its first call (host code alone, no GPU)."""
import os
import shutil
import subprocess

import pytest

from inferloop_b200.csrc.build import HERE, find_nvcc

HARNESS = r"""
#include "once_per_device.h"
#include <atomic>
#include <chrono>
#include <thread>
static std::atomic<int> device{0};
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return device == 63 ? cudaErrorNoDevice : cudaSuccess; }
static ilb::OncePerDevice once;
int main() {
  // two threads make the first call: the second must not be told that the attribute is there while the first is still setting it
  std::atomic<bool> setting{false}, there{false};
  std::thread first([&] {
    once.run([&] {
      setting = true;
      std::this_thread::sleep_for(std::chrono::milliseconds(300));
      there = true;
      return cudaSuccess;
    });
  });
  while (!setting) std::this_thread::yield();
  const bool usable = once.run([&] { there = true; return cudaSuccess; }) == cudaSuccess && there;
  first.join();
  if (!usable) return 1;
  // done: not set again; another device has its own; a failure is reported and tried again; no device: set every time
  int calls = 0;
  auto ok = [&] { ++calls; return cudaSuccess; };
  auto bad = [&] { ++calls; return cudaErrorInvalidValue; };
  if (once.run(ok) != cudaSuccess || calls != 0) return 2;
  device = 1;
  if (once.run(bad) != cudaErrorInvalidValue || calls != 1) return 3;
  if (once.run(ok) != cudaSuccess || calls != 2 || once.run(ok) != cudaSuccess || calls != 2) return 4;
  device = 0;
  if (once.run(bad) != cudaSuccess || calls != 2) return 5;
  device = 63;
  if (once.run(ok) != cudaSuccess || once.run(ok) != cudaSuccess || calls != 4) return 6;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_attributes_are_there_before_a_device_counts_as_done(tmp_path):
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(find_nvcc()))), "include")
    source, program = tmp_path / "once.cpp", tmp_path / "once"
    source.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", HERE, "-I", include, "-o", str(program), str(source)], check=True, timeout=120)
    assert subprocess.run([str(program)], timeout=60).returncode == 0
