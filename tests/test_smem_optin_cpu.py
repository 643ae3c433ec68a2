"""Opt-in to large dynamic shared memory (csrc/smem_optin.cuh), compiled against a fake
CUDA runtime of two devices: every device a kernel is launched on gets the attribute, two
threads with different sizes leave it at the limit, and no source sets it by another way."""
import shutil
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "igaops_b200" / "csrc"

PROGRAM = r"""
#include "smem_optin.cuh"
#include <stdio.h>
#include <mutex>
#include <thread>

static thread_local int device = 0;
static std::mutex lock;
static int limit_of[2] = {48 * 1024, 48 * 1024};  // the kernel's attribute per device
static int calls = 0;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 227 * 1024; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  a->sharedSizeBytes = 1024;  // static shared memory of the kernel
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
  std::lock_guard<std::mutex> g(lock);
  ++calls;
  limit_of[device] = v;
  return v + 1024 <= 227 * 1024 ? cudaSuccess : cudaErrorInvalidValue;
}
}

static iga::SmemOptIn optin;
static bool launch(int dev, size_t smem) {  // what a launch site does; does it fit?
  device = dev;
  if (optin.allow(nullptr, smem) != cudaSuccess) return false;
  std::lock_guard<std::mutex> g(lock);
  return (int)smem <= limit_of[dev];
}

int main() {
  bool ok = launch(0, 4096) && calls == 0;      // no opt-in needed
  ok = ok && launch(0, 100 * 1024);
  ok = ok && launch(1, 100 * 1024);             // a second device of the process
  ok = ok && launch(0, 200 * 1024) && launch(1, 200 * 1024) && calls == 2;
  bool fit[2] = {true, true};
  std::thread t[2];
  for (int k = 0; k < 2; ++k)
    t[k] = std::thread([&, k] {
      for (int i = 0; i < 20000; ++i) fit[k] = launch(0, (60 + 70 * k + i % 60) * 1024) && fit[k];
    });
  for (auto& x : t) x.join();
  printf("%d\n", ok && fit[0] && fit[1]);
  return 0;
}
"""


def test_opt_in_per_device_and_thread(tmp_path):
    gxx, cuda = shutil.which("g++"), Path("/usr/local/cuda/include")
    assert gxx and cuda.is_dir()
    src, exe = tmp_path / "optin.cpp", tmp_path / "optin"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", f"-I{cuda}", str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60)
    assert out.stdout.strip() == "1"


def test_every_launch_site_uses_it():
    for f in sorted(CSRC.iterdir()):
        if f.name != "smem_optin.cuh":
            assert "cudaFuncSetAttribute" not in f.read_text(), f.name
