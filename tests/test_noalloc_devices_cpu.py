"""px_derive_noalloc's report of a bad cell, per device, on a runtime of stand-ins (CPU only).

A grid entry beyond the pool is reported through a word of host memory that the kernel
writes.  The library's source is compiled here with stand-ins for the CUDA calls it makes:
a launch runs nothing but the kernel's report (the arguments it was launched with), and
waiting for device 0 lets a call on device 1 run first, as another host thread's would.
Calls on different devices share nothing, so each must see its own report.
"""
import os
import subprocess

from pixels_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STANDINS = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>
#include "pixels_gb300.h"

static int device = 0, nested = 0;
static bool bad[64];                 // device d's grid names a brick beyond its pool
static unsigned char memory[64][64]; // device d's "scratch"
static std::vector<void*> status_of[64];

static int call(int dev) {
  static const uint32_t grid[8] = {0};
  static const uint8_t tables[256] = {0};
  static uint32_t super_counts[8];
  static uint8_t density[8];
  const int before = device;
  device = dev;
  const int rc = px_derive_noalloc(grid, nullptr, 2, 2, 2, 0, tables, tables, super_counts, density, nullptr);
  device = before;
  return rc;
}

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** p, void* h, unsigned) { *p = h; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = memory[device]; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  if (device == 0 && nested == 1) {  // meanwhile, on device 1
    nested = 2;
    const int rc = call(1);
    if (rc != (bad[1] ? PX_E_INVALID_ARG : PX_OK)) { std::printf("device 1: %d\n", rc); std::exit(1); }
  }
  return cudaSuccess;
}
// noalloc_cells_kernel(grid, BX, BY, BZ, n_pool, tables, counts, call, status, super_counts, density)
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void** args) {
  uint32_t* status = *(uint32_t**)args[8];
  status_of[device].push_back(status);
  if (bad[device]) *status = *(uint32_t*)args[7];
  return cudaSuccess;
}
// what the compiler's registration of the kernels refers to; no kernel is ever launched by <<<>>>
void* __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd() {}
void __cudaUnregisterFatBinary() {}
void __cudaRegisterFunction() {}
void __cudaRegisterVar() {}
void __cudaGetKernel() { std::abort(); }
void __cudaLaunchKernel() { std::abort(); }
void __cudaPushCallConfiguration() { std::abort(); }
void __cudaPopCallConfiguration() { std::abort(); }
}

int main() {
  for (int b0 = 0; b0 < 2; b0++)
    for (int b1 = 0; b1 < 2; b1++)
      for (int first = 0; first < 2; first++) {  // alone, then with device 1's call inside
        bad[0] = b0;
        bad[1] = b1;
        nested = first;
        const int rc = call(0);
        if (rc != (b0 ? PX_E_INVALID_ARG : PX_OK)) { std::printf("device 0: %d (%d %d %d)\n", rc, b0, b1, first); return 1; }
      }
  for (int d = 0; d < 64; d++) {  // every device the library takes has a word of its own
    bad[d] = true;
    if (call(d) != PX_E_INVALID_ARG) { std::printf("device %d\n", d); return 1; }
    for (int e = 0; e < d; e++)
      if (status_of[e].back() == status_of[d].back()) { std::printf("devices %d and %d share a word\n", e, d); return 1; }
  }
  if (call(64) != PX_E_INVALID_ARG) return 1;  // more devices than it keeps addresses for
  std::puts("ok");
  return 0;
}
"""


def test_each_device_sees_its_own_report(tmp_path):
    main = tmp_path / "main.cpp"
    main.write_text(STANDINS)
    exe = tmp_path / "noalloc"
    inc = ["-I", os.path.join(ROOT, "include")]
    src = os.path.join(ROOT, "pixels_gb300", "csrc", "px_noalloc.cu")
    r = subprocess.run([build._nvcc(), *build.ARCH, "-O1", "-std=c++17", "-fmad=false", "-cudart", "none", *inc, str(main), src,
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
