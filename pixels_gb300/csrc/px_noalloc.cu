// px_derive_noalloc: the derived upload buffers (super-grid counts and the
// density bytes of GpuWorld.ts:90-101, VoxelWorld.ts:159-170) computed from a
// grid and pool the caller holds on the device, into output buffers the
// caller holds, without allocating any device memory.
//
// Who needs it: a caller that has fixed its device memory before it starts
// working and cannot let a library take more afterwards — a renderer that
// sizes all of its buffers once at upload and shares the GPU with other
// programs, a frame loop in which an allocation can stall the device for the
// length of a frame, or a process running under a hard device-memory cap.
// px_derive needs a world handle, whose buffers are allocated (and grown) by
// this library; this entry point needs none.
//
// Scratch: one opaque-voxel count per pool brick, kept in the fixed-size array
// below (2 MiB, allocated once when the library's device code is loaded), so the
// entry point's footprint is known in advance.  It limits the pool to
// PX_NOALLOC_MAX_POOL_BRICKS bricks (1 GiB of pool); larger pools are refused with
// PX_E_TOO_LARGE before any GPU work.
//
// Status: a cell that names a brick beyond the pool is reported through a word
// of host memory that the kernel can write (one per device, in a page of this
// library's own data, registered on first use and for the rest of the process): it
// stores the call's number there, so nothing is cleared before the kernels and nothing
// copied back after them.
//
// Set-up: the first call on each device, with that device current, looks up
// the array's device address (cudaGetSymbolAddress) and the status word's, and
// keeps them for later calls on that device.  Make the first call on a device
// before any stream capture is begun on it.  The kept addresses belong to the
// device's current context: after cudaDeviceReset (which unloads the library's
// device code) the array may live elsewhere, so this entry point is not to be
// called on a device that has been reset since its first call.
//
// Alignment: the pool is read as 32-bit voxel pairs (16 bytes at a time where it
// starts on a 16-byte boundary) and the grid and super counts as 32-bit words, so
// those three addresses must be multiples of 4 bytes (a uint16 pool that starts at
// an odd element is refused with PX_E_INVALID_ARG before any GPU work).
//
// Every call on a device shares its array and status word: calls on one device that
// overlap in time (from several host threads, or on several streams) race on them and
// may return wrong results.  Callers serialise them.  Calls on different devices share
// nothing.  The counts are written for every pool
// brick before they are read, so they need no clearing.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>

#include "../../include/pixels_gb300.h"
#include "jsmath.cuh"

namespace {

constexpr uint32_t MAX_POOL_BRICKS = PX_NOALLOC_MAX_POOL_BRICKS;
constexpr int MAX_DEVICES = 64;

// The only device scratch of px_derive_noalloc.  Host code never uses this name as a
// device address: the address comes from cudaGetSymbolAddress.
static __device__ __align__(256) uint16_t g_derive_scratch[MAX_POOL_BRICKS];

struct Tables {  // passed by value (512 bytes of kernel parameters)
  uint8_t opaque[256];
  uint8_t udens[256];
};

constexpr uint32_t FULL = 0xffffffffu;
constexpr uint32_t UNIFORM_FLAG = 0x80000000u;

// Opaque, non-air voxels of the voxel pair w (VoxelWorld.ts:163-169).
__device__ __forceinline__ uint32_t opaque_pair(const uint8_t* op_s, uint32_t w) {
  const uint32_t lo = w & 0xffffu, hi = w >> 16;
  return (uint32_t)(lo != 0 && op_s[lo & 0xffu]) + (uint32_t)(hi != 0 && op_s[hi & 0xffu]);
}

// Pass 1: opaque, non-air voxels of every pool brick, COUNT_BRICKS bricks per warp with
// all their loads in flight.  Bound by the pool's bytes, then by the table look-ups
// (one per voxel): the penthouse's 48 MB at 80 voxels per metre in 22 us with one
// brick per warp and 4-byte loads, 14 so (4 bricks 16.5, 8 bricks 17.4; counting each
// brick where its cell refers to it, one kernel for both passes, 78).  VEC: the pool
// starts on a 16-byte boundary.
constexpr int COUNT_BRICKS = 2;
template <bool VEC>
__global__ void __launch_bounds__(256) noalloc_count_kernel(const uint32_t* __restrict__ pool32, uint32_t n_pool,
                                                            const __grid_constant__ Tables t, uint16_t* __restrict__ counts) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // pass 2 may start: it waits for the counts itself
  __shared__ uint8_t op_s[256];
  op_s[threadIdx.x] = t.opaque[threadIdx.x];  // 256 threads
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t b0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * COUNT_BRICKS; b0 < n_pool; b0 += warps * COUNT_BRICKS) {
    uint4 v[COUNT_BRICKS][2];
#pragma unroll
    for (int q = 0; q < COUNT_BRICKS; q++) {
      if (b0 + q >= n_pool) {
        v[q][0] = v[q][1] = make_uint4(0u, 0u, 0u, 0u);
        continue;
      }
      const uint32_t* p = pool32 + (size_t)(b0 + q) * 256;
      if (VEC) {
        v[q][0] = __ldg(reinterpret_cast<const uint4*>(p) + lane);
        v[q][1] = __ldg(reinterpret_cast<const uint4*>(p) + lane + 32);
      } else {
        v[q][0] = make_uint4(__ldg(p + lane), __ldg(p + lane + 32), __ldg(p + lane + 64), __ldg(p + lane + 96));
        v[q][1] = make_uint4(__ldg(p + lane + 128), __ldg(p + lane + 160), __ldg(p + lane + 192), __ldg(p + lane + 224));
      }
    }
    uint32_t mine = 0;
#pragma unroll
    for (int q = 0; q < COUNT_BRICKS; q++) {
      uint32_t c = 0;
#pragma unroll
      for (int h = 0; h < 2; h++)
        c += opaque_pair(op_s, v[q][h].x) + opaque_pair(op_s, v[q][h].y) + opaque_pair(op_s, v[q][h].z) +
             opaque_pair(op_s, v[q][h].w);
      c = __reduce_add_sync(FULL, c);
      if (lane == q) mine = c;
    }
    if (lane < COUNT_BRICKS && b0 + lane < n_pool) counts[b0 + lane] = (uint16_t)mine;
  }
}

// Pass 2: one warp per super cell (4x4x4 bricks, two per lane): the count of
// non-empty bricks, and each brick's density byte — 0 for air, the material's
// table value for a uniform brick, Math.round(n / 512 * 255) for a pool brick.  Starts
// while pass 1 runs and reads the grid meanwhile.  The whole call: 60 us with two clears
// before and a status copy after the passes, 36 so, 32.5 with the density bytes in integers.
__global__ void __launch_bounds__(256) noalloc_cells_kernel(const uint32_t* __restrict__ grid, int BX, int BY, int BZ,
                                                            uint32_t n_pool, const __grid_constant__ Tables t,
                                                            const uint16_t* __restrict__ counts, uint32_t call, uint32_t* status,
                                                            uint32_t* __restrict__ super_counts,
                                                            uint8_t* __restrict__ density) {
  __shared__ uint8_t ud_s[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) ud_s[i] = t.udens[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int SX = (BX + 3) / 4, SY = (BY + 3) / 4, SZ = (BZ + 3) / 4;
  const long long n_super = (long long)SX * SY * SZ;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  bool counted = false;
  for (long long sc = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; sc < n_super; sc += warps) {
    const int sz = (int)(sc / ((long long)SX * SY));
    const int rem = (int)(sc - (long long)sz * SX * SY);
    const int sy = rem / SX, sx = rem - sy * SX;
    uint32_t g[2];
    size_t ci[2];
    bool cell[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int k = lane + 32 * h;
      const int bx = sx * 4 + (k & 3), by = sy * 4 + ((k >> 2) & 3), bz = sz * 4 + (k >> 4);
      cell[h] = bx < BX && by < BY && bz < BZ;
      ci[h] = (size_t)bx + (size_t)BX * ((size_t)by + (size_t)BY * (size_t)bz);
      g[h] = cell[h] ? __ldg(grid + ci[h]) : 0u;
    }
    if (!counted) asm volatile("griddepcontrol.wait;" ::: "memory");  // pass 1's counts are written
    counted = true;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (!cell[h]) continue;
      uint8_t d = 0;
      if (g[h] & UNIFORM_FLAG) {
        d = ud_s[g[h] & 0xffu];
      } else if (g[h] != 0) {
        if (g[h] - 1 < n_pool) d = density_byte(__ldcg(counts + (g[h] - 1)));
        else *(volatile uint32_t*)status = call;  // outside the caller's pool: reported, not read
      }
      density[ci[h]] = d;
    }
    const uint32_t nz = __popc(__ballot_sync(FULL, g[0] != 0)) + __popc(__ballot_sync(FULL, g[1] != 0));
    if (lane == 0) super_counts[sc] = nz;
  }
}

std::mutex g_setup_mu;
constexpr int STATUS_STRIDE = 16;  // words: a line of 64 bytes per device
// word STATUS_STRIDE d: the number of the last call on device d that met a bad cell
alignas(4096) uint32_t g_status_page[MAX_DEVICES * STATUS_STRIDE];
static_assert(sizeof g_status_page % 4096 == 0, "whole pages are registered");
bool g_registered = false;
struct Addresses {
  uint16_t* scratch;
  uint32_t* status;           // the device's word, as the device sees it
  volatile uint32_t* report;  // and as the host does
} g_addr[MAX_DEVICES];
std::atomic<uint32_t> g_calls{0};

// Addresses of the scratch and the status word on the current device (set-up on first use).
int addresses_for_current_device(Addresses* out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return PX_E_NO_DEVICE;
  }
  if (dev < 0 || dev >= MAX_DEVICES) return PX_E_INVALID_ARG;
  std::lock_guard<std::mutex> g(g_setup_mu);
  if (!g_addr[dev].scratch) {
    void *p = nullptr, *q = nullptr;
    uint32_t* const word = g_status_page + dev * STATUS_STRIDE;
    if (!g_registered && cudaHostRegister(g_status_page, sizeof g_status_page,
                                          cudaHostRegisterMapped | cudaHostRegisterPortable) != cudaSuccess) {
      cudaGetLastError();
      return PX_E_CUDA;
    }
    g_registered = true;
    if (cudaHostGetDevicePointer(&q, word, 0) != cudaSuccess || !q ||
        cudaGetSymbolAddress(&p, g_derive_scratch) != cudaSuccess || !p) {
      cudaGetLastError();
      return PX_E_CUDA;
    }
    g_addr[dev] = {(uint16_t*)p, (uint32_t*)q, word};
  }
  *out = g_addr[dev];
  return PX_OK;
}

}  // namespace

extern "C" int px_derive_noalloc(const uint32_t* grid, const uint16_t* pool, int bx, int by, int bz,
                                 uint32_t n_pool_bricks, const uint8_t* opaque256, const uint8_t* uniform_density256,
                                 uint32_t* super_counts, uint8_t* density, void* stream) {
  if (!grid || !super_counts || !density || !opaque256 || !uniform_density256 || (n_pool_bricks && !pool) ||
      bx <= 0 || by <= 0 || bz <= 0)
    return PX_E_INVALID_ARG;
  if (n_pool_bricks > MAX_POOL_BRICKS) return PX_E_TOO_LARGE;
  if (((uintptr_t)grid & 3u) || ((uintptr_t)pool & 3u) || ((uintptr_t)super_counts & 3u)) return PX_E_INVALID_ARG;
  Addresses at;
  const int rc = addresses_for_current_device(&at);
  if (rc != PX_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;

  Tables t;
  for (int i = 0; i < 256; i++) {
    t.opaque[i] = opaque256[i];
    t.udens[i] = uniform_density256[i];
  }
  uint32_t call = g_calls.fetch_add(1) + 1;
  if (call == 0) call = g_calls.fetch_add(1) + 1;  // (0: the page before any call)
  if (n_pool_bricks) {
    const uint32_t per_block = 8 * COUNT_BRICKS, blocks = (n_pool_bricks + per_block - 1) / per_block;
    const uint32_t* p32 = (const uint32_t*)pool;
    if ((uintptr_t)pool & 15u) noalloc_count_kernel<false><<<blocks, 256, 0, s>>>(p32, n_pool_bricks, t, at.scratch);
    else noalloc_count_kernel<true><<<blocks, 256, 0, s>>>(p32, n_pool_bricks, t, at.scratch);
  }
  const long long n_super = (long long)((bx + 3) / 4) * ((by + 3) / 4) * ((bz + 3) / 4);
  const long long blocks = (n_super + 7) / 8;
  // pass 2 may start while pass 1 runs (it reads the grid first and waits before it uses a count)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(blocks < 65535 ? blocks : 65535));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = n_pool_bricks ? 1 : 0;
  cudaLaunchKernelEx(&cfg, noalloc_cells_kernel, grid, bx, by, bz, n_pool_bricks, t, (const uint16_t*)at.scratch, call,
                     at.status, super_counts, density);
  if (cudaGetLastError() != cudaSuccess) return PX_E_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    return PX_E_CUDA;
  }
  return *at.report == call ? PX_E_INVALID_ARG : PX_OK;
}
