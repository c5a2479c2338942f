// Launch settings shared by the pass launchers, and the tensor maps of the
// line passes.
#pragma once
#include <atomic>
#include <cmath>
#include "kernel_set.h"

namespace wdm {

// Launch settings are device properties: each is found once per device (the
// current one at the launch) and kept in a slot per device ordinal.
constexpr int MAX_DEVICES = 64;

static int current_device() {
  int dev = 0;
  cudaGetDevice(&dev);
  return dev >= 0 && dev < MAX_DEVICES ? dev : 0;
}

// Opt a kernel in to more than 48 KB of dynamic shared memory, once per device.
template <auto K>
static cudaError_t prep_once(size_t smem) {
  if (smem <= 48 * 1024) return cudaSuccess;
  // 0: not yet, 1: done, 2 + e: failed with cudaError_t e
  static std::atomic<int> state[MAX_DEVICES];
  std::atomic<int>& st = state[current_device()];
  int v = st.load(std::memory_order_acquire);
  if (v == 0) {
    const cudaError_t e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    v = e == cudaSuccess ? 1 : 2 + (int)e;
    st.store(v, std::memory_order_release);
  }
  return v == 1 ? cudaSuccess : (cudaError_t)(v - 2);
}

// Launch K so that its CTAs may start while the stream's previous kernel drains
// (chain.cuh: the kernel waits for that one itself).
template <auto K, class... Args>
static cudaError_t launch_chained(dim3 grid, int threads, size_t smem, cudaStream_t st, const Args&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, K, args...);
  ++tl_kernel_launches;
  return cudaGetLastError();
}

// SMs of the current device.
static int sm_count() {
  static std::atomic<int> n[MAX_DEVICES];
  const int dev = current_device();
  int v = n[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    v = v > 0 ? v : 1;
    n[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

// Resident CTAs per SM of a kernel at its block size and shared memory, on the
// current device (each call site passes one fixed size).
template <auto K>
static int resident_ctas(int threads, size_t smem) {
  static std::atomic<int> n[MAX_DEVICES];
  std::atomic<int>& slot = n[current_device()];
  int v = slot.load(std::memory_order_relaxed);
  if (v == 0) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, K, threads, smem);
    v = v > 0 ? v : 1;
    slot.store(v, std::memory_order_relaxed);
  }
  return v;
}

template <int N>
struct LineMaps {
  // Tensor map of the lines of g (null view: false).
  static bool line_map(CUtensorMap* map, const float2* data, const LineGeom& g, int batch) {
    using TT = TmaTile<N>;
    if (g.axis != 1 && g.axis != 2) return false;
    if (g.nxa < LINES || g.rows <= 0) return false;  // the box stays inside the tensor along x
    const uint64_t e = sizeof(float2);
    uint64_t dims[4], strides[3];
    uint32_t box[4];
    dims[0] = (uint64_t)g.nxa;
    dims[3] = (uint64_t)batch;
    strides[0] = (uint64_t)g.pitch * e;
    strides[2] = (uint64_t)g.bstride * e;
    if (g.axis == 1) {  // [batch][rows][N][pitch]
      dims[1] = N;
      dims[2] = (uint64_t)g.rows;
      strides[1] = (uint64_t)g.pitch * N * e;
      box[0] = LINES, box[1] = TT::BOXP, box[2] = 1, box[3] = 1;
    } else {  // [batch][N][rows][pitch]
      dims[1] = (uint64_t)g.rows;
      dims[2] = N;
      strides[1] = (uint64_t)g.pitch * g.rows * e;
      box[0] = LINES, box[1] = 1, box[2] = TT::BOXP, box[3] = 1;
    }
    return encode_map_c64(map, data, dims, strides, box);
  }

  // Tensor map of the edge tiles of g (the last column when nxa = 16 m + 1,
  // 8 rows per tile; k_lfft_tma): the lines' axis outermost, a box of 2
  // columns x 8 rows x BOXP points starting at column nxa - 1, whose x offset
  // (nxa - 1) * 8 bytes must be a multiple of 16.  false: no edge tiles.
  static bool edge_map(CUtensorMap* map, const float2* data, const LineGeom& g, int batch) {
    using TT = TmaTile<N>;
    if (g.axis != 1 && g.axis != 2) return false;
    if (g.nxa % LINES != 1 || g.nxa < LINES || (g.nxa - 1) % 2 != 0 || g.rows <= 0 || g.rows % 8 != 0) return false;
    const uint64_t e = sizeof(float2);
    uint64_t dims[4] = {(uint64_t)g.nxa, (uint64_t)g.rows, (uint64_t)N, (uint64_t)batch};
    uint64_t strides[3];
    if (g.axis == 1) {  // rows (z) at pitch * N, points (y) at pitch
      strides[0] = (uint64_t)g.pitch * N * e;
      strides[1] = (uint64_t)g.pitch * e;
    } else {  // rows (y) at pitch, points (z) at pitch * rows
      strides[0] = (uint64_t)g.pitch * e;
      strides[1] = (uint64_t)g.pitch * g.rows * e;
    }
    strides[2] = (uint64_t)g.bstride * e;
    const uint32_t box[4] = {2, 8, (uint32_t)TT::BOXP, 1};
    return encode_map_c64(map, data, dims, strides, box);
  }
};

}  // namespace wdm
