// What the kernels of the copy table take, and the launchers of the kernel families (internal to the library).
#pragma once
#include <cuda_runtime.h>

#include <cstdio>

#include "common.h"
#include "m2n.h"

// The one argument of every kernel, in the constant bank.  A launch of a single op can carry it here (`ops` null): nothing
// has to be uploaded and the op is not fetched from memory.
struct M2NLaunch {
  const M2NOp* ops;
  const uint32_t* tile_start;
  uint32_t n_ops;
  uint32_t* sync;  // finished tiles, error word; may be null where nothing is signalled
  const uint64_t* signals;
  uint32_t n_signals;
  uint32_t epoch;
  int do_signal;
  M2NOp one;
};

// Makes `device` current while it lives (-1: leaves the current one). `error`: why it could not.
struct OnDevice {
  int before = -1;
  cudaError_t error;
  explicit OnDevice(int device) {
    int now = -1;
    error = cudaGetDevice(&now);
    if (error != cudaSuccess || device < 0 || device == now) return;
    error = cudaSetDevice(device);
    if (error == cudaSuccess) before = now;
    else cudaGetLastError();  // not the error of the next call
  }
  ~OnDevice() {
    if (before >= 0) cudaSetDevice(before);
  }
  OnDevice(const OnDevice&) = delete;
};

inline int m2n_cuda_error(cudaError_t e, const char* what) {
  snprintf(etha_err_buf(), ETHA_ERR_LEN, "%s: %s", what, cudaGetErrorString(e));
  return -(int)e - 1000;
}

// Launch as a programmatic dependent of the kernel before it in the stream: the CTAs may become resident, set up their
// queue and fetch their op while that kernel finishes; everything else comes after `after_previous_kernel`.
template <typename Kernel, typename... Args>
inline cudaError_t m2n_launch_dependent(Kernel kernel, uint32_t grid, int block, size_t smem, void* stream, Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(grid);
  config.blockDim = dim3(block);
  config.dynamicSmemBytes = smem;
  config.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attr;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, args...);
}

template <typename Kernel>
inline int m2n_launch(Kernel kernel, uint32_t grid, int block, size_t smem, void* stream, const M2NLaunch& args, const char* what) {
  const cudaError_t e = m2n_launch_dependent(kernel, grid, block, smem, stream, args);
  if (e == cudaSuccess) return 0;
  cudaGetLastError();
  snprintf(etha_err_buf(), ETHA_ERR_LEN, "%s kernel launch: %s", what, cudaGetErrorString(e));
  return -(int)e - 1000;
}

inline int m2n_no_instance(const char* what, int key) {
  snprintf(etha_err_buf(), ETHA_ERR_LEN, "no %s kernel instance for key 0x%x", what, key);
  return -102;
}

int m2n_launch_copy(const M2NLaunch& args, bool general, uint32_t n_tiles, int ctas_per_sm, void* stream);
int m2n_launch_bulk(const M2NLaunch& args, uint32_t n_tiles, void* stream);
int m2n_launch_typed(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream);
int m2n_launch_collapse(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream);
int m2n_launch_ragged(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream);
int m2n_launch_transpose(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream);
