// Host-side helpers shared by the C-ABI translation units: error reporting, tensor-map encoding,
// device properties.  Nothing here allocates device memory.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define KSB_OK_RC 0
#define KSB_ERR_INVALID (-1)
#define KSB_ERR_CUDA (-2)
#define KSB_ERR_UNSUPPORTED (-3)

namespace ksb {

// Stores a printf-style message retrievable with ksb_last_error() and returns `rc`.
int fail(int rc, const char* fmt, ...);

// Checks the launch error state after a kernel launch; returns 0 or KSB_ERR_CUDA.
int check_launch(const char* what);

// Encodes a 2-D tiled tensor map (row-major tensor: `inner` contiguous elements, `outer` rows,
// `row_stride_bytes` between rows).  Box rows of 128 bytes are swizzled by 128, of 64 by 64, others not.
int encode_tmap_2d(CUtensorMap* out, CUtensorMapDataType dt, int elem_bytes, const void* base, uint64_t inner,
                   uint64_t outer, uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer);

// The same for a tensor of `rank` axes (innermost first; strides in bytes of the axes behind it).
int encode_tmap(CUtensorMap* out, CUtensorMapDataType dt, int elem_bytes, const void* base, int rank, const uint64_t* dims,
                const uint64_t* stride_bytes, const uint32_t* box);

int sm_count();

// Kernels this thread has launched through launch_kernel (counts up for ever; callers take differences).
extern thread_local int t_launches;
inline int launch_count() { return t_launches; }

// Device address of the status words of the current device (resolved once per device).
int* status_words();

// Launches a kernel whose arguments are `args` (its parameters, in order), optionally as clusters of `cluster` CTAs along
// x and, with `chained`, as a programmatic dependent of the kernel before it on the stream (common.cuh: pdl_wait).
template <typename... Args>
int launch_kernel(const char* what, const void* fn, dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster, bool chained,
                  const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  void* argv[] = {const_cast<void*>(static_cast<const void*>(&args))...};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, argv);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(KSB_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  }
  ++t_launches;
  return 0;
}

// A kernel's shared-memory limit, raised once per device instead of on every launch (setting it twice from two threads
// is harmless: the value is the same).
struct DeviceOnce {
  unsigned char done[64] = {0};
  int raise_smem(const void* fn, int bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return fail(KSB_ERR_CUDA, "no current device");
    if (dev >= 0 && dev < 64 && done[dev]) return 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
      cudaGetLastError();
      return fail(KSB_ERR_CUDA, "cannot raise dynamic shared memory limit");
    }
    if (dev >= 0 && dev < 64) done[dev] = 1;
    return 0;
  }
};

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace ksb
