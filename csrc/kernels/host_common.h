// Host-side helpers shared by the kernel launchers: tensor-map encoding through
// the driver entry point (no link-time dependency on libcuda), the per-device
// status word, and the error convention of the exported C functions.
//
// Every exported launcher returns 0 on success or a negative CGK_E_* code and
// leaves a message retrievable with cgk_last_error().
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#define CGK_API extern "C" __attribute__((visibility("default")))

enum {
  CGK_E_ARG = -1,      // bad argument (shape, alignment, null pointer)
  CGK_E_CUDA = -2,     // a CUDA runtime / driver call failed
  CGK_E_LIMIT = -3,    // size beyond a stated maximum
  CGK_E_DEVICE = -4,   // the kernel reported a device-side status
};

namespace cgk {

void set_error(const char* fmt, ...);
const char* last_error();

// Device status words: int[4] per device, allocated once (lazily) per device.
int* device_status(int device);

// Encode a tiled bf16/fp32/u8 tensor map.  dims[0] is the innermost (contiguous)
// dimension.  strides_bytes[i] is the stride of dims[i+1].  Returns 0 or CGK_E_*.
enum class Swz { None = 0, B32 = 1, B64 = 2, B128 = 3 };
int encode_tmap(CUtensorMap* out, const void* base, CUtensorMapDataType dtype, int rank,
                const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box, Swz swz);

// Shorthand for a row-major 2-D bf16 matrix [rows, cols] with leading dimension
// ld (elements), box = box_rows x box_cols, 128-byte swizzle.
int encode_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols,
                        uint64_t ld, uint32_t box_rows, uint32_t box_cols);

int sm_count(int device);

#define CGK_CUDA_CHECK(expr)                                                         \
  do {                                                                               \
    cudaError_t _e = (expr);                                                         \
    if (_e != cudaSuccess) {                                                         \
      ::cgk::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, \
                       __LINE__);                                                    \
      return CGK_E_CUDA;                                                             \
    }                                                                                \
  } while (0)

#define CGK_LAUNCH_CHECK()                                                           \
  do {                                                                               \
    cudaError_t _e = cudaGetLastError();                                             \
    if (_e != cudaSuccess) {                                                         \
      ::cgk::set_error("kernel launch failed: %s (%s:%d)", cudaGetErrorString(_e),   \
                       __FILE__, __LINE__);                                          \
      return CGK_E_CUDA;                                                             \
    }                                                                                \
  } while (0)

#define CGK_REQUIRE(cond, ...)              \
  do {                                      \
    if (!(cond)) {                          \
      ::cgk::set_error(__VA_ARGS__);        \
      return CGK_E_ARG;                     \
    }                                       \
  } while (0)

// Launches a kernel that may start while its predecessor in the stream is still running (programmatic dependent launch): every
// thread of it passes pdl_wait() before it touches memory that another kernel writes or reads.  cluster: CTAs along x, 0 for none.
// Only a launch that is being captured says so: eager launches of such small kernels are bound by the host, which the attribute
// costs time (a gated-layer prompt whose host is the limit 1963 us with it, 1923 without; replayed decoding steps the same).
template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {};
  if (cluster > 0) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) (void)cudaGetLastError();
  if (capture == cudaStreamCaptureStatusActive) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Runs f(scratch) with `floats` elements from the stream's memory pool, given back in stream order (null: none wanted, or none left).
template <typename F>
int with_stream_scratch(long long floats, cudaStream_t stream, F f) {
  float* p = nullptr;
  if (floats > 0 && cudaMallocAsync((void**)&p, (size_t)floats * sizeof(float), stream) != cudaSuccess) {
    (void)cudaGetLastError();
    p = nullptr;
  }
  const int rc = f(p);
  if (p) CGK_CUDA_CHECK(cudaFreeAsync(p, stream));
  return rc;
}

}  // namespace cgk
