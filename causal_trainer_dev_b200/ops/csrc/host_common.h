// Host-side helpers shared by the launchers: error strings, tensor-map construction
// through the driver entry point (no link-time dependency on libcuda), a small cache
// of encoded maps, and the per-device status word.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <unordered_map>

#include "tc05.cuh"

#define CTB_API extern "C" __attribute__((visibility("default")))

namespace ctb {

// Last error message of the calling thread (returned by ctb_last_error()).
void set_error(const std::string& msg);
int fail(const std::string& msg);  // sets the message, returns a non-zero code

#define CTB_CUDA_OK(expr)                                                                        \
  do {                                                                                           \
    cudaError_t _e = (expr);                                                                     \
    if (_e != cudaSuccess) return ::ctb::fail(std::string(#expr) + ": " + cudaGetErrorString(_e)); \
  } while (0)

enum class Elt : int { BF16 = 0, F32 = 1 };

// A copy of an encoded tensor map.  The cache drops its own when it is full, at any later lookup of this or of another
// thread, and a launch needs several: so it hands out no pointers.
struct TensorMap {
  CUtensorMap map{};
  bool ok = false;
  explicit operator bool() const { return ok; }
};

// Encodes (or fetches from cache) a tiled tensor map over a row-major 2-D view.
//   inner/outer: extents in elements; row_stride: elements between rows;
//   box_inner/box_outer: tile; swizzle128: 128-byte swizzle or none.
// Not ok, with the error message set, on failure.
TensorMap get_tensor_map_2d(const void* base, Elt elt, uint64_t inner, uint64_t outer, uint64_t row_stride,
                            uint32_t box_inner, uint32_t box_outer, bool swizzle128);
// 4-D variant used by attention: dims {d0 (contiguous), d1, d2, d3}, element strides s1..s3.
TensorMap get_tensor_map_4d(const void* base, Elt elt, const uint64_t dims[4], const uint64_t strides[3],
                            const uint32_t box[4], bool swizzle128);

// Per-device status word in device memory (allocated on first use).
DeviceStatus* device_status();

int sm_count();

// Programmatic dependent launch: with `chained` the kernel's CTAs may start, set up and wait (wait_for_predecessor) while the
// launch before it in the stream still runs, if that one lets them (let_successor_start).  Only short calls are chained: there
// the 2 us between two launches count (two rows of 256 tokens, attention 36.5 -> 34.1 us; an MLP on 1000 rows of 1536 / 8960 299 ->
// 284; a head on 333 rows 221 -> 215); with 512 MB and 4e11 for the limits longer sequences took 0.96 to 1.15 of their time.
// These two are the most that anything chains at.  A kernel whose blocks are fewer than fit at once loses by an early start, because
// they crowd on the SMs that have room first: rotary embedding, norms, attention and the gradient of kept logits have lines of
// their own where they are launched.
constexpr long CHAINED_BYTES = 64l << 20;       // moved by a memory-bound kernel
constexpr double CHAINED_FLOPS = 6e10;          // of a product
template <typename... P, typename... A>
cudaError_t launch_chained(bool chained, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, void* stream, int cluster,
                           const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  if (cluster > 0) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  if (chained) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  cfg.attrs = attr;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();      // a refused launch is the caller's to report, not the next launch's to meet
  return e;
}

}  // namespace ctb
