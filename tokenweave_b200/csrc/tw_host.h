// Host-side helpers shared by the .cu launchers: error strings and TMA tensor-map creation
// through the driver entry point (no link-time dependency on libcuda).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tw {

// Last host-side error of a launcher, readable through tw_last_error() by the bindings.
void set_last_error(const char* fmt, ...);
const char* last_error();

// Encode a tiled tensor map for a bf16 tensor of `rank` dimensions (innermost first).
// `strides_bytes[i]` is the byte stride of dimension i+1 (dimension 0 is contiguous).
// Swizzle is always 128 bytes, out-of-bounds elements read as zero.
// Returns false (and sets the last error) if the driver refuses the encoding.
bool make_tensor_map_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                          const uint64_t* strides_bytes, const uint32_t* box);

// The same with the 64-byte swizzle (boxes whose rows are 64 bytes: the write-back blocks of the GEMM epilogue).
bool make_tensor_map_bf16_sw64(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                               const uint64_t* strides_bytes, const uint32_t* box);

// The same for a tensor of 8-bit elements (fp8 operands).
bool make_tensor_map_u8(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                        const uint64_t* strides_bytes, const uint32_t* box);

int device_sm_count();

// A launch that may start while the kernel before it on the stream still runs (if that one calls allow_dependents); the kernel
// calls wait_predecessor before it touches memory.
template <typename... Params, typename... Args>
inline cudaError_t launch_dependent(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

}  // namespace tw
