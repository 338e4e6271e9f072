// The driver's encoder of tiled tensor maps, resolved once through the runtime (no link against libcuda).
#pragma once
#include <cuda.h>  // types only
#include <cuda_runtime.h>

typedef CUresult (*tc_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// nullptr where the driver has none.
inline tc_encode_fn tc_tensor_map_encoder() {
  static const tc_encode_fn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<tc_encode_fn>(f);
  }();
  return fn;
}
