// tensormap.h -- the driver's tensor-map encoder, looked up at run time (the
// library links against the runtime only)
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace wlg {

typedef CUresult (*TensorMapEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                    const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// null if the driver has none
inline TensorMapEncode tensor_map_encode() {
  static TensorMapEncode fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &res) != cudaSuccess ||
        res != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return (TensorMapEncode)p;
  }();
  return fn;
}

}  // namespace wlg
