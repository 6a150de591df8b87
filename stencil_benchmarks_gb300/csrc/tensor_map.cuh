// Host side of the tensor memory accelerator: the driver's tensor-map encoder,
// looked up at run time (the library links the CUDA runtime only).
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"

namespace sb {

inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
        cudaGetLastError();
    });
    return fn;
}

template <class S>
CUtensorMapDataType tma_type() {
    if constexpr (sizeof(S) == 8) return CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
    else if constexpr (sizeof(S) == 4) return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    else return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
}

}  // namespace sb
