// The driver's tensor-map encoder, looked up once.
#pragma once
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

namespace tb200 {

// NULL: the driver does not have it.  The first calls of several threads are in order (initialisation of a local static).
inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &res) == cudaSuccess && res == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
        return nullptr;
    }();
    return fn;
}

}  // namespace tb200
