// Host: the driver's tensor-map encoder, resolved at run time.
#pragma once

#include "common.cuh"

#include <cuda.h>

namespace dcb
{

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Null where the driver has none.  Resolved once; threads that ask meanwhile wait.
inline EncodeTiledFn encode_tiled_fn()
{
    static const EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess
            && q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(p);
        (void) cudaGetLastError();
        return EncodeTiledFn(nullptr);
    }();
    return fn;
}

} // namespace dcb
