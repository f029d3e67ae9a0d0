// What the driver knows about a caller's buffer.
#include "common.cuh"

#include <cuda.h>

namespace gb300 {

bool inside_allocation(const void *p, size_t bytes) {
    typedef CUresult (*Attributes)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
    static const Attributes attributes = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &fn, 12000,
                                             cudaEnableDefault, &found) != cudaSuccess) {
            cudaGetLastError();
            return (Attributes) nullptr;
        }
        return found == cudaDriverEntryPointSuccess ? (Attributes)fn : nullptr;
    }();
    if (!attributes) return false;
    CUpointer_attribute which[2] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                    CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    CUdeviceptr start = 0;
    size_t size = 0;
    void *out[2] = {&start, &size};
    const CUdeviceptr at = (CUdeviceptr)(uintptr_t)p;
    if (attributes(2, which, out, at) != CUDA_SUCCESS || at < start) return false;
    return at - start <= size && bytes <= size - (at - start);
}

}  // namespace gb300
