// Where a caller's pointer lies, as far as the kernels' own stores are concerned.
#pragma once
#include <cuda_runtime_api.h>

namespace rfx {

// Whether a kernel on `device` may store through a pointer with these
// attributes: memory of that device, or managed memory.  Another GPU's memory
// is device memory too, but has no mapping on this one unless peer access was
// enabled, so results go there by a copy, which takes any device's pointer.
inline bool kernel_may_store(const cudaPointerAttributes& a, int device) {
    return a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == device);
}

}  // namespace rfx
