// Programmatic dependent launch, the way the compute kernels of a layer follow one another in a stream.
#pragma once

#include <cuda_runtime.h>
#include <cstdlib>

namespace ep {

inline bool programmatic_launches() {
    static const bool off = [] {
        const char* v = std::getenv("EP_DISABLE_PDL");
        return v != nullptr && v[0] != '\0' && v[0] != '0';
    }();
    return !off;
}

// A kernel launched like this may become resident while the kernel ahead of it in the stream drains. It calls
// dependency_wait() before it touches memory that any earlier kernel may write or still read (set-up of barriers, tensor
// memory and descriptors can go before), and launch_dependents() so that its own successor can do the same. The gap between
// dependent kernels of 2 to 3 us and the set-up of a GEMM (2 us) go away; a layer has six to twenty of them.
// (A kernel whose successor reads inputs before its own wait has to wait first and announce afterwards.)
// Every kernel launched like this calls dependency_wait() in every block before it ends, also where it needs nothing of the
// kernel ahead: the wait of the kernel behind it covers this one only, and through it what this one has waited for.
template <typename... Params, typename... Args>
cudaError_t launch_early(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem_bytes, cudaStream_t stream, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic_launches() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace ep
