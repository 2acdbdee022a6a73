// qsv_launch.h -- host launch of sweep kernels behind one another.
#pragma once
#include <cuda_runtime.h>

namespace qsv {
namespace dev {

// Launch behind the work before it in the stream without waiting for its end (programmatic dependent launch): the
// kernel itself waits before it reads the state, and a sweep lets the next one come when only its last tile's store
// is left. Interpreter and complex128 sweeps of every size gain: 12 random layers of 16 qubits 262 -> 212 us, a
// 20-qubit ansatz 153 -> 121 us, 24 qubits with Toffolis 6.37 -> 6.07 ms, a 27-qubit random circuit 17.57 -> 17.40 ms,
// complex128 at 20 / 27 qubits 480 -> 395 us / 47.1 -> 46.8 ms.
template <class... KA, class... A>
static inline cudaError_t launch_behind(void (*kernel)(KA...), unsigned grid, unsigned block, size_t smem,
                                        cudaStream_t stream, const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace dev
}  // namespace qsv
