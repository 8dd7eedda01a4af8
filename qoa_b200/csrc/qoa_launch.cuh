// qoa_launch.cuh — launches that overlap with the end of the kernel before them.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace qoa {

// Launches k with programmatic stream serialisation: its CTAs may be placed, and
// run up to their grid_wait(), while the previous kernel of the stream still
// runs (from its grid_go() on, or its end where it has none); grid_wait() then
// holds them until that kernel has finished and its writes are visible. For
// kernels that call grid_wait() before they touch anything an earlier kernel
// wrote, and before they write anything. Streams being captured launch plainly.
// It hides a launch's latency and a pass's staging behind the tail of the pass
// before: 16 passes of 20 qubits with 1024 shots 380 -> 337 us, 5 interpreter
// passes of a 16-qubit trajectory 192 -> 152 us, 13-qubit program 206 -> 184 us.
template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a[0].val.programmaticStreamSerializationAllowed = 1;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        c.attrs = a;
        c.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&c, k, std::forward<A>(args)...);
}

}  // namespace qoa
