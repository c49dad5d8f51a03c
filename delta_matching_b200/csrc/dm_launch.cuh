// Programmatic dependent launch of the composite chains: the successor in the stream is launched as its predecessor's CTAs
// finish, sets itself up (barriers, tensor memory, descriptors) and waits in pdl_wait until the predecessor's results are
// visible.  Rules: every thread of every CTA calls pdl_wait before it touches global memory that another kernel reads or writes
// (a kernel that completed without waiting would release its successor early), and all launches of such kernels go through
// launch_pdl.  Without the launch attribute pdl_wait does nothing.
// No kernel triggers its successor early (griddepcontrol.launch_dependents): a waiting successor's CTAs then take the SMs that
// the predecessor's successor-but-one, or its own last CTAs, would have used.  Eager, us per pass, plain launches / early
// triggers / this: forward B1 N512 H8 21.5 / 16.7 / 15.0; step B4 N768 H12 104 / 93 / 86; B3 N1024 H12 full 123 / 123 / 111;
// B2 N2048 H16 237 / 231 / 221; forward B4 N4096 H32 646 / 652 / 638.
#pragma once
#include <cuda_runtime.h>

namespace dm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace dm

namespace dmh {

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, void* stream, const A&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace dmh
