// launch.cuh -- launches of the kernels that follow one another in a step.
//
// A step is a chain of kernels of a few microseconds, each reading what the one
// before it wrote.  They are launched with programmatic stream serialization: a
// kernel's blocks are placed while the last blocks of the kernel before it drain,
// and wait in step_begin() until that kernel has finished and its writes are
// visible, so the launch itself no longer lies between them.  Every kernel
// launched this way calls step_begin() first, on every thread and before it
// reads or writes memory (the next kernel's wait then covers all earlier ones;
// the fluid kernel behind the solid kernels, which let it in, waits later), and reads what other kernels of the step write by ordinary loads (not
// through the read-only path, whose data must not change while a kernel
// runs).  Per stage, plain launches / graph replay: 16,384-particle 2D scene (4
// kernels) 24.8 / 18.1 us without it, 17.1 / 17.3 with it; 16,899-particle 3D
// scene (7 kernels) 65 / 54 against 50 / 52; 1.05 M particles 424 / 417 against
// 409 / 414.  Letting the next kernel's blocks in from the start
// (griddepcontrol.launch_dependents first) took 18.9 / 18.3, 53 / 54, 419 / 421.
#pragma once

#include <cuda_runtime.h>

namespace arp {

__device__ __forceinline__ void step_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Lets the next kernel's blocks in as soon as every block of this one has got here.
// For a next kernel that has work before its wait: what it reads until then must
// have been written by kernels that this one's step_begin(), or that of the
// kernel before, has waited for.  Blocks that wait hold no place that an earlier
// kernel's block still needs, all of which are resident by then.
__device__ __forceinline__ void step_let_next() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
void launch_step(void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // an error stays for cudaGetLastError
}

}  // namespace arp
