// launch.cuh -- launches of the kernels that follow one another in a step.
//
// A step is a chain of kernels of a few microseconds, each reading what the one
// before it wrote.  They are launched with programmatic stream serialization: a
// kernel's blocks are placed while the last blocks of the kernel before it drain,
// and wait in step_begin() until that kernel has finished and its writes are
// visible, so the launch itself no longer lies between them.  Every kernel
// launched this way calls step_begin() on every thread (the next kernel's wait
// then covers all earlier ones) before it reads or writes memory, and reads what
// other kernels of the step write by ordinary loads (not through the read-only
// path, whose data must not change while a kernel runs).  One kernel reads ahead
// of its step_begin(): the fluid kernel behind the solid kernels, which let it in
// (step_let_next).  What it reads there was written by kernels that the stress
// kernel's step_begin() has waited for; the wait orders those writes for the
// stress kernel, step_publish() there and step_begin_unless() here hand that
// order on (release, acquire), and a block that does not find the word set waits
// at its start like any other.  Per stage, plain launches / graph replay: 16,384-particle 2D scene (4
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
// For a next kernel that has work before its wait (see above): what it reads until
// then must have been written by kernels that this one's step_begin(), or that of
// the kernel before, has waited for.  Blocks that wait hold no place that an earlier
// kernel's block still needs, all of which are resident by then.
__device__ __forceinline__ void step_let_next() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// One thread, after its step_begin() and ahead of step_let_next(): whoever finds
// `word` set by step_begin_unless() sees what this thread's wait has waited for.
__device__ __forceinline__ void step_publish(uint32_t* word) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(word), "r"(1u) : "memory");
}
// A block's start, on all its threads: step_begin(), unless `word` (null: none)
// is found set.  The access goes to the L2, where the word was cleared by a
// kernel that the publishing one has waited for, so a value of an earlier step is
// not met.  The barrier carries thread 0's acquire to the block.  Only the blocks
// that can be resident at first (148 SMs) look at the word: later ones are placed
// when an earlier one has been through its wait, and find theirs over; an acquire
// empties its SM's L1, and with one in every block of the fluid kernel ten RK2
// steps of 1,048,576 particles took 10,046 us, now 9,940 (9,943 unordered;
// 16,899 particles under velocity Verlet 540, 537 unordered).
__device__ __forceinline__ void step_begin_unless(const uint32_t* word, uint32_t blocks_per_sm) {
    if (word && blockIdx.x < 148u * blocks_per_sm) {
        uint32_t set = 1u;
        if (threadIdx.x == 0)
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(set) : "l"(word) : "memory");
        if (__syncthreads_and((int)set)) return;
    }
    step_begin();
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
