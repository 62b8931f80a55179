// launch.cuh -- launches of step kernels that follow each other in a stream.
//
// A step kernel reads what the step before wrote, and between two ordinary launches the GPU drains, signals and
// starts again, 1-2 us that a small lattice's step does not take itself (and outside a graph whole ticks of about 2
// us).  Launched programmatically, the next kernel's CTAs are brought in while the current one's leave, and wait for
// it.  us per step: D3Q19 FP32 16^3 4.1 -> 1.8, 32^3 4.1 -> 2.2, 64^3 8.3 -> 5.7, 128^3 50.2 -> 47.8; FP64 64^2 D2Q9
// 8.3 -> 6.5, 82 x 48 D3Q19 14.4 -> 12.1, 64^3 114.9 -> 108.9; channel 192 x 48 FP32 6.2 -> 3.5.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

namespace erlbm {

// First statement of a kernel launched by launch_after, executed by every thread before any access to memory: waits
// until the kernel before it in the stream has finished and its writes are visible, then lets the next one be
// launched (to wait in its turn).  The order matters: a successor that was brought in while this kernel still waits
// could keep lines in its L1 of the buffer that the kernel before this one reads and this one writes.
// What an earlier kernel of the stream writes (the populations) is read by ordinary loads, from pointers without
// __restrict__: the read-only path (__ldg, const __restrict__) is for data that nobody writes while the kernel is
// resident, which for a kernel that comes in early includes the time before this wait, and the compiler may move such
// loads above it.
__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// CTAs of KERN that the GPU holds at a time, found once per device.
template <auto KERN, int BLOCK>
int resident_ctas(size_t smem = 0)
{
    constexpr int MAXDEV = 64;
    static std::atomic<int> cache[MAXDEV];  // host threads that race store the same value
    int dev = 0;
    cudaGetDevice(&dev);
    const int d = dev >= 0 && dev < MAXDEV ? dev : 0;
    int n = cache[d].load(std::memory_order_relaxed);
    if (n <= 0) {
        int per_sm = 0, sms = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, BLOCK, smem) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        n = per_sm * (sms > 0 ? sms : 1);
        cache[d].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Whether a grid of equal CTAs gains by coming in early.  CTAs are placed where there is room, so beside a grid that
// fills more than half of the GPU the first ones of a grid that would spread evenly over an empty GPU crowd the SMs
// with room (FP64 256^2, 1024 CTAs of 1824: 16.5 -> 21.4 us a step; 300^2, 1407: 20.6 -> 21.6).  With room for two
// grids (200^2, 625: 13.4 -> 11.2) or more than a wave of CTAs (400^2, 2500: 32.9 -> 30.9) that does not arise.
inline bool comes_early(long long grid, long long resident) { return 2 * grid <= resident || 3 * grid >= 4 * resident; }

// kern<<<grid, block, smem, s>>>(args...); early: brought in while the stream's previous kernel drains.
template <class... P, class... A>
cudaError_t launch_after(bool early, void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                         A &&...args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&c, kern, static_cast<P>(args)...);
}

// The same with the rule above, for a kernel of one CTA size.
template <auto KERN, int BLOCK, class... A>
cudaError_t launch_step_kernel(unsigned grid, cudaStream_t s, A &&...args)
{
    return launch_after(comes_early(grid, resident_ctas<KERN, BLOCK>()), KERN, grid, BLOCK, 0, s, args...);
}

}  // namespace erlbm
