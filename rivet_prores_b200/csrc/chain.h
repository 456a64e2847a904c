// chain.h -- kernels of one stream launched ahead of their turn.
//
// A call's kernels run one after another, three dozen of them for an encode,
// most of them a few microseconds long for a frame or two. Launched in
// programmatic stream order a kernel's CTAs take their places, and its
// prologue runs, while the last CTAs of the kernel before finish. Every
// kernel launched with launch_chained() calls chain_start() first, does only
// what no kernel of the chain writes (its tables), and calls chain_wait()
// before anything else and on every path: it returns when the kernel before
// has completed, and so, each having waited in turn, all kernels before that.
//
// The exceptions are k_fdct and k_alpha_size, which the counting kernels
// follow: they leave chain_start() to the end of their CTAs. With it, the next
// kernels' large CTAs took places on the SMs that their own still had use for
// (30 UHD frames 5.46 -> 5.63 ms, a batch of mixed sizes 5.06 -> 5.16).
//
// What a kernel of the chain writes is read with ordinary loads, never with
// __ldg(): its non-coherent load wants memory that is read-only for the whole
// life of the reading kernel, and that life begins while the writer may still
// run. The bitstreams, the input planes, the code and quantiser tables are in
// place before the chain and may be read either way.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace prores {

#if defined(__CUDACC__)
__device__ __forceinline__ void chain_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// An ordinary load that the compiler may move as freely as __ldg(), for data
// that the reading kernel does not write itself. Its address has to come from
// something read after chain_wait(), which keeps the load behind the wait.
// (As plain C++ loads, which stay between the stores and shuffles around them,
// k_cost took 0.6 % longer: 30 UHD frames 3388 us for 3367, the mixed batch 2590
// for 2574. With __ldg they were 3370 and 2567.)
__device__ __forceinline__ float chain_load(const float *p) {
    float v;
    asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 chain_load4(const float *p) {
    float4 v;
    asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

template <class... Params, class... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(std::forward<Args>(args))...);
}
#endif

}  // namespace prores
