/* Programmatic dependent launch (CUDA 12.3+, recorded by stream capture into graphs).
 *
 * launch_dep launches a kernel with cudaLaunchAttributeProgrammaticStreamSerialization when the
 * context allows it (GAT_TUNE_DEP_LAUNCH, on by default): the GPU may then set the kernel up
 * while the previous kernel of the stream finishes. Every kernel launched this way calls dep_wait(), which
 * returns once the previous grid has completed and its writes are visible. All but one call it first
 * and none of them triggers its dependents early, so such a grid starts only after every block of the
 * previous one has exited, and ordering in the stream is the same as without the attribute, minus the
 * launch gap. dep_wait() is a no-op for a kernel launched without the attribute.
 *
 * The exception is k_plain_groups (range_groups.cu), which lets the next query's launch of itself start at
 * once and waits late. What keeps it safe:
 *   - before its wait it reads only the index and the queries, both complete before the call's first launch
 *     (which goes without the attribute), and writes only its own shared memory;
 *   - every block of every instance reaches the wait, so that an instance completes after the one before and
 *     its completion stands for all earlier ones;
 *   - only instances of itself follow it with the attribute: a kernel behind it that took the attribute and
 *     touched memory before its own wait would run beside it. The host waits for the stream after each lot. */
#pragma once

#include <mutex>
#include <set>
#include <utility>

#include "internal.h"

namespace gat {

__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/* Sets a kernel's preferred split between L1 and shared memory (percent of the largest shared
 * size) the first time it is asked for on a device; later requests for the same kernel keep the
 * first value. An SM takes the split of the first block that lands on it while it is empty and
 * keeps it until it is empty again, so a long-running kernel fixes the split of its SMs for every
 * other stream's blocks. */
inline void prefer_split(const void* kernel, int device, int pct) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    std::lock_guard<std::mutex> lk(mu);
    if (!done.insert({kernel, device}).second) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct) != cudaSuccess)
        cudaGetLastError();
}

template <class... P, class... A>
inline cudaError_t launch_dep(const gat_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t s, A&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = ctx->dep_launch ? 1 : 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

/* zeroes n ints in stream order (a kernel, so a chain of dependent launches stays unbroken) */
__global__ void k_zero_words(int* p, int n);

}  // namespace gat
