// launch.cuh -- one way to launch every kernel of the layer loop (cudaLaunchKernelEx), so that launch attributes have one place to live.
//
// launch_pdl: programmatic dependent launch, for the kernels of the layer loop.  Such a kernel is placed on the SMs while its predecessor in
// the stream finishes; it does its own set-up and reads of weights, then calls pdl_wait() before it touches any memory that a predecessor
// wrote or still reads, and pdl_trigger() after that: its own successor may then be placed.  Since a kernel triggers only after its wait (every thread
// that triggers has waited: the first trigger in a CTA counts for the CTA; tables_kernel, launched plainly, triggers at once: all before it is complete when it starts),
// everything before its predecessor is complete when it starts: what was written two kernels ago may be read before pdl_wait (past L1).
// Not every kernel gains: norm of prefill chunks, SiLU and combine of large ones, placed early, end up unevenly spread over the SMs that happen to be
// free first (4096 tokens: combine 324 against 308 us per layer, SiLU 308 against 302; 512 tokens: norm 110 against 108); they are launched plainly.
// (Triggering before the wait, so that several kernels ahead are placed, was slower for prefill chunks: their CTAs take shared and tensor memory
// from the kernel that is still running.)
#pragma once
#include <cuda_runtime.h>
#include <string.h>

template <typename... KArgs, typename... Args>
static inline cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute at; memset(&at, 0, sizeof at);
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization; at.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = &at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif
#ifdef __CUDACC__
// Scratch that has been read for the last time: its 128-byte line at p (aligned) leaves the L2 without being written to memory.  What lies there afterwards is
// undefined until it is written again.  For gate and up rows and compact down rows (143 MB per layer of 2048 tokens, more than the L2): a layer of 511 / 843 / 2048 tokens
// 99.6 / 110.7 / 157.8 -> 97.5 / 107.3 / 156.4 us.  The pair-ordered int8 rows and the router's partial sums too: no further change.
__device__ __forceinline__ void l2_discard(const void *p) { asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory"); }
#endif
// the same, programmatically too, in clusters of `ctas` CTAs along x
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_clusters(void (*kernel)(KArgs...), dim3 grid, unsigned ctas, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute at[2]; memset(at, 0, sizeof at);
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = ctas; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
// how many of them run at the same time on an empty GPU, at most `most`
template <typename... KArgs>
static inline int clusters_at_once(void (*kernel)(KArgs...), unsigned ctas, dim3 block, size_t smem, int most) {
    cudaLaunchConfig_t cfg; memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute at; memset(&at, 0, sizeof at);
    at.id = cudaLaunchAttributeClusterDimension; at.val.clusterDim.x = ctas; at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas, most); cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.attrs = &at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); return most; }
    return n < most ? n : most;
}
// one cluster
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_cluster(void (*kernel)(KArgs...), unsigned ctas, dim3 block, cudaStream_t st, Args... args) {
    return launch_clusters(kernel, dim3(ctas), ctas, block, 0, st, args...);
}
