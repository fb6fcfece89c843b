// span.cuh -- how long a kernel ran, taken by the kernel itself from the device's clock (globaltimer: steps of 32 ns, the same for all SMs).
//
// For kernels whose launches follow one another as the host's rows arrive: a pair of events around such a launch, on a stream that is otherwise idle,
// also holds the host's time from the first record to the launch (norm and rotation of 2048 tokens: 224 to 286 us for kernels of 27 in all).
// span[0] collects the largest complement of a start, span[1] the largest end; both are zero before.  One thread per CTA calls.
#pragma once
__device__ __forceinline__ unsigned long long device_ns() { unsigned long long t; asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); return t; }
__device__ __forceinline__ void span_begin(unsigned long long *span) { if (span) atomicMax(span, ~device_ns()); }
__device__ __forceinline__ void span_end(unsigned long long *span) { if (span) { __threadfence(); atomicMax(span + 1, device_ns()); } }      // after its own stores
