// pdl.cuh — programmatic dependent launch: a kernel of this directory is launched before its predecessor on the stream
// has drained, runs its set-up (barriers, tensor memory, descriptor prefetch, cache hints) and waits on the device for
// the predecessor's completion before it touches dependent data.
//
// Four rules keep the stream's order intact:
//  * pdl_wait() comes before the first read of anything an earlier kernel may have written and before the first write to
//    global memory, in every kernel, on every path that touches global memory; a kernel does not complete before every
//    kernel ahead of it has, because some thread of each of its CTAs waits before the CTA ends;
//  * a kernel whose successor reads before its own wait (the attention forward, behind its V pre-pass) calls
//    pdl_trigger() only after pdl_wait(): everything ahead of the pair has then completed;
//  * what any kernel may do before its wait is to ask for lines of an operand to be brought into L2: a hint moves no
//    data into the SM, and L2 is where stores of the kernel ahead land, so it cannot be stale.  What only says where a hint goes
//    (lengths, a block table) may be read for it as well, past L1, if any value leads to an address inside the operand;
//  * no load of such a kernel takes the read-only path (__ldg, a const __restrict__ pointer): that is for data that nobody
//    writes while the kernel exists, so it may be served from before the wait, by the compiler or by an L1 line that the
//    wait does not invalidate.  Plain loads and the ones below are ordered behind the wait.
// Both instructions do nothing in a launch without the attribute.
//
// What it buys: the gap between two dependent kernels of a few microseconds each falls from 1.5-2.5 us to under 1 us.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sm100 {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// coherent loads
__device__ __forceinline__ uint4 ld128(const void* p) {
    uint4 r;
    asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ float4 ld128f(const void* p) {
    float4 r;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ float ld_f32(const float* p) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ int ld_s32(const int* p) {
    int r;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(r) : "l"(p) : "memory");
    return r;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// The same for a kernel that streams `bytes`.  Launched early behind one that takes most of an SM's shared memory it would find the
// SM's storage given to that, and loads in flight need lines of what is left: 28 KB hold it to two thirds of the memory's
// rate (and the kernels behind it, as long as no SM runs empty).  A large one asks for L1, which keeps its CTAs off an SM until
// that can be had; for a small one being there early is worth more (16384 rows behind a GEMM 111 -> 79 us, 16 rows 1 us slower).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_stream(size_t bytes, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = cudaSharedmemCarveoutMaxL1;
    cfg.attrs = attr;
    cfg.numAttrs = bytes >= ((size_t)16 << 20) ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace sm100
