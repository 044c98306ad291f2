// one_cluster.cuh — a per-tensor quantiser needs the maximum of the whole tensor before its first code.  For a small tensor
// (a decode step's activations, a short prompt's) the two kernels and the clearing of the maximum that this usually takes
// are three launches of 3 to 5 us each with a drain between them, for work that a few SMs do in 2 us.  Here one cluster of
// 16 CTAs does both passes: the maximum meets in distributed shared memory, nothing has to be cleared, and the second
// pass reads its input from L1 / L2.  One cluster draws about 0.9 TB/s, so larger tensors stay with the two kernels
// (as overlapped launches, with a clearing kernel in the memset's place).
//
// Loads are the coherent ones of pdl.cuh.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "pdl.cuh"

namespace sm100 {

constexpr int OC_CTAS = 16;        // more than the portable 8: a cluster of 16 fits a group of SMs of the B200
constexpr int OC_THREADS = 512;    // at most

__device__ __forceinline__ int oc_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ void oc_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void oc_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Maximum of N values over all threads of the cluster, in every thread.  All threads call it once, after one oc_arrive() at
// the kernel's start (its phase says that every CTA runs, so that its shared memory may be written).  No CTA's memory is
// touched by a peer after the return: the kernel may end.
template <int N>
__device__ __forceinline__ void oc_max(float (&m)[N]) {
    __shared__ float warp_max[N][OC_THREADS / 32];
    __shared__ float slots[N][OC_CTAS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int n = 0; n < N; n++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m[n] = fmaxf(m[n], __shfl_xor_sync(0xffffffffu, m[n], o));
        if (lane == 0) warp_max[n][warp] = m[n];
    }
    __syncthreads();
    oc_wait();
    if (threadIdx.x < OC_CTAS) {
#pragma unroll
        for (int n = 0; n < N; n++) {
            float v = warp_max[n][0];
#pragma unroll
            for (int w = 1; w < OC_THREADS / 32; w++)
                if (32 * w < (int)blockDim.x) v = fmaxf(v, warp_max[n][w]);
            const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&slots[n][oc_rank()]);
            asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.f32 [a], %2;\n\t}"
                         ::"r"(mine), "r"(threadIdx.x), "f"(v) : "memory");
        }
    }
    __syncwarp();
    oc_arrive();
    oc_wait();
#pragma unroll
    for (int n = 0; n < N; n++) {
        m[n] = slots[n][0];
#pragma unroll
        for (int c = 1; c < OC_CTAS; c++) m[n] = fmaxf(m[n], slots[n][c]);
    }
}

// Op: N maxima; ahead() runs ahead of the wait and may only ask for lines of operands; pass1(m, state) leaves this thread's maxima of
// non-negative values, pass2(m, state) is called with the tensor's; State is what a thread keeps from the one to the other
struct NoState {};
template <class Op>
__global__ void __launch_bounds__(OC_THREADS) one_cluster_kernel(const Op op) {
    oc_arrive();
    op.ahead();
    pdl_wait();
    pdl_trigger();
    typename Op::State state;
    float m[Op::N];
#pragma unroll
    for (int n = 0; n < Op::N; n++) m[n] = 0.f;
    op.pass1(m, state);
    oc_max(m);
    op.pass2(m, state);
}
__device__ __forceinline__ uint32_t oc_tid() { return (uint32_t)oc_rank() * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t oc_step() { return OC_CTAS * blockDim.x; }
constexpr uint32_t OC_STEP = OC_CTAS * OC_THREADS;   // of a full cluster

// Threads for an op of `items`, one to a thread as far as that goes.  Where there is less to do than 512 threads a CTA, a smaller CTA finds its registers on
// an SM beside the CTAs of the GEMM ahead and waits there, instead of being launched when those have gone (a step of two sequences, us, 512 threads always /
// so: 73.7 / 72.2, of three 76.1 / 74.9, of eight 85.9 / 85.2).
inline int oc_threads(size_t items) {
    const size_t t = (items + OC_CTAS * 32 - 1) / (OC_CTAS * 32) * 32;
    return (int)(t < 32 ? 32 : t > OC_THREADS ? OC_THREADS : t);
}

template <class Op>
inline cudaLaunchConfig_t oc_config(cudaLaunchAttribute* attr, cudaStream_t stream, int threads = OC_THREADS, int carveout = -1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(OC_CTAS);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = OC_CTAS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[2].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[2].val.sharedMemCarveout = carveout;
    cfg.attrs = attr;
    cfg.numAttrs = carveout < 0 ? 2 : 3;
    return cfg;
}

// whether this GPU has a group of SMs that holds the cluster (asked once per kernel and GPU)
template <class Op>
inline bool oc_fits() {
    static std::atomic<int> known[64];   // 0 not asked, 1 yes, 2 no
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int k = known[dev].load(std::memory_order_acquire);
    if (k == 0) {
        int clusters = 0;
        cudaLaunchAttribute attr[3];
        cudaLaunchConfig_t cfg = oc_config<Op>(attr, nullptr);
        cfg.numAttrs = 1;
        const bool ok = cudaFuncSetAttribute(one_cluster_kernel<Op>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&clusters, one_cluster_kernel<Op>, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) (void)cudaGetLastError();
        k = ok ? 1 : 2;
        known[dev].store(k, std::memory_order_release);
    }
    return k == 1;
}

// carveout: the per cent of an SM's storage that the kernel wants for shared memory.  With it a CTA is not put on an SM while CTAs there have
// another share.
template <class Op>
inline cudaError_t oc_launch(const Op& op, cudaStream_t stream, int threads = OC_THREADS, int carveout = -1) {
    cudaLaunchAttribute attr[3];
    const cudaLaunchConfig_t cfg = oc_config<Op>(attr, stream, threads, carveout);
    return cudaLaunchKernelEx(&cfg, one_cluster_kernel<Op>, op);
}

}  // namespace sm100
