// fp8_quantize_sm100.cu — libfp8quant.so: per-tensor FP32 -> e4m3 quantiser
// (amax reduction + scale + round-to-nearest-even, saturating conversion).
// HBM-bound: the amax pass reads 4 B/element, the conversion pass reads 4 B and
// writes 1 B per element (the second read is served from L2 when the tensor
// fits).  32-byte loads (two of 16 where the input is not 32-byte aligned), an
// 8-byte store per 8 elements, contiguous over a warp.  A small tensor is done by one
// cluster in one kernel (one_cluster.cuh).
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fp8_quantize.h"
#include "one_cluster.cuh"

namespace {

using namespace sm100;

constexpr int THREADS = 256;
// Input bytes up to which one cluster does both passes: rows of 4096, 1 / 40 / 96 rows 2.4 / 4.0 / 5.0 us; two kernels behind a
// clearing one, as overlapped launches, 4.1 at 128 rows; behind a memset and in turn, as it was, 7.1 to 8.2.
constexpr size_t OC_BYTES = 768 << 10;

__global__ void clear_word_kernel(float* w) {
    pdl_wait();
    pdl_trigger();
    *w = 0.f;
}

// Eight neighbouring values: one 32-byte load where x allows it, so that a warp's load is 1 KB in a row.
template <bool WIDE>
__device__ __forceinline__ void load8(const float* x, float (&v)[8]) {
    if (WIDE) {
        uint32_t r[8];
        asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "l"(x) : "memory");
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
    } else {
        const float4 a = ld128f(x), b = ld128f(x + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}

// BATCH: groups of 8 values in flight per thread
template <bool WIDE, int BATCH>
__device__ __forceinline__ float amax_items(const float* x, size_t n, size_t tid, size_t step) {
    const size_t n8 = n / 8;
    float m = 0.f;
    for (size_t i0 = tid; i0 < n8; i0 += BATCH * step) {
        float v[BATCH][8];
#pragma unroll
        for (int u = 0; u < BATCH; u++) load8<WIDE>(x + 8 * (i0 + u * step < n8 ? i0 + u * step : i0), v[u]);   // past the end: the first again
#pragma unroll
        for (int u = 0; u < BATCH; u++)
#pragma unroll
            for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(v[u][i]));   // NaN never wins
    }
    if (tid < (n & 7)) m = fmaxf(m, fabsf(ld_f32(x + n8 * 8 + tid)));
    return m;
}

template <bool WIDE, int BATCH>
__global__ void __launch_bounds__(THREADS) amax_kernel(const float* x, size_t n, float* amax) {
    pdl_wait();
    pdl_trigger();
    float m = amax_items<WIDE, BATCH>(x, n, (size_t)blockIdx.x * blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wm[THREADS / 32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < THREADS / 32 ? wm[threadIdx.x] : 0.f;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        // non-negative floats order like their bit patterns
        if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned int*>(amax), __float_as_uint(m));
    }
}

__device__ __forceinline__ uint32_t quant4(const float* v, float inv) {
    // x * inv (one rounding, no FMA contraction possible), clamp, RN-even satfinite
    const float a = fminf(fmaxf(__fmul_rn(v[0], inv), -448.f), 448.f);
    const float b = fminf(fmaxf(__fmul_rn(v[1], inv), -448.f), 448.f);
    const float c = fminf(fmaxf(__fmul_rn(v[2], inv), -448.f), 448.f);
    const float d = fminf(fmaxf(__fmul_rn(v[3], inv), -448.f), 448.f);
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
    return lo | (hi << 16);
}

template <bool WIDE, int BATCH>
__device__ __forceinline__ void quant_items(const float* x, uint8_t* q, size_t n, size_t tid, size_t step, float amax, float* scale_out,
                                            float divisor) {
    const float scale = (amax > 1e-12f) ? __fdiv_rn(amax, divisor) : 1.0f;
    const float inv = __fdiv_rn(1.0f, scale);
    if (tid == 0) *scale_out = scale;
    const size_t n8 = n / 8;
    uint2* q8 = reinterpret_cast<uint2*>(q);
    for (size_t i0 = tid; i0 < n8; i0 += BATCH * step) {
        float v[BATCH][8];
#pragma unroll
        for (int u = 0; u < BATCH; u++) load8<WIDE>(x + 8 * (n8 - 1 - (i0 + u * step < n8 ? i0 + u * step : i0)), v[u]);   // backwards: what pass 1 read last is still in L2
#pragma unroll
        for (int u = 0; u < BATCH; u++)
            if (i0 + u * step < n8) q8[n8 - 1 - (i0 + u * step)] = make_uint2(quant4(v[u], inv), quant4(v[u] + 4, inv));
    }
    if (tid < (n & 7)) {
        const size_t i = n8 * 8 + tid;
        const float v = fminf(fmaxf(__fmul_rn(ld_f32(x + i), inv), -448.f), 448.f);
        q[i] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
    }
}

template <bool WIDE, int BATCH>
__global__ void __launch_bounds__(THREADS) quant_kernel(const float* x, uint8_t* q, size_t n, const float* amax_ptr, float* scale_out,
                                                        float divisor) {
    pdl_wait();
    pdl_trigger();
    quant_items<WIDE, BATCH>(x, q, n, (size_t)blockIdx.x * blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x, ld_f32(amax_ptr), scale_out, divisor);
}

template <bool WIDE, int BATCH>
struct QuantOp {
    static constexpr int N = 1;
    const float* x;
    uint8_t* q;
    size_t n;
    float* scale_out;
    float* amax_out;
    float divisor;
    using State = NoState;
    __device__ void ahead() const {}
    // The step of a full cluster, known to the compiler: a smaller one has a group per thread at most.  With the step from the launch, us, alone / behind a
    // GEMM of 16 x 4096 x 4096 (before clusters had sizes; now): 32 values 2.32 / 8.38 (2.12 / 8.93; 2.05 / 8.07), 4096 2.58 / 8.53 (2.53 / 9.27; 2.32 / 8.33), 53866 3.06 / 9.08
    // (2.92 / 9.76; 2.85 / 8.86).
    __device__ void pass1(float (&m)[1], State&) const { m[0] = amax_items<WIDE, BATCH>(x, n, oc_tid(), OC_STEP); }
    __device__ void pass2(const float (&m)[1], State&) const {
        if (oc_tid() == 0) *amax_out = m[0];
        quant_items<WIDE, BATCH>(x, q, n, oc_tid(), OC_STEP, m[0], scale_out, divisor);
    }
};

__global__ void __launch_bounds__(THREADS) dequant_kernel(const uint8_t* __restrict__ q, __half* __restrict__ out,
                                                          const float* __restrict__ scale_in, int n) {
    const float s = *scale_in;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const __half_raw hr = __nv_cvt_fp8_to_halfraw(q[i], __NV_E4M3);
        out[i] = __float2half_rn(__half2float(__half(hr)) * s);
    }
}

// ---- FP16 sources: the reference's own entry point (libs1/fp8_quantize_v2.cu:176-204) has no stream, no amax
// argument and allocates its reduction buffer itself; here the amax word is a per-GPU device variable, so the
// entry allocates nothing.  Calls run on the legacy default stream like the reference's and therefore serialise.
__device__ float g_amax_fp16;

__global__ void clear_amax_fp16_kernel() { g_amax_fp16 = 0.f; }

__global__ void __launch_bounds__(THREADS) amax_fp16_kernel(const __half* __restrict__ x, int n) {
    // 8 halves (16 bytes) per step when the pointer allows it, else element by element
    float m = 0.f;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const size_t n8 = (size_t)n / 8;
        const uint4* x8 = reinterpret_cast<const uint4*>(x);
        for (size_t i = tid; i < n8; i += stride) {
            const uint4 v = __ldg(x8 + i);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
                m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
            }
        }
        for (size_t i = n8 * 8 + tid; i < (size_t)n; i += stride) m = fmaxf(m, fabsf(__half2float(x[i])));
    } else {
        for (size_t i = tid; i < (size_t)n; i += stride) m = fmaxf(m, fabsf(__half2float(x[i])));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wm[THREADS / 32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < THREADS / 32 ? wm[threadIdx.x] : 0.f;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned int*>(&g_amax_fp16), __float_as_uint(m));
    }
}

__global__ void __launch_bounds__(THREADS) quant_fp16_kernel(const __half* __restrict__ x, uint8_t* __restrict__ q, int n,
                                                             float* scale_out) {
    // operation order of libs1/fp8_quantize_v2.cu:89-121: scale = amax / 448, inv = 1 / scale, v = float(x) * inv,
    // clamp to +-448, round to nearest even
    const float amax = g_amax_fp16;
    const float scale = (amax > 1e-12f) ? __fdiv_rn(amax, 448.0f) : 1.0f;
    const float inv = __fdiv_rn(1.0f, scale);
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = scale;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool vec = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) && ((reinterpret_cast<uintptr_t>(q) & 7) == 0);
    const size_t n8 = vec ? (size_t)n / 8 : 0;
    const uint4* x8 = reinterpret_cast<const uint4*>(x);
    uint2* q8 = reinterpret_cast<uint2*>(q);
    for (size_t i = tid; i < n8; i += stride) {
        const uint4 v = __ldg(x8 + i);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t c[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
            const float a = fminf(fmaxf(__fmul_rn(f.x, inv), -448.f), 448.f);
            const float b = fminf(fmaxf(__fmul_rn(f.y, inv), -448.f), 448.f);
            c[k] = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
        }
        q8[i] = make_uint2(c[0] | (c[1] << 16), c[2] | (c[3] << 16));
    }
    for (size_t i = n8 * 8 + tid; i < (size_t)n; i += stride) {
        const float v = fminf(fmaxf(__fmul_rn(__half2float(x[i]), inv), -448.f), 448.f);
        q[i] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
    }
}

// ---- block-scaled ("MXFP8") quantiser: one ue8m0 scale per 32 consecutive elements of a row (OCP microscaling:
// scale = 2^(floor(log2(amax)) - 8), 8 = the largest e4m3 exponent; elements = e4m3_rn_satfinite(x / scale)).
// One thread per block of 32: 128 bytes read, 32 codes and one scale byte written; the scale byte goes to the tiled
// position the block-scaled GEMM copies from (fp8_gemm.h: fp8_gemm_mx).
__global__ void __launch_bounds__(THREADS) quant_mx_kernel(const float* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ sf,
                                                           int rows, int K) {
    const int kblocks = K / 32;
    const size_t total = (size_t)rows * kblocks;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int row = (int)(i / kblocks), kb = (int)(i - (size_t)row * kblocks);
        const float4* src = reinterpret_cast<const float4*>(x + (size_t)row * K + kb * 32);
        float4 v[8];
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            v[j] = __ldg(src + j);
            amax = fmaxf(fmaxf(amax, fabsf(v[j].x)), fmaxf(fabsf(v[j].y), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));  // NaN never wins
        }
        int se = 0;                                   // an all-zero block keeps scale 1
        if (amax > 0.f && amax <= 3.4028234e38f) se = ilogbf(amax) - 8;
        else if (amax > 3.4028234e38f) se = 127;      // infinity in the block
        se = max(-127, min(127, se));
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            // x * 2^-se is exact (a change of exponent) unless the result is subnormal in fp32
            const float a = fminf(fmaxf(scalbnf(v[j].x, -se), -448.f), 448.f), b = fminf(fmaxf(scalbnf(v[j].y, -se), -448.f), 448.f);
            const float c = fminf(fmaxf(scalbnf(v[j].z, -se), -448.f), 448.f), d = fminf(fmaxf(scalbnf(v[j].w, -se), -448.f), 448.f);
            const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
            const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
            w[j] = lo | (hi << 16);
        }
        uint4* dst = reinterpret_cast<uint4*>(q + (size_t)row * K + kb * 32);
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
        const size_t chunk = (size_t)(row >> 7) * (K / 128) + (kb >> 2);
        sf[chunk * 512 + (row & 31) * 16 + ((row & 127) >> 5) * 4 + (kb & 3)] = (uint8_t)(se + 127);
    }
}

int grid_for(size_t work_items, int per_sm = 8) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    size_t blocks = (work_items + THREADS - 1) / THREADS;
    const size_t cap = (size_t)sms * per_sm;  // 8 CTAs of 256 threads fit an SM
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

template <bool WIDE, int BATCH>
int quantize_in_two(const float* x, uint8_t* q, float* scale_out, float* amax_out, size_t n, float divisor, cudaStream_t s) {
    // One round of BATCH loads per thread, up to four waves of CTAs: with a fixed grid the last round of 3001 rows of 4096 was half
    // empty.  With loads and stores that are contiguous over a warp (16 values a lane before, 64 bytes apart) from the start of
    // the first pass to that of the GEMM behind the second 26.2 -> 18.4 us, 2 of them the GEMM's earlier start.
    const dim3 grid(grid_for(n / (8 * BATCH) + 1, 32));
    cudaError_t e = launch_pdl(clear_word_kernel, dim3(1), dim3(1), 0, s, amax_out);
    if (e == cudaSuccess) e = launch_pdl_stream(n * 4, amax_kernel<WIDE, BATCH>, grid, dim3(THREADS), s, x, n, amax_out);
    if (e == cudaSuccess) e = launch_pdl_stream(n * 4, quant_kernel<WIDE, BATCH>, grid, dim3(THREADS), s, x, q, n, amax_out, scale_out, divisor);
    return (int)e;
}

// Loads past the end are made all the same, of values that the thread has: a small tensor waits for them in vain.  So in one cluster a
// thread has as many groups in flight as it has to take.  Before the loads were four / with four / now, us: 4096 values 2.5 / 2.9 /
// 2.4, of an input that is only 16-byte aligned 2.5 / 3.5 / 2.5; 131072 3.1 / 3.3 / 3.0 and 3.1 / 3.8 / 3.0.  In two kernels such an
// input, whose group is two loads, has two in flight up to a million values (230000 4.5 / 4.7 / 4.3).  One per thread there, in more
// CTAs, is 0.4 us faster alone, but the few-row GEMM behind it starts late (58 x 2520 x 4528, both: 12.1 / 12.6).
template <bool WIDE>
int quantize_f32(const float* x, uint8_t* q, float* scale_out, float* amax_out, size_t n, float divisor, cudaStream_t s) {
    const size_t n8 = n / 8;
    if (n * 4 <= OC_BYTES) {
        if (n8 <= OC_STEP && oc_fits<QuantOp<WIDE, 1>>()) return (int)oc_launch(QuantOp<WIDE, 1>{x, q, n, scale_out, amax_out, divisor}, s, oc_threads(n8));
        if ((!WIDE || n8 <= 2 * OC_STEP) && oc_fits<QuantOp<WIDE, 2>>()) return (int)oc_launch(QuantOp<WIDE, 2>{x, q, n, scale_out, amax_out, divisor}, s);
        if (oc_fits<QuantOp<WIDE, 4>>()) return (int)oc_launch(QuantOp<WIDE, 4>{x, q, n, scale_out, amax_out, divisor}, s);
    }
    if (!WIDE && n < ((size_t)1 << 20)) return quantize_in_two<WIDE, 2>(x, q, scale_out, amax_out, n, divisor, s);
    return quantize_in_two<WIDE, 4>(x, q, scale_out, amax_out, n, divisor, s);
}

}  // namespace

extern "C" {

int fp8_quantize_f32(const float* x, uint8_t* q, float* scale_out, float* amax_out, size_t n, int convention,
                     void* stream) {
    if (!x || !q || !scale_out || !amax_out) return (int)cudaErrorInvalidValue;
    if (convention != FP8_QUANT_AMAX_OVER_448 && convention != FP8_QUANT_UNIT) return (int)cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(q) & 15)) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    const float divisor = convention == FP8_QUANT_UNIT ? 1.0f : 448.0f;
    return (reinterpret_cast<uintptr_t>(x) & 31) ? quantize_f32<false>(x, q, scale_out, amax_out, n, divisor, s)
                                                 : quantize_f32<true>(x, q, scale_out, amax_out, n, divisor, s);
}

int fp8_dequantize_to_fp16(const void* input_fp8, void* output_fp16, const float* scale_in, int n) {
    if (!input_fp8 || !output_fp16 || !scale_in || n < 0) return (int)cudaErrorInvalidValue;
    if (n == 0) return 0;
    dequant_kernel<<<grid_for((size_t)n), THREADS>>>((const uint8_t*)input_fp8, (__half*)output_fp16, scale_in, n);
    return (int)cudaGetLastError();
}

int fp8_quantize_fp16(const void* input_fp16, void* output_fp8, float* scale_out, int n) {
    if (!input_fp16 || !output_fp8 || !scale_out || n < 0) return (int)cudaErrorInvalidValue;
    if (reinterpret_cast<uintptr_t>(input_fp16) & 1) return (int)cudaErrorInvalidValue;
    clear_amax_fp16_kernel<<<1, 1>>>();
    if (n > 0) amax_fp16_kernel<<<grid_for((size_t)n / 8 + 1), THREADS>>>((const __half*)input_fp16, n);
    quant_fp16_kernel<<<grid_for((size_t)n / 8 + 1), THREADS>>>((const __half*)input_fp16, (uint8_t*)output_fp8, n, scale_out);
    return (int)cudaGetLastError();
}

int cuda_device_sync2(void) { return (int)cudaDeviceSynchronize(); }

int fp8_quantize_mx_f32(const float* x, uint8_t* q, uint8_t* scales, int rows, int K, void* stream) {
    if (!x || !q || !scales || rows < 0 || K <= 0 || (K % 128) != 0) return (int)cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(q) & 15)) return (int)cudaErrorInvalidValue;
    if (rows == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    // entries of the padding rows of the last 128-row tile: scale 1 (never the NaN byte)
    const size_t sf_bytes = (size_t)((rows + 127) / 128) * (size_t)(K / 128) * 512;
    cudaError_t e = cudaMemsetAsync(scales, 0x7f, sf_bytes, s);
    if (e != cudaSuccess) return (int)e;
    quant_mx_kernel<<<grid_for((size_t)rows * (K / 32)), THREADS, 0, s>>>(x, q, scales, rows, K);
    return (int)cudaGetLastError();
}

}  // extern "C"
