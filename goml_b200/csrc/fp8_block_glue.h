// fp8_block_glue.h — what the block's chain (fp8_block_chain.cu) calls inside libfp8block.so: the entry points of
// include/fp8_block.h with the clearing of their maxima taken apart.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fp8_block.h"

namespace fp8_block {

// Words that an op sets to zero before anything else; with `cleared` the op takes its own maxima as zero already.
struct Words {
    float* first = nullptr;
    int n = 0;
    bool cleared = false;
};
int rmsnorm(const float* x, const void* residual_bf16, float* h_out, bool store_h, const float* gamma, uint8_t* q, float* scale_out, float* amax_out,
            float* rstd_ws, const Words& words, int rows, int hidden, float eps, cudaStream_t s);
struct Rope {
    const void* qkv_bf16;
    const float* cos_tab;
    const float* sin_tab;
    uint8_t *q_out, *k_out, *v_out;
    float *scales, *amaxes;
    uint8_t* k_cache = nullptr;   // with k_cache set: the codes also into a cache
    uint8_t* v_cache = nullptr;
    float* cache_scales = nullptr;
    int32_t* cache_lens = nullptr;
    int batch, seq_len, s_max, heads, head_dim;
};
int rope_qkv(const Rope& r, bool cleared, cudaStream_t s);
int append(const fp8_decode_append_args_t* g, bool cleared);
// state of a maximum's word when an op is called: any value, zero, or the maximum itself (no pass over the input for it)
enum class Max { ANY, ZERO, KNOWN };
int permute_heads(const void* o_fp16, uint8_t* q, float* scale_out, float* amax, int batch, int seq_len, int heads, int head_dim, Max state,
                  cudaStream_t s);

}  // namespace fp8_block
