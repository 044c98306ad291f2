// fp8_gemm_skinny.cuh — the GEMM for few rows of A (M up to 192: the tokens of a decode step or of a short prompt).
// Included by fp8_gemm_sm100.cu, which owns the argument checks, the status word and the call of plan().
//
// Such a product reads the weight B[N,K] once and does next to no arithmetic: its floor is N*K bytes of HBM traffic.  What
// it needs is many bytes in flight from the first microsecond to the last, which the square kernel does not give it (it
// puts the tokens on the 128 MMA rows, fills half of shared memory with zero rows for them, covers N with as few as 64
// CTAs and streams a weight panel twice once M passes 128).  Here
//  * the weight rows are the MMA's M dimension and the tokens its N dimension (any multiple of 16), so a stage of the ring
//    holds 16 KB of weights and only 128 bytes per token, and every weight byte is read once;
//  * the K range of a 128-row tile is cut over a thread-block cluster of 1 to 8 CTAs; the fp32 partial sums meet in
//    distributed shared memory and are added in rank order (no atomics: the result does not depend on timing);
//  * all CTAs are resident at once, up to three to an SM, so the kernel is one wave of equal streams (an SM takes in about
//    57 bytes a nanosecond, so weights have to be spread over nearly all of them to reach the 6.5 TB/s of HBM);
//  * the kernel starts before its predecessor on the stream has drained and asks for its first weight tiles to be
//    brought into L2 while the small kernel ahead (a quantiser, usually) still runs.
// What is left is 3 us of start, fill and finish beside the stream: M = 16, 8192 x 8192 14.0 us (floor 10.3),
// 12288 x 4096 11.2 (7.7), 22016 x 4096 with SwiGLU
// 18.4 (13.8), 4096 x 11008 10.7 (6.9), 4096 x 4096 6.5 (2.6).
#pragma once

namespace skinny {

constexpr int W_ROWS = 128;                 // weight rows per tile = TMEM lanes
constexpr int W_BYTES = W_ROWS * BK;        // of one k-block
constexpr int MAX_TOKENS = 192;
constexpr int MAX_STAGES = 16;
// Most tokens whose partial sums go straight to their owners, with one meeting of the cluster behind the last MMA in the place of two and of reads from
// other CTAs (us, before / so): 16 tokens, 2048 x 2048 4.76 / 4.00, 1504 x 6000 6.47 / 5.87, 4096 x 11008 added 11.1 / 10.7, 8192 x 8192 14.4 / 14.2; 5 tokens,
// 3001 x 3008 5.70 / 5.19.  With more, 4 bytes at a time to another CTA take longer than 16 at a time from it: 64 tokens, 4096 x 4096 added 7.77 / 8.28
// (fetched, with scales asked for ahead of the meeting: 7.59), 173 tokens 10.0 / 11.8 (9.80).
constexpr int APART_TOKENS = 16;
constexpr int MAX_SPLIT = 8;                // portable cluster size
constexpr int THREADS = 192;                // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-5: read the accumulators back
constexpr int TAIL_BYTES = 1024 /*align*/ + 512 /*barriers*/;
constexpr int SMEM_ONE = 227 * 1024;        // of one CTA when it has the SM to itself
constexpr int SMEM_LONG = 160 * 1024;       // what it takes of that for a long stream
// shared memory of one of up to three CTAs on an SM (228 KB, 1 KB of it the system's for each CTA)
constexpr int smem_of(int per_sm) { return per_sm == 1 ? SMEM_ONE : per_sm == 2 ? 112 * 1024 : 75 * 1024; }

// Where the codes of the tokens come from: a matrix of them, or (a step of a few sequences) the values that they are made of, which
// every CTA quantises for itself.  Values of at most MAX_ROWS tokens, of all of K, have one scale, max|value| / 448.  A row costs the
// four products of a block 4 to 5 us, the quantisers ahead of them 15 to 18 however few rows there are: a step of a block 4096 wide, of one
// sequence 73.5 -> 65.3 us, of two 75.6 / 73.2 (a form that took more lost with three, 81.9 / 82.8, and four, 86 / 92).  How long the rows may be
// is for the caller to say: the block's chain has the line.
constexpr int MAX_ROWS = 2;
enum Source : int { CODES = 0, RMS_F32 = 1, F16 = 2, BF16_KNOWN = 3 };   // RMSNorm of fp32 rows; fp16 values; bf16 values whose maximum is known
struct Rows {
    int source;
    const void* x;         // [M, K]
    const float* gamma;    // RMS_F32
    float eps;
    const float* amax;     // BF16_KNOWN
    const float* x_in;     // accumulate mode: X = x_in + alpha A B^T
    float* zero;           // words set to 0 for later kernels
    int zeros;
    int early;             // the weight is complete when this kernel starts: its first tiles are loaded ahead of the wait
};
constexpr int TOKEN_BYTES = 8 * BK;   // a k-block of such codes: one swizzle atom of eight rows

struct Params {
    GemmParams g;
    Rows r;
    int tn;            // tokens rounded up to 16: MMA N
    int tmem_cols;
    uint32_t idesc;
    int stages;
    int slice;         // most k-blocks of a CTA
    int prefetch;      // k-blocks per CTA asked for ahead of the wait
    int vec;           // four neighbouring outputs of a token may be stored at once
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void prefetch_l2_2d(const CUtensorMap* m, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];"
                 ::"l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y) : "memory");
}
// Who finishes what.  APART: a tile's 128 weight rows are 16 pairs of 4 rows and the 4 rows 32 further on (with SwiGLU: gate rows and their up
// rows), dealt to the CTAs of the cluster in runs of up to PAIRS; the partial sums lie with the owner as [source][token][half][PAIRS][4].
// Else they lie with their source, as [token][128].
__host__ __device__ constexpr int pairs_of(int split) { return (16 + split - 1) / split; }
__host__ __device__ constexpr int apart_bytes(int split, int tokens) { return split * tokens * 2 * pairs_of(split) * 16; }
// with rows as values at least the block that the last MMAs read behind the codes
__host__ __device__ constexpr int part_room(int split, int tokens, bool values) {
    return values && apart_bytes(split, tokens) < TOKEN_BYTES ? TOKEN_BYTES : apart_bytes(split, tokens);
}
template <int SPLIT>
__device__ __forceinline__ int first_pair(int rank) { return (16 * rank + SPLIT - 1) / SPLIT; }   // owner of pair u: u * SPLIT / 16
// the sums of all sources for four rows and a token; a: where they lie in this CTA
template <int SPLIT, int APART>
__device__ __forceinline__ void gather(float4* v, uint32_t a, uint32_t source_bytes) {
#pragma unroll
    for (int s = 0; s < SPLIT; s++) {
        if (SPLIT == 1 || APART)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[s].x), "=f"(v[s].y), "=f"(v[s].z), "=f"(v[s].w) : "r"(a + s * source_bytes) : "memory");
        else
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[s].x), "=f"(v[s].y), "=f"(v[s].z), "=f"(v[s].w) : "r"(map_rank(a, s)) : "memory");
    }
}
template <int SPLIT>
__device__ __forceinline__ void add_up(const float4* v, float* r) {
    r[0] = v[0].x; r[1] = v[0].y; r[2] = v[0].z; r[3] = v[0].w;
#pragma unroll
    for (int s = 1; s < SPLIT; s++) { r[0] += v[s].x; r[1] += v[s].y; r[2] += v[s].z; r[3] += v[s].w; }
}

__device__ __forceinline__ uint32_t rows_quant4(float a, float b, float c, float d, float inv) {   // the quantiser's formula
    const float x[4] = {a, b, c, d};
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; i++) y[i] = fminf(fmaxf(__fmul_rn(x[i], inv), -448.f), 448.f);
    return pack_e4m3x4(y[0], y[1], y[2], y[3]);
}
// The codes of k-blocks [kb0, kb1) of all tokens, as a TMA load with 128-byte swizzle would leave them, and their scale.  By the four
// warps that wait for the accumulators otherwise (tid 0 .. 127); every CTA goes over all of K for the maximum, which for a few tokens is
// less than a second meeting of CTAs costs.  red: 4 * 2 * MAX_ROWS floats of shared memory.
__device__ __forceinline__ void quantise_rows(const Params& p, uint32_t tok, float* red, float* scale_out, int kb0, int kb1, int tid) {
    const Rows& r = p.r;
    const int M = p.g.M, K = p.g.K, warp = tid >> 5, lane = tid & 31;
    const float* xf = static_cast<const float*>(r.x);
    const uint8_t* xh = static_cast<const uint8_t*>(r.x);
    float amax = 0.f;
    if (r.source == BF16_KNOWN) {
        amax = ld_f32(r.amax);
    } else {
#pragma unroll 1
        for (int j = 0; j < M; j++) {
            float ss = 0.f, top = 0.f;
            if (r.source == RMS_F32) {
                const float* row = xf + (size_t)j * K;
                constexpr int U = 8;   // loads in flight: one latency for 4096 values
#pragma unroll 1
                for (int c0 = tid * 4; c0 < K; c0 += 512 * U) {
                    float4 h[U], g[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int c = c0 + u * 512;
                        h[u] = g[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (c < K) { h[u] = ld128f(row + c); g[u] = ld128f(r.gamma + c); }
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        ss = fmaf(h[u].x, h[u].x, ss); ss = fmaf(h[u].y, h[u].y, ss);
                        ss = fmaf(h[u].z, h[u].z, ss); ss = fmaf(h[u].w, h[u].w, ss);
                        top = fmaxf(fmaxf(top, fmaxf(fabsf(__fmul_rn(h[u].x, g[u].x)), fabsf(__fmul_rn(h[u].y, g[u].y)))),
                                    fmaxf(fabsf(__fmul_rn(h[u].z, g[u].z)), fabsf(__fmul_rn(h[u].w, g[u].w))));
                    }
                }
            } else {
                constexpr int U = 4;
#pragma unroll 1
                for (int c0 = tid * 8; c0 < K; c0 += 1024 * U) {
                    uint4 v[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int c = c0 + u * 1024;
                        v[u] = make_uint4(0u, 0u, 0u, 0u);
                        if (c < K) v[u] = ld128(xh + ((size_t)j * K + c) * 2);
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                            top = fmaxf(top, fmaxf(fabsf(f.x), fabsf(f.y)));   // NaN never wins
                        }
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                ss += __shfl_xor_sync(0xffffffffu, ss, o);
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            }
            if (lane == 0) {
                red[(j * 4 + warp) * 2] = ss;
                red[(j * 4 + warp) * 2 + 1] = top;
            }
        }
        named_bar_sync(1, 128);
    }
    // of row j, from the four warps' parts in a fixed order: the same in every CTA
    auto rstd_of = [&](int j) {
        return __frsqrt_rn(__fadd_rn(__fdiv_rn(((red[j * 8] + red[j * 8 + 2]) + red[j * 8 + 4]) + red[j * 8 + 6], (float)K), r.eps));
    };
    float rstd0 = 1.f;
    if (r.source != BF16_KNOWN)
        for (int j = 0; j < M; j++) {
            const float top = fmaxf(fmaxf(red[j * 8 + 1], red[j * 8 + 3]), fmaxf(red[j * 8 + 5], red[j * 8 + 7]));
            const float rstd = r.source == RMS_F32 ? rstd_of(j) : 1.f;
            if (j == 0) rstd0 = rstd;
            amax = fmaxf(amax, r.source == RMS_F32 ? __fmul_rn(top, rstd) : top);
        }
    const float scale = amax > 1e-12f ? __fdiv_rn(amax, 448.0f) : 1.0f;
    const float inv = __fdiv_rn(1.0f, scale);
    if (tid == 0) *scale_out = scale;
    const int chunks = (kb1 - kb0) * (BK / 16);   // of 16 codes; those past K are zeros
#pragma unroll 1
    for (int j = 0; j < M; j++) {
        const float rstd = r.source != RMS_F32 ? 1.f : j == 0 ? rstd0 : rstd_of(j);
        for (int it = tid; it < chunks; it += 128) {
            const int col = kb0 * BK + it * 16;
            uint4 q = make_uint4(0u, 0u, 0u, 0u);
            if (col < K) {
                float y[16];
                if (r.source == RMS_F32) {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float4 h = ld128f(xf + (size_t)j * K + col + 4 * i), g = ld128f(r.gamma + col + 4 * i);
                        y[4 * i] = __fmul_rn(__fmul_rn(h.x, g.x), rstd);
                        y[4 * i + 1] = __fmul_rn(__fmul_rn(h.y, g.y), rstd);
                        y[4 * i + 2] = __fmul_rn(__fmul_rn(h.z, g.z), rstd);
                        y[4 * i + 3] = __fmul_rn(__fmul_rn(h.w, g.w), rstd);
                    }
                } else {
                    const uint8_t* src = xh + ((size_t)j * K + col) * 2;
                    const uint4 v0 = ld128(src), v1 = ld128(src + 16);
                    const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (r.source == F16) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                            y[2 * i] = f.x;
                            y[2 * i + 1] = f.y;
                        } else {
                            y[2 * i] = __uint_as_float(w[i] << 16);
                            y[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                        }
                    }
                }
                q = make_uint4(rows_quant4(y[0], y[1], y[2], y[3], inv), rows_quant4(y[4], y[5], y[6], y[7], inv),
                               rows_quant4(y[8], y[9], y[10], y[11], inv), rows_quant4(y[12], y[13], y[14], y[15], inv));
            }
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(tok + (it >> 3) * TOKEN_BYTES + j * BK + (((it & 7) ^ j) << 4)),
                         "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
        }
    }
}

// VALUES: the tokens come as values (Rows), else as codes.  APART: the partial sums have shared memory of their own, else the ring's place.
template <int SPLIT, bool VALUES, int APART>
// Three CTAs on an SM put up to five of their warps on one of its four schedulers, whose registers hold five of 96 registers a thread: the
// bound says 224 threads so that the compiler stays there (with 104 the third CTA waits for the first to end).
__global__ void __launch_bounds__(224, 3)
fp8_gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_t, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;   // swizzle atoms are 1024 bytes
    uint8_t* ring_gen = smem_raw + (ring - smem_u32(smem_raw));
    const int stage_bytes = VALUES ? W_BYTES : W_BYTES + p.tn * BK;   // a multiple of 2048
    // VALUES: the codes of this CTA's k-blocks, eight rows each.  The MMA takes sixteen tokens; the other eight, whose sums nobody looks at, it
    // finds in the block behind, be it codes or partial sums that arrive
    const uint32_t tok = ring + p.stages * stage_bytes;
    const uint32_t tok_bytes = VALUES ? p.slice * TOKEN_BYTES : 0;
    const uint32_t part = APART ? tok + tok_bytes : ring;
    const uint32_t part_bytes = APART ? part_room(SPLIT, p.g.M, VALUES) : 0;
    const uint32_t bar_full = tok + tok_bytes + part_bytes;
    const uint32_t bar_empty = bar_full + 8 * MAX_STAGES;
    const uint32_t bar_done = bar_empty + 8 * MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring_gen + p.stages * stage_bytes + tok_bytes + part_bytes + 16 * MAX_STAGES + 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t bar_tok = bar_done + 16;
    float* scale_slot = reinterpret_cast<float*>(tmem_slot + 4);
    float* red = scale_slot + 2;                                      // 8 * MAX_ROWS floats
    static_assert(16 * MAX_STAGES + 8 + 24 + 32 * MAX_ROWS <= 512, "barriers and words fit the tail");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % SPLIT;
    const int n0 = ((int)blockIdx.x / SPLIT) * W_ROWS;
    const int kb0 = (int)((long long)rank * p.g.k_blocks / SPLIT), kb1 = (int)((long long)(rank + 1) * p.g.k_blocks / SPLIT);

    if (APART) cluster_arrive();   // its phase says that every CTA runs, so that its shared memory may be written
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_done, 1);
        if (VALUES) mbar_init(bar_tok, 128);
        *abort_flag = 0;
        fence_mbar_init();
    }
    __syncwarp();
    if (warp == 0) {
        const int pf1 = min(kb1, kb0 + p.prefetch);
        for (int kb = kb0 + lane; kb < pf1; kb += 32) prefetch_l2_2d(&tmap_w, kb * BK, n0);
        __syncwarp();
    } else if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    int kb_next = kb0;   // first k-block of the weight that is not on its way yet
    if (VALUES && p.r.early && warp == 0) {
        const bool leader = elect_one();
        for (int i = 0; i < p.stages && kb_next < kb1; i++, kb_next++) {
            if (leader) {
                mbar_arrive_expect_tx(bar_full + 8 * i, W_BYTES);
                tma_load_2d(ring + i * W_BYTES, &tmap_w, bar_full + 8 * i, kb_next * BK, n0);
            }
        }
        __syncwarp();
    }
    pdl_wait();
    pdl_trigger();
    bool acc_ready = false;   // this warp may read the accumulators
    if (VALUES && blockIdx.x == 0 && (int)threadIdx.x < p.r.zeros) p.r.zero[threadIdx.x] = 0.f;

    if (warp == 0) {
        const bool leader = elect_one();
        int stage = (kb_next - kb0) % p.stages;
        uint32_t phase = kb_next - kb0 == p.stages ? 0 : 1;
        for (int kb = kb_next; kb < kb1; kb++) {
            if (!mbar_wait_warp(bar_empty + 8 * stage, phase, abort_flag, ST_TIMEOUT_PRODUCER)) break;
            if (leader) {
                const uint32_t fb = bar_full + 8 * stage, sw = ring + stage * stage_bytes;
                mbar_arrive_expect_tx(fb, stage_bytes);   // parts of a box outside the matrix are zero-filled and counted
                tma_load_2d(sw, &tmap_w, fb, kb * BK, n0);
                if (!VALUES) tma_load_2d(sw + W_BYTES, &tmap_t, fb, kb * BK, 0);
            }
            __syncwarp();
            if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        int stage = 0;
        uint32_t phase = 0;
        bool ok = !VALUES || mbar_wait_warp(bar_tok, 0, abort_flag, ST_TIMEOUT_MMA);
        for (int kb = kb0; kb < kb1 && ok; kb++) {
            if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag, ST_TIMEOUT_MMA)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sw = ring + stage * stage_bytes;
            const uint64_t wdesc = kmajor_desc_sw128(sw), tdesc = kmajor_desc_sw128(VALUES ? tok + (kb - kb0) * TOKEN_BYTES : sw + W_BYTES);
#pragma unroll
            for (int k = 0; k < BK / 32; k++)
                if (leader) mma_f8f6f4_ss(tmem, wdesc + 2 * k, tdesc + 2 * k, p.idesc, ((kb - kb0) | k) != 0);
            if (leader) mma_commit(bar_empty + 8 * stage);
            __syncwarp();
            if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        if (ok && leader) mma_commit(bar_done);
        __syncwarp();
    } else {
        if (VALUES) {
            quantise_rows(p, tok, red, scale_slot, kb0, kb1, (int)threadIdx.x - 64);
            fence_proxy_async_smem();
            mbar_arrive(bar_tok);
            __syncwarp();
        }
        acc_ready = mbar_wait_warp(bar_done, 0, abort_flag, ST_TIMEOUT_EPILOGUE);
        tc_fence_after();
    }
    __syncwarp();

    // ---- finish: the CTAs of the cluster share the tile's outputs.  With little to hand over, a CTA's partial sums go to their owners, into memory
    // that the ring never uses, and one meeting does; else they take the ring's place (free by then: every load that was issued has been consumed by
    // an MMA that has retired), the owners fetch them behind a meeting, and nobody leaves before another.
    const GemmParams& g = p.g;
    constexpr int PAIRS = pairs_of(SPLIT);
    const int u0 = first_pair<SPLIT>(rank), pairs = first_pair<SPLIT>(rank + 1) - u0;   // APART: what this CTA owns
    const uint32_t source_bytes = g.M * 2 * PAIRS * 16;
    // asked for ahead of the meeting
    float alpha = g.alpha;
    if (!VALUES && g.scale_a) alpha *= ld_f32(g.scale_a);
    const float scale_b = g.scale_b ? ld_f32(g.scale_b) : 1.0f;
    const float scale_d = (g.D8 && g.scale_d) ? ld_f32(g.scale_d) : 1.0f;
    if (APART) cluster_wait();
    if (acc_ready) {   // neighbouring lanes write neighbouring words
        const int quad = warp & 3, row = quad * 32 + lane;
        const int u = (row >> 6) * 8 + ((row >> 2) & 7), owner = u * SPLIT / 16;
        const uint32_t dst = !APART ? part + row * 4
                                    : map_rank(part + rank * source_bytes + ((quad & 1) * PAIRS + u - first_pair<SPLIT>(owner)) * 16 + (row & 3) * 4, owner);
        constexpr int TOKEN = APART ? 2 * PAIRS * 16 : W_ROWS * 4;
        for (int j0 = 0; j0 < (APART ? g.M : p.tn); j0 += 16) {
            uint32_t acc[16];
            tmem_ld_32x32b_x16(tmem + j0 + (uint32_t(quad * 32) << 16), acc);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i++) {
                if (!APART) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (j0 + i) * TOKEN), "r"(acc[i]) : "memory");
                else if (j0 + i < g.M) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(dst + (j0 + i) * TOKEN), "r"(acc[i]) : "memory");
            }
        }
        tc_fence_before();
    }
    __syncwarp();
    cluster_arrive();
    {
        // The CTAs of the cluster finish the tile's outputs together, groups of four outputs of a token.  A thread takes several groups at a time,
        // all their loads (partial sums, and the residual stream in the accumulate mode) issued before the first use: one group at a time was bound
        // by their latency (0.35 us a round, 16 rounds for 64 tokens).
        constexpr int STEP = APART ? THREADS : SPLIT * THREADS;
        const int first = APART ? (int)threadIdx.x : rank * THREADS + (int)threadIdx.x;
        float tmax = 0.f;
        if (g.H) {
            // gate rows [64c, 64c + 32), up rows [64c + 32, 64c + 64) of the tile
            constexpr int QUADS = APART ? PAIRS : 16;   // groups of four activation columns
            constexpr int U = SPLIT == 1 ? 4 : SPLIT == 2 ? 2 : 1;
            const int items = g.M * QUADS;
            cluster_wait();
            if (VALUES) alpha *= *scale_slot;
            alpha *= scale_b;
            for (int it0 = first; it0 < items; it0 += U * STEP) {
                float4 gt[U][SPLIT], up[U][SPLIT];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int it = min(it0 + u * STEP, items - 1), j = it / QUADS, q = it % QUADS;
                    const uint32_t at = part + (APART ? (j * 2 * PAIRS + q) * 16 : j * (W_ROWS * 4) + ((q >> 3) * 64 + (q & 7) * 4) * 4);
                    gather<SPLIT, APART>(gt[u], at, source_bytes);
                    gather<SPLIT, APART>(up[u], at + (APART ? PAIRS * 16 : 32 * 4), source_bytes);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int it = it0 + u * STEP, j = it / QUADS, q = it % QUADS;
                    if (it >= items) break;
                    const int col = (n0 >> 1) + (APART ? u0 + q : q) * 4;
                    float gv[4], uv[4], h[4];
                    add_up<SPLIT>(gt[u], gv);
                    add_up<SPLIT>(up[u], uv);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float a = gv[i] * alpha;
                        float r;
                        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + __expf(-a)));
                        h[i] = a * r * (uv[i] * alpha);
                    }
                    const uint32_t w[2] = {pack_out(h[0], h[1], 1), pack_out(h[2], h[3], 1)};
                    if (col >= g.F || (APART && q >= pairs)) continue;
#pragma unroll
                    for (int i = 0; i < 2; i++)   // max of the rounded values; columns past F are zero
                        tmax = fmaxf(tmax, fmaxf(fabsf(__uint_as_float(w[i] << 16)), fabsf(__uint_as_float(w[i] & 0xffff0000u))));
                    uint16_t* dst = reinterpret_cast<uint16_t*>(g.H) + (size_t)j * g.F + col;
                    if (p.vec && col + 4 <= g.F) {
                        *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            if (col + i < g.F) dst[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
                    }
                }
            }
        } else {
            constexpr int QUADS = APART ? 2 * PAIRS : W_ROWS / 4;
            constexpr int U = SPLIT <= 2 ? 4 : SPLIT <= 4 ? 2 : 1;
            const int items = g.M * QUADS;
            auto column = [&](int r) {   // of a token's group r; none of it there: N
                if (!APART) return n0 + r * 4;
                const int half = r >= PAIRS, q = r - half * PAIRS, u = u0 + q;
                return q < pairs ? n0 + (u >> 3) * 64 + half * 32 + (u & 7) * 4 : g.N;
            };
            float x[U][4];
            auto residual = [&](int it0) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int it = min(it0 + u * STEP, items - 1), j = it / QUADS, col = column(it % QUADS);
                    const float* src = (VALUES ? p.r.x_in : g.X) + (size_t)j * g.N + col;
                    if (p.vec && col + 4 <= g.N) {
                        const float4 t = *reinterpret_cast<const float4*>(src);
                        x[u][0] = t.x; x[u][1] = t.y; x[u][2] = t.z; x[u][3] = t.w;
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++) x[u][i] = col + i < g.N ? src[i] : 0.f;
                    }
                }
            };
            if (APART && g.X) residual(first);   // only this thread writes there: it need not wait for the meeting
            __syncwarp();
            cluster_wait();
            if (VALUES) alpha *= *scale_slot;
            alpha *= scale_b;
            for (int it0 = first; it0 < items; it0 += U * STEP) {
                float4 sums[U][SPLIT];
                if (g.X && !(APART && it0 == first)) residual(it0);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int it = min(it0 + u * STEP, items - 1), j = it / QUADS, r = it % QUADS;
                    gather<SPLIT, APART>(sums[u], part + (j * QUADS + r) * 16, source_bytes);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int it = it0 + u * STEP, j = it / QUADS, col = column(it % QUADS);
                    if (it >= items) break;
                    if (col >= g.N) continue;
                    float v[4];
                    add_up<SPLIT>(sums[u], v);
                    const size_t off = (size_t)j * g.N + col;
                    const bool whole = p.vec && col + 4 <= g.N;
                    if (g.X) {
#pragma unroll
                        for (int i = 0; i < 4; i++) v[i] = fmaf(v[i], alpha, x[u][i]);
                        if (whole) {
                            *reinterpret_cast<float4*>(g.X + off) = make_float4(v[0], v[1], v[2], v[3]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                if (col + i < g.N) g.X[off + i] = v[i];
                        }
                        continue;
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] *= alpha;
                    if (g.D8) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            tmax = fmaxf(tmax, fabsf(v[i]));   // columns past N are zero
                            v[i] *= scale_d;
                        }
                        const uint32_t w = pack_e4m3x4(v[0], v[1], v[2], v[3]);
                        if (whole) {
                            *reinterpret_cast<uint32_t*>(g.D8 + off) = w;
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                if (col + i < g.N) g.D8[off + i] = (uint8_t)(w >> (8 * i));
                        }
                    } else {
                        const uint32_t w[2] = {pack_out(v[0], v[1], g.out_bf16), pack_out(v[2], v[3], g.out_bf16)};
                        uint16_t* dst = reinterpret_cast<uint16_t*>(g.C) + off;
                        if (whole) {
                            *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                if (col + i < g.N) dst[i] = (uint16_t)(w[i >> 1] >> (16 * (i & 1)));
                        }
                    }
                }
            }
        }
        if (g.amax) {
            __syncwarp();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
            if (lane == 0) atomicMax(reinterpret_cast<unsigned int*>(g.amax), __float_as_uint(tmax));
        }
    }
    // ------------------------------------------------------------- teardown
    __syncwarp();
    if (SPLIT > 1 && !APART) {   // peers have read this CTA's sums
        cluster_arrive();
        cluster_wait();
    }
    const uint32_t code = *abort_flag;
    if (code != 0) {
        if (threadIdx.x == 0) atomicCAS(&g_gemm_status, 0u, code);
        for (int i = 0; i < 200; i++) __nanosleep(1000);   // copies in flight land before shared memory is released
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, p.tmem_cols);
    }
}

using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const Params);
// kinds: codes with the sums in the ring's place or apart, values
inline Kernel kernel_for(int split, int kind) {
#define GOML_KINDS(S) {fp8_gemm_skinny_kernel<S, false, 0>, fp8_gemm_skinny_kernel<S, false, 1>, fp8_gemm_skinny_kernel<S, true, 1>}
    static const Kernel table[MAX_SPLIT][3] = {GOML_KINDS(1), GOML_KINDS(2), GOML_KINDS(3), GOML_KINDS(4), GOML_KINDS(5), GOML_KINDS(6), GOML_KINDS(7), GOML_KINDS(8)};
#undef GOML_KINDS
    return table[split - 1][kind];
}

// clusters of each size that are resident at once with one CTA to an SM (a cluster stays inside one group of SMs, so this
// is less than SMs / size); with n CTAs to an SM it is at least n times as many
struct Fit {
    int one[MAX_SPLIT + 1] = {};
};

inline void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int tiles, int split, size_t smem, cudaStream_t stream) {
    cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * split));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
}

inline cudaError_t init(Fit* fit) {
    for (int split = 1; split <= MAX_SPLIT; split++) {
        cudaError_t e = cudaSuccess;
        for (int kind = 0; kind < 3; kind++) {
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel_for(split, kind), cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ONE);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel_for(split, kind), cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        }
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        configure(cfg, attr, 1, split, SMEM_ONE, nullptr);
        cfg.numAttrs = 1;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fit->one[split], kernel_for(split, 0), &cfg);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// How a problem is cut, or split = 0 where the square kernel is the faster one.  added: the output is added to an fp32 matrix by
// the copy engine, so that the square kernel cuts a long K as well; codes: it is e4m3.
struct Plan {
    int split = 0;
    int per_sm = 1;     // CTAs that share an SM and its shared memory
};
inline Plan plan(int M, int N, int K, bool added, bool codes, int num_sms, const Fit& fit) {
    Plan r;
    if (M > MAX_TOKENS) return r;
    const long long weights = (long long)N * K;
    const long long tiles = ((long long)N + W_ROWS - 1) / W_ROWS;
    const int k_blocks = (K + BK - 1) / BK, tn = (M + 15) / 16 * 16;
    // Past 80 tokens the tokens' own traffic and the longer finish (2 us more at 128) weigh against a square kernel that
    // needs one row of tiles, for small weights whose K is short: 100 tokens, 2048 x 2048 6.7 / 6.3 us, 8192 x 2048 (128) 9.0 / 7.6, but
    // 4096 x 4096 8.4 / 9.3, 2000 x 3008 7.3 / 7.9, 1024 x 8192 8.4 / 13.6.  Past 128 that one reads the weight twice: 150 tokens, 2048
    // x 2048 7.5 / 6.5, 4096 x 4000 9.9 / 10.0, 2000 x 5008 10.4 / 14.6; 190 tokens, 1504 x 6000 12.1 / 16.5.
    // Codes cost this kernel's finish more: 100 tokens, 2048 x 3008 10.8 / 10.3, 3504 long 12.4 / 14.4.  Where the square kernel cuts K
    // too, it is ahead for all small weights: 100 tokens, 1024 x 8192 7.8 / 5.4 (behind a quantiser 9.5 / 8.2), 2048 x 11008 10.1 / 8.4,
    // 192, 512 x 8192 9.3 / 5.3, 2048 x 5504 9.8 / 8.1; 4096 x 6000 alone is not (100 tokens 10.7 / 11.9).
    const int short_k = M > 128 ? 4800 : codes ? 3500 : 3000;
    if (M > 80 && weights < (M > 128 ? 1ll << 24 : 1ll << 25) && (added || K < short_k)) return r;
    // the K range is cut as long as all slices are resident, one to an SM, and two k-blocks are left to each (16 tokens, 1 / 2 /
    // 3 / 4 slices: 8192 x 8192 17.4 / 13.9 / 14.8 / 13.7 us, of which 2 fit; 4096 x 4096 9.9 / 7.0 / 6.3 / 6.2);
    // past four slices the finish grows faster than the stream shrinks, unless less than three fifths of the SMs are in use and
    // the slices are long (4 / more: 2048 x 2048 3.9 / 4.5, 3000 x 8000 8.0 / 8.4, but 2048 x 8192 6.7 / 5.9)
    int split = tiles <= fit.one[1] ? 1 : 0;
    for (int s = 2; s <= MAX_SPLIT; s++)
        if (split > 0 && tiles <= fit.one[s] && (s <= 4 ? k_blocks >= 2 * s : k_blocks >= 10 * s && 20 * tiles < 3 * num_sms)) split = s;
    if (split > 0 && 4 * tiles * split >= 3 * num_sms) { r.split = split; return r; }
    // Too few CTAs that way (or more tiles than SMs): two to an SM.  Four stages and the partial sums have to fit in half of
    // its shared memory (80 tokens), and with fewer than one and a half CTAs per SM the imbalance costs what the spread
    // gains (16 tokens: 11008 x 4096 3 slices 10.3 us / 1 slice 12.2, 12288 x 4096 2 slices 12.1 / 12.4).
    const bool half_fits = 4 * (W_BYTES + tn * BK) <= smem_of(2) - TAIL_BYTES && tn * W_ROWS * 4 <= smem_of(2) - TAIL_BYTES;
    if (half_fits && split > 0 && k_blocks >= 24)
        for (int s = 4; s > split; s--)
            if (tiles <= 2 * fit.one[s] && 2 * tiles * s >= 3 * num_sms) { r.split = s; r.per_sm = 2; return r; }
    // Three to an SM, with four stages each (three past 16 tokens): 12288 x 4096 in 4 slices 11.1 us / 1 slice 12.4 at 16 tokens,
    // 12.3 / 12.9 at 48.
    if (M <= 48 && split > 0 && k_blocks >= 24 && tiles <= 3 * fit.one[4] && 2 * tiles >= num_sms) { r.split = 4; r.per_sm = 3; return r; }
    // With more tiles than SMs the same in two slices, instead of two whole tiles on a few SMs and one on the others, or of the
    // square kernel's short second wave (16 tokens: 22016 x 4096 19.0 us / 20.8 / 21.9, 26880 x 4096 20.4 / 21.7 / 23.1).  Past 16
    // tokens it stays ahead up to a quarter more tiles than SMs (24000 x 4096, 32 tokens 21.4 / 21.2), and with only an eighth
    // more up to 32 tokens (20000 x 4096, 48 tokens 20.0 / - / 19.7).
    if (M <= 48 && split == 0 && k_blocks >= 16 && tiles <= 3 * fit.one[2] && (M <= 16 || 4 * tiles <= 5 * num_sms) &&
        (M <= 32 || 8 * tiles >= 9 * num_sms)) {
        r.split = 2;
        r.per_sm = 3;
        return r;
    }
    if (split > 0) {
        // a third of the SMs idle: still ahead of the square kernel up to 48 tokens (12288 x 4096, 40 / 64 / 96 tokens: 12.8 / 13.4 /
        // 13.8 us against 13.2 / 13.2 / 13.4), or where that one reads the weight twice
        if (M <= 48 || M > 128 || 4 * tiles < num_sms) r.split = split;
        return r;
    }
    // Up to twice as many tiles as SMs otherwise: one wave of two to an SM (16 tokens of K = 4096: 256 tiles 22.9 us against 25.2
    // for the square kernel, 512 tiles 44.9 against 45.7), with a long K up to 48 tokens (21376 x 8192, 64 tokens 37.4 / 36.5)
    if (half_fits && M <= (k_blocks > 32 ? 48 : 64) && tiles <= 2 * fit.one[1] && 8 * tiles >= 9 * num_sms) { r.split = 1; r.per_sm = 2; }
    return r;
}

// A: tokens [M, K] (their codes; rows = nullptr) or nothing, B: weights [N, K]; g is complete but for k_blocks
inline int launch(GemmParams g, const Plan& plan, const void* A, const void* B, cudaStream_t stream, const Rows* rows = nullptr) {
    Params p;
    p.r = rows ? *rows : Rows{};
    g.k_blocks = (g.K + BK - 1) / BK;
    p.tn = (g.M + 15) / 16 * 16;
    p.tmem_cols = 32;
    while (p.tmem_cols < p.tn) p.tmem_cols *= 2;
    p.idesc = make_idesc_e4m3_f32(W_ROWS, p.tn, 0, 0);
    const int tiles = (g.N + W_ROWS - 1) / W_ROWS;
    const int slice = (g.k_blocks + plan.split - 1) / plan.split;
    const int stage_bytes = rows ? W_BYTES : W_BYTES + p.tn * BK;
    const int tok_bytes = rows ? slice * TOKEN_BYTES : 0;
    p.slice = slice;
    // A long stream of up to 32 tokens with an SM to itself has 160 KB in flight and not all 227: what is asked for beyond some 20 MB only waits in front
    // of memory.  Us, 227 KB / 160 (112 KB: a fifth slower): 16 tokens, 8192 x 8192 14.25 / 14.1, 16384 x 16384 45.2 / 44.7, 5000 x 8000 10.6 / 10.4, 4 tokens,
    // 7000 x 7008 12.8 / 12.4, 1 token 8192 x 8192 13.8 / 13.6; level or slower from 40 on, and where a CTA's 16 blocks nearly fit 9.03 / 9.17.
    const int smem = plan.per_sm == 1 && !rows && g.M <= 32 && slice > 16 ? SMEM_LONG : smem_of(plan.per_sm);
    const int room = smem - TAIL_BYTES - tok_bytes;
    auto stages_in = [&](int bytes) {
        int n = bytes / stage_bytes;
        if (rows && plan.per_sm == 3 && n > 3) n = 3;   // the rows' values wait behind what the rings have asked for: a step of one sequence of a 4096 wide block 64.6 us, with four 65.7;
                                                        // two sequences, and blocks 1024 to 6144 wide, level
        return n > slice ? slice : n > MAX_STAGES ? MAX_STAGES : n;
    };
    // Partial sums of up to 16 tokens have memory of their own where that costs no stage; a row as values has 512 to 672 bytes, by the cut, and they begin in the block
    // behind the codes, so that as long a K finds room for two stages as without them (two rows: 192, 77 and 39 k-blocks to one of one, two and three CTAs of an SM)
    const int own_bytes = part_room(plan.split, g.M, rows != nullptr);
    const bool apart = rows || (g.M <= APART_TOKENS && stages_in(room - own_bytes) == stages_in(room));
    p.stages = stages_in(apart ? room - own_bytes : room);
    if (rows && (room - own_bytes < 2 * stage_bytes || (plan.per_sm == 3 && slice > 39))) return (int)cudaErrorNotSupported;
    int ring_bytes = p.stages * stage_bytes;
    const int part_bytes = apart ? own_bytes : 0;
    while (!apart && ring_bytes < p.tn * W_ROWS * 4) { p.stages++; ring_bytes += stage_bytes; }   // the partial sums take the ring's place
    // How much of the weight is asked for ahead of the wait.  It helps as far as memory is idle until then; past that a CTA's first
    // loads stand behind hints for its last ones.  Half of a CTA's blocks up to 16 (all of up to 8), with several CTAs to an SM no more than 20 MB in
    // all, and four blocks past 80 tokens, whose first loads bring as much again in tokens, which no hint has fetched.  All / as
    // here, us: 22016 x 4096 with SwiGLU, 1 token 19.4 / 18.0, 40 tokens 21.4 / 19.3; 12288 x 4096 10.8 / 10.4; 4096 x 11008
    // 11.2 / 10.8, 173 tokens 16.7 / 16.1; a block over 40 tokens 83.2 / 80.2, a step of one sequence 79.9 / 78.3.
    p.prefetch = slice <= 8 ? slice : (slice + 1) / 2;
    if (plan.per_sm > 1 && p.prefetch > (20 << 20) / (W_BYTES * tiles * plan.split)) p.prefetch = (20 << 20) / (W_BYTES * tiles * plan.split);
    if (p.prefetch > 16) p.prefetch = 16;
    if (g.M > 80) p.prefetch = 4;
    if (p.r.early) p.prefetch = 0;
    p.vec = g.H ? (g.F % 4 == 0 && (reinterpret_cast<uintptr_t>(g.H) & 7) == 0)
          : g.X ? (g.N % 4 == 0 && ((reinterpret_cast<uintptr_t>(g.X) | (rows ? reinterpret_cast<uintptr_t>(rows->x_in) : 0)) & 15) == 0)   // both are read or written whole
          : g.D8 ? (g.N % 4 == 0 && (reinterpret_cast<uintptr_t>(g.D8) & 3) == 0)
                 : (g.N % 4 == 0 && (reinterpret_cast<uintptr_t>(g.C) & 7) == 0);
    p.g = g;
    CUtensorMap tw, tt;
    if (!make_tmap_u8_2d(&tw, B, (uint64_t)g.N, (uint64_t)g.K, W_ROWS, BK, CU_TENSOR_MAP_SWIZZLE_128B) ||
        (!rows && !make_tmap_u8_2d(&tt, A, (uint64_t)g.M, (uint64_t)g.K, (uint32_t)p.tn, BK, CU_TENSOR_MAP_SWIZZLE_128B)))
        return (int)cudaErrorInvalidValue;
    if (rows) tt = tw;   // not looked at
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure(cfg, attr, tiles, plan.split, (size_t)ring_bytes + tok_bytes + part_bytes + TAIL_BYTES, stream);
    return (int)cudaLaunchKernelEx(&cfg, kernel_for(plan.split, rows ? 2 : apart), tw, tt, p);
}

}  // namespace skinny
