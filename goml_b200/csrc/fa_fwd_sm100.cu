// fa_fwd_sm100.cu — FP8 (e4m3) FlashAttention forward for NVIDIA B200 (sm_100a).
//
// Same function as goml's libs/fa_sm120/src/_v121r_train_kernel.cu:208-723 (hd128)
// and libs/flash_attention_v89_pinregs_fp8_forward.cu:201-211 (hd64): per (batch*head),
// O = softmax(scale * Q K^T + mask) V with an online (blockwise) softmax, fp16 output
// and optional natural-log LSE — rebuilt around the Blackwell data path:
//
//   V in fp16      : exact (every e4m3 value is an fp16 value).  Long sequences: a pre-pass makes an fp16 copy in a
//                    caller-provided workspace (HBM-bound, <2% of the time).  Short ones and narrow windows, where
//                    few query tiles share a key: the kernel converts each tile in shared memory (VRAW below)
//   TMA            : swizzled tiles, 3-D maps over [BH,S,D] so a tile never crosses a head
//   S = Q K^T      : tcgen05.mma kind::f8f6f4 on the e4m3 codes, 128x64 fp32
//                    accumulator in TMEM, double buffered so the next block's scores are
//                    ready before the softmax of the current one ends
//   softmax        : 4 warps, one query row per thread (tcgen05.ld 32x32b), fp32 running
//                    max/sum in the log2 domain, scale folded into one packed FFMA per two
//                    scores, lazy O rescale (only when the max grows by more than 2^TAU)
//   P              : kept in fp16 (11-bit significand) and written back to TENSOR MEMORY
//                    over the first half of its S buffer.  The reference rounds P to e4m3 (3-bit
//                    mantissa); for zero-mean V that rounding alone costs ~2.5e-2 mean
//                    relative error, above the 1e-2 bar, so P V runs as an fp16 MMA
//   O += P V       : tcgen05.mma kind::f16, A = P read from TMEM, B = V consumed MN-major
//                    straight from the TMA tile (no shared-memory transpose), fp32
//                    accumulator in TMEM
//   epilogue       : O * (v_descale / l) -> fp16, staged per warp, 128-bit stores; LSE.
//
// The tensor core reads shared-memory operands at 128 B/clk/SM, which is what bounds both
// MMAs here; keeping P out of shared memory keeps that traffic near the exponential-unit
// time, which is the next bound (16 ex2 per clock per SM).  A CTA works on one 128-row query tile of one head at a time; 6 warps
// (4 softmax, 1 MMA issuer, 1 TMA producer), or 7 where one converts V; two CTAs share an SM so one CTA's softmax overlaps the
// other's MMAs.  With more tiles than CTAs fit, a CTA that is about to finish takes over the tile of one that has not been
// launched yet (cluster launch control), so the order and the balance are the hardware's.  Every mbarrier wait is bounded.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <stdio.h>

#include <mutex>
#include <type_traits>

#include "../../include/fa_sm120.h"
#include "fa_fwd_sm100.h"
#include "pdl.cuh"
#include "sm100_ptx.cuh"
#include "tmap.cuh"

namespace fa_sm100 {

using namespace sm100;

namespace {

constexpr int BM = 128;  // query rows per CTA (= TMEM lanes)
constexpr int BN = 64;   // keys per block
constexpr int STAGES = 3; // K / V shared-memory ring depth
constexpr int NUM_SOFTMAX_WARPS = 4;   // one thread per query row
constexpr int SMEM_ONE = 120 * 1024;   // dynamic shared memory of a CTA that is to have an SM to itself
constexpr int HEAD_GROUP = 16;         // heads whose tiles are interleaved when tiles differ in length (48 MB of K/V at S = 8192, D = 128)
constexpr long long GROUP_ELEMS = 1ll << 24;   // S * D of a larger group: as much K/V
constexpr int MMA_WARP = NUM_SOFTMAX_WARPS;
constexpr int TMA_WARP = NUM_SOFTMAX_WARPS + 1;
constexpr int CONVERT_WARP = NUM_SOFTMAX_WARPS + 2;   // where V has a warp of its own (Cfg::CONVERTER)
constexpr uint32_t IDESC_NEGATE_A = 1u << 13;   // of the instruction descriptor
constexpr float TAU = 6.0f;   // lazy-rescale threshold (log2 units)
constexpr float POFF = 2.0f;  // P is carried as P * 2^POFF (max 2^(TAU+POFF) = 256, far inside fp16)

enum : uint32_t {
    ST_TIMEOUT_LOAD = 0x201,
    ST_TIMEOUT_MMA = 0x202,
    ST_TIMEOUT_SOFTMAX = 0x203,
    ST_BAD_SMEM_ALIGN = 0x204,
    ST_TIMEOUT_SELFTEST = 0x2F0,   // fa_selftest_wait_expiry
};

__device__ uint32_t g_fa_status = 0;

// Shared memory holds the operand tiles: Q, K and the fp16 V, or (VRAW) the codes of V beside the fp16 tiles that a warp
// makes of them; two CTAs an SM either way.  Both MMAs are limited by how fast the
// tensor core can read its shared-memory operands (128 B/clk/SM), so P never goes through
// shared memory: it is written to tensor memory and read from there as the A operand.
template <int HD, bool VRAW>
struct Cfg {
    static constexpr int Q_BYTES = BM * HD;
    static constexpr int K_BYTES = BN * HD;
    static constexpr int V_BYTES = BN * HD * 2;       // fp16
    static constexpr int V_HALF_BYTES = BN * 128;     // one 64-wide (128-byte) slab of d
    // A warp of its own converts V, else the producer does.  For D = 128 a block costs a warp 900 of the 1500 clk it may take, and a
    // producer that also loads and walks falls behind at every tile's start (256 heads of 2048, causal: 291 us, with the warp 264); for
    // D = 64 it costs 500, and the warp more than it brings (64 of 3000, window 512: 57 us, with the warp 60).
    static constexpr bool CONVERTER = VRAW && HD == 128;
    static constexpr int RAW_STAGES = !VRAW ? 0 : HD == 128 ? 2 : 3;
    static constexpr int STAGE_BYTES = 2048;          // of a softmax warp, for its rows on their way out
    static constexpr int NUM_THREADS = (NUM_SOFTMAX_WARPS + 2 + CONVERTER) * 32;
    // Registers are those of eight warps, two CTAs to an SM: of fourteen warps one of its four schedulers has four, which leaves a thread
    // 128.  Of the masked forms 72 to 80 bytes spill.  With 32 registers of every other thread moved to the softmax threads (setmaxnreg) none
    // did, and 256 heads of 2048, causal, took 247 us (now 264), 1024 of 512 104 (119), 64 of 8192, window 1024, 262 (281), 256 of 1000, not
    // causal, 119 (131), 40 of 2048 45.4 (46.7), 900 of 128, causal, 16.6 (21.4).  But beside that split a small change of code, the rescale of O as a loop, raised
    // illegal accesses whose cause was not found, so registers stay where a launch puts them.
    static constexpr int BOUND_THREADS = CONVERTER ? 256 : NUM_THREADS;
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_K = OFF_Q + Q_BYTES;
    static constexpr int OFF_V = OFF_K + STAGES * K_BYTES;
    static constexpr int OFF_VRAW = OFF_V + STAGES * V_BYTES;   // codes of V, where the kernel converts them itself (D = 128: two stages, all that fits)
    static constexpr int OFF_STAGE = OFF_VRAW + RAW_STAGES * K_BYTES;
    static constexpr int OFF_BAR = OFF_STAGE + NUM_SOFTMAX_WARPS * STAGE_BYTES;
    // Behind a pre-pass a CTA asks for half of an SM's 228 KB (1 KB of which the system takes per CTA): while any CTA of the pre-pass
    // is left on an SM, no second one fits there, so that the tiles in front, a causal launch's longest, spread over all
    // SMs first.  With two to an SM from the start (88 KB, and registers for both beside a CTA of the pre-pass) one call behind
    // another took, D = 128, causal, 4 heads of 4700 65.3 us, 6 of 4790 66.1, 10 of 4608 62.0, now 52.4, 56.9, 58.1.
    static constexpr int SMEM_BYTES = VRAW ? OFF_BAR + 256 : 113 * 1024;
    static_assert(OFF_BAR + 256 <= SMEM_BYTES, "everything fits");
    // TMEM: S[0], S[1] (64 fp32 columns each; P of the same block, 32 columns of packed fp16
    //       pairs, overwrites the first half of its S buffer)   O at [128, 128 + HD)
    static constexpr int TMEM_COLS = 256;
    static constexpr int O_COL = 128;
};

struct Params {
    int bh, sl, n_qtiles;
    int causal, window;
    float scale_log2;  // scale * log2(e)
    float v_descale;
    const float* sq;   // optional device scalars (quantiser outputs)
    const float* sk;
    const float* sv;
    __half* o;
    float* lse;
    float* o_amax;             // see LaunchArgs
    const uint32_t* v_flags;
    uint32_t v_epoch;
    int v_chunks;              // chunks per head
    int group;                 // heads whose tiles are interleaved
    int few;                   // the launch leaves SMs free, and O's quantiser is not what follows: the next kernel may come at once
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Packed fp32 pairs (Blackwell fma.rn.f32x2 / add.f32x2): one issue slot for two results.
__device__ __forceinline__ void ffma2(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0, float c1) {
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void fadd2(float& d0, float& d1, float a0, float a1) {
    asm("{\n\t.reg .b64 ra, rd;\n\t"
        "mov.b64 rd, {%0, %1};\n\tmov.b64 ra, {%2, %3};\n\t"
        "add.f32x2 rd, rd, ra;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "+f"(d0), "+f"(d1)
        : "f"(a0), "f"(a1));
}
// Two products by one factor, each rounded as alone.  PACKED for D = 64 only: half the instructions of the rows out and of a rescaled O, us, 64
// heads of 3000, window 512, 52.9 / 52.0, 128 of 2048, causal, 106.4 / 105.1; for D = 128, where the compiler arranges the loops around them
// differently, 256 of 2048, causal, 273 / 277.
template <bool PACKED>
__device__ __forceinline__ void scale2(uint32_t a0, uint32_t a1, float f, float& d0, float& d1) {
    if (PACKED)
        asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
            "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\t"
            "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
            : "=f"(d0), "=f"(d1) : "r"(a0), "r"(a1), "f"(f));
    else
        d0 = __uint_as_float(a0) * f, d1 = __uint_as_float(a1) * f;
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__global__ void __launch_bounds__(32) fa_wait_expiry_selftest_kernel() {
    wait_expiry_selftest_body(&g_fa_status, ST_TIMEOUT_SELFTEST);
}

// V (e4m3) -> fp16, exact.  One CTA step = one chunk of V_CHUNK keys of one head, taken in the order the attention tiles
// ask for them; a finished chunk is published by its flag, so the attention kernel (launched behind this one without
// waiting for it) starts on the first heads while later ones are still being converted.  HBM-bound (3 bytes moved per
// element).
constexpr int V_CHUNK = 128;
constexpr int V_THREADS = 128;
constexpr int V_CTAS_PER_SM = 10;   // with 2 the first attention tiles wait for it (S = 2048 causal: 366 us a call), 4 344, 6 340, 10 337
__device__ __forceinline__ void e4m3x16_to_f16(const uint4 c, uint4& lo, uint4& hi) {
    const uint32_t w[4] = {c.x, c.y, c.z, c.w};
    uint32_t h[8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        asm("{\n\t.reg .b16 l, u;\n\tmov.b32 {l, u}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, l;\n\tcvt.rn.f16x2.e4m3x2 %1, u;\n\t}" : "=r"(h[2 * k]), "=r"(h[2 * k + 1]) : "r"(w[k]));
    }
    lo = make_uint4(h[0], h[1], h[2], h[3]);
    hi = make_uint4(h[4], h[5], h[6], h[7]);
}
template <int HD>
__global__ void __launch_bounds__(V_THREADS, 12) v_to_f16_kernel(const uint4* in, uint4* out, int chunks,
                                                                int chunks_per_head, int sl, uint32_t* flags, uint32_t epoch) {
    pdl_wait();      // V may come from the kernel ahead, and the attention of an earlier call may still read `out`
    pdl_trigger();   // after the wait: the attention kernel reads Q and K without waiting for this kernel
    constexpr int PER_KEY = HD / 16;                             // 16-byte pieces per key
    constexpr int STEPS = V_CHUNK * PER_KEY / V_THREADS;         // pieces per thread and chunk: 8 (D = 128) or 4
    constexpr int BATCH = 4;                                     // loads in flight per thread
    for (int c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int head = c / chunks_per_head, k0 = (c - head * chunks_per_head) * V_CHUNK;
        const int pieces = min(V_CHUNK, sl - k0) * PER_KEY;
        const size_t base = ((size_t)head * sl + k0) * PER_KEY;
#pragma unroll 1
        for (int i0 = 0; i0 < STEPS; i0 += BATCH) {
            uint4 v[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int at = (i0 + i) * V_THREADS + threadIdx.x;
                if (at < pieces) v[i] = ld128(in + base + at);
            }
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int at = (i0 + i) * V_THREADS + threadIdx.x;
                uint4 lo, hi;
                e4m3x16_to_f16(v[i], lo, hi);
                if (at < pieces) {
                    out[2 * (base + at)] = lo;
                    out[2 * (base + at) + 1] = hi;
                }
            }
        }
        if (flags) {
            // the readers copy with TMA (async proxy): order these stores into that proxy before the flag is released
            asm volatile("fence.proxy.async.global;" ::: "memory");
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flags + c), "r"(epoch) : "memory");
            }
        }
    }
}

// Producer-side view of the pre-pass: how many leading chunks of this head (from chunk `c` on) are known to be ready.
// The whole warp asks for 32 flags at a time, so a head of up to 4096 keys costs one load when it is complete.
// Bounded like every wait of this file.
__device__ __forceinline__ bool wait_v_chunk(const uint32_t* head_flags, int chunks_per_head, uint32_t epoch, int c, int& ready,
                                             volatile uint32_t* abort_flag) {
    if (c < ready) return true;
    const int lane = threadIdx.x & 31;
    uint64_t t0 = 0;
    for (uint32_t polls = 1;; polls++) {
        uint32_t f = epoch;
        if (c + lane < chunks_per_head)
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(head_flags + c + lane) : "memory");
        const uint32_t missing = __ballot_sync(0xffffffffu, f != epoch);
        const int n = missing ? __ffs(missing) - 1 : 32;
        if (n > 0) {
            ready = c + n;
            // the lane that issues the copy need not be the one that acquired the chunk's flag, and a vote orders no memory
            __syncwarp();
            asm volatile("fence.proxy.async.global;" ::: "memory");
            return true;
        }
        if ((polls & 255u) == 0) {
            uint32_t stop = *abort_flag;
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > SM100_WAIT_BUDGET_NS) {
                if (lane == 0) atomicCAS((uint32_t*)abort_flag, 0u, (uint32_t)ST_TIMEOUT_LOAD);
                stop = 1;
            }
            if (__any_sync(0xffffffffu, stop != 0)) return false;
        }
    }
}

// One 64-key tile of V in shared memory: codes -> fp16 in the order of a TMA load with 128-byte swizzle, one 64-column slab of
// d after the other.  By one warp, which takes 16 codes of a lane at a time; eight neighbouring lanes, whose 16-byte accesses
// share a wavefront, meet eight different bank groups on both sides.
//  D = 128 (codes swizzled too): they take four neighbouring pieces of one slab of two keys k and k ^ 5 — bit 2 of the key puts the
//   loads in different halves of the 128 bytes, bit 0 the stores on chunks of different parity;
//  D = 64 (codes as they lie in global memory): the four pieces of two neighbouring keys, 128 bytes in a row.
// In rounds of eight steps: code that is not there is not fetched (see the loops of the softmax warps).
template <int HD>
__device__ __forceinline__ void convert_v(uint32_t raw, uint32_t dst) {
    constexpr int STEPS = BN * HD / 512, BATCH = 8;   // steps of the warp, loads in flight
    const int lane = threadIdx.x & 31;
    const int slab = HD == 128 ? (lane >> 3) & 1 : 0;
    const int key = HD == 128 ? (lane >> 4) ^ ((lane & 4) ? 5 : 0) : lane >> 2;   // of step 0, below 8
    const int chunk = ((lane & 3) * 2) ^ key;
    // D = 128: a step takes four keys, {0, 5, 1, 4} and then {2, 7, 3, 6} of eight: key + 2 is key ^ 2.  D = 64: eight
    constexpr int TURN = HD == 128 ? 2 : 1;           // steps per eight keys
    uint32_t src[TURN], lo_at[TURN], hi_at[TURN];
#pragma unroll
    for (int t = 0; t < TURN; t++) {
        const int row = (key ^ (2 * t)) * 128;
        src[t] = raw + (HD == 128 ? row + (((slab * 4 + (lane & 3)) ^ key ^ (2 * t)) << 4) : lane * 16);
        lo_at[t] = dst + slab * (BN * 128) + row + ((chunk ^ (2 * t)) << 4);
        hi_at[t] = dst + slab * (BN * 128) + row + ((chunk ^ (2 * t) ^ 1) << 4);
    }
#pragma unroll 1
    for (int i0 = 0; i0 < STEPS; i0 += BATCH) {
        uint4 v[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; i++)
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w)
                         : "r"(src[i % TURN] + (i0 + i) / TURN * (8 * HD)) : "memory");
#pragma unroll
        for (int i = 0; i < BATCH; i++) {
            uint4 lo, hi;
            e4m3x16_to_f16(v[i], lo, hi);
            const int at = (i0 + i) / TURN * 1024;
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(lo_at[i % TURN] + at), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w) : "memory");
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(hi_at[i % TURN] + at), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w) : "memory");
        }
    }
}

// tile -> (head, query tile).  Tiles of equal cost go head by head, so that the CTAs in
// flight share a few heads' K/V in L2.  When the key range depends on the query tile
// (causal, window) the heads are taken in groups (heads_together), and inside a group the
// tiles with the most keys come first across all its heads: the last CTAs of the launch
// are then the short tiles of a whole group, not the long tiles of the last head.
struct Tile {
    int head, q0;
    int blk0, nblk;   // key blocks this tile can see: nblk >= 1, or 0 for no tile
    __device__ __forceinline__ Tile(int4 r) : head(r.x), q0(r.y), blk0(r.z), nblk(r.w) {}
    __device__ __forceinline__ Tile(const Params& p, int index) {
        int qt;
        if (p.causal || p.window > 0) {
            const int per_group = p.group * p.n_qtiles;
            const int g = index / per_group;
            const int r = index - g * per_group;
            const int heads_here = min(p.group, p.bh - g * p.group);
            head = g * p.group + r % heads_here;
            qt = p.n_qtiles - 1 - r / heads_here;
        } else {
            head = index / p.n_qtiles;
            qt = p.n_qtiles - 1 - (index % p.n_qtiles);
        }
        q0 = qt * BM;
        const int kv_hi = p.causal ? min(p.sl, q0 + BM) : p.sl;
        const int kv_lo = (p.window > 0) ? max(0, q0 - p.window + 1) : 0;
        blk0 = kv_lo / BN;
        nblk = (kv_hi + BN - 1) / BN - blk0;
    }
};

// The index of the tile that a request of this CTA has taken over from a CTA that had not been launched yet (its blockIdx.x), or
// -1 where none was left.  By a whole warp, once per request.
__device__ __forceinline__ int taken_tile(uint32_t response) {
    int canceled, index;
    asm volatile("{\n\t.reg .b64 lo, hi;\n\t.reg .b128 r;\n\t.reg .pred p;\n\t"
                 "ld.shared.v2.b64 {lo, hi}, [%2];\n\tmov.b128 r, {lo, hi};\n\t"
                 "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\tselp.s32 %0, 1, 0, p;\n\tmov.s32 %1, -1;\n\t"
                 "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
                 : "=r"(canceled), "=r"(index) : "r"(response) : "memory");
    fence_proxy_async_smem();   // the next response overwrites this one
    __syncwarp();
    return canceled ? index : -1;
}
__device__ __forceinline__ Tile tile_record(uint32_t at) {
    int4 r;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(at) : "memory");
    return Tile(r);
}

// VRAW = true: V arrives as codes, and a warp converts each tile in shared memory (for D = 64 the producer, while it waits for the ring).
// It shares its scheduler with one softmax warp of the CTA, and shared memory carries 24 KB more per block of D = 128; that saves the
// pre-pass: 3 bytes per element of traffic, a launch, the scratch, and the CTAs of the pre-pass, which the attention's first CTAs wait
// for.  Bit for bit the same results.
//
// MASKED = false: no key of the launch is masked (non-causal, no window, S a multiple of the block) and the host-side scale
// is positive: the masking code is not compiled into the softmax loop, and Q K^T is not asked for with a sign.  (The
// device-side scale factors are quantiser outputs, amax / 448: never negative.)
//
// AMAX = true: the largest |O| also goes to p.o_amax, for the quantiser behind (a variant of its own: the others keep their code).
// WALK = true: the CTA goes on to further tiles (walks() has the line).  The roles run through one sequence of blocks across them: the
// producer asks for a tile with the last block of the one before on its way, loads Q once the last Q K^T has read the old one, and the rings
// and the two S buffers just go on.
template <int HD, bool MASKED, bool VRAW, bool AMAX, bool WALK>
__global__ void __launch_bounds__(Cfg<HD, VRAW>::BOUND_THREADS, 2)
fa_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
              const __grid_constant__ CUtensorMap tmap_v, const Params p) {
    using C = Cfg<HD, VRAW>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bars = sbase + C::OFF_BAR;
    // Completion barriers are indexed by ring stage (block j -> j % STAGES) and double as the
    // "stage free" signals of the K and V rings: one tcgen05.commit per MMA batch instead of two.
    const uint32_t bar_q = bars;
    const uint32_t bar_kfull = bars + 8;                  // [STAGES] K tile landed
    const uint32_t bar_vfull = bar_kfull + 8 * STAGES;    // [STAGES] V tile landed
    const uint32_t bar_sfull = bar_vfull + 8 * STAGES;    // [STAGES] S = Q K^T of that block complete (K stage reusable)
    const uint32_t bar_pvdone = bar_sfull + 8 * STAGES;   // [STAGES] O += P V of that block complete (V stage reusable)
    const uint32_t bar_pfull = bars + 112;                // [2] softmax wrote P into S[b] (and rescaled O if needed); 16-byte aligned
    const uint32_t bar_vraw = bar_pfull + 16;             // [RAW_STAGES] codes of a V tile landed
    const uint32_t bar_vfree = bar_vraw + 8 * STAGES;     // [RAW_STAGES] ... and are converted
    const uint32_t bar_answer = bar_vfree + 8 * STAGES;   // the answer to a request for another tile is there
    const uint32_t bar_next = bar_answer + 8;             // the producer has written that tile's record
    const uint32_t bar_seen = bar_next + 8;               // the other warps have read it
    const uint32_t response = bars + 208, record = bars + 224;   // 16 bytes each
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + 240);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = threadIdx.x >> 5;

    if (threadIdx.x == 0) {
        mbar_init(bar_q, 1);
        for (int s = 0; s < STAGES; s++) {
            mbar_init(bar_kfull + 8 * s, 1);
            mbar_init(bar_vfull + 8 * s, 1);
            mbar_init(bar_sfull + 8 * s, 1);
            mbar_init(bar_pvdone + 8 * s, 1);
            mbar_init(bar_vraw + 8 * s, 1);
            mbar_init(bar_vfree + 8 * s, 1);
        }
        mbar_init(bar_answer, 1);
        mbar_init(bar_next, 1);
        mbar_init(bar_seen, NUM_SOFTMAX_WARPS + 1 + C::CONVERTER);
        for (int b = 0; b < 2; b++) mbar_init(bar_pfull + 8 * b, NUM_SOFTMAX_WARPS * 32);
        *abort_flag = (sbase & 1023u) ? ST_BAD_SMEM_ALIGN : 0u;
        fence_mbar_init();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_s = tmem_base;
    const uint32_t tmem_o = tmem_base + C::O_COL;
    const bool bad_start = (*abort_flag != 0);
    if (VRAW) {
        pdl_wait();   // no pre-pass has waited for what is ahead
        // The next kernel's start (its launch, barriers, tensor memory, hints) beside this one, where a launch leaves SMs free: calls behind one another, 4 heads of 256
        // keys, not causal, 5.43 / 5.05 us each, 28 of 125, causal, 5.24 / 4.91, 13 of 1251 15.2 / 15.0 (a call with nothing behind it takes what it took), in front of a GEMM of 16 x
        // 4096 x 4096 11.6 / 10.8, 11.4 / 10.4 and 21.8 / 20.7 for both; with more CTAs than SMs 9.7 / 9.9.  D = 128 loses by it (4 of 256 5.8 / 6.1, 24 of 700 11.7 / 12.5), and with the
        // trigger ahead of the rows out (32 of 512 9.7 / 9.9).  A quantiser of O behind it has little to set up and then takes longer from the wait on (7.6 / 7.5, 8.4 / 8.7, 19.9 / 20.1), so a
        // call that leaves it the maximum keeps the trigger at the end: a block of 32 heads over 100 tokens 50.4 / 50.7, 256 62.3 / 62.7, 512 84.3 / 85.0.
        if (HD == 64 && !WALK && p.few) pdl_trigger();
    }
    if (bad_start) {
        // fall through to teardown
    } else if (warp >= NUM_SOFTMAX_WARPS) {
        if (warp == TMA_WARP) {
            // ------------------------------------------------------------- TMA producer
            // The whole warp runs the loop and one elected lane issues: addresses and coordinates stay warp-uniform.
            {
                const bool leader = elect_one();
                if (leader) {
                    prefetch_tmap(&tmap_q);
                    prefetch_tmap(&tmap_k);
                    prefetch_tmap(&tmap_v);
                }
                bool ok = true;
                int s = 0, raw = 0;            // ring stages of the next block, of K and V and of the codes of V
                uint32_t ph = 0, raw_ph = 0;   // their phases
                uint32_t tph = 0;              // phase of the tile
                Tile t(p, blockIdx.x);
                for (bool first = true;; first = false) {          // first tile of this CTA: the rings are empty
                    const int before = s == 0 ? STAGES - 1 : s - 1;
                    const uint32_t before_ph = s == 0 ? ph ^ 1 : ph;
                    auto load_q = [&]() {
                        mbar_arrive_expect_tx(bar_q, C::Q_BYTES);
                        tma_load_3d(sbase + C::OFF_Q, &tmap_q, bar_q, 0, t.q0, t.head);
                    };
                    if (first && leader) load_q();
                    if constexpr (VRAW && !C::CONVERTER) {
                        auto load_k = [&](int j, int at) {
                            mbar_arrive_expect_tx(bar_kfull + 8 * at, C::K_BYTES);
                            tma_load_3d(sbase + C::OFF_K + at * C::K_BYTES, &tmap_k, bar_kfull + 8 * at, 0, (t.blk0 + j) * BN, t.head);
                        };
                        auto load_v = [&](int j, int at) {
                            mbar_arrive_expect_tx(bar_vraw + 8 * at, C::K_BYTES);
                            tma_load_3d(sbase + C::OFF_VRAW + at * C::K_BYTES, &tmap_v, bar_vraw + 8 * at, 0, (t.blk0 + j) * BN, t.head);
                        };
                        const int s0 = s;
                        const uint32_t ph0 = ph;
                        if (!first) {
                            // with the last Q K^T of the tile before, Q and all stages of the K ring are free
                            ok = mbar_wait_warp(bar_sfull + 8 * before, before_ph, abort_flag, ST_TIMEOUT_LOAD);
                            if (!ok) break;
                            if (leader) load_q();
                        }
                        if (leader) {
                            for (int j = 0; j < STAGES && j < t.nblk; j++) {
                                const int at = s0 + j < STAGES ? s0 + j : s0 + j - STAGES;
                                load_k(j, at);
                                load_v(j, at);
                            }
                        }
                        __syncwarp();
                        for (int j = 0; j < t.nblk; j++) {
                            ok = mbar_wait_warp(bar_vraw + 8 * s, ph, abort_flag, ST_TIMEOUT_LOAD) &&
                                 mbar_wait_warp(bar_pvdone + 8 * s, ph ^ 1, abort_flag, ST_TIMEOUT_LOAD);   // P V three blocks back is done
                            if (!ok) break;
                            // and with it every MMA issued before it, Q K^T two blocks back among them: its K stage is free.  (In the third
                            // block of a tile only the tile before has been waited for: there the first Q K^T is.)
                            if (j + 1 >= STAGES && j + 1 < t.nblk) {
                                if (j + 1 == STAGES) ok = mbar_wait_warp(bar_sfull + 8 * s0, ph0, abort_flag, ST_TIMEOUT_LOAD);
                                if (!ok) break;
                                if (leader) load_k(j + 1, s + 1 < STAGES ? s + 1 : 0);
                            }
                            convert_v<HD>(sbase + C::OFF_VRAW + s * C::K_BYTES, sbase + C::OFF_V + s * C::V_BYTES);
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (leader) {
                                mbar_arrive(bar_vfull + 8 * s);
                                if (j + STAGES < t.nblk) load_v(j + STAGES, s);
                            }
                            __syncwarp();
                            if (++s == STAGES) { s = 0; ph ^= 1; }
                        }
                    } else {
                        // Q and K are complete when this kernel starts (a pre-pass triggers it after its own wait); the fp16 copy
                        // of V is waited for chunk by chunk, or as a whole when the launch has no flags
                        int v_ready = 0;
                        const uint32_t* head_flags = !VRAW && p.v_flags ? p.v_flags + (size_t)t.head * p.v_chunks : nullptr;
                        for (int j = 0; j < t.nblk; j++) {
                            const int key0 = (t.blk0 + j) * BN;
                            const bool fresh = first && j < STAGES;
                            ok = fresh || mbar_wait_warp(bar_sfull + 8 * s, ph ^ 1, abort_flag, ST_TIMEOUT_LOAD);   // Q K^T three blocks back is done
                            if (!ok) break;
                            if (leader) {
                                mbar_arrive_expect_tx(bar_kfull + 8 * s, C::K_BYTES);
                                tma_load_3d(sbase + C::OFF_K + s * C::K_BYTES, &tmap_k, bar_kfull + 8 * s, 0, key0, t.head);
                            }
                            if (VRAW) {
                                ok = (first && j < C::RAW_STAGES) || mbar_wait_warp(bar_vfree + 8 * raw, raw_ph ^ 1, abort_flag, ST_TIMEOUT_LOAD);
                                if (!ok) break;
                                if (leader) {
                                    mbar_arrive_expect_tx(bar_vraw + 8 * raw, C::K_BYTES);
                                    tma_load_3d(sbase + C::OFF_VRAW + raw * C::K_BYTES, &tmap_v, bar_vraw + 8 * raw, 0, key0, t.head);
                                }
                                if (++raw == C::RAW_STAGES) { raw = 0; raw_ph ^= 1; }
                            }
                            if (!first && j == 0) {
                                // with the last Q K^T of the tile before, Q is free
                                ok = mbar_wait_warp(bar_sfull + 8 * before, before_ph, abort_flag, ST_TIMEOUT_LOAD);
                                if (!ok) break;
                                if (leader) load_q();
                            }
                            if (!VRAW) {
                                ok = fresh || mbar_wait_warp(bar_pvdone + 8 * s, ph ^ 1, abort_flag, ST_TIMEOUT_LOAD);  // P V three blocks back is done
                                if (!ok) break;
                                if (!head_flags) {
                                    if (j == 0) pdl_wait();
                                } else {
                                    ok = wait_v_chunk(head_flags, p.v_chunks, p.v_epoch, key0 / V_CHUNK, v_ready, abort_flag);
                                    if (!ok) break;
                                }
                                if (leader) {
                                    mbar_arrive_expect_tx(bar_vfull + 8 * s, C::V_BYTES);
#pragma unroll
                                    for (int h = 0; h < HD / 64; h++)  // one 64-column (128-byte) slab of d per copy
                                        tma_load_3d(sbase + C::OFF_V + s * C::V_BYTES + h * C::V_HALF_BYTES, &tmap_v, bar_vfull + 8 * s,
                                                    h * 64, key0, t.head);
                                }
                            }
                            __syncwarp();
                            if (++s == STAGES) { s = 0; ph ^= 1; }
                        }
                    }
                    if (!ok || !WALK) break;
                    // Another tile is asked for with this one's last block on its way, some three before the softmax warps finish: earlier, the
                    // launch's last tiles would go to whoever asks and not to whoever is done first.
                    if (!first && !mbar_wait_warp(bar_seen, tph ^ 1, abort_flag, ST_TIMEOUT_LOAD)) break;
                    if (leader) {
                        mbar_arrive_expect_tx(bar_answer, 16);
                        asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                                     ::"r"(response), "r"(bar_answer) : "memory");
                    }
                    __syncwarp();
                    if (!mbar_wait_warp(bar_answer, tph, abort_flag, ST_TIMEOUT_LOAD)) break;
                    const int index = taken_tile(response);
                    if (index < 0) t.nblk = 0;
                    else t = Tile(p, index);
                    if (leader) {
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(record), "r"(t.head), "r"(t.q0), "r"(t.blk0), "r"(t.nblk) : "memory");
                        mbar_arrive(bar_next);
                    }
                    __syncwarp();
                    tph ^= 1;
                    if (t.nblk == 0) break;
                }
                if (!VRAW) pdl_wait();   // this kernel completes after the pre-pass
            }
        } else if (C::CONVERTER && warp == CONVERT_WARP) {
            // ------------------------------------------------------------- V: codes -> fp16
            if constexpr (C::CONVERTER) {
                const bool leader = elect_one();
                bool ok = true;
                int s = 0, raw = 0;
                uint32_t ph = 0, raw_ph = 0, tph = 0;
                for (int nblk = Tile(p, blockIdx.x).nblk;;) {
                    for (int j = 0; j < nblk; j++) {
                        ok = mbar_wait_warp(bar_vraw + 8 * raw, raw_ph, abort_flag, ST_TIMEOUT_LOAD) &&
                             mbar_wait_warp(bar_pvdone + 8 * s, ph ^ 1, abort_flag, ST_TIMEOUT_LOAD);   // P V three blocks back is done
                        if (!ok) break;
                        convert_v<HD>(sbase + C::OFF_VRAW + raw * C::K_BYTES, sbase + C::OFF_V + s * C::V_BYTES);
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (leader) {
                            mbar_arrive(bar_vfull + 8 * s);
                            mbar_arrive(bar_vfree + 8 * raw);
                        }
                        __syncwarp();
                        if (++s == STAGES) { s = 0; ph ^= 1; }
                        if (++raw == C::RAW_STAGES) { raw = 0; raw_ph ^= 1; }
                    }
                    if (!ok || !WALK || !mbar_wait_warp(bar_next, tph, abort_flag, ST_TIMEOUT_LOAD)) break;
                    nblk = tile_record(record).nblk;
                    __syncwarp();
                    if (leader) mbar_arrive(bar_seen);
                    tph ^= 1;
                    if (nblk == 0) break;
                }
            }
        } else if (warp == MMA_WARP) {
            // -------------------------------------------------------------- MMA issuer
            // Whole warp, one elected lane issues (descriptors stay in uniform registers).
            {
                const bool leader = elect_one();
                // a negative scale: the scores come out of the tensor core with the sign that their maximum is taken with
                float sign = p.scale_log2;
                if (MASKED && p.sq) sign *= ld_f32(p.sq);
                if (MASKED && p.sk) sign *= ld_f32(p.sk);
                const uint32_t idesc_qk = make_idesc_e4m3_f32(BM, BN, 0, 0) | (MASKED && sign < 0.f ? IDESC_NEGATE_A : 0u);
                constexpr uint32_t idesc_pv = make_idesc_f16_f32(BM, HD, 0, 1);  // A = P from TMEM, V is MN-major
                auto qk_desc = [&](uint32_t addr) { return HD == 128 ? kmajor_desc_sw128(addr) : kmajor_desc_sw64(addr); };
                // K ring position of the next Q K^T, V ring position of the next P V
                int ks = 0, vs = 0;
                uint32_t kph = 0, vph = 0;
                bool ok = true;
                uint32_t kb = 0, vb = 0;      // S buffers of the next Q K^T and of the next P V
                uint32_t pph = 0;             // bit b: phase of P in S[b]
                uint32_t tph = 0, qph = 0;    // phases of the next tile's record and of Q
                auto issue_qk = [&]() {       // S[kb] = Q K^T of the next block
                    ok = mbar_wait_warp(bar_kfull + 8 * ks, kph, abort_flag, ST_TIMEOUT_MMA);
                    if (!ok) return;
                    tc_fence_after();
                    const uint64_t qd = qk_desc(sbase + C::OFF_Q);
                    const uint64_t kd = qk_desc(sbase + C::OFF_K + ks * C::K_BYTES);
                    if (leader) {
#pragma unroll
                        for (int k = 0; k < HD / 32; k++)
                            mma_f8f6f4_ss(tmem_s + kb * BN, qd + 2 * k, kd + 2 * k, idesc_qk, k != 0);
                        mma_commit(bar_sfull + 8 * ks);
                    }
                    __syncwarp();
                    kb ^= 1;
                    if (++ks == STAGES) { ks = 0; kph ^= 1; }
                };
                // Two blocks' scores are ahead of the P V, across the end of a tile too: behind this tile's last but one P V follows the
                // next one's first Q K^T, so that the softmax warps have its scores to work on until the last P V is done.
                int nblk = Tile(p, blockIdx.x).nblk, next = -1;   // blocks of this tile and of the next (-1: not known yet, 0: none)
                int qk = 0;                                       // Q K^T issued of this tile or, once next >= 0, of the next
                ok = mbar_wait_warp(bar_q, 0, abort_flag, ST_TIMEOUT_MMA);
                for (; nblk > 0 && ok;) {
                    for (int j = 0; j < nblk && ok; j++) {
                        while (ok && (next < 0 ? qk : nblk + qk) < j + 2) {
                            if (next < 0 && qk == nblk) {
                                if (!WALK) { next = 0; break; }
                                ok = mbar_wait_warp(bar_next, tph, abort_flag, ST_TIMEOUT_MMA);
                                if (!ok) break;
                                next = tile_record(record).nblk;
                                __syncwarp();
                                if (leader) mbar_arrive(bar_seen);
                                tph ^= 1;
                                qk = 0;
                                if (next > 0) {
                                    qph ^= 1;
                                    ok = mbar_wait_warp(bar_q, qph, abort_flag, ST_TIMEOUT_MMA);
                                }
                            }
                            if (!ok || (next >= 0 && qk == next)) break;
                            issue_qk();
                            qk++;
                        }
                        if (!ok) break;
                        const uint32_t b = vb;
                        ok = mbar_wait_warp(bar_vfull + 8 * vs, vph, abort_flag, ST_TIMEOUT_MMA) &&
                             mbar_wait_warp(bar_pfull + 8 * b, (pph >> b) & 1, abort_flag, ST_TIMEOUT_MMA);
                        if (!ok) break;
                        pph ^= 1u << b;
                        vb ^= 1;
                        tc_fence_after();
                        const uint32_t vaddr = sbase + C::OFF_V + vs * C::V_BYTES;
                        if (leader) {
#pragma unroll
                            for (int k = 0; k < BN / 16; k++) {  // 16 keys per MMA: 8 TMEM columns of P, 16 rows of V
                                const uint64_t vd = mnmajor_desc_sw128(vaddr + k * 16 * 128, C::V_HALF_BYTES);
                                mma_f16_ts(tmem_o, tmem_s + b * BN + 8 * k, vd, idesc_pv, (j | k) != 0);
                            }
                            mma_commit(bar_pvdone + 8 * vs);
                        }
                        __syncwarp();
                        if (++vs == STAGES) { vs = 0; vph ^= 1; }
                        // S[b] is rewritten by the Q K^T two blocks ahead; it is issued behind this P V on the
                        // same in-order tensor pipe, so P(j) has been read before S(j+2) lands on it
                    }
                    nblk = next;   // its first P V, which overwrites O, waits for a P that is published after O has been read
                    next = -1;
                }
            }
        }
    } else {
        // ------------------------------------------- softmax / correction / epilogue
        const int r = threadIdx.x;               // row of the tile = TMEM lane (one thread per row)
        const uint32_t lane_off = uint32_t(warp * 32) << 16;
        float scale_log2 = p.scale_log2;
        if (p.sq) scale_log2 *= ld_f32(p.sq);
        if (p.sk) scale_log2 *= ld_f32(p.sk);
        const float vds = p.sv ? p.v_descale * ld_f32(p.sv) : p.v_descale;
        float ascale = fabsf(scale_log2);        // the scores have the scale's sign already
        if (ascale == 0.f) ascale = 1e-30f;      // keeps -inf * scale = -inf for masked keys
        int rs = 0;           // ring stage of the next block and its phase; those of the block before
        uint32_t rph = 0;
        int rs_prev = 0;
        uint32_t rph_prev = 0;
        uint32_t tph = 0;     // phase of the next tile's record
        uint32_t s_addr = tmem_s + lane_off, p_bar = bar_pfull;   // S buffer of the next block and the barrier of its P (^ BN, ^ 8: the other one)
        float m_ref, m_thr, nmsub, l0, l1, l2, l3;
        auto start_tile = [&]() {
            m_ref = -INFINITY;                   // reference max used in the exponent (log2 units)
            m_thr = -INFINITY;                   // m_ref + TAU
            nmsub = 0.f;                         // POFF - m_ref (0 while no finite score has been seen)
            l0 = l1 = l2 = l3 = 0.f;             // running sum of P * 2^POFF, in four partial sums
        };
        Tile t(p, blockIdx.x);

        // The scores of key block j of the tile, in the S buffer at sa, and what they do to the reference.  EDGE: the block may hold
        // masked keys.
        uint32_t sreg[BN];
        bool hidden[BN / 32];                    // no row of this warp sees these 32 keys: their P is zero
        auto scores = [&](const int j, const uint32_t sa, auto edge) -> bool {
            constexpr bool EDGE = decltype(edge)::value;
            if (!mbar_wait_warp(bar_sfull + 8 * rs, rph, abort_flag, ST_TIMEOUT_SOFTMAX)) return false;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < BN / 32; c++) tmem_ld_32x32b_x32(sa + c * 32, sreg + c * 32);
            tmem_ld_wait();

            hidden[0] = hidden[1] = false;
            if (EDGE) {
                // last and first visible key of this row, and the same of the first and the last row of its warp
                const int wq0 = t.q0 + warp * 32;
                const int hi_key = p.causal ? min(t.q0 + r, p.sl - 1) : p.sl - 1, lo_key = p.window > 0 ? t.q0 + r - p.window + 1 : 0;
                const int hi_key_first = p.causal ? min(wq0, p.sl - 1) : p.sl - 1, hi_key_last = p.causal ? min(wq0 + 31, p.sl - 1) : p.sl - 1;
                const int lo_key_first = p.window > 0 ? wq0 - p.window + 1 : 0, lo_key_last = p.window > 0 ? lo_key_first + 31 : 0;
                // What an edge leaves to do is decided per warp and 32 keys: most such chunks are visible to all rows of the
                // warp or to none, and only those cut by the edge are masked key by key.
#pragma unroll
                for (int g = 0; g < BN / 32; g++) {
                    const int k0 = (t.blk0 + j) * BN + g * 32;
                    hidden[g] = k0 > hi_key_last || k0 + 31 < lo_key_first;
                    if (hidden[g]) {
#pragma unroll
                        for (int c = 0; c < 32; c++) sreg[g * 32 + c] = 0xff800000u;  // -inf
                    } else if (k0 + 31 > hi_key_first || k0 < lo_key_last) {
                        // bit c: this row sees key k0 + c
                        const int hi = hi_key - k0, lo = lo_key - k0;
                        uint32_t seen = hi < 0 ? 0u : 0xffffffffu >> (31 - min(hi, 31));
                        seen = lo > 31 ? 0u : seen & (0xffffffffu << max(lo, 0));
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (!(seen & (1u << c))) sreg[g * 32 + c] = 0xff800000u;
                    }
                }
            }
            float mxa[8];  // eight short dependency chains
#pragma unroll
            for (int t = 0; t < 8; t++) mxa[t] = fmaxf(__uint_as_float(sreg[2 * t]), __uint_as_float(sreg[2 * t + 1]));
#pragma unroll
            for (int c = 16; c < BN; c += 16) {
#pragma unroll
                for (int t = 0; t < 8; t++)
                    mxa[t] = max3(mxa[t], __uint_as_float(sreg[c + 2 * t]), __uint_as_float(sreg[c + 2 * t + 1]));
            }
            const float mx = fmaxf(max3(max3(mxa[0], mxa[1], mxa[2]), max3(mxa[3], mxa[4], mxa[5]), mxa[6]), mxa[7]) * ascale;

            // The reference moves only when some row's maximum exceeds it by more than 2^TAU (always on the first finite
            // maximum: m_thr starts at -inf); everything that depends on it is state updated in this rare branch, so the
            // common path is one compare and one vote.
            if (__any_sync(0xffffffffu, mx > m_thr)) {
                const bool bump = mx > m_thr;
                const float m_new = bump ? mx : m_ref;
                if (j > 0) {
                    // O is final only once the previous P V has finished
                    if (!mbar_wait_warp(bar_pvdone + 8 * rs_prev, rph_prev, abort_flag, ST_TIMEOUT_SOFTMAX)) return false;
                    tc_fence_after();
                    const float f = bump ? ex2(m_ref - m_new) : 1.0f;  // m_ref = -inf -> 0
                    l0 *= f; l1 *= f; l2 *= f; l3 *= f;
#pragma unroll
                    for (int c = 0; c < HD / 16; c++) {
                        uint32_t o[16];
                        tmem_ld_32x32b_x16(tmem_o + lane_off + c * 16, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            float x0, x1;
                            scale2<HD == 64>(o[i], o[i + 1], f, x0, x1);
                            o[i] = __float_as_uint(x0);
                            o[i + 1] = __float_as_uint(x1);
                        }
                        tmem_st_32x32b_x16(tmem_o + lane_off + c * 16, o);
                    }
                }
                m_ref = m_new;
                m_thr = m_ref + TAU;
                nmsub = (m_ref == -INFINITY) ? 0.f : POFF - m_ref;
            }
            return true;
        };
        // P of 32 keys of the block: 16 words of packed fp16 pairs, and their part of the row sum
        auto exponentials = [&](const int g, uint32_t* w, auto edge) {
            if (decltype(edge)::value && hidden[g]) {
#pragma unroll
                for (int q = 0; q < 16; q++) w[q] = 0;
            } else {
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    float x0, x1;
                    ffma2(x0, x1, __uint_as_float(sreg[g * 32 + q * 2 + 0]), __uint_as_float(sreg[g * 32 + q * 2 + 1]),
                          ascale, ascale, nmsub, nmsub);
                    const float p0 = ex2(x0);
                    const float p1 = ex2(x1);
                    if (q & 1) fadd2(l2, l3, p0, p1); else fadd2(l0, l1, p0, p1);
                    w[q] = pack_half2(p0, p1);
                }
            }
        };
        auto publish = [&](const uint32_t pb) {   // P is in tensor memory
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(pb);
            rs_prev = rs;
            rph_prev = rph;
            if (++rs == STAGES) { rs = 0; rph ^= 1; }
        };
        auto block = [&](const int j, const uint32_t sa, const uint32_t pb, auto edge) -> bool {
            if (!scores(j, sa, edge)) return false;
#pragma unroll
            for (int g = 0; g < BN / 32; g++) {  // 32 keys -> 16 TMEM columns
                uint32_t w[16];
                exponentials(g, w, edge);
                tmem_st_32x32b_x16(sa + g * 16, w);  // P overwrites the first half of its S buffer
            }
            publish(pb);
            return true;
        };
        // Blocks [j, end) of one kind.  What these loops cost is also their code: four warps run through it in turn with the other roles', and
        // past the instruction cache it is fetched again and again.  With the clear loop unrolled by two, a sign flip of 64 instructions
        // in the edge loop and the conversion of V unrolled in full, us: 256 heads of 2048 of 128, causal, 298 (now 279), 64 of 8192, window
        // 1024, 327 (287), 64 of 3000 of 64, window 512, 57.1 (52.9), 256 of 1000 of 128, not causal, 139 (131).  One loop with the edge
        // as a test in it keeps more registers alive: 300, 305, 57.5, 143.  (All at the power cap, and those of 128 with registers moved
        // between the warps.)
        // A CTA with a tile of its own keeps the clear loop unrolled by two: its calls are few and long (1 head of 8192 of 128, causal, 92.8 / 85.7).
        auto edge_blocks = [&](int& j, const int end) -> bool {
#pragma unroll 1
            for (; j < end; j++) {
                if (!block(j, s_addr, p_bar, std::true_type())) return false;
                s_addr ^= BN;
                p_bar ^= 8;
            }
            return true;
        };
        auto clear_blocks = [&](int& j, const int end) -> bool {
            const int n = max(end - j, 0);
            constexpr int UNROLL = WALK ? 1 : 2;
#pragma unroll UNROLL
            for (int i = 0; i < n; i++) {
                if (!block(j + i, s_addr, p_bar, std::false_type())) return false;
                s_addr ^= BN;
                p_bar ^= 8;
            }
            j += n;
            return true;
        };

        // O / l (times the V dequantisation scale) -> fp16, and the LSE, of a tile whose last P V has this ring stage
        auto epilogue = [&](const int head, const int q0, const float l, const float m, const int stage_pv, const uint32_t phase_pv) -> bool {
            if (!mbar_wait_warp(bar_pvdone + 8 * stage_pv, phase_pv, abort_flag, ST_TIMEOUT_SOFTMAX)) return false;
            tc_fence_after();
            const int qi = q0 + r;
            const float inv = (l > 0.f) ? vds / l : 0.f;
            __half2 top = __float2half2_rn(0.f);
            // O leaves through shared memory: a thread owns one row, which written straight to global makes every store instruction of a
            // warp touch 32 lines.  32 columns at a time, each warp stages its 32 rows of 64 bytes — 16-byte
            // chunk c of row r at chunk c ^ (r / 2 % 4), so that both the row-wise writes and the read-back are free of bank conflicts —
            // and stores 8 rows an instruction.
            uint8_t* stage = smem + C::OFF_STAGE + warp * C::STAGE_BYTES;
            const int lane = threadIdx.x & 31;
            __half* obase = p.o + ((size_t)head * p.sl + q0 + warp * 32 + (lane >> 2)) * HD + (lane & 3) * 8;
            const int rows_left = p.sl - (q0 + warp * 32 + (lane >> 2));   // rows of this warp inside the sequence, from the lane's first on
#pragma unroll
            for (int c = 0; c < HD / 32; c++) {
                uint32_t o[32];
                tmem_ld_32x32b_x32(tmem_o + lane_off + c * 32, o);
                tmem_ld_wait();
                if (c > 0) __syncwarp();   // the columns before have been read back
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        float x0, x1;
                        scale2<HD == 64>(o[8 * v + 2 * i], o[8 * v + 2 * i + 1], inv, x0, x1);
                        w[i] = pack_half2(x0, x1);
                        if (AMAX) top = __hmax2(top, __habs2(*reinterpret_cast<const __half2*>(&w[i])));   // of the rounded values; NaN never wins
                    }
                    *reinterpret_cast<uint4*>(stage + lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int rr = i * 8 + (lane >> 2);
                    const uint4 w = *reinterpret_cast<const uint4*>(stage + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
                    if (i * 8 < rows_left) *reinterpret_cast<uint4*>(obase + (size_t)i * 8 * HD + c * 32) = w;
                }
            }
            if (WALK) __syncwarp();   // the next tile's rows are staged here too
            if (AMAX) {
                float top1 = qi < p.sl ? fmaxf(__low2float(top), __high2float(top)) : 0.f;
#pragma unroll
                for (int i = 16; i > 0; i >>= 1) top1 = fmaxf(top1, __shfl_xor_sync(0xffffffffu, top1, i));
                if (lane == 0) atomicMax(reinterpret_cast<unsigned int*>(p.o_amax), __float_as_uint(top1));   // ordered like their bits
            }
            if (p.lse && qi < p.sl) {
                // sum_j exp(s_j) = l * 2^(m_ref - POFF)  ->  natural-log LSE
                p.lse[(size_t)head * p.sl + qi] = (l > 0.f) ? (m - POFF + log2f(l)) * 0.6931471805599453f : -INFINITY;
            }
            return true;
        };

        start_tile();
        for (int j = 0;;) {   // one tile per trip, from block j on
            // Blocks without masked keys (uniform across the CTA) lie between those that start before the window of the tile's
            // last query, below j_lo, and those that reach past the sequence end or past the tile's first query (causal), from
            // j_hi on.  They run in a loop of their own.  (One loop with the test in it, masking key by key: 75.4 us for 64 heads of 3000 keys
            // of 64, window 512, then 71.2; 8192 keys causal 477 / 475.)
            // With 64-key blocks and 128-query tiles: (blk0 + j + 1) * BN > sl  <=>  j >= sl / BN - blk0;
            // (blk0 + j + 1) * BN - 1 > q0  <=>  j >= q0 / BN - blk0;  (blk0 + j) * BN < q0 + BM - window  <=>  j < ceil(..) - blk0.
            bool ok;
            if (!MASKED) {
                ok = clear_blocks(j, t.nblk);
            } else {
                int j_hi = p.sl / BN - t.blk0;
                if (p.causal) j_hi = min(j_hi, t.q0 / BN - t.blk0);
                int j_lo = (p.window > 0 && t.q0 + BM - p.window > 0) ? (t.q0 + BM - p.window + BN - 1) / BN - t.blk0 : 0;
                j_lo = min(j_lo, t.nblk);
                // one copy of each loop: edge, clear, edge
                ok = true;
                for (int stop = j_lo;; stop = t.nblk) {
                    ok = edge_blocks(j, stop);
                    if (!ok || j == t.nblk) break;
                    ok = clear_blocks(j, j_hi);
                    if (!ok) break;
                }
            }
            if (!ok) break;
            const float l = (l0 + l1) + (l2 + l3), m = m_ref;
            const int head = t.head, q0 = t.q0, stage_pv = rs_prev;
            const uint32_t phase_pv = rph_prev;
            if (WALK) {
                if (!mbar_wait_warp(bar_next, tph, abort_flag, ST_TIMEOUT_SOFTMAX)) break;
                t = tile_record(record);
                __syncwarp();
                if ((threadIdx.x & 31) == 0) mbar_arrive(bar_seen);
                tph ^= 1;
            }
            if (!WALK || MASKED || t.nblk == 0) {
                if (!epilogue(head, q0, l, m, stage_pv, phase_pv) || !WALK || t.nblk == 0) break;
                start_tile();
                j = 0;
                continue;
            }
            // The next tile's first block is worked on while this tile's last P V runs; its P is published once O has been read.  (512 heads
            // of 512, D = 64, 61.6 -> 51.8 us, of which this is 3.  With it the masked kernel, whose loops are twice the code, loses 2 to 17 %.)
            start_tile();
            if (!scores(0, s_addr, std::false_type())) break;
            uint32_t w[BN / 2];
#pragma unroll
            for (int g = 0; g < BN / 32; g++) exponentials(g, w + 16 * g, std::false_type());
            if (!epilogue(head, q0, l, m, stage_pv, phase_pv)) break;
#pragma unroll
            for (int g = 0; g < BN / 32; g++) tmem_st_32x32b_x16(s_addr + g * 16, w + 16 * g);
            publish(p_bar);
            s_addr ^= BN;
            p_bar ^= 8;
            j = 1;
        }
    }
    // ----------------------------------------------------------------- teardown
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    // Triggered at the end of a CTA, not at its start: the next call's pre-pass is spread over the SMs that have room when
    // it is launched, and during this kernel's last wave those are few (S = 2048 causal: 525 us a call against 343).  (Few tiles of D = 64: above.)
    pdl_trigger();
    const uint32_t code = *abort_flag;
    if (code != 0) {
        if (threadIdx.x == 0) atomicCAS(&g_fa_status, 0u, code);
        for (int i = 0; i < 200; i++) __nanosleep(1000);  // let copies already in flight land
        __syncthreads();
    }
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

struct DeviceState {
    std::once_flag once;   // first call on this device, from whichever host thread gets there first
    cudaError_t init_error = cudaSuccess;
    int num_sms = 148;
};
DeviceState g_dev[64];

void init_device(DeviceState* st, int dev);

// Whether the kernel converts V itself.  What a tile's conversion costs is paid once for every query tile that reads the key
// block, what the pre-pass costs once per key block: the line lies at a number of queries per key.  Measured with the pre-pass /
// in the kernel (us), one call behind another: D = 128, not causal, 128 heads of 1024 67 / 60, 64 of 1536 76 / 73, 64 of 2048 114 / 110, 24 of 4096
// 178 / 181; causal, half of whose queries see a key, but the last ones of every sequence see all: 512 heads of 512 74 / 63, 256 of
// 2048 277 / 265, 60 of 2500 98 / 96, 60 of 3000 132 / 131; window 1300, 20 heads of 8000, 112 / 109, 300, 128 of 2500, 113 / 107.
// D = 64 converts half as much per block: 64 of 2048 99 / 95, 42 of 3072 142 / 139, 32 of 4096 187 / 184; causal 40 of 4000 127 / 126, 64 of 5000
// 299 / 303; window 512 of 3000, 64 heads, 61 / 54.  Behind the kernel that has just written V the pre-pass costs more (both kernels, 32 of
// 1536 of 128, not causal, 75.0 / 64.0, 64 of 2048 173 / 164, 24 of 4096 223 / 223).  Past the lines the two forms differ by 3 % up to
// twice the keys, to either side.  Where no more than half of the SMs have a tile, nothing hides the conversion behind another
// CTA and its cost adds up along the longest tile: 8 heads of 1024 15.4 / 13.6, 4 of 1280 17.5 / 16.8, behind that kernel 24.5 / 26.5 and 24.3 /
// 23.5; 1 of 8192, with the producer converting, 75 / 92.
bool converts_v(const LaunchArgs& a, int num_sms) {
    const int limit = a.hd == 128 ? 1536 : 2560;
    const int span = a.causal && a.window > 0 && a.window < a.sl - BM ? a.window + BM : a.sl;   // keys of the longest tile
    const long long tiles = (long long)a.bh * ((a.sl + BM - 1) / BM);
    if (2 * tiles <= num_sms) return span <= 1024;
    return (a.causal && span == a.sl ? (long long)a.sl * 3 / 5 : span) <= limit;
}

// Heads whose tiles are interleaved, the longest of all of them first, where tiles differ in length.  In groups of 16 the long tiles of
// the last few heads end the launch, so it is one group, or equal ones, of as many heads as 48 MB of K and V allow.  Full groups stay
// where there is little to balance, up to 1.6 tiles per SM.  Causal, one call behind another, in groups of 16 / in as few as that, us: D = 128, 17
// heads of 2560 47.3 / 36.3, 24 of 2048 34.6 / 31.1, 40 of 2048 55.3 / 46.5, 256 of 2048 268 / 266, 32 of 1300 25.1 / 22.3, 48 of 1100 27.4 /
// 23.8, 48 of 600 15.1 / 13.9, but 32 of 850 15.9 / 16.8, 48 of 500 11.3 / 12.2, 32 of 600 11.6 / 12.1; D = 64, 18 of 3000 58.2 / 37.1, 64 of 700 16.4 /
// 13.7, 32 of 700 10.6 / 10.5; a window of 300, 128 of 2500 of 128 106.6 / 107.1.
int heads_together(const LaunchArgs& a, long long tiles, int num_sms) {
    const bool full = a.bh % HEAD_GROUP == 0 || a.bh % HEAD_GROUP >= HEAD_GROUP - 2;
    long long most = GROUP_ELEMS / ((long long)a.sl * a.hd);
    if (most < HEAD_GROUP || (full && 5 * tiles <= 8ll * num_sms)) most = HEAD_GROUP;
    const long long groups = (a.bh + most - 1) / most;
    return (int)((a.bh + groups - 1) / groups);
}

// Whether a CTA asks for more than half of an SM's shared memory, so that no two share one.  The CTAs of an early launch go where
// the kernel ahead has drained first, two to such an SM, and with few more tiles than SMs the longest ones of a causal launch, in
// front, then pair up while other SMs have a short one.  One to an SM, the short ones start where middle ones have finished.  Up to
// one and a half tiles per SM that was the faster form or level for up to 16 heads; with more heads a sequence has so few tiles that
// their start and finish count, which two to an SM hide (32 heads of 700 keys of 64, 192 tiles: 11 / 13 us).
// Behind the kernel that writes Q, K and V, us for both kernels, two to an SM / one: D = 64, 5 heads of 4000 60.4 / 49.7, 6 of 3500 57.2 / 45.0, 8 of
// 3000 50.9 / 40.5, 16 of 1500 32.4 / 27.3; D = 128, 4 of 4700 70.4 / 66.5, 8 of 2000 43.9 / 37.2, 16 of 1200 34.5 / 30.9.  One call behind
// another: the same 39.7 / 39.6, 35.6 / 35.3, 31.4 / 30.7, 17.9 / 17.6; 50.2 / 50.0, 24.5 / 24.5, 17.8 / 16.5; D = 128, 6 of 3500 50.7 / 39.2.
bool one_to_an_sm(const LaunchArgs& a, long long tiles, int num_sms) {
    return a.causal && (a.window <= 0 || a.window >= a.sl) && a.bh <= HEAD_GROUP && 2 * tiles <= 3ll * num_sms;
}

// Whether a CTA goes on to further tiles: as soon as there are more than fit at once.  That saves a tile its CTA's start (barriers,
// tensor memory, the first loads' latency: 3000 clk) and part of its end, which the other CTA of the SM hides in part.  A CTA per tile / a
// walk, us, one call behind another, below the power cap: D = 128, causal, 1500 heads of 128 41.0 / 33.8, 500 of 384 49.9 / 42.8, 88 of 2100 112 / 98.6;
// not causal 1500 of 128 32.8 / 24.5, 500 of 384 49.4 / 40.0, 136 of 1300 125 / 112, 58 of 3300 258 / 246; D = 64, causal, 500 of 384 36.6 / 28.6, 88 of
// 2100 88.2 / 81.8; not causal 500 of 384 39.0 / 31.5, 58 of 3300 237 / 225; window 512, 64 of 3000, 60.0 / 52.4.  Just past that line a few
// calls lose (D = 128, 340 to 400 of 128, causal, 12.0 to 12.6 / 12.9 to 13.1, 133 of 384, not causal, 15.5 / 16.4; D = 64, 12 to 27 of 3300 to 1300,
// causal, 3 %) and most gain (36 of 1300 of 128 25.8 / 23.1, 24 of 2100 33.7 / 30.7; 300 of 128 of 64 9.2 / 7.8).
bool walks(long long tiles, int num_sms) { return tiles > 2ll * num_sms; }

template <int HD, bool VRAW>
cudaError_t launch_hd(const LaunchArgs& a, int num_sms) {
    using C = Cfg<HD, VRAW>;
    const long long grid = (long long)a.bh * ((a.sl + BM - 1) / BM);
    const int v_chunks = (a.sl + V_CHUNK - 1) / V_CHUNK;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
    CUtensorMap tq, tk, tv;
    const CUtensorMapSwizzle swz = (HD == 128) ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    if (!make_tmap_u8_3d(&tq, a.q, a.bh, a.sl, HD, BM, HD, swz) ||
        !make_tmap_u8_3d(&tk, a.k, a.bh, a.sl, HD, BN, HD, swz) ||
        !(VRAW ? make_tmap_u8_3d(&tv, a.v, a.bh, a.sl, HD, BN, HD, HD == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE)
               : make_tmap_u16_3d(&tv, a.v16_workspace, a.bh, a.sl, HD, BN, 64, CU_TENSOR_MAP_SWIZZLE_128B)))
        return cudaErrorInvalidValue;
    Params p;
    p.group = heads_together(a, grid, num_sms);
    p.few = grid <= num_sms && !a.o_amax;
    p.bh = a.bh; p.sl = a.sl; p.n_qtiles = (a.sl + BM - 1) / BM;
    p.causal = a.causal; p.window = a.window;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.v_descale = a.v_descale;
    p.sq = a.scale_q_dev; p.sk = a.scale_k_dev; p.sv = a.scale_v_dev;
    p.o = reinterpret_cast<__half*>(a.o);
    p.lse = a.lse;
    p.o_amax = a.o_amax;
    p.v_flags = a.v_flags; p.v_epoch = a.v_epoch; p.v_chunks = v_chunks;
    if (!VRAW) {
        // pre-pass: V codes -> fp16 workspace
        const long long chunks = (long long)a.bh * v_chunks, cap = (long long)num_sms * V_CTAS_PER_SM;
        const cudaError_t e = launch_pdl(v_to_f16_kernel<HD>, (unsigned)(chunks < cap ? chunks : cap), V_THREADS, 0, a.stream,
                                         reinterpret_cast<const uint4*>(a.v), reinterpret_cast<uint4*>(a.v16_workspace), (int)chunks, v_chunks,
                                         a.sl, a.v_flags, a.v_epoch);
        if (e != cudaSuccess) return e;
    }
    const bool masked = a.causal || a.window > 0 || (a.sl % BN) != 0 || !(a.scale > 0.f);
    const size_t smem = one_to_an_sm(a, grid, num_sms) ? SMEM_ONE : C::SMEM_BYTES;
    auto start = [&](auto kernel) { return launch_pdl(kernel, (unsigned)grid, C::NUM_THREADS, smem, a.stream, tq, tk, tv, p); };
    const bool walk = walks(grid, num_sms);
    if (a.o_amax) return walk ? start(fa_fwd_kernel<HD, true, VRAW, true, true>) : start(fa_fwd_kernel<HD, true, VRAW, true, false>);   // the masked kernel serves every call
    if (walk) return masked ? start(fa_fwd_kernel<HD, true, VRAW, false, true>) : start(fa_fwd_kernel<HD, false, VRAW, false, true>);
    return masked ? start(fa_fwd_kernel<HD, true, VRAW, false, false>) : start(fa_fwd_kernel<HD, false, VRAW, false, false>);
}

}  // namespace

namespace {
void init_device(DeviceState* st, int dev) {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto kernel, int bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes > SMEM_ONE ? bytes : SMEM_ONE);
    };
    auto set_hd = [&](auto hd, auto vraw, auto walk) {
        constexpr int HD = decltype(hd)::value;
        constexpr bool VRAW = decltype(vraw)::value, WALK = decltype(walk)::value;
        set(fa_fwd_kernel<HD, true, VRAW, false, WALK>, Cfg<HD, VRAW>::SMEM_BYTES);
        set(fa_fwd_kernel<HD, false, VRAW, false, WALK>, Cfg<HD, VRAW>::SMEM_BYTES);
        set(fa_fwd_kernel<HD, true, VRAW, true, WALK>, Cfg<HD, VRAW>::SMEM_BYTES);
    };
    auto set_all = [&](auto vraw, auto walk) {
        set_hd(std::integral_constant<int, 128>(), vraw, walk);
        set_hd(std::integral_constant<int, 64>(), vraw, walk);
    };
    set_all(std::false_type(), std::false_type());
    set_all(std::false_type(), std::true_type());
    set_all(std::true_type(), std::false_type());
    set_all(std::true_type(), std::true_type());
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&st->num_sms, cudaDevAttrMultiProcessorCount, dev);
    st->init_error = e;
}
}  // namespace

bool needs_no_scratch(const LaunchArgs& a) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::call_once(g_dev[dev].once, init_device, &g_dev[dev], dev);
    return g_dev[dev].init_error == cudaSuccess && converts_v(a, g_dev[dev].num_sms);
}
size_t workspace_bytes(int bh, int sl, int hd) { return (size_t)bh * sl * hd * 2; }
size_t v_flag_count(int bh, int sl) { return (size_t)bh * ((sl + V_CHUNK - 1) / V_CHUNK); }

cudaError_t launch(const LaunchArgs& a) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::call_once(g_dev[dev].once, init_device, &g_dev[dev], dev);
    if (g_dev[dev].init_error != cudaSuccess) return g_dev[dev].init_error;
    if (converts_v(a, g_dev[dev].num_sms)) return a.hd == 128 ? launch_hd<128, true>(a, g_dev[dev].num_sms) : launch_hd<64, true>(a, g_dev[dev].num_sms);
    if (!a.v16_workspace || (reinterpret_cast<uintptr_t>(a.v16_workspace) & 127)) return cudaErrorInvalidValue;
    return a.hd == 128 ? launch_hd<128, false>(a, g_dev[dev].num_sms) : launch_hd<64, false>(a, g_dev[dev].num_sms);
}

cudaError_t launch_wait_expiry_selftest(cudaStream_t stream) {
    fa_wait_expiry_selftest_kernel<<<1, 32, 0, stream>>>();
    return cudaGetLastError();
}

int device_status() {
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return -(int)e;
    uint32_t code = 0, zero = 0;
    e = cudaMemcpyFromSymbol(&code, g_fa_status, sizeof(code));
    if (e != cudaSuccess) return -(int)e;
    if (code != 0) cudaMemcpyToSymbol(g_fa_status, &zero, sizeof(zero));
    return (int)code;
}

// ----------------------------------------------------------------------------------------
// Forward pass for callers that must not allocate.
//
// The regular entry points borrow their scratch (the fp16 copy of V) from a memory pool.
// Some callers cannot do that: code embedded in a framework that reserved the whole GPU up
// front and forbids any later cudaMalloc-family call, and real-time or safety-certified
// processes whose device memory map is frozen after start-up.  For them the scratch lives in
// the fixed device array below, which every GPU that loads this library carries until the
// process exits (32 MiB).  That caps one call at FA_NOALLOC_MAX_ELEMS elements of V.
//
// The array is shared by every call on that GPU and keeps the previous call's contents.
// Nothing in it has to start at zero: the pre-pass rewrites every element the kernel will read
// before the kernel runs.  Two calls whose GPU work overlaps (different streams) race on it;
// issue them on one stream or serialise them.  The first call on each device also looks up the
// array's device address and sets kernel attributes; make that first call before starting any
// stream capture.
// ----------------------------------------------------------------------------------------
constexpr size_t FA_NOALLOC_MAX_ELEMS = (size_t)16 << 20;  // batch_heads * seq_len * head_dim <= 16 Mi
static __device__ __align__(256) uint16_t g_noalloc_v16[FA_NOALLOC_MAX_ELEMS];

namespace {
// In host code `g_noalloc_v16` is only a stand-in for the device array; the device address is
// looked up once per device (with that device current) and cached.
struct NoallocState {
    std::once_flag once;
    fa_status_t status = FA_OK;
    cudaError_t cuda_error = cudaSuccess;
    void* ptr = nullptr;
};
NoallocState g_noalloc[64];

// One-time set-up for a device, run with that device current (do it before any stream capture): architecture
// check and the device address of the scratch array.  With lazy module loading this is also where the driver
// reserves the array's 32 MiB on that GPU.
void noalloc_init(NoallocState* st, int dev) {
    int major = 0;
    cudaError_t e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (e != cudaSuccess) { st->status = FA_ERR_CUDA; st->cuda_error = e; return; }
    if (major != 10) { st->status = FA_ERR_UNSUPPORTED_ARCH; return; }
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_noalloc_v16);
    if (e != cudaSuccess || !ptr) { st->status = FA_ERR_CUDA; st->cuda_error = e; return; }
    st->ptr = ptr;
}

void write_msg(char* err, int err_len, const char* msg) {
    if (err && err_len > 0) snprintf(err, (size_t)err_len, "%s", msg);
}
}  // namespace

}  // namespace fa_sm100

extern "C" __attribute__((visibility("default")))
fa_status_t fa_forward_noalloc(const fa_forward_args_t* g, char* err, int err_len) {
    using namespace fa_sm100;
    if (err && err_len > 0) err[0] = '\0';
    if (!g) { write_msg(err, err_len, "fa_forward_noalloc: null argument block"); return FA_ERR_INVALID_ARG; }
    if (!g->q || !g->k || !g->v || !g->o) { write_msg(err, err_len, "fa_forward_noalloc: null pointer in q/k/v/o"); return FA_ERR_INVALID_ARG; }
    if (g->batch_heads <= 0 || g->seq_len <= 0) { write_msg(err, err_len, "fa_forward_noalloc: bh/sl must be > 0"); return FA_ERR_INVALID_ARG; }
    if (g->head_dim != 64 && g->head_dim != 128) { write_msg(err, err_len, "fa_forward_noalloc: head_dim must be 64 or 128"); return FA_ERR_UNSUPPORTED_HD; }
    if (g->window < 0 || g->window > g->seq_len) { write_msg(err, err_len, "fa_forward_noalloc: window must be in [0, seq_len]"); return FA_ERR_INVALID_ARG; }
    if (g->causal != 0 && g->causal != 1) { write_msg(err, err_len, "fa_forward_noalloc: causal must be 0 or 1"); return FA_ERR_INVALID_ARG; }
    const uintptr_t align_or = reinterpret_cast<uintptr_t>(g->q) | reinterpret_cast<uintptr_t>(g->k) |
                               reinterpret_cast<uintptr_t>(g->v) | reinterpret_cast<uintptr_t>(g->o);
    if (align_or & 15) { write_msg(err, err_len, "fa_forward_noalloc: q/k/v/o must be 16-byte aligned"); return FA_ERR_INVALID_ARG; }
    if (reinterpret_cast<uintptr_t>(g->l_out) & 3) { write_msg(err, err_len, "fa_forward_noalloc: l_out must be 4-byte aligned"); return FA_ERR_INVALID_ARG; }
    const size_t elems = (size_t)g->batch_heads * (size_t)g->seq_len * (size_t)g->head_dim;
    if (elems > FA_NOALLOC_MAX_ELEMS) {
        if (err && err_len > 0)
            snprintf(err, (size_t)err_len,
                     "fa_forward_noalloc: batch_heads*seq_len*head_dim = %zu exceeds the fixed scratch of %zu elements "
                     "(32 MiB); split the batch or use fa_forward_ex", elems, FA_NOALLOC_MAX_ELEMS);
        return FA_ERR_UNSUPPORTED_SHAPE;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) { write_msg(err, err_len, "fa_forward_noalloc: cudaGetDevice failed"); return FA_ERR_CUDA; }
    NoallocState& st = g_noalloc[dev];
    std::call_once(st.once, noalloc_init, &st, dev);
    if (st.status == FA_ERR_UNSUPPORTED_ARCH) { write_msg(err, err_len, "fa_forward_noalloc: GPU is not compute capability 10.x"); return st.status; }
    if (st.status != FA_OK) {
        if (err && err_len > 0) snprintf(err, (size_t)err_len, "fa_forward_noalloc: set-up (cudaGetSymbolAddress): %s", cudaGetErrorString(st.cuda_error));
        return st.status;
    }
    // same dispatcher consultation as the other entries, so FA_SM120_DEBUG traces every forward call alike
    if (fa_dispatch_select(g->batch_heads, g->seq_len, g->head_dim, g->causal, g->window) == FA_KERNEL_NONE) {
        write_msg(err, err_len, "fa_forward_noalloc: no kernel matches this configuration");
        return FA_ERR_UNSUPPORTED_SHAPE;
    }
    LaunchArgs a{};
    a.q = g->q; a.k = g->k; a.v = g->v; a.o = g->o; a.lse = static_cast<float*>(g->l_out);
    a.bh = g->batch_heads; a.sl = g->seq_len; a.hd = g->head_dim; a.causal = g->causal; a.window = g->window;
    a.scale = g->scale; a.v_descale = (g->v_descale == 0.0f) ? 1.0f : g->v_descale;
    a.scale_q_dev = g->scale_q_dev; a.scale_k_dev = g->scale_k_dev; a.scale_v_dev = g->scale_v_dev;
    a.v16_workspace = st.ptr;
    a.stream = reinterpret_cast<cudaStream_t>(g->stream);
    e = launch(a);
    if (e != cudaSuccess) {
        if (err && err_len > 0) snprintf(err, (size_t)err_len, "fa_forward_noalloc: launch: %s", cudaGetErrorString(e));
        return FA_ERR_CUDA;
    }
    return FA_OK;
}

// Context-free twin of fa_device_status for callers of fa_forward_noalloc, which have no fa_ctx_t (creating one
// would create a memory pool, the very thing they avoid).  Synchronises the current device; allocates nothing.
extern "C" __attribute__((visibility("default")))
int fa_noalloc_device_status(void) { return fa_sm100::device_status(); }
