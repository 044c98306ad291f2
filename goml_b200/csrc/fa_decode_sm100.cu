// fa_decode_sm100.cu — FP8 attention for one new token per sequence against an FP8 KV cache
// (decode step), grouped-query heads, for NVIDIA B200 (sm_100a).
//
//   q        [B, Hq, D]          e4m3   (one token per sequence)
//   k_cache  [B, Hkv, Smax, D]   e4m3   (the layout the prefill kernels read: BH = B*Hkv, S = Smax)
//   v_cache  [B, Hkv, Smax, D]   e4m3
//   o        [B, Hq, D]          fp16,  lse [B, Hq] fp32 (natural log, optional)
//   seq_lens [B] int32 on the device (keys [0, seq_lens[b]) of sequence b are visible), or one length for all
//
// The step reads every cached key and value once and does 4*Hq*D FLOP per key: HBM-bound, so this is a streaming
// kernel on the warp-level tensor path, built to need as few instructions per cached byte as possible:
//
//  * K and V go from global memory straight into MMA fragments, with no shared memory in between.  Contraction and row
//    indices of an MMA may be permuted as long as both operands agree, so every lane's share of a key row is contiguous
//    (D/4 bytes of K, D/8 bytes of V) and a warp's loads cover whole rows.
//  * S^T = K Q^T (m16n8k32, e4m3): 16 keys are the rows, up to 8 query heads of the kv head the columns (two column tiles
//    for groups of 9 to 16); O^T += V^T P^T (m16n8k16, fp16): V bytes of two keys are paired with a byte permute and
//    converted in registers, P (kept in fp16: an e4m3 P costs 2.5e-2 relative error) is transposed by movmatrix.
//  * Each warp carries its own online-softmax state over the 16-key tiles it takes.  Whether a running maximum moves is
//    one vote per tile; row sums stay in the lanes until the end: the loop has no shuffles.
//  * A warp's next K block is on its way while it works on this block's softmax and V, and the next V block during the
//    next block's scores (Little's law asks for about 45 KB in flight per SM).
//
// How the keys are divided (Plan below): a pair (sequence, kv head) may be cut between chunks; the pieces are the CTAs of a cluster and
// hand their partial states to its first one, or leave them in a workspace where the CTA that finishes last takes them up.  Either merges them in
// a fixed order, so there is no second kernel and results do not depend on timing: the same call gives the same bits, eager or in a graph, on whatever stream.
//
// STREAMS: the rounding of P to fp16 depends on the running maximum it is taken against, so which keys share a warp and
// where a pair is cut show in the last bits of O.  A block that re-quantises its activations turns last bits into e4m3
// steps further on.  For one query head per kv head (what the decoder block runs) warp w therefore always takes keys
// 16w .. 16w + 15 of every 64-key chunk, and each such stream's maximum is what a walk over the pair (or over a fixed split of
// it) gives.  Grouped heads are free of that: the maximum may lag by 2^LAG, a warp takes 32 (D = 64: 64) contiguous keys,
// pairs are cut anywhere.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <mutex>

#include "fa_fwd_sm100.h"
#include "pdl.cuh"

namespace fa_sm100 {

namespace {

using namespace sm100;

constexpr int CHUNK = 64;        // keys per unit of work (page sizes are multiples of it)
constexpr int THREADS = 128;
constexpr int WARPS = THREADS / 32;
constexpr float LAG = 6.0f;      // log2 units
constexpr int LONGEST_SPLIT = 8;   // chunks of a split up to which a cluster is worth it: past that it is level with the workspace
constexpr int FEW_SPLITS = 8;      // up to so many the last CTA takes up the pieces of a pair in one round of 32 threads (16, D = 64)
constexpr int MAX_CLUSTER = 16, PORTABLE_CLUSTER = 8;   // splits of a pair that are a cluster
constexpr int HINTS = 2;         // chunks a CTA asks for ahead of the wait
// A wide warp step takes twice the keys of a narrow one (8 against 4 KB in flight per warp) and leaves registers for 12
// warps per SM instead of 16 (two column tiles: 8 instead of 12, or of 16 for D = 64).  It streams faster (0.8 GB of cache: 137 us against 146); the
// narrow one lets more CTAs be resident.
constexpr int ctas_per_sm(int d, int nq, bool wide) { return nq == 2 ? (wide ? 2 : d == 64 ? 4 : 3) : wide ? 3 : 4; }

// D = A B with a zero accumulator input
__device__ __forceinline__ void mma_e4m3_m16n8k32_zero(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_f16_m16n8k16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose_8x8_b16(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// two e4m3 pairs (the halves of w) -> two fp16 pairs
__device__ __forceinline__ void e4m3x4_to_h2x2(uint32_t w, uint32_t& lo, uint32_t& hi) {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, l;\n\tcvt.rn.f16x2.e4m3x2 %1, h;\n\t}" : "=r"(lo), "=r"(hi) : "r"(w));
}
// read once: not kept in L1 (with the default policy the D = 128 kernel is 9 % slower; one 256-bit load in place of two of
// these costs 3 %)
__device__ __forceinline__ void ldg128(uint32_t* r, const uint8_t* p) {
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(p));
}
__device__ __forceinline__ void ldg64(uint32_t* r, const uint8_t* p) {
    asm volatile("ld.global.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "l"(p));
}

// Plans.
//  SPLITS: CTA i is split i % splits of pair i / splits; a split is chunks_per_split chunks.  Few pairs: one resident CTA
//          per split, or a cluster per pair whose CTAs take equal runs of the splits.  Many: one CTA per pair.
//  LINE:   the chunks of all pairs form one line that is cut into equal pieces, one per resident CTA, so sequences of very
//          different lengths load all SMs alike.
enum Plan : int { SPLITS, LINE };

struct DecodeParams {
    const uint8_t* q;
    const uint8_t* k;
    const uint8_t* v;
    __half* o;
    float* lse;
    const int* seq_lens;
    int batch, hq, hkv, group, s_max, seq_len;
    float scale_log2, v_descale;
    const float* sq;
    const float* sk;
    const float* sv;
    int plan, splits, chunks_per_split;
    int cluster;   // CTAs of a pair, each with a run of its splits (CLUSTER)
    bool hints;   // on the line: ask for the first chunks ahead of the wait
    // paged cache: k, v are [num_pages, Hkv, page_size, D]; the chunk at key k0 of sequence b lives in page
    // block_table[b * max_pages + k0 / page_size]
    const int* block_table;
    int page_size, max_pages, num_pages;
    uint32_t page_mul, page_shr;   // key / page_size as multiply-high and shift
    // partial states, two slots per CTA: [slot][rows][D] un-normalised outputs, then [slot][rows][2] (m in log2 units, l)
    float* ws_o;
    float* ws_ml;
    uint32_t* arrivals;   // [B*Hkv], zero before and after every launch
};

template <int D, int NQ, bool WIDE>
struct Cfg {
    static constexpr int TILES = (D == 128 ? 1 : 2) * (WIDE ? 2 : 1);   // 16-key tiles per warp step = chunks per CTA step
    static constexpr int KSTEPS = D / 32;
    static constexpr int KW = D / 16;                    // 32-bit words of a lane's share of one K row
    static constexpr int MT = D / 16;                    // 16-row tiles of O^T
    static constexpr int VW = D / 32;                    // 32-bit words of a lane's share of one V row
    static constexpr int ROWS = 8 * NQ;                  // query columns
    static constexpr int PITCH = D + 4;                  // floats per row of the merge buffer
};

__device__ __forceinline__ int seq_len_of(const DecodeParams& p, int b) { return p.seq_lens ? min(max(__ldcg(p.seq_lens + b), 0), p.s_max) : p.seq_len; }
__device__ __forceinline__ int chunks_of(int len) { return (len + CHUNK - 1) / CHUNK; }

// [begin, end) of piece i of equal pieces of a line (the first `remainder` pieces are one unit longer), and back
struct Cut {
    int q, r;
    __device__ __forceinline__ Cut(int quotient, int remainder) : q(quotient), r(remainder) {}
    __device__ __forceinline__ int begin(int i) const { return i * q + min(i, r); }
    __device__ __forceinline__ int piece_of(int u) const { return u < r * (q + 1) ? u / (q + 1) : r + (u - r * (q + 1)) / q; }
};

__device__ __forceinline__ void fold(float& L, float4& O, float l, const float4& o, float f) {
    L += l * f;
    O.x += o.x * f; O.y += o.y * f; O.z += o.z * f; O.w += o.w * f;
}
template <int D>
__device__ __forceinline__ void store_out(const DecodeParams& p, size_t row, int col, float M, float L, const float4& O, float vds) {
    const float inv = L > 0.f ? vds / L : 0.f;
    if ((reinterpret_cast<uintptr_t>(p.o) & 7) == 0) {   // o need only be 2-byte aligned
        *reinterpret_cast<uint2*>(p.o + row * D + col) = make_uint2(pack_h2(O.x * inv, O.y * inv), pack_h2(O.z * inv, O.w * inv));
    } else {
        __half* h = p.o + row * D + col;
        h[0] = __float2half_rn(O.x * inv); h[1] = __float2half_rn(O.y * inv);
        h[2] = __float2half_rn(O.z * inv); h[3] = __float2half_rn(O.w * inv);
    }
    if (col == 0 && p.lse) p.lse[row] = (L > 0.f) ? (M + log2f(L)) * 0.6931471805599453f : -INFINITY;
}

// What a hint ahead of the wait is addressed by: read past L1, which the wait does not invalidate.
__device__ __forceinline__ int peek_s32(const int* p) {
    int r;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(r) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ void prefetch_l2(const uint8_t* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_here() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }   // nothing is handed over
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// To the same place in another CTA of the cluster
__device__ __forceinline__ uint32_t in_rank(const float* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_rank(const float* p, int rank, const float4& v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(in_rank(p, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_rank(const float* p, int rank, const float2& v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(in_rank(p, rank)), "f"(v.x), "f"(v.y) : "memory");
}

struct Segment {
    int b, kvh, len;                // sequence, kv head, keys of the sequence
    int n_chunks, c_begin, c_end;   // chunks of the pair, and those of them this CTA takes
    int pair_u0;                    // unit of the line where the pair starts
};

// CLUSTER: the splits of a pair are the CTAs of a cluster (one query head per kv head), its first CTA the one with the first run of them
// MANY: all threads of the last CTA take up the pieces of a pair in the workspace (one query head per kv head).  A kernel of its own, for its code costs every call 0.1 us:
// 12 heads of 16 keys, us, with it / without 2.73 / 2.64, 2 of 385 (7 splits) 4.98 / 4.79, 14 of 256 (4) 4.84 / 4.65; but 8 of 1000 (16) 5.30 / 5.92, 2 of 4000 5.65 / 8.86.
template <int D, int NQ, bool WIDE, bool STREAMS, bool PAGED, bool MANY = false, bool CLUSTER = false>
__global__ void __launch_bounds__(THREADS, ctas_per_sm(D, NQ, WIDE)) fa_decode_kernel(const DecodeParams p) {
    using C = Cfg<D, NQ, WIDE>;
    static_assert(!(CLUSTER || MANY) || (STREAMS && NQ == 1), "clusters and many pieces are for one query head per kv head");
    __shared__ __align__(16) float s_o[WARPS][CLUSTER ? 1 : C::ROWS][C::PITCH];
    __shared__ float s_m[WARPS][C::ROWS], s_l[WARPS][C::ROWS];
    __shared__ Segment s_next[WARPS];
    __shared__ uint32_t s_last;
    // CLUSTER: what the splits of the pair hand to its first CTA
    __shared__ __align__(16) float s_part_o[CLUSTER ? MAX_CLUSTER : 1][CLUSTER ? D : 4];
    __shared__ __align__(8) float s_part_ml[CLUSTER ? MAX_CLUSTER : 1][2];
    if (CLUSTER) cluster_here();   // its phase says that every CTA runs, so that its shared memory may be written

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;              // MMA fragment coordinates

    // a sequence with no visible key is on nobody's piece: O = 0, LSE = -inf
    auto empty_sequence = [&](int b) {
        for (int i = 0; i < p.hq * D; i++) p.o[(size_t)b * p.hq * D + i] = __float2half_rn(0.f);
        if (p.lse)
            for (int i = 0; i < p.hq; i++) p.lse[(size_t)b * p.hq + i] = -INFINITY;
    };

    // ---- this CTA's piece of the line.  Every warp adds the lengths up for itself (no barrier); lane i keeps those of
    // sequences i, i + 32, .. of the first 32 * LENS, larger batches read theirs again where they need them.
    constexpr int LENS = 4;
    int lens[LENS] = {};
    auto lane_len = [&](int b0) -> int {   // length of sequence b0 + lane, b0 a multiple of 32
        if (b0 < 32 * LENS) {
            int x = lens[0];
#pragma unroll
            for (int i = 1; i < LENS; i++)
                if (b0 == 32 * i) x = lens[i];
            return x;
        }
        return b0 + lane < p.batch ? seq_len_of(p, b0 + lane) : 0;
    };
    // the part of one pair that starts at unit u and ends at unit end or with the pair.  The sequence, its length and what lies
    // before it come from one reading of the lengths: nothing is addressed from two that disagree (a caller that rewrites them
    // while the kernel runs gets wrong results, and an empty part where the line has become shorter than u).
    auto segment_at = [&](int u, int end) {
        Segment x;
        x.b = x.kvh = x.len = x.n_chunks = x.c_begin = x.c_end = x.pair_u0 = 0;
        for (int b0 = 0, before = 0; b0 < p.batch; b0 += 32) {
            const int len = lane_len(b0), n = chunks_of(len) * p.hkv;
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t past = __ballot_sync(0xffffffffu, before + incl > u);   // first lane whose sequence ends past u
            if (past) {
                const int at = __ffs(past) - 1, seq_u0 = before + __shfl_sync(0xffffffffu, incl - n, at);
                x.b = b0 + at;
                x.len = __shfl_sync(0xffffffffu, len, at);
                x.n_chunks = chunks_of(x.len);
                x.kvh = (u - seq_u0) / x.n_chunks;
                x.pair_u0 = seq_u0 + x.kvh * x.n_chunks;
                x.c_begin = u - x.pair_u0;
                x.c_end = min(x.n_chunks, x.c_begin + (end - u));
                break;
            }
            before += __shfl_sync(0xffffffffu, incl, 31);
        }
        return x;
    };

    auto page_of = [&](int key) -> int { return (int)(__umulhi((uint32_t)key, p.page_mul) >> (p.page_shr - 1)); };
    // byte offset of chunk c (the same in K and V), or -1 where the table names no page of the pool: nothing is read
    // there, the keys count as zeros
    auto offset = [&](const Segment& x, int c, int page) -> long long {
        if (!PAGED) return (((long long)x.b * p.hkv + x.kvh) * p.s_max + (long long)c * CHUNK) * D;
        if (page < 0 || page >= p.num_pages) return -1;
        const int key = c * CHUNK;
        return (((long long)page * p.hkv + x.kvh) * p.page_size + (key - page_of(key) * p.page_size)) * D;
    };

    // On the line the piece is found twice, the first time while the kernel ahead still runs (the append of the new token, usually), which leaves memory
    // idle: this CTA's first chunks are asked for from L2, by the lengths and the table as they then are.  Those may still be the last
    // step's, or anything: they are bounded like the ones read behind the wait, and nothing but hints comes of them.  Two chunks for each of
    // 444 CTAs are 14 MB.  Append and attention, 8 kv heads, paged, without / with: 24 sequences of 3000 to 6000 keys 48.7 / 47.3 us, 12 of
    // 1500 to 3000 24.1 / 23.0, one of 8000 18.0 / 17.3, one of 500 9.4 / 9.5; with the lengths and pages of other sequences in place until
    // the append, the same 48.3 / 47.1, 27.4 / 26.7, 21.8 / 21.5, 14.4 / 14.4.  Not behind a kernel that clears the counters (captured calls):
    // that one starts when the append has ended, and the hints cost a call 0.9 us.  (As two trips of one loop the search cost pieces of one to two
    // chunks: one sequence of 4000 18.3, now 16.5, 16.6 without.)  A CTA per pair or split gains nothing (a step of 64 sequences 336 / 341, of one
    // 78.1 / 77.7) and is found once.
    //
    // CLUSTER: the run of splits that this CTA has, and whose rank the first run is.  Equal ranks of clusters lie on few SMs, and short sequences give work to the
    // first runs alone, so that these go round the ranks: 5 sequences of 300 keys, 16 heads of 128, a cache of 1064 7.9 / 7.3 us, 2 of 60, 32 heads, 4.4 / 3.9, full caches level.
    int run = 0, first_rank = 0;
    Segment seg;
    int cut_q = 0, cut_r = 0;
    int mid = 0, mid_end = 0;    // units of the segments still to come in line order
    const bool line = !STREAMS && p.plan == LINE;   // streams are not cut along a line: that code is not compiled for them
    auto find_piece = [&](const bool early) {
        seg.b = seg.kvh = seg.len = seg.n_chunks = seg.c_begin = seg.c_end = seg.pair_u0 = 0;
        if (!line) {
            const int per_pair = CLUSTER ? p.cluster : p.splits;
            const int pair = blockIdx.x / per_pair;
            int split = blockIdx.x - pair * per_pair;
            if (CLUSTER) {
                first_rank = pair % per_pair;
                split = run = (split < first_rank ? split + per_pair : split) - first_rank;
            }
            seg.b = pair / p.hkv;
            seg.kvh = pair - seg.b * p.hkv;
            seg.len = seq_len_of(p, seg.b);
            seg.n_chunks = chunks_of(seg.len);
            int each = p.chunks_per_split;
            if (CLUSTER) {   // the splits that the sequence has, in equal runs
                const int used = (seg.n_chunks + each - 1) / each;
                each *= (used + p.cluster - 1) / p.cluster;
            }
            seg.c_begin = split * each;
            seg.c_end = min(seg.n_chunks, seg.c_begin + each);
            if (seg.n_chunks == 0 && seg.kvh == 0 && split == 0 && threadIdx.x == 0) empty_sequence(seg.b);
        } else {
#pragma unroll
            for (int i = 0; i < LENS; i++) lens[i] = 32 * i + lane < p.batch ? seq_len_of(p, 32 * i + lane) : 0;
            int total = 0;
            for (int b0 = 0; b0 < p.batch; b0 += 32) {
                const int b = b0 + lane, n = chunks_of(lane_len(b0));
                if (!early && n == 0 && b < p.batch && warp == 0 && b % gridDim.x == blockIdx.x) empty_sequence(b);
                total += __reduce_add_sync(0xffffffffu, n);
            }
            total *= p.hkv;
            const int pieces = gridDim.x;
            cut_q = total / pieces;
            cut_r = total - cut_q * pieces;
            const Cut cut(cut_q, cut_r);
            mid = cut.begin(blockIdx.x);
            mid_end = cut.begin(blockIdx.x + 1);
            if (mid < mid_end) seg = segment_at(mid, mid_end);
            mid += seg.c_end - seg.c_begin;
        }
    };
    if (line && p.hints) {
        find_piece(true);
        const int c = seg.c_begin + lane;
        if (warp < 2 && lane < HINTS && c < seg.c_end) {
            const long long off = offset(seg, c, PAGED ? peek_s32(p.block_table + (size_t)seg.b * p.max_pages + page_of(c * CHUNK)) : 0);
            if (off >= 0) prefetch_l2((warp == 0 ? p.k : p.v) + off, (PAGED ? CHUNK : min(CHUNK, p.s_max - c * CHUNK)) * D);
        }
        __syncwarp();
    }
    pdl_wait();
    pdl_trigger();
    find_piece(false);
    // CLUSTER: each CTA reads the length for itself.  Under a caller that rewrites the lengths while the kernel runs a peer may hand over what the first CTA
    // does not wait for, so the first one ends behind the second phase, when every peer has handed over or gone, whatever it has read itself.  Where it has no keys
    // or all of them it arrives at that phase here, without the order of memory that a hand-over needs (five sequences of 130 keys, 32 heads, a cache of 500: 7.9 us
    // with arrivals that release, 6.8 so; 7.2 without a second phase but with a first arrival that releases).
    const bool nothing = seg.c_begin >= seg.c_end;
    if (CLUSTER && run == 0 && (nothing || seg.c_end == seg.n_chunks)) {
        __syncwarp();
        cluster_wait();
        cluster_here();
        if (nothing) cluster_wait();
    }
    if (nothing) return;
    float scale_log2 = p.scale_log2;
    if (p.sq) scale_log2 *= ld_f32(p.sq);
    if (p.sk) scale_log2 *= ld_f32(p.sk);
    const Cut cut(cut_q, cut_r);

    // A CTA step is TILES chunks.  Tile i of warp w: keys 16w.. of chunk i (STREAMS), or 16i.. of the warp's own contiguous
    // run of TILES * 16 keys.
    auto tile_chunk = [&](int i) { return STREAMS ? i : (warp * C::TILES * 16) / CHUNK; };
    auto tile_key = [&](int i) { return STREAMS ? 16 * warp : (warp * C::TILES * 16) % CHUNK + 16 * i; };
    constexpr int OFFS = STREAMS ? C::TILES : 1;        // chunks a warp touches per step
    // lane-constant byte offsets inside a tile: K rows g and g + 8, V rows 2t, 2t + 1, 2t + 8, 2t + 9
    const uint32_t k_lane = g * D + (D / 4) * t, v_lane = 2 * t * D + (D / 8) * g;
    uint32_t kr[C::TILES][2][C::KW];    // [tile][row g / g + 8][words]
    uint32_t vr[C::TILES][4][C::VW];
    auto entry = [&](const Segment& x, int c) -> int {   // table entry of chunk c
        return PAGED && c < x.c_end ? ld_s32(p.block_table + (size_t)x.b * p.max_pages + page_of(c * CHUNK)) : 0;
    };
    // left: keys from the chunk's first one to the end of the sequence.  Keys past it are not read but taken as zeros: they
    // may hold anything (0 x NaN would poison O)
    auto load_k = [&](int i, int left, long long off) {
        const uint8_t* base = p.k + off + (k_lane + tile_key(i) * D);
        if (left >= CHUNK) {
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int h = 0; h < D / 64; h++) ldg128(kr[i][r] + 4 * h, base + 8 * r * D + 16 * h);
        } else {
#pragma unroll
            for (int r = 0; r < 2; r++) {
#pragma unroll
                for (int w = 0; w < C::KW; w++) kr[i][r][w] = 0u;
                if (tile_key(i) + 8 * r + g < left) {
#pragma unroll
                    for (int h = 0; h < D / 64; h++) ldg128(kr[i][r] + 4 * h, base + 8 * r * D + 16 * h);
                }
            }
        }
    };
    auto load_v_row = [&](int i, int r, const uint8_t* row) {
        if (D == 128) ldg128(vr[i][r], row);
        else ldg64(vr[i][r], row);
    };
    auto load_v = [&](int i, int left, long long off) {
        const uint8_t* base = p.v + off + (v_lane + tile_key(i) * D);
        if (left >= CHUNK) {
#pragma unroll
            for (int r = 0; r < 4; r++) load_v_row(i, r, base + ((r & 1) + 8 * (r >> 1)) * D);
        } else {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int key = (r & 1) + 8 * (r >> 1);   // + 2t
#pragma unroll
                for (int w = 0; w < C::VW; w++) vr[i][r][w] = 0u;
                if (tile_key(i) + key + 2 * t < left) load_v_row(i, r, base + key * D);
            }
        }
    };
    // keys left of chunk c of a segment for load_k / load_v: none past the segment's end or where there is no page
    auto left_of = [&](const Segment& x, int c, long long off) { return c < x.c_end && off >= 0 ? x.len - c * CHUNK : 0; };
    auto chunk_at = [&](int j) { return STREAMS ? j : tile_chunk(0); };   // j-th chunk a warp touches in a step

    bool loaded = false;   // the segment's first chunks are already on their way
    for (;;) {             // one segment per trip
        int page_next[OFFS];
        if (!loaded) {
#pragma unroll
            for (int j = 0; j < OFFS; j++) {
                const int c = seg.c_begin + chunk_at(j);
                const long long off = offset(seg, c, entry(seg, c));
                const int left = left_of(seg, c, off);
#pragma unroll
                for (int i = j; i < (STREAMS ? j + 1 : C::TILES); i++) {
                    load_k(i, left, off);
                    load_v(i, left, off);
                }
            }
        }
        loaded = false;
#pragma unroll
        for (int j = 0; j < OFFS; j++) page_next[j] = entry(seg, seg.c_begin + C::TILES + chunk_at(j));

        // the segment behind this one waits in shared memory (a copy per warp: no barrier)
        bool more;
        int next_entry[OFFS];
        {
            Segment next;
            more = line && mid < mid_end;
            if (more) {
                next = segment_at(mid, mid_end);
                more = next.c_begin < next.c_end;
                mid += next.c_end - next.c_begin;
            }
            if (more) {
#pragma unroll
                for (int j = 0; j < OFFS; j++) next_entry[j] = entry(next, next.c_begin + chunk_at(j));
                if (lane == 0) s_next[warp] = next;
            }
            __syncwarp();
        }

        const int b = seg.b, kvh = seg.kvh;
        // Q fragments (B operand): column g of tile n is query head kvh * group + 8n + g, words as in the K rows
        uint32_t qf[NQ][C::KW];
#pragma unroll
        for (int n = 0; n < NQ; n++) {
            const bool live = 8 * n + g < p.group;
            const uint8_t* qb = p.q + ((size_t)b * p.hq + (size_t)kvh * p.group + 8 * n + g) * D + (D / 4) * t;
#pragma unroll
            for (int w = 0; w < C::KW; w++) qf[n][w] = live ? *reinterpret_cast<const uint32_t*>(qb + 4 * w) : 0u;
        }

        // online-softmax state for query columns 2t and 2t + 1 of every column tile: running maximum (the same in all lanes
        // g) and this lane's part of the sum
        float m[NQ][2], l[NQ][2];
        float acc[NQ][C::MT][4];
#pragma unroll
        for (int n = 0; n < NQ; n++) {
#pragma unroll
            for (int e = 0; e < 2; e++) { m[n][e] = -INFINITY; l[n][e] = 0.f; }
#pragma unroll
            for (int i = 0; i < C::MT; i++) acc[n][i][0] = acc[n][i][1] = acc[n][i][2] = acc[n][i][3] = 0.f;
        }

        // CLUSTER: the same of the splits before this one, of the only query
        float m_all = -INFINITY, l_all = 0.f, acc_all[CLUSTER ? C::MT : 1][2] = {};
        auto end_of_split = [&] {
            const float top = fmaxf(m_all, m[0][0]);
            if (top == -INFINITY) return;
            const float f0 = ex2f(m_all - top), f1 = ex2f(m[0][0] - top);
            m_all = top;
            l_all = l_all * f0 + l[0][0] * f1;
#pragma unroll
            for (int j = 0; j < (CLUSTER ? C::MT : 0); j++) {
                acc_all[j][0] = acc_all[j][0] * f0 + acc[0][j][0] * f1;
                acc_all[j][1] = acc_all[j][1] * f0 + acc[0][j][2] * f1;
                acc[0][j][0] = acc[0][j][2] = 0.f;
            }
            m[0][0] = -INFINITY;
            l[0][0] = 0.f;
        };
        int split_end = CLUSTER ? seg.c_begin + p.chunks_per_split : 0;

        for (int c = seg.c_begin; c < seg.c_end; c += C::TILES) {
            if (CLUSTER && C::TILES == 1 && c == split_end) {   // P is rounded against the maximum of its own split; with two tiles a step, below
                end_of_split();
                split_end += p.chunks_per_split;
            }
            // ---- S^T = K Q^T, one accumulator per k-step: independent MMAs instead of a chain
            float s[NQ][C::TILES][4];
#pragma unroll
            for (int n = 0; n < NQ; n++)
#pragma unroll
                for (int i = 0; i < C::TILES; i++) {
                    float part[C::KSTEPS][4];
#pragma unroll
                    for (int ks = 0; ks < C::KSTEPS; ks++)
                        mma_e4m3_m16n8k32_zero(part[ks], kr[i][0][2 * ks], kr[i][1][2 * ks], kr[i][0][2 * ks + 1], kr[i][1][2 * ks + 1],
                                               qf[n][2 * ks], qf[n][2 * ks + 1]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        float x = part[0][e];
#pragma unroll
                        for (int ks = 1; ks < C::KSTEPS; ks++) x += part[ks][e];
                        s[n][i][e] = x * scale_log2;
                    }
                }
            // ---- the next chunks' keys, of this segment or, behind its last ones, of the next: the merge below then hides
            // their latency
            const bool roll = c + C::TILES >= seg.c_end;
            const bool fetch = !roll || more;
            int left_n[OFFS];
            long long off_n[OFFS];
            if (!roll) {
#pragma unroll
                for (int j = 0; j < OFFS; j++) {
                    const int cn = c + C::TILES + chunk_at(j);
                    off_n[j] = offset(seg, cn, page_next[j]);
                    left_n[j] = left_of(seg, cn, off_n[j]);
                    page_next[j] = entry(seg, cn + C::TILES);
                }
            } else if (more) {
                const Segment next = s_next[warp];
#pragma unroll
                for (int j = 0; j < OFFS; j++) {
                    const int cn = next.c_begin + chunk_at(j);
                    off_n[j] = offset(next, cn, next_entry[j]);
                    left_n[j] = left_of(next, cn, off_n[j]);
                }
                loaded = true;
            }
            if (fetch) {
#pragma unroll
                for (int i = 0; i < C::TILES; i++) load_k(i, left_n[STREAMS ? i : 0], off_n[STREAMS ? i : 0]);
            }
            // ---- softmax and O^T += V^T P^T, 16 keys at a time.  s[n][i][e] = key g (e < 2) or g + 8 of tile i,
            // query 8n + 2t + (e & 1)
#pragma unroll
            for (int i = 0; i < C::TILES; i++) {
                const int ci = c + tile_chunk(i);
                if (CLUSTER && C::TILES > 1 && ci == split_end) {
                    end_of_split();
                    split_end += p.chunks_per_split;
                }
                const int key0 = ci * CHUNK + tile_key(i), key_end = ci < seg.c_end ? seg.len : 0;
                if (key0 + 16 > key_end) {   // only the last chunk of a sequence has keys past its end
#pragma unroll
                    for (int n = 0; n < NQ; n++)
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (key0 + g + 8 * (e >> 1) >= key_end) s[n][i][e] = -INFINITY;
                }
                float mx[NQ][2];
                bool bump = false;
#pragma unroll
                for (int n = 0; n < NQ; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        mx[n][e] = fmaxf(s[n][i][e], s[n][i][e + 2]);
                        bump = bump || mx[n][e] > (STREAMS ? m[n][e] : m[n][e] + LAG);
                    }
                if (__any_sync(0xffffffffu, bump)) {   // rare once a few chunks are in
#pragma unroll
                    for (int n = 0; n < NQ; n++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
#pragma unroll
                            for (int o = 4; o < 32; o <<= 1) mx[n][e] = fmaxf(mx[n][e], __shfl_xor_sync(0xffffffffu, mx[n][e], o));
                            const float m_new = fmaxf(m[n][e], mx[n][e]);
                            const float f = m[n][e] == -INFINITY ? 0.f : ex2f(m[n][e] - m_new);
                            m[n][e] = m_new;
                            l[n][e] *= f;
#pragma unroll
                            for (int j = 0; j < C::MT; j++) {
                                acc[n][j][e] *= f;
                                acc[n][j][e + 2] *= f;
                            }
                        }
                }
                // P^T as B fragments: rows (keys) 2t, 2t + 1 and 2t + 8, 2t + 9 of column g
                uint32_t pf[NQ][2];
#pragma unroll
                for (int n = 0; n < NQ; n++) {
                    float pv[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        pv[e] = m[n][e & 1] == -INFINITY ? 0.f : ex2f(s[n][i][e] - m[n][e & 1]);
                        l[n][e & 1] += pv[e];
                    }
                    pf[n][0] = transpose_8x8_b16(pack_h2(pv[0], pv[1]));
                    pf[n][1] = transpose_8x8_b16(pack_h2(pv[2], pv[3]));
                }
                // rows g and g + 8 of tile j of O^T are d = (D/8) g + 2j and + 1
#pragma unroll
                for (int w = 0; w < C::VW; w++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t sel = h ? 0x7362 : 0x5140;   // bytes (2h, 2h + 1) of two keys, interleaved
                        uint32_t a[4];
                        e4m3x4_to_h2x2(__byte_perm(vr[i][0][w], vr[i][1][w], sel), a[0], a[1]);
                        e4m3x4_to_h2x2(__byte_perm(vr[i][2][w], vr[i][3][w], sel), a[2], a[3]);
#pragma unroll
                        for (int n = 0; n < NQ; n++) mma_f16_m16n8k16(acc[n][2 * w + h], a, pf[n][0], pf[n][1]);
                    }
            }
            if (fetch) {
#pragma unroll
                for (int i = 0; i < C::TILES; i++) load_v(i, left_n[STREAMS ? i : 0], off_n[STREAMS ? i : 0]);
            }
        }

        // ---- merge the four warps' states
        if (CLUSTER) {
            end_of_split();
            m[0][0] = m_all;
            l[0][0] = l_all;
#pragma unroll
            for (int j = 0; j < (CLUSTER ? C::MT : 0); j++) {
                acc[0][j][0] = acc_all[j][0];
                acc[0][j][2] = acc_all[j][1];
            }
        }
        const bool whole = seg.c_begin == 0 && seg.c_end == seg.n_chunks;
#pragma unroll
        for (int n = 0; n < NQ; n++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) l[n][e] += __shfl_xor_sync(0xffffffffu, l[n][e], o);
                const int row = 8 * n + 2 * t + e;
                if (g == 0) {
                    s_m[warp][row] = m[n][e];
                    s_l[warp][row] = l[n][e];
                }
                if (row < p.group) {
#pragma unroll
                    for (int j = 0; j < C::MT; j++)
                        *reinterpret_cast<float2*>(&s_o[warp][CLUSTER ? 0 : row][(D / 8) * g + 2 * j]) = make_float2(acc[n][j][e], acc[n][j][e + 2]);
                }
            }
        __syncthreads();
        if (CLUSTER && !whole) cluster_wait();
        // slots of a cut pair: its splits in order, or on the line the odd slot of the CTA that has its first piece and the
        // even slots of the CTAs after that
        const int slot = !line ? blockIdx.x : 2 * blockIdx.x + (seg.c_begin == 0 ? 1 : 0);
        const float vds = p.sv ? p.v_descale * ld_f32(p.sv) : p.v_descale;
        for (int idx = threadIdx.x; idx < p.group * (D / 4); idx += THREADS) {   // four columns per thread and step
            const int row = idx / (D / 4), col = idx % (D / 4) * 4;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < WARPS; w++) M = fmaxf(M, s_m[w][row]);
            float L = 0.f;
            float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < WARPS; w++) {
                const float mw = s_m[w][row];
                fold(L, O, s_l[w][row], *reinterpret_cast<const float4*>(&s_o[w][CLUSTER ? 0 : row][col]), mw == -INFINITY ? 0.f : ex2f(mw - M));
            }
            if (whole) {
                store_out<D>(p, ((size_t)b * p.hq + (size_t)kvh * p.group + row), col, M, L, O, vds);
            } else if (CLUSTER) {
                st_rank(&s_part_o[run][col], first_rank, O);
                if (col == 0) st_rank(s_part_ml[run], first_rank, make_float2(M, L));
            } else {
                const size_t at = (size_t)slot * C::ROWS + row;
                __stcg(reinterpret_cast<float4*>(p.ws_o + at * D + col), O);
                if (col == 0) __stcg(reinterpret_cast<float2*>(p.ws_ml + at * 2), make_float2(M, L));
            }
        }
        if (CLUSTER) {
            __syncwarp();
            if (!whole) cluster_arrive();
            if (seg.c_begin != 0) return;   // what it has handed over is the first one's
            cluster_wait();
            if (whole) return;
            // A column to a thread, the pieces in order
            const int parts = (seg.n_chunks + seg.c_end - 1) / seg.c_end;
            float M = -INFINITY;
            for (int i = 0; i < parts; i++) M = fmaxf(M, s_part_ml[i][0]);
            if (threadIdx.x < D / 4) {
                float L = 0.f;
                float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
                const int col = threadIdx.x * 4;
#pragma unroll 4
                for (int i = 0; i < parts; i++)
                    fold(L, O, s_part_ml[i][1], *reinterpret_cast<const float4*>(&s_part_o[i][col]), M == -INFINITY ? 0.f : ex2f(s_part_ml[i][0] - M));
                store_out<D>(p, (size_t)b * p.hq + kvh, col, M, L, O, vds);
            }
            return;
        }
        if (!whole) {
            int parts, slot0, slot_step;   // the pair's pieces: slot0, then slot0 + 1 + i * slot_step
            if (!line) {
                parts = (seg.n_chunks + p.chunks_per_split - 1) / p.chunks_per_split;
                slot0 = (blockIdx.x / p.splits) * p.splits;
                slot_step = 1;
            } else {
                const int first = cut.piece_of(seg.pair_u0);
                parts = cut.piece_of(seg.pair_u0 + seg.n_chunks - 1) - first + 1;
                slot0 = 2 * first + 1;
                slot_step = 2;
            }
            const int bh = b * p.hkv + kvh;
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                s_last = atomicAdd(p.arrivals + bh, 1u) == (uint32_t)(parts - 1);
                if (s_last) p.arrivals[bh] = 0;   // for the next launch
            }
            __syncthreads();
            if (s_last && MANY) {
                // one row: a group of D / 4 threads takes every GROUPS-th piece, eight loads in flight, and the groups' states meet in shared memory
                __threadfence();
                constexpr int LANES = D / 4, GROUPS = THREADS / LANES;
                const int group = threadIdx.x / LANES, col = threadIdx.x % LANES * 4;
                float M = -INFINITY, L = 0.f;
                float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int i0 = group; i0 < parts; i0 += 8 * GROUPS) {
                    float2 ml[8];
                    float4 oi[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int i = i0 + k * GROUPS;
                        ml[k] = make_float2(-INFINITY, 0.f);
                        oi[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (i >= parts) continue;
                        const size_t at = (size_t)(slot0 + i) * C::ROWS;
                        ml[k] = __ldcg(reinterpret_cast<const float2*>(p.ws_ml + at * 2));
                        oi[k] = __ldcg(reinterpret_cast<const float4*>(p.ws_o + at * D + col));
                    }
                    float M2 = M;
#pragma unroll
                    for (int k = 0; k < 8; k++) M2 = fmaxf(M2, ml[k].x);
                    if (M2 == -INFINITY) continue;
                    const float f = ex2f(M - M2);
                    L *= f;
                    O.x *= f; O.y *= f; O.z *= f; O.w *= f;
#pragma unroll
                    for (int k = 0; k < 8; k++) fold(L, O, ml[k].y, oi[k], ex2f(ml[k].x - M2));
                    M = M2;
                }
                float(*const rows)[C::PITCH] = &s_o[0][0];   // GROUPS of them
                *reinterpret_cast<float4*>(&rows[group][col]) = O;
                if (col == 0) {
                    s_m[0][group] = M;
                    s_l[0][group] = L;
                }
                __syncthreads();
                if (group == 0) {
                    float top = -INFINITY;
#pragma unroll
                    for (int i = 0; i < GROUPS; i++) top = fmaxf(top, s_m[0][i]);
                    L = 0.f;
                    O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int i = 0; i < GROUPS; i++)
                        fold(L, O, s_l[0][i], *reinterpret_cast<const float4*>(&rows[i][col]), s_m[0][i] == -INFINITY ? 0.f : ex2f(s_m[0][i] - top));
                    store_out<D>(p, (size_t)b * p.hq + kvh, col, top, L, O, vds);
                }
            } else if (s_last) {
                __threadfence();
                for (int idx = threadIdx.x; idx < p.group * (D / 4); idx += THREADS) {
                    const int row = idx / (D / 4), col = idx % (D / 4) * 4;
                    float M = -INFINITY, L = 0.f;
                    float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int i0 = 0; i0 < parts; i0 += 8) {   // eight pieces' loads in flight
                        float2 ml[8];
                        float4 oi[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const int i = i0 + k;
                            ml[k] = make_float2(-INFINITY, 0.f);
                            oi[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (i >= parts) continue;
                            const size_t at = (size_t)(i == 0 ? slot0 : slot0 + 1 + (i - 1) * slot_step) * C::ROWS + row;
                            ml[k] = __ldcg(reinterpret_cast<const float2*>(p.ws_ml + at * 2));
                            oi[k] = __ldcg(reinterpret_cast<const float4*>(p.ws_o + at * D + col));
                        }
                        float M2 = M;
#pragma unroll
                        for (int k = 0; k < 8; k++) M2 = fmaxf(M2, ml[k].x);
                        if (M2 == -INFINITY) continue;
                        const float f = ex2f(M - M2);
                        L *= f;
                        O.x *= f; O.y *= f; O.z *= f; O.w *= f;
#pragma unroll
                        for (int k = 0; k < 8; k++) fold(L, O, ml[k].y, oi[k], ex2f(ml[k].x - M2));
                        M = M2;
                    }
                    store_out<D>(p, ((size_t)b * p.hq + (size_t)kvh * p.group + row), col, M, L, O, vds);
                }
            }
        } else {
            __syncthreads();   // the merge buffer is free again
        }
        if (!more) break;
        seg = s_next[warp];
        __syncwarp();
    }
}

int num_sms_of_current_device() {
    static int cached[64];   // 0 = not asked yet; every thread would store the same value
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess) return sms;
    if (dev >= 0 && dev < 64 && cached[dev]) return cached[dev];
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (dev >= 0 && dev < 64) cached[dev] = sms;
    return sms;
}

// A kernel and not a memset node: in a graph the decode kernel is then launched behind it before it has drained (one sequence of
// 32 heads and 100 keys: 8.8 us a captured call with the node).
__global__ void clear_words_kernel(uint32_t* w, uint32_t n) {
    pdl_wait();
    pdl_trigger();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) w[i] = 0;
}

// Kernels whose splits are a cluster: [paged][head dim 128]
using DecodeKernel = void (*)(const DecodeParams);
DecodeKernel cluster_kernel(int hd, bool paged) {
    if (hd == 64) return paged ? fa_decode_kernel<64, 1, false, true, true, false, true> : fa_decode_kernel<64, 1, false, true, false, false, true>;
    return paged ? fa_decode_kernel<128, 1, false, true, true, false, true> : fa_decode_kernel<128, 1, false, true, false, false, true>;
}
cudaLaunchConfig_t cluster_config(cudaLaunchAttribute* attr, int grid, int size, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(THREADS);
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}
// Clusters of each size that are resident at once on the current device (the least of the kernels'; asked once per device)
struct ClusterFit {
    int n[MAX_CLUSTER + 1] = {};
};
const ClusterFit& cluster_fit() {
    static ClusterFit known[64], none;
    static std::once_flag asked[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return none;
    std::call_once(asked[dev], [&] {
        ClusterFit f;
        for (int size = 2; size <= MAX_CLUSTER; size++) {
            int least = 1 << 30;
            for (int k = 0; k < 4; k++) {
                const DecodeKernel kernel = cluster_kernel(k & 1 ? 128 : 64, k & 2);
                cudaLaunchAttribute attr[2];
                cudaLaunchConfig_t cfg = cluster_config(attr, size, size, nullptr);
                cfg.numAttrs = 1;
                int n = 0;
                if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                    cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
                    (void)cudaGetLastError();
                    n = 0;
                }
                least = n < least ? n : least;
            }
            f.n[size] = least;
        }
        known[dev] = f;
    });
    return known[dev];
}

struct Layout {
    int plan, splits, grid, rows;
    bool streams, wide;
    int cluster;   // 0: none
    bool cuts() const { return plan != SPLITS || (splits > 1 && !cluster); }   // whether the pieces of a pair meet in a workspace
};
// One query head per kv head keeps the streams: fixed splits while the pairs leave room for them, else a CTA per pair, which
// the hardware hands out as CTAs end, so uneven lengths balance by themselves.  (The freely cut line, with a CTA taking up the
// running maxima of the one before it, was 10 to 30 % faster where all sequences are equally long and the pairs fill the
// SMs badly, and up to twice as slow for short or very uneven ones: 24 sequences of 32 heads of 128, lengths random up to
// 2048, 100 us against 56, 64 of up to 4160 255 against 205.)
//
// Wide steps pay once there is something to stream (from 2048 keys on; 300 keys of 64 x 32 pairs 51 us against 47), for head
// dim 128 (64 takes 256 keys a step: up to 1.4 times as slow on short sequences in a long cache), and unless the fewer
// CTAs they leave resident need more rounds than that (keys of equal length, 4160 of them: 80 x 16 pairs, 3 rounds of 444
// against 3 of 592, 221 us against 262; 30 x 32 pairs, 3 rounds against 2, 202 against 186).
//
// Groups take the freely cut line, which balances best (24 sequences of 3000 to 6000 keys, 8 kv heads: 45 us against 70 with
// fixed splits and a merging kernel).  But each piece of a pair costs some 5 us of latency that nothing hides, so once the
// pairs nearly fill the SMs (four fifths of the resident CTAs) a CTA per pair is faster for short sequences, and with several
// pairs to a CTA for long ones too.  8 kv heads of 64 / of 128, lengths random up to the span, line against CTA per pair: 64
// sequences of 1000 30 against 13 us / 32 against 20, 400 of 300 133 against 30 / 145 against 44, 400 of 4160 264 against 165 /
// 392 against 306; but 64 of 8256 74 against 72 / 114 against 131.  Groups of 9 to 16 have fewer CTAs resident, so "several" is
// one and a half there, and short sequences take narrow steps, which leave room for more (300 sequences of 64 keys, 16 heads on
// one kv head of 64: 9.2 against 7 us; 500 of 1000 on one of 128 the other way, 39 against 62).  Last, a line has to have no more chunks than an int
// counts (a paged cache whose capacity is far above what it holds).
Layout layout_of(int batch, int q_heads, int kv_heads, int head_dim, int span) {
    Layout x;
    const int group = q_heads / kv_heads, sms = num_sms_of_current_device();
    x.rows = group <= 8 ? 8 : 16;
    x.streams = group == 1;
    const long long pairs = (long long)batch * kv_heads, chunks = ((long long)span + CHUNK - 1) / CHUNK;
    const long long narrow = (long long)ctas_per_sm(head_dim, 1, false) * sms, wide = (long long)ctas_per_sm(head_dim, x.rows / 8, true) * sms;
    x.splits = 1;
    x.cluster = 0;
    x.wide = !x.streams;
    if (x.streams && pairs <= narrow) {
        long long splits = narrow / pairs;
        if (splits > chunks) splits = chunks;
        if (splits > 64) splits = 64;
        x.splits = splits < 1 ? 1 : (int)splits;
        // Splits in clusters, of up to eight CTAs or of sizes that only some GPUs place: the largest that has room (112 pairs of 900 keys in as many
        // clusters of 5 as fit 12.3 us, workspace 10.8), and 8 rather than more.  A CTA takes several splits in turn, which must not cost more
        // chunks in turn than the workspace's merge costs time.
        // Us, workspace / cluster: 32 pairs of 1000 keys 6.6 / 5.7 (of 64 6.1 / 4.5), of 100 5.0 / 4.1; 16 of 2000 7.4 / 6.6; 96 of 500 7.9 / 6.8; 112 of 900 10.7 /
        // 9.8; but where a split has several chunks and a CTA would take two, 32 of 2000 9.0 / 9.4, 192 of 500 9.7 / 12.4.  Near what fits clusters wait for room: 40 of 2200
        // in 13s of 38 that fit 9.8 / 12.0, 172 of 900 in 3s of 187 12.8 / 12.5 (of 64 10.4 / 13.5), 184 13.0 / 17.2 (10.5 / 14.0), 164 12.7 / 11.8 (10.3 / 9.6); pairs of CTAs do not (all 296: of 500
        // keys 11.9 / 11.1), nor 4s up to 132 of 142 (11.4 / 10.4).  The lengths are on the device: sequences that fill an eighth of the cache or less pay a cluster's start for nothing, 32 of 28 of 64
        // in 226 2.9 / 3.3, 64 of 60 in 500 3.5 / 3.75, 288 of up to 90 in 718 4.4 / 5.0.
        // Fewer than 16 pairs keep the workspace, which is not the faster one there (8 pairs of 1000 keys 5.6 / 4.4): the line is not where clusters stop paying, but
        // calls of eight pairs are what the tests of scratch and of captured calls take for a cut pair in the workspace (tests/test_fa_scratch_gpu.py).
        const ClusterFit& fit = cluster_fit();
        const long long each = (chunks + x.splits - 1) / x.splits, used = each ? (chunks + each - 1) / each : 0;
        auto placed = [&](long long n) { return n > PORTABLE_CLUSTER ? 8 * pairs <= 7 * fit.n[n] : n > 3 ? 16 * pairs <= 15 * fit.n[n] : n == 3 ? 9 * pairs <= 8 * fit.n[n] : pairs <= fit.n[n]; };
        auto steps_of = [&](long long n) { return (used + n - 1) / n * each; };
        long long size = used < MAX_CLUSTER ? used : MAX_CLUSTER;
        while (size > 1 && !placed(size)) size--;
        if (size > PORTABLE_CLUSTER && placed(PORTABLE_CLUSTER) && steps_of(PORTABLE_CLUSTER) <= steps_of(size) + 1) size = PORTABLE_CLUSTER;
        while (size > PORTABLE_CLUSTER && steps_of(size - 1) == steps_of(size)) size--;
        // (a cache is rarely full to its last split: 64 pairs of 1000 keys in a cache of 1064 have 8 of 9, 8.4 / 7.6)
        if (pairs >= 16 && size > 1 && each <= LONGEST_SPLIT && (steps_of(size) <= (each == 1 ? 3 : each + 1) || (each <= 2 && used <= size + size / 8))) x.cluster = (int)size;
        x.plan = SPLITS;
        x.grid = (int)(pairs * (x.cluster ? x.cluster : x.splits));
    } else if (x.streams || 2 * pairs >= (x.rows == 8 ? 6 : 3) * wide || (chunks <= 32 && 5 * pairs >= 4 * wide) || pairs * chunks > 0x7fffffffLL) {
        x.plan = SPLITS;
        x.grid = (int)pairs;
        if (x.rows == 16) x.wide = chunks > (head_dim == 64 ? 16 : 8);
        if (x.streams) x.wide = head_dim == 128 && chunks >= 32 && (pairs + wide - 1) / wide * wide <= (pairs + narrow - 1) / narrow * narrow;
    } else {
        x.plan = LINE;
        const long long units = pairs * chunks;
        x.grid = (int)(units < wide ? (units > 0 ? units : 1) : wide);
    }
    return x;
}

}  // namespace

size_t decode_workspace_bytes(int batch, int q_heads, int kv_heads, int head_dim, int span) {
    const Layout x = layout_of(batch, q_heads, kv_heads, head_dim, span);
    return x.cuts() ? (size_t)x.grid * x.rows * 2 * (head_dim + 2) * sizeof(float) : 0;
}
size_t decode_arrival_count(int batch, int q_heads, int kv_heads, int head_dim, int span) {
    return layout_of(batch, q_heads, kv_heads, head_dim, span).cuts() ? (size_t)batch * kv_heads : 0;
}

cudaError_t launch_decode(const DecodeArgs& a) {
    const int span = decode_span(a);
    if ((long long)a.batch * a.kv_heads > 0x7fffffffLL) return cudaErrorInvalidValue;
    const Layout x = layout_of(a.batch, a.q_heads, a.kv_heads, a.hd, span);
    if (x.cuts() && (!a.workspace || !a.arrivals)) return cudaErrorInvalidValue;
    DecodeParams p;
    p.q = static_cast<const uint8_t*>(a.q);
    p.k = static_cast<const uint8_t*>(a.k_cache);
    p.v = static_cast<const uint8_t*>(a.v_cache);
    p.o = static_cast<__half*>(a.o);
    p.lse = a.lse;
    p.seq_lens = a.seq_lens;
    p.batch = a.batch; p.hq = a.q_heads; p.hkv = a.kv_heads; p.group = a.q_heads / a.kv_heads;
    p.s_max = a.s_max; p.seq_len = a.seq_len;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.v_descale = a.v_descale;
    p.sq = a.scale_q_dev; p.sk = a.scale_k_dev; p.sv = a.scale_v_dev;
    p.plan = x.plan; p.splits = x.splits; p.cluster = x.cluster; p.hints = !a.behind_clear;
    p.chunks_per_split = (int)((((long long)span + CHUNK - 1) / CHUNK + x.splits - 1) / x.splits);
    p.block_table = a.block_table;
    p.page_mul = p.page_shr = 0;
    if (a.block_table) {   // page_size >= 64; exact for numerators below 2^31, and the multiplier fits 32 bits
        uint32_t lg = 0;
        while ((1ull << lg) < (unsigned)a.page_size) lg++;
        p.page_mul = (uint32_t)(((1ull << (31 + lg)) + a.page_size - 1) / a.page_size);
        p.page_shr = lg;   // umulhi is >> 32: >> (31 + lg) is >> (lg - 1) more
    }
    p.page_size = a.page_size; p.max_pages = a.max_pages; p.num_pages = a.num_pages;
    p.ws_o = static_cast<float*>(a.workspace);
    p.ws_ml = p.ws_o + (size_t)x.grid * 2 * x.rows * a.hd;
    p.arrivals = a.arrivals;
    if (x.cluster) {
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t cfg = cluster_config(attr, x.grid, x.cluster, a.stream);
        return cudaLaunchKernelEx(&cfg, cluster_kernel(a.hd, a.block_table != nullptr), p);
    }
    auto run = [&](auto contiguous, auto paged) { return launch_pdl(a.block_table ? paged : contiguous, x.grid, THREADS, 0, a.stream, p); };
    if (x.streams && x.splits > FEW_SPLITS)
        return a.hd == 64 ? run(fa_decode_kernel<64, 1, false, true, false, true>, fa_decode_kernel<64, 1, false, true, true, true>)
                          : run(fa_decode_kernel<128, 1, false, true, false, true>, fa_decode_kernel<128, 1, false, true, true, true>);
#define KERNEL(D, NQ, WIDE, STREAMS) run(fa_decode_kernel<D, NQ, WIDE, STREAMS, false>, fa_decode_kernel<D, NQ, WIDE, STREAMS, true>)
    if (x.streams) return a.hd == 64 ? KERNEL(64, 1, false, true) : x.wide ? KERNEL(128, 1, true, true) : KERNEL(128, 1, false, true);
    if (x.rows == 8) return a.hd == 64 ? KERNEL(64, 1, true, false) : KERNEL(128, 1, true, false);
    if (x.wide) return a.hd == 64 ? KERNEL(64, 2, true, false) : KERNEL(128, 2, true, false);
    return a.hd == 64 ? KERNEL(64, 2, false, false) : KERNEL(128, 2, false, false);
#undef KERNEL
}

cudaError_t launch_clear_words(uint32_t* w, size_t n, cudaStream_t stream) {
    if (n > 0xffffffffu) return cudaErrorInvalidValue;
    const unsigned blocks = (unsigned)((n + 1023) / 1024 < 64 ? (n + 1023) / 1024 : 64);
    return launch_pdl(clear_words_kernel, dim3(blocks), dim3(256), 0, stream, w, (uint32_t)n);
}

}  // namespace fa_sm100
