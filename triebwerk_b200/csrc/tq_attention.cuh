// GQA decode attention over the TurboQuant packed cache, sm_100a.
//
// Replaces turbo_gqa_attention_batch_kernel / turbo_gqa_attention_kernel (reference
// engine/kernels.cu:1641-1870).  Same mathematics -- score = (q_rot . centroids[codesK]) * k_norm / sqrt(128),
// softmax over positions 0..pos with denominator + 1e-8, V accumulated in rotated space as
// sum w * v_norm * centroids[codesV], one multiplication by R^T per head -- evaluated as a split-K
// online-softmax (flash-decoding) so that no score ever goes to global memory.
//
// Decomposition
//   * The (sequence, 32-token tile) pairs of the whole batch form one flat list (lengths come from the
//     device-side positions, so the launch geometry never depends on them and the launch can be captured in
//     a CUDA graph).  The list is cut into equal contiguous slices, one per WORKER; a CTA holds two workers
//     (16 warps on the SM for latency hiding), each a group of Hkv warps with its own named barrier.  Every SM
//     gets the same number of bytes whatever the mix of sequence lengths.
//   * Inside a worker warp w owns KV head w and all of its query heads (2 for Qwen3-0.6B, 4 for Qwen3-8B):
//     every cache byte is fetched from HBM once, not once per query head as in the reference.
//   * A worker streams its tiles through a ring of shared-memory stages filled by the TMA engine (no multicast):
//     the K codes of 32 token rows arrive as [32 rows][128 B] boxes (two heads' bytes per row, four boxes for eight
//     heads) through a 2-D tensor map with the 128-byte swizzle, likewise V, and the fp16 norms as two small
//     contiguous bulk copies; completion on one mbarrier per stage.  (An optional cp.async.bulk.prefetch.L2 of tiles
//     further ahead exists, TQ_ATTN_L2_AHEAD; it is off by default because it did not pay on B200.)  The last warp of the
//     worker to finish a stage (one shared-memory atomic per warp and tile) re-arms it: nobody waits for a slower
//     warp.  In the layer form and in whole steps of enough tiles a copy warp does, which the warps tell through a barrier per part: without the list's
//     cursor, the atomics and the fences 664 -> 630 warp instructions per warp and tile (28 layers of 64 x 4096 tokens
//     2007 -> 1863 us, ragged 128 sequences 2319 -> 2135; shared memory 74 % busy, issue slots 64 %, and
//     with two stages the time from hand-back to copy counts: a thread that polls and sleeps 64 ns, 4 layers 2-bit 64 x 3000
//     198 us, one suspended in the wait 180).  With the swizzle, and with the eight tokens of a score block taken in the order 0,5,2,7,4,1,6,3, every
//     16-, 8- and 4-byte read of packed codes is free of bank conflicts.
//   * Codes are turned into fp16 centroids one BYTE at a time (2 codes for 4-bit, 4 for 2-bit) through a
//     shared-memory table with one private column per lane (bank-conflict free); the table sits at shared
//     address 0x10000 so that a single PRMT builds the lookup address from the packed word.
//   * The dot products run on the tensor cores with warp-level mma.sync.m16n8k16 (fp16 in, fp32 accumulate):
//     scores as K(16 tokens x 16 coordinates) * Q^T(16 x 8 columns), and the value sum in transposed form
//     V^T(16 coords x 16 tokens) * P^T(16 tokens x 8 columns); the token pairs the V^T fragment needs are
//     formed by interleaving the nibbles of two tokens' words BEFORE the table lookup.  With eight KV heads a head
//     has two columns (PAIR): a lane's scores are of one head, half the exponentials, and 580 instead of 622 warp
//     instructions per warp and 4-bit tile (28 layers of 64 x 4096 tokens 1902 -> 1874 us).
//   * 2-bit scores need no table there (PLANES): a centroid is affine in its code's two bits, so every bit of the code bytes,
//     masked in place, is an operand of mma.sync.m16n8k32 (u8 x s8) against 16-bit fixed-point queries; one mask per four
//     codes and plane, as many products as before.  The table look-ups of K were 64 of a tile's 176 shared-memory wavefronts: that
//     pipe 67 -> 49 % busy, 550 -> 484 warp instructions, 8 layers of 64 x 4096 tokens (32/8 heads) 456 -> 423 us in the whole-step form.
//     What is left is instruction issue (65 %) and the ALU (56 %).  V keeps the table: its operand is the weights, whose
//     range fixed point does not cover.  Scalar fp32 FMAs cannot
//     keep up with HBM3e on this path: 512 FMAs per 132-byte row is more than the SMs can issue.
//   * A worker that finishes its part of a sequence writes (acc[128], m, l) per query head to the workspace.  A kernel behind
//     this one merges the parts and multiplies by R^T on the tensor cores (normalised accumulators split into fp16
//     high + low parts as the A operand, R^T as B); in MODE 0 the last worker to arrive does, found by a ticket: a single
//     atomicAdd, nobody spins on anybody.
//   * Layer form (MODE 1): append and query rotation in a launch before (tq_layer_prep.cuh), merge in one behind, so that a tile loop with
//     copy warps and nothing else is left, which starts with table and ring ready.  With all of it in one launch a tile took
//     1.76 us for 1.47 and the first one began 4 us later: 32 x 8192 tokens 2-bit, 32/8 heads 69.6 -> 57.9 us a layer (issue
//     slots 51 -> 64 % busy, DRAM 24 -> 32 %), 4-bit 32 x 4096 49.8 -> 41.8, 128 x 64 18.7 -> 17.0.
#pragma once

#include <type_traits>

#include "tq_common.cuh"

namespace tq {

constexpr uint32_t LUT_ABS = 0x10000u;        // absolute shared address of the byte -> centroid table
constexpr uint32_t REGION_B_ABS = 0x20000u;   // more stage blocks live above the table
constexpr int ATTN_MAX_HEADS = 32;
constexpr size_t ATTN_DYN_SMEM = 226 * 1024;  // requested dynamic shared memory
constexpr int ATTN_GROUPS = 2;                // workers per CTA
constexpr int ATTN_MAX_STAGES = 4;            // shared-memory stages per worker (as many as fit, at most this)
constexpr int ATTN_L2_AHEAD = 0;              // tiles prefetched into L2 beyond the ring; 0 = off (measured: no gain on B200)
constexpr int MERGE_ROW = 136;                // halves per row of the merge A-operand (padded: conflict-free)

struct AttnParams {
    const uint8_t* ck;         // packed K codes [rows][kvp]
    const uint8_t* cv;
    const __half* kn;          // norms [rows][Hkv]
    const __half* vn;
    const float* q_rot;        // [G][H][128], pre-scaled by log2(e)/sqrt(128)
    const __half* rotation_t;  // R transposed: rotation_t[d][k] = R[k][d]
    __half* out;               // [G][q_dim]
    float* out_f32;            // optional [G][H][128]: the same results before the rounding to fp16 (error reports), or null
    const int* positions;      // device [G] or null
    const long long* row_base;
    // Shared prefixes (optional, both null otherwise): the first prefix_tiles[g] tiles of sequence g are read from the rows
    // prefix_base[g] + 32 * tile (another sequence's slot, which holds the common prompt once); every later tile j from
    // row_base[g] + 32 * j as usual -- row_base[g] then already has the prefix length subtracted.
    const long long* prefix_base;
    const int* prefix_tiles;
    const int* tile_start;     // [G+1]
    const int* worker_g;       // first sequence of each worker's slice, or null (then it is searched for)
    int* tickets;              // [G]
    float* partials;           // [workers+G][H][PART_STRIDE]
    int* status;
    long long total_rows;      // rows of the cache arrays (copies are clipped to it)
    int pos_value;
    int max_seq_len;
    int G, H, Hkv, q_dim;
    // layer form (MODE 1): after layer_prep_kernel (tq_layer_prep.cuh), whose predecessors have finished when this kernel starts:
    // positions and cache rows are read before that launch has, but for the tiles it writes the new tokens to
    int appends;               // 1: layer_prep_kernel appends, to the last tile of every sequence
    const float* q_rot32;      // rotated queries as fp32 [G][H][128] instead of q_rot16 (2-bit with eight KV heads, for the planes), coordinate
                               // 32 a + 4 b + c at 16 b + 4 a + c: what the four lanes of a head load together lies side by side (in the
                               // order of the coordinates their loads met on one bank: 32 x 8192, 32 heads, 58.9 us a layer)
    int l2_ahead;              // tiles prefetched into L2 beyond the shared-memory ring
    // whole-step form (MODE 2): ONE launch streams the layers [layer0, layer0 + n_layers) back to back -- every worker
    // walks its slice of the tile list once per layer, its ring of stages never drains in between -- and only PUBLISHES its
    // split-K partials, per layer; merge_partials_kernel finishes the step.
    // ck/cv/kn/vn are the arrays of layer0, the tensor maps have the layer as their outermost coordinate.
    int layer0, n_layers;
    long long norm_layer_stride;   // halves between consecutive layers' norm arrays
    long long part_layer_stride;   // floats between consecutive layers' partial areas
    int* table_out;                // [G + 4]: the tile table, then {workers taking part, total tiles}, for the merge kernel
    const __half* q_rot16;         // layer and whole-step form: pre-rotated, pre-scaled fp16 queries of layer0, [layers][G][H][128]
                                   // (layer_prep_kernel, rotate_queries_kernel); a sequence's block reaches shared memory by one bulk copy
#ifdef TQ_TIMING_SWITCHES
    int debug;                 // timing-experiment builds only: bit 0 = skip the math, bit 1 = skip the loads, ... (results are then wrong)
    unsigned long long* stamps;  // timing-experiment builds only: [8] summed clock deltas of the tile loop's sections
#endif
};

// Switches that leave parts of the kernel out, for timing experiments.  They exist only in builds made with
// -DTQ_TIMING_SWITCHES; in the library they are the constant false and the compiler removes the branches.
#ifdef TQ_TIMING_SWITCHES
#define TQ_DBG(bit) ((p.debug & (bit)) != 0)
#define TQ_DBG_FACTOR (p.debug >> 8)
#define TQ_STAMP(i) do { const long long _t = clock64(); stamp_acc[i] += _t - stamp_last; stamp_last = _t; } while (0)
#else
#define TQ_DBG(bit) false
#define TQ_DBG_FACTOR 0
#define TQ_STAMP(i) do { } while (0)
#endif

template <int BITS>
struct AttnGeom {
    static constexpr int BPH = (BITS == 4) ? 64 : 32;  // code bytes per head per token
};

// Region A (below the table): barriers, control words, merge operands, then stage blocks.
struct RegionA {
    static constexpr uint32_t BAR_OFF = 0;       // per group: full[ATTN_MAX_STAGES] mbarriers (8 B each)
    static constexpr uint32_t CNT_OFF = 128;     // per group: done-counters, one u32 per stage
    static constexpr uint32_t CTRL_OFF = 256;    // one word per group
    static constexpr uint32_t MERGE_OFF = 512;   // per group: hi + lo [16][MERGE_ROW] halves
    static constexpr uint32_t MERGE_GROUP_BYTES = 2 * 16 * MERGE_ROW * 2;  // 8704
    static constexpr uint32_t BLOCKS_OFF = MERGE_OFF + ATTN_GROUPS * MERGE_GROUP_BYTES;
    static constexpr uint32_t Q32_GROUP_BYTES = ATTN_MAX_HEADS * HEAD_DIM * 4;  // in the merge operands' place: a sequence's fp32 queries
    // layer and whole-step form, `area` bytes per group in that place: tile table of the launch, then the stage blocks
    __host__ __device__ static constexpr uint32_t scan_off(uint32_t area) { return MERGE_OFF + ATTN_GROUPS * area; }   // 32 ints of scan scratch
    __host__ __device__ static constexpr uint32_t ts_off(uint32_t area) { return scan_off(area) + 128; }               // tile_start[G + 1], G <= FUSED_MAX_G
    __host__ __device__ static constexpr uint32_t blocks_off(uint32_t area) { return ts_off(area) + 4096; }
};
constexpr int FUSED_MAX_G = 1023;

__device__ __forceinline__ void group_barrier(int group, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(nthreads) : "memory");
}

__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t atom_add_shared(uint32_t addr, uint32_t v) {
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
    return old;
}
// Loads whose ordering is carried by data dependence (their address derives from a value produced after the
// barrier wait), so the compiler may schedule them freely among the arithmetic of a tile.
__device__ __forceinline__ uint32_t ldsp32(uint32_t addr) {
    uint32_t r;
    asm("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint2 ldsp64(uint32_t addr) {
    uint2 r;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint4 ldsp128(uint32_t addr) {
    uint4 r;
    asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
    return r;
}
// The same loads kept in program order relative to barriers and other volatile accesses (staging buffers that are
// rewritten between uses).
__device__ __forceinline__ uint2 ldsv64(uint32_t addr) {
    uint2 r;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(addr));
    return r;
}
__device__ __forceinline__ uint4 ldsv128(uint32_t addr) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
    return r;
}
__device__ __forceinline__ float ldsv_h2f(uint32_t addr) {  // one fp16 from shared memory as float, kept in program order
    unsigned short h;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(addr));
    return __half2float(__ushort_as_half(h));
}
// Transpose of an 8 x 8 matrix of 16-bit elements held by the warp, one 32-bit register per lane: lane (r, c) holds
// the elements (row r, columns 2c and 2c + 1) before and after.
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
// Sixteen bytes from global memory, requested where they stand (a later griddepcontrol.wait does not pull the load behind it).
__device__ __forceinline__ uint4 ldg128_now(const void* src) {
    uint4 r;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(src));
    return r;
}
// The same, and a word, past L1: for what an earlier kernel of the stream has written that is known to have finished, though this launch has
// not waited yet.
__device__ __forceinline__ uint4 ldg128_l2(const void* src) {
    uint4 r;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(src));
    return r;
}
__device__ __forceinline__ int ldg32_l2(const int* src) {
    int r;
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(r) : "l"(src));
    return r;
}
__device__ __forceinline__ float ldsp_h2f(uint32_t addr) {  // one fp16 from shared memory as float
    unsigned short h;
    asm("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(addr));
    return __half2float(__ushort_as_half(h));
}

// Split-K merge of one sequence: combines the `parts` partials (acc[128], m, l) of every query head, normalises, and
// multiplies by R^T on the tensor cores (normalised accumulators split into fp16 high + low parts as the A operand, R^T
// as B).  Run by NW warps (`head` = warp index among them) that share the named barrier `bar_group` and the staging
// area `merge_s` ([2][16][MERGE_ROW] halves of shared memory).  part0: the first part's rows, [H][PART_STRIDE]; parts
// follow each other H * PART_STRIDE floats apart.  out_row(h) / out_row_f32(h): where head h's 128 outputs go, or null.
template <int NW, typename OutRow, typename OutRowF32>
__device__ __forceinline__ void merge_sequence(const float* part0, int parts, int H, uint32_t merge_s, const __half* rotation_t,
                                               int head, int lane, int bar_group, int nthreads, OutRow out_row,
                                               OutRowF32 out_row_f32, bool rotated_out = false) {
    const int gl = lane >> 2, t4 = lane & 3;
    constexpr int RH = 2, FLIGHT = 16 / RH;  // heads per warp at a time, parts whose loads are in flight together
    for (int hb = 0; hb < H; hb += 16) {
        // ---- phase A: heads hb .. hb+15, two heads per warp at a time with all their loads in flight
        //      together: combine the parts, normalise, split into fp16 high + low, store as the A operand
        //      [16][MERGE_ROW]
        for (int hh0 = head; hh0 < 16; hh0 += RH * NW) {
            float4 a[RH];
#pragma unroll
            for (int r = 0; r < RH; ++r) a[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            const size_t pstride = (size_t)H * PART_STRIDE;
            if (parts <= FLIGHT) {
                // common case: one round trip for everything, weights afterwards
                float4 v[RH][FLIGHT];
                float2 ml[RH];
#pragma unroll
                for (int r = 0; r < RH; ++r) {
                    const int hq = hb + hh0 + r * NW;
                    const float* base = part0 + (size_t)hq * PART_STRIDE;
                    const bool on = hq < H && hh0 + r * NW < 16;
                    ml[r] = make_float2(-1e30f, 0.0f);
                    if (on && lane < parts) ml[r] = __ldcg(reinterpret_cast<const float2*>(base + lane * pstride + HEAD_DIM));
#pragma unroll
                    for (int j = 0; j < FLIGHT; ++j)
                        v[r][j] = (on && j < parts) ? __ldcg(reinterpret_cast<const float4*>(base + j * pstride) + lane)
                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int r = 0; r < RH; ++r) {
                    float M = ml[r].x;
#pragma unroll
                    for (int o = FLIGHT / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
                    M = __shfl_sync(0xffffffffu, M, 0);
                    const float e = lane < parts ? ex2_approx(ml[r].x - M) : 0.0f;
                    float Z = ml[r].y * e;
#pragma unroll
                    for (int o = FLIGHT / 2; o > 0; o >>= 1) Z += __shfl_xor_sync(0xffffffffu, Z, o);
                    Z = __shfl_sync(0xffffffffu, Z, 0);
                    const float sc = e / (Z + 1e-8f);
#pragma unroll
                    for (int j = 0; j < FLIGHT; ++j) {
                        const float wj = __shfl_sync(0xffffffffu, sc, j);
                        a[r].x = fmaf(wj, v[r][j].x, a[r].x); a[r].y = fmaf(wj, v[r][j].y, a[r].y);
                        a[r].z = fmaf(wj, v[r][j].z, a[r].z); a[r].w = fmaf(wj, v[r][j].w, a[r].w);
                    }
                }
            } else {
                // many parts: one round trip for all (max, sum) pairs, then the vectors 16 at a time
#pragma unroll
                for (int r = 0; r < RH; ++r) {
                    const int hq = hb + hh0 + r * NW;
                    if (hq >= H || hh0 + r * NW >= 16) continue;
                    const float* base = part0 + (size_t)hq * PART_STRIDE;
                    float M = -1e30f, Z = 0.0f, m0 = -1e30f;  // m0: the max of part `lane` (parts 0 .. 31)
                    for (int j0 = 0; j0 < parts; j0 += 32) {
                        float2 t = make_float2(-1e30f, 0.0f);
                        if (j0 + lane < parts) t = __ldcg(reinterpret_cast<const float2*>(base + (j0 + lane) * pstride + HEAD_DIM));
                        if (j0 == 0) m0 = t.x;
                        const float Mn = fmaxf(M, t.x);
                        Z = Z * ex2_approx(M - Mn) + t.y * ex2_approx(t.x - Mn);
                        M = Mn;
                    }
                    float Mw = M;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) Mw = fmaxf(Mw, __shfl_xor_sync(0xffffffffu, Mw, o));
                    Z *= ex2_approx(M - Mw);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) Z += __shfl_xor_sync(0xffffffffu, Z, o);
                    const float inv = 1.0f / (Z + 1e-8f);
                    for (int j0 = 0; j0 < parts; j0 += 32) {
                        float mj = m0;
                        if (j0 > 0) mj = j0 + lane < parts ? __ldcg(base + (j0 + lane) * pstride + HEAD_DIM) : -1e30f;
                        const float sc = j0 + lane < parts ? ex2_approx(mj - Mw) * inv : 0.0f;
#pragma unroll 1
                        for (int j1 = j0; j1 < parts && j1 < j0 + 32; j1 += 16) {
                            float4 v[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                v[j] = j1 + j < parts ? __ldcg(reinterpret_cast<const float4*>(base + (j1 + j) * pstride) + lane)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const float wj = __shfl_sync(0xffffffffu, sc, (j1 - j0) + j);
                                a[r].x = fmaf(wj, v[j].x, a[r].x); a[r].y = fmaf(wj, v[j].y, a[r].y);
                                a[r].z = fmaf(wj, v[j].z, a[r].z); a[r].w = fmaf(wj, v[j].w, a[r].w);
                            }
                        }
                    }
                }
            }
            if (rotated_out) {
                // the consumer's weights carry R^T (tq_fold_rotation_into_projection): the normalised sums leave as they are
#pragma unroll
                for (int r = 0; r < RH; ++r) {
                    const int hh = hh0 + r * NW;
                    if (hh >= 16) continue;
                    if (__half* o = out_row(hb + hh)) {
                        const __half2 h01 = __floats2half2_rn(a[r].x, a[r].y), h23 = __floats2half2_rn(a[r].z, a[r].w);
                        *reinterpret_cast<uint2*>(o + 4 * lane) = make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
                    }
                    if (float* o = out_row_f32(hb + hh)) *reinterpret_cast<float4*>(o + 4 * lane) = a[r];
                }
                continue;
            }
#pragma unroll
            for (int r = 0; r < RH; ++r) {
                const int hh = hh0 + r * NW;
                if (hh >= 16) continue;
                __half2 h01 = __floats2half2_rn(a[r].x, a[r].y), h23 = __floats2half2_rn(a[r].z, a[r].w);
                float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
                const uint32_t dst = merge_s + (uint32_t)(hh * MERGE_ROW + 4 * lane) * 2u;
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst), "r"(*reinterpret_cast<uint32_t*>(&h01)),
                             "r"(*reinterpret_cast<uint32_t*>(&h23)) : "memory");
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst + 16u * MERGE_ROW * 2u),
                             "r"(pack_half2(a[r].x - f01.x, a[r].y - f01.y)), "r"(pack_half2(a[r].z - f23.x, a[r].w - f23.y)) : "memory");
            }
        }
        if (rotated_out) continue;
        // ---- phase B: out[h][d] = sum_k a[h][k] * R[k][d]  ==  A(16 x 128) * B with B[k][n=d] = rotation_t[d][k].
        //      Two column blocks of 8 per warp and pass; their B fragments are fetched before the barrier so that
        //      the round trip overlaps the other warps' phase A.
        for (int nb0 = head; nb0 < 16; nb0 += RH * NW) {
            uint32_t bfrag[RH][8][2];
#pragma unroll
            for (int i = 0; i < RH; ++i) {
                const int nb = nb0 + i * NW;
                const __half* rt = rotation_t + (size_t)(8 * (nb < 16 ? nb : 0) + gl) * HEAD_DIM + 2 * t4;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    bfrag[i][j][0] = __ldg(reinterpret_cast<const unsigned int*>(rt + 16 * j));
                    bfrag[i][j][1] = __ldg(reinterpret_cast<const unsigned int*>(rt + 16 * j + 8));
                }
            }
            if (nb0 == head) group_barrier(bar_group, nthreads);  // phase A of every warp is in shared memory
#pragma unroll
            for (int i = 0; i < RH; ++i) {
                const int nb = nb0 + i * NW;
                if (nb >= 16) continue;
                float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t r0 = merge_s + (uint32_t)(gl * MERGE_ROW + 16 * j + 2 * t4) * 2u;
                    const uint32_t r8 = r0 + 8u * MERGE_ROW * 2u;
                    const uint32_t lo_off = 16u * MERGE_ROW * 2u;
                    mma16816(c, lds32(r0), lds32(r8), lds32(r0 + 16u), lds32(r8 + 16u), bfrag[i][j][0], bfrag[i][j][1]);
                    mma16816(c, lds32(r0 + lo_off), lds32(r8 + lo_off), lds32(r0 + lo_off + 16u), lds32(r8 + lo_off + 16u),
                             bfrag[i][j][0], bfrag[i][j][1]);
                }
                const int d = 8 * nb + 2 * t4;
                if (__half* o = out_row(hb + gl))
                    *reinterpret_cast<__half2*>(o + d) = __floats2half2_rn(c[0], c[1]);
                if (__half* o = out_row(hb + gl + 8))
                    *reinterpret_cast<__half2*>(o + d) = __floats2half2_rn(c[2], c[3]);
                if (float* o = out_row_f32(hb + gl)) *reinterpret_cast<float2*>(o + d) = make_float2(c[0], c[1]);
                if (float* o = out_row_f32(hb + gl + 8)) *reinterpret_cast<float2*>(o + d) = make_float2(c[2], c[3]);
            }
        }
        group_barrier(bar_group, nthreads);  // the A operand may be overwritten (next 16 heads, next segment)
    }
}

// MODE 0: queries pre-rotated and tile table built by append_rotate_kernel, merge in the kernel.  In the other modes the kernel builds
// its table and publishes its partials, the queries are rotated and the new tokens appended already: 1: one layer, after
// layer_prep_kernel, merge_layer_kernel follows; 2: whole-step form, see AttnParams; 4: as 2 without the copy warps.
// Modes 1 and 2 have two warps more, which issue the copies of one worker each.  With 16 warps at work it is a warpgroup more:
// the launch brings 640 x 96 registers, of which the workers' warps take 112 each and the copy warps keep 32.
template <int HKV, int MODE>
constexpr int attn_threads() { return ATTN_GROUPS * 32 * HKV + (MODE == 1 || MODE == 2 ? (HKV == 8 ? 128 : 64) : 0); }
constexpr int ATTN_REGS_WORK = 112, ATTN_REGS_COPY = 32;
template <int BITS, int HKV, int MODE>
__global__ void __launch_bounds__(attn_threads<HKV, MODE>(), 1)
decode_attention_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                        const AttnParams p) {
    using Geo = AttnGeom<BITS>;
    constexpr bool LAYER = MODE == 1;
    constexpr bool PERSIST = MODE == 2 || MODE == 4;
    constexpr bool PUBLISH = LAYER || PERSIST;
    constexpr bool COPIER = MODE == 1 || MODE == 2;
    // Eight KV heads have at most four query heads each (ATTN_MAX_HEADS), half of a product's eight columns.  Head h takes the columns
    // 2 h and 2 h + 1: a lane's two score columns are ONE head, so that it has half the exponentials; in the value product the even
    // column sums the first eight tokens of a step, the odd one the other eight.
    constexpr bool PAIR = HKV == 8;
    constexpr int NE = PAIR ? 1 : 2;               // query heads per lane in the score layout
    // 2-bit: a centroid is affine in its code's two bits, so the scores need no table: every bit of the code bytes, masked in place, is
    // a plane of an integer product with 16-bit fixed-point queries (see make_planes).
    constexpr bool PLANES = PAIR && BITS == 2;
    extern __shared__ __align__(1024) uint8_t dyn_smem[];

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    constexpr int Hkv = HKV;  // compile time: row pitches, tile sizes and norm strides fold into immediates
    // lane 0 of each worker's copy warp keeps its ring filled
    const bool copier = COPIER && warp >= ATTN_GROUPS * Hkv;
    const int group = copier ? ((warp - ATTN_GROUPS * Hkv) & 1) : warp / Hkv;  // worker within the CTA
    const int head = warp - group * Hkv; // KV head of this warp
    const int gl = lane >> 2;            // mma "group id": token (K side), coordinate row (V side), head (S layout)
    const int t4 = lane & 3;             // mma "thread in group"
    const int grp = p.H / Hkv;           // query heads per KV head (<= 8)
    constexpr int gthreads = 32 * Hkv;   // threads of a worker
    const int gtid = tid - group * gthreads;
    constexpr uint32_t kvp = (uint32_t)Hkv * Geo::BPH;               // code bytes per token row (all heads)
    constexpr uint32_t code_tile = TILE_TOKENS * kvp;                // one K (or V) tile
    constexpr uint32_t norm_tile = TILE_TOKENS * (uint32_t)Hkv * 2u; // one norm tile
    // a stage starts on a 1024-byte boundary: the 128-byte swizzle of the tensor-map copies goes by the shared address
    constexpr uint32_t stage_bytes = (2u * code_tile + 2u * norm_tile + 1023u) & ~1023u;

    // ---- shared memory map (absolute shared addresses) ----
    const uint32_t dyn_base = smem_u32(dyn_smem);
    const uint32_t a_base = (dyn_base + 1023u) & ~1023u;
    constexpr bool Q_WIDE = LAYER && PLANES;  // rotated queries as fp32 (two groups' areas still leave room for three stages)
    constexpr uint32_t MERGE_AREA = Q_WIDE ? RegionA::Q32_GROUP_BYTES : RegionA::MERGE_GROUP_BYTES;
    const uint32_t blocks_a = (a_base + (PUBLISH ? RegionA::blocks_off(MERGE_AREA) : RegionA::BLOCKS_OFF) + 1023u) & ~1023u;
    const uint32_t n_a = blocks_a < LUT_ABS ? (LUT_ABS - blocks_a) / stage_bytes : 0u;
    const uint32_t dyn_end = dyn_base + (uint32_t)ATTN_DYN_SMEM;
    const uint32_t n_b = dyn_end > REGION_B_ABS ? (dyn_end - REGION_B_ABS) / stage_bytes : 0u;
    const int s_fit = (int)((n_a + n_b) / ATTN_GROUPS);
    // 4-bit: a power of two (stage index and parity are masks and shifts).  2-bit stages are half the size and three of
    // them fit where two 4-bit ones do: there the index and the parity are carried along instead.
    const int S = s_fit >= 4 ? 4 : ((BITS == 2 && s_fit == 3) ? 3 : 2);
    const int s_log = s_fit >= 4 ? 2 : 1;
    auto stage_addr = [&](int s) -> uint32_t {
        const uint32_t blk = (uint32_t)(group * S + s);
        return blk < n_a ? blocks_a + blk * stage_bytes : REGION_B_ABS + (blk - n_a) * stage_bytes;
    };
    bool layout_ok = !(blocks_a >= LUT_ABS || s_fit < 2 || dyn_end < REGION_B_ABS);
    if (!layout_ok) {
        if (tid == 0) atomicMax(p.status, ST_SMEM_LAYOUT);
        return;
    }
    // two barriers and two done-counters per stage: the K part (codes + norms) and the V part are filled, waited for
    // and handed back separately, so that a stage's K half is on its way again while its V half is still being read
    const uint32_t bar0 = a_base + RegionA::BAR_OFF + (uint32_t)group * (ATTN_MAX_STAGES * 16u);
    const uint32_t cnt0 = a_base + RegionA::CNT_OFF + (uint32_t)group * (ATTN_MAX_STAGES * 8u);
    const uint32_t ebar0 = a_base + RegionA::CNT_OFF + (uint32_t)group * (ATTN_MAX_STAGES * 16u);  // copy warps: "part handed back" barriers
    const uint32_t ctrl_s = a_base + RegionA::CTRL_OFF + (uint32_t)group * 16u;
    const uint32_t merge_s = a_base + RegionA::MERGE_OFF + (uint32_t)group * MERGE_AREA;

    // (modes with a table of their own let their successor start only once they have themselves seen their predecessor finish)
    if (!PUBLISH) pdl_launch_dependents();
    if (TQ_DBG(32)) { pdl_wait(); pdl_launch_dependents(); return; }
    const int G = p.G;

    // (layer form: the first positions are on their way while the look-up table is written)
    int first_pos = p.pos_value;
    if (LAYER && p.positions && tid < G) first_pos = ldg32_l2(p.positions + tid);
    // ---- byte -> centroid table, one column per lane ----
    if (TQ_DBG(16)) {
    } else if (BITS == 4) {
        for (int idx = tid; idx < 256 * 8; idx += blockDim.x) {  // four lanes' columns at a time
            int v = idx >> 3, l = idx & 7;
            uint32_t val = pack_half2(kCent4[v & 15], kCent4[v >> 4]);
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(LUT_ABS + (uint32_t)v * 256u + (uint32_t)l * 16u), "r"(val) : "memory");
        }
    } else {
        for (int idx = tid; idx < 256 * 16; idx += blockDim.x) {  // two lanes' columns at a time
            int v = idx >> 4, l = idx & 15;
            // (c0, c2), (c1, c3): the low and the high nibble each give one value to either word.  For K a byte is four
            // coordinates of one token (the query fragments are packed in the same order); for V a byte is put together
            // from the nibbles of two tokens, and either word is then one coordinate of that token pair.
            uint32_t lo2 = pack_half2(kCent2[v & 3], kCent2[(v >> 4) & 3]);
            uint32_t hi2 = pack_half2(kCent2[(v >> 2) & 3], kCent2[(v >> 6) & 3]);
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %1, %2};" ::"r"(LUT_ABS + (uint32_t)v * 256u + (uint32_t)l * 16u),
                         "r"(lo2), "r"(hi2) : "memory");
        }
    }
    if (gtid == 0) {
        for (int s = 0; s < 2 * ATTN_MAX_STAGES; ++s) {
            mbar_init(bar0 + 8u * s, 1);
            if (COPIER) mbar_init(ebar0 + 8u * s, Hkv);
            else asm volatile("st.shared.u32 [%0], %1;" ::"r"(cnt0 + 4u * s), "r"(0u) : "memory");
        }
        if (PUBLISH) mbar_init(a_base + 320u + 8u * (uint32_t)group, 1);
        fence_mbar_init();
        fence_proxy_async_smem();
    }
    // Everything above touches only shared memory and may overlap the tail of the previous kernel in the stream.
    if (!LAYER) {
        pdl_wait();
        if (PUBLISH) pdl_launch_dependents();
    }
    // Tile table.  Built here, in shared memory, from the positions (every CTA the same table); the plain form reads the one the
    // append kernel left in the workspace.
    const int* ts;
    if constexpr (PUBLISH) {
        int* ts_s = reinterpret_cast<int*>(dyn_smem + (a_base - dyn_base) + RegionA::ts_off(MERGE_AREA));
        int* scan_s = reinterpret_cast<int*>(dyn_smem + (a_base - dyn_base) + RegionA::scan_off(MERGE_AREA));
        int carry = 0;
        for (int base = 0; base < G; base += (int)blockDim.x) {
            const int gq = base + tid;
            int n = 0;
            if (gq < G) {
                int pos = LAYER && base == 0 ? first_pos : p.positions ? __ldcg(p.positions + gq) : p.pos_value;
                if (pos < 0) pos = 0;
                n = (pos + TILE_TOKENS) / TILE_TOKENS;
            }
            int incl = n;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += v;
            }
            if (lane == 31) scan_s[warp] = incl;
            __syncthreads();
            int before = 0, all = 0;
            for (int w2 = 0; w2 < (int)(blockDim.x >> 5); ++w2) {
                const int v = scan_s[w2];
                before += (w2 < warp) ? v : 0;
                all += v;
            }
            if (gq < G) ts_s[gq] = carry + before + incl - n;
            carry += all;
            __syncthreads();
        }
        if (tid == 0) ts_s[G] = carry;
        ts = ts_s;
        if constexpr (PERSIST) {
            if (blockIdx.x == 0) {  // the merge kernel reads the table from global memory
                __syncthreads();
                for (int i = tid; i <= G; i += (int)blockDim.x) p.table_out[i] = ts_s[i];
            }
        }
    } else {
        ts = p.tile_start;
    }
    __syncthreads();
    const int N = ts[G];  // (the host refuses caches of 2^31 rows or more)

    // ---- work slice of this worker ----
    // At most min(workers, N) workers take part, so that every participant owns at least one tile: the ticket
    // count of a sequence is then simply (last owner - first owner + 1).  Fewer when the list is short.
    const long long w_all = (long long)gridDim.x * ATTN_GROUPS;
    const int W = attention_workers(w_all, N, G, TQ_DBG_FACTOR ? TQ_DBG_FACTOR : 16);
    const int wid = blockIdx.x * ATTN_GROUPS + group;
    if (PERSIST && blockIdx.x == 0 && tid == 0) {
        p.table_out[G + 1] = W;
        p.table_out[G + 2] = N;
    }
    if (wid >= W && !copier) return;  // uniform for the worker; no CTA-wide barrier follows
    // Worker w takes the tiles [w * N / W, (w + 1) * N / W).
    const int n_each = N / W, n_over = N - n_each * W;  // (N < 2^26, W <= 1024)
    const int lo = wid * n_each + wid * n_over / W, hi = (wid + 1) * n_each + (wid + 1) * n_over / W;
    int g;  // first sequence of the slice: largest g with tile_start[g] <= lo
    if (!PUBLISH && p.worker_g && !TQ_DBG_FACTOR) {
        g = p.worker_g[wid];
    } else {
        int a = 0, b = G;  // invariant: tile_start[a] <= lo < tile_start[b]
        while (b - a > 1) {
            int mid = (a + b) >> 1;
            if (ts[mid] <= lo) a = mid; else b = mid;
        }
        g = a;
    }

    const bool idle = copier && (lane > 0 || wid >= W);  // nothing to copy (it returns further down)
    if (idle) g = 0;
    // ---- load cursor over the flat tile list (warp-uniform, advanced in step by every warp of the worker) ----
    // Tile counts and row numbers fit 32 bits (the host refuses caches of 2^31 rows or more).
    const int lo_i = idle ? 0 : lo, hi_i = idle ? 0 : hi;
    int cl_tile = lo_i;                         // next tile to load into shared memory
    int cl_g = g;
    int cl_gend = ts[g + 1];
    // first cache row of tile j of sequence gq (j counted from the sequence's first tile)
    auto tile_row = [&](int gq, int j) -> int {
        if (p.prefix_tiles && j < p.prefix_tiles[gq]) return (int)p.prefix_base[gq] + j * TILE_TOKENS;
        return (int)(p.row_base ? p.row_base[gq] : (long long)gq * p.max_seq_len) + j * TILE_TOKENS;
    };
    const int row_lo = tile_row(g, lo_i - ts[g]);
    int cl_switch = p.prefix_tiles ? ts[g] + p.prefix_tiles[g] : -1;  // flat index of the current sequence's first private tile
    int cl_row = row_lo;
    int cl_layer = 0;                           // whole-step form: layer (relative to layer0) the cursor is in
    const int g_lo = g;
    const int n_layers = PERSIST ? p.n_layers : 1;
    auto cursor_advance = [&]() {
        ++cl_tile;
        cl_row += TILE_TOKENS;
        if (PERSIST && cl_tile == hi_i) {  // the same slice again, one layer on
            ++cl_layer;
            cl_tile = lo_i;
            cl_g = g_lo;
            cl_gend = ts[g_lo + 1];
            cl_row = row_lo;
            if (p.prefix_tiles) cl_switch = ts[g_lo] + p.prefix_tiles[g_lo];
        } else if (cl_tile == cl_gend && cl_tile < hi_i) {
            ++cl_g;
            cl_gend = ts[cl_g + 1];
            cl_row = tile_row(cl_g, 0);
            if (p.prefix_tiles) cl_switch = cl_tile + p.prefix_tiles[cl_g];
        } else if (cl_tile == cl_switch) {  // from the shared prefix into the sequence's own rows
            cl_row = tile_row(cl_g, cl_tile - ts[cl_g]);
        }
    };
    auto cursor_more = [&]() -> bool { return PERSIST ? cl_layer < n_layers : cl_tile < hi_i; };
    // the rotated queries of a segment's sequence arrive by a bulk copy into the (otherwise idle) merge
    // area of the worker, completion on a barrier of their own; the copy for the next segment goes out as soon as every
    // warp has taken its fragments of the current one
    const uint32_t qbar = a_base + 320u + 8u * (uint32_t)group;
    const uint32_t q_block_bytes = (uint32_t)p.H * HEAD_DIM * (Q_WIDE ? 4u : 2u);
    uint32_t q_par = 0;
    auto issue_queries = [&](int layer, int gq) {
        mbar_arrive_expect_tx(qbar, q_block_bytes);
        const char* const src = Q_WIDE ? reinterpret_cast<const char*>(p.q_rot32) : reinterpret_cast<const char*>(p.q_rot16);
        bulk_load(merge_s, src + ((size_t)layer * p.G + (size_t)gq) * q_block_bytes, q_block_bytes, qbar);
    };
    int consumed = 0;
    int s_idx = 0;          // 2-bit form: stage of the tile being consumed and the parity of its barrier
    uint32_t s_par = 0;
    bool dead = false;  // a bounded wait gave up: keep the control flow, stop touching the pipeline
    const bool loads_on = !TQ_DBG(2);
    const int total_rows_i = (int)p.total_rows;

    // One elected thread issues the two copies of a tile's K part (codes, norms) or V part, clipped to the end of the
    // arrays; rows past a sequence's position only ever reach masked tokens.
    auto issue_part = [&](int row, int s, int part, int layer) {
        int nrows = total_rows_i - row;
        if (nrows > TILE_TOKENS) nrows = TILE_TOKENS;
        if (nrows < 0) nrows = 0;
        const uint32_t nb = (uint32_t)nrows * (uint32_t)Hkv * 2u;
        const uint32_t bar = bar0 + 16u * s + 8u * part;
        const uint32_t dst = stage_addr(s);
        // a tensor-map box always delivers its full size (rows past the end of the array arrive as zeros)
        mbar_arrive_expect_tx(bar, code_tile + nb);
        const size_t noff = (size_t)row * Hkv + (PERSIST ? (size_t)layer * (size_t)p.norm_layer_stride : (size_t)0);
        if (part == 0) {
            if (PERSIST) tma_load_4d(dst, &tmK, bar, 0, row, 0, p.layer0 + layer);
            else tma_load_3d(dst, &tmK, bar, 0, row, 0);
            if (nrows > 0) bulk_load(dst + 2u * code_tile, p.kn + noff, nb, bar);
        } else {
            if (PERSIST) tma_load_4d(dst + code_tile, &tmV, bar, 0, row, 0, p.layer0 + layer);
            else tma_load_3d(dst + code_tile, &tmV, bar, 0, row, 0);
            if (nrows > 0) bulk_load(dst + 2u * code_tile + norm_tile, p.vn + noff, nb, bar);
        }
    };
    auto issue_tile = [&](int row, int s, int layer) {
        issue_part(row, s, 0, layer);
        issue_part(row, s, 1, layer);
    };
    // L2 prefetch of the tile ATTN_L2_AHEAD further on, when it belongs to the same sequence (rows are then contiguous)
    auto prefetch_ahead = [&](int row, int tile_idx, int gend) {
        if (tile_idx + p.l2_ahead < gend && tile_idx + p.l2_ahead < hi_i) {  // own slice only: others fetch theirs
            const int prow = row + p.l2_ahead * TILE_TOKENS;
            int nrows = total_rows_i - prow;
            if (nrows > TILE_TOKENS) nrows = TILE_TOKENS;
            if (nrows > 0) {
                bulk_prefetch_l2(p.ck + (size_t)prow * kvp, (uint32_t)nrows * kvp);
                bulk_prefetch_l2(p.cv + (size_t)prow * kvp, (uint32_t)nrows * kvp);
            }
        }
    };
    auto fill_ring = [&]() {  // prologue: fill the ring (and prefetch a few tiles beyond each)
        for (int s = 0; s < S; ++s) {
            if (cursor_more()) {
                if (gtid == 0 && loads_on) {
                    issue_tile(cl_row, s, cl_layer);
                    prefetch_ahead(cl_row, cl_tile, cl_gend);
                }
                cursor_advance();
            }
        }
    };
    if (PERSIST && !COPIER && gtid == 0 && loads_on) issue_queries(0, g);
    if constexpr (COPIER) {
        if (copier) {
            // One thread per worker walks the worker's list and re-arms every part as soon as all its warps have handed it back.
            // (When the last warp to hand a part back did this itself, the cursor over the list, the counter's atomic and the
            // fences were in all 16 warps' instruction streams.)  Its own wait is bounded like theirs, and it leaves only when
            // the copies it issued have landed.
            if constexpr (HKV == 8) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ATTN_REGS_COPY));
            if (warp >= ATTN_GROUPS * (Hkv + 1) || lo_i >= hi_i) return;
            int n = 0;
            bool stuck = false, waited = !LAYER || !p.appends;
            for (; cursor_more() && loads_on && !stuck; ++n, cursor_advance()) {
                if (!waited && cl_tile + 1 == cl_gend) {  // the tile of a new token: not before the launch that appends has finished
                    pdl_wait();
                    waited = true;
                }
                const int st = n % S;
                const uint32_t par = ((uint32_t)(n / S) & 1u) ^ 1u;  // of the hand-back that this tile's copies wait for
                for (int part = 0; part < 2 && !stuck; ++part) {
                    if (n >= S) {
                        uint32_t ok = 0;
                        for (uint32_t it = 0; it < (1u << 15) && !ok; ++it)
                            ok = mbar_try_wait_hint(ebar0 + 16u * (uint32_t)st + 8u * (uint32_t)part, par, 20000u);
                        if (!ok) {
                            stuck = true;
                            atomicMax(p.status, ST_TMA_WAIT_TIMEOUT);
                            break;
                        }
                    }
                    issue_part(cl_row, st, part, cl_layer);
                }
                if (!stuck) prefetch_ahead(cl_row, cl_tile, cl_gend);
            }
            for (int m = n > S ? n - S : 0; m < n; ++m) {
                mbar_wait_bounded(bar0 + 16u * (uint32_t)(m % S), (uint32_t)(m / S) & 1u, 1u << 16);
                mbar_wait_bounded(bar0 + 16u * (uint32_t)(m % S) + 8u, (uint32_t)(m / S) & 1u, 1u << 16);
            }
            return;
        }
        if constexpr (HKV == 8) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ATTN_REGS_WORK));
        if (LAYER) {
            pdl_wait();
            pdl_launch_dependents();
        }
        if (gtid == 0 && loads_on) issue_queries(0, g);
    } else {
        fill_ring();
    }

    if (TQ_DBG(64)) return;
    const uint32_t lutlane = LUT_ABS | ((uint32_t)lane << (BITS == 4 ? 2 : 3));
    // ---- swizzled addressing.  A box holds [32 rows][128 B]; the 16-byte chunk c of row r sits at chunk c ^ (r & 7).
    // Tokens of an 8-token score block are taken in the order tau(n) = n ^ ((n & 1) << 2), which keeps both the
    // K reads (lane <-> token tau(gl)) and the V reads (lane <-> tokens tau(2*t4), tau(2*t4+1)) conflict free.
    const uint32_t hbyte = (uint32_t)head * Geo::BPH;          // this head's first byte within the token row
    const uint32_t box_off = (hbyte >> 7) * 4096u;              // which box
    const uint32_t hchunk = (hbyte & 127u) >> 4;                // first 16-byte chunk of the head inside the box row
    const uint32_t tauK = (uint32_t)gl ^ (((uint32_t)gl & 1u) << 2);
    const uint32_t tokA = 2u * (uint32_t)t4, tokB = (2u * (uint32_t)t4 + 1u) ^ 4u;   // tau(2*t4), tau(2*t4+1)
    uint32_t k_off, vA_off, vB_off;
    if (BITS == 4) {
        k_off = box_off + tauK * 128u + (((hchunk + (uint32_t)t4) ^ tauK) << 4);
        const uint32_t vch = hchunk + ((uint32_t)gl >> 1), vsub = ((uint32_t)gl & 1u) * 8u;
        vA_off = box_off + tokA * 128u + ((vch ^ tokA) << 4) + vsub;
        vB_off = box_off + tokB * 128u + ((vch ^ tokB) << 4) + vsub;
    } else {
        k_off = box_off + tauK * 128u + (((hchunk + ((uint32_t)t4 >> 1)) ^ tauK) << 4) + ((uint32_t)t4 & 1u) * 8u;
        const uint32_t vch = hchunk + ((uint32_t)gl >> 2), vsub = ((uint32_t)gl & 3u) * 4u;
        vA_off = box_off + tokA * 128u + ((vch ^ tokA) << 4) + vsub;
        vB_off = box_off + tokB * 128u + ((vch ^ tokB) << 4) + vsub;
    }

#ifdef TQ_TIMING_SWITCHES
    long long stamp_acc[16] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    long long stamp_last = clock64();
#endif
    for (int layer = 0; layer < n_layers; ++layer) {  // (one pass unless this is the whole-step form)
    int tile = lo_i;
    g = g_lo;
    while (tile < hi_i) {
        // ================= one segment: tiles [tile, seg_end) of sequence g =================
        const int ts_g = ts[g];
        const int ts_g1 = ts[g + 1];
        const int seg_end = hi_i < ts_g1 ? hi_i : ts_g1;
        const int pos = p.positions ? p.positions[g] : p.pos_value;
        const int L = (pos < 0 ? 0 : pos) + 1;
        TQ_STAMP(8);   // loop tail + publishing of the previous segment + this segment's table / position reads
        // query fragments (B operand of the score product): lane (gl, t4) holds coordinates 32*t4 .. 32*t4+31 of head
        // head*grp + gl as fp16
        uint32_t qb[8][2];
        const int q_col = PAIR ? gl >> 1 : gl;                                       // query head of this lane's column
        const bool q_on = q_col < grp && !(PAIR && !PLANES && (gl & 1));             // (fp16 queries: the odd columns stay zero)
        float s_scale = 0.0f, s_zero = 0.0f;  // PLANES: score = (sum * s_scale + s_zero) * K norm, of head t4
        // PLANES: the queries as integers Q, |Q| <= 32639, in two signed bytes: the even column of a head has the high ones, the odd
        // column the low ones.  Code 2 b1 + b0 stands for -c3 + (c3 - c2) b0 + (c3 + c2) b1, c2 and c3 the positive centroids.  Bit b of
        // a byte's coordinate j is worth 2^(2 j + b) where it stands: the query of that plane is divided by it (by 2^(2 (j mod 2) + b): the
        // coordinates 0, 1 and 2, 3 have sums of their own, 16 apart).  The sum's offset is minus half the sum with all bits set.
        // Rounding: half a weight (1 and 4, 2 and 8) of the 32639 C_b / C0 steps to the largest coordinate: 1.5e-5 to 6.6e-5 of it at most.
        // The queries are fp32, but in the whole-step form, which holds them as fp16: there up to 4.9e-4 of every coordinate on top, and
        // queries that do not fit fp16 rotated and scaled, infinities here, give NaN.
        auto make_planes = [&](const float (&x)[32]) {
            constexpr float C0 = 0.13351f - 0.04003f, C1 = 0.13351f + 0.04003f;
            uint32_t top = 0u;  // of the magnitudes' bits: an infinity or a NaN comes out on top
#pragma unroll
            for (int i = 0; i < 32; ++i) top = max(top, __float_as_uint(x[i]) & 0x7fffffffu);
            top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float mx = __uint_as_float(top);
            const bool some = mx > 1e-30f;
            const float k = some ? 32639.0f / (mx * C0) : 0.0f;
            const float scale = top >= 0x7f800000u ? __uint_as_float(0x7fffffffu) : some ? mx * (C0 / (16.0f * 32639.0f)) : 0.0f;
            const uint32_t bias = (gl & 1) ? 0u : 128u, sel = (gl & 1) ? 0x0040u : 0x0051u;
            const float magic = 12582912.0f + (float)bias;  // 1.5 * 2^23: the sum's low bits are the rounded integer
            uint32_t all = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const uint32_t weight = 1u << (2 * (j & 1) + b);
                    const float kk = k * ((b ? C1 : C0) / (float)weight);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        uint32_t u[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            u[i] = __float_as_uint(fmaf(x[16 * r + 4 * i + j], kk, magic));
                            all += weight * u[i];
                        }
                        qb[2 * j + b][r] = prmt(prmt(u[0], u[1], sel), prmt(u[2], u[3], sel), 0x5410u);
                    }
                }
            all -= 240u * (0x4b400000u + bias);  // 8 bytes' weights
            all += __shfl_xor_sync(0xffffffffu, all, 1);
            all += __shfl_xor_sync(0xffffffffu, all, 2);
            const float zero = -8.0f * (float)(int)all * scale;
            s_scale = __shfl_sync(0xffffffffu, scale, 8 * t4);
            s_zero = __shfl_sync(0xffffffffu, zero, 8 * t4);
        };
        // lane (gl, t4): the 32 coordinates 32*t4 .. of its head from the merge area, rows `pitch` bytes apart
        auto take_fragments = [&]() {
            constexpr uint32_t pitch = HEAD_DIM * 2u;
            if constexpr (Q_WIDE) {
                float x[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint4 u = make_uint4(0u, 0u, 0u, 0u);
                    if (q_on && !dead) u = ldsv128(merge_s + (uint32_t)(head * grp + q_col) * (HEAD_DIM * 4u) + (uint32_t)(4 * i + t4) * 16u);
                    x[4 * i] = __uint_as_float(u.x); x[4 * i + 1] = __uint_as_float(u.y);
                    x[4 * i + 2] = __uint_as_float(u.z); x[4 * i + 3] = __uint_as_float(u.w);
                }
                make_planes(x);
                return;
            }
            uint4 qw[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                qw[i] = make_uint4(0u, 0u, 0u, 0u);
                if (q_on && !dead) qw[i] = ldsv128(merge_s + (uint32_t)(head * grp + q_col) * pitch + (uint32_t)(32 * t4 + 8 * i) * 2u);
            }
            if constexpr (PLANES) {
                float x[32];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half2* h2 = reinterpret_cast<const __half2*>(&qw[i]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(h2[e]);
                        x[8 * i + 2 * e] = f.x;
                        x[8 * i + 2 * e + 1] = f.y;
                    }
                }
                make_planes(x);
                return;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t w4[4] = {qw[i].x, qw[i].y, qw[i].z, qw[i].w};
#pragma unroll
                for (int h2 = 0; h2 < 2; ++h2) {
                    // step j = 2*i + h2 takes the coordinates 4j .. 4j+3: (4j, 4j+1), (4j+2, 4j+3) -- the 2-bit table
                    // returns the four values of a byte as (0, 2), (1, 3)
                    const uint32_t a = w4[2 * h2], b = w4[2 * h2 + 1];
                    qb[2 * i + h2][0] = BITS == 2 ? prmt(a, b, 0x5410u) : a;
                    qb[2 * i + h2][1] = BITS == 2 ? prmt(a, b, 0x7632u) : b;
                }
            }
        };
        if constexpr (PUBLISH) {
            uint32_t ok = (dead || !loads_on) ? 1u : 0u;
            for (uint32_t it = 0; it < (1u << 14) && !ok; ++it) ok = mbar_try_wait_hint(qbar, q_par, 20000u);
            if (!ok) {
                dead = true;
                if (lane == 0) atomicMax(p.status, ST_TMA_WAIT_TIMEOUT);
            }
            dead = __any_sync(0xffffffffu, dead);
            q_par ^= 1u;
            TQ_STAMP(9);   // wait for the query block
            take_fragments();
            TQ_STAMP(10);  // fragments
            group_barrier(group, gthreads);  // every warp holds its fragments: the area may take the next block
            TQ_STAMP(11);  // barrier of the worker's warps
            if (gtid == 0 && !dead && loads_on) {
                fence_proxy_async_smem();
                if (seg_end < hi_i) issue_queries(layer, g + 1);
                else if (layer + 1 < n_layers) issue_queries(layer + 1, g_lo);
            }
        } else {
            float qv[32];
            if (q_on && !TQ_DBG(8)) {
                const float4* src =
                    reinterpret_cast<const float4*>(p.q_rot + ((size_t)g * p.H + (size_t)head * grp + q_col) * HEAD_DIM + 32 * t4);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float4 f = __ldg(src + i);
                    qv[4 * i] = f.x; qv[4 * i + 1] = f.y; qv[4 * i + 2] = f.z; qv[4 * i + 3] = f.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) qv[i] = 0.0f;
            }
            if constexpr (PLANES) make_planes(qv);
#pragma unroll
            for (int j = 0; j < (PLANES ? 0 : 8); ++j) {
                // the 2-bit table returns the four values of a byte as (0, 2), (1, 3)
                const float x0 = qv[4 * j], x1 = BITS == 2 ? qv[4 * j + 2] : qv[4 * j + 1];
                const float x2 = BITS == 2 ? qv[4 * j + 1] : qv[4 * j + 2], x3 = qv[4 * j + 3];
                qb[j][0] = pack_half2(x0, x1);
                qb[j][1] = pack_half2(x2, x3);
            }
        }

        // running maximum and (per lane: over its own token rows) sum of the heads of this lane's score columns
        float m_run[NE], l_run[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) { m_run[e] = -1e30f; l_run[e] = 0.0f; }
        float acc[8][4];
#pragma unroll
        for (int b = 0; b < 8; ++b) { acc[b][0] = acc[b][1] = acc[b][2] = acc[b][3] = 0.0f; }

        for (; tile < seg_end; ++tile) {
            const int t0 = (tile - ts_g) * TILE_TOKENS;
            const bool full = t0 + TILE_TOKENS <= L;  // warp-uniform: no token of the tile is masked
            const int s = BITS == 2 ? s_idx : (consumed & (S - 1));
            const uint32_t parity = BITS == 2 ? s_par : ((uint32_t)(consumed >> s_log) & 1u);
            // the tile that takes this stage's place (warp-uniform; every warp of the worker advances the cursor in step)
            const int next_row = cl_row, next_tile = cl_tile, next_gend = cl_gend, next_layer = cl_layer;
            const bool more = !COPIER && cursor_more();
            if (more) cursor_advance();
            // Wait for one part (0: K codes and norms, 1: V codes and norms) of the stage.  Returns 0 at run time, as a
            // value PRODUCED by the wait: the part's loads take it into their address and so cannot move above the wait.
            auto wait_part = [&](int part) -> uint32_t {
                uint32_t token = 0;
                if (!dead && loads_on) {
                    const uint32_t bar = bar0 + 16u * s + 8u * part;
                    uint32_t ok = mbar_try_wait_hint(bar, parity, 20000u);
                    if (!ok) {
                        for (uint32_t it = 0; it < (1u << 14) && !ok; ++it) ok = mbar_try_wait_hint(bar, parity, 20000u);
                        if (!ok) {  // (lane by lane: one that gave up computes on, on whatever is there, and waits for nothing more)
                            dead = true;
                            atomicMax(p.status, ST_TMA_WAIT_TIMEOUT);
                            ok = 1u;
                        }
                    }
                    __syncwarp();
                    token = ok ^ 1u;
                }
                return token;
            };
            // Hand a part back: everything this warp read from it has been consumed by (ordered) instructions above.  The
            // last warp of the worker to get here re-arms the part with the same part of the tile S ahead; nobody waits.
            auto release_part = [&](int part) {
                __syncwarp();
                if constexpr (COPIER) {
                    if (lane == 0) mbar_arrive(ebar0 + 16u * (uint32_t)s + 8u * (uint32_t)part);
                    return;
                }
                if (lane == 0 && more && !dead && loads_on) {
                    __threadfence_block();  // this warp's reads of the part are ordered before the hand-over below
                    const uint32_t cnt = cnt0 + 8u * s + 4u * part;
                    const uint32_t old = atom_add_shared(cnt, 1u);
                    if (old == (uint32_t)Hkv - 1u) {
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(cnt), "r"(0u) : "memory");
                        fence_proxy_async_smem();
                        issue_part(next_row, s, part, next_layer);
                        if (part == 1) prefetch_ahead(next_row, next_tile, next_gend);
                    }
                }
            };
            // The tile body exists twice: for tiles in which every token is attended to (all but the last tile of a
            // sequence) without any masking code, and for the last, partly filled tile with it.
            auto tile_body = [&](auto full_tag) {
                constexpr bool FULLT = decltype(full_tag)::value;
                constexpr uint32_t nstride = (uint32_t)Hkv * 2u;
                TQ_STAMP(0);
                const uint32_t tokK = wait_part(0);
                TQ_STAMP(1);
                const uint32_t kt = stage_addr(s) + tokK;
                const uint32_t kns = kt + 2u * code_tile + (uint32_t)head * 2u;

                // ---------------- scores: S^T = K (16 token rows x 16 coordinates) * Q^T (16 coordinates x 8 heads), two
                // blocks of 16 token rows.  Row r of block rb is token 16*rb + 8*(r >> 3) + tau(r & 7) of the tile; the
                // eight 16-coordinate steps of a row block form one accumulator chain.
                float c[2][4];
                int t_lo[2][4], t_hi[2][4];  // PLANES: sums of the coordinates 0, 1 and 2, 3 of every byte
                {
                    uint32_t w[4][4];
#pragma unroll
                    for (int blk = 0; blk < 4; ++blk) {
                        if (BITS == 4) {
                            const uint4 kw = ldsp128(kt + (uint32_t)blk * 1024u + k_off);
                            w[blk][0] = kw.x; w[blk][1] = kw.y; w[blk][2] = kw.z; w[blk][3] = kw.w;
                        } else {
                            const uint2 kw = ldsp64(kt + (uint32_t)blk * 1024u + k_off);
                            w[blk][0] = kw.x; w[blk][1] = kw.y; w[blk][2] = w[blk][3] = 0u;
                        }
                    }
#pragma unroll
                    for (int rb = 0; rb < 2; ++rb) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            c[rb][e] = 0.0f;
                            t_lo[rb][e] = t_hi[rb][e] = 0;
                        }
                    }
                    if constexpr (PLANES) {
#pragma unroll
                        for (int pl = 0; pl < 4; ++pl)
#pragma unroll
                            for (int rb = 0; rb < 2; ++rb) {
                                const uint32_t m = 0x01010101u << pl, n = m << 4;
                                mma16832(t_lo[rb], w[2 * rb][0] & m, w[2 * rb + 1][0] & m, w[2 * rb][1] & m, w[2 * rb + 1][1] & m, qb[pl][0], qb[pl][1]);
                                mma16832(t_hi[rb], w[2 * rb][0] & n, w[2 * rb + 1][0] & n, w[2 * rb][1] & n, w[2 * rb + 1][1] & n, qb[4 + pl][0], qb[4 + pl][1]);
                            }
                    }
#pragma unroll
                    for (int j = 0; j < (PLANES ? 0 : 8); ++j) {
#pragma unroll
                        for (int rb = 0; rb < 2; ++rb) {
                            uint32_t a0, a1, a2, a3;  // rows gl / gl + 8, coordinate pairs (4j, 4j+1) / (4j+2, 4j+3) of the lane's 32
                            if (BITS == 4) {
                                const uint32_t sel0 = (j & 1) ? 0x7624u : 0x7604u, sel1 = (j & 1) ? 0x7634u : 0x7614u;
                                const uint32_t wlo = w[2 * rb][j >> 1], whi = w[2 * rb + 1][j >> 1];
                                a0 = ldsp32(prmt(wlo, lutlane, sel0));
                                a1 = ldsp32(prmt(whi, lutlane, sel0));
                                a2 = ldsp32(prmt(wlo, lutlane, sel1));
                                a3 = ldsp32(prmt(whi, lutlane, sel1));
                            } else {
                                const uint32_t sel = 0x7604u | ((uint32_t)(j & 3) << 4);
                                const uint2 lo2 = ldsp64(prmt(w[2 * rb][j >> 2], lutlane, sel));
                                const uint2 hi2 = ldsp64(prmt(w[2 * rb + 1][j >> 2], lutlane, sel));
                                a0 = lo2.x; a1 = hi2.x; a2 = lo2.y; a3 = hi2.y;
                            }
                            mma16816(c[rb], a0, a1, a2, a3, qb[j][0], qb[j][1]);
                        }
                    }
                }
                // K norms of this lane's four token rows (ordered loads: they precede the hand-over of the K part)
                float kn4[4];
#pragma unroll
                for (int blk = 0; blk < 4; ++blk) kn4[blk] = ldsv_h2f(kns + ((uint32_t)(8 * blk) + tauK) * nstride);
                release_part(0);
                TQ_STAMP(2);

                // ---------------- online softmax: sv[blk][e] = score of token row (block blk, tau(gl)) and head t4 (PAIR), 2*t4 + e.
                // Columns of heads >= grp carry zeros and are never read.
                float sv[4][NE];
#pragma unroll
                for (int blk = 0; blk < 4; ++blk) {
                    const int rb = blk >> 1, at = 2 * (blk & 1);
                    if constexpr (PLANES) {
                        const int t = t_lo[rb][at] * 4096 + t_lo[rb][at + 1] * 16 + t_hi[rb][at] * 256 + t_hi[rb][at + 1];  // (below 2^30)
                        sv[blk][0] = fmaf((float)t, s_scale, s_zero) * kn4[blk];
                    } else {
#pragma unroll
                        for (int e = 0; e < NE; ++e) sv[blk][e] = c[rb][at + e] * kn4[blk];
                    }
                }
                if constexpr (!FULLT) {  // rows past the position may hold anything (even NaN norms): force them out
#pragma unroll
                    for (int blk = 0; blk < 4; ++blk) {
                        const int tok = t0 + 8 * blk + (int)tauK;
#pragma unroll
                        for (int e = 0; e < NE; ++e)
                            if (tok >= L) sv[blk][e] = -1e30f;
                    }
                }
                float mx[NE];
                bool grown = false;
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    mx[e] = fmaxf(fmaxf(sv[0][e], sv[1][e]), fmaxf(sv[2][e], sv[3][e]));
                    grown = grown || mx[e] > m_run[e];
                }
                // (the maximum over the row lanes is only looked for in the few tiles that hold a new one)
                if (__any_sync(0xffffffffu, grown)) {
                    float cf[NE];
#pragma unroll
                    for (int e = 0; e < NE; ++e) {
#pragma unroll
                        for (int o = 4; o < 32; o <<= 1) mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], o));
                        const float mn = fmaxf(m_run[e], mx[e]);
                        cf[e] = ex2_approx(m_run[e] - mn);  // 1 when unchanged, 0 at the first tile; the lane's accumulators are of its own heads
                        l_run[e] *= cf[e];
                        m_run[e] = mn;
                    }
#pragma unroll
                    for (int b = 0; b < 8; ++b)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[b][e] *= cf[PAIR ? 0 : e & 1];
                }
                float pv[4][NE];
#pragma unroll
                for (int blk = 0; blk < 4; ++blk)
#pragma unroll
                    for (int e = 0; e < NE; ++e) pv[blk][e] = ex2_approx(sv[blk][e] - m_run[e]);
                if constexpr (!FULLT) {
#pragma unroll
                    for (int blk = 0; blk < 4; ++blk) {
                        const int tok = t0 + 8 * blk + (int)tauK;
#pragma unroll
                        for (int e = 0; e < NE; ++e)
                            if (tok >= L) pv[blk][e] = 0.0f;
                    }
                }
#pragma unroll
                for (int e = 0; e < NE; ++e) l_run[e] += (pv[0][e] + pv[1][e]) + (pv[2][e] + pv[3][e]);

                // ---------------- values: 2 blocks of 16 tokens ----------------
                TQ_STAMP(3);
                const uint32_t tokV = wait_part(1);
                TQ_STAMP(4);
                const uint32_t vt = stage_addr(s) + code_tile + tokV;
                const uint32_t vns = stage_addr(s) + tokV + 2u * code_tile + norm_tile + (uint32_t)head * 2u;
                // weights times V norms as fp16 pairs (heads 2*t4, 2*t4 + 1) of this lane's token rows, then transposed
                // across the warp into the B operand of the value product: lane (gl, t4) receives head gl of the token
                // rows tau(2*t4), tau(2*t4 + 1) of every 8-row block
                // (PAIR: the pairs are one head's rows of two blocks; the even lanes gl get the first block's, the odd ones the second's)
                uint32_t pb[4];
                float vn[4];
#pragma unroll
                for (int blk = 0; blk < 4; ++blk) {
                    vn[blk] = ldsp_h2f(vns + ((uint32_t)(8 * blk) + tauK) * nstride);
                    if constexpr (!FULLT) {  // 0 * NaN would poison the accumulators
                        if (t0 + 8 * blk + (int)tauK >= L) vn[blk] = 0.0f;
                    }
                }
                if constexpr (PAIR) {
#pragma unroll
                    for (int gam = 0; gam < 2; ++gam) {
                        const uint32_t t = movmatrix_trans(pack_half2(pv[2 * gam][0] * vn[2 * gam], pv[2 * gam + 1][0] * vn[2 * gam + 1]));
                        pb[2 * gam] = (gl & 1) ? 0u : t;
                        pb[2 * gam + 1] = (gl & 1) ? t : 0u;
                    }
                } else {
#pragma unroll
                    for (int blk = 0; blk < 4; ++blk) pb[blk] = movmatrix_trans(pack_half2(pv[blk][0] * vn[blk], pv[blk][NE - 1] * vn[blk]));
                }
#pragma unroll
                for (int gam = 0; gam < 2; ++gam) {
                    // token rows of this lane: A, B from score block 2*gam, C, D from block 2*gam+1
                    const uint32_t pb0 = pb[2 * gam], pb1 = pb[2 * gam + 1];
                    if (BITS == 4) {
                        // lane reads bytes 8*gl .. 8*gl+7 (coordinates 16*gl .. 16*gl+15) of token rows A, B, C = A+8, D = B+8
                        const uint32_t vg = vt + (uint32_t)gam * 2048u;
                        const uint2 xa = ldsp64(vg + vA_off);
                        const uint2 xb = ldsp64(vg + vB_off);
                        const uint2 xc = ldsp64(vg + vA_off + 1024u);
                        const uint2 xd = ldsp64(vg + vB_off + 1024u);
                        // Interleave the nibbles of two tokens: byte b of `ev` = (code of token A, code of token B) for the
                        // EVEN coordinate of byte b, `od` for the odd one.  The table then returns the (A, B) pair directly.
                        const uint32_t wa[2] = {xa.x, xa.y}, wb[2] = {xb.x, xb.y}, wc[2] = {xc.x, xc.y}, wd[2] = {xd.x, xd.y};
#pragma unroll
                        for (int w2 = 0; w2 < 2; ++w2) {
                            const uint32_t ev_ab = (wa[w2] & 0x0f0f0f0fu) | ((wb[w2] << 4) & 0xf0f0f0f0u);
                            const uint32_t od_ab = ((wa[w2] >> 4) & 0x0f0f0f0fu) | (wb[w2] & 0xf0f0f0f0u);
                            const uint32_t ev_cd = (wc[w2] & 0x0f0f0f0fu) | ((wd[w2] << 4) & 0xf0f0f0f0u);
                            const uint32_t od_cd = ((wc[w2] >> 4) & 0x0f0f0f0fu) | (wd[w2] & 0xf0f0f0f0u);
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                const uint32_t sel = 0x7604u | ((uint32_t)b << 4);
                                const uint32_t a0 = ldsp32(prmt(ev_ab, lutlane, sel));
                                const uint32_t a1 = ldsp32(prmt(od_ab, lutlane, sel));
                                const uint32_t a2 = ldsp32(prmt(ev_cd, lutlane, sel));
                                const uint32_t a3 = ldsp32(prmt(od_cd, lutlane, sel));
                                mma16816(acc[4 * w2 + b], a0, a1, a2, a3, pb0, pb1);
                            }
                        }
                    } else {
                        const uint32_t vg = vt + (uint32_t)gam * 2048u;
                        const uint32_t xa = ldsp32(vg + vA_off);
                        const uint32_t xb = ldsp32(vg + vB_off);
                        const uint32_t xc = ldsp32(vg + vA_off + 1024u);
                        const uint32_t xd = ldsp32(vg + vB_off + 1024u);
                        // As in the 4-bit form: byte b of `ev` = (low nibble of token A, low nibble of token B), `od` the high
                        // nibbles; the table turns it into the (A, B) pairs of two coordinates, which are two rows of the operand.
                        const uint32_t ev_ab = (xa & 0x0f0f0f0fu) | ((xb << 4) & 0xf0f0f0f0u);
                        const uint32_t od_ab = ((xa >> 4) & 0x0f0f0f0fu) | (xb & 0xf0f0f0f0u);
                        const uint32_t ev_cd = (xc & 0x0f0f0f0fu) | ((xd << 4) & 0xf0f0f0f0u);
                        const uint32_t od_cd = ((xc >> 4) & 0x0f0f0f0fu) | (xd & 0xf0f0f0f0u);
#pragma unroll
                        for (int bb = 0; bb < 4; ++bb) {
                            const uint32_t sel = 0x7604u | ((uint32_t)bb << 4);
                            const uint2 eab = ldsp64(prmt(ev_ab, lutlane, sel));
                            const uint2 ecd = ldsp64(prmt(ev_cd, lutlane, sel));
                            const uint2 oab = ldsp64(prmt(od_ab, lutlane, sel));
                            const uint2 ocd = ldsp64(prmt(od_cd, lutlane, sel));
                            mma16816(acc[2 * bb], eab.x, eab.y, ecd.x, ecd.y, pb0, pb1);
                            mma16816(acc[2 * bb + 1], oab.x, oab.y, ocd.x, ocd.y, pb0, pb1);
                        }
                    }
                }
            };
            if (!TQ_DBG(1)) {
                if (full) tile_body(std::true_type{});
                else tile_body(std::false_type{});
            }
            TQ_STAMP(5);
            if (TQ_DBG(1)) {  // timing experiments: the copies without the arithmetic
                wait_part(0);
                release_part(0);
                wait_part(1);
            }
            release_part(1);
            ++consumed;
            if (BITS == 2) {
                if (++s_idx == S) {
                    s_idx = 0;
                    s_par ^= 1u;
                }
            }
        }

        TQ_STAMP(12);  // (zero-length marker: everything up to here went to the tile stamps)
        // ================= end of segment: publish the partial, maybe merge =================
        const int slot = wid + g;
        float* const part_base = p.partials + (PERSIST ? (size_t)layer * (size_t)p.part_layer_stride : (size_t)0);
        if (!TQ_DBG(8)) {
            float lsum[NE];  // per lane over its own token rows: sum over the eight row lanes
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                lsum[e] = l_run[e];
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) lsum[e] += __shfl_xor_sync(0xffffffffu, lsum[e], o);
            }
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const int hq = NE * t4 + e;
                if (hq < grp) {
                    float* dst = part_base + ((size_t)slot * p.H + (size_t)head * grp + hq) * PART_STRIDE;
                    if (gl == 0) {
                        dst[HEAD_DIM] = m_run[e];
                        dst[HEAD_DIM + 1] = lsum[e];
                    }
                    auto sum = [&](int b, int row) { return PAIR ? acc[b][2 * row] + acc[b][2 * row + 1] : acc[b][2 * row + e]; };
#pragma unroll
                    for (int b2 = 0; b2 < 4; ++b2)
                        *reinterpret_cast<float4*>(dst + 16 * gl + 4 * b2) = make_float4(sum(2 * b2, 0), sum(2 * b2, 1), sum(2 * b2 + 1, 0), sum(2 * b2 + 1, 1));
                }
            }
        }
        if (TQ_DBG(4)) { ++g; continue; }
        if constexpr (PUBLISH) {  // the partials are merged by a launch of its own
            ++g;
            continue;
        }
        // number of workers that hold a part of sequence g: owners of the sequence's first and last tile
        const int first_w = (int)(((long long)(ts_g + 1) * W - 1) / N);
        const int last_w = (int)(((long long)ts_g1 * W - 1) / N);
        const int parts = last_w - first_w + 1;
        group_barrier(group, gthreads);  // every warp's partial is written (happens-before the fence below)
        uint32_t is_last = 1u;
        if (parts > 1) {
            if (gtid == 0) {
                __threadfence();  // cumulative: orders the whole worker's partials before the ticket
                const int old = atomicAdd(p.tickets + g, 1);
                const uint32_t flag = (old == parts - 1) ? 1u : 0u;
                if (flag) {
                    p.tickets[g] = 0;  // everybody has arrived: leave the ticket ready for the next launch
                }
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(ctrl_s), "r"(flag) : "memory");
            }
            group_barrier(group, gthreads);
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(is_last) : "r"(ctrl_s) : "memory");
        }
        if (is_last) {
            const int H = p.H;
            // where row vh of this sequence's output goes (null: nowhere)
            auto out_row = [&](int vh) -> __half* {
                if (vh >= H) return nullptr;
                return p.out + (size_t)g * p.q_dim + (size_t)vh * HEAD_DIM;
            };
            // optional copy of the results before their rounding to fp16
            auto out_row_f32 = [&](int vh) -> float* {
                if (!p.out_f32 || vh >= H) return nullptr;
                return p.out_f32 + ((size_t)g * H + (size_t)vh) * HEAD_DIM;
            };
            merge_sequence<Hkv>(p.partials + (size_t)(first_w + g) * H * PART_STRIDE, parts, H, merge_s, p.rotation_t, head, lane,
                                group, gthreads, out_row, out_row_f32);
        }
        ++g;
    }
    }

#ifdef TQ_TIMING_SWITCHES
    if (p.stamps && lane == 0) {
        TQ_STAMP(6);
        for (int i = 0; i < 15; ++i) atomicAdd(p.stamps + i, (unsigned long long)stamp_acc[i]);
        atomicAdd(p.stamps + 15, 1ull);
    }
#endif
    // A warp that gave up on a wait may still have copies in flight: give them a bounded chance to land
    // before the CTA (and its shared memory) goes away.
    if (!COPIER && dead) {
        for (int n = consumed; n < consumed + S && n < (int)(hi - lo) * n_layers; ++n) {
            mbar_wait_bounded(bar0 + 16u * (uint32_t)(n % S), (uint32_t)(n / S) & 1u, 1u << 16);
            mbar_wait_bounded(bar0 + 16u * (uint32_t)(n % S) + 8u, (uint32_t)(n / S) & 1u, 1u << 16);
        }
    }
}

// ---- merge of the partials that modes 1 and 2 publish -----------------------------------------------------------------
struct MergeParams {
    const float* partials;       // [layers][workers + G][H][PART_STRIDE]
    const int* table;            // tile table [G + 1], then {workers that took part, total tiles}
    const __half* rotation_t;
    __half* out;                 // [layers][G][q_dim]
    float* out_f32;              // optional [layers][G][H][128]
    long long part_layer_stride; // floats
    long long q_layer_stride;    // halves
    int G, H, q_dim;
    int rotated_out;             // 1: leave the results in rotated space (the consumer's weights carry R^T)
};

// Merge of a whole step's partials: one CTA of 8 warps per (sequence, layer), two heads per warp.
__global__ void __launch_bounds__(256) merge_partials_kernel(const MergeParams p) {
    __shared__ __align__(16) uint8_t merge_buf[RegionA::MERGE_GROUP_BYTES];
    pdl_wait();  // the partials and the table come from the previous kernel in the stream
    const int g = blockIdx.x, layer = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long t0 = p.table[g], t1 = p.table[g + 1], W = p.table[p.G + 1], N = p.table[p.G + 2];
    if (N <= 0 || W <= 0) return;
    // owners of the sequence's first and last tile: worker w holds the tiles [w * N / W, (w + 1) * N / W)
    const int first_w = (int)(((t0 + 1) * W - 1) / N);
    const int last_w = (int)((t1 * W - 1) / N);
    const int parts = last_w - first_w + 1;
    const int H = p.H;
    auto out_row = [&](int vh) -> __half* {
        if (vh >= H) return nullptr;
        return p.out + (size_t)layer * (size_t)p.q_layer_stride + (size_t)g * p.q_dim + (size_t)vh * HEAD_DIM;
    };
    auto out_row_f32 = [&](int vh) -> float* {
        if (!p.out_f32 || vh >= H) return nullptr;
        return p.out_f32 + (((size_t)layer * p.G + (size_t)g) * H + (size_t)vh) * HEAD_DIM;
    };
    merge_sequence<8>(p.partials + (size_t)layer * (size_t)p.part_layer_stride + (size_t)(first_w + g) * H * PART_STRIDE,
                      parts, H, smem_u32(merge_buf), p.rotation_t, warp, lane, 0, 256, out_row, out_row_f32, p.rotated_out != 0);
}

// The merge of one layer's partials (mode 1), the tail of that layer: bound by latency.  One CTA per (sequence, 8 heads), a warp per
// head, its parts' loads in flight together.  Under the attention's last tiles, before the wait: R's fragments and which workers had
// a part, from the positions (which that launch does not write).  Both may be the work of a launch shortly before: the attention lets this one
// start behind its own wait, when layer_prep_kernel, which transposes a caller's R, and all before that have finished; the loads pass
// by L1, in which an SM may still have what it read in the layer before.
// From the wait to the end 2.4 to 3.1 us (32 x 8192 tokens, 32 heads); by the last arriving worker inside the attention 5.6.
// PER_SM: with 141 registers one CTA fills an SM, which is the fastest where that is enough (32 x 8192 tokens, 2-bit, 58.3 us a layer, with 128
// registers 59.1) and a queue where there are many sequences: longer than the attention at 1000 x 100 tokens, 73 us of a layer's 140.6;
// with room for two 113.1, 128 x 300 32.6 -> 29.2.
struct MergeLayerParams {
    const float* partials;       // [workers + G][H][PART_STRIDE]
    const int* positions;        // device [G] or null: pos_value
    const __half* rotation_t;
    __half* out;                 // [G][q_dim]
    float* out_f32;              // optional [G][H][128]
    int pos_value, G, H, q_dim;
    int workers;                 // workers of the attention launch
};
// HEADS = 1: a CTA per (sequence, head) instead, an eighth of its parts for every warp: for few sequences, which are cut into many parts
// each (launch_merge_layer, tq_host.cuh).
constexpr int MERGE_WARPS = 8;
template <int HEADS, int PER_SM>
__global__ void __launch_bounds__(MERGE_WARPS * 32, PER_SM) merge_layer_kernel(const MergeLayerParams p) {
    static_assert(HEADS == 1 || HEADS == MERGE_WARPS, "a warp per head, or all warps for one");
    constexpr bool SPLIT = HEADS == 1;
    __shared__ __align__(16) __half a_op[2 * MERGE_WARPS * MERGE_ROW];  // rows 0-7: high parts, 8-15: low parts (SPLIT: rows 0 and 8 alone are used)
    __shared__ int sums[2][MERGE_WARPS];
    __shared__ float4 acc_s[SPLIT ? MERGE_WARPS : 1][32];
    __shared__ float2 ml_s[SPLIT ? MERGE_WARPS : 1];
    pdl_launch_dependents();
    const int g = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane >> 2, t4 = lane & 3;
    const int h = HEADS * (int)blockIdx.y + (SPLIT ? 0 : warp);
    // out[h][d] = sum_k a[h][k] R[k][d]: B fragments of the column blocks `warp` and `warp + 8`
    uint4 bf[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int m = 0; m < 4; ++m)  // (step (m, e) of lane t4 covers k = 32m + 8*t4 + 4e .. +3, on both sides)
            bf[i][m] = ldg128_l2(reinterpret_cast<const uint4*>(p.rotation_t + (size_t)(8 * (warp + MERGE_WARPS * i) + gl) * HEAD_DIM) + t4 + 4 * m);
    auto tiles_of = [&](int i) {
        const int pos = p.positions ? __ldcg(p.positions + i) : p.pos_value;
        return ((pos < 0 ? 0 : pos) + TILE_TOKENS) / TILE_TOKENS;
    };
    int before = 0, all = 0;  // tiles before sequence g, of all sequences
    for (int i = threadIdx.x; i < p.G; i += MERGE_WARPS * 32) {
        const int n = tiles_of(i);
        all += n;
        before += i < g ? n : 0;
    }
    const int own = tiles_of(g);
    all = __reduce_add_sync(0xffffffffu, all);
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) {
        sums[0][warp] = all;
        sums[1][warp] = before;
    }
    __syncthreads();
    all = before = 0;
#pragma unroll
    for (int w = 0; w < MERGE_WARPS; ++w) {
        all += sums[0][w];
        before += sums[1][w];
    }
    // owners of the sequence's first and last tile, as in the attention kernel's cut of the list
    const long long W = attention_workers(p.workers, all, p.G);
    const int first_w = (int)(((long long)(before + 1) * W - 1) / all);
    const int all_parts = (int)(((long long)(before + own) * W - 1) / all) - first_w + 1;
    const int part_lo = SPLIT ? all_parts * warp / MERGE_WARPS : 0, parts = SPLIT ? all_parts * (warp + 1) / MERGE_WARPS - part_lo : all_parts;
    const size_t pstride = (size_t)p.H * PART_STRIDE;
    const float* const part0 = p.partials + ((size_t)(first_w + g) * p.H + h) * PART_STRIDE + (size_t)part_lo * pstride;
    pdl_wait();
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (h < p.H) {
        constexpr int FLIGHT = 16;
        float M = -1e30f, Z = 0.0f;
        for (int j0 = 0; j0 < parts; j0 += FLIGHT) {
            const int n = parts - j0;
            float2 ml = make_float2(-1e30f, 0.0f);
            if (lane < FLIGHT && lane < n) ml = __ldcg(reinterpret_cast<const float2*>(part0 + (size_t)(j0 + lane) * pstride + HEAD_DIM));
            float4 v[FLIGHT];
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j)
                v[j] = j < n ? __ldcg(reinterpret_cast<const float4*>(part0 + (size_t)(j0 + j) * pstride) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            float Mn = ml.x;
#pragma unroll
            for (int o = FLIGHT / 2; o > 0; o >>= 1) Mn = fmaxf(Mn, __shfl_xor_sync(0xffffffffu, Mn, o));
            Mn = fmaxf(M, __shfl_sync(0xffffffffu, Mn, 0));
            const float e = lane < FLIGHT && lane < n ? ex2_approx(ml.x - Mn) : 0.0f, f = ex2_approx(M - Mn);
            float z = ml.y * e;
#pragma unroll
            for (int o = FLIGHT / 2; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            Z = Z * f + __shfl_sync(0xffffffffu, z, 0);
            M = Mn;
            a.x *= f; a.y *= f; a.z *= f; a.w *= f;
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j) {
                const float wj = __shfl_sync(0xffffffffu, e, j);
                a.x = fmaf(wj, v[j].x, a.x); a.y = fmaf(wj, v[j].y, a.y);
                a.z = fmaf(wj, v[j].z, a.z); a.w = fmaf(wj, v[j].w, a.w);
            }
        }
        if constexpr (SPLIT) {  // the warps' shares meet in shared memory, in their order
            acc_s[warp][lane] = a;
            if (lane == 0) ml_s[warp] = make_float2(M, Z);
            __syncthreads();
            M = ml_s[0].x;
#pragma unroll
            for (int w = 1; w < MERGE_WARPS; ++w) M = fmaxf(M, ml_s[w].x);
            a = make_float4(0.f, 0.f, 0.f, 0.f);
            Z = 0.0f;
#pragma unroll
            for (int w = 0; w < MERGE_WARPS; ++w) {
                const float f = ex2_approx(ml_s[w].x - M);
                const float4 v = acc_s[w][lane];
                Z = fmaf(ml_s[w].y, f, Z);
                a.x = fmaf(v.x, f, a.x); a.y = fmaf(v.y, f, a.y); a.z = fmaf(v.z, f, a.z); a.w = fmaf(v.w, f, a.w);
            }
        }
        const float inv = 1.0f / (Z + 1e-8f);
        a.x *= inv; a.y *= inv; a.z *= inv; a.w *= inv;
    }
    if (!SPLIT || warp == 0) {
        *reinterpret_cast<uint2*>(a_op + warp * MERGE_ROW + 4 * lane) = make_uint2(pack_half2(a.x, a.y), pack_half2(a.z, a.w));
        *reinterpret_cast<uint2*>(a_op + (warp + MERGE_WARPS) * MERGE_ROW + 4 * lane) = make_uint2(pack_low_half2(a.x, a.y), pack_low_half2(a.z, a.w));
    }
    __syncthreads();
    float c[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[i][0][e] = c[i][1][e] = 0.0f;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const uint4 hi = *reinterpret_cast<const uint4*>(a_op + gl * MERGE_ROW + 32 * m + 8 * t4);
        const uint4 lo = *reinterpret_cast<const uint4*>(a_op + (gl + MERGE_WARPS) * MERGE_ROW + 32 * m + 8 * t4);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mma16816(c[i][0], hi.x, lo.x, hi.y, lo.y, bf[i][m].x, bf[i][m].y);
            mma16816(c[i][1], hi.z, lo.z, hi.w, lo.w, bf[i][m].z, bf[i][m].w);
        }
    }
    const int ho = HEADS * (int)blockIdx.y + gl;
    if (gl >= HEADS || ho >= p.H) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float o0 = (c[i][0][0] + c[i][1][0]) + (c[i][0][2] + c[i][1][2]), o1 = (c[i][0][1] + c[i][1][1]) + (c[i][0][3] + c[i][1][3]);
        const size_t at = (size_t)ho * HEAD_DIM + 8 * (warp + MERGE_WARPS * i) + 2 * t4;
        *reinterpret_cast<__half2*>(p.out + (size_t)g * p.q_dim + at) = __floats2half2_rn(o0, o1);
        if (p.out_f32) *reinterpret_cast<float2*>(p.out_f32 + (size_t)g * p.H * HEAD_DIM + at) = make_float2(o0, o1);
    }
}

}  // namespace tq
