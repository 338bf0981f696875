// Decode attention of small batches, one launch per layer: a thread-block cluster per (sequence, KV head), sm_100a.
//
// The streaming kernel (tq_attention.cuh) is built for caches that take many microseconds to read; a layer of a small
// batch (4 sequences x 600 tokens: 2.6 MB) costs it 19 us, nearly all of it start-up: tile table, ring fill, tensor-map
// round trips, a 16-row append on one worker, per-sequence tickets and a merge through global memory.  Here the work is
// cut so that the longest dependent chain is short:
//   * a cluster of S CTAs (1 to 16, chosen by the host) owns one sequence and one KV head with up to 8 of its query heads
//     (more query heads: further clusters).  Its 8 * S warps (8 * (S - 1) where a CTA is the new token's alone, see below) take the
//     sequence's tiles of 32 tokens, or of 16 where that leaves each warp one, in turn, first all CTAs' warp 0, then warp 1 ..., with plain 16- and 8-byte loads that land in registers in fragment order: no shared-memory
//     ring, no table of tiles, any head layout, ragged slots and shared prefixes by row arithmetic alone.
//   * codes become fp16 through a shared-memory table with a private column per lane (one entry per code byte at 4-bit,
//     per nibble at 2-bit); table and R are staged before griddepcontrol.wait, i.e. under the previous kernel's tail, and
//     so are, in a chain of layers, the cache rows of the warp's first tile.
//   * positions and R are requested first, the table is written while they are on their way; K rows of a single tile per warp are
//     looked up there too, so that only products are left once the queries have arrived.
//   * the step's token is quantised by the cluster's last CTA (its owner): its raw K and V vectors are two more
//     rows of the A operand of the query rotation (rows 8 and 9, otherwise idle), scaled by 1/norm afterwards; a
//     coordinate within CD_MARGIN of a decision bound is recomputed with the reference's exact fp32 chain, as in
//     tq_prefill_tc.cuh, so the stored bytes are the reference's.  It is in no tile: its score is a dot product of one warp per
//     head, its value row enters the CTA's sum of the warps' results, in fp32; it goes to the cache at the very end, so that no
//     barrier has to wait for a global write.  In clusters of four CTAs or more the owner takes nothing else: quantising costs no
//     more time than the others' tiles then.
//   * S^T = K Q^T and O^T += V^T P^T on mma.sync with tokens / coordinates in the M dimension as in the streaming kernel.
//     The warps' partial results meet in shared memory; every CTA normalises its own and multiplies it by R (fp16 high
//     parts as rows 0-7 of the A operand, low parts as rows 8-15) and sends every other CTA its share of the output coordinates with asynchronous stores into that CTA's
//     shared memory, counted by that CTA's mbarrier; a CTA adds up its share, weighted, when all of it has arrived.  (A
//     cluster barrier in that place costs 0.8 us more: its release waits for the remote stores to be acknowledged.)
//   * Head layouts that the streaming kernels do not serve took a kernel with fp32 queries, centroids and weights.  Here they are
//     fp16 high + low parts (EXACT: three products for one, a second table): the results' error is that kernel's.  With the high
//     parts alone it was 2.9 (4-bit), 3.8 (2-bit) and 1.12 (fp16 rows) times as large.
// Bound by latency: one round trip for the inputs, the rotation, one tile, three CTA barriers, one trip across the cluster, about
// 700 + 800 + 1500 + 600 + 900 + 900 + 1500 cycles.  With the token as a row of the last tile (its CTA 1600 cycles behind the others),
// divisions by the cluster's size in the exchange, the low parts' products with R of their own and the look-ups behind the queries:
// 1 layer of 4 x 612 tokens 7.0 us, now 5.9; 28 layers of 1 x 1500 188 us, now 157 with fewer CTAs (4-bit, 16/8 heads, one call after
// the other, caches from HBM; 8 layers, which stay in L2, 5.3 us each).
#pragma once

#include <type_traits>

#include "tq_attention.cuh"

namespace tq {

constexpr int CD_WARPS = 8;
constexpr int CD_THREADS = CD_WARPS * 32;
constexpr int CD_MAX_CLUSTER = 16;
constexpr int CD_HEADS = 8;                    // query heads of a KV head per cluster (the N side of the score product)
constexpr float CD_MARGIN = 1.7e-5f;           // see tq_prefill_tc.cuh
// Fixed shared addresses (relative to the CTA's window).  The table has one entry per 256 bytes, so that one PRMT makes a
// look-up address from the packed word; the entry itself is 128 bytes (32 lanes).  At 4-bit the 256 unused halves hold R.
constexpr uint32_t CD_LUT_ABS = 0x8000u;
constexpr uint32_t CD_MAX_BASE = 0x480u;       // dynamic shared memory starts at or below this address (1 KB is the driver's)

struct ClusterDecodeParams {
    const uint8_t* ck;           // packed codes [rows][kvp], or fp16 rows [rows][kv_dim] (BITS = 0)
    const uint8_t* cv;
    const __half* kn;
    const __half* vn;
    const __half* q;             // [G][q_dim], not rotated
    const __half* new_k;         // [G][kv_dim] or null: nothing is appended
    const __half* new_v;
    const __half* rotation;      // R row-major
    __half* out;                 // [G][q_dim]
    float* out_f32;              // optional [G][H][128]
    const int* positions;        // device [G] or null
    const long long* row_base;   // [G] or null: g * max_seq_len
    const int* seq_capacity;     // [G] or null: capacity_rows
    const long long* prefix_base;  // shared prefixes, as in AttnParams
    const int* prefix_tiles;
    int* status;                 // or null
    int pos_value, max_seq_len, capacity_rows;
    int G, H, Hkv, q_dim;
    // Several layers in one launch (a decode step that has all layers' queries, keys and values at once): grid.z = layers * G,
    // the pointers above are the first layer's, the others lie these strides behind (bytes of the code arrays, halves elsewhere).
    long long code_layer_stride, norm_layer_stride, q_layer_stride, kv_layer_stride;
    int head_blocks;             // clusters per KV head: ceil(query heads per KV head / 8)
    int early;                   // as in AttnParams: positions and old rows may be read before the previous kernel has finished
    int static_rotation;         // R is not written by any kernel of the stream: staged before the wait
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// (volatile: the instruction is undefined for a rank outside the cluster, so it must not be executed ahead of its condition)
__device__ __forceinline__ uint32_t map_shared(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Eight bytes to another CTA's shared memory, counted by the mbarrier `bar` of that CTA.
__device__ __forceinline__ void st_async_f32x2(uint32_t addr, float a, float b, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr), "r"(__float_as_uint(a)),
                 "r"(__float_as_uint(b)), "r"(bar) : "memory");
}

// Loads that stay behind griddepcontrol.wait (volatile: never moved across it), zero where `on` is 0.
__device__ __forceinline__ uint4 lds128_if(uint32_t addr, bool on) { return on ? lds128(addr) : make_uint4(0u, 0u, 0u, 0u); }
__device__ __forceinline__ uint4 ldg128_if(const void* src, bool on) {
    uint4 r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
                 "@p ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "=&r"(r.x), "=&r"(r.y), "=&r"(r.z), "=&r"(r.w) : "l"(src), "r"((uint32_t)on));
    return r;
}
__device__ __forceinline__ uint2 ldg64_if(const void* src, bool on) {
    uint2 r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t@p ld.global.v2.u32 {%0, %1}, [%2];\n\t}"
                 : "=&r"(r.x), "=&r"(r.y) : "l"(src), "r"((uint32_t)on));
    return r;
}
__device__ __forceinline__ uint32_t ldg32_if(const void* src, bool on) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t@p ld.global.u32 %0, [%1];\n\t}"
                 : "=&r"(r) : "l"(src), "r"((uint32_t)on));
    return r;
}
__device__ __forceinline__ __half ldg_half_if(const __half* src, bool on) {
    unsigned short r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u16 %0, 0;\n\t@p ld.global.u16 %0, [%1];\n\t}"
                 : "=&h"(r) : "l"(src), "r"((uint32_t)on));
    return __ushort_as_half(r);
}

// A warp's partial result, or that of a warp without tiles: maximum, sum, one or four coordinates.
__device__ __forceinline__ void part_if(uint32_t ml, uint32_t acc, bool on, float& m, float& l, float (&a)[4]) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %8, 0;\n\tmov.f32 %0, 0fF149F2CA;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\t"
                 "mov.f32 %3, 0f00000000;\n\tmov.f32 %4, 0f00000000;\n\tmov.f32 %5, 0f00000000;\n\t"
                 "@p ld.shared.v2.f32 {%0, %1}, [%6];\n\t@p ld.shared.v4.f32 {%2, %3, %4, %5}, [%7];\n\t}"
                 : "=&f"(m), "=&f"(l), "=&f"(a[0]), "=&f"(a[1]), "=&f"(a[2]), "=&f"(a[3]) : "r"(ml), "r"(acc), "r"((uint32_t)on));
}
__device__ __forceinline__ void part_if(uint32_t ml, uint32_t acc, bool on, float& m, float& l, float (&a)[1]) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.f32 %0, 0fF149F2CA;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\t"
                 "@p ld.shared.v2.f32 {%0, %1}, [%3];\n\t@p ld.shared.f32 %2, [%4];\n\t}"
                 : "=&f"(m), "=&f"(l), "=&f"(a[0]) : "r"(ml), "r"(acc), "r"((uint32_t)on));
}

// Shared memory of a CTA below the table, from the dynamic base: the small arrays and, when they fit, the warps' partial
// results (otherwise those lie behind table and R).
struct CdSmem {
    static constexpr uint32_t NEW_OFF = 0;                               // new token: K codes [128 B], V codes [128 B]
    static constexpr uint32_t RAW_OFF = 256;                             // new token: K, V as they arrived, [2][128] fp16
    static constexpr uint32_t WP_OFF = RAW_OFF + 512;                    // warp sums of squares [2][4] fp32
    static constexpr uint32_t NN_OFF = WP_OFF + 32;                      // K and V norm of the new token, fp32 values of the stored halves
    static constexpr uint32_t Q_OFF = NN_OFF + 32;                       // rotated queries [8][136] fp16, later merge operand high part
    static constexpr uint32_t LO_OFF = Q_OFF + CD_HEADS * MERGE_ROW * 2; // merge operand low part
    static constexpr uint32_t BND_OFF = LO_OFF + CD_HEADS * MERGE_ROW * 2;  // decision bounds, fp32, between -inf and +inf
    static constexpr uint32_t BAR_OFF = BND_OFF + 80;                    // mbarrier of what the cluster's CTAs send
    static constexpr uint32_t CENT_OFF = BND_OFF + 96;                   // centroids, fp32
    static constexpr uint32_t NS_OFF = CENT_OFF + 64;                    // new token: its score with each query head
    static constexpr uint32_t CP_OFF = NS_OFF + 32;                      // [CTA][head][this CTA's share of the coordinates] fp32, from all CTAs
    static constexpr uint32_t MZ_OFF = CP_OFF + CD_HEADS * HEAD_DIM * 4; // [CTA][head] maximum and sum
    static constexpr uint32_t WARP_OFF = MZ_OFF + CD_MAX_CLUSTER * CD_HEADS * 8;  // the warps' partial results [8][heads][PART_STRIDE] fp32
};
__host__ __device__ constexpr uint32_t cd_low_table(int bits) { return bits == 4 ? 0x10000u : 0x1000u + 0x8000u; }  // the low parts' table, from the first one
__host__ __device__ constexpr uint32_t cd_table_bytes(int bits, bool exact) {                                       // with R
    return bits == 0 ? 0u : cd_low_table(bits) + (!exact ? 0u : bits == 4 ? 0x10000u : 0x1000u);
}
// (the host: bytes of dynamic shared memory for `heads` query heads per cluster, counted from address 0: what the driver
// reserves at the start is slack)
inline size_t cd_smem_bytes(int bits, int heads, bool exact) {
    const uint32_t warps = (uint32_t)CD_WARPS * heads * PART_STRIDE * 4u;
    uint32_t top = CD_LUT_ABS + cd_table_bytes(bits, exact);
    if (CD_MAX_BASE + CdSmem::WARP_OFF + warps > CD_LUT_ABS) top += warps;
    return (size_t)top;
}

// MB: 16-token blocks per tile (2 for throughput, 1 where every warp gets a single tile anyway and its latency counts)
// HOST: q, new_k, new_v (and out) are pinned host memory: every byte of them is fetched once per CTA, not once per warp
// EXACT: rotated queries, centroids and weights as fp16 high + low parts (see above)
template <int BITS, int MB, bool HOST, bool EXACT>
__global__ void __launch_bounds__(CD_THREADS, EXACT && BITS != 0 ? 1 : 2) cluster_decode_kernel(const ClusterDecodeParams p_in) {
    extern __shared__ __align__(1024) uint8_t cd_smem[];
    ClusterDecodeParams p = p_in;
    constexpr int BPH = BITS == 0 ? 256 : (BITS == 4 ? 64 : 32);  // bytes of a head's row
    constexpr int TT = 16 * MB;                                   // tokens per tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gl = lane >> 2, t4 = lane & 3;
    const uint32_t rank = cluster_ctarank(), S = cluster_nctarank();
    const int kvh = blockIdx.y / p.head_blocks, hblk = blockIdx.y - kvh * p.head_blocks;
    const int layer = (int)blockIdx.z / p.G, g = (int)blockIdx.z - layer * p.G;
    if (layer > 0) {
        p.ck += layer * p.code_layer_stride; p.cv += layer * p.code_layer_stride;
        p.kn += layer * p.norm_layer_stride; p.vn += layer * p.norm_layer_stride;
        p.q += layer * p.q_layer_stride; p.out += layer * p.q_layer_stride;
        p.new_k += layer * p.kv_layer_stride; p.new_v += layer * p.kv_layer_stride;
        if (p.out_f32) p.out_f32 += (long long)layer * p.G * p.H * HEAD_DIM;
    }
    const int grp = p.H / p.Hkv;
    const int nh = min(CD_HEADS, grp - CD_HEADS * hblk);  // query heads of this cluster
    const int head0 = kvh * grp + CD_HEADS * hblk;
    const int kvp = p.Hkv * BPH;

    // (in a cluster the upper byte of a shared address is the CTA's rank: the fixed addresses are relative to it)
    const uint32_t window = smem_u32(cd_smem) & 0xff000000u;
    const uint32_t base = (smem_u32(cd_smem) + 127u) & ~127u;
    const uint32_t lut_s = window + CD_LUT_ABS;
    const uint32_t warps_low = base + CdSmem::WARP_OFF;
    const uint32_t warp_bytes = (uint32_t)(CD_WARPS * nh * PART_STRIDE * 4);
    const uint32_t warps_s = warps_low + warp_bytes <= lut_s ? warps_low : lut_s + cd_table_bytes(BITS, EXACT);
    if (base - window > CD_MAX_BASE) {  // the dynamic part does not start where cd_smem_bytes counts on: no CTA of the launch goes on
        if (tid == 0 && p.status) atomicMax(p.status, ST_SMEM_LAYOUT);
        return;
    }
    // R in 16-byte pieces (row, k / 8): eight rows share 128 bytes, rotated by 2 (k / 8) pieces, so that the fragment loads of
    // both products and the exact chains are free of bank conflicts
    constexpr uint32_t RS = BITS == 4 ? 256u : 128u;
    const uint32_t r_s = lut_s + (BITS == 4 ? 128u : 0x1000u);
    auto r_piece = [&](int row, int k8) -> uint32_t { return r_s + (uint32_t)(k8 * 16 + (row >> 3)) * RS + (uint32_t)(((row + 2 * k8) & 7) << 4); };

    // ---- positions, rows, and the cache rows of a tile ----
    const bool owner = p.new_k != nullptr && rank == S - 1u;  // the CTA of the new token
    int pos = 0, cap = 0;
    bool appends = false, pos_ok = false;
    int tile = 0, tile_end = 0, tile_step = 1;  // this warp's tiles
    int n_act = 0;                              // warps of this CTA that have any
    int lim = 0;                                // cached tokens: those below lim
    long long row0 = 0, prow0 = 0;
    int ptok = 0;  // tokens below ptok are read from the shared prefix
    uint2 row0_w = make_uint2(0u, 0u), prow0_w = make_uint2(0u, 0u);
    auto fetch_position = [&]() {  // (volatile loads, all in flight together before anything waits for one)
        pos = (int)ldg32_if(p.positions + g, p.positions != nullptr);
        cap = (int)ldg32_if(p.seq_capacity + g, p.seq_capacity != nullptr);
        row0_w = ldg64_if(p.row_base + g, p.row_base != nullptr);
        ptok = (int)ldg32_if(p.prefix_tiles + g, p.prefix_tiles != nullptr);
        prow0_w = ldg64_if(p.prefix_base + g, p.prefix_tiles != nullptr);
    };
    auto use_position = [&]() {
        if (!p.positions) pos = p.pos_value;
        if (!p.seq_capacity) cap = p.capacity_rows;
        pos_ok = pos >= 0 && (cap <= 0 || pos < cap);
        int L = (pos < 0 ? 0 : pos) + 1;
        if (cap > 0 && L > cap) L = cap;  // a position outside its slot is reported; rows outside the slot are not read
        appends = p.new_k != nullptr && pos_ok;
        lim = appends ? L - 1 : L;        // (the row this very step writes is never read from the cache)
        const int W = p.new_k != nullptr && S >= 4u ? (int)S - 1 : (int)S;  // CTAs that take the cached tokens
        tile_end = (int)rank < W ? (lim + TT - 1) / TT : 0;
        tile = warp * W + (int)rank;
        tile_step = CD_WARPS * W;
        for (int w = 0, t = (int)rank; w < CD_WARPS && t < tile_end; ++w, t += W) n_act = w + 1;
        auto join = [](uint2 w) { return (long long)((unsigned long long)w.y << 32 | w.x); };
        row0 = p.row_base ? join(row0_w) : (long long)g * p.max_seq_len;
        ptok *= TILE_TOKENS;
        prow0 = join(prow0_w);
    };
    constexpr int KV4 = BITS == 0 ? 4 : 1, VV4 = BITS == 0 ? 2 : 1;  // 16-byte pieces per lane and row
    uint4 kw[MB][2][KV4];                      // K rows gl, gl + 8 of a block: the lane's 32 coordinates 32 t4 ..
    uint4 vw[MB][4][VV4];                      // V rows 2 t4, 2 t4 + 1, 2 t4 + 8, 2 t4 + 9: the lane's 16 coordinates 16 gl ..
    __half kn_h[MB][2], vn_h[MB][2];           // norms of rows gl, gl + 8
    auto token_row = [&](int t) -> size_t { return (size_t)(t < ptok ? prow0 + t : row0 + t); };
    // rows at or past `lim` are not read: they count as zero codes with zero norm, and are masked anyway
    auto load_k = [&](int tile, int lim) {
#pragma unroll
        for (int b = 0; b < MB; ++b)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = tile * TT + 16 * b + 8 * r + gl;
                const bool on = t < lim;
                const size_t row = token_row(t);
                const uint8_t* src = p.ck + row * kvp + (size_t)kvh * BPH;
                if constexpr (BITS == 4) {
                    kw[b][r][0] = ldg128_if(src + 16 * t4, on);
                } else if constexpr (BITS == 2) {
                    const uint2 w = ldg64_if(src + 8 * t4, on);
                    kw[b][r][0].x = w.x; kw[b][r][0].y = w.y;
                } else {
#pragma unroll
                    for (int i = 0; i < KV4; ++i) kw[b][r][i] = ldg128_if(src + 64 * t4 + 16 * i, on);
                }
                if constexpr (BITS != 0) kn_h[b][r] = ldg_half_if(p.kn + row * p.Hkv + kvh, on);
            }
    };
    auto load_v = [&](int tile, int lim) {
#pragma unroll
        for (int b = 0; b < MB; ++b) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int t = tile * TT + 16 * b + 2 * t4 + (r & 1) + 8 * (r >> 1);
                const bool on = t < lim;
                const uint8_t* src = p.cv + token_row(t) * kvp + (size_t)kvh * BPH;
                if constexpr (BITS == 4) {
                    const uint2 w = ldg64_if(src + 8 * gl, on);
                    vw[b][r][0].x = w.x; vw[b][r][0].y = w.y;
                } else if constexpr (BITS == 2) {
                    vw[b][r][0].x = ldg32_if(src + 4 * gl, on);
                } else {
#pragma unroll
                    for (int i = 0; i < VV4; ++i) vw[b][r][i] = ldg128_if(src + 32 * gl + 16 * i, on);
                }
            }
            if constexpr (BITS != 0) {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int t = tile * TT + 16 * b + 8 * r + gl;
                    vn_h[b][r] = ldg_half_if(p.vn + token_row(t) * p.Hkv + kvh, t < lim);
                }
            }
        }
    };
    auto first_tile = [&]() {
        use_position();
        if (tile < tile_end) {
            load_k(tile, lim);
            load_v(tile, lim);
        }
    };
    const bool staged = BITS == 0 || HOST || p.static_rotation != 0;  // R may be read now (HOST waits for the previous kernel before all else)
    uint4 ru[8];
    auto fetch_rotation = [&]() {
#pragma unroll
        for (int i = 0; i < 8; ++i) ru[i] = ldg128_if(reinterpret_cast<const uint4*>(p.rotation) + tid + CD_THREADS * i, true);
    };
    auto store_rotation = [&]() {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = tid + CD_THREADS * i;
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(r_piece(at >> 4, at & 15)), "r"(ru[i].x), "r"(ru[i].y), "r"(ru[i].z), "r"(ru[i].w) : "memory");
        }
    };

    // Host inputs take longer than all else: they are requested first, one 16-byte piece per thread, and everything else is done while
    // they are on the bus.  (Many CTAs follow each other on an SM; only the first could have started under a previous kernel.  Behind the
    // first rows and the barrier, 28 layers of 16 x 2019 tokens take 420 us instead of 397.)
    const size_t new_at = ((size_t)g * p.Hkv + kvh) * HEAD_DIM;
    uint4 in_w = make_uint4(0u, 0u, 0u, 0u);
    // (fp16 rows: one place where the first rows are requested, before or after the wait -- two places cost registers that
    // the loop needs, and a spilled value read back there comes behind the loads of the next rows: 4 layers of 16 x 1000 tokens 57 us, now 53.6)
    constexpr bool ROWS16 = BITS == 0 && !HOST;
    if (ROWS16 && !p.early) {
        pdl_wait();
        pdl_launch_dependents();
    }
    if constexpr (HOST) {
        pdl_wait();
        pdl_launch_dependents();
        const int r = tid >> 4;
        const uint4* src = r < nh ? reinterpret_cast<const uint4*>(p.q + (size_t)g * p.q_dim + (size_t)head0 * HEAD_DIM) + tid
                                  : reinterpret_cast<const uint4*>((r == nh ? p.new_k : p.new_v) + new_at) + (tid & 15);
        in_w = ldg128_if(src, tid < (nh + (owner ? 2 : 0)) * 16);
    }
    // ---- before the wait: positions and R on their way, table and bounds meanwhile, then the first tile ----
    const bool early = HOST || ROWS16 || p.early != 0;
    if (early) fetch_position();
    if (BITS != 0 && staged) fetch_rotation();
    const uint32_t bar = base + CdSmem::BAR_OFF;
    if (S > 1) {
        if (tid == 0) {
            mbar_init(bar, 1);
            fence_mbar_init();
            mbar_arrive_expect_tx(bar, (uint32_t)nh * (HEAD_DIM * 4u + S * 8u));
        }
        __syncwarp();
        cluster_arrive();  // (the wait comes before the first store to another CTA: it has started then, its barrier is set)
    }
    constexpr int NBND = BITS == 4 ? 15 : 3;
    if (BITS != 0 && tid <= NBND + 1) {
        const float bound = tid == 0 ? -3.4e38f : (tid > NBND ? 3.4e38f : (BITS == 4 ? kBnd4[(tid - 1) & 15] : kBnd2[(tid - 1) & 3]));
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + CdSmem::BND_OFF + 4u * (uint32_t)tid), "f"(bound) : "memory");
    }
    if (BITS != 0 && tid >= 32 && tid < 48)
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + CdSmem::CENT_OFF + 4u * (uint32_t)(tid - 32)), "f"(BITS == 4 ? kCent4[tid & 15] : kCent2[tid & 3]) : "memory");
    constexpr uint32_t LOW = cd_low_table(BITS);
    auto table_entry = [&](uint32_t at, float c0, float c1) {  // four lanes' copies of two centroids
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at), "r"(pack_half2(c0, c1)) : "memory");
        if (EXACT) asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at + LOW), "r"(pack_low_half2(c0, c1)) : "memory");
    };
    if constexpr (BITS == 4) {
        const float lo = kCent4[(tid >> 3) & 15];
#pragma unroll
        for (int i = 0; i < 8; ++i)  // entry (tid >> 3) + 32 i, lanes 4 (tid & 7) .. + 3
            table_entry(lut_s + (uint32_t)((tid >> 3) + 32 * i) * 256u + (uint32_t)(tid & 7) * 16u, lo, kCent4[(tid >> 7) + 2 * i]);
    } else if constexpr (BITS == 2) {
        if (tid < 128) table_entry(lut_s + (uint32_t)(tid >> 3) * 256u + (uint32_t)(tid & 7) * 16u, kCent2[(tid >> 3) & 3], kCent2[tid >> 5]);
    }
    if (BITS != 0 && staged) store_rotation();
    uint32_t lutlane;  // produced behind the barrier that the table waits for: the look-ups, which take it into their address, cannot move above it
    auto after_table = [&]() { asm volatile("mov.u32 %0, %1;" : "=r"(lutlane) : "r"(window | ((uint32_t)lane << 2)) : "memory"); };
    auto lut = [&](uint32_t w, int byte) -> uint32_t {  // the table's entry for a byte of w: two halves
        uint32_t r;
        asm("ld.shared.u32 %0, [%1 + %2];" : "=r"(r) : "r"(prmt(w, lutlane, 0x7604u | ((uint32_t)byte << 4))), "n"(CD_LUT_ABS));
        return r;
    };
    auto lut_low = [&](uint32_t w, int byte) -> uint32_t {  // EXACT: the low parts
        uint32_t r;
        asm("ld.shared.u32 %0, [%1 + %2];" : "=r"(r) : "r"(prmt(w, lutlane, 0x7604u | ((uint32_t)byte << 4))), "n"(CD_LUT_ABS + LOW));
        return r;
    };
    // One tile per warp: the K rows' operands are looked up as soon as the rows are there, in a chain of layers under the previous
    // kernel's tail.
    constexpr bool PRE = BITS != 0 && MB == 1 && !EXACT;
    uint32_t ka[PRE ? 8 : 1][4];
    auto look_up_k = [&]() {
        auto now = [&](uint32_t w, int byte) -> uint32_t {  // (volatile: not behind the wait, where it would be on the critical path)
            uint32_t r;
            asm volatile("ld.shared.u32 %0, [%1 + %2];" : "=r"(r) : "r"(prmt(w, lutlane, 0x7604u | ((uint32_t)byte << 4))), "n"(CD_LUT_ABS));
            return r;
        };
#pragma unroll
        for (int j = 0; j < (PRE ? 8 : 0); ++j) {
            if constexpr (BITS == 4) {
                const uint4 lo4 = kw[0][0][0], hi4 = kw[0][1][0];
                const uint32_t lo = j < 2 ? lo4.x : (j < 4 ? lo4.y : (j < 6 ? lo4.z : lo4.w)), hi = j < 2 ? hi4.x : (j < 4 ? hi4.y : (j < 6 ? hi4.z : hi4.w));
                ka[j][0] = now(lo, 2 * (j & 1)); ka[j][1] = now(hi, 2 * (j & 1));
                ka[j][2] = now(lo, 2 * (j & 1) + 1); ka[j][3] = now(hi, 2 * (j & 1) + 1);
            } else {
                const uint32_t lo = j < 4 ? kw[0][0][0].x : kw[0][0][0].y, hi = j < 4 ? kw[0][1][0].x : kw[0][1][0].y;
                ka[j][0] = now(lo & 0x0f0f0f0fu, j & 3); ka[j][1] = now(hi & 0x0f0f0f0fu, j & 3);
                ka[j][2] = now((lo >> 4) & 0x0f0f0f0fu, j & 3); ka[j][3] = now((hi >> 4) & 0x0f0f0f0fu, j & 3);
            }
        }
    };
    if (early) first_tile();
    if (BITS != 0 && staged) {
        __syncthreads();  // table, R: under the previous kernel's tail too
        after_table();
        if (PRE && early && tile < tile_end) look_up_k();
    }
    if (ROWS16 && p.early) {
        pdl_wait();
        pdl_launch_dependents();
    }
    if constexpr (!HOST && !ROWS16) {
        pdl_wait();
        pdl_launch_dependents();
        if (!early) fetch_position();
        if (!staged) fetch_rotation();
    }

    // ---- queries ----
    uint32_t qb[8][2];  // B fragments of the score product: lane (gl, t4) holds head gl, step j coordinates 32 t4 + 4 j ..
    uint32_t ql[EXACT && BITS != 0 ? 8 : 1][2];  // their low parts
    uint4 qw[4];
    const uint32_t in_s = warps_s;  // host inputs: [nh] queries, K, V, 256 bytes each, where the warps' results will be
    if constexpr (HOST) {
        if (tid < (nh + (owner ? 2 : 0)) * 16)
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(in_s + (uint32_t)tid * 16u), "r"(in_w.x), "r"(in_w.y), "r"(in_w.z), "r"(in_w.w) : "memory");
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int c = BITS == 0 ? 4 * t4 + m : 4 * m + t4;
        const __half* src = p.q + (size_t)g * p.q_dim + (size_t)(head0 + gl) * HEAD_DIM;
        qw[m] = HOST ? lds128_if(in_s + (uint32_t)(gl * 256 + 16 * c), gl < nh) : ldg128_if(src + 8 * c, gl < nh);
    }
    // the owner takes the new token: K and V are rows 8 and 9 of the rotation's A operand
    const int vec = tid >> 7, d = tid & 127;
    uint4 nw[4];
#pragma unroll
    for (int m = 0; m < (BITS != 0 ? 4 : 0); ++m) {
        const bool on = owner && gl < 2;
        nw[m] = HOST ? lds128_if(in_s + (uint32_t)((nh + gl) * 256 + 16 * (4 * m + t4)), on)
                              : ldg128_if((gl == 0 ? p.new_k : p.new_v) + new_at + 8 * (4 * m + t4), on);
    }
    uint2 q4 = make_uint2(0u, 0u);  // fp16 rows: coordinates 4 lane .. of the head whose score with the new token this warp takes
    __half xh = __ushort_as_half((unsigned short)0);
    if (owner) {
        if constexpr (HOST) {
            unsigned short u;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(in_s + (uint32_t)((nh + vec) * 256 + 2 * d)));
            xh = __ushort_as_half(u);
            if (BITS == 0 && CD_WARPS - 1 - warp < nh) q4 = lds64(in_s + (uint32_t)((CD_WARPS - 1 - warp) * 256 + 8 * lane));
        } else {
            xh = ldg_half_if((vec == 0 ? p.new_k : p.new_v) + new_at + d, true);
            if (BITS == 0) q4 = ldg64_if(p.q + (size_t)g * p.q_dim + (size_t)(head0 + CD_WARPS - 1 - warp) * HEAD_DIM + 4 * lane, CD_WARPS - 1 - warp < nh);
        }
    }
    if (!staged) store_rotation();
    if (!HOST && !ROWS16 && !early) first_tile();
    if (owner) {
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(base + CdSmem::RAW_OFF + 2u * (uint32_t)tid), "h"(__half_as_ushort(xh)) : "memory");
        if (!pos_ok && tid == 0 && p.status) atomicMax(p.status, ST_BAD_POSITION);
        if constexpr (BITS != 0) {  // sum of squares in the reference's order (tq_append.cuh)
            const float xv = __half2float(xh);
            float sq = mul_ftz(xv, xv);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sq = add_ftz(sq, __shfl_down_sync(0xffffffffu, sq, off));
            if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + CdSmem::WP_OFF + 4u * (uint32_t)warp), "f"(sq) : "memory");
        }
    }
    // warp sums, raw token; a rotation that was not staged before the wait, and the table; host inputs, which lie where the warps' results
    // will be: in the packed modes the rotation's barrier stands between their last reads and the first result, with fp16 rows only this one
    if (owner || !staged || (HOST && BITS == 0)) __syncthreads();
    if (!staged) after_table();
    if constexpr (BITS != 0) {
        // rotated queries, rot[h][n] = sum_k q[h][k] R[n][k]: warp w takes the coordinate blocks w and w + 8
        float nc[4];  // rows 8 (lanes gl = 0: K) and 9 (gl = 1: V): coordinates 8 warp + 2 t4, + 1, and the same + 64
        float rc[2][2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) rc[i][0][e] = rc[i][1][e] = 0.0f;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            uint4 b4[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) b4[i] = lds128(r_piece(8 * (warp + CD_WARPS * i) + gl, 4 * m + t4));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mma16816(rc[i][0], qw[m].x, nw[m].x, qw[m].y, nw[m].y, b4[i].x, b4[i].y);
                mma16816(rc[i][1], qw[m].z, nw[m].z, qw[m].w, nw[m].w, b4[i].z, b4[i].w);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float c[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) c[e] = rc[i][0][e] + rc[i][1][e];
            const float sc = 0.12751743074602467f;  // log2(e) / sqrt(128)
            const uint32_t q_at = base + CdSmem::Q_OFF + (uint32_t)(gl * MERGE_ROW + 8 * (warp + CD_WARPS * i) + 2 * t4) * 2u;
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(q_at), "r"(pack_half2(c[0] * sc, c[1] * sc)) : "memory");
            if (EXACT)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(q_at + (CdSmem::LO_OFF - CdSmem::Q_OFF)), "r"(pack_low_half2(c[0] * sc, c[1] * sc)) : "memory");
            nc[2 * i] = c[2];
            nc[2 * i + 1] = c[3];
        }
        if (owner) {  // uniform for the CTA
            // one coordinate per lane: lane (gl, t4) takes vector gl & 1, value gl >> 1 of lane (gl & 1, t4)
            const int nv = gl & 1, ni = gl >> 1, from = nv * 4 + t4;
            const float r0 = __shfl_sync(0xffffffffu, nc[0], from), r1 = __shfl_sync(0xffffffffu, nc[1], from);
            const float r2 = __shfl_sync(0xffffffffu, nc[2], from), r3 = __shfl_sync(0xffffffffu, nc[3], from);
            const float raw = ni == 0 ? r0 : (ni == 1 ? r1 : (ni == 2 ? r2 : r3));
            const int nd = 8 * (warp + CD_WARPS * (ni >> 1)) + 2 * t4 + (ni & 1);
            const uint32_t wp = base + CdSmem::WP_OFF + 16u * (uint32_t)nv;
            float w4[4];
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w4[0]), "=f"(w4[1]), "=f"(w4[2]), "=f"(w4[3]) : "r"(wp));
            const float ss = add_ftz(add_ftz(w4[0], w4[2]), add_ftz(w4[1], w4[3]));
            const float t = add_ftz(ss, 1e-12f);
            const float inv = rsqrt_approx_ftz(t);
            float x = mul_ftz(raw, inv);
            if (!(t < 3.0e38f)) x = __int_as_float(0x7fc00000);  // an infinity or a NaN among the inputs: NaN everywhere, as in the reference
            const bool zero = ss == 0.0f && raw == 0.0f;          // all zero: every coordinate is 0, on a bound but exact
            if (zero) x = 0.0f;
            // the code: how many bounds the coordinate has reached (NaN: as the reference's comparisons fall out)
            const uint32_t bnd = base + CdSmem::BND_OFF;
            auto lds_bound = [&](int i) { float f; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(bnd + 4u * (uint32_t)i)); return f; };
            auto search = [&](float y) -> int {
                int c = 0;
#pragma unroll
                for (int step = (NBND + 1) / 2; step > 0; step >>= 1)
                    if (y >= lds_bound(c + step)) c += step;
                return BITS == 4 && y != y ? 15 : c;
            };
            int code = search(x);
            const float dist = fminf(x - lds_bound(code), lds_bound(code + 1) - x);
            if (!zero && dist < CD_MARGIN) {
                // about 1 coordinate in 700: the reference's k-ascending chain
                float acc = 0.0f;
                const uint32_t xs = base + CdSmem::RAW_OFF + 256u * (uint32_t)nv;
#pragma unroll 2
                for (int k8 = 0; k8 < 16; ++k8) {
                    const uint4 r4 = lds128(r_piece(nd, k8)), x4 = lds128(xs + 16u * (uint32_t)k8);
                    const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w}, xw[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 rf = __half22float2(*reinterpret_cast<const __half2*>(&rw[e])), xf = __half22float2(*reinterpret_cast<const __half2*>(&xw[e]));
                        acc = fma_ftz(rf.x, mul_ftz(xf.x, inv), acc);
                        acc = fma_ftz(rf.y, mul_ftz(xf.y, inv), acc);
                    }
                }
                code = search(acc);
            }
            __syncwarp();
            uint32_t v = (uint32_t)code;
            // coordinates nd, nd + 1 are in lanes 8 apart, nd + 2, nd + 3 in the next t4
            v |= __shfl_down_sync(0xffffffffu, v, 8) << BITS;
            if (BITS == 2) v |= __shfl_down_sync(0xffffffffu, v, 1) << 4;
            if ((ni & 1) == 0 && (BITS == 4 || (t4 & 1) == 0))
                asm volatile("st.shared.u8 [%0], %1;" ::"r"(base + CdSmem::NEW_OFF + 128u * (uint32_t)nv + (uint32_t)(nd * BITS >> 3)), "r"(v & 0xffu) : "memory");
            if (warp == 0 && lane < 8 && t4 == 0)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + CdSmem::NN_OFF + 4u * (uint32_t)nv), "f"(__half2float(__float2half_rn(sqrt_approx_ftz(t)))) : "memory");
        }
        __syncthreads();  // rotated queries, the new token's codes
        const uint32_t qa = base + CdSmem::Q_OFF + (uint32_t)(gl * MERGE_ROW + 32 * t4) * 2u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 w = gl < nh ? lds128(qa + 16u * i) : make_uint4(0u, 0u, 0u, 0u);
            qb[2 * i][0] = w.x; qb[2 * i][1] = w.y;
            qb[2 * i + 1][0] = w.z; qb[2 * i + 1][1] = w.w;
            if constexpr (EXACT) {
                const uint4 l = gl < nh ? lds128(qa + (CdSmem::LO_OFF - CdSmem::Q_OFF) + 16u * i) : make_uint4(0u, 0u, 0u, 0u);
                ql[2 * i][0] = l.x; ql[2 * i][1] = l.y;
                ql[2 * i + 1][0] = l.z; ql[2 * i + 1][1] = l.w;
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            qb[2 * i][0] = qw[i].x; qb[2 * i][1] = qw[i].y;
            qb[2 * i + 1][0] = qw[i].z; qb[2 * i + 1][1] = qw[i].w;
        }
    }

    auto lds_f32 = [&](uint32_t a) { float f; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(a)); return f; };
    auto new_codes = [&](int v, int k) -> uint32_t {  // the new token's K (0) or V (1): codes of the coordinates k .. k + 3
        const uint32_t at = base + CdSmem::NEW_OFF + 128u * (uint32_t)v + (uint32_t)(k * BITS >> 3);
        uint32_t w;
        if (BITS == 4) asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(w) : "r"(at));
        else asm volatile("ld.shared.u8 %0, [%1];" : "=r"(w) : "r"(at));
        return w;
    };
    auto centroid = [&](uint32_t w, int e) { return lds_f32(base + CdSmem::CENT_OFF + 4u * ((w >> (BITS * e)) & ((1u << BITS) - 1u))); };
    const bool takes_new = owner && appends;  // uniform for the CTA

    // ---- the new token, in its owner: one of the last warps, which have the fewest tiles, takes its score with a query head (its weight
    // in the CTA's result follows below).  Behind the tiles: in front of them it holds up launches of many CTAs (28 layers of 32 x 128 tokens,
    // 2-bit 32/8 heads, 178 us, behind them 168).  Not in EXACT's packed modes, whose one CTA per SM has longer tiles, which the compiler
    // orders better without it behind them (4-bit 40/8 heads 21 x 5198 tokens, 4 layers, 158 us, in front of them 153). ----
    const int new_h = CD_WARPS - 1 - warp;  // this warp's query head
    auto new_score = [&]() {
        if (!takes_new || new_h >= nh) return;
        float q[4], k[4];
        auto halves = [&](uint2 u, float (&f)[4]) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
            f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
        };
        float scale = 0.12751743074602467f;
        if constexpr (BITS == 0) {
            halves(q4, q);
            halves(lds64(base + CdSmem::RAW_OFF + 8u * (uint32_t)lane), k);
        } else {
            const uint32_t at = base + CdSmem::Q_OFF + (uint32_t)(new_h * MERGE_ROW + 4 * lane) * 2u;
            halves(lds64(at), q);
            if constexpr (EXACT) {
                float ql4[4];
                halves(lds64(at + (CdSmem::LO_OFF - CdSmem::Q_OFF)), ql4);
#pragma unroll
                for (int e = 0; e < 4; ++e) q[e] += ql4[e];
            }
            const uint32_t w = new_codes(0, 4 * lane);
#pragma unroll
            for (int e = 0; e < 4; ++e) k[e] = centroid(w, e);
            scale = lds_f32(base + CdSmem::NN_OFF);
        }
        float dot = fmaf(q[0], k[0], q[1] * k[1]) + fmaf(q[2], k[2], q[3] * k[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + CdSmem::NS_OFF + 4u * (uint32_t)new_h), "f"(dot * scale) : "memory");
    };
    constexpr bool SCORE_FIRST = EXACT && BITS != 0;
    if (SCORE_FIRST) new_score();

    // ---- tiles ----
    const bool any_tile = tile < tile_end;
    if (PRE && !(staged && early) && any_tile) look_up_k();
    float m_run[2] = {-1e30f, -1e30f}, l_run[2] = {0.0f, 0.0f};
    float acc[8][4];
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[b][0] = acc[b][1] = acc[b][2] = acc[b][3] = 0.0f;
    for (; tile < tile_end; tile += tile_step) {
        const int t0 = tile * TT;
        // ---- scores: rows gl and gl + 8 of each block, heads 2 t4 and 2 t4 + 1 ----
        float c[MB][4], ce[MB][4];  // ce: EXACT, the products with one low part; a single block: every other step, for two short chains
#pragma unroll
        for (int b = 0; b < MB; ++b) c[b][0] = c[b][1] = c[b][2] = c[b][3] = ce[b][0] = ce[b][1] = ce[b][2] = ce[b][3] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int b = 0; b < MB; ++b) {
                uint32_t a0, a1, a2, a3;
                auto low_product = [&](uint32_t wlo, int blo, uint32_t whi, int bhi, uint32_t wlo2, int blo2, uint32_t whi2, int bhi2) {
                    if constexpr (EXACT && BITS != 0) {
                        mma16816(ce[b], a0, a1, a2, a3, ql[j][0], ql[j][1]);
                        mma16816(ce[b], lut_low(wlo, blo), lut_low(whi, bhi), lut_low(wlo2, blo2), lut_low(whi2, bhi2), qb[j][0], qb[j][1]);
                    }
                };
                if constexpr (PRE) {
                    a0 = ka[j][0]; a1 = ka[j][1]; a2 = ka[j][2]; a3 = ka[j][3];
                } else if constexpr (BITS == 4) {
                    const uint4 lo4 = kw[b][0][0], hi4 = kw[b][1][0];
                    const uint32_t lo = j < 2 ? lo4.x : (j < 4 ? lo4.y : (j < 6 ? lo4.z : lo4.w)), hi = j < 2 ? hi4.x : (j < 4 ? hi4.y : (j < 6 ? hi4.z : hi4.w));
                    a0 = lut(lo, 2 * (j & 1)); a1 = lut(hi, 2 * (j & 1));
                    a2 = lut(lo, 2 * (j & 1) + 1); a3 = lut(hi, 2 * (j & 1) + 1);
                    low_product(lo, 2 * (j & 1), hi, 2 * (j & 1), lo, 2 * (j & 1) + 1, hi, 2 * (j & 1) + 1);
                } else if constexpr (BITS == 2) {
                    // byte j & 3 of the word: low nibble coordinates 4 j, 4 j + 1, high nibble 4 j + 2, 4 j + 3
                    const uint32_t lo = j < 4 ? kw[b][0][0].x : kw[b][0][0].y, hi = j < 4 ? kw[b][1][0].x : kw[b][1][0].y;
                    a0 = lut(lo & 0x0f0f0f0fu, j & 3); a1 = lut(hi & 0x0f0f0f0fu, j & 3);
                    a2 = lut((lo >> 4) & 0x0f0f0f0fu, j & 3); a3 = lut((hi >> 4) & 0x0f0f0f0fu, j & 3);
                    low_product(lo & 0x0f0f0f0fu, j & 3, hi & 0x0f0f0f0fu, j & 3, (lo >> 4) & 0x0f0f0f0fu, j & 3, (hi >> 4) & 0x0f0f0f0fu, j & 3);
                } else {
                    const uint4 lo = kw[b][0][j >> 1], hi = kw[b][1][j >> 1];
                    a0 = (j & 1) ? lo.z : lo.x; a1 = (j & 1) ? hi.z : hi.x;
                    a2 = (j & 1) ? lo.w : lo.y; a3 = (j & 1) ? hi.w : hi.y;
                }
                mma16816(MB == 1 && BITS != 0 && !EXACT && (j & 1) ? ce[b] : c[b], a0, a1, a2, a3, qb[j][0], qb[j][1]);
            }
        if (BITS != 0 && (EXACT || MB == 1)) {
#pragma unroll
            for (int b = 0; b < MB; ++b)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[b][e] += ce[b][e];
        }
        float sv[2 * MB][2];
#pragma unroll
        for (int b = 0; b < MB; ++b)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float n = BITS == 0 ? 0.12751743074602467f : __half2float(kn_h[b][r]);
                const int t = t0 + 16 * b + 8 * r + gl;
                const bool on = t < lim;
                sv[2 * b + r][0] = on ? c[b][2 * r] * n : -1e30f;
                sv[2 * b + r][1] = on ? c[b][2 * r + 1] * n : -1e30f;
            }
        const int next = tile + tile_step;
        if (next < tile_end) load_k(next, lim);
        float mx0 = sv[0][0], mx1 = sv[0][1];
#pragma unroll
        for (int i = 1; i < 2 * MB; ++i) {
            mx0 = fmaxf(mx0, sv[i][0]);
            mx1 = fmaxf(mx1, sv[i][1]);
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        }
        const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
        if (__any_sync(0xffffffffu, mn0 > m_run[0] || mn1 > m_run[1])) {
            const float f0 = ex2_approx(m_run[0] - mn0), f1 = ex2_approx(m_run[1] - mn1);
            l_run[0] *= f0;
            l_run[1] *= f1;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                acc[b][0] *= f0; acc[b][2] *= f0;
                acc[b][1] *= f1; acc[b][3] *= f1;
            }
            m_run[0] = mn0;
            m_run[1] = mn1;
        }
        uint32_t pb[2 * MB], pl[EXACT ? 2 * MB : 1];  // weights times norms, their low parts
#pragma unroll
        for (int i = 0; i < 2 * MB; ++i) {
            const int t = t0 + 16 * (i >> 1) + 8 * (i & 1) + gl;
            const bool on = t < lim;
            const float p0 = on ? ex2_approx(sv[i][0] - m_run[0]) : 0.0f, p1 = on ? ex2_approx(sv[i][1] - m_run[1]) : 0.0f;
            l_run[0] += p0;
            l_run[1] += p1;
            const float n = BITS == 0 ? 1.0f : (on ? __half2float(vn_h[i >> 1][i & 1]) : 0.0f);
            pb[i] = movmatrix_trans(pack_half2(p0 * n, p1 * n));
            if constexpr (EXACT) pl[i] = movmatrix_trans(pack_low_half2(p0 * n, p1 * n));
        }
        // ---- values ----
#pragma unroll
        for (int b = 0; b < MB; ++b) {
            const uint32_t pb0 = pb[2 * b], pb1 = pb[2 * b + 1], pl0 = EXACT ? pl[2 * b] : 0u, pl1 = EXACT ? pl[2 * b + 1] : 0u;
            auto value_product = [&](float (&d)[4], uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, int byte) {
                const uint32_t a0 = lut(w0, byte), a1 = lut(w1, byte), a2 = lut(w2, byte), a3 = lut(w3, byte);
                mma16816(d, a0, a1, a2, a3, pb0, pb1);
                if constexpr (EXACT) {
                    mma16816(d, a0, a1, a2, a3, pl0, pl1);
                    mma16816(d, lut_low(w0, byte), lut_low(w1, byte), lut_low(w2, byte), lut_low(w3, byte), pb0, pb1);
                }
            };
            if constexpr (BITS == 4) {
                const uint32_t wa[2] = {vw[b][0][0].x, vw[b][0][0].y}, wb[2] = {vw[b][1][0].x, vw[b][1][0].y};
                const uint32_t wc[2] = {vw[b][2][0].x, vw[b][2][0].y}, wd[2] = {vw[b][3][0].x, vw[b][3][0].y};
#pragma unroll
                for (int w2 = 0; w2 < 2; ++w2) {  // (code of token A, code of token B) per byte, even and odd coordinates
                    const uint32_t ev_ab = (wa[w2] & 0x0f0f0f0fu) | ((wb[w2] << 4) & 0xf0f0f0f0u);
                    const uint32_t od_ab = ((wa[w2] >> 4) & 0x0f0f0f0fu) | (wb[w2] & 0xf0f0f0f0u);
                    const uint32_t ev_cd = (wc[w2] & 0x0f0f0f0fu) | ((wd[w2] << 4) & 0xf0f0f0f0u);
                    const uint32_t od_cd = ((wc[w2] >> 4) & 0x0f0f0f0fu) | (wd[w2] & 0xf0f0f0f0u);
#pragma unroll
                    for (int i = 0; i < 4; ++i) value_product(acc[4 * w2 + i], ev_ab, od_ab, ev_cd, od_cd, i);
                }
            } else if constexpr (BITS == 2) {
                const uint32_t wa = vw[b][0][0].x, wb = vw[b][1][0].x, wc = vw[b][2][0].x, wd = vw[b][3][0].x;
                const uint32_t ev_ab = (wa & 0x33333333u) | ((wb << 2) & 0xccccccccu), od_ab = ((wa >> 2) & 0x33333333u) | (wb & 0xccccccccu);
                const uint32_t ev_cd = (wc & 0x33333333u) | ((wd << 2) & 0xccccccccu), od_cd = ((wc >> 2) & 0x33333333u) | (wd & 0xccccccccu);
#pragma unroll
                for (int i = 0; i < 8; ++i) {  // coordinates 2 i, 2 i + 1 of the lane's 16: nibble i of `ev`, `od`
                    auto nib = [&](uint32_t w) { return ((i & 1) ? w >> 4 : w) & 0x0f0f0f0fu; };
                    value_product(acc[i], nib(ev_ab), nib(od_ab), nib(ev_cd), nib(od_cd), i >> 1);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {  // (token A, token B) per even and odd coordinate
                    auto word = [&](int r) -> uint32_t {
                        const uint4 u = vw[b][r][i >> 2];
                        return (i & 3) == 0 ? u.x : ((i & 3) == 1 ? u.y : ((i & 3) == 2 ? u.z : u.w));
                    };
                    const uint32_t a0 = prmt(word(0), word(1), 0x5410u), a1 = prmt(word(0), word(1), 0x7632u);
                    const uint32_t a2 = prmt(word(2), word(3), 0x5410u), a3 = prmt(word(2), word(3), 0x7632u);
                    mma16816(acc[i], a0, a1, a2, a3, pb0, pb1);
                    if (EXACT) mma16816(acc[i], a0, a1, a2, a3, pl0, pl1);
                }
            }
        }
        if (next < tile_end) {
            load_v(next, lim);
            if (PRE) look_up_k();
        }
    }

    // ---- the warps' results: acc[b]: coordinates 16 gl + 2 b (and + 1), heads 2 t4, 2 t4 + 1 ----
    if (any_tile) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], o);
            l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], o);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int h = 2 * t4 + e;
            if (h < nh) {
                const uint32_t dst = warps_s + (uint32_t)((warp * nh + h) * PART_STRIDE) * 4u;
#pragma unroll
                for (int b2 = 0; b2 < 4; ++b2)
                    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)(16 * gl + 4 * b2) * 4u), "f"(acc[2 * b2][e]),
                                 "f"(acc[2 * b2][2 + e]), "f"(acc[2 * b2 + 1][e]), "f"(acc[2 * b2 + 1][2 + e]) : "memory");
                if (gl == 0)
                    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dst + HEAD_DIM * 4u), "f"(m_run[e]), "f"(l_run[e]) : "memory");
            }
        }
    }
    if (!SCORE_FIRST) new_score();
    __syncthreads();
    // ---- the CTA's result, normalised: maximum and sum beside it ----
    // where coordinate n of head h goes in the CTA that adds up its share: [this CTA][head][coordinate of the share]
    const uint32_t s_log = 31u - (uint32_t)__clz((int)S), share_log = 7u - s_log;  // (S is a power of two)
    auto send = [&](int h, int n, float v0, float v1) {  // coordinates n, n + 1
        const uint32_t r = (uint32_t)n >> share_log;
        st_async_f32x2(map_shared(base + CdSmem::CP_OFF + ((((rank * (uint32_t)nh + (uint32_t)h) << share_log) + ((uint32_t)n & ((1u << share_log) - 1u))) << 2), r), v0, v1,
                       map_shared(bar, r));
    };
    // Host results of a single CTA meet in shared memory and leave in whole lines: the bus takes a write in the pieces it arrives in.  As
    // the products leave them, 16 bytes at a time, those were what L2 happened to put together: a step of many short sequences took up to
    // 1.7 times as long for a change of the instructions in front of them (28 layers, 2-bit 32/4 heads 16 x 300 tokens 140 or 230 us, now 137).
    auto stage_out = [&](int at, uint32_t two) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + CdSmem::CP_OFF + 2u * (uint32_t)at), "r"(two) : "memory"); };
    if (S > 1) cluster_wait();  // every CTA of the cluster has started
    // The warps' results are added up by a warp per head, a lane per four coordinates: maxima and exponentials once for four (a lane per
    // coordinate costs steps of many short sequences with 8 heads 5 %).  Clusters with up to two heads, whose launches wait for their
    // longest chain, take a lane per coordinate, four warps per head.
    auto sum_up = [&](auto c_) {
        constexpr int C = decltype(c_)::value;
        const int h = C == 1 ? warp >> 2 : warp, k = C == 1 ? tid & (HEAD_DIM - 1) : C * lane;
        if (h >= nh) return;
        const uint32_t src = warps_s + (uint32_t)(h * PART_STRIDE) * 4u, wstride = (uint32_t)(nh * PART_STRIDE) * 4u;
        float mw[CD_WARPS], lw[CD_WARPS], aw[CD_WARPS][C], vn[C], M = -1e30f, m_new = -1e30f;
#pragma unroll
        for (int w = 0; w < CD_WARPS; ++w) {
            const uint32_t at = src + (uint32_t)w * wstride;
            part_if(at + HEAD_DIM * 4u, at + (uint32_t)k * 4u, w < n_act, mw[w], lw[w], aw[w]);
        }
#pragma unroll
        for (int i = 0; i < C; ++i) vn[i] = 0.0f;
        if (takes_new) {
            if constexpr (BITS == 0) {
                const uint2 u = lds64(base + CdSmem::RAW_OFF + 256u + 2u * (uint32_t)(k & ~3));
                const float2 v0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), v1 = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
                const float v[4] = {v0.x, v0.y, v1.x, v1.y};
                if constexpr (C == 4) { vn[0] = v[0]; vn[1] = v[1]; vn[2] = v[2]; vn[3] = v[3]; }
                else vn[0] = (k & 2) ? ((k & 1) ? v[3] : v[2]) : ((k & 1) ? v[1] : v[0]);
            } else {
                const uint32_t w = new_codes(1, k & ~3);
                const float n = lds_f32(base + CdSmem::NN_OFF + 4u);
#pragma unroll
                for (int i = 0; i < C; ++i) vn[i] = n * centroid(w, C == 1 ? k & 3 : i);
            }
            m_new = lds_f32(base + CdSmem::NS_OFF + 4u * (uint32_t)h);
            M = fmaxf(M, m_new);
        }
#pragma unroll
        for (int w = 0; w < CD_WARPS; ++w) M = fmaxf(M, mw[w]);
        const float e_new = takes_new ? ex2_approx(m_new - M) : 0.0f;
        float a[C], z = e_new;
#pragma unroll
        for (int i = 0; i < C; ++i) a[i] = takes_new ? e_new * vn[i] : 0.0f;
#pragma unroll
        for (int w = 0; w < CD_WARPS; ++w) {
            const float e = ex2_approx(mw[w] - M);  // (a warp without tiles: times zero)
#pragma unroll
            for (int i = 0; i < C; ++i) a[i] = fmaf(e, aw[w][i], a[i]);
            z = fmaf(e, lw[w], z);
        }
        // one CTA: the reference's denominator; several: the part's own sum (none: no token), the rest follows below (there, and here for
        // several, 1 and 2 units of fp32 off a correctly rounded quotient: those cost 1 to 3 % of a small layer)
#pragma unroll
        for (int i = 0; i < C; ++i) a[i] = S == 1 ? a[i] / (z + 1e-8f) : (z > 0.0f || z != z ? a[i] * rcp_approx_ftz(z) : 0.0f);
        const int r = C == 1 ? k : lane;
        if (S > 1 && r < (int)S)
            st_async_f32x2(map_shared(base + CdSmem::MZ_OFF + (uint32_t)((int)rank * nh + h) * 8u, (uint32_t)r), M, z, map_shared(bar, (uint32_t)r));
        if constexpr (BITS == 0) {
            __half* const o = p.out + (size_t)g * p.q_dim + (size_t)(head0 + h) * HEAD_DIM + k;
            if constexpr (C == 1) {
                const float a1 = __shfl_down_sync(0xffffffffu, a[0], 1);
                if (S == 1) *o = __float2half_rn(a[0]);
                else if ((k & 1) == 0) send(h, k, a[0], a1);
            } else if (HOST && S == 1) {
                stage_out(h * HEAD_DIM + k, pack_half2(a[0], a[1]));
                stage_out(h * HEAD_DIM + k + 2, pack_half2(a[2], a[3]));
            } else if (S == 1) {
                reinterpret_cast<__half2*>(o)[0] = __floats2half2_rn(a[0], a[1]);
                reinterpret_cast<__half2*>(o)[1] = __floats2half2_rn(a[2], a[3]);
            } else {
                send(h, k, a[0], a[1]);
                send(h, k + 2, a[2], a[3]);
            }
        } else {
            const uint32_t o = base + CdSmem::Q_OFF + (uint32_t)(h * MERGE_ROW + k) * 2u;
            constexpr uint32_t low = CdSmem::LO_OFF - CdSmem::Q_OFF;
            if constexpr (C == 1) {
                const __half ahi = __float2half_rn(a[0]);
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(o), "h"(__half_as_ushort(ahi)) : "memory");
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(o + low), "h"(__half_as_ushort(__float2half_rn(a[0] - __half2float(ahi)))) : "memory");
            } else {
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(o), "r"(pack_half2(a[0], a[1])), "r"(pack_half2(a[2], a[3])) : "memory");
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(o + low), "r"(pack_low_half2(a[0], a[1])), "r"(pack_low_half2(a[2], a[3])) : "memory");
            }
        }
    };
    if (nh <= 2) sum_up(std::integral_constant<int, 1>());
    else sum_up(std::integral_constant<int, 4>());
    if constexpr (BITS != 0) {
        __syncthreads();
        // times R: o[h][n] = sum_k a[h][k] R[k][n], two blocks of 8 output coordinates per warp.  The high parts are rows 0-7 of the A
        // operand, the low parts rows 8-15 (rows >= nh are never read back)
        uint32_t ah[4][4], al[4][4];  // two 16-k steps each
        const uint32_t a_at = base + CdSmem::Q_OFF + (uint32_t)((lane & 7) * MERGE_ROW + 8 * (lane >> 3)) * 2u;
#pragma unroll
        for (int j2 = 0; j2 < 4; ++j2) {
            ldmatrix_x4(ah[j2], a_at + 64u * j2);
            ldmatrix_x4(al[j2], a_at + (CdSmem::LO_OFF - CdSmem::Q_OFF) + 64u * j2);
        }
        float oc[2][2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) oc[i][0][e] = oc[i][1][e] = 0.0f;
#pragma unroll
        for (int j2 = 0; j2 < 4; ++j2) {  // two steps of 16 k each per ldmatrix
            uint32_t b[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) ldmatrix_x4_trans(b[i], r_piece(32 * j2 + lane, warp + CD_WARPS * i));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mma16816(oc[i][0], ah[j2][0], al[j2][0], ah[j2][1], al[j2][1], b[i][0], b[i][1]);
                mma16816(oc[i][1], ah[j2][2], al[j2][2], ah[j2][3], al[j2][3], b[i][2], b[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int nb = warp + CD_WARPS * i;
            if (gl < nh) {
                const float o0 = (oc[i][0][0] + oc[i][1][0]) + (oc[i][0][2] + oc[i][1][2]), o1 = (oc[i][0][1] + oc[i][1][1]) + (oc[i][0][3] + oc[i][1][3]);
                if (S == 1) {
                    const size_t at = (size_t)(head0 + gl) * HEAD_DIM + 8 * nb + 2 * t4;
                    if (HOST) stage_out(gl * HEAD_DIM + 8 * nb + 2 * t4, pack_half2(o0, o1));
                    else *reinterpret_cast<__half2*>(p.out + (size_t)g * p.q_dim + at) = __floats2half2_rn(o0, o1);
                    if (p.out_f32) *reinterpret_cast<float2*>(p.out_f32 + (size_t)g * p.H * HEAD_DIM + at) = make_float2(o0, o1);
                } else {
                    send(gl, 8 * nb + 2 * t4, o0, o1);
                }
            }
        }
    }
    if (HOST && S == 1 && (BITS != 0 || nh > 2)) {
        __syncthreads();
        uint32_t* const o = reinterpret_cast<uint32_t*>(p.out + (size_t)g * p.q_dim + (size_t)head0 * HEAD_DIM);
        for (int i = tid; i < nh * (HEAD_DIM / 2); i += CD_THREADS) o[i] = lds32(base + CdSmem::CP_OFF + 4u * (uint32_t)i);
    }
    if (S > 1) {
        if (!mbar_wait_bounded_hint(bar, 0u, 1u << 14, 20000u) && p.status) atomicMax(p.status, ST_TMA_WAIT_TIMEOUT);
        // ---- this CTA's share of the coordinates: one lane per (coordinate, CTA), the S lanes of a coordinate side by side ----
        for (int i = tid; i < nh * HEAD_DIM; i += CD_THREADS) {
            const int r = i & ((int)S - 1), o = i >> s_log;
            const int h = o >> share_log, n = o & ((1 << share_log) - 1);
            const float v = lds_f32(base + CdSmem::CP_OFF + (uint32_t)(((r * nh + h) << share_log) + n) * 4u);
            float m, z;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m), "=f"(z) : "r"(base + CdSmem::MZ_OFF + (uint32_t)(r * nh + h) * 8u));
            float M = m;
#pragma unroll
            for (int w = 1; w < CD_MAX_CLUSTER; w <<= 1)
                if (w < (int)S) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, w));
            float Z = ex2_approx(m - M) * z, a = Z * v;
#pragma unroll
            for (int w = 1; w < CD_MAX_CLUSTER; w <<= 1)
                if (w < (int)S) {
                    Z += __shfl_xor_sync(0xffffffffu, Z, w);
                    a += __shfl_xor_sync(0xffffffffu, a, w);
                }
            if (r == 0) {
                a = __fdividef(a, Z + 1e-8f);
                const size_t at = (size_t)(head0 + h) * HEAD_DIM + ((int)rank << share_log) + n;
                p.out[(size_t)g * p.q_dim + at] = __float2half_rn(a);
                if (p.out_f32) p.out_f32[(size_t)g * p.H * HEAD_DIM + at] = a;
            }
        }
    }
    // ---- the new token goes to the cache (one of the KV head's clusters) ----
    if (owner && hblk == 0 && pos_ok) {
        uint8_t* dst = const_cast<uint8_t*>(vec == 0 ? p.ck : p.cv) + (size_t)(row0 + pos) * kvp + (size_t)kvh * BPH;
        const uint32_t src = base + (BITS == 0 ? CdSmem::RAW_OFF + 256u * (uint32_t)vec : CdSmem::NEW_OFF + 128u * (uint32_t)vec);
        if (d < BPH / 4) *reinterpret_cast<uint32_t*>(dst + 4 * d) = lds32(src + 4u * (uint32_t)d);
        if (BITS != 0 && d == 0)
            const_cast<__half*>(vec == 0 ? p.kn : p.vn)[(size_t)(row0 + pos) * p.Hkv + kvh] = __float2half_rn(lds_f32(base + CdSmem::NN_OFF + 4u * (uint32_t)vec));
    }
}

}  // namespace tq
