// Causal prefill attention on the 5th-generation tensor cores (tcgen05 + tensor memory), sm_100a.
//
// Query token t of a prompt attends to cache rows 0 .. t (reference engine/kernels.cu:1874-1960 packed, :1071-1158 fp16).
// One CTA has two SLOTS that work in turn, so that the tensor core always has a product of one slot while the softmax of the
// other runs.  A slot = 128 score rows (128 / GRP query tokens x the GRP query heads of one KV head) = the M dimension,
// eight softmax warps (16 rows each, four threads per row), 128 columns of tensor memory for S and 128 for O:
//   * long prompts (MT = 2): the slots are two consecutive query blocks that share every K and V tile;
//   * short ones (MT = 1): both slots hold the same query block and take the even and the odd tiles; their results are
//     combined at the end.  Twice the CTAs and half the chain when there are not enough blocks for the GPU.
// Tiles are 128 cache rows.  K lies in shared memory as [coordinate half][128 rows][128 B] (K-major B operand of S = Q K^T),
// V in the same form, read as an MN-major B operand of O += P V: no transposition anywhere, both arrive by one tensor-map
// copy.  Packed caches are turned into fp16 centroids (unscaled: the same operands as ever) and fp32 norms by
// dequantize_rows_kernel (short prompts: by the append, tq_prefill_tc.cuh) first, once per prompt and layer instead of once per query block: done by producer warps inside
// this kernel the table look-ups and operand stores took as much of the shared-memory pipe as the products themselves (8192
// tokens, 16/8 heads, 4-bit, eight softmax warps: 617 us against 439).  Prompts of a single tile are the exception (DIRECT).  P (times the V norm, fp16) replaces S in tensor memory and is read from
// there as the A operand.
//   warps 0-15   softmax of slots 0 and 1: S -> registers (16x256b loads: a thread holds two rows' column pairs as in an mma
//                fragment, so a row's maximum is two shuffles), K norm, causal limit, exponentials, P -> tensor memory.  The
//                exponentials' reference point follows the row maximum only when that has grown by more than PFT_SLACK (in
//                powers of two; packed tiles with very large V norms: at all): weights stay below 2^PFT_SLACK and O is rescaled in
//                place in the first tiles only.
//   warp 16      issues the copies; warp 17 issues every product, in the order P(i) V -> S(i + 1) per slot, slots alternating: the
//                products of one thread execute in order, so S(i + 1) may overwrite the P(i) that the one before it reads.
// Numbers of query heads per KV head other than 1, 2, 4, 8 and 16 took a kernel with fp32 queries, centroids and weights.  Here they
// are fp16 high + low parts (EXACT: three products for one, two for fp16 caches): the results' error is that kernel's.  With the high
// parts alone it was 2.4 (4-bit), 2.9 (2-bit) and 1.2 (fp16) times as large.
// Packed forms: Q R^T at the start and (O / l) R at the end (fp16 high + low parts) are tcgen05 products too.  Behind the append the first of
// them is done before the wait: the append lets this launch start when everything before it has finished, and its own stores have nothing
// to do with queries and R.  Per layer, 16/8 heads, 4-bit: 300 tokens 21.6 -> 20.1 us, 777 28.4 -> 27.0, 16 x 256 50.2 -> 47.1.
// Every wait on a barrier is bounded; a wait that runs out raises the status word and the kernel runs to its end.
// Bound by the softmax threads (exponentials, tensor-memory loads) against the tensor core at long prompts, by the chain copy ->
// S -> softmax -> O of a single block at short ones.  Per layer, 8 KV heads, cache write included, the one-block kernel with V
// transposed through shared memory -> this one: fp16 8192 tokens 32 heads 2811 -> 478 us in runs of a few milliseconds (1150 TFLOP/s
// of causal arithmetic), 557 (987) under the power cap of longer ones; 4-bit 777 tokens 16 heads 43.7 -> 26.3.  (With one thread per row, eight softmax warps, S read twice: 530, 379, 34.2.)
#pragma once

#include "tq_prefill_tc.cuh"

namespace tq {

constexpr int PFT_ROWS = 128;     // score rows of a slot
constexpr float PFT_SLACK = 4.0f;
constexpr float PFT_SCALE = 0.12751743074602467f;  // log2(e) / sqrt(128); packed forms: carried by the rotated queries
constexpr uint32_t PFT_TILE = 32768u;  // an operand tile: [2 halves of the coordinates][128 rows][128 B]
constexpr uint32_t PFT_NORM_BYTES = PFT_NORMS * 4u;

constexpr int PFT_SOFT_WARPS = 16;
constexpr int PFT_THREADS = 32 * PFT_SOFT_WARPS + 128;  // softmax, then one warp for the copies, one for the products, two idle (a full warpgroup)
// Registers per thread of the softmax warpgroups and of the last one after the split.  The launch must bring at least their sum
// (the host checks what the kernel was built with): 640 x 96 = 512 x 104 + 128 x 64.
constexpr int PFT_REGS_SOFT = 104, PFT_REGS_REST = 64;
constexpr int PFT_REGS_LAUNCH = (32 * PFT_SOFT_WARPS * PFT_REGS_SOFT + 128 * PFT_REGS_REST + PFT_THREADS - 1) / PFT_THREADS;

struct PrefillAttnParams {
    const __half* q;          // queries [n_seq][T][q_tok_stride] as the model makes them
    long long q_tok_stride;   // halves between the queries of consecutive tokens
    const uint8_t* ck;        // packed codes [rows][kvp] or fp16 rows [rows][Hkv * 128]; read through maps, but for DIRECT
    const uint8_t* cv;
    const __half* kn;         // [rows][Hkv], packed caches (read by DIRECT)
    const __half* vn;
    int early;                // packed, behind prefill_append_tc_kernel (or a launch behind it), which lets its successor start once all before it
                              // has finished: queries and R may be read and rotated before the wait
    const __half* rotation;   // packed: R row-major [128][128]
    int low_row;              // packed, EXACT: rows from the high parts to the low parts of ck, cv
    const float* norms;       // packed: fp32 [n_seq][Hkv][tiles][PFT_NORMS] (dequantize_rows_kernel)
    int tiles;                // of PFT_KT cache rows per prompt
    int* status;              // optional device status word (a bounded wait that gave up raises it)
    __half* out;              // [n_seq][T][q_dim]
    int q_dim;
    int T;                    // query tokens of a prompt = cache rows in use
    int H, Hkv, grp;          // grp query heads per KV head
    // Several prompts of the same length in one launch (grid.x = Hkv * n_seq): the cache rows of prompt i start at row_base[i]
    // (or i * seq_rows).
    int n_seq;
    long long seq_rows;
    const long long* row_base;
};

struct PftSmem {
    static constexpr uint32_t Q = 0;                    // MT tiles; at the end: high parts of the results
    static constexpr uint32_t K = 2 * PFT_TILE;         // 2 stages; at the end: low parts
    static constexpr uint32_t V = K + 2 * PFT_TILE;     // 2 stages
    static constexpr uint32_t R = V + 2 * PFT_TILE;     // packed: R [row][column]
    static constexpr uint32_t NORM = R + PFT_TILE;      // [2 stages][PFT_NORMS] floats; MT = 1, at the end: [2 slots][128][maximum, sum]
    static constexpr uint32_t CTRL = NORM + 2u * PFT_NORM_BYTES;  // mbarriers, tensor-memory base
    static constexpr uint32_t BYTES = CTRL + 256u;
};

// Packed prompts for the kernel below: rows first_row .. of one KV cache array pair as fp16 centroids [n_seq][T][kv_dim] and fp32
// norms [n_seq][Hkv][tiles][PFT_NORMS] (zero behind the prompt).  One thread per 8 codes; bound by HBM / L2 writes of the fp16 rows.
struct DequantParams {
    const uint8_t* ck;
    const uint8_t* cv;
    const __half* kn;
    const __half* vn;
    const long long* row_base;   // [n_seq] or null: seq_rows * i
    long long seq_rows;
    __half* k16;
    __half* v16;
    float* norms;
    int T, tiles, Hkv;           // Hkv: heads of this pass; ck, cv, kn, vn point at the first one's
    int row_heads;               // heads per row of the cache
    long long low;               // EXACT: halves from a value's high part to its low part
    int code_blocks;             // CTAs (per prompt) for the codes; those behind them take the norms, a warp per tile and KV head
};
template <int BITS, bool EXACT>
__global__ void __launch_bounds__(256) dequantize_rows_kernel(const DequantParams p) {
    // byte (4-bit) or nibble (2-bit) -> two centroids; eight copies, so that at most four lanes of a warp share a bank
    constexpr int ENTRIES = BITS == 4 ? 256 : 16;
    __shared__ uint32_t luts[(EXACT ? 2 : 1) * ENTRIES * 8];  // EXACT: then their low parts
    for (int i = threadIdx.x; i < ENTRIES * 8; i += 256) {
        const int e = i >> 3;
        const float c0 = BITS == 4 ? kCent4[e & 15] : kCent2[e & 3], c1 = BITS == 4 ? kCent4[e >> 4] : kCent2[(e >> 2) & 3];
        luts[i] = pack_half2(c0, c1);
        if (EXACT) luts[ENTRIES * 8 + i] = pack_low_half2(c0, c1);
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();  // the rows come from the append before this launch
    const int seq = blockIdx.y;
    const long long row0 = p.row_base ? p.row_base[seq] : (long long)seq * p.seq_rows;
    if ((int)blockIdx.x >= p.code_blocks) {
        const int lane = threadIdx.x & 31, blocks = (int)gridDim.x - p.code_blocks;
        for (int w = ((int)blockIdx.x - p.code_blocks) * 8 + (threadIdx.x >> 5); w < p.Hkv * p.tiles; w += blocks * 8) {
            const int h = w / p.tiles, tile = w - h * p.tiles;
            float* const dst = p.norms + (((long long)seq * p.Hkv + h) * p.tiles + tile) * PFT_NORMS;
            uint32_t top = 0u;  // of the V norms' words: they order as the values do, and what is not a number lies above them all
#pragma unroll
            for (int i = 0; i < PFT_KT; i += 32) {
                const int t = tile * PFT_KT + i + lane;
                const long long at = (row0 + t) * p.row_heads + h;
                const float kn = t < p.T ? __half2float(p.kn[at]) : 0.0f, vn = t < p.T ? __half2float(p.vn[at]) : 0.0f;
                dst[i + lane] = kn;
                dst[PFT_KT + i + lane] = vn;
                top = max(top, __float_as_uint(vn));
            }
            top = __reduce_max_sync(0xffffffffu, top);
            // (as a half, exactly; what is not a number stays above the infinity)
            if (lane == 0) *reinterpret_cast<uint4*>(dst + 2 * PFT_KT) = make_uint4(__half_as_ushort(__float2half_rn(__uint_as_float(top))), 0u, 0u, 0u);
        }
        return;
    }
    const int words = p.Hkv * 16;  // 8-code pieces per row
    const long long n = (long long)p.T * words;
    const int copy = threadIdx.x & 7;
    // (four pieces' loads in flight at a time, not four round trips one after the other)
    constexpr int FLIGHT = 4;
    const long long step = (long long)p.code_blocks * 256;
    for (long long i0 = (long long)blockIdx.x * 256 + threadIdx.x; i0 < 2 * n; i0 += FLIGHT * step) {
        uint32_t codes[FLIGHT];
#pragma unroll
        for (int f = 0; f < FLIGHT; ++f) {
            const long long i = i0 + f * step;
            const bool is_v = i >= n;
            const long long w = is_v ? i - n : i;
            const long long at = row0 * (p.row_heads * 16) + (p.row_heads == p.Hkv ? w : w / words * (p.row_heads * 16) + w % words);
            codes[f] = 0u;
            if (i < 2 * n)
                codes[f] = BITS == 4 ? *(reinterpret_cast<const uint32_t*>(is_v ? p.cv : p.ck) + at)
                                     : (uint32_t)*(reinterpret_cast<const unsigned short*>(is_v ? p.cv : p.ck) + at);
        }
#pragma unroll
        for (int f = 0; f < FLIGHT; ++f) {
            const long long i = i0 + f * step;
            if (i >= 2 * n) break;
            const bool is_v = i >= n;
            const uint32_t c = codes[f];
            uint4* const dst = reinterpret_cast<uint4*>(is_v ? p.v16 : p.k16) + (long long)seq * n + (is_v ? i - n : i);
#pragma unroll
            for (int part = 0; part < (EXACT ? 2 : 1); ++part) {
                const uint32_t* const lut = luts + part * ENTRIES * 8;
                uint4 u;
                if (BITS == 4) {
                    u.x = lut[(c & 0xffu) * 8 + copy]; u.y = lut[((c >> 8) & 0xffu) * 8 + copy];
                    u.z = lut[((c >> 16) & 0xffu) * 8 + copy]; u.w = lut[(c >> 24) * 8 + copy];
                } else {
                    u.x = lut[(c & 0xfu) * 8 + copy]; u.y = lut[((c >> 4) & 0xfu) * 8 + copy];
                    u.z = lut[((c >> 8) & 0xfu) * 8 + copy]; u.w = lut[(c >> 12) * 8 + copy];
                }
                dst[part ? p.low / 8 : 0] = u;
            }
        }
    }
}

// 16 lanes x 32 (64) consecutive 32-bit columns.  Thread (g = lane / 4, t = lane % 4) holds of column block j (8 columns) the
// columns 8 j + 2 t, + 1 of row g in r[4 j], r[4 j + 1] and of row g + 8 in r[4 j + 2], r[4 j + 3].
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_frag32(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// 16 lanes x 32 columns of words that pack two halves each: of word block j (4 words) word 4 j + t of row g in r[2 j], of row g + 8
// in r[2 j + 1] -- what the two values of a fragment pack to
__device__ __forceinline__ void tmem_st_pack32(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// Four 8 x 8 matrices of halves to shared memory: lane l holds (row l / 4, columns 2 (l % 4), + 1) of each and names the address of row
// l % 8 of matrix l / 8 (16 bytes).
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The same products with the descriptors as their low words; the high word is common to all operand tiles of this kernel (groups
// of 8 rows 1024 bytes apart, descriptor version, 128-byte swizzle).  Few registers, few instructions: the thread that issues
// them is on the critical path of every tile.
constexpr uint32_t PFT_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void umma_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 a, {%1, %5};\n\t"
        "mov.b64 b, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t"
        "}\n" ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(PFT_DESC_HI)
        : "memory");
}
// A from tensor memory: row = lane, two halves per 32-bit column
__device__ __forceinline__ void umma_lo_ta(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 b, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(PFT_DESC_HI)
        : "memory");
}
// fp16 x fp16 -> fp32, M = 128, N = 128; B K-major (rows = N) or MN-major (rows = K)
constexpr uint32_t PFT_IDESC_K = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t PFT_IDESC_MN = PFT_IDESC_K | (1u << 16);
// Low descriptor word of a K-major operand tile at shared address `addr`; step ks of 16 k lies pft_kstep(ks) further on
__device__ __forceinline__ uint32_t pft_lo_k(uint32_t addr) { return ((addr >> 4) & 0x3fffu) | (1u << 16); }
__host__ __device__ constexpr uint32_t pft_kstep(int ks) { return (uint32_t)(ks >> 2) * (PFT_TILE / 2 / 16) + (uint32_t)(ks & 3) * 2u; }
// ... of an MN-major one (64 N elements per 128-byte row, the N halves PFT_TILE / 2 apart): 2048 bytes per step of 16 k
__device__ __forceinline__ uint32_t pft_lo_mn(uint32_t addr) { return ((addr >> 4) & 0x3fffu) | ((PFT_TILE / 2 / 16) << 16); }
// byte offset of the 16-byte chunk `ch` (8 halves; 0 .. 15) of row `row` in an operand tile
__device__ __forceinline__ uint32_t pft_chunk(int row, int ch) {
    return (uint32_t)(ch >> 3) * (PFT_TILE / 2) + (uint32_t)row * 128u + (uint32_t)(((ch & 7) ^ (row & 7)) << 4);
}
template <int N>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// PACKED: but for DIRECT, ck, cv are the fp16 centroids [n_seq * T][kv_dim] of dequantize_rows_kernel (seq_rows = T, no row_base), p.norms its norms
// EXACT: queries, centroids and weights as fp16 high + low parts; packed with MT = 1 only: one stage of K and V, the low parts in
// the other one's place, the queries' in the second query tile's
// DIRECT (4 or 2 bits, prompts of one tile): the softmax warps turn the tile's codes into centroids themselves, while the queries arrive
// and are rotated.  Every query block of a head repeats that, but dequantize_rows_kernel's launch is saved: a layer of 35 tokens,
// 16/8 heads, 4-bit 20.4 -> 15.5 us, 16 prompts of 32 tokens, 2-bit 24.9 -> 19.9, 16 of 128, 4-bit 33.0 -> 25.8.
// EARLY (DIRECT only; elsewhere p.early says it): queries and R before the wait, the codes behind the rotation.
template <bool PACKED, int MT, bool EXACT, int DIRECT, bool EARLY = false>
__global__ void __launch_bounds__(PFT_THREADS, 1)
prefill_attention_fa_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ,
                            const __grid_constant__ CUtensorMap tmR, const PrefillAttnParams p) {
    extern __shared__ __align__(1024) uint8_t pft_smem_base[];
    const uint32_t sb = smem_u32(pft_smem_base);
    uint8_t* const gb = pft_smem_base;
    if ((sb & 1023u) != 0u) {  // operand tiles want 1024-byte alignment; nothing static lies before the dynamic part
        if (threadIdx.x == 0 && p.status) atomicMax(p.status, ST_SMEM_LAYOUT);
        return;
    }
    constexpr int COPY_WARP = PFT_SOFT_WARPS, MMA_WARP = PFT_SOFT_WARPS + 1;
    constexpr bool LOW = PACKED && EXACT;  // low parts of the operands in shared memory
    static_assert(!LOW || MT == 1, "the second query block's places hold the low parts");
    static_assert(!EARLY || DIRECT, "decided by p.early");
    static_assert(!DIRECT || (PACKED && !EXACT), "a packed form");
    // DIRECT: byte (4-bit) or nibble (2-bit) -> two centroids, eight copies, in the idle second stage of K
    constexpr int CODES = DIRECT == 4 ? 256 : 16;
    uint32_t* const lut = reinterpret_cast<uint32_t*>(gb + PftSmem::K + PFT_TILE);
    // tile j's data are in stage j % STAGES; its barriers are number j & 1 also where there is one stage (a slot waits for every other
    // tile only, so that it must not meet the one between them on the same barrier)
    constexpr int STAGES = LOW ? 1 : 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int GRP = p.grp, QT = PFT_ROWS / GRP;
    const int qb = (int)gridDim.y - 1 - (int)blockIdx.y;  // the longest causal prefixes of all heads and prompts first
    const int seq = (int)blockIdx.x / p.Hkv, kvh = (int)blockIdx.x - seq * p.Hkv;
    const int q0 = qb * MT * QT;
    // tiles of each slot, and where slot s's i-th tile lies
    auto tiles_to = [&](int first) { return first < p.T ? (min(first + QT, p.T) - 1) / PFT_KT + 1 : 0; };
    const int n_all = tiles_to(q0);
    const int n0 = MT == 2 ? n_all : (n_all + 1) / 2, n1 = MT == 2 ? tiles_to(q0 + QT) : n_all / 2;
    const int n_tiles = MT == 2 ? max(n0, n1) : n_all;
    auto tile_of = [&](int s, int i) { return MT == 2 ? i : 2 * i + s; };
    const long long seq_row0 = p.row_base ? p.row_base[seq] : (long long)seq * p.seq_rows;
    __half* const out_seq = p.out + (size_t)seq * (size_t)p.T * (size_t)p.q_dim;

    const uint32_t ctrl = sb + PftSmem::CTRL;
    const uint32_t bar_kfull = ctrl, bar_vfull = ctrl + 16u, bar_kfree = ctrl + 32u, bar_vfree = ctrl + 48u;  // [2 stages] each
    const uint32_t bar_sfull = ctrl + 64u, bar_pfull = ctrl + 80u;                                            // [2 slots] each
    const uint32_t bar_rot = ctrl + 96u, bar_done = ctrl + 104u, bar_tail = ctrl + 112u, bar_q = ctrl + 120u;
    volatile uint32_t* const tmem_slot = reinterpret_cast<volatile uint32_t*>(gb + PftSmem::CTRL + 128);
    bool dead = false;
    auto wait_bar = [&](uint32_t bar, uint32_t parity) {
        if (!dead && !mbar_wait_bounded_hint(bar, parity, 1u << 17, 2000u)) {
            dead = true;
            if (p.status) atomicMax(p.status, ST_TMA_WAIT_TIMEOUT);
        }
    };

    auto ready = [&](uint32_t bar, uint32_t parity) {  // (two blocks: most waits are over when they are asked for)
        if (MT == 1 || !mbar_try_wait(bar, parity)) wait_bar(bar, parity);
    };

    // ---- once: tensor memory, barriers, table, queries, R ----
    if (warp == 0) {
        tmem_alloc(ctrl + 128u, 512u);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_kfull + 8u * i, 1);
            mbar_init(bar_vfull + 8u * i, 1);
            mbar_init(bar_kfree + 8u * i, 1);
            mbar_init(bar_vfree + 8u * i, 1);
            mbar_init(bar_sfull + 8u * i, 1);
            mbar_init(bar_pfull + 8u * i, 16 * PFT_SOFT_WARPS);
        }
        mbar_init(bar_rot, 1);
        mbar_init(bar_done, 1);
        mbar_init(bar_tail, 1);
        mbar_init(bar_q, 1);
        fence_mbar_init();
    }
    if (DIRECT) {
        for (int i = tid; i < CODES * 8; i += PFT_THREADS) {
            const int e = i >> 3;
            lut[i] = DIRECT == 4 ? pack_half2(kCent4[e & 15], kCent4[(e >> 4) & 15]) : pack_half2(kCent2[e & 3], kCent2[(e >> 2) & 3]);
        }
        if (tid == 0) *reinterpret_cast<uint32_t*>(gb + PftSmem::NORM + 8u * PFT_KT) = 0u;  // the largest V norm
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const bool early = DIRECT ? EARLY : PACKED && p.early != 0;
    if (!early) {
        pdl_wait();
        pdl_launch_dependents();  // (the next launch waits for this one's end before it reads or writes anything of the caller's)
    }
    // this block's queries, row (token, head), and R: one copy each (rows behind GRP * QT and tokens past the prompt: whatever comes
    // -- a row's garbage stays in that row and is never stored)
    if (tid == 32 * COPY_WARP) {
        mbar_arrive_expect_tx(bar_q, (uint32_t)(MT * QT * GRP) * 256u + (PACKED ? PFT_TILE : 0u));
        for (int m = 0; m < MT; ++m) {  // a box narrower than the tile: the coordinate halves separately
            tma_load_4d(sb + PftSmem::Q + m * PFT_TILE, &tmQ, bar_q, 0, kvh * GRP, seq * p.T + q0 + m * QT, 0);
            tma_load_4d(sb + PftSmem::Q + m * PFT_TILE + PFT_TILE / 2, &tmQ, bar_q, 0, kvh * GRP, seq * p.T + q0 + m * QT, 1);
        }
        if (PACKED) tma_load_3d(sb + PftSmem::R, &tmR, bar_q, 0, 0, 0);
    }
    const uint32_t tmem = *tmem_slot;
    // softmax warps: slot, 16 score rows (= tensor-memory lanes) row0 ..; a thread's rows row0 + g and row0 + g + 8
    const int slot = (warp >> 2) & 1, row0 = 32 * (warp & 3) + 16 * (warp >> 3), g = lane >> 2, t4 = lane & 3;
    const int my_first = q0 + (MT == 2 ? slot * QT : 0);
    // row / GRP by a multiplication, exact below 128; (made anew where it is used: not live through the tiles)
    auto make_by_grp = [&]() {
        uint32_t d = (uint32_t)GRP;
        asm volatile("" : "+r"(d));
        return (65536u + d - 1u) / d;
    };
    auto token_in = [&](int row, uint32_t by_grp) { return (int)(((uint32_t)row * by_grp) >> 16); };
    auto token_of = [&](int row, uint32_t by_grp) { return token_in(row, by_grp) < QT ? my_first + token_in(row, by_grp) : p.T; };  // (p.T: a row of no query)
    const uint32_t my_lanes = tmem + ((uint32_t)row0 << 16);
    // the warp's rows, columns c0 .. c0 + 63, of an operand tile from a 64-column fragment.  (Pair by pair, with 32 columns of
    // tensor memory at a time and a division per stored row, the way from the last tile to the end took 3.4 us.)
    auto put_frag = [&](uint32_t tile, int c0, const float (&y)[32]) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                auto two = [&](int b) { return pack_half2(y[4 * b + 2 * h], y[4 * b + 2 * h + 1]); };
                stmatrix_x4(sb + tile + pft_chunk(row0 + 8 * h + (lane & 7), (c0 >> 3) + j + (lane >> 3)), two(j), two(j + 1), two(j + 2), two(j + 3));
            }
    };
    // in the products before and after the tiles a warp takes 128 columns of its slot's rows, or with one query block, whose rows
    // both slots' warps share, 64
    constexpr int PCOLS = MT == 2 ? 128 : 64;
    const int pcol0 = MT == 2 ? 0 : 64 * slot;
    const uint32_t pslot = MT == 2 ? (uint32_t)slot : 0u;

    if (PACKED) {
        // ---- q_rot = Q . R^T (reference engine/kernels.cu:1896-1903), scaled by log2(e) / sqrt(128), back into the Q tiles ----
        if (warp == MMA_WARP && lane == 0) {
            wait_bar(bar_q, 0u);
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_lo(tmem + 128u * m, pft_lo_k(sb + PftSmem::Q + m * PFT_TILE) + pft_kstep(ks), pft_lo_k(sb + PftSmem::R) + pft_kstep(ks), PFT_IDESC_K, ks != 0);
            umma_commit(bar_rot);
        }
        auto make_operands = [&]() {
            constexpr int PIECES = 2 * PFT_KT * 16 / (32 * PFT_SOFT_WARPS);  // of 8 codes per thread: K rows, then V rows
            uint32_t c[PIECES];
            const size_t head0 = ((size_t)seq_row0 * p.Hkv + kvh) * 16;
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int row = (tid >> 4) + 32 * (i % (PIECES / 2));
                const size_t at = head0 + (size_t)row * p.Hkv * 16 + (tid & 15);
                const uint8_t* const codes = i < PIECES / 2 ? p.ck : p.cv;
                c[i] = 0u;
                if (row < p.T) c[i] = DIRECT == 4 ? reinterpret_cast<const uint32_t*>(codes)[at] : (uint32_t)reinterpret_cast<const unsigned short*>(codes)[at];
            }
            if (tid < PFT_KT) {
                const size_t at = ((size_t)seq_row0 + tid) * p.Hkv + kvh;
                const float kn = tid < p.T ? __half2float(p.kn[at]) : 0.0f, vn = tid < p.T ? __half2float(p.vn[at]) : 0.0f;
                float* const norms = reinterpret_cast<float*>(gb + PftSmem::NORM);
                norms[tid] = kn;
                norms[PFT_KT + tid] = vn;
                const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(vn));
                if (lane == 0) atomicMax(reinterpret_cast<uint32_t*>(norms + 2 * PFT_KT), top);
            }
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int row = (tid >> 4) + 32 * (i % (PIECES / 2)), copy = tid & 7;
                uint4 u = make_uint4(0u, 0u, 0u, 0u);  // (rows past the prompt)
                if (row < p.T) {
                    constexpr int W = DIRECT == 4 ? 8 : 4;
                    constexpr uint32_t M = CODES - 1;
                    u.x = lut[(c[i] & M) * 8 + copy]; u.y = lut[((c[i] >> W) & M) * 8 + copy];
                    u.z = lut[((c[i] >> (2 * W)) & M) * 8 + copy]; u.w = lut[((c[i] >> (3 * W)) & M) * 8 + copy];
                }
                *reinterpret_cast<uint4*>(gb + (i < PIECES / 2 ? PftSmem::K : PftSmem::V) + pft_chunk(row, tid & 15)) = u;
            }
        };
        if (warp < PFT_SOFT_WARPS) {
            if constexpr (DIRECT && !EARLY) make_operands();
            wait_bar(bar_rot, 0u);
            tc_fence_after();
#pragma unroll 1
            for (int c0 = pcol0; c0 < pcol0 + PCOLS; c0 += 64) {
                uint32_t r[32];
                tmem_ld_frag64(my_lanes + 128u * pslot + (uint32_t)c0, r);
                tmem_ld_wait();
                float y[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) y[e] = __uint_as_float(r[e]) * PFT_SCALE;
                put_frag(PftSmem::Q + pslot * PFT_TILE, c0, y);
                if (LOW) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) y[e] = low_part(y[e]);
                    put_frag(PftSmem::Q + PFT_TILE, c0, y);
                }
            }
            if constexpr (EARLY) {
                pdl_wait();
                make_operands();
            }
        }
        if (warp < PFT_SOFT_WARPS || warp == MMA_WARP) {  // the rotated queries are in place (the copies of the first tiles are on their way already)
            fence_proxy_async_smem();
            tc_fence_before();
            named_barrier(1, 32 * PFT_SOFT_WARPS + 32);
            tc_fence_after();
        }
    }

    if (warp >= PFT_SOFT_WARPS) {
      regs_dec<PFT_REGS_REST>();
      if (warp == COPY_WARP) {
        if (early) {  // (every other warp gets what the launches before this one made from this one's copies)
            pdl_wait();
            pdl_launch_dependents();
        }
        // ================= the copies of every tile =================
        // (fp16 caches, the prompt's last tile: rows past the prompt may hold anything, and 0 x NaN is NaN, so its V rows are blanked)
        const int x_row = (int)seq_row0;
        const float* const norms = PACKED ? p.norms + ((size_t)seq * p.Hkv + kvh) * p.tiles * PFT_NORMS : nullptr;
        for (int j = 0; j < (DIRECT ? 0 : n_tiles); ++j) {
            const int st = j % STAGES, b = j & 1, last = j - STAGES;  // last: the tile that was in this stage
            if (last >= 0) wait_bar(bar_kfree + 8u * (last & 1), (uint32_t)((last >> 1) & 1));
            if (lane == 0 && !dead) {
                mbar_arrive_expect_tx(bar_kfull + 8u * b, (LOW ? 2u : 1u) * PFT_TILE);
                tma_load_3d(sb + PftSmem::K + st * PFT_TILE, &tmK, bar_kfull + 8u * b, 0, x_row + j * PFT_KT, 2 * kvh);
                if (LOW) tma_load_3d(sb + PftSmem::K + PFT_TILE, &tmK, bar_kfull + 8u * b, 0, p.low_row + x_row + j * PFT_KT, 2 * kvh);
            }
            // (V free: the value products of that tile are done, hence its softmax has read its norms)
            if (last >= 0) wait_bar(bar_vfree + 8u * (last & 1), (uint32_t)((last >> 1) & 1));
            const int valid = p.T - j * PFT_KT;
            const bool tail = !PACKED && valid < PFT_KT;
            const uint32_t bar = tail ? bar_tail : bar_vfull + 8u * b;
            if (lane == 0 && !dead) {
                mbar_arrive_expect_tx(bar, (LOW ? 2u : 1u) * PFT_TILE + (PACKED ? PFT_NORM_BYTES : 0u));
                if (PACKED) bulk_load(sb + PftSmem::NORM + st * PFT_NORM_BYTES, norms + (size_t)j * PFT_NORMS, PFT_NORM_BYTES, bar);
                tma_load_3d(sb + PftSmem::V + st * PFT_TILE, &tmV, bar, 0, x_row + j * PFT_KT, 2 * kvh);
                if (LOW) tma_load_3d(sb + PftSmem::V + PFT_TILE, &tmV, bar, 0, p.low_row + x_row + j * PFT_KT, 2 * kvh);
            }
            if (tail) {
                wait_bar(bar_tail, 0u);
                for (int i = lane; i < (PFT_KT - valid) * 16; i += 32)
                    *reinterpret_cast<uint4*>(gb + PftSmem::V + st * PFT_TILE + pft_chunk(valid + (i >> 4), i & 15)) = make_uint4(0u, 0u, 0u, 0u);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_vfull + 8u * b);
            }
        }
      } else if (warp == MMA_WARP) {
        // ================= one thread issues every product =================
        if (lane == 0) {
            // (Two blocks: the products follow each other closely and this thread's own time counts: a wait on a barrier that is complete
            // costs it 100 cycles and more, in which they run out.  So a slot's turn waits for K and V ahead of its weights, and the second
            // slot, which shares them, does not: 8192 tokens, 32 heads, fp16 503 -> 478 us a layer, 4-bit 629 -> 607.  With one block a slot's next
            // tile is two further on and not to be waited for before the values.)
            auto issue_scores = [&](int s, int i) {
                const int j = tile_of(s, i), st = j % STAGES;
                if (MT == 1) {
                    if (!DIRECT) wait_bar(bar_kfull + 8u * (j & 1), (uint32_t)((j >> 1) & 1));
                    tc_fence_after();
                }
                if (dead) return;
                const uint32_t a = pft_lo_k(sb + PftSmem::Q + (MT == 2 ? s * PFT_TILE : 0u)), b = pft_lo_k(sb + PftSmem::K + st * PFT_TILE);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) umma_lo(tmem + 128u * s, a + pft_kstep(ks), b + pft_kstep(ks), PFT_IDESC_K, ks != 0);
                if (LOW) {
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        umma_lo(tmem + 128u * s, a + PFT_TILE / 16u + pft_kstep(ks), b + pft_kstep(ks), PFT_IDESC_K, 1u);
                        umma_lo(tmem + 128u * s, a + pft_kstep(ks), b + PFT_TILE / 16u + pft_kstep(ks), PFT_IDESC_K, 1u);
                    }
                }
                umma_commit(bar_sfull + 8u * s);
                if (MT == 1 || s == (j < n1 ? 1 : 0)) umma_commit(bar_kfree + 8u * (j & 1));  // its last reader
            };
            auto issue_values = [&](int s, int i) {
                const int j = tile_of(s, i), st = j % STAGES;
                if (MT == 1) {
                    if (!DIRECT) wait_bar(bar_vfull + 8u * (j & 1), (uint32_t)((j >> 1) & 1));
                    wait_bar(bar_pfull + 8u * s, (uint32_t)(i & 1));
                    tc_fence_after();
                }
                if (dead) return;
                const uint32_t b = pft_lo_mn(sb + PftSmem::V + st * PFT_TILE);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_lo_ta(tmem + 256u + 128u * s, tmem + 128u * s + 8u * ks, b + 128u * ks, PFT_IDESC_MN, ks == 0 ? (uint32_t)(i != 0) : 1u);
                if (EXACT) {
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks) {
                        umma_lo_ta(tmem + 256u + 128u * s, tmem + 128u * s + 64u + 8u * ks, b + 128u * ks, PFT_IDESC_MN, 1u);
                        if (LOW) umma_lo_ta(tmem + 256u + 128u * s, tmem + 128u * s + 8u * ks, b + PFT_TILE / 16u + 128u * ks, PFT_IDESC_MN, 1u);
                    }
                }
                if (MT == 1 || s == (j < n1 ? 1 : 0)) umma_commit(bar_vfree + 8u * (j & 1));
            };
            if (!PACKED) wait_bar(bar_q, 0u);
            if (MT == 2) {  // (the first block has tiles)
                if (!DIRECT) ready(bar_kfull, 0u);
                tc_fence_after();
            }
            if (n0 > 0) issue_scores(0, 0);
            if (n1 > 0) issue_scores(1, 0);
            if constexpr (MT == 2) {
                auto turn = [&](int s, int i, int n) {
                    if (i >= n) return;
                    if (!DIRECT && (s == 0 || i >= n0)) {
                        ready(bar_vfull + 8u * (i & 1), (uint32_t)((i >> 1) & 1));
                        if (i + 1 < n) ready(bar_kfull + 8u * ((i + 1) & 1), (uint32_t)(((i + 1) >> 1) & 1));
                    } else if (!DIRECT && i + 1 < n && i + 1 >= n0) {  // (the first block ends here)
                        ready(bar_kfull + 8u * ((i + 1) & 1), (uint32_t)(((i + 1) >> 1) & 1));
                    }
                    ready(bar_pfull + 8u * s, (uint32_t)(i & 1));
                    tc_fence_after();
                    issue_values(s, i);
                    if (i + 1 < n) issue_scores(s, i + 1);
                };
                for (int i = 0; i < max(n0, n1); ++i) {
                    turn(0, i, n0);
                    turn(1, i, n1);
                }
            } else
            for (int i = 0; i < max(n0, n1); ++i) {
                if (i < n0) {
                    issue_values(0, i);
                    if (i + 1 < n0) issue_scores(0, i + 1);
                }
                if (i < n1) {
                    issue_values(1, i);
                    if (i + 1 < n1) issue_scores(1, i + 1);
                }
            }
            umma_commit(bar_done);
        }
        __syncwarp();
        if (PACKED) {
            // out[d] = sum_k R[k][d] * acc[k] (reference engine/kernels.cu:1957): the results' high and low parts times R
            named_barrier(1, 32 * PFT_SOFT_WARPS + 32);
            tc_fence_after();
            if (lane == 0 && !dead) {
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int part = 0; part < 2; ++part)
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)
                            umma_lo(tmem + 128u * m, pft_lo_k(sb + (part ? PftSmem::K : PftSmem::Q) + m * PFT_TILE) + pft_kstep(ks),
                                    pft_lo_mn(sb + PftSmem::R) + 128u * ks, PFT_IDESC_MN, (part | ks) != 0);
                umma_commit(bar_rot);
            }
            __syncwarp();
        }
      }
    } else {
        // ================= softmax of slot `slot`, rows row0 + g and row0 + g + 8 =================
        regs_inc<PFT_REGS_SOFT>();
        const uint32_t s_col = my_lanes + 128u * slot, o_col = my_lanes + 256u + 128u * slot;
        const int nt = slot ? n1 : n0;
        const uint32_t by_grp0 = make_by_grp();
        const int tok0 = token_of(row0 + g, by_grp0), tok1 = token_of(row0 + g + 8, by_grp0);
        float m_run[2] = {-1e30f, -1e30f}, l_run[2] = {0.0f, 0.0f};  // (sums: of this thread's columns)
        for (int i = 0; i < nt; ++i) {
            const int j = tile_of(slot, i), st = j % STAGES, col0 = j * PFT_KT;
            if (PACKED && !DIRECT) ready(bar_vfull + 8u * (j & 1), (uint32_t)((j >> 1) & 1));  // (for the tile's norms)
            ready(bar_sfull + 8u * slot, (uint32_t)(i & 1));
            tc_fence_after();
            const bool diagonal = col0 + PFT_KT - 1 > my_first;  // (uniform for the slot)
            const float2* const nrm = reinterpret_cast<const float2*>(gb + PftSmem::NORM + (uint32_t)st * PFT_NORM_BYTES) + t4;
            float v_top = 0.0f;  // the tile's largest V norm: one word, or the largest of eight halves
            if constexpr (DIRECT != 0) {
                v_top = *reinterpret_cast<const float*>(gb + PftSmem::NORM + 8u * PFT_KT);
            } else if constexpr (PACKED) {
                const uint4 u = *reinterpret_cast<const uint4*>(gb + PftSmem::NORM + (uint32_t)st * PFT_NORM_BYTES + 8u * PFT_KT);
                const uint32_t m = __vmaxu2(__vmaxu2(u.x, u.y), __vmaxu2(u.z, u.w));
                v_top = __half2float(__ushort_as_half((unsigned short)max(m & 0xffffu, m >> 16)));
            }
            // ---- scores, scaled (packed: by the K norms), masked; row maxima ----
            uint32_t sr[2][32];
            tmem_ld_frag64(s_col, sr[0]);
            tmem_ld_frag64(s_col + 64u, sr[1]);
            tmem_ld_wait();
            float2 x[2][16];  // [row][column block]
            float mx[2] = {-1e30f, -1e30f};
#pragma unroll
            for (int b = 0; b < 16; ++b) {
                float2 k2;
                if constexpr (PACKED) k2 = nrm[4 * b];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    x[h][b] = make_float2(__uint_as_float(sr[b >> 3][4 * (b & 7) + 2 * h]), __uint_as_float(sr[b >> 3][4 * (b & 7) + 2 * h + 1]));
                    if constexpr (PACKED) x[h][b] = mul2(x[h][b], k2);
                }
            }
            if (diagonal) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int lim = (h ? tok1 : tok0) - col0 - 2 * t4;  // columns up to here count
#pragma unroll
                    for (int b = 0; b < 16; ++b) {
                        if (8 * b > lim) x[h][b].x = -1e30f;
                        if (8 * b + 1 > lim) x[h][b].y = -1e30f;
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float m2 = -1e30f;
#pragma unroll
                for (int b = 0; b < 16; b += 2) {
                    mx[h] = fmaxf(mx[h], fmaxf(x[h][b].x, x[h][b].y));
                    m2 = fmaxf(m2, fmaxf(x[h][b + 1].x, x[h][b + 1].y));
                }
                mx[h] = fmaxf(mx[h], m2);
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
                if (!PACKED) mx[h] *= mx[h] <= -1e30f ? 1.0f : PFT_SCALE;
            }
            // (weights of up to 2^PFT_SLACK times a norm of 4094 still fit fp16; a tile with a larger one keeps its weights below 1)
            const float slack = !PACKED || v_top <= 65504.0f / (float)(1 << (int)PFT_SLACK) ? PFT_SLACK : 0.0f;
            const bool grew0 = mx[0] > m_run[0] + slack, grew1 = mx[1] > m_run[1] + slack;
            if (__any_sync(0xffffffffu, grew0 || grew1)) {
                const float mn0 = grew0 ? mx[0] : m_run[0], mn1 = grew1 ? mx[1] : m_run[1];
                const float corr0 = ex2_approx(m_run[0] - mn0), corr1 = ex2_approx(m_run[1] - mn1);
                m_run[0] = mn0; m_run[1] = mn1;
                l_run[0] *= corr0; l_run[1] *= corr1;
                if (i > 0) {  // S(i) is there, so P(i - 1) V has finished: O is at rest
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t r[16];
                        tmem_ld_frag32(o_col + 32u * c, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * ((e & 2) ? corr1 : corr0));
                        tmem_st_frag32(o_col + 32u * c, r);
                    }
                }
            }
            // ---- P (times the V norm) as fp16 over S ----
            float2 lsum[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
            float2 minus[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)  // (no column counts yet: all weights 0)
                minus[h] = m_run[h] <= -1e29f ? make_float2(0.0f, 0.0f) : make_float2(-m_run[h], -m_run[h]);
            const float2 sc2 = make_float2(PFT_SCALE, PFT_SCALE);
            auto weights = [&](auto masked_is_zero) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t pr[16], pl[EXACT ? 16 : 1];  // EXACT: the low parts behind the high ones, columns 64 ..
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        float2 v2;
                        if constexpr (PACKED) v2 = nrm[64 + 32 * c + 4 * b];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float2 a = PACKED ? add2(x[h][8 * c + b], minus[h]) : fma2(x[h][8 * c + b], sc2, minus[h]);
                            a = make_float2(ex2_approx(a.x), ex2_approx(a.y));
                            lsum[h] = add2(lsum[h], a);
                            if constexpr (PACKED && decltype(masked_is_zero)::value) {
                                a = make_float2(x[h][8 * c + b].x <= -1e30f ? 0.0f : a.x * v2.x, x[h][8 * c + b].y <= -1e30f ? 0.0f : a.y * v2.y);
                            } else if constexpr (PACKED) {
                                a = mul2(a, v2);
                            }
                            pr[2 * b + h] = pack_half2(a.x, a.y);
                            if constexpr (EXACT) pl[2 * b + h] = pack_low_half2(a.x, a.y);
                        }
                    }
                    tmem_st_pack32(s_col + 32u * c, pr);
                    if constexpr (EXACT) tmem_st_pack32(s_col + 64u + 32u * c, pl);
                }
            };
            // a masked weight is 0, and 0 times a V norm that is not finite is not: a tile with such a norm selects instead
            if (PACKED && diagonal && !(v_top < INFINITY)) weights(std::true_type{});
            else weights(std::false_type{});
            l_run[0] += lsum[0].x + lsum[0].y;
            l_run[1] += lsum[1].x + lsum[1].y;
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(bar_pfull + 8u * slot);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
            l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
        }
        wait_bar(bar_done, 0u);  // every product has completed (and nobody reads the norms any more)
        tc_fence_after();

        // ================= results =================
        // MT = 2: a slot's rows are its own.  MT = 1: the slots' sums over the same rows meet; slot s finishes the columns 64 s ..
        float w0[2], w1[2] = {0.0f, 0.0f};  // by row: weights of the slots' sums, normalised (MT = 2: of its own)
        if constexpr (MT == 1) {
            float2* const xch = reinterpret_cast<float2*>(gb + PftSmem::NORM);
            if (t4 == 0) {
                xch[slot * 128 + row0 + g] = make_float2(m_run[0], l_run[0]);
                xch[slot * 128 + row0 + g + 8] = make_float2(m_run[1], l_run[1]);
            }
            named_barrier(2, 32 * PFT_SOFT_WARPS);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 a = xch[row0 + g + 8 * h], b = xch[128 + row0 + g + 8 * h];
                const float M = fmaxf(a.x, b.x), e0 = ex2_approx(a.x - M), e1 = n1 > 0 ? ex2_approx(b.x - M) : 0.0f;
                const float inv = 1.0f / (a.y * e0 + b.y * e1 + 1e-8f);
                w0[h] = e0 * inv;
                w1[h] = e1 * inv;
            }
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) w0[h] = 1.0f / (l_run[h] + 1e-8f);
        }
        const bool has_rows = MT == 1 || nt > 0;
        auto result = [&](int c0, float (&y)[32]) {  // columns c0 .. c0 + 63, normalised, in fragment order
            uint32_t r[32];
            tmem_ld_frag64((MT == 2 ? o_col : my_lanes + 256u) + (uint32_t)c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) y[e] = __uint_as_float(r[e]) * w0[(e >> 1) & 1];
            if (MT == 1 && n1 > 0) {
                tmem_ld_frag64(my_lanes + 384u + (uint32_t)c0, r);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) y[e] = fmaf(__uint_as_float(r[e]), w1[(e >> 1) & 1], y[e]);
            }
        };
        const uint32_t qtile = PftSmem::Q + pslot * PFT_TILE, ktile = PftSmem::K + pslot * PFT_TILE;
        if constexpr (PACKED) {
            // out[d] = sum_k R[k][d] * acc[k]: the normalised rows, split into fp16 high and low parts, over the Q and K tiles
            if (has_rows) {
#pragma unroll 1
                for (int c0 = pcol0; c0 < pcol0 + PCOLS; c0 += 64) {
                    float y[32];
                    result(c0, y);
                    put_frag(qtile, c0, y);
#pragma unroll
                    for (int e = 0; e < 32; ++e) y[e] = low_part(y[e]);
                    put_frag(ktile, c0, y);
                }
            }
            fence_proxy_async_smem();
            tc_fence_before();
            named_barrier(1, 32 * PFT_SOFT_WARPS + 32);
            wait_bar(bar_rot, 1u);
            tc_fence_after();
        }
        if (has_rows) {
            // the finished values as fp16 through the (consumed) query tile, so that 16 lanes store 256 contiguous bytes of a row
#pragma unroll 1
            for (int c0 = pcol0; c0 < pcol0 + PCOLS; c0 += 64) {
                float y[32];
                if constexpr (PACKED) {
                    uint32_t r[32];
                    tmem_ld_frag64(my_lanes + 128u * pslot + (uint32_t)c0, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) y[e] = __uint_as_float(r[e]);
                } else {
                    result(c0, y);
                }
                put_frag(qtile, c0, y);
            }
            __syncwarp();
            constexpr int CH = PCOLS / 8;  // 16-byte pieces per row
            const uint32_t by_grp = make_by_grp();
#pragma unroll
            for (int k = 0; k < CH / 2; ++k) {
                const int at = 32 * k + lane, row = row0 + at / CH, ch = (pcol0 >> 3) + at % CH, tok = token_of(row, by_grp);
                if (tok < p.T) {
                    const uint4 u = *reinterpret_cast<const uint4*>(gb + qtile + pft_chunk(row, ch));
                    *(reinterpret_cast<uint4*>(out_seq + (size_t)tok * p.q_dim + (size_t)(kvh * GRP + row - token_in(row, by_grp) * GRP) * HEAD_DIM) + ch) = u;
                }
            }
        }
        tc_fence_before();
    }
    if (dead) {  // copies and products may still be in flight: a bounded chance to land before shared and tensor memory go away
        for (int i = 0; i < 4; ++i) {
            mbar_wait_bounded_hint(bar_kfull + 8u * i, 0u, 1u << 10, 2000u);  // (kfull[2], vfull[2])
            mbar_wait_bounded_hint(bar_kfull + 8u * i, 1u, 1u << 10, 2000u);
        }
        mbar_wait_bounded_hint(bar_done, 0u, 1u << 10, 2000u);
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512u);
}

}  // namespace tq
