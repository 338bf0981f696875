// Causal prefill attention on the 5th-generation tensor cores (tcgen05 + tensor memory), sm_100a.
//
// Query token t of a prompt attends to cache rows 0 .. t (reference engine/kernels.cu:1874-1960 packed, :1071-1158 fp16).
// One CTA has two SLOTS that work in turn, so that the tensor core always has a product of one slot while the softmax of the
// other runs.  A slot = 128 score rows (128 / GRP query tokens x the GRP query heads of one KV head) = the M dimension,
// a warpgroup of softmax threads (one thread per row), 128 columns of tensor memory for S and 128 for O:
//   * long prompts (MT = 2): the slots are two consecutive query blocks that share every K and V tile;
//   * short ones (MT = 1): both slots hold the same query block and take the even and the odd tiles; their results are
//     combined at the end.  Twice the CTAs and half the chain when there are not enough blocks for the GPU.
// Tiles are 128 cache rows.  K lies in shared memory as [coordinate half][128 rows][128 B] (K-major B operand of S = Q K^T),
// V in the same form, read as an MN-major B operand of O += P V: no transposition anywhere, both arrive by one tensor-map
// copy.  Packed caches are turned into fp16 centroids (unscaled: the same operands as ever) and fp32 norms by
// dequantize_rows_kernel first, once per prompt and layer instead of once per query block: done by producer warps inside
// this kernel the table look-ups and operand stores took as much of the shared-memory pipe as the products themselves (8192
// tokens, 16/8 heads, 4-bit: 617 us against 439).  P (times the V norm, fp16) replaces S in tensor memory and is read from
// there as the A operand.
//   warps 0-7    softmax of slots 0 and 1: S -> registers, K norm, causal limit, exponentials, P -> tensor memory.  The
//                exponentials' reference point follows the row maximum only when that has grown by more than PFT_SLACK (in
//                powers of two): weights stay below 2^PFT_SLACK and O is rescaled in place in the first tiles only.
//   warp 8       issues the copies; warp 9 issues every product, in the order P(i) V -> S(i + 1) per slot, slots alternating: the
//                products of one thread execute in order, so S(i + 1) may overwrite the P(i) that the one before it reads.
// Packed forms: Q R^T at the start and (O / l) R at the end (fp16 high + low parts) are tcgen05 products too.
// Every wait on a barrier is bounded; a wait that runs out raises the status word and the kernel runs to its end.
// Bound by the softmax threads (exponentials, tensor-memory loads) against the tensor core at long prompts, by the chain copy ->
// S -> softmax -> O of a single block at short ones.  Per layer, 8 KV heads, cache write included, the one-block kernel with V
// transposed through shared memory -> this one: fp16 8192 tokens 32 heads 2811 -> 530 us (1040 TFLOP/s of causal arithmetic), 777
// tokens 59 -> 31; 4-bit 8192 tokens 16 heads 763 -> 379 us, 777 tokens 43.7 -> 34.2.
#pragma once

#include "tq_prefill_tc.cuh"

namespace tq {

constexpr int PFT_ROWS = 128;     // score rows of a slot
constexpr int PFT_KT = 128;       // cache rows per tile
constexpr float PFT_SLACK = 4.0f;
constexpr float PFT_SCALE = 0.12751743074602467f;  // log2(e) / sqrt(128); packed forms: carried by the rotated queries
constexpr uint32_t PFT_TILE = 32768u;  // an operand tile: [2 halves of the coordinates][128 rows][128 B]

constexpr int PFT_THREADS = 384;  // 8 softmax warps, one for the copies, one for the products, two idle (a full warpgroup)
// Registers per thread of the softmax and the other warpgroup after the split.  The launch must bring at least their sum (the
// host checks what the kernel was built with): 384 x 168 >= 256 x 200 + 128 x 88.
constexpr int PFT_REGS_SOFT = 200, PFT_REGS_REST = 88;
constexpr int PFT_REGS_LAUNCH = (256 * PFT_REGS_SOFT + 128 * PFT_REGS_REST + PFT_THREADS - 1) / PFT_THREADS;

struct PrefillAttnParams {
    const __half* q;          // queries [n_seq][T][q_tok_stride] as the model makes them
    long long q_tok_stride;   // halves between the queries of consecutive tokens
    const uint8_t* ck;        // (host) packed codes [rows][kvp] or fp16 rows [rows][Hkv * 128]; the kernel reads through its maps
    const uint8_t* cv;
    const __half* kn;         // (host) [rows][Hkv], packed caches
    const __half* vn;
    const __half* rotation;   // packed: R row-major [128][128]
    const float* norms;       // packed: fp32 [n_seq][Hkv][K, V][t_pad] (dequantize_rows_kernel)
    int t_pad;
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
    static constexpr uint32_t NORM = R + PFT_TILE;      // [2 stages][K, V][128] floats; MT = 1, at the end: [2 slots][128][maximum, sum]
    static constexpr uint32_t CTRL = NORM + 2048u;      // mbarriers, tensor-memory base
    static constexpr uint32_t BYTES = CTRL + 256u;
};

// Packed prompts for the kernel below: rows first_row .. of one KV cache array pair as fp16 centroids [n_seq][T][kv_dim] and fp32
// norms [n_seq][Hkv][K, V][t_pad] (zero behind the prompt).  One thread per 8 codes; bound by HBM / L2 writes of the fp16 rows.
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
    int T, t_pad, Hkv;
};
template <int BITS>
__global__ void __launch_bounds__(256) dequantize_rows_kernel(const DequantParams p) {
    // byte (4-bit) or nibble (2-bit) -> two centroids; eight copies, so that at most four lanes of a warp share a bank
    constexpr int ENTRIES = BITS == 4 ? 256 : 16;
    __shared__ uint32_t lut[ENTRIES * 8];
    for (int i = threadIdx.x; i < ENTRIES * 8; i += 256) {
        const int e = i >> 3;
        lut[i] = BITS == 4 ? pack_half2(kCent4[e & 15], kCent4[e >> 4]) : pack_half2(kCent2[e & 3], kCent2[(e >> 2) & 3]);
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();  // the rows come from the append before this launch
    const int seq = blockIdx.y;
    const long long row0 = p.row_base ? p.row_base[seq] : (long long)seq * p.seq_rows;
    const int words = p.Hkv * 16;  // 8-code pieces per row
    const long long n = (long long)p.T * words;
    const int copy = threadIdx.x & 7;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < 2 * n; i += (long long)gridDim.x * 256) {
        const bool is_v = i >= n;
        const long long w = is_v ? i - n : i;
        uint4 u;
        if (BITS == 4) {
            const uint32_t c = *(reinterpret_cast<const uint32_t*>(is_v ? p.cv : p.ck) + row0 * words + w);
            u.x = lut[(c & 0xffu) * 8 + copy]; u.y = lut[((c >> 8) & 0xffu) * 8 + copy];
            u.z = lut[((c >> 16) & 0xffu) * 8 + copy]; u.w = lut[(c >> 24) * 8 + copy];
        } else {
            const uint32_t c = *(reinterpret_cast<const unsigned short*>(is_v ? p.cv : p.ck) + row0 * words + w);
            u.x = lut[(c & 0xfu) * 8 + copy]; u.y = lut[((c >> 4) & 0xfu) * 8 + copy];
            u.z = lut[((c >> 8) & 0xfu) * 8 + copy]; u.w = lut[(c >> 12) * 8 + copy];
        }
        *(reinterpret_cast<uint4*>(is_v ? p.v16 : p.k16) + (long long)seq * n + w) = u;
    }
    const long long m = (long long)p.t_pad * p.Hkv;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < 2 * m; i += (long long)gridDim.x * 256) {
        const bool is_v = i >= m;
        const long long w = is_v ? i - m : i;
        const int t = (int)(w / p.Hkv), h = (int)(w - (long long)t * p.Hkv);
        const float x = t < p.T ? __half2float((is_v ? p.vn : p.kn)[(row0 + t) * p.Hkv + h]) : 0.0f;
        p.norms[(((long long)seq * p.Hkv + h) * 2 + (is_v ? 1 : 0)) * p.t_pad + t] = x;
    }
}

// 32 lanes x 32 consecutive 32-bit columns, registers -> tensor memory (the counterpart of tmem_ld32)
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
        "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
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

// PACKED: ck, cv are the fp16 centroids [n_seq * T][kv_dim] of dequantize_rows_kernel (seq_rows = T, no row_base), p.norms its norms
template <bool PACKED, int MT>
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
    constexpr int MMA_WARP = 9;
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
            mbar_init(bar_pfull + 8u * i, PFT_ROWS);
        }
        mbar_init(bar_rot, 1);
        mbar_init(bar_done, 1);
        mbar_init(bar_tail, 1);
        mbar_init(bar_q, 1);
        fence_mbar_init();
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    // this block's queries, row (token, head), and R: one copy each (rows behind GRP * QT and tokens past the prompt: whatever comes
    // -- a row's garbage stays in that row and is never stored)
    if (tid == 256) {
        mbar_arrive_expect_tx(bar_q, (uint32_t)(MT * QT * GRP) * 256u + (PACKED ? PFT_TILE : 0u));
        for (int m = 0; m < MT; ++m) {  // a box narrower than the tile: the coordinate halves separately
            tma_load_4d(sb + PftSmem::Q + m * PFT_TILE, &tmQ, bar_q, 0, kvh * GRP, seq * p.T + q0 + m * QT, 0);
            tma_load_4d(sb + PftSmem::Q + m * PFT_TILE + PFT_TILE / 2, &tmQ, bar_q, 0, kvh * GRP, seq * p.T + q0 + m * QT, 1);
        }
        if (PACKED) tma_load_3d(sb + PftSmem::R, &tmR, bar_q, 0, 0, 0);
    }
    const uint32_t tmem = *tmem_slot;
    // softmax threads: slot, score row = tensor-memory lane, the row's token and query head
    const int slot = warp >> 2, srow = (warp & 3) * 32 + lane;
    const int my_t = srow / GRP, my_first = q0 + (MT == 2 ? slot * QT : 0);
    const int my_tok = my_t < QT ? my_first + my_t : p.T;  // (p.T: a row of no query)
    const int my_head = kvh * GRP + (srow - my_t * GRP);
    const uint32_t my_lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);

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
        if (warp < 4 * MT) {
            wait_bar(bar_rot, 0u);
            tc_fence_after();
#pragma unroll 1
            for (int c2 = 0; c2 < 4; ++c2) {
                uint32_t r[32];
                tmem_ld32(my_lanes + 128u * slot + 32u * c2, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float sc = PFT_SCALE;
                    uint4 u;
                    u.x = pack_half2(__uint_as_float(r[8 * i]) * sc, __uint_as_float(r[8 * i + 1]) * sc);
                    u.y = pack_half2(__uint_as_float(r[8 * i + 2]) * sc, __uint_as_float(r[8 * i + 3]) * sc);
                    u.z = pack_half2(__uint_as_float(r[8 * i + 4]) * sc, __uint_as_float(r[8 * i + 5]) * sc);
                    u.w = pack_half2(__uint_as_float(r[8 * i + 6]) * sc, __uint_as_float(r[8 * i + 7]) * sc);
                    *reinterpret_cast<uint4*>(gb + PftSmem::Q + slot * PFT_TILE + pft_chunk(srow, 4 * c2 + i)) = u;
                }
            }
        }
        if (warp < 8 || warp == MMA_WARP) {  // the rotated queries are in place (the copies of the first tiles are on their way already)
            fence_proxy_async_smem();
            tc_fence_before();
            named_barrier(1, 288);
            tc_fence_after();
        }
    }

    float m_run = -1e30f, l_run = 0.0f;
    if (warp >= 8) {
      regs_dec<PFT_REGS_REST>();
      if (warp == 8) {
        // ================= the copies of every tile =================
        // (fp16 caches, the prompt's last tile: rows past the prompt may hold anything, and 0 x NaN is NaN, so its V rows are blanked)
        const int x_row = (int)seq_row0;
        const float* const norms = PACKED ? p.norms + ((size_t)seq * p.Hkv + kvh) * 2 * p.t_pad : nullptr;
        for (int j = 0; j < n_tiles; ++j) {
            const int st = j & 1;
            const uint32_t again = (uint32_t)(((j >> 1) - 1) & 1);
            if (j > 1) wait_bar(bar_kfree + 8u * st, again);
            if (lane == 0 && !dead) {
                mbar_arrive_expect_tx(bar_kfull + 8u * st, PFT_TILE);
                tma_load_3d(sb + PftSmem::K + st * PFT_TILE, &tmK, bar_kfull + 8u * st, 0, x_row + j * PFT_KT, 2 * kvh);
            }
            // (V free: the value products of the tile two back are done, hence its softmax has read its norms)
            if (j > 1) wait_bar(bar_vfree + 8u * st, again);
            const int valid = p.T - j * PFT_KT;
            const bool tail = !PACKED && valid < PFT_KT;
            const uint32_t bar = tail ? bar_tail : bar_vfull + 8u * st;
            if (lane == 0 && !dead) {
                mbar_arrive_expect_tx(bar, PFT_TILE + (PACKED ? 1024u : 0u));
                if (PACKED) {
                    bulk_load(sb + PftSmem::NORM + st * 1024u, norms + j * PFT_KT, 512u, bar);
                    bulk_load(sb + PftSmem::NORM + st * 1024u + 512u, norms + p.t_pad + j * PFT_KT, 512u, bar);
                }
                tma_load_3d(sb + PftSmem::V + st * PFT_TILE, &tmV, bar, 0, x_row + j * PFT_KT, 2 * kvh);
            }
            if (tail) {
                wait_bar(bar_tail, 0u);
                for (int i = lane; i < (PFT_KT - valid) * 16; i += 32)
                    *reinterpret_cast<uint4*>(gb + PftSmem::V + st * PFT_TILE + pft_chunk(valid + (i >> 4), i & 15)) = make_uint4(0u, 0u, 0u, 0u);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_vfull + 8u * st);
            }
        }
      } else if (warp == MMA_WARP) {
        // ================= one thread issues every product =================
        if (lane == 0) {
            auto issue_scores = [&](int s, int i) {
                const int j = tile_of(s, i), st = j & 1;
                wait_bar(bar_kfull + 8u * st, (uint32_t)((j >> 1) & 1));
                tc_fence_after();
                if (dead) return;
                const uint32_t a = pft_lo_k(sb + PftSmem::Q + (MT == 2 ? s * PFT_TILE : 0u)), b = pft_lo_k(sb + PftSmem::K + st * PFT_TILE);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) umma_lo(tmem + 128u * s, a + pft_kstep(ks), b + pft_kstep(ks), PFT_IDESC_K, ks != 0);
                umma_commit(bar_sfull + 8u * s);
                if (MT == 1 || s == (j < n1 ? 1 : 0)) umma_commit(bar_kfree + 8u * st);  // its last reader
            };
            auto issue_values = [&](int s, int i) {
                const int j = tile_of(s, i), st = j & 1;
                wait_bar(bar_vfull + 8u * st, (uint32_t)((j >> 1) & 1));
                wait_bar(bar_pfull + 8u * s, (uint32_t)(i & 1));
                tc_fence_after();
                if (dead) return;
                const uint32_t b = pft_lo_mn(sb + PftSmem::V + st * PFT_TILE);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_lo_ta(tmem + 256u + 128u * s, tmem + 128u * s + 8u * ks, b + 128u * ks, PFT_IDESC_MN, ks == 0 ? (uint32_t)(i != 0) : 1u);
                if (MT == 1 || s == (j < n1 ? 1 : 0)) umma_commit(bar_vfree + 8u * st);
            };
            if (!PACKED) wait_bar(bar_q, 0u);
            if (n0 > 0) issue_scores(0, 0);
            if (n1 > 0) issue_scores(1, 0);
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
            named_barrier(1, 288);
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
        // ================= softmax of slot `slot`, row `srow` =================
        regs_inc<PFT_REGS_SOFT>();
        const uint32_t s_col = my_lanes + 128u * slot, o_col = my_lanes + 256u + 128u * slot;
        const int nt = slot ? n1 : n0;
        for (int i = 0; i < nt; ++i) {
            const int j = tile_of(slot, i), st = j & 1, col0 = j * PFT_KT;
            if (PACKED) wait_bar(bar_vfull + 8u * st, (uint32_t)((j >> 1) & 1));  // (for the tile's norms)
            wait_bar(bar_sfull + 8u * slot, (uint32_t)(i & 1));
            tc_fence_after();
            const bool diagonal = col0 + PFT_KT - 1 > my_first;  // (uniform for the slot)
            const int lim = my_tok - col0;                        // columns up to here count
            const float4* const nrm = reinterpret_cast<const float4*>(gb + PftSmem::NORM + (uint32_t)st * 1024u);
            // S comes out of tensor memory twice, 64 columns at a time: once for the row maximum, once for the weights.  Holding
            // all 128 columns in between would save four loads and cost an unrolled body of several thousand instructions, which a
            // short prompt spends its time fetching (777 tokens, 16/8 heads, 4-bit: 38.9 us a layer that way, 35.2 this way).
            auto load64 = [&](int c, float2 (&x)[32]) {  // 64 scores, scaled (packed: by the K norms), masked
                uint32_t r[2][32];
                tmem_ld32(s_col + 64u * c, r[0]);
                tmem_ld32(s_col + 64u * c + 32u, r[1]);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    const uint32_t* w = &r[e >> 4][2 * (e & 15)];
                    x[e] = make_float2(__uint_as_float(w[0]), __uint_as_float(w[1]));
                    x[e + 1] = make_float2(__uint_as_float(w[2]), __uint_as_float(w[3]));
                    if constexpr (PACKED) {
                        const float4 k4 = nrm[16 * c + (e >> 1)];
                        x[e] = mul2(x[e], make_float2(k4.x, k4.y));
                        x[e + 1] = mul2(x[e + 1], make_float2(k4.z, k4.w));
                    }
                }
                if (diagonal) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        if (64 * c + 2 * e > lim) x[e].x = -1e30f;
                        if (64 * c + 2 * e + 1 > lim) x[e].y = -1e30f;
                    }
                }
            };
            float mx = -1e30f;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                float2 x[32];
                load64(c, x);
                float m2 = -1e30f;
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    mx = fmaxf(mx, fmaxf(x[e].x, x[e].y));
                    m2 = fmaxf(m2, fmaxf(x[e + 1].x, x[e + 1].y));
                }
                mx = fmaxf(mx, m2);
            }
            if (!PACKED) mx *= mx <= -1e30f ? 1.0f : PFT_SCALE;
            const bool grew = mx > m_run + PFT_SLACK;
            const float mn = grew ? mx : m_run;
            const float corr = ex2_approx(m_run - mn);
            m_run = mn;
            if (i > 0 && __any_sync(0xffffffffu, grew)) {  // S(i) is there, so P(i - 1) V has finished: O is at rest
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld32(o_col + 32u * c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * corr);
                    tmem_st32(o_col + 32u * c, r);
                }
            }
            // ---- P (times the V norm) as fp16 over S: the columns a store covers have been read by then ----
            float2 lsum2 = make_float2(0.0f, 0.0f);
            const float2 sc2 = make_float2(PFT_SCALE, PFT_SCALE);
            const float2 minus = mn <= -1e29f ? make_float2(0.0f, 0.0f) : make_float2(-mn, -mn);  // (no column counts yet: all weights 0)
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                float2 x[32];
                load64(c, x);
                uint32_t pr[2][16];
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    float4 v4;
                    if constexpr (PACKED) v4 = nrm[32 + 16 * c + (e >> 1)];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float2 a = PACKED ? add2(x[e + h], minus) : fma2(x[e + h], sc2, minus);
                        a = make_float2(ex2_approx(a.x), ex2_approx(a.y));
                        lsum2 = add2(lsum2, a);
                        if constexpr (PACKED) a = mul2(a, h ? make_float2(v4.z, v4.w) : make_float2(v4.x, v4.y));
                        pr[e >> 4][(e & 15) + h] = pack_half2(a.x, a.y);
                    }
                }
                tmem_st16(s_col + 32u * c, pr[0]);
                tmem_st16(s_col + 32u * c + 16u, pr[1]);
            }
            l_run = l_run * corr + (lsum2.x + lsum2.y);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(bar_pfull + 8u * slot);
        }
        wait_bar(bar_done, 0u);  // every product has completed (and nobody reads the norms any more)
        tc_fence_after();

        // ================= results =================
        // MT = 2: a slot's rows are its own.  MT = 1: the slots' sums over the same rows meet; slot s finishes the coordinate half s.
        float inv, w0 = 0.0f, w1 = 0.0f;
        if constexpr (MT == 1) {
            float2* const xch = reinterpret_cast<float2*>(gb + PftSmem::NORM);
            xch[slot * 128 + srow] = make_float2(m_run, l_run);
            named_barrier(2, 256);
            const float2 a = xch[srow], b = xch[128 + srow];
            const float M = fmaxf(a.x, b.x), e0 = ex2_approx(a.x - M), e1 = n1 > 0 ? ex2_approx(b.x - M) : 0.0f;
            inv = 1.0f / (a.y * e0 + b.y * e1 + 1e-8f);
            w0 = e0 * inv;
            w1 = e1 * inv;
        } else {
            inv = 1.0f / (l_run + 1e-8f);
        }
        auto result = [&](int c2, float (&x)[32]) {  // this row's columns 32 c2 .., normalised
            uint32_t r[32];
            tmem_ld32(MT == 2 ? o_col + 32u * c2 : my_lanes + 256u + 32u * c2, r);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) x[e] = __uint_as_float(r[e]) * (MT == 2 ? inv : w0);
            if (MT == 1 && n1 > 0) {
                tmem_ld32(my_lanes + 384u + 32u * c2, r);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) x[e] = fmaf(__uint_as_float(r[e]), w1, x[e]);
            }
        };
        const int c_begin = MT == 2 ? 0 : 2 * slot, c_end = MT == 2 ? 4 : 2 * slot + 2;
        __half* const dst = out_seq + (size_t)my_tok * p.q_dim + (size_t)my_head * HEAD_DIM;
        const bool has_rows = MT == 1 || nt > 0, stores = my_tok < p.T;
        auto store32 = [&](int c2, const float (&x)[32]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint4 u;
                u.x = pack_half2(x[8 * i], x[8 * i + 1]); u.y = pack_half2(x[8 * i + 2], x[8 * i + 3]);
                u.z = pack_half2(x[8 * i + 4], x[8 * i + 5]); u.w = pack_half2(x[8 * i + 6], x[8 * i + 7]);
                *reinterpret_cast<uint4*>(dst + 32 * c2 + 8 * i) = u;
            }
        };
        if constexpr (!PACKED) {
            if (has_rows) {
#pragma unroll 1
                for (int c2 = c_begin; c2 < c_end; ++c2) {
                    float x[32];
                    result(c2, x);
                    if (stores) store32(c2, x);
                }
            }
        } else {
            // the normalised rows, split into fp16 high and low parts, over the Q and K tiles
            const int m = MT == 2 ? slot : 0;
            if (has_rows) {
#pragma unroll 1
                for (int c2 = c_begin; c2 < c_end; ++c2) {
                    float x[32];
                    result(c2, x);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 uh, ul;
                        uint32_t* ph = &uh.x;
                        uint32_t* pl = &ul.x;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float x0 = x[8 * i + 2 * e], x1 = x[8 * i + 2 * e + 1];
                            const __half2 h = __floats2half2_rn(x0, x1);
                            const float2 f = __half22float2(h);
                            ph[e] = *reinterpret_cast<const uint32_t*>(&h);
                            pl[e] = pack_half2(x0 - f.x, x1 - f.y);
                        }
                        *reinterpret_cast<uint4*>(gb + PftSmem::Q + m * PFT_TILE + pft_chunk(srow, 4 * c2 + i)) = uh;
                        *reinterpret_cast<uint4*>(gb + PftSmem::K + m * PFT_TILE + pft_chunk(srow, 4 * c2 + i)) = ul;
                    }
                }
            }
            fence_proxy_async_smem();
            tc_fence_before();
            named_barrier(1, 288);
            wait_bar(bar_rot, 1u);
            tc_fence_after();
            if (has_rows) {
#pragma unroll 1
                for (int c2 = c_begin; c2 < c_end; ++c2) {
                    uint32_t r[32];
                    float x[32];
                    tmem_ld32(my_lanes + 128u * m + 32u * c2, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) x[e] = __uint_as_float(r[e]);
                    if (stores) store32(c2, x);
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
