// Host side of the library: tensor-map encoding, launch wrappers with argument checks, the per-device
// workspace used by the reference-compatible launchers, and the KV arena / engine state that the
// reference keeps inside InferenceEngine (engine/engine.cpp:292-409, 893-1022, 1338-1620).
#pragma once

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <random>
#include <tuple>
#include <vector>

#include <cudaTypedefs.h>

#include "../../include/triebwerk_b200.h"
#include "tq_append.cuh"
#include "tq_prefill_tc.cuh"
#include "tq_attention.cuh"
#include "tq_common.cuh"
#include "tq_decode_cluster.cuh"
#include "tq_fp16.cuh"
#include "tq_fp16_tc.cuh"
#include "tq_layer_prep.cuh"
#include "tq_qrot.cuh"
#include "tq_generic.cuh"
#include "tq_prefill_fa.cuh"

namespace tq {

inline int cuda_status(cudaError_t e) { return e == cudaSuccess ? TQ_OK : (int)e; }

#define TQ_CUDA(call)                                  \
    do {                                               \
        cudaError_t _e = (call);                       \
        if (_e != cudaSuccess) return (int)_e;         \
    } while (0)

struct DeviceProps {
    int sm_count = 0;
};

inline DeviceProps& device_props() {
    static std::mutex mu;
    static std::map<int, DeviceProps> props;
    std::lock_guard<std::mutex> lock(mu);
    int dev = 0;
    cudaGetDevice(&dev);
    DeviceProps& d = props[dev];
    if (d.sm_count == 0) {
        cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (d.sm_count <= 0) d.sm_count = 1;
    }
    return d;
}

// ---- TMA descriptors ----------------------------------------------------------------------------------------------
inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

// Code array viewed as uint8 [rows][kvp]; box = 128 bytes x TILE_TOKENS rows, 128-byte swizzle in shared memory.
inline int make_code_map(CUtensorMap* m, const void* base, long long rows, int kvp) {
    auto fn = encode_fn();
    if (!fn) return TQ_ERR_UNSUPPORTED;
    if (((uintptr_t)base & 15u) != 0 || rows <= 0 || rows >= (1ll << 31) || kvp % 128 != 0) return TQ_ERR_ARG;
    // Three dimensions: 128 bytes of a row, the rows, and the 128-byte column blocks of a row.  One box covers a whole
    // tile (32 rows x all column blocks) and lands in shared memory as [column block][row][128 B]: one copy
    // instruction per tile and array, and the 128-byte swizzle still goes by the row number.
    cuuint64_t dims[3] = {128u, (cuuint64_t)rows, (cuuint64_t)(kvp / 128)};
    cuuint64_t strides[2] = {(cuuint64_t)kvp, 128u};
    cuuint32_t box[3] = {128u, (cuuint32_t)TILE_TOKENS, (cuuint32_t)(kvp / 128)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TQ_OK : TQ_ERR_ARG;
}

// fp16 K or V array [rows][kv_dim] viewed as bytes for fp16_tc_decode_attention_kernel: box = one head's 256 bytes
// (two 128-byte blocks) x 16 rows, 128-byte swizzle.
inline int make_fp16_rows_map(CUtensorMap* m, const void* base, long long rows, int kv_dim) {
    auto fn = encode_fn();
    if (!fn) return TQ_ERR_UNSUPPORTED;
    const long long row_bytes = (long long)kv_dim * 2;
    if (((uintptr_t)base & 15u) != 0 || rows <= 0 || rows >= (1ll << 31) || row_bytes % 256 != 0) return TQ_ERR_ARG;
    cuuint64_t dims[3] = {128u, (cuuint64_t)rows, (cuuint64_t)(row_bytes / 128)};
    cuuint64_t strides[2] = {(cuuint64_t)row_bytes, 128u};
    cuuint32_t box[3] = {128u, (cuuint32_t)FP16TC_BLOCK, 2u};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TQ_OK : TQ_ERR_ARG;
}

// All layers' code arrays (layer_stride bytes apart) as ONE map with the layer as the fourth coordinate; same boxes.
inline int make_code_map_layers(CUtensorMap* m, const void* base, long long rows, int kvp, int layers, size_t layer_stride) {
    auto fn = encode_fn();
    if (!fn) return TQ_ERR_UNSUPPORTED;
    if (((uintptr_t)base & 15u) != 0 || rows <= 0 || rows >= (1ll << 31) || kvp % 128 != 0 || layers <= 0 ||
        (layer_stride & 15u) != 0 || layer_stride < (size_t)rows * kvp)
        return TQ_ERR_ARG;
    cuuint64_t dims[4] = {128u, (cuuint64_t)rows, (cuuint64_t)(kvp / 128), (cuuint64_t)layers};
    cuuint64_t strides[3] = {(cuuint64_t)kvp, 128u, (cuuint64_t)layer_stride};
    cuuint32_t box[4] = {128u, (cuuint32_t)TILE_TOKENS, (cuuint32_t)(kvp / 128), 1u};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TQ_OK : TQ_ERR_ARG;
}

// fp16 K or V input of an append, [tokens][kv_dim] halves, for prefill_append_tc_kernel's TMA form: one box = the 128 head
// vectors of a tile (128 / Hkv tokens x Hkv heads), landing in shared memory as [half of the vector][token][head][128 B]
// with the 128-byte swizzle -- the K-major operand layout of the tensor core, no instruction of the SM involved.
inline int make_append_input_map(CUtensorMap* m, const void* base, long long tokens, int Hkv, int kv_dim) {
    auto fn = encode_fn();
    if (!fn) return TQ_ERR_UNSUPPORTED;
    const long long row_bytes = (long long)kv_dim * 2;
    if (((uintptr_t)base & 15u) != 0 || tokens <= 0 || tokens >= (1ll << 31) || Hkv <= 0 || Hkv > TC_TILE || TC_TILE % Hkv != 0 ||
        row_bytes % 16 != 0 || kv_dim < Hkv * HEAD_DIM)
        return TQ_ERR_ARG;
    cuuint64_t dims[4] = {128u, (cuuint64_t)Hkv, (cuuint64_t)tokens, 2u};
    cuuint64_t strides[3] = {256u, (cuuint64_t)row_bytes, 128u};
    cuuint32_t box[4] = {128u, (cuuint32_t)Hkv, (cuuint32_t)(TC_TILE / Hkv), 2u};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TQ_OK : TQ_ERR_ARG;
}

// ---- workspace ------------------------------------------------------------------------------------------------------
// The carve of tq_common.cuh plus the transposed rotation; the fp16 twin's ticket/partial area aliases the packed path's partials.
struct FullWorkspace {
    Workspace w;
    __half* rot_t;         // [128][128] transposed rotation (for callers that only hand over R)
    size_t bytes;
};

inline FullWorkspace carve_full(void* base, int G, int H) {
    FullWorkspace f;
    f.w = carve_workspace(base, G, H);
    size_t off = f.w.bytes;
    char* p = (char*)base;
    f.rot_t = (__half*)(p + off);
    off += (size_t)HEAD_DIM * HEAD_DIM * sizeof(__half);
    f.bytes = off;
    return f;
}

inline size_t fp16_partials_bytes(int G, int H, int max_seq_len) {
    int nchunk = (max_seq_len + FP16_CHUNK - 1) / FP16_CHUNK;
    return (size_t)G * H * nchunk * PART_STRIDE * sizeof(float);
}

// ---- shape checks -------------------------------------------------------------------------------------------------------
// What the entry points accept: any head layout the reference accepts (head_dim 128, num_heads a multiple of num_kv_heads).
inline int check_shape(int G, int H, int Hkv, int head_dim, int q_dim, int kv_dim, int bits, bool packed) {
    if (head_dim != HEAD_DIM) return TQ_ERR_UNSUPPORTED;
    if (G <= 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0) return TQ_ERR_ARG;
    if (kv_dim != Hkv * head_dim || q_dim < H * head_dim) return TQ_ERR_ARG;
    if (packed && bits != 2 && bits != 4) return TQ_ERR_ARG;
    return TQ_OK;
}

// What the streaming kernels serve; every other layout takes generic_decode_attention_kernel (one CTA per sequence
// and query head, every cache byte read once per query head, as the reference does).
inline bool fast_shape(int H, int Hkv, bool packed) {
    if (packed) return Hkv % 4 == 0 && Hkv <= 8 && H / Hkv <= 8 && H <= ATTN_MAX_HEADS;
    const int grp = H / Hkv;
    return grp == 1 || grp == 2 || grp == 4 || grp == 8;
}

inline int launch_generic_attention(const GenericAttnParams& p, bool fp16, cudaStream_t s) {
    if (p.G <= 0 || p.H <= 0 || p.G > 2147483647 / 1 || p.H > 65535) return TQ_ERR_ARG;
    dim3 grid((unsigned)p.G, (unsigned)p.H);
    if (fp16) generic_decode_attention_kernel<true><<<grid, GENERIC_WARPS * 32, 0, s>>>(p);
    else generic_decode_attention_kernel<false><<<grid, GENERIC_WARPS * 32, 0, s>>>(p);
    return cuda_status(cudaGetLastError());
}

// ---- launches -------------------------------------------------------------------------------------------------------------
// Launch with the programmatic-serialisation attribute: the kernel may start while the previous kernel of the
// stream is still running; the kernels themselves wait (griddepcontrol.wait) before touching dependent data.
template <typename Kernel, typename Params>
inline int launch_kernel(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl, const Params& p) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cuda_status(cudaLaunchKernelEx(&cfg, kernel, p));
}

constexpr size_t APPEND_SMEM = (size_t)HEAD_DIM * HEAD_DIM * sizeof(float);  // R as fp32

// Opt-in to large dynamic shared memory, once per (device, kernel); safe to call from several host threads.
inline int ensure_dynamic_smem(const void* func, size_t bytes, bool big_clusters = false) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, bool> done;
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    bool& d = done[std::make_pair(dev, func)];
    if (!d) {
        TQ_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        if (big_clusters) TQ_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        d = true;
    }
    return TQ_OK;
}

template <int NV>
inline int launch_append_t(const AppendParams& p, dim3 grid, cudaStream_t s, bool pdl) {
    int r = ensure_dynamic_smem((const void*)append_rotate_kernel<NV>, APPEND_SMEM);
    if (r != TQ_OK) return r;
    return launch_kernel(append_rotate_kernel<NV>, grid, dim3(APPEND_THREADS), APPEND_SMEM, s, pdl && p.rot_prep, p);  // (it reads a caller's R before the wait)
}

// Whole prompts (token form, K and/or V, no queries) go to the tensor-core kernel; TQ_PREFILL_TC=0 keeps them on
// the fp32-chain kernel.  Both store the same bytes.
// producer: the form that applies QK-norm and rotary embedding to the K vectors on the way in (PrefillTcParams)
// rows_made: set where the launch makes the rows and norms that t.k16 asks for as well (ROWS16)
inline int launch_prefill_tc_params(const PrefillTcParams& t, cudaStream_t s, bool pdl, bool producer = false, bool* rows_made = nullptr) {
    const long long tokens = (long long)t.n_seq * t.T;
    const long long tiles = ((tokens * t.Hkv + TC_TILE - 1) / TC_TILE) * ((t.k_buf ? 1 : 0) + (t.v_buf ? 1 : 0));
    long long grid = (long long)(producer ? 2 : TC_CTAS_PER_SM) * device_props().sm_count;
    if (grid > tiles) grid = tiles;
    if (grid < 1) return TQ_OK;
    // The vectors reach the operand tile by tensor-map copies where the layout allows it (TQ_PREFILL_TMA=0: through
    // registers, as in the producer form, whose K vectors are computed on the way in).
    static const bool tma_allowed = !(getenv("TQ_PREFILL_TMA") && atoi(getenv("TQ_PREFILL_TMA")) == 0);
    CUtensorMap tmk{}, tmv{};
    bool tma = !producer && tma_allowed;
    if (tma && t.k_buf) tma = make_append_input_map(&tmk, t.k_buf, tokens, t.Hkv, t.kv_dim) == TQ_OK;
    if (tma && t.v_buf) tma = make_append_input_map(&tmv, t.v_buf, tokens, t.Hkv, t.kv_dim) == TQ_OK;
    PrefillTcParams ts = t;
    const bool rows16 = tma && rows_made && t.k16;
    if (rows_made) *rows_made = rows16;
    if (rows16) grid = std::min<long long>(tiles, 2ll * device_props().sm_count);
    const size_t smem = rows16 ? (size_t)TC_ROWS_END : TC_DYN_SMEM;
    const void* kernel = producer ? (const void*)prefill_append_tc_kernel<true, false>
                         : rows16 ? (const void*)prefill_append_tc_kernel<false, true, true>
                                  : (tma ? (const void*)prefill_append_tc_kernel<false, true> : (const void*)prefill_append_tc_kernel<false, false>);
    int ar = ensure_dynamic_smem(kernel, smem);
    if (ar != TQ_OK) return ar;
#ifdef TQ_TIMING_SWITCHES
    static unsigned long long* d_stamps = nullptr;
    static int stamp_calls = 0;
    if (getenv("TQ_TC_STAMPS")) {
        if (!d_stamps) { cudaMalloc(&d_stamps, 256); cudaMemset(d_stamps, 0, 256); }
        ts.stamps = d_stamps;
    }
#endif
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaError_t le;
    if (producer) le = cudaLaunchKernelEx(&cfg, prefill_append_tc_kernel<true, false>, tmk, tmv, ts);
    else if (rows16) le = cudaLaunchKernelEx(&cfg, prefill_append_tc_kernel<false, true, true>, tmk, tmv, ts);
    else if (tma) le = cudaLaunchKernelEx(&cfg, prefill_append_tc_kernel<false, true>, tmk, tmv, ts);
    else le = cudaLaunchKernelEx(&cfg, prefill_append_tc_kernel<false, false>, tmk, tmv, ts);
    if (le != cudaSuccess) return (int)le;
#ifdef TQ_TIMING_SWITCHES
    if (ts.stamps && ++stamp_calls == 40) {
        unsigned long long h[32];
        cudaStreamSynchronize(s);
        cudaMemcpy(h, d_stamps, 256, cudaMemcpyDeviceToHost);
        for (int w = 0; w < 2; ++w) {
            const double n = (double)h[16 * w + 15] * (double)((tiles + grid - 1) / grid);
            fprintf(stderr, "append stamps, warp %d (cycles per tile): top %.0f | loads %.0f | tree %.0f | wait for the chain warp %.0f | operand + barrier B %.0f | "
                            "mma issue + per-vector %.0f | mma wait + barrier C %.0f | epilogue %.0f | barrier D %.0f | loop back %.0f\n",
                    w ? 7 : 0, h[16 * w] / n, h[16 * w + 1] / n, h[16 * w + 2] / n, h[16 * w + 3] / n, h[16 * w + 4] / n, h[16 * w + 5] / n,
                    h[16 * w + 6] / n, h[16 * w + 7] / n, h[16 * w + 8] / n, h[16 * w + 9] / n);
        }
    }
#endif
    return cuda_status(cudaGetLastError());
}

// Where a packed prompt's rows as fp16 and its norms go (PrefillTcParams), and whether the append made them.
struct PrefillRows {
    __half* k16;
    __half* v16;
    float* norms;
    int tiles;
    bool made;
    bool behind;  // the append was the tensor-core kernel: what comes next may read everything before it at once
};
inline int launch_prefill_tc(const AppendParams& p, cudaStream_t s, bool pdl, int n_seq = 1, long long seq_stride_rows = 0,
                             const long long* seq_row_base = nullptr, PrefillRows* rows = nullptr) {
    PrefillTcParams t{};
    t.ck = p.ck; t.kn = p.kn; t.cv = p.cv; t.vn = p.vn;
    t.k_buf = p.k_buf; t.v_buf = p.v_buf; t.rotation = p.rotation; t.positions = p.positions; t.pos_value = p.pos_value; t.status = p.status;
    t.token_row0 = p.token_row0; t.capacity_rows = p.capacity_rows;
    t.seq_stride_rows = seq_stride_rows; t.row_base = seq_row_base; t.n_seq = n_seq;
    t.T = p.n_src; t.Hkv = p.Hkv; t.kv_dim = p.kv_dim; t.bits = p.bits;
    t.static_rotation = p.rot_prep ? 1 : 0;  // (the engine's own R)
    if (rows) { t.k16 = rows->k16; t.v16 = rows->v16; t.norms = rows->norms; t.norm_tiles = rows->tiles; }
    if (rows) rows->behind = true;
    return launch_prefill_tc_params(t, s, pdl, false, rows ? &rows->made : nullptr);
}

inline bool prefill_tc_on() {
    static const bool on = !(getenv("TQ_PREFILL_TC") && atoi(getenv("TQ_PREFILL_TC")) == 0);
    return on;
}
inline int launch_append(const AppendParams& p, cudaStream_t s, bool pdl = false, PrefillRows* rows = nullptr) {
    const bool prefill_tc = prefill_tc_on();
    // (the tensor-core kernel moves 16 bytes at a time: every array it touches has to be 16-byte aligned)
    const uintptr_t align_or = (uintptr_t)p.k_buf | (uintptr_t)p.v_buf | (uintptr_t)p.ck | (uintptr_t)p.cv | (uintptr_t)p.rotation;
    if (prefill_tc && p.token_mode && !p.q && (p.k_buf || p.v_buf) && (align_or & 15u) == 0 &&
        p.kv_dim == p.Hkv * HEAD_DIM && (long long)p.n_src * p.Hkv >= 4 * TC_TILE && (long long)p.n_src * p.Hkv < (1ll << 31))
        return launch_prefill_tc(p, s, pdl, 1, 0, nullptr, rows);
    const int nk = p.k_buf ? p.Hkv : 0, nv = p.v_buf ? p.Hkv : 0, nq = p.q ? p.H : 0;
    const long long total = (long long)p.n_src * (nk + nv + nq);
    const bool tables = p.tile_start != nullptr && !p.token_mode;
    if (total <= 0 && !tables) return TQ_OK;
    if (total >= (1ll << 31)) return TQ_ERR_CAPACITY;
    // A few vectors and nothing else to do: one CTA each (16-byte loads of R's rows, 4-byte stores of code words).
    if (!p.q && !tables && total <= (long long)APPEND_VECTOR_MAX_PER_SM * device_props().sm_count && (((uintptr_t)p.rotation & 15u) == 0) &&
        ((((uintptr_t)p.ck | (uintptr_t)p.cv) & 3u) == 0))
        return p.bits == 4 ? launch_kernel(append_vector_kernel<4>, dim3((unsigned)total), dim3(HEAD_DIM), 0, s, pdl, p)
                           : launch_kernel(append_vector_kernel<2>, dim3((unsigned)total), dim3(HEAD_DIM), 0, s, pdl, p);
    // One CTA per SM at most.  As few vectors per group as still fit the whole launch into that one wave: short
    // dependent chains when the batch is small, amortised staging of R when it is large (then the CTAs loop).
    const long long slots = (long long)device_props().sm_count - 1;
    int nvec = 1;
    while (nvec < APPEND_MAX_NV && (total + nvec * APPEND_GROUPS - 1) / (nvec * APPEND_GROUPS) > slots) nvec *= 2;
    long long blocks = (total + nvec * APPEND_GROUPS - 1) / (nvec * APPEND_GROUPS);
    if (blocks > slots) blocks = slots;
    if (blocks < 1) blocks = 1;
    const dim3 grid((unsigned)(blocks + (tables ? 1 : 0)));
    if (nvec == 1) return launch_append_t<1>(p, grid, s, pdl);
    if (nvec == 2) return launch_append_t<2>(p, grid, s, pdl);
    return launch_append_t<4>(p, grid, s, pdl);
}

// Number of attention CTAs: one per SM (each holds ATTN_GROUPS workers), fewer when the cache cannot hold that
// many tiles.
inline int attention_ctas(int G, int max_seq_len) {
    long long tiles = (long long)G * ((max_seq_len + TILE_TOKENS - 1) / TILE_TOKENS);
    long long w = device_props().sm_count;
    if (w * ATTN_GROUPS > MAX_WORKERS) w = MAX_WORKERS / ATTN_GROUPS;
    long long need = (tiles + ATTN_GROUPS - 1) / ATTN_GROUPS;
    if (need < w) w = need;
    return (int)(w < 1 ? 1 : w);
}

template <int BITS, int HKV, int MODE>
inline int launch_attention_t(const CUtensorMap& tmK, const CUtensorMap& tmV, const AttnParams& p, int ctas, cudaStream_t s,
                              bool pdl) {
    int ar = ensure_dynamic_smem((const void*)decode_attention_kernel<BITS, HKV, MODE>, ATTN_DYN_SMEM);
    if (ar != TQ_OK) return ar;
    if constexpr ((MODE == 1 || MODE == 2) && HKV == 8) {
        // the register split inside the kernel draws on what the launch brings: never launch with less
        static const int regs = [] {
            cudaFuncAttributes f{};
            return cudaFuncGetAttributes(&f, (const void*)decode_attention_kernel<BITS, HKV, MODE>) == cudaSuccess ? f.numRegs : 0;
        }();
        if (regs * attn_threads<HKV, MODE>() < 32 * (ATTN_GROUPS * HKV * ATTN_REGS_WORK + 4 * ATTN_REGS_COPY)) return TQ_ERR_UNSUPPORTED;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(attn_threads<HKV, MODE>());
    cfg.dynamicSmemBytes = ATTN_DYN_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cuda_status(cudaLaunchKernelEx(&cfg, decode_attention_kernel<BITS, HKV, MODE>, tmK, tmV, p));
}

// mode 0: after append_rotate_kernel (rotated queries and tile table in the workspace, merge in the kernel); 1: one layer, after
// layer_prep_kernel, the merge left to merge_layer_kernel; 2: whole-step form over AttnParams::n_layers layers; 4: as 2 without the
// copy warps (8 KV heads only).
inline int launch_attention(int bits, const CUtensorMap& tmK, const CUtensorMap& tmV, const AttnParams& p, int ctas,
                            cudaStream_t s, bool pdl = false, int mode = 0) {
    if (p.Hkv != 8 && p.Hkv != 4) return TQ_ERR_UNSUPPORTED;
#define TQ_ATTN_DISPATCH(MODE)                                                                                  \
    if (p.Hkv == 8)                                                                                             \
        return bits == 4 ? launch_attention_t<4, 8, MODE>(tmK, tmV, p, ctas, s, pdl)                            \
                         : launch_attention_t<2, 8, MODE>(tmK, tmV, p, ctas, s, pdl);                           \
    return bits == 4 ? launch_attention_t<4, 4, MODE>(tmK, tmV, p, ctas, s, pdl)                                \
                     : launch_attention_t<2, 4, MODE>(tmK, tmV, p, ctas, s, pdl);
    if (mode == 4) return bits == 4 ? launch_attention_t<4, 8, 4>(tmK, tmV, p, ctas, s, pdl) : launch_attention_t<2, 8, 4>(tmK, tmV, p, ctas, s, pdl);
    if (mode == 2) { TQ_ATTN_DISPATCH(2) }
    if (mode == 1) { TQ_ATTN_DISPATCH(1) }
    TQ_ATTN_DISPATCH(0)
#undef TQ_ATTN_DISPATCH
}

// Two CTAs per SM at most: each fetches R once and loops.  Where R is transposed too, 64 at least, an element per thread: by the CTAs of a few
// sequences alone that took longer than all the rest (one sequence of 30000 tokens, 2-bit, 4/4 heads, one CTA: 24.6 -> 16.0 us).
inline int launch_layer_prep(int bits, const LayerPrepParams& p, cudaStream_t s, bool pdl) {
    const long long vectors = (p.new_k ? p.G : 0) + ((long long)p.G * p.H + 15) / 16, items = p.rotation_t ? std::max(vectors, 64ll) : vectors;
    const dim3 grid((unsigned)std::min(items, 2ll * device_props().sm_count));
    return bits == 4 ? launch_kernel(layer_prep_kernel<4>, grid, dim3(PREP_THREADS), 0, s, pdl, p)
                     : launch_kernel(layer_prep_kernel<2>, grid, dim3(PREP_THREADS), 0, s, pdl, p);
}

// One cluster per (sequence, KV head, block of 8 query heads): tq_decode_cluster.cuh.  `max_tokens`: rows a sequence may hold.
constexpr size_t CD_ONE_PER_SM = 118 * 1024;  // more than half of an SM's shared memory
template <int BITS, int MB, bool HOST, bool EXACT>
inline int launch_cluster_decode_t(const ClusterDecodeParams& p, int S, int layers, cudaStream_t s, bool pdl) {
    const void* kernel = (const void*)cluster_decode_kernel<BITS, MB, HOST, EXACT>;
    int r = ensure_dynamic_smem(kernel, std::max(cd_smem_bytes(BITS, CD_HEADS, EXACT), CD_ONE_PER_SM), true);
    if (r != TQ_OK) return r;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)S, (unsigned)(p.Hkv * p.head_blocks), (unsigned)(p.G * layers));
    cfg.blockDim = dim3(CD_THREADS);
    cfg.dynamicSmemBytes = cd_smem_bytes(BITS, std::min(CD_HEADS, p.H / p.Hkv), EXACT);
    // One CTA per SM where they fit and none starts under a launch of its own kind (its room would be needed then): small clusters come
    // two to an SM otherwise, with SMs idle (launchers, 2-bit 32/8 heads 8 x 1023 tokens 18.5 us a layer, one per SM 17.5; 4-bit 16/8
    // 8 x 1500 22.4 / 20.5).  Clusters of 4 and more find no room that way (4-bit 4 x 600 13.5 / 14.2, 1 x 3000 15.1 / 19.4).
    if (S <= 2 && !p.early && !p.static_rotation && (long long)S * cfg.gridDim.y * cfg.gridDim.z <= device_props().sm_count)
        cfg.dynamicSmemBytes = std::max(cfg.dynamicSmemBytes, CD_ONE_PER_SM);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, cluster_decode_kernel<BITS, MB, HOST, EXACT>, p));
}
// CTAs per cluster.  As many as give every warp a 16-token block of its own, up to one CTA per SM over the whole launch: two share
// the SM's L1 and issue slots, and the CTAs of the next launch find no room for their prologue (8 sequences x 1023 tokens through
// the launchers 24 us a layer with two, 19 with one).  16 only where 8 leave a warp two blocks and more: seven of the GPU's
// processing clusters hold one cluster of 16 beside the previous launch's, an eighth waits (1 sequence, 8 KV heads, 4-bit: 600 tokens 5.2 us
// with 8 and 7.9 with 16, 1500 tokens 5.5 / 6.2, 3000 tokens 7.4 / 6.8; fp16 1500 5.3 / 5.6, 3000 11.0 / 7.9; layers
// that stay in L2.  1 and 2 sequences of 1100 to 2019 tokens, all modes and layouts, 1.0 to 1.25 times as fast as with 16, EXACT up to 2.)  Clusters of 4 and more leave some of a processing cluster's SMs over (136
// of 148 serve fours, 128 eights): one cluster more than fits waits for a whole turn (72 clusters of 4 at two CTAs per SM 1.5
// times the time of 72 of 2).  Where a warp goes through many tiles, more than the launch's fixed part costs, a second CTA per SM
// hides the latency of the first one's loads: above 12 tiles 0.6 to 0.95 of the time (4 x 8192 tokens, 8 KV heads, 44 -> 28 us),
// above 4 for fp16, whose rows are four times as long.  Not with more than 4 query heads per cluster in a packed mode: the warps'
// partial results leave room for one CTA per SM there.
// Where those are one layer's (`layer`), 4-bit, and as many as fit, the next layer's clusters of 8 and 16 find no room beside this one's: they are
// halved (32/4 heads 2 x 4000 tokens 17.1 -> 10.1 us, 2 x 8000 20.9 -> 13.8, 4 x 4000 19.9 -> 14.5; 40/8 1 x 2048 13.8 -> 8.3, 1 x 12000 25.6 -> 20.4,
// 1 x 32000 52.1 -> 49.0, 2 x 520 11.5 -> 5.9, 2 x 6000 25.2 -> 22.1).  Layouts without a streaming form (`streams` false) keep clusters of 8 where 4
// would have chains of more than 20 tiles (40/8 2 x 10000 37.5 -> 37.0, 2 x 12000 43.1 -> 44.0, 2 x 16000 53.0 -> 56.5).  With a cluster's room and more to
// spare only short slots are, where the shorter exchange pays (full / halved: 32/4 3 x 700 7.2 / 6.2, 3 x 1300 7.7 / 7.7, 3 x 4000 10.8 / 14.4, 3 x 8000 14.4 /
// 23.0; 8 heads over 5, 6 and 7 KV heads, 80 to 120 CTAs: 700 tokens 1.05 to 1.18 of the time, 1300 0.87 to 0.99, 4000 0.67 to 0.73; 16 CTAs from 2100 on 0.98 to 1.1).
inline int cluster_split(int bits, long long clusters, int heads, int max_tokens, bool layer, bool streams) {
    const long long sms = device_props().sm_count, blocks = (max_tokens + 15) / 16;
    auto half = [&](int n) {
        if (n < 8 || !layer || bits != 4 || heads <= 4) return false;
        return clusters * n > sms - 28 ? streams || n > 8 || blocks <= 20 * 4 * CD_WARPS : blocks <= n * CD_WARPS;
    };
    auto fit = [&](int n) { return half(n) ? (sms - 20) / 2 : sms - (n >= 8 ? 20 : n >= 4 ? 12 : 0); };
    int S = 1;
    auto longer = [&](int n) { return n == 8 ? 2 * n * CD_WARPS <= blocks : n * CD_WARPS < blocks; };
    while (S < CD_MAX_CLUSTER && longer(S) && clusters * S * 2 <= fit(2 * S)) S *= 2;
    if (S <= 4 && clusters * S * 8 <= 7 * sms && clusters * S * 2 <= 2 * fit(2 * S) && blocks > (bits ? 12 : 4) * CD_WARPS * S &&
        (heads <= 4 || bits == 0))
        S *= 2;
    return S;
}
// Is one layer faster in the cluster form than in the streaming one?  Both times, in us, are lines in what bounds them, measured
// over 1 to 128 sequences of 64 to 16384 tokens, equal and ragged, and 8 KV heads of 2 and 4 query heads, 4 of 8.  Packed: the
// cluster form 4.6 + 0.4 per tile of its longest warp + 0.3 more per turn of the SMs + 0.023 per 1000 rows and KV heads + 0.007 to
// 0.009 per cluster, the streaming form 14.6 + 0.030 per 1000 rows and KV heads + 0.4 per 1000 tokens of the longest sequence.  Long
// chains of tiles cost the cluster form more than those lines say, and with 8 heads in 4-bit, one CTA per SM, more turns: 12 tiles at
// most, with many rows a few more (cluster / streaming: 4-bit 32/8 heads 8 x 8000 39.4 / 29.7 us, 2-bit 32/4 8 x 8000 29.3 / 21.4, 4-bit
// 32/4 48 x 1023 26.0 / 21.5, 2 x 16000 23.3 / 21.5, 96 x 600 31.8 / 26.7, 24 x 1500 17.2 / 17.6).  fp16: a tile costs the cluster form 1 us more than the streaming form's
// share of it where there is one turn, less with more turns and with 8 query heads,
// and that form starts 7 us later.  Above 640 clusters their number counts for more than in the lines fitted below it (128 x 64
// tokens, 16/8 heads, 4-bit 25.7 / 19.7 us, 96 x 64 19.8 / 19.0, 64 x 64 13.5 / 17.2; 32/8 heads 128 x 64 26.8 / 24.9, 96 x 64 20 / 23;
// fp16 128 x 300 43.0 / 39.1, 96 x 300 32.6 / 33.2).
// fp16 slots of one chunk of the streaming form, which has nothing to merge there and in an engine starts under the write of the new rows, go
// to it where the cluster form has one CTA per sequence and KV head and its warps enough tiles (cluster / streaming, slots of 288, 352, 416 and
// 512 rows: 16/8 heads 96 clusters 5.9 / 6.7, 7.1 / 7.2, 8.9 / 7.9, 11.7 / 9.3 us, 160 7.5 / 8.0, 10.5 / 10.0, 13.0 / 10.9, 14.4 / 11.8, 384 18.2 / 16.6,
// 22.3 / 18.5, 26.5 / 20.3, 29.7 / 23.0; 8/8 96 5.6 / 7.3, 6.9 / 7.9, 8.5 / 8.6, 11.3 / 10.0, 512 18.3 / 19.2, 22.4 / 21.1), unless those just
// fill two CTAs per SM (16/8 296 10.1 / 11.9, 12.1 / 13.0, 14.3 / 14.7, 16.1 / 17.0).
// Launchers: their streaming fp16 form has its clears and writes in launches of their own (3 us); packed, the layer form has the same
// three launches, and the cluster form, which cannot start under the appends, is 3 us ahead in 2-bit only (2-bit 32/4 heads 128 x 600
// tokens 38.9 us a layer with the appends, streaming 40.9; 4-bit 32/4 48 x 2500 58.9 / 36.3, 16/8 64 x 1500 64.7 / 44.4).
enum class LayerCaller { Engine, Launchers };
inline bool cluster_layer_faster(int bits, int G, int Hkv, int heads, long long rows, int max_tokens, LayerCaller caller) {
    const long long clusters = (long long)G * Hkv, sms = device_props().sm_count;
    const int S = cluster_split(bits, clusters, heads, max_tokens, true, true);
    const double chain = ((max_tokens + 15) / 16) / (double)(S * CD_WARPS), turns = (double)((clusters * S + sms - 1) / sms);
    const double extra = caller == LayerCaller::Launchers && bits != 4 ? 3.0 : 0.0;  // us the streaming form's launches cost on top
    if (bits == 0 && caller == LayerCaller::Engine && S == 1 && heads <= 4 && max_tokens <= FP16_CHUNK && (2 * clusters <= 3 * sms || clusters > 2 * sms) &&
        chain > (clusters > 2 * sms ? 2.2 : 4 * clusters > 3 * sms ? 2.5 : 2.8))
        return false;
    if (bits == 0) return (heads > 4 ? 0.5 : 1.0) * chain < 7.0 + 1.5 * turns + extra && !(clusters > 768 && chain > 2.0);
    const double many = heads > 2 ? 0.0015 * std::max(0ll, clusters - 800) : 0.02 * std::max(0ll, clusters - 640);
    if (bits == 4 && heads > 4 ? chain * turns > 12.0 : chain > 12.0 + 5e-6 * (double)rows * Hkv) return false;
    return 0.4 * chain + 0.3 * chain * turns + 0.009 * clusters + many < 10.0 + 7e-6 * (double)rows * Hkv + 0.0004 * max_tokens + extra;
}
// split_layers: the number of layers the cut of the work is made for (a step's layers give the same bits in one launch or several)
inline int cluster_launch_split(int bits, int G, int split_layers, int H, int Hkv, int max_tokens) {
    const int head_blocks = (H / Hkv + CD_HEADS - 1) / CD_HEADS;
    const bool streams = fast_shape(H, Hkv, bits != 0), one_per_sm = bits != 0 && !streams;  // (EXACT, packed: as with 8 heads)
    return cluster_split(bits, (long long)G * split_layers * Hkv * head_blocks, one_per_sm ? CD_HEADS : std::min(CD_HEADS, H / Hkv), max_tokens, split_layers == 1, streams);
}
template <bool HOST, bool EXACT>
inline int launch_cluster_decode_e(int bits, const ClusterDecodeParams& p, int layers, int split_layers, int max_tokens, cudaStream_t s, bool pdl) {
    const int blocks = (max_tokens + 15) / 16;
    const int S = cluster_launch_split(bits, p.G, split_layers, p.H, p.Hkv, max_tokens);
    if (bits == 0) return launch_cluster_decode_t<0, 1, HOST, EXACT>(p, S, layers, s, pdl);
    // 16-token tiles where every warp of the cluster has one at most.  (From four CTAs on the new token's takes none, so that the last
    // S-th of a full slot is a second tile for some warps.  Two blocks per tile there: 8 layers of 1 x 980 tokens in 1024 rows, 4-bit 16/8
    // heads, 46.3 -> 42.5 us, but of 4 x 300 in 512 rows 44.3 -> 46.3: the contexts that fit are seven eighths or three quarters.)
    const bool one = S * CD_WARPS >= blocks;
    if (bits == 4) return one ? launch_cluster_decode_t<4, 1, HOST, EXACT>(p, S, layers, s, pdl) : launch_cluster_decode_t<4, 2, HOST, EXACT>(p, S, layers, s, pdl);
    return one ? launch_cluster_decode_t<2, 1, HOST, EXACT>(p, S, layers, s, pdl) : launch_cluster_decode_t<2, 2, HOST, EXACT>(p, S, layers, s, pdl);
}
template <bool HOST = false>
inline int launch_cluster_decode(int bits, const ClusterDecodeParams& p, int layers, int split_layers, int max_tokens, cudaStream_t s, bool pdl) {
    return fast_shape(p.H, p.Hkv, bits != 0) ? launch_cluster_decode_e<HOST, false>(bits, p, layers, split_layers, max_tokens, s, pdl)
                                             : launch_cluster_decode_e<HOST, true>(bits, p, layers, split_layers, max_tokens, s, pdl);
}

// Merge of a layer's partials.  Few sequences are cut into many parts each, and a warp that adds up a head's alone, 16 in flight, was up to
// half of the layer: from 14 workers per sequence on, a CTA per head, while these are not many more than the SMs (eight heads per CTA / one, 4-bit
// 16/8 heads 3 x 30000 tokens 51.3 / 34.4 us a layer, 5 x 16384 40.7 / 31.7, 10 x 8192 35.0 / 31.3, 2-bit 32/8 8 x 8000 29.0 / 26.0; 288 heads: 9 x 8000 28.3 /
// 28.7, 4-bit 16/8 18 x 6000 37.2 / 38.0; nine parts: 8/8 36 x 2000 27.7 / 30.3).
inline int launch_merge_layer(const MergeLayerParams& p, cudaStream_t s, bool pdl) {
    const long long sms = device_props().sm_count, each = (long long)p.G * p.H;
    const dim3 threads(MERGE_WARPS * 32);
    if (p.workers >= 14 * p.G && 4 * each <= 7 * sms) {
        const dim3 grid((unsigned)p.G, (unsigned)p.H);
        return each <= sms ? launch_kernel(merge_layer_kernel<1, 1>, grid, threads, 0, s, pdl, p) : launch_kernel(merge_layer_kernel<1, 2>, grid, threads, 0, s, pdl, p);
    }
    const dim3 grid((unsigned)p.G, (unsigned)((p.H + MERGE_WARPS - 1) / MERGE_WARPS));
    return (long long)grid.x * grid.y <= sms ? launch_kernel(merge_layer_kernel<MERGE_WARPS, 1>, grid, threads, 0, s, pdl, p)
                                             : launch_kernel(merge_layer_kernel<MERGE_WARPS, 2>, grid, threads, 0, s, pdl, p);
}

__global__ void transpose_rotation_kernel(__half* dst, const __half* src) {
    // dst[d][k] = src[k][d]; one block per 32x32 tile would be overkill for 32 KB: a plain strided copy
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < HEAD_DIM * HEAD_DIM; i += gridDim.x * blockDim.x) {
        const int d = i >> 7, k = i & 127;
        dst[i] = src[k * HEAD_DIM + d];
    }
}

// Tensor-core form of the twin (tq_fp16_tc.cuh): every query head of a KV head from one pass, whatever their number.
template <int GRP>
inline int launch_fp16_tc_t(const CUtensorMap& tmK, const CUtensorMap& tmV, const Fp16AttnParams& p, cudaStream_t s, bool pdl) {
    int ar = ensure_dynamic_smem((const void*)fp16_tc_decode_attention_kernel<GRP>, FP16TC_SMEM);
    if (ar != TQ_OK) return ar;
    dim3 grid(p.Hkv, p.nchunk_max, p.G);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(FP16TC_WARPS * 32);
    cfg.dynamicSmemBytes = FP16TC_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cuda_status(cudaLaunchKernelEx(&cfg, fp16_tc_decode_attention_kernel<GRP>, tmK, tmV, p));
}
inline int launch_fp16_tc_attention(const CUtensorMap& tmK, const CUtensorMap& tmV, const Fp16AttnParams& p, cudaStream_t s, bool pdl) {
    switch (p.H / p.Hkv) {
        case 1: return launch_fp16_tc_t<1>(tmK, tmV, p, s, pdl);
        case 2: return launch_fp16_tc_t<2>(tmK, tmV, p, s, pdl);
        case 4: return launch_fp16_tc_t<4>(tmK, tmV, p, s, pdl);
        case 8: return launch_fp16_tc_t<8>(tmK, tmV, p, s, pdl);
        default: return TQ_ERR_UNSUPPORTED;
    }
}

// What the causal prefill attention (tq_prefill_fa.cuh) serves: a slot holds at least one token's query heads.
inline bool prefill_attn_shape(int H, int Hkv) { return Hkv > 0 && H % Hkv == 0 && H / Hkv <= PFT_ROWS; }
// fp16 K or V array [rows][kv_dim] viewed as bytes for prefill_attention_fa_kernel: box = one head's 256 bytes (two 128-byte
// blocks) x 128 rows, 128-byte swizzle.
inline int make_prefill_rows_map(CUtensorMap* m, const void* base, long long rows, int kv_dim) {
    auto fn = encode_fn();
    if (!fn) return TQ_ERR_UNSUPPORTED;
    const long long row_bytes = (long long)kv_dim * 2;
    if (((uintptr_t)base & 15u) != 0 || rows <= 0 || rows >= (1ll << 31)) return TQ_ERR_ARG;
    cuuint64_t dims[3] = {128u, (cuuint64_t)rows, (cuuint64_t)(row_bytes / 128)};
    cuuint64_t strides[2] = {(cuuint64_t)row_bytes, 128u};
    cuuint32_t box[3] = {128u, (cuuint32_t)PFT_KT, 2u};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TQ_OK : TQ_ERR_ARG;
}
// Queries [tokens][q_stride] halves: box = one half (128 bytes) of the coordinates of `grp` heads of `qt` tokens, landing as
// [token][head][128 B] with the 128-byte swizzle = the rows of a query operand tile.
inline int make_prefill_query_map(CUtensorMap* m, const void* base, long long tokens, int H, int grp, int qt, long long q_stride) {
    auto fn = encode_fn();
    if (!fn) return TQ_ERR_UNSUPPORTED;
    if (((uintptr_t)base & 15u) != 0 || q_stride % 8 != 0 || tokens <= 0 || tokens >= (1ll << 31)) return TQ_ERR_ARG;
    cuuint64_t dims[4] = {128u, (cuuint64_t)H, (cuuint64_t)tokens, 2u};
    cuuint64_t strides[3] = {256u, (cuuint64_t)q_stride * 2u, 128u};
    cuuint32_t box[4] = {128u, (cuuint32_t)grp, (cuuint32_t)qt, 1u};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? TQ_OK : TQ_ERR_ARG;
}
template <bool PACKED, int MT, bool EXACT = false, int DIRECT = 0, bool EARLY = false>
inline int launch_prefill_fa_t(const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmQ, const CUtensorMap& tmR, const PrefillAttnParams& p,
                               dim3 grid, cudaStream_t s) {
    int r = ensure_dynamic_smem((const void*)prefill_attention_fa_kernel<PACKED, MT, EXACT, DIRECT, EARLY>, PftSmem::BYTES);
    if (r != TQ_OK) return r;
    // the register split inside the kernel draws on what the launch brings: never launch with less
    static const int regs = [] {
        cudaFuncAttributes a{};
        return cudaFuncGetAttributes(&a, (const void*)prefill_attention_fa_kernel<PACKED, MT, EXACT, DIRECT, EARLY>) == cudaSuccess ? a.numRegs : 0;
    }();
    if (regs < PFT_REGS_LAUNCH) return TQ_ERR_UNSUPPORTED;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(PFT_THREADS);
    cfg.dynamicSmemBytes = PftSmem::BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, prefill_attention_fa_kernel<PACKED, MT, EXACT, DIRECT, EARLY>, tmK, tmV, tmQ, tmR, p));
}
// Which layouts keep fp32's precision (tq_prefill_fa.cuh): those that neither this kernel's predecessor nor the streaming kernels took.
inline bool prefill_exact(int bits, int H, int Hkv) {
    const int grp = H / Hkv;
    return !(grp == 1 || grp == 2 || grp == 4 || grp == 8 || grp == 16) && !fast_shape(H, Hkv, bits != 0);
}
// Bytes of scratch a packed prompt of T tokens needs: fp16 centroids of K and V (exact: high and low parts), fp32 norms.
inline int prefill_tiles(int T) { return (T + PFT_KT - 1) / PFT_KT; }
inline size_t prefill_scratch_bytes(int T, int Hkv, bool exact) {
    return 2 * align_up((size_t)(exact ? 2 : 1) * T * Hkv * HEAD_DIM * sizeof(__half), 256) + align_up((size_t)Hkv * prefill_tiles(T) * PFT_NORM_BYTES, 256);
}
// Causal prefill attention.  `total_rows`: rows of the arrays ck and cv point into (from where they point); `scratch`: packed
// modes, device memory for at least one KV head of one prompt (prompts go through it in groups; one that is too long for it as a
// whole, some of its KV heads at a time).  Prompts of one tile need none: their blocks convert the codes themselves.
// rows_made: the append has left the rows and norms of all prompts in the scratch (prefill_rows_in).
struct PrefillScratch {
    __half* k16;
    __half* v16;
    float* norms;
    long long rows;  // of each array, low parts included
};
inline PrefillScratch prefill_rows_in(void* scratch, int n_seq, int T, int Hkv, bool low) {
    PrefillScratch c{};
    c.rows = (long long)n_seq * T * (low ? 2 : 1);
    const size_t bytes = align_up((size_t)c.rows * Hkv * HEAD_DIM * sizeof(__half), 256);
    c.k16 = (__half*)scratch; c.v16 = (__half*)((char*)scratch + bytes); c.norms = (float*)((char*)scratch + 2 * bytes);
    return c;
}
inline int launch_prefill_attention(int bits, PrefillAttnParams p, long long total_rows, void* scratch, size_t scratch_bytes, cudaStream_t s, bool rows_made = false) {
    p.grp = p.H / p.Hkv;
    const bool exact = prefill_exact(bits, p.H, p.Hkv), low = exact && bits != 0;
    if (p.n_seq <= 0) p.n_seq = 1;
    if (p.T <= 0) return TQ_OK;
    const int qt = PFT_ROWS / p.grp;
    int group = p.n_seq, heads = p.Hkv;  // prompts and KV heads per launch (fp16 caches: all of them)
    const bool direct = bits != 0 && !exact && p.T <= PFT_KT;  // prompts of one tile: no rows in between
    if (bits != 0 && !direct) {
        if (!scratch) return TQ_ERR_WORKSPACE;
        while (heads > 0 && prefill_scratch_bytes(p.T, heads, exact) > scratch_bytes) --heads;
        if (heads == 0) return TQ_ERR_WORKSPACE;
        const int passes = (p.Hkv + heads - 1) / heads;
        heads = (p.Hkv + passes - 1) / passes;  // of about the same size
        group = (int)std::min<long long>(p.n_seq, (long long)(scratch_bytes / prefill_scratch_bytes(p.T, heads, exact)));
    }
    for (int s0 = 0; s0 < p.n_seq; s0 += group) {
        for (int h0 = 0; h0 < p.Hkv; h0 += heads) {
            PrefillAttnParams a = p;
            a.n_seq = std::min(group, p.n_seq - s0);
            a.Hkv = std::min(heads, p.Hkv - h0);
            a.H = a.Hkv * p.grp;
            const size_t col = (size_t)h0 * p.grp * HEAD_DIM;
            const int kv_dim = a.Hkv * HEAD_DIM;
            a.q = p.q + (size_t)s0 * p.T * p.q_tok_stride + col;
            a.out = p.out + (size_t)s0 * p.T * p.q_dim + col;
            CUtensorMap tmK{}, tmV{}, tmQ{}, tmR{};
            int r = make_prefill_query_map(&tmQ, a.q, (long long)a.n_seq * p.T, a.H, p.grp, qt, p.q_tok_stride);
            if (r != TQ_OK) return r;
            if (bits == 0) {
                r = make_prefill_rows_map(&tmK, p.ck, total_rows, kv_dim);
                if (r == TQ_OK) r = make_prefill_rows_map(&tmV, p.cv, total_rows, kv_dim);
            } else if (direct) {
                r = make_prefill_rows_map(&tmR, p.rotation, HEAD_DIM, HEAD_DIM);
            } else {
                DequantParams d{};
                const size_t rows = p.row_base ? 0 : (size_t)s0 * p.seq_rows, head_bytes = bits == 4 ? 64 : 32;
                d.ck = p.ck + (rows * p.Hkv + h0) * head_bytes; d.cv = p.cv + (rows * p.Hkv + h0) * head_bytes;
                d.kn = p.kn + rows * p.Hkv + h0; d.vn = p.vn + rows * p.Hkv + h0;
                d.row_base = p.row_base ? p.row_base + s0 : nullptr;
                d.seq_rows = p.seq_rows; d.T = p.T; d.tiles = prefill_tiles(p.T); d.Hkv = a.Hkv; d.row_heads = p.Hkv;
                const long long rows_hi = (long long)a.n_seq * p.T;  // the low parts behind the high ones
                const PrefillScratch c = prefill_rows_in(scratch, a.n_seq, p.T, a.Hkv, low);
                const long long rows_all = c.rows;
                d.low = rows_hi * kv_dim;
                d.k16 = c.k16; d.v16 = c.v16; d.norms = c.norms;
                const long long pieces = 2ll * p.T * a.Hkv * 16;
                d.code_blocks = (int)std::min<long long>((pieces + 1023) / 1024, 8ll * device_props().sm_count);
                const int norm_blocks = (int)std::min<long long>(((long long)a.Hkv * d.tiles + 7) / 8, device_props().sm_count);
                const dim3 grid((unsigned)(d.code_blocks + norm_blocks), (unsigned)a.n_seq);
                if (rows_made) r = TQ_OK;
                else if (low) r = bits == 4 ? launch_kernel(dequantize_rows_kernel<4, true>, grid, dim3(256), 0, s, true, d)
                                       : launch_kernel(dequantize_rows_kernel<2, true>, grid, dim3(256), 0, s, true, d);
                else r = bits == 4 ? launch_kernel(dequantize_rows_kernel<4, false>, grid, dim3(256), 0, s, true, d)
                                   : launch_kernel(dequantize_rows_kernel<2, false>, grid, dim3(256), 0, s, true, d);
                a.ck = (const uint8_t*)d.k16; a.cv = (const uint8_t*)d.v16; a.norms = d.norms; a.tiles = d.tiles;
                a.row_base = nullptr;
                a.seq_rows = p.T;
                a.low_row = (int)rows_hi;
                if (r == TQ_OK) r = make_prefill_rows_map(&tmR, p.rotation, HEAD_DIM, HEAD_DIM);
                if (r == TQ_OK) r = make_prefill_rows_map(&tmK, d.k16, rows_all, kv_dim);
                if (r == TQ_OK) r = make_prefill_rows_map(&tmV, d.v16, rows_all, kv_dim);
            }
            if (r != TQ_OK) return r;
            // Two query blocks per CTA, which share every tile, once there are enough of them for the GPU; below that twice the
            // CTAs with one block each, whose two slots take the even and the odd tiles.  Per layer, one block / two (8 KV heads,
            // 4-bit): 2048 tokens 16 heads (128 pairs of blocks) 55 / 67 us, 3000 tokens (188) 88 / 85, 32 heads 2048 tokens (256)
            // 91 / 76, 8192 tokens 16 heads (512) 381 / 352; fp16 2048 tokens 16 heads 31 / 43, 32 heads 57 / 48.
            const long long blocks2 = (p.T + 2 * qt - 1) / (2 * qt), cols = (long long)a.Hkv * a.n_seq;
            // Prompts of up to two tiles have no long CTAs, there the turns of the SMs decide, of which one with two blocks costs about
            // 4/3 of one with one: 12 prompts of 70 tokens 29.4 / 23.8 us, of 163 39.5 / 44.4, 16 of 250 62.6 / 51.6.
            const long long sms = device_props().sm_count, blocks1 = (p.T + qt - 1) / qt;
            const long long turns1 = (blocks1 * cols + sms - 1) / sms, turns2 = (blocks2 * cols + sms - 1) / sms;
            const int mt = low ? 1 : (p.T <= 2 * PFT_KT ? 3 * turns1 >= 4 * turns2 : 4 * blocks2 * cols >= 5 * sms) ? 2 : 1;
            const long long blocks = mt == 2 ? blocks2 : blocks1;
            if (cols > 2147483647ll || blocks > 65535) return TQ_ERR_CAPACITY;
            dim3 grid((unsigned)cols, (unsigned)blocks);
            // Where the blocks convert the codes themselves, that comes behind the rotation in the early form: taken where append and attention
            // fit the GPU side by side (28 layers, 2-bit, 120 tokens 435 -> 407 us, 64 4-bit 400 -> 390, but 8 of 16 x 100 188 -> 191).
            const bool early = direct && a.early && mt == 1 && cols * blocks + 2ll * a.n_seq * p.T * a.Hkv / TC_TILE <= sms;
            if (early) r = bits == 4 ? launch_prefill_fa_t<true, 1, false, 4, true>(tmK, tmV, tmQ, tmR, a, grid, s) : launch_prefill_fa_t<true, 1, false, 2, true>(tmK, tmV, tmQ, tmR, a, grid, s);
            else if (direct) r = bits == 4 ? (mt == 2 ? launch_prefill_fa_t<true, 2, false, 4>(tmK, tmV, tmQ, tmR, a, grid, s) : launch_prefill_fa_t<true, 1, false, 4>(tmK, tmV, tmQ, tmR, a, grid, s))
                                      : (mt == 2 ? launch_prefill_fa_t<true, 2, false, 2>(tmK, tmV, tmQ, tmR, a, grid, s) : launch_prefill_fa_t<true, 1, false, 2>(tmK, tmV, tmQ, tmR, a, grid, s));
            else if (low) r = launch_prefill_fa_t<true, 1, true>(tmK, tmV, tmQ, tmR, a, grid, s);
            else if (bits != 0) r = mt == 2 ? launch_prefill_fa_t<true, 2>(tmK, tmV, tmQ, tmR, a, grid, s) : launch_prefill_fa_t<true, 1>(tmK, tmV, tmQ, tmR, a, grid, s);
            else if (exact) r = mt == 2 ? launch_prefill_fa_t<false, 2, true>(tmK, tmV, tmQ, tmR, a, grid, s) : launch_prefill_fa_t<false, 1, true>(tmK, tmV, tmQ, tmR, a, grid, s);
            else r = mt == 2 ? launch_prefill_fa_t<false, 2>(tmK, tmV, tmQ, tmR, a, grid, s) : launch_prefill_fa_t<false, 1>(tmK, tmV, tmQ, tmR, a, grid, s);
            if (r != TQ_OK) return r;
        }
    }
    return TQ_OK;
}

inline int launch_fp16_attention(const Fp16AttnParams& p_in, cudaStream_t s) {
    // A CTA serves at most two query heads per pass over the rows (more cost it its occupancy: 47 % of the copy
    // bandwidth with four, 23 % with eight).  With 4 or 8 query heads per KV head, 2 or 4 CTAs share the rows of a KV
    // head as "virtual" KV heads; they are neighbours in the grid, so all but the first read the rows from L2.
    const int grp = p_in.H / p_in.Hkv;
    Fp16AttnParams p = p_in;
    p.Hkv = p_in.Hkv << (grp == 4 ? 1 : (grp == 8 ? 2 : 0));
    dim3 grid(p.Hkv, p.nchunk_max, p.G);  // KV heads fastest: CTAs that run together read the same 2 KB rows (DRAM page locality)
    dim3 block(FP16_WARPS * 32);
    switch (grp) {
        case 1: fp16_decode_attention_kernel<1, 0><<<grid, block, 0, s>>>(p); break;
        case 2: fp16_decode_attention_kernel<2, 0><<<grid, block, 0, s>>>(p); break;
        case 4: fp16_decode_attention_kernel<2, 1><<<grid, block, 0, s>>>(p); break;
        case 8: fp16_decode_attention_kernel<2, 2><<<grid, block, 0, s>>>(p); break;
        default: return TQ_ERR_UNSUPPORTED;
    }
    return cuda_status(cudaGetLastError());
}

// ---- per-device workspace of the compat launchers + descriptor cache ----------------------------------------------------------
// The reference's launchers get every buffer from their caller; the kernels here need scratch of their own (rotated
// queries, tile table, split-K partials), which the reference-compatible launchers keep per device.  All of this state
// is guarded by ONE mutex that a launcher holds from its first look at the state until its kernels are enqueued: the
// compat launchers serialise per process (their host part is a few microseconds).
struct CompatState {
    void* ws = nullptr;
    size_t ws_bytes = 0;
    std::vector<void*> retired;  // outgrown workspaces: kernels already enqueued may still use them, so they stay allocated
    std::map<std::tuple<const void*, long long, int>, CUtensorMap> maps;  // descriptors by (base, rows, row bytes)
};

inline std::recursive_mutex& compat_mutex() {
    static std::recursive_mutex mu;
    return mu;
}

// Call with compat_mutex() held.
inline CompatState& compat_state() {
    static std::map<int, CompatState> st;
    int dev = 0;
    cudaGetDevice(&dev);
    return st[dev];
}

// Call with compat_mutex() held.  The workspace only ever grows, and by at least a factor of two (first allocation:
// 64 MiB or the request), so a serving loop reaches its final size after a few calls; growth allocates a new buffer
// and retires the old one without waiting for the device.
inline int compat_workspace(size_t need, void** out, cudaStream_t s) {
    CompatState& c = compat_state();
    if (c.ws_bytes < need) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(s, &cs);
        if (cs != cudaStreamCaptureStatusNone) return TQ_ERR_WORKSPACE;  // cannot allocate while capturing
        size_t bytes = std::max(need, std::max(c.ws_bytes * 2, (size_t)64 << 20));
        void* fresh = nullptr;
        if (cudaMalloc(&fresh, bytes) != cudaSuccess) {
            cudaGetLastError();
            bytes = need;
            TQ_CUDA(cudaMalloc(&fresh, bytes));
        }
        TQ_CUDA(cudaMemsetAsync(fresh, 0, bytes, s));
        if (c.ws) c.retired.push_back(c.ws);
        c.ws = fresh;
        c.ws_bytes = bytes;
    }
    *out = c.ws;
    return TQ_OK;
}

// Call with compat_mutex() held.  The fp16 twin's descriptors share the cache (key: minus the row bytes).
inline int cached_fp16_map(CUtensorMap* out, const void* base, long long rows, int kv_dim) {
    CompatState& c = compat_state();
    auto key = std::make_tuple(base, rows, -2 * kv_dim);
    auto it = c.maps.find(key);
    if (it == c.maps.end()) {
        CUtensorMap m;
        int r = make_fp16_rows_map(&m, base, rows, kv_dim);
        if (r != TQ_OK) return r;
        if (c.maps.size() > 4096) c.maps.clear();
        it = c.maps.emplace(key, m).first;
    }
    *out = it->second;
    return TQ_OK;
}

// Call with compat_mutex() held.
inline int cached_code_map(CUtensorMap* out, const void* base, long long rows, int kvp) {
    CompatState& c = compat_state();
    auto key = std::make_tuple(base, rows, kvp);
    auto it = c.maps.find(key);
    if (it == c.maps.end()) {
        CUtensorMap m;
        int r = make_code_map(&m, base, rows, kvp);
        if (r != TQ_OK) return r;
        if (c.maps.size() > 4096) c.maps.clear();
        it = c.maps.emplace(key, m).first;
    }
    *out = it->second;
    return TQ_OK;
}

}  // namespace tq

// =====================================================================================================================
// Engine state (opaque to C callers)
// =====================================================================================================================
struct tq_engine {
    tq_model_shape shape{};
    int ctor_max_seq_len = 0;
    int kv_bits = 0;
    int device = 0;

    // arena
    char* arena = nullptr;
    size_t arena_cap = 0;
    bool arena_external = false;
    bool asleep = false;
    // The last thing this engine put on `chain_stream` was a fused decode launch: positions and caches are as that
    // launch saw them, so the next fused launch may read them before it has seen its predecessor finish.
    bool chain_ok = false;
    cudaStream_t chain_stream = nullptr;
    bool fused = !(getenv("TQ_FUSED") && atoi(getenv("TQ_FUSED")) == 0);  // the layer form, not the two-launch form (packed modes)

    // current carving
    int G = 0;
    int msl = 0;          // dense slot size, or the largest capacity in ragged mode
    bool ragged = false;
    long long total_rows = 0;
    std::vector<int> capacities;       // rows of every slot (ragged: rounded up to 32; dense: the slot size)
    std::vector<long long> h_row_base; // first row of every slot
    // Shared prefixes: sequence g reads its first prefix_tokens[g] tokens (a multiple of 32) from the slot of
    // prefix_owner[g]; its own slot then starts at token prefix_tokens[g].  0 / -1: nothing shared.
    std::vector<int> prefix_tokens, prefix_owner;
    bool shared_active = false;
    long long* d_prefix_base = nullptr;  // [G] first row of the shared tiles
    int* d_prefix_tiles = nullptr;       // [G] number of shared tiles
    // the slot table the kernels see (null in the dense layout without shared prefixes: row = g * max_seq_len + pos)
    const long long* rb() const { return (ragged || shared_active) ? d_row_base : nullptr; }
    const int* caps() const { return (ragged || shared_active) ? d_capacities : nullptr; }
    long long row0_eff(int g) const { return h_row_base[g] - prefix_tokens[g]; }   // row of token 0 if the slot started there
    int cap_eff(int g) const { return capacities[g] + prefix_tokens[g]; }          // positions the sequence may reach

    struct Layer {
        void* k = nullptr;
        void* v = nullptr;
        void* kn = nullptr;
        void* vn = nullptr;
        CUtensorMap tmK{}, tmV{};  // packed modes: descriptors of the code arrays
    };
    std::vector<Layer> layers;

    // whole-step form: all layers' code arrays as one tensor map each, per-layer split-K partials, the tile table
    CUtensorMap tmK4{}, tmV4{};
    size_t code_layer_stride = 0;      // bytes between consecutive layers' K (and V) code arrays
    size_t norm_layer_stride = 0;      // bytes between consecutive layers' norm arrays
    float* step_partials = nullptr;    // [layers][workers + G][H][PART_STRIDE]
    size_t step_part_stride = 0;       // floats per layer
    int* step_table = nullptr;         // [G + 4]
    void* step_qrot = nullptr;         // [layers][G][H][128] fp16: pre-rotated, pre-scaled queries
    void* step_kpost = nullptr;        // [layers][G][kv_dim] fp16: K after QK-norm and rotary embedding (producer form)
    void* prefill_scratch = nullptr;   // packed modes: fp16 rows and fp32 norms of prompts (launch_prefill_attention)
    size_t prefill_scratch_bytes = 0;
    // Its users are calls on any stream of any host thread: a call on another stream than the last one's waits for that one's kernels.
    std::mutex prefill_mutex;
    cudaEvent_t ev_prefill = nullptr;           // behind the last use
    unsigned long long prefill_stream_id = 0;   // whose stream it was (0: none yet)
    bool whole_step = !(getenv("TQ_WHOLE_STEP") && atoi(getenv("TQ_WHOLE_STEP")) == 0);
    float* out_f32 = nullptr;          // optional [layers][G][H][128]: results before the fp16 rounding (outside the arena)
    cudaEvent_t ev_attn[2] = {nullptr, nullptr};  // optional: recorded around the attention launch of the whole-step form

    int* d_positions = nullptr;
    int* d_capacities = nullptr;       // [G] positions each sequence may reach (slot rows + shared prefix tokens)
    long long* d_row_base = nullptr;   // [G] first row of every slot, minus the sequence's shared prefix tokens
    void* workspace = nullptr;
    size_t ws_bytes = 0;
    void* stage_q = nullptr;   // [layers][G][q_dim]
    void* stage_k = nullptr;   // [layers][G][kv_dim]
    void* stage_v = nullptr;
    void* stage_out = nullptr; // [layers][G][q_dim]
    // host-buffer steps: copy streams and events that let the copies of one group of layers overlap the kernels of another
    static constexpr int HOST_STEP_CHUNKS = 9;
    cudaStream_t st_in = nullptr, st_out = nullptr;
    cudaEvent_t ev_begin = nullptr, ev_done = nullptr;
    cudaEvent_t ev_in[HOST_STEP_CHUNKS] = {}, ev_out[HOST_STEP_CHUNKS] = {};

    // rotation: host copy kept across sleep, device copies (R and R transposed, 32 KB each) outside the arena
    std::vector<uint16_t> h_rotation;
    void* d_rotation = nullptr;
    void* d_rotation_t = nullptr;
    float* d_rotation_prep = nullptr;  // fp32, in the append kernel's shared-memory order
    void* d_rotation_rep = nullptr;    // R row-major, several copies, for layer_prep_kernel

    // sleep that keeps the sequences: every sequence's written rows as a blob in host memory (see tq_engine_export_sequence)
    struct Kept {
        bool valid = false;
        int G = 0, max_seq_len = 0;
        bool ragged = false;
        std::vector<int> capacities, positions;
        std::vector<std::vector<unsigned char>> blobs;
    } kept;

    int q_dim() const { return shape.num_heads * shape.head_dim; }
    int kv_dim() const { return shape.num_kv_heads * shape.head_dim; }
    int vpb() const { return kv_bits == 2 ? 4 : 2; }
    // bytes per cache row (all KV heads) of one of K / V: engine/engine.cpp:292-294 for the packed modes
    size_t code_row_bytes() const { return kv_bits == 0 ? (size_t)kv_dim() * 2 : (size_t)kv_dim() / vpb(); }
};

namespace tq {

// Walks the arena exactly as tq_engine_alloc_batch carves it.  base == nullptr only measures.
struct ArenaPlan {
    size_t bytes = 0;
    long long total_rows = 0;
};

inline size_t bump(size_t& off, size_t bytes) {
    off = (off + 255) & ~(size_t)255;  // 256-byte alignment, as GpuArena::alloc (engine/model.h:264-279)
    size_t at = off;
    off += bytes;
    return at;
}

inline long long plan_rows(int G, int max_seq_len, const int* capacities, std::vector<int>* caps_out,
                           std::vector<long long>* base_out) {
    long long rows = 0;
    if (capacities == nullptr) {
        for (int g = 0; g < G; ++g) {
            if (caps_out) caps_out->push_back(max_seq_len);
            if (base_out) base_out->push_back((long long)g * max_seq_len);
        }
        return (long long)G * max_seq_len;
    }
    for (int g = 0; g < G; ++g) {
        int c = capacities[g] < 1 ? 1 : capacities[g];
        c = (c + TILE_TOKENS - 1) / TILE_TOKENS * TILE_TOKENS;
        if (caps_out) caps_out->push_back(c);
        if (base_out) base_out->push_back(rows);
        rows += c;
    }
    return rows;
}

}  // namespace tq
