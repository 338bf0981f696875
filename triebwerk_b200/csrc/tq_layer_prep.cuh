// What a decode layer needs before its attention over a packed cache: the step's new token appended and the queries rotated, sm_100a.
//
// One launch in front of decode_attention_kernel's layer form (tq_attention.cuh).  The rotation of all vectors runs on
// mma.sync.m16n8k16: 16 query heads, or one sequence's 2 * Hkv new K and V head vectors, are the rows of the A operand as they
// arrive, R is the B operand and stays in registers (16 coordinates per warp).  Queries leave scaled by log2(e) / sqrt(128).  The new
// token's coordinates are divided by the norm afterwards; one within PREP_MARGIN of a decision bound is recomputed with the
// reference's exact fp32 chain, as in tq_prefill_tc.cuh, so that the stored bytes are the reference's.
// Bound by latency: one round trip for the vectors, the products, the stores (R's trip lies under the previous kernel where
// no kernel writes R).  When the attention kernel did this itself, every worker fetched R and rotated its sequences' queries between
// the previous layer's end and its first tile, a few workers had the append on top, and its warps the registers of all that
// in their tile loop, without copy warps.
// From the wait on (32 x 8192 tokens, 2-bit, 32/8 heads): rotated queries stored after 2.1 us, the appends after 2.8 to 4.3; inside the
// attention kernel 3.7 and 7.  A piece of 16 vectors per CTA while two CTAs per SM hold all pieces; beyond that CTAs loop.
#pragma once

#include "tq_attention.cuh"

namespace tq {

constexpr int PREP_THREADS = 256;
// Twice the bound on either sum's rounding, 128 terms whose magnitudes sum to 1 at most (7.7e-6 each), and 1.5e-6 for the norm's two places: on
// every term in the exact chain, on the sum here.  The two chains of products here round less often than that; largest difference measured to the exact
// chain 8.4e-7 (1.9e9 coordinates: normal, heavy-tailed, all terms of one sign, 1e-5 to 65504).  Bytes against the two-launch form's: 2.15e9
// coordinates of those kinds, none differ.
constexpr float PREP_MARGIN = 1.7e-5f;
constexpr int PREP_ROW = HEAD_DIM + 8;  // halves per row of R in shared memory

struct LayerPrepParams {
    uint8_t* ck;                 // the layer's cache arrays
    uint8_t* cv;
    __half* kn;
    __half* vn;
    const __half* new_k;         // [G][Hkv * 128], or null: nothing is appended
    const __half* new_v;
    const __half* q;             // [G][q_dim]
    const __half* rotation;      // R row-major, rot_copies copies back to back
    int rot_copies;              // CTA b reads copy b % rot_copies: all of them fetch the same 32 KB at once
    int static_rotation;         // R is not written by any kernel of the stream: fetched before the wait
    __half* q_rot16;             // [G][H][128], or as fp32:
    float* q_rot32;              // (in AttnParams::q_rot32's order)
    __half* rotation_t;          // or null: R transposed goes here, for the merge
    const int* positions;        // device [G] or null: pos_value
    const long long* row_base;   // [G] or null: g * max_seq_len
    const int* seq_capacity;     // [G] or null: capacity_rows
    int* status;
    int pos_value, max_seq_len, capacity_rows;
    int G, H, Hkv, q_dim;
};

template <int BITS>
__global__ void __launch_bounds__(PREP_THREADS, 2) layer_prep_kernel(const LayerPrepParams p) {
    __shared__ __align__(16) __half raw[16][HEAD_DIM];  // the new token's vectors as they arrived
    __shared__ __align__(16) __half r_s[HEAD_DIM][PREP_ROW];  // R, for the exact chains
    __shared__ float inv_s[16], ss_s[16];
    __shared__ float bound_s[17];  // decision bounds between -inf and +inf
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gl = lane >> 2, t4 = lane & 3;
    const long long n_vec = (long long)p.G * p.H;
    const long long n_app = p.new_k ? p.G : 0, n_items = n_app + (n_vec + 15) / 16;
    const __half* const R = p.rotation + (size_t)(blockIdx.x % p.rot_copies) * (HEAD_DIM * HEAD_DIM);
    // B fragments of the coordinate blocks 2 warp and 2 warp + 1; step (m, e) of lane t4 covers k = 32m + 8*t4 + 4e .. +3, on both sides
    uint4 bf[2][4];
    auto fetch_rotation = [&]() {
        if (blockIdx.x >= n_items) return;  // (a CTA that only helps with the transposition)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int m = 0; m < 4; ++m) bf[i][m] = ldg128_now(reinterpret_cast<const uint4*>(R + (size_t)(8 * (2 * warp + i) + gl) * HEAD_DIM) + t4 + 4 * m);
    };
    // (the exact chains read R from here: four round trips to L2 for a few lanes were half of the append's 5 us)
    auto stage_rotation = [&]() {
        if (!p.new_k || blockIdx.x >= p.G) return;  // no append among this CTA's items
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int m = 0; m < 4; ++m) *reinterpret_cast<uint4*>(&r_s[8 * (2 * warp + i) + gl][32 * m + 8 * t4]) = bf[i][m];
    };
    constexpr int NBND = BITS == 4 ? 15 : 3;
    if (tid <= NBND + 1) bound_s[tid] = tid == 0 ? -3.4e38f : (tid > NBND ? 3.4e38f : (BITS == 4 ? kBnd4[(tid - 1) & 15] : kBnd2[(tid - 1) & 3]));
    if (p.static_rotation) {
        fetch_rotation();
        stage_rotation();
    }
    pdl_wait();
    pdl_launch_dependents();  // (what came before this launch has finished: the attention may read positions and old rows)
    if (!p.static_rotation) {
        fetch_rotation();
        stage_rotation();
    }
    if (p.rotation_t)
        for (int i = (int)blockIdx.x * PREP_THREADS + tid; i < HEAD_DIM * HEAD_DIM; i += (int)gridDim.x * PREP_THREADS)
            p.rotation_t[i] = R[(i & (HEAD_DIM - 1)) * HEAD_DIM + (i >> 7)];
    const int nvec = 2 * p.Hkv;
    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        const bool app = item < n_app;
        // rows gl and gl + 8 of the A operand
        const __half* src[2];
        bool on[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int v = gl + 8 * r;
            if (app) {
                on[r] = v < nvec;
                src[r] = (v < p.Hkv ? p.new_k : p.new_v) + ((size_t)item * p.Hkv + (v < p.Hkv ? v : v - p.Hkv)) * HEAD_DIM;
            } else {
                const long long vec = (item - n_app) * 16 + v, g = vec / p.H;
                on[r] = vec < n_vec;
                src[r] = p.q + (size_t)g * p.q_dim + (size_t)(vec - g * p.H) * HEAD_DIM;
            }
        }
        uint4 a[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                a[r][m] = make_uint4(0u, 0u, 0u, 0u);
                if (on[r]) a[r][m] = ldg128_now(reinterpret_cast<const uint4*>(src[r]) + t4 + 4 * m);
            }
        int pos = p.pos_value, cap = p.capacity_rows;
        long long row = 0;
        float x4[2][4];  // append: the vectors 2 warp and 2 warp + 1, coordinates lane + 32 c
        if (app) {
            if (p.positions) pos = p.positions[item];
            if (p.seq_capacity) cap = p.seq_capacity[item];
            row = p.row_base ? p.row_base[item] : (long long)item * p.max_seq_len;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int v = 2 * warp + i;
                const __half* const x = (v < p.Hkv ? p.new_k : p.new_v) + ((size_t)item * p.Hkv + (v < p.Hkv ? v : v - p.Hkv)) * HEAD_DIM;
#pragma unroll
                for (int c = 0; c < 4; ++c) x4[i][c] = v < nvec ? __half2float(x[lane + 32 * c]) : 0.0f;
            }
        }
        const bool ok = pos >= 0 && (cap <= 0 || pos < cap);
        row += pos;
        float c[2][2][4];  // [block][chain]
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) c[i][0][e] = c[i][1][e] = 0.0f;
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mma16816(c[i][0], a[0][m].x, a[1][m].x, a[0][m].y, a[1][m].y, bf[i][m].x, bf[i][m].y);
                mma16816(c[i][1], a[0][m].z, a[1][m].z, a[0][m].w, a[1][m].w, bf[i][m].z, bf[i][m].w);
            }
        if (!app) {
            constexpr float sc = 0.12751743074602467f;  // log2(e) / sqrt(128)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float y0 = (c[i][0][2 * r] + c[i][1][2 * r]) * sc, y1 = (c[i][0][2 * r + 1] + c[i][1][2 * r + 1]) * sc;
                    const size_t vec = (size_t)((item - n_app) * 16 + gl + 8 * r) * HEAD_DIM;
                    if (!on[r]) continue;
                    if (p.q_rot32) *reinterpret_cast<float2*>(p.q_rot32 + vec + 16 * (4 * (warp & 1) + 2 * i + (t4 >> 1)) + 4 * (warp >> 1) + 2 * (t4 & 1)) = make_float2(y0, y1);
                    else *reinterpret_cast<__half2*>(p.q_rot16 + vec + 8 * (2 * warp + i) + 2 * t4) = __floats2half2_rn(y0, y1);
                }
            continue;
        }
        if (warp == 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int m = 0; m < 4; ++m) *reinterpret_cast<uint4*>(&raw[gl + 8 * r][32 * m + 8 * t4]) = a[r][m];
        }
        // sums of squares in the reference's order (tq_append.cuh); norms
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float sq[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) sq[k] = mul_ftz(x4[i][k], x4[i][k]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) sq[k] = add_ftz(sq[k], __shfl_down_sync(0xffffffffu, sq[k], off));
            const int v = 2 * warp + i;
            if (lane == 0) {
                const float ss = add_ftz(add_ftz(sq[0], sq[2]), add_ftz(sq[1], sq[3])), t = add_ftz(ss, 1e-12f);
                ss_s[v] = ss;
                inv_s[v] = rsqrt_approx_ftz(t);
                if (v < nvec && ok) (v < p.Hkv ? p.kn : p.vn)[(size_t)row * p.Hkv + (v < p.Hkv ? v : v - p.Hkv)] = __float2half_rn(sqrt_approx_ftz(t));
            }
        }
        if (tid == 0 && !ok) atomicMax(p.status, ST_BAD_POSITION);
        __syncthreads();
        // the codes: how many bounds a coordinate has reached (NaN: as the reference's comparisons fall out); value 4 r + e: row gl + 8 r,
        // block e >> 1, coordinate 2 t4 + (e & 1) of it.  (All eight a step at a time: their look-ups are in flight together.)
        auto search = [&](const float* y, auto count, uint32_t* n) {
            constexpr int C = decltype(count)::value;
#pragma unroll
            for (int i = 0; i < C; ++i) n[i] = 0u;
#pragma unroll
            for (uint32_t step = (NBND + 1) / 2; step > 0; step >>= 1) {
                float b[C];
#pragma unroll
                for (int i = 0; i < C; ++i) b[i] = bound_s[n[i] + step];
#pragma unroll
                for (int i = 0; i < C; ++i) n[i] += y[i] >= b[i] ? step : 0u;
            }
            if (BITS == 4) {
#pragma unroll
                for (int i = 0; i < C; ++i) n[i] = y[i] != y[i] ? 15u : n[i];
            }
        };
        float x[8];
        uint32_t n8[8], codes = 0u, near = 0u, zeros = 0u;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float inv = inv_s[gl + 8 * r], ss = ss_s[gl + 8 * r];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 4 * r + e;
                const float rot = c[e >> 1][0][2 * r + (e & 1)] + c[e >> 1][1][2 * r + (e & 1)];
                x[i] = mul_ftz(rot, inv);
                if (!(add_ftz(ss, 1e-12f) < 3.0e38f)) x[i] = __int_as_float(0x7fc00000);  // an infinity or a NaN among the inputs: NaN everywhere, as in the reference
                const bool zero = ss == 0.0f && rot == 0.0f;  // all zero: every coordinate is 0, on a bound but exact
                if (zero) x[i] = 0.0f;
                if (zero || gl + 8 * r >= nvec) zeros |= 1u << i;
            }
        }
        search(x, std::integral_constant<int, 8>(), n8);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            codes |= n8[i] << (4 * i);
            near |= fminf(x[i] - bound_s[n8[i]], bound_s[n8[i] + 1] - x[i]) < PREP_MARGIN ? 1u << i : 0u;
        }
        near &= ~zeros;
        while (near) {  // about 1 coordinate in 700: the reference's k-ascending chain
            const int at = __ffs((int)near) - 1, v = gl + 8 * (at >> 2), d = 8 * (2 * warp + ((at >> 1) & 1)) + 2 * t4 + (at & 1);
            near &= near - 1u;
            const float inv = inv_s[v];
            float acc = 0.0f;
#pragma unroll 4
            for (int k = 0; k < 16; ++k) {
                const uint4 rv = *reinterpret_cast<const uint4*>(&r_s[d][8 * k]), xv = *reinterpret_cast<const uint4*>(&raw[v][8 * k]);
                const __half2* const rh = reinterpret_cast<const __half2*>(&rv);
                const __half2* const xh = reinterpret_cast<const __half2*>(&xv);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 rf = __half22float2(rh[e]), xf = __half22float2(xh[e]);
                    acc = fma_ftz(rf.x, mul_ftz(xf.x, inv), acc);
                    acc = fma_ftz(rf.y, mul_ftz(xf.y, inv), acc);
                }
            }
            uint32_t n;
            search(&acc, std::integral_constant<int, 1>(), &n);
            codes = (codes & ~(15u << (4 * at))) | n << (4 * at);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int v = gl + 8 * r;
            // the 16 coordinates 16 warp .. of row v: from its four lanes into 8 (4) bytes
            uint32_t w0, w1 = 0u;
            if (BITS == 4) {
                w0 = ((codes >> (16 * r)) & 0xffu) << (8 * t4);
                w1 = ((codes >> (16 * r + 8)) & 0xffu) << (8 * t4);
            } else {
                auto pair = [&](int e) { return ((codes >> (4 * (4 * r + e))) & 3u) | ((codes >> (4 * (4 * r + e) + 4)) & 3u) << 2; };
                w0 = pair(0) << (4 * t4) | pair(2) << (4 * t4 + 16);
            }
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                w0 |= __shfl_xor_sync(0xffffffffu, w0, o);
                if (BITS == 4) w1 |= __shfl_xor_sync(0xffffffffu, w1, o);
            }
            if (t4 == 0 && v < nvec && ok) {
                constexpr int BPH = HEAD_DIM * BITS / 8;
                uint8_t* const dst = (v < p.Hkv ? p.ck : p.cv) + ((size_t)row * p.Hkv + (v < p.Hkv ? v : v - p.Hkv)) * BPH + 2 * BITS * warp;
                if (BITS == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(w0, w1);
                else *reinterpret_cast<uint32_t*>(dst) = w0;
            }
        }
        __syncthreads();  // (the next item's vectors)
    }
}

}  // namespace tq
