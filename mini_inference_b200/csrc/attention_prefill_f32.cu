// Paged attention for prompt portions in true float32, head size 64 or 128: tiles of 64 query rows x 32 keys, both products on the
// CUDA cores with the packed two-float multiply-add, online softmax in between.  Masks, sink, distance terms, cap, kept keys and gate as
// csrc/attention_masked.cu states them (keys and values of one size); plain causal attention is the case with all of them off.
//
// The kernel with a warp per query row read every key and value once per row (501 tokens x 32 heads: 3.1 ms).  Here a key
// is read from the pages once per 64 rows and an operand from shared memory once per 4 (rows) or 4 to 16 (columns) multiply-adds a lane;
// the float32 FMA rate is the bound.  64 rows leave two blocks of 110 KB an SM and enough blocks for short prompts; 128 rows need fewer
// loads but their longest tile alone takes twice as long.  A Qwen3-4B-size layer of 501 tokens went from 8.7 to 3.05 ms with this kernel and
// the float32 product's tiles; 3.0 ms of the gain are this kernel's.
//
// The arithmetic of a row depends on its own position only: tiles lie at multiples of 32 keys from the start of the sequence, and a tile
// without visible keys changes no bit (its weights are zeros, the factor that rescales is one).
#include "common.cuh"
#include <math.h>
#include <type_traits>

using namespace mi;

namespace {

constexpr int BQ = 64, BK = 32, THREADS = 128;

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

struct Terms {
    int block, window, sink, keep, bias_last, gate_stride;
    float cap;
    const float *sink_values, *bias, *slopes, *gate;          // bias [bias_last + 1, H]
};

template <int D>
struct Smem {
    static constexpr int LQ = D + 4, LP = BK + 4;             // rows padded by 16 bytes: a quarter warp's eight rows in different banks
    static constexpr int Q = 0, K = Q + BQ * LQ, V = K + 2 * BK * LQ, P = V + 2 * BK * D, FLOATS = P + BQ * LP;
};

template <int D, bool PLAIN>
__global__ void __launch_bounds__(THREADS, 2)
attn_prefill_f32_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                        float* __restrict__ out, const int* __restrict__ tiles, const int* __restrict__ seg_q_start,
                        const int* __restrict__ seg_pos0, const int* __restrict__ block_table, const int* __restrict__ table_rows,
                        int table_stride, int H, int KV, int ps, float scale, const Terms t) {
    using L = Smem<D>;
    constexpr int CH = D / 4, DV = D / 32;                    // 16-byte pieces of a row; pieces of four output columns a lane owns
    extern __shared__ __align__(16) float smem[];
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lm = lane >> 3, ln = lane & 7;
    const int tile = gridDim.y - 1 - blockIdx.y;              // the longest tile of every head first
    const int seg = tiles[2 * tile], r0 = tiles[2 * tile + 1];
    const int h = blockIdx.x, kvh = h / (H / KV);
    const int qs = seg_q_start[seg], n = seg_q_start[seg + 1] - qs, pos0 = seg_pos0[seg];
    const int rows = min(BQ, n - r0);
    const int* table_row = block_table + (size_t)(table_rows ? table_rows[seg] : seg) * table_stride;
    const int p_first = pos0 + r0, p_last = p_first + rows - 1;
    auto first_key = [&](int p) { return max(t.block > 0 ? p / t.block * t.block : 0, t.window > 0 ? p - t.window + 1 : 0); };
    const int kt_first = first_key(p_first) / BK, kt_hi = p_last / BK;
    // the tiles of the kept keys come first (those that the window's tiles do not hold anyway)
    const int kept_tiles = !PLAIN && t.window > 0 ? min((t.keep + BK - 1) / BK, kt_first) : 0;
    const int kt_lo = kt_first - kept_tiles;
    auto kt_of = [&](int it) { return it < kt_first ? it - kt_lo : it; };

    auto load_kv = [&](int it) {
        const int kt = kt_of(it), buf = (it - kt_lo) & 1;
        for (int id = tid; id < BK * CH; id += THREADS) {
            const int row = id / CH, ch = id % CH, j = kt * BK + row;
            const bool ok = j <= p_last;
            const size_t off = ok ? ((size_t)(table_row[j / ps] * KV + kvh) * ps + j % ps) * D + ch * 4 : 0;
            cp16(s0 + (L::K + (buf * BK + row) * L::LQ + ch * 4) * 4, k_cache + off, ok);
            cp16(s0 + (L::V + (buf * BK + row) * D + ch * 4) * 4, v_cache + off, ok);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    load_kv(kt_lo);
    for (int id = tid; id < BQ * CH; id += THREADS) {
        const int row = id / CH, ch = id % CH;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows) v = *reinterpret_cast<const float4*>(q + (size_t)(qs + r0 + row) * q_stride + (size_t)h * D + ch * 4);
        *reinterpret_cast<float4*>(smem + L::Q + row * L::LQ + ch * 4) = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
    }
    // a lane's rows are warp * 16 + lm + 4 i; its keys of a tile ln + 8 j; its output columns 4 ln + 32 c ..
    const int row0 = warp * 16 + lm;
    const float slope = !PLAIN && t.slopes ? t.slopes[h] : 0.f;
    const float m_start = !PLAIN && t.sink ? (t.sink_values ? t.sink_values[h] : 0.f) : -INFINITY;
    float m[4], l[4];
    float2 o[4][2 * DV];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = m_start;
        l[i] = !PLAIN && t.sink ? 1.f : 0.f;
#pragma unroll
        for (int c = 0; c < 2 * DV; ++c) o[i][c] = make_float2(0.f, 0.f);
    }
    for (int it = kt_lo; it <= kt_hi; ++it) {
        const int kt = kt_of(it), buf = (it - kt_lo) & 1;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                                       // the tile (and, the first time, q) is there; the other buffer is free
        if (it < kt_hi) load_kv(it + 1);
        // ---- scores
        float2 acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
        const float* qp = smem + L::Q + row0 * L::LQ;
        const float* kp = smem + L::K + (buf * BK + ln) * L::LQ;
#pragma unroll 8
        for (int d = 0; d < D; d += 4) {
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(kp + 8 * j * L::LQ + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(qp + 4 * i * L::LQ + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(a.x, a.y), make_float2(b[j].x, b[j].y), acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(a.z, a.w), make_float2(b[j].z, b[j].w), acc[i][j]);
            }
        }
        // ---- terms, mask, online softmax; the weights go to this warp's rows of P
        const int p_warp = p_first + warp * 16;                // a key that a row does not see may hold anything, and 0 * inf is no 0: its weight is marked
        const bool whole = kt * BK + BK - 1 <= p_warp && (kt * BK >= first_key(p_warp + 15) || (!PLAIN && kt * BK + BK <= t.keep));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = p_first + row0 + 4 * i, lo = first_key(p);
            float s[4], mx = -INFINITY;
            bool seen[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = kt * BK + ln + 8 * j;
                s[j] = acc[i][j].x + acc[i][j].y;
                if (!PLAIN) {
                    const int dist = p - key;
                    if (t.bias && dist >= 0) s[j] += t.bias[(size_t)min(dist, t.bias_last) * H + h];
                    if (slope != 0.f) s[j] -= slope * (float)dist;
                    if (t.cap > 0.f) s[j] = t.cap * tanhf(s[j] / t.cap);
                }
                seen[j] = key <= p && (key >= lo || (!PLAIN && key < t.keep));
                s[j] = seen[j] ? s[j] : -INFINITY;
                mx = fmaxf(mx, s[j]);
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            const float m_new = fmaxf(m[i], mx), z = m_new == -INFINITY ? 0.f : m_new;       // a row that has seen no key yet
            const float alpha = expf(m[i] - z);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float w = expf(s[j] - z);
                sum += w;
                smem[L::P + (row0 + 4 * i) * L::LP + ln + 8 * j] = seen[j] ? w : -1.f;
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 2 * DV; ++c) o[i][c] = make_float2(o[i][c].x * alpha, o[i][c].y * alpha);
        }
        __syncwarp();
        // ---- the weighted sum; a tile that some row of the warp does not see whole leaves the marked weights out
        const float* pp = smem + L::P + row0 * L::LP;
        const float* vp = smem + L::V + buf * BK * D + 4 * ln;
        auto add_values = [&](auto marked) {
#pragma unroll 2
            for (int k = 0; k < BK; k += 4) {
                float w[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 v = *reinterpret_cast<const float4*>(pp + 4 * i * L::LP + k);
                    w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int c = 0; c < DV; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(vp + (k + e) * D + 32 * c);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (decltype(marked)::value && w[i][e] < 0.f) continue;
                            const float2 ww = make_float2(w[i][e], w[i][e]);
                            o[i][2 * c] = __ffma2_rn(ww, make_float2(v.x, v.y), o[i][2 * c]);
                            o[i][2 * c + 1] = __ffma2_rn(ww, make_float2(v.z, v.w), o[i][2 * c + 1]);
                        }
                    }
            }
        };
        if (whole) add_values(std::false_type{}); else add_values(std::true_type{});
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + 4 * i;
        if (r >= rows) continue;
        const size_t tok = (size_t)(qs + r0 + r);
        float* orow = out + (tok * H + h) * D + 4 * ln;
        const float* grow = !PLAIN && t.gate ? t.gate + tok * t.gate_stride + (size_t)h * D + 4 * ln : nullptr;
#pragma unroll
        for (int c = 0; c < DV; ++c) {
            float v[4] = {o[i][2 * c].x / l[i], o[i][2 * c].y / l[i], o[i][2 * c + 1].x / l[i], o[i][2 * c + 1].y / l[i]};
            if (grow)
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = v[e] / (1.f + expf(-grow[32 * c + e]));
            *reinterpret_cast<float4*>(orow + 32 * c) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

}  // namespace

// tiles: (entry, first row) of 64-row tiles; out [T, H D].  plain: causal with an optional window, the other terms off.
MI_EXPORT int mi_attn_prefill_f32(const float* q, int q_stride, const float* k_cache, const float* v_cache, float* out, const int* tiles,
                                  int num_tiles, const int* seg_q_start, const int* seg_pos0, const int* block_table, const int* table_rows,
                                  int table_stride, int H, int KV, int D, int ps, int tile_rows, float scale, int block, int window, int sink,
                                  const float* sink_values, const float* bias, int bias_last, const float* slopes, float cap, int keep,
                                  const float* gate, int gate_stride, cudaStream_t stream) {
    if (num_tiles == 0) return 0;
    if ((D != 64 && D != 128) || H % KV || tile_rows != BQ || q_stride % 4 || ((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) % 16) return -2;
    const Terms t{block, window, sink, window > 0 ? keep : 0, bias_last, gate_stride, cap, sink_values, bias, slopes, gate};
    const bool plain = block <= 0 && !sink && !bias && !slopes && cap <= 0.f && t.keep <= 0 && !gate;
    const dim3 grid(H, num_tiles);
#define LAUNCH(DD, PP) do { \
        constexpr int bytes = Smem<DD>::FLOATS * 4; \
        static bool configured = false; \
        if (!configured) { \
            cudaError_t e = cudaFuncSetAttribute(attn_prefill_f32_kernel<DD, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); \
            if (e != cudaSuccess) return (int)e; \
            configured = true; \
        } \
        attn_prefill_f32_kernel<DD, PP><<<grid, THREADS, bytes, stream>>>(q, q_stride, k_cache, v_cache, out, tiles, seg_q_start, seg_pos0, \
                                                                         block_table, table_rows, table_stride, H, KV, ps, scale, t); \
    } while (0)
    if (D == 128) { if (plain) LAUNCH(128, true); else LAUNCH(128, false); }
    else { if (plain) LAUNCH(64, true); else LAUNCH(64, false); }
#undef LAUNCH
    return (int)cudaGetLastError();
}
