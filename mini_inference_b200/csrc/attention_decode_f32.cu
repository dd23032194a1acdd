// Decoded tokens in true float32 over the pages: one block per (request, key head, piece of the keys), its eight warps take eight keys at a time in turn,
// each with an online softmax of its own that the block merges at the end.
//
// Bound by the keys' and values' bytes: a warp reads a key's row as one line (a lane D / 32 neighbouring entries), once for all query heads of the key
// head, eight keys and eight values in flight.  The 8 G partial products of a lane are summed over lanes together (31 shuffles for 32 sums), lane
// l ends with the score of key l / G and head l % G and makes its weight.
// The kernels with a lane per key (attention_generic.cu, attention_masked.cu) wait for a row's pieces one after the other: 15 to 20 us for 32 keys,
// whatever else runs.  A float32 Qwen3-4B-size layer's decoded tokens, microseconds there / here: one of 78 keys 44 / 6; five of 20 to 3,069 keys 286 / 24;
// with slopes, one of 901 keys 169 / 11.
#include "attention_decode_f32.cuh"
#include <math.h>

using namespace mi;

namespace {

constexpr int WARPS = 8, NK = 8;                                // warps of a block, keys of a warp's step

template <int N> __device__ __forceinline__ void load_n(const float* p, float (&v)[N]) {
    if constexpr (N == 4) load16(p, v);
    else load2(p, v[0], v[1]);
}

// G query heads of a key head, HG of them at a time (HG NK sums, at most 32)
template <int D, int G, bool PLAIN>
__global__ void __launch_bounds__(32 * WARPS) decode_f32_kernel(const DecodeF32 a) {
    constexpr int R = D / 32, HG = G < 4 ? G : 4, NV = HG * NK, TURNS = G / HG;
    __shared__ float acc_s[WARPS][G][D], m_s[WARPS][G], l_s[WARPS][G];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int seg = a.decode_segs[blockIdx.x], kvh = blockIdx.y, S = gridDim.z, s = blockIdx.z;
    const int tok = a.seg_q_start[seg], len = a.seg_kv_len[seg], p = len - 1;
    // a request's visible keys (the kept ones first, then the range from lo0) in S pieces of whole 32-key chunks
    const int lo0 = max(a.block > 0 ? p / a.block * a.block : 0, a.window > 0 ? p - a.window + 1 : 0);
    const int kept = min(a.keep, lo0), seen = kept + len - lo0, shift = lo0 - kept;
    const int piece = ((seen + S - 1) / S + 31) / 32 * 32, first = s * piece, last = min(first + piece, seen);
    const int* table_row = a.block_table + (size_t)(a.table_rows ? a.table_rows[seg] : seg) * a.table_stride;
    float q[G][R], acc[G][R], m[TURNS], l[TURNS];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        load_n<R>(a.q + (size_t)tok * a.q_stride + (size_t)(kvh * G + g) * D + R * lane, q[g]);
#pragma unroll
        for (int r = 0; r < R; ++r) { q[g][r] *= a.scale; acc[g][r] = 0.f; }
    }
#pragma unroll
    for (int t = 0; t < TURNS; ++t) { m[t] = -INFINITY; l[t] = 0.f; }
    const int my_key = lane % NV / HG, my_head = lane % HG;
    for (int base = first + warp * NK; base < last; base += WARPS * NK) {
        long long off = 0;
        if (lane < NK && base + lane < last) {
            const int idx = base + lane, j = idx < kept ? idx : idx + shift;
            off = ((long long)(table_row[j / a.ps] * a.KV + kvh) * a.ps + j % a.ps) * D;
        }
        float k[NK][R], v[NK][R];
#pragma unroll
        for (int i = 0; i < NK; ++i) {
            const long long o = __shfl_sync(0xffffffffu, off, i) + R * lane;
#pragma unroll
            for (int r = 0; r < R; ++r) k[i][r] = v[i][r] = 0.f;
            if (base + i < last) { load_n<R>(a.k_cache + o, k[i]); load_n<R>(a.v_cache + o, v[i]); }
        }
        const int idx = base + my_key, dist = p - (idx < kept ? idx : idx + shift);
#pragma unroll
        for (int t = 0; t < TURNS; ++t) {
            float y[NV];
#pragma unroll
            for (int i = 0; i < NK; ++i)
#pragma unroll
                for (int g = 0; g < HG; ++g) {
                    float d = q[t * HG + g][0] * k[i][0];
#pragma unroll
                    for (int r = 1; r < R; ++r) d = fmaf(q[t * HG + g][r], k[i][r], d);
                    y[i * HG + g] = d;
                }
            float score = sum_spread<NV>(y, lane);
            if (!PLAIN) {
                const int h = kvh * G + t * HG + my_head;
                if (a.bias) score += a.bias[(size_t)max(0, min(dist, a.bias_last)) * a.H + h];
                if (a.slopes) score -= a.slopes[h] * (float)dist;
                if (a.cap > 0.f) score = a.cap * tanhf(score / a.cap);
            }
            if (idx >= last) score = -INFINITY;
            float mx = score;
#pragma unroll
            for (int w = HG; w < NV; w <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float m_new = fmaxf(m[t], mx), z = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = expf(m[t] - z), weight = idx < last ? expf(score - z) : 0.f;
            float sum = weight;
#pragma unroll
            for (int w = HG; w < NV; w <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[t] = l[t] * alpha + sum;
            m[t] = m_new;
            if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
                for (int g = 0; g < HG; ++g) {
                    const float f = __shfl_sync(0xffffffffu, alpha, g);
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[t * HG + g][r] *= f;
                }
            }
#pragma unroll
            for (int i = 0; i < NK; ++i)
#pragma unroll
                for (int g = 0; g < HG; ++g) {
                    const float f = __shfl_sync(0xffffffffu, weight, i * HG + g);
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[t * HG + g][r] = fmaf(f, v[i][r], acc[t * HG + g][r]);
                }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int r = 0; r < R; ++r) acc_s[warp][g][R * lane + r] = acc[g][r];
#pragma unroll
    for (int t = 0; t < TURNS; ++t)
        if (lane < HG) { m_s[warp][t * HG + lane] = m[t]; l_s[warp][t * HG + lane] = l[t]; }
    __syncthreads();
    for (int id = threadIdx.x; id < G * D; id += 32 * WARPS) {
        const int g = id / D, d = id % D, h = kvh * G + g;
        const bool own_sink = !PLAIN && a.sink && S == 1;       // with several pieces the merge adds the sink's term
        const float sink = own_sink ? (a.sink_values ? a.sink_values[h] : 0.f) : -INFINITY;
        float mx = sink;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) mx = fmaxf(mx, m_s[w][g]);
        const float z = mx == -INFINITY ? 0.f : mx;
        float den = own_sink ? expf(sink - z) : 0.f, num = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = expf(m_s[w][g] - z);
            den = fmaf(f, l_s[w][g], den);
            num = fmaf(f, acc_s[w][g][d], num);
        }
        const float o = den > 0.f ? num / den : den == 0.f ? 0.f : num / den;       // an empty piece: output 0, lse -inf; NaN stays NaN
        if (S == 1) {
            const float gate = PLAIN || !a.gate ? 0.f : a.gate[(size_t)tok * a.gate_stride + (size_t)h * D + d];
            a.out[((size_t)tok * a.H + h) * D + d] = PLAIN || !a.gate ? o : o / (1.f + expf(-gate));
        } else {
            const size_t at = ((size_t)blockIdx.x * a.H + h) * S + s;
            a.o_part[at * D + d] = o;
            if (d == 0) a.lse_part[at] = den == 0.f ? -INFINITY : mx + logf(den);
        }
    }
}

template <int D, int G>
int launch(const DecodeF32& a, cudaStream_t stream) {
    const bool plain = a.block <= 0 && !a.sink && !a.bias && !a.slopes && a.cap <= 0.f && a.keep <= 0 && !a.gate;
    const dim3 grid(a.num_decode, a.KV, a.splits);
    if (plain) decode_f32_kernel<D, G, true><<<grid, 32 * WARPS, 0, stream>>>(a);
    else decode_f32_kernel<D, G, false><<<grid, 32 * WARPS, 0, stream>>>(a);
    return (int)cudaGetLastError();
}
template <int D>
int launch(const DecodeF32& a, cudaStream_t stream) {
    switch (a.H / a.KV) {
        case 1: return launch<D, 1>(a, stream);
        case 2: return launch<D, 2>(a, stream);
        case 4: return launch<D, 4>(a, stream);
        default: return launch<D, 8>(a, stream);
    }
}

}  // namespace

namespace mi {

bool takes_decode_f32(const DecodeF32& a) {
    const int g = a.KV > 0 && a.H % a.KV == 0 ? a.H / a.KV : 0;
    return (a.D == 64 || a.D == 128) && (g == 1 || g == 2 || g == 4 || g == 8) && a.q_stride % 4 == 0 && a.KV <= 65535 && a.splits <= 65535 &&
           ((uintptr_t)a.q | (uintptr_t)a.k_cache | (uintptr_t)a.v_cache) % 16 == 0;
}

int decode_f32(const DecodeF32& a, cudaStream_t stream) { return a.D == 128 ? launch<128>(a, stream) : launch<64>(a, stream); }

}  // namespace mi
