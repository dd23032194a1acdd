// One token per request for the matrix-state recurrences of recurrent.cu (decode steps), in float32:
//   delta       S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//   constant    S <- d S + k v^T;  o = S^T q     (q, k, v the silu of the rows as projected)
// The state's bytes bound it: 64 requests x 16 heads of 128 x 128 read and write 134 MB (20 us).  A block owns one (request, head); its 256
// threads hold the whole state in registers, four neighbouring columns of every 8th (16th) row each, so that all of a block's loads, whole
// rows of 16-byte pieces, are in flight at once and nothing is staged; the two sums over rows go through shared memory.  A token's numbers
// are requested behind the state.  47 -> 25 us (delta), 46 -> 24 us (constant, with the silu that was a kernel before) against the scan that
// stages tokens and keeps 32 columns a block; that one stays for other sizes.
#include "common.cuh"
#include <math.h>

using namespace mi;

namespace {

constexpr int THREADS = 256;
__device__ __forceinline__ float silu(float x) { return x / (1.f + expf(-x)); }

struct StepSource {             // where a token's numbers are: q, k (+ kv head * D), g (+ head * D), v (+ head * V), beta (+ head) in rows of ld entries
    int ld, q, k, v, g, beta;
};

// grid (heads, requests)
template <typename T, bool DELTA, int D, int V>
__global__ void __launch_bounds__(THREADS) state_step_kernel(const T* __restrict__ in, const StepSource L, const float* __restrict__ decay,
                                                             float* __restrict__ state, long long state_stride, float* __restrict__ out,
                                                             const int* __restrict__ seg_q_start, const int* __restrict__ seg_slot, int H, int KV) {
    constexpr int TPR = V / 4, RPP = THREADS / TPR, R = D / RPP;       // threads of a row, rows of a pass, rows a thread holds
    __shared__ __align__(16) float qs[D], ks[D], gs[D], vs[V], part[RPP][V];
    const int h = blockIdx.x, seg = blockIdx.y, tid = threadIdx.x, c = tid % TPR * 4, r0 = tid / TPR;
    float* S = state + (long long)seg_slot[seg] * state_stride + (long long)h * D * V + c;
    float4 s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) s[i] = *reinterpret_cast<const float4*>(S + (size_t)(r0 + RPP * i) * V);
    const int tok = seg_q_start[seg];
    const T* row = in + (size_t)tok * L.ld;
    const int kvh = h / (H / KV);
    for (int i = tid; i < D; i += THREADS) {
        const float q = to_f32(row[L.q + kvh * D + i]), k = to_f32(row[L.k + kvh * D + i]);
        qs[i] = DELTA ? q : silu(q);
        ks[i] = DELTA ? k : silu(k);
        if (DELTA) gs[i] = to_f32(row[L.g + h * D + i]);
    }
    for (int i = tid; i < V; i += THREADS) { const float v = to_f32(row[L.v + h * V + i]); vs[i] = DELTA ? v : silu(v); }
    const float beta = DELTA ? to_f32(row[L.beta + h]) : 0.f, d1 = DELTA ? 0.f : decay[h];
    __syncthreads();
    float4 u = *reinterpret_cast<const float4*>(vs + c);
    if (DELTA) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float g = gs[r0 + RPP * i], k = ks[r0 + RPP * i];
            s[i].x *= g; s[i].y *= g; s[i].z *= g; s[i].w *= g;
            a.x = fmaf(s[i].x, k, a.x); a.y = fmaf(s[i].y, k, a.y); a.z = fmaf(s[i].z, k, a.z); a.w = fmaf(s[i].w, k, a.w);
        }
        *reinterpret_cast<float4*>(&part[r0][c]) = a;
        __syncthreads();
        float4 dot = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < RPP; ++i) {
            const float4 p = *reinterpret_cast<const float4*>(&part[i][c]);
            dot.x += p.x; dot.y += p.y; dot.z += p.z; dot.w += p.w;
        }
        u = make_float4(beta * (u.x - dot.x), beta * (u.y - dot.y), beta * (u.z - dot.z), beta * (u.w - dot.w));
        __syncthreads();                                               // everyone has read the sums
    }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const float k = ks[r0 + RPP * i], q = qs[r0 + RPP * i];
        if (DELTA) {
            s[i].x = fmaf(k, u.x, s[i].x); s[i].y = fmaf(k, u.y, s[i].y); s[i].z = fmaf(k, u.z, s[i].z); s[i].w = fmaf(k, u.w, s[i].w);
        } else {
            s[i].x = fmaf(d1, s[i].x, k * u.x); s[i].y = fmaf(d1, s[i].y, k * u.y); s[i].z = fmaf(d1, s[i].z, k * u.z); s[i].w = fmaf(d1, s[i].w, k * u.w);
        }
        *reinterpret_cast<float4*>(S + (size_t)(r0 + RPP * i) * V) = s[i];
        o.x = fmaf(s[i].x, q, o.x); o.y = fmaf(s[i].y, q, o.y); o.z = fmaf(s[i].z, q, o.z); o.w = fmaf(s[i].w, q, o.w);
    }
    *reinterpret_cast<float4*>(&part[r0][c]) = o;
    __syncthreads();
    for (int i = tid; i < V; i += THREADS) {
        float acc = 0.f;
#pragma unroll
        for (int p = 0; p < RPP; ++p) acc += part[p][i];
        out[(size_t)tok * H * V + (size_t)h * V + i] = acc;
    }
}

template <typename T, bool DELTA>
int run(const T* in, const StepSource& L, const float* decay, float* state, long long state_stride, float* out, const int* seg_q_start, const int* seg_slot,
        int num_segs, int H, int KV, int D, int V, cudaStream_t stream) {
    if (num_segs == 0) return 0;
    if ((D != 64 && D != 128) || (V != 64 && V != 128) || H % KV || num_segs > 65535 || state_stride % 4 || (uintptr_t)state % 16) return -2;
    const dim3 grid(H, num_segs);
#define GO(DD, VV) state_step_kernel<T, DELTA, DD, VV><<<grid, THREADS, 0, stream>>>(in, L, decay, state, state_stride, out, seg_q_start, seg_slot, H, KV)
    if (D == 128) { if (V == 128) GO(128, 128); else GO(128, 64); }
    else { if (V == 128) GO(64, 128); else GO(64, 64); }
#undef GO
    return (int)cudaGetLastError();
}

}  // namespace

// Every entry brings one token.  prep [T, ld] float32 = q [KV D] | k [KV D] | v [H V] | g [H D] | beta [H]; out float32 [T, H V]
MI_EXPORT int mi_delta_step(const float* prep, int ld, float* state, long long state_stride, float* out, const int* seg_q_start, const int* seg_slot,
                            int num_segs, int H, int KV, int D, int V, cudaStream_t stream) {
    const int channels = 2 * KV * D + H * V;
    return run<float, true>(prep, StepSource{ld, 0, KV * D, 2 * KV * D, channels, channels + H * D}, nullptr, state, state_stride, out, seg_q_start, seg_slot,
                            num_segs, H, KV, D, V, stream);
}

// p [T, ldp] bfloat16 = q | k | v before silu; decay [H]
MI_EXPORT int mi_lightning_step(const void* p, int ldp, const float* decay, float* state, long long state_stride, float* out, const int* seg_q_start,
                                const int* seg_slot, int num_segs, int H, int D, int V, cudaStream_t stream) {
    return run<__nv_bfloat16, false>((const __nv_bfloat16*)p, StepSource{ldp, 0, H * D, 2 * H * D, 0, 0}, decay, state, state_stride, out, seg_q_start, seg_slot,
                                     num_segs, H, H, D, V, stream);
}
