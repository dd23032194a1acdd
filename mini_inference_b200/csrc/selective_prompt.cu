// Selective state-space scan for steps that bring prompt portions: per channel c and state n, token by token,
//     S[c, n] <- exp(step_c A[c, n]) S[c, n] + step_c x_c B_n;   y_c = sum_n S[c, n] C_n + D_c x_c;   out = y * silu(z),
// step = softplus(dt + dt_b).  All float32; the slot's first I N floats are S.
//
// Instruction issue bounds it: per token, channel and state one exponential and four more operations, 134 M of each for 2,048 tokens x
// 4,096 channels x 16 states.  Only the update itself is a chain from token to token.  Eight lanes share a channel and hold
// two states each in one packed pair (N = 16), so 4,096 channels are 1,024 warps, two per scheduler; exponentials run on the
// FMA pipe, two at a time.  A block is 32 channels: eight warps walk the tokens, eight more make the next chunk of 32 tokens ready (steps, inputs, B, C to
// shared memory) and finish the previous one (skip term, gate, store), so neither softplus nor a load is waited for; one barrier a chunk.
// Eight tokens' partial sums are added up over the eight lanes together (seven shuffles instead of 24).  2,048 tokens: 490 -> 148 us.  The kernel in
// which all warps do everything in turn (recurrent.cu) stays for decode steps, where there is one token a request, for other N, and for
// float32 runs: it takes every step, so a request's bits there depend on nothing but its own tokens.
#include "common.cuh"
#include <math.h>
#include <type_traits>

using namespace mi;

namespace {

constexpr int TC = 32, CB = 32, HELPERS = 256;

// e^(step A) of two states at once.  hi + lo is A log2(e) to twice float32's bits, so the rounded product of step and A enters nowhere:
// n = round(step hi), f = step hi - n + step lo, e^(step A) = 2^n 2^f, 2^f a polynomial of degree 6 fitted to (2^f - 1) / f on |f| <= 1/2
// (weighted minimax, 2e-9).  Largest and mean error relative to e^(step A) of the exact product: 9.5e-8 and 2.3e-8 for step A down to -86,
// falling with f towards 1, where a decay acts hundreds of times in a row (expf(step * A): 1.4e-7 and 3.2e-8 even where the product is
// exact, up to 4e-6 at -86 where it is not).  Below 2^-125 the exponent stays there: about 2e-38 instead of less.
// Takes -1000 <= A <= 0 and 0 <= step <= 1e6 (f stays small where n is past the integers that float32 holds): other numbers go to expf.
__device__ __forceinline__ float2 decay2(float step, float2 hi, float2 lo) {
    const float2 st = make_float2(step, step), big = make_float2(12582912.f, 12582912.f);        // 1.5 * 2^23: the sum's low bits are the rounded integer
    const float2 t = __ffma2_rn(st, hi, big);
    const float2 f = __ffma2_rn(st, lo, __ffma2_rn(st, hi, __ffma2_rn(t, make_float2(-1.f, -1.f), big)));
    float2 p = make_float2(1.5476350e-4f, 1.5476350e-4f);
    p = __ffma2_rn(p, f, make_float2(1.3400323e-3f, 1.3400323e-3f));
    p = __ffma2_rn(p, f, make_float2(9.6180039e-3f, 9.6180039e-3f));
    p = __ffma2_rn(p, f, make_float2(5.5503275e-2f, 5.5503275e-2f));
    p = __ffma2_rn(p, f, make_float2(0.24022651f, 0.24022651f));
    p = __ffma2_rn(p, f, make_float2(0.69314718f, 0.69314718f));
    p = __ffma2_rn(p, f, make_float2(1.f, 1.f));
    const float ex = fmaxf(t.x, 12582912.f - 125.f), ey = fmaxf(t.y, 12582912.f - 125.f);
    return make_float2(__int_as_float(__float_as_int(p.x) + (__float_as_int(ex) << 23)), __int_as_float(__float_as_int(p.y) + (__float_as_int(ey) << 23)));
}
constexpr float LEAST_A = -1000.f, MOST_STEP = 1e6f;

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }

// grid (entries, ceil(I / 32)); L lanes of NS states each, N = L NS
template <int L, int NS>
__global__ void __launch_bounds__(CB * L + HELPERS, 1) selective_prompt_kernel(
    const __nv_bfloat16* __restrict__ x, const float* __restrict__ dt, const float* __restrict__ dt_b, const float* __restrict__ A,
    const __nv_bfloat16* __restrict__ B, int ldb, const __nv_bfloat16* __restrict__ Cm, int ldc, const float* __restrict__ Dv, const __nv_bfloat16* __restrict__ z, int ldz,
    float* __restrict__ state, long long state_stride, __nv_bfloat16* __restrict__ out, const int* __restrict__ seg_q_start,
    const int* __restrict__ seg_slot, int I) {
    constexpr int N = L * NS;
    __shared__ __align__(16) float Bs[2][TC][N], Cs[2][TC][N], ys[2][TC][CB];
    __shared__ __align__(16) float2 in[2][TC][CB];                  // step, step * x
    const int seg = blockIdx.x, qs = seg_q_start[seg], n = seg_q_start[seg + 1] - qs, c0 = blockIdx.y * CB;
    const int chunks = (n + TC - 1) / TC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= L) {
        // ---------------- helpers: a warp takes 32 channels of a token; what an iteration works on was requested an iteration earlier
        const int ht = threadIdx.x - CB * L, hw = ht >> 5, cc = c0 + lane;
        const bool live = cc < I;
        const float bias = live ? dt_b[cc] : 0.f, skip = live ? Dv[cc] : 0.f;
        constexpr int HW = HELPERS / 32, R = TC / HW, RB = (TC * N + HELPERS - 1) / HELPERS;
        float rs[R];
        __nv_bfloat16 rx[R], rB[RB], rC[RB], fx[R], fz[R];
        auto request = [&](int k) {                                 // chunk k for making ready, chunk k - 2 for finishing
            const int ta = k * TC, tb = ta - 2 * TC;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int tt = hw + HW * r;
                if (live && ta + tt < n) {
                    rs[r] = dt[(size_t)(qs + ta + tt) * I + cc];
                    rx[r] = x[(size_t)(qs + ta + tt) * I + cc];
                }
                if (live && tb >= 0 && tb + tt < n) {
                    fx[r] = x[(size_t)(qs + tb + tt) * I + cc];
                    fz[r] = z[(size_t)(qs + tb + tt) * ldz + cc];
                }
            }
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const int i = ht + HELPERS * r, tt = i / N, nn = i % N;
                if (tt < TC && ta + tt < n) {
                    rB[r] = B[(size_t)(qs + ta + tt) * ldb + nn];
                    rC[r] = Cm[(size_t)(qs + ta + tt) * ldc + nn];
                }
            }
        };
        request(0);
        int unusual = 0;                                            // a step of the chunk made ready last is none that decay2 takes
        for (int k = -1; k <= chunks; ++k) {                        // makes chunk k + 1 ready, finishes chunk k - 1
            if (k >= 0) __syncthreads_or(unusual);
            unusual = 0;
            const int ta = (k + 1) * TC, tb = (k - 1) * TC, b = (k + 1) & 1;        // chunks k - 1 and k + 1 use the same buffers
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int tt = hw + HW * r;
                if (live && tb >= 0 && tb + tt < n) {
                    const float xv = to_f32(fx[r]), zv = to_f32(fz[r]);
                    out[(size_t)(qs + tb + tt) * I + cc] = __float2bfloat16_rn((ys[b][tt][lane] + skip * xv) * silu(zv));
                }
            }
            if (ta < n) {
#pragma unroll
                for (int r = 0; r < R; ++r) {                       // tokens behind the entry's last: a step of 0 changes no state
                    const int tt = hw + HW * r;
                    float2 v = make_float2(0.f, 0.f);
                    if (live && ta + tt < n) {
                        const float d = rs[r] + bias;
                        v.x = d > 20.f ? d : log1pf(expf(d));
                        if (!(v.x <= MOST_STEP)) unusual = 1;
                        v.y = v.x * to_f32(rx[r]);
                    }
                    in[b][tt][lane] = v;
                }
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const int i = ht + HELPERS * r, tt = i / N, nn = i % N;
                    if (tt < TC) {
                        const bool ok = ta + tt < n;
                        Bs[b][tt][nn] = ok ? to_f32(rB[r]) : 0.f;
                        Cs[b][tt][nn] = ok ? to_f32(rC[r]) : 0.f;
                    }
                }
            }
            request(k + 2);
        }
        return;
    }
    // ---------------- the scan: lane l of L holds the states NS l .. NS l + NS - 1
    constexpr int CW = 32 / L;                                      // channels of a warp
    const int l = lane % L, cl = warp * CW + lane / L, c = c0 + cl;
    const bool live = c < I;
    float* S = state + (long long)seg_slot[seg] * state_stride + (size_t)(live ? c : 0) * N + l * NS;
    const float* ar = A + (size_t)(live ? c : 0) * N + l * NS;
    float2 s[NS / 2], hi[NS / 2], lo[NS / 2];
    bool usual = true;
#pragma unroll
    for (int g = 0; g < NS / 2; ++g) {
        s[g] = hi[g] = lo[g] = make_float2(0.f, 0.f);
        if (live) {
            constexpr float H = 1.44269504f, R = 1.92596299e-8f;    // log2(e) = H + R
            s[g] = make_float2(S[2 * g], S[2 * g + 1]);
            const float2 a = make_float2(ar[2 * g], ar[2 * g + 1]);
            hi[g] = make_float2(a.x * H, a.y * H);
            lo[g] = make_float2(fmaf(a.x, R, fmaf(a.x, H, -hi[g].x)), fmaf(a.y, R, fmaf(a.y, H, -hi[g].y)));
            usual = usual && a.x >= LEAST_A && a.x <= 0.f && a.y >= LEAST_A && a.y <= 0.f;
        }
    }
    usual = __all_sync(0xffffffffu, usual);
    for (int k = 0; k <= chunks; ++k) {
        const bool fast = !__syncthreads_or(0) && usual;
        if (k == chunks) break;                                     // the helpers finish the last chunk
        const int b = k & 1;
        auto walk = [&](auto usual_numbers) {                       // one loop body each: a branch between decays and chain would keep them from overlapping
#pragma unroll 1
            for (int t0 = 0; t0 < TC; t0 += L) {
                float y[L];
                float2 decay[L][NS / 2];                            // not part of the chain from token to token: made side by side
#pragma unroll
                for (int e = 0; e < L; ++e) {
                    const float step = in[b][t0 + e][cl].x;
                    const bool behind = k * TC + t0 + e >= n;       // a token behind the entry's last: no decay, whatever A is
#pragma unroll
                    for (int g = 0; g < NS / 2; ++g) {
                        if (decltype(usual_numbers)::value) decay[e][g] = decay2(step, hi[g], lo[g]);
                        else decay[e][g] = behind ? make_float2(1.f, 1.f) : make_float2(expf(step * ar[2 * g]), expf(step * ar[2 * g + 1]));
                    }
                }
#pragma unroll
                for (int e = 0; e < L; ++e) {
                    const float sx = in[b][t0 + e][cl].y;
                    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                    for (int g = 0; g < NS / 2; ++g) {
                        const float2 bv = *reinterpret_cast<const float2*>(&Bs[b][t0 + e][l * NS + 2 * g]);
                        const float2 cv = *reinterpret_cast<const float2*>(&Cs[b][t0 + e][l * NS + 2 * g]);
                        s[g] = __ffma2_rn(decay[e][g], s[g], __fmul2_rn(make_float2(sx, sx), bv));
                        sum = __ffma2_rn(s[g], cv, sum);
                    }
                    y[e] = sum.x + sum.y;
                }
                // L sums over L lanes together: half of what is left changes hands at every step, lane l ends with token t0 + l
#pragma unroll
                for (int w = 1; w < L; w <<= 1)
#pragma unroll
                    for (int e = 0; e < L; e += 2 * w) {
                        const float got = __shfl_xor_sync(0xffffffffu, l & w ? y[e] : y[e + w], w);
                        y[e] = (l & w ? y[e + w] : y[e]) + got;
                    }
                ys[b][t0 + l][cl] = y[0];
            }
        };
        if (fast) walk(std::true_type{}); else walk(std::false_type{});
    }
    if (live) {
#pragma unroll
        for (int g = 0; g < NS / 2; ++g) { S[2 * g] = s[g].x; S[2 * g + 1] = s[g].y; }
    }
}

}  // namespace

// x [T, I] and out [T, I] contiguous bfloat16; dt float32 [T, I] (before bias and softplus); B, C, z: strided bfloat16 views; A float32
// [I, N], N one of 8, 16, 32.
MI_EXPORT int mi_selective_prompt(const void* x, const float* dt, const float* dt_b, const float* A, const void* B, int ldb, const void* C, int ldc,
                                  const float* Dv, const void* z, int ldz, float* state, long long state_stride, void* out,
                                  const int* seg_q_start, const int* seg_slot, int num_segs, int I, int N, cudaStream_t stream) {
    if (num_segs == 0 || I == 0) return 0;
    const dim3 grid(num_segs, (I + CB - 1) / CB);
#define GO(L, NS) selective_prompt_kernel<L, NS><<<grid, CB * L + HELPERS, 0, stream>>>((const __nv_bfloat16*)x, dt, dt_b, A, (const __nv_bfloat16*)B, ldb, \
        (const __nv_bfloat16*)C, ldc, Dv, (const __nv_bfloat16*)z, ldz, state, state_stride, (__nv_bfloat16*)out, seg_q_start, seg_slot, I)
    if (N == 16) GO(8, 2); else if (N == 8) GO(4, 2); else if (N == 32) GO(8, 4); else return -2;
#undef GO
    return (int)cudaGetLastError();
}
