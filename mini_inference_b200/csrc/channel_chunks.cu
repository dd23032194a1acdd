// The delta rule with a decay per head and key channel over prompt portions of bfloat16 runs, 32 tokens at a time on the tensor cores, every
// operand in three bfloat16 parts (split3.cuh: float32 products).  With S_0 before a chunk, G_ij = g_{j+1} .. g_i and G_i = g_0 .. g_i (products of
// decays, row by row, never more than 1), A_ij = beta_i k_i^T G_ij k_j below the diagonal and B_ij = q_i^T G_ij k_j up to it:
//   W = (I + A)^-1 [beta_i G_i k_i],  U_0 = (I + A)^-1 [beta_i v_i]          do not depend on the state
//   U = U_0 - W S_0;      O = [G_i q_i] S_0 + B U;      S = G_31 S_0 + [G_31,j k_j]^T U
//
// chunk_kernel, a block per (chunk, head): W, U_0, B and the decayed queries and keys of all chunks at once.  A warp owns eight tokens, inside which
// every G_ij is a product of its own; between them the decays go by way of the bounds of the eights, so that no factor is above 1 and none is divided by.
// pass_kernel, a block per (entry, head, 16 columns): walks an entry's chunks with S^T [columns x rows] in the registers of four warps, a warp's 32
// rows.  The accumulator of S^T is, two tiles at a time, laid out as the left operand of the next product, so the state never goes through shared
// memory: a warp multiplies its own rows, and the four partial sums of U^T and O^T meet there.  One more warp brings chunks by bulk copies.
//
// mma.sync and not tcgen05: the walk is a chain, and what counts is how many SMs share it.  A tcgen05 product has 128 rows, all columns of a
// head (16 blocks for one prompt), where 16 columns a block make 128.
//
// 16 heads of 128 x 128 on 8 key heads, microseconds by state_octets.cu / here: 2,048 tokens 238 / 162, 1,300 + 517 + 231 249 / 160, 4 x 512 202 / 151,
// 8 x 1,024 680 / 508, 16 x 64 105 / 85, 400 54 / 44, 192 31 / 29.  Of the 162 the first kernel takes 52 (a third of the issue slots: forward
// substitution and the products between eights), the second 110: 2,600 clocks a chunk, 156 products a warp of 8.5 each (the rate of one
// scheduler) and half as much again waiting between the operands' cutting, the products and the partial sums' way around.  Error against 64 bits
// (2-norm, 1,034 tokens): outputs 1.7e-7 there, 1.5e-7 here, states 5.1e-8 and 4.0e-8.
// Measured and left: outputs made by four more warps (as fast: they share the schedulers' product rate and the shared memory), operands cut
// by the first kernel (6 bytes a number instead of 4: as fast, and half as much scratch again), 32 columns by eight warps (64 blocks for one prompt: 227).
//
// Numbers that the parts do not hold are found where U is cut into parts, or when a chunk is made ready: from the first such token on the chunk is
// computed token by token, the tokens before it keep their bits.  These are infinities and NaN, W, Q, K, B and U beyond 2^60, a query or a key whose largest
// magnitude is below 2^-50 (so that B's parts are whole), a token's 16 columns of U that are all below 2^-100.  All else is as exact as float32 sums are
// against the vectors' norms; what decays below 2^-100 of a query, a key or a state may keep fewer bits than it has in float32, and a query times a state
// beyond 2^127 is an infinity also where a chunk's later additions would have taken it back.
// Token by token costs 1.4 us a token and block: 2,048 tokens and 16 heads 164 us, 199 with one small key, 2,800 with an infinity that stays in a state.
#include "split3.cuh"
#include <math.h>
#include <algorithm>

using namespace mi;
using namespace mi::sm100;
using namespace mi::split3;

namespace {

constexpr int C = 32, D = 128, OCT = 8, NOCT = C / OCT, VC = 16;        // tokens of a chunk; rows of a state; columns of four warps
constexpr float LEAST = 0x1p-100f, MOST = 0x1p60f, LEAST_SCORED = 0x1p-50f;

// What chunk_kernel leaves per (chunk, head), float32: W, Q, K and B in the order in which lanes take them as right operands of m16n8k16 (a lane's
// four numbers of a tile side by side); pass_kernel cuts them into parts
constexpr int MATRIX = D * C * 4;
constexpr int W_OFF = 0, Q_OFF = MATRIX, K_OFF = 2 * MATRIX, P_OFF = 3 * MATRIX, DEC_OFF = P_OFF + C * C * 4, ODD_OFF = DEC_OFF + D * 4;
constexpr int U_OFF = ODD_OFF + 16, UPITCH = C + 4;                     // U_0: [column][token] float32, rows apart so that reads of a tile meet few banks twice
__host__ __device__ constexpr int record_bytes(int V) { return U_OFF + V * UPITCH * 4; }

// An entry's chunks lie behind floor(first token / 32) + entry slots: entries never share one.
__host__ __device__ __forceinline__ int first_slot(int qs, int seg) { return qs / C + seg; }

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// the largest magnitude of N numbers as float bits (NaN above all)
template <int N> __device__ __forceinline__ uint32_t largest(const float (&x)[N]) {
    float m = 0.f;
#pragma unroll
    for (int e = 0; e < N; ++e) asm("max.NaN.f32 %0, %0, %1;\n" : "+f"(m) : "f"(fabsf(x[e])));
    return __float_as_uint(m);
}

struct Rows { const float* at; int ld, k, v, g, beta, group; };         // q at 0 (+ key head * D), k (+ key head * D), v (+ head * V), g (+ head * D), beta (+ head)

// ------------------------------------------------------------------ what the state does not enter
constexpr int PITCH = D + 4;
struct ChunkSmem {
    float kd[C][PITCH], qd[C][PITCH], kh[C][PITCH], g[NOCT][D];
    float ab[C][C];                                                     // -beta A below the diagonal, B^T on and above it (four blocks an SM)
    float beta[C];
    int odd;
};

// float index of (k, n) of a right operand: steps of 16 k, tiles of 8 n; the n's 32 numbers of a step side by side, lanes' fours in a row
__device__ __forceinline__ int four(int k, int n, int tiles) { return ((k / 16 * tiles + n / 8) * 32 + n % 8 * 4 + k % 8 / 2) * 4 + (k % 16 / 8) * 2 + (k & 1); }
// 32 tokens' numbers of column n of a right operand whose k are the tokens
__device__ __forceinline__ void store_by_token(float* to, int n, int tiles, const float (&x)[C]) {
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            *reinterpret_cast<float4*>(to + four(16 * ks + 2 * c, n, tiles)) = make_float4(x[16 * ks + 2 * c], x[16 * ks + 2 * c + 1], x[16 * ks + 2 * c + 8], x[16 * ks + 2 * c + 9]);
}
__device__ __forceinline__ void async4(uint32_t dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// grid (slots, heads): 4 warps, a warp eight tokens
__global__ void __launch_bounds__(128, 4) chunk_kernel(const Rows L, unsigned char* __restrict__ work, const int* __restrict__ seg_q_start, int num_segs, int h0, int V) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ChunkSmem& sm = *reinterpret_cast<ChunkSmem*>(smem_raw);
    const int slot = blockIdx.x, h = h0 + blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int lo = 0, hi = num_segs - 1;                                      // the entry whose chunks hold this slot
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (first_slot(seg_q_start[mid], mid) <= slot) lo = mid; else hi = mid - 1;
    }
    const int qs = seg_q_start[lo], t0 = C * (slot - first_slot(qs, lo)), n = seg_q_start[lo + 1] - qs - t0;     // tokens from this chunk on
    if (n <= 0) return;
    const float* first = L.at + (size_t)(qs + t0) * L.ld;
    const int kvh = h / L.group;
    {   // ---- eight tokens a warp, four neighbouring rows a lane
        float4 q4[OCT], k4[OCT], g4[OCT];
#pragma unroll
        for (int i = 0; i < OCT; ++i) {
            const int t = OCT * warp + i;
            const float* row = first + (size_t)t * L.ld;
            q4[i] = k4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            g4[i] = make_float4(1.f, 1.f, 1.f, 1.f);                    // a token behind the last: no decay, no key, beta 0
            if (t < n) {
                q4[i] = *reinterpret_cast<const float4*>(row + kvh * D + 4 * lane);
                k4[i] = *reinterpret_cast<const float4*>(row + L.k + kvh * D + 4 * lane);
                g4[i] = *reinterpret_cast<const float4*>(row + L.g + h * D + 4 * lane);
            }
        }
        if (tid < C) sm.beta[tid] = tid < n ? first[(size_t)tid * L.ld + L.beta + h] : 0.f;
        if (tid == 0) sm.odd = C;
        __syncthreads();
        int tiny = C;                                                   // the warp's first token whose query or key is small but for zeros
#pragma unroll
        for (int i = OCT - 1; i >= 0; --i) {
            const float q[4] = {q4[i].x, q4[i].y, q4[i].z, q4[i].w}, k[4] = {k4[i].x, k4[i].y, k4[i].z, k4[i].w};
            const uint32_t mq = __reduce_max_sync(0xffffffffu, largest(q)), mk = __reduce_max_sync(0xffffffffu, largest(k));
            if (min(mq - 1, mk - 1) < __float_as_uint(LEAST_SCORED) - 1) tiny = OCT * warp + i;
        }
        if (tiny < C && lane == 0) atomicMin(&sm.odd, tiny);
        float y[32], z[32], last[4] = {0.f, 0.f, 0.f, 0.f};             // 28 A_ij at i (i - 1) / 2 + j, 36 B_ij at i (i + 1) / 2 + j
        float G[4] = {1.f, 1.f, 1.f, 1.f}, kh[OCT][4];
#pragma unroll
        for (int e = 0; e < 32; ++e) y[e] = z[e] = 0.f;
#pragma unroll
        for (int i = 0; i < OCT; ++i) {
            const float q[4] = {q4[i].x, q4[i].y, q4[i].z, q4[i].w}, k[4] = {k4[i].x, k4[i].y, k4[i].z, k4[i].w}, g[4] = {g4[i].x, g4[i].y, g4[i].z, g4[i].w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                G[r] *= g[r];
                kh[i][r] = k[r];
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    if (j < i) {
                        kh[j][r] *= g[r];
                        y[i * (i - 1) / 2 + j] = fmaf(k[r], kh[j][r], y[i * (i - 1) / 2 + j]);
                    }
                    const int e = i * (i + 1) / 2 + j;
                    if (e < 32) z[e] = fmaf(q[r], kh[j][r], z[e]);
                    else last[e - 32] = fmaf(q[r], kh[j][r], last[e - 32]);
                }
            }
            *reinterpret_cast<float4*>(&sm.kd[OCT * warp + i][4 * lane]) = make_float4(k[0] * G[0], k[1] * G[1], k[2] * G[2], k[3] * G[3]);
            *reinterpret_cast<float4*>(&sm.qd[OCT * warp + i][4 * lane]) = make_float4(q[0] * G[0], q[1] * G[1], q[2] * G[2], q[3] * G[3]);
        }
#pragma unroll
        for (int i = 0; i < OCT; ++i) *reinterpret_cast<float4*>(&sm.kh[OCT * warp + i][4 * lane]) = make_float4(kh[i][0], kh[i][1], kh[i][2], kh[i][3]);
        *reinterpret_cast<float4*>(&sm.g[warp][4 * lane]) = make_float4(G[0], G[1], G[2], G[3]);
        const float b_sum = sum_spread<32>(z, lane), b_last = sum_spread<4>(last, lane), a_sum = sum_spread<32>(y, lane);
        int i = 0;
        while ((i + 1) * (i + 2) / 2 <= lane) ++i;                      // row of entry `lane` in a lower triangle with its diagonal
        const int j = lane - i * (i + 1) / 2, o = OCT * warp;
        sm.ab[o + j][o + i] = b_sum;
        if (lane < 4) sm.ab[o + 4 + lane][o + 7] = b_last;
        if (lane < 28) sm.ab[o + i + 1][o + j] = -sm.beta[o + i + 1] * a_sum;
    }
    __syncthreads();
    // ---- between eights: six pairs of them, half of the rows at a time; a lane 2 x 4 tokens of both matrices and a quarter of that half
    {
        const int dq = lane >> 3, i0 = (lane & 3) * 2, j0 = (lane >> 2 & 1) * 4;
#pragma unroll 1
        for (int u = warp; u < 12; u += 4) {
            const int pair = u < 6 ? u : u - 6, half = u < 6 ? 0 : 1, a = pair < 1 ? 1 : pair < 3 ? 2 : 3, b = pair - a * (a - 1) / 2;      // (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
            float2 ka[2][4] = {}, qa[2][4] = {};                        // of even and odd rows
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int d = half * 64 + s * 16 + dq * 4;
                float4 e = make_float4(1.f, 1.f, 1.f, 1.f);
                for (int m = b + 1; m < a; ++m) {
                    const float4 t = *reinterpret_cast<const float4*>(&sm.g[m][d]);
                    e.x *= t.x; e.y *= t.y; e.z *= t.z; e.w *= t.w;
                }
                float4 k[2], q[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    k[i] = *reinterpret_cast<const float4*>(&sm.kd[OCT * a + i0 + i][d]);
                    q[i] = *reinterpret_cast<const float4*>(&sm.qd[OCT * a + i0 + i][d]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 t = *reinterpret_cast<const float4*>(&sm.kh[OCT * b + j0 + j][d]);
                    const float2 x0 = __fmul2_rn(make_float2(t.x, t.y), make_float2(e.x, e.y)), x1 = __fmul2_rn(make_float2(t.z, t.w), make_float2(e.z, e.w));
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        ka[i][j] = __ffma2_rn(make_float2(k[i].x, k[i].y), x0, ka[i][j]);
                        qa[i][j] = __ffma2_rn(make_float2(q[i].x, q[i].y), x0, qa[i][j]);
                        ka[i][j] = __ffma2_rn(make_float2(k[i].z, k[i].w), x1, ka[i][j]);
                        qa[i][j] = __ffma2_rn(make_float2(q[i].z, q[i].w), x1, qa[i][j]);
                    }
                }
            }
            float sums[16];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { sums[4 * i + j] = ka[i][j].x + ka[i][j].y; sums[8 + 4 * i + j] = qa[i][j].x + qa[i][j].y; }
            float some[4];                                              // lanes of quarter dq end with sums 4 dq ..
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float got = __shfl_xor_sync(0xffffffffu, dq & 2 ? sums[e] : sums[e + 8], 16);
                sums[e] = (dq & 2 ? sums[e + 8] : sums[e]) + got;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float got = __shfl_xor_sync(0xffffffffu, dq & 1 ? sums[e] : sums[e + 4], 8);
                some[e] = (dq & 1 ? sums[e + 4] : sums[e]) + got;
            }
            const int row = OCT * a + i0 + (dq & 1), col = OCT * b + j0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float* to = dq & 2 ? &sm.ab[col + j][row] : &sm.ab[row][col + j];
                const float v = dq & 2 ? some[j] : -sm.beta[row] * some[j];
                *to = half ? *to + v : v;
            }
            __syncthreads();                                            // a pair's second half comes a turn or two after its first
        }
    }
    unsigned char* rec = work + ((size_t)blockIdx.y * gridDim.x + slot) * record_bytes(V);
    // ---- a thread a row of the state (a column of kh, qd, kd) and a column of the values, which take the place of kh.  (Loops: as one long run of
    // 5,900 instructions this kernel waited for them.)
    auto fetch_values = [&](int v) {
#pragma unroll 8
        for (int i = 0; i < C; ++i)
            if (i < n && v < V) async4(smem_u32(&sm.kh[i][tid]), first + (size_t)i * L.ld + L.v + h * V + v);
            else sm.kh[i][tid] = 0.f;
    };
    float g[NOCT];
#pragma unroll
    for (int o = 0; o < NOCT; ++o) g[o] = sm.g[o][tid];
    auto put = [&](int what, float (&f)[NOCT]) {                        // 0: K, 1: Q, 2: W; a factor per eight tokens
        const float* from = what == 0 ? &sm.kh[0][tid] : what == 1 ? &sm.qd[0][tid] : &sm.kd[0][tid];
        float x[C];
#pragma unroll
        for (int i = 0; i < C; ++i) x[i] = from[i * PITCH] * f[i / OCT];
        const uint32_t mx = largest(x);
        if (!(mx <= __float_as_uint(MOST))) {
            int odd = C - 1;                                            // K goes into the state alone (also what a later decay did to it)
            if (what) for (int i = C - 1; i >= 0; --i) if (!(fabsf(from[i * PITCH] * (i < 8 ? f[0] : i < 16 ? f[1] : i < 24 ? f[2] : f[3])) <= MOST)) odd = i;
            atomicMin(&sm.odd, odd);
        }
        if (what == 0) {
            store_by_token(reinterpret_cast<float*>(rec + K_OFF) + (tid / 32) * 1024, tid % 32, 4, x);
        } else {                                                        // k is the row, n the token
            float* to = reinterpret_cast<float*>(rec + (what == 1 ? Q_OFF : W_OFF));
#pragma unroll
            for (int i = 0; i < C; ++i) to[four(tid, i, 4)] = x[i];
        }
    };
    float f[NOCT];
#pragma unroll 1
    for (int what = 0; what < 3; ++what) {
        if (what == 0) {                                                // decays of the eights behind each
            f[3] = 1.f; f[2] = g[3]; f[1] = g[2] * f[2]; f[0] = g[1] * f[1];
        } else if (what == 1) {                                         // ... before each
            f[0] = 1.f; f[1] = g[0]; f[2] = f[1] * g[1]; f[3] = f[2] * g[2];
            reinterpret_cast<float*>(rec + DEC_OFF)[tid] = f[3] * g[3];
            fetch_values(tid);
        } else {                                                        // W and U_0 by forward substitution, eight tokens after eight, in place
            async_wait();
            for (int v = tid; v < (V + 127) / 128 * 128; v += 128) {
                const bool keys = v < 128;
                if (!keys) { fetch_values(v); async_wait(); }
#pragma unroll 1
                for (int o = 0; o < NOCT; ++o) {
                    float x[OCT], u[OCT];
                    const float fo = o == 0 ? f[0] : o == 1 ? f[1] : o == 2 ? f[2] : f[3];
#pragma unroll
                    for (int i = 0; i < OCT; ++i) {
                        const float beta = sm.beta[OCT * o + i];
                        x[i] = beta * (sm.kd[OCT * o + i][tid] * fo);
                        u[i] = beta * sm.kh[OCT * o + i][tid];
                    }
#pragma unroll 1
                    for (int e = 0; e < o; ++e)
#pragma unroll
                        for (int j = 0; j < OCT; j += 4) {
                            float xj[4], uj[4];
#pragma unroll
                            for (int c = 0; c < 4; ++c) { xj[c] = sm.kd[OCT * e + j + c][tid]; uj[c] = sm.kh[OCT * e + j + c][tid]; }
#pragma unroll
                            for (int i = 0; i < OCT; ++i) {
                                const float4 a = *reinterpret_cast<const float4*>(&sm.ab[OCT * o + i][OCT * e + j]);
                                x[i] = fmaf(a.x, xj[0], x[i]); u[i] = fmaf(a.x, uj[0], u[i]);
                                x[i] = fmaf(a.y, xj[1], x[i]); u[i] = fmaf(a.y, uj[1], u[i]);
                                x[i] = fmaf(a.z, xj[2], x[i]); u[i] = fmaf(a.z, uj[2], u[i]);
                                x[i] = fmaf(a.w, xj[3], x[i]); u[i] = fmaf(a.w, uj[3], u[i]);
                            }
                        }
#pragma unroll
                    for (int i = 1; i < OCT; ++i) {
                        float a[OCT];
                        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&sm.ab[OCT * o + i][OCT * o]);
                        if (i > 4) *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&sm.ab[OCT * o + i][OCT * o + 4]);
#pragma unroll
                        for (int j = 0; j < i; ++j) { x[i] = fmaf(a[j], x[j], x[i]); u[i] = fmaf(a[j], u[j], u[i]); }
                    }
#pragma unroll
                    for (int i = 0; i < OCT; ++i) {
                        if (keys) sm.kd[OCT * o + i][tid] = x[i];
                        sm.kh[OCT * o + i][tid] = u[i];
                    }
                    if (v < V) {
                        float4* to = reinterpret_cast<float4*>(rec + U_OFF) + (size_t)v * (UPITCH / 4) + o * (OCT / 4);
                        to[0] = make_float4(u[0], u[1], u[2], u[3]);
                        to[1] = make_float4(u[4], u[5], u[6], u[7]);
                    }
                }
            }
            f[0] = f[1] = f[2] = f[3] = 1.f;
        }
        put(what, f);
    }
    if (tid < C) {                                                      // B's rows
        float x[C];
#pragma unroll
        for (int j = 0; j < C; ++j) x[j] = j <= tid ? sm.ab[j][tid] : 0.f;
        if (!(largest(x) <= __float_as_uint(MOST))) atomicMin(&sm.odd, tid);
        store_by_token(reinterpret_cast<float*>(rec + P_OFF) + (tid / 8) * 256, tid % 8, 1, x);
    }
    __syncthreads();
    if (tid == 0) *reinterpret_cast<int*>(rec + ODD_OFF) = sm.odd;
}

// ------------------------------------------------------------------ the walk over an entry's chunks
constexpr int U_BYTES = VC * UPITCH * 4;
// A chunk in shared memory, in pieces that are refilled when they have been read: W, the flag and U_0 | Q | K, B, the decays
constexpr int P_AT = P_OFF - K_OFF, DEC_AT = DEC_OFF - K_OFF, K_BYTES = ODD_OFF - K_OFF;
// DEEP: three whole chunks as they lie in memory (all pieces on the first one's barriers) and a block an SM.  Else two of the first piece and one of
// the others, which a walk waits for a little (0.2 us a chunk), and two blocks an SM, which use each other's waits.
template <bool DEEP> struct Ring {
    static constexpr int W = DEEP ? 3 : 2, R = DEEP ? 3 : 1;            // chunks of the first piece, of the others
    static constexpr int FLAG_AT = DEEP ? ODD_OFF : MATRIX, U_AT = FLAG_AT + 16, W_BYTES = MATRIX + 16 + U_BYTES;
    static constexpr int W_STEP = (U_AT + U_BYTES + 127) / 128 * 128, R_STEP = DEEP ? W_STEP : 0;
    static constexpr int Q_AT = DEEP ? Q_OFF : W * W_STEP, K_AT = Q_AT + MATRIX;
    static constexpr int BYTES = DEEP ? W * W_STEP : (K_AT + K_BYTES + 127) / 128 * 128, BARS = W + 2 * R;
};
struct Exchange {
    float4 u_part[4][4][32];                                            // W S of a warp's rows: [warp][tile of 8 tokens][lane]; token by token: the state's columns
    float4 o_part[2][4][4][32];                                         // Q S, two chunks in turn
    float red[256];
    uint2 u[PARTS][4][32];                                              // the parts of U^T as a left operand: [part][tile][lane]
    int odd[2];
    uint64_t bars[2 * 9];
};
template <bool DEEP> constexpr int PASS_SMEM = Ring<DEEP>::BYTES + sizeof(Exchange);

// The chunk's tokens one after the other for 16 columns, by 128 threads: a thread has 16 rows of a column, the state (before the chunk) in st [D][VC].
__device__ __noinline__ void by_token(float* st, float* red, const Rows L, const float* first, int n, int from, int h, int kvh, int V, int v0, float* out, int H,
                                      int t) {
    const int c = t & 15, r0 = (t >> 4) * 16;
    auto meet = [] { asm volatile("bar.sync 1, 128;\n" ::: "memory"); };
    for (int i = 0; i < n; ++i) {
        const float* row = first + (size_t)i * L.ld;
        float y = 0.f;
        for (int r = r0; r < r0 + 16; ++r) {
            const float s = st[r * VC + c] * row[L.g + h * D + r];
            st[r * VC + c] = s;
            y = fmaf(s, row[L.k + kvh * D + r], y);
        }
        red[t] = y;
        meet();
        y = 0.f;
        for (int e = 0; e < 8; ++e) y += red[16 * e + c];
        const float u = row[L.beta + h] * (row[L.v + h * V + v0 + c] - y);
        y = 0.f;
        for (int r = r0; r < r0 + 16; ++r) {
            const float s = fmaf(row[L.k + kvh * D + r], u, st[r * VC + c]);
            st[r * VC + c] = s;
            y = fmaf(s, row[kvh * D + r], y);
        }
        red[128 + t] = y;
        meet();
        if (t < 16 && i >= from) {
            y = 0.f;
            for (int e = 0; e < 8; ++e) y += red[128 + 16 * e + c];
            out[(size_t)i * H * V + c] = y;
        }
    }
}

// grid (V / 16, heads, entries); four warps and one that copies.  Products are laid where a warp would wait for the others: those of O while the
// sums of U go round.  The outputs of a chunk are added up when the sums of the next one have met.
template <bool DEEP>
__global__ void __launch_bounds__(160, DEEP ? 1 : 2) pass_kernel(const unsigned char* __restrict__ work, int slots, const Rows L, float* __restrict__ state,
                                                      long long state_stride, float* __restrict__ out, const int* __restrict__ seg_q_start,
                                                      const int* __restrict__ seg_slot, int H, int h0, int V, int* __restrict__ error_word) {
    using G = Ring<DEEP>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Exchange& ex = *reinterpret_cast<Exchange*>(smem + G::BYTES);
    const uint32_t full = smem_u32(ex.bars), empty = full + 8 * G::BARS, base = smem_u32(smem);
    const int seg = blockIdx.z, h = h0 + blockIdx.y, v0 = blockIdx.x * VC;
    const int qs = seg_q_start[seg], n = seg_q_start[seg + 1] - qs, chunks = (n + C - 1) / C;
    if (chunks == 0) return;
    const size_t step = record_bytes(V);
    if (threadIdx.x == 0) {
        for (int s = 0; s < G::BARS; ++s) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 4); }
        mbar_init_fence();
        ex.odd[0] = ex.odd[1] = C;
    }
    __syncthreads();
    if (w == 4) {
        const unsigned char* rec = work + ((size_t)blockIdx.y * slots + first_slot(qs, seg)) * step;
        if (lane == 0)
            for (int k = 0; k < chunks; ++k, rec += step) {
                bool ok = true;
                for (int i = 0; i < (DEEP ? 1 : 3) && ok; ++i) {
                    const int depth = i ? G::R : G::W, slot = k % depth, bar_no = i == 0 ? slot : i == 1 ? G::W + slot : G::W + G::R + slot;
                    const uint32_t bar = full + 8 * bar_no, dst = base + slot * G::W_STEP;
                    if (k >= depth && !mbar_wait(empty + 8 * bar_no, (k / depth - 1) & 1)) { atomicExch(error_word, 91); ok = false; break; }
                    mbar_expect_tx(bar, DEEP ? U_OFF + U_BYTES : i == 0 ? G::W_BYTES : i == 1 ? MATRIX : K_BYTES);
                    if (i == 0) {
                        bulk_load(dst, rec, DEEP ? U_OFF : MATRIX, bar);
                        if (!DEEP) bulk_load(dst + G::FLAG_AT, rec + ODD_OFF, 16, bar);
                        bulk_load(dst + G::U_AT, rec + U_OFF + blockIdx.x * U_BYTES, U_BYTES, bar);
                    } else if (i == 1) {
                        bulk_load(base + G::Q_AT, rec + Q_OFF, MATRIX, bar);
                    } else {
                        bulk_load(base + G::K_AT, rec + K_OFF, K_BYTES, bar);
                    }
                }
                if (!ok) break;
            }
        return;
    }
    const int g = lane >> 2, c2 = 2 * (lane & 3);
    bool alive = true;
    auto await = [&](uint32_t bar, int phase) {                         // a wait that ran out is recorded once; no further ones follow
        if (alive && !mbar_spin(bar, phase & 1)) { alive = false; if (lane == 0) atomicExch(error_word, 92); }
    };
    bool there = false;                                                 // the next chunk was there when this one's sums had met
    auto meet = [] { asm volatile("bar.sync 1, 128;\n" ::: "memory"); };
    auto arrive = [&](uint32_t bar) { __syncwarp(); if (lane == 0) mbar_arrive(bar); };
    using Right = uint32_t[PARTS][4][2];                                // the parts of 16 x 32 numbers as a right operand
    auto fetch_right = [&](Right& b, const unsigned char* at, int ks) { // the warp's rows and 16 rows (W, Q) or tokens (K) of them
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            float4 x = reinterpret_cast<const float4*>(at)[((2 * w + ks) * 4 + t) * 32 + lane];
#pragma unroll
            for (int p = 0; p < PARTS; ++p) { b[p][t][0] = take_part(x.x, x.y); b[p][t][1] = take_part(x.z, x.w); }
        }
    };
    struct Sums { float lead[4][4], small[4][4]; };                     // the leading products apart: the tensor core cuts off where it adds
    auto clear = [&](Sums& x) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) x.lead[t][e] = x.small[t][e] = 0.f;
    };
    auto product = [&](Sums& x, const uint32_t (&a)[PARTS][4], const Right& b) {
#pragma unroll
        for (int p = 0; p < PRODUCTS; ++p)
#pragma unroll
            for (int t = 0; t < 4; ++t) mma16816(p < PRODUCTS - 1 ? x.small[t] : x.lead[t], a[PART_A[p]], b[PART_B[p]][t][0], b[PART_B[p]][t][1]);
    };
    auto put = [&](float4 (&to)[4][32], const Sums& x) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
            to[t][lane] = make_float4(x.lead[t][0] + x.small[t][0], x.lead[t][1] + x.small[t][1], x.lead[t][2] + x.small[t][2], x.lead[t][3] + x.small[t][3]);
    };
    float* S = state + (long long)seg_slot[seg] * state_stride + (long long)h * D * V + v0;
    // S^T: tile nt has rows 32 w + 8 nt + c2, + 1 of columns g (first two) and g + 8
    float s[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[nt][e] = S[(size_t)(32 * w + 8 * nt + c2 + (e & 1)) * V + g + (e >> 1) * 8];
    float own[4];                                                       // U^T B^T of the warp's eight tokens
    int left = 0;                                                       // tokens of the chunk before that are not made one by one
    auto store = [&](int k) {                                           // the outputs of chunk k
        float o[4] = {own[0], own[1], own[2], own[3]};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float4 a = ex.o_part[k & 1][e][w][lane];
            o[0] += a.x; o[1] += a.y; o[2] += a.z; o[3] += a.w;
        }
        float* to = out + (size_t)(qs + k * C) * H * V + (size_t)h * V + v0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int tok = OCT * w + c2 + (e & 1);
            if (tok < left) to[(size_t)tok * H * V + g + (e >> 1) * 8] = o[e];
        }
    };
    for (int k = 0; k < chunks; ++k) {
        const int ws = k % G::W, wr = k / G::W, rs = k % G::R, rr = k / G::R;       // the pieces' slots, and how often those were filled before
        const unsigned char *first = smem + ws * G::W_STEP, *queries = smem + G::Q_AT + rs * G::R_STEP, *keys = queries + MATRIX;
        const int q_bar = 8 * (G::W + rs), k_bar = q_bar + 8 * G::R;
        uint32_t sa[2][PARTS][4];                                       // the accumulators' layout is the left operand's, two tiles at a time
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            float x[2][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) { x[0][e] = s[2 * ks][e]; x[1][e] = s[2 * ks + 1][e]; }
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                sa[ks][p][0] = take_part(x[0][0], x[0][1]);
                sa[ks][p][1] = take_part(x[0][2], x[0][3]);
                sa[ks][p][2] = take_part(x[1][0], x[1][1]);
                sa[ks][p][3] = take_part(x[1][2], x[1][3]);
            }
        }
        if (!there) await(full + 8 * ws, wr);
        Sums q;
        Right b0, b1;
        {
            Sums x;
            clear(x);
            const bool q_there = DEEP || mbar_test(full + q_bar, rr & 1);           // (a wait for what is there takes 170 clocks, an answer that is read later none)
            fetch_right(b0, first, 0);
            fetch_right(b1, first, 1);
            product(x, sa[0], b0);
            if (!q_there) await(full + q_bar, rr);
            fetch_right(b0, queries, 0);
            product(x, sa[1], b1);
            put(ex.u_part[w], x);
        }
        clear(q);
        fetch_right(b1, queries, 1);
        const bool k_there = DEEP || mbar_test(full + k_bar, rr & 1);
        product(q, sa[0], b0);
        meet();
        {
            float u[4] = {0.f, 0.f, 0.f, 0.f};                          // the warp's eight tokens: W S over all rows
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 a = ex.u_part[e][w][lane];
                u[0] += a.x; u[1] += a.y; u[2] += a.z; u[3] += a.w;
            }
            const float* u0 = reinterpret_cast<const float*>(first + G::U_AT) + g * UPITCH + OCT * w + c2;
            const float2 ua = *reinterpret_cast<const float2*>(u0), ub = *reinterpret_cast<const float2*>(u0 + 8 * UPITCH);
            u[0] = ua.x - u[0];
            u[1] = ua.y - u[1];
            u[2] = ub.x - u[2];
            u[3] = ub.y - u[3];
            float v[4] = {u[0], u[1], u[2], u[3]};
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                uint2 t;
                t.x = take_part(v[0], v[1]);
                t.y = take_part(v[2], v[3]);
                ex.u[p][w][lane] = t;
            }
            int odd = *reinterpret_cast<const int*>(first + G::FLAG_AT);
            if (!DEEP) arrive(empty + 8 * ws);                          // W, U_0 and the flag have been read
            const uint32_t mx = __reduce_max_sync(0xffffffffu, largest(u));
            if (mx > __float_as_uint(MOST)) {
                const int mine = !(fabsf(u[0]) <= MOST && fabsf(u[2]) <= MOST) ? OCT * w + c2 : !(fabsf(u[1]) <= MOST && fabsf(u[3]) <= MOST) ? OCT * w + c2 + 1 : C;
                odd = min(odd, __reduce_min_sync(0xffffffffu, mine));
            }
            uint32_t low = 0xffffffffu;
#pragma unroll
            for (int e = 0; e < 4; ++e) low = min(low, __float_as_uint(fabsf(u[e])) - 1);
            if (__any_sync(0xffffffffu, low < __float_as_uint(LEAST) - 1)) {        // rare: is it the largest of its token's?
                float t0 = fmaxf(fabsf(u[0]), fabsf(u[2])), t1 = fmaxf(fabsf(u[1]), fabsf(u[3]));
#pragma unroll
                for (int x = 4; x < 32; x <<= 1) {
                    t0 = fmaxf(t0, __shfl_xor_sync(0xffffffffu, t0, x));
                    t1 = fmaxf(t1, __shfl_xor_sync(0xffffffffu, t1, x));
                }
                const int mine = t0 != 0.f && t0 < LEAST ? OCT * w + c2 : t1 != 0.f && t1 < LEAST ? OCT * w + c2 + 1 : C;
                odd = min(odd, __reduce_min_sync(0xffffffffu, mine));
            }
            if (odd < C && lane == 0) atomicMin(&ex.odd[k & 1], odd);
        }
        if (!DEEP) arrive(empty + q_bar);                               // ... and Q
        if (!k_there) await(full + k_bar, rr);
        fetch_right(b0, keys, 0);
        product(q, sa[1], b1);
        fetch_right(b1, keys, 1);
        uint32_t pb[PARTS][4];
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            float4 x = reinterpret_cast<const float4*>(keys + P_AT)[(2 * w + ks) * 32 + lane];
#pragma unroll
            for (int p = 0; p < PARTS; ++p) { pb[p][2 * ks] = take_part(x.x, x.y); pb[p][2 * ks + 1] = take_part(x.z, x.w); }
        }
        if (k) store(k - 1);
        put(ex.o_part[k & 1][w], q);
        there = k + 1 < chunks && mbar_test(full + 8 * ((k + 1) % G::W), (k + 1) / G::W & 1);
        meet();
        const int odd = ex.odd[k & 1];
        float so[4][4];                                                 // the state before the chunk
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) so[nt][e] = s[nt][e];
        {   // ---- S^T = decay S^T + U^T K (the warp's rows);  U^T B^T (its tokens)
            uint32_t a[2][PARTS][4];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                for (int p = 0; p < PARTS; ++p) {
                    const uint2 t0 = ex.u[p][2 * ks][lane], t1 = ex.u[p][2 * ks + 1][lane];
                    a[ks][p][0] = t0.x; a[ks][p][1] = t0.y; a[ks][p][2] = t1.x; a[ks][p][3] = t1.y;
                }
            if (odd < C) {                                              // nothing of tokens from `odd` on goes into sums of the tokens before it
#pragma unroll
                for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                    for (int p = 0; p < PARTS; ++p)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int tok = 16 * ks + (e >> 1) * 8 + c2;
                            if (tok >= odd) a[ks][p][e] = 0;
                            else if (tok + 1 >= odd) a[ks][p][e] &= 0xffffu;
                        }
            }
            Sums x;
            clear(x);
            float lead[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
            product(x, a[0], b0);
            product(x, a[1], b1);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                for (int p = 0; p < PRODUCTS; ++p) mma16816(p < PRODUCTS - 1 ? small : lead, a[ks][PART_A[p]], pb[PART_B[p]][2 * ks], pb[PART_B[p]][2 * ks + 1]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float2 dec = *reinterpret_cast<const float2*>(keys + DEC_AT + 4 * (32 * w + 8 * nt + c2));
#pragma unroll
                for (int e = 0; e < 4; ++e) s[nt][e] = fmaf(s[nt][e], e & 1 ? dec.y : dec.x, x.lead[nt][e] + x.small[nt][e]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) own[e] = lead[e] + small[e];
        }
        left = min(n - k * C, odd);
        if (threadIdx.x == 0) ex.odd[(k + 1) & 1] = C;                  // all have read it: they had this chunk's sums before it
        arrive(empty + (DEEP ? 8 * ws : k_bar));
        if (odd < C) {
            float* cols = reinterpret_cast<float*>(&ex.u_part[0][0][0]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) cols[(32 * w + 8 * nt + c2 + (e & 1)) * VC + g + (e >> 1) * 8] = so[nt][e];
            meet();
            by_token(cols, ex.red, L, L.at + (size_t)(qs + k * C) * L.ld, min(C, n - k * C), odd, h, h / L.group, V, v0,
                     out + (size_t)(qs + k * C) * H * V + (size_t)h * V + v0, H, threadIdx.x);
            meet();
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[nt][e] = cols[(32 * w + 8 * nt + c2 + (e & 1)) * VC + g + (e >> 1) * 8];
            meet();
        }
    }
    meet();
    store(chunks - 1);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[(size_t)(32 * w + 8 * nt + c2 + (e & 1)) * V + g + (e >> 1) * 8] = s[nt][e];
}

}  // namespace

// bytes of scratch a head takes for T tokens in num_segs entries; more heads at a time run side by side
MI_EXPORT long long mi_channel_chunk_bytes(int T_, int num_segs, int V) { return (long long)(T_ / C + num_segs) * record_bytes(V); }

// prep [T, ld] float32 = q [KV D] | k [KV D] | v [H V] | g [H D] | beta [H] (rows on 16 bytes); out float32 [T, H V]; work on 16 bytes
MI_EXPORT int mi_channel_chunks(const float* prep, int ld, void* work, long long work_bytes, float* state, long long state_stride, float* out,
                                const int* seg_q_start, const int* seg_slot, int T_, int num_segs, int longest, int H, int KV, int D_, int V, int* error_word, cudaStream_t stream) {
    if (num_segs == 0 || T_ == 0) return 0;
    if (D_ != D || V % VC || H > 65535 || num_segs > 65535 || H % KV || ld % 4 || ((uintptr_t)prep | (uintptr_t)work) % 16) return -2;
    const int slots = T_ / C + num_segs, at_once = (int)std::min<long long>(H, work_bytes / mi_channel_chunk_bytes(T_, num_segs, V));
    if (at_once < 1) return -2;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(ChunkSmem));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(pass_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PASS_SMEM<true>);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(pass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PASS_SMEM<false>);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int channels = 2 * KV * D + H * V;
    const Rows L{prep, ld, KV * D, 2 * KV * D, channels, channels + H * D, H / KV};
    for (int h0 = 0; h0 < H; h0 += at_once) {
        const int heads = std::min(at_once, H - h0);
        chunk_kernel<<<dim3(slots, heads), 128, sizeof(ChunkSmem), stream>>>(L, (unsigned char*)work, seg_q_start, num_segs, h0, V);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
        // A block an SM where every block then has one (2,048 tokens 162 us against 177 with two), or where there are more than two and the longest
        // entry's walk is two thirds and more of what an SM walks on average (an entry counted as two chunks more than it has: 1,500 + 300 + 200 tokens
        // 159 and 191, 1,300 + 517 + 231 160 and 176, 300 + 700 + 200 113 and 100, 4 x 512 168 and 151, 900 + 500 125 and 113, 8 x 1,024 556 and 508).
        const long long blocks = (long long)heads * num_segs * (V / VC), all = (long long)(T_ / C + 2 * num_segs) * heads * (V / VC);
        const long long sms = device_sms();
        const bool deep = blocks <= sms || (blocks > 2 * sms && 20 * sms * (longest / C + 2) >= 13 * all);
        auto walk = deep ? pass_kernel<true> : pass_kernel<false>;
        walk<<<dim3(V / VC, heads, num_segs), 160, deep ? PASS_SMEM<true> : PASS_SMEM<false>, stream>>>((const unsigned char*)work, slots, L, state, state_stride, out, seg_q_start,
                                                                                                    seg_slot, H, h0, V, error_word);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}
