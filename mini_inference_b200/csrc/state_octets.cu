// Matrix-state recurrences over prompt portions, EIGHT tokens at a time, in float32 (the forms of recurrent.cu that it states token by token):
//   delta       S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q      (a decay per head and key channel)
//   constant    S <- d S + k v^T;  o = S^T q                                            (one decay per head)
// Unrolled over an octet with S_0 before it, G_ij = g_{j+1} .. g_i (products of decays, never more than 1) and G_i = g_0 .. g_i, row by row:
//   w_i = beta_i (v_i - (G_i k_i)^T S_0);   u_i = w_i - beta_i sum_{j<i} A_ij u_j,            A_ij = sum k_i G_ij k_j
//   o_i = (G_i q_i)^T S_0 + sum_{j<=i} B_ij u_j,  B_ij = sum q_i G_ij k_j;       S = G_7 S_0 + sum_j (G_7j k_j) u_j^T
// (constant: u = v, no A).  That is 3 1/8 (2 1/8) multiply-adds per state entry and token instead of 4 (3), and the chain from token to token,
// S^T k summed over lanes by shuffles before anything else can go on, is walked once per octet.
//
// octet_kernel, a warp per (octet, head): the row vectors k G_i, q G_i, G_7j k_j, G_7 and the scalars A beta, B, beta, written as one record, and the
// values in float32 (constant: the silu of q, k and v first).
// scan_kernel, a block per (entry, head, 16 columns): a warp owns four columns and its 32 lanes the rows, so that a vector of the record is read from
// shared memory once per four columns.  A 16-byte load of a warp takes the shared-memory pipe four clocks even where lanes read the same
// words, so with 8 lanes to a pair of columns the loads were 65 % of that pipe's time.  The 32 sums over lanes (eight tokens, four columns)
// are made together, lane l ends with sum l; u goes around through shared memory.  One more warp brings the records by bulk copies into
// a ring: a head's records lie one behind the other, and so do its values of the block's columns, so an octet is two copies.  (A record
// and a row of values per token took the copying thread 480 ns for four tokens, whatever the compute warps did.)
// Scan with its octet_kernel, 16 heads of 128 x 128: 2,048 tokens 553 -> 234 us (delta), 286 -> 166 us (constant, silu included); 4 x 512
// tokens 449 -> 198 and 197 -> 135 us; 16 x 64 tokens 212 -> 101 and 113 -> 71 us.  One warp a scheduler issues every 2.4 clocks: what is left
// is the latency of one warp's own instructions.  (Two groups of 16 lanes with four columns each in a warp need 40 % fewer instructions per
// column, but half as many warps share one prompt: 297 and 198 us.)
#include "sm100.cuh"
#include <math.h>

using namespace mi;
using namespace mi::sm100;

namespace {

constexpr int C = 8, NC = 4, WARPS = 4, COLS = NC * WARPS;      // tokens at a time; columns of a warp, warps and columns of a block
constexpr int STAGES = 6, SCALARS = 2 * C * C + C + 8;      // N [8][8] | B [8][8] | beta [8] | d^8 - 1 | unused
constexpr int B_OFF = C * C, BETA_OFF = 2 * C * C, D8_OFF = BETA_OFF + C;

template <bool DELTA> __host__ __device__ constexpr int vectors() { return DELTA ? 3 * C + 1 : 2 * C; }
template <bool DELTA> __host__ __device__ constexpr int record_floats(int D) { return vectors<DELTA>() * D + SCALARS; }

// An entry's octets lie behind floor(first token / 8) + entry slots: entries never share one.
__device__ __forceinline__ int first_slot(int qs, int seg) { return qs / C + seg; }

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ float silu(float x) { return x / (1.f + expf(-x)); }

// R (2 or 4) neighbouring entries in one access
template <int R> __device__ __forceinline__ void load_n(const float* p, float (&v)[R]) {
    if constexpr (R == 4) { const float4 t = *reinterpret_cast<const float4*>(p); v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
    else { const float2 t = *reinterpret_cast<const float2*>(p); v[0] = t.x; v[1] = t.y; }
}
template <int R> __device__ __forceinline__ void load_n(const __nv_bfloat16* p, float (&v)[R]) {
    if constexpr (R == 4) {
        const uint2 t = *reinterpret_cast<const uint2*>(p);
        v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u); v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
    } else {
        const uint32_t t = *reinterpret_cast<const uint32_t*>(p);
        v[0] = __uint_as_float(t << 16); v[1] = __uint_as_float(t & 0xffff0000u);
    }
}
template <int R> __device__ __forceinline__ void store_n(float* p, const float (&v)[R]) {
    if constexpr (R == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

struct Source {                 // where a token's numbers are: q, k, g (+ head * D), v (+ head * V), beta (+ head) in rows of ld entries
    int ld, q, k, v, g, beta;
};

// grid (slots, heads / 4), 4 warps: a warp owns one octet of one head.  DELTA: in is the float32 prologue's rows; else the rows as projected.
template <typename T, bool DELTA, bool SILU, int D>
__global__ void __launch_bounds__(128) octet_kernel(const T* __restrict__ in, const Source L, const float* __restrict__ decay, float* __restrict__ rec,
                                                   float* __restrict__ v_out, const int* __restrict__ seg_q_start, int num_segs, int H, int KV, int V) {
    constexpr int R = D / 32;                                       // neighbouring rows a lane owns
    const int slot = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (h >= H) return;
    int lo = 0, hi = num_segs - 1;                                  // the entry whose octets hold this slot
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (first_slot(seg_q_start[mid], mid) <= slot) lo = mid; else hi = mid - 1;
    }
    const int qs = seg_q_start[lo], n = seg_q_start[lo + 1] - qs, t0 = C * (slot - first_slot(qs, lo));
    if (t0 >= n) return;
    const int kvh = h / (H / KV);
    float q[C][R], k[C][R], g[C][R];
    const float d1 = DELTA ? 0.f : decay[h];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const bool ok = t0 + i < n;                                 // a token behind the last: no decay, no key, beta 0
        const T* row = in + (size_t)(qs + t0 + (ok ? i : 0)) * L.ld;
        load_n<R>(row + L.q + kvh * D + lane * R, q[i]);
        load_n<R>(row + L.k + kvh * D + lane * R, k[i]);
        if (DELTA) load_n<R>(row + L.g + h * D + lane * R, g[i]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (SILU) { q[i][r] = silu(q[i][r]); k[i][r] = silu(k[i][r]); }
            if (!DELTA) g[i][r] = d1;
            if (!ok) { q[i][r] = k[i][r] = 0.f; g[i][r] = 1.f; }
        }
    }
    for (int c = 2 * lane; c < V; c += 64) {                        // values: [head][column block][slot][8][COLS] float32, zeros behind the last token
        float t[C][2];
#pragma unroll
        for (int i = 0; i < C; ++i) {
            t[i][0] = t[i][1] = 0.f;
            if (t0 + i < n) load_n<2>(in + (size_t)(qs + t0 + i) * L.ld + L.v + h * V + c, t[i]);
        }
        float* to = v_out + (((size_t)h * (V / COLS) + c / COLS) * gridDim.x + slot) * C * COLS + c % COLS;
#pragma unroll
        for (int i = 0; i < C; ++i)
            *reinterpret_cast<float2*>(to + i * COLS) = SILU ? make_float2(silu(t[i][0]), silu(t[i][1])) : make_float2(t[i][0], t[i][1]);
    }
    float* o = rec + ((size_t)h * gridDim.x + slot) * record_floats<DELTA>(D);
    float* kd = o;                                                  // DELTA: k_i G_i
    float* qd = o + (DELTA ? C * D : 0);
    float* kh = qd + C * D;
    float* sc = o + vectors<DELTA>() * D;
    float G[R], khat[C][R], y[32], z[32];                           // 28 A_ij (j < i) at i (i - 1) / 2 + j; 36 B_ij (j <= i) at i (i + 1) / 2 + j
#pragma unroll
    for (int e = 0; e < 32; ++e) y[e] = z[e] = 0.f;
    float last[4] = {0.f, 0.f, 0.f, 0.f};                           // B_ij from 32 on
#pragma unroll
    for (int r = 0; r < R; ++r) G[r] = 1.f;
#pragma unroll
    for (int i = 0; i < C; ++i) {
        float a[R], b[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            G[r] *= g[i][r];
            a[r] = k[i][r] * G[r];
            b[r] = q[i][r] * G[r];
            khat[i][r] = k[i][r];
#pragma unroll
            for (int j = 0; j <= i; ++j) {
                if (j < i) {
                    khat[j][r] *= g[i][r];                          // now G_ij k_j
                    if (DELTA) y[i * (i - 1) / 2 + j] = fmaf(k[i][r], khat[j][r], y[i * (i - 1) / 2 + j]);
                }
                const int e = i * (i + 1) / 2 + j;
                if (e < 32) z[e] = fmaf(q[i][r], khat[j][r], z[e]);
                else last[e - 32] = fmaf(q[i][r], khat[j][r], last[e - 32]);
            }
        }
        if (DELTA) store_n<R>(kd + i * D + lane * R, a);
        store_n<R>(qd + i * D + lane * R, b);
    }
#pragma unroll
    for (int j = 0; j < C; ++j) store_n<R>(kh + j * D + lane * R, khat[j]);
    if (DELTA) store_n<R>(kh + C * D + lane * R, G);
    // lane l ends with the l-th of each; the squares' other entries are zeros
    const float b_sum = sum_spread<32>(z, lane), b_last = sum_spread<4>(last, lane), a_sum = DELTA ? sum_spread<32>(y, lane) : 0.f;
    for (int e = lane; e < B_OFF + C * C; e += 32) sc[e] = 0.f;
    __syncwarp();
    auto row_of = [](int e) { int i = 0; while ((i + 1) * (i + 2) / 2 <= e) ++i; return i; };       // of e in a lower triangle with its diagonal
    {
        const int i = row_of(lane), j = lane - i * (i + 1) / 2;
        sc[B_OFF + C * i + j] = b_sum;
        if (lane < 4) sc[B_OFF + C * 7 + 4 + lane] = b_last;        // B_74 .. B_77
        if (DELTA && lane < 28)
            sc[C * (i + 1) + j] = t0 + i + 1 < n ? a_sum * to_f32(in[(size_t)(qs + t0 + i + 1) * L.ld + L.beta + h]) : 0.f;
    }
    if (lane < C) sc[BETA_OFF + lane] = DELTA && t0 + lane < n ? to_f32(in[(size_t)(qs + t0 + lane) * L.ld + L.beta + h]) : 0.f;
    if (!DELTA && lane == C) {                                      // d^m - 1 for the octet's m tokens: s + s (d^m - 1) keeps the last bits of a decay near 1
        double p = 1.0;
        for (int m = 0; m < min(C, n - t0); ++m) p *= (double)decay[h];
        sc[D8_OFF] = (float)(p - 1.0);
    }
}

// grid (V / COLS, heads, entries); WARPS compute warps and one that copies
template <bool DELTA, int D>
__global__ void __launch_bounds__(32 * WARPS + 32, DELTA ? 2 : 3) scan_kernel(const float* __restrict__ rec, const float* __restrict__ v, int slots, float* __restrict__ state,
                                                                  long long state_stride, float* __restrict__ out, const int* __restrict__ seg_q_start,
                                                                  const int* __restrict__ seg_slot, int H, int V, int* __restrict__ error_word) {
    constexpr int RF = record_floats<DELTA>(D), STAGE = RF + C * COLS, R = D / 32, RP = R / 2, NV = C * NC;
    static_assert(NV == 32, "a lane per sum");
    extern __shared__ __align__(128) float sm[];
    float* around = sm + STAGES * STAGE;                            // [2][WARPS][C][NC]: w (delta), two octets in turn
    uint64_t* bars = reinterpret_cast<uint64_t*>(around + 2 * WARPS * NV);
    const uint32_t full = smem_u32(bars), empty = smem_u32(bars + STAGES);
    const int seg = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * COLS;
    const int qs = seg_q_start[seg], n = seg_q_start[seg + 1] - qs, octets = (n + C - 1) / C;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, WARPS); }
        mbar_init_fence();
    }
    __syncthreads();
    if (warp == WARPS) {
        // ---------------- copies: an octet's record, and its values of the block's columns
        if (lane == 0) {
            const float* src = rec + ((size_t)h * slots + first_slot(qs, seg)) * RF;
            const float* vs = v + (((size_t)h * (V / COLS) + blockIdx.x) * slots + first_slot(qs, seg)) * C * COLS;
            for (int k = 0; k < octets; ++k) {
                const int st = k % STAGES;
                if (k >= STAGES && !mbar_wait(empty + 8 * st, (k / STAGES - 1) & 1)) { atomicExch(error_word, 41); break; }
                const uint32_t dst = smem_u32(sm + st * STAGE);
                mbar_expect_tx(full + 8 * st, STAGE * 4);
                bulk_load(dst, src + (size_t)k * RF, RF * 4, full + 8 * st);
                bulk_load(dst + RF * 4, vs + (size_t)k * C * COLS, C * COLS * 4, full + 8 * st);
            }
        }
        return;
    }
    const int cw = warp * NC;                                       // the warp's first column in the block
    float* S = state + (long long)seg_slot[seg] * state_stride + (long long)h * D * V + (size_t)(R * lane) * V + col0 + cw;
    float2 s[NC][RP];                                               // rows R lane + 2 p, + 1 of column c
#pragma unroll
    for (int p = 0; p < RP; ++p)
#pragma unroll
        for (int c = 0; c < NC; c += 2) {
            const float2 a = *reinterpret_cast<const float2*>(S + (size_t)(2 * p) * V + c), b = *reinterpret_cast<const float2*>(S + (size_t)(2 * p + 1) * V + c);
            s[c][p] = make_float2(a.x, b.x);
            s[c + 1][p] = make_float2(a.y, b.y);
        }
    const int my_i = lane / NC, my_c = lane % NC;             // the sum a lane ends up with: token my_i, column my_c
    float* out_at = out + (size_t)(qs + my_i) * H * V + (size_t)h * V + col0 + cw + my_c;
    auto fetch = [&](float2 (&x)[C][RP], const float* r, int vec) {  // C vectors, this lane's rows
#pragma unroll
        for (int i = 0; i < C; ++i) {
            if constexpr (RP == 2) {
                const float4 t = *reinterpret_cast<const float4*>(r + (vec + i) * D);
                x[i][0] = make_float2(t.x, t.y); x[i][RP - 1] = make_float2(t.z, t.w);
            } else {
                x[i][0] = *reinterpret_cast<const float2*>(r + (vec + i) * D);
            }
        }
    };
    auto dots = [&](const float2 (&x)[C][RP], float (&y)[NV]) {      // y[i NC + c]: this lane's rows of vector i with column c
#pragma unroll
        for (int i = 0; i < C; ++i)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float2 a = __fmul2_rn(s[c][0], x[i][0]);
                if (RP == 2) a = __ffma2_rn(s[c][RP - 1], x[i][RP - 1], a);
                y[i * NC + c] = a.x + a.y;
            }
    };
    bool there = false;                                             // the next record was there when this one was begun
    for (int k = 0; k < octets; ++k) {
        const int st = k % STAGES, st1 = (k + 1) % STAGES;
        if (!there && !mbar_spin(full + 8 * st, (k / STAGES) & 1)) { if (lane == 0) atomicExch(error_word, 42); break; }
        const float* r = sm + st * STAGE + R * lane;
        const float* sc = sm + st * STAGE + vectors<DELTA>() * D;
        const float* vv = sm + st * STAGE + RF + cw;
        float2 x[C][RP], xq[C][RP], u[C][NC / 2];                    // u[i][c / 2]: two columns
        float z[NV], own[C];                                         // own: u of this lane's column
        if constexpr (DELTA) {
            float2 dec[RP];
            fetch(x, r, 0);
            fetch(xq, r, C);
            there = k + 1 < octets && mbar_test(full + 8 * st1, ((k + 1) / STAGES) & 1);
            float y[NV];
            dots(x, y);
            fetch(x, r, 2 * C);
            if constexpr (RP == 2) {
                const float4 t = *reinterpret_cast<const float4*>(r + 3 * C * D);
                dec[0] = make_float2(t.x, t.y); dec[RP - 1] = make_float2(t.z, t.w);
            } else {
                dec[0] = *reinterpret_cast<const float2*>(r + 3 * C * D);
            }
            const float beta = sc[BETA_OFF + my_i], value = vv[my_i * COLS + my_c];
            const float dot = sum_spread<NV>(y, lane);
            float* w = around + ((k & 1) * WARPS + warp) * NV;
            w[lane] = beta * (value - dot);                          // 0 behind the last token
            dots(xq, z);                                             // what the state before the octet gives to the outputs; u does not wait for it
            __syncwarp();
#pragma unroll
            for (int i = 0; i < C; ++i) {
                const float4 t = *reinterpret_cast<const float4*>(w + i * NC);
                u[i][0] = make_float2(t.x, t.y); u[i][1] = make_float2(t.z, t.w);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int p = 0; p < RP; ++p) s[c][p] = __fmul2_rn(s[c][p], dec[p]);
#pragma unroll
            for (int i = 1; i < C; ++i) {
                float a[C];
                *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(sc + C * i);
                if (i > 4) *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(sc + C * i + 4);
#pragma unroll
                for (int m = 0; m < i; ++m)
#pragma unroll
                    for (int c = 0; c < NC / 2; ++c) u[i][c] = __ffma2_rn(make_float2(-a[m], -a[m]), u[m][c], u[i][c]);
            }
#pragma unroll
            for (int i = 0; i < C; ++i) {
                const float2 t = my_c & 2 ? u[i][1] : u[i][0];
                own[i] = my_c & 1 ? t.y : t.x;
            }
        } else {
            fetch(xq, r, 0);
            fetch(x, r, C);
            there = k + 1 < octets && mbar_test(full + 8 * st1, ((k + 1) / STAGES) & 1);
            const float d8 = sc[D8_OFF];                             // d^8 - 1
#pragma unroll
            for (int i = 0; i < C; ++i) {
                const float4 t = *reinterpret_cast<const float4*>(vv + i * COLS);
                u[i][0] = make_float2(t.x, t.y); u[i][1] = make_float2(t.z, t.w);
                own[i] = vv[i * COLS + my_c];
            }
            dots(xq, z);
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int p = 0; p < RP; ++p) s[c][p] = __ffma2_rn(s[c][p], make_float2(d8, d8), s[c][p]);
        }
#pragma unroll
        for (int i = 0; i < C; ++i)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float uc = c & 1 ? u[i][c / 2].y : u[i][c / 2].x;
#pragma unroll
                for (int p = 0; p < RP; ++p) s[c][p] = __ffma2_rn(x[i][p], make_float2(uc, uc), s[c][p]);
            }
        float o = sum_spread<NV>(z, lane);
        const float4 b0 = *reinterpret_cast<const float4*>(sc + B_OFF + C * my_i), b1 = *reinterpret_cast<const float4*>(sc + B_OFF + C * my_i + 4);      // zeros above the diagonal
        // a later token's number may be anything, and 0 * inf is no 0.  (Selections cost a mixer 1.7 %; masks held in registers 1 to 4 %, a second
        // sum where the first is not finite 2 to 4 %: the branch ends what overlaps between octets.)
        auto known = [&](int j) { return j <= my_i ? own[j] : 0.f; };
        float o2 = b1.x * known(4);
        o = fmaf(b0.x, known(0), o); o2 = fmaf(b1.y, known(5), o2);
        o = fmaf(b0.y, known(1), o); o2 = fmaf(b1.z, known(6), o2);
        o = fmaf(b0.z, known(2), o); o2 = fmaf(b1.w, known(7), o2);
        o = fmaf(b0.w, known(3), o) + o2;
        if (C * k + my_i < n) *out_at = o;
        out_at += (size_t)C * H * V;
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * st);
    }
#pragma unroll
    for (int p = 0; p < RP; ++p)
#pragma unroll
        for (int c = 0; c < NC; c += 2) {
            *reinterpret_cast<float2*>(S + (size_t)(2 * p) * V + c) = make_float2(s[c][p].x, s[c + 1][p].x);
            *reinterpret_cast<float2*>(S + (size_t)(2 * p + 1) * V + c) = make_float2(s[c][p].y, s[c + 1][p].y);
        }
}

template <bool DELTA, int D>
int run_scan(const float* rec, const float* values, int slots, float* state, long long state_stride, float* out, const int* seg_q_start, const int* seg_slot,
             int num_segs, int H, int V, int* error_word, cudaStream_t stream) {
    constexpr int bytes = (STAGES * (record_floats<DELTA>(D) + C * COLS) + 2 * WARPS * C * NC) * 4 + 2 * STAGES * 8;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(scan_kernel<DELTA, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    scan_kernel<DELTA, D><<<dim3(V / COLS, H, num_segs), 32 * WARPS + 32, bytes, stream>>>(rec, values, slots, state, state_stride, out, seg_q_start, seg_slot,
                                                                                        H, V, error_word);
    return (int)cudaGetLastError();
}

template <typename T, bool DELTA, bool SILU>
int run(const T* in, const Source& L, const float* decay, float* rec, float* values, float* state, long long state_stride, float* out,
        const int* seg_q_start, const int* seg_slot, int T_, int num_segs, int H, int KV, int D, int V, int* error_word, cudaStream_t stream) {
    if (num_segs == 0 || T_ == 0) return 0;
    if ((D != 64 && D != 128) || V % COLS || H > 65535 || num_segs > 65535 || H % KV || state_stride % 2 || (uintptr_t)state % 8) return -2;
    if (L.ld % 4 || (uintptr_t)in % 16 || (uintptr_t)values % 16 || (uintptr_t)rec % 16) return -2;       // every head starts on a multiple of 16 entries
    const int slots = T_ / C + num_segs;
    const dim3 ogrid(slots, (H + 3) / 4);
    if (D == 128) octet_kernel<T, DELTA, SILU, 128><<<ogrid, 128, 0, stream>>>(in, L, decay, rec, values, seg_q_start, num_segs, H, KV, V);
    else octet_kernel<T, DELTA, SILU, 64><<<ogrid, 128, 0, stream>>>(in, L, decay, rec, values, seg_q_start, num_segs, H, KV, V);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    if (D == 128) return run_scan<DELTA, 128>(rec, values, slots, state, state_stride, out, seg_q_start, seg_slot, num_segs, H, V, error_word, stream);
    return run_scan<DELTA, 64>(rec, values, slots, state, state_stride, out, seg_q_start, seg_slot, num_segs, H, V, error_word, stream);
}

}  // namespace

// floats of scratch for T tokens in num_segs entries: the records; the values lie behind them
MI_EXPORT long long mi_octet_floats(int T_, int num_segs, int H, int D, int V, int delta) {
    return (long long)(T_ / C + num_segs) * H * ((delta ? record_floats<true>(D) : record_floats<false>(D)) + C * V);
}

// prep [T, ld] float32 = q [KV D] | k [KV D] | v [H V] | g [H D] | beta [H] (rows on 16 bytes); out float32 [T, H V]; scratch: mi_octet_floats
MI_EXPORT int mi_delta_octets(const float* prep, int ld, float* scratch, float* state, long long state_stride, float* out, const int* seg_q_start,
                              const int* seg_slot, int T_, int num_segs, int H, int KV, int D, int V, int* error_word, cudaStream_t stream) {
    const int channels = 2 * KV * D + H * V;
    float* values = scratch + (size_t)(T_ / C + num_segs) * H * record_floats<true>(D);
    return run<float, true, false>(prep, Source{ld, 0, KV * D, 2 * KV * D, channels, channels + H * D}, nullptr, scratch, values, state, state_stride, out, seg_q_start,
                            seg_slot, T_, num_segs, H, KV, D, V, error_word, stream);
}

// rows [T, 2 H D + H V] float32 = q | k | v as they enter the recurrence; decay [H]; otherwise as mi_delta_octets
MI_EXPORT int mi_constant_octets(const float* rows, float* scratch, const float* decay, float* state, long long state_stride, float* out, const int* seg_q_start,
                                 const int* seg_slot, int T_, int num_segs, int H, int D, int V, int* error_word, cudaStream_t stream) {
    float* values = scratch + (size_t)(T_ / C + num_segs) * H * record_floats<false>(D);
    return run<float, false, false>(rows, Source{2 * H * D + H * V, 0, H * D, 2 * H * D, 0, 0}, decay, scratch, values, state, state_stride, out, seg_q_start,
                                    seg_slot, T_, num_segs, H, H, D, V, error_word, stream);
}

// p [T, ldp] bfloat16 = q | k | v before silu; decay [H]; otherwise as mi_delta_octets
MI_EXPORT int mi_lightning_octets(const void* p, int ldp, float* scratch, const float* decay, float* state, long long state_stride, float* out,
                                  const int* seg_q_start, const int* seg_slot, int T_, int num_segs, int H, int D, int V, int* error_word, cudaStream_t stream) {
    float* values = scratch + (size_t)(T_ / C + num_segs) * H * record_floats<false>(D);
    return run<__nv_bfloat16, false, true>((const __nv_bfloat16*)p, Source{ldp, 0, H * D, 2 * H * D, 0, 0}, decay, scratch, values, state, state_stride, out, seg_q_start,
                                           seg_slot, T_, num_segs, H, H, D, V, error_word, stream);
}
