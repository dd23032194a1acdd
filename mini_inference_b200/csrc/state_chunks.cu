// The recurrence with a constant decay per head, S <- d S + k v^T; o = S^T q (lightning attention, retention), over prompt portions of bfloat16 runs,
// 128 tokens at a time on the tensor cores, every operand in three bfloat16 parts (split3.cuh: float32 products).  With S_0 before a chunk of n tokens:
//   S_n = d^n S_0 + sum_j d^(n-1-j) k_j v_j^T;       o_i = d^(i+1) S_0^T q_i + sum_{j<=i} d^(i-j) (q_i . k_j) v_j
// Three kernels, so that all chunks of a prompt are worked on at once and only an addition walks from chunk to chunk:
//   chunk_state_kernel   a block per (chunk, head, 128 columns): the sum that the chunk adds to the state, [D x tokens] [tokens x V]
//   chunk_scan_kernel    every state entry on its own: the state before each chunk takes the place of the chunk's sum, the last one the slot's
//   chunk_out_kernel     a block per (chunk, head, 128 columns): Q K^T, masked and decayed, times V, and Q S_0
// Operands whose rows are the product's M side (K^T, Q, the masked scores) go to tensor memory, a thread a row; the others to shared memory in the
// 128-byte swizzle.  state_octets.cu walks a prompt eight tokens at a time: bound by the latency of one warp's instructions, whatever the chip has free.
//
// 16 heads of 128 x 128, silu included, microseconds there / here: 2,048 tokens 167 / 73, 4 x 512 137 / 76, 700 + 3 65 / 38, 400 41 / 36, 256 31 / 36.
// Error against 64 bits (2-norm, 2,048 tokens): outputs 9.6e-8 / 8.9e-8, states 2.3e-7 / 8.2e-8.  A block of the last kernel takes some 38,000 clocks of
// which the tensor pipe needs 9,200: 4,600 instructions a warp (silu 1,500, parts 1,100, sums 700), a third of the issue slots used, each product
// waiting for the operand before it.  Scores of all 128 columns in one sum in tensor memory cost 2.2e-7 of error, of 32 columns 1.2e-7, the leading
// products of parts of 32 on their own 8.9e-8.
//
// Numbers that the parts do not hold are taken out of the products; the outputs from their token on are computed once more token by token in float32, those
// before it have the bits they have without it.  These are infinities and NaN; a query (a quarter of it) or a key whose largest magnitude is not in
// [2^-50, 2^36], so that scores stay where their parts are whole; 8 values beyond [2^-90, 2^36] and 8 entries of a state beyond [2^-90, 2^60].  All else is
// as exact as float32 sums are against |q| |k| |v| as vectors; what decays below 2^-100 of that may keep fewer bits than it has in float32.
#include "split3.cuh"
#include <algorithm>

using namespace mi;
using namespace mi::sm100;
using namespace mi::split3;

namespace {

constexpr int C = 128, D = 128, VC = 128;                       // tokens of a chunk, rows of a state, columns of a block
constexpr int WORKERS = 512, THREADS = WORKERS + 32;            // 16 warps, a thread one row and a quarter of its columns; one warp issues the products
constexpr int BLOCK64 = C * 128, PART_BYTES = 2 * BLOCK64, OPERAND = PARTS * PART_BYTES;      // 128 rows of 64 bfloat16; an operand's part; its parts
constexpr int ROW_OUT = VC + 4;                                 // floats of a result's row in shared memory
struct Range { float least, most; };
constexpr Range SCORED{0x1p-50f, 0x1p36f}, ADDED{0x1p-90f, 0x1p36f}, STATE{0x1p-90f, 0x1p60f};      // q and k; v, and k on its way into the state; the state

// An entry's chunks lie behind floor(first token / 128) + entry slots: entries never share one.
__host__ __device__ __forceinline__ int first_slot(int qs, int seg) { return qs / C + seg; }

__device__ __noinline__ float silu(float x) { return x / (1.f + expf(-x)); }
// x / (1 + e^-x).  The quotient by one of Newton's steps on its remainder (Markstein, 1990) is a third of a division that also takes 1 + e^-x
// beyond 2^126; inputs down there go to that division, once for all N numbers.  An infinity becomes NaN here: both do not fit, and their tokens are
// computed again with the division.
template <int N> __device__ __forceinline__ void silu(float (&v)[N]) {
    float least = INFINITY;
#pragma unroll
    for (int e = 0; e < N; ++e) least = fminf(least, v[e]);
    if (least > -80.f) {                                        // NaN stays NaN on either way
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const float y = 1.f + expf(-v[e]);
            float r;
            asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(y));
            const float q = v[e] * r;
            v[e] = fmaf(fmaf(-q, y, v[e]), r, q);
        }
    } else {
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] = silu(v[e]);
    }
}

struct Source { int ld, q, k, v; };                             // columns of q, k (+ head * D), v (+ head * V) in rows of ld entries

struct Chunk { int seg, qs, t0, n; };                           // entry, its first token, the chunk's first token in it, its tokens (0: no chunk here)
__device__ __forceinline__ Chunk chunk_of(int slot, const int* __restrict__ seg_q_start, int num_segs) {
    int lo = 0, hi = num_segs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (first_slot(seg_q_start[mid], mid) <= slot) lo = mid; else hi = mid - 1;
    }
    Chunk c;
    c.seg = lo;
    c.qs = seg_q_start[lo];
    c.t0 = C * (slot - first_slot(c.qs, lo));
    c.n = max(0, min(C, seg_q_start[lo + 1] - c.qs - c.t0));
    return c;
}

__device__ __forceinline__ double power(double d, int m) {      // d^m, m >= 0
    double p = 1.0;
    for (; m; m >>= 1, d *= d) if (m & 1) p *= d;
    return p;
}

template <int N> __device__ __forceinline__ void clear(float (&v)[N]) {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = 0.f;
}
template <typename T, int N> __device__ __forceinline__ void load_n(const T* p, float (&v)[N]) {
#pragma unroll
    for (int e = 0; e < N; e += Vec16<T>::N) load16(p + e, v + e);
}
template <bool SILU, int N> __device__ __forceinline__ void activate(float (&v)[N]) {
    if constexpr (SILU) silu(v);
}
template <int N> __device__ __forceinline__ float largest(const float (&v)[N]) {       // NaN if there is one
    float mx = 0.f;
#pragma unroll
    for (int e = 0; e < N; ++e) asm("max.NaN.f32 %0, %0, %1;\n" : "+f"(mx) : "f"(fabsf(v[e])));
    return mx;
}
// Whether the parts hold numbers of which this is the largest magnitude; if not they become zeros
template <int N> __device__ __forceinline__ bool fits(float (&v)[N], float mx, Range range) {
    const bool ok = mx <= range.most && (mx == 0.f || mx >= range.least);
    if (!ok) clear(v);
    return ok;
}
// 128 rows of 128 numbers as they lie in global memory, in registers: a thread has 8 neighbouring numbers of 4 rows, 16 threads a row (whole lines)
template <typename T> struct Tile { uint4 w[4][8 / Vec16<T>::N]; };
template <typename T>
__device__ __forceinline__ void fetch(Tile<T>& t, const T* src, size_t ld, int rows) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int id = i * WORKERS + threadIdx.x, row = id >> 4, c = id & 15;
#pragma unroll
        for (int j = 0; j < 8 / Vec16<T>::N; ++j)
            t.w[i][j] = row < rows ? *reinterpret_cast<const uint4*>(src + row * ld + 8 * c + j * Vec16<T>::N) : make_uint4(0, 0, 0, 0);
    }
}
// ... -> the three parts in shared memory, the 16-byte pieces of a row by 8 threads side by side.  Answers with the first row that does not fit (C: none).
// ROW: judged by the whole row, else by 8 numbers.
template <typename T, bool SILU, bool ROW = false>
__device__ __forceinline__ int to_shared(unsigned char* operand, const Tile<T>& t, Range range) {
    int odd = C;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int id = i * WORKERS + threadIdx.x, row = id >> 4, c = id & 15;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8 / Vec16<T>::N; ++j) load16(reinterpret_cast<const T*>(&t.w[i][j]), v + j * Vec16<T>::N);
        activate<SILU>(v);
        float mx = largest(v);
        if (ROW) {
#pragma unroll
            for (int w = 1; w < 16; w <<= 1) asm("max.NaN.f32 %0, %0, %1;\n" : "+f"(mx) : "f"(__shfl_xor_sync(0xffffffffu, mx, w)));
        }
        if (!fits(v, mx, range)) odd = min(odd, row);
        unsigned char* at = operand + (c >> 3) * BLOCK64 + row * 128 + (((c ^ row) & 7) << 4);
#pragma unroll
        for (int p = 0; p < PARTS; ++p) {
            uint4 w;
            w.x = take_part(v[0], v[1]);
            w.y = take_part(v[2], v[3]);
            w.z = take_part(v[4], v[5]);
            w.w = take_part(v[6], v[7]);
            *reinterpret_cast<uint4*>(at + p * PART_BYTES) = w;
        }
    }
    return odd;
}
// ... -> rows in shared memory, PITCH bytes apart: the threads that have rows or columns to themselves read them there
template <typename T> constexpr int PITCH = D * (int)sizeof(T) + 16;
template <typename T>
__device__ __forceinline__ void stage(unsigned char* rows, const Tile<T>& t) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int id = i * WORKERS + threadIdx.x, row = id >> 4, c = id & 15;
#pragma unroll
        for (int j = 0; j < 8 / Vec16<T>::N; ++j) *reinterpret_cast<uint4*>(rows + row * PITCH<T> + 8 * c * sizeof(T) + 16 * j) = t.w[i][j];
    }
}
// 32 numbers of a row -> the three parts in tensor memory: part p's 64 columns from 64 p on, of which this is quarter `quarter`
__device__ __forceinline__ void to_tensor(uint32_t lanes, int quarter, float (&v)[32]) {
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) w[e] = take_part(v[2 * e], v[2 * e + 1]);
        tmem_st16(lanes + 64 * p + 16 * quarter, w);
    }
}
__device__ __forceinline__ void shared_is_written() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// The products of a block, by one thread: A's parts in tensor memory from `a` on, B's in shared memory (MN: stored [k][n], else [n][k]).  The tensor
// core cuts off where it adds, half a unit in the last place each time and always towards zero, so long sums stay out of it: the five small products of
// parts of all of K are one sum (what that loses does not count), the leading ones are added 32 of K at a time.  Two accumulators take turns; the
// workers add up in float32, rounded to nearest.
constexpr int GROUPS = 5;
struct Sums { uint32_t tmem, full, empty; };                    // two accumulators of 128 columns from column 192 on; their barriers
template <bool MN>
__device__ __forceinline__ bool product(const Sums& d, int& turn, uint32_t a, uint32_t b) {
    const uint32_t idesc = umma_idesc_bf16(128, 128, MN);
    const uint64_t desc = MN ? umma_desc_sw128(b, BLOCK64, 1024) : umma_desc_sw128(b, 16, 1024);
#pragma unroll 1
    for (int g = 0; g < GROUPS; ++g, ++turn) {
        const int s = turn & 1;
        if (turn >= 2 && !mbar_spin(d.empty + 8 * s, ((turn >> 1) - 1) & 1)) return false;
        tc_fence_after();
        auto step = [&](int p, int ks, bool add) {
            const uint32_t off = PART_B[p] * PART_BYTES + (MN ? ks * 2048 : ks / 4 * BLOCK64 + ks % 4 * 32);
            umma_ts(d.tmem + 192 + 128 * s, a + PART_A[p] * 64 + ks * 8, desc + (off >> 4), idesc, add);
        };
        if (g == 1) {                                           // the long one in second place: the first is fetched under it
#pragma unroll 1
            for (int p = 0; p < PRODUCTS - 1; ++p)
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) step(p, ks, (p | ks) != 0);
        } else {
            const int ks = g ? 2 * g - 2 : 0;
            step(PRODUCTS - 1, ks, false);
            step(PRODUCTS - 1, ks + 1, true);
        }
        umma_commit(d.full + 8 * s);
    }
    return true;
}
// ... and the worker's side: the sums of its row and quarter
__device__ __forceinline__ bool add_up(const Sums& d, int& turn, uint32_t lanes, int quarter, float (&acc)[32]) {
    clear(acc);
    bool ok = true;
#pragma unroll 1
    for (int g = 0; g < GROUPS; ++g, ++turn) {
        const int s = turn & 1;
        ok &= mbar_wait(d.full + 8 * s, (turn >> 1) & 1);
        tc_fence_after();
        uint32_t r[32];
        tmem_ld32(lanes + 192 + 128 * s + 32 * quarter, r);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(d.empty + 8 * s);
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[e] += __uint_as_float(r[e]);
    }
    return ok;
}
__device__ __forceinline__ void workers_meet() { asm volatile("bar.sync 1, %0;\n" :: "n"(WORKERS) : "memory"); }
// a block's 128 x 128 result by way of shared memory: whole rows of 512 bytes at a time
__device__ __forceinline__ void store_rows(float* staged, const float (&acc)[32], int row, int quarter, float* to, size_t ld, int rows) {
#pragma unroll
    for (int e = 0; e < 32; e += 4)
        *reinterpret_cast<float4*>(staged + row * ROW_OUT + 32 * quarter + e) = make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]);
    workers_meet();
    const int lane = threadIdx.x & 31;
#pragma unroll 4
    for (int r = threadIdx.x >> 5; r < rows; r += WORKERS / 32)
        *reinterpret_cast<float4*>(to + r * ld + 4 * lane) = *reinterpret_cast<const float4*>(staged + r * ROW_OUT + 4 * lane);
}

struct Tail { float pw[C + 4]; uint64_t bars[8]; uint32_t tmem; int first_odd; };      // behind the operands: d^0 .. d^128
template <typename T> constexpr int STATE_SMEM = 1024 + OPERAND + C * PITCH<T> + sizeof(Tail);
constexpr int OUT_SMEM = 1024 + 2 * OPERAND + sizeof(Tail);

// grid (slots, heads, V / VC): sums [head][slot][D][V].  Tensor memory: K^T's parts, two accumulators; shared memory: V's parts, then the result.
template <typename T, bool SILU>
__global__ void __launch_bounds__(THREADS, 1) chunk_state_kernel(const T* __restrict__ in, const Source L, const float* __restrict__ decay, float* __restrict__ sums,
                                                                 const int* __restrict__ seg_q_start, int num_segs, int V, int* __restrict__ error_word) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* rows = base + OPERAND;
    Tail& tail = *reinterpret_cast<Tail*>(rows + C * PITCH<T>);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = (warp & 3) * 32 + lane, quarter = warp >> 2;
    const int slot = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * VC;
    const Chunk ch = chunk_of(slot, seg_q_start, num_segs);
    pdl_trigger();
    if (ch.n == 0) return;
    const T* first = in + (size_t)(ch.qs + ch.t0) * L.ld;
    Tile<T> k, x;
    if (warp < 16) {
        fetch(k, first + L.k + h * D, L.ld, ch.n);
        fetch(x, first + L.v + h * V + col0, L.ld, ch.n);
    }
    const uint32_t bar = smem_u32(tail.bars), ready = bar + 32;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1); mbar_init(bar + 8, 1); mbar_init(bar + 16, 16); mbar_init(bar + 24, 16); mbar_init(ready, WORKERS);
        mbar_init_fence();
        tail.first_odd = C;
    }
    if (warp == 16) tmem_alloc(smem_u32(&tail.tmem), 512);
    else if (threadIdx.x < C) tail.pw[threadIdx.x] = (float)power((double)decay[h], threadIdx.x);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tail.tmem, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const Sums d{tmem, bar, bar + 16};
    int turn = 0;
    if (warp == 16) {
        if (lane == 0) {
            bool ok = mbar_wait(ready, 0);
            tc_fence_after();
            ok = ok && product<true>(d, turn, tmem, smem_u32(base));
            if (!ok) atomicExch(error_word, 71);
        }
    } else {
        stage(rows, k);
        workers_meet();
        float v[32];                                            // row `row` of K^T: 32 tokens' entry `row`, decayed to the chunk's end
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = to_f32(*reinterpret_cast<const T*>(rows + (32 * quarter + j) * PITCH<T> + row * sizeof(T)));
        activate<SILU>(v);
        bool ok = fits(v, largest(v), ADDED);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] *= tail.pw[max(0, ch.n - 1 - 32 * quarter - j)];
        to_tensor(lanes, quarter, v);
        ok &= to_shared<T, SILU>(base, x, ADDED) == C;
        if (!ok) tail.first_odd = 0;
        shared_is_written();
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(ready);
        if (!add_up(d, turn, lanes, quarter, v) && lane == 0) atomicExch(error_word, 72);
        workers_meet();                                         // ... and first_odd is everyone's
        if (tail.first_odd == 0) {                              // the same sums by multiply-adds; V's rows take the place of its parts
            float* values = reinterpret_cast<float*>(base);     // [C][VC]
            for (int id = threadIdx.x; id < ch.n * VC; id += WORKERS) {
                const float x = to_f32(first[(size_t)(id / VC) * L.ld + L.v + h * V + col0 + id % VC]);
                values[id] = SILU ? silu(x) : x;
            }
            workers_meet();
            clear(v);
            for (int j = 0; j < ch.n; ++j) {
                float k = to_f32(first[(size_t)j * L.ld + L.k + h * D + row]);
                if (SILU) k = silu(k);
                k *= tail.pw[ch.n - 1 - j];
                const float* x = values + j * VC + 32 * quarter;
#pragma unroll
                for (int c = 0; c < 32; ++c) v[c] = fmaf(k, x[c], v[c]);
            }
            workers_meet();
        }
        store_rows(reinterpret_cast<float*>(base), v, row, quarter, sums + ((size_t)h * gridDim.x + slot) * D * V + col0, V, D);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// grid (D V / 1024, heads, entries): a thread has four state entries (V is a multiple of 128).  No __restrict__ on sums: the kernel ahead writes them while
// this one already runs, and loads through a pointer that promises to be the only one may be moved ahead of the wait.
// Bound by memory: the sums and the states once each way.  Eight blocks an SM, an entry of one chunk without a loop, and the powers by two threads of a
// block (64-bit products are slow): eight sums in flight a thread left four blocks an SM (64 heads, microseconds there / here: 16 entries of 64 tokens
// 390 / 59, 2,048 tokens beside 18 single ones 496 / 101, 1,000 + 6 x 100 102 / 35, 2,048 25 / 17).
__global__ void __launch_bounds__(256, 8) chunk_scan_kernel(float* sums, const float* __restrict__ decay, float* __restrict__ state, long long state_stride,
                                                            const int* __restrict__ seg_q_start, const int* __restrict__ seg_slot, int slots, int V) {
    constexpr int AT_ONCE = 4;
    __shared__ float less_one[2];
    pdl_trigger();
    const int seg = blockIdx.z, h = blockIdx.y, at = 4 * (blockIdx.x * 256 + threadIdx.x);
    const int qs = seg_q_start[seg], n = seg_q_start[seg + 1] - qs, chunks = (n + C - 1) / C;
    if (chunks == 0) return;
    // d^m - 1: s + s (d^m - 1) keeps the last bits of a decay near 1 (an infinity stays one)
    if (threadIdx.x < 2) less_one[threadIdx.x] = (float)(power((double)decay[h], threadIdx.x ? n - (chunks - 1) * C : C) - 1.0);
    const bool lasts = decay[h] > 0.f;
    auto step_on = [&](float4 s, float m, const float4& t) {
        auto next = [&](float s, float t) { return (fabsf(s) == INFINITY && lasts ? s : fmaf(s, m, s)) + t; };
        return make_float4(next(s.x, t.x), next(s.y, t.y), next(s.z, t.z), next(s.w, t.w));
    };
    float* S = state + (long long)seg_slot[seg] * state_stride + (long long)h * D * V + at;
    float* ws = sums + ((size_t)h * slots + first_slot(qs, seg)) * D * V + at;
    const size_t step = (size_t)D * V;
    const float2 s01 = *reinterpret_cast<const float2*>(S), s23 = *reinterpret_cast<const float2*>(S + 2);
    float4 s = make_float4(s01.x, s01.y, s23.x, s23.y);
    __syncthreads();
    const float whole = less_one[0], last = less_one[1];
    pdl_wait();
    if (chunks == 1) {
        const float4 t = *reinterpret_cast<const float4*>(ws);
        *reinterpret_cast<float4*>(ws) = s;
        s = step_on(s, last, t);
    } else {
        for (int c = 0; c < chunks; c += AT_ONCE) {
            float4 t[AT_ONCE];
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i) if (c + i < chunks) t[i] = *reinterpret_cast<const float4*>(ws + (c + i) * step);
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i) {
                if (c + i >= chunks) break;
                *reinterpret_cast<float4*>(ws + (c + i) * step) = s;
                s = step_on(s, c + i == chunks - 1 ? last : whole, t[i]);
            }
        }
    }
    *reinterpret_cast<float2*>(S) = make_float2(s.x, s.y);
    *reinterpret_cast<float2*>(S + 2) = make_float2(s.z, s.w);
}

// A chunk's tokens one after the other, by the workers: a thread has a quarter of a column of the state in registers.  Queries and keys of eight tokens at a
// time are made once and lie in shared memory, the quarters' sums meet there.  (2,048 tokens and 16 heads with one key beyond the parts: 3,657 us with a column a
// thread, all queries and keys made by each; 184 so, 78 without such a key.  An infinity in every head's state, from which on every chunk is so: 7,800, 398.)
template <typename T, bool SILU>
__device__ __noinline__ void by_token(float* shared, const T* first, const Source L, const float* S0, float decay, int h, int V, int col0, int n, int from,
                                      float* out, int H) {
    constexpr int OCT = 8, ROWS = D / 4;
    float *qs = shared, *ks = qs + OCT * D, *part = ks + OCT * D;       // [token][row] twice; [quarter][token][column]
    const int c = threadIdx.x % VC, quarter = threadIdx.x / VC, r0 = quarter * ROWS;
    float S[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) S[r] = S0[(size_t)(r0 + r) * V + c];
    for (int i0 = 0; i0 < n; i0 += OCT) {
        for (int id = threadIdx.x; id < 2 * OCT * D; id += WORKERS) {
            const int i = i0 + id % (OCT * D) / D;
            const float x = i < n ? to_f32(first[(size_t)i * L.ld + (id < OCT * D ? L.q : L.k) + h * D + id % D]) : 0.f;
            shared[id] = SILU ? silu(x) : x;
        }
        workers_meet();
        for (int i = 0; i < min(OCT, n - i0); ++i) {
            float x = to_f32(first[(size_t)(i0 + i) * L.ld + L.v + h * V + col0 + c]), y = 0.f;
            if (SILU) x = silu(x);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                S[r] = fmaf(S[r], decay, ks[i * D + r0 + r] * x);
                y = fmaf(S[r], qs[i * D + r0 + r], y);
            }
            part[(quarter * OCT + i) * VC + c] = y;
        }
        workers_meet();
        for (int i = quarter; i < min(OCT, n - i0); i += 4)
            if (i0 + i >= from)
                out[(size_t)(i0 + i) * H * V + (size_t)h * V + col0 + c] =
                    (part[i * VC + c] + part[(OCT + i) * VC + c]) + (part[(2 * OCT + i) * VC + c] + part[(3 * OCT + i) * VC + c]);
    }
}

// grid (slots, heads, V / VC); before [head][slot][D][V]: the state before each chunk (no __restrict__ here either).  Tensor memory: Q's parts, then those of the decayed scores; two
// accumulators.  Shared memory: K, then V; S_0, then the result.
template <typename T, bool SILU>
__global__ void __launch_bounds__(THREADS, 1) chunk_out_kernel(const T* __restrict__ in, const Source L, const float* __restrict__ decay, const float* before,
                                                               float* __restrict__ out, const int* __restrict__ seg_q_start, int num_segs, int H, int V,
                                                               int* __restrict__ error_word) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sbuf = base + OPERAND;
    Tail& tail = *reinterpret_cast<Tail*>(base + 2 * OPERAND);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = (warp & 3) * 32 + lane, quarter = warp >> 2;
    const int slot = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * VC;
    const Chunk ch = chunk_of(slot, seg_q_start, num_segs);
    if (ch.n == 0) return;
    const T* first = in + (size_t)(ch.qs + ch.t0) * L.ld;
    const float* S0 = before + ((size_t)h * gridDim.x + slot) * D * V + col0;
    Tile<T> q, k;
    if (warp < 16) {
        fetch(q, first + L.q + h * D, L.ld, ch.n);
        fetch(k, first + L.k + h * D, L.ld, ch.n);
    }
    const uint32_t bar = smem_u32(tail.bars), qk_ready = bar + 32, s_ready = bar + 40, pv_ready = bar + 48;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1); mbar_init(bar + 8, 1); mbar_init(bar + 16, 16); mbar_init(bar + 24, 16);
        mbar_init(qk_ready, WORKERS); mbar_init(s_ready, WORKERS); mbar_init(pv_ready, WORKERS);
        mbar_init_fence();
        tail.first_odd = C;
    }
    if (warp == 16) tmem_alloc(smem_u32(&tail.tmem), 512);
    else if (threadIdx.x <= C) tail.pw[threadIdx.x] = (float)power((double)decay[h], threadIdx.x);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tail.tmem, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const Sums d{tmem, bar, bar + 16};
    int turn = 0;
    if (warp == 16) {
        if (lane == 0) {
            bool ok = mbar_wait(qk_ready, 0);
            ok = ok && product<false>(d, turn, tmem, smem_u32(base));
            ok = ok && mbar_wait(s_ready, 0) && product<true>(d, turn, tmem, smem_u32(sbuf));
            ok = ok && mbar_wait(pv_ready, 0) && product<true>(d, turn, tmem, smem_u32(base));
            if (!ok) atomicExch(error_word, 73);
        }
    } else {
        stage(sbuf, q);
        workers_meet();
        float s[32], o[32];
        load_n(reinterpret_cast<const T*>(sbuf + row * PITCH<T> + 32 * quarter * sizeof(T)), s);
        activate<SILU>(s);
        int odd = fits(s, largest(s), SCORED) ? C : row;
        to_tensor(lanes, quarter, s);
        odd = min(odd, to_shared<T, SILU, true>(base, k, SCORED));
        shared_is_written();
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(qk_ready);
        fetch(k, first + L.v + h * V + col0, L.ld, ch.n);       // V
        pdl_wait();
        {
            Tile<float> t;
            fetch(t, S0, V, D);
            workers_meet();                                     // everyone has its row of Q
            if (to_shared<float, false>(sbuf, t, STATE) < C) odd = 0;
        }
        shared_is_written();
        mbar_arrive(s_ready);
        bool ok = add_up(d, turn, lanes, quarter, s);           // the scores; K is done with
        odd = min(odd, to_shared<T, SILU>(base, k, ADDED));
        shared_is_written();
        if (odd < C) atomicMin(&tail.first_odd, odd);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const int back = row - 32 * quarter - j;
            s[j] = back >= 0 ? s[j] * tail.pw[max(0, back)] : 0.f;
        }
        ok &= add_up(d, turn, lanes, quarter, o);               // Q S_0; Q is done with
        tc_fence_after();
        to_tensor(lanes, quarter, s);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(pv_ready);
        ok &= add_up(d, turn, lanes, quarter, s);
        if (!ok && lane == 0) atomicExch(error_word, 74);
        const float p = tail.pw[row + 1];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = fmaf(p, o[e], s[e]);
        store_rows(reinterpret_cast<float*>(sbuf), o, row, quarter, out + (size_t)(ch.qs + ch.t0) * H * V + (size_t)h * V + col0, (size_t)H * V, ch.n);
        workers_meet();
        const int from = tail.first_odd;
        if (from < ch.n) by_token<T, SILU>(reinterpret_cast<float*>(base), first, L, S0, decay[h], h, V, col0, ch.n, from, out + (size_t)(ch.qs + ch.t0) * H * V, H);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

template <typename K, typename... A>
int launch(K kernel, dim3 grid, int threads, int smem, bool early, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename T, bool SILU>
int run(const T* in, const Source& L, float* sums, const float* decay, float* state, long long state_stride, float* out, const int* seg_q_start, const int* seg_slot,
        int T_, int num_segs, int H, int D_, int V, int* error_word, cudaStream_t stream) {
    if (num_segs == 0 || T_ == 0) return 0;
    if (D_ != D || V % VC || H > 65535 || num_segs > 65535 || state_stride % 2 || (uintptr_t)state % 8) return -2;
    if (L.ld % Vec16<T>::N || (uintptr_t)in % 16 || (uintptr_t)sums % 16 || (uintptr_t)out % 16) return -2;      // every head starts on a multiple of 128 entries
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<T, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, STATE_SMEM<T>);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_out_kernel<T, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int slots = T_ / C + num_segs;
    int rc = launch(chunk_state_kernel<T, SILU>, dim3(slots, H, V / VC), THREADS, STATE_SMEM<T>, false, stream, in, L, decay, sums, seg_q_start, num_segs, V, error_word);
    if (rc == 0) rc = launch(chunk_scan_kernel, dim3(D * V / 1024, H, num_segs), 256, 0, true, stream, sums, decay, state, state_stride, seg_q_start, seg_slot, slots, V);
    if (rc == 0) rc = launch(chunk_out_kernel<T, SILU>, dim3(slots, H, V / VC), THREADS, OUT_SMEM, true, stream, in, L, decay, (const float*)sums, out, seg_q_start,
                             num_segs, H, V, error_word);
    return rc;
}

}  // namespace

// floats of scratch for T tokens in num_segs entries
MI_EXPORT long long mi_chunk_floats(int T_, int num_segs, int H, int D_, int V) { return (long long)(T_ / C + num_segs) * H * D_ * V; }

// rows [T, 2 H D + H V] float32 = q | k | v as they enter the recurrence; decay [H]; scratch: mi_chunk_floats; out float32 [T, H V]
MI_EXPORT int mi_constant_chunks(const float* rows, float* scratch, const float* decay, float* state, long long state_stride, float* out, const int* seg_q_start,
                                 const int* seg_slot, int T_, int num_segs, int H, int D_, int V, int* error_word, cudaStream_t stream) {
    return run<float, false>(rows, Source{2 * H * D_ + H * V, 0, H * D_, 2 * H * D_}, scratch, decay, state, state_stride, out, seg_q_start, seg_slot, T_, num_segs,
                             H, D_, V, error_word, stream);
}

// p [T, ldp] bfloat16 = q | k | v before silu; otherwise as mi_constant_chunks
MI_EXPORT int mi_lightning_chunks(const void* p, int ldp, float* scratch, const float* decay, float* state, long long state_stride, float* out,
                                  const int* seg_q_start, const int* seg_slot, int T_, int num_segs, int H, int D_, int V, int* error_word, cudaStream_t stream) {
    return run<__nv_bfloat16, true>((const __nv_bfloat16*)p, Source{ldp, 0, H * D_, 2 * H * D_}, scratch, decay, state, state_stride, out, seg_q_start, seg_slot, T_,
                                    num_segs, H, D_, V, error_word, stream);
}
