// True 32-bit matrix product C[M,N] = A[M,K] * W[N,K]^T on the tensor cores: every float32 is cut exactly into three bfloat16 numbers, six products of
// parts stand for one product (split3.cuh).
//
// Exactness.  The tensor core cuts off instead of rounding when it adds, so no sum stays there for long: 64 of K (24 instructions, the small
// products first) go into a fresh accumulator in tensor memory, and the epilogue warps add it in float32, rounded to nearest, to sums that they
// keep in registers.  The order depends on N and K alone (segments of K by segments(), 64 of K at a time within one), not on M or on the tile: a
// token's numbers are the same bits whatever else is in the batch.
// Values that three bfloat16 numbers do not hold: a row of A or W whose largest magnitude is not in [2^-60, 2^60] (infinities, NaN, numbers near
// the ends of float32's range; a row of zeros is fine) has its results computed over again by float32 multiply-adds at the end of a tile.
// The promise is one about vectors: an error of some 2^-23 of |x| |w|, as float32 sums of any order give it.  It is not one about sum |x_k w_k|: a number
// below 2^-110 in a row that also holds large ones keeps what is above 2^-133 of it.
//
// W is the tensor core's A operand (128 of its rows a tile, read from tensor memory), tokens are its N side (NT = 32, 64 or 128 of them):
//   warp 0       W as it lies, float32, by TMA into a ring of stages of 64 of K (starts before the kernel ahead is done)
//   warp 1       the MMAs of a stage: 6 products x 4 steps of K
//   warps 2-9    two groups that take turns: a thread reads a row's 64 numbers of a stage and writes their three parts to tensor memory
//   warps 10-17  the sums: a thread has one row of W and half of the tile's tokens
//   warp 18      the tokens' parts, made once by split_rows_kernel, by TMA
// The rows' largest magnitudes go from the converting to the adding warps in two slots that take turns and are not handed back: an item has at least
// three stages (tc_segments in gemm_f32.cu), so both groups have converted a stage that lies five or more behind item i before they end item i + 2, and
// one four stages earlier, of a later item than i, was added up by then.
// Tensor memory: two stages of W's parts (2 x 96 columns) and two accumulators (2 x NT columns).
//
// Against gemm_f32.cu's multiply-adds (microseconds; N x K = 6,144 x 2,560, 2,560 x 4,096, 19,456 x 2,560, 2,560 x 9,728): 501 rows 492, 332, 1,355, 668
// -> 95, 78, 273, 144; 48 rows 107, 87, 301, 154 -> 30, 25, 111, 47; one row 69, 45, 138, 81 -> 29, 26, 107, 41.  Error against 64 bits (2-norm)
// 4.1e-7 .. 6.5e-7 -> 1.0e-7 .. 1.4e-7.  At 501 rows the tensor pipe is active 64 % of the time and a fifth of it goes to the last wave; a stage
// brings 80 KB for 1,536 clocks of products, close to what a block can load (53 bytes a clock).  With one row a stage of W is 1,128 clocks
// of products (an instruction of 32 tokens takes as long as one of 64).
#include "split3.cuh"
#include <algorithm>

using namespace mi;
using namespace mi::sm100;
using namespace mi::split3;

namespace {

constexpr int BN = 128, BK = 64;
constexpr int W_BOX = BN * 32 * 4, W_STAGE = 2 * W_BOX;         // a box is 32 floats (128 bytes) of 128 rows
constexpr int THREADS = 32 * 19;
constexpr int A_COLS = PARTS * BK / 2;                          // tensor-memory columns of a stage of W's parts

constexpr int x_stage(int nt) { return PARTS * nt * BK * 2; }
constexpr int w_stages(int nt) { return nt == 128 ? 2 : nt == 64 ? 4 : 5; }
constexpr int x_stages(int nt) { return nt == 128 ? 3 : nt == 64 ? 3 : 4; }
constexpr int smem_bytes(int nt) { return 1024 + w_stages(nt) * W_STAGE + x_stages(nt) * x_stage(nt) + 2 * 2 * BN * 4 + 512; }

constexpr float LEAST = 0x1p-60f, MOST = 0x1p60f;               // of a row's largest magnitude

// parts[3][M][ldp] of A [M, K]; columns K .. ldp are zeros.  flag[m]: the row does not fit three bfloat16 numbers.  One block a row.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, int lda, __nv_bfloat16* __restrict__ parts, int ldp,
                                                         unsigned char* __restrict__ flag, int M, int K, int vec) {
    pdl_trigger();
    const int m = blockIdx.x;
    const float* row = A + (size_t)m * lda;
    const size_t plane = (size_t)M * ldp;
    float mx = 0.f;
    bool bad = false;
    for (int k = 4 * threadIdx.x; k < ldp; k += 1024) {
        float v[4];
        if (vec && k + 4 <= K) load16(row + k, v);
        else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = k + e < K ? row[k + e] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) { mx = fmaxf(mx, fabsf(v[e])); bad |= !(fabsf(v[e]) <= MOST); }
#pragma unroll
        for (int p = 0; p < PARTS; ++p) {
            const uint2 w = make_uint2(take_part(v[0], v[1]), take_part(v[2], v[3]));
            *reinterpret_cast<uint2*>(parts + p * plane + (size_t)m * ldp + k) = w;
        }
    }
    const int any_bad = __syncthreads_or(bad), any = __syncthreads_or(mx > 0.f), enough = __syncthreads_or(mx >= LEAST);
    if (threadIdx.x == 0) flag[m] = any_bad || (any && !enough);
}

struct Item { int n0, m0, k_first, k_end, seg, stages; };

struct Shape {
    int M, N, K, lda, ldp, ldc;
    int n_tiles, m_tiles, segments, segment;
};

// items: tokens fastest, so that the blocks that run together share W's tiles in L2
template <int NT>
__device__ __forceinline__ Item item_of(const Shape& sh, int i) {
    Item it;
    const int mt = i % sh.m_tiles, rest = i / sh.m_tiles;
    it.seg = rest % sh.segments;
    it.n0 = rest / sh.segments * BN;
    it.m0 = mt * NT;
    it.k_first = it.seg * sh.segment;
    it.k_end = it.seg + 1 == sh.segments ? sh.K : it.k_first + sh.segment;
    it.stages = (it.k_end - it.k_first + BK - 1) / BK;
    return it;
}

// x . w over [k0, k1) by multiply-adds for R of the warp's rows of W, by the whole warp, a lane every 32nd of K; lane r stores row r's
template <int R>
__device__ __forceinline__ void plain_rows(const float* x, const float* w, int K, int k0, int k1, unsigned& rows, float* to) {
    const int lane = threadIdx.x & 31;
    int r[R];
    float sum[R];
#pragma unroll
    for (int e = 0; e < R; ++e) { r[e] = __ffs(rows) - 1; rows &= rows - 1; sum[e] = 0.f; }
#pragma unroll 4
    for (int k = k0 + lane; k < k1; k += 32) {
        const float v = x[k];
#pragma unroll
        for (int e = 0; e < R; ++e) sum[e] = fmaf(v, w[(size_t)r[e] * K + k], sum[e]);
    }
#pragma unroll
    for (int e = 0; e < R; ++e) {
        sum[e] = warp_sum(sum[e]);
        if (lane == r[e]) *to = sum[e];
    }
}
// ... for all of `rows` (w: the first of the 32).  A call, which leaves the main loop its registers (inlined: 3 to 5 % of a product).  With a lane a
// result 501 rows of 6,144 x 2,560 took 1,420 us beside one row of W beyond the parts; so 320 (multiply-adds alone 489).
__device__ __noinline__ void plain_sums(const float* x, const float* w, int K, int k0, int k1, unsigned rows, float* to) {
    while (__popc(rows) >= 4) plain_rows<4>(x, w, K, k0, k1, rows, to);
    while (rows) plain_rows<1>(x, w, K, k0, k1, rows, to);
}

template <int NT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const Shape sh, const float* __restrict__ A,
                   const float* __restrict__ W, const unsigned char* token_flag, float* __restrict__ out, int* __restrict__ error_word) {
    constexpr int WS = w_stages(NT), XS = x_stages(NT), X_STAGE = x_stage(NT), HALF = NT / 2;
    constexpr uint32_t TMEM_COLS = 512, D_COL = 2 * A_COLS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* row_max = reinterpret_cast<float*>(base + WS * W_STAGE + XS * X_STAGE);          // [items in turn][conversion groups][BN]
    uint64_t* bars = reinterpret_cast<uint64_t*>(row_max + 2 * 2 * BN);
    const uint32_t sW = smem_u32(base), sX = sW + WS * W_STAGE;
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * WS, x_full = w_empty + 8 * WS, x_empty = x_full + 8 * XS,
                   a_full = x_empty + 8 * XS, a_empty = a_full + 16, d_full = a_empty + 16, d_empty = d_full + 16, m_full = d_empty + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * WS + 2 * XS + 10);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < WS; ++s) { mbar_init(w_full + 8 * s, 1); mbar_init(w_empty + 8 * s, 4); }
        for (int s = 0; s < XS; ++s) { mbar_init(x_full + 8 * s, 1); mbar_init(x_empty + 8 * s, 1); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(a_full + 8 * s, 4); mbar_init(a_empty + 8 * s, 1); mbar_init(d_full + 8 * s, 1); mbar_init(d_empty + 8 * s, 8);
            mbar_init(m_full + 8 * s, 8);
        }
        mbar_init_fence();
        tma_prefetch_desc(&wmap); tma_prefetch_desc(&xmap);
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int items = sh.n_tiles * sh.m_tiles * sh.segments;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0, turn = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item it = item_of<NT>(sh, i);
                for (int k = 0; k < it.stages; ++k) {
                    if (turn > 0 && !mbar_wait(w_empty + 8 * s, (turn - 1) & 1)) { atomicExch(error_word, 81); ok = false; break; }
                    mbar_expect_tx(w_full + 8 * s, W_STAGE);
                    const int x = it.k_first + k * BK;
                    tma_load_2d(sW + s * W_STAGE, &wmap, x, it.n0, w_full + 8 * s);
                    tma_load_2d(sW + s * W_STAGE + W_BOX, &wmap, x + 32, it.n0, w_full + 8 * s);
                    if (++s == WS) { s = 0; ++turn; }
                }
            }
        }
    } else if (warp == 18) {
        pdl_wait();
        if (lane == 0) {
            int s = 0, turn = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item it = item_of<NT>(sh, i);
                for (int k = 0; k < it.stages; ++k) {
                    if (turn > 0 && !mbar_wait(x_empty + 8 * s, (turn - 1) & 1)) { atomicExch(error_word, 82); ok = false; break; }
                    mbar_expect_tx(x_full + 8 * s, X_STAGE);
#pragma unroll
                    for (int p = 0; p < PARTS; ++p)
                        tma_load_2d(sX + s * X_STAGE + p * (NT * 128), &xmap, it.k_first + k * BK, p * sh.M + it.m0, x_full + 8 * s);
                    if (++s == XS) { s = 0; ++turn; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16(BN, NT, false);
            int n = 0, xs = 0, x_turn = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item it = item_of<NT>(sh, i);
                for (int k = 0; k < it.stages; ++k, ++n) {
                    const int b = n & 1;
                    if (n >= 2 && !mbar_spin(d_empty + 8 * b, ((n >> 1) - 1) & 1)) { atomicExch(error_word, 83); ok = false; break; }
                    if (!mbar_spin(x_full + 8 * xs, x_turn & 1)) { atomicExch(error_word, 84); ok = false; break; }
                    if (!mbar_spin(a_full + 8 * b, (n >> 1) & 1)) { atomicExch(error_word, 85); ok = false; break; }
                    tc_fence_after();
                    const uint32_t d = tmem + D_COL + b * NT, a = tmem + b * A_COLS;
                    const uint64_t x = umma_desc_sw128(sX + xs * X_STAGE, 16, 1024);
#pragma unroll
                    for (int p = 0; p < PRODUCTS; ++p)
#pragma unroll
                        for (int ks = 0; ks < BK / 16; ++ks)
                            umma_ts(d, a + PART_A[p] * (BK / 2) + ks * 8, x + ((PART_B[p] * NT * 128 + ks * 32) >> 4), idesc, (p | ks) != 0);
                    umma_commit(a_empty + 8 * b);
                    umma_commit(x_empty + 8 * xs);
                    umma_commit(d_full + 8 * b);
                    if (++xs == XS) { xs = 0; ++x_turn; }
                }
            }
        }
    } else if (warp < 10) {
        // ---------------- W's parts: group g takes the stages n with n % 2 == g
        const int g = (warp - 2) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + g * A_COLS;
        int n = 0, s = 0, turn = 0, turn_of_item = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++turn_of_item) {
            const Item it = item_of<NT>(sh, i);
            __nv_bfloat162 mx = __floats2bfloat162_rn(0.f, 0.f);
            for (int k = 0; k < it.stages; ++k, ++n) {
                if ((n & 1) == g) {
                    if (!mbar_wait(w_full + 8 * s, turn & 1)) { atomicExch(error_word, 86); ok = false; break; }
                    if (n >= 2) {
                        if (!mbar_wait(a_empty + 8 * g, ((n >> 1) - 1) & 1)) { atomicExch(error_word, 87); ok = false; break; }
                        tc_fence_after();
                    }
                    const unsigned char* at = base + s * W_STAGE + row * 128;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v[32];
#pragma unroll
                        for (int c = 0; c < 8; ++c) load16(reinterpret_cast<const float*>(at + h * W_BOX + ((c ^ (row & 7)) * 16)), v + 4 * c);
                        if (h == 1) { __syncwarp(); if (lane == 0) mbar_arrive(w_empty + 8 * s); }
#pragma unroll
                        for (int p = 0; p < PARTS; ++p) {
                            uint32_t w[16];
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                w[e] = take_part(v[2 * e], v[2 * e + 1]);
                                if (p == 0) mx = __hmax2_nan(mx, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[e])));
                            }
                            tmem_st16(lanes + p * (BK / 2) + h * 16, w);
                        }
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full + 8 * g);
                }
                if (++s == WS) { s = 0; ++turn; }
            }
            const float lo = __low2float(mx), hi = __high2float(mx);
            row_max[((turn_of_item & 1) * 2 + g) * BN + row] = lo == lo && hi == hi ? fmaxf(lo, hi) : INFINITY;
            __syncwarp();
            if (lane == 0) mbar_arrive(m_full + 8 * (turn_of_item & 1));
        }
    } else {
        // ---------------- sums
        const int half = (warp - 10) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + D_COL + half * HALF;
        pdl_wait();
        int n = 0, turn_of_item = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++turn_of_item) {
            const Item it = item_of<NT>(sh, i);
            float acc[HALF];
#pragma unroll
            for (int c = 0; c < HALF; ++c) acc[c] = 0.f;
            for (int k = 0; k < it.stages; ++k, ++n) {
                const int b = n & 1;
                if (!mbar_wait(d_full + 8 * b, (n >> 1) & 1)) { atomicExch(error_word, 88); ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < HALF; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(lanes + b * NT + c, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[c + e] += __uint_as_float(r[e]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty + 8 * b);
            }
            if (!ok) break;
            const int nrow = it.n0 + row, m_first = it.m0 + half * HALF;
            float* to = out + ((size_t)it.seg * sh.M + m_first) * sh.ldc + nrow;
#pragma unroll
            for (int c = 0; c < HALF; ++c)
                if (nrow < sh.N && m_first + c < sh.M) to[(size_t)c * sh.ldc] = acc[c];
            if (!mbar_wait(m_full + 8 * (turn_of_item & 1), (turn_of_item >> 1) & 1)) { atomicExch(error_word, 89); ok = false; break; }
            const float* rm = row_max + (turn_of_item & 1) * 2 * BN + row;
            const float most = fmaxf(rm[0], rm[BN]);
            const bool odd_row = !(most <= MOST) || (most > 0.f && most < LEAST);
            const int mine = m_first + lane;
            const unsigned odd0 = __ballot_sync(0xffffffffu, lane < HALF && mine < sh.M && token_flag[mine]);
            const unsigned odd1 = HALF > 32 ? __ballot_sync(0xffffffffu, mine + 32 < sh.M && token_flag[mine + 32]) : 0u;
            if (__builtin_expect(__any_sync(0xffffffffu, odd_row) || odd0 || odd1, 0)) {
                const unsigned rows = __ballot_sync(0xffffffffu, nrow < sh.N), odd_rows = __ballot_sync(0xffffffffu, odd_row) & rows;
                const float* w = W + (size_t)(nrow - lane) * sh.K;
                for (int c = 0; c < HALF && m_first + c < sh.M; ++c) {
                    const bool odd_token = ((c < 32 ? odd0 >> c : odd1 >> (c - 32)) & 1) != 0;
                    plain_sums(A + (size_t)(m_first + c) * sh.lda, w, sh.K, it.k_first, it.k_end, odd_token ? rows : odd_rows, to + (size_t)c * sh.ldc);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

template <int NT>
int launch(const CUtensorMap& wmap, const CUtensorMap& xmap, Shape sh, const float* A, const float* W, const unsigned char* flag, float* out, int* error_word,
           cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(NT));
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    sh.m_tiles = (sh.M + NT - 1) / NT;
    const int items = sh.n_tiles * sh.m_tiles * sh.segments;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(std::min(items, device_sms()));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes(NT);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<NT>, wmap, xmap, sh, A, W, flag, out, error_word);
}

bool map_2d(CUtensorMap* m, CUtensorMapDataType type, int size, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols) {
    auto fn = sm100_host::encoder();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * size};
    const cuuint32_t box[2] = {box_cols, box_rows}, estr[2] = {1, 1};
    return fn(m, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int round_up(int v, int to) { return (v + to - 1) / to * to; }

}  // namespace

namespace mi {

// bytes of the tokens' parts and flags
long long gemm_f32_tc_parts(int M, int K) { return (long long)PARTS * M * round_up(K, BK) * 2 + round_up(M, 16); }        // a multiple of 16

// Which number of tokens a tile: the waves of blocks times a stage's MMAs (an instruction of 32 or 64 tokens takes 47 clocks, one of 128 takes 64)
int gemm_f32_tc_tile(int M, int N, int S) {
    const long long n = (long long)((N + BN - 1) / BN) * S;
    const int sms = device_sms();
    auto cost = [&](int nt, int clocks) { return (n * ((M + nt - 1) / nt) + sms - 1) / sms * clocks; };
    if (M <= 32) return 32;
    return cost(128, 64) <= cost(64, 47) ? 128 : 64;
}

int gemm_f32_tc(const float* A, int lda, const float* W, float* out, int ldc, int M, int N, int K, int S, int segment, int nt, void* parts_ws,
                int* error_word, cudaStream_t stream) {
    const int ldp = round_up(K, BK);
    __nv_bfloat16* parts = reinterpret_cast<__nv_bfloat16*>(parts_ws);
    unsigned char* flag = reinterpret_cast<unsigned char*>(parts + (size_t)PARTS * M * ldp);
    CUtensorMap wmap, xmap;
    if (!map_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, W, N, K, K, BN, 32) ||
        !map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, parts, (uint64_t)PARTS * M, ldp, ldp, nt, BK)) return -2;
    const int vec = lda % 4 == 0 && (uintptr_t)A % 16 == 0;
    split_rows_kernel<<<M, 256, 0, stream>>>(A, lda, parts, ldp, flag, M, K, vec);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    Shape sh{M, N, K, lda, ldp, ldc, (N + BN - 1) / BN, 0, S, segment};
    if (nt == 128) return launch<128>(wmap, xmap, sh, A, W, flag, out, error_word, stream);
    if (nt == 64) return launch<64>(wmap, xmap, sh, A, W, flag, out, error_word, stream);
    return launch<32>(wmap, xmap, sh, A, W, flag, out, error_word, stream);
}

}  // namespace mi
