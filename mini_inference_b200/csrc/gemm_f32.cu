// True 32-bit matrix product C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores: IEEE float32
// multiply-add, no TF32, no reduced-precision staging.  It serves the float32 path of the
// whole model, whose purpose is to show faults that bfloat16 rounding hides, so the summation
// order is fixed: K is cut into segments by a rule on N and K alone; in a segment every output
// element adds its products over the even k and over the odd k in ascending order and then those
// two sums, and the segments' sums are added in order.  Neither M nor the tile that computes an
// element changes a bit, hence a token's logits do not depend on what else is in the batch.
// (The reference reaches float32 by running its library path with DTYPE=float32 on the CPU,
// tests/test_batching.py:57; it has no float32 GPU path.)
//
// Matrices of a million entries and more go to the tensor cores (gemm_f32_tc.cu: the same precision, an order of its own).  The
// kernel here is bound by the float32 FMA rate (74 TFLOP/s) for many rows, by the weight's bytes for few.  The
// packed two-float multiply-add of this architecture does two neighbouring k per instruction:
// both operands lie along K as they are stored, so tiles go to shared memory untransposed by
// cp.async (16 bytes, or 4 where rows do not start on 16) and pairs need no shuffling.  Rows are
// padded by 16 bytes: the eight rows that a quarter warp reads lie in different banks.  501 rows,
// N x K = 6,144 x 2,560, 2,560 x 4,096, 19,456 x 2,560, 2,560 x 9,728: 482, 334, 1,357, 672 us (32 to
// 37 TFLOP/s; a 64 x 64 tile with scalar multiply-adds and no pipeline took 862, 737, 2,366, 1,727).
// The packed multiply-add pipe is active 59 % of the time; tiles of 8 x 4 or 4 x 8 a thread with twice
// the warps, steps of 16 of K, and scalar multiply-adds (33 TFLOP/s at 3,000 rows against 37) are slower.
#include "common.cuh"

namespace mi {                                  // gemm_f32_tc.cu: the same product on the tensor cores
long long gemm_f32_tc_parts(int M, int K);
int gemm_f32_tc_tile(int M, int N, int S);
int gemm_f32_tc(const float* A, int lda, const float* W, float* out, int ldc, int M, int N, int K, int S, int segment, int nt, void* parts,
                int* error_word, cudaStream_t stream);
}

namespace {

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" :: "r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

constexpr int BK_MAX = 64;

// A warp's lanes are 4 (rows) x 8 (columns); a lane owns TM x TN outputs, rows 4 apart, columns 8 apart, so a warp covers
// 4 TM x 8 TN and the block WM x WN of those.
template <int TM, int TN, int WM, int WN, int BK, int STAGES>
struct Tile {
    static constexpr int BM = 4 * TM * WM, BN = 8 * TN * WN, THREADS = 32 * WM * WN, LD = BK + 4;
    static constexpr int STAGE = (BM + BN) * LD, SMEM = STAGES * STAGE * 4;
};

// grid (column tiles, row tiles, segments of K); segment z writes out + z * M * ldc
template <int TM, int TN, int WM, int WN, int BK, int STAGES, bool VEC>
__global__ void __launch_bounds__(32 * WM * WN) gemm_f32_nt_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W,
                                                                   float* __restrict__ out, int ldc, int M, int N, int K, int segment) {
    using L = Tile<TM, TN, WM, WN, BK, STAGES>;
    extern __shared__ __align__(16) float smem[];
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * L::BM, n0 = blockIdx.x * L::BN;
    const int row_a = (warp / WN) * 4 * TM + (lane >> 3), row_b = (warp % WN) * 8 * TN + (lane & 7);
    const int k_first = blockIdx.z * segment, k_end = min(K, k_first + segment);
    const int steps = (k_end - k_first + BK - 1) / BK;

    auto load = [&](int step) {
        const uint32_t dst = s0 + (step % STAGES) * L::STAGE * 4;
        const int k0 = k_first + step * BK;
        constexpr int PIECE = VEC ? 4 : 1, PER_ROW = BK / PIECE;
        for (int id = tid; id < (L::BM + L::BN) * PER_ROW; id += L::THREADS) {
            const int r = id / PER_ROW, k = k0 + id % PER_ROW * PIECE;
            const bool is_a = r < L::BM;
            const int g = is_a ? m0 + r : n0 + r - L::BM;
            const bool ok = k < k_end && g < (is_a ? M : N);
            const float* src = !ok ? A : is_a ? A + (size_t)g * lda + k : W + (size_t)g * K + k;
            const uint32_t at = dst + (r * L::LD + id % PER_ROW * PIECE) * 4;
            if (VEC) cp16(at, src, ok); else cp4(at, src, ok);
        }
    };
    float2 acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" :: "n"(STAGES - 2) : "memory");
        __syncthreads();                       // the stage is there for everyone, and everyone is done with the one loaded next
        if (step + STAGES - 1 < steps) load(step + STAGES - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* a_s = smem + (step % STAGES) * L::STAGE + row_a * L::LD;
        const float* b_s = smem + (step % STAGES) * L::STAGE + (L::BM + row_b) * L::LD;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float4 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(b_s + 8 * j * L::LD + kk);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + 4 * i * L::LD + kk);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(a.x, a.y), make_float2(b[j].x, b[j].y), acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(a.z, a.w), make_float2(b[j].z, b[j].w), acc[i][j]);
            }
        }
    }
    out += (size_t)blockIdx.z * M * ldc;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + row_a + 4 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + row_b + 8 * j;
            if (n < N) out[(size_t)m * ldc + n] = acc[i][j].x + acc[i][j].y;
        }
    }
}

// C = the segments' sums, added in order; ws [S, M, N].  VEC neighbouring columns a thread.
template <int VEC>
__global__ void add_segments_kernel(const float* __restrict__ ws, float* __restrict__ C, int ldc, int M, int N, int S) {
    const size_t plane = (size_t)M * N;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC; i < plane; i += (size_t)gridDim.x * blockDim.x * VEC) {
        float v[VEC];
        if constexpr (VEC == 4) mi::load16(ws + i, v); else v[0] = ws[i];
        for (int s = 1; s < S; ++s) {
            float u[VEC];
            if constexpr (VEC == 4) mi::load16(ws + s * plane + i, u); else u[0] = ws[s * plane + i];
#pragma unroll
            for (int e = 0; e < VEC; ++e) v[e] += u[e];
        }
        float* to = C + i / N * ldc + i % N;
        if constexpr (VEC == 4) *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]); else *to = v[0];
    }
}

template <int TM, int TN, int WM, int WN, int BK, int STAGES>
int launch(const float* A, int lda, const float* W, float* out, int ldc, int M, int N, int K, int S, int segment, cudaStream_t stream) {
    using L = Tile<TM, TN, WM, WN, BK, STAGES>;
    static_assert(BK_MAX % BK == 0, "a segment is a whole number of every tile's steps");
    const dim3 grid((N + L::BN - 1) / L::BN, (M + L::BM - 1) / L::BM, S);
    const bool vec = K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
    auto kernel = vec ? gemm_f32_nt_kernel<TM, TN, WM, WN, BK, STAGES, true> : gemm_f32_nt_kernel<TM, TN, WM, WN, BK, STAGES, false>;
    static bool configured[2] = {false, false};
    if (!configured[vec]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured[vec] = true;
    }
    kernel<<<grid, L::THREADS, L::SMEM, stream>>>(A, lda, W, out, ldc, M, N, K, segment);
    return (int)cudaGetLastError();
}

// Narrow products have few column tiles: their K is cut until a row tile alone gives about one block per SM, in pieces of at least
// 1,024 (501 rows, N 2,560, K 9,728 in one segment: 80 blocks of 128 x 128, 1,093 us; in 8: 672 us).
int segments(int N, int K, int* segment) {
    const int tiles = (N + 127) / 128;
    int S = K / 1024 < 8 ? K / 1024 : 8;
    if (S > 160 / tiles) S = 160 / tiles;
    if (S < 1) S = 1;
    *segment = K < BK_MAX ? BK_MAX : ((K + S - 1) / S + BK_MAX - 1) / BK_MAX * BK_MAX;
    return (K + *segment - 1) / *segment > 1 ? (K + *segment - 1) / *segment : 1;
}

constexpr int ROWS_AT_ONCE = 1024;             // rows per pass of a product that needs a workspace: bounds it

// Which products run on the tensor cores: by N and K alone (and that W's rows start on 16 bytes, as TMA reads them), so that a row's bits do not
// depend on M.  Smaller matrices are a few tiles for 148 blocks and keep the multiply-adds.  At the low end of N and K a few rows pay for the many
// (microseconds by multiply-adds / here: 2,048 x 512 one row 8.4 / 14.9, 33 rows 27 / 16, 1,000 rows 63 / 20; 128 x 8,192 18 / 27, 24 / 29, 87 / 38;
// 1,024 x 1,024 15.0 / 16.5, 17.1 / 17.5, 81 / 23; from 256 x 4,096 on one row is faster here too); the error is a third everywhere.
bool on_tensor_cores(int N, int K) { return K % 4 == 0 && K >= 512 && N >= 128 && (long long)N * K >= 1 << 20; }

// Their K is cut until a tile of tokens alone gives about one block per SM, in pieces of at least 512 (148 is a
// constant of the format here, like 512: a row's bits go with it).  The last piece takes the rest, at least three stages of 64: gemm_f32_tc.cu hands its
// rows' maxima over between items of that length only.
int tc_segments(int N, int K, int* segment) {
    int S = K / 512 < 8 ? K / 512 : 8;
    if (S > 148 / ((N + 127) / 128)) S = 148 / ((N + 127) / 128);
    if (S < 1) S = 1;
    *segment = ((K + S - 1) / S + BK_MAX - 1) / BK_MAX * BK_MAX;
    S = (K + *segment - 1) / *segment;
    return S > 1 && K - (S - 1) * *segment <= 2 * BK_MAX ? S - 1 : S;
}

int add_up(const float* ws, float* C, int ldc, int M, int N, int S, cudaStream_t stream) {
    const bool vec = N % 4 == 0 && ldc % 4 == 0 && (uintptr_t)C % 16 == 0 && (uintptr_t)ws % 16 == 0;
    const size_t n = ((size_t)M * N + (vec ? 3 : 0)) / (vec ? 4 : 1);
    const int blocks = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
    if (vec) add_segments_kernel<4><<<blocks, 256, 0, stream>>>(ws, C, ldc, M, N, S);
    else add_segments_kernel<1><<<blocks, 256, 0, stream>>>(ws, C, ldc, M, N, S);
    return (int)cudaGetLastError();
}

// The tile whose last wave wastes least, by the area an SM works through (relative rates measured with every SM full).
int pick_tile(int M, int N, int S) {
    static const int bm[5] = {128, 64, 64, 32, 16}, bn[5] = {128, 128, 64, 64, 16};
    static const float rate[5] = {1.f, 1.f, 0.94f, 0.8f, 0.3f};
    int best = 0;
    float least = 0.f;
    const int sms = mi::device_sms();
    for (int t = 0; t < 5; ++t) {
        const long long blocks = (long long)((M + bm[t] - 1) / bm[t]) * ((N + bn[t] - 1) / bn[t]) * S;
        const float cost = (float)((blocks + sms - 1) / sms) * bm[t] * bn[t] / rate[t];
        if (t == 0 || cost < least) { least = cost; best = t; }
    }
    return best;
}

int run_tile(const float* A, int lda, const float* W, float* out, int ldc, int M, int N, int K, int S, int segment, int tile, cudaStream_t stream) {
    switch (tile) {
        case 0: return launch<8, 8, 4, 2, 32, 3>(A, lda, W, out, ldc, M, N, K, S, segment, stream);
        case 1: return launch<8, 8, 2, 2, 32, 3>(A, lda, W, out, ldc, M, N, K, S, segment, stream);
        case 2: return launch<8, 8, 2, 1, 32, 3>(A, lda, W, out, ldc, M, N, K, S, segment, stream);
        case 3: return launch<8, 4, 1, 2, 32, 4>(A, lda, W, out, ldc, M, N, K, S, segment, stream);
        default: return launch<2, 2, 2, 1, 64, 6>(A, lda, W, out, ldc, M, N, K, S, segment, stream);
    }
}

}  // namespace

// floats of workspace that a product of this shape needs (0: none)
MI_EXPORT long long mi_gemm_f32_workspace(int M, int N, int K) {
    int segment;
    const int rows = M < ROWS_AT_ONCE ? M : ROWS_AT_ONCE;
    int S = segments(N, K, &segment);
    const long long plain = S > 1 ? (long long)S * rows * N : 0;      // also for a W of this shape that does not start on 16 bytes
    if (!on_tensor_cores(N, K)) return plain;
    S = tc_segments(N, K, &segment);
    const long long parts = mi::gemm_f32_tc_parts(rows, K) / 4 + (S > 1 ? (long long)S * rows * N : 0);
    return parts > plain ? parts : plain;
}

// Where K is cut for the tensor cores: the pieces, and how long all but the last are (0 pieces: multiply-adds)
MI_EXPORT int mi_gemm_f32_pieces(int N, int K, int* length) { return on_tensor_cores(N, K) ? tc_segments(N, K, length) : 0; }

// kernels that mi_gemm_f32_nt launches
MI_EXPORT int mi_gemm_f32_launches(const float* W, int M, int N, int K) {
    if (M == 0 || N == 0) return 0;
    int segment;
    const int passes = (M + ROWS_AT_ONCE - 1) / ROWS_AT_ONCE;
    if (on_tensor_cores(N, K) && (uintptr_t)W % 16 == 0) return passes * (tc_segments(N, K, &segment) > 1 ? 3 : 2);
    return segments(N, K, &segment) > 1 ? passes * 2 : 1;
}

// tile < 0: chosen here (every tile gives the same bits)
MI_EXPORT int mi_gemm_f32_nt(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K, float* ws, int tile, int* error_word,
                             cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    int segment;
    if (on_tensor_cores(N, K) && (uintptr_t)W % 16 == 0) {
        if (!ws) return -2;
        static const int tokens[5] = {128, 128, 64, 64, 32};
        const int S = tc_segments(N, K, &segment);
        for (int m = 0; m < M; m += ROWS_AT_ONCE) {
            const int rows = M - m < ROWS_AT_ONCE ? M - m : ROWS_AT_ONCE;
            float* to = C + (size_t)m * ldc;
            float* shares = ws + mi::gemm_f32_tc_parts(rows, K) / 4;
            int rc = mi::gemm_f32_tc(A + (size_t)m * lda, lda, W, S > 1 ? shares : to, S > 1 ? N : ldc, rows, N, K, S, segment,
                                     tile >= 0 ? tokens[tile] : mi::gemm_f32_tc_tile(rows, N, S), ws, error_word, stream);
            if (rc == 0 && S > 1) rc = add_up(shares, to, ldc, rows, N, S, stream);
            if (rc) return rc;
        }
        return 0;
    }
    const int S = segments(N, K, &segment);
    if (S > 1 && !ws) return -2;
    const int step = S > 1 ? ROWS_AT_ONCE : M;
    for (int m = 0; m < M; m += step) {
        const int rows = M - m < step ? M - m : step;
        const int t = tile >= 0 ? tile : pick_tile(rows, N, S);
        int rc = run_tile(A + (size_t)m * lda, lda, W, S > 1 ? ws : C + (size_t)m * ldc, S > 1 ? N : ldc, rows, N, K, S, segment, t, stream);
        if (rc == 0 && S > 1) rc = add_up(ws, C + (size_t)m * ldc, ldc, rows, N, S, stream);
        if (rc) return rc;
    }
    return 0;
}
