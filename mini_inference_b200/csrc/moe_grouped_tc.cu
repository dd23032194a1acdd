// Grouped products of routed experts on the tcgen05 tensor cores, for steps in which an expert gets many rows.
//
// plan_kernel sorts the (token, choice) pairs by expert, an expert's rows from a multiple of 32 on, and cuts them into tiles of at most 256 rows, as
// even as 32 allows, so that a tile belongs to ONE expert.  A product is then taken the other way round: 256 rows of the expert's matrix are the M
// side and the tile's tokens the N side (32 to 256), so that an expert of 270 rows costs 288 and not three tiles of 128.  Two blocks on
// neighbouring SMs (a cluster of 2) share a product: each loads ITS 128 rows of the matrix and ITS half of the tokens, and one thread of the even
// block issues tcgen05.mma.cta_group::2, which leaves 128 accumulator rows (features) x tokens in each block's tensor memory.  The protocol
// (barriers, hand-over, allocation) is that of gemm_tc2.cu: a persistent grid, ring stages of 128 of K, two accumulators in turn.
//   MODE 0 ("in"):  the expert's matrix is [gate rows | up rows]; a block's 128 rows are 64 gate rows and the 64 up rows of the SAME outputs.  Gate and
//                   up of an output are then in lanes of two warps, which exchange half of each 32 tokens through shared memory and write
//                   g = min(g, limit), u = clamp(u, -limit, limit), g * sigmoid(slope * g) * (u + shift) to the sorted rows.
//   MODE 1 ("out"): a row is written to its pair's own row of the result.
// In both the block's 32 x 32 pieces are turned over in shared memory, so that a token's 64 bytes are stored together.  The
// exponential is the fast one, whose error grows with its argument (2 + 1.2 |x| units in the last place), and counts where e^-x does beside 1: at
// most 2^-18.6 of the result at x = -16, 2^-16.3 at -88, below the bfloat16 rounding of it (2^-9).  The reciprocal is rounded correctly.
// Every wait is bounded; a wait that runs out sets the error word, and all roles go on without waiting.
//
// Both products, microseconds with one-block tiles of 128 rows x 256 columns (bound by the operands' way through shared memory) / here: 2,048 tokens,
// 4 of 32 experts of 1,024 on 2,048 167 / 131; the whole op 210 / 165, 4,096 tokens 301 / 225, 8,192 tokens 8 of 128 experts of 768 1,042 / 703, 50 rows
// an expert 110 / 108.  A product of 256 x 256 takes 0.85 us per 128 of K and hardly less with fewer columns (what gemm_tc2.cu takes too), so the
// number of tiles counts.  Measured and left: tiles of up to 384 rows as two products on one piece of the matrix (165 us), stages of 64 of K
// (177), tokens in boxes of 32 and 16 rows (157: the copying thread was the bound).
#include "pair.cuh"
#include <math.h>

using namespace mi;
using namespace mi::sm100;

namespace {

constexpr int BM = 128, BK = 64, KSUB = 2, STAGES = 3;                  // rows of a block; k of a box; boxes along k in a stage
constexpr int A_SUB = BM * BK * 2, B_SUB = 128 * BK * 2, SUB = A_SUB + B_SUB, STAGE = KSUB * SUB;
constexpr int EPILOGUE_WARPS = 8, THREADS = 64 + 32 * EPILOGUE_WARPS, ACC_COLS = 256;
constexpr int TURN_BYTES = 4096;                                        // per epilogue warp: 32 x 32 bfloat16 to be stored, 16 x 32 float32 from its partner
constexpr int SMEM = 1024 + STAGES * STAGE + EPILOGUE_WARPS * TURN_BYTES + 128;
constexpr int TILE = 256, STEP = 32;                                    // most rows of a tile; rows of tiles come in steps

__device__ __forceinline__ float gated(float g, float u, float limit, float slope, float shift) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g * __frcp_rn(1.f + __expf(-slope * g)) * (u + shift);
}

// plan: [number of tiles, 0, 0, 0 | per tile: first row, rows, expert, 0]
struct Tiles {
    const int* __restrict__ plan;
    int count, per_tile;                                                // tiles of rows; products per tile
    __device__ int4 operator()(int u) const {
        return u < count * per_tile ? *reinterpret_cast<const int4*>(plan + 4 + 4 * (u / per_tile)) : make_int4(0, 0, 0, 0);
    }
};

// the tokens' boxes of 16, 32 .. 128 rows: one copy a tile
struct Boxes { CUtensorMap of[TILE / 2 / 16]; };

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ Boxes xmaps,
                __nv_bfloat16* __restrict__ out, int ldo, const int* __restrict__ sorted_pair, const int* __restrict__ plan, int N, int K, float limit,
                float slope, float shift, int* __restrict__ error_word) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* turn = base + STAGES * STAGE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(turn + EPILOGUE_WARPS * TURN_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    const uint32_t stage0 = smem_u32(base), full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const uint32_t acc_full0 = smem_u32(bars + 2 * STAGES), acc_empty0 = smem_u32(bars + 2 * STAGES + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t rank = cta_rank_in_cluster();                        // 0: the block that issues the products
    const int nk = (K + KSUB * BK - 1) / (KSUB * BK);                   // a box beyond K reads zeros
    constexpr int WIDE = MODE == 0 ? BM : 2 * BM;                       // outputs of a product
    const Tiles tiles{plan, plan[0], (N + WIDE - 1) / WIDE};
    const int units = tiles.count * tiles.per_tile;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full0 + 8 * b, 1); mbar_init(acc_empty0 + 8 * b, 2 * EPILOGUE_WARPS); }
        mbar_init_fence();
        tma_prefetch_desc(&wmap);
    }
    __syncthreads();
    if (warp == 1) tmem_alloc_pair(smem_u32(tmem_slot), 2 * ACC_COLS);
    tc_fence_before();
    cluster_barrier();                                                  // both blocks' barriers exist before either signals the other's
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t full_even0 = map_to_rank(full0, 0);
            int s = 0, round = 0;
            bool ok = true;
            int4 next = tiles(pair);
            for (int u = pair; ok && u < units; u += pairs) {
                const int4 t = next;
                next = tiles(u + pairs);
                const int half = t.y / 2, x0 = t.x + (int)rank * half, f0 = u % tiles.per_tile * WIDE;
                const CUtensorMap* xmap = &xmaps.of[half / 16 - 1];
                tma_prefetch_desc(xmap);
                const int w0 = MODE == 0 ? t.z * 2 * N + f0 + (int)rank * 64 : t.z * N + f0 + (int)rank * 128;
                for (int kc = 0; kc < nk; ++kc) {
                    if (round > 0 && !mbar_spin(empty0 + 8 * s, (round - 1) & 1)) { atomicExch(error_word, 61); ok = false; break; }
                    const uint32_t dst = stage0 + s * STAGE, bar = full_even0 + 8 * s;
                    if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * KSUB * (A_SUB + half * BK * 2));      // the bytes of both blocks
#pragma unroll
                    for (int i = 0; i < KSUB; ++i) {
                        const int x = (kc * KSUB + i) * BK;
                        const uint32_t a = dst + i * SUB, b = a + A_SUB;
                        tma_load_2d_pair(a, &wmap, x, w0, bar);         // the block's 128 rows of the matrix
                        if (MODE == 0) tma_load_2d_pair(a + A_SUB / 2, &wmap, x, w0 + N, bar);
                        tma_load_2d_pair(b, xmap, x, x0, bar);
                    }
                    if (++s == STAGES) { s = 0; ++round; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && lane == 0) {
            const uint64_t desc_a0 = umma_desc_sw128(stage0, 16, 1024), desc_b0 = umma_desc_sw128(stage0 + A_SUB, 16, 1024);
            int s = 0, round = 0, turn_no = 0;
            bool ok = true;
            int4 next = tiles(pair);
            for (int u = pair; ok && u < units; u += pairs, ++turn_no) {
                const int b = turn_no & 1;
                const uint32_t idesc = umma_idesc_bf16(2 * BM, next.y, false);
                next = tiles(u + pairs);
                if (turn_no >= 2 && !mbar_wait(acc_empty0 + 8 * b, ((turn_no >> 1) - 1) & 1)) { atomicExch(error_word, 64); break; }
                tc_fence_after();
                const uint32_t acc = tmem + b * ACC_COLS;
                for (int kc = 0; kc < nk; ++kc) {
                    if (!mbar_spin(full0 + 8 * s, round & 1)) { atomicExch(error_word, 62); ok = false; break; }
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((uint32_t)(s * STAGE) >> 4);
#pragma unroll
                    for (int k = 0; k < KSUB * BK / 16; ++k)
                        umma_ss_pair(acc, desc_a0 + off + (k >> 2) * (SUB >> 4) + 2 * (k & 3), desc_b0 + off + (k >> 2) * (SUB >> 4) + 2 * (k & 3), idesc, (kc | k) != 0);
                    umma_commit_pair(empty0 + 8 * s, 3);                // the stage is free in both blocks once these have read it
                    if (++s == STAGES) { s = 0; ++round; }
                }
                if (!ok) break;
                umma_commit_pair(acc_full0 + 8 * b, 3);                 // the accumulator is complete in both blocks
            }
        }
    } else {
        // ---------------- warp's quarter of the lanes (features), every other group of 32 columns (tokens)
        const int q = warp & 3, part = (warp - 2) >> 2, slot = warp - 2, partner = slot ^ 2;
        const uint32_t acc_empty_even0 = map_to_rank(acc_empty0, 0);
        unsigned char* box = turn + slot * TURN_BYTES;                  // rows of 32 features, 64 bytes
        float* from = reinterpret_cast<float*>(turn + slot * TURN_BYTES + 2048);
        float* to_partner = reinterpret_cast<float*>(turn + partner * TURN_BYTES + 2048);
        const int bar = 1 + (q & 1) + 2 * part;                         // the two warps with gate and up of the same outputs
        auto meet = [&] { asm volatile("bar.sync %0, 64;\n" :: "r"(bar) : "memory"); };
        auto put = [&](int row, float v) { *reinterpret_cast<__nv_bfloat16*>(box + row * 64 + lane * 2) = __float2bfloat16_rn(v); };
        const int row8 = lane >> 2, piece = lane & 3;                   // a lane's 16 bytes of eight rows
        bool alive = true;
        int turn_no = 0;
        int4 next = tiles(pair);
        for (int u = pair; u < units; u += pairs, ++turn_no) {
            const int4 t = next;
            next = tiles(u + pairs);
            const int b = turn_no & 1, f0 = u % tiles.per_tile * WIDE;
            if (alive && !mbar_wait(acc_full0 + 8 * b, (turn_no >> 1) & 1)) { alive = false; if (lane == 0) atomicExch(error_word, 63); }
            tc_fence_after();
            const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + b * ACC_COLS;
            for (int c = part; c < t.y / STEP; c += 2) {
                uint32_t r[32];
                tmem_ld32(acc + c * 32, r);
                tmem_wait_ld();
                const int pos = t.x + c * 32;
                if (MODE == 1) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) put(i, __uint_as_float(r[i]));
                    __syncwarp();
                    const int col = f0 + (int)rank * 128 + q * 32 + piece * 8;
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        const int pr = sorted_pair[pos + i + row8];
                        if (pr >= 0 && col < N) *reinterpret_cast<uint4*>(out + (size_t)pr * ldo + col) = *reinterpret_cast<const uint4*>(box + (i + row8) * 64 + piece * 16);
                    }
                } else {
                    const bool up = q >= 2;                             // the gate's warp makes tokens 0 .. 15, the other one the rest
                    meet();                                             // the partner has read what it was sent before
#pragma unroll
                    for (int i = 0; i < 16; ++i) to_partner[i * 32 + lane] = __uint_as_float(up ? r[i] : r[16 + i]);
                    meet();
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float own = __uint_as_float(up ? r[16 + i] : r[i]), got = from[i * 32 + lane];
                        put(i, gated(up ? got : own, up ? own : got, limit, slope, shift));
                    }
                    __syncwarp();
                    const int col = f0 + (int)rank * 64 + (q & 1) * 32 + piece * 8;
#pragma unroll
                    for (int i = 0; i < 16; i += 8)
                        if (col < N)
                            *reinterpret_cast<uint4*>(out + (size_t)(pos + (up ? 16 : 0) + i + row8) * ldo + col) = *reinterpret_cast<const uint4*>(box + (i + row8) * 64 + piece * 16);
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_empty_even0 + 8 * b);
        }
    }
    tc_fence_before();
    cluster_barrier();            // neither block leaves while the other may still read its shared memory or signal its barriers
    if (warp == 1) tmem_dealloc_pair(tmem, 2 * ACC_COLS);
}

// One block: the pairs by expert and the tiles (see Tiles).  A pair's place among its expert's is what the counting's atomics answer.
constexpr int PLAN_THREADS = 1024, HELD = 16;
__global__ void __launch_bounds__(PLAN_THREADS) plan_kernel(const int* __restrict__ chosen, int P, int E, int* __restrict__ sorted_pair, int cap_pos, int* __restrict__ plan) {
    extern __shared__ int plan_smem[];
    int* count = plan_smem;                                             // [E]; then an expert's next free place when pairs are counted twice
    int* first = count + E;                                             // [E + 1]
    int* first_tile = first + E + 1;                                    // [E + 1]
    const int tid = threadIdx.x;
    for (int e = tid; e < E; e += PLAN_THREADS) count[e] = 0;
    int e_of[HELD], place[HELD];                                        // chosen is read once, and all at once (12.4 -> 8.2 us for 8,192 pairs)
#pragma unroll
    for (int i = 0; i < HELD; ++i) e_of[i] = i * PLAN_THREADS + tid < P ? chosen[i * PLAN_THREADS + tid] : -1;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < HELD; ++i) if (e_of[i] >= 0) place[i] = atomicAdd(&count[e_of[i]], 1);
    if (P > HELD * PLAN_THREADS) __syncthreads();                       // the pairs that are held come first
    for (int p = HELD * PLAN_THREADS + tid; p < P; p += PLAN_THREADS) atomicAdd(&count[chosen[p]], 1);
    __syncthreads();
    if (tid < 32) {                                                     // sums before each expert
        int rows = 0, tiles = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + tid, n = e < E ? count[e] : 0;
            int a = (n + STEP - 1) / STEP * STEP, b = (n + TILE - 1) / TILE;
            const int own_a = a, own_b = b;
#pragma unroll
            for (int w = 1; w < 32; w <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, a, w), y = __shfl_up_sync(0xffffffffu, b, w);
                if (tid >= w) { a += x; b += y; }
            }
            if (e < E) { first[e] = rows + a - own_a; first_tile[e] = tiles + b - own_b; }
            rows += __shfl_sync(0xffffffffu, a, 31);
            tiles += __shfl_sync(0xffffffffu, b, 31);
        }
        if (tid == 0) { first[E] = rows; plan[0] = tiles; }
    }
    __syncthreads();
    for (int e = tid; e < E; e += PLAN_THREADS) {
        const int n = count[e], tiles = (n + TILE - 1) / TILE, at = first[e], end = at + (n + STEP - 1) / STEP * STEP;
        const int rows = tiles ? ((n + tiles - 1) / tiles + STEP - 1) / STEP * STEP : 0;
        for (int i = 0; i < tiles; ++i)
            *reinterpret_cast<int4*>(plan + 4 + 4 * (first_tile[e] + i)) = make_int4(at + i * rows, min(rows, end - at - i * rows), e, 0);
        for (int r = at + n; r < end; ++r) sorted_pair[r] = -1;
    }
    for (int r = first[E] + tid; r < cap_pos; r += PLAN_THREADS) sorted_pair[r] = -1;
#pragma unroll
    for (int i = 0; i < HELD; ++i) if (e_of[i] >= 0) sorted_pair[first[e_of[i]] + place[i]] = i * PLAN_THREADS + tid;
    if (P > HELD * PLAN_THREADS) {                                      // the pairs that were only counted: behind the others, again by atomics
        __syncthreads();
        for (int e = tid; e < E; e += PLAN_THREADS) count[e] = 0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < HELD; ++i) if (e_of[i] >= 0) atomicMax(&count[e_of[i]], place[i] + 1);
        __syncthreads();
        for (int p = HELD * PLAN_THREADS + tid; p < P; p += PLAN_THREADS) {
            const int e = chosen[p];
            sorted_pair[first[e] + atomicAdd(&count[e], 1)] = p;
        }
    }
}

// sorted[pos] = h[sorted_pair[pos] / top] (zeros where the position is padding): the rows of the first grouped product
__global__ void moe_gather_rows_kernel(const __nv_bfloat16* __restrict__ h, int ldh, const int* __restrict__ sorted_pair, int top,
                                       __nv_bfloat16* __restrict__ sorted, int K, const float* __restrict__ weights) {
    const int pr = sorted_pair[blockIdx.x];
    uint4* dst = reinterpret_cast<uint4*>(sorted + (size_t)blockIdx.x * K);
    if (pr < 0) {
        for (int i = threadIdx.x; i < K / 8; i += blockDim.x) dst[i] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    const uint4* src = reinterpret_cast<const uint4*>(h + (size_t)(pr / top) * ldh);
    if (!weights) {
        for (int i = threadIdx.x; i < K / 8; i += blockDim.x) dst[i] = src[i];
        return;
    }
    const float w = weights[pr];                                    // the pair's score multiplies the expert's input
    for (int i = threadIdx.x; i < K / 8; i += blockDim.x) {
        uint4 raw = src[i];
        __nv_bfloat162* v = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(v[j]); v[j] = __floats2bfloat162_rn(w * f.x, w * f.y); }
        dst[i] = raw;
    }
}

}  // namespace

MI_EXPORT int mi_moe_gather_rows(const void* h, int ldh, const int* sorted_pair, int top, void* sorted, int cap_pos, int K, const float* weights,
                                 cudaStream_t stream) {
    if (cap_pos == 0) return 0;
    if (K % 8 || ldh % 8 || ((uintptr_t)h % 16) || ((uintptr_t)sorted % 16)) return -2;
    moe_gather_rows_kernel<<<cap_pos, 128, 0, stream>>>((const __nv_bfloat16*)h, ldh, sorted_pair, top, (__nv_bfloat16*)sorted, K, weights);
    return (int)cudaGetLastError();
}

// rows of the sorted activations, and ints of the plan, for P pairs over E experts
MI_EXPORT int mi_moe_plan_rows(int P, int E) { return ((P + STEP - 1) / STEP + min(E, P)) * STEP; }
MI_EXPORT int mi_moe_plan_ints(int P, int E) { return 4 + 4 * ((P + TILE - 1) / TILE + min(E, P)); }

// chosen [P]: experts below E; sorted_pair [mi_moe_plan_rows], -1 where a row has no pair; plan [mi_moe_plan_ints] on 16 bytes
MI_EXPORT int mi_moe_plan(const int* chosen, int P, int E, int* sorted_pair, int cap_pos, int* plan, cudaStream_t stream) {
    if (P == 0) return 0;
    if (E > 4095 || cap_pos < mi_moe_plan_rows(P, E) || (uintptr_t)plan % 16) return -2;
    plan_kernel<<<1, PLAN_THREADS, (3 * E + 2) * sizeof(int), stream>>>(chosen, P, E, sorted_pair, cap_pos, plan);
    return (int)cudaGetLastError();
}

// A [cap_pos, K] contiguous bfloat16 (sorted rows); W [E, mode 0 ? 2 N : N, K] contiguous; out: mode 0 [cap_pos, N] (ldo = N), mode 1 [pairs, N].
// K % 64 == 0, N % 8 == 0.
MI_EXPORT int mi_moe_gemm_tcgen05(const void* A, const void* W, int E, void* out, int ldo, const int* sorted_pair, const int* plan, int cap_pos, int N, int K,
                                  float limit, float slope, float shift, int mode, int* error_word, cudaStream_t stream) {
    if (cap_pos == 0) return 0;
    if (K % BK || K < BK || N % 8 || ldo % 8 || ((uintptr_t)A % 16) || ((uintptr_t)W % 16) || ((uintptr_t)out % 16) || ((uintptr_t)plan % 16)) return -2;
    auto kern = mode == 0 ? moe_pair_kernel<0> : moe_pair_kernel<1>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM; cfg.stream = stream; cfg.attrs = attr; cfg.numAttrs = 1;
    static int pairs[2] = {0, 0};
    if (!pairs[mode]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        cfg.gridDim = dim3(2);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) { (void)cudaGetLastError(); return -2; }
        pairs[mode] = n;
    }
    CUtensorMap wmap;
    Boxes xmaps;
    if (!sm100_host::make_map_bf16(&wmap, W, (uint64_t)E * (mode == 0 ? 2 : 1) * N, K, K, mode == 0 ? 64 : 128, BK)) return -5;
    for (int i = 0; i < TILE / 2 / 16; ++i)
        if (!sm100_host::make_map_bf16(&xmaps.of[i], A, cap_pos, K, K, 16 * (i + 1), BK)) return -5;
    const long long most = ((long long)cap_pos / STEP) * ((N + (mode == 0 ? BM : 2 * BM) - 1) / (mode == 0 ? BM : 2 * BM));      // products there can be
    cfg.gridDim = dim3((unsigned)(2 * (most < pairs[mode] ? most : pairs[mode])));
    return (int)cudaLaunchKernelEx(&cfg, kern, wmap, xmaps, (__nv_bfloat16*)out, ldo, sorted_pair, plan, N, K, limit, slope, shift, error_word);
}
