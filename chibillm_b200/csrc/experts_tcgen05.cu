// The products of a feed-forward of experts on the 5th-generation tensor cores.
//
// The rows (one per (token, choice) pair) lie sorted by expert in one bfloat16 array
// [pairs, K]; all experts' matrices are one array [experts * rows_w, K].  A tile map made on
// the device by route_by_table (layer_ops.cu) names, for every tile of 128 rows, its expert
// and its first row, the tiles in use first; a tile never holds rows of two experts that it writes.
//
// MODE 1 (gated): an expert's matrix holds blocks of 16 gate rows followed by their 16 up rows,
// so 32 sums are 16 gate sums and their 16 up sums; out[r, f] = act(gate) * up
// in bfloat16.  MODE 2: out[r, n] = act(sum) in bfloat16 (an expert without a gate).
// MODE 0: out is 32-bit [pairs, rows_w].
//
// Many tokens: a persistent CTA an SM walks over tiles of 128 rows x 256 weight rows.  TMA brings the
// K blocks of 64 of both operands (128-byte swizzle) through a ring of stages, one elected thread
// issues tcgen05.mma (128 x 256 x 16) into one of two TMEM accumulators, and eight warps
// read the other back with tcgen05.ld.  Bound by what an SM can take in (48 KB to 128 x 256 x 64
// multiply-adds) and by the epilogue: a CTA a tile of 128 x 128, which this replaces, wanted 64 KB for as many
// and began and ended each tile by itself, and with four epilogue warps the gate bounds the tiles (the whole
// feed-forward, two of eight experts a token, three sets of weights in turn, more than L2 holds: 2,048 tokens of
// 2,048 x 3,072 231 us before, 176 now, of 4,096 x 6,144 770 -> 650; with weights that L2 holds 232 before, 221 with four
// warps, 176 with eight).  The gate is made with CUDA's exact exponential and division, 1.6 % of the first of these.
// Rows past the expert's last row are computed (they are the next expert's rows,
// or zeros past the array's end) and not written.
//
// Few tokens: an expert has few rows and the weights' way from memory bounds the products.  The
// operands are swapped: a CTA takes 128 weight rows as the instruction's rows and the tile's rows, 16, 32 or
// 64 at a time, as its columns, so that beside 16 KB of weights a stage brings 2 to 8 KB of rows
// instead of 16 (8 tokens, the same experts: 109 -> 58.4 us).
//
// Warp roles: warp 0 loads, warp 1 owns TMEM and issues, the others are the
// epilogue (warp w reads TMEM lanes 32 * (w % 4) ..).  Every wait has a limit; a wait that
// runs out records a code in the error word and the CTA goes on to free its TMEM.
#define CHIBI_UNIT experts_tcgen05
#define CHIBI_UNIT_ID 10
#include "common.cuh"
#include "sm100.cuh"
#include "tensor_map.cuh"

namespace chibi {

using namespace sm100;

constexpr int XT_M = 128, XT_K = 64, XT_UMMA_K = 16, XT_THREADS = 192, XT_MANY_THREADS = 320;
template <int XT_N> struct ManyTile {
    static constexpr int STAGES = XT_N == 256 ? 4 : 6, A_BYTES = XT_M * XT_K * 2, STAGE_BYTES = A_BYTES + XT_N * XT_K * 2;
    static constexpr size_t SMEM = STAGES * STAGE_BYTES + (2 * STAGES + 4) * 8 + 16 + 1024;
};

struct ExpertTileParams {
    const int* offsets;        // [experts + 1]: first sorted row of every expert
    const int* tile_expert;    // [max_tiles]: -1 = unused
    const int* tile_row0;      // [max_tiles]
    int max_tiles;
    int rows_w;                // rows of one expert's matrix (2 F when gated)
    int k_blocks;              // K / 64
    void* out;
    long long out_stride;
    int kind;                  // activation of the gate
    const float* row_weight;   // [pairs] or null: gated sums of pair p's row are multiplied by row_weight[p] first
    const int* pair_of_row;    // [pairs]
    int* error;
};

template <int MODE, int XT_N>
__global__ void __launch_bounds__(XT_MANY_THREADS)
expert_rows_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      const ExpertTileParams p)
{
    constexpr int XT_STAGES = ManyTile<XT_N>::STAGES, XT_A_BYTES = ManyTile<XT_N>::A_BYTES,
                  XT_STAGE_BYTES = ManyTile<XT_N>::STAGE_BYTES;
    pdl_enter();                                   // the tile map is the kernel before's work
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + XT_STAGES * XT_STAGE_BYTES);
    uint64_t* empty_bar = full_bar + XT_STAGES;
    uint64_t* tmem_full_bar = empty_bar + XT_STAGES;                 // [2]
    uint64_t* tmem_empty_bar = tmem_full_bar + 2;                    // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = (p.rows_w + XT_N - 1) / XT_N;
    // the CTA's tile number `it`: false past the last
    auto tile_at = [&](int it, int& expert, int& row0, int& n0) {
        const int t = (int)blockIdx.x + it * (int)gridDim.x, j = t / tiles_n;
        if (j >= p.max_tiles)
            return false;
        expert = p.tile_expert[j];
        row0 = p.tile_row0[j];
        n0 = (t - j * tiles_n) * XT_N;
        return expert >= 0;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < XT_STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tmem_full_bar[b], 1);
            mbar_init(&tmem_empty_bar[b], 256);        // every epilogue thread arrives
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 2 * XT_N);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    int expert, row0, n0;
    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_descriptor(&map_a);
            tma_prefetch_descriptor(&map_b);
            uint32_t i = 0;
            bool ok = true;
            for (int it = 0; ok && tile_at(it, expert, row0, n0); ++it)
                for (int kb = 0; kb < p.k_blocks; ++kb, ++i) {
                    const uint32_t s = i % XT_STAGES, round = i / XT_STAGES;
                    if (round > 0 && !mbar_wait(&empty_bar[s], (round - 1) & 1, p.error, 31)) {
                        ok = false;
                        break;
                    }
                    uint8_t* a_dst = smem + s * XT_STAGE_BYTES;
                    mbar_arrive_expect_tx(&full_bar[s], XT_STAGE_BYTES);
                    tma_load_2d(a_dst, &map_a, &full_bar[s], kb * XT_K, row0);
                    tma_load_2d(a_dst + XT_A_BYTES, &map_b, &full_bar[s], kb * XT_K, expert * p.rows_w + n0);
                }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc_bf16_f32(XT_M, XT_N);
            uint32_t i = 0;
            bool ok = true;
            for (int it = 0; ok && tile_at(it, expert, row0, n0); ++it) {
                const uint32_t buf = it & 1, use = it >> 1;
                if (use > 0 && !mbar_wait(&tmem_empty_bar[buf], (use - 1) & 1, p.error, 34))
                    break;
                tcgen05_fence_after();
                for (int kb = 0; kb < p.k_blocks; ++kb, ++i) {
                    const uint32_t s = i % XT_STAGES, round = i / XT_STAGES;
                    if (!mbar_wait(&full_bar[s], round & 1, p.error, 32)) {
                        ok = false;
                        break;
                    }
                    tcgen05_fence_after();
                    const uint32_t a_addr = smem_addr(smem + s * XT_STAGE_BYTES);
                    const uint32_t b_addr = a_addr + XT_A_BYTES;
#pragma unroll
                    for (int k = 0; k < XT_K / XT_UMMA_K; ++k) {
                        const uint64_t a_desc = make_kmajor_sw128_desc(a_addr + k * XT_UMMA_K * 2);
                        const uint64_t b_desc = make_kmajor_sw128_desc(b_addr + k * XT_UMMA_K * 2);
                        tcgen05_mma_bf16(tmem_base + buf * XT_N, a_desc, b_desc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    tcgen05_commit(&empty_bar[s]);     // the stage is free once these MMAs have read it
                }
                if (ok)
                    tcgen05_commit(&tmem_full_bar[buf]);
            }
        }
    } else {
        // two warps to a quarter of the rows, each with half of the columns
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        for (int it = 0; tile_at(it, expert, row0, n0); ++it) {
            const uint32_t buf = it & 1, use = it >> 1;
            if (!mbar_wait_warp(&tmem_full_bar[buf], use & 1, p.error, 33))
                break;
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + buf * XT_N + (static_cast<uint32_t>(quarter * 32) << 16);
            const int r = row0 + quarter * 32 + lane;
            const bool write = r < min(row0 + XT_M, p.offsets[expert + 1]);
            const float wr = (MODE == 1 && write && p.row_weight) ? p.row_weight[p.pair_of_row[r]] : 1.f;
#pragma unroll 1
            for (int c0 = half * (XT_N / 2); c0 < (half + 1) * (XT_N / 2); c0 += 32) {
                uint32_t v[32];
                // every lane of the warp takes part in the load, whether its row is written or not
                tmem_load_32x32(taddr + c0, v);
                tmem_load_wait();
                if (!write)
                    continue;
                if (MODE == 2) {
                    if (n0 + c0 >= p.rows_w)
                        continue;
                    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + (size_t)r * p.out_stride + n0 + c0;
                    __nv_bfloat162 h[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        h[j] = __floats2bfloat162_rn(activate(__uint_as_float(v[2 * j]), p.kind),
                                                     activate(__uint_as_float(v[2 * j + 1]), p.kind));
                    if (n0 + c0 + 32 <= p.rows_w && p.out_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            reinterpret_cast<uint4*>(dst)[j] = reinterpret_cast<uint4*>(h)[j];
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            if (n0 + c0 + 2 * j < p.rows_w)
                                dst[2 * j] = h[j].x;
                            if (n0 + c0 + 2 * j + 1 < p.rows_w)
                                dst[2 * j + 1] = h[j].y;
                        }
                    }
                } else if (MODE == 1) {
                    const int col = (n0 + c0) / 2;          // 32 accumulator columns = 16 features
                    if (col >= p.rows_w / 2)
                        continue;
                    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + (size_t)r * p.out_stride + col;
                    __nv_bfloat162 h[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        h[j] = __floats2bfloat162_rn(
                            activate(wr * __uint_as_float(v[2 * j]), p.kind) * (wr * __uint_as_float(v[16 + 2 * j])),
                            activate(wr * __uint_as_float(v[2 * j + 1]), p.kind) * (wr * __uint_as_float(v[16 + 2 * j + 1])));
                    if (p.out_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0) {
                        reinterpret_cast<uint4*>(dst)[0] = reinterpret_cast<uint4*>(h)[0];
                        reinterpret_cast<uint4*>(dst)[1] = reinterpret_cast<uint4*>(h)[1];
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            dst[2 * j] = h[j].x;
                            dst[2 * j + 1] = h[j].y;
                        }
                    }
                } else {
                    float* dst = static_cast<float*>(p.out) + (size_t)r * p.out_stride + n0 + c0;
                    if (n0 + c0 + 32 <= p.rows_w && p.out_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            reinterpret_cast<float4*>(dst)[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                                            __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (n0 + c0 + j < p.rows_w)
                                dst[j] = __uint_as_float(v[j]);
                    }
                }
            }
            tcgen05_fence_before();
            mbar_arrive(&tmem_empty_bar[buf]);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 2 * XT_N);
    }
}

// Few tokens: grid (blocks of 128 weight rows, tiles of the map), XN rows of the tile at a time.  (Where an expert has more
// rows than XN the weights are fetched once more for each XN.)
template <int XN> struct FewTile {
    static constexpr int STAGES = XN == 16 ? 6 : XN == 32 ? 5 : 4;      // two CTAs to an SM
    static constexpr int A_BYTES = 128 * XT_K * 2, STAGE_BYTES = A_BYTES + XN * XT_K * 2;
    static constexpr size_t SMEM = STAGES * STAGE_BYTES + (2 * STAGES + 1) * 8 + 16 + 1024;
};

template <int MODE, int XN>
__global__ void __launch_bounds__(XT_THREADS)
expert_few_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                       const ExpertTileParams p)
{
    pdl_enter();                                   // the tile map is the kernel before's work
    using F = FewTile<XN>;
    constexpr uint32_t TMEM_COLS = XT_M;           // a column for every row that a tile can hold
    const int expert = p.tile_expert[blockIdx.y];
    if (expert < 0)
        return;                                    // the whole CTA, before any barrier or TMEM
    const int row0 = p.tile_row0[blockIdx.y];
    const int row_end = min(row0 + XT_M, p.offsets[expert + 1]);
    const int n0 = blockIdx.x * 128, subs = (row_end - row0 + XN - 1) / XN;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + F::STAGES * F::STAGE_BYTES);
    uint64_t* empty_bar = full_bar + F::STAGES;
    uint64_t* tmem_full_bar = empty_bar + F::STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full_bar + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < F::STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(tmem_full_bar, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int turns = subs * p.k_blocks;

    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_descriptor(&map_w);
            tma_prefetch_descriptor(&map_x);
            for (int i = 0; i < turns; ++i) {
                const uint32_t s = i % F::STAGES, round = i / F::STAGES;
                if (round > 0 && !mbar_wait(&empty_bar[s], (round - 1) & 1, p.error, 31))
                    break;
                const int sub = i / p.k_blocks, kb = i - sub * p.k_blocks;
                uint8_t* dst = smem + s * F::STAGE_BYTES;
                mbar_arrive_expect_tx(&full_bar[s], F::STAGE_BYTES);
                tma_load_2d(dst, &map_w, &full_bar[s], kb * XT_K, expert * p.rows_w + n0);
                tma_load_2d(dst + F::A_BYTES, &map_x, &full_bar[s], kb * XT_K, row0 + sub * XN);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc_bf16_f32(128, XN);
            for (int i = 0; i < turns; ++i) {
                const uint32_t s = i % F::STAGES, round = i / F::STAGES;
                if (!mbar_wait(&full_bar[s], round & 1, p.error, 32))
                    break;
                tcgen05_fence_after();
                const int sub = i / p.k_blocks, kb = i - sub * p.k_blocks;
                const uint32_t w_addr = smem_addr(smem + s * F::STAGE_BYTES), x_addr = w_addr + F::A_BYTES;
#pragma unroll
                for (int k = 0; k < XT_K / XT_UMMA_K; ++k) {
                    const uint64_t w_desc = make_kmajor_sw128_desc(w_addr + k * XT_UMMA_K * 2);
                    const uint64_t x_desc = make_kmajor_sw128_desc(x_addr + k * XT_UMMA_K * 2);
                    tcgen05_mma_bf16(tmem_base + sub * XN, w_desc, x_desc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                }
                tcgen05_commit(&empty_bar[s]);
            }
            tcgen05_commit(tmem_full_bar);
        }
    } else {
        const int quarter = warp & 3, n = n0 + quarter * 32 + lane;
        const bool ok = mbar_wait_warp(tmem_full_bar, 0, p.error, 33);
        tcgen05_fence_after();
#pragma unroll 1
        for (int c0 = 0; ok && c0 < row_end - row0; c0 += 16) {
            uint32_t v[16];
            tmem_load_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c0, v);
            tmem_load_wait();
            if (MODE == 1) {
                // lanes 0 to 15 hold gate sums, 16 to 31 their up sums: of two rows each half finishes one
                const bool upper = lane >= 16;
                const int f = (n0 + quarter * 32) / 2 + (lane & 15);
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    const float mine = __uint_as_float(upper ? v[c + 1] : v[c]);
                    const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, upper ? v[c] : v[c + 1], 16));
                    const int r = row0 + c0 + c + (upper ? 1 : 0);
                    if (r < row_end && f < p.rows_w / 2) {
                        const float wr = p.row_weight ? p.row_weight[p.pair_of_row[r]] : 1.f;
                        const float gate = upper ? other : mine, up = upper ? mine : other;
                        static_cast<__nv_bfloat16*>(p.out)[(size_t)r * p.out_stride + f] =
                            __float2bfloat16_rn(activate(wr * gate, p.kind) * (wr * up));
                    }
                }
            } else if (n < p.rows_w) {
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    const int r = row0 + c0 + c;
                    if (r < row_end) {
                        if (MODE == 2)
                            static_cast<__nv_bfloat16*>(p.out)[(size_t)r * p.out_stride + n] =
                                __float2bfloat16_rn(activate(__uint_as_float(v[c]), p.kind));
                        else
                            static_cast<float*>(p.out)[(size_t)r * p.out_stride + n] = __uint_as_float(v[c]);
                    }
                }
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int MODE, int XN>
static int launch_expert_few(const void* a, const void* w, long long pairs, int experts, int K, const ExpertTileParams& p,
                             cudaStream_t stream)
{
    CUtensorMap map_w, map_x;
    if (!tensor_map_2d(w, (long long)experts * p.rows_w, K, K, 128, &map_w) || !tensor_map_2d(a, pairs, K, K, XN, &map_x))
        return CHIBI_ERR_UNSUPPORTED;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(expert_few_rows_kernel<MODE, XN>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FewTile<XN>::SMEM);
        if (e != cudaSuccess)
            return (int)e;
        configured = true;
    }
    launch(expert_few_rows_kernel<MODE, XN>, dim3((unsigned)((p.rows_w + 127) / 128), (unsigned)p.max_tiles), dim3(XT_THREADS),
           FewTile<XN>::SMEM, stream, map_w, map_x, p);
    return launch_status();
}

template <int MODE, int XT_N>
static int launch_expert_many(const void* a, const void* w, long long pairs, int experts, int K, const ExpertTileParams& p,
                              cudaStream_t stream)
{
    CUtensorMap map_a, map_b;
    if (!tensor_map_2d(a, pairs, K, K, XT_M, &map_a) || !tensor_map_2d(w, (long long)experts * p.rows_w, K, K, XT_N, &map_b))
        return CHIBI_ERR_UNSUPPORTED;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(expert_rows_tc_kernel<MODE, XT_N>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ManyTile<XT_N>::SMEM);
        if (e != cudaSuccess)
            return (int)e;
        configured = true;
    }
    const long long tiles = (long long)((p.rows_w + XT_N - 1) / XT_N) * p.max_tiles, sms = device_sm_count();
    launch(expert_rows_tc_kernel<MODE, XT_N>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(XT_MANY_THREADS),
           ManyTile<XT_N>::SMEM, stream, map_a, map_b, p);
    return launch_status();
}

template <int MODE>
static int launch_expert_rows(const void* a, const void* w, long long pairs, int experts, int K, long long tokens,
                              const ExpertTileParams& p, cudaStream_t stream)
{
    if (tokens <= 16)
        return launch_expert_few<MODE, 16>(a, w, pairs, experts, K, p, stream);
    if (tokens <= 32)
        return launch_expert_few<MODE, 32>(a, w, pairs, experts, K, p, stream);
    // Few columns as long as an expert's rows mostly fit 64 of them: 128 tokens of 8 experts of 1,024 x 1,536, two a
    // token, weights that L2 holds, 29.5 us, 37.4 in tiles; 300 tokens (128 columns) 41.4, 40.9 in tiles.
    if (tokens <= 64 || pairs <= 32LL * experts)
        return launch_expert_few<MODE, 64>(a, w, pairs, experts, K, p, stream);
    // (as many tiles as the pairs make if they spread over the experts)  Narrow ones where they leave no SM a second.
    const long long spread = pairs / XT_M + (pairs < experts ? pairs : experts);
    if (spread * ((p.rows_w + 127) / 128) <= device_sm_count())
        return launch_expert_many<MODE, 128>(a, w, pairs, experts, K, p, stream);
    return launch_expert_many<MODE, 256>(a, w, pairs, experts, K, p, stream);
}

} // namespace chibi

using namespace chibi;

// One product of the routed rows on tcgen05.  a: [pairs, K] bfloat16, contiguous, sorted by expert;
// w: [experts, rows_w, K] bfloat16, contiguous (gated: rows_w = 2 F, interleaved in blocks of 16);
// route: as route_by_table lays it out for tiles of 128 rows.  out: gated == 1: bfloat16 [pairs, F]
// with out_stride (row_weight [pairs], may be null: see ExpertTileParams); gated == 2: bfloat16 [pairs, rows_w], act(sum); else float [pairs, rows_w].  CHIBI_ERR_UNSUPPORTED for sizes it does not take.
CHIBI_API int chibi_expert_rows_tc(const void* a, const void* w, void* out, long long out_stride, const int* route,
                                   long long pairs, long long tokens, int experts, int rows_w, int K, int gated,
                                   int kind, const float* row_weight, int* error, cudaStream_t stream)
{
    if (pairs <= 0)
        return CHIBI_OK;
    if (!a || !w || !out || !route || experts <= 0 || rows_w <= 0 || K <= 0 || (row_weight && gated != 1))
        return CHIBI_ERR_ARGUMENT;
    if (K % XT_K != 0 || (gated == 1 && rows_w % 32 != 0) || (reinterpret_cast<uintptr_t>(a) & 15)
        || (reinterpret_cast<uintptr_t>(w) & 15) || pairs > 2147483647LL - XT_M
        || (long long)experts * rows_w > 2147483647LL - 256)
        return CHIBI_ERR_UNSUPPORTED;
    const int max_tiles = (int)((pairs + XT_M - 1) / XT_M) + experts;
    if (max_tiles > 65535)
        return CHIBI_ERR_UNSUPPORTED;
    ExpertTileParams p {};
    p.offsets = route;
    p.tile_expert = route + experts + 1 + 2 * pairs;
    p.tile_row0 = p.tile_expert + max_tiles;
    p.rows_w = rows_w;
    p.k_blocks = K / XT_K;
    p.out = out;
    p.out_stride = out_stride;
    p.kind = kind;
    p.row_weight = row_weight;
    p.pair_of_row = route + experts + 1;
    p.error = error;
    p.max_tiles = max_tiles;
    if (gated == 1)
        return launch_expert_rows<1>(a, w, pairs, experts, K, tokens, p, stream);
    if (gated == 2)
        return launch_expert_rows<2>(a, w, pairs, experts, K, tokens, p, stream);
    return launch_expert_rows<0>(a, w, pairs, experts, K, tokens, p, stream);
}
