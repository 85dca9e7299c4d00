// out[M, N] = x[M, K] * w[N, K]^T (+ residual[M, N]), all 32-bit, on the 5th-generation tensor cores.
//
// A 32-bit number is the sum of three bfloat16 numbers (its leading 8 bits, the next 8 of what is left, and the last 8;
// each rounded to nearest), so a product of two is the sum of nine exact products of 8 by 8 bits.  The three
// smallest of them (below 2^-26 of the whole) are left out, the other six are tcgen05.mma with 32-bit accumulators.
// What limits the precision is the accumulator, which the tensor core cuts off instead of rounding: so a block of 64 places
// has an accumulator of its own, that takes the five small products of all its places first and the large one last (four
// roundings at the size of the sum), and the blocks are added up in plain 32-bit arithmetic.  Relative error against 64 bits
// (2-norm, normal numbers, K = 128 / 1,024 / 3,072 / 6,144): XX; by multiply-adds (fma.rn.f32x2) before 1.5e-7 / 1.5e-7 /
// 1.9e-7 / 2.6e-7.
//
// The order of a sum depends on K alone: the blocks of 64 places lie in at most eight runs, a run's blocks are added in
// order, the first four runs in order, the other four in order, and the two halves at last.  So a row's result does not
// depend on the rows beside it, nor on how many CTAs share a sum (a cluster of 1, 2, 4 or 8 takes the runs in order).
//
// A number that is none, or too large for bfloat16, would leave its row by the products with zeros that are exact: rows of
// x and w with such a number are marked, and their outputs are summed by multiply-adds instead.
//
// A CTA owns 128 rows of w (the M of the MMA) and up to 128 rows of x (its N).  Eight warps bring both from memory (in
// registers, one block ahead), split them and write the six tiles to one of two stages in shared memory in
// the swizzled K-major layout; one thread of the first issues the MMAs; and while they run, all eight read the accumulator of
// the block before, in one of two buffers in TMEM, and add it up.  (A ninth warp for the MMAs would leave 168 registers a
// thread instead of 255, and 128 columns do not fit them.)
#define CHIBI_UNIT gemm_f32_tcgen05
#define CHIBI_UNIT_ID 18
#include "common.cuh"
#include "sm100.cuh"

namespace chibi {

using namespace sm100;

constexpr int F3_ROWS = 128, F3_KB = 64;         // rows of w; places of a block
constexpr int F3_RUNS = 8;
constexpr int F3_THREADS = 256;
constexpr int F3_W_PLANE = F3_ROWS * F3_KB * 2;

struct F3Params {
    const float* x;
    const float* w;
    float* out;
    const float* residual;
    long long x_stride, w_stride, out_stride, res_stride;
    int M, N, K;
    int cols;                                    // rows of x of a CTA, a multiple of 16
    int ranks;                                   // CTAs of a cluster, which share a sum's runs
    int run_blocks, runs;                        // blocks of a run; runs that there are
    int* error;
};

template <int NT> constexpr int f3_stage() { return 3 * (F3_W_PLANE + NT * F3_KB * 2); }
template <int NT> constexpr size_t f3_smem() { return 1024 + 2 * f3_stage<NT>() + 64 + 4 * (F3_ROWS + NT) + 16; }

__device__ __forceinline__ float f3_peer(const void* local, int rank)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(peer_smem_addr(smem_addr(local), rank)) : "memory");
    return v;
}

// Four places of a row, zeros past K.
__device__ __forceinline__ float4 f3_fetch(const float* row, int k, int K)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k + 4 <= K) {
        asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(row + k) : "memory");
    } else if (k < K) {
        v.x = row[k];
        if (k + 1 < K)
            v.y = row[k + 1];
        if (k + 2 < K)
            v.z = row[k + 2];
    }
    return v;
}

__device__ __forceinline__ uint32_t f3_pair(float a, float b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
// What is left of two numbers without their bfloat16 parts (exact).
__device__ __forceinline__ void f3_rest(float& a, float& b, uint32_t pair)
{
    a -= __uint_as_float(pair << 16);
    b -= __uint_as_float(pair & 0xffff0000u);
}
__device__ __forceinline__ void f3_put(uint32_t at, uint32_t a, uint32_t b)
{
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(a), "r"(b) : "memory");
}
// Writes the three parts of four places, `plane` bytes apart; true if a number has no such parts.
__device__ __forceinline__ bool f3_split(float4 v, uint32_t at, uint32_t plane)
{
    uint32_t a = f3_pair(v.x, v.y), b = f3_pair(v.z, v.w);
    f3_put(at, a, b);
    f3_rest(v.x, v.y, a);
    f3_rest(v.z, v.w, b);
    a = f3_pair(v.x, v.y), b = f3_pair(v.z, v.w);
    f3_put(at + plane, a, b);
    f3_rest(v.x, v.y, a);
    f3_rest(v.z, v.w, b);
    f3_put(at + 2 * plane, f3_pair(v.x, v.y), f3_pair(v.z, v.w));
    const float rest = (v.x + v.y) + (v.z + v.w);        // (infinite parts leave infinities or no numbers)
    return !(fabsf(rest) < INFINITY);
}

template <int COUNT> __device__ __forceinline__ void f3_tmem_load(uint32_t at, uint32_t (&r)[COUNT])
{
    if constexpr (COUNT == 32) {
        tmem_load_32x32(at, r);
    } else if constexpr (COUNT == 16) {
        tmem_load_32x16(at, r);
    } else {
        static_assert(COUNT == 8);
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(at) : "memory");
    }
}
template <int COUNT> __device__ __forceinline__ void f3_tmem_store(uint32_t at, const uint32_t (&r)[COUNT])
{
    if constexpr (COUNT == 32)
        tmem_store_32x32(at, r);
    else if constexpr (COUNT == 16)
        tmem_store_32x16(at, r);
    else
        tmem_store_32x8(at, r);
}

// An output of a marked row, by multiply-adds (a rare event, out of line: its registers don't count against the loop).
__device__ __noinline__ float f3_by_hand(const float* x, const float* w, int K)
{
    float v = 0.f;
    for (int k = 0; k < K; ++k)
        v = fmaf(x[k], w[k], v);
    return v;
}

template <int NT>
__global__ void __launch_bounds__(F3_THREADS, NT == 16 ? 2 : 1)
gemm_f32_tc_kernel(const F3Params p)
{
    pdl_trigger();
    constexpr int STAGE = f3_stage<NT>(), X_PLANE = NT * F3_KB * 2, TMEM = 4 * NT;
    constexpr int HALF = NT / 2, PIECE = HALF < 32 ? HALF : 32, PIECES = HALF / PIECE;    // columns of a warp, and at a time
    constexpr int W_EACH = F3_ROWS / 16, X_EACH = NT / 16;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + 2 * STAGE);
    uint64_t* const full = bars;                 // [2] all threads: the stage is written, the accumulator's last sums are taken
    uint64_t* const done = bars + 2;             // [2] MMA commit: the stage is read, the accumulator is finished
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
    int* const marked = reinterpret_cast<int*>(bars + 8);        // [0] any; [1 + row of w], [129 + row of x]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ranks = p.ranks, rank = ranks > 1 ? (int)(blockIdx.x % ranks) : 0;
    const int n0 = (int)(blockIdx.x / ranks) * F3_ROWS, m0 = blockIdx.y * p.cols;
    const int all_blocks = (p.K + F3_KB - 1) / F3_KB;
    const int own = F3_RUNS / ranks;             // runs of a rank
    const int first_block = min(rank * own * p.run_blocks, all_blocks);
    const int blocks = min((rank + 1) * own * p.run_blocks, all_blocks) - first_block;

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], F3_THREADS);
            mbar_init(&done[i], 1);
        }
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, TMEM);
        tmem_relinquish();
    }
    for (int i = tid; i < 1 + F3_ROWS + NT; i += F3_THREADS)
        marked[i] = 0;
    // the first weights are asked for in L2 (and read after the wait: the kernel ahead may write them)
    if (tid < F3_ROWS && n0 + tid < p.N)
        for (int b = 0; b < min(blocks, 2); ++b) {
            const float* at = p.w + (size_t)(n0 + tid) * p.w_stride + (first_block + b) * F3_KB;
            prefetch_l2(at);
            if ((first_block + b) * F3_KB + 32 < p.K)
                prefetch_l2(at + 32);
        }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();

    const int quarter = warp & 3, half = warp >> 2;              // a warp's TMEM lanes and its columns
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + half * HALF;
    const uint32_t idesc = make_idesc_bf16_f32(F3_ROWS, p.cols);
    auto multiply = [&](int st) {
        const uint32_t w_s = smem_addr(smem + st * STAGE), x_s = w_s + 3 * F3_W_PLANE;
        auto product = [&](int pw, int px, int ks, uint32_t more) {
            tcgen05_mma_bf16(tmem + st * NT, make_kmajor_sw128_desc(w_s + pw * F3_W_PLANE + ks * 32),
                             make_kmajor_sw128_desc(x_s + px * X_PLANE + ks * 32), idesc, more);
        };
#pragma unroll
        for (int ks = 0; ks < F3_KB / 16; ++ks) {
            product(2, 0, ks, ks > 0 ? 1u : 0u);
            product(1, 1, ks, 1u);
            product(1, 0, ks, 1u);
            product(0, 2, ks, 1u);
            product(0, 1, ks, 1u);
        }
#pragma unroll
        for (int ks = 0; ks < F3_KB / 16; ++ks)
            product(0, 0, ks, 1u);
        tcgen05_commit(&done[st]);
    };
    {
        const int quad = tid & 15, r0 = tid >> 4;                // four places of rows r0 + 16 i
        const float* const w_row = p.w + (size_t)(n0 + r0) * p.w_stride;
        const float* const x_row = p.x + (size_t)(m0 + r0) * p.x_stride;
        const uint32_t to = smem_addr(smem) + (r0 >> 3) * 1024 + (r0 & 7) * 128 + (((quad >> 1) ^ (r0 & 7)) << 4) + (quad & 1) * 8;
        float4 wv[W_EACH], xv[X_EACH];
        auto fetch = [&](int i) {
            const int k = (first_block + i) * F3_KB + 4 * quad;
#pragma unroll
            for (int j = 0; j < W_EACH; ++j)
                wv[j] = f3_fetch(w_row + 16 * j * p.w_stride, k, n0 + r0 + 16 * j < p.N ? p.K : 0);
#pragma unroll
            for (int j = 0; j < X_EACH; ++j)
                xv[j] = f3_fetch(x_row + 16 * j * p.x_stride, k, m0 + r0 + 16 * j < p.M && r0 + 16 * j < p.cols ? p.K : 0);
        };
        float run[HALF];
        // Adds block i's accumulator to its run, and a run that is finished to what came before it, in TMEM: by halves, or, where
        // a rank has two runs or one, each by itself.
        auto take = [&](int i) {
            const int st = i & 1, at = first_block + i;
            const bool opens = at % p.run_blocks == 0, closes = (at + 1) % p.run_blocks == 0 || i + 1 == blocks;
            tcgen05_fence_after();
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
                uint32_t v[PIECE];
                f3_tmem_load(lanes + st * NT + c * PIECE, v);
                tmem_load_wait();
#pragma unroll
                for (int u = 0; u < PIECE; ++u)
                    run[c * PIECE + u] = opens ? __uint_as_float(v[u]) : run[c * PIECE + u] + __uint_as_float(v[u]);
            }
            if (closes) {
                const int r = at / p.run_blocks;
                const int slot = ranks >= 4 ? r - rank * own : ranks == 2 ? 0 : r / 4;
                const bool joins = ranks <= 2 && r % 4 != 0;
#pragma unroll
                for (int c = 0; c < PIECES; ++c) {
                    uint32_t v[PIECE];
                    if (joins) {
                        f3_tmem_load(lanes + (2 + slot) * NT + c * PIECE, v);
                        tmem_load_wait();
                    }
#pragma unroll
                    for (int u = 0; u < PIECE; ++u)
                        v[u] = __float_as_uint(joins ? __uint_as_float(v[u]) + run[c * PIECE + u] : run[c * PIECE + u]);
                    f3_tmem_store(lanes + (2 + slot) * NT + c * PIECE, v);
                }
                tmem_store_wait();
            }
        };
        if (blocks > 0)
            fetch(0);
        for (int i = 0; i < blocks; ++i) {
            const int st = i & 1;
            if (i >= 2) {
                mbar_wait_warp(&done[st], ((i >> 1) - 1) & 1, p.error, 61);
                take(i - 2);
            }
#pragma unroll
            for (int j = 0; j < W_EACH; ++j)
                if (f3_split(wv[j], to + st * STAGE + j * 2048, F3_W_PLANE))
                    marked[1 + r0 + 16 * j] = marked[0] = 1;
#pragma unroll
            for (int j = 0; j < X_EACH; ++j)
                if (f3_split(xv[j], to + st * STAGE + 3 * F3_W_PLANE + j * 2048, X_PLANE))
                    marked[1 + F3_ROWS + r0 + 16 * j] = marked[0] = 1;
            fence_proxy_async();
            tcgen05_fence_before();
            mbar_arrive(&full[st]);
            if (i + 1 < blocks)
                fetch(i + 1);
            if (warp == 0) {
                if (elect_one()) {
                    mbar_wait(&full[st], (i >> 1) & 1, p.error, 62);
                    tcgen05_fence_after();
                    multiply(st);
                }
                __syncwarp();
            }
        }
        for (int i = max(blocks - 2, 0); i < blocks; ++i) {
            mbar_wait_warp(&done[i & 1], (i >> 1) & 1, p.error, 63);
            take(i);
        }
    }
    // ---- the whole sums: of this CTA alone, or of the cluster's through shared memory
    const int kept = ranks >= 4 ? own : 1;                       // sums of a rank
    float* const sums = reinterpret_cast<float*>(smem);          // [kept][column][row] (the stages are read)
    auto finish = [&](int m, int n, float v, bool by_hand) {
        if (m >= p.M || n >= p.N)
            return;
        if (by_hand)
            v = f3_by_hand(p.x + (size_t)m * p.x_stride, p.w + (size_t)n * p.w_stride, p.K);
        if (p.residual)
            v = p.residual[(size_t)m * p.res_stride + n] + v;
        p.out[(size_t)m * p.out_stride + n] = v;
    };
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    {
        const int slots = ranks == 1 ? (p.runs > 4 ? 2 : 1) : kept;
        const bool any = ranks == 1 && marked[0];
        const int row = quarter * 32 + lane;
#pragma unroll
        for (int c = 0; c < PIECES; ++c) {
            uint32_t a[PIECE], b[PIECE];
            const int col = half * HALF + c * PIECE;
            f3_tmem_load(lanes + 2 * NT + c * PIECE, a);
            if (slots > 1)
                f3_tmem_load(lanes + 3 * NT + c * PIECE, b);
            tmem_load_wait();
            if (ranks == 1) {
#pragma unroll
                for (int u = 0; u < PIECE; ++u)
                    if (col + u < p.cols)
                        finish(m0 + col + u, n0 + row, __uint_as_float(a[u]) + (slots > 1 ? __uint_as_float(b[u]) : 0.f),
                               any && (marked[1 + row] || marked[1 + F3_ROWS + col + u]));
            } else {
#pragma unroll
                for (int u = 0; u < PIECE; ++u) {
                    sums[(col + u) * F3_ROWS + row] = __uint_as_float(a[u]);
                    if (slots > 1)
                        sums[(NT + col + u) * F3_ROWS + row] = __uint_as_float(b[u]);
                }
            }
        }
    }
    if (ranks > 1) {
        cluster_sync();
        {
            bool any = false;
            for (int r = 0; r < ranks; ++r)
                any = any || __float_as_int(f3_peer(marked, r)) != 0;
            const int each = ranks >= 4 ? 1 : 4;                 // runs of a kept sum
            for (int i = rank * F3_THREADS + tid; i < p.cols * F3_ROWS; i += ranks * F3_THREADS) {
                const int col = i / F3_ROWS, row = i % F3_ROWS;
                float s[F3_RUNS];
#pragma unroll
                for (int r = 0; r < F3_RUNS; ++r)
                    if (r % each == 0 && r < p.runs)
                        s[r] = f3_peer(sums + (ranks >= 4 ? r % own : 0) * NT * F3_ROWS + i, r / own);
                float v = s[0], w = 0.f;
                if (each == 1) {
#pragma unroll
                    for (int r = 1; r < 4; ++r)
                        if (r < p.runs)
                            v += s[r];
                }
                if (p.runs > 4) {
                    w = s[4];
                    if (each == 1) {
#pragma unroll
                        for (int r = 5; r < 8; ++r)
                            if (r < p.runs)
                                w += s[r];
                    }
                    v += w;
                }
                bool by_hand = false;
                if (any)
                    for (int r = 0; r < ranks; ++r)
                        by_hand = by_hand || __float_as_int(f3_peer(marked + 1 + row, r)) || __float_as_int(f3_peer(marked + 1 + F3_ROWS + col, r));
                finish(m0 + col, n0 + row, v, by_hand);
            }
        }
        cluster_sync();                                          // nobody leaves while its sums are read
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) {
        tcgen05_fence_after();
        tmem_dealloc(tmem, TMEM);
    }
}

template <int NT>
static int f3_launch(const F3Params& p, cudaStream_t stream)
{
    auto kernel = gemm_f32_tc_kernel<NT>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f3_smem<NT>());
        if (e != cudaSuccess)
            return (int)e;
        configured = true;
    }
    const dim3 grid((unsigned)((p.N + F3_ROWS - 1) / F3_ROWS * p.ranks), (unsigned)((p.M + p.cols - 1) / p.cols));
    if (p.ranks > 1)
        launch_cluster_x(kernel, grid, dim3(F3_THREADS), f3_smem<NT>(), stream, p.ranks, p);
    else
        launch(kernel, grid, dim3(F3_THREADS), f3_smem<NT>(), stream, p);
    return launch_status();
}

} // namespace chibi

using namespace chibi;

// All three operands 32-bit, rows of x and w on 16-byte boundaries, K > 0; CHIBI_ERR_UNSUPPORTED otherwise.
CHIBI_API int chibi_gemm_f32(const float* x, const float* w, float* out, const float* residual, int M, int N, int K,
                             long long x_stride, long long w_stride, long long out_stride, long long res_stride,
                             int cols, int ranks, int* error, cudaStream_t stream)
{
    if (M <= 0 || N <= 0)
        return CHIBI_OK;
    if (K < 0 || cols < 0 || ranks < 0)
        return CHIBI_ERR_ARGUMENT;
    if (K == 0 || ((uintptr_t)x | (uintptr_t)w) % 16 != 0 || x_stride % 4 != 0 || w_stride % 4 != 0)
        return CHIBI_ERR_UNSUPPORTED;
    F3Params p = { x, w, out, residual, x_stride, w_stride, out_stride, res_stride, M, N, K, 0, 1, 0, 0, error };
    const int blocks = (K + F3_KB - 1) / F3_KB;
    p.run_blocks = (blocks + F3_RUNS - 1) / F3_RUNS;
    p.runs = (blocks + p.run_blocks - 1) / p.run_blocks;
    // TODO rule
    const int tiles = (N + F3_ROWS - 1) / F3_ROWS, sms = device_sm_count();
    double least = 0.0;
    for (int parts = (M + 127) / 128; parts <= (M + 15) / 16; ++parts) {
        const int width = ((M + parts - 1) / parts + 15) / 16 * 16;
        if ((M + width - 1) / width != parts)
            continue;
        for (int r = 1; r <= F3_RUNS; r *= 2) {
            if ((r - 1) * (F3_RUNS / r) >= p.runs)
                break;                                           // (a CTA without a run)
            const long long ctas = (long long)tiles * parts * r, slots = width <= 16 ? 2 * sms : sms;
            const double rounds = (double)((ctas + slots - 1) / slots);
            const double block = 700.0 + 13.0 * width;
            const double cost = rounds * ((F3_RUNS / r < p.runs ? F3_RUNS / r : p.runs) * p.run_blocks * block + 3500.0 + (r > 1 ? 1500.0 + 10.0 * width : 0.0));
            if (p.cols == 0 || cost < least) {
                least = cost;
                p.cols = width;
                p.ranks = r;
            }
        }
    }
    if (cols > 0)
        p.cols = cols;
    if (ranks > 0)
        p.ranks = ranks;
    if (p.cols % 16 != 0 || p.cols > 128 || (p.ranks & (p.ranks - 1)) || p.ranks > F3_RUNS)
        return CHIBI_ERR_ARGUMENT;
    if ((M + p.cols - 1) / p.cols > 65535)
        return CHIBI_ERR_UNSUPPORTED;
    return p.cols <= 16 ? f3_launch<16>(p, stream) : p.cols <= 32 ? f3_launch<32>(p, stream)
        : p.cols <= 64 ? f3_launch<64>(p, stream) : f3_launch<128>(p, stream);
}
