// out[M, N] = x[M, K] * w[N, K]^T (+ residual[M, N]), all 32-bit, on the 5th-generation tensor cores.
//
// Numbers are split into three bfloat16 parts (split_f32.cuh), and six of the nine partial products are tcgen05.mma with
// 32-bit accumulators.  What limits the precision is the accumulator, which the tensor core cuts off instead of rounding:
// so a block of 64 places has an accumulator of its own, that takes the five small products of all its places first and the
// large one last (four roundings at the size of the sum), and the blocks are added up in plain 32-bit arithmetic.  Relative
// error against 64 bits
// (2-norm, normal numbers, K = 64 / 128 / 1,024 / 3,072 / 12,300): 7.9e-8 / 8.3e-8 / 9.6e-8 / 1.0e-7 / 1.3e-7; by multiply-adds
// (fma.rn.f32x2) before 1.1e-7 / 1.5e-7 / 1.6e-7 / 1.9e-7 / 3.6e-7.  What is cut off has a sign: operands of one sign (the same numbers
// without theirs) come out 0.84e-7 low at every K and lose 9.3e-8 in all, by multiply-adds 6.9e-8 / 9.2e-8 / 5.3e-8 / 4.4e-8 /
// 5.8e-8; the largest error of a result is 2.7e-7, and was 4.2e-7.
//
// The order of a sum depends on K alone: the blocks of 64 places lie in at most eight runs, a run's blocks are added in
// order, the first four runs in order, the other four in order, and the two halves at last.  So a row's result does not
// depend on the rows beside it, nor on which kernel makes it or how many CTAs share a sum (a cluster of 1, 2, 4 or 8 takes the
// runs in order).
//
// Sums are 2^32 as large as they should be until the end.  What has no parts (no number, or from 2^112 on) makes all sums of its row
// of x or w come out as no number.  Sums that do, and sums from 2^96 on, which come out infinite, are made by hand instead.
// (No loop looks for such numbers, which pays for the scaling: 300 rows through the feed-forward of 1,024 x 3,072 75.1 us with
// rows marked and w not scaled, 70.2 so.)
//
// A CTA owns 128 rows of w (the M of the MMA) and up to 128 rows of x (its N).  Eight or sixteen warps bring both from
// memory (in registers, one block ahead), split them and write the six tiles to one of two stages in shared memory in
// the swizzled K-major layout; a warp of its own issues the MMAs (an issuing thread waits while they run); and while they
// do, the others read the accumulator of the block before, in one of two buffers in TMEM, and add it up.  Bound by that work
// beside 24 MMAs a block (64 cycles each with 128 columns, and shared memory as long); tiles of 64 x 64 by multiply-adds were
// bound by their reads of shared memory.  Us by multiply-adds and so, in a replayed graph, weights in turn that L2 does not
// hold: 300 rows of 6,144 x 1,024 134 and 34, of 12,288 x 2,048 449 and 120, 1,200 rows 1,564 and 429 (141 TFLOP/s, 6 times as many
// products), 64 rows of 1,024 x 3,072 26 and 14.4.
#define CHIBI_UNIT gemm_f32_tcgen05
#define CHIBI_UNIT_ID 18
#include "common.cuh"
#include "sm100.cuh"
#include "split_f32.cuh"

namespace chibi {

using namespace sm100;

constexpr int F3_ROWS = 128, F3_KB = 64;         // rows of w; places of a block
constexpr int F3_RUNS = 8;
constexpr int F3_FEW_MANY = 8;                   // tiles an SM from which on there are many
constexpr int F3_FEW_WARPS = 16, F3_FEW_SHARED = 208 * 1024;     // of the kernel for few rows, on an SM
constexpr int F3_REGS = 96, F3_REGS_FEW = 32, F3_REGS_MANY = 112;    // of a thread at launch, of the first four warps', of the others' (sixteen)
static_assert(F3_REGS_FEW + 4 * F3_REGS_MANY <= 5 * F3_REGS, "more registers than the block has");
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
template <int NT> constexpr size_t f3_smem() { return 1024 + 2 * f3_stage<NT>() + 64; }

__device__ __forceinline__ float4 f3_peer4(const void* local, int rank)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(peer_smem_addr(smem_addr(local), rank)) : "memory");
    return v;
}

__device__ __forceinline__ float4 f3_load(const float* at)
{
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at) : "memory");
    return v;
}
// Four places of a row, zeros past K.
__device__ __forceinline__ float4 f3_load_end(const float* row, int k, int K)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < K)
        v.x = row[k];
    if (k + 1 < K)
        v.y = row[k + 1];
    if (k + 2 < K)
        v.z = row[k + 2];
    if (k + 3 < K)
        v.w = row[k + 3];
    return v;
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

// Outputs that the tensor cores cannot make (a rare event, out of line: its registers don't count against the loop, if they are not
// many: four outputs at a time cost a call of few rows 4 of 14 us without any such output), by a whole warp: of lane's `count`
// ones, (m + u * dm, n + u * dn), those with bit u of `bad`.  The warp reads the rows of one at a time in whole lines; sums are 64-bit, so
// that their order does not matter.  300 (4) rows of 6,144 x 1,024 without such a row 42 us (14); one row with an infinity 108 (112),
// one row that is no number 45 (17), all rows 58 (17), a row of w with an infinity 125 (18); by a chain of multiply-adds of one
// thread each 168 (134), 174 (141), 7,816 (162), 1,495 (39).
__device__ __noinline__ void f3_by_hand(const F3Params& p, uint32_t bad, int count, int m, int n, int dm, int dn)
{
    const int lane = threadIdx.x & 31;
    auto store = [&](int mm, int nn, float v) {
        p.out[(size_t)mm * p.out_stride + nn] = p.residual ? p.residual[(size_t)mm * p.res_stride + nn] + v : v;
    };
    for (int u = 0; u < count; ++u) {
        const int own_m = m + u * dm, own_n = n + u * dn;
        bool mine = bad >> u & 1u;
        if (mine) {
            // (a row of which nothing is a number is one from its first place on: every lane looks for itself)
            const float a = p.x[(size_t)own_m * p.x_stride], b = p.w[(size_t)own_n * p.w_stride];
            if (a != a || b != b) {
                store(own_m, own_n, NAN);
                mine = false;
            }
        }
        for (uint32_t left = __ballot_sync(0xffffffffu, mine); left; left &= left - 1) {
            const int from = __ffs(left) - 1, mm = __shfl_sync(0xffffffffu, own_m, from), nn = __shfl_sync(0xffffffffu, own_n, from);
            const float* const x = p.x + (size_t)mm * p.x_stride;
            const float* const w = p.w + (size_t)nn * p.w_stride;
            double s = 0.0;
            for (int k0 = 4 * lane; k0 < (p.K + 511) / 512 * 512; k0 += 512) {
                float4 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = k0 + 128 * i;
                    a[i] = k + 4 <= p.K ? *reinterpret_cast<const float4*>(x + k) : f3_load_end(x, k, p.K);
                    b[i] = k + 4 <= p.K ? *reinterpret_cast<const float4*>(w + k) : f3_load_end(w, k, p.K);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s = fma((double)a[i].x, (double)b[i].x, s);
                    s = fma((double)a[i].y, (double)b[i].y, s);
                    s = fma((double)a[i].z, (double)b[i].z, s);
                    s = fma((double)a[i].w, (double)b[i].w, s);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == from)
                store(mm, nn, (float)s);
            __syncwarp();
        }
    }
}

template <int NT, int WORKERS>
__global__ void __launch_bounds__(WORKERS == 256 ? 288 : 640, WORKERS == 256 ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ F3Params p)
{
    pdl_trigger();
    constexpr int OTHERS = WORKERS == 256 ? 32 : 128;
    constexpr int STAGE = f3_stage<NT>(), X_PLANE = NT * F3_KB * 2, TMEM = 4 * NT;
    constexpr int SHARES = WORKERS / F3_ROWS, COLS = NT / SHARES;        // threads of a row of w; a thread's rows of x
    constexpr int PIECE = COLS < 16 ? COLS : 16, PIECES = COLS / PIECE;
    constexpr int PASS = WORKERS / 16, W_EACH = F3_ROWS / PASS, X_EACH = NT / PASS;
    static_assert(NT % PASS == 0);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + 2 * STAGE);
    uint64_t* const full = bars;                 // [2] workers: the stage is written
    uint64_t* const done = bars + 2;             // [2] MMA commit: the stage is read, the accumulator is finished
    uint64_t* const taken = bars + 4;            // [2] workers: the accumulator is read
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ranks = p.ranks, rank = ranks > 1 ? (int)(blockIdx.x % ranks) : 0;
    const int n0 = (int)(blockIdx.x / ranks) * F3_ROWS, m0 = blockIdx.y * p.cols;
    const int all_blocks = (p.K + F3_KB - 1) / F3_KB;
    const int own = F3_RUNS / ranks;             // runs of a rank
    const int first_block = min(rank * own * p.run_blocks, all_blocks);
    const int blocks = min((rank + 1) * own * p.run_blocks, all_blocks) - first_block;

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], WORKERS);
            mbar_init(&done[i], 1);
            mbar_init(&taken[i], WORKERS);
        }
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, TMEM);
        tmem_relinquish();
    }
    // the first weights are asked for in L2 (and read after the wait: the kernel ahead may write them)
    if (tid >= OTHERS && tid < OTHERS + F3_ROWS && n0 + tid - OTHERS < p.N)
        for (int b = 0; b < min(blocks, 4); ++b) {
            const float* at = p.w + (size_t)(n0 + tid - OTHERS) * p.w_stride + (first_block + b) * F3_KB;
            prefetch_l2(at);
            if ((first_block + b) * F3_KB + 32 < p.K)
                prefetch_l2(at + 32);
        }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();

    const int quarter = warp & 3, share = (tid - OTHERS) / F3_ROWS;      // a worker's TMEM lanes and its columns
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + share * COLS;
    if (tid < OTHERS) {
        if (WORKERS == 512)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F3_REGS_FEW));
        if (warp == 0 && elect_one()) {
            const uint32_t idesc = make_idesc_bf16_f32(F3_ROWS, p.cols);
            const uint32_t w_s = smem_addr(smem);
            for (int i = 0; i < blocks; ++i) {
                const int st = i & 1;
                uint64_t a = make_kmajor_sw128_desc(w_s + st * STAGE), b = make_kmajor_sw128_desc(w_s + st * STAGE + 3 * F3_W_PLANE);
                asm volatile("" : "+l"(a), "+l"(b));     // (or sums of constants wait in registers from block to block)
                mbar_wait(&full[st], (i >> 1) & 1, p.error, 61);
                if (i >= 2)
                    mbar_wait(&taken[st], ((i >> 1) - 1) & 1, p.error, 62);
                tcgen05_fence_after();
                const uint32_t d = tmem + st * NT;
                auto product = [&](int pw, int px, int ks, uint32_t more) {
                    tcgen05_mma_bf16(d, a + ((pw * F3_W_PLANE + ks * 32) >> 4), b + ((px * X_PLANE + ks * 32) >> 4), idesc, more);
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
            }
        }
        __syncwarp();
        if (ranks > 1) {                                         // (as the others below)
            cluster_sync();
            cluster_sync();
        }
    } else {
        if (WORKERS == 512)
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(F3_REGS_MANY));
        const int worker = tid - OTHERS, quad = worker & 15, line = worker >> 4;     // four places of rows line + PASS i
        // (rows past the end bring the last one's numbers: what they give is not stored)
        const float* const w0 = p.w + (size_t)n0 * p.w_stride;
        const float* const x0 = p.x + (size_t)m0 * p.x_stride;
        const int w_last = p.N - 1 - n0, x_last = min(p.M - 1 - m0, p.cols - 1);
        const uint32_t to = smem_addr(smem) + (line >> 3) * 1024 + (line & 7) * 128 + (((quad >> 1) ^ (line & 7)) << 4) + (quad & 1) * 8;
        float4 wv[W_EACH], xv[X_EACH];
        auto fetch = [&](int i) {
            const int k = (first_block + i) * F3_KB + 4 * quad;
            if ((first_block + i + 1) * F3_KB <= p.K) {
#pragma unroll
                for (int j = 0; j < W_EACH; ++j)
                    wv[j] = f3_load(w0 + min(line + PASS * j, w_last) * p.w_stride + k);
#pragma unroll
                for (int j = 0; j < X_EACH; ++j)
                    xv[j] = f3_load(x0 + min(line + PASS * j, x_last) * p.x_stride + k);
            } else {
#pragma unroll
                for (int j = 0; j < W_EACH; ++j)
                    wv[j] = f3_load_end(w0 + min(line + PASS * j, w_last) * p.w_stride, k, p.K);
#pragma unroll
                for (int j = 0; j < X_EACH; ++j)
                    xv[j] = f3_load_end(x0 + min(line + PASS * j, x_last) * p.x_stride, k, p.K);
            }
        };
        auto spread = [&](int st) {
#pragma unroll
            for (int j = 0; j < W_EACH; ++j)
                split_to_shared(wv[j], to + st * STAGE + j * (PASS / 8) * 1024, F3_W_PLANE);
#pragma unroll
            for (int j = 0; j < X_EACH; ++j)
                split_to_shared(xv[j], to + st * STAGE + 3 * F3_W_PLANE + j * (PASS / 8) * 1024, X_PLANE);
        };
        uint64_t run[COLS / 2];
        // Adds block i's accumulator to its run, and a run that is finished to what came before it, in TMEM: by halves, or, where
        // a rank has two runs or one, each by itself.
        auto take = [&](int i) {
            const int st = i & 1, at = first_block + i;
            mbar_wait_warp(&done[st], (i >> 1) & 1, p.error, 64);
            tcgen05_fence_after();
            if (at % p.run_blocks == 0) {
#pragma unroll
                for (int c = 0; c < COLS / 2; ++c)
                    run[c] = 0;
            }
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
                uint32_t v[PIECE];
                f3_tmem_load(lanes + st * NT + c * PIECE, v);
                tmem_load_wait();
#pragma unroll
                for (int u = 0; u < PIECE / 2; ++u)
                    run[c * PIECE / 2 + u] = pair_fma(run[c * PIECE / 2 + u], PAIR_ONES, pair_of(__uint_as_float(v[2 * u]), __uint_as_float(v[2 * u + 1])));
            }
            tcgen05_fence_before();
            mbar_arrive(&taken[st]);
            if ((at + 1) % p.run_blocks == 0 || i + 1 == blocks) {
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
                    for (int u = 0; u < PIECE / 2; ++u) {
                        const float2 h = halves_of(run[c * PIECE / 2 + u]);
                        v[2 * u] = __float_as_uint(joins ? __uint_as_float(v[2 * u]) + h.x : h.x);
                        v[2 * u + 1] = __float_as_uint(joins ? __uint_as_float(v[2 * u + 1]) + h.y : h.y);
                    }
                    f3_tmem_store(lanes + (2 + slot) * NT + c * PIECE, v);
                }
                tmem_store_wait();
            }
        };
        if (blocks > 0)
            fetch(0);
        for (int i = 0; i < blocks; ++i) {
            const int st = i & 1;
            if (i >= 2)
                mbar_wait_warp(&done[st], ((i >> 1) - 1) & 1, p.error, 63);
            spread(st);
            if (i + 1 < blocks)
                fetch(i + 1);
            fence_proxy_async();
            mbar_arrive(&full[st]);
            if (i >= 2)
                take(i - 2);
        }
        for (int i = max(blocks - 2, 0); i < blocks; ++i)
            take(i);
        // ---- the whole sums: of this CTA alone, or of the cluster's through shared memory
        const int kept = ranks >= 4 ? own : 1;                       // sums of a rank
        float* const sums = reinterpret_cast<float*>(smem);          // [kept][column][row] (the stages are read: this thread has
                                                                     // waited for the last products)
        // stores an output; true if it is to be made by hand
        auto finish = [&](int m, int n, float v) {
            if (m >= p.M || n >= p.N)
                return false;
            v *= SPLIT_DOWN;
            if (!(fabsf(v) < INFINITY))
                return true;
            if (p.residual)
                v = p.residual[(size_t)m * p.res_stride + n] + v;
            p.out[(size_t)m * p.out_stride + n] = v;
            return false;
        };
        {
            const int slots = ranks == 1 ? (p.runs > 4 ? 2 : 1) : kept;
            const int row = quarter * 32 + lane;
#pragma unroll
            for (int c = 0; c < PIECES; ++c) {
                uint32_t a[PIECE], b[PIECE];
                const int col = share * COLS + c * PIECE;
                f3_tmem_load(lanes + 2 * NT + c * PIECE, a);
                if (slots > 1)
                    f3_tmem_load(lanes + 3 * NT + c * PIECE, b);
                tmem_load_wait();
                if (ranks == 1) {
                    uint32_t bad = 0;
#pragma unroll
                    for (int u = 0; u < PIECE; ++u)
                        if (col + u < p.cols
                            && finish(m0 + col + u, n0 + row, __uint_as_float(a[u]) + (slots > 1 ? __uint_as_float(b[u]) : 0.f)))
                            bad |= 1u << u;
                    if (__any_sync(0xffffffffu, bad != 0))
                        f3_by_hand(p, bad, PIECE, m0 + col, n0 + row, 1, 0);
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
                // (four rows of w at a time: what bounds this is the number of reads from the other CTAs)
                const int each = ranks >= 4 ? 1 : 4;                 // runs of a kept sum
                for (int i = 4 * (rank * WORKERS + tid - OTHERS); i < p.cols * F3_ROWS; i += 4 * ranks * WORKERS) {
                    const int col = i / F3_ROWS, row = i % F3_ROWS;
                    if (m0 + col >= p.M)                             // (a warp has one column; rows past the end are not stored)
                        continue;
                    float4 s[F3_RUNS];
#pragma unroll
                    for (int r = 0; r < F3_RUNS; ++r)
                        if (r % each == 0 && r < p.runs)
                            s[r] = f3_peer4(sums + (ranks >= 4 ? r % own : 0) * NT * F3_ROWS + i, r / own);
                    float4 v = s[0];
                    auto add = [](float4& to, float4 x) { to.x += x.x, to.y += x.y, to.z += x.z, to.w += x.w; };
                    if (each == 1) {
#pragma unroll
                        for (int r = 1; r < 4; ++r)
                            if (r < p.runs)
                                add(v, s[r]);
                    }
                    if (p.runs > 4) {
                        float4 w = s[4];
                        if (each == 1) {
#pragma unroll
                            for (int r = 5; r < 8; ++r)
                                if (r < p.runs)
                                    add(w, s[r]);
                        }
                        add(v, w);
                    }
                    uint32_t bad = finish(m0 + col, n0 + row, v.x) ? 1u : 0u;
                    bad |= finish(m0 + col, n0 + row + 1, v.y) ? 2u : 0u;
                    bad |= finish(m0 + col, n0 + row + 2, v.z) ? 4u : 0u;
                    bad |= finish(m0 + col, n0 + row + 3, v.w) ? 8u : 0u;
                    if (__any_sync(0xffffffffu, bad != 0))
                        f3_by_hand(p, bad, 4, m0 + col, n0 + row, 0, 1);
                }
            }
            cluster_sync();                                          // nobody leaves while its sums are read
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) {
        tcgen05_fence_after();
        tmem_dealloc(tmem, TMEM);
    }
}

// ---------------------------------------------------------------- few rows
// The same sums, bit for bit, by mma.sync m16n8k16 straight from registers (the tensor core adds up sixteen places the same way
// whichever instruction asks for it, and whatever their order): no TMEM, swizzled tiles or barriers on the way, which cost a call
// of few rows more than its weights.  A CTA has tiles of 16 rows of w, its warps take a tile's blocks in turn.  A warp brings
// 16 x 64 numbers (eight pieces of 16 bytes a lane, a row's 64 bytes by four lanes; the places of a fragment are taken as they
// lie), splits sixteen places, asks for the next block's in their stead and multiplies; a block's or a run's sums go to shared
// memory, where they are put together in order.  Bound by the weights' way from memory, with many of them by mma.sync's rate.  Us by
// multiply-adds and so, one / four / eight / sixteen rows, in a replayed graph, weights in turn that L2 does not hold (the same
// weights again, where they fit: 0.3 to 2 less): 4,096 x 1,024 5.8, 6.4, 7.8, 11.3 and 5.7, 5.7, 5.8, 8.6; 1,024 x 3,072 7.1, 8.1, 10.1, 13.7
// and 7.0, 7.1, 7.3, 10.9; 6,144 x 1,024 7.2, 8.3, 10.9, 16.1 and 8.1, 8.0, 8.1, 13.0; 2,048 x 6,144 12.7, 14.1, 18.4, 25.6 and 13.3, 13.7, 14.2,
// 20.9; 151,936 x 1,024 107, 131, 137, 176 and 103, 115, 116, 177.
template <int TILES, int WARPS, bool KEPT>                   // eights of rows of x; warps; x stays split in shared memory
__global__ void __launch_bounds__(32 * WARPS, F3_FEW_WARPS / WARPS)
gemm_f32_few_kernel(const __grid_constant__ F3Params p, int w_tiles)
{
    pdl_trigger();
    // sixteen warps take the blocks in turn; eight a run each, so that there is less to put together
    constexpr int XS = 8 * TILES, THREADS = 32 * WARPS, OWN = WARPS < 16 ? F3_RUNS / WARPS : 0;
    extern __shared__ __align__(16) float kept_sums[];       // [block, or turn and run][row of x][row of w]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int blocks = (p.K + F3_KB - 1) / F3_KB;
    const int begin = OWN ? min(warp * OWN * p.run_blocks, blocks) : warp, end = OWN ? min((warp + 1) * OWN * p.run_blocks, blocks) : blocks;
    constexpr int STEP = OWN ? 1 : WARPS;                    // a warp's blocks
    // the first weights are asked for in L2 (and read after the wait: the kernel ahead may write them); a line to a lane
    for (int b = begin; b < min(end, begin + 2 * STEP); b += STEP) {
        const int n = blockIdx.x * 16 + (lane >> 1), k = b * F3_KB + 32 * (lane & 1);
        if (n < p.N && k < p.K)
            prefetch_l2(p.w + (size_t)n * p.w_stride + k);
    }
    pdl_wait();

    float4 wn[2][4], xn[TILES][4];                           // rows g and g + 8 of the tile, row g of every eight of x (if not KEPT)
    const float* at_w[2];                                    // where the block to be fetched lies in those rows
    const float* at_x[TILES];
    int at_k = 0;
    auto aim = [&](int tile, int block) {
        at_k = block * F3_KB;
#pragma unroll
        for (int i = 0; i < 2; ++i)                          // (rows past the end: not stored)
            at_w[i] = p.w + min(tile * 16 + g + 8 * i, p.N - 1) * p.w_stride + at_k + 4 * t;
        if (!KEPT) {
#pragma unroll
            for (int i = 0; i < TILES; ++i)
                at_x[i] = p.x + min(8 * i + g, p.M - 1) * p.x_stride + at_k + 4 * t;
        }
    };
    auto fetch = [&](int ks) {                               // places 16 ks + 4 t .. + 3
        if (at_k + F3_KB <= p.K) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
                wn[i][ks] = f3_load(at_w[i] + 16 * ks);
            if (!KEPT) {
#pragma unroll
                for (int i = 0; i < TILES; ++i)
                    xn[i][ks] = *reinterpret_cast<const float4*>(at_x[i] + 16 * ks);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i)
                wn[i][ks] = f3_load_end(at_w[i] + 16 * ks, 0, p.K - at_k - 16 * ks - 4 * t);
            if (!KEPT) {
#pragma unroll
                for (int i = 0; i < TILES; ++i)
                    xn[i][ks] = f3_load_end(at_x[i] + 16 * ks, 0, p.K - at_k - 16 * ks - 4 * t);
            }
        }
    };
    // (KEPT) the parts of a block's sixteen places of eight rows of x: two words of each part, a lane's beside its neighbours'
    uint4* const kept4 = reinterpret_cast<uint4*>(kept_sums + 2 * F3_RUNS * XS * 16);
    uint2* const kept2 = reinterpret_cast<uint2*>(kept4 + blocks * 4 * TILES * 32);
    auto kept_at = [&](int b, int ks, int i) { return ((b * 4 + ks) * TILES + i) * 32 + lane; };
    if (begin < end && (int)blockIdx.x < w_tiles) {
        aim(blockIdx.x, begin);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
            fetch(ks);
    }
    if (KEPT) {                                              // (every warp those of its own blocks)
        for (int b = begin; b < end; ++b)
#pragma unroll
            for (int i = 0; i < TILES; ++i) {
                const float* const row = p.x + min(8 * i + g, p.M - 1) * p.x_stride;
                float4 v[4];
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    const int k = b * F3_KB + 16 * ks + 4 * t;
                    v[ks] = k + 4 <= p.K ? *reinterpret_cast<const float4*>(row + k) : f3_load_end(row, k, p.K);
                }
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    uint32_t parts[3][2];
                    split_parts(v[ks], parts);
                    kept4[kept_at(b, ks, i)] = make_uint4(parts[0][0], parts[0][1], parts[1][0], parts[1][1]);
                    kept2[kept_at(b, ks, i)] = make_uint2(parts[2][0], parts[2][1]);
                }
            }
        __syncwarp();
    }
    int turn = 0;
    for (int tile = blockIdx.x; tile < w_tiles; tile += gridDim.x, turn ^= 1) {
        float* const sums = kept_sums + (OWN ? turn * F3_RUNS * XS * 16 : 0);
        float run[TILES][4];
        for (int b = begin; b < end; b += STEP) {
            // (the next block of this tile, or the first of the next one)
            const bool same = b + STEP < end, more = same || tile + (int)gridDim.x < w_tiles;
            if (more)
                aim(same ? tile : tile + (int)gridDim.x, same ? b + STEP : begin);
            float d[TILES][4];
            uint32_t w0[4][4], x0[TILES][4][2];              // the leading parts, for the large products at last
#pragma unroll
            for (int i = 0; i < TILES; ++i)
                d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.f;
            auto product = [&](const uint32_t (&wf)[4], int i, uint32_t low, uint32_t high) {
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                             "{%0, %1, %2, %3};"
                             : "+f"(d[i][0]), "+f"(d[i][1]), "+f"(d[i][2]), "+f"(d[i][3])
                             : "r"(wf[0]), "r"(wf[1]), "r"(wf[2]), "r"(wf[3]), "r"(low), "r"(high));
            };
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t low[3][2], high[3][2], wf[3][4], xf[TILES][3][2];
                if (KEPT) {
#pragma unroll
                    for (int i = 0; i < TILES; ++i) {
                        const uint4 a = kept4[kept_at(b, ks, i)];
                        const uint2 c = kept2[kept_at(b, ks, i)];
                        xf[i][0][0] = a.x, xf[i][0][1] = a.y, xf[i][1][0] = a.z, xf[i][1][1] = a.w, xf[i][2][0] = c.x, xf[i][2][1] = c.y;
                    }
                }
                split_parts(wn[0][ks], low);
                split_parts(wn[1][ks], high);
                if (!KEPT) {
#pragma unroll
                    for (int i = 0; i < TILES; ++i)
                        split_parts(xn[i][ks], xf[i]);
                }
                if (more)
                    fetch(ks);
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    wf[j][0] = low[j][0], wf[j][1] = high[j][0], wf[j][2] = low[j][1], wf[j][3] = high[j][1];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    w0[ks][c] = wf[0][c];
                constexpr int pw[5] = { 2, 1, 1, 0, 0 }, px[5] = { 0, 1, 0, 2, 1 };
#pragma unroll
                for (int q = 0; q < 5; ++q)
#pragma unroll
                    for (int i = 0; i < TILES; ++i)
                        product(wf[pw[q]], i, xf[i][px[q]][0], xf[i][px[q]][1]);
#pragma unroll
                for (int i = 0; i < TILES; ++i)
                    x0[i][ks][0] = xf[i][0][0], x0[i][ks][1] = xf[i][0][1];
            }
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                for (int i = 0; i < TILES; ++i)
                    product(w0[ks], i, x0[i][ks][0], x0[i][ks][1]);
            const bool opens = OWN && b % p.run_blocks == 0;
            if (OWN) {
#pragma unroll
                for (int i = 0; i < TILES; ++i)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        run[i][c] = opens ? d[i][c] : run[i][c] + d[i][c];
            }
            if (!OWN || (b + 1) % p.run_blocks == 0 || b + 1 == end) {
                float* const to = sums + (OWN ? b / p.run_blocks : b) * XS * 16;
#pragma unroll
                for (int i = 0; i < TILES; ++i)
#pragma unroll
                    for (int c = 0; c < 4; ++c)              // columns 2 t, 2 t + 1 of rows g, g + 8
                        to[(8 * i + 2 * t + (c & 1)) * 16 + g + 8 * (c >> 1)] = OWN ? run[i][c] : d[i][c];
            }
        }
        __syncthreads();
        for (int o = threadIdx.x; o < XS * 16; o += THREADS) {       // (whole warps)
            const int m = o / 16, n = tile * 16 + o % 16;
            float s[F3_RUNS];
            if (OWN) {
#pragma unroll
                for (int r = 0; r < F3_RUNS; ++r)
                    if (r < p.runs)
                        s[r] = sums[r * XS * 16 + o];
            } else {
#pragma unroll
                for (int r = 0; r < F3_RUNS; ++r)            // (all runs at a time: eight short chains)
                    if (r < p.runs)
                        s[r] = sums[r * p.run_blocks * XS * 16 + o];
                for (int b = 1; b < p.run_blocks; ++b)
#pragma unroll
                    for (int r = 0; r < F3_RUNS; ++r)
                        if (r * p.run_blocks + b < blocks)
                            s[r] += sums[(r * p.run_blocks + b) * XS * 16 + o];
            }
            float v = s[0];
#pragma unroll
            for (int r = 1; r < 4; ++r)
                if (r < p.runs)
                    v += s[r];
            if (p.runs > 4) {
                float half = s[4];
#pragma unroll
                for (int r = 5; r < 8; ++r)
                    if (r < p.runs)
                        half += s[r];
                v += half;
            }
            v *= SPLIT_DOWN;
            const bool in = m < p.M && n < p.N, bad = in && !(fabsf(v) < INFINITY);
            if (in && !bad)
                p.out[(size_t)m * p.out_stride + n] = p.residual ? p.residual[(size_t)m * p.res_stride + n] + v : v;
            if (__any_sync(0xffffffffu, bad))
                f3_by_hand(p, bad ? 1u : 0u, 1, m, n, 0, 0);
        }
        // (the sums of a turn are written again only behind the next turn's barrier; there is one tile to a CTA of sixteen warps, or
        // few)
        if (!OWN)
            __syncthreads();
    }
}

template <int TILES, int WARPS, bool KEPT>
static int f3_few(const F3Params& p, size_t shared, cudaStream_t stream)
{
    auto kernel = gemm_f32_few_kernel<TILES, WARPS, KEPT>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F3_FEW_SHARED);
        if (e != cudaSuccess)
            return (int)e;
        configured = true;
    }
    const int w_tiles = (p.N + 15) / 16, walkers = device_sm_count() * F3_FEW_WARPS / WARPS;
    launch(kernel, dim3((unsigned)(w_tiles < walkers ? w_tiles : walkers)), dim3(32 * WARPS), shared, stream, p, w_tiles);
    return launch_status();
}

// Which form of it, by how many tiles of 16 rows of w there are: one CTA of sixteen warps an SM where every tile has one at once
// (1,024 x 2,048, eight rows, 5.0 us; eight warps 6.0), or two rounds and a half do (6,144 x 1,024 7.6 and 8.2); eight warps
// where two to an SM have one round (4,096 x 1,024 5.1 and 5.6) or many (12,288 x 2,048 21.0 and 24.0); from eight
// tiles an SM on, x is split once and kept (151,936 x 1,024 103 and 114; 12,288 x 2,048 29.0).
template <int TILES>
static int f3_few_rows(const F3Params& p, int form, cudaStream_t stream)
{
    const int w_tiles = (p.N + 15) / 16, sms = device_sm_count(), blocks = (p.K + F3_KB - 1) / F3_KB;
    const size_t tile = (size_t)TILES * 8 * 16 * sizeof(float), runs = 2 * F3_RUNS * tile;
    const size_t split = runs + (size_t)blocks * 4 * TILES * 32 * 24;    // with all of x split
    const bool keeps = split <= (size_t)F3_FEW_SHARED / 2;
    if (form == 0)
        form = w_tiles <= sms || (w_tiles > 2 * sms && w_tiles <= 3 * sms) ? 16 : w_tiles < F3_FEW_MANY * sms || !keeps ? 8 : 4;
    if (form == 16 && (size_t)blocks * tile <= (size_t)F3_FEW_SHARED)
        return f3_few<TILES, 16, false>(p, blocks * tile, stream);
    return form == 4 && keeps ? f3_few<TILES, 8, true>(p, split, stream) : f3_few<TILES, 8, false>(p, runs, stream);
}

template <int NT, int WORKERS>
static int f3_launch(const F3Params& p, cudaStream_t stream)
{
    auto kernel = gemm_f32_tc_kernel<NT, WORKERS>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f3_smem<NT>());
        // (threads that asked for more registers than the block was launched with would wait for good)
        cudaFuncAttributes attr {};
        const cudaError_t a = e == cudaSuccess ? cudaFuncGetAttributes(&attr, kernel) : e;
        if (a != cudaSuccess)
            return (int)a;
        if (WORKERS == 512 && attr.numRegs < F3_REGS)
            return CHIBI_ERR_ARGUMENT;
        configured = true;
    }
    const int threads = WORKERS == 256 ? 288 : 640;
    const dim3 grid((unsigned)((p.N + F3_ROWS - 1) / F3_ROWS * p.ranks), (unsigned)((p.M + p.cols - 1) / p.cols));
    if (p.ranks > 1)
        launch_cluster_x(kernel, grid, dim3(threads), f3_smem<NT>(), stream, p.ranks, p);
    else
        launch(kernel, grid, dim3(threads), f3_smem<NT>(), stream, p);
    return launch_status();
}

} // namespace chibi

using namespace chibi;

// All three operands 32-bit, rows of x and w on 16-byte boundaries, K > 0; CHIBI_ERR_UNSUPPORTED otherwise.  cols and ranks are
// chosen if 0.  Any choice gives the same sums: `cols` rows of x to a CTA (a multiple of 16 up to 128) and `ranks` CTAs to a
// sum's runs, or, for at most 16 rows, the kernel for few with a form of -cols (4: x split once, 8 or 16 warps to a CTA).
CHIBI_API int chibi_gemm_f32(const float* x, const float* w, float* out, const float* residual, int M, int N, int K,
                             long long x_stride, long long w_stride, long long out_stride, long long res_stride,
                             int cols, int ranks, int* error, cudaStream_t stream)
{
    if (M <= 0 || N <= 0)
        return CHIBI_OK;
    if (K < 0 || ranks < 0)
        return CHIBI_ERR_ARGUMENT;
    if (K == 0 || ((uintptr_t)x | (uintptr_t)w) % 16 != 0 || x_stride % 4 != 0 || w_stride % 4 != 0)
        return CHIBI_ERR_UNSUPPORTED;
    F3Params p = { x, w, out, residual, x_stride, w_stride, out_stride, res_stride, M, N, K, 0, 1, 0, 0, error };
    const int blocks = (K + F3_KB - 1) / F3_KB;
    p.run_blocks = (blocks + F3_RUNS - 1) / F3_RUNS;
    p.runs = (blocks + p.run_blocks - 1) / p.run_blocks;
    // To 16 rows the kernel for few; but mma.sync does 16 x 8 x 16 products in 32 cycles of a quarter of an SM, and with
    // 9 to 16 rows and many rows of w that is what bounds it (151,936 x 1,024: 232 us and 176 here, 8 rows 107).
    const int sms = device_sm_count();
    if (cols <= 0 && (M <= 8 || (M <= 16 && (N + 15) / 16 < F3_FEW_MANY * sms)))
        return M <= 8 ? f3_few_rows<1>(p, -cols, stream) : f3_few_rows<2>(p, -cols, stream);
    // The rows of x in parts of equal width, a tile's runs shared by 1, 2, 4 or 8 CTAs: the least of what was measured, about
    // 0.75 us a block and 0.0075 for a row of x, 6 for a CTA's start and end, and what putting shared runs together
    // takes by the row of x.  (Clusters of eight do not fill every SM.)
    const int tiles = (N + F3_ROWS - 1) / F3_ROWS;
    double least = 0.0;
    for (int width = 128; width >= 16; width -= 16) {
        const int parts = (M + width - 1) / width;
        if (((M + parts - 1) / parts + 15) / 16 * 16 != width)
            continue;                                            // (as many parts of less width are enough)
        for (int r = 1; r <= F3_RUNS; r *= 2) {
            if ((r - 1) * (F3_RUNS / r) >= p.runs)
                break;                                           // (a CTA without a run)
            const int slots = (width <= 16 ? 2 : 1) * (r == 1 ? sms : r == 2 ? sms * 36 / 37 : r == 4 ? sms * 32 / 37 : sms * 26 / 37);
            const double rounds = (double)(((long long)tiles * parts * r + slots - 1) / slots);
            const int each = F3_RUNS / r < p.runs ? F3_RUNS / r : p.runs;
            const double together = r == 1 ? 0.0 : r == 2 ? 0.02 : r == 4 ? 0.04 : 0.027;
            const double cost = rounds * (each * p.run_blocks * (0.75 + 0.0075 * width) * (width <= 16 ? 2.0 : 1.0) + 6.0) + together * width;
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
    return p.cols <= 16 ? f3_launch<16, 256>(p, stream) : p.cols <= 32 ? f3_launch<32, 512>(p, stream)
        : p.cols <= 64 ? f3_launch<64, 512>(p, stream) : f3_launch<128, 512>(p, stream);
}
