// out[M, N] = x[M, K] * w[N, K]^T (+ residual[M, N]) with plain 32-bit FMAs.
//
// This is the matrix product of the true 32-bit path (no tensor-core mode, so
// no reduced-precision inputs or accumulators) and the fall-back of the
// bfloat16 path for shapes the tensor-core kernel refuses.  Operands that are all
// 32-bit, with rows on 16-byte boundaries, run the two kernels further down; the first one
// takes the rest: every output element is one thread's sequential sum over k = 0..K-1.  In
// both the result of a row does not depend on how many rows the call has.
#define CHIBI_UNIT gemm_simt
#define CHIBI_UNIT_ID 2
#include "common.cuh"

namespace chibi {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TO* __restrict__ out,
                 const float* __restrict__ residual, int M, int N, int K, long long x_stride,
                 long long w_stride, long long out_stride, long long res_stride)
{
    pdl_enter();
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4; // 16 x 16 threads, each TM x TN outputs
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
            acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k = 1024 elements per operand, 4 per thread
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + i * 256;
            const int r = e >> 4, kk = e & 15;
            const int k = k0 + kk;
            float xv = 0.f, wv = 0.f;
            if (k < K) {
                if (m0 + r < M)
                    xv = to_f32(x[(size_t)(m0 + r) * x_stride + k]);
                if (n0 + r < N)
                    wv = to_f32(w[(size_t)(n0 + r) * w_stride + k]);
            }
            xs[kk][r] = xv;
            ws[kk][r] = wv;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i)
                a[i] = xs[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j)
                b[j] = ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j)
                    acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M)
            continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N)
                continue;
            float v = acc[i][j];
            if (residual)
                v = residual[(size_t)m * res_stride + n] + v;
            out[(size_t)m * out_stride + n] = from_f32<TO>(v);
        }
    }
}

// ---------------------------------------------------------------- all three operands 32-bit, rows on 16-byte boundaries
//
// The order of a sum depends on K alone, so the result of a row does not depend on how many rows the call has,
// although few and many rows run different kernels: K is cut into at most 16 parts of `part` places (a
// multiple of 32, at least 128); a part's even and its odd places are summed one after the other, the two are
// added, four neighbouring parts are added in order, and then those groups in order.  The even and the odd
// sum are the two halves of one 64-bit register: fma.rn.f32x2 takes two neighbouring places of both operands
// as they lie in shared memory (each half rounded like fmaf), so neither operand is transposed or
// doubled on its way.  Rows lie 36 floats apart there: the 16 bytes of eight rows fall on all 32 banks.
constexpr int F32_KB = 32, F32_ROW = F32_KB + 4;        // places of a stage; floats from row to row
constexpr int F32_GROUP = 4;                            // parts of a group
constexpr int F32_GROUPS = 4;                           // most groups of a sum
constexpr int F32_TILE_STAGES = 3;
constexpr int F32_MAX_SHARED = 200 * 1024;

struct F32Params {
    const float* x;
    const float* w;
    float* out;
    const float* residual;
    long long x_stride, w_stride, out_stride, res_stride;
    int M, N, K, part, parts;                           // part: places of a part
    int ranks;                                          // CTAs of a cluster, which share a tile's parts
    int tiles;                                          // of the few-row kernel
};

__device__ __forceinline__ uint64_t f32_fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float f32_halves_sum(uint64_t v)
{
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a + b;
}
// 16 bytes, of which those beyond the first `bytes` are zeros and not read.
__device__ __forceinline__ void f32_copy16(float* dst, const float* src, int bytes)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void f32_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
// A value of CTA `rank` of this cluster at the same place of shared memory.
__device__ __forceinline__ float f32_peer(const float* local, int rank)
{
    uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local)), b;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(b) : "memory");
    return v;
}
__device__ __forceinline__ void f32_store(const F32Params& p, int m, int n, float v)
{
    if (p.residual)
        v = p.residual[(size_t)m * p.res_stride + n] + v;
    p.out[(size_t)m * p.out_stride + n] = v;
}

// Many rows: a tile of 64 x 64 sums, 4 rows and 8 columns to a thread, three stages of 32 places by cp.async.  Bound by
// the way out of shared memory: four places of a thread's tile are 12 reads of 16 bytes (48 cycles of the
// SM's 128 bytes a cycle for a warp) and 64 double multiply-adds (32 cycles for a warp on each of the four
// schedulers).  8 x 8 sums to a thread would be 64 to 64, but their pairs take 128 registers, and the eight warps
// that are left room for hide less (the same 0.56 of the multiply-adds' rate, and half of it where tiles are
// few).  Where the tiles are fewer than the SMs can take, a cluster of 2 or 4 CTAs shares a tile's groups of
// parts: each leaves its groups' sums in its shared memory, and each adds up some of the tile over all of them.
__global__ void __launch_bounds__(128)
gemm_f32_tile_kernel(const F32Params p)
{
    pdl_enter();
    constexpr int BM = 64, TM = 4, TY = BM / TM, THREADS = 8 * TY, STAGES = F32_TILE_STAGES, STAGE = (BM + 64) * F32_ROW;
    constexpr int QUADS = F32_KB / 4, RUN = THREADS / QUADS, COPIES = BM / RUN;     // rows at a time; a thread's copies
    extern __shared__ __align__(16) float f32_sm[];
    float* const sums = f32_sm + STAGES * STAGE;        // [own group][BM][64], or the total
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const int ranks = p.ranks, rank = ranks > 1 ? (int)(blockIdx.x % ranks) : 0;
    const int n0 = (int)(blockIdx.x / ranks) * 64, m0 = blockIdx.y * BM;
    const int groups = (p.parts + F32_GROUP - 1) / F32_GROUP;
    const int own = (groups + ranks - 1) / ranks;       // groups of a rank (the last ones may have fewer)
    const int first = min(rank * own, groups), last = min(first + own, groups);
    const int k_begin = first * F32_GROUP * p.part, k_end = min(last * F32_GROUP * p.part, p.K);
    const int blocks = k_end > k_begin ? (k_end - k_begin + F32_KB - 1) / F32_KB : 0;

    const int at = 4 * (tid % QUADS), row = tid / QUADS;
    const float* x[COPIES];
    const float* w[COPIES];
#pragma unroll
    for (int i = 0; i < COPIES; ++i) {
        const int m = m0 + row + RUN * i, n = n0 + row + RUN * i;
        x[i] = m < p.M ? p.x + (size_t)m * p.x_stride + k_begin + at : nullptr;
        w[i] = n < p.N ? p.w + (size_t)n * p.w_stride + k_begin + at : nullptr;
    }
    auto fetch = [&](int kb) {
        if (kb < blocks) {
            float* const dst = f32_sm + (kb % STAGES) * STAGE + row * F32_ROW + at;
            const int left = min(max(k_end - k_begin - at - kb * F32_KB, 0), 4) * 4;
#pragma unroll
            for (int i = 0; i < COPIES; ++i)
                f32_copy16(dst + RUN * i * F32_ROW, x[i] && left ? x[i] + kb * F32_KB : p.x, x[i] ? left : 0);
#pragma unroll
            for (int i = 0; i < COPIES; ++i)
                f32_copy16(dst + (BM + RUN * i) * F32_ROW, w[i] && left ? w[i] + kb * F32_KB : p.w, w[i] ? left : 0);
        }
        f32_commit();
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        fetch(s);

    uint64_t acc[TM][8];
    float kept[TM][8];                                  // the group's sum
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            acc[i][j] = 0;
    const int part_blocks = p.part / F32_KB;
    int in_part = 0, part = 0;
    for (int kb = 0; kb < blocks; ++kb) {
        f32_wait<STAGES - 2>();
        __syncthreads();                                // the stage is there; everyone is through with the one before
        fetch(kb + STAGES - 1);
        const float* xs = f32_sm + (kb % STAGES) * STAGE + ty * F32_ROW;
        const float* ws = f32_sm + (kb % STAGES) * STAGE + (BM + tx) * F32_ROW;
#pragma unroll
        for (int k = 0; k < F32_KB; k += 4) {
            ulonglong2 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i)
                a[i] = *reinterpret_cast<const ulonglong2*>(xs + TY * i * F32_ROW + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * F32_ROW + k);
#pragma unroll
                for (int i = 0; i < TM; ++i)
                    acc[i][j] = f32_fma2(a[i].x, b.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
                    acc[i][j] = f32_fma2(a[i].y, b.y, acc[i][j]);
            }
        }
        if (++in_part == part_blocks || kb + 1 == blocks) {
            in_part = 0;
            const bool opens = part % F32_GROUP == 0;
            ++part;
            const bool closes = part % F32_GROUP == 0 || kb + 1 == blocks;
            const int g = (part - 1) / F32_GROUP;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float s = f32_halves_sum(acc[i][j]);
                    acc[i][j] = 0;
                    if (!opens)
                        s = kept[i][j] + s;
                    if (!closes) {
                        kept[i][j] = s;
                    } else {
                        float* const t = sums + ((ranks > 1 ? g * BM : 0) + ty + TY * i) * 64 + tx + 8 * j;
                        *t = ranks > 1 || g == 0 ? s : *t + s;
                    }
                }
        }
    }
    if (ranks > 1)
        f32_cluster_sync();
    else
        __syncthreads();
    for (int i = rank * THREADS + tid; i < BM * 64; i += ranks * THREADS) {
        const int m = m0 + i / 64, n = n0 + (i & 63);
        if (m < p.M && n < p.N) {
            if (ranks == 1) {
                f32_store(p, m, n, sums[i]);
                continue;
            }
            float s[F32_GROUPS];
#pragma unroll
            for (int g = 0; g < F32_GROUPS; ++g)
                if (g < groups)
                    s[g] = f32_peer(sums + (g % own) * BM * 64 + i, g / own);
            float v = s[0];
#pragma unroll
            for (int g = 1; g < F32_GROUPS; ++g)
                if (g < groups)
                    v += s[g];
            f32_store(p, m, n, v);
        }
    }
    if (ranks > 1)
        f32_cluster_sync();                             // nobody leaves while its sums are read
}

// Few rows, MT at a time (padded to that): bound by the weights' way from memory.  A warp brings 32 NR of the weights'
// rows, NR rows to a lane, 32 places a stage by its own cp.async ring (no barrier between warps on the way),
// the rows of x beside them, which all lanes read at the same place: MT + NR reads of 16 bytes (four cycles
// each) to 16 NR bytes of weights a lane, so more rows of x want more rows of weights to a lane to stay behind
// memory.  The four warps of a CTA, and the CTAs of a cluster where the tiles of 32 NR rows are few, take
// the parts in turn; a CTA that is alone with its tiles walks over several.  The first weights are asked for in L2
// before the wait for the kernel ahead, and read after it, because that kernel may be the one that writes them (fetched into
// shared memory before the wait, one row of 4,096 x 1,024 / 1,024 x 3,072 / 151,936 x 1,024 takes 5.5, 5.8, 94.8 us; so 5.8,
// 7.0, 103.6).
template <int MT, int NR, int STAGES>
__global__ void __launch_bounds__(128)
gemm_f32_few_kernel(const F32Params p)
{
    pdl_trigger();
    constexpr int ROWS = 32 * NR, STAGE = ROWS * F32_ROW + MT * F32_KB, QUADS = F32_KB / 4, RUN = 32 / QUADS;
    extern __shared__ __align__(16) float f32_sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ranks = p.ranks, rank = ranks > 1 ? (int)(blockIdx.x % ranks) : 0;
    float* const ring = f32_sm + warp * STAGES * STAGE;
    float* const sums = f32_sm + 4 * STAGES * STAGE;    // [own parts of the CTA, or a group][MT][ROWS]
    const int walkers = gridDim.x / ranks;              // CTAs (or clusters) that walk over the tiles
    const int slots = 4 * ranks, slot = 4 * rank + warp;
    const int part_blocks = p.part / F32_KB;
    const int mine = slot < p.parts ? (p.parts - slot + slots - 1) / slots : 0;      // this warp's parts of a tile
    const int all_blocks = (p.K + F32_KB - 1) / F32_KB;
    const int m0 = MT * blockIdx.y, rows = min(p.M - m0, MT);
    const float* const x0 = p.x + (size_t)m0 * p.x_stride;

    // where the loads are: tile, own part, block of the part
    struct Place { int tile, part, block; };
    auto advance = [&](Place& at) {
        const int blocks = min(part_blocks, all_blocks - (slot + at.part * slots) * part_blocks);
        if (++at.block >= blocks) {
            at.block = 0;
            if (++at.part >= mine) {
                at.part = 0;
                at.tile += walkers;
            }
        }
    };
    auto fetch_w = [&](const Place& at, int stage) {
        float* const ws = ring + stage * STAGE;
        const int quad = 4 * (lane % QUADS), k = ((slot + at.part * slots) * part_blocks + at.block) * F32_KB + quad;
#pragma unroll
        for (int i = 0; i < ROWS / RUN; ++i) {
            const int r = lane / QUADS + RUN * i, n = at.tile * ROWS + r;
            const int bytes = n < p.N ? min(max(p.K - k, 0), 4) * 4 : 0;
            f32_copy16(ws + r * F32_ROW + quad, bytes ? p.w + (size_t)n * p.w_stride + k : p.w, bytes);
        }
    };
    auto fetch_x = [&](const Place& at, int stage) {
        float* const xs = ring + stage * STAGE + ROWS * F32_ROW;
        const int quad = 4 * (lane % QUADS), k = ((slot + at.part * slots) * part_blocks + at.block) * F32_KB + quad;
#pragma unroll
        for (int i = 0; i < (MT + RUN - 1) / RUN; ++i) {
            const int r = lane / QUADS + RUN * i;
            if (r < MT) {
                const int bytes = r < rows ? min(max(p.K - k, 0), 4) * 4 : 0;
                f32_copy16(xs + r * F32_KB + quad, bytes ? x0 + (size_t)r * p.x_stride + k : p.x, bytes);
            }
        }
    };
    const int first_tile = blockIdx.x / ranks;
    Place ahead = { first_tile, 0, 0 };
    if (mine > 0) {
        Place at = ahead;
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s)
            if (at.tile < p.tiles) {
                const int k = ((slot + at.part * slots) * part_blocks + at.block) * F32_KB;
#pragma unroll
                for (int j = 0; j < NR; ++j) {
                    const int n = at.tile * ROWS + 32 * j + lane;
                    if (n < p.N && k < p.K)
                        prefetch_l2(p.w + (size_t)n * p.w_stride + k);
                }
                advance(at);
            }
    }
    pdl_wait();
    if (mine > 0) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) {
            if (ahead.tile < p.tiles) {
                fetch_w(ahead, s);
                fetch_x(ahead, s);
                advance(ahead);
            }
            f32_commit();
        }
    }
    int stage = 0;
    auto one_part = [&](int q) {                        // own part q, its sums to shared memory
        const int blocks = min(part_blocks, all_blocks - (slot + q * slots) * part_blocks);
        uint64_t acc[NR][MT];
#pragma unroll
        for (int j = 0; j < NR; ++j)
#pragma unroll
            for (int i = 0; i < MT; ++i)
                acc[j][i] = 0;
        for (int b = 0; b < blocks; ++b) {
            f32_wait<STAGES - 2>();
            __syncwarp();
            {
                const int next = stage == 0 ? STAGES - 1 : stage - 1;
                if (ahead.tile < p.tiles) {
                    fetch_w(ahead, next);
                    fetch_x(ahead, next);
                    advance(ahead);
                }
                f32_commit();
            }
            const float* ws = ring + stage * STAGE + lane * F32_ROW;
            const float* xs = ring + stage * STAGE + ROWS * F32_ROW;
#pragma unroll
            for (int k = 0; k < F32_KB; k += 4) {
                ulonglong2 w[NR];
#pragma unroll
                for (int j = 0; j < NR; ++j)
                    w[j] = *reinterpret_cast<const ulonglong2*>(ws + 32 * j * F32_ROW + k);
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(xs + i * F32_KB + k);
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        acc[j][i] = f32_fma2(x.x, w[j].x, acc[j][i]);
                        acc[j][i] = f32_fma2(x.y, w[j].y, acc[j][i]);
                    }
                }
            }
            stage = stage + 1 == STAGES ? 0 : stage + 1;
        }
        const int kept = ranks > 1 ? 4 * q + warp : warp;
#pragma unroll
        for (int j = 0; j < NR; ++j)
#pragma unroll
            for (int i = 0; i < MT; ++i)
                sums[(kept * MT + i) * ROWS + 32 * j + lane] = f32_halves_sum(acc[j][i]);
    };
    if (ranks == 1) {
        // a group of parts at a time joins the total, which a thread holds for its places of the tile
        constexpr int PLACES = (MT * ROWS + 127) / 128;
        for (int tile = first_tile; tile < p.tiles; tile += walkers) {
            float total[PLACES];
            for (int q = 0; F32_GROUP * q < p.parts; ++q) {
                if (q < mine)
                    one_part(q);
                __syncthreads();
                const int there = min(F32_GROUP, p.parts - F32_GROUP * q);
#pragma unroll
                for (int u = 0; u < PLACES; ++u) {
                    const int i = tid + 128 * u;
                    if (i < MT * ROWS) {
                        float s[F32_GROUP];
#pragma unroll
                        for (int v = 0; v < F32_GROUP; ++v)
                            s[v] = v < there ? sums[v * MT * ROWS + i] : 0.f;
                        float t = s[0];
#pragma unroll
                        for (int v = 1; v < F32_GROUP; ++v)
                            if (v < there)
                                t += s[v];
                        total[u] = q == 0 ? t : total[u] + t;
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int u = 0; u < PLACES; ++u) {
                const int i = tid + 128 * u, m = i / ROWS, n = tile * ROWS + i % ROWS;
                if (m < rows && n < p.N)
                    f32_store(p, m0 + m, n, total[u]);
            }
        }
        return;
    }
    for (int q = 0; q < mine; ++q)
        one_part(q);
    f32_cluster_sync();
    for (int i = rank * 128 + tid; i < rows * ROWS; i += ranks * 128) {
        const int m = i / ROWS, n = first_tile * ROWS + i % ROWS;
        // (part q: the CTA's number 4 (q / slots) + q % 4 of CTA (q % slots) / 4)
        if (n < p.N) {
            float s[F32_GROUPS * F32_GROUP];
#pragma unroll
            for (int q = 0; q < F32_GROUPS * F32_GROUP; ++q)
                if (q < p.parts)
                    s[q] = f32_peer(sums + (4 * (q / slots) + (q & 3)) * MT * ROWS + i, (q % slots) >> 2);
            float total = 0.f;
#pragma unroll
            for (int g = 0; g < F32_GROUPS; ++g)
                if (F32_GROUP * g < p.parts) {
                    float v = s[F32_GROUP * g];
#pragma unroll
                    for (int u = 1; u < F32_GROUP; ++u)
                        if (F32_GROUP * g + u < p.parts)
                            v += s[F32_GROUP * g + u];
                    total = g == 0 ? v : total + v;
                }
            f32_store(p, m0 + m, n, total);
        }
    }
    f32_cluster_sync();                                 // nobody leaves while its sums are read
}

template <auto KERNEL>
static int f32_launch(dim3 grid, int ranks, size_t smem, cudaStream_t stream, const F32Params& p)
{
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, F32_MAX_SHARED);
        if (e != cudaSuccess)
            return (int)e;
        configured = true;
    }
    if (ranks > 1)
        launch_cluster_x(KERNEL, grid, dim3(128), smem, stream, ranks, p);
    else
        launch(KERNEL, grid, dim3(128), smem, stream, p);
    return launch_status();
}

template <int MT, int NR, int STAGES>
static int f32_few(F32Params p, cudaStream_t stream)
{
    // Two CTAs to an SM.  The tiles fill them, or the parts of a tile are shared by 2 or 4 CTAs while that needs no
    // second round and leaves every warp a part.
    p.tiles = (p.N + 32 * NR - 1) / (32 * NR);
    const int blocks = (p.M + MT - 1) / MT, slots = 2 * device_sm_count() / blocks;
    p.ranks = 1;
    while (p.ranks < 4 && p.tiles * p.ranks * 2 <= slots && 8 * p.ranks <= p.parts)
        p.ranks *= 2;
    const int kept = p.ranks > 1 ? (p.parts + 4 * p.ranks - 1) / (4 * p.ranks) : 1;
    const size_t smem = sizeof(float) * ((size_t)4 * STAGES * (32 * NR * F32_ROW + MT * F32_KB) + (size_t)4 * kept * MT * 32 * NR);
    const int grid = p.ranks > 1 ? p.tiles * p.ranks : (p.tiles < slots ? p.tiles : slots);
    return f32_launch<gemm_f32_few_kernel<MT, NR, STAGES>>(dim3(grid, blocks), p.ranks, smem, stream, p);
}

static int f32_tiles(F32Params p, cudaStream_t stream)
{
    // How many CTAs share a tile.  An SM holds two CTAs (the registers; with bounds for three the sums spill, 128 rows of
    // 1,024 x 2,048 38 -> 50 us), and one alone takes 0.8 of the time of two (512 rows of 1,024 x 2,048, 128 tiles: 134 us
    // whole, 76 shared).  The busiest SM's time in groups of parts, with an eighth of one for a CTA's start and end.
    const long long tiles = (long long)((p.N + 63) / 64) * ((p.M + 63) / 64);
    const int groups = (p.parts + F32_GROUP - 1) / F32_GROUP, sms = device_sm_count();
    double least = 0.0;
    for (int ranks = 1; ranks <= groups; ranks *= 2) {
        const long long ctas = (tiles * ranks + sms - 1) / sms;
        const double cost = ((double)(ctas / 2) + (ctas % 2 ? 0.8 : 0.0)) * ((groups + ranks - 1) / ranks + 0.125);
        if (ranks == 1 || cost < least) {
            p.ranks = ranks;
            least = cost;
        }
    }
    const int own = p.ranks > 1 ? (groups + p.ranks - 1) / p.ranks : 1;
    const size_t smem = sizeof(float) * ((size_t)F32_TILE_STAGES * 128 * F32_ROW + (size_t)own * 64 * 64);
    return f32_launch<gemm_f32_tile_kernel>(dim3((p.N + 63) / 64 * p.ranks, (p.M + 63) / 64), p.ranks, smem, stream, p);
}

static int gemm_f32(const float* x, const float* w, float* out, const float* residual, int M, int N, int K,
                    long long x_stride, long long w_stride, long long out_stride, long long res_stride, cudaStream_t stream)
{
    F32Params p = { x, w, out, residual, x_stride, w_stride, out_stride, res_stride, M, N, K, 0, 0, 1, 0 };
    const int sixteenth = (K + 15) / 16;
    p.part = (sixteenth + F32_KB - 1) / F32_KB * F32_KB;
    p.part = p.part < 128 ? 128 : p.part;
    p.parts = (K + p.part - 1) / p.part;
    // Few rows to 48 (blocks of 16 above 8), to 128 where N is small: 4,096 x 1,024 / 1,024 x 3,072 take 6.7, 8.1 us with
    // 4 rows, 30, 26 us with 48 (50 in tiles of 64 rows), 30, 26 with 64 (37, 43), 58, 44 with 128 (39, 53); the
    // kernel for all before this 150, 180 us from one row to 64.  From 5 rows on, where the weights'
    // tiles fill the SMs (N >= 64 x 148), a lane takes two of their rows (151,936 x 1,024: 8 rows 155 -> 130 us, 16 rows
    // 246 -> 173; with fewer tiles two rows a lane leave SMs idle, 4,096 x 1,024: 7.9 -> 10.9).
    if (M <= 1)
        return f32_few<1, 1, 6>(p, stream);
    if (M <= 2)
        return f32_few<2, 1, 4>(p, stream);
    if (M <= 4)
        return f32_few<4, 1, 4>(p, stream);
    const bool wide = N >= 64 * device_sm_count();
    if (M <= 8)
        return wide ? f32_few<8, 2, 2>(p, stream) : f32_few<8, 1, 4>(p, stream);
    if (M <= 48 || (M <= 128 && (long long)((N + 31) / 32) * ((M + 15) / 16) <= 512))
        return wide ? f32_few<16, 2, 2>(p, stream) : f32_few<16, 1, 3>(p, stream);
    return f32_tiles(p, stream);
}

} // namespace chibi

using namespace chibi;

CHIBI_API int chibi_gemm_simt(const void* x, int x_type, const void* w, int w_type, void* out,
                              int out_type, const float* residual, int M, int N, int K,
                              long long x_stride, long long w_stride, long long out_stride,
                              long long res_stride, cudaStream_t stream)
{
    if (M <= 0 || N <= 0)
        return CHIBI_OK;
    if (K < 0)
        return CHIBI_ERR_ARGUMENT;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535)
        return CHIBI_ERR_UNSUPPORTED;
    // (copies of 16 bytes: rows that start elsewhere, and mixed types, stay with the plain kernel)
    if (x_type == CHIBI_F32 && w_type == CHIBI_F32 && out_type == CHIBI_F32 && K > 0
        && ((uintptr_t)x | (uintptr_t)w) % 16 == 0 && x_stride % 4 == 0 && w_stride % 4 == 0)
        return gemm_f32((const float*)x, (const float*)w, (float*)out, residual, M, N, K, x_stride, w_stride, out_stride,
                        res_stride, stream);
    CHIBI_DISPATCH_TYPE(x_type, TX, CHIBI_DISPATCH_TYPE(w_type, TW, CHIBI_DISPATCH_TYPE(out_type, TO, {
        launch(gemm_simt_kernel<TX, TW, TO>, dim3(grid), dim3(256), 0, stream, 
            (const TX*)x, (const TW*)w, (TO*)out, residual, M, N, K, x_stride, w_stride,
            out_stride, res_stride);
    })));
    return launch_status();
}
