// Causal grouped-query attention for prompt portions on the 5th-generation
// tensor cores, for one head size per compiled library (-DCHIBI_HEAD_DIM=d,
// d = 64 or 128).
//
// One CTA owns 128 query rows of one kv head -- the rows are (token, head of the
// group) pairs, so the group's heads share every key and value tile -- and walks
// over the keys in tiles of 128:
//
//   warp 0      loads the query rows (where a tile of 128 is whole tokens) and the K and V tiles with TMA, one box per
//               cache page and 64-wide half of the head (128-byte swizzle);
//   warp 1      issues the MMAs:  S = Q K^T  (both K-major) into one of two TMEM
//               buffers, and  O += P V  with P from TMEM and V as the
//               MN-major operand (V is stored [key][d]), accumulating in a third TMEM buffer;
//   warps 4..11 softmax: two threads own a query row, each half of a tile's keys.  A thread reads its 64 scores from
//               TMEM, keeps the running maximum and its sum in registers and writes
//               P = exp2(S * scale - max) as packed bfloat16 over the first 64 columns of that S.  The output accumulates
//               in TMEM over all tiles; it is rescaled there only when a row's maximum has grown by
//               more than 2^8, and read out once at the end.
//
// The MMA of the next S tile is issued before the P V product of the current
// one, so it runs while the softmax threads work.  All waits are bounded.
#define CHIBI_UNIT attention_tcgen05
#define CHIBI_UNIT_ID 7
#include "common.cuh"
#include "sm100.cuh"
#include "attention_tc.cuh"
#include "split_f32.cuh"
#include "tensor_map.cuh"

#ifndef CHIBI_HEAD_DIM
#define CHIBI_HEAD_DIM 128
#endif

namespace chibi {

using namespace sm100;

constexpr int D = CHIBI_HEAD_DIM;
static_assert(D == 64 || D == 128, "the tcgen05 attention kernel takes head sizes 64 and 128");
constexpr int ROWS = 128;                    // query rows per CTA = UMMA M
constexpr int KEYS = 128;                    // keys per tile
constexpr int HALVES = D / 64;               // 64-wide (128-byte) slices of a head
constexpr int ATC_THREADS = 384;
constexpr int Q_BYTES = ROWS * D * 2;
constexpr int KV_TILE_BYTES = KEYS * D * 2;  // one K or V tile
constexpr int SMEM_TILES = Q_BYTES + 4 * KV_TILE_BYTES;
constexpr int NUM_BARS = 15;
constexpr int COLS = KEYS / 2;               // scores of a softmax thread
constexpr size_t ATC_SMEM = SMEM_TILES + NUM_BARS * 8 + 16 + 2 * ROWS * 4 + 1024;

// Options of the score, compiled in: 0 none; 1 any of them (a soft cap, a bias of either kind); 2 a bias linear in
// the distance and nothing else, which costs a multiply-add or two a score; 3 a soft cap and nothing else.
constexpr int OPT_NONE = 0, OPT_ANY = 1, OPT_LINEAR = 2, OPT_CAP = 3;

// v[i] = cap tanh(v[i] scale / cap) in units of log2, by the same operations as among the other options, so that a cap alone
// gives the bits of a cap with a bias of zeros.  What it saves is the bias's logarithm, one of four special-function
// operations a score, of which an SM does 16 a cycle, and its multiplications: four prompts of up to 700 tokens of 16
// heads of 128 59.6 -> 35.5 us.  (No model of the package has a cap without a bias; programs that call attention() do.)
template <int N>
__device__ __forceinline__ void cap_scores(uint32_t (&v)[N], float scale, float cap, float two_over_cap_log2)
{
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const float x = __uint_as_float(v[i]) * scale;
        v[i] = __float_as_uint(cap * (1.f - __fdividef(2.f, fast_exp2(x * two_over_cap_log2) + 1.f)) * 1.4426950408889634f);
    }
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// The output accumulator's columns of this thread *= f, in TMEM (a rare event: piece by piece, so that it takes few registers).
__device__ __forceinline__ void rescale_output_row(uint32_t o_addr, float f)
{
#pragma unroll 1
    for (int c0 = 0; c0 < D / 2; c0 += 16) {
        uint32_t ov[16];
        tmem_load_32x16(o_addr + c0, ov);
        tmem_load_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i)
            ov[i] = __float_as_uint(__uint_as_float(ov[i]) * f);
        tmem_store_32x16(o_addr + c0, ov);
    }
    tmem_store_wait();
}

// A warp pair's vote and barrier: whether any of the 64 threads says yes.
__device__ __forceinline__ bool pair_any(int barrier, bool yes)
{
    uint32_t r;
    asm volatile("{\n"
                 ".reg .pred p, q;\n"
                 "setp.ne.u32 q, %2, 0;\n"
                 "barrier.cta.red.or.pred.aligned p, %1, 64, q;\n"
                 "selp.u32 %0, 1, 0, p;\n"
                 "}\n" : "=r"(r) : "r"(barrier), "r"((uint32_t)yes) : "memory");
    return r != 0;
}
__device__ __forceinline__ void pair_sync(int barrier)
{
    asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(barrier) : "memory");
}

// ------------------------------------------------------------------ what both kernels' threads do
// Lane i of the loader brings page i of every 128-key tile (at most 16 pages: page_size >= 8): the row of the cache view
// where its page of tile j begins.
struct KeyPages {
    const int* table;
    int key_begin, key_end, kv_head, per_tile;
    __device__ __forceinline__ long long row_of(const AttnTcParams& p, int j, int lane) const
    {
        const int key = key_begin + j * KEYS + lane * p.page_size;
        if (lane >= per_tile || key >= key_end)
            return p.cache_rows;          // past the context: read outside the array, zeros
        const int page = table[key / p.page_size];
        if (page < 0 || page >= p.num_pages) {
            if (p.error)
                atomicExch(p.error, 3);
            return p.cache_rows;
        }
        return ((long long)page * p.nkv + kv_head) * p.page_size;
    }
};

// Brings tile j of the keys (or values) into its stage; the whole warp, `row` from KeyPages.
__device__ __forceinline__ void load_tile(const AttnTcParams& p, const CUtensorMap* map, uint8_t* stages, uint64_t* full,
                                          uint64_t* empty, int j, long long row, int per_tile, int lane)
{
    const int st = j & 1;
    if (lane == 0) {
        if (j >= 2)
            mbar_wait(&empty[st], ((j >> 1) - 1) & 1, p.error, 41);
        mbar_arrive_expect_tx(&full[st], KV_TILE_BYTES);
    }
    __syncwarp();
    if (lane < per_tile) {
        for (int h = 0; h < HALVES; ++h)
            tma_load_2d(stages + st * KV_TILE_BYTES + h * (KEYS * 128) + lane * p.page_size * 128, map, &full[st], h * 64, (int)row);
    }
}

// TILES tiles of 128 query rows from row0 on -> shared memory in the swizzled K-major layout, by all threads; all of a
// thread's loads before the first store.
template <int TILES, int THREADS>
__device__ __forceinline__ void gather_queries(const AttnTcParams& p, uint8_t* q_s, int row0, int rows_total, int t0, int kv_head)
{
    constexpr int PIECES = (TILES * ROWS * (D / 8) + THREADS - 1) / THREADS;
    uint4 v[PIECES];
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int c = threadIdx.x + i * THREADS;
        const int row = c / (D / 8), chunk = c - row * (D / 8), r = row0 + row;
        v[i] = make_uint4(0, 0, 0, 0);
        if (c < TILES * ROWS * (D / 8) && r < rows_total) {
            const int tok = r / p.group, h = r - tok * p.group;
            v[i] = *reinterpret_cast<const uint4*>(p.q + ((size_t)(t0 + tok) * p.nq + kv_head * p.group + h) * D + chunk * 8);
        }
    }
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int c = threadIdx.x + i * THREADS;
        const int row = c / (D / 8), chunk = c - row * (D / 8);
        if (c < TILES * ROWS * (D / 8))
            *reinterpret_cast<uint4*>(q_s + (row >> 7) * Q_BYTES + (chunk >> 3) * (ROWS * 128) + swizzled_chunk(row & 127, chunk & 7)) = v[i];
    }
    fence_proxy_async();                  // the tensor core reads what these threads wrote
}
// The same by TMA, one thread.
__device__ __forceinline__ void load_queries(const AttnTcParams& p, const CUtensorMap* map, uint8_t* q_s, uint64_t* full, int row0,
                                             int t0, int kv_head)
{
    mbar_arrive_expect_tx(full, Q_BYTES);
    for (int h = 0; h < HALVES; ++h)
        tma_load_3d(q_s + h * (ROWS * 128), map, full, h * 64, kv_head * p.group, t0 + row0 / p.group);
}

// A softmax thread's query row.
struct QueryRow {
    bool live;
    int tok, head, pos, first;            // its token in the sequence and query head; its position and first visible key
    float r1, r2, two_over_cap_log2;
    bool linear_bias;                     // r1 * distance instead of r1 * ln(1 + r2 * distance)
    float m, l;                           // the maximum that the exponents are taken against, the sum
};
__device__ __forceinline__ QueryRow query_row(const AttnTcParams& p, int r, int rows_total, int pos0, int kv_head)
{
    QueryRow w;
    w.live = r < rows_total;
    w.tok = w.live ? r / p.group : 0;
    w.head = kv_head * p.group + (w.live ? r - w.tok * p.group : 0);       // (rows past the end have none)
    w.pos = w.live ? pos0 + w.tok : -1;
    w.first = first_visible_key(w.pos, p.window, p.chunk);
    w.r1 = p.bias_r1 ? p.bias_r1[w.head] : 0.f;
    w.r2 = p.bias_r2 ? p.bias_r2[w.head] : 0.f;
    w.linear_bias = p.bias_r1 && !p.bias_r2;
    w.two_over_cap_log2 = p.softcap > 0.f ? 2.f * 1.4426950408889634f / p.softcap : 0.f;
    w.m = -INFINITY;
    w.l = 0.f;
    return w;
}

// Half a row of S (keys key0 on, in TMEM at s_addr, finished) -> its probabilities, over the row's first columns at p_addr.
// The output accumulates in TMEM over all tiles.  `m` follows the true maximum only when that has grown by more than 2^8
// (then the output so far is rescaled in TMEM, a rare event after the first tiles), so the probabilities stay below
// 2^8 and most tiles need no rescaling at all; `landed` waits until the products so far have.  So the two threads of a row
// tell each other their maxima (through `maxima`, [2][128]) only if one of their warps has such a row; that vote is also the
// barrier behind which S has been read and may be written over.
template <int OPT, typename LANDED>
__device__ __forceinline__ void softmax_row(const AttnTcParams& p, QueryRow& w, uint32_t s_addr, uint32_t p_addr, uint32_t o_addr, int key0,
                                            bool first_tile, int barrier, float* maxima, int half, int thread, LANDED landed)
{
    // with options of the score a row is brought to its final form (in units of log2) right after it is read, and the
    // scale below is 1
    constexpr bool options = OPT == OPT_ANY || OPT == OPT_CAP;
    const float sl2 = OPT != OPT_NONE ? 1.f : p.scale_log2;
    uint32_t sv[COLS];
#pragma unroll
    for (int c0 = 0; c0 < COLS; c0 += 32)
        tmem_load_32x32(s_addr + c0, *reinterpret_cast<uint32_t(*)[32]>(&sv[c0]));
    tmem_load_wait();
    if (OPT == OPT_LINEAR) {
        // score - slope * (pos - key), in units of log2; keys after pos are masked below
        const float slope = w.r1 * 1.4426950408889634f, at0 = slope * (float)(key0 - w.pos);
#pragma unroll
        for (int i = 0; i < COLS; ++i)
            sv[i] = __float_as_uint(fmaf(__uint_as_float(sv[i]), p.scale_log2, fmaf((float)i, slope, at0)));
    }
    if (OPT == OPT_CAP) {
        cap_scores(sv, p.scale, p.softcap, w.two_over_cap_log2);
    } else if (options) {
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
            float x = __uint_as_float(sv[i]) * p.scale;
            if (p.softcap > 0.f)                     // c * tanh(x / c) = c * (1 - 2 / (exp(2 x / c) + 1))
                x = p.softcap * (1.f - __fdividef(2.f, fast_exp2(x * w.two_over_cap_log2) + 1.f));
            const int dist = w.pos - (key0 + i);
            x -= w.linear_bias ? w.r1 * (float)(dist > 0 ? dist : 0) : w.r1 * __logf(1.f + w.r2 * (float)(dist > 0 ? dist : 0));
            sv[i] = __float_as_uint(x * 1.4426950408889634f);
        }
    }
    // masks only where a row's visible range ends inside the tile; the warp takes one path
    if (__any_sync(0xffffffffu, key0 + COLS - 1 > w.pos || key0 < w.first)) {
#pragma unroll
        for (int i = 0; i < COLS; ++i) {
            const int key = key0 + i;
            if (!(key <= w.pos && key >= w.first))
                sv[i] = 0xff800000u;                 // -inf
        }
    }
    float mx4[4];                                    // four short chains, not one long one
#pragma unroll
    for (int u = 0; u < 4; ++u)
        mx4[u] = max3(__uint_as_float(sv[u]), __uint_as_float(sv[u + 4]), __uint_as_float(sv[u + 8]));
#pragma unroll
    for (int i = 12; i < COLS - 4; i += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            mx4[u] = max3(mx4[u], __uint_as_float(sv[i + u]), __uint_as_float(sv[i + 4 + u]));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        mx4[u] = fmaxf(mx4[u], __uint_as_float(sv[COLS - 4 + u]));
    float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
    mx *= sl2;                                       // the scale is positive
    tcgen05_fence_before();                          // (the other warp's probabilities are written over these scores)
    const bool any = pair_any(barrier, mx > w.m + 8.f);      // also for the first visible key (m = -inf)
    tcgen05_fence_after();
    if (any) {
        maxima[half * ROWS + thread] = mx;
        pair_sync(barrier);
        mx = fmaxf(mx, maxima[(half ^ 1) * ROWS + thread]);
        pair_sync(barrier);                          // (read before the next tile's are written)
        const bool grow = mx > w.m + 8.f;
        if (__any_sync(0xffffffffu, grow && w.m != -INFINITY && !first_tile)) {
            landed();
            tcgen05_fence_after();
            rescale_output_row(o_addr, (grow && w.m != -INFINITY) ? fast_exp2(w.m - mx) : 1.f);
        }
        if (grow) {
            w.l *= (w.m == -INFINITY) ? 0.f : fast_exp2(w.m - mx);
            w.m = mx;
        }
        __syncwarp();
    }
    const float base = w.m == -INFINITY ? 0.f : w.m;
    const uint64_t scale2 = pair_of(sl2, sl2), base2 = pair_of(-base, -base);
    uint64_t sum2[4] = { 0, 0, 0, 0 };
#pragma unroll
    for (int c0 = 0; c0 < COLS; c0 += 32) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint64_t s2 = pair_of(__uint_as_float(sv[c0 + 2 * i]), __uint_as_float(sv[c0 + 2 * i + 1]));
            const float2 e = halves_of(OPT == OPT_NONE ? pair_fma(s2, scale2, base2) : pair_add(s2, base2));
            const float p0 = fast_exp2(e.x), p1 = fast_exp2(e.y);
            sum2[i & 3] = pair_add(sum2[i & 3], pair_of(p0, p1));
            const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
            packed[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        tmem_store_32x16(p_addr + (c0 >> 1), packed);
    }
    const float2 s01 = halves_of(pair_add(sum2[0], sum2[1])), s23 = halves_of(pair_add(sum2[2], sum2[3]));
    w.l += (s01.x + s01.y) + (s23.x + s23.y);
}

// Values past the context may be anything (a page is loaded whole): make them zero, so that 0 * value stays 0.  Only a
// CTA's last tile can hold such keys; the 256 threads of a softmax group.
__device__ __forceinline__ void clear_values(uint8_t* v_tile, int past, int thread)
{
    for (int c = thread; c < (KEYS - past) * (D / 8); c += 2 * ROWS) {
        const int row = past + c / (D / 8), chunk = c % (D / 8);
        *reinterpret_cast<uint4*>(v_tile + (chunk >> 3) * (KEYS * 128) + swizzled_chunk(row, chunk & 7)) = make_uint4(0, 0, 0, 0);
    }
    fence_proxy_async();
}

// The finished output rows of a pair of warps (32, from warp_row0 on; a thread has half of a row's columns): normalised, and
// written by way of the tile's query rows in shared memory, which are done with: neighbouring lanes then store neighbouring
// pieces of a row.
__device__ __forceinline__ void write_rows(const AttnTcParams& p, QueryRow& w, uint32_t o_addr, uint8_t* mine, int warp_row0, int rows_total,
                                           int t0, int kv_head, int lane, int barrier, int half)
{
    w.l += sink_weight(p.sink, w.head, w.m);
    const float inv = w.l > 0.f ? 1.f / w.l : 0.f;
    constexpr int CHUNKS = D / 8;
    uint32_t ov[D / 2];
#pragma unroll
    for (int c0 = 0; c0 < D / 2; c0 += 32)
        tmem_load_32x32(o_addr + c0, *reinterpret_cast<uint32_t(*)[32]>(&ov[c0]));
    tmem_load_wait();
#pragma unroll
    for (int c = 0; c < CHUNKS / 2; ++c) {
        __nv_bfloat162 h[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            h[u] = __floats2bfloat162_rn(__uint_as_float(ov[8 * c + 2 * u]) * inv, __uint_as_float(ov[8 * c + 2 * u + 1]) * inv);
        *reinterpret_cast<uint4*>(mine + lane * (D * 2) + (((c + half * (CHUNKS / 2)) ^ (lane & 7)) << 4)) = *reinterpret_cast<uint4*>(h);
    }
    pair_sync(barrier);
#pragma unroll 4
    for (int i = lane + half * (16 * CHUNKS); i < (half + 1) * (16 * CHUNKS); i += 32) {
        const int rr = i / CHUNKS, c = i % CHUNKS, at = warp_row0 + rr;
        if (at < rows_total) {
            const int t = at / p.group, h = at - t * p.group;
            *reinterpret_cast<uint4*>(p.out + ((size_t)(t0 + t) * p.nq + kv_head * p.group + h) * D + 8 * c) =
                *reinterpret_cast<const uint4*>(mine + rr * (D * 2) + ((c ^ (rr & 7)) << 4));
        }
    }
}

// The sum of a row whose two threads hold half each, through `sums` ([2][128]).
__device__ __forceinline__ void join_sums(QueryRow& w, float* sums, int barrier, int half, int thread)
{
    sums[half * ROWS + thread] = w.l;
    pair_sync(barrier);
    w.l = sums[thread] + sums[ROWS + thread];
}

// ------------------------------------------------------------------ one query tile per CTA
// Two S buffers: the next tile's scores are there when a row's probabilities are written, so a thread goes on without a
// wait, and the time of a key tile is that of its softmax, or, with pages of 16 keys, of its 64 TMA boxes (8,192 tokens of
// 32 heads of 128: 770 us, 523 with pages of 128).  P stays in TMEM (through shared memory and with one thread to a row:
// 4 prompts of 100 tokens 10.1 us, 8.0 so; 600 tokens of 32 heads 18.3 and 14.9; 300 after 6,000 in key ranges 100 and 90).
template <int OPT>
__global__ void __launch_bounds__(ATC_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const AttnTcParams p)
{
    pdl_enter();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_s = smem;
    uint8_t* k_s = q_s + Q_BYTES;                  // two stages
    uint8_t* v_s = k_s + 2 * KV_TILE_BYTES;        // two stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SMEM_TILES);
    uint64_t* k_full = bars;          // [2] TMA
    uint64_t* v_full = bars + 2;      // [2] TMA
    uint64_t* k_empty = bars + 4;     // [2] MMA commit
    uint64_t* v_empty = bars + 6;     // [2] MMA commit
    uint64_t* s_full = bars + 8;      // [2] MMA commit
    uint64_t* p_full = bars + 10;     // [2] 256 threads
    uint64_t* o_full = bars + 12;     // [2] MMA commit: O holds tile j
    uint64_t* q_full = bars + 14;     // TMA
    float* maxima = reinterpret_cast<float*>(bars + NUM_BARS);   // [2][128]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(maxima + 2 * ROWS);

    // CTAs start in the order of their linear index: the row tiles with the most keys come first,
    // for all kv heads, so that the long ones do not start last
    const int seq = blockIdx.z / p.kv_splits, split = blockIdx.z - seq * p.kv_splits;
    const int linear = blockIdx.x + gridDim.x * blockIdx.y;
    const int kv_head = linear % gridDim.y, tile_rank = linear / gridDim.y;
    const int t0 = p.q_start[seq];
    const int q_len = p.q_start[seq + 1] - t0;
    const int rows_total = q_len * p.group;
    const int row0 = (gridDim.x - 1 - tile_rank) * ROWS;
    if (q_len <= 0 || (q_len == 1 && p.skip_single) || row0 >= rows_total)
        return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos0 = p.ctx_len[seq] - q_len;

    const int last_row = min(rows_total, row0 + ROWS) - 1;
    const int min_pos = pos0 + row0 / p.group, max_pos = pos0 + last_row / p.group;
    int key_begin = first_visible_key(min_pos, p.window, p.chunk);
    key_begin = key_begin / p.page_size * p.page_size;           // tiles start on a page
    const int key_end = max_pos + 1;
    int n_tiles = (key_end - key_begin + KEYS - 1) / KEYS;
    if (p.kv_splits > 1) {
        // this CTA's range of the row tile's key tiles (it may be empty)
        const int per = (n_tiles + p.kv_splits - 1) / p.kv_splits;
        const int lo = split * per;
        n_tiles = max(0, min(per, n_tiles - lo));
        key_begin += lo * KEYS;
    }
    const KeyPages pages { p.block_table + (size_t)(p.seq_rows ? p.seq_rows[seq] : seq) * p.table_stride, key_begin, key_end, kv_head,
                           KEYS / p.page_size };

    long long next_row = 0;
    if (warp == 0) {
        // the loader starts by itself: queries, first keys and first values are on their way while the others set up
        if (lane == 0) {
            for (int i = 0; i < 2; ++i) {
                mbar_init(&k_full[i], 1);
                mbar_init(&v_full[i], 1);
                mbar_init(&k_empty[i], 1);
                mbar_init(&v_empty[i], 1);
                mbar_init(&s_full[i], 1);
                mbar_init(&p_full[i], 2 * ROWS);
                mbar_init(&o_full[i], 1);
            }
            mbar_init(q_full, 1);
            fence_barrier_init();
            if (p.q_by_tma && n_tiles > 0)
                load_queries(p, &map_q, q_s, q_full, row0, t0, kv_head);
        }
        if (n_tiles > 0) {
            const long long row = pages.row_of(p, 0, lane);
            next_row = n_tiles > 1 ? pages.row_of(p, 1, lane) : 0;
            __syncwarp();
            load_tile(p, &map_k, k_s, k_full, k_empty, 0, row, pages.per_tile, lane);
            load_tile(p, &map_v, v_s, v_full, v_empty, 0, row, pages.per_tile, lane);
        }
    } else if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (!p.q_by_tma)
        gather_queries<1, ATC_THREADS>(p, q_s, row0, rows_total, t0, kv_head);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    constexpr uint32_t TMEM_O = 256;               // S at columns 0 and 128

    if (warp == 0) {
        // (a lane looks its page up one tile ahead, so the dependent read of the block table is over when the stage is free)
        for (int j = 1; j < n_tiles; ++j) {
            const long long row = next_row;
            next_row = j + 1 < n_tiles ? pages.row_of(p, j + 1, lane) : 0;
            load_tile(p, &map_k, k_s, k_full, k_empty, j, row, pages.per_tile, lane);
            load_tile(p, &map_v, v_s, v_full, v_empty, j, row, pages.per_tile, lane);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc_qk = make_idesc_bf16_f32(ROWS, KEYS);
            constexpr uint32_t idesc_pv = make_idesc_bf16_f32(ROWS, D) | (1u << 16);    // B is MN-major
            const uint64_t q_desc = make_kmajor_sw128_desc(smem_addr(q_s)), k_desc = make_kmajor_sw128_desc(smem_addr(k_s));
            const uint64_t v_desc = make_mnmajor_sw128_desc(smem_addr(v_s), KEYS * 128);
            auto issue_qk = [&](int j) {
                const int st = j & 1;
                mbar_wait(&k_full[st], (j >> 1) & 1, p.error, 22);
                tcgen05_fence_after();
                const uint64_t b = k_desc + st * (KV_TILE_BYTES >> 4);
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint32_t off = ((ks >> 2) * (ROWS * 128) + (ks & 3) * 32) >> 4;
                    tcgen05_mma_bf16(tmem_base + st * 128, q_desc + off, b + off, idesc_qk, ks > 0 ? 1u : 0u);
                }
                tcgen05_commit(&s_full[st]);
                tcgen05_commit(&k_empty[st]);
            };
            if (n_tiles > 0) {
                if (p.q_by_tma)
                    mbar_wait(q_full, 0, p.error, 23);
                issue_qk(0);
            }
            for (int j = 0; j < n_tiles; ++j) {
                // runs while the softmax threads work on tile j; S of tile j - 1 may be overwritten: the products of one thread
                // run in order
                if (j + 1 < n_tiles)
                    issue_qk(j + 1);
                const int st = j & 1;
                mbar_wait(&v_full[st], (j >> 1) & 1, p.error, 25);
                mbar_wait(&p_full[st], (j >> 1) & 1, p.error, 24);    // P(j) is in TMEM
                tcgen05_fence_after();
                const uint64_t b = v_desc + st * (KV_TILE_BYTES >> 4);
                const uint32_t more = j > 0 ? 1u : 0u;
#pragma unroll
                for (int ks = 0; ks < KEYS / 16; ++ks)
                    tcgen05_mma_bf16_a_tmem(tmem_base + TMEM_O, tmem_base + st * 128 + ks * 8, b + ks * (16 * 128 >> 4), idesc_pv,
                                            ks > 0 ? 1u : more);
                tcgen05_commit(&o_full[st]);
                tcgen05_commit(&v_empty[st]);
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        // the thread's query row = its TMEM lane; its half of a tile's keys, and of the output's columns
        const int quarter = warp & 3, half = (warp - 4) >> 2, thread = quarter * 32 + lane, barrier = 1 + quarter;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16), o_addr = lane_addr + TMEM_O + half * (D / 2);
        QueryRow w = query_row(p, row0 + thread, rows_total, pos0, kv_head);
        for (int j = 0; j < n_tiles; ++j) {
            const int st = j & 1, key0 = key_begin + j * KEYS;
            mbar_wait_warp(&s_full[st], (j >> 1) & 1, p.error, 26);
            tcgen05_fence_after();
            softmax_row<OPT>(p, w, lane_addr + st * 128 + half * COLS, lane_addr + st * 128 + half * (COLS / 2), o_addr,
                             key0 + half * COLS, j == 0, barrier, maxima, half, thread,
                             [&] { mbar_wait_warp(&o_full[(j - 1) & 1], ((j - 1) >> 1) & 1, p.error, 27); });
            if (key0 + KEYS > key_end) {
                mbar_wait(&v_full[st], (j >> 1) & 1, p.error, 29);
                clear_values(v_s + st * KV_TILE_BYTES, key_end - key0, half * ROWS + thread);
                __syncwarp();
            }
            tmem_store_wait();
            tcgen05_fence_before();
            mbar_arrive(&p_full[st]);
        }
        // the last product has landed: normalise and write the rows out
        if (n_tiles > 0)
            mbar_wait_warp(&o_full[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, p.error, 30);
        tcgen05_fence_after();
        join_sums(w, maxima, barrier, half, thread);
        if (p.kv_splits > 1) {
            // one of several key ranges: the row as it stands, with its maximum and sum
            const size_t slot = ((size_t)(t0 + w.tok) * p.nq + w.head) * p.kv_splits + split;
            float* dst = p.part_o + slot * D + half * (D / 2);
#pragma unroll
            for (int c0 = 0; c0 < D / 2; c0 += 32) {
                uint32_t ov[32];
                if (n_tiles > 0) {
                    tmem_load_32x32(o_addr + c0, ov);
                    tmem_load_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        ov[i] = 0;
                }
                if (w.live) {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        reinterpret_cast<uint4*>(dst + c0)[c] = make_uint4(ov[4 * c], ov[4 * c + 1], ov[4 * c + 2], ov[4 * c + 3]);
                }
                __syncwarp();
            }
            if (w.live && half == 0) {
                p.part_ml[slot * 2] = w.m;
                p.part_ml[slot * 2 + 1] = w.l;
            }
        } else {
            write_rows(p, w, o_addr, q_s + quarter * 32 * (D * 2), row0 + quarter * 32, rows_total, t0, kv_head, lane, barrier, half);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ------------------------------------------------------------------ two query tiles per CTA
// The same attention with 256 query rows per CTA: two tiles of 128 rows share
// every key and value tile, each tile has a softmax warp group of its own, and
// P never leaves TMEM (it overwrites the first 64 columns of its S buffer as
// packed bfloat16 and is the A operand of the P V product).  While one group
// works on its S tile the tensor core multiplies for the other.
//
//   warp 0       TMA loader: the query rows (where a tile of 128 is whole tokens), then keys and values as above
//   warp 1       MMA issuer:  S_q = Q_q K^T,  O_q += P_q V  for q = 0, 1 in turn
//   warps 2, 3   none (registers are given back by warp groups of four)
//   warps 4..11  softmax of tile 0;  warps 12..19  softmax of tile 1
//
// What bounds it over long rows is each tile's chain softmax -> P V -> next Q K^T beside full tensor cores and
// special-function units (each needs 2,048 cycles for a pair of tiles, which takes about 2,900), over short ones a CTA's start and
// end.  A softmax thread holds its scores, so that they leave TMEM once for both the maximum and the exponentials (the
// first four warps give registers back); scale, differences and sums are made two at a time (fma.rn.f32x2); two threads to
// a row halve the chain.  The queries come by TMA, asked for together with the first keys and values before anything else is
// set up, and the output goes out by way of shared memory in whole lines.  32 heads of 128 on 8 key heads, 2,048 / 8,192
// tokens: 70.6 / 649 us with two readings of S in pieces, queries through registers and rows written lane by lane, 45.0 /
// 455 with one thread to a row (168 registers for all, then 224 for these), 44.7 / 467 with two (0.47 / 0.73 of the measured
// product rate); with a soft cap, 4 prompts of 700 tokens of 16 heads of 128, 35.2, 31.7 and 28.8.
//
// TMEM: S_0 at column 0, S_1 at 128, O_0 at 256, O_1 at 384.
constexpr int ATC2_THREADS = 640;
constexpr int SMEM2_TILES = 2 * Q_BYTES + 4 * KV_TILE_BYTES;
constexpr int NUM_BARS2 = 16;
constexpr size_t ATC2_SMEM = SMEM2_TILES + NUM_BARS2 * 8 + 16 + 4 * ROWS * 4 + 1024;
// Registers of a thread: what the block is launched with, and what the loader's and the softmax groups' threads have then.
constexpr int ATC2_REGS = 96, ATC2_REGS_FEW = 48, ATC2_REGS_MANY = 104;
static_assert(ATC2_REGS_FEW + 4 * ATC2_REGS_MANY <= 5 * ATC2_REGS, "more registers than the block has");

template <int OPT>
__global__ void __launch_bounds__(ATC2_THREADS, 1)
attn_prefill_tc2_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const AttnTcParams p)
{
    pdl_enter();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_s = smem;                           // two tiles
    uint8_t* k_s = q_s + 2 * Q_BYTES;              // two stages
    uint8_t* v_s = k_s + 2 * KV_TILE_BYTES;        // two stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SMEM2_TILES);
    uint64_t* k_full = bars;          // [2] TMA
    uint64_t* v_full = bars + 2;      // [2] TMA
    uint64_t* k_empty = bars + 4;     // [2] MMA commit
    uint64_t* v_empty = bars + 6;     // [2] MMA commit
    uint64_t* s_full = bars + 8;      // [2] per query tile, MMA commit
    uint64_t* p_full = bars + 10;     // [2] per query tile, 256 threads
    uint64_t* o_done = bars + 12;     // [2] per query tile, MMA commit
    uint64_t* q_full = bars + 14;     // [2] per query tile, TMA
    float* maxima = reinterpret_cast<float*>(bars + NUM_BARS2);  // [query tile][2][128]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(maxima + 4 * ROWS);

    const int seq = blockIdx.z;
    const int linear = blockIdx.x + gridDim.x * blockIdx.y;        // longest row tiles first, for all kv heads
    const int kv_head = linear % gridDim.y, tile_rank = linear / gridDim.y;
    const int t0 = p.q_start[seq];
    const int q_len = p.q_start[seq + 1] - t0;
    const int rows_total = q_len * p.group;
    const int row0 = (gridDim.x - 1 - tile_rank) * (2 * ROWS);
    if (q_len <= 0 || (q_len == 1 && p.skip_single) || row0 >= rows_total)
        return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos0 = p.ctx_len[seq] - q_len;

    // key tiles: all start at key_begin (a page boundary at or before the first key that the
    // CTA's first row sees); tile q needs nt[q] of them, nt[0] <= nt[1] when tile 1 has rows
    const int min_pos = pos0 + row0 / p.group;
    int key_begin = first_visible_key(min_pos, p.window, p.chunk);
    key_begin = key_begin / p.page_size * p.page_size;
    int nt[2], key_end = 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int lo = row0 + q * ROWS;
        if (lo < rows_total) {
            const int last_row = min(rows_total, lo + ROWS) - 1;
            const int end = pos0 + last_row / p.group + 1;
            nt[q] = (end - key_begin + KEYS - 1) / KEYS;
            key_end = max(key_end, end);
        } else {
            nt[q] = 0;
        }
    }
    const int n_tiles = max(nt[0], nt[1]);

    const KeyPages pages { p.block_table + (size_t)(p.seq_rows ? p.seq_rows[seq] : seq) * p.table_stride, key_begin, key_end, kv_head,
                           KEYS / p.page_size };
    long long next_row = 0;
    if (warp == 0) {
        // the loader starts by itself: queries, first keys and first values are on their way while the others set up
        if (lane == 0) {
            for (int i = 0; i < 2; ++i) {
                mbar_init(&k_full[i], 1);
                mbar_init(&v_full[i], 1);
                mbar_init(&k_empty[i], 1);
                mbar_init(&v_empty[i], 1);
                mbar_init(&s_full[i], 1);
                mbar_init(&p_full[i], 2 * ROWS);
                mbar_init(&o_done[i], 1);
                mbar_init(&q_full[i], 1);
            }
            fence_barrier_init();
            if (p.q_by_tma) {
                for (int q = 0; q < 2; ++q)
                    if (nt[q] > 0)
                        load_queries(p, &map_q, q_s + q * Q_BYTES, &q_full[q], row0 + q * ROWS, t0, kv_head);
            }
        }
        const long long row = pages.row_of(p, 0, lane);
        next_row = n_tiles > 1 ? pages.row_of(p, 1, lane) : 0;
        __syncwarp();
        load_tile(p, &map_k, k_s, k_full, k_empty, 0, row, pages.per_tile, lane);
        load_tile(p, &map_v, v_s, v_full, v_empty, 0, row, pages.per_tile, lane);
    } else if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (!p.q_by_tma)
        gather_queries<2, ATC2_THREADS>(p, q_s, row0, rows_total, t0, kv_head);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    timeline_mark(0);                  // barriers and TMEM are there (and the query rows, if not by TMA)
    const uint32_t tmem_base = *tmem_slot;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ATC2_REGS_FEW));
        if (warp == 0) {
            for (int j = 1; j < n_tiles; ++j) {
                const long long row = next_row;
                next_row = j + 1 < n_tiles ? pages.row_of(p, j + 1, lane) : 0;
                load_tile(p, &map_k, k_s, k_full, k_empty, j, row, pages.per_tile, lane);
                load_tile(p, &map_v, v_s, v_full, v_empty, j, row, pages.per_tile, lane);
            }
        } else if (warp == 1 && elect_one()) {
            constexpr uint32_t idesc_qk = make_idesc_bf16_f32(ROWS, KEYS);
            constexpr uint32_t idesc_pv = make_idesc_bf16_f32(ROWS, D) | (1u << 16);    // B is MN-major
            // tile 1 is the last user of a key/value tile that it needs at all
            auto last_user = [&](int q, int j) { return q == (j < nt[1] ? 1 : 0); };
            // (descriptors of a tile's first 16 columns or keys; the others are constants away in units of 16 bytes)
            const uint64_t q_desc = make_kmajor_sw128_desc(smem_addr(q_s)), k_desc = make_kmajor_sw128_desc(smem_addr(k_s));
            const uint64_t v_desc = make_mnmajor_sw128_desc(smem_addr(v_s), KEYS * 128);
            auto issue_qk = [&](int q, int j) {
                const int st = j & 1;
                if (j == 0 && p.q_by_tma)
                    mbar_wait(&q_full[q], 0, p.error, 49);
                mbar_wait(&k_full[st], (j >> 1) & 1, p.error, 42);
                tcgen05_fence_after();
                const uint64_t a = q_desc + q * (Q_BYTES >> 4), b = k_desc + st * (KV_TILE_BYTES >> 4);
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint32_t off = ((ks >> 2) * (ROWS * 128) + (ks & 3) * 32) >> 4;
                    tcgen05_mma_bf16(tmem_base + q * 128, a + off, b + off, idesc_qk, ks > 0 ? 1u : 0u);
                }
                tcgen05_commit(&s_full[q]);
                if (last_user(q, j))
                    tcgen05_commit(&k_empty[st]);
            };
            auto issue_pv = [&](int q, int j) {
                const int st = j & 1;
                mbar_wait(&v_full[st], (j >> 1) & 1, p.error, 44);
                mbar_wait(&p_full[q], j & 1, p.error, 43);            // P_q(j) is in TMEM
                tcgen05_fence_after();
                const uint64_t b = v_desc + st * (KV_TILE_BYTES >> 4);
                const uint32_t more = j > 0 ? 1u : 0u;
#pragma unroll
                for (int ks = 0; ks < KEYS / 16; ++ks)
                    tcgen05_mma_bf16_a_tmem(tmem_base + 256 + q * 128, tmem_base + q * 128 + ks * 8, b + ks * (16 * 128 >> 4),
                                            idesc_pv, ks > 0 ? 1u : more);
                tcgen05_commit(&o_done[q]);
                if (last_user(q, j))
                    tcgen05_commit(&v_empty[st]);
            };
            // one turn for each tile in order, the products of tile j - 1's probabilities before tile j's scores (S_q may be
            // overwritten: the products of one thread run in order)
#pragma unroll 1
            for (int turn = 0; turn < 2 * (n_tiles + 1); ++turn) {
                const int q = turn & 1, j = turn >> 1;
                if (j > 0 && j - 1 < nt[q])
                    issue_pv(q, j - 1);
                if (j < nt[q])
                    issue_qk(q, j);
            }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ATC2_REGS_MANY));
        const int q = warp >= 12 ? 1 : 0;                    // these warps' query tile
        const int quarter = warp & 3, half = ((warp - 4) >> 2) & 1, thread = quarter * 32 + lane, barrier = 1 + 4 * q + quarter;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16), o_addr = lane_addr + 256 + q * 128 + half * (D / 2);
        const int my_tiles = nt[q];
        QueryRow w = query_row(p, row0 + q * ROWS + thread, rows_total, pos0, kv_head);
        for (int j = 0; j < my_tiles; ++j) {
            const int st = j & 1, key0 = key_begin + j * KEYS;
            mbar_wait_warp(&s_full[q], j & 1, p.error, 45);
            tcgen05_fence_after();
            softmax_row<OPT>(p, w, lane_addr + q * 128 + half * COLS, lane_addr + q * 128 + half * (COLS / 2), o_addr,
                             key0 + half * COLS, j == 0, barrier, maxima + q * 2 * ROWS, half, thread,
                             [&] { mbar_wait_warp(&o_done[q], (j - 1) & 1, p.error, 46); });
            if (key0 + KEYS > key_end) {
                mbar_wait(&v_full[st], (j >> 1) & 1, p.error, 47);
                clear_values(v_s + st * KV_TILE_BYTES, key_end - key0, half * ROWS + thread);
                __syncwarp();
            }
            tmem_store_wait();
            tcgen05_fence_before();
            mbar_arrive(&p_full[q]);
            if (j == 0)
                timeline_mark(1);      // the first tile's probabilities are written
        }
        timeline_mark(2);              // the last tile's probabilities are written
        // the last product has landed: normalise and write the rows out
        if (my_tiles > 0) {
            mbar_wait_warp(&o_done[q], (my_tiles - 1) & 1, p.error, 48);
            tcgen05_fence_after();
            join_sums(w, maxima + q * 2 * ROWS, barrier, half, thread);
            write_rows(p, w, o_addr, q_s + q * Q_BYTES + quarter * 32 * (D * 2), row0 + q * ROWS + quarter * 32, rows_total, t0, kv_head, lane,
                       barrier, half);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// Whether the kernel with one query tile per CTA finishes a plain causal step before the one with two, although that
// would give every SM a CTA: with hardly more CTAs than SMs, the time is that of the CTA with the most keys, and a
// CTA with two tiles takes 1.76 (heads of 64) or 1.5 (128) times as long for a key tile as one with one.  In units of one tile's
// time for 128 keys, 1.5 for a CTA's start and end: the longer of the longest CTA and of all work spread over the SMs,
// the columns of CTAs taken as so many of the longest sequence as the step has tokens for; the estimate has to be 1.08.  Of
// 63 steps of 1 to 4 sequences, up to 3,000 tokens and 6,000 keys before them, both kernels timed, this and the rule of one CTA
// an SM choose the faster one, or one at most 1.09 times as long, but for 4 portions of 220 tokens after 895 (128 CTAs
// with two tiles: 39 us with one, 32 with two).
static bool one_tile_is_faster(long long rows, int group, int max_q_len, int max_ctx_len, long long tokens, int nkv,
                               int window, int chunk, int sms)
{
    const double pair_cost = D == 64 ? 1.76 : 1.5, start = 1.5;
    const long long tiles1 = (rows + ROWS - 1) / ROWS, tiles2 = (rows + 2 * ROWS - 1) / (2 * ROWS);
    const double columns = (double)nkv * (tokens > 0 ? (double)tokens / max_q_len : 1.0);
    int most = max_ctx_len;                       // keys that a row can see
    if (window > 0 && window + ROWS / group < most)
        most = window + ROWS / group;
    if (chunk > 0 && chunk < most)
        most = chunk;
    auto keys = [&](long long rows_before) {      // key tiles of a CTA whose last row is number rows_before - 1
        const long long seen = max_ctx_len - max_q_len + (rows_before < rows ? rows_before : rows) / group;
        return (double)(((seen < most ? seen : most) + KEYS - 1) / KEYS);
    };
    const double longest = keys(rows);
    if (longest < 4.0)
        return false;                             // (four prompts of up to 300 tokens, four heads to a key head: 21.3 and 20.0 us)
    double all1 = 0.0, all2 = 0.0;
    for (long long i = 1; i <= tiles1; ++i)
        all1 += keys(i * ROWS) + start;
    for (long long i = 1; i <= tiles2; ++i)
        all2 += keys(i * 2 * ROWS) * pair_cost + start;
    const double t1 = fmax(longest + start, all1 * columns / sms), t2 = fmax(longest * pair_cost + start, all2 * columns / sms);
    return t2 > 1.08 * t1;
}

} // namespace chibi

using namespace chibi;

CHIBI_API int chibi_attention_tc_head_dim() { return D; }

// Attention of the sequences that bring more than one token (all sequences when
// skip_single is 0).  Returns CHIBI_ERR_UNSUPPORTED for page sizes it does not
// take (the page size must divide 128 and be at least 8).  variant: 0 chooses
// between the kernel with one query tile per CTA (1) and the one with two (2).
CHIBI_API int chibi_attention_prefill_tc(const void* q, const void* k_cache, const void* v_cache, void* out,
                                         const int* block_table, int table_stride, const int* seq_rows,
                                         const int* q_start, const int* ctx_len, int seqs, int nq, int nkv,
                                         int page_size, int num_pages, float scale, int window, int chunk,
                                         int skip_single, int max_q_len, int max_ctx_len, int variant, int kv_splits,
                                         float* scratch, long long scratch_floats, long long tokens,
                                         float softcap, const float* bias_r1, const float* bias_r2,
                                         const float* sink, int* error, cudaStream_t stream)
{
    if (seqs <= 0)
        return CHIBI_OK;
    if (nkv <= 0 || nq % nkv != 0 || window < 0 || chunk < 0 || variant < 0 || variant > 2 || softcap < 0.f
        || (bias_r2 != nullptr && bias_r1 == nullptr))
        return CHIBI_ERR_ARGUMENT;

    if (page_size < 8 || page_size > 128 || KEYS % page_size != 0
        || (reinterpret_cast<uintptr_t>(k_cache) & 15) || (reinterpret_cast<uintptr_t>(v_cache) & 15)
        || (reinterpret_cast<uintptr_t>(q) & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
        return CHIBI_ERR_UNSUPPORTED;
    AttnTcParams p {};
    p.q = static_cast<const __nv_bfloat16*>(q);
    p.out = static_cast<__nv_bfloat16*>(out);
    p.block_table = block_table;
    p.table_stride = table_stride;
    p.seq_rows = seq_rows;
    p.q_start = q_start;
    p.ctx_len = ctx_len;
    p.nq = nq;
    p.nkv = nkv;
    p.group = nq / nkv;
    p.page_size = page_size;
    p.num_pages = num_pages;
    p.cache_rows = (long long)num_pages * nkv * page_size;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.window = window;
    p.chunk = chunk;
    p.skip_single = skip_single;
    p.error = error;
    p.kv_splits = 1;
    p.scale = scale;
    p.softcap = softcap;
    p.bias_r1 = bias_r1;
    p.bias_r2 = bias_r2;
    p.sink = sink;
    const int options = bias_r2 || (softcap > 0.f && bias_r1) ? OPT_ANY
        : softcap > 0.f ? OPT_CAP : (bias_r1 ? OPT_LINEAR : OPT_NONE);
    CUtensorMap mk, mv;
    if (!tensor_map_2d(k_cache, p.cache_rows, D, D, page_size, &mk)
        || !tensor_map_2d(v_cache, p.cache_rows, D, D, page_size, &mv))
        return CHIBI_ERR_UNSUPPORTED;
    CUtensorMap mq = mk;                                  // (not used where a tile's rows are not whole tokens)
    p.q_by_tma = tokens > 0 && ROWS % p.group == 0 && tensor_map_of_heads(q, tokens, nq, D, p.group, ROWS / p.group, &mq);
    using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const AttnTcParams);
    static const Kernel one_tile[4] = { attn_prefill_tc_kernel<OPT_NONE>, attn_prefill_tc_kernel<OPT_ANY>,
                                        attn_prefill_tc_kernel<OPT_LINEAR>, attn_prefill_tc_kernel<OPT_CAP> };
    static const Kernel two_tiles[4] = { attn_prefill_tc2_kernel<OPT_NONE>, attn_prefill_tc2_kernel<OPT_ANY>,
                                         attn_prefill_tc2_kernel<OPT_LINEAR>, attn_prefill_tc2_kernel<OPT_CAP> };
    static bool configured = false;
    if (!configured) {
        for (int i = 0; i < 4; ++i) {
            cudaError_t e = cudaFuncSetAttribute(one_tile[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ATC_SMEM);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(two_tiles[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ATC2_SMEM);
            // (a softmax group that asked for more registers than the block was launched with would wait for good)
            cudaFuncAttributes attr {};
            if (e == cudaSuccess)
                e = cudaFuncGetAttributes(&attr, two_tiles[i]);
            if (e == cudaSuccess && attr.numRegs < ATC2_REGS)
                return CHIBI_ERR_ARGUMENT;
            if (e != cudaSuccess)
                return (int)e;
        }
        configured = true;
    }
    const long long rows = (long long)max_q_len * p.group;
    // Two query tiles per CTA share the key and value tiles and keep the tensor core busier, but
    // halve the number of CTAs: taken when that still gives every SM a CTA (or when asked for).
    const long long ctas2 = ((rows + 2 * ROWS - 1) / (2 * ROWS)) * nkv * seqs;
    int sms = 148, device = 0;
    if (cudaGetDevice(&device) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // (with max_ctx_len 0, not known, that is all the rule)
    const bool two = ctas2 >= sms
        && !(options == OPT_NONE && max_ctx_len > 0 && ctas2 < 2 * sms
             && one_tile_is_faster(rows, p.group, max_q_len, max_ctx_len, tokens, nkv, window, chunk, sms));
    if (variant == 2 || (variant == 0 && two)) {
        const dim3 grid2((unsigned)((rows + 2 * ROWS - 1) / (2 * ROWS)), nkv, seqs);
        launch(two_tiles[options], grid2, dim3(ATC2_THREADS), ATC2_SMEM, stream, mq, mk, mv, p);
        return launch_status();
    }
    if (kv_splits > 1) {
        // key ranges: only this kernel (one query tile per CTA) has them
        if (kv_splits > 64 || !scratch || tokens <= 0 || scratch_floats < tokens * nq * kv_splits * (long long)(D + 2)
            || (long long)seqs * kv_splits > 65535)
            return CHIBI_ERR_ARGUMENT;
        p.kv_splits = kv_splits;
        p.part_o = scratch;
        p.part_ml = scratch + (size_t)tokens * nq * kv_splits * D;
    }
    const dim3 grid((unsigned)((rows + ROWS - 1) / ROWS), nkv, seqs * p.kv_splits);
    launch(one_tile[options], grid, dim3(ATC_THREADS), ATC_SMEM, stream, mq, mk, mv, p);
    int st = launch_status();
    if (st == CHIBI_OK && p.kv_splits > 1) {
        launch(attn_prefill_merge_kernel<D>, dim3(nq, max_q_len, seqs), dim3(D), 0, stream, p);
        st = launch_status();
    }
    return st;
}
