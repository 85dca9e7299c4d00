// Causal grouped-query attention of the 32-bit path over the paged cache, head sizes 64 and 128: all operands and
// results 32-bit (attention_generic.cu says what is computed and which options
// the scores have; it takes the other sizes and types).  Two kernels, one for the sequences that bring one token to a step
// and one for those that bring more.  In both, the order of a row's operations depends on its own position (and on
// whether it came alone), never on the batch around it.
#define CHIBI_UNIT attention_f32
#define CHIBI_UNIT_ID 17
#include "common.cuh"
#include "sm100.cuh"
#include "split_f32.cuh"

namespace chibi {

using namespace sm100;

struct AttentionF32 {
    const float* q;
    const float* k_cache;
    const float* v_cache;
    float* out;
    const int* block_table;
    int table_stride;
    const int* q_start;
    const int* ctx_len;
    const int* seq_rows;
    int nq, nkv, page_size, num_pages;
    float scale;
    int window, chunk;
    float softcap;
    const float* bias_r1;
    const float* bias_r2;
    const float* sink;
    int* error;
};

__device__ __forceinline__ void af_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
// What lies at the same place of the shared memory of CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t af_peer_address(const float* local, int rank)
{
    uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local)), b;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
    return b;
}
__device__ __forceinline__ float af_peer(const float* local, int rank)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(af_peer_address(local, rank)) : "memory");
    return v;
}
// What becomes of a dot product; `distance`: query position - key position.
__device__ __forceinline__ float af_score(const AttentionF32& p, float dot, float r1, float r2, int distance)
{
    float s = dot * p.scale;
    if (p.softcap > 0.f)
        s = p.softcap * tanhf(s / p.softcap);
    if (p.bias_r1)
        s -= p.bias_r2 ? r1 * log1pf(r2 * (float)distance) : r1 * (float)distance;
    return s;
}
// exp(m - m_new), with nothing kept of a maximum that was none yet.
__device__ __forceinline__ float af_keep(float m, float m_new) { return m == -INFINITY ? 0.f : expf(m - m_new); }

// ---------------------------------------------------------------- sequences that bring several tokens
// On the 5th-generation tensor cores: numbers are split into three bfloat16 parts (split_f32.cuh), and six of the nine partial
// products are tcgen05.mma with 32-bit accumulators.  What limits the precision is the accumulator, which the tensor core cuts
// off instead of rounding: so every sum over 64 features or keys has an accumulator of its own, that takes the five small
// products first and the large one last, and those sums are added in plain 32-bit arithmetic.  Relative error against 64 bits,
// 3 prompts of up to 400 tokens: 1.6e-7, by multiply-adds (fma.rn.f32x2) before 2.1e-7 (values of one sign 1.05e-7 and 1.0e-7, for
// the accumulators are cut off downwards).
//
// A CTA owns 128 query rows of one kv head, (token, head of the group) pairs, and walks over the keys in blocks of 64, counted
// from the sequence's start: what a row gives does not depend on the rows beside it (a key that it does not see has
// probability 0 and leaves its sums as they are).  Warp 0 issues the MMAs.  Warps 4 to 19 do the rest: four threads own a
// row, a quarter of a block's keys and of the output's columns each; all of them bring queries, keys and values (in registers, a
// block ahead), split them and write the parts into the swizzled tiles that the MMAs read; probabilities go through TMEM as the
// A operand.  S = Q K^T of the next block runs while a block's softmax is made, O = P V while the next keys are split.
// Bound by the products beside the threads' work: 48 MMAs of 128 x 64 x 16 (shared memory: 48 cycles each) and 24 of
// 128 x D x 16 (64) a block, 3,900 cycles for heads of 128.  An issuing thread waits while they run (issued by one of the
// working warps a block took 11,400).  Heads of 128, us by multiply-adds (64 rows a CTA, four CTAs to a row tile's keys) and
// so: with keys and values that are not in
// L2: 3 prompts of up to 400 tokens of 16 heads 104 and 45 (in L2 109 and 37), 4 of 600 after 800 of 32 heads 1,536 and 383, 64 tokens
// after 800 of 16 heads 84 and 76, 100 after 4,000 315 and 285, 4 after 800 82 and 70; 2,000 tokens, heads of 64, 393 and 145.
//
// Scores and outputs are 2^32 as large as they should be until they are used.  A query or key without parts (no number, or from
// 2^112 on) makes its scores no number; those, and scores from 2^96 on, are summed by multiply-adds.  Such values are marked
// and taken out, because they would spoil the rows that do not see them: what is no number adds itself to its column of the rows
// that do, and rows that see a large one, or whose sums are too large, are made by hand.
constexpr int AT_ROWS = 128, AT_KEYS = 64, AT_WORKERS = 512, AT_THREADS = 128 + AT_WORKERS;
constexpr int AT_REGS = 96, AT_REGS_FEW = 32, AT_REGS_MANY = 112;    // of a thread at launch, of the first four warps', of the others'
static_assert(AT_REGS_FEW + 4 * AT_REGS_MANY <= 5 * AT_REGS, "more registers than the block has");
constexpr int AT_SHARE = AT_WORKERS / AT_ROWS, AT_OWN = AT_KEYS / AT_SHARE;     // threads of a row; keys of a thread

template <int D> struct AtShape {
    static constexpr int SLICES = D / 64;                        // 64 features are a swizzled line
    static constexpr int Q_PLANE = AT_ROWS * D * 2, KV_PLANE = AT_KEYS * D * 2;
    static constexpr int TILES = 3 * Q_PLANE + 6 * KV_PLANE;
    static constexpr size_t SHARED = 1024 + TILES + 64 + 4 * (3 * AT_SHARE * AT_ROWS + 12);
    static constexpr uint32_t S_COLS = 64 * SLICES;              // TMEM: two buffers of S, three parts of P, O
    static constexpr uint32_t P_AT = 2 * S_COLS, O_AT = P_AT + 96, TMEM = O_AT + D <= 256 ? 256 : 512;
};

// Writes the parts of four numbers without what has none (2^16 times it is infinite as bfloat16, or it is no number); true if
// there was one.
__device__ __noinline__ bool at_split_odd(float4 v, uint32_t at, uint32_t plane)
{
    bool found = false;
    auto one = [&](float& x) {
        if ((__float_as_uint(x) & 0x7fffffffu) >= 0x777f8000u) {
            x = 0.f;
            found = true;
        }
    };
    one(v.x), one(v.y), one(v.z), one(v.w);
    if (found)
        split_to_shared(v, at, plane);
    return found;
}
__device__ __noinline__ float at_dot(const float* a, const float* b, int d)
{
    float s[4] = { 0.f, 0.f, 0.f, 0.f };
    for (int i = 0; i < d; i += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a + i), y = *reinterpret_cast<const float4*>(b + i);
        s[0] = fmaf(x.x, y.x, s[0]);
        s[1] = fmaf(x.y, y.y, s[1]);
        s[2] = fmaf(x.z, y.z, s[2]);
        s[3] = fmaf(x.w, y.w, s[3]);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
}
// A thread's part of a row's output (COLS columns, by pieces of four in swizzled places), the scores and the sums of the products
// anew, in 64 bits what could be too large for 32: exponents against `top`, times `inv` at the end.
template <int D, bool OPTIONS>
__device__ __noinline__ void at_row_by_hand(const AttentionF32& p, const int* table, int token, int h, int kv_head, int pos, int first,
                                            int part, float top, float inv, float* out, int swizzle)
{
    constexpr int COLS = D / AT_SHARE, PIECES = COLS / 4;
    const float* const q = p.q + ((size_t)token * p.nq + h) * D;
    const float r1 = p.bias_r1 ? p.bias_r1[h] : 0.f, r2 = p.bias_r2 ? p.bias_r2[h] : 0.f, least = top == -INFINITY ? 0.f : top;
    double sum[COLS];
    for (int c = 0; c < COLS; ++c)
        sum[c] = 0.0;
    for (int key = first; key <= pos; ++key) {
        const int page = table[key / p.page_size];
        if (page < 0 || page >= p.num_pages)
            continue;
        const size_t at = (size_t)((page * p.nkv + kv_head) * p.page_size + key % p.page_size) * D;
        const float dot = at_dot(q, p.k_cache + at, D);
        const double e = expf((OPTIONS ? af_score(p, dot, r1, r2, pos - key) : dot * p.scale) - least);
        for (int c = 0; c < COLS; ++c)
            sum[c] = fma(e, (double)p.v_cache[at + part * COLS + c], sum[c]);
    }
    for (int c = 0; c < COLS; ++c)
        reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(out) + (((part * PIECES + c / 4) ^ (swizzle & 7)) << 4))[c & 3] = (float)(sum[c] * inv);
}
// A thread's scores that the tensor cores could not make (infinite or no number), by multiply-adds; those of hidden keys stay.
template <int D, bool OPTIONS>
__device__ __noinline__ void at_scores_in_memory(const AttentionF32& p, float* s, const int* table, int token, int h, int kv_head, int key0,
                                                 int first, int pos)
{
    const float* const q = p.q + ((size_t)token * p.nq + h) * D;
    for (int i = 0; i < AT_OWN; ++i) {
        const int key = key0 + i;
        if (fabsf(s[i]) < INFINITY || key > pos || key < first)
            continue;
        const int page = table[key / p.page_size];
        if (page < 0 || page >= p.num_pages)
            continue;
        const float* const k = p.k_cache + (size_t)((page * p.nkv + kv_head) * p.page_size + key % p.page_size) * D;
        if (q[0] != q[0] || k[0] != k[0])                        // (a row of which nothing is a number: it is none already)
            continue;
        const float dot = at_dot(q, k, D);
        s[i] = OPTIONS ? dot : dot * p.scale;
    }
}
// (By way of memory: with the registers indexed here, and this call among them, all calls took 4 to 7 % longer.)
template <int D, bool OPTIONS>
__device__ __forceinline__ void at_scores_by_hand(const AttentionF32& p, float (&s)[AT_OWN], const int* table, int token, int h, int kv_head,
                                                  int key0, int first, int pos)
{
    float there[AT_OWN];
#pragma unroll
    for (int i = 0; i < AT_OWN; ++i)
        there[i] = s[i];
    at_scores_in_memory<D, OPTIONS>(p, there, table, token, h, kv_head, key0, first, pos);
#pragma unroll
    for (int i = 0; i < AT_OWN; ++i)
        s[i] = there[i];
}
// The warps that share 32 rows.
__device__ __forceinline__ void at_row_sync(int barrier)
{
    asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(barrier), "n"(32 * AT_SHARE) : "memory");
}
// MN-major operand (V: [key][d]) in swizzled slices of 64 columns, `slice` bytes apart.
__device__ __forceinline__ uint64_t at_values_desc(uint32_t smem_byte_addr, uint32_t slice)
{
    return static_cast<uint64_t>((smem_byte_addr & 0x3ffff) >> 4) | static_cast<uint64_t>((slice >> 4) & 0x3fff) << 16
        | static_cast<uint64_t>(1024 >> 4) << 32 | static_cast<uint64_t>(1) << 46 | static_cast<uint64_t>(2) << 61;
}

template <int COUNT> __device__ __forceinline__ void at_tmem_load(uint32_t at, uint32_t (&r)[COUNT])
{
    static_assert(COUNT == 16 || COUNT == 32);
    if constexpr (COUNT == 32)
        tmem_load_32x32(at, r);
    else
        tmem_load_32x16(at, r);
}

template <int D, bool OPTIONS>
__global__ void __launch_bounds__(AT_THREADS, 1)
attention_f32_prompt_kernel(const __grid_constant__ AttentionF32 p)
{
    pdl_enter();
    using Shape = AtShape<D>;
    constexpr int QUADS = D / 4, PASS = AT_WORKERS / QUADS;      // rows that all threads bring at a time
    constexpr int KV_EACH = AT_KEYS / PASS, Q_EACH = AT_ROWS / PASS;
    extern __shared__ uint8_t at_raw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(at_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t q_s = smem_addr(smem), k_s = q_s + 3 * Shape::Q_PLANE, v_s = k_s + 3 * Shape::KV_PLANE;
    uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + Shape::TILES);
    uint64_t* const keys_there = bars;           // working threads: the keys are written
    uint64_t* const p_there = bars + 1;          // working threads: probabilities and values are written
    uint64_t* const s_done = bars + 2;           // MMA commit
    uint64_t* const o_done = bars + 3;           // MMA commit
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
    float* const exchange = reinterpret_cast<float*>(bars + 8);          // [4][128]
    // marks of values that have no parts: [4][2], of a block's 64 keys (block j in place j % 4), and whether there are any at all
    uint32_t* const odd_values = reinterpret_cast<uint32_t*>(exchange + AT_SHARE * AT_ROWS);
    uint32_t* const odd_any = odd_values + 8;
    // [512] of each working thread: the columns that a value which is no number has added itself to; whether a value that is too
    // large is among what it sees (rare events: in memory they take no registers)
    uint32_t* const spoiled = odd_any + 4;
    uint32_t* const large = spoiled + AT_WORKERS;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int seq = blockIdx.z, kv_head = blockIdx.y, G = p.nq / p.nkv;
    const int row0 = p.q_start[seq], q_len = p.q_start[seq + 1] - row0;
    if (q_len <= 1)
        return;                                                  // (a single token is the other kernel's)
    const int all_rows = q_len * G, tile = (all_rows + AT_ROWS - 1) / AT_ROWS - 1 - (int)blockIdx.x;     // most keys first
    if (tile < 0)
        return;
    const int pos0 = p.ctx_len[seq] - q_len;                     // the first token's position
    const int* const table = p.block_table + (size_t)(p.seq_rows ? p.seq_rows[seq] : seq) * p.table_stride;
    const int first_row = tile * AT_ROWS, last_pos = pos0 + (min(first_row + AT_ROWS, all_rows) - 1) / G;
    const int oldest = first_visible_key(pos0 + first_row / G, p.window, p.chunk);      // (older pages may be gone)
    const int begin = oldest / AT_KEYS * AT_KEYS, blocks = (last_pos - begin) / AT_KEYS + 1;

    if (tid == 0) {
        mbar_init(keys_there, AT_WORKERS);
        mbar_init(p_there, AT_WORKERS);
        mbar_init(s_done, 1);
        mbar_init(o_done, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, Shape::TMEM);
        tmem_relinquish();
    }
    if (tid < 12)
        odd_values[tid] = 0;

    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AT_REGS_FEW));
        if (warp == 0 && elect_one()) {
            constexpr uint32_t idesc_s = make_idesc_bf16_f32(AT_ROWS, AT_KEYS), idesc_o = make_idesc_bf16_f32(AT_ROWS, D) | (1u << 16);
            const uint64_t q_desc = make_kmajor_sw128_desc(q_s), k_desc = make_kmajor_sw128_desc(k_s);
            const uint64_t v_desc = at_values_desc(v_s, AT_KEYS * 128);
            auto scores = [&](int j) {
                uint64_t a = q_desc, b = k_desc;
                asm volatile("" : "+l"(a), "+l"(b));                 // (or 48 sums of constants wait in registers from block to block)
                mbar_wait(keys_there, j & 1, p.error, 71);
                tcgen05_fence_after();
#pragma unroll
                for (int slice = 0; slice < Shape::SLICES; ++slice) {
                    const uint32_t d = tmem + (j & 1) * Shape::S_COLS + slice * 64;
                    auto product = [&](int pq, int pk, int ks, uint32_t more) {
                        tcgen05_mma_bf16(d, a + ((pq * Shape::Q_PLANE + slice * AT_ROWS * 128 + ks * 32) >> 4),
                                         b + ((pk * Shape::KV_PLANE + slice * AT_KEYS * 128 + ks * 32) >> 4), idesc_s, more);
                    };
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        product(2, 0, ks, ks > 0 ? 1u : 0u);
                        product(1, 1, ks, 1u);
                        product(1, 0, ks, 1u);
                        product(0, 2, ks, 1u);
                        product(0, 1, ks, 1u);
                    }
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        product(0, 0, ks, 1u);
                }
                tcgen05_commit(s_done);
            };
            auto outputs = [&](int j) {
                uint64_t b = v_desc;
                asm volatile("" : "+l"(b));
                mbar_wait(p_there, j & 1, p.error, 72);
                tcgen05_fence_after();
                auto product = [&](int pp, int pv, int ks, uint32_t more) {
                    tcgen05_mma_bf16_a_tmem(tmem + Shape::O_AT, tmem + Shape::P_AT + pp * 32 + ks * 8,
                                            b + ((pv * Shape::KV_PLANE + ks * 16 * 128) >> 4), idesc_o, more);
                };
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    product(2, 0, ks, ks > 0 ? 1u : 0u);
                    product(1, 1, ks, 1u);
                    product(1, 0, ks, 1u);
                    product(0, 2, ks, 1u);
                    product(0, 1, ks, 1u);
                }
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    product(0, 0, ks, 1u);
                tcgen05_commit(o_done);
            };
            scores(0);
            for (int j = 0; j < blocks; ++j) {
                if (j + 1 < blocks)
                    scores(j + 1);
                outputs(j);
            }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AT_REGS_MANY));
        // four columns of rows line + PASS i of a tile: where they lie in a part of the queries, and of the keys or values
        static_assert(PASS % 8 == 0);
        const int worker = tid - (AT_THREADS - AT_WORKERS), quad = worker % QUADS, line = worker / QUADS;
        const uint32_t inside = (uint32_t)((line >> 3) * 1024 + (line & 7) * 128 + ((((4 * quad & 63) >> 3) ^ (line & 7)) << 4) + (quad & 1) * 8);
        const uint32_t q_at = (quad >> 4) * (AT_ROWS * 128) + inside, kv_at = (quad >> 4) * (AT_KEYS * 128) + inside;
        // Which rows of the cache a warp brings of a block's keys and values (-1: none): lane i looks up the i-th.
        constexpr int WARP_ROWS = 32 / QUADS > 1 ? 32 / QUADS : 1, FOUND = KV_EACH * WARP_ROWS;
        static_assert(AT_WORKERS % QUADS == 0 && QUADS <= 32 && FOUND <= 32);
        auto lookup = [&](int base) {                                // the page, as it stands in the table
            const int u = base + worker / QUADS / WARP_ROWS * WARP_ROWS + lane % WARP_ROWS + PASS * (lane / WARP_ROWS);
            return lane < FOUND && u >= oldest && u <= last_pos ? table[u / p.page_size] : -2;
        };
        auto row_in = [&](int base, int page) {                      // and the key's row there
            const int u = base + worker / QUADS / WARP_ROWS * WARP_ROWS + lane % WARP_ROWS + PASS * (lane / WARP_ROWS);
            if (page < 0 || page >= p.num_pages) {
                if (page != -2 && p.error)
                    atomicExch(p.error, 3);
                return -1;
            }
            return (page * p.nkv + kv_head) * p.page_size + u % p.page_size;
        };
        auto fetch = [&](const float* cache, int found, float4 (&v)[KV_EACH]) {
#pragma unroll
            for (int i = 0; i < KV_EACH; ++i) {
                const int at = __shfl_sync(0xffffffffu, found, WARP_ROWS * i + lane / QUADS);
                v[i] = at >= 0 ? *reinterpret_cast<const float4*>(cache + (size_t)at * D + 4 * quad) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        auto spread = [&](const float4 (&v)[KV_EACH], uint32_t to) {
            uint64_t last = 0;
#pragma unroll
            for (int i = 0; i < KV_EACH; ++i)
                last = pair_add(split_to_shared(v[i], to + kv_at + i * (PASS / 8) * 1024, Shape::KV_PLANE), last);
            return last;
        };
        auto spread_values = [&](const float4 (&v)[KV_EACH], uint32_t* flags) {
            if (pair_is_none(spread(v, v_s))) {
#pragma unroll
                for (int i = 0; i < KV_EACH; ++i) {
                    const int r = line + PASS * i;
                    if (at_split_odd(v[i], v_s + kv_at + i * (PASS / 8) * 1024, Shape::KV_PLANE)) {
                        atomicOr(&flags[r >> 5], 1u << (r & 31));
                        *odd_any = 1;
                    }
                }
            }
            __syncwarp();
        };
        float4 kn[KV_EACH], vn[KV_EACH];
        int page[3], found[2];                                       // pages of blocks j + 1 .. j + 3 (looked up long before they are
                                                                     // looked at); rows of blocks j + 1 and j + 2
        {
            const int first_page = lookup(begin);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                page[i] = lookup(begin + (i + 1) * AT_KEYS);
            found[0] = row_in(begin, first_page);
        }
        fetch(p.k_cache, found[0], kn);
        fetch(p.v_cache, found[0], vn);
        found[0] = row_in(begin + AT_KEYS, page[0]);
        found[1] = row_in(begin + 2 * AT_KEYS, page[1]);
        int ahead = page[2];
        // the queries, in two goes
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float4 v[Q_EACH / 2];
#pragma unroll
            for (int i = 0; i < Q_EACH / 2; ++i) {
                const int row = first_row + line + PASS * (i + half * (Q_EACH / 2));
                v[i] = row < all_rows ? *reinterpret_cast<const float4*>(p.q + ((size_t)(row0 + row / G) * p.nq + kv_head * G + row % G) * D + 4 * quad)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < Q_EACH / 2; ++i)
                split_to_shared(v[i], q_s + q_at + (i + half * (Q_EACH / 2)) * (PASS / 8) * 1024, Shape::Q_PLANE);
        }
        spread(kn, k_s);
        fence_proxy_async();
        mbar_arrive(keys_there);
        if (blocks > 1)
            fetch(p.k_cache, found[0], kn);

        // ---- a thread's row, its part of the keys and of the columns
        const int quarter = warp & 3, part = (warp - 4) >> 2, r = quarter * 32 + lane, barrier = 1 + quarter;
        const int row = min(first_row + r, all_rows - 1), h = kv_head * G + row % G, pos = pos0 + row / G;
        const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
        const float r1 = p.bias_r1 ? p.bias_r1[h] : 0.f, r2 = p.bias_r2 ? p.bias_r2[h] : 0.f;
        const int first = first_visible_key(pos, p.window, p.chunk);
        constexpr int COLS = D / AT_SHARE;
        uint64_t O[COLS / 2];
        const float down = OPTIONS ? SPLIT_DOWN : p.scale * SPLIT_DOWN;
        const uint64_t down2 = pair_of(down, down);
        float m = -INFINITY, l = 0.f;
        spoiled[worker] = large[worker] = 0;
#pragma unroll
        for (int c = 0; c < COLS / 2; ++c)
            O[c] = 0;
        auto key_at = [&](int key) -> long long {                    // where a key's numbers begin, -1 if its page is none of the pool's
            const int page = table[key / p.page_size];
            return page < 0 || page >= p.num_pages ? -1 : (long long)((page * p.nkv + kv_head) * p.page_size + key % p.page_size) * D;
        };
        auto add_output = [&](int j) {                // what block j's product has found
            mbar_wait_warp(o_done, j & 1, p.error, 74);
            tcgen05_fence_after();
            uint32_t v[COLS];
            at_tmem_load(lanes + Shape::O_AT + part * COLS, v);
            tmem_load_wait();
#pragma unroll
            for (int c = 0; c < COLS / 2; ++c)
                O[c] = pair_fma(O[c], PAIR_ONES, pair_of(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1])));
            if (*odd_any) {
                uint32_t found = 0;                                  // columns, as in `spoiled`
                bool too_large = false, left = false;                // (nothing is left to spoil where all are none)
#pragma unroll
                for (int c = 0; c < COLS / 2; ++c) {
                    const float2 o = halves_of(O[c]);
                    left |= o.x == o.x || o.y == o.y;
                }
                for (int i = 0; i < AT_KEYS && left; ++i) {
                    const int key = begin + j * AT_KEYS + i;
                    if ((odd_values[2 * (j & 3) + (i >> 5)] >> (i & 31) & 1) && key <= pos && key >= first) {
                        const float* const v = p.v_cache + key_at(key) + part * COLS;        // (what is marked has been read)
#pragma unroll
                        for (int c = 0; c < COLS / 2; ++c) {
                            const float x = v[2 * c], y = v[2 * c + 1];
                            const bool no_x = !(fabsf(x) < INFINITY), no_y = !(fabsf(y) < INFINITY);
                            const float2 o = halves_of(O[c]);
                            O[c] = pair_of(o.x + (no_x ? x : 0.f), o.y + (no_y ? y : 0.f));
                            found |= (no_x ? 1u : 0u) << (2 * c) | (no_y ? 2u : 0u) << (2 * c);
                            too_large |= (!no_x && fabsf(x) >= 0x1p111f) || (!no_y && fabsf(y) >= 0x1p111f);
                        }
                    }
                }
                spoiled[worker] |= found;
                large[worker] |= too_large;
            }
            __syncwarp();
        };
        for (int j = 0; j < blocks; ++j) {
            const int base = begin + j * AT_KEYS;
            mbar_wait_warp(s_done, j & 1, p.error, 73);
            tcgen05_fence_after();
            // (a place of a block that all threads are through with: everyone has written keys j)
            if (worker < 2)
                odd_values[2 * ((j + 1) & 3) + worker] = 0;
            // the next block's scores are made while this one's are worked on
            if (j + 1 < blocks) {
                spread(kn, k_s);
                fence_proxy_async();
                tcgen05_fence_before();
                mbar_arrive(keys_there);
                if (j + 2 < blocks)
                    fetch(p.k_cache, found[1], kn);
            }
            float s[AT_OWN];
            uint64_t none = 0;                                       // (no number, or infinite, if a score is)
            {
                uint32_t v[Shape::SLICES][AT_OWN];
#pragma unroll
                for (int slice = 0; slice < Shape::SLICES; ++slice)
                    at_tmem_load(lanes + (j & 1) * Shape::S_COLS + slice * 64 + part * AT_OWN, v[slice]);
                tmem_load_wait();
                uint64_t pairs[AT_OWN / 2];
#pragma unroll
                for (int i = 0; i < AT_OWN / 2; ++i) {
                    pairs[i] = pair_of(__uint_as_float(v[0][2 * i]), __uint_as_float(v[0][2 * i + 1]));
                    if (Shape::SLICES > 1)
                        pairs[i] = pair_add(pairs[i], pair_of(__uint_as_float(v[Shape::SLICES - 1][2 * i]), __uint_as_float(v[Shape::SLICES - 1][2 * i + 1])));
                    pairs[i] = pair_mul(pairs[i], down2);
                    if (i % 2)
                        none = pair_fma(pairs[i - 1], pairs[i], none);
                    const float2 h = halves_of(pairs[i]);
                    s[2 * i] = h.x;
                    s[2 * i + 1] = h.y;
                }
            }
            const int key0 = base + part * AT_OWN;
            if (pair_is_none(none))
                at_scores_by_hand<D, OPTIONS>(p, s, table, row0 + row / G, h, kv_head, key0, first, pos);
            // every row sees every key of these?
            const bool whole = __all_sync(0xffffffffu, key0 + AT_OWN - 1 <= pos && key0 >= first);
            float most = -INFINITY;
            if (OPTIONS) {
#pragma unroll
                for (int i = 0; i < AT_OWN; ++i)
                    s[i] = af_score(p, s[i], r1, r2, pos - key0 - i);
            }
            if (!whole) {
#pragma unroll
                for (int i = 0; i < AT_OWN; ++i)
                    if (key0 + i > pos || key0 + i < first)
                        s[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < AT_OWN; ++i)
                most = fmaxf(most, s[i]);
            exchange[part * AT_ROWS + r] = most;
            at_row_sync(barrier);
            float m_new = m;
#pragma unroll
            for (int x = 0; x < AT_SHARE; ++x)
                m_new = fmaxf(m_new, exchange[x * AT_ROWS + r]);
            at_row_sync(barrier);                                    // (read before the next block's are written)
            const float keep = af_keep(m, m_new), least = m_new == -INFINITY ? 0.f : m_new;
            m = m_new;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < AT_OWN; ++i) {
                s[i] = expf(s[i] - least);                           // (of a hidden key: 0)
                sum += s[i];
            }
            l = l * keep + sum;
            if (j > 0)
                add_output(j - 1);
            const uint64_t keep2 = pair_of(keep, keep);
#pragma unroll
            for (int c = 0; c < COLS / 2; ++c)
                O[c] = pair_mul(O[c], keep2);
            uint64_t s2[AT_OWN / 2];
#pragma unroll
            for (int i = 0; i < AT_OWN / 2; ++i)
                s2[i] = pair_mul(pair_of(s[2 * i], s[2 * i + 1]), SPLIT_UP);
#pragma unroll
            for (int plane = 0; plane < 3; ++plane) {
                uint32_t pairs[AT_OWN / 2];
#pragma unroll
                for (int i = 0; i < AT_OWN / 2; ++i) {
                    pairs[i] = bf16_pair(s2[i]);
                    s2[i] = without_bf16_pair(s2[i], pairs[i]);
                }
                tmem_store_32x8(lanes + Shape::P_AT + plane * 32 + part * (AT_OWN / 2), pairs);
            }
            spread_values(vn, odd_values + 2 * (j & 3));
            tmem_store_wait();
            fence_proxy_async();
            tcgen05_fence_before();
            mbar_arrive(p_there);
            if (j + 1 < blocks)
                fetch(p.v_cache, found[0], vn);
            found[0] = found[1];
            found[1] = row_in(base + 3 * AT_KEYS, ahead);
            ahead = lookup(base + 4 * AT_KEYS);
        }
        add_output(blocks - 1);
        // ---- the row's sum of all its threads, and the rows by way of the queries' place: neighbouring lanes store neighbouring pieces
        exchange[part * AT_ROWS + r] = l;
        at_row_sync(barrier);
        l = 0.f;
#pragma unroll
        for (int x = 0; x < AT_SHARE; ++x)
            l += exchange[x * AT_ROWS + r];
        float top = m;
        if (p.sink) {
            const float sink = p.sink[h];
            top = fmaxf(sink, m);
            const float keep = af_keep(m, top);
            l = l * keep + af_keep(sink, top);
            const uint64_t keep2 = pair_of(keep, keep);
#pragma unroll
            for (int c = 0; c < COLS / 2; ++c)
                O[c] = pair_mul(O[c], keep2);
        }
        const float inv = l > 0.f ? 1.f / l : 0.f, inv_down = inv * SPLIT_DOWN;
        uint32_t none = 0;                                           // columns whose sums are no number, or too large for one
#pragma unroll
        for (int c = 0; c < COLS / 2; ++c) {
            const float2 o = halves_of(O[c]);
            none |= (fabsf(o.x) < INFINITY ? 0u : 1u) << (2 * c) | (fabsf(o.y) < INFINITY ? 0u : 2u) << (2 * c);
        }
        const bool by_hand = l == l && ((none & ~spoiled[worker]) || large[worker]);     // (with a score that is none all of the row is)
        constexpr int CHUNKS = D / 4, SHARE = CHUNKS / AT_SHARE;     // pieces of 16 bytes of a row, and a thread's
        uint8_t* const rows = smem + quarter * 32 * (D * 4);
#pragma unroll
        for (int c = 0; c < SHARE; ++c) {
            const float2 a = halves_of(O[2 * c]), b = halves_of(O[2 * c + 1]);
            *reinterpret_cast<float4*>(rows + lane * (D * 4) + (((part * SHARE + c) ^ (lane & 7)) << 4)) =
                make_float4(a.x * inv_down, a.y * inv_down, b.x * inv_down, b.y * inv_down);
        }
        if (by_hand)
            at_row_by_hand<D, OPTIONS>(p, table, row0 + row / G, h, kv_head, pos, first, part, top, inv,
                                       reinterpret_cast<float*>(rows + lane * (D * 4)), lane);
        __syncwarp();
        at_row_sync(barrier);
#pragma unroll 4
        for (int i = part * 32 * SHARE + lane; i < (part + 1) * 32 * SHARE; i += 32) {
            const int rr = i / CHUNKS, c = i % CHUNKS, to = first_row + quarter * 32 + rr;
            if (to < all_rows)
                *reinterpret_cast<float4*>(p.out + ((size_t)(row0 + to / G) * p.nq + kv_head * G + to % G) * D + 4 * c) =
                    *reinterpret_cast<const float4*>(rows + rr * (D * 4) + ((c ^ (rr & 7)) << 4));
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) {
        tcgen05_fence_after();
        tmem_dealloc(tmem, Shape::TMEM);
    }
}

// ---------------------------------------------------------------- sequences that bring one token
// A cluster of up to eight CTAs to a sequence, kv head and GT of its query heads; each takes a range of the keys (an
// eighth of them, 64 at least) in its four warps.  Eight lanes share a key, each with an eighth of its
// features in 16-byte pieces, four keys to a warp at a time, and keep a softmax of their own; the four of a warp,
// the warps and the CTAs are put together at the end.  Bound by the keys' and values' way from memory; the next
// keys are on their way while these are used.
template <int D, int GT>
__global__ void __launch_bounds__(128)
attention_f32_token_kernel(const AttentionF32 p, int ranks, int head_blocks)
{
    pdl_enter();
    constexpr int N = D / 32;                           // 16-byte pieces of a lane
    __shared__ float part_m[4][GT], part_l[4][GT], part_o[4][GT][D];
    __shared__ float range_m[GT], range_l[GT], range_o[GT][D];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, at = lane & 7;
    const int seq = blockIdx.z, kv_head = blockIdx.y / head_blocks, G = p.nq / p.nkv;
    const int h0 = kv_head * G + GT * ((int)blockIdx.y % head_blocks), heads = min(GT, kv_head * G + G - h0);
    const int row = p.q_start[seq], rank = blockIdx.x;
    if (p.q_start[seq + 1] - row != 1)
        return;                                         // (all CTAs of the cluster alike)
    const int pos = p.ctx_len[seq] - 1, first = first_visible_key(pos, p.window, p.chunk);
    const int* const table = p.block_table + (size_t)(p.seq_rows ? p.seq_rows[seq] : seq) * p.table_stride;
    const int keys = pos + 1 - first;
    const int range = max(64, (keys + 255) / 256 * 32); // an eighth, in steps of 32

    uint64_t q[GT][N][2], o[GT][N][2];
    float m[GT], l[GT], r1[GT], r2[GT];
#pragma unroll
    for (int g = 0; g < GT; ++g) {
        const int h = h0 + min(g, heads - 1);
        m[g] = -INFINITY;
        l[g] = 0.f;
        r1[g] = p.bias_r1 ? p.bias_r1[h] : 0.f;
        r2[g] = p.bias_r2 ? p.bias_r2[h] : 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p.q + ((size_t)row * p.nq + h) * D + 4 * at + 32 * i);
            q[g][i][0] = v.x;
            q[g][i][1] = v.y;
            o[g][i][0] = o[g][i][1] = 0;
        }
    }
    for (int start = first + rank * range; start <= pos; start += ranks * range) {
        const int end = min(start + range, pos + 1);
        // (key, its row of the cache) of a turn; a row is -1 past the end and where the page is not one of the pool's
        auto row_of = [&](int u) -> long long {
            if (u >= end)
                return -1;
            const int page = table[u / p.page_size];
            if (page < 0 || page >= p.num_pages) {
                if (p.error)
                    atomicExch(p.error, 3);
                return -1;
            }
            return (((long long)page * p.nkv + kv_head) * p.page_size + u % p.page_size) * D;
        };
        ulonglong2 k[N], v[N];
        auto fetch = [&](const float* cache, long long from, ulonglong2 (&dst)[N]) {
#pragma unroll
            for (int i = 0; i < N; ++i)
                dst[i] = from >= 0 ? __ldcg(reinterpret_cast<const ulonglong2*>(cache + from + 4 * at + 32 * i))
                                   : make_ulonglong2(0, 0);
        };
        int u = start + 4 * warp + (lane >> 3);
        long long here = row_of(u);
        fetch(p.k_cache, here, k);
        fetch(p.v_cache, here, v);
        // (a warp's four keys go together: the sums over a key's lanes are shuffles of the whole warp)
        for (int turn = start + 4 * warp; turn < end; turn += 16, u += 16) {
            const long long next = row_of(u + 16);
            ulonglong2 kn[N], vn[N];
            fetch(p.k_cache, next, kn);
            fetch(p.v_cache, next, vn);
#pragma unroll
            for (int g = 0; g < GT; ++g) {
                uint64_t d0 = 0, d1 = 0;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    d0 = pair_fma(q[g][i][0], k[i].x, d0);
                    d1 = pair_fma(q[g][i][1], k[i].y, d1);
                }
                const float2 a = halves_of(d0), b = halves_of(d1);
                float dot = (a.x + a.y) + (b.x + b.y);
#pragma unroll
                for (int x = 4; x > 0; x >>= 1)
                    dot += __shfl_xor_sync(0xffffffffu, dot, x);
                if (here >= 0) {
                    const float s = af_score(p, dot, r1[g], r2[g], pos - u);
                    const float m_new = fmaxf(m[g], s);
                    const float keep = af_keep(m[g], m_new), e = s == -INFINITY ? 0.f : expf(s - m_new);
                    const uint64_t k2 = pair_of(keep, keep), e2 = pair_of(e, e);
                    l[g] = l[g] * keep + e;
                    m[g] = m_new;
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        o[g][i][0] = pair_fma(e2, v[i].x, pair_mul(o[g][i][0], k2));
                        o[g][i][1] = pair_fma(e2, v[i].y, pair_mul(o[g][i][1], k2));
                    }
                }
            }
            here = next;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                k[i] = kn[i];
                v[i] = vn[i];
            }
        }
    }
    // the warp's four softmaxes become one
#pragma unroll
    for (int g = 0; g < GT; ++g) {
        float top = m[g];
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
        const float keep = af_keep(m[g], top);
        float sum = l[g] * keep;
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                float2 a = halves_of(o[g][i][x]);
                a.x *= keep;
                a.y *= keep;
                a.x += __shfl_xor_sync(0xffffffffu, a.x, 8);
                a.y += __shfl_xor_sync(0xffffffffu, a.y, 8);
                a.x += __shfl_xor_sync(0xffffffffu, a.x, 16);
                a.y += __shfl_xor_sync(0xffffffffu, a.y, 16);
                if (lane < 8)
                    *reinterpret_cast<float2*>(&part_o[warp][g][4 * at + 32 * i + 2 * x]) = a;
            }
        if (lane == 0) {
            part_m[warp][g] = top;
            part_l[warp][g] = sum;
        }
    }
    __syncthreads();
    for (int i = tid; i < GT * D; i += 128) {
        const int g = i / D, c = i % D;
        float top = part_m[0][g];
#pragma unroll
        for (int w = 1; w < 4; ++w)
            top = fmaxf(top, part_m[w][g]);
        float sum = 0.f, v = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float keep = af_keep(part_m[w][g], top);
            sum = fmaf(part_l[w][g], keep, sum);
            v = fmaf(part_o[w][g][c], keep, v);
        }
        range_o[g][c] = v;
        if (c == 0) {
            range_m[g] = top;
            range_l[g] = sum;
        }
    }
    auto sync = [&]() {
        if (ranks > 1)
            af_cluster_sync();
        else
            __syncthreads();
    };
    sync();
    for (int i = rank * 128 + tid; i < heads * D; i += ranks * 128) {
        const int g = i / D, c = i % D;
        float pm[8], pl[8], po[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            pm[r] = -INFINITY;
            pl[r] = po[r] = 0.f;
            if (r < ranks) {
                pm[r] = af_peer(&range_m[g], r);
                pl[r] = af_peer(&range_l[g], r);
                po[r] = af_peer(&range_o[g][c], r);
            }
        }
        float top = p.sink ? p.sink[h0 + g] : -INFINITY;
        float sum = p.sink ? 1.f : 0.f, v = 0.f;
        const float own = top;
#pragma unroll
        for (int r = 0; r < 8; ++r)
            top = fmaxf(top, pm[r]);
        sum *= af_keep(own, top);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float keep = af_keep(pm[r], top);
            sum = fmaf(pl[r], keep, sum);
            v = fmaf(po[r], keep, v);
        }
        p.out[((size_t)row * p.nq + h0 + g) * D + c] = v * (sum > 0.f ? 1.f / sum : 0.f);
    }
    sync();                                             // nobody leaves while its sums are read
}

template <int D>
static int attention_f32(const AttentionF32& p, int seqs, int max_q_len, int min_q_len, int ranks, cudaStream_t stream)
{
    const int G = p.nq / p.nkv;
    if (max_q_len > 1) {
        // (a scale whose 2^-32th is no normal number goes the way of the other options)
        const bool options = p.softcap > 0.f || p.bias_r1 || fabsf(p.scale) < 0x1p-90f;
        const auto kernel = options ? attention_f32_prompt_kernel<D, true> : attention_f32_prompt_kernel<D, false>;
        static bool configured[2] = { false, false };
        if (!configured[options]) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AtShape<D>::SHARED);
            // (threads that asked for more registers than the block was launched with would wait for good)
            cudaFuncAttributes attr {};
            const cudaError_t a = e == cudaSuccess ? cudaFuncGetAttributes(&attr, kernel) : e;
            if (a != cudaSuccess)
                return (int)a;
            if (attr.numRegs < AT_REGS)
                return CHIBI_ERR_ARGUMENT;
            configured[options] = true;
        }
        const long long tiles = ((long long)max_q_len * G + AT_ROWS - 1) / AT_ROWS;
        if (tiles > 2147483647LL || (long long)p.num_pages * p.nkv * p.page_size > 2147483647LL)
            return CHIBI_ERR_UNSUPPORTED;
        launch(kernel, dim3((unsigned)tiles, p.nkv, seqs), dim3(AT_THREADS), AtShape<D>::SHARED, stream, p);
        if (const int status = launch_status())
            return status;
    }
    if (max_q_len == 1 || min_q_len <= 1) {
        const int blocks = G <= 1 ? 1 : G <= 2 ? 1 : (G + 3) / 4;
        const dim3 grid(ranks, p.nkv * blocks, seqs);
        if (G <= 1)
            launch_cluster_x(attention_f32_token_kernel<D, 1>, grid, dim3(128), 0, stream, ranks, p, ranks, blocks);
        else if (G <= 2)
            launch_cluster_x(attention_f32_token_kernel<D, 2>, grid, dim3(128), 0, stream, ranks, p, ranks, blocks);
        else
            launch_cluster_x(attention_f32_token_kernel<D, 4>, grid, dim3(128), 0, stream, ranks, p, ranks, blocks);
    }
    return launch_status();
}

} // namespace chibi

using namespace chibi;

// Which of its two kernels run: one for sequences of several tokens if max_q_len > 1, one for single tokens if
// min_q_len <= 1 (0: not known).  ranks (1, 2, 4 or 8): CTAs that share a single token's keys; fewer than its ranges take
// several each.
CHIBI_API int chibi_attention_f32(const float* q, const float* k_cache, const float* v_cache, float* out,
                                  const int* block_table, int table_stride, const int* q_start, const int* ctx_len,
                                  const int* seq_rows, int seqs, int nq, int nkv, int d, int page_size, int num_pages,
                                  float scale, int window, int chunk, int max_q_len, int min_q_len, int ranks,
                                  float softcap, const float* bias_r1, const float* bias_r2, const float* sink, int* error,
                                  cudaStream_t stream)
{
    if (seqs <= 0 || max_q_len <= 0)
        return CHIBI_OK;
    // (pieces of 16 bytes; the grid's limits)
    if ((d != 64 && d != 128) || nkv <= 0 || nq % nkv != 0 || window < 0 || chunk < 0 || softcap < 0.f || page_size <= 0
        || (bias_r2 != nullptr && bias_r1 == nullptr) || seqs > 65535 || (ranks != 1 && ranks != 2 && ranks != 4 && ranks != 8) || nq > 65535
        || ((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) % 16 != 0)
        return CHIBI_ERR_UNSUPPORTED;
    const AttentionF32 p = { q, k_cache, v_cache, out, block_table, table_stride, q_start, ctx_len, seq_rows, nq, nkv,
                             page_size, num_pages, scale, window, chunk, softcap, bias_r1, bias_r2, sink, error };
    return d == 64 ? attention_f32<64>(p, seqs, max_q_len, min_q_len, ranks, stream)
                   : attention_f32<128>(p, seqs, max_q_len, min_q_len, ranks, stream);
}
