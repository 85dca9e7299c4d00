// Causal grouped-query attention of the 32-bit path over the paged cache, head sizes 64 and 128: all operands and
// results 32-bit, scores and sums by 32-bit multiply-adds (attention_generic.cu says what is computed and which options
// the scores have; it takes the other sizes and types).  Two kernels, one for the sequences that bring one token to a step
// and one for those that bring more.  In both, the order of a row's operations depends on its own position (and on
// whether it came alone), never on the batch around it.
#define CHIBI_UNIT attention_f32
#define CHIBI_UNIT_ID 17
#include "common.cuh"

namespace chibi {

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

__device__ __forceinline__ uint64_t af_pair(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 af_halves(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t af_fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t af_mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// 16 bytes, zeros where `bytes` is 0 (nothing is read then).
__device__ __forceinline__ void af_copy16(float* dst, const float* src, int bytes)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

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
__device__ __forceinline__ float4 af_peer4(const float* local, int rank)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(af_peer_address(local, rank)) : "memory");
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
// grid (4 CTAs for each row tile, kv heads, sequences), 128 threads.  A tile is 64 rows, the group's heads of
// neighbouring tokens; the keys are taken 32 at a time, from a multiple of 32 on, and blocks of 64 keys (counted from the
// sequence's start) go to the four CTAs of a cluster in turn, which add up what they found at the end: a causal
// tile's keys spread evenly, and few rows make four times the CTAs (three prompts of up to 400 tokens of 16 heads:
// 137 us with one CTA a tile).  A thread owns rows ty + 16 i; of the scores
// the keys tx + 8 j, of the output the columns 4 tx + 32 j .. + 3, so a row's eight threads sit side by side in a warp:
// its maximum and sum are three shuffles, and its probabilities reach them through shared memory without a block
// barrier.  The next keys are fetched while the values are used and the other way round.  Scores take two
// neighbouring features at a time (fma.rn.f32x2), the output two neighbouring columns.  Bound by the reads of
// shared memory beside the multiply-adds (8 reads of 16 bytes, 32 cycles, to 16 cycles of multiply-adds for the
// scores; 80 to 64 for the output); 76 KB a CTA, three to an SM.
constexpr int AF_ROWS = 64, AF_KEYS = 32, AF_P = AF_KEYS + 4, AF_RANKS = 4, AF_BLOCK = 64;

template <int D> constexpr size_t af_shared()
{
    return sizeof(float) * (AF_ROWS * (D + 4) + AF_KEYS * (D + 4) + AF_KEYS * D + AF_ROWS * AF_P);
}

template <int D>
__global__ void __launch_bounds__(128, 3)
attention_f32_prompt_kernel(const AttentionF32 p)
{
    pdl_enter();
    constexpr int DS = D + 4, QUADS = D / 4, CJ = D / 32;
    extern __shared__ __align__(16) float af_sm[];
    float* const Q = af_sm;                             // [AF_ROWS][DS]
    float* const K = Q + AF_ROWS * DS;                  // [AF_KEYS][DS]
    float* const V = K + AF_KEYS * DS;                  // [AF_KEYS][D]
    float* const P = V + AF_KEYS * D;                   // [AF_ROWS][AF_P]
    const int tid = threadIdx.x, lane = tid & 31, tx = tid & 7, ty = tid >> 3;
    const int seq = blockIdx.z, kv_head = blockIdx.y, G = p.nq / p.nkv;
    const int row0 = p.q_start[seq], q_len = p.q_start[seq + 1] - row0;
    if (q_len <= 1)
        return;                                         // (a single token is the other kernel's)
    const int all_rows = q_len * G, tiles = (all_rows + AF_ROWS - 1) / AF_ROWS;
    const int pos0 = p.ctx_len[seq] - q_len;            // the first token's position
    const int* const table = p.block_table + (size_t)(p.seq_rows ? p.seq_rows[seq] : seq) * p.table_stride;

    const int rank = blockIdx.x % AF_RANKS;
    float* const ml = P;                                // at the end: [AF_ROWS] maxima, [AF_ROWS] sums
    float* const part = K;                              // and, over keys and values, [AF_ROWS][D] sums

    // the tiles with the most keys first
    for (int tile = tiles - 1 - (int)blockIdx.x / AF_RANKS; tile >= 0; tile -= gridDim.x / AF_RANKS) {
        const int first_row = tile * AF_ROWS, last_row = min(first_row + AF_ROWS, all_rows) - 1;
        const int last_pos = pos0 + last_row / G;
        const int oldest = first_visible_key(pos0 + first_row / G, p.window, p.chunk);      // (older pages may be gone)
        const int visible = oldest & ~(AF_KEYS - 1);
        // this CTA's blocks: those whose number is rank modulo AF_RANKS
        const int block = visible / AF_BLOCK, mine = block + (rank + AF_RANKS - block % AF_RANKS) % AF_RANKS;
        const int begin = mine == block ? visible : mine * AF_BLOCK;
        auto after = [&](int base) {
            const int next = base + AF_KEYS;
            return next % AF_BLOCK ? next : next + (AF_RANKS - 1) * AF_BLOCK;
        };
        __syncthreads();                                // (the tile before is through)
        for (int c = tid; c < AF_ROWS * QUADS; c += 128) {
            const int r = c / QUADS, at = 4 * (c % QUADS), row = first_row + r;
            const bool there = row < all_rows;
            af_copy16(Q + r * DS + at,
                      there ? p.q + ((size_t)(row0 + row / G) * p.nq + kv_head * G + row % G) * D + at : p.q, there ? 16 : 0);
        }
        // rows of keys or values: lane l looks the page of key l up, a row is copied by QUADS threads
        unsigned usable = 0;                            // keys of the tile whose page is one of the pool's
        auto fetch = [&](const float* cache, float* dst, int stride, int base) {
            const int u = base + lane;
            long long at = -1;
            if (u >= oldest && u <= last_pos) {
                const int page = table[u / p.page_size];
                if (page < 0 || page >= p.num_pages) {
                    if (p.error)
                        atomicExch(p.error, 3);
                } else {
                    at = (((long long)page * p.nkv + kv_head) * p.page_size + u % p.page_size) * D;
                }
            }
#pragma unroll
            for (int i = 0; i < AF_KEYS * QUADS / 128; ++i) {
                const int c = tid + 128 * i, r = c / QUADS, x = 4 * (c % QUADS);
                const long long from = __shfl_sync(0xffffffffu, at, r);
                af_copy16(dst + r * stride + x, from >= 0 ? cache + from + x : cache, from >= 0 ? 16 : 0);
            }
            af_commit();
            return __ballot_sync(0xffffffffu, at >= 0);
        };

        int pos[4];
        float r1[4], r2[4], m[4], l[4];
        uint64_t O[4][CJ][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = min(first_row + ty + 16 * i, all_rows - 1), h = kv_head * G + row % G;
            pos[i] = pos0 + row / G;
            r1[i] = p.bias_r1 ? p.bias_r1[h] : 0.f;
            r2[i] = p.bias_r2 ? p.bias_r2[h] : 0.f;
            m[i] = -INFINITY;
            l[i] = 0.f;
#pragma unroll
            for (int j = 0; j < CJ; ++j)
                O[i][j][0] = O[i][j][1] = 0;
        }
        usable = fetch(p.k_cache, K, DS, begin);        // (one group with the queries)
        for (int base = begin; base <= last_pos; base = after(base)) {
            const unsigned keys = usable;
            af_wait<0>();
            __syncthreads();                            // the keys are there; everyone is through with the values before
            fetch(p.v_cache, V, D, base);
            uint64_t S[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    S[i][j] = 0;
#pragma unroll 4
            for (int c = 0; c < D; c += 4) {
                ulonglong2 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    a[i] = *reinterpret_cast<const ulonglong2*>(Q + (ty + 16 * i) * DS + c);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(K + (tx + 8 * j) * DS + c);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        S[i][j] = af_fma2(a[i].x, b.x, S[i][j]);
                        S[i][j] = af_fma2(a[i].y, b.y, S[i][j]);
                    }
                }
            }
            // every row sees every key of this tile?
            const bool whole = base + AF_KEYS - 1 <= pos0 + first_row / G && keys == 0xffffffffu
                && base >= first_visible_key(last_pos, p.window, p.chunk);
            int low[4], high[4];                        // the keys of the tile that a row sees
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                low[i] = whole ? 0 : max(first_visible_key(pos[i], p.window, p.chunk) - base, 0);
                high[i] = whole ? AF_KEYS - 1 : min(pos[i] - base, AF_KEYS - 1);
                float s[4], most = -INFINITY;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int kk = tx + 8 * j;
                    const float2 halves = af_halves(S[i][j]);
                    s[j] = af_score(p, halves.x + halves.y, r1[i], r2[i], pos[i] - base - kk);
                    if (kk < low[i] || kk > high[i] || !(keys >> kk & 1))
                        s[j] = -INFINITY;
                    most = fmaxf(most, s[j]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
                    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                const float m_new = fmaxf(m[i], most);
                const float keep = af_keep(m[i], m_new);
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float e = s[j] == -INFINITY ? 0.f : expf(s[j] - m_new);
                    P[(ty + 16 * i) * AF_P + tx + 8 * j] = e;
                    sum += e;
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
                    sum += __shfl_xor_sync(0xffffffffu, sum, o);
                l[i] = l[i] * keep + sum;
                m[i] = m_new;
                const uint64_t k2 = af_pair(keep, keep);
#pragma unroll
                for (int j = 0; j < CJ; ++j) {
                    O[i][j][0] = af_mul2(O[i][j][0], k2);
                    O[i][j][1] = af_mul2(O[i][j][1], k2);
                }
            }
            af_wait<0>();
            __syncthreads();                            // the values are there (and the row's probabilities)
            if (after(base) <= last_pos)
                usable = fetch(p.k_cache, K, DS, after(base));
            auto values = [&](bool all) {
#pragma unroll 2
                for (int kk = 0; kk < AF_KEYS; kk += 4) {
                    float4 e[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        e[i] = *reinterpret_cast<const float4*>(P + (ty + 16 * i) * AF_P + kk);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        ulonglong2 v[CJ];
#pragma unroll
                        for (int j = 0; j < CJ; ++j)
                            v[j] = *reinterpret_cast<const ulonglong2*>(V + (kk + u) * D + 4 * tx + 32 * j);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float w = u == 0 ? e[i].x : u == 1 ? e[i].y : u == 2 ? e[i].z : e[i].w;
                            const uint64_t w2 = af_pair(w, w);
                            // (a key that the row does not see adds nothing, whatever its value holds)
                            if (all || (kk + u >= low[i] && kk + u <= high[i])) {
#pragma unroll
                                for (int j = 0; j < CJ; ++j) {
                                    O[i][j][0] = af_fma2(w2, v[j].x, O[i][j][0]);
                                    O[i][j][1] = af_fma2(w2, v[j].y, O[i][j][1]);
                                }
                            }
                        }
                    }
                }
            };
            if (whole)
                values(true);
            else
                values(false);
        }
        af_wait<0>();
        __syncthreads();                                // keys and values are through: their place takes the sums
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty + 16 * i;
#pragma unroll
            for (int j = 0; j < CJ; ++j)
                *reinterpret_cast<ulonglong2*>(part + r * D + 4 * tx + 32 * j) = make_ulonglong2(O[i][j][0], O[i][j][1]);
            if (tx == 0) {
                ml[r] = m[i];
                ml[AF_ROWS + r] = l[i];
            }
        }
        af_cluster_sync();
        // each CTA finishes a quarter of the rows
        constexpr int OWN = AF_ROWS / AF_RANKS;
        for (int c = tid; c < OWN * QUADS; c += 128) {
            const int r = rank * OWN + c / QUADS, at = 4 * (c % QUADS), row = first_row + r;
            if (row >= all_rows)
                continue;
            float pm[AF_RANKS], pl[AF_RANKS];
            float4 po[AF_RANKS];
#pragma unroll
            for (int x = 0; x < AF_RANKS; ++x) {
                pm[x] = af_peer(ml + r, x);
                pl[x] = af_peer(ml + AF_ROWS + r, x);
                po[x] = af_peer4(part + r * D + at, x);
            }
            const int h = kv_head * G + row % G;
            const float sink = p.sink ? p.sink[h] : -INFINITY;
            float top = sink;
#pragma unroll
            for (int x = 0; x < AF_RANKS; ++x)
                top = fmaxf(top, pm[x]);
            float sum = p.sink ? af_keep(sink, top) : 0.f;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int x = 0; x < AF_RANKS; ++x) {
                const float keep = af_keep(pm[x], top);
                sum = fmaf(pl[x], keep, sum);           // (a CTA without a key for the row has zeros)
                v.x = fmaf(po[x].x, keep, v.x);
                v.y = fmaf(po[x].y, keep, v.y);
                v.z = fmaf(po[x].z, keep, v.z);
                v.w = fmaf(po[x].w, keep, v.w);
            }
            const float inv = sum > 0.f ? 1.f / sum : 0.f;
            *reinterpret_cast<float4*>(p.out + ((size_t)(row0 + row / G) * p.nq + h) * D + at) =
                make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv);
        }
        af_cluster_sync();                              // nobody goes on while its sums are read
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
                    d0 = af_fma2(q[g][i][0], k[i].x, d0);
                    d1 = af_fma2(q[g][i][1], k[i].y, d1);
                }
                const float2 a = af_halves(d0), b = af_halves(d1);
                float dot = (a.x + a.y) + (b.x + b.y);
#pragma unroll
                for (int x = 4; x > 0; x >>= 1)
                    dot += __shfl_xor_sync(0xffffffffu, dot, x);
                if (here >= 0) {
                    const float s = af_score(p, dot, r1[g], r2[g], pos - u);
                    const float m_new = fmaxf(m[g], s);
                    const float keep = af_keep(m[g], m_new), e = s == -INFINITY ? 0.f : expf(s - m_new);
                    const uint64_t k2 = af_pair(keep, keep), e2 = af_pair(e, e);
                    l[g] = l[g] * keep + e;
                    m[g] = m_new;
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        o[g][i][0] = af_fma2(e2, v[i].x, af_mul2(o[g][i][0], k2));
                        o[g][i][1] = af_fma2(e2, v[i].y, af_mul2(o[g][i][1], k2));
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
                float2 a = af_halves(o[g][i][x]);
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
        static bool configured = false;
        if (!configured) {
            const cudaError_t e = cudaFuncSetAttribute(attention_f32_prompt_kernel<D>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)af_shared<D>());
            if (e != cudaSuccess)
                return (int)e;
            configured = true;
        }
        const long long tiles = ((long long)max_q_len * G + AF_ROWS - 1) / AF_ROWS;
        if (tiles * AF_RANKS > 2147483647LL)
            return CHIBI_ERR_UNSUPPORTED;
        launch_cluster_x(attention_f32_prompt_kernel<D>, dim3((unsigned)tiles * AF_RANKS, p.nkv, seqs), dim3(128), af_shared<D>(),
                         stream, AF_RANKS, p);
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
