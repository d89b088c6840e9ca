// Causal grouped-query attention over the block cache, for any key size and any value size
// up to 256 (the two may differ), in float32 or bfloat16 storage with float32 arithmetic,
// optionally with a per-head sink term in the softmax denominator, capped scores, a bias that grows with the
// distance between query and key (a slope per head), and a sigmoid gate on the output (see AttnExtra).
// Prompts with heads of up to 128 numbers go in tiles of 32 queries (below).  One kernel serves everything else: a warp owns one (token, query head, split)
// and walks that token's visible keys 32 at a time with a running softmax; with more
// than one split the partial (max, sum, accumulator) triples are merged by a second
// kernel.  This is the exact path (every product and sum in float32 FMA) and the
// fallback of the tensor-core kernels for head sizes they do not take.
//
// Counterparts in random-unknown-username/Thintensor: _single_token_gqa_attention_kernel
// thinruntime/triton_kernels.py:14-109 and the split pair
// _split_gqa_attention_partial_kernel / _reduce_kernel thinruntime/triton_kernels.py:112-245
// (one token, one sequence); the formula is thinruntime/gpu_runtime.py:8913-8961.
#include "attention_kernels.cuh"

template <bool VALUE> struct AtBool { static constexpr bool value = VALUE; };

// Prompts: a CTA takes 32 queries of one sequence and head and walks the cache blocks they see, 64 keys at a time, with both
// products as tiles in registers (4 x 4 scores, 4 x SIZE / 16 outputs a thread) from operands staged in shared memory, so that a key
// or a value is fetched for 32 queries instead of one and read from shared memory for four.  Scores, the running softmax and the
// sums are float32 as in the kernel that takes a query a warp; that one was bound by its reads of the values, 32 cache lines an
// instruction.  A row's arithmetic does not depend on which queries share its tile.  193 tokens of 32 heads of 64, float32: 226 -> 41 us.
// SIZE: key and value heads of up to so many numbers (64 or 128).
constexpr int AT_QUERIES = 32, AT_THREADS = 128, AT_PLD = TT_BLOCK_TOKENS + 4;

template <int SIZE>
constexpr size_t at_shared() { return (size_t)((AT_QUERIES + TT_BLOCK_TOKENS) * (SIZE + 4) + (SIZE + AT_QUERIES) * AT_PLD) * sizeof(float); }

template <typename T, int SIZE>
__global__ void __launch_bounds__(AT_THREADS)
attention_tiles_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool, const int* __restrict__ table, int table_width,
                       int pool_blocks, const int* __restrict__ cu, const int* __restrict__ len_before, int sequences, int heads, int kv_heads, int head_dim,
                       int value_dim, float scale, const float* __restrict__ sinks, int window, T* __restrict__ out, unsigned* status, AttnExtra extra) {
    constexpr int LD = SIZE + 4, DIMS = SIZE / 16;
    extern __shared__ __align__(16) float at_shared_memory[];
    float* Qs = at_shared_memory;                               // [32][LD], times scale
    float* Ks = Qs + AT_QUERIES * LD;                           // [64][LD]
    float* Vs = Ks + TT_BLOCK_TOKENS * LD;                      // [SIZE][AT_PLD]
    float* Ps = Vs + SIZE * AT_PLD;                             // [32][AT_PLD]
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    // tiles of a sequence: slots from cu[b] / 32 + b on, room for all of them before the next sequence's first
    const int slot = blockIdx.x, h = blockIdx.y, kh = h / (heads / kv_heads);
    int lo = 0, hi = sequences;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cu[mid] / AT_QUERIES + mid <= slot) lo = mid; else hi = mid;
    }
    const int first = cu[lo], i0 = (slot - (first / AT_QUERIES + lo)) * AT_QUERIES, count = min(AT_QUERIES, cu[lo + 1] - first - i0);
    if (count <= 0) return;
    const int pos0 = len_before[lo] + i0;                       // position of the tile's first query
    const int* table_row = table + (size_t)lo * table_width;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;

    for (int e = threadIdx.x; e < AT_QUERIES * SIZE; e += AT_THREADS) {
        const int r = e / SIZE, d = e % SIZE;
        Qs[r * LD + d] = r < count && d < head_dim ? tt_to_float(q[((size_t)(first + i0 + r) * heads + h) * head_dim + d]) * scale : 0.0f;
    }
    const float slope = extra.slopes ? __ldg(extra.slopes + h) : 0.0f;
    const float cap = extra.softcap, inv_cap = cap > 0.0f ? 1.0f / cap : 0.0f;
    float m[4], l[4], acc[4][DIMS];
    int seen_from[4], pos[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = ty + 8 * r;
        pos[r] = i < count ? pos0 + i : -1;                     // rows that do not exist see nothing
        seen_from[r] = i < count ? tt_first_key(pos[r], window) : 0;
        m[r] = sinks ? __ldg(sinks + h) : -INFINITY;
        l[r] = sinks ? 1.0f : 0.0f;
#pragma unroll
        for (int d = 0; d < DIMS; ++d) acc[r][d] = 0.0f;
    }
    const int from = tt_first_key(pos0, window), last = pos0 + count - 1;
    constexpr int N = Vec16<T>::N;                              // numbers of a 16-byte piece
    const bool vec = head_dim % N == 0;
    for (int block = from / TT_BLOCK_TOKENS; block <= last / TT_BLOCK_TOKENS; ++block) {
        const int base = block * TT_BLOCK_TOKENS, id = table_row[block];
        if (id < 0 || id >= pool_blocks) {                      // every thread sees the same
            if (threadIdx.x == 0 && status) atomicOr(status, TT_STATUS_BAD_BLOCK);
            continue;
        }
        const T* kb = k_pool + ((size_t)id * kv_heads + kh) * TT_BLOCK_TOKENS * head_dim;
        const T* vb = v_pool + ((size_t)id * kv_heads + kh) * TT_BLOCK_TOKENS * value_dim;
        __syncthreads();                                        // the last block's operands are read
        constexpr int KP = SIZE / N, VP = TT_BLOCK_TOKENS / N;
        for (int e = threadIdx.x; e < TT_BLOCK_TOKENS * KP; e += AT_THREADS) {
            const int j = e / KP, d = (e % KP) * N;
            const bool live = base + j >= from && base + j <= last;
            float x[N];
            if (vec && live && d < head_dim) {
                const uint4 raw = *reinterpret_cast<const uint4*>(kb + (size_t)j * head_dim + d);
                const T* p = reinterpret_cast<const T*>(&raw);
#pragma unroll
                for (int i = 0; i < N; ++i) x[i] = tt_to_float(p[i]);
            } else {
#pragma unroll
                for (int i = 0; i < N; ++i) x[i] = live && d + i < head_dim ? tt_to_float(kb[(size_t)j * head_dim + d + i]) : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(Ks + j * LD + d + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
        }
        for (int e = threadIdx.x; e < SIZE * VP; e += AT_THREADS) {
            const int d = e / VP, j = (e % VP) * N;
            float x[N];
            if (d < value_dim && base + j + N > from && base + j <= last) {
                const uint4 raw = *reinterpret_cast<const uint4*>(vb + (size_t)d * TT_BLOCK_TOKENS + j);
                const T* p = reinterpret_cast<const T*>(&raw);
#pragma unroll
                for (int i = 0; i < N; ++i) x[i] = base + j + i >= from && base + j + i <= last ? tt_to_float(p[i]) : 0.0f;      // other places may hold anything
            } else {
#pragma unroll
                for (int i = 0; i < N; ++i) x[i] = 0.0f;
            }
#pragma unroll
            for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(Vs + d * AT_PLD + j + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
        }
        __syncthreads();
        float s[4][4], s2[4][4];                                // two sums a score, added up: a long chain of additions loses more
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[r][c] = s2[r][c] = 0.0f;
#pragma unroll 4
        for (int d = 0; d < SIZE; d += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(Qs + (ty + 8 * r) * LD + d);
#pragma unroll
            for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * c) * LD + d);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[r][c] = fmaf(a[r].x, b[c].x, s[r][c]);
                    s[r][c] = fmaf(a[r].y, b[c].y, s[r][c]);
                    s2[r][c] = fmaf(a[r].z, b[c].z, s2[r][c]);
                    s2[r][c] = fmaf(a[r].w, b[c].w, s2[r][c]);
                }
        }
        bool whole = true;                                      // the warp's queries see every key of the block
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float top = -INFINITY;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int key = base + tx + 16 * c;
                float v = s[r][c] + s2[r][c];
                if (cap > 0.0f) v = cap * tanhf(v * inv_cap);
                v -= slope * (float)(pos[r] - key);
                const bool seen = key >= seen_from[r] && key <= pos[r];
                whole = whole && seen;
                s[r][c] = seen ? v : -INFINITY;
                top = fmaxf(top, s[r][c]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m[r], top);
            const float corr = m_new == -INFINITY ? 1.0f : expf(m[r] - m_new);
            float sum = 0.0f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[r][c] = s[r][c] == -INFINITY ? 0.0f : expf(s[r][c] - m_new);
                sum += s[r][c];
                Ps[(ty + 8 * r) * AT_PLD + tx + 16 * c] = s[r][c];
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l[r] = l[r] * corr + sum;
            m[r] = m_new;
#pragma unroll
            for (int d = 0; d < DIMS; ++d) acc[r][d] *= corr;
        }
        whole = __all_sync(0xffffffffu, whole);                 // a warp's rows and weights are its own
        __syncwarp();
        auto weigh = [&](auto guarded) {                        // the block's sums, then added to the running ones
            float part[4][DIMS];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int d = 0; d < DIMS; ++d) part[r][d] = 0.0f;
#pragma unroll 2
            for (int j = 0; j < TT_BLOCK_TOKENS; j += 4) {
                float4 p[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) p[r] = *reinterpret_cast<const float4*>(Ps + (ty + 8 * r) * AT_PLD + j);
#pragma unroll
                for (int d = 0; d < DIMS; ++d) {
                    const float4 v = *reinterpret_cast<const float4*>(Vs + (tx + 16 * d) * AT_PLD + j);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        // a weight of zero does not touch its value: what a query does not see may be no number
                        if (!decltype(guarded)::value || p[r].x != 0.0f) part[r][d] = fmaf(p[r].x, v.x, part[r][d]);
                        if (!decltype(guarded)::value || p[r].y != 0.0f) part[r][d] = fmaf(p[r].y, v.y, part[r][d]);
                        if (!decltype(guarded)::value || p[r].z != 0.0f) part[r][d] = fmaf(p[r].z, v.z, part[r][d]);
                        if (!decltype(guarded)::value || p[r].w != 0.0f) part[r][d] = fmaf(p[r].w, v.w, part[r][d]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int d = 0; d < DIMS; ++d) acc[r][d] += part[r][d];
        };
        if (whole) weigh(AtBool<false>()); else weigh(AtBool<true>());
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = ty + 8 * r, t = first + i0 + i;
        if (i >= count) continue;
        const float inv = l[r] > 0.0f ? 1.0f / l[r] : 0.0f;
#pragma unroll
        for (int d = 0; d < DIMS; ++d) {
            const int c = tx + 16 * d;
            if (c >= value_dim) continue;
            float o = acc[r][d] * inv;
            if (extra.gate) o *= attn_gate(extra, t, h, value_dim, c);
            out[((size_t)t * heads + h) * value_dim + c] = tt_from_float<T>(o);
        }
    }
}

template <typename T, int SIZE>
static int attention_tiles_launch(const void* q, const void* k_pool, const void* v_pool, const int* table, int table_width, int pool_blocks, const int* cu,
                                  const int* len_before, int sequences, int n_tokens, int heads, int kv_heads, int head_dim, int value_dim, float scale,
                                  const float* sinks, int window, void* out, unsigned* status, const AttnExtra& extra, cudaStream_t stream) {
    const cudaError_t code = tt_allow_shared(attention_tiles_kernel<T, SIZE>, at_shared<SIZE>());
    if (code != cudaSuccess) return (int)code;
    tt_launch_pdl(attention_tiles_kernel<T, SIZE>, dim3((unsigned)(n_tokens / AT_QUERIES + sequences), (unsigned)heads), dim3(AT_THREADS), at_shared<SIZE>(), stream,
                  (const T*)q, (const T*)k_pool, (const T*)v_pool, table, table_width, pool_blocks, cu, len_before, sequences, heads, kv_heads, head_dim, value_dim,
                  scale, sinks, window, (T*)out, status, extra);
    TT_LAUNCH_CHECK();
}

// Whether a step's queries go in tiles: prompts (eight tokens a sequence on average fill a quarter of a tile, which already pays), heads of up to
// 128 numbers, the cache on 16-byte boundaries.  Where the block table is one block wide, a query meets so few keys that tiles have to be full, or a
// query a warp has to keep the SMs busy, for tiles to be faster.  Measured without a past, a query a warp against tiles (us, heads of 64): one prompt of 16 tokens, 32
// heads 9.0 and 10.8, of 24 10.9 and 10.2, of 40 24 and 13; 8 prompts of 16 17 and 14; 16 of 8 24 and 28, of 12 42 and 30; one of 32 tokens, 8 heads 12.3 and 13.1.
static bool attention_in_tiles(const void* k_pool, const void* v_pool, int table_width, int sequences, int n_tokens, int heads, int head_dim, int value_dim, int splits) {
    const long long warps = (long long)n_tokens * heads;
    const bool enough = table_width > 1 ? n_tokens >= 8 * sequences : n_tokens >= 40 * sequences || (n_tokens >= 24 * sequences && warps >= 1024)
        || (n_tokens >= 16 * sequences && warps >= 2048) || (n_tokens >= 12 * sequences && warps >= 6144);
    return splits == 1 && enough && head_dim <= 128 && value_dim <= 128 && heads <= 65535
        && (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0;
}

// part_acc: float32 [tokens * heads * splits * value_dim], part_ml: float32
// [tokens * heads * splits * 2]; both may be null when splits == 1.
extern "C" int tt_attention(const void* q, const void* k_pool, const void* v_pool, int dtype, const int* table,
                            int table_width, int pool_blocks, const int* cu, const int* len_before, int sequences,
                            int n_tokens, int heads, int kv_heads, int head_dim, int value_dim, float scale, const float* sinks,
                            int window, int splits, void* out, float* part_acc, float* part_ml, unsigned* status,
                            float softcap, const float* slopes, const float* gate, int gate_splits, long long gate_split_stride,
                            int gate_row, int gate_per_head, cudaStream_t stream) {
    const AttnExtra extra{softcap, slopes, gate, gate_splits, gate_split_stride, gate_row, gate_per_head};
    if (n_tokens <= 0) return 0;
    if (head_dim <= 0 || head_dim > ATTN_MAX_HEAD_DIM || value_dim <= 0 || value_dim > ATTN_MAX_HEAD_DIM || heads % kv_heads || splits < 1 || splits > 65535)
        return (int)cudaErrorInvalidValue;
    if (splits > 1 && (!part_acc || !part_ml)) return (int)cudaErrorInvalidValue;
    if (attention_in_tiles(k_pool, v_pool, table_width, sequences, n_tokens, heads, head_dim, value_dim, splits)) {
#define TT_TILES(T, SIZE) attention_tiles_launch<T, SIZE>(q, k_pool, v_pool, table, table_width, pool_blocks, cu, len_before, sequences, n_tokens, heads, kv_heads, head_dim, value_dim, scale, sinks, window, out, status, extra, stream)
        const bool small = head_dim <= 64 && value_dim <= 64;
        if (dtype == TT_F32) return small ? TT_TILES(float, 64) : TT_TILES(float, 128);
        return small ? TT_TILES(__nv_bfloat16, 64) : TT_TILES(__nv_bfloat16, 128);
#undef TT_TILES
    }
    const long long rows = (long long)n_tokens * heads;
    const dim3 grid((unsigned)((rows + ATTN_WARPS - 1) / ATTN_WARPS), (unsigned)splits);
    const size_t shared = (size_t)ATTN_WARPS * head_dim * sizeof(float);
    if (dtype == TT_F32) {
        attention_rows_kernel<float><<<grid, ATTN_WARPS * 32, shared, stream>>>((const float*)q, (const float*)k_pool, (const float*)v_pool, table, table_width, pool_blocks, cu, len_before, sequences, n_tokens, heads, kv_heads, head_dim, value_dim, scale, sinks, window, splits, (float*)out, part_acc, part_ml, status, extra);
        if (splits > 1)
            attention_merge_kernel<float><<<grid.x, ATTN_WARPS * 32, 0, stream>>>(part_acc, part_ml, splits, value_dim, rows, (float*)out, extra, heads);
    } else {
        attention_rows_kernel<__nv_bfloat16><<<grid, ATTN_WARPS * 32, shared, stream>>>((const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, table, table_width, pool_blocks, cu, len_before, sequences, n_tokens, heads, kv_heads, head_dim, value_dim, scale, sinks, window, splits, (__nv_bfloat16*)out, part_acc, part_ml, status, extra);
        if (splits > 1)
            attention_merge_kernel<__nv_bfloat16><<<grid.x, ATTN_WARPS * 32, 0, stream>>>(part_acc, part_ml, splits, value_dim, rows, (__nv_bfloat16*)out, extra, heads);
    }
    TT_LAUNCH_CHECK();
}
