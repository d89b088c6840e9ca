// Routing of a mixture of experts.
//
// tt_route_topk: one warp per token.  Scores are the softmax of the router's logits over all experts (float32).
// Experts form `groups` equal groups of neighbours; a group's score is its largest expert score, and only experts of
// the `keep` groups with the largest scores can be chosen.  Of those the `top` largest are chosen (ties: the lower
// index), and their weights are their scores divided by the sum of the chosen scores (+ 1e-20).  The kernel writes
// the chosen experts and weights ([tokens][top]) and the same as a dense table ([tokens][experts], zero where an
// expert is not chosen).
//
// Options (RouteOptions): sigmoid scores instead of the softmax, a correction added for the choice only, groups scored by
// their two best, weights left as the scores, and gates of always-on experts from further rows of the router's matrix.
//
// tt_route_rows: the same with the router's product in front, from the token's row and the router's matrix.
//
// tt_expert_activation: the clamped gated unit of every expert's columns times the token's gate for that expert.
//
// tt_expert_unary_activation: the same for experts without a gate projection.
//
// tt_scale_expert_columns: act[t][e * width + j] *= gates[t][e] for the first experts * width columns of act; the next
// shared_width columns (an always-on expert's) are multiplied by gates[t][experts], and columns behind those stay as they are.
#include "common.cuh"

constexpr int ROUTE_MAX_EXPERTS = 512;      // a lane holds ROUTE_MAX_EXPERTS / 32 scores
constexpr int ROUTE_WARPS = 4;

// the largest value among the lanes' candidates and the lowest index that has it
__device__ __forceinline__ void route_argmax(float& value, int& index) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, value, o);
        const int i = __shfl_xor_sync(0xffffffffu, index, o);
        if (v > value || (v == value && i < index)) { value = v; index = i; }
    }
}

// How the scores are made and used (all zero: softmax scores, a group scored by its best expert, weights renormalised).
//   sigmoid: scores are sigmoid(logit) instead of the softmax over all experts.
//   correction (float32 [experts] or null): added to the scores for the CHOICE only (groups and top); weights use the scores.
//   group_top2: a group's score is the sum of its two largest choice scores (its only one, for groups of one expert).
//   plain_weights: the weights are the chosen scores themselves instead of score / (sum of the chosen + 1e-20).
//   weight_scale: a factor on the weights, however they are made (not on the always-on experts' gates).
//   extra: so many more logits follow the experts'; gates[t][experts + k] = sigmoid(logit) for each (the gate of an
//   expert that every token uses).  A row of `gates` has experts + extra numbers.
struct RouteOptions {
    int sigmoid;
    const float* correction;
    int group_top2;
    int plain_weights;
    int extra;
    float weight_scale;
};

// One warp routes token t from its logits (`splits` partial sums `split_stride` apart); group_best: 32 floats of the warp's own.
__device__ __forceinline__ void route_token(const float* __restrict__ logits, int splits, size_t split_stride, int t, int experts,
                                            int top, int groups, int keep, float* __restrict__ gates, int* __restrict__ chosen,
                                            float* __restrict__ weights, float* group_best_row, const RouteOptions opt) {
    const int lane = threadIdx.x & 31;
    constexpr int PER = ROUTE_MAX_EXPERTS / 32;
    float s[PER];                                               // score of expert lane + 32 * i
    float c[PER];                                               // its choice score; -inf: cannot be chosen (any more)
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int e = lane + 32 * i;
        s[i] = -INFINITY;
        if (e < experts) {
            float z = 0.0f;
            for (int k = 0; k < splits; ++k) z += logits[(size_t)k * split_stride + e];
            s[i] = z;
            m = fmaxf(m, z);
        }
    }
    if (opt.sigmoid) {
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (lane + 32 * i < experts) s[i] = 1.0f / (1.0f + expf(-s[i]));
    } else {
        m = tt_warp_max(m);
        float total = 0.0f;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (lane + 32 * i < experts) { s[i] = expf(s[i] - m); total += s[i]; }
        total = tt_warp_sum(total);
        const float inv = 1.0f / total;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (lane + 32 * i < experts) s[i] *= inv;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int e = lane + 32 * i;
        c[i] = e < experts ? s[i] + (opt.correction ? __ldg(opt.correction + e) : 0.0f) : -INFINITY;
    }
    const int row = experts + opt.extra;
    if (lane < opt.extra) {                                     // gates of the always-on experts
        float z = 0.0f;
        for (int k = 0; k < splits; ++k) z += logits[(size_t)k * split_stride + experts + lane];
        gates[(size_t)t * row + experts + lane] = 1.0f / (1.0f + expf(-z));
    }

    // groups: a bit per group that stays (groups <= 32)
    const int size = experts / groups;
    unsigned kept = 0xffffffffu;
    if (groups > 1 && keep < groups) {
        for (int g = 0; g < groups; ++g) {
            float best = -INFINITY;
            int where = 0x7fffffff;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int e = lane + 32 * i;
                if (e < experts && e / size == g && c[i] > best) { best = c[i]; where = e; }
            }
            route_argmax(best, where);
            if (opt.group_top2 && size > 1) {
                float second = -INFINITY;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int e = lane + 32 * i;
                    if (e < experts && e / size == g && e != where) second = fmaxf(second, c[i]);
                }
                best += tt_warp_max(second);
            }
            if (lane == 0) group_best_row[g] = best;
        }
        __syncwarp();
        kept = 0u;
        for (int round = 0; round < keep; ++round) {
            float v = (lane < groups && !((kept >> lane) & 1u)) ? group_best_row[lane] : -INFINITY;
            int g = (lane < groups && !((kept >> lane) & 1u)) ? lane : 0x7fffffff;
            route_argmax(v, g);
            if (g < groups) kept |= 1u << g;
        }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int e = lane + 32 * i;
        if (e < experts) gates[(size_t)t * row + e] = 0.0f;
        if (e < experts && !((kept >> (e / size)) & 1u)) c[i] = -INFINITY;
    }
    __syncwarp();

    float sum = 0.0f;
    int mine = -1;                                              // lane r keeps the r-th choice (top <= 32)
    float mine_score = 0.0f;
    for (int round = 0; round < top; ++round) {
        float v = -INFINITY;
        int e = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (c[i] > v) { v = c[i]; e = lane + 32 * i; }      // a lane's experts rise with i: the first largest is the lowest
        route_argmax(v, e);
        if (e == 0x7fffffff) break;                             // fewer allowed experts than top
        float score = 0.0f;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (lane + 32 * i == e) { score = s[i]; c[i] = -INFINITY; }
        score = __shfl_sync(0xffffffffu, score, e & 31);
        sum += score;
        if (lane == round) { mine = e; mine_score = score; }
    }
    const float scale = opt.weight_scale * (opt.plain_weights ? 1.0f : 1.0f / (sum + 1e-20f));
    if (lane < top) {
        chosen[(size_t)t * top + lane] = mine;
        weights[(size_t)t * top + lane] = mine >= 0 ? mine_score * scale : 0.0f;
        if (mine >= 0) gates[(size_t)t * row + mine] = mine_score * scale;
    }
}

__global__ void route_topk_kernel(const float* __restrict__ logits, int splits, size_t split_stride, int n_tokens, int experts,
                                  int top, int groups, int keep, float* __restrict__ gates, int* __restrict__ chosen,
                                  float* __restrict__ weights, RouteOptions opt) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    __shared__ float group_best[ROUTE_WARPS][32];
    const int warp = threadIdx.x >> 5;
    const int t = blockIdx.x * ROUTE_WARPS + warp;
    if (t >= n_tokens) return;
    route_token(logits + (size_t)t * (experts + opt.extra), splits, split_stride, t, experts, top, groups, keep, gates, chosen, weights,
                group_best[warp], opt);
}

// The router's product and the routing in one kernel, one block per token: the token's row goes to shared memory as
// float32, every warp takes experts in turn (lanes across the row, float32 sums), and the first warp then routes the token
// from the logits in shared memory.
template <typename TX, typename TW>
__global__ void route_rows_kernel(const TX* __restrict__ x, const TW* __restrict__ w, int hidden, int n_tokens, int experts, int top,
                                  int groups, int keep, float* __restrict__ gates, int* __restrict__ chosen,
                                  float* __restrict__ weights, RouteOptions opt) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    extern __shared__ float route_shared[];                     // hidden, then experts + extra, then 32
    float* logits = route_shared + hidden;
    const int t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int j = threadIdx.x; j < hidden; j += blockDim.x) route_shared[j] = tt_to_float(x[(size_t)t * hidden + j]);
    __syncthreads();
    for (int e = warp; e < experts + opt.extra; e += warps) {
        const TW* row = w + (size_t)e * hidden;
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        int j = lane;
        for (; j + 96 < hidden; j += 128) {                     // four loads in flight, four sums
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = tt_to_float(row[j + 32 * i]);
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = fmaf(v[i], route_shared[j + 32 * i], a[i]);
        }
        for (; j < hidden; j += 32) a[0] = fmaf(tt_to_float(row[j]), route_shared[j], a[0]);
        const float z = tt_warp_sum((a[0] + a[1]) + (a[2] + a[3]));
        if (lane == 0) logits[e] = z;
    }
    __syncthreads();
    if (warp == 0) route_token(logits, 1, 0, t, experts, top, groups, keep, gates, chosen, weights, logits + experts + opt.extra, opt);
}

// The same for prompts in bfloat16: a warp a token, its row in the lanes' registers (16 bytes each, up to RT_PIECES of them; instances
// for rows of up to 2,048, 2,560, 3,584 and 4,096 numbers, because pieces without numbers cost as much as others), so that
// the router's rows, which the block's eight warps read together, come out of the L1 and no barrier stands between a token's steps.
// 2,048 tokens of 2,048 numbers, 16 experts: 30 -> 16 us (a block a token staged its row and re-read the matrix from the L2).
constexpr int RT_WARPS = 8, RT_PIECES = 16;                     // rows of up to 4,096 numbers

template <int PIECES>
__global__ void __launch_bounds__(32 * RT_WARPS)
route_tokens_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, int hidden, int n_tokens, int experts, int top, int groups, int keep,
                    float* __restrict__ gates, int* __restrict__ chosen, float* __restrict__ weights, RouteOptions opt) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    extern __shared__ float route_shared[];                     // per warp: experts + extra, then 32
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, total = experts + opt.extra;
    float* logits = route_shared + warp * (total + 32);
    const int t = blockIdx.x * RT_WARPS + warp;
    if (t >= n_tokens) return;
    uint4 mine[PIECES];
#pragma unroll
    for (int c = 0; c < PIECES; ++c) {
        const int j = 8 * (lane + 32 * c);
        mine[c] = j < hidden ? __ldg(reinterpret_cast<const uint4*>(x + (size_t)t * hidden + j)) : make_uint4(0u, 0u, 0u, 0u);
    }
    for (int e = 0; e < total; ++e) {
        const __nv_bfloat16* row = w + (size_t)e * hidden;
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int c = 0; c < PIECES; ++c) {
            const int j = 8 * (lane + 32 * c);
            if (j >= hidden) continue;
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row + j));
            const uint32_t p[4] = {raw.x, raw.y, raw.z, raw.w}, q[4] = {mine[c].x, mine[c].y, mine[c].z, mine[c].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[i] = fmaf(__uint_as_float(p[i] << 16), __uint_as_float(q[i] << 16), a[i]);
                a[i] = fmaf(__uint_as_float(p[i] & 0xffff0000u), __uint_as_float(q[i] & 0xffff0000u), a[i]);
            }
        }
        const float z = tt_warp_sum((a[0] + a[1]) + (a[2] + a[3]));
        if (lane == 0) logits[e] = z;
    }
    __syncwarp();
    route_token(logits, 1, 0, t, experts, top, groups, keep, gates, chosen, weights, logits + total, opt);
}

template <typename T>
__global__ void scale_expert_columns_kernel(T* __restrict__ act, int row_stride, int width, int experts,
                                            const float* __restrict__ gates, int gate_row, int shared_width, long long total) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int per_row = experts * width + shared_width;
    const long long t = i / per_row;
    const int c = (int)(i - t * per_row);
    const float g = gates[t * gate_row + (c < experts * width ? c / width : experts)];
    T* p = act + t * row_stride + c;
    *p = tt_from_float<T>(g == 0.0f ? 0.0f : tt_to_float(*p) * g);     // an expert the token did not choose adds nothing, whatever it made
}

extern "C" int tt_route_topk(const float* logits, int splits, long long split_stride, int n_tokens, int experts, int top, int groups,
                             int keep, float* gates, int* chosen, float* weights, int sigmoid, const float* correction,
                             int group_top2, int plain_weights, int extra, float weight_scale, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (experts <= 0 || experts > ROUTE_MAX_EXPERTS || top < 1 || top > 32 || top > experts || groups < 1 || groups > 32 ||
        experts % groups || keep < 1 || keep > groups || extra < 0 || extra > 32)
        return (int)cudaErrorInvalidValue;
    const RouteOptions opt{sigmoid, correction, group_top2, plain_weights, extra, weight_scale};
    tt_launch_pdl(route_topk_kernel, dim3((n_tokens + ROUTE_WARPS - 1) / ROUTE_WARPS), dim3(ROUTE_WARPS * 32), 0, stream, logits, splits,
                  (size_t)split_stride, n_tokens, experts, top, groups, keep, gates, chosen, weights, opt);
    TT_LAUNCH_CHECK();
}

// The same, PIECES pieces of 16 bytes a thread (width and row_stride are multiples of N numbers).  The weights of a thread's pieces are
// asked for together, then the pieces that have one: 8,192 tokens of eight experts of 1,024 with one chosen 47 -> 33 us, with all chosen 47 ->
// 42 (a piece a thread, its weight first: 39 and 55).  Few tokens: a piece a thread, asked for with its weight (64 tokens of 8,192 numbers 1.9 us,
// in four pieces 2.8).
template <typename T, int N, int PIECES>
__global__ void scale_expert_columns_vec_kernel(T* __restrict__ act, int row_stride, int width, int experts,
                                                const float* __restrict__ gates, int gate_row, int shared_width, long long total) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int per_row = experts * width + shared_width;
    uint4* p[PIECES];
    float g[PIECES];
    uint4 raw[PIECES];
#pragma unroll
    for (int k = 0; k < PIECES; ++k) {
        const long long i = (((long long)blockIdx.x * PIECES + k) * blockDim.x + threadIdx.x) * N;
        p[k] = nullptr;
        if (i >= total) continue;
        const long long t = i / per_row;
        const int c = (int)(i - t * per_row);
        g[k] = gates[t * gate_row + (c < experts * width ? c / width : experts)];
        p[k] = reinterpret_cast<uint4*>(act + t * row_stride + c);
    }
#pragma unroll
    for (int k = 0; k < PIECES; ++k)
        if (p[k] && (PIECES == 1 || g[k] != 0.0f)) raw[k] = *p[k];
#pragma unroll
    for (int k = 0; k < PIECES; ++k) {
        if (!p[k]) continue;
        if (g[k] == 0.0f) {                                     // an expert the token did not choose
            *p[k] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        T* v = reinterpret_cast<T*>(&raw[k]);
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] = tt_from_float<T>(tt_to_float(v[e]) * g[k]);
        *p[k] = raw[k];
    }
}

// sms: the device's multiprocessors
extern "C" int tt_route_rows(const void* x, int x_dtype, const void* w, int w_dtype, int hidden, int n_tokens, int experts, int top,
                             int groups, int keep, float* gates, int* chosen, float* weights, int sigmoid, const float* correction,
                             int group_top2, int plain_weights, int extra, float weight_scale, int sms, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (experts <= 0 || experts > ROUTE_MAX_EXPERTS || top < 1 || top > 32 || top > experts || groups < 1 || groups > 32 ||
        experts % groups || keep < 1 || keep > groups || extra < 0 || extra > 32)
        return (int)cudaErrorInvalidValue;
    const RouteOptions opt{sigmoid, correction, group_top2, plain_weights, extra, weight_scale};
    const size_t shared = (size_t)(hidden + experts + extra + 32) * sizeof(float);
    if (shared > 48 * 1024) return (int)cudaErrorInvalidValue;
    // A warp a token.  It pays a reduction for every expert, so rows have to be long enough for their products to outweigh it, the longer the
    // more experts there are; and tokens enough for a block of eight on every SM, or rows so long that 129 blocks do.  Measured, a block a
    // token against a warp a token (us): 2,048 tokens of 2,048 numbers, 16 experts 30 and 16, 256 experts 321 and 167; 512 numbers, 8 experts
    // 12.7 and 10.0, 64 experts 32 and 37; 768 numbers, 64 experts 43 and 38, but 3,000 tokens a sixth the other way; 1,024 numbers, 256 experts
    // 169 and 133, 3,000 tokens 6 % the other way; 1,183 tokens of 1,536 numbers, 4 experts 9.0 and 7.1; 1,025 of them, 64 experts 7 % the other
    // way, of 1,792 numbers a seventh less.
    const int row_from = experts + extra <= 8 ? 512 : experts + extra <= 16 ? 768 : 1024;
    const int row_least = n_tokens > RT_WARPS * sms ? row_from : n_tokens > (RT_WARPS - 1) * sms ? 1536 : 1792;
    if (n_tokens > 1024 && hidden >= row_least && x_dtype == TT_BF16 && w_dtype == TT_BF16 && hidden % 8 == 0 && hidden <= 32 * 8 * RT_PIECES && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
        const size_t each = (size_t)RT_WARPS * (experts + extra + 32) * sizeof(float);
#define TT_ROUTE_TOKENS(PIECES) tt_launch_pdl(route_tokens_kernel<PIECES>, dim3((n_tokens + RT_WARPS - 1) / RT_WARPS), dim3(32 * RT_WARPS), each, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, hidden, n_tokens, experts, top, groups, keep, gates, chosen, weights, opt)
        const int pieces = (hidden + 255) / 256;
        if (pieces <= 8) TT_ROUTE_TOKENS(8);
        else if (pieces <= 10) TT_ROUTE_TOKENS(10);
        else if (pieces <= 14) TT_ROUTE_TOKENS(14);
        else TT_ROUTE_TOKENS(RT_PIECES);
#undef TT_ROUTE_TOKENS
        TT_LAUNCH_CHECK();
    }
#define TT_ROUTE(TX, TW) tt_launch_pdl(route_rows_kernel<TX, TW>, dim3(n_tokens), dim3(n_tokens <= 256 ? 512 : 128), shared, stream, (const TX*)x, (const TW*)w, hidden, n_tokens, experts, top, groups, keep, gates, chosen, weights, opt)
    if (x_dtype == TT_F32 && w_dtype == TT_F32) TT_ROUTE(float, float);
    else if (x_dtype == TT_F32) TT_ROUTE(float, __nv_bfloat16);
    else if (w_dtype == TT_F32) TT_ROUTE(__nv_bfloat16, float);
    else TT_ROUTE(__nv_bfloat16, __nv_bfloat16);
#undef TT_ROUTE
    TT_LAUNCH_CHECK();
}

extern "C" int tt_scale_expert_columns(void* act, int dtype, int n_tokens, int row_stride, int width, int experts, const float* gates,
                                       int gate_row, int shared_width, cudaStream_t stream) {
    const long long total = (long long)n_tokens * ((long long)experts * width + shared_width);
    if (total <= 0) return 0;
    const int threads = 256;
    const int n = dtype == TT_F32 ? 4 : 8;
    if (width % n == 0 && shared_width % n == 0 && row_stride % n == 0 && ((uintptr_t)act & 15) == 0) {
        const int pieces = total / n >= 4LL * threads * 512 ? 4 : 1;        // four where that leaves several blocks an SM
        const long long blocks = (total / n + threads * pieces - 1) / (threads * pieces);
        if (blocks > 2147483647LL) return (int)cudaErrorInvalidValue;
#define TT_SCALE(T, N, PIECES) tt_launch_pdl(scale_expert_columns_vec_kernel<T, N, PIECES>, dim3((unsigned)blocks), dim3(threads), 0, stream, (T*)act, row_stride, width, experts, gates, gate_row, shared_width, total)
        if (dtype == TT_F32) { if (pieces == 4) TT_SCALE(float, 4, 4); else TT_SCALE(float, 4, 1); }
        else if (pieces == 4) TT_SCALE(__nv_bfloat16, 8, 4);
        else TT_SCALE(__nv_bfloat16, 8, 1);
#undef TT_SCALE
        TT_LAUNCH_CHECK();
    }
    const long long blocks = (total + threads - 1) / threads;
    if (blocks > 2147483647LL) return (int)cudaErrorInvalidValue;
    if (dtype == TT_F32)
        tt_launch_pdl(scale_expert_columns_kernel<float>, dim3((unsigned)blocks), dim3(threads), 0, stream, (float*)act, row_stride, width, experts, gates, gate_row, shared_width, total);
    else
        tt_launch_pdl(scale_expert_columns_kernel<__nv_bfloat16>, dim3((unsigned)blocks), dim3(threads), 0, stream, (__nv_bfloat16*)act, row_stride, width, experts, gates, gate_row, shared_width, total);
    TT_LAUNCH_CHECK();
}

// ------------------------------------------------------------------------------------
// The clamped gated unit of a mixture's experts, with the routing weights applied on the way.
// gate_up: float32 [splits][tokens][2 * cols], gate columns first; cols = experts * width + shared_width (the routed
// experts side by side, an always-on expert behind them).  With g' = min(g, limit) and u' = clamp(u, -limit, limit)
//   act[t][c] = g' * sigmoid(alpha * g') * (u' + 1) * gates[t][c / width]            (routed columns, limit)
//   act[t][c] = the same with shared_limit, times gates[t][experts] if shared_gated  (the always-on expert's columns)
// limit <= 0: no clamp.  Everything is float32 until the one narrowing at the end.
// ------------------------------------------------------------------------------------
template <typename TAct>
__global__ void expert_activation_kernel(const float* __restrict__ gate_up, int splits, size_t split_stride, TAct* __restrict__ act,
                                         int experts, int width, int shared_width, float limit, float shared_limit, float alpha,
                                         const float* __restrict__ gates, int gate_row, int shared_gated, long long total) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int cols = experts * width + shared_width;
    const long long t = i / cols;
    const int c = (int)(i - t * cols);
    const bool routed = c < experts * width;
    const float weight = routed ? gates[t * gate_row + c / width] : (shared_gated ? gates[t * gate_row + experts] : 1.0f);
    if (weight == 0.0f) { act[i] = tt_from_float<TAct>(0.0f); return; }          // an expert the token did not choose
    const float* row = gate_up + (size_t)t * (2 * (size_t)cols) + c;
    float g = 0.0f, u = 0.0f;
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
        g += __ldg(row + s * split_stride);
        u += __ldg(row + s * split_stride + cols);
    }
    const float lim = routed ? limit : shared_limit;
    if (lim > 0.0f) { g = fminf(g, lim); u = fminf(fmaxf(u, -lim), lim); }
    act[i] = tt_from_float<TAct>(g / (1.0f + expf(-alpha * g)) * (u + 1.0f) * weight);
}

extern "C" int tt_expert_activation(const float* gate_up, int splits, long long split_stride, void* act, int act_dtype, int n_tokens,
                                    int experts, int width, int shared_width, float limit, float shared_limit, float alpha,
                                    const float* gates, int gate_row, int shared_gated, cudaStream_t stream) {
    const long long total = (long long)n_tokens * ((long long)experts * width + shared_width);
    if (total <= 0) return 0;
    const int threads = 256;
    const long long blocks = (total + threads - 1) / threads;
    if (blocks > 2147483647LL || experts < 0 || width < 0 || shared_width < 0 || (shared_gated && gate_row <= experts))
        return (int)cudaErrorInvalidValue;
    if (act_dtype == TT_F32)
        tt_launch_pdl(expert_activation_kernel<float>, dim3((unsigned)blocks), dim3(threads), 0, stream, gate_up, splits, (size_t)split_stride, (float*)act, experts, width, shared_width, limit, shared_limit, alpha, gates, gate_row, shared_gated, total);
    else
        tt_launch_pdl(expert_activation_kernel<__nv_bfloat16>, dim3((unsigned)blocks), dim3(threads), 0, stream, gate_up, splits, (size_t)split_stride, (__nv_bfloat16*)act, experts, width, shared_width, limit, shared_limit, alpha, gates, gate_row, shared_gated, total);
    TT_LAUNCH_CHECK();
}

// ------------------------------------------------------------------------------------
// Experts without a gate projection: act[t][c] = f(sum over slices of up[s][t][c]) * gates[t][c / width].
// up: float32 [splits][tokens][experts * width].  f by `activation`: 0 silu, 1 relu, 2 the tanh form of gelu, 4 the exact gelu, 5 the
// square of relu.  Columns of experts the token did not choose are zero without being read.  A thread takes VEC neighbouring
// columns of one expert.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float expert_unary(float z, int activation) {
    if (activation == 5) { const float p = fmaxf(z, 0.0f); return p * p; }
    if (activation == 1) return fmaxf(z, 0.0f);
    if (activation == 2) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    if (activation == 4) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
    return z / (1.0f + expf(-z));
}

template <typename T, int N> struct alignas(N * sizeof(T)) ExpertPack { T v[N]; };

template <typename TAct, int VEC>
__global__ void expert_unary_activation_kernel(const float* __restrict__ up, int splits, size_t split_stride, TAct* __restrict__ act, int experts,
                                               int width, int activation, const float* __restrict__ gates, int gate_row, long long total) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
    if (i >= total) return;
    const int cols = experts * width;
    const long long t = i / cols;
    const int c = (int)(i - t * cols);
    const float weight = gates[t * gate_row + c / width];
    float z[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) z[e] = 0.0f;
    if (weight != 0.0f) {
        for (int s = 0; s < splits; ++s) {
            const ExpertPack<float, VEC> x = *reinterpret_cast<const ExpertPack<float, VEC>*>(up + (size_t)s * split_stride + i);
#pragma unroll
            for (int e = 0; e < VEC; ++e) z[e] += x.v[e];
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) z[e] = expert_unary(z[e], activation) * weight;
    }
    ExpertPack<TAct, VEC> o;
#pragma unroll
    for (int e = 0; e < VEC; ++e) o.v[e] = tt_from_float<TAct>(z[e]);
    *reinterpret_cast<ExpertPack<TAct, VEC>*>(act + i) = o;
}

extern "C" int tt_expert_unary_activation(const float* up, int splits, long long split_stride, void* act, int act_dtype, int n_tokens, int experts,
                                          int width, int activation, const float* gates, int gate_row, cudaStream_t stream) {
    const long long total = (long long)n_tokens * experts * width;
    if (total <= 0) return 0;
    if (activation < 0 || activation > 5 || activation == 3 || gate_row < experts) return (int)cudaErrorInvalidValue;
    const bool wide = width % 4 == 0 && split_stride % 4 == 0 && (((uintptr_t)up | (uintptr_t)act) & 15) == 0;
    const int threads = 256;
    const long long per_block = (long long)threads * (wide ? 4 : 1), blocks = (total + per_block - 1) / per_block;
    if (blocks > 2147483647LL) return (int)cudaErrorInvalidValue;
#define TT_UNARY(T, V) tt_launch_pdl(expert_unary_activation_kernel<T, V>, dim3((unsigned)blocks), dim3(threads), 0, stream, up, splits, (size_t)split_stride, (T*)act, experts, width, activation, gates, gate_row, total)
    if (act_dtype == TT_F32) { if (wide) TT_UNARY(float, 4); else TT_UNARY(float, 1); }
    else { if (wide) TT_UNARY(__nv_bfloat16, 4); else TT_UNARY(__nv_bfloat16, 1); }
#undef TT_UNARY
    TT_LAUNCH_CHECK();
}

// ------------------------------------------------------------------------------------
// Tokens sorted by the experts they chose, for prompts (products of few rows with an expert's weights each: tt_gemm_tcgen05_experts).
//   chosen [tokens][top] (an expert, or -1)  ->  xs: x's rows, expert after expert, each expert's from a multiple of 256 rows on;
//   place [tokens][top]: the row of xs (-1: none); tile_expert: the expert of every 256 rows; tile_count: how many such tiles there are.
// The first kernel, a block an expert, counts its tokens and ranks them in their order; the second copies, a warp a row.  Both are bound by their
// latency and the copies: 2,048 tokens of 2,048 numbers, 4 of 16 experts:
// 15 us together (66 MB), and 21 us the sum of the products at the end (101 MB), where every expert for every token took 180 more.
// ------------------------------------------------------------------------------------
constexpr int SORT_TILE = 256, SORT_THREADS = 1024, SORT_ROWS = 8;

__global__ void __launch_bounds__(SORT_THREADS)
rank_tokens_kernel(const int* __restrict__ chosen, int items, int* __restrict__ place, int* __restrict__ counts) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    __shared__ int sums[2][32];
    const int expert = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int before = 0;
    for (int i0 = 0, round = 0; i0 < items; i0 += 4 * SORT_THREADS, round ^= 1) {
        bool mine[4];
        int count = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = i0 + 4 * threadIdx.x + e;
            mine[e] = i < items && __ldg(chosen + i) == expert;
            count += mine[e];
        }
        int rank = count;                                       // sum over this and the lanes before it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, rank, o);
            if (lane >= o) rank += other;
        }
        if (lane == 31) sums[round][warp] = rank;
        __syncthreads();
        int all = sums[round][lane], first = lane < warp ? all : 0;
        all = __reduce_add_sync(0xffffffffu, all);
        rank += __reduce_add_sync(0xffffffffu, first) - count + before;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (mine[e]) place[i0 + 4 * threadIdx.x + e] = rank++;
        before += all;
    }
    if (threadIdx.x == 0) counts[expert] = before;
}

__device__ __forceinline__ int sort_first_row(const int* __restrict__ counts, int expert, int lane) {      // by a whole warp
    int sum = 0;
    for (int e = lane; e < expert; e += 32) sum += (__ldg(counts + e) + SORT_TILE - 1) / SORT_TILE * SORT_TILE;
    return __reduce_add_sync(0xffffffffu, sum);
}

__global__ void __launch_bounds__(32 * SORT_ROWS)
gather_tokens_kernel(const __nv_bfloat16* __restrict__ x, int hidden, const int* __restrict__ chosen, int items, int top, int experts, const int* __restrict__ counts,
                     int* __restrict__ place, __nv_bfloat16* __restrict__ xs, int* __restrict__ tile_expert, int* __restrict__ tile_count) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x == gridDim.x - 1) {                          // the last block: the tiles' experts
        for (int e = warp; e < experts; e += SORT_ROWS) {
            const int first = sort_first_row(counts, e, lane) / SORT_TILE, n = (__ldg(counts + e) + SORT_TILE - 1) / SORT_TILE;
            for (int i = lane; i < n; i += 32) tile_expert[first + i] = e;
            if (e == experts - 1 && lane == 0) {
                *tile_count = first + n;
                if (first + n == 0) tile_expert[0] = 0;         // nobody has a choice: the products still look at their first tile's expert
            }
        }
        return;
    }
    const int item = blockIdx.x * SORT_ROWS + warp;
    if (item >= items) return;
    const int expert = __ldg(chosen + item);
    if (expert < 0 || expert >= experts) {
        if (lane == 0) place[item] = -1;
        return;
    }
    const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)(item / top) * hidden);
    const int row = sort_first_row(counts, expert, lane) + place[item];
    __syncwarp();
    uint4* to = reinterpret_cast<uint4*>(xs + (size_t)row * hidden);
#pragma unroll 8
    for (int i = lane; i < hidden / 8; i += 32) to[i] = __ldg(from + i);
    if (lane == 0) place[item] = row;
}

// xs holds at least (items + 255 * min(experts, items)) / 256 tiles of 256 rows, tile_expert a number a tile
extern "C" int tt_sort_tokens(const void* x, int hidden, const int* chosen, int n_tokens, int top, int experts, int* counts, int* place, void* xs,
                              int* tile_expert, int* tile_count, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    const long long items = (long long)n_tokens * top;
    if (experts < 1 || experts > 65535 || top < 1 || items > 1000000000LL || hidden % 8 || (((uintptr_t)x | (uintptr_t)xs) & 15)) return (int)cudaErrorInvalidValue;
    tt_launch_pdl(rank_tokens_kernel, dim3(experts), dim3(SORT_THREADS), 0, stream, chosen, (int)items, place, counts);
    tt_launch_pdl(gather_tokens_kernel, dim3((unsigned)((items + SORT_ROWS - 1) / SORT_ROWS + 1)), dim3(32 * SORT_ROWS), 0, stream, (const __nv_bfloat16*)x, hidden, chosen,
                  (int)items, top, experts, (const int*)counts, place, (__nv_bfloat16*)xs, tile_expert, tile_count);
    TT_LAUNCH_CHECK();
}

// out[t] += sum over a token's choices of weights[t][c] * y[place[t][c]]  (float32; first the choices in their order, then the sum is
// added; a weight of zero counts for nothing, whatever y holds).  Four numbers a thread.
__global__ void __launch_bounds__(256)
combine_experts_kernel(const float* __restrict__ y, const int* __restrict__ place, const float* __restrict__ weights, int top, float* __restrict__ out, int hidden) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int t = blockIdx.x, c = 4 * (blockIdx.y * 256 + threadIdx.x);
    if (c >= hidden) return;
    float4* to = reinterpret_cast<float4*>(out + (size_t)t * hidden + c);
    const float4 old = *to;
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
        const int row = __ldg(place + (size_t)t * top + k);
        const float w = __ldg(weights + (size_t)t * top + k);
        if (row < 0 || w == 0.0f) continue;
        const float4 v = __ldg(reinterpret_cast<const float4*>(y + (size_t)row * hidden + c));
        sum.x = fmaf(w, v.x, sum.x); sum.y = fmaf(w, v.y, sum.y); sum.z = fmaf(w, v.z, sum.z); sum.w = fmaf(w, v.w, sum.w);
    }
    *to = make_float4(old.x + sum.x, old.y + sum.y, old.z + sum.z, old.w + sum.w);
}

extern "C" int tt_combine_experts(const float* y, const int* place, const float* weights, int n_tokens, int top, float* out, int hidden, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (top < 1 || hidden % 4 || (((uintptr_t)y | (uintptr_t)out) & 15)) return (int)cudaErrorInvalidValue;
    tt_launch_pdl(combine_experts_kernel, dim3(n_tokens, (hidden + 1023) / 1024), dim3(256), 0, stream, y, place, weights, top, out, hidden);
    TT_LAUNCH_CHECK();
}
