// Recurrences with one decay per head and token, for prompts: a chunk of 64 tokens at a time.
//
//   S_t = a_t S_(t-1) + dt_t B_t x_t^T,   y_t = S_t^T C_t + D x_t        (S: N x P per head; Mamba-2, and with a constant
//                                                                          decay and dt = 1 linear attention: B = k, C = q, x = v)
//
// With f(i, j) = a_(j+1) * .. * a_i, e_i = a_0 * .. * a_i and w_j = f(63, j) dt_j, a chunk that starts from state S gives
//   y_i = e_i (S^T C_i) + sum_(j<=i) f(i, j) dt_j (C_i . B_j) x_j + D x_i,     S <- e_63 S + sum_j w_j B_j x_j^T
// so the token-by-token chain of row products becomes four matrix products a chunk.  They run on the tensor cores with every operand in three
// bfloat16 parts (split_mma.cuh); the rows that a state of fast decays is made of are added by multiply-adds (ck_tail).  Error against 64 bits by decay, relative to
// token by token (and of float32 multiply-adds in chunks): outputs 0.999 a token 0.25 (0.73), 0.9 0.77 (0.92), 0.5 0.93 (1.05), 0.1 0.89 (1.01); states 0.23 (0.75),
// 0.67 (0.83), 1.00 (1.00), 1.00 (1.00).  The decays only ever enter as products of decays (never as quotients, never as differences of sums of logarithms): nothing
// cancels, and a constant decay may have any sign.  Up to 64 of them are multiplied before they meet a state, so none may exceed one (callers see to
// it).  Products of decays are formed in float64 from the float32 decays and rounded once inside an 8-token block and in e, w and e_63; across
// blocks f(i, j) dt_j is the product of three such numbers (in float32 here: five roundings; in float64, rounded once, for the delta rule below).
// Numbers that are not finite reach the tokens they reach in the recurrence and no others: the first kernel leaves them out and says which
// token of a chunk is the first with one, the walk takes the columns they reach from that token on one by one.
//
// Two kernels.  The first, parallel over chunks, makes what the columns of a head share: C and B of every chunk and group, and the scores times
// the factors f(i, j) dt_j of every chunk and head, in parts and in the order in which the walk's lanes take them, and e, w, e_63.  The second
// walks a sequence's chunks with the state of 16 to 128 columns of one head in its warps' accumulators.
//
// What bounds it: latency, with two warps a scheduler for want of registers (64 heads of 64 x 128: tensor pipe 45 % busy, issue slots 31 %, shared memory 34 %; a warp
// waits for fixed latencies, then for the pipe, then for shared memory): half of a chunk's time is its products, the rest splitting states and x, adding up outputs and
// waiting for one another.  16 warps with half the registers were slower at every size (64 heads of 64 x 128, 2,048
// tokens: 222 against 169 us), as was fetching the operands with 16-byte copies by all threads instead of the copy engine (198).
// Token by token, in chunks of float32 multiply-adds, and now (us, one B200, back to back): 64 heads of 64 x 128, one sequence of 2,048 tokens
// 748, 227, 171 (180 where every chunk has a tail), four of 731 423, 340, 236; 16 heads of 256 x 128, four of
// 1,024 590, 476, 313 (334).
#include "common.cuh"
#include "split_mma.cuh"
#include "tcgen05.cuh"

constexpr int CK_TOKENS = 64, CK_THREADS = 256, CK_WARPS = 8;          // threads: of the first kernel
constexpr int CK_MLD = CK_TOKENS + 4;
// a chunk's factors for one head: u [64], v [64] (times dt), e [64], w [64] (times dt), E [8][8], diagonal blocks [8][8][8] (times dt), e_63
constexpr int CK_U = 0, CK_V = 64, CK_E = 128, CK_W = 192, CK_BLOCKS = 256, CK_DIAG = 320, CK_ALL = 832, CK_FACTORS = 836;

__device__ __forceinline__ uint32_t ck_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ck_copy16(float* to, const float* from, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ck_smem(to)), "l"(from), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ck_copy4(float* to, const float* from, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ck_smem(to)), "l"(from), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void ck_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ck_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 64 rows of `width` numbers (at most WIDTH, a power of two; row stride `stride`) into shared memory, rows from `rows` on as zeros;
// vec: 16-byte pieces
template <int WIDTH, int THREADS = CK_THREADS>
__device__ __forceinline__ void ck_stage(float* to, int to_stride, const float* from, size_t stride, int rows, int width, bool vec) {
    if (vec) {
        constexpr int PER_ROW = WIDTH / 4, STEP = THREADS / PER_ROW, EACH = (CK_TOKENS + STEP - 1) / STEP;
        const int r0 = threadIdx.x / PER_ROW, c = 4 * (threadIdx.x % PER_ROW);
        if (c < width && (STEP <= CK_TOKENS || r0 < CK_TOKENS)) {
            to += r0 * to_stride + c;
            const float* at = from + c;
#pragma unroll
            for (int k = 0; k < EACH; ++k) {
                const int r = r0 + k * STEP;
                ck_copy16(to + k * STEP * to_stride, at + (r < rows ? (size_t)r * stride : 0), r < rows);
            }
        }
    } else {
        for (int e = threadIdx.x; e < CK_TOKENS * WIDTH; e += THREADS) {
            const int r = e / WIDTH, c = e % WIDTH;
            if (c < width) ck_copy4(to + r * to_stride + c, from + (r < rows ? (size_t)r * stride : 0) + c, r < rows);
        }
    }
}

// Where a sequence's chunks lie among the slots of scratch memory: sequence b's first is cu[b] / 64 + b, which leaves room for
// every chunk before the next sequence's first, whatever the lengths are.  n_tokens / 64 + sequences slots are enough.
__device__ __forceinline__ int ck_first_slot(const int* __restrict__ cu, int b) { return cu[b] / CK_TOKENS + b; }

// sum over the k-slices of a projection, in slice order
__device__ __forceinline__ float ck_sum_slices(const float* __restrict__ p, int splits, size_t split_stride) {
    float total = 0.0f;
    for (int s = 0; s < splits; ++s) total += __ldg(p + (size_t)s * split_stride);
    return total;
}

constexpr int CK_MBLOCKS = 10;                                  // blocks of 16 x 16 on and below the diagonal of 64 x 64
// a chunk's record for one head: e [64], w [64] (times dt; zero for the tail's tokens), e_63, the first token with a number that is not finite, the first
// token of the tail, the tail's w [8] (so far in shared memory in the walk), then decay [64] and dt [64]
constexpr int CK_R_E = 0, CK_R_W = 64, CK_R_ALL = 128, CK_R_BAD = 129, CK_R_TAIL = 130, CK_R_TAIL_W = 132, CK_NEAR = 140, CK_R_DECAY = 140, CK_R_DT = 204, CK_RECORD = 268;

// The rows of a chunk's last 8 tokens (its tail) are added to the state by multiply-adds, token after token, instead of by products on the tensor
// cores, where their decays multiply to less than CK_SHORT (0.77 a token).  Those rows are most of the state then, and a sum that a few products
// dominate is right to half a unit as a chain of multiply-adds, while the tensor cores truncate it.  The first kernel writes the 8 rows of B, or of w K.  Error of a state against 64 bits relative to token by
// token, without tails and with them: 0.8 a token 0.89 and 0.89, 0.7 1.03 and 0.93, 0.5 1.41 and 1.00, 0.1 2.28 and 1.00.  So are all rows of a chunk of up to 8
// tokens.  CK_TOKENS: no tail.
constexpr int CK_TAIL_ROWS = 8;
constexpr float CK_SHORT = 1.0f / 8.0f;
__device__ __forceinline__ int ck_tail(const float* decay, int count, int lane) {       // by a whole warp
    if (count <= CK_TAIL_ROWS) return 0;
    float last = fabsf(decay[count - CK_TAIL_ROWS + (lane & 7)]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) last *= __shfl_xor_sync(0xffffffffu, last, o);
    return last < CK_SHORT ? count - CK_TAIL_ROWS : CK_TOKENS;
}
// where a state row's number lies in a row of the tail: a lane's rows of two tiles of 8 (2 q, 2 q + 1, 2 q + 8, 2 q + 9) side by side
__device__ __forceinline__ int ck_tail_place(int row) { return (row & ~15) + 4 * ((row & 7) >> 1) + 2 * ((row >> 3) & 1) + (row & 1); }
// s += x times the tail's row for this lane's two columns; at: the row at the warp's first state row and the lane's four numbers
template <int TILES>
__device__ __forceinline__ void ck_add_row(float (&s)[TILES][4], float x0, float x1, const float* at) {
#pragma unroll
    for (int k = 0; k < TILES; k += 2) {
        const float4 v = *reinterpret_cast<const float4*>(at + 8 * k);
        s[k][0] = fmaf(x0, v.x, s[k][0]);
        s[k][1] = fmaf(x0, v.y, s[k][1]);
        s[k][2] = fmaf(x1, v.x, s[k][2]);
        s[k][3] = fmaf(x1, v.y, s[k][3]);
        s[k + 1][0] = fmaf(x0, v.z, s[k + 1][0]);
        s[k + 1][1] = fmaf(x0, v.w, s[k + 1][1]);
        s[k + 1][2] = fmaf(x1, v.z, s[k + 1][2]);
        s[k + 1][3] = fmaf(x1, v.w, s[k + 1][3]);
    }
}
struct ScanChunks {
    const float* x;             // float32 rows of `stride` numbers: x of head h at + h * P, B and C of group g at + g * N
    const float* b;
    const float* c;
    size_t stride;
    const float* proj;          // Mamba-2: column dt_col + h of the partial sums is the raw step size
    int splits, cols, dt_col;
    size_t split_stride;
    const float* dt_bias;
    const float* a_log;
    const float* d_skip;        // or null
    const float* fixed_decay;   // a constant decay per head (then step sizes are one), or null
    float* state;               // [slots][heads][P][N]
    float* y;                   // [tokens][heads * P]
    unsigned* status;           // or null
    unsigned char* scratch;     // [slots][groups]: C and B as operands of the walk, B's rows of the tail; [slots][heads]: scores times factors as an operand, the record
    int max_slots;
    const int* cu;
    const int* slots;
    int sequences, heads, groups, P, N, vec, together;
    static __host__ __device__ constexpr size_t group_bytes(int padded) { return (size_t)2 * padded / 16 * 4 * SPLIT_BLOCK_BYTES + CK_TAIL_ROWS * padded * sizeof(float); }
    static __host__ __device__ constexpr size_t head_bytes() { return (size_t)CK_MBLOCKS * SPLIT_BLOCK_BYTES + CK_RECORD * sizeof(float); }
    template <int NP> __device__ uint4* group_scratch(int slot, int g) const {
        return reinterpret_cast<uint4*>(scratch + ((size_t)slot * groups + g) * group_bytes(NP));
    }
    template <int NP> __device__ uint4* head_scratch(int slot, int h) const {
        return reinterpret_cast<uint4*>(scratch + (size_t)max_slots * groups * group_bytes(NP) + ((size_t)slot * heads + h) * head_bytes());
    }
};

// ------------------------------------------------------------------------------------------- what a chunk's columns share
// the rows of outputs of a block of scores: blocks 0; 1, 2; 3 .. 5; 6 .. 9
__device__ __forceinline__ int ck_block_row(int block) { return block < 1 ? 0 : block < 3 ? 1 : block < 6 ? 2 : 3; }
// finite, and its first bfloat16 part too
__device__ __forceinline__ bool ck_usable(float x) { return fabsf(x) <= 3.3e38f; }

// The factors of one chunk and head, by one warp, into shared memory; lane l brings the decays and step sizes of tokens l and l + 32.
__device__ __forceinline__ void ck_factors(float* out, float a0, float a1, float dt0, float dt1, int lane, float* decay, float* step) {
    decay[lane] = a0; decay[lane + 32] = a1;
    step[lane] = dt0; step[lane + 32] = dt1;
    __syncwarp();
    // products inside a block of 8 tokens: of the decays up to the token's (u) and of those behind it (v)
    const int t = lane & 7;
    double u[2] = {(double)a0, (double)a1}, v[2] = {1.0, 1.0}, block[8];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const double other = __shfl_up_sync(0xffffffffu, u[half], o, 8);
            if (t >= o) u[half] *= other;
        }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const double next = __shfl_down_sync(0xffffffffu, half ? (double)a1 : (double)a0, 1, 8);
        if (t < 7) v[half] = next;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const double other = __shfl_down_sync(0xffffffffu, v[half], o, 8);
            if (t + o < 8) v[half] *= other;
        }
#pragma unroll
    for (int k = 0; k < 8; ++k) block[k] = __shfl_sync(0xffffffffu, u[k >> 2], 8 * (k & 3) + 7);
    double before[2] = {1.0, 1.0}, after[2] = {1.0, 1.0}, e[2] = {1.0, 1.0}, p[2] = {(double)dt0, (double)dt1};
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = lane + 32 * half, b = i >> 3;
            if (k < b) before[half] *= block[k];
            if (k > b) after[half] *= block[k];
            // E[b][t]: the blocks strictly between; column t of the diagonal block b: f(i', i) dt_i for i' = 0 .. 7 (zero above the diagonal)
            if (k > t && k < b) e[half] *= block[k];
            if (k > t) p[half] *= (double)decay[8 * b + k];
            out[CK_DIAG + b * 64 + k * 8 + t] = k < t ? 0.0f : (float)p[half];
        }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = lane + 32 * half;
        const double dt = half ? (double)dt1 : (double)dt0;
        out[CK_U + i] = (float)u[half];
        out[CK_V + i] = (float)(v[half] * dt);
        out[CK_E + i] = (float)(before[half] * u[half]);
        out[CK_W + i] = (float)(v[half] * after[half] * dt);
        out[CK_BLOCKS + i] = (float)e[half];
        if (i == CK_TOKENS - 1) out[CK_ALL] = (float)(before[half] * u[half]);
    }
    __syncwarp();
}

template <int NP>
struct CkPrepare {
    // C and B in parts: [C, B][hi, mid, lo][64][PITCH bytes] (rows 16 bytes further than a multiple of 128: no bank conflicts); then, in their place,
    // the scores and the factors of CK_WARPS heads; a lone head's factors, formed while C and B are on their way
    static constexpr int PITCH = 2 * NP + 16, PART = CK_TOKENS * PITCH, ONE = 6 * PART, BYTES = ONE + CK_FACTORS * 4;
    static_assert((CK_TOKENS * CK_MLD + CK_WARPS * CK_FACTORS) * 4 <= ONE, "scores and factors lie where C and B were");
};
// four 8 x 8 matrices of bfloat16; lane l names row l % 8 of matrix l / 8
__device__ __forceinline__ uint4 ck_matrices(uint32_t at) {
    uint4 v;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ck_matrices_turned(uint32_t at) {
    uint4 v;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}

template <int NP>
__global__ void __launch_bounds__(CK_THREADS, 2)
scan_chunks_prepare_kernel(const ScanChunks a) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    using L = CkPrepare<NP>;
    constexpr int KS = NP / 16;
    extern __shared__ __align__(16) float ck_shared[];
    float* gs = ck_shared;
    float* factors = ck_shared + CK_TOKENS * CK_MLD;
    float* one = ck_shared + L::ONE / 4;
    __shared__ float scalars[CK_WARPS][2][CK_TOKENS];
    __shared__ int bad, bad_head[CK_WARPS];
    // blockIdx.z: `together` heads of the group (each of these CTAs forms the scores for itself)
    const int slot = blockIdx.x, g = blockIdx.y;
    int lo = 0, hi = a.sequences;                               // the sequence whose slots reach this one
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ck_first_slot(a.cu, mid) <= slot) lo = mid; else hi = mid;
    }
    const int first = a.cu[lo], n = a.cu[lo + 1] - first, c0 = (slot - ck_first_slot(a.cu, lo)) * CK_TOKENS;
    if (c0 >= n) return;
    const int count = min(CK_TOKENS, n - c0);
    if (threadIdx.x == 0) bad = CK_TOKENS;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per_group = a.heads / a.groups;
    // the warps' heads; a lone head is the last warp's, which has one block of scores
    const bool lone = a.together == 1;
    const int own = lone ? CK_WARPS - 1 - warp : warp, h0 = g * per_group + blockIdx.z * a.together, h = h0 + own;
    const int here = min(a.together, per_group - (int)blockIdx.z * a.together);            // heads of this CTA
    float decay[2] = {1.0f, 1.0f}, step[2] = {0.0f, 0.0f};      // first the raw step sizes
    if (own < here && !a.fixed_decay)
#pragma unroll
        for (int half = 0; half < 2; ++half)
            if (lane + 32 * half < count) step[half] = ck_sum_slices(a.proj + (size_t)(first + c0 + lane + 32 * half) * a.cols + a.dt_col + h, a.splits, a.split_stride);
    // C and B into their parts.  Numbers that are not finite are left out: the walk takes such a token and what follows it in the chunk one by one.
    {
        constexpr int PIECES = NP / 4, EACH = CK_TOKENS * PIECES / CK_THREADS;
        const size_t row = (size_t)(first + c0) * a.stride + (size_t)g * a.N;
        float4 v[2][EACH];
#pragma unroll
        for (int matrix = 0; matrix < 2; ++matrix)
#pragma unroll
            for (int e = 0; e < EACH; ++e) {
                const int r = (threadIdx.x + e * CK_THREADS) / PIECES, c = 4 * ((threadIdx.x + e * CK_THREADS) % PIECES);
                const float* at = (matrix ? a.b : a.c) + row + (size_t)r * a.stride + c;
                float4& x = v[matrix][e];
                x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (r >= count || c >= a.N) continue;
                if (a.vec) x = __ldg(reinterpret_cast<const float4*>(at));
                else {
                    x.x = __ldg(at);
                    if (c + 1 < a.N) x.y = __ldg(at + 1);
                    if (c + 2 < a.N) x.z = __ldg(at + 2);
                    if (c + 3 < a.N) x.w = __ldg(at + 3);
                }
            }
#pragma unroll
        for (int matrix = 0; matrix < 2; ++matrix)
#pragma unroll
            for (int e = 0; e < EACH; ++e) {
                const int r = (threadIdx.x + e * CK_THREADS) / PIECES, c = 4 * ((threadIdx.x + e * CK_THREADS) % PIECES);
                float4& x = v[matrix][e];
                if (!(ck_usable(x.x) && ck_usable(x.y) && ck_usable(x.z) && ck_usable(x.w))) {
                    atomicMin(&bad, r);
                    x = make_float4(ck_usable(x.x) ? x.x : 0.0f, ck_usable(x.y) ? x.y : 0.0f, ck_usable(x.z) ? x.z : 0.0f, ck_usable(x.w) ? x.w : 0.0f);
                }
                if (const int tail = r - max(count - CK_TAIL_ROWS, 0); matrix && blockIdx.z == 0 && tail >= 0 && tail < CK_TAIL_ROWS) {
                    float* to = reinterpret_cast<float*>(a.group_scratch<NP>(slot, g) + 2 * KS * 4 * (SPLIT_BLOCK_BYTES / 16)) + tail * NP;
                    *reinterpret_cast<float2*>(to + ck_tail_place(c)) = make_float2(x.x, x.y);
                    *reinterpret_cast<float2*>(to + ck_tail_place(c + 2)) = make_float2(x.z, x.w);
                }
                uint2 hi, mid, lo;
                split_pair(x.x, x.y, hi.x, mid.x, lo.x);
                split_pair(x.z, x.w, hi.y, mid.y, lo.y);
                unsigned char* at = reinterpret_cast<unsigned char*>(ck_shared) + matrix * 3 * L::PART + r * L::PITCH + 2 * c;
                *reinterpret_cast<uint2*>(at) = hi;
                *reinterpret_cast<uint2*>(at + L::PART) = mid;
                *reinterpret_cast<uint2*>(at + 2 * L::PART) = lo;
            }
    }
    if (own < here) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (lane + 32 * half >= count) continue;
            if (a.fixed_decay) {
                decay[half] = __ldg(a.fixed_decay + h);
                step[half] = 1.0f;
            } else {
                const float raw = step[half] + __ldg(a.dt_bias + h);
                step[half] = raw > 20.0f ? raw : log1pf(expf(raw));
                decay[half] = expf(-expf(__ldg(a.a_log + h)) * step[half]);
            }
        }
    }
    float* f = lone ? one : factors + own * CK_FACTORS;
    __syncthreads();                                            // C and B are there
    if (lone && own == 0) ck_factors(f, decay[0], decay[1], step[0], step[1], lane, scalars[0][0], scalars[0][1]);
    const int t2 = 2 * (lane & 3), gq = lane >> 2;
    const uint32_t c_parts = tc::smem_u32(ck_shared), b_parts = c_parts + 3 * L::PART;
    // rows 16 q .. of a matrix and 16 of its columns: as an operand whose columns the rows are (pieces x, y, z, w; as one whose rows they are: x, z, y, w)
    const uint32_t plain = ((lane & 7) + 8 * (lane >> 4)) * L::PITCH + 16 * ((lane >> 3) & 1), turned = (lane & 15) * L::PITCH + 16 * (lane >> 4);
    // the scores C B^T on and below the diagonal, in tiles of 16 x 8 (two or three a warp); sums of 32 are added in float64: long chains lose more
    constexpr int TILES = (2 * CK_MBLOCKS + CK_WARPS - 1) / CK_WARPS;
    const uint32_t columns = (lane & 7) * L::PITCH + 16 * (lane >> 3);
    float scores[TILES][4];
#pragma unroll
    for (int mine = 0; mine < TILES; ++mine) {
        const int block = (warp + CK_WARPS * mine) >> 1, tile = warp & 1;
        if (block >= CK_MBLOCKS) continue;
        const int q = ck_block_row(block), s = block - q * (q + 1) / 2;
        double total[4] = {};
        float rest[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < KS; ks += 2) {
            float sum[2][4];
            SplitA A[2];
            uint4 v[3];                                         // columns' parts: x and y of 16 k, z and w of the next
#pragma unroll
            for (int part = 0; part < 3; ++part) {
                v[part] = ck_matrices(b_parts + part * L::PART + (16 * s + 8 * tile) * L::PITCH + 32 * ks + columns);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4 x = ck_matrices(c_parts + part * L::PART + 16 * q * L::PITCH + 32 * (ks + k) + plain);
                    uint32_t (&to)[4] = part == 0 ? A[k].hi : part == 1 ? A[k].mid : A[k].lo;
                    to[0] = x.x; to[1] = x.z; to[2] = x.y; to[3] = x.w;
                }
            }
            split_mma(rest[0], A[0].lo, v[0].x, v[0].y);
            split_mma(rest[1], A[1].lo, v[0].z, v[0].w);
            split_mma_zero(sum[0], A[0].hi, v[0].x, v[0].y);
            split_mma_zero(sum[1], A[1].hi, v[0].z, v[0].w);
            split_mma(rest[0], A[0].hi, v[2].x, v[2].y);
            split_mma(rest[1], A[1].hi, v[2].z, v[2].w);
            split_mma(rest[0], A[0].mid, v[1].x, v[1].y);
            split_mma(rest[1], A[1].mid, v[1].z, v[1].w);
            split_mma(rest[0], A[0].mid, v[0].x, v[0].y);
            split_mma(rest[1], A[1].mid, v[0].z, v[0].w);
            split_mma(rest[0], A[0].hi, v[1].x, v[1].y);
            split_mma(rest[1], A[1].hi, v[1].z, v[1].w);
#pragma unroll
            for (int e = 0; e < 4; ++e) total[e] += (double)(sum[0][e] + sum[1][e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) scores[mine][e] = (float)(total[e] + (double)(rest[0][e] + rest[1][e]));
    }
    if (blockIdx.z == 0) {
        // C: k = state rows, columns = tokens; B: k = tokens, columns = state rows
        uint4* out = a.group_scratch<NP>(slot, g) + lane;
#pragma unroll 2
        for (int item = warp; item < KS * 8; item += CK_WARPS) {
            const int s = (item - KS * 4) / KS, q = (item - KS * 4) % KS;
            uint4 v[3];
#pragma unroll
            for (int part = 0; part < 3; ++part)
                v[part] = item < KS * 4 ? ck_matrices(c_parts + part * L::PART + 16 * (item & 3) * L::PITCH + 32 * (item >> 2) + plain)
                                        : ck_matrices_turned(b_parts + part * L::PART + 16 * s * L::PITCH + 32 * q + turned);
#pragma unroll
            for (int part = 0; part < 3; ++part) out[item * (SPLIT_BLOCK_BYTES / 16) + 32 * part] = v[part];
        }
    }
    __syncthreads();                                            // C and B are read
#pragma unroll
    for (int mine = 0; mine < TILES; ++mine) {
        const int block = (warp + CK_WARPS * mine) >> 1;
        if (block >= CK_MBLOCKS) continue;
        const int q = ck_block_row(block), s = block - q * (q + 1) / 2;
#pragma unroll
        for (int half = 0; half < 2; ++half)
            *reinterpret_cast<float2*>(gs + (16 * q + gq + 8 * half) * CK_MLD + 16 * s + 8 * (warp & 1) + t2) = make_float2(scores[mine][2 * half], scores[mine][2 * half + 1]);
    }
    if (!lone && own < here) ck_factors(f, decay[0], decay[1], step[0], step[1], lane, scalars[own][0], scalars[own][1]);
    if (own < here) {
        int first_bad = bad;
#pragma unroll
        for (int half = 0; half < 2; ++half)
            if (!ck_usable(decay[half]) || !ck_usable(step[half])) first_bad = min(first_bad, lane + 32 * half);
        first_bad = __reduce_min_sync(0xffffffffu, first_bad);
        float* record = reinterpret_cast<float*>(a.head_scratch<NP>(slot, h) + CK_MBLOCKS * (SPLIT_BLOCK_BYTES / 16));
        const int tail = ck_tail(scalars[own][0], count, lane);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = lane + 32 * half;
            record[CK_R_E + i] = f[CK_E + i];
            record[CK_R_W + i] = i < tail ? f[CK_W + i] : 0.0f;
            if (i >= tail && i < tail + CK_TAIL_ROWS) record[CK_R_TAIL_W + i - tail] = f[CK_W + i];
            record[CK_R_DECAY + i] = decay[half];
            record[CK_R_DT + i] = step[half];
        }
        if (lane == 0) {
            record[CK_R_ALL] = f[CK_ALL];
            record[CK_R_TAIL] = __int_as_float(tail);
            bad_head[own] = first_bad;
        }
    }
    __syncthreads();
    // scores times factors, in blocks of 16 x 16 (q: tokens of the outputs, s: tokens they see)
    for (int item = warp; item < here * CK_MBLOCKS; item += CK_WARPS) {
        const int head = item / CK_MBLOCKS, block = item - head * CK_MBLOCKS, q = ck_block_row(block), s = block - q * (q + 1) / 2;
        const float* f = lone ? one : factors + head * CK_FACTORS;
        int first_bad = CK_TOKENS;
        float v[2][4], odd = 0.0f;
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
            const int i = 16 * q + 8 * tile + gq, bi = 2 * q + tile;
            const float2 e = *reinterpret_cast<const float2*>(f + CK_BLOCKS + bi * 8 + 2 * s);
            const float u = f[CK_U + i];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int j = 16 * s + 8 * half + t2;
                const float2 score = *reinterpret_cast<const float2*>(gs + i * CK_MLD + j);
                float2 m;
                if (q > s) {
                    const float2 step = *reinterpret_cast<const float2*>(f + CK_V + j);
                    const float between = u * (half ? e.y : e.x);
                    m = make_float2(score.x * (between * step.x), score.y * (between * step.y));
                } else if (tile > half) {
                    const float2 step = *reinterpret_cast<const float2*>(f + CK_V + j);
                    const float between = u * e.x;
                    m = make_float2(score.x * (between * step.x), score.y * (between * step.y));
                } else if (tile == half) {                      // (the scores above the diagonal need not be finite)
                    const float2 factor = *reinterpret_cast<const float2*>(f + CK_DIAG + bi * 64 + (i & 7) * 8 + t2);
                    m = make_float2(j <= i ? score.x * factor.x : 0.0f, j + 1 <= i ? score.y * factor.y : 0.0f);
                } else {
                    m = make_float2(0.0f, 0.0f);
                }
                odd = fmaxf(odd, fmaxf(ck_usable(m.x) ? 0.0f : 1.0f, ck_usable(m.y) ? 0.0f : 1.0f));
                v[tile][2 * half] = m.x;
                v[tile][2 * half + 1] = m.y;
            }
        }
        if (odd != 0.0f) {
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!ck_usable(v[tile][e])) {
                        first_bad = min(first_bad, 16 * q + 8 * tile + gq);
                        v[tile][e] = 0.0f;
                    }
        }
        split_store(a.head_scratch<NP>(slot, h0 + head) + block * (SPLIT_BLOCK_BYTES / 16), lane, v);
        if (first_bad < CK_TOKENS) atomicMin(bad_head + head, first_bad);
    }
    __syncthreads();
    if (threadIdx.x < here)
        reinterpret_cast<int*>(a.head_scratch<NP>(slot, h0 + threadIdx.x) + CK_MBLOCKS * (SPLIT_BLOCK_BYTES / 16))[CK_R_BAD] = bad_head[threadIdx.x];
}

// -------------------------------------------------------------------------------------------------- the walk over the chunks
// All products are transposed: 16 value columns on the rows of a tile (x^T, S^T), tokens or state rows on its columns, so that the state
// S^T [columns x rows] that the update leaves in a warp's accumulators is, split, the operand with which the next chunk's tokens read it.
// A warp holds 16 columns and a slice of NP / NS state rows; the NS warps of 16 columns add their parts of the outputs through
// shared memory, PB times 16 columns are a CTA's.
template <int NP, int PB, int NS>
struct CkWalk {
    static constexpr int THREADS = 32 * PB * NS, TP = 16 * PB, LDX = TP + 4, KS = NP / 16, KL = KS / NS;
    static constexpr int C = 0, B = C + KS * 4 * SPLIT_BLOCK_BYTES, TAIL = B + KS * 4 * SPLIT_BLOCK_BYTES, M = TAIL + CK_TAIL_ROWS * NP * 4, X = M + CK_MBLOCKS * SPLIT_BLOCK_BYTES;
    static constexpr int X_BYTES = CK_TOKENS * LDX * 4, R = X + 2 * X_BYTES, PARTS = R + 2 * CK_NEAR * 4;
    static constexpr int W = PARTS + (NS > 1 ? PB * (NS - 1) * 8 * 512 : 0), BAD = W + (NS > 1 ? PB * 4 * SPLIT_BLOCK_BYTES : 0), BAR = BAD + TP * 4, BYTES = BAR + 16;
    static_assert(BYTES + 16 <= 227 * 1024, "a CTA's shared memory");
    static constexpr int FIRST_BYTES = CK_NEAR * 4 + CK_MBLOCKS * SPLIT_BLOCK_BYTES + KS * 4 * SPLIT_BLOCK_BYTES, B_BYTES = KS * 4 * SPLIT_BLOCK_BYTES;
    // Which 16 tokens' x (j) a warp multiplies with the scores of which outputs (q >= j): a block each, about as many for the warps of
    // every scheduler
    static constexpr int XA = NS >= 4 ? 1 : 4 / NS;
    static __device__ __forceinline__ int x_block(int pb, int ns, int at) {
        if (NS == 1) return at;
        if (NS == 2) return ns == 0 ? 3 * at : 1 + at;
        const int w = pb & 1 ? NS - 1 - ns : ns;
        return NS == 4 ? w : w < 3 ? 0 : w < 5 ? 1 : w < 7 ? 2 : 3;
    }
    static __device__ __forceinline__ bool takes(int pb, int ns, int q, int at) {
        if (x_block(pb, ns, at) > q) return false;
        if (NS < 8) return true;
        const int w = pb & 1 ? NS - 1 - ns : ns;
        return w == 0 ? q < 2 : w == 3 ? q < 3 : w == 1 ? q == 2 : w == 5 ? q == 2 : q == 3;
    }
};

// a piece of memory by the copy engine (both addresses on 16 bytes); its bytes are counted on the barrier
__device__ __forceinline__ void ck_fetch(void* to, const void* from, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::smem_u32(to)), "l"(from), "r"(bytes), "r"(bar) : "memory");
}
// whether one of the numbers that this thread copied with ck_stage is not finite (after its copies have arrived)
template <int WIDTH, int THREADS>
__device__ __forceinline__ bool ck_staged_odd(const float* to, int to_stride, int width, bool vec) {
    bool odd = false;
    if (vec) {
        constexpr int PER_ROW = WIDTH / 4, STEP = THREADS / PER_ROW, EACH = (CK_TOKENS + STEP - 1) / STEP;
        const int r0 = threadIdx.x / PER_ROW, c = 4 * (threadIdx.x % PER_ROW);
        if (c < width && (STEP <= CK_TOKENS || r0 < CK_TOKENS)) {
#pragma unroll
            for (int k = 0; k < EACH; ++k) {
                const float4 v = *reinterpret_cast<const float4*>(to + (r0 + k * STEP) * to_stride + c);
                odd |= !(ck_usable(v.x) && ck_usable(v.y) && ck_usable(v.z) && ck_usable(v.w));
            }
        }
    } else {
        for (int e = threadIdx.x; e < CK_TOKENS * WIDTH; e += THREADS)
            if (e % WIDTH < width) odd |= !ck_usable(to[e / WIDTH * to_stride + e % WIDTH]);
    }
    return odd;
}

// One column's chunk token by token, by one warp: for chunks with numbers that are not finite.  Outputs from token `from` on.
__device__ __noinline__ void ck_scan_column(const ScanChunks& a, const float* record, int token, int count, int h, int g, int p, float* S, int from) {
    const int lane = threadIdx.x & 31;
    const float skip = a.d_skip ? __ldg(a.d_skip + h) : 0.0f;
    float s[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] = lane + 32 * k < a.N ? S[lane + 32 * k] : 0.0f;
    for (int i = 0; i < count; ++i) {
        const size_t row = (size_t)(token + i) * a.stride;
        const float x = a.x[row + (size_t)h * a.P + p], decay = record[CK_R_DECAY + i], dx = record[CK_R_DT + i] * x;
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int n = lane + 32 * k;
            if (n < a.N) {
                s[k] = fmaf(dx, a.b[row + (size_t)g * a.N + n], decay * s[k]);
                sum = fmaf(s[k], a.c[row + (size_t)g * a.N + n], sum);
            }
        }
        sum = tt_warp_sum(sum);
        if (lane == 0 && i >= from) a.y[(size_t)(token + i) * a.heads * a.P + (size_t)h * a.P + p] = fmaf(skip, x, sum);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (lane + 32 * k < a.N) S[lane + 32 * k] = s[k];
}

template <int NP, int PB, int NS>
__global__ void __launch_bounds__(32 * PB * NS, 1)
scan_chunks_kernel(const ScanChunks a) {
    using L = CkWalk<NP, PB, NS>;
    constexpr int THREADS = L::THREADS, TP = L::TP, LDX = L::LDX, KL = L::KL, PAIR = KL > 1 ? 2 : 1;
    extern __shared__ __align__(16) unsigned char ck_bytes[];
    __shared__ int late;                                        // twice the chunk whose wait ran out, and one for its second wait
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int h = blockIdx.x, b = blockIdx.y, p0 = blockIdx.z * TP;
    const int first = a.cu[b], n = a.cu[b + 1] - first;
    if (n <= 0) return;
    const int g = h / (a.heads / a.groups), P = a.P, N = a.N, inner = a.heads * P, width = min(TP, P - p0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pb = warp / NS, ns = warp % NS;
    const int t2 = 2 * (lane & 3), gq = lane >> 2;
    const float skip = a.d_skip ? __ldg(a.d_skip + h) : 0.0f;
    const int chunks = (n + CK_TOKENS - 1) / CK_TOKENS, slot0 = ck_first_slot(a.cu, b);
    const bool vec_x = a.vec && (width & 3) == 0;
    const uint4* Cs = reinterpret_cast<const uint4*>(ck_bytes + L::C) + ns * KL * 4 * (SPLIT_BLOCK_BYTES / 16);
    const uint4* Bs = reinterpret_cast<const uint4*>(ck_bytes + L::B) + ns * KL * (SPLIT_BLOCK_BYTES / 16);
    const uint4* Ms = reinterpret_cast<const uint4*>(ck_bytes + L::M);
    uint4* Ws = reinterpret_cast<uint4*>(ck_bytes + L::W) + pb * 4 * (SPLIT_BLOCK_BYTES / 16);
    float4* parts = reinterpret_cast<float4*>(ck_bytes + L::PARTS) + pb * (NS - 1) * 8 * 32 + lane;          // [another warp][tile of 8 tokens][lane]
    int* bad_from = reinterpret_cast<int*>(ck_bytes + L::BAD);
    const float* tail = reinterpret_cast<const float*>(ck_bytes + L::TAIL) + ns * (NP / NS) + 4 * (lane & 3);
    for (int e = threadIdx.x; e < 2 * CK_TOKENS * LDX; e += THREADS) reinterpret_cast<float*>(ck_bytes + L::X)[e] = 0.0f;      // what no copy writes is zero
    const uint32_t bar = tc::smem_u32(ck_bytes + L::BAR), bar_b = bar + 8;
    if (threadIdx.x == 0) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(bar_b, 1);
        tc::fence_barrier_init();
    }
    __syncthreads();
    bool in_time = true;                                        // no wait has run out; else nothing more is fetched

    auto xs = [&](int chunk) { return reinterpret_cast<float*>(ck_bytes + L::X + (chunk & 1) * L::X_BYTES); };
    auto records = [&](int chunk) { return reinterpret_cast<float*>(ck_bytes + L::R) + (chunk & 1) * CK_NEAR; };
    auto fetch_first = [&](int chunk) {                         // x, C, scores and factors
        if (chunk >= chunks) return;
        const int c0 = chunk * CK_TOKENS;
        const uint4* head = a.head_scratch<NP>(slot0 + chunk, h);
        ck_stage<TP, THREADS>(xs(chunk), LDX, a.x + (size_t)(first + c0) * a.stride + (size_t)h * P + p0, a.stride, min(CK_TOKENS, n - c0), width, vec_x);
        ck_commit();
        if (threadIdx.x == 0 && in_time) {
            tc::mbar_expect_tx(bar, L::FIRST_BYTES);
            ck_fetch(ck_bytes + L::C, a.group_scratch<NP>(slot0 + chunk, g), L::B_BYTES, bar);
            ck_fetch(ck_bytes + L::M, head, CK_MBLOCKS * SPLIT_BLOCK_BYTES, bar);
            ck_fetch(records(chunk), head + CK_MBLOCKS * (SPLIT_BLOCK_BYTES / 16), CK_NEAR * 4, bar);
        }
    };
    fetch_first(0);

    // this warp's state: tile k: columns pb * 16 + gq (and 8 further), rows row0 + 8 k + t2 and the next
    const int row0 = ns * (NP / NS);
    float* S = a.state + (((size_t)a.slots[b] * a.heads + h) * P + p0) * N;
    float s[2 * KL][4];
    auto load_state = [&](int half) {
        const int p = pb * 16 + gq + 8 * half;
#pragma unroll
        for (int k = 0; k < 2 * KL; ++k)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = row0 + 8 * k + t2 + e;
                s[k][2 * half + e] = p < width && r < N ? S[(size_t)p * N + r] : 0.0f;
            }
    };
    auto store_state = [&]() {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int p = pb * 16 + gq + 8 * half;
#pragma unroll
            for (int k = 0; k < 2 * KL; ++k)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = row0 + 8 * k + t2 + e;
                    if (p < width && r < N) S[(size_t)p * N + r] = s[k][2 * half + e];
                }
        }
    };
    load_state(0);
    load_state(1);
    // 16 tokens' x (times w) of this warp's columns as an operand
    auto split_x = [&](SplitA& A, const float* X, int j) {
        const float* at = X + (16 * j + t2) * LDX + pb * 16 + gq;
        split_pair(at[0], at[LDX], A.hi[0], A.mid[0], A.lo[0]);
        split_pair(at[8], at[LDX + 8], A.hi[1], A.mid[1], A.lo[1]);
        split_pair(at[8 * LDX], at[9 * LDX], A.hi[2], A.mid[2], A.lo[2]);
        split_pair(at[8 * LDX + 8], at[9 * LDX + 8], A.hi[3], A.mid[3], A.lo[3]);
    };
    auto split_wx = [&](SplitA& A, const float* X, const float* F, int j) {
        const float* at = X + (16 * j + t2) * LDX + pb * 16 + gq;
        const float2 w = *reinterpret_cast<const float2*>(F + CK_R_W + 16 * j + t2), v = *reinterpret_cast<const float2*>(F + CK_R_W + 16 * j + t2 + 8);
        split_pair(w.x * at[0], w.y * at[LDX], A.hi[0], A.mid[0], A.lo[0]);
        split_pair(w.x * at[8], w.y * at[LDX + 8], A.hi[1], A.mid[1], A.lo[1]);
        split_pair(v.x * at[8 * LDX], v.y * at[9 * LDX], A.hi[2], A.mid[2], A.lo[2]);
        split_pair(v.x * at[8 * LDX + 8], v.y * at[9 * LDX + 8], A.hi[3], A.mid[3], A.lo[3]);
    };

    for (int chunk = 0; chunk < chunks; ++chunk) {
        float* X = xs(chunk);
        const float* F = records(chunk);
        const int left = n - chunk * CK_TOKENS;
        ck_wait<0>();
        // (the same in two forms: with the branch the compiler's schedule of 128 columns is 3 % slower, without it that of the others 1 to 4 %)
        if constexpr (NS == 1) in_time = in_time && tc::mbar_wait(bar, chunk & 1);
        else if (in_time && !tc::mbar_wait(bar, chunk & 1)) { in_time = false; late = 2 * chunk; }
        bool odd = ck_staged_odd<TP, THREADS>(X, LDX, width, vec_x);
#pragma unroll
        for (int k = 0; k < 2 * KL; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e) odd |= !ck_usable(s[k][e]);
        // x, C, scores and factors are there; B, the weighted rows and the parts of the chunk before are read
        bool some_bad = __syncthreads_or(odd);
        some_bad |= __float_as_int(F[CK_R_BAD]) < CK_TOKENS;
        const int count = min(CK_TOKENS, left), tail0 = __float_as_int(F[CK_R_TAIL]);
        if (threadIdx.x == 0 && in_time) {
            const uint32_t bytes = L::B_BYTES + (tail0 < CK_TOKENS ? CK_TAIL_ROWS * NP * 4 : 0);
            tc::mbar_expect_tx(bar_b, bytes);
            ck_fetch(ck_bytes + L::B, a.group_scratch<NP>(slot0 + chunk, g) + L::KS * 4 * (SPLIT_BLOCK_BYTES / 16), bytes, bar_b);
        }
        if (some_bad) {
            // columns from their first token on that is, or meets, a number that is not finite go token by token; the others as ever
            for (int p = threadIdx.x; p < TP; p += THREADS) bad_from[p] = __float_as_int(F[CK_R_BAD]);
            __syncthreads();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                bool mine = false;
#pragma unroll
                for (int k = 0; k < 2 * KL; ++k) mine |= !ck_usable(s[k][2 * half]) || !ck_usable(s[k][2 * half + 1]);
                if (mine) atomicMin(bad_from + pb * 16 + gq + 8 * half, 0);
            }
            for (int e = threadIdx.x; e < CK_TOKENS * TP; e += THREADS)
                if (float* x = X + e / TP * LDX + e % TP; !ck_usable(*x)) {
                    atomicMin(bad_from + e % TP, e / TP);
                    *x = 0.0f;
                }
            store_state();
            __syncthreads();
            const float* record = reinterpret_cast<const float*>(a.head_scratch<NP>(slot0 + chunk, h) + CK_MBLOCKS * (SPLIT_BLOCK_BYTES / 16));
            for (int p = warp; p < width; p += THREADS / 32)
                if (bad_from[p] < count) ck_scan_column(a, record, first + chunk * CK_TOKENS, count, h, g, p0 + p, S + (size_t)p * N, bad_from[p]);
            __syncthreads();
        }
        float* out = a.y + (size_t)(first + chunk * CK_TOKENS) * inner + (size_t)h * P + p0 + pb * 16 + gq;
        const float* own = X + pb * 16 + gq;
        const int limit[2] = {pb * 16 + gq < width ? min(left, some_bad ? bad_from[pb * 16 + gq] : CK_TOKENS) : 0,
                              pb * 16 + gq + 8 < width ? min(left, some_bad ? bad_from[pb * 16 + gq + 8] : CK_TOKENS) : 0};
        auto write = [&](int tile, const float (&o)[4]) {       // the outputs of 8 tokens: skip times x is added last
            float* to = out + (size_t)(8 * tile + t2) * inner;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 8 * tile + t2 + (e & 1), half = e >> 1;
                const float v = a.d_skip ? fmaf(skip, own[i * LDX + 8 * half], o[e]) : o[e];
                if (i < limit[half]) to[(e & 1 ? inner : 0) + 8 * half] = v;
            }
        };
        float mine[NS > 1 ? 8 / NS : 1][4];
        {
            SplitA A, xa[L::XA];
            if (NS > 1 && (NS <= 4 || ns < 4)) {                // the rows of the update, shared out among the warps that take them
#pragma unroll
                for (int j = 0; j < (NS < 4 ? 4 / NS : 1); ++j) {
                    const int block = NS < 4 ? ns * (4 / NS) + j : ns;
                    split_wx(A, X, F, block);
                    split_store(Ws + block * (SPLIT_BLOCK_BYTES / 16), lane, A);
                }
            }
            auto split_state = [&](SplitA& to, int k) {
                split_pair(s[2 * k][0], s[2 * k][1], to.hi[0], to.mid[0], to.lo[0]);
                split_pair(s[2 * k][2], s[2 * k][3], to.hi[1], to.mid[1], to.lo[1]);
                split_pair(s[2 * k + 1][0], s[2 * k + 1][1], to.hi[2], to.mid[2], to.lo[2]);
                split_pair(s[2 * k + 1][2], s[2 * k + 1][3], to.hi[3], to.mid[3], to.lo[3]);
            };
            // y: C times the state for the tiles of blocks q0 and q0 + 1; then the scores times x, and out with it
            auto outputs = [&](int q0, float (*y)[4]) {
                float sum[4][4] = {}, rest[4][4] = {};
#pragma unroll
                for (int q = q0; q < q0 + 2; ++q)
#pragma unroll
                    for (int j = 0; j < L::XA; ++j)
                        if (L::takes(pb, ns, q, j))
                            split_products<1, false>(sum + 2 * (q - q0), rest + 2 * (q - q0), xa[j], Ms + (q * (q + 1) / 2 + L::x_block(pb, ns, j)) * (SPLIT_BLOCK_BYTES / 16), lane);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 e = *reinterpret_cast<const float2*>(F + CK_R_E + 16 * q0 + 8 * i + t2);
                    const float o[4] = {fmaf(e.x, y[i][0], rest[i][0]) + sum[i][0], fmaf(e.y, y[i][1], rest[i][1]) + sum[i][1],
                                        fmaf(e.x, y[i][2], rest[i][2]) + sum[i][2], fmaf(e.y, y[i][3], rest[i][3]) + sum[i][3]};
                    constexpr int EACH = 8 / NS;                // a warp adds up and writes EACH tiles
                    const int tile = 2 * q0 + i, owner = tile / EACH;
                    if (NS == 1) write(tile, o);
                    else if (owner != ns) parts[((ns - (ns > owner)) * 8 + tile) * 32] = make_float4(o[0], o[1], o[2], o[3]);
                    else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) mine[tile % EACH][e] = o[e];
                    }
                }
            };
            if constexpr (THREADS <= 256) {                     // registers for all outputs: the state is split as it is used
                float y[8][4], rest[8][4];
#pragma unroll
                for (int k = 0; k < KL; ++k) {
                    split_state(A, k);
                    const uint4* block = Cs + k * 4 * (SPLIT_BLOCK_BYTES / 16);
                    if (k == 0) { split_products<2, true>(y, rest, A, block, lane); split_products<2, true>(y + 4, rest + 4, A, block + 2 * (SPLIT_BLOCK_BYTES / 16), lane); }
                    else { split_products<2, false>(y, rest, A, block, lane); split_products<2, false>(y + 4, rest + 4, A, block + 2 * (SPLIT_BLOCK_BYTES / 16), lane); }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[i][e] += rest[i][e];
#pragma unroll
                for (int j = 0; j < L::XA; ++j) split_x(xa[j], X, L::x_block(pb, ns, j));
                outputs(0, y);
                outputs(2, y + 4);
            } else {
                SplitA As[KL];
#pragma unroll
                for (int k = 0; k < KL; ++k) split_state(As[k], k);
#pragma unroll
                for (int j = 0; j < L::XA; ++j) split_x(xa[j], X, L::x_block(pb, ns, j));
#pragma unroll
                for (int q0 = 0; q0 < 4; q0 += 2) {
                    float y[4][4], rest[4][4];
                    split_products<2, true>(y, rest, As[0], Cs + q0 * (SPLIT_BLOCK_BYTES / 16), lane);
#pragma unroll
                    for (int k = 1; k < KL; ++k) split_products<2, false>(y, rest, As[k], Cs + (k * 4 + q0) * (SPLIT_BLOCK_BYTES / 16), lane);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) y[i][e] += rest[i][e];
                    outputs(q0, y);
                }
            }
        }
        __syncthreads();                                        // the weighted rows and the parts are there; C and the scores are read
        fetch_first(chunk + 1);
        // S^T <- e_63 S^T + (w x)^T B; the larger part is added last: one rounding at the size of the sum
        if constexpr (NS == 1) in_time = in_time && tc::mbar_wait(bar_b, chunk & 1);
        else if (in_time && !tc::mbar_wait(bar_b, chunk & 1)) { in_time = false; late = 2 * chunk + 1; }
        const float all = F[CK_R_ALL];
        const bool long_memory = fabsf(all) > 0.25f;
        SplitA wa[NS > 1 ? 1 : 4];
        if (NS == 1)
#pragma unroll
            for (int j = 0; j < 4; ++j) split_wx(wa[NS > 1 ? 0 : j], X, F, j);
#pragma unroll
        for (int k = 0; k < KL; k += PAIR) {
            float sum[2 * PAIR][4], rest[2 * PAIR][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (NS > 1) split_load(wa[0], Ws + j * (SPLIT_BLOCK_BYTES / 16), lane);
                const uint4* block = Bs + (j * L::KS + k) * (SPLIT_BLOCK_BYTES / 16);
                if (j == 0) split_products<PAIR, true>(sum, rest, wa[0], block, lane);
                else split_products<PAIR, false>(sum, rest, wa[NS > 1 ? 0 : j], block, lane);
            }
#pragma unroll
            for (int i = 0; i < 2 * PAIR; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float& v = s[2 * k + i][e];
                    v = long_memory ? fmaf(all, v, sum[i][e] + rest[i][e]) : fmaf(all, v, rest[i][e]) + sum[i][e];
                }
        }
        if (tail0 < CK_TOKENS) {
            const float* x = own + tail0 * LDX;
            const float4 w[2] = {reinterpret_cast<const float4*>(F + CK_R_TAIL_W)[0], reinterpret_cast<const float4*>(F + CK_R_TAIL_W)[1]};
#pragma unroll
            for (int i = 0; i < CK_TAIL_ROWS; ++i) {            // (zeros behind the last token)
                const float wi = i & 2 ? (i & 1 ? w[i >> 2].w : w[i >> 2].z) : (i & 1 ? w[i >> 2].y : w[i >> 2].x);
                ck_add_row(s, wi * x[i * LDX], wi * x[i * LDX + 8], tail + i * NP);
            }
        }
        if (NS > 1) {
#pragma unroll
            for (int i = 0; i < 8 / NS; ++i) {
                const int tile = ns * (8 / NS) + i;
                float o[4] = {};
#pragma unroll
                for (int k = 0; k < NS - 1; ++k) {
                    const float4 q = parts[(k * 8 + tile) * 32];
                    o[0] += q.x; o[1] += q.y; o[2] += q.z; o[3] += q.w;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) o[e] += mine[i][e];
                write(tile, o);
            }
        }
        if (some_bad) {
            if (bad_from[pb * 16 + gq] < count) load_state(0);
            if (bad_from[pb * 16 + gq + 8] < count) load_state(1);
        }
    }
    if (!in_time && a.status) atomicOr(a.status, TT_STATUS_WAIT_EXPIRED);
    if (!in_time && threadIdx.x == 0) {                         // its copies that may still be on their way to this shared memory
        if (NS == 1)
            for (int phase = 0; phase < 2; ++phase) { tc::mbar_wait(bar, phase); tc::mbar_wait(bar_b, phase); }
        else {
            if (late & 1) tc::mbar_wait(bar_b, (late >> 1) & 1);
            if (const int chunk = (late + 1) >> 1; chunk < chunks) tc::mbar_wait(bar, chunk & 1);
        }
    }
    store_state();
}

template <int NP, int PB, int NS>
static int scan_chunks_launch(const ScanChunks& a, int max_slots, cudaStream_t stream) {
    using L = CkWalk<NP, PB, NS>;
    constexpr size_t prepare_bytes = CkPrepare<NP>::BYTES;
    cudaError_t code = tt_allow_shared(scan_chunks_prepare_kernel<NP>, prepare_bytes);
    if (code == cudaSuccess) code = tt_allow_shared(scan_chunks_kernel<NP, PB, NS>, L::BYTES);
    if (code != cudaSuccess) return (int)code;
    tt_launch_pdl(scan_chunks_prepare_kernel<NP>, dim3(max_slots, a.groups, (a.heads / a.groups + a.together - 1) / a.together), dim3(CK_THREADS), prepare_bytes, stream, a);
    tt_launch_pdl(scan_chunks_kernel<NP, PB, NS>, dim3(a.heads, a.sequences, (a.P + L::TP - 1) / L::TP), dim3(L::THREADS), (size_t)L::BYTES, stream, a);
    TT_LAUNCH_CHECK();
}

// Columns of a CTA of the walk: rounds of the SMs times what a chunk takes a CTA (hundredths of a microsecond, measured with the GPU to itself: 128 rows 16 columns
// 333, 32 453, 64 766, 128 1,363; 64 rows 32 columns 300, 64 500, 128 810, and 16 columns no less than 32).
extern "C" int tt_scan_chunks_columns(int heads, int sequences, int P, int N, int sms) {
    const long long one = (long long)heads * sequences;
    auto cost = [&](int columns, int chunk) { return (one * ((P + columns - 1) / columns) + sms - 1) / sms * chunk; };
    const bool small = N <= 64;
    const long long c16 = cost(16, 333), c32 = cost(32, small ? 300 : 453), c64 = cost(64, small ? 500 : 766), c128 = cost(128, small ? 810 : 1363);
    if (c128 <= c64 && c128 <= c32 && c128 <= c16) return 128;
    if (c64 <= c32 && c64 <= c16) return 64;
    return small || c32 <= c16 ? 32 : 16;
}

// Bytes of scratch memory for max_slots chunks.
extern "C" long long tt_scan_chunks_scratch_bytes(int max_slots, int heads, int groups, int N) {
    return (long long)max_slots * ((long long)groups * ScanChunks::group_bytes(N <= 64 ? 64 : 128) + (long long)heads * ScanChunks::head_bytes());
}

// rows: [tokens][width] with x, B and C from the given columns on (see ScanChunks).  max_slots: n_tokens / 64 + sequences.  scratch:
// tt_scan_chunks_scratch_bytes, on a 16-byte boundary (the walk copies it in 16-byte pieces whatever the rows' alignment).  sms: the device's multiprocessors.
extern "C" int tt_scan_chunks(const float* rows, int width, int x_col, int b_col, int c_col, const float* proj, int splits, long long split_stride,
                              int cols, int dt_col, const float* dt_bias, const float* a_log, const float* d_skip, const float* fixed_decay, float* state,
                              float* y, float* scratch, const int* cu, const int* slots, int sequences, int max_slots, int heads,
                              int groups, int P, int N, int sms, unsigned* status, cudaStream_t stream) {
    if (sequences <= 0 || max_slots <= 0) return 0;
    if (N <= 0 || N > 128 || P <= 0 || groups <= 0 || groups > 65535 || heads % groups || sequences > 65535) return (int)cudaErrorInvalidValue;
    if (!rows || !scratch || ((uintptr_t)scratch & 15) || (!fixed_decay && (!proj || !dt_bias || !a_log))) return (int)cudaErrorInvalidValue;
    const float *x = rows + x_col, *b = rows + b_col, *c = rows + c_col;
    const uintptr_t bases = (uintptr_t)x | (uintptr_t)b | (uintptr_t)c | (uintptr_t)y;
    // heads of a CTA of the first kernel: as few as one wave of two CTAs an SM has room for (a head takes a warp ten blocks of scores, eight heads all of them)
    int together = 1;
    while (together < CK_WARPS && (long long)max_slots * groups * ((heads / groups + together - 1) / together) > 2LL * sms) together *= 2;
    together = together < heads / groups ? together : heads / groups;
    const ScanChunks a{x, b, c, (size_t)width, proj, splits, cols, dt_col, (size_t)split_stride, dt_bias, a_log, d_skip, fixed_decay, state, y, status,
                       reinterpret_cast<unsigned char*>(scratch), max_slots, cu, slots, sequences, heads, groups, P, N,
                       (bases & 15) == 0 && !(width & 3) && !(N & 3) && !(P & 3) ? 1 : 0, together};
    const bool small = N <= 64;
    switch (tt_scan_chunks_columns(heads, sequences, P, N, sms)) {
        case 128: return small ? scan_chunks_launch<64, 8, 1>(a, max_slots, stream) : scan_chunks_launch<128, 8, 1>(a, max_slots, stream);
        case 64: return small ? scan_chunks_launch<64, 4, 2>(a, max_slots, stream) : scan_chunks_launch<128, 4, 2>(a, max_slots, stream);
        case 32: return small ? scan_chunks_launch<64, 2, 4>(a, max_slots, stream) : scan_chunks_launch<128, 2, 4>(a, max_slots, stream);
    }
    return scan_chunks_launch<128, 1, 8>(a, max_slots, stream);
}

// ------------------------------------------------------------------------------------------------------ the gated delta rule
//   q = q / |q| * scale, k = k / |k|;  S <- a_t S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t
// (lengths with 1e-6 under the root, scale = D^-1/2).  Inside a chunk that starts from state S
//   u_i = beta_i v_i - beta_i e_i S^T k_i - sum_(j<i) beta_i f(i, j) (k_i . k_j) u_j
// is a unit lower triangular system, (I + A) U = beta V - (beta e K) S, whose solution is U = U0 - W S with (I + A) U0 = beta V and
// (I + A) W = beta e K: neither needs the state, so the first kernel solves for both, parallel over chunks and heads, and the second
// walks the chunks with   U = U0 - W S,   o = e Q S + P U (P_ij = f(i, j) q_i . k_j, j <= i),   S <- e_63 S + (w K)^T U.
// All products are the split products of split_mma.cuh, in the systems too (what the rows before a block of 16 take off it; the triangle of the 16
// is float32 multiply-adds, a column a thread); lengths, and products of factors with scores, are formed in float64 and rounded once; a chunk's tail is
// added to the state as in the scan.  Error against 64 bits by decay, relative to token by token (and of float32 multiply-adds in chunks), 22 heads of 128 x 128: outputs
// 0.999 a token 1.00 (1.00), 0.9 0.79 (0.77), 0.5 0.61 (0.69), 0.1 0.62 (0.66); states 1.01 (1.01), 1.03 (1.01), 0.92 (0.92), 0.87 (0.87).
// 16 heads of 128 x 128 on 4,097 tokens, us: token by token 1,900, chunks of float32 multiply-adds 485, now 385 (392 where every chunk has a tail), of which the first kernel takes 150
// (issue around splitting its operands, 44 % of the slots at two CTAs an SM, and barriers; with scores and systems of multiply-adds 172) and the walk 246 (three barriers a
// chunk and the latency of what lies between them; tensor pipe 38 % busy, issue slots 26 %).
constexpr int CD_THREADS = 256;

struct DeltaChunks {
    const float* qkv;           // float32 rows [q | k | v]: query/key head g at g * D, value head h at 2 * qk_heads * D + h * V
    size_t stride;
    const float* proj;          // columns b_col + h and a_col + h of the partial sums: raw write strength, raw decay input
    int splits, cols, b_col, a_col;
    size_t split_stride;
    const float* dt_bias;
    const float* a_log;
    float* state;               // [slots][heads][V][D]
    float* out;                 // [tokens][heads * V]
    unsigned* status;           // or null
    unsigned char* scratch;     // [slots][qk_heads]: q as an operand of the walk; [slots][heads]: W, w K and the scores P as operands, w K's rows of the tail, the record, U0 [64][V]
    const int* cu;
    const int* slots;
    int sequences, max_slots, heads, qk_heads, D, V, vec;
    static __host__ __device__ constexpr size_t matrix_bytes(int padded) { return (size_t)padded / 16 * 4 * SPLIT_BLOCK_BYTES; }
    static __host__ __device__ constexpr size_t record_at(int padded) { return 2 * matrix_bytes(padded) + CK_MBLOCKS * SPLIT_BLOCK_BYTES + CK_TAIL_ROWS * padded * sizeof(float); }
    static __host__ __device__ constexpr size_t operand_bytes(int padded) { return record_at(padded) + CK_RECORD * sizeof(float); }
    __host__ __device__ size_t head_bytes(int padded) const { return operand_bytes(padded) + (size_t)CK_TOKENS * V * sizeof(float); }
    template <int NP> __device__ uint4* group_scratch(int slot, int g) const { return reinterpret_cast<uint4*>(scratch + ((size_t)slot * qk_heads + g) * matrix_bytes(NP)); }
    template <int NP> __device__ uint4* head_scratch(int slot, int h) const {
        return reinterpret_cast<uint4*>(scratch + (size_t)max_slots * qk_heads * matrix_bytes(NP) + ((size_t)slot * heads + h) * head_bytes(NP));
    }
    template <int NP> __device__ float* values(int slot, int h) const { return reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(head_scratch<NP>(slot, h)) + operand_bytes(NP)); }
};

template <int NP>
struct CdPrepare {
    static constexpr int LD = NP + 4;
    static constexpr size_t BYTES = (size_t)(2 * CK_TOKENS * LD + 2 * CK_TOKENS * CK_MLD + CK_FACTORS + 7 * CK_TOKENS) * sizeof(float);
};

template <int NP>
__global__ void __launch_bounds__(CD_THREADS, 2)
delta_chunks_prepare_kernel(const DeltaChunks a) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    constexpr int LD = NP + 4;
    extern __shared__ __align__(16) float ck_shared[];
    float* ks = ck_shared;                                      // [64][LD]
    float* qs = ks + CK_TOKENS * LD;                            // [64][LD]
    float* As = qs + CK_TOKENS * LD;                            // [64][CK_MLD]
    float* Ps = As + CK_TOKENS * CK_MLD;                        // [64][CK_MLD]
    float* f = Ps + CK_TOKENS * CK_MLD;                         // [CK_FACTORS]
    double* nq = reinterpret_cast<double*>(f + CK_FACTORS);     // [64] each: D^-1/2 / |q|, 1 / |k|; then beta
    double* nk = nq + CK_TOKENS;
    float* beta = reinterpret_cast<float*>(nk + CK_TOKENS);
    float* scalars = beta + CK_TOKENS;                          // [2][64]; then the rows' factors of W's right-hand side
    __shared__ int bad, tail;                                   // the first token with a number that is not finite, the tail's first
    __shared__ float tail_w[CK_TAIL_ROWS];
    const int slot = blockIdx.x, h = blockIdx.y, D = a.D, V = a.V;
    int lo = 0, hi = a.sequences;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ck_first_slot(a.cu, mid) <= slot) lo = mid; else hi = mid;
    }
    const int first = a.cu[lo], n = a.cu[lo + 1] - first, c0 = (slot - ck_first_slot(a.cu, lo)) * CK_TOKENS;
    if (c0 >= n) return;
    const int count = min(CK_TOKENS, n - c0), g = h / (a.heads / a.qk_heads);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) bad = CK_TOKENS;
    if (D < NP)
        for (int e = threadIdx.x; e < 2 * CK_TOKENS * LD; e += CD_THREADS) ck_shared[e] = 0.0f;
    __syncthreads();
    uint4* head = a.head_scratch<NP>(slot, h);
    float* record = reinterpret_cast<float*>(head) + DeltaChunks::record_at(NP) / 4;
    const float* rows = a.qkv + (size_t)(first + c0) * a.stride;
    ck_stage<NP, CD_THREADS>(qs, LD, rows + (size_t)g * D, a.stride, count, D, a.vec);
    ck_stage<NP, CD_THREADS>(ks, LD, rows + (size_t)(a.qk_heads + g) * D, a.stride, count, D, a.vec);
    ck_commit();
    float raw_a[2] = {}, raw_b[2] = {};                         // the first warp's: what the chunk's decays and write strengths are made of
    if (warp == 0)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float* row = a.proj + (size_t)(first + c0 + lane + 32 * half) * a.cols + h;
            if (lane + 32 * half < count) {
                raw_a[half] = ck_sum_slices(row + a.a_col, a.splits, a.split_stride);
                raw_b[half] = ck_sum_slices(row + a.b_col, a.splits, a.split_stride);
            }
        }
    ck_wait<0>();
    __syncthreads();
    // numbers that are not finite are left out here: the walk takes such a token and what follows it in the chunk one by one
    for (int e = threadIdx.x; e < 2 * CK_TOKENS * (NP / 4); e += CD_THREADS) {
        const int row = e / (NP / 4);
        float* at = ck_shared + row * LD + 4 * (e % (NP / 4));
        const float4 v = *reinterpret_cast<const float4*>(at);
        if (!(ck_usable(v.x) && ck_usable(v.y) && ck_usable(v.z) && ck_usable(v.w))) {
            atomicMin(&bad, row & (CK_TOKENS - 1));
            *reinterpret_cast<float4*>(at) = make_float4(ck_usable(v.x) ? v.x : 0.0f, ck_usable(v.y) ? v.y : 0.0f, ck_usable(v.z) ? v.z : 0.0f, ck_usable(v.w) ? v.w : 0.0f);
        }
    }
    __syncthreads();
    // lengths: four lanes a row
    for (int item = threadIdx.x >> 2; item < 2 * CK_TOKENS; item += CD_THREADS / 4) {
        const float* row = (item < CK_TOKENS ? qs : ks) + (item & (CK_TOKENS - 1)) * LD;
        double sum = 0.0, more = 0.0;                           // (zeros behind D)
        for (int c = threadIdx.x & 3; c < NP; c += 8) {
            sum = fma((double)row[c], (double)row[c], sum);
            more = fma((double)row[c + 4], (double)row[c + 4], more);
        }
        sum += more;
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (!(threadIdx.x & 3)) (item < CK_TOKENS ? nq : nk)[item & (CK_TOKENS - 1)] = 1.0 / sqrt((sum + 1e-6) * (item < CK_TOKENS ? (double)D : 1.0));
    }
    // k . k and q . k on and below the diagonal, a warp 16 rows of the one or the other; the first, whose rows are the shortest, makes the factors too
    const int t2 = 2 * (lane & 3), gq = lane >> 2;
    if (warp == 0) {
        float decay[2];
        const float neg_a = -expf(__ldg(a.a_log + h)), bias = __ldg(a.dt_bias + h);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = lane + 32 * half;
            decay[half] = 1.0f;
            float write = 0.0f;
            if (i < count) {
                const float raw = raw_a[half] + bias;
                decay[half] = expf(neg_a * (raw > 20.0f ? raw : log1pf(expf(raw))));
                write = 1.0f / (1.0f + expf(-raw_b[half]));
            }
            if (!ck_usable(decay[half]) || !ck_usable(write)) atomicMin(&bad, i);
            beta[i] = ck_usable(write) ? write : 0.0f;
            record[CK_R_DECAY + i] = decay[half];
            record[CK_R_DT + i] = write;
        }
        ck_factors(f, decay[0], decay[1], 1.0f, 1.0f, lane, scalars, scalars + CK_TOKENS);
        const int first_of_tail = ck_tail(scalars, count, lane);
        if (lane == 0) record[CK_R_TAIL] = __int_as_float(tail = first_of_tail);
    }
    {
        const int q = warp >> 1;
        float sums[4][2][4] = {}, rest[4][2][4] = {};
        auto rows_of = [&](const float* m, int row, int k, float2 (&v)[2]) {
            const float* at = m + row * LD + 16 * k + t2;
            v[0] = *reinterpret_cast<const float2*>(at);
            v[1] = *reinterpret_cast<const float2*>(at + 8);
        };
#pragma unroll 1
        for (int k = 0; k < NP / 16; ++k) {
            SplitA A;
            float2 v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                rows_of(warp & 1 ? qs : ks, 16 * q + gq + 8 * e, k, v);
                split_pair(v[0].x, v[0].y, A.hi[e], A.mid[e], A.lo[e]);
                split_pair(v[1].x, v[1].y, A.hi[2 + e], A.mid[2 + e], A.lo[2 + e]);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                if (s > q) continue;
                uint32_t hi[2][2], mid[2][2], lo[2][2];
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) {
                    rows_of(ks, 16 * s + 8 * tile + gq, k, v);
#pragma unroll
                    for (int e = 0; e < 2; ++e) split_pair(v[e].x, v[e].y, hi[tile][e], mid[tile][e], lo[tile][e]);
                }
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) split_mma(rest[s][tile], A.lo, hi[tile][0], hi[tile][1]);
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) split_mma_add(sums[s][tile], A.hi, hi[tile][0], hi[tile][1]);
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) split_mma(rest[s][tile], A.hi, lo[tile][0], lo[tile][1]);
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) split_mma(rest[s][tile], A.mid, mid[tile][0], mid[tile][1]);
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) split_mma(rest[s][tile], A.mid, hi[tile][0], hi[tile][1]);
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) split_mma(rest[s][tile], A.hi, mid[tile][0], mid[tile][1]);
            }
        }
        __syncthreads();                                        // lengths, factors and write strengths are there
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (s > q) continue;
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = 16 * q + gq + 8 * (e >> 1), j = 16 * s + 8 * tile + t2 + (e & 1), bi = 2 * q + (e >> 1), bj = 2 * s + tile;
                    // products of the factors in float64, rounded once
                    const double fij = bi > bj ? (double)f[CK_U + i] * (double)f[CK_BLOCKS + bi * 8 + bj] * (double)f[CK_V + j]
                                     : bi == bj ? (double)f[CK_DIAG + bi * 64 + (i & 7) * 8 + (j & 7)] : 0.0;
                    const double product = fij * nk[j] * ((double)sums[s][tile][e] + (double)rest[s][tile][e]);
                    float m = warp & 1 ? (j <= i ? (float)(nq[i] * product) : 0.0f) : (j < i ? -(float)((double)beta[i] * nk[i] * product) : 0.0f);        // P, -A
                    if (!ck_usable(m)) {
                        atomicMin(&bad, i);
                        m = 0.0f;
                    }
                    (warp & 1 ? Ps : As)[i * CK_MLD + j] = m;
                }
        }
    }
    if (threadIdx.x < CK_TOKENS) {
        const int i = threadIdx.x;
        const float start = (float)((double)beta[i] * (double)f[CK_E + i] * nk[i]), w = (float)((double)f[CK_W + i] * nk[i]);
        record[CK_R_E + i] = (float)((double)f[CK_E + i] * nq[i]);
        scalars[i] = ck_usable(start) ? start : 0.0f;
        scalars[CK_TOKENS + i] = ck_usable(w) && i < tail ? w : 0.0f;       // (not usable: no column's state comes from these products)
        if (i >= tail && i < tail + CK_TAIL_ROWS) tail_w[i - tail] = w;
        if (i == 0) record[CK_R_ALL] = f[CK_ALL];
    }
    __syncthreads();
    if (tail < CK_TOKENS)
        for (int e = threadIdx.x; e < CK_TAIL_ROWS * NP; e += CD_THREADS) {     // (zeros behind the last token)
            const int r = e / NP, c = e % NP;
            (record - CK_TAIL_ROWS * NP)[r * NP + ck_tail_place(c)] = tail_w[r] * ks[(tail + r) * LD + c];
        }
    // the operands that do not need the systems: w K (k = tokens, columns = state rows), and by the first head of a group q (k = state rows, columns = tokens)
    constexpr int KS = NP / 16, BLOCK = SPLIT_BLOCK_BYTES / 16;
    auto by_token = [&](const float* m, int item, float (&v)[2][4]) {           // k = the matrix' columns, columns = its rows
        const int ks = item >> 2, q = item & 3;
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
            const float* at = m + (16 * q + 8 * tile + gq) * LD + 16 * ks + t2;
            const float2 x = *reinterpret_cast<const float2*>(at), y = *reinterpret_cast<const float2*>(at + 8);
            v[tile][0] = x.x; v[tile][1] = x.y; v[tile][2] = y.x; v[tile][3] = y.y;
        }
    };
    for (int item = warp; item < KS * 4; item += CD_THREADS / 32) {
        float v[2][4];
        const int j = item / KS, q = item % KS;
#pragma unroll
        for (int tile = 0; tile < 2; ++tile)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int token = 16 * j + t2 + (e & 1) + 8 * (e >> 1);
                v[tile][e] = scalars[CK_TOKENS + token] * ks[token * LD + 16 * q + 8 * tile + gq];
            }
        split_store(head + DeltaChunks::matrix_bytes(NP) / 16 + item * BLOCK, lane, v);
        if (h % (a.heads / a.qk_heads) == 0) {
            by_token(qs, item, v);
            split_store(a.group_scratch<NP>(slot, g) + item * BLOCK, lane, v);
        }
    }
    __syncthreads();                                            // keys and queries are read
    // (I + A) x = r for the columns of beta e K (made W) and of beta V (made U0), 16 rows at a time: what the rows before contribute as a product on the
    // tensor cores, a warp its 32 columns, then the triangle of the 16, a column a thread.  Half of the CTA takes the keys'
    // columns, in place, and every second tile of NP value columns; the other half the other tiles, where the queries lay.
    const int half = threadIdx.x / (CD_THREADS / 2), col = threadIdx.x % (CD_THREADS / 2);
    float* xs = (half ? qs : ks) + col;
    const float* values = rows + (size_t)2 * a.qk_heads * D + (size_t)h * V;
    auto solve = [&](int job) {                                 // job 0: the keys; job t: value columns from (t - 1) * NP on
        const int c = (job ? (job - 1) * NP : 0) + col, width = job ? V : D;
        if (col - lane >= NP || c - lane >= width) return;      // the same for the whole warp
        const bool live = c < width;
        float* to = a.values<NP>(slot, h) + c;
        float raw[16];                                          // the next 16 rows' values, fetched ahead
        auto fetch = [&](int i0) {
            if (!job) return;
#pragma unroll
            for (int r = 0; r < 16; ++r) raw[r] = live && i0 + r < count ? __ldg(values + (size_t)(i0 + r) * a.stride + c) : 0.0f;
        };
        fetch(0);
#pragma unroll 1
        for (int i0 = 0; i0 < CK_TOKENS; i0 += 16) {
            // the right-hand side, and what the rows before take off it, summed apart: many small terms added to x one by one would each round it
            float x[16], before[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) x[r] = job ? beta[i0 + r] * raw[r] : scalars[i0 + r] * xs[(i0 + r) * LD];
            if (i0 + 16 < CK_TOKENS) fetch(i0 + 16);
            if (i0) {
                float sums[4][4] = {}, rest[4][4] = {};
                const float* mine = xs - lane;
#pragma unroll 1
                for (int j0 = 0; j0 < i0; j0 += 16) {
                    SplitA A;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 v = *reinterpret_cast<const float2*>(As + (i0 + gq + 8 * (e & 1)) * CK_MLD + j0 + t2 + 8 * (e >> 1));
                        split_pair(v.x, v.y, A.hi[e], A.mid[e], A.lo[e]);
                    }
#pragma unroll
                    for (int tile = 0; tile < 4; ++tile) {
                        uint32_t hi[2], mid[2], lo[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float* at = mine + (j0 + t2 + 8 * e) * LD + 8 * tile + gq;
                            split_pair(at[0], at[LD], hi[e], mid[e], lo[e]);
                        }
                        split_mma(rest[tile], A.lo, hi[0], hi[1]);
                        split_mma_add(sums[tile], A.hi, hi[0], hi[1]);
                        split_mma(rest[tile], A.hi, lo[0], lo[1]);
                        split_mma(rest[tile], A.mid, mid[0], mid[1]);
                        split_mma(rest[tile], A.mid, hi[0], hi[1]);
                        split_mma(rest[tile], A.hi, mid[0], mid[1]);
                    }
                }
                __syncwarp();                                   // the right-hand sides are read: the sums take their place on the way to their columns' threads
                float* out = xs - lane + (i0 + gq) * LD + t2;
#pragma unroll
                for (int tile = 0; tile < 4; ++tile)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        *reinterpret_cast<float2*>(out + 8 * e * LD + 8 * tile) = make_float2(sums[tile][2 * e] + rest[tile][2 * e], sums[tile][2 * e + 1] + rest[tile][2 * e + 1]);
                __syncwarp();
#pragma unroll
                for (int r = 0; r < 16; ++r) before[r] = xs[(i0 + r) * LD];
            } else {
#pragma unroll
                for (int r = 0; r < 16; ++r) before[r] = 0.0f;
            }
            x[0] += before[0];
#pragma unroll
            for (int r = 1; r < 16; ++r) {
#pragma unroll
                for (int j = 0; j < r; j += 4) {
                    const float4 m = *reinterpret_cast<const float4*>(As + (i0 + r) * CK_MLD + i0 + j);
                    before[r] = fmaf(m.x, x[j], before[r]);
                    if (j + 1 < r) before[r] = fmaf(m.y, x[j + 1], before[r]);
                    if (j + 2 < r) before[r] = fmaf(m.z, x[j + 2], before[r]);
                    if (j + 3 < r) before[r] = fmaf(m.w, x[j + 3], before[r]);
                }
                x[r] += before[r];
            }
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                xs[(i0 + r) * LD] = x[r];
                if (job && live) to[(size_t)(i0 + r) * width] = x[r];
            }
            __syncwarp();
        }
    };
    for (int job = half; (job - 1) * NP < V; job += 2) {
        solve(job);
        if (job == 0) {                                         // W lies where the keys were: as an operand, before value columns take its place
            asm volatile("bar.sync 1, %0;" ::"n"(CD_THREADS / 2) : "memory");
            for (int item = warp; item < KS * 4 + CK_MBLOCKS; item += CD_THREADS / 64) {
                float v[2][4];
                if (item < KS * 4) {
                    by_token(ks, item, v);
#pragma unroll
                    for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (!ck_usable(v[tile][e])) {
                                atomicMin(&bad, 16 * (item & 3) + 8 * tile + gq);
                                v[tile][e] = 0.0f;
                            }
                    split_store(head + item * BLOCK, lane, v);
                } else {
                    const int block = item - KS * 4, q = ck_block_row(block), s = block - q * (q + 1) / 2;
#pragma unroll
                    for (int tile = 0; tile < 2; ++tile) {
                        const float* at = Ps + (16 * q + 8 * tile + gq) * CK_MLD + 16 * s + t2;
                        const float2 x = *reinterpret_cast<const float2*>(at), y = *reinterpret_cast<const float2*>(at + 8);
                        v[tile][0] = x.x; v[tile][1] = x.y; v[tile][2] = y.x; v[tile][3] = y.y;
                    }
                    split_store(head + 2 * DeltaChunks::matrix_bytes(NP) / 16 + block * BLOCK, lane, v);
                }
            }
            if (V > NP) asm volatile("bar.sync 1, %0;" ::"n"(CD_THREADS / 2) : "memory");
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) reinterpret_cast<int*>(record)[CK_R_BAD] = bad;
}

// One column's chunk token by token, by one warp: for chunks with numbers that are not finite.  Outputs from token `from` on.
__device__ __noinline__ void ck_delta_column(const DeltaChunks& a, const float* record, int token, int count, int h, int g, int p, float* S, int from) {
    const int lane = threadIdx.x & 31, D = a.D;
    float s[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) s[r] = lane + 32 * r < D ? S[lane + 32 * r] : 0.0f;
    for (int i = 0; i < count; ++i) {
        const float* row = a.qkv + (size_t)(token + i) * a.stride;
        float q[4], k[4], qq = 0.0f, kk = 0.0f, sk = 0.0f, o = 0.0f;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int n = lane + 32 * r;
            q[r] = n < D ? row[(size_t)g * D + n] : 0.0f;
            k[r] = n < D ? row[(size_t)(a.qk_heads + g) * D + n] : 0.0f;
            qq = fmaf(q[r], q[r], qq);
            kk = fmaf(k[r], k[r], kk);
        }
        const float nq = rsqrtf(tt_warp_sum(qq) + 1e-6f) * rsqrtf((float)D), nk = rsqrtf(tt_warp_sum(kk) + 1e-6f), decay = record[CK_R_DECAY + i];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            k[r] *= nk;
            s[r] *= decay;
            if (lane + 32 * r < D) sk = fmaf(s[r], k[r], sk);
        }
        const float u = record[CK_R_DT + i] * (row[(size_t)2 * a.qk_heads * D + (size_t)h * a.V + p] - tt_warp_sum(sk));
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (lane + 32 * r < D) {
                s[r] = fmaf(k[r], u, s[r]);
                o = fmaf(s[r], q[r] * nq, o);
            }
        o = tt_warp_sum(o);
        if (lane == 0 && i >= from) a.out[(size_t)(token + i) * a.heads * a.V + (size_t)h * a.V + p] = o;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
        if (lane + 32 * r < D) S[lane + 32 * r] = s[r];
}

// The walk, transposed and split like the scan's: a warp holds 16 value columns and a slice of the state's rows.  W S and Q S of a chunk are added up over
// the slices through shared memory, and of what comes of it U^T goes back as the operand of both products that need it; a warp that adds up a tile
// of 8 tokens also makes its outputs.  w is in K already, which the first kernel wrote.
template <int NP, int PB, int NS>
struct CdWalk {
    static constexpr int THREADS = 32 * PB * NS, TP = 16 * PB, KS = NP / 16, KL = KS / NS, EACH = 8 / NS;
    static constexpr int MATRIX = KS * 4 * SPLIT_BLOCK_BYTES;
    static constexpr int W = 0, Q = W + MATRIX, K = Q + MATRIX, M = K + MATRIX, TAIL = M + CK_MBLOCKS * SPLIT_BLOCK_BYTES, R = TAIL + CK_TAIL_ROWS * NP * 4, PARTS = R + 2 * CK_NEAR * 4;
    static constexpr int U = PARTS + 2 * PB * (NS - 1) * 8 * 512, BAD = U + PB * 4 * SPLIT_BLOCK_BYTES, BAR = BAD + TP * 4, TAIL_U = BAR + 16;
    static constexpr int BYTES = TAIL_U + CK_TAIL_ROWS * TP * 4, REST_BYTES = R - K;
    static_assert(BYTES + 16 <= 227 * 1024, "a CTA's shared memory");
};

template <int NP, int PB, int NS>
__global__ void __launch_bounds__(32 * PB * NS, 1)
delta_chunks_kernel(const DeltaChunks a) {
    using L = CdWalk<NP, PB, NS>;
    constexpr int THREADS = L::THREADS, TP = L::TP, KL = L::KL, EACH = L::EACH, BLOCK = SPLIT_BLOCK_BYTES / 16, PAIR = KL > 1 ? 2 : 1;
    extern __shared__ __align__(16) unsigned char ck_bytes[];
    __shared__ int late;                                        // twice the chunk whose wait ran out, and one for its second wait
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int h = blockIdx.x, b = blockIdx.y, p0 = blockIdx.z * TP;
    const int first = a.cu[b], n = a.cu[b + 1] - first;
    if (n <= 0) return;
    const int g = h / (a.heads / a.qk_heads), V = a.V, D = a.D, width = min(TP, V - p0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pb = warp / NS, ns = warp % NS;
    const int t2 = 2 * (lane & 3), gq = lane >> 2;
    const int chunks = (n + CK_TOKENS - 1) / CK_TOKENS, slot0 = ck_first_slot(a.cu, b);
    const uint4* Ws = reinterpret_cast<const uint4*>(ck_bytes + L::W) + ns * KL * 4 * BLOCK;
    const uint4* Qs = reinterpret_cast<const uint4*>(ck_bytes + L::Q) + ns * KL * 4 * BLOCK;
    const uint4* Ks = reinterpret_cast<const uint4*>(ck_bytes + L::K) + ns * KL * BLOCK;
    const uint4* Ms = reinterpret_cast<const uint4*>(ck_bytes + L::M);
    uint4* Us = reinterpret_cast<uint4*>(ck_bytes + L::U) + pb * 4 * BLOCK;
    float4* parts_w = reinterpret_cast<float4*>(ck_bytes + L::PARTS) + pb * (NS - 1) * 8 * 32 + lane;          // [another warp][tile of 8 tokens][lane]
    float4* parts_q = parts_w + PB * (NS - 1) * 8 * 32;
    int* bad_from = reinterpret_cast<int*>(ck_bytes + L::BAD);
    const float* tail = reinterpret_cast<const float*>(ck_bytes + L::TAIL) + ns * (NP / NS) + 4 * (lane & 3);
    float* tail_u = reinterpret_cast<float*>(ck_bytes + L::TAIL_U) + pb * 16 + 2 * gq;                                                             // [token][columns c and c + 8 side by side]
    const uint32_t bar = tc::smem_u32(ck_bytes + L::BAR), bar_rest = bar + 8;
    if (threadIdx.x == 0) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(bar_rest, 1);
        tc::fence_barrier_init();
    }
    __syncthreads();
    bool in_time = true;                                        // no wait has run out; else nothing more is fetched

    auto records = [&](int chunk) { return reinterpret_cast<float*>(ck_bytes + L::R) + (chunk & 1) * CK_NEAR; };
    auto fetch_first = [&](int chunk) {                         // what meets the state, and the record
        if (threadIdx.x || chunk >= chunks || !in_time) return;
        const uint4* head = a.head_scratch<NP>(slot0 + chunk, h);
        tc::mbar_expect_tx(bar, 2 * L::MATRIX + CK_NEAR * 4);
        ck_fetch(ck_bytes + L::W, head, L::MATRIX, bar);
        ck_fetch(ck_bytes + L::Q, a.group_scratch<NP>(slot0 + chunk, g), L::MATRIX, bar);
        ck_fetch(records(chunk), head + DeltaChunks::record_at(NP) / 16, CK_NEAR * 4, bar);
    };
    auto fetch_rest = [&](int chunk) {                          // K, the scores and the tail
        if (threadIdx.x || chunk >= chunks || !in_time) return;
        tc::mbar_expect_tx(bar_rest, L::REST_BYTES);
        ck_fetch(ck_bytes + L::K, a.head_scratch<NP>(slot0 + chunk, h) + L::MATRIX / 16, L::REST_BYTES, bar_rest);
    };
    fetch_first(0);
    fetch_rest(0);

    // this warp's state: tile k: columns pb * 16 + gq (and 8 further), rows row0 + 8 k + t2 and the next
    const int row0 = ns * (NP / NS);
    float* S = a.state + (((size_t)a.slots[b] * a.heads + h) * V + p0) * D;
    float s[2 * KL][4];
    auto load_state = [&](int half) {
        const int p = pb * 16 + gq + 8 * half;
#pragma unroll
        for (int k = 0; k < 2 * KL; ++k)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = row0 + 8 * k + t2 + e;
                s[k][2 * half + e] = p < width && r < D ? S[(size_t)p * D + r] : 0.0f;
            }
    };
    auto store_state = [&]() {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int p = pb * 16 + gq + 8 * half;
#pragma unroll
            for (int k = 0; k < 2 * KL; ++k)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = row0 + 8 * k + t2 + e;
                    if (p < width && r < D) S[(size_t)p * D + r] = s[k][2 * half + e];
                }
        }
    };
    load_state(0);
    load_state(1);

    for (int chunk = 0; chunk < chunks; ++chunk) {
        const float* F = records(chunk);
        const int left = n - chunk * CK_TOKENS;
        // this warp's tiles of U0, on their way while the products run
        float u[EACH][4];
        const float* from = a.values<NP>(slot0 + chunk, h) + p0 + pb * 16 + gq;
#pragma unroll
        for (int i = 0; i < EACH; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int token = 8 * (ns * EACH + i) + t2 + (e & 1), p = 8 * (e >> 1);
                u[i][e] = pb * 16 + gq + p < width ? __ldg(from + (size_t)token * V + p) : 0.0f;
            }
        if (in_time && !tc::mbar_wait(bar, chunk & 1)) { in_time = false; late = 2 * chunk; }
        const int count = min(CK_TOKENS, left), tail0 = __float_as_int(F[CK_R_TAIL]);
        for (int p = threadIdx.x; p < TP; p += THREADS) bad_from[p] = __float_as_int(F[CK_R_BAD]);
        float qs[EACH][4], ws[EACH][4];                         // this warp's tiles
        {
            SplitA A[KL];
#pragma unroll
            for (int k = 0; k < KL; ++k) {
                split_pair(s[2 * k][0], s[2 * k][1], A[k].hi[0], A[k].mid[0], A[k].lo[0]);
                split_pair(s[2 * k][2], s[2 * k][3], A[k].hi[1], A[k].mid[1], A[k].lo[1]);
                split_pair(s[2 * k + 1][0], s[2 * k + 1][1], A[k].hi[2], A[k].mid[2], A[k].lo[2]);
                split_pair(s[2 * k + 1][2], s[2 * k + 1][3], A[k].hi[3], A[k].mid[3], A[k].lo[3]);
            }
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                const uint4* operand = which ? Qs : Ws;
                float4* parts = which ? parts_q : parts_w;
                float (&own)[EACH][4] = which ? qs : ws;
#pragma unroll
                for (int q0 = 0; q0 < 4; q0 += 2) {
                    float y[4][4], rest[4][4];
                    split_products<2, true>(y, rest, A[0], operand + q0 * BLOCK, lane);
#pragma unroll
                    for (int k = 1; k < KL; ++k) split_products<2, false>(y, rest, A[k], operand + (k * 4 + q0) * BLOCK, lane);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int tile = 2 * q0 + i, owner = tile / EACH;
                        const float4 v = make_float4(y[i][0] + rest[i][0], y[i][1] + rest[i][1], y[i][2] + rest[i][2], y[i][3] + rest[i][3]);
                        if (owner == ns) { own[tile % EACH][0] = v.x; own[tile % EACH][1] = v.y; own[tile % EACH][2] = v.z; own[tile % EACH][3] = v.w; }
                        else parts[((ns - (ns > owner)) * 8 + tile) * 32] = v;
                    }
                }
            }
        }
        __syncthreads();                                        // the parts are there; W and Q are read
        fetch_first(chunk + 1);
        bool odd = false;
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            const int tile = ns * EACH + i;
            float sum[4] = {};
            float more[4] = {};
#pragma unroll
            for (int k = 0; k < NS - 1; ++k) {
                const float4 v = parts_w[(k * 8 + tile) * 32], w = parts_q[(k * 8 + tile) * 32];
                sum[0] += v.x; sum[1] += v.y; sum[2] += v.z; sum[3] += v.w;
                more[0] += w.x; more[1] += w.y; more[2] += w.z; more[3] += w.w;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                u[i][e] -= ws[i][e] + sum[e];
                qs[i][e] += more[e];
                if (!ck_usable(u[i][e])) {
                    odd = true;
                    atomicMin(bad_from + pb * 16 + gq + 8 * (e >> 1), 8 * tile + t2 + (e & 1));
                    u[i][e] = 0.0f;
                }
            }
            if (8 * tile + 8 > tail0) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (const int r = 8 * tile + t2 + (e & 1) - tail0; r >= 0 && r < CK_TAIL_ROWS) tail_u[r * TP + (e >> 1)] = u[i][e];
            }
            uint32_t part[3][2];
            split_pair(u[i][0], u[i][1], part[0][0], part[1][0], part[2][0]);
            split_pair(u[i][2], u[i][3], part[0][1], part[1][1], part[2][1]);
#pragma unroll
            for (int k = 0; k < 3; ++k)
                reinterpret_cast<uint2*>(Us + (tile >> 1) * BLOCK + 32 * k + lane)[tile & 1] = make_uint2(part[k][0], part[k][1]);
        }
        bool some_bad = __syncthreads_or(odd);                  // U is there
        some_bad |= __float_as_int(F[CK_R_BAD]) < CK_TOKENS;
        if (some_bad) {                                         // as in the scan: columns from their first such token on go token by token
            store_state();
            __syncthreads();
            const float* record = reinterpret_cast<const float*>(a.head_scratch<NP>(slot0 + chunk, h) + DeltaChunks::record_at(NP) / 16);
            for (int p = warp; p < width; p += THREADS / 32)
                if (bad_from[p] < count) ck_delta_column(a, record, first + chunk * CK_TOKENS, count, h, g, p0 + p, S + (size_t)p * D, bad_from[p]);
            __syncthreads();
        }
        if (in_time && !tc::mbar_wait(bar_rest, chunk & 1)) { in_time = false; late = 2 * chunk + 1; }
        // S^T <- e_63 S^T + U^T (w K); the larger part is added last
        const float all = F[CK_R_ALL];
        const bool long_memory = fabsf(all) > 0.25f;
        SplitA A;
#pragma unroll
        for (int k = 0; k < KL; k += PAIR) {
            float sum[2 * PAIR][4], rest[2 * PAIR][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                split_load(A, Us + j * BLOCK, lane);
                if (j == 0) split_products<PAIR, true>(sum, rest, A, Ks + (j * L::KS + k) * BLOCK, lane);
                else split_products<PAIR, false>(sum, rest, A, Ks + (j * L::KS + k) * BLOCK, lane);
            }
#pragma unroll
            for (int i = 0; i < 2 * PAIR; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float& v = s[2 * k + i][e];
                    v = long_memory ? fmaf(all, v, sum[i][e] + rest[i][e]) : fmaf(all, v, rest[i][e]) + sum[i][e];
                }
        }
        if (tail0 < CK_TOKENS) {
#pragma unroll
            for (int i = 0; i < CK_TAIL_ROWS; ++i) {
                const float2 u = *reinterpret_cast<const float2*>(tail_u + i * TP);
                ck_add_row(s, u.x, u.y, tail + i * NP);
            }
        }
        // outputs: Q S times its factor and the scores times U, for this warp's tiles
        float* out = a.out + (size_t)(first + chunk * CK_TOKENS) * a.heads * V + (size_t)h * V + p0 + pb * 16 + gq;
        const int limit[2] = {pb * 16 + gq < width ? min(left, some_bad ? bad_from[pb * 16 + gq] : CK_TOKENS) : 0,
                              pb * 16 + gq + 8 < width ? min(left, some_bad ? bad_from[pb * 16 + gq + 8] : CK_TOKENS) : 0};
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            const int tile = ns * EACH + i, q = tile >> 1;
            float sum[4] = {}, rest[4] = {}, more[4] = {};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j > q) continue;
                split_load(A, Us + j * BLOCK, lane);
                const uint2* block = reinterpret_cast<const uint2*>(Ms + (q * (q + 1) / 2 + j) * BLOCK + lane) + (tile & 1);
                const uint2 hi = block[0], mid = block[64], lo = block[128];
                split_mma(rest, A.lo, hi.x, hi.y);
                split_mma(more, A.mid, mid.x, mid.y);
                split_mma_add(sum, A.hi, hi.x, hi.y);
                split_mma(rest, A.hi, lo.x, lo.y);
                split_mma(more, A.mid, hi.x, hi.y);
                split_mma(rest, A.hi, mid.x, mid.y);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) rest[k] += more[k];
            const float2 e = *reinterpret_cast<const float2*>(F + CK_R_E + 8 * tile + t2);
            float* to = out + (size_t)(8 * tile + t2) * a.heads * V;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float o = fmaf(k & 1 ? e.y : e.x, qs[i][k], rest[k]) + sum[k];
                if (8 * tile + t2 + (k & 1) < limit[k >> 1]) to[(k & 1 ? (size_t)a.heads * V : 0) + 8 * (k >> 1)] = o;
            }
        }
        if (some_bad) {
            if (bad_from[pb * 16 + gq] < count) load_state(0);
            if (bad_from[pb * 16 + gq + 8] < count) load_state(1);
        }
        __syncthreads();                                        // K, the scores and U are read
        fetch_rest(chunk + 1);
    }
    if (!in_time && a.status) atomicOr(a.status, TT_STATUS_WAIT_EXPIRED);
    if (!in_time && threadIdx.x == 0) {                         // its copies that may still be on their way to this shared memory
        tc::mbar_wait(bar_rest, (late >> 1) & 1);
        if (const int chunk = (late + 1) >> 1; chunk < chunks) tc::mbar_wait(bar, chunk & 1);
    }
    store_state();
}

template <int NP, int PB, int NS>
static int delta_chunks_launch(const DeltaChunks& a, int max_slots, cudaStream_t stream) {
    using L = CdWalk<NP, PB, NS>;
    constexpr size_t prepare_bytes = CdPrepare<NP>::BYTES;
    cudaError_t code = tt_allow_shared(delta_chunks_prepare_kernel<NP>, prepare_bytes);
    if (code == cudaSuccess) code = tt_allow_shared(delta_chunks_kernel<NP, PB, NS>, L::BYTES);
    if (code != cudaSuccess) return (int)code;
    tt_launch_pdl(delta_chunks_prepare_kernel<NP>, dim3(max_slots, a.heads), dim3(CD_THREADS), prepare_bytes, stream, a);
    tt_launch_pdl(delta_chunks_kernel<NP, PB, NS>, dim3(a.heads, a.sequences, (a.V + L::TP - 1) / L::TP), dim3(L::THREADS), (size_t)L::BYTES, stream, a);
    TT_LAUNCH_CHECK();
}

// columns of a CTA, as for the scan: a chunk takes a CTA of 16, 32 and 64 columns 3.5, 5.5 and 10.7 us with keys of 128, 3.7, 5.4 and 8.4 with keys of 64
extern "C" int tt_delta_chunks_columns(int heads, int sequences, int D, int V, int sms) {
    const long long one = (long long)heads * sequences;
    auto cost = [&](int columns, int chunk) { return (one * ((V + columns - 1) / columns) + sms - 1) / sms * chunk; };
    const bool small = D <= 64;
    const long long c16 = cost(16, small ? 370 : 352), c32 = cost(32, small ? 540 : 550), c64 = cost(64, small ? 840 : 1070);
    return c64 <= c32 && c64 <= c16 ? 64 : c32 <= c16 ? 32 : 16;
}

extern "C" long long tt_delta_chunks_scratch_bytes(int max_slots, int heads, int qk_heads, int D, int V) {
    const int padded = D <= 64 ? 64 : 128;
    return (long long)max_slots * ((long long)qk_heads * DeltaChunks::matrix_bytes(padded) + (long long)heads * (DeltaChunks::operand_bytes(padded) + (long long)CK_TOKENS * V * sizeof(float)));
}

// scratch: tt_delta_chunks_scratch_bytes, on a 16-byte boundary; max_slots as for tt_scan_chunks
extern "C" int tt_delta_chunks(const float* qkv, int qkv_cols, const float* proj, int splits, long long split_stride, int cols, int b_col, int a_col,
                               const float* dt_bias, const float* a_log, float* state, float* out, float* scratch, const int* cu, const int* slots,
                               int sequences, int max_slots, int heads, int qk_heads, int D, int V, int sms, unsigned* status, cudaStream_t stream) {
    if (sequences <= 0 || max_slots <= 0) return 0;
    if (D <= 0 || D > 128 || V <= 0 || qk_heads <= 0 || heads % qk_heads || heads > 65535 || sequences > 65535) return (int)cudaErrorInvalidValue;
    if (!qkv || !proj || !dt_bias || !a_log || !scratch || ((uintptr_t)scratch & 15)) return (int)cudaErrorInvalidValue;
    const int vec = ((uintptr_t)qkv & 15) == 0 && !(qkv_cols & 3) && !(D & 3);
    const DeltaChunks a{qkv, (size_t)qkv_cols, proj, splits, cols, b_col, a_col, (size_t)split_stride, dt_bias, a_log, state, out, status,
                        reinterpret_cast<unsigned char*>(scratch), cu, slots, sequences, max_slots, heads, qk_heads, D, V, vec};
    const bool small = D <= 64;
    switch (tt_delta_chunks_columns(heads, sequences, D, V, sms)) {
        case 64: return small ? delta_chunks_launch<64, 4, 2>(a, max_slots, stream) : delta_chunks_launch<128, 4, 2>(a, max_slots, stream);
        case 32: return small ? delta_chunks_launch<64, 2, 4>(a, max_slots, stream) : delta_chunks_launch<128, 2, 4>(a, max_slots, stream);
    }
    return small ? delta_chunks_launch<64, 1, 4>(a, max_slots, stream) : delta_chunks_launch<128, 1, 8>(a, max_slots, stream);
}
