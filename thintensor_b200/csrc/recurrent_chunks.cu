// Recurrences with one decay per head and token, for prompts: a chunk of 64 tokens at a time.
//
//   S_t = a_t S_(t-1) + dt_t B_t x_t^T,   y_t = S_t^T C_t + D x_t        (S: N x P per head; Mamba-2, and with a constant
//                                                                          decay and dt = 1 linear attention: B = k, C = q, x = v)
//
// With f(i, j) = a_(j+1) * .. * a_i, e_i = a_0 * .. * a_i and w_j = f(63, j) dt_j, a chunk that starts from state S gives
//   y_i = e_i (S^T C_i) + sum_(j<=i) f(i, j) dt_j (C_i . B_j) x_j + D x_i,     S <- e_63 S + sum_j w_j B_j x_j^T
// so the token-by-token chain of row products becomes four matrix products a chunk, all of them float32 multiply-adds (the scores' short sums
// are added in float64, so that outputs are as close to 64 bits as token by token: 30 runs, at most 3 % further off, 7 % closer in the mean).  The
// decays only ever enter as products of decays (never as quotients, never as differences of sums of logarithms): nothing cancels, and a
// constant decay may have any sign.  Up to 64 of them are multiplied before they meet a state, so none may exceed one (callers see to
// it), and the scores C_i . B_j are formed undecayed: they overflow where |C| |B| does, which the recurrence, that meets dt x and the decays
// in between, need not.  Numbers that are not finite reach the tokens they reach in the recurrence and no others.  Products of decays are
// formed in float64 from the float32 decays and rounded once inside an 8-token block and in e, w and e_63; across blocks f(i, j) dt_j is
// the product of three such numbers (in float32 here: five roundings; in float64, rounded once, for the delta rule below).
//
// Two kernels.  The first, parallel over chunks, makes what the columns of a head share: G_ij = C_i . B_j for every chunk and
// group, and the factors of every chunk and head (u, v, E, diagonal blocks: f(i, j) is a product of three numbers across
// 8-token blocks, and is stored inside one).  The second walks a sequence's chunks with the state of TP columns of one head in
// registers (256 threads) and, for the products that read it, in shared memory.
//
// What bounds it: shared memory's delivery of operands and the latency of two warps a scheduler (one CTA of 8 warps an SM; the
// multiply-add pipe is 43 % busy); the copies of the next chunk run under this one's products.  16 warps with half the registers
// spilled and were slower (348 against 227 us at the first size below), rows of operands used for two instead of four outputs
// too (305).  Against the kernels that go token by token, whose chain of row products a token bounds them (us, one B200, back to back):
// 64 heads of 64 x 128, one sequence of 2,048 tokens 748 -> 226, four of 731 423 -> 340; 16 heads of 256 x 128, four of 1,024 590 -> 476.
#include "common.cuh"

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

__device__ __forceinline__ void ck_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long ck_pair(float lo, float hi) {
    return ((unsigned long long)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
__device__ __forceinline__ float ck_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float ck_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }

// Where a sequence's chunks lie among the slots of scratch memory: sequence b's first is cu[b] / 64 + b, which leaves room for
// every chunk before the next sequence's first, whatever the lengths are.  n_tokens / 64 + sequences slots are enough.
__device__ __forceinline__ int ck_first_slot(const int* __restrict__ cu, int b) { return cu[b] / CK_TOKENS + b; }

// sum over the k-slices of a projection, in slice order
__device__ __forceinline__ float ck_sum_slices(const float* __restrict__ p, int splits, size_t split_stride) {
    float total = 0.0f;
    for (int s = 0; s < splits; ++s) total += __ldg(p + (size_t)s * split_stride);
    return total;
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
    float* scores;              // scratch: [slots][groups][64][64]
    float* factors;             // scratch: [slots][heads][CK_FACTORS]
    const int* cu;
    const int* slots;
    int sequences, heads, groups, P, N, vec;
};

// ------------------------------------------------------------------------------------------- what a chunk's columns share
// The factors of one chunk and head, by one warp; lane l brings the decays and step sizes of tokens l and l + 32.
__device__ __forceinline__ void ck_factors(float* __restrict__ out, float a0, float a1, float dt0, float dt1, int lane, float* decay, float* step) {
    decay[lane] = a0; decay[lane + 32] = a1;
    step[lane] = dt0; step[lane + 32] = dt1;
    __syncwarp();
    // lane l < 8: its block's product; then everyone has all eight
    double mine = 1.0;
    if (lane < 8)
        for (int t = 0; t < 8; ++t) mine *= (double)decay[8 * lane + t];
    double block[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) block[k] = __shfl_sync(0xffffffffu, mine, k);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = lane + 32 * half, b = i >> 3, t = i & 7;
        double u = 1.0, v = 1.0, before = 1.0, after = 1.0;
        for (int k = 0; k <= t; ++k) u *= (double)decay[8 * b + k];
        for (int k = t + 1; k < 8; ++k) v *= (double)decay[8 * b + k];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k < b) before *= block[k];
            if (k > b) after *= block[k];
        }
        const double dt = (double)step[i];
        out[CK_U + i] = (float)u;
        out[CK_V + i] = (float)(v * dt);
        out[CK_E + i] = (float)(before * u);
        out[CK_W + i] = (float)(v * after * dt);
        // column t of the diagonal block: f(i', i) dt_i for i' = 0 .. 7 (zero above the diagonal)
        double p = dt;
        for (int k = 0; k < 8; ++k) {
            if (k > t) p *= (double)decay[8 * b + k];
            out[CK_DIAG + b * 64 + k * 8 + t] = k < t ? 0.0f : (float)p;
        }
        // E[bi][bj]: the blocks strictly between
        const int bi = i >> 3, bj = i & 7;
        double e = 1.0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k > bj && k < bi) e *= block[k];
        out[CK_BLOCKS + i] = (float)e;
        if (i == CK_TOKENS - 1) out[CK_ALL] = (float)(before * u);
    }
    __syncwarp();
}

template <int NP>
__global__ void __launch_bounds__(CK_THREADS, 2)
scan_chunks_prepare_kernel(const ScanChunks a) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    constexpr int LD = NP + 4;
    extern __shared__ __align__(16) float ck_shared[];
    float* cs = ck_shared;
    float* bs = cs + CK_TOKENS * LD;
    __shared__ float scalars[CK_WARPS][2][CK_TOKENS];
    // blockIdx.z: the scores and the first CK_WARPS heads' factors, or the factors of CK_WARPS further heads of the group
    const int slot = blockIdx.x, g = blockIdx.y;
    int lo = 0, hi = a.sequences;                               // the sequence whose slots reach this one
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ck_first_slot(a.cu, mid) <= slot) lo = mid; else hi = mid;
    }
    const int first = a.cu[lo], n = a.cu[lo + 1] - first, c0 = (slot - ck_first_slot(a.cu, lo)) * CK_TOKENS;
    if (c0 >= n) return;
    const int count = min(CK_TOKENS, n - c0);
    if (blockIdx.z == 0 && a.N < NP) {
        for (int e = threadIdx.x; e < 2 * CK_TOKENS * LD; e += CK_THREADS) ck_shared[e] = 0.0f;
        __syncthreads();
    }
    const size_t row = (size_t)(first + c0) * a.stride;
    if (blockIdx.z == 0) {
        ck_stage<NP>(cs, LD, a.c + row + (size_t)g * a.N, a.stride, count, a.N, a.vec);
        ck_stage<NP>(bs, LD, a.b + row + (size_t)g * a.N, a.stride, count, a.N, a.vec);
        ck_commit();
    }

    // the factors of the group's heads, while the rows are on their way
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per_group = a.heads / a.groups;
    if (const int k = blockIdx.z * CK_WARPS + warp; k < per_group) {
        const int h = g * per_group + k;
        float decay[2], step[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = lane + 32 * half;
            decay[half] = 1.0f;
            step[half] = 0.0f;
            if (i < count) {
                if (a.fixed_decay) {
                    decay[half] = __ldg(a.fixed_decay + h);
                    step[half] = 1.0f;
                } else {
                    const float raw = ck_sum_slices(a.proj + (size_t)(first + c0 + i) * a.cols + a.dt_col + h, a.splits, a.split_stride) + __ldg(a.dt_bias + h);
                    step[half] = raw > 20.0f ? raw : log1pf(expf(raw));
                    decay[half] = expf(-expf(__ldg(a.a_log + h)) * step[half]);
                }
            }
        }
        ck_factors(a.factors + ((size_t)slot * a.heads + h) * CK_FACTORS, decay[0], decay[1], step[0], step[1], lane, scalars[warp][0], scalars[warp][1]);
    }
    if (blockIdx.z) return;
    ck_wait<0>();
    __syncthreads();
    // G: 16 x 16 threads, rows and columns 16 apart
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double total[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) total[i][j] = 0.0;
    // sums of 8, for states of 128 rows added up to 32, those in float64: long chains lose more
    constexpr int MIDDLE = NP > 64 ? 32 : 8;
    for (int k0 = 0; k0 < NP; k0 += MIDDLE) {
        float part[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) part[i][j] = 0.0f;
#pragma unroll 2
        for (int k1 = k0; k1 < k0 + MIDDLE; k1 += 8) {
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll
            for (int k = k1; k < k1 + 8; k += 4) {
                float4 c[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    c[i] = *reinterpret_cast<const float4*>(cs + (ty + 16 * i) * LD + k);
                    b[i] = *reinterpret_cast<const float4*>(bs + (tx + 16 * i) * LD + k);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j <= i; ++j) {              // columns behind the row's block are not used
                        acc[i][j] = fmaf(c[i].x, b[j].x, acc[i][j]);
                        acc[i][j] = fmaf(c[i].y, b[j].y, acc[i][j]);
                        acc[i][j] = fmaf(c[i].z, b[j].z, acc[i][j]);
                        acc[i][j] = fmaf(c[i].w, b[j].w, acc[i][j]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) part[i][j] += acc[i][j];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) total[i][j] += (double)part[i][j];
    }
    float* out = a.scores + ((size_t)slot * a.groups + g) * CK_TOKENS * CK_TOKENS;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)                             // zeros above the diagonal: a later token's score may be no number
            out[(ty + 16 * i) * CK_TOKENS + tx + 16 * j] = tx + 16 * j <= ty + 16 * i ? (float)total[i][j] : 0.0f;
}

// -------------------------------------------------------------------------------------------------- the walk over the chunks
// The products of a chunk's 64 output rows are shared out over the warps in blocks of rows and, so that a lane can hold four rows of
// four neighbouring columns (an operand piece read from shared memory then serves four outputs, which is what bounds these
// products), over slices of k: PL = TP / 4 lanes lie across the columns, RL = 32 / PL across the rows.
// acc[r] += sum over k of A[row r][k] * B[k][columns], four k a step, k = k0, k0 + stride, ..; the next step's numbers are
// on their way while this one's are multiplied.
template <int RL>
__device__ __forceinline__ void ck_product(unsigned long long (&acc)[4][2], const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb, int k0, int stride, int k_end) {
    float4 av[4], an[4];
    ulonglong2 bv[4], bn[4];
    auto load = [&](float4 (&x)[4], ulonglong2 (&y)[4], int k) {
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(A + r * RL * lda + k);
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = *reinterpret_cast<const ulonglong2*>(B + (k + e) * ldb);
    };
    auto multiply = [&](const float4 (&x)[4], const ulonglong2 (&y)[4]) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float v = e == 0 ? x[r].x : e == 1 ? x[r].y : e == 2 ? x[r].z : x[r].w;
                const unsigned long long twice = ck_pair(v, v);
                ck_fma2(acc[r][0], twice, y[e].x);
                ck_fma2(acc[r][1], twice, y[e].y);
            }
    };
    if (k0 >= k_end) return;
    load(av, bv, k0);
    for (int k = k0; k < k_end; k += 2 * stride) {
        if (k + stride < k_end) load(an, bn, k + stride);
        multiply(av, bv);
        if (k + stride >= k_end) break;
        if (k + 2 * stride < k_end) load(av, bv, k + 2 * stride);
        multiply(an, bn);
    }
}

// The same with what lies behind a row left out instead of multiplied by the zeros that stand there: for a chunk with numbers in B
// that are not finite, which must not reach the tokens before them (0 * inf is no number).  row: this lane's first.
template <int RL>
__device__ __forceinline__ void ck_causal_product(unsigned long long (&acc)[4][2], const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb, int k0, int stride, int k_end, int row) {
#pragma unroll 1
    for (int k = k0; k < k_end; k += stride)
#pragma unroll 1
        for (int e = 0; e < 4; ++e) {
            const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(B + (k + e) * ldb);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (k + e > row + RL * r) continue;
                const float v = A[r * RL * lda + k + e];
                const unsigned long long twice = ck_pair(v, v);
                ck_fma2(acc[r][0], twice, y.x);
                ck_fma2(acc[r][1], twice, y.y);
            }
        }
}
// zero for finite numbers, no number otherwise
__device__ __forceinline__ float ck_not_finite(const float4& x) { return fmaf(x.x, 0.0f, fmaf(x.y, 0.0f, fmaf(x.z, 0.0f, x.w * 0.0f))); }

// Two such products with the same B (k0 .. k0 + K - 1 in sums of 32, which are added up: a long chain of additions loses more)
template <int RL, int K>
__device__ __forceinline__ void ck_two_products(unsigned long long (&acc0)[4][2], const float* __restrict__ A0, unsigned long long (&acc1)[4][2],
                                                const float* __restrict__ A1, int lda, const float* __restrict__ B, int ldb, int k0) {
    constexpr int SUM = K < 32 ? K : 32;
    float4 x0[2][4], x1[2][4];
    ulonglong2 y[2][4];
    auto load = [&](int at, int k) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            x0[at][r] = *reinterpret_cast<const float4*>(A0 + r * RL * lda + k);
            x1[at][r] = *reinterpret_cast<const float4*>(A1 + r * RL * lda + k);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) y[at][e] = *reinterpret_cast<const ulonglong2*>(B + (k + e) * ldb);
    };
    load(0, k0);
#pragma unroll 1
    for (int ks = 0; ks < K; ks += SUM) {
        unsigned long long p0[4][2], p1[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) p0[r][0] = p0[r][1] = p1[r][0] = p1[r][1] = 0ull;
#pragma unroll
        for (int step = 0; step < SUM / 4; ++step) {
            const int at = step & 1, next = ks + 4 * (step + 1);
            if (next < K) load(at ^ 1, k0 + next);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float v0 = e == 0 ? x0[at][r].x : e == 1 ? x0[at][r].y : e == 2 ? x0[at][r].z : x0[at][r].w;
                    const float v1 = e == 0 ? x1[at][r].x : e == 1 ? x1[at][r].y : e == 2 ? x1[at][r].z : x1[at][r].w;
                    const unsigned long long t0 = ck_pair(v0, v0), t1 = ck_pair(v1, v1);
                    ck_fma2(p0[r][0], t0, y[at][e].x);
                    ck_fma2(p0[r][1], t0, y[at][e].y);
                    ck_fma2(p1[r][0], t1, y[at][e].x);
                    ck_fma2(p1[r][1], t1, y[at][e].y);
                }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                acc0[r][c] = ck_pair(ck_lo(acc0[r][c]) + ck_lo(p0[r][c]), ck_hi(acc0[r][c]) + ck_hi(p0[r][c]));
                acc1[r][c] = ck_pair(ck_lo(acc1[r][c]) + ck_lo(p1[r][c]), ck_hi(acc1[r][c]) + ck_hi(p1[r][c]));
            }
    }
}

// acc += A * B over K numbers of k from k0 on, in sums of 32 (a long chain of additions loses more)
template <int RL, int K>
__device__ __forceinline__ void ck_state_product(unsigned long long (&acc)[4][2], const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb, int k0) {
    constexpr int SUM = K < 32 ? K : 32;
#pragma unroll 1
    for (int k = k0; k < k0 + K; k += SUM) {
        unsigned long long part[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) part[r][0] = part[r][1] = 0ull;
        ck_product<RL>(part, A, lda, B, ldb, k, 4, k + SUM);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            acc[r][0] = ck_pair(ck_lo(acc[r][0]) + ck_lo(part[r][0]), ck_hi(acc[r][0]) + ck_hi(part[r][0]));
            acc[r][1] = ck_pair(ck_lo(acc[r][1]) + ck_lo(part[r][1]), ck_hi(acc[r][1]) + ck_hi(part[r][1]));
        }
    }
}

// S <- all S + sum over the chunk's tokens of B[j] (w x)[j]^T: NL state rows and four columns of a lane; B: row j at j * NP
template <int NP, int NL>
__device__ __forceinline__ void ck_update(unsigned long long (&s)[NL][2], float all, const float* __restrict__ B, const float* __restrict__ XW, int ldx) {
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        s[i][0] = ck_pair(ck_lo(s[i][0]) * all, ck_hi(s[i][0]) * all);
        s[i][1] = ck_pair(ck_lo(s[i][1]) * all, ck_hi(s[i][1]) * all);
    }
#pragma unroll 8
    for (int j = 0; j < CK_TOKENS; ++j) {
        float bv[NL];
        if constexpr (NL == 4) {
            const float4 q = *reinterpret_cast<const float4*>(B + j * NP);
            bv[0] = q.x; bv[1] = q.y; bv[2] = q.z; bv[3] = q.w;
        } else if constexpr (NL == 2) {
            const float2 q = *reinterpret_cast<const float2*>(B + j * NP);
            bv[0] = q.x; bv[1] = q.y;
        } else {
            bv[0] = B[j * NP];
        }
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(XW + j * ldx);
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            const unsigned long long twice = ck_pair(bv[i], bv[i]);
            ck_fma2(s[i][0], twice, x.x);
            ck_fma2(s[i][1], twice, x.y);
        }
    }
}

// A chunk's outputs: this lane's sums and the other slices', then skip times own (if there is one); rows from `left` on do not exist
template <int RL, int SLICES>
__device__ __forceinline__ void ck_outputs(const unsigned long long (&acc)[4][2], const float* __restrict__ parts, int ldx, int row, int col, int width, int left,
                                           bool vec, float skip, const float4* own, float* __restrict__ out, int stride) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = row + RL * r;
        float o[4] = {ck_lo(acc[r][0]), ck_hi(acc[r][0]), ck_lo(acc[r][1]), ck_hi(acc[r][1])};
#pragma unroll
        for (int k = 0; k < SLICES - 1; ++k) {
            const float4 q = *reinterpret_cast<const float4*>(parts + (k * CK_TOKENS + i) * ldx + col);
            o[0] += q.x; o[1] += q.y; o[2] += q.z; o[3] += q.w;
        }
        if (own) {
            o[0] = fmaf(skip, own[r].x, o[0]); o[1] = fmaf(skip, own[r].y, o[1]);
            o[2] = fmaf(skip, own[r].z, o[2]); o[3] = fmaf(skip, own[r].w, o[3]);
        }
        if (i >= left || col >= width) continue;
        float* to = out + (size_t)i * stride + col;
        if (vec) {
            *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (col + e < width) to[e] = o[e];
        }
    }
}

template <int NP, int TP>
struct CkLayout {
    static constexpr int LDA = NP + 4, LDX = TP + 4;
    static constexpr int PL = TP / 4, RL = 32 / PL, ROWS = 4 * RL;          // lanes across columns and rows; output rows of a warp
    static constexpr int THREADS = CK_THREADS, WARPS = THREADS / 32;
    static constexpr int SLICES = WARPS * ROWS / CK_TOKENS;                 // of k
    static constexpr int A = 0, S = A + CK_TOKENS * LDA, XW = S + NP * LDX, PARTS = XW + CK_TOKENS * LDX, STAGE = PARTS + (SLICES - 1) * CK_TOKENS * LDX;
    static constexpr int B = 0, X = B + CK_TOKENS * NP, M = X + CK_TOKENS * LDX, F = M + CK_TOKENS * CK_MLD, STAGE_FLOATS = F + CK_FACTORS;
    static constexpr size_t BYTES = (size_t)(STAGE + 2 * STAGE_FLOATS) * sizeof(float);
};

template <int NP, int TP>
__global__ void __launch_bounds__(CkLayout<NP, TP>::THREADS, 1)
scan_chunks_kernel(const ScanChunks a) {
    using L = CkLayout<NP, TP>;
    constexpr int THREADS = L::THREADS, PL = L::PL, RL = L::RL, ROW_BLOCKS = CK_TOKENS / L::ROWS;
    constexpr int NL = NP * TP / (THREADS * 4);              // state rows of a lane
    extern __shared__ __align__(16) float ck_shared[];
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int h = blockIdx.x, b = blockIdx.y, p0 = blockIdx.z * TP;
    const int first = a.cu[b], n = a.cu[b + 1] - first;
    if (n <= 0) return;
    const int g = h / (a.heads / a.groups), P = a.P, N = a.N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = 4 * (lane % PL), width = min(TP, P - p0), inner = a.heads * P;
    // row blocks are dealt to the warps so that the warps of a scheduler (w, w + 4, ..) together have equally long causal sums
    const int slice = warp / ROW_BLOCKS, block = (warp + (warp >> 2)) % ROW_BLOCKS;
    const int row = block * L::ROWS + lane / PL;                // first of this lane's four rows, RL apart
    const int srow = warp * (NP / L::WARPS) + (lane / PL) * NL;        // first of this lane's state rows
    const float skip = a.d_skip ? __ldg(a.d_skip + h) : 0.0f;
    float* As = ck_shared + L::A;
    float* Ss = ck_shared + L::S;
    float* XW = ck_shared + L::XW;
    const int chunks = (n + CK_TOKENS - 1) / CK_TOKENS, slot0 = ck_first_slot(a.cu, b);
    const bool vec_x = a.vec && (width & 3) == 0;

    for (int e = threadIdx.x; e < L::STAGE + 2 * L::STAGE_FLOATS; e += THREADS) ck_shared[e] = 0.0f;     // what no copy writes is zero
    __syncthreads();
    auto fetch_a = [&](int chunk) {
        if (chunk < chunks) {
            const int c0 = chunk * CK_TOKENS;
            ck_stage<NP, THREADS>(As, L::LDA, a.c + (size_t)(first + c0) * a.stride + (size_t)g * N, a.stride, min(CK_TOKENS, n - c0), N, a.vec);
        }
        ck_commit();
    };
    auto fetch_rest = [&](int chunk) {
        if (chunk < chunks) {
            const int c0 = chunk * CK_TOKENS, count = min(CK_TOKENS, n - c0);
            float* stage = ck_shared + L::STAGE + (chunk & 1) * L::STAGE_FLOATS;
            const size_t at = (size_t)(first + c0) * a.stride;
            ck_stage<NP, THREADS>(stage + L::B, NP, a.b + at + (size_t)g * N, a.stride, count, N, a.vec);
            ck_stage<TP, THREADS>(stage + L::X, L::LDX, a.x + at + (size_t)h * P + p0, a.stride, count, width, vec_x);
            ck_stage<CK_TOKENS, THREADS>(stage + L::M, CK_MLD, a.scores + ((size_t)(slot0 + chunk) * a.groups + g) * CK_TOKENS * CK_TOKENS, CK_TOKENS, CK_TOKENS, CK_TOKENS, true);
            const float* factors = a.factors + ((size_t)(slot0 + chunk) * a.heads + h) * CK_FACTORS;
            for (int e = threadIdx.x; e < CK_FACTORS / 4; e += THREADS) ck_copy16(stage + L::F + 4 * e, factors + 4 * e, true);
        }
        ck_commit();
    };
    fetch_rest(0);
    fetch_a(0);

    float* S = a.state + (((size_t)a.slots[b] * a.heads + h) * P + p0 + col) * N;
    unsigned long long s[NL][2];
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = srow + i < N && p0 + col + e < P ? S[(size_t)e * N + srow + i] : 0.0f;
        s[i][0] = ck_pair(v[0], v[1]);
        s[i][1] = ck_pair(v[2], v[3]);
        *reinterpret_cast<float4*>(Ss + (srow + i) * L::LDX + col) = make_float4(v[0], v[1], v[2], v[3]);
    }

    for (int chunk = 0; chunk < chunks; ++chunk) {
        float* stage = ck_shared + L::STAGE + (chunk & 1) * L::STAGE_FLOATS;
        const float* X = stage + L::X;
        float* M = stage + L::M;
        const float* F = stage + L::F;
        fetch_rest(chunk + 1);
        ck_wait<1>();
        __syncthreads();                                        // this chunk's numbers and the state are there

        // the decays into the scores, and the rows the update adds
        float odd = 0.0f;                                       // no longer zero: an x of the chunk is not finite
        {
            const int j = 4 * (threadIdx.x & 15), bj = j >> 3;
            const float4 v = *reinterpret_cast<const float4*>(F + CK_V + j);
#pragma unroll
            for (int k = 0; k < 16 * CK_TOKENS / THREADS; ++k) {
                const int i = (threadIdx.x >> 4) + THREADS / 16 * k, bi = i >> 3;
                float4* at = reinterpret_cast<float4*>(M + i * CK_MLD + j);
                float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (bi > bj) {
                    const float u = F[CK_U + i] * F[CK_BLOCKS + bi * 8 + bj];
                    f = make_float4(u * v.x, u * v.y, u * v.z, u * v.w);
                } else if (bi == bj) {
                    f = *reinterpret_cast<const float4*>(F + CK_DIAG + bi * 64 + (i & 7) * 8 + (j & 7));
                }
                if (bi >= bj) {                                 // what lies above is not read
                    const float4 m = *at;
                    *at = make_float4(m.x * f.x, m.y * f.y, m.z * f.z, m.w * f.w);
                } else {
                    *at = f;
                }
            }
            for (int e = threadIdx.x; e < CK_TOKENS * PL; e += THREADS) {
                const int t = e / PL, c = 4 * (e - t * PL);
                const float4 x = *reinterpret_cast<const float4*>(X + t * L::LDX + c);
                const float w = F[CK_W + t];
                odd += ck_not_finite(x);
                *reinterpret_cast<float4*>(XW + t * L::LDX + c) = make_float4(w * x.x, w * x.y, w * x.z, w * x.w);
            }
        }
        unsigned long long acc[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0ull;
        constexpr int K = NP / L::SLICES;
        ck_state_product<RL, K>(acc, As + row * L::LDA, L::LDA, Ss + col, L::LDX, slice * K);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float e = F[CK_E + row + RL * r];
            acc[r][0] = ck_pair(ck_lo(acc[r][0]) * e, ck_hi(acc[r][0]) * e);
            acc[r][1] = ck_pair(ck_lo(acc[r][1]) * e, ck_hi(acc[r][1]) * e);
        }
        const bool finite = !__syncthreads_or(odd != 0.0f);     // scores and weighted rows are written, C and the old state are read
        fetch_a(chunk + 1);
        if (finite) ck_product<RL>(acc, M + row * CK_MLD, CK_MLD, X + col, L::LDX, 4 * slice, 4 * L::SLICES, block * L::ROWS + L::ROWS);
        else ck_causal_product<RL>(acc, M + row * CK_MLD, CK_MLD, X + col, L::LDX, 4 * slice, 4 * L::SLICES, block * L::ROWS + L::ROWS, row);
        if (slice > 0) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                *reinterpret_cast<float4*>(ck_shared + L::PARTS + ((slice - 1) * CK_TOKENS + row + RL * r) * L::LDX + col) =
                    make_float4(ck_lo(acc[r][0]), ck_hi(acc[r][0]), ck_lo(acc[r][1]), ck_hi(acc[r][1]));
        }
        float4 own[4];                                          // added last, to the whole sum: one rounding at its size
#pragma unroll
        for (int r = 0; r < 4; ++r) own[r] = slice == 0 ? *reinterpret_cast<const float4*>(X + (row + RL * r) * L::LDX + col) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        // S <- e_63 S + B^T (w x)
        ck_update<NP, NL>(s, F[CK_ALL], stage + L::B + srow, XW + col, L::LDX);
#pragma unroll
        for (int i = 0; i < NL; ++i)
            *reinterpret_cast<float4*>(Ss + (srow + i) * L::LDX + col) = make_float4(ck_lo(s[i][0]), ck_hi(s[i][0]), ck_lo(s[i][1]), ck_hi(s[i][1]));
        __syncthreads();                                        // this stage may be filled again, the weighted rows be written again
        if (slice == 0)                                         // the other slices' sums are there: the chunk's outputs
            ck_outputs<RL, L::SLICES>(acc, ck_shared + L::PARTS, L::LDX, row, col, width, n - chunk * CK_TOKENS, vec_x, skip, own,
                                      a.y + (size_t)(first + chunk * CK_TOKENS) * inner + (size_t)h * P + p0, inner);
    }
    ck_wait<0>();
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        const float v[4] = {ck_lo(s[i][0]), ck_hi(s[i][0]), ck_lo(s[i][1]), ck_hi(s[i][1])};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (srow + i < N && p0 + col + e < P) S[(size_t)e * N + srow + i] = v[e];
    }
}

// on every launch: it holds for the current device alone, and an engine may run on any of the process's
template <typename Kernel>
static cudaError_t ck_allow(Kernel kernel, size_t bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); }

template <int NP, int TP>
static int scan_chunks_launch(const ScanChunks& a, int max_slots, cudaStream_t stream) {
    constexpr size_t prepare_bytes = (size_t)2 * CK_TOKENS * (NP + 4) * sizeof(float);
    cudaError_t code = ck_allow(scan_chunks_prepare_kernel<NP>, prepare_bytes);
    if (code == cudaSuccess) code = ck_allow(scan_chunks_kernel<NP, TP>, CkLayout<NP, TP>::BYTES);
    if (code != cudaSuccess) return (int)code;
    tt_launch_pdl(scan_chunks_prepare_kernel<NP>, dim3(max_slots, a.groups, (a.heads / a.groups + CK_WARPS - 1) / CK_WARPS), dim3(CK_THREADS), prepare_bytes, stream, a);
    tt_launch_pdl(scan_chunks_kernel<NP, TP>, dim3(a.heads, a.sequences, (a.P + TP - 1) / TP), dim3(CkLayout<NP, TP>::THREADS), CkLayout<NP, TP>::BYTES, stream, a);
    TT_LAUNCH_CHECK();
}

// rows: [tokens][width] with x, B and C from the given columns on (see ScanChunks).  max_slots: n_tokens / 64 + sequences.  scratch: so many
// times the scores of every group (64 * 64 numbers) and the factors of every head (CK_FACTORS), on a 16-byte boundary: the walk copies
// it in 16-byte pieces whatever the rows' alignment.  sms: the device's multiprocessors.
extern "C" int tt_scan_chunks(const float* rows, int width, int x_col, int b_col, int c_col, const float* proj, int splits, long long split_stride,
                              int cols, int dt_col, const float* dt_bias, const float* a_log, const float* d_skip, const float* fixed_decay, float* state,
                              float* y, float* scratch, const int* cu, const int* slots, int sequences, int max_slots, int heads,
                              int groups, int P, int N, int sms, cudaStream_t stream) {
    if (sequences <= 0 || max_slots <= 0) return 0;
    if (N <= 0 || N > 128 || P <= 0 || groups <= 0 || groups > 65535 || heads % groups || sequences > 65535) return (int)cudaErrorInvalidValue;
    if (!rows || !scratch || ((uintptr_t)scratch & 15) || (!fixed_decay && (!proj || !dt_bias || !a_log))) return (int)cudaErrorInvalidValue;
    const float *x = rows + x_col, *b = rows + b_col, *c = rows + c_col;
    float *scores = scratch, *factors = scratch + (size_t)max_slots * groups * CK_TOKENS * CK_TOKENS;
    const uintptr_t bases = (uintptr_t)x | (uintptr_t)b | (uintptr_t)c | (uintptr_t)y;
    const ScanChunks a{x, b, c, (size_t)width, proj, splits, cols, dt_col, (size_t)split_stride, dt_bias, a_log, d_skip, fixed_decay, state, y, scores, factors,
                       cu, slots, sequences, heads, groups, P, N, (bases & 15) == 0 && !(width & 3) && !(N & 3) && !(P & 3) ? 1 : 0};
    // 32 columns a CTA use a number of C twice; 16 where that grid would leave half of the SMs without one
    const bool narrow = (long long)heads * sequences * ((P + 31) / 32) * 2 <= sms + sms / 4;
    if (N <= 64) return narrow ? scan_chunks_launch<64, 16>(a, max_slots, stream) : scan_chunks_launch<64, 32>(a, max_slots, stream);
    return narrow ? scan_chunks_launch<128, 16>(a, max_slots, stream) : scan_chunks_launch<128, 32>(a, max_slots, stream);
}

// ------------------------------------------------------------------------------------------------------ the gated delta rule
//   q = q / |q| * scale, k = k / |k|;  S <- a_t S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t
// (lengths with 1e-6 under the root, scale = D^-1/2).  Inside a chunk that starts from state S
//   u_i = beta_i v_i - beta_i e_i S^T k_i - sum_(j<i) beta_i f(i, j) (k_i . k_j) u_j
// is a unit lower triangular system, (I + A) U = beta V - (beta e K) S, whose solution is U = U0 - W S with (I + A) U0 = beta V and
// (I + A) W = beta e K: neither needs the state, so the first kernel solves for both, parallel over chunks and heads, and the second
// walks the chunks with   U = U0 - W S,   o = e Q S + P U (P_ij = f(i, j) q_i . k_j, j <= i),   S <- e_63 S + (w K)^T U.
// Products and sums are float32 multiply-adds (lengths, and products of factors with scores, float64 rounded once: in float32 throughout the
// outputs were 14 % further from 64 bits than token by token, now 15 % closer, for 2 % of the time); the systems are solved by forward
// substitution, a column a thread.  16 heads of 128 x 128 on 4,097 tokens: 1,900 us token by token, now 486: the first kernel 130 (bound by issue and shared memory; two columns a thread and half the
// threads 229, the whole substitution unrolled 278), the second 345 (bound like the one above; the two products with the state,
// W S and Q S, take an operand of S from shared memory once for both: one after the other 408).
constexpr int CD_THREADS = 256;
constexpr int CD_E = 0, CD_W = 64, CD_ALL = 128, CD_FACTORS = 136;        // of a chunk and head, for the second kernel

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
    float* scratch;             // [slots][heads]: W [64][D], U0 [64][V], P [64][64], factors [CD_FACTORS]
    const int* cu;
    const int* slots;
    int sequences, heads, qk_heads, D, V, vec, vec_v;
    __host__ __device__ size_t chunk_floats() const { return (size_t)CK_TOKENS * (D + V + CK_TOKENS) + CD_FACTORS; }
    __device__ float* chunk_scratch(int slot, int h) const { return scratch + ((size_t)slot * heads + h) * chunk_floats(); }
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
    float* f = As + CK_TOKENS * CK_MLD;                         // [CK_FACTORS]
    double* nq = reinterpret_cast<double*>(f + CK_FACTORS);     // [64] each: D^-1/2 / |q|, 1 / |k|; then beta
    double* nk = nq + CK_TOKENS;
    float* beta = reinterpret_cast<float*>(nk + CK_TOKENS);
    float* scalars = beta + CK_TOKENS;                          // [2][64]; then the rows' factors of W's right-hand side
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
    if (D < NP) {
        for (int e = threadIdx.x; e < 2 * CK_TOKENS * LD; e += CD_THREADS) ck_shared[e] = 0.0f;
        __syncthreads();
    }
    const float* rows = a.qkv + (size_t)(first + c0) * a.stride;
    ck_stage<NP, CD_THREADS>(qs, LD, rows + (size_t)g * D, a.stride, count, D, a.vec);
    ck_stage<NP, CD_THREADS>(ks, LD, rows + (size_t)(a.qk_heads + g) * D, a.stride, count, D, a.vec);
    ck_commit();
    if (warp == 0) {
        float decay[2];
        const float neg_a = -expf(__ldg(a.a_log + h)), bias = __ldg(a.dt_bias + h);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = lane + 32 * half;
            const float* row = a.proj + (size_t)(first + c0 + i) * a.cols + h;
            decay[half] = 1.0f;
            float write = 0.0f;
            if (i < count) {
                const float raw = ck_sum_slices(row + a.a_col, a.splits, a.split_stride) + bias;
                decay[half] = expf(neg_a * (raw > 20.0f ? raw : log1pf(expf(raw))));
                write = 1.0f / (1.0f + expf(-ck_sum_slices(row + a.b_col, a.splits, a.split_stride)));
            }
            beta[i] = write;
        }
        ck_factors(f, decay[0], decay[1], 1.0f, 1.0f, lane, scalars, scalars + CK_TOKENS);
    }
    ck_wait<0>();
    __syncthreads();
    // lengths: four lanes a row
    for (int item = threadIdx.x >> 2; item < 2 * CK_TOKENS; item += CD_THREADS / 4) {
        const float* row = (item < CK_TOKENS ? qs : ks) + (item & (CK_TOKENS - 1)) * LD;
        double sum = 0.0;
        for (int c = threadIdx.x & 3; c < D; c += 4) sum = fma((double)row[c], (double)row[c], sum);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (!(threadIdx.x & 3)) (item < CK_TOKENS ? nq : nk)[item & (CK_TOKENS - 1)] = 1.0 / sqrt((sum + 1e-6) * (item < CK_TOKENS ? (double)D : 1.0));
    }
    __syncthreads();
    float* scratch = a.chunk_scratch(slot, h);
    float* P = scratch + (size_t)CK_TOKENS * (D + V);
    // k . k and q . k: 16 x 16 threads, rows and columns 16 apart
    {
        const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
        float kk[4][4], qk[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) kk[r][c] = qk[r][c] = 0.0f;
#pragma unroll 1
        for (int k0 = 0; k0 < NP; k0 += 32) {                   // sums of 8, added up to 32, added up: long chains lose more
            float hk[4][4], hq[4][4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) hk[r][c] = hq[r][c] = 0.0f;
#pragma unroll 1
            for (int k1 = k0; k1 < k0 + 32; k1 += 8) {
                float pk[4][4], pq[4][4];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) pk[r][c] = pq[r][c] = 0.0f;
#pragma unroll
                for (int k = k1; k < k1 + 8; k += 4) {
                    float4 b[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(ks + (tx + 16 * c) * LD + k);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float4 x = *reinterpret_cast<const float4*>(ks + (ty + 16 * r) * LD + k), y = *reinterpret_cast<const float4*>(qs + (ty + 16 * r) * LD + k);
#pragma unroll
                        for (int c = 0; c <= r; ++c) {              // the others lie above the diagonal
                            pk[r][c] = fmaf(x.x, b[c].x, pk[r][c]); pk[r][c] = fmaf(x.y, b[c].y, pk[r][c]);
                            pk[r][c] = fmaf(x.z, b[c].z, pk[r][c]); pk[r][c] = fmaf(x.w, b[c].w, pk[r][c]);
                            pq[r][c] = fmaf(y.x, b[c].x, pq[r][c]); pq[r][c] = fmaf(y.y, b[c].y, pq[r][c]);
                            pq[r][c] = fmaf(y.z, b[c].z, pq[r][c]); pq[r][c] = fmaf(y.w, b[c].w, pq[r][c]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c <= r; ++c) { hk[r][c] += pk[r][c]; hq[r][c] += pq[r][c]; }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c <= r; ++c) { kk[r][c] += hk[r][c]; qk[r][c] += hq[r][c]; }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = ty + 16 * r, bi = i >> 3;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = tx + 16 * c, bj = j >> 3;
                if (c > r) {
                    As[i * CK_MLD + j] = P[i * CK_TOKENS + j] = 0.0f;
                    continue;
                }
                // products of the factors in float64, rounded once
                const double fij = bi > bj ? (double)f[CK_U + i] * (double)f[CK_BLOCKS + bi * 8 + bj] * (double)f[CK_V + j] : bi == bj ? (double)f[CK_DIAG + bi * 64 + (i & 7) * 8 + (j & 7)] : 0.0;
                const double fk = fij * nk[j];
                As[i * CK_MLD + j] = j < i ? -(float)((double)beta[i] * nk[i] * fk * (double)kk[r][c]) : 0.0f;         // -A
                P[i * CK_TOKENS + j] = j <= i ? (float)(nq[i] * fk * (double)qk[r][c]) : 0.0f;
            }
        }
    }
    if (threadIdx.x < CK_TOKENS) {
        float* factors = P + CK_TOKENS * CK_TOKENS;
        factors[CD_E + threadIdx.x] = (float)((double)f[CK_E + threadIdx.x] * nq[threadIdx.x]);
        factors[CD_W + threadIdx.x] = (float)((double)f[CK_W + threadIdx.x] * nk[threadIdx.x]);
        scalars[threadIdx.x] = (float)((double)beta[threadIdx.x] * (double)f[CK_E + threadIdx.x] * nk[threadIdx.x]);
        if (threadIdx.x == 0) factors[CD_ALL] = f[CK_ALL];
    }
    __syncthreads();
    // (I + A) x = r for the columns of beta e K (made W) and of beta V (made U0), one a thread, 16 rows at a time: what the rows
    // before contribute as a product (sums of 16 added up), then the triangle of the 16.  Half of the CTA takes the keys'
    // columns, in place, and every second tile of NP value columns; the other half the other tiles, where the queries lay.
    const int half = threadIdx.x / (CD_THREADS / 2), col = threadIdx.x % (CD_THREADS / 2);
    float* xs = (half ? qs : ks) + col;
    const float* values = rows + (size_t)2 * a.qk_heads * D + (size_t)h * V;
    for (int job = half; (job - 1) * NP < V; job += 2) {       // job 0: the keys; job t: value columns from (t - 1) * NP on
        const int c = (job ? (job - 1) * NP : 0) + col, width = job ? V : D;
        if (col >= NP || c >= width) continue;
        float* to = scratch + (job ? (size_t)CK_TOKENS * D : 0) + c;
        float raw[16];                                          // the next 16 rows' values, fetched ahead
        auto fetch = [&](int i0) {
            if (!job) return;
#pragma unroll
            for (int r = 0; r < 16; ++r) raw[r] = i0 + r < count ? __ldg(values + (size_t)(i0 + r) * a.stride + c) : 0.0f;
        };
        fetch(0);
#pragma unroll 1
        for (int i0 = 0; i0 < CK_TOKENS; i0 += 16) {
            // the right-hand side, and what the rows before take off it, summed apart: many small terms added to x one by one would each round it
            float x[16], before[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = i0 + r;
                before[r] = 0.0f;
                x[r] = job ? beta[i] * raw[r] : scalars[i] * xs[i * LD];
            }
            if (i0 + 16 < CK_TOKENS) fetch(i0 + 16);
#pragma unroll 1
            for (int j0 = 0; j0 < i0; j0 += 16) {
                float sum[16];
#pragma unroll
                for (int r = 0; r < 16; ++r) sum[r] = 0.0f;
#pragma unroll
                for (int j = j0; j < j0 + 16; j += 4) {
                    float y[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[e] = xs[(j + e) * LD];
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const float4 m = *reinterpret_cast<const float4*>(As + (i0 + r) * CK_MLD + j);
                        sum[r] = fmaf(m.x, y[0], sum[r]);
                        sum[r] = fmaf(m.y, y[1], sum[r]);
                        sum[r] = fmaf(m.z, y[2], sum[r]);
                        sum[r] = fmaf(m.w, y[3], sum[r]);
                    }
                }
#pragma unroll
                for (int r = 0; r < 16; ++r) before[r] += sum[r];
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
                to[(size_t)(i0 + r) * width] = x[r];
            }
        }
    }
}

template <int NP, int TP>
struct CdLayout {
    using L = CkLayout<NP, TP>;                                 // lanes, rows and slices as above
    static constexpr int LDA = L::LDA, LDX = L::LDX;
    static constexpr int Q = 0, W = Q + CK_TOKENS * LDA, S = W + CK_TOKENS * LDA, XW = S + NP * LDX, PARTS = XW + CK_TOKENS * LDX;
    static constexpr int STAGE = PARTS + (L::SLICES - 1) * CK_TOKENS * LDX;
    static constexpr int K = 0, X = K + CK_TOKENS * NP, M = X + CK_TOKENS * LDX, F = M + CK_TOKENS * CK_MLD, STAGE_FLOATS = F + CD_FACTORS;
    static constexpr size_t BYTES = (size_t)(STAGE + 2 * STAGE_FLOATS) * sizeof(float);
};

template <int NP, int TP>
__global__ void __launch_bounds__(CK_THREADS, 1)
delta_chunks_kernel(const DeltaChunks a) {
    using D_ = CdLayout<NP, TP>;
    using L = CkLayout<NP, TP>;
    constexpr int PL = L::PL, RL = L::RL, ROW_BLOCKS = CK_TOKENS / L::ROWS, SLICE_K = NP / L::SLICES;
    constexpr int NL = NP * TP / (CK_THREADS * 4);              // state rows of a lane
    extern __shared__ __align__(16) float ck_shared[];
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int h = blockIdx.x, b = blockIdx.y, p0 = blockIdx.z * TP;
    const int first = a.cu[b], n = a.cu[b + 1] - first;
    if (n <= 0) return;
    const int g = h / (a.heads / a.qk_heads), V = a.V, D = a.D;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = 4 * (lane % PL), width = min(TP, V - p0);
    const int slice = warp / ROW_BLOCKS, block = (warp + (warp >> 2)) % ROW_BLOCKS;
    const int row = block * L::ROWS + lane / PL;
    const int srow = warp * (NP / CK_WARPS) + (lane / PL) * NL;
    float* Qs = ck_shared + D_::Q;
    float* Ws = ck_shared + D_::W;
    float* Ss = ck_shared + D_::S;
    float* XW = ck_shared + D_::XW;
    const int chunks = (n + CK_TOKENS - 1) / CK_TOKENS, slot0 = ck_first_slot(a.cu, b);
    const bool vec_x = a.vec_v && (width & 3) == 0;

    for (int e = threadIdx.x; e < D_::STAGE + 2 * D_::STAGE_FLOATS; e += CK_THREADS) ck_shared[e] = 0.0f;
    __syncthreads();
    auto fetch_first = [&](int chunk) {                         // what meets the state: q and W
        if (chunk < chunks) {
            const int c0 = chunk * CK_TOKENS;
            ck_stage<NP>(Qs, D_::LDA, a.qkv + (size_t)(first + c0) * a.stride + (size_t)g * D, a.stride, min(CK_TOKENS, n - c0), D, a.vec);
            ck_stage<NP>(Ws, D_::LDA, a.chunk_scratch(slot0 + chunk, h), D, CK_TOKENS, D, !(D & 3));
        }
        ck_commit();
    };
    auto fetch_rest = [&](int chunk) {
        if (chunk < chunks) {
            const int c0 = chunk * CK_TOKENS;
            float* stage = ck_shared + D_::STAGE + (chunk & 1) * D_::STAGE_FLOATS;
            const float* scratch = a.chunk_scratch(slot0 + chunk, h);
            ck_stage<NP>(stage + D_::K, NP, a.qkv + (size_t)(first + c0) * a.stride + (size_t)(a.qk_heads + g) * D, a.stride, min(CK_TOKENS, n - c0), D, a.vec);
            ck_stage<TP>(stage + D_::X, D_::LDX, scratch + (size_t)CK_TOKENS * D + p0, V, CK_TOKENS, width, vec_x);
            const float* P = scratch + (size_t)CK_TOKENS * (D + V);
            ck_stage<CK_TOKENS>(stage + D_::M, CK_MLD, P, CK_TOKENS, CK_TOKENS, CK_TOKENS, true);
            for (int e = threadIdx.x; e < CD_FACTORS / 4; e += CK_THREADS) ck_copy16(stage + D_::F + 4 * e, P + CK_TOKENS * CK_TOKENS + 4 * e, true);
        }
        ck_commit();
    };
    fetch_rest(0);
    fetch_first(0);

    float* S = a.state + (((size_t)a.slots[b] * a.heads + h) * V + p0 + col) * D;
    unsigned long long s[NL][2];
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = srow + i < D && p0 + col + e < V ? S[(size_t)e * D + srow + i] : 0.0f;
        s[i][0] = ck_pair(v[0], v[1]);
        s[i][1] = ck_pair(v[2], v[3]);
        *reinterpret_cast<float4*>(Ss + (srow + i) * D_::LDX + col) = make_float4(v[0], v[1], v[2], v[3]);
    }

    for (int chunk = 0; chunk < chunks; ++chunk) {
        float* stage = ck_shared + D_::STAGE + (chunk & 1) * D_::STAGE_FLOATS;
        float* X = stage + D_::X;
        const float* M = stage + D_::M;
        const float* F = stage + D_::F;
        fetch_rest(chunk + 1);
        ck_wait<1>();
        __syncthreads();                                        // this chunk's numbers and the state are there
        unsigned long long acc[4][2], ws[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = ws[r][0] = ws[r][1] = 0ull;
        ck_two_products<RL, SLICE_K>(ws, Ws + row * D_::LDA, acc, Qs + row * D_::LDA, D_::LDA, Ss + col, D_::LDX, slice * SLICE_K);
        {                                                       // W S: the first slice's sums lie where the weighted rows will
            float* to = slice == 0 ? XW : ck_shared + D_::PARTS + (slice - 1) * CK_TOKENS * D_::LDX;
#pragma unroll
            for (int r = 0; r < 4; ++r)
                *reinterpret_cast<float4*>(to + (row + RL * r) * D_::LDX + col) = make_float4(ck_lo(ws[r][0]), ck_hi(ws[r][0]), ck_lo(ws[r][1]), ck_hi(ws[r][1]));
        }
        __syncthreads();                                        // W S is whole; q, W and the old state are read
        fetch_first(chunk + 1);
        float odd = 0.0f;                                       // no longer zero: a number of U is not finite
        for (int e = threadIdx.x; e < CK_TOKENS * PL; e += CK_THREADS) {           // U = U0 - W S, and the rows the update adds
            const int t = e / PL, c = 4 * (e % PL);
            float4 u = *reinterpret_cast<const float4*>(X + t * D_::LDX + c);
            float4 ws = *reinterpret_cast<const float4*>(XW + t * D_::LDX + c);
#pragma unroll
            for (int k = 0; k < L::SLICES - 1; ++k) {
                const float4 q = *reinterpret_cast<const float4*>(ck_shared + D_::PARTS + (k * CK_TOKENS + t) * D_::LDX + c);
                ws.x += q.x; ws.y += q.y; ws.z += q.z; ws.w += q.w;
            }
            u.x -= ws.x; u.y -= ws.y; u.z -= ws.z; u.w -= ws.w;
            const float w = F[CD_W + t];
            odd += ck_not_finite(u);
            *reinterpret_cast<float4*>(X + t * D_::LDX + c) = u;
            *reinterpret_cast<float4*>(XW + t * D_::LDX + c) = make_float4(w * u.x, w * u.y, w * u.z, w * u.w);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float e = F[CD_E + row + RL * r];
            acc[r][0] = ck_pair(ck_lo(acc[r][0]) * e, ck_hi(acc[r][0]) * e);
            acc[r][1] = ck_pair(ck_lo(acc[r][1]) * e, ck_hi(acc[r][1]) * e);
        }
        const bool finite = !__syncthreads_or(odd != 0.0f);     // U is there
        if (finite) ck_product<RL>(acc, M + row * CK_MLD, CK_MLD, X + col, D_::LDX, 4 * slice, 4 * L::SLICES, block * L::ROWS + L::ROWS);
        else ck_causal_product<RL>(acc, M + row * CK_MLD, CK_MLD, X + col, D_::LDX, 4 * slice, 4 * L::SLICES, block * L::ROWS + L::ROWS, row);
        if (slice > 0) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                *reinterpret_cast<float4*>(ck_shared + D_::PARTS + ((slice - 1) * CK_TOKENS + row + RL * r) * D_::LDX + col) =
                    make_float4(ck_lo(acc[r][0]), ck_hi(acc[r][0]), ck_lo(acc[r][1]), ck_hi(acc[r][1]));
        }
        const float all = F[CD_ALL];
        ck_update<NP, NL>(s, all, stage + D_::K + srow, XW + col, D_::LDX);
#pragma unroll
        for (int i = 0; i < NL; ++i)
            *reinterpret_cast<float4*>(Ss + (srow + i) * D_::LDX + col) = make_float4(ck_lo(s[i][0]), ck_hi(s[i][0]), ck_lo(s[i][1]), ck_hi(s[i][1]));
        __syncthreads();
        if (slice == 0)
            ck_outputs<RL, L::SLICES>(acc, ck_shared + D_::PARTS, D_::LDX, row, col, width, n - chunk * CK_TOKENS, vec_x, 0.0f, nullptr,
                                      a.out + (size_t)(first + chunk * CK_TOKENS) * (a.heads * V) + (size_t)h * V + p0, a.heads * V);
    }
    ck_wait<0>();
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        const float v[4] = {ck_lo(s[i][0]), ck_hi(s[i][0]), ck_lo(s[i][1]), ck_hi(s[i][1])};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (srow + i < D && p0 + col + e < V) S[(size_t)e * D + srow + i] = v[e];
    }
}

template <int NP, int TP>
static int delta_chunks_launch(const DeltaChunks& a, int max_slots, cudaStream_t stream) {
    constexpr size_t prepare_bytes = (size_t)(2 * CK_TOKENS * (NP + 4) + CK_TOKENS * CK_MLD + CK_FACTORS + 7 * CK_TOKENS) * sizeof(float);
    cudaError_t code = ck_allow(delta_chunks_prepare_kernel<NP>, prepare_bytes);
    if (code == cudaSuccess) code = ck_allow(delta_chunks_kernel<NP, TP>, CdLayout<NP, TP>::BYTES);
    if (code != cudaSuccess) return (int)code;
    tt_launch_pdl(delta_chunks_prepare_kernel<NP>, dim3(max_slots, a.heads), dim3(CD_THREADS), prepare_bytes, stream, a);
    tt_launch_pdl(delta_chunks_kernel<NP, TP>, dim3(a.heads, a.sequences, (a.V + TP - 1) / TP), dim3(CK_THREADS), CdLayout<NP, TP>::BYTES, stream, a);
    TT_LAUNCH_CHECK();
}

// scratch: max_slots * heads * (64 * (D + V + 64) + CD_FACTORS) floats on a 16-byte boundary; max_slots as for tt_scan_chunks
extern "C" int tt_delta_chunks(const float* qkv, int qkv_cols, const float* proj, int splits, long long split_stride, int cols, int b_col, int a_col,
                               const float* dt_bias, const float* a_log, float* state, float* out, float* scratch, const int* cu, const int* slots,
                               int sequences, int max_slots, int heads, int qk_heads, int D, int V, int sms, cudaStream_t stream) {
    if (sequences <= 0 || max_slots <= 0) return 0;
    if (D <= 0 || D > 128 || V <= 0 || qk_heads <= 0 || heads % qk_heads || heads > 65535 || sequences > 65535) return (int)cudaErrorInvalidValue;
    if (!qkv || !proj || !dt_bias || !a_log || !scratch || ((uintptr_t)scratch & 15)) return (int)cudaErrorInvalidValue;
    const int vec = ((uintptr_t)qkv & 15) == 0 && !(qkv_cols & 3) && !(D & 3);
    const DeltaChunks a{qkv, (size_t)qkv_cols, proj, splits, cols, b_col, a_col, (size_t)split_stride, dt_bias, a_log, state, out, scratch, cu, slots,
                        sequences, heads, qk_heads, D, V, vec, ((uintptr_t)out & 15) == 0 && !(V & 3) ? 1 : 0};
    const bool narrow = (long long)heads * sequences * ((V + 31) / 32) * 2 <= sms + sms / 4;        // as for tt_scan_chunks
    if (D <= 64) return narrow ? delta_chunks_launch<64, 16>(a, max_slots, stream) : delta_chunks_launch<64, 32>(a, max_slots, stream);
    return narrow ? delta_chunks_launch<128, 16>(a, max_slots, stream) : delta_chunks_launch<128, 32>(a, max_slots, stream);
}
