// Recurrences with one decay per head and token, for prompts: a chunk of 64 tokens at a time.
//
//   S_t = a_t S_(t-1) + dt_t B_t x_t^T,   y_t = S_t^T C_t + D x_t        (S: N x P per head; Mamba-2, and with a constant
//                                                                          decay and dt = 1 linear attention: B = k, C = q, x = v)
//
// With f(i, j) = a_(j+1) * .. * a_i, e_i = a_0 * .. * a_i and w_j = f(63, j) dt_j, a chunk that starts from state S gives
//   y_i = e_i (S^T C_i) + sum_(j<=i) f(i, j) dt_j (C_i . B_j) x_j + D x_i,     S <- e_63 S + sum_j w_j B_j x_j^T
// so the token-by-token chain of row products becomes four matrix products a chunk, all of them float32 multiply-adds.  The
// decays only ever enter as products of decays (never as quotients, never as differences of sums of logarithms): nothing can
// overflow that does not overflow in the recurrence, nothing cancels, and a constant decay may have any sign.  The products are
// formed in float64 from the float32 decays and rounded once.
//
// Two kernels.  The first, parallel over chunks, makes what the columns of a head share: G_ij = C_i . B_j for every chunk and
// group, and the factors of every chunk and head (u, v, E, diagonal blocks: f(i, j) is a product of three numbers across
// 8-token blocks, and is stored inside one).  The second walks a sequence's chunks with the state of TP columns of one head in
// registers (256 threads) and, for the products that read it, in shared memory.
//
// What bounds it: shared memory's delivery of operands and the latency of two warps a scheduler (one CTA of 8 warps an SM; the
// multiply-add pipe is 43 % busy); the copies of the next chunk run under this one's products.  16 warps with half the registers
// spilled and were slower (348 against 227 us at the first size below), rows of operands used for two instead of four outputs
// too (305).  Against the kernels that go token by token, whose chain of row products a token bounds them (us, one B200): 64 heads of
// 64 x 128, one sequence of 2,048 tokens 895 -> 228, four of 731 545 -> 332; 16 heads of 256 x 128, four of 1,024 740 -> 455.
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
__global__ void __launch_bounds__(CK_THREADS)
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
    float total[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) total[i][j] = 0.0f;
    for (int k0 = 0; k0 < NP; k0 += 32) {                       // short sums, added up: a long chain of additions loses more
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 4
        for (int k = k0; k < k0 + 32; k += 4) {
            float4 c[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                c[i] = *reinterpret_cast<const float4*>(cs + (ty + 16 * i) * LD + k);
                b[i] = *reinterpret_cast<const float4*>(bs + (tx + 16 * i) * LD + k);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {                  // columns behind the row's block are not used
                    acc[i][j] = fmaf(c[i].x, b[j].x, acc[i][j]);
                    acc[i][j] = fmaf(c[i].y, b[j].y, acc[i][j]);
                    acc[i][j] = fmaf(c[i].z, b[j].z, acc[i][j]);
                    acc[i][j] = fmaf(c[i].w, b[j].w, acc[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) total[i][j] += acc[i][j];
    }
    float* out = a.scores + ((size_t)slot * a.groups + g) * CK_TOKENS * CK_TOKENS;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[(ty + 16 * i) * CK_TOKENS + tx + 16 * j] = j <= i ? total[i][j] : 0.0f;
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
                *reinterpret_cast<float4*>(XW + t * L::LDX + c) = make_float4(w * x.x, w * x.y, w * x.z, w * x.w);
            }
        }
        unsigned long long acc[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0ull;
        constexpr int K = NP / L::SLICES;
        ck_product<RL>(acc, As + row * L::LDA, L::LDA, Ss + col, L::LDX, slice * K, 4, slice * K + K);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float e = F[CK_E + row + RL * r];
            acc[r][0] = ck_pair(ck_lo(acc[r][0]) * e, ck_hi(acc[r][0]) * e);
            acc[r][1] = ck_pair(ck_lo(acc[r][1]) * e, ck_hi(acc[r][1]) * e);
        }
        __syncthreads();                                        // scores and weighted rows are written, C and the old state are read
        fetch_a(chunk + 1);
        ck_product<RL>(acc, M + row * CK_MLD, CK_MLD, X + col, L::LDX, 4 * slice, 4 * L::SLICES, block * L::ROWS + L::ROWS);
        if (slice > 0) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                *reinterpret_cast<float4*>(ck_shared + L::PARTS + ((slice - 1) * CK_TOKENS + row + RL * r) * L::LDX + col) =
                    make_float4(ck_lo(acc[r][0]), ck_hi(acc[r][0]), ck_lo(acc[r][1]), ck_hi(acc[r][1]));
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float4 x = *reinterpret_cast<const float4*>(X + (row + RL * r) * L::LDX + col);
                acc[r][0] = ck_pair(fmaf(skip, x.x, ck_lo(acc[r][0])), fmaf(skip, x.y, ck_hi(acc[r][0])));
                acc[r][1] = ck_pair(fmaf(skip, x.z, ck_lo(acc[r][1])), fmaf(skip, x.w, ck_hi(acc[r][1])));
            }
        }
        // S <- e_63 S + B^T (w x)
        const float all = F[CK_ALL];
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            s[i][0] = ck_pair(ck_lo(s[i][0]) * all, ck_hi(s[i][0]) * all);
            s[i][1] = ck_pair(ck_lo(s[i][1]) * all, ck_hi(s[i][1]) * all);
        }
        const float* B = stage + L::B + srow;
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
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(XW + j * L::LDX + col);
#pragma unroll
            for (int i = 0; i < NL; ++i) {
                const unsigned long long twice = ck_pair(bv[i], bv[i]);
                ck_fma2(s[i][0], twice, x.x);
                ck_fma2(s[i][1], twice, x.y);
            }
        }
#pragma unroll
        for (int i = 0; i < NL; ++i)
            *reinterpret_cast<float4*>(Ss + (srow + i) * L::LDX + col) = make_float4(ck_lo(s[i][0]), ck_hi(s[i][0]), ck_lo(s[i][1]), ck_hi(s[i][1]));
        __syncthreads();                                        // this stage may be filled again, the weighted rows be written again
        if (slice == 0) {                                       // the other slices' sums are there: the chunk's outputs
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = row + RL * r, t = chunk * CK_TOKENS + i;
                float o[4] = {ck_lo(acc[r][0]), ck_hi(acc[r][0]), ck_lo(acc[r][1]), ck_hi(acc[r][1])};
#pragma unroll
                for (int k = 0; k < L::SLICES - 1; ++k) {
                    const float4 q = *reinterpret_cast<const float4*>(ck_shared + L::PARTS + (k * CK_TOKENS + i) * L::LDX + col);
                    o[0] += q.x; o[1] += q.y; o[2] += q.z; o[3] += q.w;
                }
                if (t >= n || col >= width) continue;
                float* to = a.y + (size_t)(first + t) * inner + (size_t)h * P + p0 + col;
                if (vec_x) {
                    *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (col + e < width) to[e] = o[e];
                }
            }
        }
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

template <typename Kernel>
static cudaError_t ck_allow(Kernel kernel, size_t bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); }

template <int NP, int TP>
static int scan_chunks_launch(const ScanChunks& a, int max_slots, cudaStream_t stream) {
    constexpr size_t prepare_bytes = (size_t)2 * CK_TOKENS * (NP + 4) * sizeof(float);
    static bool allowed = false;
    if (!allowed) {
        cudaError_t code = ck_allow(scan_chunks_prepare_kernel<NP>, prepare_bytes);
        if (code == cudaSuccess) code = ck_allow(scan_chunks_kernel<NP, TP>, CkLayout<NP, TP>::BYTES);
        if (code != cudaSuccess) return (int)code;
        allowed = true;
    }
    tt_launch_pdl(scan_chunks_prepare_kernel<NP>, dim3(max_slots, a.groups, (a.heads / a.groups + CK_WARPS - 1) / CK_WARPS), dim3(CK_THREADS), prepare_bytes, stream, a);
    tt_launch_pdl(scan_chunks_kernel<NP, TP>, dim3(a.heads, a.sequences, (a.P + TP - 1) / TP), dim3(CkLayout<NP, TP>::THREADS), CkLayout<NP, TP>::BYTES, stream, a);
    TT_LAUNCH_CHECK();
}

// x, b, c: rows of `stride` numbers (see ScanChunks).  max_slots: n_tokens / 64 + sequences (scratch for scores and factors holds as many).
// sms: the device's multiprocessors.
extern "C" int tt_scan_chunks(const float* x, const float* b, const float* c, long long stride, const float* proj, int splits, long long split_stride,
                              int cols, int dt_col, const float* dt_bias, const float* a_log, const float* d_skip, const float* fixed_decay, float* state,
                              float* y, float* scores, float* factors, const int* cu, const int* slots, int sequences, int max_slots, int heads,
                              int groups, int P, int N, int sms, cudaStream_t stream) {
    if (sequences <= 0 || max_slots <= 0) return 0;
    if (N <= 0 || N > 128 || P <= 0 || groups <= 0 || groups > 65535 || heads % groups || sequences > 65535) return (int)cudaErrorInvalidValue;
    if (!fixed_decay && (!proj || !dt_bias || !a_log)) return (int)cudaErrorInvalidValue;
    const uintptr_t bases = (uintptr_t)x | (uintptr_t)b | (uintptr_t)c | (uintptr_t)y;
    const ScanChunks a{x, b, c, (size_t)stride, proj, splits, cols, dt_col, (size_t)split_stride, dt_bias, a_log, d_skip, fixed_decay, state, y, scores, factors,
                       cu, slots, sequences, heads, groups, P, N, (bases & 15) == 0 && !(stride & 3) && !(N & 3) && !(P & 3) ? 1 : 0};
    // 32 columns a CTA use a number of C twice; 16 where that grid would leave half of the SMs without one
    const bool narrow = (long long)heads * sequences * ((P + 31) / 32) * 2 <= sms + sms / 4;
    if (N <= 64) return narrow ? scan_chunks_launch<64, 16>(a, max_slots, stream) : scan_chunks_launch<64, 32>(a, max_slots, stream);
    return narrow ? scan_chunks_launch<128, 16>(a, max_slots, stream) : scan_chunks_launch<128, 32>(a, max_slots, stream);
}
