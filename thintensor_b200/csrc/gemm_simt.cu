// out[s][m][n] = sum over the s-th slice of k of x[m][k] * w[n][k]  (+ bias[n] in s = 0)
//
// The exact matrix product: float32 FMA on CUDA cores, no tensor-core mode of any
// kind, float32 or bfloat16 operands widened exactly.  It is the product of the true
// 32-bit path, the oracle of the tensor-core kernel in tests, and what a bfloat16 model
// falls back to for a weight that its checkpoint stores in float32.  Any m, n, k.
//
// Weights are [out_features, in_features] row-major as checkpoints store them and are
// applied as W x, like torch.mv(W, x) at thinruntime/gpu_runtime.py:10112; the Triton
// counterparts are _matvec_kernel / _matvec_looped_kernel / _matvec_split_k_kernel,
// thinruntime/triton_kernels.py:484-535, 2959-2986, 3022-3083.
#include "common.cuh"

// Tiles of 64 x 128 outputs by 128 threads, an 8 x 8 square of outputs in each thread's registers, so that an operand number
// read from shared memory serves eight multiply-adds; two shared-memory stages of 16 k, the next stage's numbers on their way
// from global memory while this one is multiplied.  Neighbouring outputs of a row are one packed instruction (two multiply-adds,
// each rounded as ever): no faster on the FMA pipe, but half the instructions, and the form with single ones lost a sixth of its
// issue slots to register conflicts.  Warps whose 32 rows all lie behind m skip the arithmetic.  Bound by issue: 1,000 x 4,096 x
// 4,096 runs at 51 TFLOP/s of the pipe's 74 (single multiply-adds on stages filled by asynchronous copies: 43).  4 x 4 outputs a
// thread and one stage, the form before, was bound by shared memory and the loads' latency: at 193 rows 16,384 features of 2,048 took
// 695 us against 334 (in 4 slices of k), 2,048 of 8,192 574 against 203 (8 slices), 3,072 of 2,048 216 against 72 (6 slices).
constexpr int GS_BM = 64, GS_BK = 16, GS_THREADS = 128;
constexpr int GS_XLD = GS_BM + 4;

__device__ __forceinline__ void gs_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// four neighbouring numbers, widened; vec: they lie on a boundary of their own size
__device__ __forceinline__ void gs_load4(float (&v)[4], const float* p, int count, bool vec) {
    if (vec && count == 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = e < count ? __ldg(p + e) : 0.0f;
    }
}
__device__ __forceinline__ void gs_load4(float (&v)[4], const __nv_bfloat16* p, int count, bool vec) {
    if (vec && count == 4) {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
        v[0] = __uint_as_float(q.x << 16); v[1] = __uint_as_float(q.x & 0xffff0000u);
        v[2] = __uint_as_float(q.y << 16); v[3] = __uint_as_float(q.y & 0xffff0000u);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = e < count ? __bfloat162float(p[e]) : 0.0f;
    }
}

// The same as they lie in memory, for the tiles, which widen them where they go to shared memory: widened at once, a load was waited for before
// the next was asked for.
template <typename T> struct GsFour;
template <> struct GsFour<float> {
    float4 q;
    __device__ __forceinline__ void load(const float* p, int count, bool vec) {
        if (vec && count == 4) q = __ldg(reinterpret_cast<const float4*>(p));
        else q = make_float4(count > 0 ? __ldg(p) : 0.0f, count > 1 ? __ldg(p + 1) : 0.0f, count > 2 ? __ldg(p + 2) : 0.0f, count > 3 ? __ldg(p + 3) : 0.0f);
    }
    __device__ __forceinline__ float at(int e) const { return e == 0 ? q.x : e == 1 ? q.y : e == 2 ? q.z : q.w; }
};
template <> struct GsFour<__nv_bfloat16> {
    uint2 q;
    __device__ __forceinline__ void load(const __nv_bfloat16* p, int count, bool vec) {
        if (vec && count == 4) {
            q = __ldg(reinterpret_cast<const uint2*>(p));
        } else {
            const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
            const unsigned a = count > 0 ? __ldg(h) : 0u, b = count > 1 ? __ldg(h + 1) : 0u, c = count > 2 ? __ldg(h + 2) : 0u, d = count > 3 ? __ldg(h + 3) : 0u;
            q = make_uint2(a | b << 16, c | d << 16);
        }
    }
    __device__ __forceinline__ float at(int e) const { const unsigned w = e < 2 ? q.x : q.y; return __uint_as_float(e & 1 ? w & 0xffff0000u : w << 16); }
};

// BN: the tile's columns, 128 or, for grids that leave SMs without a tile anyway, 64 (8 x 4 outputs a thread).
template <typename TX, typename TW, int BN>
__global__ void __launch_bounds__(GS_THREADS)
gemm_simt_kernel(const TX* __restrict__ x, long long ldx, const TW* __restrict__ w, long long ldw,
                 const float* __restrict__ bias, float* __restrict__ out, long long ldo, long long split_stride,
                 int m, int n, int k, int k_per_split, int vec_x, int vec_w, int vec_o) {
    __shared__ __align__(16) float xs[2][GS_BK][GS_XLD];
    __shared__ __align__(16) float ws[2][GS_BK][BN + 4];
    constexpr int COLS = BN / 32, WP = BN / 32;                  // packed columns of a thread; its pieces of w
    tt_pdl_launch_dependents();
    const int m0 = blockIdx.y * GS_BM, n0 = blockIdx.x * BN;
    const int split = blockIdx.z;
    const int k_begin = split * k_per_split;
    const int k_end = min(k, k_begin + k_per_split);
    // warps 2 x 2 over the tile (32 rows x half of the columns each), lanes 4 x 8; a thread's rows are two runs of four 16 apart, its
    // columns one or two runs of four 32 apart, so that the lanes' 16-byte reads lie side by side
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = (warp >> 1) * 32 + (lane >> 3) * 4, col = (warp & 1) * (BN / 2) + (lane & 7) * 4;
    const bool busy = m0 + (warp >> 1) * 32 < m;
    unsigned long long acc[8][COLS];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[i][j] = 0ull;

    // piece i of a thread: row (threadIdx.x + i * 128) / 4 of the operand's tile, four k from 4 * (threadIdx.x % 4)
    const int load_row = threadIdx.x >> 2, load_k = (threadIdx.x & 3) * 4;
    GsFour<TX> xr[2];
    GsFour<TW> wr[WP];
    auto fetch = [&](int kk) {
        const int count = max(0, min(4, k_end - kk - load_k));
#pragma unroll
        for (int i = 0; i < WP; ++i) {
            const int gn = n0 + load_row + 32 * i;
            wr[i].load(w + (size_t)gn * ldw + kk + load_k, gn < n ? count : 0, vec_w);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int gm = m0 + load_row + 32 * i;
            xr[i].load(x + (size_t)gm * ldx + kk + load_k, gm < m ? count : 0, vec_x);
        }
    };
    auto put = [&](int stage) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int i = 0; i < 2; ++i) xs[stage][load_k + e][load_row + 32 * i] = xr[i].at(e);
#pragma unroll
            for (int i = 0; i < WP; ++i) ws[stage][load_k + e][load_row + 32 * i] = wr[i].at(e);
        }
    };
    tt_pdl_wait();                                              // before either operand: a caller's weights may be fresh
    fetch(k_begin);
    put(0);
    __syncthreads();
    int stage = 0;
    for (int kk = k_begin; kk < k_end; kk += GS_BK, stage ^= 1) {
        const bool more = kk + GS_BK < k_end;
        if (more) fetch(kk + GS_BK);
        if (busy) {
#pragma unroll
            for (int e = 0; e < GS_BK; ++e) {
                const float4 a0 = *reinterpret_cast<const float4*>(&xs[stage][e][row]), a1 = *reinterpret_cast<const float4*>(&xs[stage][e][row + 16]);
                ulonglong2 b[COLS / 2];
#pragma unroll
                for (int j = 0; j < COLS / 2; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(&ws[stage][e][col + 32 * j]);
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned long long twice = ((unsigned long long)__float_as_uint(a[i]) << 32) | __float_as_uint(a[i]);
#pragma unroll
                    for (int j = 0; j < COLS / 2; ++j) {
                        gs_fma2(acc[i][2 * j], twice, b[j].x);
                        gs_fma2(acc[i][2 * j + 1], twice, b[j].y);
                    }
                }
            }
        }
        if (more) {
            put(stage ^ 1);                                     // the stage that the round before read: everyone has passed its barrier
            __syncthreads();
        }
    }
    float* o = out + (size_t)split * split_stride;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + row + (i & 3) + 16 * (i >> 2);
        if (gm >= m) continue;
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) {
            const int gn = n0 + col + 32 * j;
            float v[4] = {__uint_as_float((unsigned)acc[i][2 * j]), __uint_as_float((unsigned)(acc[i][2 * j] >> 32)),
                          __uint_as_float((unsigned)acc[i][2 * j + 1]), __uint_as_float((unsigned)(acc[i][2 * j + 1] >> 32))};
            if (bias && split == 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] += gn + e < n ? bias[gn + e] : 0.0f;
            }
            float* to = o + (size_t)gm * ldo + gn;
            if (vec_o && gn + 4 <= n) {
                *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
                continue;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (gn + e < n) to[e] = v[e];
        }
    }
}

// Skinny form for few rows of x (decoding, the few wanted rows of a head): a warp takes four output columns and up to 8 rows of x
// at a time, its lanes stride over k four numbers each, so that a lane has four 16-byte loads of weights in flight, a round ahead
// of their use, and a number of x that it fetched (from the L1) serves four columns.  Where there are too few columns for eight warps an SM,
// the four warps of a block take the same columns and walk k by turns.  Bound by reading the weights (us against a warp per
// column with 4-byte loads, float32): 1 and 4 rows of 128,256 x 2,048 761 -> 157 (6.7 TB/s) and 823 -> 205, 8 of 16,384 x 2,048 181 -> 92,
// 8 of 2,048 x 8,192 238 -> 34, 3 of 3,072 x 2,048 35 -> 11.
// GR_ROWS: rows of x at a time (1, 4 or 8, the least that holds m: fewer sums a lane, more warps an SM).
constexpr int GR_COLS = 4, GR_WARPS = 4;

// SIDE: a block takes its own GR_ROWS rows (blockIdx.y) instead of all rows in turn; an instance of its own, because the shift cost the others registers.
template <typename TX, typename TW, int GR_ROWS, bool SIDE = false>
__global__ void __launch_bounds__(GR_WARPS * 32)
gemm_rows_kernel(const TX* __restrict__ x, long long ldx, const TW* __restrict__ w, long long ldw,
                 const float* __restrict__ bias, float* __restrict__ out, long long ldo, int m, int n,
                 int k, int vec_x, int vec_w, int k_warps) {
    __shared__ float sums[GR_WARPS][GR_ROWS][GR_COLS];
    tt_pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // k_warps (1 or all): so many warps share four columns and walk k by turns
    const int col = (k_warps > 1 ? (int)blockIdx.x : (int)blockIdx.x * GR_WARPS + warp) * GR_COLS, k0 = (k_warps > 1 ? warp * 128 : 0) + lane * 4, step = 128 * k_warps;
    if (col >= n) return;                                       // with shared columns the whole block leaves
    float wv[GR_COLS][4];
    auto weights = [&](int kk) {
        const int count = max(0, min(4, k - kk));
#pragma unroll
        for (int c = 0; c < GR_COLS; ++c) gs_load4(wv[c], w + (size_t)min(col + c, n - 1) * ldw + kk, count, vec_w);
    };
    tt_pdl_wait();
    if constexpr (SIDE) {
        const int m_first = blockIdx.y * GR_ROWS;
        x += (size_t)m_first * ldx;
        out += (size_t)m_first * ldo;
        m = min(GR_ROWS, m - m_first);
    }
    for (int m0 = 0; m0 < m; m0 += GR_ROWS) {
        weights(k0);
        float acc[GR_ROWS][GR_COLS];
#pragma unroll
        for (int i = 0; i < GR_ROWS; ++i)
#pragma unroll
            for (int c = 0; c < GR_COLS; ++c) acc[i][c] = 0.0f;
        for (int kk = k0; kk < k; kk += step) {
            float now[GR_COLS][4];
#pragma unroll
            for (int c = 0; c < GR_COLS; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) now[c][e] = wv[c][e];
            if (kk + step < k) weights(kk + step);
            const int count = min(4, k - kk);
#pragma unroll
            for (int i = 0; i < GR_ROWS; ++i) {
                if (m0 + i >= m) break;
                float xv[4];
                gs_load4(xv, x + (size_t)(m0 + i) * ldx + kk, count, vec_x);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int c = 0; c < GR_COLS; ++c) acc[i][c] = fmaf(xv[e], now[c][e], acc[i][c]);
            }
        }
        if (k_warps > 1) __syncthreads();                       // the rows before are written
#pragma unroll
        for (int i = 0; i < GR_ROWS; ++i) {
            if (m0 + i >= m) break;
#pragma unroll
            for (int c = 0; c < GR_COLS; ++c) {
                const float total = tt_warp_sum(acc[i][c]);
                if (lane) continue;
                if (k_warps > 1) sums[warp][i][c] = total;
                else if (col + c < n) out[(size_t)(m0 + i) * ldo + col + c] = total + (bias ? bias[col + c] : 0.0f);
            }
        }
        if (k_warps > 1) {
            __syncthreads();
            const int i = threadIdx.x / GR_COLS, c = threadIdx.x % GR_COLS;
            if (i < GR_ROWS && m0 + i < m && col + c < n) {
                float total = 0.0f;
#pragma unroll
                for (int s = 0; s < GR_WARPS; ++s) total += sums[s][i][c];
                out[(size_t)(m0 + i) * ldo + col + c] = total + (bias ? bias[col + c] : 0.0f);
            }
        }
    }
}

// four neighbouring numbers of every row lie on a boundary of their size
template <typename T>
static int vec4(const void* p, long long ld) { return ((uintptr_t)p % (4 * sizeof(T))) == 0 && ld % 4 == 0; }

template <typename TX, typename TW>
static int launch(const void* x, long long ldx, const void* w, long long ldw, const float* bias, float* out,
                  long long ldo, long long split_stride, int m, int n, int k, int splits, int sms, cudaStream_t stream) {
    const int vec_x = vec4<TX>(x, ldx), vec_w = vec4<TW>(w, ldw);
    if (m <= 16 && splits == 1) {
        // fewer than eight warps an SM: the four warps of a block share its columns
        const int k_warps = n < 8 * GR_COLS * sms ? GR_WARPS : 1, cols = k_warps > 1 ? GR_COLS : GR_WARPS * GR_COLS;
        // nine rows and more side by side where the weights are few enough to be read twice at no cost (16 rows of 64 x 64 7.2 -> 4.2 us, of 16 x 2,048
        // 16 -> 9, of 3,072 x 2,048 35 -> 28; of 2,048 x 8,192 66 the one way and 72 the other)
        const bool side = m > 8 && k_warps > 1 && (long long)n * k <= 8 << 20;
#define TT_ROWS(ROWS, ...) tt_launch_pdl(gemm_rows_kernel<TX, TW, ROWS, ##__VA_ARGS__>, dim3((n + cols - 1) / cols, side ? (m + (ROWS) - 1) / (ROWS) : 1), dim3(GR_WARPS * 32), 0, stream, (const TX*)x, ldx, (const TW*)w, ldw, bias, out, ldo, m, n, k, vec_x, vec_w, k_warps)
        if (m == 1) TT_ROWS(1); else if (m <= 4) TT_ROWS(4); else if (side) TT_ROWS(8, true); else TT_ROWS(8);
#undef TT_ROWS
        TT_LAUNCH_CHECK();
    }
    int k_per_split = (k + splits - 1) / splits;
    k_per_split = (k_per_split + GS_BK - 1) / GS_BK * GS_BK;
    const int rows = (m + GS_BM - 1) / GS_BM;
    if (rows > 65535) return (int)cudaErrorInvalidValue;
    // tiles of half the width where even they leave SMs free: a tile alone on its SM takes half the time
    const bool half = (long long)rows * splits * ((n + 63) / 64) <= sms;
#define TT_TILES(BN) tt_launch_pdl(gemm_simt_kernel<TX, TW, BN>, dim3((n + (BN) - 1) / (BN), rows, splits), dim3(GS_THREADS), 0, stream, (const TX*)x, ldx, (const TW*)w, ldw, bias, out, ldo, split_stride, m, n, k, k_per_split, vec_x, vec_w, vec4<float>(out, ldo) && split_stride % 4 == 0)
    if (half) TT_TILES(64); else TT_TILES(128);
#undef TT_TILES
    TT_LAUNCH_CHECK();
}

// sms: the device's multiprocessors
extern "C" int tt_gemm_simt(const void* x, int x_dtype, long long ldx, const void* w, int w_dtype, long long ldw,
                            const float* bias, float* out, long long ldo, long long split_stride, int m, int n, int k,
                            int splits, int sms, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0 || splits < 1 || splits > 64) return (int)cudaErrorInvalidValue;
    if (x_dtype == TT_F32 && w_dtype == TT_F32) return launch<float, float>(x, ldx, w, ldw, bias, out, ldo, split_stride, m, n, k, splits, sms, stream);
    if (x_dtype == TT_BF16 && w_dtype == TT_BF16) return launch<__nv_bfloat16, __nv_bfloat16>(x, ldx, w, ldw, bias, out, ldo, split_stride, m, n, k, splits, sms, stream);
    if (x_dtype == TT_BF16 && w_dtype == TT_F32) return launch<__nv_bfloat16, float>(x, ldx, w, ldw, bias, out, ldo, split_stride, m, n, k, splits, sms, stream);
    if (x_dtype == TT_F32 && w_dtype == TT_BF16) return launch<float, __nv_bfloat16>(x, ldx, w, ldw, bias, out, ldo, split_stride, m, n, k, splits, sms, stream);
    return (int)cudaErrorInvalidValue;
}
