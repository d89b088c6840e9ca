// out[s][m][n] = sum over the s-th slice of k of x[m][k] * w[n][k]  (+ bias[n] in s = 0), float32 operands, on the tensor cores
//
// The 32-bit product of prompts.  Every operand is cut into three bfloat16 numbers (x = hi + mid + lo, each what the parts before leave,
// rounded to nearest: see split_mma.cuh), and six of the nine products of parts (all but mid lo, lo mid and lo lo: together 2^-23
// of the product at most, 2^-27 rms) go through tcgen05.mma, whose products of bfloat16 are exact.  What the tensor cores do to a sum is the other
// half: they truncate, so that a sum that runs through all of k in tensor memory drifts.  So tensor memory only ever holds
// the sum over 64 k, the small products of them first and the large ones behind; it is then read and added to float32 sums in
// registers.  Sums of many terms are nearer to 64 bits than those of the float32 multiply-adds of gemm_simt.cu (see there for the reference's entry
// points): 0.16 to 0.52 of their error for normal numbers, 0.36 to 0.87 for numbers of one sign (the truncation takes 0.6e-7 to 0.8e-7 of a sum), 0.12 to 0.42 where
// sums cancel; a product that stands alone is right to a unit or two in the last place instead of half of one (4.7e-8 against 2.7e-8).
//
// A CTA pair (cta_group::2) has 256 output features and up to 256 tokens: the weights are the 256-row operand, so they are read and cut
// up once for all those tokens.  Sixteen warps of each CTA cut the pair's weights up as they come from memory (straight into the
// swizzled rows that the products read; they would be too many bytes to cut up beforehand) and read the accumulators; another
// fetches the activations' parts, which a small kernel before wrote; one more, of the even CTA, issues.  Two stages of 64 k, two accumulators: while the
// products of a block of 64 k run, the warps add up the block before and cut up the one behind.
//
// What bounds it: the six products (a block of 64 k of 224 tokens is 24 of them, 2,690 of the 3,000 cycles a block takes; tensor pipe 76 % busy over a whole launch); below about 100
// tokens the way of a block through the kernel, 2,700 cycles; few features the pairs' start and end.  The rows of weights go behind the arrival
// of the block before: with loads ahead of it the fence took 750 cycles more a block.  What the odd CTA's warps wrote has to be released to the
// cluster, which took every warp 1,700 cycles when each did it (its fence waits for the warp's loads): they arrive at a barrier of their own CTA, and one thread
// without loads passes that on.  us with a cold L2 (about 8 of them the events'), multiply-adds of gemm_simt.cu and now: 193 rows, 16,384 features of 2,048 349 -> 69, 2,048 of 8,192
// 215 -> 44, 3,072 of 2,048 78 -> 28, 256 of 2,048 21.5 -> 17.4; 17 rows, 16,384 of 2,048 79 -> 60, 64 of 512 19.5 -> 13.3; 2,048 rows, 16,384 of 2,048 2,660 -> 546.  Relative error
// against 64 bits, normal numbers: 193 rows, 2,048 of 8,192 6.6e-7 -> 1.1e-7, 17 rows, 40 of 72 1.6e-7 -> 0.8e-7.
//
// A sum that comes out infinite or NaN (an operand that is, one that rounds up to infinity, parts of infinite products of opposite
// signs) is formed again by multiply-adds, by the thread that has it: such outputs are what gemm_simt.cu makes of them.  So is a sum below 2^-90: the third
// part of a number below 2^-109 falls under the smallest bfloat16 number, 2^-133, and is lost (x of 1e-36: errors of 2.6e-5 instead of 1.5e-7).  Sums of
// such numbers times others that reach 2^-90 all the same (others above 2^18 / k) keep the bits that two parts have.
#include <algorithm>

#include <cooperative_groups.h>

#include "split_mma.cuh"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;
using namespace tc;

namespace {

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int WORKERS = 512, WARPS = WORKERS / 32, THREADS = WORKERS + 128;
// registers: 640 x 96 = 512 x 104 + 128 x 64
constexpr int REGS_WORKER = 104, REGS_ISSUER = 64;
constexpr int PARTS = 3;
constexpr int A_BYTES = BM * BK * 2;                            // one part of a CTA's weights of a stage
constexpr int MAX_HALF = 128;                                   // rows of activations of a CTA
constexpr int STAGE_BYTES = PARTS * A_BYTES + PARTS * MAX_HALF * BK * 2;
constexpr int AHEAD = 4;                                        // blocks of 64 k that are asked for into the L2
constexpr int SHARED = 2 * STAGE_BYTES + 1024;

// The activations' parts [3][m][kp] (kp: k rounded up to 8, the padding never read), four numbers a thread.  A product is preceded by one
// such launch; cutting them up with the weights, in every CTA that reads them, would double that work there.
__global__ void __launch_bounds__(256) cut_kernel(const float* __restrict__ x, long long ldx, __nv_bfloat16* __restrict__ parts, int m, int k, int kp, int vec) {
    tt_pdl_launch_dependents();
    tt_pdl_wait();
    const int quads = kp >> 2;
    const long long plane = (long long)m * kp;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < (long long)m * quads; i += (long long)gridDim.x * 256) {
        const int row = (int)(i / quads), at = (int)(i % quads) * 4;
        const float* p = x + (size_t)row * ldx + at;
        float v[4];
        if (vec && at + 4 <= k) {
            const float4 q = *reinterpret_cast<const float4*>(p);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = at + e < k ? p[e] : 0.0f;
        }
        uint2 hi, mid, lo;
        split_pair(v[0], v[1], hi.x, mid.x, lo.x);
        split_pair(v[2], v[3], hi.y, mid.y, lo.y);
        __nv_bfloat16* to = parts + (size_t)row * kp + at;
        *reinterpret_cast<uint2*>(to) = hi;
        *reinterpret_cast<uint2*>(to + plane) = mid;
        *reinterpret_cast<uint2*>(to + 2 * plane) = lo;
    }
}

constexpr float LEAST = 8.077935669463161e-28f;                 // 2^-90: smaller sums, but zeros, are formed again

struct Args {
    const float* x;
    const float* w;
    const float* bias;
    float* out;
    unsigned* status;
    long long ldx, ldw, ldo, split_stride;
    int m, n, k, k_blocks_per_split;
    int tokens;                                                 // rows of a token tile, a multiple of 32
    int vec_w;
};

__global__ void __launch_bounds__(THREADS, 1) gemm_split_kernel(const __grid_constant__ CUtensorMap map_x, const Args args) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full_bar[2], done_bar[2], cut_bar[2];
    __shared__ uint32_t tmem_base_shared;

    tt_pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster.block_rank();
    const int feature0 = ((int)blockIdx.x >> 1) * 2 * BM + rank * BM, token0 = blockIdx.y * args.tokens;
    const int half = args.tokens >> 1;                          // rows of activations that each CTA fetches
    const int kb0 = blockIdx.z * args.k_blocks_per_split;
    const int steps = max(0, min((args.k + BK - 1) / BK - kb0, args.k_blocks_per_split));

    if (threadIdx.x == 0) {
        // full (the even CTA's): the announced copies, its workers' warps, and one arrival for all of the odd CTA's; cut (the odd CTA's): its workers'
        // warps; done: the products of a stage
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 2 + WARPS);
            mbar_init(smem_u32(&cut_bar[s]), WARPS);
            mbar_init(smem_u32(&done_bar[s]), 1);
        }
        fence_barrier_init();
    }
    cluster.sync();
    if (warp == WARPS + 1) tmem_alloc_pair(smem_u32(&tmem_base_shared), 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = tmem_base_shared;
    tt_pdl_wait();                                              // before either operand: a caller's weights may be fresh

    if (warp >= WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUER));
        if (warp == WARPS && lane == 0) {
            for (int i = 0; i < steps; ++i) {
                const int s = i & 1;
                if (i >= 2 && !mbar_wait(smem_u32(&done_bar[s]), ((i >> 1) & 1) ^ 1)) { atomicOr(args.status, TT_STATUS_WAIT_EXPIRED); break; }
                const uint32_t bar = smem_u32(&full_bar[s]);
                if (rank == 0) mbar_expect_tx(bar, 2u * PARTS * half * BK * 2);         // both CTAs' copies
                const uint32_t to = smem_u32(smem + (size_t)s * STAGE_BYTES + PARTS * A_BYTES);
                for (int p = 0; p < PARTS; ++p)
                    asm volatile(
                        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                        ::"r"(to + p * half * BK * 2), "l"(&map_x), "r"((kb0 + i) * BK), "r"(token0 + rank * half), "r"(p), "r"(bar & PEER_MASK) : "memory");
            }
            // every copy has landed once the products that read it are done, for which the workers wait; where a wait ran out, theirs or this one, the
            // copies before it were asked for a limit ago
        }
        if (warp == WARPS + 1 && lane == 0 && rank == 0) {
            const uint32_t idesc = instr_desc(2 * BM, args.tokens);
            for (int i = 0; i < steps; ++i) {
                const int s = i & 1;
                if (!mbar_wait<true>(smem_u32(&full_bar[s]), (i >> 1) & 1)) { atomicOr(args.status, TT_STATUS_WAIT_EXPIRED); break; }
                fence_after_sync();
                const uint32_t a = smem_u32(smem + (size_t)s * STAGE_BYTES), b = a + PARTS * A_BYTES, acc = tmem_base + s * 256;
                // parts of (weights, activations), the smallest products first
                constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int kk = 0; kk < BK / UMMA_K; ++kk)
                        umma_bf16_pair(acc, smem_desc(a + PA[p] * A_BYTES + kk * UMMA_K * 2), smem_desc(b + PB[p] * half * BK * 2 + kk * UMMA_K * 2), idesc,
                                       (p > 0 || kk > 0) ? 1u : 0u);
                umma_commit_pair(smem_u32(&done_bar[s]), 3);
            }
        }
        if (warp == WARPS + 1 && lane == 0 && rank == 1) {
            // the odd CTA's rows of weights, and its reading of the accumulator two blocks ago, handed to the issuer
            for (int i = 0; i < steps; ++i) {
                const int s = i & 1;
                if (!mbar_wait(smem_u32(&cut_bar[s]), (i >> 1) & 1)) { atomicOr(args.status, TT_STATUS_WAIT_EXPIRED); break; }
                fence_after_sync();
                fence_before_sync();
                mbar_release_even_cta(smem_u32(&full_bar[s]));
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_WORKER));
        // rows of weights: a warp 8, two at a time, 16 lanes a row of 64 k
        const int load_row = warp * 8 + (lane >> 4), load_k = (lane & 15) * 4;
        float4 raw[4];
        auto fetch = [&](int i, int j) {
            const int at = (kb0 + i) * BK + load_k, row = feature0 + load_row + 2 * j;
            const float* p = args.w + (size_t)row * args.ldw + at;
            if (row < args.n && args.vec_w && at + 4 <= args.k) raw[j] = __ldg(reinterpret_cast<const float4*>(p));
            else {
                const int count = row < args.n ? args.k - at : 0;
                raw[j] = make_float4(count > 0 ? __ldg(p) : 0.0f, count > 1 ? __ldg(p + 1) : 0.0f, count > 2 ? __ldg(p + 2) : 0.0f, count > 3 ? __ldg(p + 3) : 0.0f);
            }
        };
        // the lines of a block further ahead into the L2, one a thread: as far as memory is away
        auto ask = [&](int i) {
            const int row = feature0 + (threadIdx.x >> 1), at = (kb0 + i) * BK + (threadIdx.x & 1) * 32;
            if (threadIdx.x < 2 * BM && i < steps && row < args.n && at < args.k)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(args.w + (size_t)row * args.ldw + at));
        };
        // sums: 32 lanes' features, a quarter of the tile's tokens in blocks of 16 (half of the last one may be another warp's)
        const int quarter = warp & 3, width = half >> 1, column0 = (warp >> 2) * width;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + column0;
        float acc[4][16];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[b][e] = 0.0f;
        auto drain = [&](int i) -> bool {
            const int s = i & 1;
            if (!mbar_wait(smem_u32(&done_bar[s]), (i >> 1) & 1)) return false;
            fence_after_sync();
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (b * 16 >= width) break;
                float v[16];
                tmem_load16(lane_addr + s * 256 + b * 16, v);
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[b][e] += v[e];
            }
            fence_before_sync();
            return true;
        };
        bool ok = true;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (steps > 0) fetch(0, j);
        for (int i = 1; i < AHEAD; ++i) ask(i);
        for (int i = 0; i < steps; ++i) {
            // the stage is free: the products of block i - 2 were waited for when its sums were added up
            const uint32_t to = smem_u32(smem + (size_t)(i & 1) * STAGE_BYTES);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = load_row + 2 * j;
                const uint32_t at = to + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8;
                uint2 hi, mid, lo;
                split_pair(raw[j].x, raw[j].y, hi.x, mid.x, lo.x);
                split_pair(raw[j].z, raw[j].w, hi.y, mid.y, lo.y);
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(hi.x), "r"(hi.y) : "memory");
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + A_BYTES), "r"(mid.x), "r"(mid.y) : "memory");
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + 2 * A_BYTES), "r"(lo.x), "r"(lo.y) : "memory");
            }
            fence_async_shared();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(rank ? &cut_bar[i & 1] : &full_bar[i & 1]));
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + 1 < steps) fetch(i + 1, j);                // behind the arrival: the fence before it would wait for them
            ask(i + AHEAD);
            if (i > 0 && !drain(i - 1)) { ok = false; break; }
        }
        if (ok && steps > 0) ok = drain(steps - 1);
        if (!ok && lane == 0) atomicOr(args.status, TT_STATUS_WAIT_EXPIRED);

        const int feature = feature0 + quarter * 32 + lane;
        if (ok && feature < args.n) {
            const float bias = args.bias && blockIdx.z == 0 ? args.bias[feature] : 0.0f;
            float* out = args.out + (size_t)blockIdx.z * args.split_stride + feature;
            const int first = token0 + column0, count = min(width, args.m - first);
            float least = INFINITY, odd = 0.0f;                 // the smallest sum's size; NaN once a sum is not finite
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                float* to = out + (size_t)(first + b * 16) * args.ldo;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    if (b * 16 + e < count) {
                        to[0] = acc[b][e] + bias;
                        least = fminf(least, fabsf(acc[b][e]));
                        odd = fmaf(acc[b][e], 0.0f, odd);
                    }
                    to += args.ldo;
                }
            }
            if (!(least >= LEAST) || odd != 0.0f) {             // (asked once for all sums: asked for each, the 32-bit prompt took 1 % more)
                unsigned again[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    again[b] = 0;
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (b * 16 + e < count && acc[b][e] != 0.0f && !(fabsf(acc[b][e]) >= LEAST && fabsf(acc[b][e]) <= 3.402823466e38f)) again[b] |= 1u << e;
                }
#pragma unroll 1
                for (int b = 0; b < 4; ++b) {
                    unsigned left = b == 0 ? again[0] : b == 1 ? again[1] : b == 2 ? again[2] : again[3];
                    for (; left; left &= left - 1) {
                        const int token = first + b * 16 + __ffs(left) - 1;
                        const float *xr = args.x + (size_t)token * args.ldx, *wr = args.w + (size_t)feature * args.ldw;
                        float v = 0.0f;
                        for (int kk = kb0 * BK; kk < min(args.k, (kb0 + steps) * BK); ++kk) v = fmaf(xr[kk], wr[kk], v);
                        out[(size_t)token * args.ldo] = v + bias;
                    }
                }
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    cluster.sync();                                             // nobody's shared or tensor memory goes while the other CTA may touch it
    if (warp == WARPS + 1) tmem_dealloc_pair(tmem_base, 512);
}

}  // namespace

// parts: bfloat16 [3][m][k rounded up to 8], scratch
extern "C" int tt_gemm_split(const float* x, long long ldx, const float* w, long long ldw, const float* bias, float* out, long long ldo,
                             long long split_stride, void* parts, unsigned* status, int m, int n, int k, int splits, int sms, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0 || splits < 1 || splits > 64) return (int)cudaErrorInvalidValue;
    const int kp = (k + 7) / 8 * 8;
    const int tiles = (m + 255) / 256, tokens = ((m + tiles - 1) / tiles + 31) / 32 * 32;
    if (tiles > 65535) return (int)cudaErrorInvalidValue;
    cudaError_t err = tt_allow_shared(gemm_split_kernel, SHARED);
    if (err != cudaSuccess) return (int)err;
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)m, PARTS};
    const cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)m * kp * 2};
    const cuuint32_t box[3] = {BK, (cuuint32_t)(tokens / 2), 1};
    if (!tc::make_map(&map, parts, 3, dims, strides, box)) return (int)cudaErrorInvalidValue;
    const long long quads = (long long)m * (kp / 4);
    const int blocks = (int)std::min((quads + 255) / 256, (long long)sms * 8);
    err = tt_launch_pdl(cut_kernel, dim3(blocks), dim3(256), 0, stream, x, ldx, (__nv_bfloat16*)parts, m, k, kp,
                                    (int)((uintptr_t)x % 16 == 0 && ldx % 4 == 0));
    if (err != cudaSuccess) return (int)err;
    Args args = {x, w, bias, out, status, ldx, ldw, ldo, split_stride, m, n, k, ((k + BK - 1) / BK + splits - 1) / splits, tokens,
                 (int)((uintptr_t)w % 16 == 0 && ldw % 4 == 0)};
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(2 * ((n + 2 * BM - 1) / (2 * BM)), (m + tokens - 1) / tokens, splits);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = SHARED;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    attribute[1].id = cudaLaunchAttributeClusterDimension;
    attribute[1].val.clusterDim.x = 2;
    attribute[1].val.clusterDim.y = 1;
    attribute[1].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 2;
    err = cudaLaunchKernelEx(&config, gemm_split_kernel, map, args);
    return err != cudaSuccess ? (int)err : (int)cudaGetLastError();
}
