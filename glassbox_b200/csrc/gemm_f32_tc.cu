// C[M, N] (+)= A[M, K] * W[N, K]^T of float32 activations (and float32 or bfloat16 weights) on the 5th-generation tensor cores,
// with the exactness of float32 FMA.
//
// Every float32 operand is the exact sum of three bfloat16 numbers, each what is left rounded to the nearest (a bfloat16 weight is one;
// Henry, Tang and Heinecke 2019). Eight of the nine products of two operands' terms stay: what is left out lies below 2^-34 of a
// product (with six, and terms cut off instead of rounded, it was up to 2^-21, always towards zero). Operands below some 2^-110 lose their
// last terms to bfloat16's smallest number: 2^-134 each. The tensor core's accumulator cuts instead of rounding, 1.1e-8 of the sum per 16
// of K, always downwards: a product over K 576 in one accumulator is off by 5.4e-7 where FMA is by 1.7e-7. So the products of the first terms
// get an accumulator for every 32 of K, and these sums are added in registers, rounded to nearest; all other products, at most
// 2^-8 of those, keep theirs to the end.
// Measured against 64 bits, float32 weights (2-norm of the error over that of the result), this / FMA: normal operands, K 64 5.3e-8 / 1.4e-7,
// K 576 9.4e-8 / 4.3e-7, K 1536 1.4e-7 / 7.0e-7, K 4096 2.2e-7 / 1.2e-6; rows of one number 2.5e-8 / 2.5e-8 (largest 6.0e-8 of a
// product for both), of two 2.6e-8 / 3.1e-8, of eight 2.9e-8 / 5.4e-8.
//
// A block computes one 128 x BN tile, 32 of K at a time. Sixteen warps do the same: bring float32 values into registers (two steps ahead),
// split them and store the terms as 64-byte-swizzled K-major tiles (two stages), then add the accumulator of the step before (of two) to
// their sums. A thread of a seventeenth issues the products, M 128, N BN, K 16.
// Bound by the workers' chain of a step (values, split, stores, the fence in front of the tensor core, the sums): 0.67 us at BN 64 and 0.89 at
// 128, where the products' operands alone keep shared memory busy for 0.3 and 0.4. One product takes two of W's terms side by side
// where it can and reads A's once for both (eight products apart: 22.1 us in the place of 20.6 for the first of the following).
// Measured, us, the FMA tiles (bound by the operands' way through shared memory at half of the FMA rate) and this: 2,047 rows N 960, K 576
// 67 -> 21; N 576, K 576 37 -> 15; N 3072, K 576 175 -> 58; N 576, K 1536 95 -> 35; 1,200 rows N 960, K 2560 150 -> 75; 9 rows N 576, K
// 576 17 -> 13; bfloat16 weights, 2,048 rows N 1024, K 64 10.2 -> 5.3. A step's products issued by a worker instead: 1.2 us a step.
//
// A result that is no finite number is formed again by FMA, one product after the other (an infinite operand's lesser terms are not
// numbers). Each output element's order of sums depends on K alone. Every wait is bounded (GB_STATUS_WAIT_TIMEOUT); there are no TMA
// copies to wait for.
#include "tcgen05.cuh"

constexpr int F3_BM = 128, F3_BK = 32, F3_WORKERS = 512, F3_THREADS = F3_WORKERS + 32, F3_ROW = F3_BK * 2;       // bytes of a row of one term

struct __align__(8) F3Shared {
    uint64_t full[2], done[2];
    uint32_t tmem_base;
    int abort_flag;
};

// K-major rows of 64 bytes, 64-byte swizzle: 8-row groups are 512 bytes apart
__device__ __forceinline__ uint64_t f3_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

__device__ __forceinline__ float4 f3_load(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 f3_load(const __nv_bfloat16* p) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xffff0000u), __uint_as_float(t.y << 16), __uint_as_float(t.y & 0xffff0000u));
}

template <int BN, typename TW>
__global__ void __launch_bounds__(F3_THREADS, 1) gemm_f32_tc_kernel(const float* __restrict__ A, const TW* __restrict__ W, float* __restrict__ C,
                                                                    int M, int N, int K, long long lda, long long ldw, long long ldc, int add,
                                                                    int* __restrict__ status) {
    constexpr int WT = sizeof(TW) == 4 ? 3 : 1;                       // terms of a weight
    constexpr int A_TERM = F3_BM * F3_ROW, W_TERM = BN * F3_ROW, STAGE = 3 * A_TERM + WT * W_TERM;
    constexpr int LR = F3_WORKERS / 8, AL = F3_BM / LR, WL = BN / LR; // 16-byte loads of a thread and step
    // accumulators side by side, BN columns each: two that take turns for the products of the first terms, then LESSER for all others
    constexpr int LESSER = WT == 1 ? 1 : 2, TMEM = 4 * BN;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* tiles = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    __shared__ F3Shared sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * F3_BM, n0 = blockIdx.y * BN, steps = (K + F3_BK - 1) / F3_BK;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sh.full[s], F3_WORKERS / 32);
            mbar_init(&sh.done[s], 1);
        }
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    volatile int* abort_flag = &sh.abort_flag;
    gb_pdl_launch_dependents();
    gb_pdl_wait();

    if (warp == F3_WORKERS / 32) {
        // (a warp of its own: the issuing thread is held up about as long as the products take)
        if (elect_one()) {
            const uint64_t a_desc = f3_desc(smem_u32(tiles)), w_desc = f3_desc(smem_u32(tiles) + 3 * A_TERM);
            for (int step = 0; step < steps; ++step) {
                const int s = step & 1;
                if (!mbar_wait(&sh.full[s], (step >> 1) & 1, abort_flag, status)) break;
                tc_fence_after();
                const uint64_t da = a_desc + ((s * STAGE) >> 4), dw = w_desc + ((s * STAGE) >> 4);
                // A's term `a` by `n` of W's terms from `w` on, which lie one behind the other: one product of n * BN columns reads A once
                auto product = [&](int a, int w, int n, int column, bool first) {
#pragma unroll
                    for (int k = 0; k < F3_BK / 16; ++k)
                        umma_bf16(tmem + (uint32_t)column, da + ((a * A_TERM) >> 4) + k * 2, dw + ((w * W_TERM) >> 4) + k * 2, umma_idesc(F3_BM, n * BN),
                                  first && k == 0 ? 0u : 1u);
                };
                if (WT == 1) {
                    product(2, 0, 1, 2 * BN, step == 0);
                    product(1, 0, 1, 2 * BN, false);
                } else {
                    product(2, 0, 2, 2 * BN, step == 0);
                    product(1, 2, 1, 2 * BN, false);
                    product(1, 0, 2, 2 * BN, false);
                    product(0, 1, 2, 2 * BN, false);
                }
                product(0, 0, 1, s * BN, true);
                umma_commit(&sh.done[s]);
            }
        }
    } else {
        // a thread fetches four k's of every 64th row; a row's 16-byte pieces of a term lie in an order that its number turns
        const int lr = tid >> 3, lk = (tid & 7) * 4;
        const int put = lr * F3_ROW + (((lk >> 3) ^ ((lr >> 1) & 3)) << 4) + (lk & 4) * 2;     // (the same turn 64 rows on)
        struct Ahead { float4 a[AL], w[WL]; } ahead[2];                   // the values of this step and the next
        auto fetch = [&](int step, Ahead& to) {
            const int k = step * F3_BK + lk;
#pragma unroll
            for (int i = 0; i < AL; ++i) {
                const int m = m0 + lr + LR * i;
                to.a[i] = m < M && k < K ? f3_load(A + (size_t)m * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < WL; ++i) {
                const int n = n0 + lr + LR * i;
                to.w[i] = n < N && k < K ? f3_load(W + (size_t)n * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        constexpr int CW = BN / (F3_WORKERS / 128), PIECES = CW / 4;      // a warp's columns, their 16-byte pieces
        const int q = warp & 3, col0 = (warp >> 2) * CW;                  // the quarter of the accumulator's rows and the first of its columns of this warp
        const uint32_t t_base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)col0;
        float acc[CW];
#pragma unroll
        for (int j = 0; j < CW; ++j) acc[j] = 0.f;
        bool ok = true;
        auto collect = [&](int step) {                                    // adds a finished step's accumulator to the sums
            ok = mbar_wait_warp(&sh.done[step & 1], (step >> 1) & 1, abort_flag, status);
            if (!ok) return;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < CW; c += 16) {
                uint32_t r[16];
                tmem_load16(t_base + (uint32_t)((step & 1) * BN + c), r);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(r[j]);
            }
            tc_fence_before();                                            // (the next arrival at `full` of this stage hands the accumulator back)
        };
        fetch(0, ahead[0]);
        if (steps > 1) fetch(1, ahead[1]);
        auto turn = [&](int step, int s, Ahead& own) {
            // the stage is free: the products of two steps before were waited for when their sums were collected
            unsigned char* at = tiles + s * STAGE + put;
            auto split = [&](const float4& v, unsigned char* to, int terms, int stride) {
                uint32_t lo[3], hi[3];
                gb_split_bf16(v.x, v.y, lo);
                gb_split_bf16(v.z, v.w, hi);
#pragma unroll
                for (int e = 0; e < terms; ++e) *reinterpret_cast<uint2*>(to + e * stride) = make_uint2(lo[e], hi[e]);
            };
#pragma unroll
            for (int i = 0; i < AL; ++i) split(own.a[i], at + i * LR * F3_ROW, 3, A_TERM);
#pragma unroll
            for (int i = 0; i < WL; ++i) split(own.w[i], at + 3 * A_TERM + i * LR * F3_ROW, WT, W_TERM);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads what was stored
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.full[s]);
            __syncwarp();
            if (step + 2 < steps) fetch(step + 2, own);
            if (step > 0) collect(step - 1);
        };
        for (int step = 0; step < steps && ok; step += 2) {
            turn(step, 0, ahead[0]);
            if (step + 1 < steps && ok) turn(step + 1, 1, ahead[1]);
        }
        if (ok) collect(steps - 1);
        if (ok) {
#pragma unroll
            for (int c = 0; c < CW; c += 16) {                            // the sums of the lesser terms' products
                float sum[16] = {};
#pragma unroll
                for (int e = 0; e < LESSER; ++e) {
                    uint32_t r[16];
                    tmem_load16(t_base + (uint32_t)((2 + e) * BN + c), r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[j] += __uint_as_float(r[j]);
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += sum[j];
            }
            const int row = m0 + q * 32 + lane;
            bool odd = false;
#pragma unroll
            for (int j = 0; j < CW; ++j) odd |= !(fabsf(acc[j]) <= FLT_MAX);
            if (__any_sync(0xffffffffu, odd && row < M)) {
#pragma unroll
                for (int j = 0; j < CW; ++j) {
                    const int n = n0 + col0 + j;
                    if (fabsf(acc[j]) <= FLT_MAX || row >= M || n >= N) continue;
                    float v = 0.f;
                    for (int k = 0; k < K; ++k) v = fmaf(A[(size_t)row * lda + k], gb_to_float(W[(size_t)n * ldw + k]), v);
                    acc[j] = v;
                }
                __syncwarp();
            }
            // a lane has piece `lane % PIECES` of every (32 / PIECES)th row
            constexpr int RR = 32 / PIECES;
            const int rows_here = min(32, M - (m0 + q * 32)), lrow = lane / PIECES, piece = lane % PIECES, col = n0 + col0 + 4 * piece;
            const bool vec = ((uintptr_t)C & 15) == 0 && (ldc & 3) == 0;
            float* base = C + (size_t)(m0 + q * 32) * ldc + col;
            // every product has been formed: the stages serve as the warps' tiles in which rows turn, so that an instruction writes whole rows
            uint4* stage = reinterpret_cast<uint4*>(tiles) + warp * (32 * PIECES);
            auto place = [&](int r, int p) { return r * PIECES + (p ^ (PIECES == 8 ? r & 7 : (r >> 1) & 3)); };
#pragma unroll
            for (int p = 0; p < PIECES; ++p)
                stage[place(lane, p)] = make_uint4(__float_as_uint(acc[4 * p]), __float_as_uint(acc[4 * p + 1]), __float_as_uint(acc[4 * p + 2]),
                                                   __float_as_uint(acc[4 * p + 3]));
            float4 old[PIECES];
            if (add) {
#pragma unroll
                for (int i = 0; i < PIECES; ++i) {
                    const int rr = RR * i + lrow;
                    const float* src = base + (size_t)rr * ldc;
                    old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (rr >= rows_here) continue;
                    if (vec && col + 4 <= N) {
                        old[i] = *reinterpret_cast<const float4*>(src);
                    } else {
                        if (col < N) old[i].x = src[0];
                        if (col + 1 < N) old[i].y = src[1];
                        if (col + 2 < N) old[i].z = src[2];
                        if (col + 3 < N) old[i].w = src[3];
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int rr = RR * i + lrow;
                float4 v = *reinterpret_cast<const float4*>(&stage[place(rr, piece)]);
                if (add) v = make_float4(old[i].x + v.x, old[i].y + v.y, old[i].z + v.z, old[i].w + v.w);
                if (rr < rows_here) tc_store4_f32(base + (size_t)rr * ldc, v, col, N, vec);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM) : "memory");
}

template <int BN, typename TW>
static int f3_launch(const float* a, const TW* w, float* c, int M, int N, int K, long long lda, long long ldw, long long ldc, int add, int* status,
                     cudaStream_t stream) {
    constexpr int SMEM = 2 * (3 * F3_BM + (sizeof(TW) == 4 ? 3 : 1) * BN) * F3_ROW + 1024;
    static_assert(SMEM - 1024 >= F3_BM * BN * 4, "the warps' turning tiles lie in the stages");
    auto kernel = gemm_f32_tc_kernel<BN, TW>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    GB_REQUIRE(e == cudaSuccess, "gb_gemm_f32_tc: %d bytes of shared memory refused: %s", SMEM, cudaGetErrorString(e));
    e = gb_launch(GB_PDL_GEMM, kernel, dim3(gb_ceil_div(M, F3_BM), gb_ceil_div(N, BN)), dim3(F3_THREADS), SMEM, stream, a, w, c, M, N, K, lda, ldw,
                  ldc, add, status);
    GB_REQUIRE(e == cudaSuccess, "gb_gemm_f32_tc: launch failed: %s", cudaGetErrorString(e));
    return gb_check_launch("gb_gemm_f32_tc");
}

// 1 if the product takes these operands: rows of whole four-number pieces, 16-byte aligned bases.
GB_EXPORT int gb_gemm_f32_tc_supported(const void* a, const void* w, int N, int K, long long lda, long long ldw) {
    return N > 0 && K > 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0 &&
           gb_ceil_div(N, 64) <= 65535;
}

GB_EXPORT int gb_gemm_f32_tc(const void* a, const void* w, int w_dtype, void* c, int accumulate, int M, int N, int K, long long lda, long long ldw,
                             long long ldc, int* status, cudaStream_t stream) {
    GB_REQUIRE(gb_gemm_f32_tc_supported(a, w, N, K, lda, ldw) && status != nullptr && M >= 0,
               "gb_gemm_f32_tc: rows must be whole aligned 16-byte pieces (M=%d N=%d K=%d)", M, N, K);
    GB_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gb_gemm_f32_tc: a leading dimension is smaller than its row");
    if (M == 0) return 0;
    // The width whose rounds of tiles end soonest: a tile takes 0.67 us a step and 2.9 beside it at BN 64, 0.89 and 3.4 at 128 (from launches
    // of one round). Both add in the same order.
    const int steps = gb_ceil_div(K, F3_BK);
    const long long tiles_m = gb_ceil_div(M, F3_BM), r64 = (tiles_m * gb_ceil_div(N, 64) + 147) / 148, r128 = (tiles_m * gb_ceil_div(N, 128) + 147) / 148;
    const bool wide = (float)r128 * (0.89f * (float)steps + 3.4f) < (float)r64 * (0.67f * (float)steps + 2.9f);
#define F3_CASE(BN_, TW_) f3_launch<BN_, TW_>((const float*)a, (const TW_*)w, (float*)c, M, N, K, lda, ldw, ldc, accumulate, status, stream)
    if (w_dtype == GB_F32) return wide ? F3_CASE(128, float) : F3_CASE(64, float);
    GB_REQUIRE(w_dtype == GB_BF16, "gb_gemm_f32_tc: unsupported weights' dtype %d", w_dtype);
    return wide ? F3_CASE(128, __nv_bfloat16) : F3_CASE(64, __nv_bfloat16);
#undef F3_CASE
}
