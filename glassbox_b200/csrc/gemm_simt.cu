// C[M, N] (+)= A[M, K] * W[N, K]^T on the CUDA cores with float32 FMA only.
//
// The generic product for any mix of float32 / bfloat16 operands at any size, and the one for up to eight float32 rows. (More of them run
// gemm_f32_tc.cu where K is 64 or more and rows are whole 16-byte pieces.) The kernels:
//   * register-tiled kernels with packed FMA for M > 8 (float32 activations, rows aligned to 16 bytes: the products of K below 64),
//   * a 64x64x16 register-tiled kernel for every other M > 8,
//   * weight-streaming kernels for M <= 8 (a block or a warp per four output columns, or a warp per column), which is what a
//     decode step needs: every weight is read once, coalesced along K.
// Each output element is reduced over K in an order that depends only on K and N (and on whether M > 8: all tiled kernels
// add one product after the other from k = 0, so they give the same bits), never on M or on the element's place in the batch.
// Row-major [out, in] weights as in crates/glassbox-core/src/kernels.rs:381, 586-655.
#include "common.cuh"

enum { OUT_STORE = 0, OUT_ACCUMULATE = 1 };

template <typename T> struct Vec4Load;
template <> struct Vec4Load<float> {
    static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
        float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
};
template <> struct Vec4Load<__nv_bfloat16> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[4]) {
        uint2 t = *reinterpret_cast<const uint2*>(p);
        __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&t.x);
        __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&t.y);
        v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
    }
};

template <typename TC>
__device__ __forceinline__ void store_out(TC* c, float v, int mode) {
    if (mode == OUT_ACCUMULATE) *c = gb_from_float<TC>(gb_to_float(*c) + v);
    else *c = gb_from_float<TC>(v);
}

// ------------------------------------------------------------------------------- tiled kernel
constexpr int BM = 64, BN = 64, BK = 16;

template <typename TA, typename TW, typename TC, bool VEC>
__global__ void __launch_bounds__(256) gemm_tiled_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                         TC* __restrict__ C, int M, int N, int K, long long lda,
                                                         long long ldw, long long ldc, int mode) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;  // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    const int lr = tid / 4;        // 0..63: tile row this thread loads
    const int lk = (tid % 4) * 4;  // 0,4,8,12: first k of its 4 elements
    for (int k0 = 0; k0 < K; k0 += BK) {
        float a[4] = {0.f, 0.f, 0.f, 0.f}, w[4] = {0.f, 0.f, 0.f, 0.f};
        int gm = m0 + lr, gn = n0 + lr, gk = k0 + lk;
        if (gm < M) {
            const TA* p = A + (size_t)gm * lda + gk;
            if (VEC && gk + 3 < K) Vec4Load<TA>::load(p, a);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) if (gk + e < K) a[e] = gb_to_float(p[e]);
        }
        if (gn < N) {
            const TW* p = W + (size_t)gn * ldw + gk;
            if (VEC && gk + 3 < K) Vec4Load<TW>::load(p, w);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) if (gk + e < K) w[e] = gb_to_float(p[e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            As[lk + e][lr] = a[e];
            Ws[lk + e][lr] = w[e];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int gn = n0 + tx * 4 + j;
            if (gn < N) store_out<TC>(C + (size_t)gm * ldc + gn, acc[i][j], mode);
        }
    }
}

// ------------------------------------------------------------------------ packed tiled kernels
// Tiles of BM x BN outputs, 128 threads of TM x TN outputs each, k in slices of KS double-buffered in shared memory (the next
// slice's loads are in flight while one is worked on; one barrier per slice). A packed FMA does two neighbouring rows. Bound by
// shared memory: a load costs its bytes to every lane whoever shares them, so the 64 x 64 tile of 256 threads (8 words for 16
// products, no loads in flight) reached 26-32 TFLOP/s; 8 x 4 outputs a thread read 12 words for 32. Two shapes: 64 x 64, and
// 32 x 64 where all tiles of that shape have an SM of their own (a lone block's time is its chain of slices, and a smaller slice
// is a shorter one). Measured, us for 576 x 576 at 200 / 800 / 2,047 rows: 31 / 32 / 50 before, 27 / 28 / 38 in 64 x 64, 19 / 29 /
// 54 in 32 x 64; 960 x 2560: 132 / 212 / 374, 109 / 155 / 281, 74 / 166 / 375; 3072 x 576: 49 / 106 / 227, 37 / 84 / 173, 40 / 111 /
// 252. (128 x 64 and 128 x 128 tiles: no better but for the last, 163.)
typedef unsigned long long simt_pair;

// WM x WN warps of LM x (32 / LM) lanes
template <int WM, int WN, int LM, int TM, int TN, int KS> struct PackedTile {
    static constexpr int LN = 32 / LM, THREADS = WM * WN * 32, BM = WM * LM * TM, BN = WN * LN * TN;
    static constexpr int WARPS_M = WM, LANES_M = LM, ROWS = TM, COLS = TN, SLICE = KS;
    static constexpr int FETCH_ROWS = THREADS / (KS / 4), FA = BM / FETCH_ROWS, FW = BN / FETCH_ROWS;
    static_assert(BM % FETCH_ROWS == 0 && BN % FETCH_ROWS == 0 && TM % 4 == 0 && TN % 4 == 0, "whole rounds of 16-byte loads");
};
typedef PackedTile<2, 2, 4, 8, 4, 16> Packed64x64;
typedef PackedTile<2, 2, 4, 4, 4, 32> Packed32x64;

template <typename P, typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(P::THREADS, 4) gemm_packed_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, int M,
                                                                    int N, int K, long long lda, long long ldw, long long ldc, int mode) {
    constexpr int TM = P::ROWS, TN = P::COLS, KS = P::SLICE, LM = P::LANES_M, LN = P::LN;
    __shared__ __align__(16) float As[2][KS][P::BM + 4];
    __shared__ __align__(16) float Ws[2][KS][P::BN + 4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // a thread's rows: four at m1, four 4 * LM further on, ...; its columns likewise
    const int m1 = (warp % P::WARPS_M) * LM * TM + (lane / LN) * 4, n1 = (warp / P::WARPS_M) * LN * TN + (lane % LN) * 4;
    const int m0 = blockIdx.y * P::BM, n0 = blockIdx.x * P::BN;
    const int lr = tid / (KS / 4), lk = (tid % (KS / 4)) * 4;      // the row (and those FETCH_ROWS further on) and the k's this thread fetches
    simt_pair acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
    float fa[P::FA][4], fw[P::FW][4];
    auto fetch = [&](int k0) {
        const int gk = k0 + lk;
#pragma unroll
        for (int h = 0; h < P::FA; ++h) {
            const int gm = m0 + lr + P::FETCH_ROWS * h;
            if (gm < M && gk < K) Vec4Load<TA>::load(A + (size_t)gm * lda + gk, fa[h]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) fa[h][e] = 0.f;
        }
#pragma unroll
        for (int h = 0; h < P::FW; ++h) {
            const int gn = n0 + lr + P::FETCH_ROWS * h;
            if (gn < N && gk < K) Vec4Load<TW>::load(W + (size_t)gn * ldw + gk, fw[h]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) fw[h][e] = 0.f;
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int h = 0; h < P::FA; ++h) As[buf][lk + e][lr + P::FETCH_ROWS * h] = fa[h][e];
#pragma unroll
            for (int h = 0; h < P::FW; ++h) Ws[buf][lk + e][lr + P::FETCH_ROWS * h] = fw[h][e];
        }
    };
    fetch(0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += KS, buf ^= 1) {
        const bool more = k0 + KS < K;
        if (more) fetch(k0 + KS);
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            simt_pair a[TM / 2];
            float w[TN];
#pragma unroll
            for (int g = 0; g < TM / 4; ++g) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&As[buf][kk][m1 + g * LM * 4]);
                a[2 * g] = t.x;
                a[2 * g + 1] = t.y;
            }
#pragma unroll
            for (int g = 0; g < TN / 4; ++g) *reinterpret_cast<float4*>(w + 4 * g) = *reinterpret_cast<const float4*>(&Ws[buf][kk][n1 + g * LN * 4]);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                simt_pair both;
                asm("mov.b64 %0, {%1, %1};" : "=l"(both) : "f"(w[j]));
#pragma unroll
                for (int i = 0; i < TM / 2; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a[i]), "l"(both));
            }
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
    const bool whole = N % 4 == 0 && ldc % 4 == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + m1 + (i / 4) * LM * 4 + i % 4;
        if (gm >= M) continue;
#pragma unroll
        for (int g = 0; g < TN / 4; ++g) {
            const int gn = n0 + n1 + g * LN * 4;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float lo, hi;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i / 2][g * 4 + j]));
                v[j] = i & 1 ? hi : lo;
            }
            TC* dst = C + (size_t)gm * ldc + gn;
            if (sizeof(TC) == 4 && whole) {
                if (gn >= N) continue;
                float4* d4 = reinterpret_cast<float4*>(dst);
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (mode == OUT_ACCUMULATE) {
                    const float4 o = *d4;
                    r = make_float4(o.x + r.x, o.y + r.y, o.z + r.z, o.w + r.w);
                }
                *d4 = r;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (gn + j < N) store_out<TC>(dst + j, v[j], mode);
            }
        }
    }
}

template <typename P, typename TA, typename TW, typename TC>
static void packed_launch(const TA* A, const TW* W, TC* C, int M, int N, int K, long long lda, long long ldw, long long ldc, int mode,
                          cudaStream_t stream) {
    gemm_packed_kernel<P, TA, TW, TC><<<dim3(gb_ceil_div(N, P::BN), gb_ceil_div(M, P::BM)), P::THREADS, 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc,
                                                                                                                 mode);
}

// ------------------------------------------------------------------- weight-streaming kernel
// One warp per output column n. Lanes stride over K four elements at a time; up to 8 rows of A
// are reduced against the same weight row, so the weight matrix is read exactly once.
template <typename TA, typename TW, typename TC, bool VEC>
__global__ void __launch_bounds__(256) gemm_skinny_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                          TC* __restrict__ C, int M, int N, int K, long long lda,
                                                          long long ldw, long long ldc, int mode) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * (blockDim.x >> 5) + warp;
    if (n >= N) return;
    float acc[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m] = 0.f;
    const TW* wrow = W + (size_t)n * ldw;
    for (int k = lane * 4; k < K; k += 128) {
        float w[4] = {0.f, 0.f, 0.f, 0.f};
        if (VEC && k + 3 < K) Vec4Load<TW>::load(wrow + k, w);
        else
#pragma unroll
            for (int e = 0; e < 4; ++e) if (k + e < K) w[e] = gb_to_float(wrow[k + e]);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m < M) {
                float a[4] = {0.f, 0.f, 0.f, 0.f};
                const TA* arow = A + (size_t)m * lda + k;
                if (VEC && k + 3 < K) Vec4Load<TA>::load(arow, a);
                else
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (k + e < K) a[e] = gb_to_float(arow[e]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m] = fmaf(a[e], w[e], acc[m]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        if (m < M) {
            float v = gb_warp_sum(acc[m]);
            if (lane == 0) store_out<TC>(C + (size_t)m * ldc + n, v, mode);
        }
    }
}

// The same four columns at a time, twelve 16-byte loads of a lane under way per 128 of K, the 32 sums of a lane brought together
// by 31 shuffles. SPLIT: the block is the unit, K dealt out to its eight warps in slices of 128 (a lane holds four consecutive
// k) whose sums meet in shared memory; else a warp takes its four columns alone, in the order, and so with the bits, of the
// kernel above. That one walks K alone, nine loads and their latency after the other, and re-reads the activations for every
// column: latency, a tenth of the copy rate at best. Measured, 8 rows float32: N 960, K 576 10.8 -> 2.3 us (split); N 576, K
// 1536 22.5 -> 3.3 (split); N 3072, K 576 12.1 -> 6.9; N 49152, K 576 62.7 -> 38.1 (113 MB). With the weights ahead of the wait and
// of the products, and (no split) two warps a block, which spread N 3072 over every SM: 2.3 -> 2.0, 3.3 -> 2.8, 6.9 -> 6.5, 38.0 -> 34.0;
// N 3072, K 2048 18.2 -> 17.4. (The activations one round ahead as well: N 8192 7.3 -> 11.6 for want of warps.) Weights of 16 bits, whose
// conversions then stand between the requests, gain nothing so and keep eight warps a block and no round ahead: 8 rows, N 1600, K 960 4.3 ->
// 4.0; N 8192, K 2048 20.4 -> 19.7.
template <typename TW> constexpr bool SK4_EARLY = sizeof(TW) == 4;
template <typename TA, typename TW, typename TC, bool SPLIT>
__global__ void __launch_bounds__(SPLIT || !SK4_EARLY<TW> ? 256 : 64) gemm_skinny4_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, int M, int N,
                                                           int K, long long lda, long long ldw, long long ldc, int mode) {
    __shared__ float part[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = (SPLIT ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + warp) * 4;
    gb_pdl_launch_dependents();
    // EARLY: the weights, which no kernel of a step writes, are asked for before the wait for the kernel before, and those of the next
    // round before this one's products.
    constexpr bool EARLY = SK4_EARLY<TW>;
    constexpr int STEP = SPLIT ? 1024 : 128;
    float wn[4][4];
    auto weights = [&](int k) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (n0 + c < N && k < K) Vec4Load<TW>::load(W + (size_t)(n0 + c) * ldw + k, wn[c]);
            else wn[c][0] = wn[c][1] = wn[c][2] = wn[c][3] = 0.f;
        }
    };
    const int k0 = (SPLIT ? warp * 128 : 0) + lane * 4;
    if (EARLY) weights(k0);
    gb_pdl_wait();
    float acc[32];                                      // [row][column]
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    for (int k = k0; k < K; k += STEP) {
        float w[4][4], a[8][4];
        if (!EARLY) weights(k);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) w[c][e] = wn[c][e];
        if (EARLY && k + STEP < K) weights(k + STEP);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m < M) Vec4Load<TA>::load(A + (size_t)m * lda + k, a[m]);
            else a[m][0] = a[m][1] = a[m][2] = a[m][3] = 0.f;
        }
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m >= M) break;
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m * 4 + c] = fmaf(a[m][e], w[c][e], acc[m * 4 + c]);
        }
    }
    // lane l ends up with the warp's sum number l: in each round the half of the sums that the partner keeps is sent to it
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float keep = up ? acc[i + o] : acc[i], send = up ? acc[i] : acc[i + o];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    float v = acc[0];
    if (SPLIT) {
        part[warp][lane] = v;
        __syncthreads();
        if (warp > 0) return;
#pragma unroll
        for (int i = 1; i < 8; ++i) v += part[i][lane];
    }
    {
        const int m = lane >> 2, n = n0 + (lane & 3);
        if (m < M && n < N) store_out<TC>(C + (size_t)m * ldc + n, v, mode);
    }
}

template <typename TA, typename TW, typename TC>
static int launch_gemm(const void* a, const void* w, void* c, int M, int N, int K, long long lda, long long ldw,
                       long long ldc, int mode, cudaStream_t stream) {
    bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && ((uintptr_t)a % 16 == 0) &&
               ((uintptr_t)w % 16 == 0);
    const TA* A = (const TA*)a;
    const TW* W = (const TW*)w;
    TC* C = (TC*)c;
    if (M <= 8) {
        int warps = 8;
        dim3 grid(gb_ceil_div(N, warps));
        // Up to 2,048 columns (512 blocks of four: one round of the chip) the split form is the faster at every number of rows
        // (N 2048, K 576, one row: 3.9 us against 5.1; K 8192: 18 against 40); beyond, its blocks are small change against their
        // barriers (N 8192, K 576, one row: 12.3 against 6.2). There four columns a warp pay from three rows of 32-bit and five
        // of 16-bit activations, whose conversions cost more (N 49152, K 576: one row 29.9 against 27.4, four 33.1 / 39.6, eight
        // 38.1 / 62.7; bfloat16 four rows 46.8 / 42.3, eight 50.5 / 66.0). The line between these two is the only one that
        // depends on M, and both sides give the same bits.
        if (vec && N <= 2048)
            gb_launch(GB_PDL_GEMM, gemm_skinny4_kernel<TA, TW, TC, true>, dim3(gb_ceil_div(N, 4)), dim3(256), 0, stream, A, W, C, M, N, K, lda, ldw, ldc, mode);
        else if (vec && M > (sizeof(TA) == 4 ? 2 : 4))
            gb_launch(GB_PDL_GEMM, gemm_skinny4_kernel<TA, TW, TC, false>, dim3(gb_ceil_div(N, SK4_EARLY<TW> ? 8 : 32)), dim3(SK4_EARLY<TW> ? 64 : 256), 0, stream, A, W, C, M, N, K, lda, ldw, ldc, mode);
        else if (vec) gemm_skinny_kernel<TA, TW, TC, true><<<grid, warps * 32, 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, mode);
        else gemm_skinny_kernel<TA, TW, TC, false><<<grid, warps * 32, 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, mode);
    } else {
        if constexpr (sizeof(TA) == 4 && sizeof(TC) == 4) {
            if (vec) {
                if ((long long)gb_ceil_div(M, Packed32x64::BM) * gb_ceil_div(N, Packed32x64::BN) <= 148)
                    packed_launch<Packed32x64>(A, W, C, M, N, K, lda, ldw, ldc, mode, stream);
                else packed_launch<Packed64x64>(A, W, C, M, N, K, lda, ldw, ldc, mode, stream);
                return gb_check_launch("gb_gemm_simt");
            }
        }
        dim3 grid(gb_ceil_div(N, BN), gb_ceil_div(M, BM));
        if (vec) gemm_tiled_kernel<TA, TW, TC, true><<<grid, 256, 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, mode);
        else gemm_tiled_kernel<TA, TW, TC, false><<<grid, 256, 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, mode);
    }
    return gb_check_launch("gb_gemm_simt");
}

// C dtype float32 with accumulate=1 adds into C (the residual stream); otherwise C is stored.
GB_EXPORT int gb_gemm_simt(const void* a, int a_dtype, const void* w, int w_dtype, void* c, int c_dtype,
                           int accumulate, int M, int N, int K, long long lda, long long ldw, long long ldc,
                           cudaStream_t stream) {
    GB_REQUIRE(M >= 0 && N > 0 && K > 0, "gb_gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
    GB_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gb_gemm_simt: a leading dimension is smaller than its row");
    GB_REQUIRE(!accumulate || c_dtype == GB_F32, "gb_gemm_simt: accumulation needs a float32 output");
    if (M == 0) return 0;
    int mode = accumulate ? OUT_ACCUMULATE : OUT_STORE;
#define GB_CASE(TA_, ta, TW_, tw, TC_, tc)                                                              \
    if (a_dtype == ta && w_dtype == tw && c_dtype == tc)                                                \
        return launch_gemm<TA_, TW_, TC_>(a, w, c, M, N, K, lda, ldw, ldc, mode, stream);
    GB_CASE(float, GB_F32, float, GB_F32, float, GB_F32)
    GB_CASE(__nv_bfloat16, GB_BF16, __nv_bfloat16, GB_BF16, __nv_bfloat16, GB_BF16)
    GB_CASE(__nv_bfloat16, GB_BF16, __nv_bfloat16, GB_BF16, float, GB_F32)
    GB_CASE(__nv_bfloat16, GB_BF16, float, GB_F32, __nv_bfloat16, GB_BF16)
    GB_CASE(__nv_bfloat16, GB_BF16, float, GB_F32, float, GB_F32)
    GB_CASE(float, GB_F32, __nv_bfloat16, GB_BF16, float, GB_F32)
#undef GB_CASE
    GB_REQUIRE(false, "gb_gemm_simt: unsupported dtype combination a=%d w=%d c=%d", a_dtype, w_dtype, c_dtype);
}
