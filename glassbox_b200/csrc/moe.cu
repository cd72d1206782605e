// A routed feed-forward (mixture of experts) with sigmoid scores, a choice bias and a limit to the best groups of experts.
//
//   moe_route        per row: logits = W_router h in float32 (h in the activation dtype), scores s = sigmoid(logits);
//                    experts are chosen by s + correction, the weights use s alone. The experts form `groups` equal runs of
//                    neighbours; a run's score is the sum of its two largest choice scores (its only one, if it has one
//                    member); only experts of the `keep` best runs can be chosen, the others count as minus infinity. The
//                    `top` largest are taken (among equals the lowest index), each with the weight s * route_scale, not
//                    renormalised. Also the gate of a shared expert, sigmoid(w_gate . h), one number per row.
//                    With softmax_chosen the scores are the logits themselves (plus a stored bias per expert), the `top`
//                    largest are taken and their weights are the softmax over the chosen logits alone.
//                    With softmax scores s = softmax(logits) over all experts; a run's score is the largest in it (run_best
//                    1; else the sum of its two largest), and with renorm_eps >= 0 the chosen scores are divided by
//                    (their sum + renorm_eps).
//                    An expert is either W_down relu(W_up h)^2 or (UNIT) W_down unit(W_gate h, W_up h) with one of the gated
//                    units of gb_gated_unit (the clamped one, gelu_tanh(gate) * up or silu(gate) * up); its
//                    up matrix then holds gate row f and up row f as rows 2f and 2f + 1.
//   moe_expert_rows  one block per (row, chosen expert): act = relu(W_up[e] h)^2 in shared memory, then W_down[e] act,
//                    written as float32 per (row, choice). Reads the two matrices of one expert once per block: the
//                    form for few rows (decoding), and the float32 path's form for any number.
//   moe_combine      out[row] (+)= sum_k weight[row, k] * pair[row, k] + gate[row] * shared[row]; a fixed order of sums.
#include "common.cuh"

#include <math.h>

constexpr int MOE_MAX_EXPERTS = 512;
enum { MOE_SIGMOID = 0, MOE_SOFTMAX_CHOSEN = 1, MOE_SOFTMAX = 2 };      // how logits become scores and weights
constexpr int MOE_ROUTE_THREADS = 1024;      // at most; the launch takes a warp per expert (and one for the shared gate)

__device__ __forceinline__ float moe_sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }

// sum over K of w[k] * x[k]; x float32 in shared memory, w a row of a matrix in global memory; all lanes get the sum
template <typename T>
__device__ __forceinline__ float moe_warp_dot(const T* __restrict__ w, const float* __restrict__ x, int K, int lane);

template <>
__device__ __forceinline__ float moe_warp_dot<float>(const float* __restrict__ w, const float* __restrict__ x, int K, int lane) {
    float d = 0.f;
    if (K % 4 == 0 && ((uintptr_t)w & 15) == 0) {
#pragma unroll 4
        for (int i = lane * 4; i < K; i += 128) {
            const float4 v = *reinterpret_cast<const float4*>(w + i);
            d = fmaf(v.x, x[i], d); d = fmaf(v.y, x[i + 1], d); d = fmaf(v.z, x[i + 2], d); d = fmaf(v.w, x[i + 3], d);
        }
    } else {
        for (int i = lane; i < K; i += 32) d = fmaf(w[i], x[i], d);
    }
    return gb_warp_sum(d);
}

template <>
__device__ __forceinline__ float moe_warp_dot<__nv_bfloat16>(const __nv_bfloat16* __restrict__ w, const float* __restrict__ x, int K,
                                                             int lane) {
    float d = 0.f;
    if (K % 8 == 0 && ((uintptr_t)w & 15) == 0) {
#pragma unroll 4
        for (int i = lane * 8; i < K; i += 256) {
            const uint4 raw = *reinterpret_cast<const uint4*>(w + i);
            const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float2 f = __bfloat1622float2(p[t]);
                d = fmaf(f.x, x[i + 2 * t], d);
                d = fmaf(f.y, x[i + 2 * t + 1], d);
            }
        }
    } else {
        for (int i = lane; i < K; i += 32) d = fmaf(__bfloat162float(w[i]), x[i], d);
    }
    return gb_warp_sum(d);
}

// index of the largest of v[0 .. count) (lowest index among equals) over a warp; every lane gets it; -1 if all are -inf
__device__ __forceinline__ int moe_warp_argmax(const float* v, int count, int lane) {
    float best = -INFINITY;
    int at = -1;
    for (int i = lane; i < count; i += 32) {
        const float c = v[i];
        if (c > best) { best = c; at = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (oa >= 0 && (at < 0 || ob > best || (ob == best && oa < at))) { best = ob; at = oa; }
    }
    return at;
}

// The choice for one row, by one warp: `score`, `choice` (score + correction), `run_score` and `kept` are the row's arrays.
__device__ __forceinline__ void moe_choose(const float* score, float* choice, float* run_score, unsigned char* kept, int E, int top,
                                           int groups, int keep, float route_scale, int* choice_out, float* weight_out, int lane,
                                           int scoring, int run_best, float renorm_eps) {
    const bool softmax_chosen = scoring == MOE_SOFTMAX_CHOSEN;
    if (groups > 1 && keep < groups) {
        const int per = E / groups;
        for (int g = lane; g < groups; g += 32) {
            float a = -INFINITY, b = -INFINITY;          // the two largest of the run
            for (int i = 0; i < per; ++i) {
                const float c = choice[g * per + i];
                if (c > a) { b = a; a = c; } else if (c > b) { b = c; }
            }
            run_score[g] = per > 1 && !run_best ? a + b : a;
            kept[g] = 0;
        }
        __syncwarp();
        for (int k = 0; k < keep; ++k) {
            const int g = moe_warp_argmax(run_score, groups, lane);
            __syncwarp();
            if (lane == 0 && g >= 0) { run_score[g] = -INFINITY; kept[g] = 1; }
            __syncwarp();
        }
        for (int e = lane; e < E; e += 32)
            if (!kept[e / per]) choice[e] = -INFINITY;
        __syncwarp();
    }
    // The chosen values wait in the row's run_score (its use above is over) and reach global memory once, at the end: a
    // store and a load of the same address per choice would put a trip to memory into each turn of this chain.
    for (int k = 0; k < top; ++k) {
        const int e = moe_warp_argmax(choice, E, lane);
        __syncwarp();
        if (lane == 0) {
            choice_out[k] = e;                                               // -1: fewer experts could be chosen than `top`
            run_score[k] = e >= 0 ? score[e] * route_scale : (softmax_chosen ? -INFINITY : 0.f);
            if (e >= 0) choice[e] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (softmax_chosen) {
            // run_score holds the chosen logits, the largest first: softmax over them alone
            const float m = run_score[0];
            float sum = 0.f;
            for (int k = 0; k < top; ++k) {
                const float w = run_score[k] > -INFINITY ? expf(run_score[k] - m) : 0.f;
                run_score[k] = w;
                sum += w;
            }
            const float inv = 1.0f / sum;
            for (int k = 0; k < top; ++k) weight_out[k] = run_score[k] * inv;
        } else {
            float f = 1.0f;
            if (renorm_eps >= 0.f) {
                float sum = renorm_eps;
                for (int k = 0; k < top; ++k) sum += run_score[k];
                f = 1.0f / sum;
            }
            for (int k = 0; k < top; ++k) weight_out[k] = run_score[k] * f;
        }
    }
}

// RB rows per block: a warp per expert (and one for the shared gate) reads its row of the router matrix once and dots it
// with the block's RB rows; then a warp per row chooses. RB = 1 for a handful of rows (shortest chain), 8 for many (the
// router matrix is read an eighth as often). EMAX bounds the experts (the arrays' size).
template <typename T, int RB, int EMAX>
__global__ void __launch_bounds__(RB > 1 ? MOE_ROUTE_THREADS / 2 : MOE_ROUTE_THREADS) moe_route_kernel(
    const T* __restrict__ h, int d, const float* __restrict__ w_router, const float* __restrict__ correction,
    const float* __restrict__ w_gate, const int* __restrict__ positions, int n, int E, int top, int groups, int keep,
    float route_scale, int* __restrict__ choice_out, float* __restrict__ weight_out, float* __restrict__ gate_out,
    const float* __restrict__ router_bias, int scoring, int run_best, float renorm_eps) {
    extern __shared__ __align__(16) float moe_smem[];
    float* hx = moe_smem;                       // RB rows of d numbers (rows start 16-byte aligned: ldh is a multiple of 4)
    const int ldh = (d + 3) & ~3;
    __shared__ float score[RB][EMAX], choice[RB][EMAX], run_score[RB][EMAX];
    __shared__ unsigned char kept[RB][EMAX];
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int row0 = blockIdx.x * RB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)(blockDim.x >> 5);
    int pos[RB];                                // every row's position asked for before the first is used
#pragma unroll
    for (int r = 0; r < RB; ++r) pos[r] = row0 + r < n ? positions[row0 + r] : -1;
    unsigned live = 0;
#pragma unroll
    for (int r = 0; r < RB; ++r) live |= (pos[r] >= 0 ? 1u : 0u) << r;
    if (!live) return;
    constexpr int PIECE = 16 / sizeof(T);
    if (RB > 1 && d % PIECE == 0 && ((uintptr_t)h & 15) == 0) {
        // 16 bytes a load, four of them in flight (one number a load and a row after the other: 37 us for 2,048 rows of 1,024 and
        // 16 experts, now 21)
        const int per_row = d / PIECE, total = RB * per_row;
        for (int i0 = threadIdx.x; i0 < total; i0 += 4 * blockDim.x) {
            uint4 raw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * blockDim.x, r = i / per_row;
                raw[u] = i < total && (live >> r & 1) ? *reinterpret_cast<const uint4*>(h + (size_t)(row0 + r) * d + (i % per_row) * PIECE)
                                                      : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * blockDim.x;
                if (i >= total) break;
                const T* v = reinterpret_cast<const T*>(&raw[u]);
                float* dst = hx + (i / per_row) * ldh + (i % per_row) * PIECE;
#pragma unroll
                for (int c = 0; c < PIECE; c += 4)
                    *reinterpret_cast<float4*>(dst + c) = make_float4(gb_to_float(v[c]), gb_to_float(v[c + 1]), gb_to_float(v[c + 2]), gb_to_float(v[c + 3]));
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const bool on = live >> r & 1;
            const T* src = h + (size_t)(on ? row0 + r : 0) * d;
            for (int i = threadIdx.x; i < d; i += blockDim.x) hx[r * ldh + i] = on ? gb_to_float(src[i]) : 0.f;
        }
    }
    __syncthreads();
    auto settle = [&](int e, const float (&acc)[RB]) {      // a logit per row, or the shared gate's
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const float z = gb_warp_sum(acc[r]);
            const int row = row0 + r;
            if (lane == 0 && (live >> r & 1)) {
                const float sg = moe_sigmoid(z);
                if (e < E && scoring != MOE_SIGMOID) {
                    score[r][e] = choice[r][e] = z + (router_bias ? router_bias[e] : 0.f);
                } else if (e < E) {
                    score[r][e] = sg;
                    choice[r][e] = sg + (correction ? correction[e] : 0.f);
                } else {
                    gate_out[row] = sg;
                }
            }
        }
    };
    int e_from = 0;
    if (RB > 1 && d % 4 == 0 && ((uintptr_t)w_router & 15) == 0) {
        // two experts a warp: the rows come out of shared memory half as often
        for (int e = 2 * warp; e + 1 < E; e += 2 * warps) {
            const float* w0 = w_router + (size_t)e * d;
            float a0[RB], a1[RB];
#pragma unroll
            for (int r = 0; r < RB; ++r) a0[r] = a1[r] = 0.f;
#pragma unroll 4
            for (int i = lane * 4; i < d; i += 128) {
                const float4 v = *reinterpret_cast<const float4*>(w0 + i), u = *reinterpret_cast<const float4*>(w0 + d + i);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const float4 x = *reinterpret_cast<const float4*>(hx + r * ldh + i);
                    a0[r] = fmaf(v.x, x.x, a0[r]); a0[r] = fmaf(v.y, x.y, a0[r]); a0[r] = fmaf(v.z, x.z, a0[r]); a0[r] = fmaf(v.w, x.w, a0[r]);
                    a1[r] = fmaf(u.x, x.x, a1[r]); a1[r] = fmaf(u.y, x.y, a1[r]); a1[r] = fmaf(u.z, x.z, a1[r]); a1[r] = fmaf(u.w, x.w, a1[r]);
                }
            }
            settle(e, a0);
            settle(e + 1, a1);
        }
        e_from = E & ~1;
    }
    for (int e = e_from + warp; e < E + (w_gate ? 1 : 0); e += warps) {
        const float* wrow = e < E ? w_router + (size_t)e * d : w_gate;
        float acc[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) acc[r] = 0.f;
        if (d % 4 == 0 && ((uintptr_t)wrow & 15) == 0) {
#pragma unroll 4
            for (int i = lane * 4; i < d; i += 128) {
                const float4 v = *reinterpret_cast<const float4*>(wrow + i);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const float4 x = *reinterpret_cast<const float4*>(hx + r * ldh + i);
                    acc[r] = fmaf(v.x, x.x, acc[r]); acc[r] = fmaf(v.y, x.y, acc[r]);
                    acc[r] = fmaf(v.z, x.z, acc[r]); acc[r] = fmaf(v.w, x.w, acc[r]);
                }
            }
        } else {
            for (int i = lane; i < d; i += 32) {
                const float v = wrow[i];
#pragma unroll
                for (int r = 0; r < RB; ++r) acc[r] = fmaf(v, hx[r * ldh + i], acc[r]);
            }
        }
        settle(e, acc);
    }
    __syncthreads();
    for (int r = warp; r < RB; r += warps) {
        const int row = row0 + r;
        if (live >> r & 1) {
            if (scoring == MOE_SOFTMAX) {        // the row's logits become its softmax over all experts, by this row's warp
                float m = -INFINITY, sum = 0.f;
                for (int e = lane; e < E; e += 32) m = fmaxf(m, score[r][e]);
                m = gb_warp_max(m);
                for (int e = lane; e < E; e += 32) sum += expf(score[r][e] - m);
                sum = gb_warp_sum(sum);
                for (int e = lane; e < E; e += 32) score[r][e] = choice[r][e] = expf(score[r][e] - m) / sum;
                __syncwarp();
            }
            moe_choose(score[r], choice[r], run_score[r], kept[r], E, top, groups, keep,
                       scoring == MOE_SOFTMAX_CHOSEN ? 1.0f : route_scale, choice_out + (size_t)row * top,
                       weight_out + (size_t)row * top, lane, scoring, run_best, renorm_eps);
        }
    }
}

// The logits of many bfloat16 rows on the tensor cores (mma.sync): 16 rows a block, the K of their products dealt out to 16 warps in pieces
// of 32, sums over the warps in shared memory, then a warp per row chooses. A router weight is the exact sum of three bfloat16 numbers, all of
// whose products with a row's are kept; the largest product of 16 channels has an accumulator of its own and is added in float32 (the
// tensor core cuts what it adds to).
// Operands come straight from memory in 16-byte loads: a lane's eight neighbouring channels stand for the fragment's pairs, the same way
// on both sides. The FMA form brings every row through shared memory as float32 for every two experts: bound by those reads.
// Measured, 16 experts, width 1,024, FMA / this, us: 300 rows 14.0 / 7.7, 2,048 rows 15.4 / 7.9;
// width 2,048 17.4 / 9.2 and 19.5 / 9.5; 128 experts 36 / 27 and 72 / 27.
constexpr int MR_ROWS = 16, MR_WARPS = 16, MR_COLS = 32, MR_EMAX = 128;
struct MrShared {
    float part[MR_WARPS][MR_ROWS][MR_COLS + 1];
    float score[MR_ROWS][MR_EMAX], choice[MR_ROWS][MR_EMAX], run_score[MR_ROWS][MR_EMAX];
    unsigned char kept[MR_ROWS][MR_EMAX];
};

__device__ __forceinline__ void mr_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(MR_WARPS * 32) moe_route_mma_kernel(
    const __nv_bfloat16* __restrict__ h, int d, const float* __restrict__ w_router, const float* __restrict__ correction,
    const float* __restrict__ w_gate, const int* __restrict__ positions, int n, int E, int top, int groups, int keep, float route_scale,
    int* __restrict__ choice_out, float* __restrict__ weight_out, float* __restrict__ gate_out, const float* __restrict__ router_bias,
    int scoring, int run_best, float renorm_eps) {
    extern __shared__ __align__(16) unsigned char mr_mem[];
    MrShared& sh = *reinterpret_cast<MrShared*>(mr_mem);
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int row0 = blockIdx.x * MR_ROWS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int cols = E + (w_gate ? 1 : 0);
    auto column = [&](int e) { return e < E ? w_router + (size_t)e * d : e < cols ? w_gate : nullptr; };
    for (int e0 = 0; e0 < cols; e0 += MR_COLS) {
        float hi[MR_COLS / 8][4] = {}, lo[MR_COLS / 8][4] = {};
        for (int k = warp * 32 + 8 * t4; k - 8 * t4 < d; k += MR_WARPS * 32) {
            const uint4 none = make_uint4(0, 0, 0, 0);
            const bool in = k < d;
            const uint4 x0 = in && row0 + g < n ? *reinterpret_cast<const uint4*>(h + (size_t)(row0 + g) * d + k) : none;
            const uint4 x1 = in && row0 + g + 8 < n ? *reinterpret_cast<const uint4*>(h + (size_t)(row0 + g + 8) * d + k) : none;
            float4 w[MR_COLS / 8][2];
#pragma unroll
            for (int c = 0; c < MR_COLS / 8; ++c) {
                const float* src = column(e0 + 8 * c + g);
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    w[c][s] = in && src ? *reinterpret_cast<const float4*>(src + k + 4 * s) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int c = 0; c < MR_COLS / 8; ++c) {
                if (e0 + 8 * c >= cols) break;                          // (uniform for the block)
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    uint32_t b0[3], b1[3];
                    gb_split_bf16(w[c][s].x, w[c][s].y, b0);
                    gb_split_bf16(w[c][s].z, w[c][s].w, b1);
                    const uint32_t a0 = s ? x0.z : x0.x, a1 = s ? x1.z : x1.x, a2 = s ? x0.w : x0.y, a3 = s ? x1.w : x1.y;
                    float sum[4] = {0.f, 0.f, 0.f, 0.f};
                    mr_mma(lo[c], a0, a1, a2, a3, b0[2], b1[2]);
                    mr_mma(lo[c], a0, a1, a2, a3, b0[1], b1[1]);
                    mr_mma(sum, a0, a1, a2, a3, b0[0], b1[0]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) hi[c][i] += sum[i];
                }
            }
        }
#pragma unroll
        for (int c = 0; c < MR_COLS / 8; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) sh.part[warp][g + 8 * (i >> 1)][8 * c + 2 * t4 + (i & 1)] = hi[c][i] + lo[c][i];
        __syncthreads();
        {
            const int r = threadIdx.x / MR_COLS, e = e0 + threadIdx.x % MR_COLS, row = row0 + r;
            if (e < cols && row < n && positions[row] >= 0) {
                float z = 0.f;
#pragma unroll
                for (int i = 0; i < MR_WARPS; ++i) z += sh.part[i][r][e - e0];
                if (!(fabsf(z) <= FLT_MAX)) {                           // (an infinite operand's lesser terms are no numbers)
                    const float* src = column(e);
                    z = 0.f;
                    for (int k = 0; k < d; ++k) z = fmaf(__bfloat162float(h[(size_t)row * d + k]), src[k], z);
                }
                const float sg = moe_sigmoid(z);
                if (e == E) gate_out[row] = sg;
                else if (scoring != MOE_SIGMOID) sh.score[r][e] = sh.choice[r][e] = z + (router_bias ? router_bias[e] : 0.f);
                else {
                    sh.score[r][e] = sg;
                    sh.choice[r][e] = sg + (correction ? correction[e] : 0.f);
                }
            }
        }
        __syncthreads();
    }
    const int r = warp, row = row0 + r;
    if (row >= n || positions[row] < 0) return;
    if (scoring == MOE_SOFTMAX) {                                       // the row's logits become its softmax over all experts
        float m = -INFINITY, sum = 0.f;
        for (int e = lane; e < E; e += 32) m = fmaxf(m, sh.score[r][e]);
        m = gb_warp_max(m);
        for (int e = lane; e < E; e += 32) sum += expf(sh.score[r][e] - m);
        sum = gb_warp_sum(sum);
        for (int e = lane; e < E; e += 32) sh.score[r][e] = sh.choice[r][e] = expf(sh.score[r][e] - m) / sum;
        __syncwarp();
    }
    moe_choose(sh.score[r], sh.choice[r], sh.run_score[r], sh.kept[r], E, top, groups, keep, scoring == MOE_SOFTMAX_CHOSEN ? 1.0f : route_scale,
               choice_out + (size_t)row * top, weight_out + (size_t)row * top, lane, scoring, run_best, renorm_eps);
}

template <typename T, int RB, int EMAX>
static void moe_route_launch(const void* h, int d, const float* w_router, const float* correction, const float* w_gate,
                             const int* positions, int n, int E, int top, int groups, int keep, float route_scale, int* choice_out,
                             float* weight_out, float* gate_out, const float* router_bias, int scoring, int run_best, float renorm_eps,
                             cudaStream_t stream) {
    const size_t smem = (size_t)RB * ((d + 3) & ~3) * 4;
    int warps = RB > 1 ? (E + 1) / 2 : E + (w_gate ? 1 : 0);
    const int most = (RB > 1 ? MOE_ROUTE_THREADS / 2 : MOE_ROUTE_THREADS) / 32, least = RB > 4 ? RB : 4;
    warps = warps < least ? least : (warps > most ? most : warps);
    if (smem > 32 * 1024) cudaFuncSetAttribute(moe_route_kernel<T, RB, EMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gb_launch(GB_PDL_ELEMENTWISE, moe_route_kernel<T, RB, EMAX>, dim3(gb_ceil_div(n, RB)), dim3(32 * warps), smem, stream, (const T*)h, d,
              w_router, correction, w_gate, positions, n, E, top, groups, keep, route_scale, choice_out, weight_out, gate_out, router_bias,
              scoring, run_best, renorm_eps);
}

GB_EXPORT int gb_moe_route(const void* h, int h_dtype, int d, const float* w_router, const float* correction, const float* w_gate,
                           const int* positions, int n, int E, int top, int groups, int keep, float route_scale, int* choice_out,
                           float* weight_out, float* gate_out, const float* router_bias, int scoring, int run_best, float renorm_eps,
                           cudaStream_t stream) {
    GB_REQUIRE(scoring >= MOE_SIGMOID && scoring <= MOE_SOFTMAX, "gb_moe_route: unknown scoring %d", scoring);
    GB_REQUIRE(scoring == MOE_SIGMOID || correction == nullptr, "gb_moe_route: a choice correction goes with sigmoid scores");
    GB_REQUIRE(scoring != MOE_SOFTMAX_CHOSEN || groups == 1, "gb_moe_route: softmax over the chosen logits goes without groups");
    GB_REQUIRE(n >= 0 && d > 0 && E > 0 && E <= MOE_MAX_EXPERTS && top > 0 && top <= E, "gb_moe_route: bad sizes (experts %d, top %d)", E,
               top);
    GB_REQUIRE(groups >= 1 && E % groups == 0 && keep >= 1 && keep <= groups, "gb_moe_route: %d experts in %d groups, %d kept", E, groups,
               keep);
    GB_REQUIRE((size_t)d * 4 <= 160 * 1024, "gb_moe_route: a row of %d numbers does not fit shared memory", d);
    GB_REQUIRE(w_gate == nullptr || gate_out != nullptr, "gb_moe_route: a gate needs its output");
    GB_REQUIRE(h_dtype == GB_F32 || h_dtype == GB_BF16, "gb_moe_route: unsupported dtype %d", h_dtype);
    if (n == 0) return 0;
    // From the rows on for which the FMA form takes eight rows a block: 256 rows, a row a block, 16 experts 5.7 us against 7.7, 128 experts
    // 24 against 27. The sums over K are taken in another order here, so a logit's low bits, and with them the choice between experts that
    // are all but equal, depend on whether 256 rows or more are routed together (as a bfloat16 row's hidden numbers do on the products'
    // forms, which are chosen by rows too).
    if (h_dtype == GB_BF16 && n > 256 && E <= MR_EMAX && d % 8 == 0 && (((uintptr_t)h | (uintptr_t)w_router | (uintptr_t)w_gate) & 15) == 0) {
        cudaError_t e = cudaFuncSetAttribute(moe_route_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MrShared));
        GB_REQUIRE(e == cudaSuccess, "gb_moe_route: %d bytes of shared memory refused: %s", (int)sizeof(MrShared), cudaGetErrorString(e));
        gb_launch(GB_PDL_ELEMENTWISE, moe_route_mma_kernel, dim3(gb_ceil_div(n, MR_ROWS)), dim3(MR_WARPS * 32), sizeof(MrShared), stream,
                  (const __nv_bfloat16*)h, d, w_router, correction, w_gate, positions, n, E, top, groups, keep, route_scale, choice_out, weight_out,
                  gate_out, router_bias, scoring, run_best, renorm_eps);
        return gb_check_launch("gb_moe_route");
    }
    // eight rows per block when there are many rows, the experts are few enough for the block's arrays and eight rows fit
    const bool many = n > 256 && E <= 128 && (size_t)8 * ((d + 3) & ~3) * 4 <= 160 * 1024;      // (below: too few blocks to fill the GPU)
#define MOE_ROUTE_GO(T)                                                                                                              \
    if (many)                                                                                                                        \
        moe_route_launch<T, 8, 128>(h, d, w_router, correction, w_gate, positions, n, E, top, groups, keep, route_scale, choice_out,  \
                                    weight_out, gate_out, router_bias, scoring, run_best, renorm_eps, stream);                       \
    else                                                                                                                             \
        moe_route_launch<T, 1, MOE_MAX_EXPERTS>(h, d, w_router, correction, w_gate, positions, n, E, top, groups, keep, route_scale,  \
                                                choice_out, weight_out, gate_out, router_bias, scoring, run_best, renorm_eps, stream);
    if (h_dtype == GB_F32) { MOE_ROUTE_GO(float) } else { MOE_ROUTE_GO(__nv_bfloat16) }
#undef MOE_ROUTE_GO
    return gb_check_launch("gb_moe_route");
}

// ----------------------------------------------------------------------------------------------
// One block per (row, choice k): pair[row, k, :] = W_down[e] relu(W_up[e] h[row])^2, e = choice[row, k].
// w_up [E * ff, d], w_down [E * d, ff] (the experts' matrices stacked by rows).
// ----------------------------------------------------------------------------------------------
constexpr int MOE_ROWS_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(MOE_ROWS_THREADS) moe_expert_rows_kernel(
    const T* __restrict__ h, int d, const T* __restrict__ w_up, const T* __restrict__ w_down, int ff, const int* __restrict__ choice,
    const int* __restrict__ positions, int n, int E, int top, float* __restrict__ pair) {
    extern __shared__ __align__(16) float moe_smem[];
    float* hx = moe_smem;            // d
    float* act = moe_smem + ((d + 3) & ~3);     // ff
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int row = blockIdx.x, k = blockIdx.y;
    if (row >= n || positions[row] < 0) return;
    const int e = choice[(size_t)row * top + k];
    float* dst = pair + ((size_t)row * top + k) * d;
    if (e < 0 || e >= E) {
        for (int i = threadIdx.x; i < d; i += MOE_ROWS_THREADS) dst[i] = 0.f;
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* src = h + (size_t)row * d;
    for (int i = threadIdx.x; i < d; i += MOE_ROWS_THREADS) hx[i] = gb_to_float(src[i]);
    __syncthreads();
    const T* up = w_up + (size_t)e * ff * d;
    for (int f = warp; f < ff; f += MOE_ROWS_THREADS / 32) {
        const float a = fmaxf(moe_warp_dot<T>(up + (size_t)f * d, hx, d, lane), 0.f);
        if (lane == 0) act[f] = a * a;
    }
    __syncthreads();
    const T* down = w_down + (size_t)e * d * ff;
    for (int c = warp; c < d; c += MOE_ROWS_THREADS / 32) {
        const float o = moe_warp_dot<T>(down + (size_t)c * ff, act, ff, lane);
        if (lane == 0) dst[c] = o;
    }
}

GB_EXPORT int gb_moe_expert_rows(const void* h, int dtype, int d, const void* w_up, const void* w_down, int ff, const int* choice,
                                 const int* positions, int n, int E, int top, float* pair, cudaStream_t stream) {
    GB_REQUIRE(n >= 0 && d > 0 && ff > 0 && E > 0 && top > 0, "gb_moe_expert_rows: bad sizes");
    const size_t smem = ((size_t)((d + 3) & ~3) + ff) * 4;
    GB_REQUIRE(smem <= 200 * 1024, "gb_moe_expert_rows: a row of %d and %d hidden numbers do not fit shared memory", d, ff);
    if (n == 0) return 0;
    dim3 grid(n, top);
    if (dtype == GB_F32) {
        if (smem > 32 * 1024) cudaFuncSetAttribute(moe_expert_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        gb_launch(GB_PDL_GEMM, moe_expert_rows_kernel<float>, grid, dim3(MOE_ROWS_THREADS), smem, stream, (const float*)h, d,
                  (const float*)w_up, (const float*)w_down, ff, choice, positions, n, E, top, pair);
    } else if (dtype == GB_BF16) {
        if (smem > 32 * 1024)
            cudaFuncSetAttribute(moe_expert_rows_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        gb_launch(GB_PDL_GEMM, moe_expert_rows_kernel<__nv_bfloat16>, grid, dim3(MOE_ROWS_THREADS), smem, stream, (const __nv_bfloat16*)h,
                  d, (const __nv_bfloat16*)w_up, (const __nv_bfloat16*)w_down, ff, choice, positions, n, E, top, pair);
    } else {
        GB_REQUIRE(false, "gb_moe_expert_rows: unsupported dtype %d", dtype);
    }
    return gb_check_launch("gb_moe_expert_rows");
}

// ----------------------------------------------------------------------------------------------
// out[row, :] (+)= sum_k weight[row, k] * pair[row, k, :] + gate[row] * shared[row, :]
// ----------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ pair, const float* __restrict__ weight, int top,
                                                          const float* __restrict__ shared, long long lds, const float* __restrict__ gate,
                                                          const int* __restrict__ positions, float* __restrict__ out, long long ldo,
                                                          int n, int d, int accumulate, int vec) {
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int row = blockIdx.x;
    if (row >= n || positions[row] < 0) return;
    const float g = gate ? gate[row] : 1.f;
    if (vec) {         // four columns a thread, four choices' loads in flight (8,192 pairs of 1,024: 15 -> 7.5 us)
        for (int j = threadIdx.x * 4; j < d; j += blockDim.x * 4) {
            const float* src = pair + (size_t)row * top * d + j;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            float4* o = reinterpret_cast<float4*>(out + (size_t)row * ldo + j);
            const float4 old = accumulate ? *o : a, s = shared ? *reinterpret_cast<const float4*>(shared + (size_t)row * lds + j) : a;
            for (int k0 = 0; k0 < top; k0 += 4) {
                float4 v[4];
                float w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k0 + k < top) {
                        v[k] = *reinterpret_cast<const float4*>(src + (size_t)(k0 + k) * d);
                        w[k] = weight[(size_t)row * top + k0 + k];
                    }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k0 + k < top) {
                        a.x = fmaf(w[k], v[k].x, a.x); a.y = fmaf(w[k], v[k].y, a.y);
                        a.z = fmaf(w[k], v[k].z, a.z); a.w = fmaf(w[k], v[k].w, a.w);
                    }
            }
            if (shared) { a.x = fmaf(g, s.x, a.x); a.y = fmaf(g, s.y, a.y); a.z = fmaf(g, s.z, a.z); a.w = fmaf(g, s.w, a.w); }
            if (accumulate) { a.x = old.x + a.x; a.y = old.y + a.y; a.z = old.z + a.z; a.w = old.w + a.w; }
            *o = a;
        }
        return;
    }
    for (int j = threadIdx.x; j < d; j += blockDim.x) {
        float a = 0.f;
        for (int k = 0; k < top; ++k) a = fmaf(weight[(size_t)row * top + k], pair[((size_t)row * top + k) * d + j], a);
        if (shared) a = fmaf(g, shared[(size_t)row * lds + j], a);
        float* o = out + (size_t)row * ldo + j;
        *o = accumulate ? *o + a : a;
    }
}

GB_EXPORT int gb_moe_combine(const float* pair, const float* weight, int top, const float* shared, long long lds, const float* gate,
                             const int* positions, float* out, long long ldo, int n, int d, int accumulate, cudaStream_t stream) {
    GB_REQUIRE(n >= 0 && d > 0 && top > 0, "gb_moe_combine: bad sizes");
    if (n == 0) return 0;
    const bool vec = d % 4 == 0 && ldo % 4 == 0 && lds % 4 == 0 && (((uintptr_t)pair | (uintptr_t)out | (uintptr_t)shared) & 15) == 0;
    gb_launch(GB_PDL_ELEMENTWISE, moe_combine_kernel, dim3(n), dim3(256), 0, stream, pair, weight, top, shared, lds, gate, positions, out,
              ldo, n, d, accumulate, vec ? 1 : 0);
    return gb_check_launch("gb_moe_combine");
}

// ----------------------------------------------------------------------------------------------
// The two halves of moe_expert_rows as kernels of their own, many blocks per (row, choice): the form for a handful of rows
// (decoding), where one block per pair would leave most of the GPU idle. act float32 [n * top, ff].
//   up:   act[pair, f]  = relu(W_up[e][f, :] . h[row])^2         grid (pairs, ceil(ff / 8)), a warp per f
//   down: pair[pair, c] = W_down[e][c, :] . act[pair, :]         grid (pairs, ceil(d / 8)), a warp per c
// ----------------------------------------------------------------------------------------------
template <typename T, bool UP>
__global__ void __launch_bounds__(256) moe_half_rows_kernel(const void* __restrict__ in_, long long ld_in, const T* __restrict__ w, int N,
                                                            int K, const int* __restrict__ choice, const int* __restrict__ positions,
                                                            int n, int E, int top, float* __restrict__ out, long long ld_out,
                                                            int unit, float limit, float slope) {
    extern __shared__ __align__(16) float moe_smem[];
    float* x = moe_smem;       // K numbers: the row h (UP) or the pair's activations (DOWN)
    const int pair = blockIdx.x, row = pair / top;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.y * 8 + warp;
    gb_pdl_launch_dependents();
    gb_pdl_wait();                // (the choice is the router kernel's output: nothing of it may be read before this)
    const int e = (row < n && positions[row] >= 0) ? choice[pair] : -2;
    // (with the gated unit an expert has 2N rows: output c reads its gate row 2c and its up row 2c + 1)
    const T* wrow = (e >= 0 && e < E && c < N) ? w + ((size_t)e * N + c) * K * (UP && unit ? 2 : 1) : nullptr;
    if (e == -2) return;
    if (e < 0 || e >= E) {
        if (c < N && lane == 0) out[(size_t)pair * ld_out + c] = 0.f;
        return;
    }
    if (UP) {
        const T* src = (const T*)in_ + (size_t)row * ld_in;
        for (int i = threadIdx.x; i < K; i += 256) x[i] = gb_to_float(src[i]);
    } else {
        const float* src = (const float*)in_ + (size_t)pair * ld_in;
        for (int i = threadIdx.x; i < K; i += 256) x[i] = src[i];
    }
    __syncthreads();
    if (wrow == nullptr) return;
    float v = moe_warp_dot<T>(wrow, x, K, lane);
    if (UP && unit) {
        v = gb_gated_unit(v, moe_warp_dot<T>(wrow + K, x, K, lane), limit, slope);
    } else if (UP) {
        v = fmaxf(v, 0.f);
        v *= v;
    }
    if (lane == 0) out[(size_t)pair * ld_out + c] = v;
}

// The same with four matrix rows a warp (32 a block): the 16-byte loads of four rows are under way together and a block's copy of
// its input serves four times the weights. One row a warp had at most four loads in flight and a barrier per 32 KB of weights.
// For K in whole 16-byte pieces of aligned matrices. Measured, 8 rows, two of 16 experts, 2048 x 2048 bfloat16 (16 pairs,
// 134 MB of which about 84 distinct): up half 28.7 -> 19.2 us, down half 28.4 -> 17.1; with the first loads after the staging
// instead of before it 26.5 and 28.8.
constexpr int MH_STEPS = 4;     // 16-byte loads a lane and row under way: the first are requested before the input is staged

template <typename T, bool UP>
__global__ void __launch_bounds__(256) moe_half_rows4_kernel(const void* __restrict__ in_, long long ld_in, const T* __restrict__ w, int N,
                                                             int K, const int* __restrict__ choice, const int* __restrict__ positions,
                                                             int n, int E, int top, float* __restrict__ out, long long ld_out,
                                                             int unit, float limit, float slope) {
    constexpr int PN = 16 / sizeof(T);
    extern __shared__ __align__(16) float moe_smem[];
    float* x = moe_smem;
    const int pair = blockIdx.x, row = pair / top;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool gated = UP && unit;
    const int rows = gated ? 2 * N : N, r0 = blockIdx.y * 32 + warp * 4;
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int e = (row < n && positions[row] >= 0) ? choice[pair] : -2;
    if (e == -2) return;
    float* dst = out + (size_t)pair * ld_out;
    if (e < 0 || e >= E) {
        for (int c = blockIdx.y * (gated ? 16 : 32) + threadIdx.x; c < min(N, (int)(blockIdx.y + 1) * (gated ? 16 : 32)); c += 256) dst[c] = 0.f;
        return;
    }
    const T* base = w + ((size_t)e * rows + r0) * K;
    uint4 raw[MH_STEPS][4];
    auto request = [&](int k0) {
#pragma unroll
        for (int s = 0; s < MH_STEPS; ++s) {
            const int i = k0 + (s * 32 + lane) * PN;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                raw[s][j] = (i < K && r0 + j < rows) ? __ldg(reinterpret_cast<const uint4*>(base + (size_t)j * K + i)) : make_uint4(0, 0, 0, 0);
        }
    };
    request(0);
    if (UP) {
        const T* src = (const T*)in_ + (size_t)row * ld_in;
        for (int i = threadIdx.x; i < K; i += 256) x[i] = gb_to_float(src[i]);
    } else {
        const float* src = (const float*)in_ + (size_t)pair * ld_in;
        for (int i = threadIdx.x; i < K; i += 256) x[i] = src[i];
    }
    __syncthreads();
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = 0; k0 < K; k0 += MH_STEPS * 32 * PN) {
        if (k0 > 0) request(k0);
#pragma unroll
        for (int s = 0; s < MH_STEPS; ++s) {
            const int i = k0 + (s * 32 + lane) * PN;
            if (i >= K) break;
            float xv[PN];
#pragma unroll
            for (int t = 0; t < PN; t += 4) *reinterpret_cast<float4*>(xv + t) = *reinterpret_cast<const float4*>(x + i + t);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t p[4] = {raw[s][j].x, raw[s][j].y, raw[s][j].z, raw[s][j].w};
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if constexpr (sizeof(T) == 2) {
                        v[j] = fmaf(__uint_as_float(p[t] << 16), xv[2 * t], v[j]);
                        v[j] = fmaf(__uint_as_float(p[t] & 0xffff0000u), xv[2 * t + 1], v[j]);
                    } else {
                        v[j] = fmaf(__uint_as_float(p[t]), xv[t], v[j]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = gb_warp_sum(v[j]);
    if (lane > 0) return;
    if (gated) {
#pragma unroll
        for (int j = 0; j < 4; j += 2)
            if (r0 + j < rows) dst[(r0 + j) >> 1] = gb_gated_unit(v[j], v[j + 1], limit, slope);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (r0 + j >= rows) break;
            const float a = UP ? fmaxf(v[j], 0.f) : v[j];
            dst[r0 + j] = UP ? a * a : a;
        }
    }
}

template <typename T, bool UP>
static void moe_half_rows_one(const void* in, long long ld_in, const T* w, int N, int K, const int* choice, const int* positions, int n, int E,
                              int top, float* out, long long ld_out, int unit, float limit, float slope, cudaStream_t stream) {
    const size_t smem = (size_t)K * 4;
    const long long rows = UP && unit ? 2LL * N : N;
    // (at no size slower than a row a warp: 8 rows of 512 x 512 18.4 us the feed-forward against 21.9, one row 16.4 both)
    const bool four = K % (16 / sizeof(T)) == 0 && K % 4 == 0 && (uintptr_t)w % 16 == 0;
    auto kernel = four ? moe_half_rows4_kernel<T, UP> : moe_half_rows_kernel<T, UP>;
    if (smem > 32 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int blocks = four ? (int)((rows + 31) / 32) : gb_ceil_div(N, 8);
    gb_launch(GB_PDL_GEMM, kernel, dim3(n * top, blocks), dim3(256), smem, stream, in, ld_in, w, N, K, choice, positions, n, E, top, out, ld_out,
              unit, limit, slope);
}

template <typename T>
static int moe_half_rows_launch(const void* h, int d, const T* w_up, const T* w_down, int ff, const int* choice, const int* positions,
                                int n, int E, int top, float* act, float* pair, int unit, float limit, float slope, cudaStream_t stream) {
    moe_half_rows_one<T, true>(h, d, w_up, ff, d, choice, positions, n, E, top, act, ff, unit, limit, slope, stream);
    int rc = gb_check_launch("gb_moe_expert_halves (up)");
    if (rc) return rc;
    moe_half_rows_one<T, false>(act, ff, w_down, d, ff, choice, positions, n, E, top, pair, d, 0, 0.f, 0.f, stream);
    return gb_check_launch("gb_moe_expert_halves (down)");
}

GB_EXPORT int gb_moe_expert_halves(const void* h, int dtype, int d, const void* w_up, const void* w_down, int ff, const int* choice,
                                   const int* positions, int n, int E, int top, float* act, float* pair, int unit, float limit, float slope,
                                   cudaStream_t stream) {
    GB_REQUIRE(n >= 0 && d > 0 && ff > 0 && E > 0 && top > 0, "gb_moe_expert_halves: bad sizes");
    GB_REQUIRE((size_t)d * 4 <= 200 * 1024 && (size_t)ff * 4 <= 200 * 1024, "gb_moe_expert_halves: rows of %d / %d numbers do not fit", d, ff);
    if (n == 0) return 0;
    if (dtype == GB_F32)
        return moe_half_rows_launch<float>(h, d, (const float*)w_up, (const float*)w_down, ff, choice, positions, n, E, top, act, pair, unit,
                                           limit, slope, stream);
    if (dtype == GB_BF16)
        return moe_half_rows_launch<__nv_bfloat16>(h, d, (const __nv_bfloat16*)w_up, (const __nv_bfloat16*)w_down, ff, choice, positions,
                                                   n, E, top, act, pair, unit, limit, slope, stream);
    GB_REQUIRE(false, "gb_moe_expert_halves: unsupported dtype %d", dtype);
}

// ----------------------------------------------------------------------------------------------
// Many rows (prompt portions, large batches), bfloat16: the (row, choice) pairs are sorted by expert, and the experts'
// products run as one grouped product per half on the tensor cores (moe_tcgen05.cu).
//   moe_sort            one block: counts per expert, where each expert's pairs start (offsets [E + 1]) and sorted[slot] = pair.
//                       The order of an expert's pairs is not fixed from run to run; no result depends on it (a pair's
//                       numbers do not depend on its slot).
// A thread keeps up to 16 pairs' experts in registers, asked for together: the two passes over the pairs cost one trip to
// memory between them.
// ----------------------------------------------------------------------------------------------
constexpr int MS_THREADS = 1024, MS_KEEP = 16;

__global__ void __launch_bounds__(MS_THREADS) moe_sort_kernel(const int* __restrict__ choice, const int* __restrict__ positions, int n, int E,
                                                              int top, int* __restrict__ offsets, int* __restrict__ sorted) {
    __shared__ int count[MOE_MAX_EXPERTS], cursor[MOE_MAX_EXPERTS];
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    for (int e = threadIdx.x; e < E; e += MS_THREADS) count[e] = 0;
    const int pairs = n * top;
    auto expert_of = [&](int p) {
        if (p >= pairs) return -1;
        const int e = positions[p / top] >= 0 ? choice[p] : -1;
        return e >= 0 && e < E ? e : -1;
    };
    int own[MS_KEEP];
#pragma unroll
    for (int i = 0; i < MS_KEEP; ++i) own[i] = expert_of(threadIdx.x + i * MS_THREADS);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MS_KEEP; ++i)
        if (own[i] >= 0) atomicAdd(&count[own[i]], 1);
    for (int p = threadIdx.x + MS_KEEP * MS_THREADS; p < pairs; p += MS_THREADS) {
        const int e = expert_of(p);
        if (e >= 0) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int before = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + threadIdx.x, c = e < E ? count[e] : 0;
            int sum = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, o);
                if ((int)threadIdx.x >= o) sum += v;
            }
            if (e < E) offsets[e] = cursor[e] = before + sum - c;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (threadIdx.x == 0) offsets[E] = before;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MS_KEEP; ++i)
        if (own[i] >= 0) sorted[atomicAdd(&cursor[own[i]], 1)] = threadIdx.x + i * MS_THREADS;
    for (int p = threadIdx.x + MS_KEEP * MS_THREADS; p < pairs; p += MS_THREADS) {
        const int e = expert_of(p);
        if (e >= 0) sorted[atomicAdd(&cursor[e], 1)] = p;
    }
}

// The same for up to MS_FEW experts and MS_KEEP pairs a thread, without two pairs ever meeting at one counter: a thread counts its own pairs in
// a column of its own, a warp per expert turns the counts of its row into the threads' first slots, and the thread deals them out. (8,192
// pairs of 16 experts were 2 x 256 additions of 32 lanes to a handful of addresses, a division a pair and scattered stores: 7.8 us, 6.0 so.) An expert's pairs come in a fixed order.
// What it costs whatever the pairs (columns to clear and to add up) pays from 3,072 pairs on, of more than 32 experts from 96 an expert. By
// additions / by columns, us: 16 experts 256 pairs 3.3 / 4.4, 2,048 4.3 / 4.5, 3,072 4.9 / 4.7, 16,384 13.2 / 8.4; 32 experts 2,048 4.5 /
// 5.0, 3,072 5.6 / 5.2; 64 experts 512 3.4 / 6.0, 4,096 6.5 / 6.8, 6,144 8.4 / 7.0, 8,192 10.0 / 7.7.
constexpr int MS_FEW = 64, MS_MANY = 3072;

__global__ void __launch_bounds__(MS_THREADS) moe_sort_columns_kernel(const int* __restrict__ choice, const int* __restrict__ positions, int n,
                                                                      int E, int top, int* __restrict__ offsets, int* __restrict__ sorted) {
    extern __shared__ __align__(16) unsigned char ms_mem[];
    unsigned short* cell = reinterpret_cast<unsigned short*>(ms_mem);      // [E][MS_THREADS]: a thread's pairs of an expert, then its first slot's
    __shared__ int start[MS_FEW + 1];                                      // distance from the expert's first
    int* slots = reinterpret_cast<int*>(ms_mem + (size_t)E * MS_THREADS * 2);      // [pairs]: the pairs by slot
    gb_pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < E * MS_THREADS / 8; i += MS_THREADS) reinterpret_cast<uint4*>(cell)[i] = make_uint4(0, 0, 0, 0);
    gb_pdl_wait();
    const int pairs = n * top;
    int own[MS_KEEP];                                                      // of quads of pairs 4 (tid + i * MS_THREADS) ..: one division each
    {
        int pos[MS_KEEP];
#pragma unroll
        for (int i = 0; i < MS_KEEP / 4; ++i) {
            const int p = 4 * (tid + i * MS_THREADS);
            int row = p / top, rest = p - row * top;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = p + u < pairs;
                own[4 * i + u] = in ? choice[p + u] : -1;
                pos[4 * i + u] = in ? positions[row] : -1;
                if (++rest == top) {
                    rest = 0;
                    ++row;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < MS_KEEP; ++i)
            if (pos[i] < 0 || own[i] >= E) own[i] = -1;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MS_KEEP; ++i)
        if (own[i] >= 0) ++cell[own[i] * MS_THREADS + tid];
    __syncthreads();
    for (int e = warp; e < E; e += MS_THREADS / 32) {                      // a lane has 32 threads' counts, two in every 32nd word
        uint32_t* row = reinterpret_cast<uint32_t*>(cell + e * MS_THREADS) + lane;
        uint32_t w[MS_THREADS / 64];
        int total = 0;
#pragma unroll
        for (int i = 0; i < MS_THREADS / 64; ++i) {
            w[i] = row[32 * i];
            total += (int)(w[i] & 0xffffu) + (int)(w[i] >> 16);
        }
        int sum = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        int before = sum - total;
#pragma unroll
        for (int i = 0; i < MS_THREADS / 64; ++i) {
            const int low = (int)(w[i] & 0xffffu);
            row[32 * i] = (uint32_t)before | (uint32_t)(before + low) << 16;
            before += low + (int)(w[i] >> 16);
        }
        if (lane == 31) start[e + 1] = sum;
    }
    __syncthreads();
    if (warp == 0) {
        int before = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane, c = e < E ? start[e + 1] : 0;
            int sum = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += v;
            }
            __syncwarp();                                                  // (start[e + 1] has been read by all before it is an expert's start)
            if (e < E) offsets[e] = start[e] = before + sum - c;
            before += __shfl_sync(0xffffffffu, sum, 31);
            __syncwarp();
        }
        if (lane == 0) offsets[E] = start[E] = before;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MS_KEEP; ++i)
        if (own[i] >= 0) slots[start[own[i]] + cell[own[i] * MS_THREADS + tid]++] = 4 * (tid + i / 4 * MS_THREADS) + i % 4;
    __syncthreads();
    // (by way of shared memory: 8,192 scattered stores of one multiprocessor take 8,300 cycles)
    for (int i = tid; i < start[E]; i += MS_THREADS) sorted[i] = slots[i];
}

GB_EXPORT int gb_moe_sort(const int* choice, const int* positions, int n, int E, int top, int* offsets, int* sorted, cudaStream_t stream) {
    GB_REQUIRE(n >= 0 && E > 0 && E <= MOE_MAX_EXPERTS && top > 0, "gb_moe_sort: bad sizes");
    if (n == 0) return 0;
    const long long pairs = (long long)n * top;
    if (E <= MS_FEW && pairs <= (long long)MS_KEEP * MS_THREADS && pairs >= MS_MANY && pairs >= 96 * E) {
        // (the limit is the most that any sizes need: a kernel has one, and a thread with few pairs must not lower it under another's launch)
        constexpr int most = MS_FEW * MS_THREADS * (int)sizeof(unsigned short) + MS_KEEP * MS_THREADS * (int)sizeof(int);
        const int smem = E * MS_THREADS * (int)sizeof(unsigned short) + n * top * (int)sizeof(int);
        cudaError_t e = cudaFuncSetAttribute(moe_sort_columns_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        GB_REQUIRE(e == cudaSuccess, "gb_moe_sort: %d bytes of shared memory refused: %s", most, cudaGetErrorString(e));
        e = gb_launch(GB_PDL_ELEMENTWISE, moe_sort_columns_kernel, dim3(1), dim3(MS_THREADS), smem, stream, choice, positions, n, E, top, offsets, sorted);
        GB_REQUIRE(e == cudaSuccess, "gb_moe_sort: launch failed: %s", cudaGetErrorString(e));
        return gb_check_launch("gb_moe_sort");
    }
    gb_launch(GB_PDL_ELEMENTWISE, moe_sort_kernel, dim3(1), dim3(MS_THREADS), 0, stream, choice, positions, n, E, top, offsets, sorted);
    return gb_check_launch("gb_moe_sort");
}
