// The gated delta rule over prompt portions, 32 tokens at a time (the walk token by token is in delta_rule.cu).
//
// With S_0 the state in front of a chunk, P_i the product of the chunk's decays up to and including token i (per key channel)
// and D_ij that of the decays after token j up to token i, the recurrence S <- diag(g) S; u = beta (v - S^T k); S <- S + k u^T;
// o = S^T q unrolls to
//     u_i + beta_i sum_{j<i} A_ij u_j = beta_i (v_i - (k_i P_i)^T S_0),      A_ij = sum_c k_i[c] D_ij[c] k_j[c]
//     o_i = (q_i P_i)^T S_0 + sum_{j<=i} B_ij u_j,                            B_ij = sum_c q_i[c] D_ij[c] k_j[c]
//     S_32 = diag(P_32) S_0 + sum_j (k_j D_(32)j) u_j^T
// (the WY form of a product of Householder-like factors; Bischof and Van Loan 1987, with decays as in gated linear
// attention). With T = (1 + diag(beta) A)^(-1) diag(beta) (A strictly lower triangular: forward substitution) and M = B T a
// chunk is W = V - (K P) S_0, U = T W, O = (Q P) S_0 + M W, S_32 = P_32 S_0 + (K D)^T U: products, and nothing but S passes
// from chunk to chunk. Decays only ever appear as products of themselves, never as quotients, so nothing overflows
// however fast a channel forgets. Everything is float32, sums and operands, as in the walk.
//
//   delta_prepare_kernel  every (chunk, head) side by side: unit vectors, decays, A, B, T, M into a workspace
//   delta_scan_kernel     a block per (request, head, 8 columns of S): chunk after chunk, S in shared memory
//
// What bounds it: the walk was a chain of 0.3 us per token whatever the chip could do (one warp's dependent instructions);
// here a block pays a chunk's shared-memory traffic (a 16-byte load takes the pipe four cycles whoever shares it: 1,280 of 4,000
// cycles a chunk in the first product alone) and six barriers, 0.07 us per token.
// Measured, 8 heads x 128 x 128, 2,048 tokens of one request: walk 724 us; prepare 44 + scan 139 us (16 heads 85 + 215 us).
#include "common.cuh"

constexpr int DC_C = 32;                            // tokens of a chunk
constexpr int DC_K = 128;                           // key channels (smaller key sizes are padded: k = q = 0, decay 1)
constexpr int DC_COLS = 8;                          // columns of S of a scanning block
constexpr int DC_RP = DC_K + 4;                     // floats from row to row of K P and Q P: 8 lanes on 8 rows hit 32 banks
constexpr int DC_TP = DC_C + 4;                     // ... of T and M
constexpr int DC_THREADS = 256;
// the workspace of a (chunk, head): K P [32][132], Q P [32][132] | T [32][36], M [32][36] | K D [32][128], P_32 [128]
constexpr int DC_WS_KQ = 2 * DC_C * DC_RP, DC_WS_TM = 2 * DC_C * DC_TP, DC_WS_KD = DC_C * DC_K + DC_K;
constexpr int DC_WS = DC_WS_KQ + DC_WS_TM + DC_WS_KD;
constexpr float DC_UNIT_EPS = 1e-6f;

struct DeltaChunkArgs {
    const float* qkv;       // [n, ldq]: q (kvh * dk), k (kvh * dk), v (heads * dv), after convolution and SiLU
    long long ldq;
    const float* beta;      // [n, ldb]: logits of beta, one per head
    long long ldb;
    const float* a;         // [n, lda]: decay logits before the bias, heads * decay_channels
    long long lda;
    const float* dt_bias;   // [heads * decay_channels]
    const float* a_log;     // [heads]
    float* state;           // per slot `state_stride` numbers; S is [heads, dk, dv] at the start
    long long state_stride;
    float* out;             // [n, heads * dv]: o before its norm
    const int* seq_first_row;
    const int* seq_start_pos;
    const int* seq_slots;
    float* ws;
    int heads, kv_heads, dk, dv, num_slots, write_state, decay_channels;
    int* status;
};

typedef unsigned long long dc_pair;                 // two floats in one 64-bit register
__device__ __forceinline__ dc_pair dc_pack(float lo, float hi) {
    dc_pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float dc_sum(dc_pair v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}
__device__ __forceinline__ void dc_fma(dc_pair& c, dc_pair a, dc_pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ dc_pair dc_mul(dc_pair a, dc_pair b) {
    dc_pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void dc_cp16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void dc_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void dc_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

// where a request's chunks lie in the workspace: requests own rows one after the other, so r0 / 32 + seq leaves room for
// each one's last, ragged chunk
__device__ __forceinline__ size_t dc_slot(int r0, int seq, int chunk, int heads, int head) {
    return ((size_t)(r0 / DC_C + seq + chunk) * heads + head) * DC_WS;
}

// Sums v[0..31] over the warp's lanes; lane l receives the sum of v[l].
__device__ __forceinline__ float dc_transpose_sum(float (&v)[32], int lane) {
#pragma unroll
    for (int half = 16; half >= 1; half >>= 1) {
        const bool upper = lane & half;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return v[0];
}

__global__ void __launch_bounds__(DC_THREADS, 2) delta_prepare_kernel(DeltaChunkArgs p) {
    extern __shared__ __align__(16) float dc_mem[];
    float* Q = dc_mem, *K = Q + DC_C * DC_RP, *G = K + DC_C * DC_RP;       // [32][132] each
    __shared__ __align__(16) float A[DC_C][DC_TP], B[DC_C][DC_TP], Tm[DC_C][DC_TP];
    __shared__ float beta_s[DC_C];
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int chunk = blockIdx.x, head = blockIdx.y, seq = blockIdx.z;
    if (p.seq_start_pos[seq] < 0) return;
    const int r0 = p.seq_first_row[seq], r1 = p.seq_first_row[seq + 1];
    const int c0 = r0 + chunk * DC_C, nt = min(DC_C, r1 - c0);
    if (nt <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dk = p.dk, kvh = head / (p.heads / p.kv_heads), dc = p.decay_channels;
    float* ws = p.ws + dc_slot(r0, seq, chunk, p.heads, head);
    const float rate = expf(p.a_log[head]);

    // rows of the chunk: a token past its end is k = q = 0, decay 1, beta 0 and changes nothing
    {
        const int c = tid & (DC_K - 1);
        const size_t ai = (size_t)head * dc + (dc > 1 ? c : 0);
        const float bias = c < dk ? p.dt_bias[ai] : 0.f;
        for (int t0 = tid >> 7; t0 < DC_C; t0 += 16) {                     // eight tokens' loads in flight
            float qv[8], kv[8], zv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + 2 * u;
                const size_t row = (size_t)(c0 + t);
                const bool in = t < nt && c < dk;
                qv[u] = in ? p.qkv[row * p.ldq + (size_t)kvh * dk + c] : 0.f;
                kv[u] = in ? p.qkv[row * p.ldq + (size_t)(p.kv_heads + kvh) * dk + c] : 0.f;
                zv[u] = in ? p.a[row * p.lda + ai] + bias : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + 2 * u;
                const float sp = zv[u] > 15.f ? zv[u] : __logf(1.0f + __expf(zv[u]));     // (as in the walk)
                Q[t * DC_RP + c] = qv[u];
                K[t * DC_RP + c] = kv[u];
                G[t * DC_RP + c] = t < nt && c < dk ? __expf(-rate * sp) : 1.f;
            }
        }
        if (tid < DC_C) beta_s[tid] = tid < nt ? 1.0f / (1.0f + __expf(-p.beta[(size_t)(c0 + tid) * p.ldb + head])) : 0.f;
    }
    __syncthreads();
    const float q_scale = 1.0f / sqrtf((float)dk);
#pragma unroll
    for (int u = 0; u < DC_C / 8; ++u) {                                   // unit vectors, a warp per token
        const int t = warp + 8 * u;
        float4* q4 = reinterpret_cast<float4*>(Q + t * DC_RP) + lane;
        float4* k4 = reinterpret_cast<float4*>(K + t * DC_RP) + lane;
        float4 q = *q4, k = *k4;
        const float sq = gb_warp_sum(fmaf(q.x, q.x, fmaf(q.y, q.y, fmaf(q.z, q.z, q.w * q.w))));
        const float sk = gb_warp_sum(fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, k.w * k.w))));
        const float iq = q_scale / sqrtf(sq + DC_UNIT_EPS), ik = 1.0f / sqrtf(sk + DC_UNIT_EPS);
        *q4 = make_float4(q.x * iq, q.y * iq, q.z * iq, q.w * iq);
        *k4 = make_float4(k.x * ik, k.y * ik, k.z * ik, k.w * ik);
    }
    __syncthreads();
    // products of decays: from the front for K P and Q P (half of the block), from the back for K D (the other half)
    if (tid < DC_K) {
        float d = 1.f;
#pragma unroll 8
        for (int t = 0; t < DC_C; ++t) {
            d *= G[t * DC_RP + tid];
            ws[t * DC_RP + tid] = K[t * DC_RP + tid] * d;
            ws[(DC_C + t) * DC_RP + tid] = Q[t * DC_RP + tid] * d;
        }
        ws[DC_WS_KQ + DC_WS_TM + DC_C * DC_K + tid] = d;
    } else {
        const int c = tid - DC_K;
        float d = 1.f;
#pragma unroll 8
        for (int t = DC_C - 1; t >= 0; --t) {
            ws[DC_WS_KQ + DC_WS_TM + t * DC_K + c] = K[t * DC_RP + c] * d;
            d *= G[t * DC_RP + c];
        }
    }
    // A and B: a warp takes four rows, a lane four channels; walking j downwards, the decays between the tokens grow factor
    // by factor. The sums over the lanes go 32 at a time (four j of four rows and two matrices).
    {
        const int i0 = warp * 4;
        dc_pair qi[4][2], ki[4][2], d[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Q + (i0 + r) * DC_RP + 4 * lane);
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(K + (i0 + r) * DC_RP + 4 * lane);
            qi[r][0] = q.x; qi[r][1] = q.y; ki[r][0] = k.x; ki[r][1] = k.y;
            d[r][0] = d[r][1] = dc_pack(1.f, 1.f);
        }
        for (int j0 = i0; j0 >= 0; j0 -= 4) {
            float sums[32];
#pragma unroll
            for (int jj = 3; jj >= 0; --jj) {
                const int j = j0 + jj;
                const ulonglong2 kj = *reinterpret_cast<const ulonglong2*>(K + j * DC_RP + 4 * lane);
                const ulonglong2 gj = *reinterpret_cast<const ulonglong2*>(G + j * DC_RP + 4 * lane);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    dc_pair a = 0ull, b = 0ull;
                    if (j <= i0 + r) {
                        const dc_pair x = dc_mul(d[r][0], kj.x), y = dc_mul(d[r][1], kj.y);
                        a = dc_mul(ki[r][0], x);
                        b = dc_mul(qi[r][0], x);
                        dc_fma(a, ki[r][1], y);
                        dc_fma(b, qi[r][1], y);
                        d[r][0] = dc_mul(d[r][0], gj.x);
                        d[r][1] = dc_mul(d[r][1], gj.y);
                    }
                    sums[jj * 8 + r * 2] = dc_sum(a);
                    sums[jj * 8 + r * 2 + 1] = dc_sum(b);
                }
            }
            const float total = dc_transpose_sum(sums, lane);
            const int j = j0 + (lane >> 3), i = i0 + ((lane >> 1) & 3);
            if (lane & 1) B[i][j] = total;
            else A[i][j] = total;
        }
    }
    __syncthreads();
    // T by forward substitution, a lane per column
    if (warp == 0) {
        float t[DC_C];
#pragma unroll
        for (int i = 0; i < DC_C; ++i) {
            const float bi = beta_s[i];
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < i; ++j) s[j & 3] = fmaf(A[i][j], t[j], s[j & 3]);
            t[i] = bi * ((lane == i ? 1.f : 0.f) - ((s[0] + s[1]) + (s[2] + s[3])));
            Tm[i][lane] = t[i];
            ws[DC_WS_KQ + i * DC_TP + lane] = t[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {                                          // M = B T, sums over j .. i
        const int i = warp + 8 * u, j = lane;
        float s = 0.f;
        for (int l = 0; l <= i; ++l)
            if (l >= j) s = fmaf(B[i][l], Tm[l][j], s);
        ws[DC_WS_KQ + (DC_C + i) * DC_TP + j] = s;
    }
}

// (two blocks share an SM where there are that many)
constexpr int DC_SCAN_SMEM = (2 * DC_WS_KQ + 2 * DC_WS_TM + DC_WS_KD + DC_COLS * DC_RP + 2 * DC_COLS * DC_TP) * 4;

__global__ void __launch_bounds__(DC_THREADS, 2) delta_scan_kernel(DeltaChunkArgs p) {
    extern __shared__ __align__(16) float dc_mem[];
    float* KQ = dc_mem;                                     // two of [64][132]: K P, then Q P
    float* TM = KQ + 2 * DC_WS_KQ;                          // two of [64][36]: T, then M
    float* KD = TM + 2 * DC_WS_TM;                          // [32][128], then P_32 [128]
    float* Ss = KD + DC_WS_KD;                              // S by columns: [8][132]
    float* Wt = Ss + DC_COLS * DC_RP;                       // W and U by columns: [8][36] each
    float* Ut = Wt + DC_COLS * DC_TP;
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z;
    if (p.seq_start_pos[seq] < 0) return;
    const int slot = p.seq_slots[seq];
    if (slot < 0 || slot >= p.num_slots) {
        if (threadIdx.x == 0) atomicOr(p.status, GB_STATUS_BAD_SLOT);
        return;
    }
    const int r0 = p.seq_first_row[seq], r1 = p.seq_first_row[seq + 1];
    const int chunks = (r1 - r0 + DC_C - 1) / DC_C;
    if (chunks <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dk = p.dk, dv = p.dv, col0 = blockIdx.x * DC_COLS;
    float* sbase = p.state + (size_t)slot * p.state_stride + (size_t)head * dk * dv;
    const float* ws0 = p.ws + dc_slot(r0, seq, 0, p.heads, head);
    const size_t ws_step = (size_t)p.heads * DC_WS;

    auto load_first = [&](int chunk) {                      // what the first two phases of a chunk read
        const float* src = ws0 + chunk * ws_step;
        float* kq = KQ + (chunk & 1) * DC_WS_KQ, *tm = TM + (chunk & 1) * DC_WS_TM;
        for (int i = tid; i < DC_WS_KQ / 4; i += DC_THREADS) dc_cp16(kq + 4 * i, src + 4 * i);
        for (int i = tid; i < DC_WS_TM / 4; i += DC_THREADS) dc_cp16(tm + 4 * i, src + DC_WS_KQ + 4 * i);
        dc_commit();
    };
    auto load_last = [&](int chunk) {                       // ... and its third
        const float* src = ws0 + chunk * ws_step + DC_WS_KQ + DC_WS_TM;
        for (int i = tid; i < DC_WS_KD / 4; i += DC_THREADS) dc_cp16(KD + 4 * i, src + 4 * i);
        dc_commit();
    };
    load_first(0);
    load_last(0);
    for (int i = tid; i < DC_K * DC_COLS; i += DC_THREADS) {
        const int d = i / DC_COLS, c = i % DC_COLS;
        Ss[c * DC_RP + d] = d < dk && col0 + c < dv ? sbase[(size_t)d * dv + col0 + c] : 0.f;
    }
    // a thread's token and column in the second phase; its value is asked for a chunk ahead
    const int ti = tid >> 3, tc = tid & 7;
    const bool col_in = col0 + tc < dv;
    const float* vcol = p.qkv + (size_t)2 * p.kv_heads * dk + (size_t)head * dv + col0 + tc;
    auto value_of = [&](int chunk) {
        const int row = r0 + chunk * DC_C + ti;
        return col_in && row < r1 ? vcol[(size_t)row * p.ldq] : 0.f;
    };
    float v_next = value_of(0);

    for (int chunk = 0; chunk < chunks; ++chunk) {
        const float* kq = KQ + (chunk & 1) * DC_WS_KQ, *tm = TM + (chunk & 1) * DC_WS_TM;
        // [8 warps][64 rows][8 columns], later the second half of the update: where the chunk's K P and Q P were
        float* red = KQ + (chunk & 1) * DC_WS_KQ;
        dc_wait<1>();                                       // this chunk's first half (its last part may still be under way)
        __syncthreads();                                    // ... for everyone; S is complete; the other buffers are free
        if (chunk + 1 < chunks) load_first(chunk + 1);
        else dc_commit();
        const float v = v_next;
        if (chunk + 1 < chunks) v_next = value_of(chunk + 1);

        // (K P) S and (Q P) S: a warp takes 16 channels, a lane rows `lane` and `lane + 32` against all columns
        {
            dc_pair acc[2][DC_COLS];
#pragma unroll
            for (int c = 0; c < DC_COLS; ++c) acc[0][c] = acc[1][c] = 0ull;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int d = warp * 16 + 4 * s;
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(kq + lane * DC_RP + d);
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(kq + (lane + 32) * DC_RP + d);
#pragma unroll
                for (int c = 0; c < DC_COLS; ++c) {
                    const ulonglong2 sv = *reinterpret_cast<const ulonglong2*>(Ss + c * DC_RP + d);
                    dc_fma(acc[0][c], x.x, sv.x);
                    dc_fma(acc[1][c], y.x, sv.x);
                    dc_fma(acc[0][c], x.y, sv.y);
                    dc_fma(acc[1][c], y.y, sv.y);
                }
            }
            __syncthreads();                                // everyone has read K P and Q P
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // (the two 16-byte halves of a row change places by row, so that eight lanes hit 32 banks)
                float* dst = red + (warp * 64 + lane + 32 * h) * DC_COLS;
                const float4 lo = make_float4(dc_sum(acc[h][0]), dc_sum(acc[h][1]), dc_sum(acc[h][2]), dc_sum(acc[h][3]));
                const float4 hi = make_float4(dc_sum(acc[h][4]), dc_sum(acc[h][5]), dc_sum(acc[h][6]), dc_sum(acc[h][7]));
                const int flip = (lane >> 2) & 1;
                reinterpret_cast<float4*>(dst)[flip] = lo;
                reinterpret_cast<float4*>(dst)[flip ^ 1] = hi;
            }
        }
        __syncthreads();
        float qs = 0.f;
        {
            const int at = tc ^ (((ti >> 2) & 1) << 2);
            float ks = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                ks += red[(w * 64 + ti) * DC_COLS + at];
                qs += red[(w * 64 + 32 + ti) * DC_COLS + at];
            }
            Wt[tc * DC_TP + ti] = v - ks;
        }
        __syncthreads();
        // U = T W and O = (Q P) S + M W; a token never meets a later one's numbers, not even times zero
        {
            float u = 0.f, o = qs;
            const float* trow = tm + ti * DC_TP, *mrow = tm + (DC_C + ti) * DC_TP, *wcol = Wt + tc * DC_TP;
            const int last = (ti | 3);                      // the largest token of this warp
            for (int j = 0; j <= last; j += 4) {
                const float4 t4 = *reinterpret_cast<const float4*>(trow + j);
                const float4 m4 = *reinterpret_cast<const float4*>(mrow + j);
                const float4 w4 = *reinterpret_cast<const float4*>(wcol + j);
                if (j <= ti) { u = fmaf(t4.x, w4.x, u); o = fmaf(m4.x, w4.x, o); }
                if (j + 1 <= ti) { u = fmaf(t4.y, w4.y, u); o = fmaf(m4.y, w4.y, o); }
                if (j + 2 <= ti) { u = fmaf(t4.z, w4.z, u); o = fmaf(m4.z, w4.z, o); }
                if (j + 3 <= ti) { u = fmaf(t4.w, w4.w, u); o = fmaf(m4.w, w4.w, o); }
            }
            Ut[tc * DC_TP + ti] = u;
            const int row = r0 + chunk * DC_C + ti;
            if (row < r1 && col_in) p.out[(size_t)row * p.heads * dv + (size_t)head * dv + col0 + tc] = o;
        }
        dc_wait<1>();                                       // K D (the next chunk's first half may still be under way)
        __syncthreads();
        // S <- P S + (K D)^T U: warps 0 to 3 take tokens 0 to 15, the others 16 to 31; a warp 64 channels of four columns
        {
            const int half = warp >> 2, cg = (warp >> 1) & 1, d = (warp & 1) * 64 + 2 * lane;
            dc_pair acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                float u4[4][4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    *reinterpret_cast<float4*>(u4[c]) = *reinterpret_cast<const float4*>(Ut + (cg * 4 + c) * DC_TP + half * 16 + j);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const dc_pair k = *reinterpret_cast<const dc_pair*>(KD + (half * 16 + j + e) * DC_K + d);
#pragma unroll
                    for (int c = 0; c < 4; ++c) dc_fma(acc[c], k, dc_pack(u4[c][e], u4[c][e]));
                }
            }
            dc_pair* other = reinterpret_cast<dc_pair*>(red);                  // [4 warps][4 columns][32 lanes]
            if (half) {
#pragma unroll
                for (int c = 0; c < 4; ++c) other[((warp & 3) * 4 + c) * 32 + lane] = acc[c];
            }
            __syncthreads();
            if (!half) {
                const dc_pair decay = *reinterpret_cast<const dc_pair*>(KD + DC_C * DC_K + d);
                const dc_pair one = dc_pack(1.f, 1.f);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    dc_pair* s = reinterpret_cast<dc_pair*>(Ss + (cg * 4 + c) * DC_RP + d);
                    dc_fma(acc[c], decay, *s);
                    dc_fma(acc[c], one, other[((warp & 3) * 4 + c) * 32 + lane]);
                    *s = acc[c];
                }
            }
        }
        __syncthreads();                                    // K D has been read: the next chunk's may come
        if (chunk + 1 < chunks) load_last(chunk + 1);
        else dc_commit();
    }
    if (p.write_state) {
        for (int i = tid; i < DC_K * DC_COLS; i += DC_THREADS) {
            const int d = i / DC_COLS, c = i % DC_COLS;
            if (d < dk && col0 + c < dv) sbase[(size_t)d * dv + col0 + c] = Ss[c * DC_RP + d];
        }
    }
}

GB_EXPORT int gb_delta_chunk_rows() { return DC_C; }
GB_EXPORT int gb_delta_chunk_floats() { return DC_WS; }            // workspace of a (chunk, head)

// As gb_channel_delta (delta_rule.cu) for key sizes up to 128, with a workspace of n / 32 + S chunks of heads *
// gb_delta_chunk_floats() numbers, 16-byte aligned. max_rows: the most rows that a request brings.
GB_EXPORT int gb_channel_delta_chunks(const float* qkv, long long ldq, const float* beta, long long ldb, const float* a, long long lda,
                                      const float* dt_bias, const float* a_log, float* state, long long state_stride, float* out,
                                      const int* seq_first_row, const int* seq_start_pos, const int* seq_slots, int S, int max_rows, int heads,
                                      int kv_heads, int dk, int dv, int num_slots, int write_state, int* status, int decay_channels,
                                      float* ws, cudaStream_t stream) {
    GB_REQUIRE(S >= 0 && S <= 65535 && heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0,
               "gb_channel_delta_chunks: heads %d must be a multiple of key heads %d", heads, kv_heads);
    GB_REQUIRE(decay_channels == 1 || decay_channels == dk, "gb_channel_delta_chunks: %d decays per head (one, or one per key channel)",
               decay_channels);
    GB_REQUIRE(dk > 0 && dk <= DC_K && dv > 0, "gb_channel_delta_chunks: a key size of %d is outside 1..%d", dk, DC_K);
    GB_REQUIRE((uintptr_t)ws % 16 == 0, "gb_channel_delta_chunks: the workspace must be 16-byte aligned");
    if (S == 0 || max_rows <= 0) return 0;
    DeltaChunkArgs p = {qkv, ldq, beta, ldb, a, lda, dt_bias, a_log, state, state_stride, out, seq_first_row, seq_start_pos, seq_slots,
                        ws, heads, kv_heads, dk, dv, num_slots, write_state, decay_channels, status};
    const int prepare_smem = 3 * DC_C * DC_RP * 4;
    cudaError_t e = cudaFuncSetAttribute(delta_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, prepare_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_SCAN_SMEM);
    GB_REQUIRE(e == cudaSuccess, "gb_channel_delta_chunks: %d bytes of shared memory refused: %s", DC_SCAN_SMEM, cudaGetErrorString(e));
    gb_launch(GB_PDL_ATTENTION, delta_prepare_kernel, dim3(gb_ceil_div(max_rows, DC_C), heads, S), dim3(DC_THREADS), prepare_smem, stream, p);
    int rc = gb_check_launch("gb_channel_delta_chunks (prepare)");
    if (rc) return rc;
    gb_launch(GB_PDL_ATTENTION, delta_scan_kernel, dim3(gb_ceil_div(dv, DC_COLS), heads, S), dim3(DC_THREADS), DC_SCAN_SMEM, stream, p);
    return gb_check_launch("gb_channel_delta_chunks");
}
