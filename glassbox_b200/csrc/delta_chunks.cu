// The gated delta rule over prompt portions, 32 tokens at a time (the walk token by token is in delta_rule.cu).
//
// With S_0 the state in front of a chunk, P_i the product of the chunk's decays up to and including token i (per key channel)
// and D_ij that of the decays after token j up to token i, the recurrence S <- diag(g) S; u = beta (v - S^T k); S <- S + k u^T;
// o = S^T q unrolls to
//     u_i + beta_i sum_{j<i} A_ij u_j = beta_i (v_i - (k_i P_i)^T S_0),      A_ij = sum_c k_i[c] D_ij[c] k_j[c]
//     o_i = (q_i P_i)^T S_0 + sum_{j<=i} B_ij u_j,                            B_ij = sum_c q_i[c] D_ij[c] k_j[c]
//     S_32 = diag(P_32) S_0 + sum_j (k_j D_(32)j) u_j^T
// (the WY form of a product of Householder-like factors; Bischof and Van Loan 1987, with decays as in gated linear
// attention). With T = (1 + diag(beta) A)^(-1) diag(beta) (A strictly lower triangular: forward substitution) a chunk is
// U = T V - (T K P) S_0, O = (Q P) S_0 + B U, S_32 = P_32 S_0 + (K D)^T U: products, and nothing but S passes from chunk to
// chunk. Decays only ever appear as products of themselves, never as quotients, so nothing overflows however fast a channel
// forgets.
//
//   delta_prepare_kernel  every (chunk, head) side by side: unit vectors, decays, A, B, T K P and T V into a workspace
//   delta_scan_kernel     a block per (request, head, 8 or 16 columns of S): U and S chunk after chunk, S in registers
//   delta_out_kernel      every (chunk, head) side by side: O from the chunk's S_0 and U
//
// Each lets the next start only when it is about to end. A scanning block takes a multiprocessor's whole register file: when all three let
// their successors in at once, blocks of the calls to come held most multiprocessors waiting, and the few blocks of a short prompt's
// preparation and read-out ran two to a multiprocessor beside them (one request of 96 rows, 8 heads: 37.8 us; 28.6 so).
// Everything is float32. The products run on the tensor cores with every float32 operand as three bfloat16 numbers whose sum it is
// exactly, each what is left rounded to the nearest (Henry, Tang and Heinecke 2019), and six products of them, the largest in an
// accumulator of its own: what is left out is below 2^-24 of a product and has either sign. Measured against 64 bits, random inputs
// (2-norm of the error over that of the result, read-out / state), 160 and 700 tokens of one request: 1.3e-7 / 1.2e-7 and 1.4e-7 /
// 1.2e-7; by the walk 2.4e-7 / 2.0e-7 and 2.6e-7 / 2.3e-7; nothing written and a state of one number a head 7.0e-7 / 1.2e-6 and 2.8e-6 /
// 4.8e-6, by the walk 1.1e-6 / 1.8e-6 and 4.2e-6 / 7.2e-6 (the decays' product).
// What bounds the scan: a chain of 1,350 cycles a chunk (two products, two barriers and a sum over the warps) and a chunk's two operands
// for a block, 48 KB from L2 (with all operands in L1 45 us of the 68). A warp owns 16 channels of S: S never leaves its registers
// (movmatrix turns the accumulators into the next product's operand); the sums over the channels meet in shared memory. Operands come
// in the order of the fragments, two chunks ahead, straight into registers. 16 columns a block where 8 would make more blocks than
// multiprocessors: the operands' way counts once for both.
// Measured, 2,048 tokens of one request, prepare + scan + read-out: 8 heads x 128 x 128 45 + 70 + 21 us (the chunk's products by FMA from
// shared memory, read-out in the scan: 37 + 126), 16 heads 81 + 107 + 41 (78 + 200); 96 tokens, 8 heads, 16.5 + 5.0 + 7.1 (15.8 + 9.4).
#include "common.cuh"

constexpr int DC_C = 32;                            // tokens of a chunk
constexpr int DC_K = 128;                           // key channels (smaller key sizes are padded: k = q = 0, decay 1)
constexpr int DC_V = 128;                           // columns of S that one pass takes
constexpr int DC_RP = DC_K + 8;                     // floats from row to row in shared memory: a fragment's 8-byte loads hit 32 banks
constexpr int DC_TP = DC_C + 4;                     // ... of A and B
constexpr int DC_THREADS = 256;
// The workspace of a (chunk, head), in 32-bit words (162 KB; with the operands as float32 and no S_0 it was 60). Fragments of mma.m16n8k16, [tile][3 terms][32 lanes][4 words]:
//   T K P   [8 groups of 16 channels][2 groups of 16 tokens]       rows tokens, k channels
//   K D     [8 groups of 16 channels][2 halves of each 8 tokens]   rows channels, k tokens (lane t of four: 8 t + 4 half ..)
//   Q P     as T K P
//   B       [2 groups of 16 tokens][2 groups of 16 tokens]         zero above the diagonal
// float32: P_32 [128], T V and later U [32 tokens][128 columns], S_0 [16 groups of 8 columns][8 groups of 16 channels][32 lanes][4]
constexpr int DC_FRAG = 3 * 32 * 4;
constexpr int DC_AT_KT = 0, DC_AT_KD = DC_AT_KT + 16 * DC_FRAG, DC_AT_QP = DC_AT_KD + 16 * DC_FRAG, DC_AT_B = DC_AT_QP + 16 * DC_FRAG;
constexpr int DC_AT_P = DC_AT_B + 4 * DC_FRAG, DC_AT_U = DC_AT_P + DC_K, DC_AT_S = DC_AT_U + DC_C * DC_V;
constexpr int DC_WS = DC_AT_S + DC_K * DC_V;
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
    int heads, kv_heads, dk, dv, num_slots, write_state, decay_channels, num_seqs;
    int col0, cols;         // the columns of S of this pass: at most DC_V
    int window, room;       // the chunks of this pass, by their places: `room` of them from `window` on
    const float* from;      // S of the request that began in the pass before, [heads][128][128]
    float* to;              // ... of the one that goes on in the next
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
__device__ __forceinline__ uint32_t dc_turn(uint32_t v) {       // an 8 x 8 matrix of 16-bit numbers, a row per four lanes, transposed
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ void dc_mma(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// The largest of an operand pair's products: 8 and 8 of the 16 channels or tokens apart, their sums added as float32 adds. The tensor
// core cuts what lies below its window: over 16 numbers near one an error of 2.5e-8 of the result, so 2.3e-8, in a chain of FMA 2.2e-8.
__device__ __forceinline__ void dc_mma_add(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    float d[4], f[4];
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a.x), "r"(a.y), "r"(b0), "f"(0.f));
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(a.z), "r"(a.w), "r"(b1), "f"(0.f));
#pragma unroll
    for (int e = 0; e < 4; ++e) c[e] += d[e] + f[e];
}
// The six products of two operands of three terms, the smallest first: (a's term, b's term); the last has its own accumulator.
constexpr int DC_PRODUCTS = 6;
__device__ constexpr int DC_A_TERM[DC_PRODUCTS] = {2, 0, 1, 1, 0, 0}, DC_B_TERM[DC_PRODUCTS] = {0, 2, 1, 0, 1, 0};

// A chunk's place: requests own rows one after the other, so r0 / 32 + seq leaves room for each one's last, ragged chunk. The workspace
// holds the places of a pass.
__device__ __forceinline__ size_t dc_slot(const DeltaChunkArgs& p, int r0, int seq, int chunk, int head) {
    return ((size_t)(r0 / DC_C + seq + chunk - p.window) * p.heads + head) * DC_WS;
}
// What a block of prepare or read-out works on. SEARCH: x is a place of the pass, y the head, and a warp looks the request up, the last whose
// first place is no higher; else x is the chunk and z the request.
struct DcPlace {
    int seq, chunk, start, slot, r0, r1;
};
template <bool SEARCH> __device__ __forceinline__ DcPlace dc_place(const DeltaChunkArgs& p) {
    DcPlace at = {(int)blockIdx.z, (int)blockIdx.x, -1, -1, 0, 0};
    if (!SEARCH) {
        at.start = p.seq_start_pos[at.seq]; at.slot = p.seq_slots[at.seq];                                  // (requested together)
        at.r0 = p.seq_first_row[at.seq]; at.r1 = p.seq_first_row[at.seq + 1];
        return at;
    }
    const int lane = threadIdx.x & 31, place = p.window + (int)blockIdx.x;
    for (int s0 = 0; s0 < p.num_seqs; s0 += 32) {
        const int s = min(s0 + lane, p.num_seqs - 1), r0 = p.seq_first_row[s], r1 = p.seq_first_row[s + 1], start = p.seq_start_pos[s], slot = p.seq_slots[s];
        const unsigned up_to = __ballot_sync(0xffffffffu, s0 + lane < p.num_seqs && r0 / DC_C + s <= place);
        if (up_to == 0) break;
        const int l = 31 - __clz(up_to);
        at.seq = s0 + l;
        at.start = __shfl_sync(0xffffffffu, start, l); at.slot = __shfl_sync(0xffffffffu, slot, l);
        at.r0 = __shfl_sync(0xffffffffu, r0, l); at.r1 = __shfl_sync(0xffffffffu, r1, l);
        if (up_to != 0xffffffffu) break;
    }
    at.chunk = place - (at.r0 / DC_C + at.seq);
    return at;
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

template <bool SEARCH>
__global__ void __launch_bounds__(DC_THREADS, 2) delta_prepare_kernel(DeltaChunkArgs p) {
    extern __shared__ __align__(16) float dc_mem[];
    float* Q = dc_mem, *K = Q + DC_C * DC_RP, *G = K + DC_C * DC_RP;       // [32][136] each
    __shared__ __align__(16) float A[DC_C][DC_TP], B[DC_C][DC_TP];
    __shared__ float beta_s[DC_C];
    gb_pdl_wait();
    const DcPlace at = dc_place<SEARCH>(p);
    const int head = blockIdx.y, c0 = at.r0 + at.chunk * DC_C, nt = min(DC_C, at.r1 - c0);
    if (at.start < 0 || nt <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dk = p.dk, kvh = head / (p.heads / p.kv_heads), dc = p.decay_channels;
    float* ws = p.ws + dc_slot(p, at.r0, at.seq, at.chunk, head);
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
                const float sp = zv[u] > 15.f ? zv[u] : log1pf(expf(zv[u]));
                Q[t * DC_RP + c] = qv[u];
                K[t * DC_RP + c] = kv[u];
                G[t * DC_RP + c] = t < nt && c < dk ? expf(-rate * sp) : 1.f;
            }
        }
        if (tid < DC_C) beta_s[tid] = tid < nt ? 1.0f / (1.0f + expf(-p.beta[(size_t)(c0 + tid) * p.ldb + head])) : 0.f;
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
    // A and B: a warp takes four rows, a lane four channels; walking j downwards, the decays between the tokens grow factor
    // by factor. The sums over the lanes go 32 at a time (four j of four rows and two matrices).
    {
        const int i0 = (warp < 4 ? warp : 11 - warp) * 4;  // (a scheduler's two warps have nine groups of four rows between them)
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
    // A thread per column of [K P | V]: forward substitution gives T K P and T V without T (row i needs rows in front of it alone, so
    // a token never meets a later one's numbers, not even times zero). Half of the block also leaves Q P and K D where Q and K were.
    {
        float x[DC_C];
        const int c = tid & (DC_K - 1);
        const bool keys = tid < DC_K;
        if (keys) {
            float d = 1.f;
#pragma unroll
            for (int t = 0; t < DC_C; ++t) {
                d *= G[t * DC_RP + c];
                x[t] = K[t * DC_RP + c] * d;
                Q[t * DC_RP + c] *= d;
            }
            ws[DC_AT_P + c] = d;
            d = 1.f;
#pragma unroll
            for (int t = DC_C - 1; t >= 0; --t) {
                K[t * DC_RP + c] *= d;
                d *= G[t * DC_RP + c];
            }
        } else {
            const float* v = p.qkv + (size_t)2 * p.kv_heads * dk + (size_t)head * p.dv + p.col0 + c;
#pragma unroll
            for (int t = 0; t < DC_C; ++t) x[t] = t < nt && c < p.cols ? v[(size_t)(c0 + t) * p.ldq] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < DC_C; ++i) {
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < i; j += 4) {
                const float4 a = *reinterpret_cast<const float4*>(&A[i][j]);
                s[0] = fmaf(a.x, x[j], s[0]);
                if (j + 1 < i) s[1] = fmaf(a.y, x[j + 1], s[1]);
                if (j + 2 < i) s[2] = fmaf(a.z, x[j + 2], s[2]);
                if (j + 3 < i) s[3] = fmaf(a.w, x[j + 3], s[3]);
            }
            x[i] = beta_s[i] * (x[i] - ((s[0] + s[1]) + (s[2] + s[3])));
        }
#pragma unroll
        for (int t = 0; t < DC_C; ++t) {
            if (keys) G[t * DC_RP + c] = x[t];
            else ws[DC_AT_U + t * DC_V + c] = x[t];
        }
    }
    __syncthreads();
    gb_pdl_launch_dependents();
    // the operands in the order of the fragments
    const int g = lane >> 2, t4 = lane & 3;
    for (int it = warp; it < 52; it += DC_THREADS / 32) {
        float2 v[4];
        int at;
        if (it < 32) {                                                     // T K P, then Q P
            const int tile = it & 15;
            const float* src = (it < 16 ? G : Q) + ((tile & 1) * 16 + g) * DC_RP + (tile >> 1) * 16 + 2 * t4;
            at = (it < 16 ? DC_AT_KT : DC_AT_QP) + tile * DC_FRAG;
            v[0] = *reinterpret_cast<const float2*>(src);
            v[1] = *reinterpret_cast<const float2*>(src + 8 * DC_RP);
            v[2] = *reinterpret_cast<const float2*>(src + 8);
            v[3] = *reinterpret_cast<const float2*>(src + 8 * DC_RP + 8);
        } else if (it < 48) {                                              // K D
            const int tile = it - 32;
            const float* src = K + (8 * t4 + 4 * (tile & 1)) * DC_RP + (tile >> 1) * 16 + g;
            at = DC_AT_KD + tile * DC_FRAG;
            v[0] = make_float2(src[0], src[DC_RP]);
            v[1] = make_float2(src[8], src[DC_RP + 8]);
            v[2] = make_float2(src[2 * DC_RP], src[3 * DC_RP]);
            v[3] = make_float2(src[2 * DC_RP + 8], src[3 * DC_RP + 8]);
        } else {                                                           // B (above its diagonal nothing was written)
            const int tile = it - 48, i = (tile >> 1) * 16 + g, j = (tile & 1) * 16 + 2 * t4;
            at = DC_AT_B + tile * DC_FRAG;
            auto b = [&](int r, int c) { return make_float2(c <= r ? B[r][c] : 0.f, c + 1 <= r ? B[r][c + 1] : 0.f); };
            v[0] = b(i, j); v[1] = b(i + 8, j); v[2] = b(i, j + 8); v[3] = b(i + 8, j + 8);
        }
        uint32_t w[4][3];
#pragma unroll
        for (int r = 0; r < 4; ++r) gb_split_bf16(v[r].x, v[r].y, w[r]);
#pragma unroll
        for (int e = 0; e < 3; ++e)
            *reinterpret_cast<uint4*>(ws + at + e * 128 + lane * 4) = make_uint4(w[0][e], w[1][e], w[2][e], w[3][e]);
    }
}

// S of a warp's 16 channels and 8 columns as the right operand of a product over the channels
__device__ __forceinline__ void dc_right(const float (&s)[4], uint32_t (&b)[3][2]) {
    uint32_t lo[3], hi[3];
    gb_split_bf16<true>(s[0], s[1], lo);
    gb_split_bf16<true>(s[2], s[3], hi);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        b[e][0] = dc_turn(lo[e]);
        b[e][1] = dc_turn(hi[e]);
    }
}

template <int NT> struct DeltaOperands {                     // what a chunk brings to a thread
    uint4 kt[2][3], kd[2][3];
    float decay[2], tv[NT];
};

template <int NT>
__global__ void __launch_bounds__(DC_THREADS, 1) delta_scan_kernel(DeltaChunkArgs p) {
    __shared__ __align__(16) float red[NT][8][DC_C][8];      // T K P S by warp (16 channels each): [column group][warp][token][column]
    __shared__ __align__(16) unsigned short Ub[NT][3][8][DC_C];     // U's terms by column
    gb_pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z;
    const int start = p.seq_start_pos[seq], slot = p.seq_slots[seq], r0 = p.seq_first_row[seq], r1 = p.seq_first_row[seq + 1];
    if (start < 0) return;
    if (slot < 0 || slot >= p.num_slots) {
        if (threadIdx.x == 0) atomicOr(p.status, GB_STATUS_BAD_SLOT);
        return;
    }
    // its chunks in this pass
    const int place = r0 / DC_C + seq, all = (r1 - r0 + DC_C - 1) / DC_C;
    const int chunk0 = max(p.window - place, 0), chunks = min(all, p.window + p.room - place) - chunk0;
    if (chunks <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int dk = p.dk, dv = p.dv, col0 = blockIdx.x * 8 * NT;              // (of this pass)
    float* sbase = p.state + (size_t)slot * p.state_stride + (size_t)head * dk * dv + p.col0;
    float* ws0 = p.ws + dc_slot(p, r0, seq, chunk0, head);
    const size_t ws_step = (size_t)p.heads * DC_WS;
    const int ti = tid >> 3, tc = tid & 7;                   // a thread's token and column between the two products
    const int ch = warp * 16 + g;

    float S[NT][4];                                          // channels ch and ch + 8, columns 2 t4 and 2 t4 + 1 of each group
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = ch + 8 * (e >> 1), c = col0 + 8 * n + 2 * t4 + (e & 1);
            S[n][e] = d < dk && c < p.cols ? (chunk0 ? p.from[((size_t)head * DC_K + d) * DC_V + c] : sbase[(size_t)d * dv + c]) : 0.f;
        }
    auto load = [&](int chunk, DeltaOperands<NT>& o) {
        const float* ws = ws0 + chunk * ws_step;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                o.kt[m][e] = *reinterpret_cast<const uint4*>(ws + DC_AT_KT + (warp * 2 + m) * DC_FRAG + e * 128 + lane * 4);
                o.kd[m][e] = *reinterpret_cast<const uint4*>(ws + DC_AT_KD + (warp * 2 + m) * DC_FRAG + e * 128 + lane * 4);
            }
        o.decay[0] = ws[DC_AT_P + ch];
        o.decay[1] = ws[DC_AT_P + ch + 8];
#pragma unroll
        for (int n = 0; n < NT; ++n) o.tv[n] = ws[DC_AT_U + ti * DC_V + col0 + 8 * n + tc];
    };
    auto step = [&](int chunk, const DeltaOperands<NT>& o) {
        float* ws = ws0 + chunk * ws_step;
#pragma unroll
        for (int n = 0; n < NT; ++n)
            *reinterpret_cast<float4*>(ws + DC_AT_S + ((blockIdx.x * NT + n) * 8 + warp) * 128 + lane * 4) = make_float4(S[n][0], S[n][1], S[n][2], S[n][3]);
        {
            uint32_t b[NT][3][2];
            float hi[2][NT][4] = {}, lo[2][NT][2][4] = {};
#pragma unroll
            for (int n = 0; n < NT; ++n) dc_right(S[n], b[n]);
#pragma unroll
            for (int k = 0; k < DC_PRODUCTS; ++k)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if (k < DC_PRODUCTS - 1) dc_mma(lo[m][n][k & 1], o.kt[m][DC_A_TERM[k]], b[n][DC_B_TERM[k]][0], b[n][DC_B_TERM[k]][1]);
                        else dc_mma_add(hi[m][n], o.kt[m][DC_A_TERM[k]], b[n][DC_B_TERM[k]][0], b[n][DC_B_TERM[k]][1]);
                    }
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = hi[m][n][e] + (lo[m][n][0][e] + lo[m][n][1][e]);
                    *reinterpret_cast<float2*>(&red[n][warp][m * 16 + g][2 * t4]) = make_float2(v[0], v[1]);
                    *reinterpret_cast<float2*>(&red[n][warp][m * 16 + g + 8][2 * t4]) = make_float2(v[2], v[3]);
                }
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float r[8];
#pragma unroll
            for (int w = 0; w < 8; ++w) r[w] = red[n][w][ti][tc];
            const float u = o.tv[n] - (((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7])));
            ws[DC_AT_U + ti * DC_V + col0 + 8 * n + tc] = u;
            uint32_t term[3];
            gb_split_bf16<true>(u, 0.f, term);
#pragma unroll
            for (int e = 0; e < 3; ++e) Ub[n][e][tc][ti] = (unsigned short)term[e];
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            uint4 u[3];
            float hi[2][4] = {}, lo[2][2][4] = {};
#pragma unroll
            for (int e = 0; e < 3; ++e) u[e] = *reinterpret_cast<const uint4*>(&Ub[n][e][g][8 * t4]);
#pragma unroll
            for (int k = 0; k < DC_PRODUCTS; ++k)
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const uint4& r = u[DC_B_TERM[k]];
                    if (k < DC_PRODUCTS - 1) dc_mma(lo[s][k & 1], o.kd[s][DC_A_TERM[k]], s ? r.z : r.x, s ? r.w : r.y);
                    else dc_mma_add(hi[s], o.kd[s][DC_A_TERM[k]], s ? r.z : r.x, s ? r.w : r.y);
                }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                S[n][e] = fmaf(o.decay[e >> 1], S[n][e], (hi[0][e] + hi[1][e]) + ((lo[0][0][e] + lo[0][1][e]) + (lo[1][0][e] + lo[1][1][e])));
        }
    };
    DeltaOperands<NT> o[3];
    load(0, o[0]);
    if (chunks > 1) load(1, o[1]);
    for (int chunk = 0; chunk < chunks; chunk += 3) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (chunk + i >= chunks) break;
            if (chunk + i + 2 < chunks) load(chunk + i + 2, o[(i + 2) % 3]);
            step(chunk + i, o[i]);
        }
    }
    gb_pdl_launch_dependents();
    const bool goes_on = chunk0 + chunks < all;
    if (goes_on || p.write_state) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = ch + 8 * (e >> 1), c = col0 + 8 * n + 2 * t4 + (e & 1);
                if (d < dk && c < p.cols) *(goes_on ? p.to + ((size_t)head * DC_K + d) * DC_V + c : sbase + (size_t)d * dv + c) = S[n][e];
            }
    }
}

// O = (Q P) S_0 + B U: a warp takes two groups of 8 columns.
template <bool SEARCH>
__global__ void __launch_bounds__(DC_THREADS, 2) delta_out_kernel(DeltaChunkArgs p) {
    __shared__ uint4 left[20 * DC_FRAG / 4];                 // the left operands: Q P, then B
    gb_pdl_wait();
    gb_pdl_launch_dependents();
    const DcPlace at = dc_place<SEARCH>(p);
    const int head = blockIdx.y, c0 = at.r0 + at.chunk * DC_C, r1 = at.r1;
    if (at.start < 0 || at.slot < 0 || at.slot >= p.num_slots || c0 >= r1) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const float* ws = p.ws + dc_slot(p, at.r0, at.seq, at.chunk, head);
    for (int i = threadIdx.x; i < 20 * DC_FRAG / 4; i += DC_THREADS) dc_cp16(left + i, ws + DC_AT_QP + 4 * i);      // Q P and B
    asm volatile("cp.async.commit_group;");
    // (a group of columns past this pass's last has a slot, which nothing wrote: its sums are not stored)
    auto state = [&](int k16, float4 (&s)[2]) {
#pragma unroll
        for (int n = 0; n < 2; ++n) s[n] = *reinterpret_cast<const float4*>(ws + DC_AT_S + ((warp * 2 + n) * 8 + k16) * 128 + lane * 4);
    };
    float4 next[2][2];                                       // S_0, two groups of channels ahead
    state(0, next[0]);
    state(1, next[1]);
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();
    if (warp * 16 >= p.cols) return;
    float hi[2][2][4] = {}, lo[2][2][4] = {};                // [16 tokens][8 columns]
#pragma unroll
    for (int k16 = 0; k16 < DC_K / 16; ++k16) {
        uint4 a[2][3];
        uint32_t b[2][3][2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float4 s4 = next[k16 & 1][n];
            const float s[4] = {s4.x, s4.y, s4.z, s4.w};
            dc_right(s, b[n]);
        }
        if (k16 + 2 < DC_K / 16) state(k16 + 2, next[k16 & 1]);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int e = 0; e < 3; ++e) a[m][e] = left[((k16 * 2 + m) * DC_FRAG + e * 128) / 4 + lane];
#pragma unroll
        for (int k = 0; k < DC_PRODUCTS; ++k)
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    if (k < DC_PRODUCTS - 1) dc_mma(lo[m][n], a[m][DC_A_TERM[k]], b[n][DC_B_TERM[k]][0], b[n][DC_B_TERM[k]][1]);
                    else dc_mma_add(hi[m][n], a[m][DC_A_TERM[k]], b[n][DC_B_TERM[k]][0], b[n][DC_B_TERM[k]][1]);
                }
    }
    // U's rows as the right operand. A token must not meet a later one's numbers, not even times zero: what is not finite is left out
    // here and added below for the tokens that see it.
    const float* U = ws + DC_AT_U + warp * 16 + g;
    float u[2][2][4];
    bool odd = false;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int k16 = 0; k16 < 2; ++k16)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float v = U[(k16 * 16 + 2 * t4 + (e & 1) + 8 * (e >> 1)) * DC_V + 8 * n];
                const bool finite = fabsf(v) <= FLT_MAX;
                odd |= !finite;
                u[n][k16][e] = finite ? v : 0.f;
            }
    const bool plain = __any_sync(0xffffffffu, odd);
#pragma unroll
    for (int k16 = 0; k16 < 2; ++k16) {
        uint32_t b[2][2][3];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            gb_split_bf16<true>(u[n][k16][0], u[n][k16][1], b[n][0]);
            gb_split_bf16<true>(u[n][k16][2], u[n][k16][3], b[n][1]);
        }
#pragma unroll
        for (int m = k16; m < 2; ++m) {
            uint4 a[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) a[e] = left[((16 + m * 2 + k16) * DC_FRAG + e * 128) / 4 + lane];
#pragma unroll
            for (int k = 0; k < DC_PRODUCTS; ++k)
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    if (k < DC_PRODUCTS - 1) dc_mma(lo[m][n], a[DC_A_TERM[k]], b[n][0][DC_B_TERM[k]], b[n][1][DC_B_TERM[k]]);
                    else dc_mma_add(hi[m][n], a[DC_A_TERM[k]], b[n][0][DC_B_TERM[k]], b[n][1][DC_B_TERM[k]]);
                }
        }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = m * 16 + g + 8 * (e >> 1), c = (warp * 2 + n) * 8 + 2 * t4 + (e & 1);
                float o = hi[m][n][e] + lo[m][n][e];
                if (plain) {
                    const unsigned short* words = reinterpret_cast<const unsigned short*>(ws + DC_AT_B);
                    for (int j = 0; j <= i; ++j) {
                        const float v = ws[DC_AT_U + j * DC_V + c];
                        if (fabsf(v) <= FLT_MAX) continue;
                        const int lane_of = (i & 7) * 4 + ((j & 7) >> 1), word = ((i >> 3) & 1) + 2 * ((j >> 3) & 1);
                        const int at = (((i >> 4) * 2 + (j >> 4)) * DC_FRAG + lane_of * 4 + word) * 2 + (j & 1);
                        float bij = 0.f;
                        for (int e3 = 2; e3 >= 0; --e3) bij += __uint_as_float((uint32_t)words[at + e3 * 256] << 16);
                        o = fmaf(bij, v, o);
                    }
                }
                if (c0 + i < r1 && c < p.cols) p.out[(size_t)(c0 + i) * p.heads * p.dv + (size_t)head * p.dv + p.col0 + c] = o;
            }
}

GB_EXPORT int gb_delta_chunk_rows() { return DC_C; }
GB_EXPORT int gb_delta_chunk_floats() { return DC_WS; }                 // workspace of a (chunk, head)
GB_EXPORT int gb_delta_carry_floats() { return 2 * DC_K * DC_V; }       // ... of a head beside the chunks', where a call takes several passes

// As gb_channel_delta (delta_rule.cu) for key sizes up to 128 (value columns in passes of 128), with a workspace of `room` chunks of heads *
// gb_delta_chunk_floats() numbers, 16-byte aligned. A call of n rows in S requests has n / 32 + S places for chunks; where room is less,
// it takes them in passes, one behind the other, and heads * gb_delta_carry_floats() numbers lie behind the chunks.
// max_rows: the most rows that a request brings.
GB_EXPORT int gb_channel_delta_chunks(const float* qkv, long long ldq, const float* beta, long long ldb, const float* a, long long lda,
                                      const float* dt_bias, const float* a_log, float* state, long long state_stride, float* out,
                                      const int* seq_first_row, const int* seq_start_pos, const int* seq_slots, int n, int S, int max_rows, int heads,
                                      int kv_heads, int dk, int dv, int num_slots, int write_state, int* status, int decay_channels,
                                      float* ws, int room, cudaStream_t stream) {
    GB_REQUIRE(n >= 0 && S >= 0 && S <= 65535 && heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0,
               "gb_channel_delta_chunks: heads %d must be a multiple of key heads %d", heads, kv_heads);
    GB_REQUIRE(decay_channels == 1 || decay_channels == dk, "gb_channel_delta_chunks: %d decays per head (one, or one per key channel)",
               decay_channels);
    GB_REQUIRE(dk > 0 && dk <= DC_K && dv > 0, "gb_channel_delta_chunks: a key size of %d is outside 1..%d", dk, DC_K);
    GB_REQUIRE((uintptr_t)ws % 16 == 0 && room > 0, "gb_channel_delta_chunks: the workspace must be 16-byte aligned and hold a chunk");
    if (S == 0 || max_rows <= 0) return 0;
    DeltaChunkArgs p = {qkv, ldq, beta, ldb, a, lda, dt_bias, a_log, state, state_stride, out, seq_first_row, seq_start_pos, seq_slots,
                        ws, heads, kv_heads, dk, dv, num_slots, write_state, decay_channels, S, 0, 0, 0, room, nullptr, nullptr, status};
    const int places = n / DC_C + S, chunks = gb_ceil_div(max_rows, DC_C);
    float* carry = ws + (size_t)room * heads * DC_WS;
    // A recorded step gives its shape's longest possible portion, with which a grid of requests by chunks is mostly empty: beyond twice the
    // places the request is looked up (8 heads, 32 prompts of 16 tokens as one step 90 us with that grid, 74 so; 64 of 64 394 and 254).
    const bool search = places > room || (long long)S * chunks > 2LL * places;
    auto prepare = search ? delta_prepare_kernel<true> : delta_prepare_kernel<false>;
    auto read_out = search ? delta_out_kernel<true> : delta_out_kernel<false>;
    const int prepare_smem = 3 * DC_C * DC_RP * 4;
    cudaError_t e = cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, prepare_smem);
    GB_REQUIRE(e == cudaSuccess, "gb_channel_delta_chunks: %d bytes of shared memory refused: %s", prepare_smem, cudaGetErrorString(e));
    for (p.col0 = 0; p.col0 < dv; p.col0 += DC_V) {
        p.cols = dv - p.col0 < DC_V ? dv - p.col0 : DC_V;
        int pass = 0;
        for (p.window = 0; p.window < places; p.window += room, ++pass) {
            const int here = places - p.window < room ? places - p.window : room;
            const dim3 every = search ? dim3(here, heads) : dim3(chunks, heads, S);
            p.from = carry + (size_t)((pass + 1) & 1) * heads * DC_K * DC_V;
            p.to = carry + (size_t)(pass & 1) * heads * DC_K * DC_V;
            gb_launch(GB_PDL_ATTENTION, prepare, every, dim3(DC_THREADS), prepare_smem, stream, p);
            int rc = gb_check_launch("gb_channel_delta_chunks (prepare)");
            if (rc) return rc;
            const long long narrow = (long long)gb_ceil_div(p.cols, 8) * heads * S;
            if (narrow <= 148)
                gb_launch(GB_PDL_ATTENTION, delta_scan_kernel<1>, dim3(gb_ceil_div(p.cols, 8), heads, S), dim3(DC_THREADS), 0, stream, p);
            else
                gb_launch(GB_PDL_ATTENTION, delta_scan_kernel<2>, dim3(gb_ceil_div(p.cols, 16), heads, S), dim3(DC_THREADS), 0, stream, p);
            rc = gb_check_launch("gb_channel_delta_chunks (scan)");
            if (rc) return rc;
            gb_launch(GB_PDL_ATTENTION, read_out, every, dim3(DC_THREADS), 0, stream, p);
            rc = gb_check_launch("gb_channel_delta_chunks (read-out)");
            if (rc) return rc;
        }
    }
    return 0;
}
