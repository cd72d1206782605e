// Single decoded tokens of the talking-heads attention (talking_attention.cu) on the tensor cores (mma.sync m16n8k16), bfloat16
// queries and cache. One block = one row x 16 query heads x one share of the row's keys, all key/value heads' values.
//
// The keys pass in steps of KT. Per step: (1) every warp forms the scores of KT/8 keys, its keys straight from memory as right
// operands (a lane reads 16-byte pieces of a key; the order of the channels within a product is the same for the queries), each
// key/value head against the 16 rows of a head tile, of which the rows of its group are kept; (2) the scores meet in shared memory,
// a warp takes whole heads: running maximum, weights, denominator, and the weights' three bfloat16 terms, whose sum a weight is
// exactly; (3) O += (terms) V: a warp has an eighth of the wide value row's channels for all heads, and brings these itself
// (cp.async, 64 KB a block under way), so that values need no barrier. The sums of 32 keys start at zero and are added to the
// running ones in float32. A sum that is no finite number is formed again by FMA (an infinite value times the terms of a weight, of
// which some are zero or negative, would be NaN).
//
// What bounds it: per step of 128 keys some 2 us of latency (keys, two barriers, 32 dependent products) and the products themselves, 11
// cycles each on a scheduler: 3 terms x 16 heads x 256 channels. With two blocks an SM, 32 rows of 16 heads, 4 value heads of 64, contexts
// of 1,024 to 2,047 (51 MB): 16 us (3.1 TB/s). By FMA, four heads a block, so that four groups of heads each read every value again,
// and a key a lane (talking_attention_decode_kernel) it takes 48. Smaller ones, there / here: 1 row, 100 keys 8.5 / 6.7; 8 rows, 1,200 keys
// 13.3 / 9; 128 rows, 1,000 keys 89 / 35; 32 heads: 4 rows, 600 keys 13.3 / 9.5; 32 rows, 2,047 keys 164 / 64. Error against 64 bits 1.4e-7
// where FMA has 2.0e-7 to 3.3e-7 (sums of 64 keys instead of 32 under way: 2.5e-7, 1 us less). One block for 32 heads: values read once, but
// one block an SM: 54 instead of 64 us for 32 rows, 14 instead of 7 for few.
#include "common.cuh"
#include "paged_rows.cuh"

constexpr int TDM_WARPS = 8, TDM_THREADS = TDM_WARPS * 32;

__device__ __forceinline__ void tdm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool TRANS> __device__ __forceinline__ void tdm_ldmatrix(uint32_t (&r)[4], const void* smem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s) : "memory");
    else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s) : "memory");
}

// tanh(y) for |y| < 0.6, y + y t c(t) with t = y^2 and c the interpolation of (tanh(sqrt t) / sqrt t - 1) / t at the Chebyshev nodes of
// [0, 0.36]: as exact as a call of tanhf there (1.1 units in the last place). Most caps lie far above the scores.
__device__ __forceinline__ float tdm_tanh_small(float y) {
    const float t = y * y;
    float w = fmaf(-0.0062691197f, t, 0.021110959f);
    w = fmaf(w, t, -0.05387395f);
    w = fmaf(w, t, 0.13332915f);
    w = fmaf(w, t, -0.3333333135f);
    return fmaf(y, w * t, y);
}

template <int NT> struct TdmShape {
    static constexpr int WIDE = 64 * NT, HEADS = 16;
    static constexpr int KT = 32768 / WIDE < 128 ? 32768 / WIDE : 128;      // keys a step
    static constexpr int LDP = KT + 8, LDS = KT + 8;      // rows 16 bytes longer: no bank twice
    static constexpr int V_BYTES = KT * WIDE * 2, P_BYTES = 3 * HEADS * LDP * 2, S_BYTES = HEADS * LDS * 4;
    static constexpr int BYTES = V_BYTES + P_BYTES + S_BYTES + HEADS * 3 * 4 + 2 * KT * 4;
};

// q [n][H][D], out / ml as of gb_talking_attention_decode. D = 64 * DP; the wide value row has 64 * NT channels, 8 * NT a warp.
template <int NT, int DP>
__global__ void __launch_bounds__(TDM_THREADS, 2) talking_decode_mma_kernel(
    const __nv_bfloat16* __restrict__ q, float* __restrict__ out, float* __restrict__ ml, const __nv_bfloat16* __restrict__ kcache,
    const __nv_bfloat16* __restrict__ vcache, const int* __restrict__ block_tables, int max_pages, const int* __restrict__ row_seq,
    const int* __restrict__ positions, int n, int H, int G, int V, int page_size, long long num_pages, float scale, float cap, float unit,
    int window, int shares, int* __restrict__ status) {
    using Sh = TdmShape<NT>;
    constexpr int KT = Sh::KT, LDP = Sh::LDP, LDS = Sh::LDS, HEADS = Sh::HEADS, WIDE = Sh::WIDE, D = 64 * DP;
    constexpr int SN = KT / 64;                         // 8-key tiles of scores a warp forms in a step
    constexpr int PIECES = NT;                          // 16-byte pieces of a key's values a warp brings
    extern __shared__ __align__(128) unsigned char tdm_smem[];
    unsigned char* sv = tdm_smem;                                                          // [KT][WIDE] bfloat16, 16-byte pieces turned by the key
    __nv_bfloat16* sp = reinterpret_cast<__nv_bfloat16*>(sv + Sh::V_BYTES);                // [3][HEADS][LDP]: the weights' terms
    float* ss = reinterpret_cast<float*>(sv + Sh::V_BYTES + Sh::P_BYTES);                  // [HEADS][LDS]: scores
    float* s_corr = ss + HEADS * LDS;                                                      // [HEADS], then maxima, then denominators
    float* s_m = s_corr + HEADS, *s_l = s_m + HEADS;
    int* s_at = reinterpret_cast<int*>(s_l + HEADS);                                       // [2][KT]: page * G * page_size + offset, or -1
    gb_pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = lane & 3, lrow = lane >> 2;
    const int row = blockIdx.x, head0 = blockIdx.y * HEADS, share = blockIdx.z;
    const int pos = positions[row];
    if (pos < 0) return;
    if (pos / page_size >= max_pages) {
        if (tid == 0) atomicOr(status, GB_STATUS_BAD_POSITION);
        return;
    }
    const int* table = block_tables + (size_t)row_seq[row] * max_pages;
    const int first = (window > 0 && pos + 1 > window) ? pos + 1 - window : 0;
    // this block's share of the visible keys, [k_lo, k_hi): whole chunks of 32, the same count for every share but the last
    const int chunks = (pos - first) / 32 + 1, per_share = (chunks + shares - 1) / shares;
    const int k_lo = first + share * per_share * 32, k_hi = min(pos + 1, k_lo + per_share * 32);
    const int steps = k_hi > k_lo ? (k_hi - k_lo + KT - 1) / KT : 0;
    const int per = H / G;

    auto look_up = [&](int step) {                       // where the step's keys lie
        for (int i = tid; i < KT; i += TDM_THREADS) {
            const int key = k_lo + step * KT + i;
            int at = -1;
            if (key < k_hi) {
                const long long page = table[key / page_size];
                if (page < 0 || page >= num_pages) atomicOr(status, GB_STATUS_BAD_SLOT);
                else at = (int)(page * G * page_size + key % page_size);
            }
            s_at[(step & 1) * KT + i] = at;
        }
    };
    // a warp's channels are [warp * 8 NT, + 8 NT) of the wide row; half of a step's keys is one group of copies
    auto bring_values = [&](int step, int half) {
        if (step < steps) {
            constexpr int KEYS = 32 / PIECES;            // keys an instruction
            const int piece = lane % PIECES, ch = warp * 8 * NT + piece * 8;
            const long long head_off = (long long)(ch / V) * page_size * V + ch % V;
#pragma unroll 4
            for (int i = 0; i < KT / 2 / KEYS; ++i) {
                const int key = half * (KT / 2) + i * KEYS + lane / PIECES;
                const int at = s_at[(step & 1) * KT + key];
                sat_cp16(sv + key * (WIDE * 2) + (((warp * NT + piece) ^ (key & 7)) << 4), vcache + (at < 0 ? 0 : (long long)at * V + head_off), at >= 0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    if (steps > 0) look_up(0);
    if (steps > 1) look_up(1);
    gb_pdl_wait();
    __syncthreads();

    // queries as left operands: product k of a pair of pieces takes word k of pieces `quad` and `quad + 4` (8 channels each)
    uint4 qa[DP][4];
#pragma unroll
        for (int dp = 0; dp < DP; ++dp)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int head = head0 + lrow + (i & 1) * 8;
                qa[dp][i] = head < H ? *reinterpret_cast<const uint4*>(q + ((size_t)row * H + head) * D + dp * 64 + (quad + (i >> 1) * 4) * 8)
                                         : make_uint4(0, 0, 0, 0);
            }
    const float inv_cap = cap > 0.f ? 1.0f / cap : 0.f;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    constexpr int NH = Sh::HEADS / TDM_WARPS;            // heads whose weights a warp forms
    float m_run[NH], l_run[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        m_run[h] = -INFINITY;
        l_run[h] = 0.f;
    }
    const int g_lo = head0 / per, g_hi = min(G - 1, (min(H, head0 + HEADS) - 1) / per);

    for (int step = 0; step < steps; ++step) {
        // ---- scores of this warp's keys
        int at[SN];
#pragma unroll
        for (int t = 0; t < SN; ++t) at[t] = s_at[(step & 1) * KT + (warp * SN + t) * 8 + lrow];
        constexpr int GB = 8 / (SN * DP);   // key/value heads whose loads are under way together
        for (int g0 = g_lo; g0 <= g_hi; g0 += GB) {
            uint4 kb[GB][SN][DP][2];
#pragma unroll
            for (int u = 0; u < GB; ++u)
#pragma unroll
                for (int t = 0; t < SN; ++t) {
                    const __nv_bfloat16* kp = kcache + ((at[t] < 0 ? 0 : (long long)at[t]) + (long long)min(g0 + u, g_hi) * page_size) * D;
#pragma unroll
                    for (int dp = 0; dp < DP; ++dp) {
                        kb[u][t][dp][0] = *reinterpret_cast<const uint4*>(kp + dp * 64 + quad * 8);
                        kb[u][t][dp][1] = *reinterpret_cast<const uint4*>(kp + dp * 64 + (quad + 4) * 8);
                    }
                }
            if (step == 0 && g0 == g_lo) {               // (the first step's values are asked for behind its first keys)
                bring_values(0, 0);
                bring_values(0, 1);
            }
#pragma unroll
            for (int u = 0; u < GB; ++u) {
                const int g = g0 + u;
                if (g > g_hi) break;
                const bool mine0 = (head0 + lrow) / per == g, mine1 = (head0 + lrow + 8) / per == g;
                {
#pragma unroll
                    for (int t = 0; t < SN; ++t) {
                        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int dp = 0; dp < DP; ++dp) {
                            const uint4 (&a)[4] = qa[dp];
                            const uint4 (&b)[2] = kb[u][t][dp];
                            tdm_mma(c, {a[0].x, a[1].x, a[2].x, a[3].x}, b[0].x, b[1].x);
                            tdm_mma(c, {a[0].y, a[1].y, a[2].y, a[3].y}, b[0].y, b[1].y);
                            tdm_mma(c, {a[0].z, a[1].z, a[2].z, a[3].z}, b[0].z, b[1].z);
                            tdm_mma(c, {a[0].w, a[1].w, a[2].w, a[3].w}, b[0].w, b[1].w);
                        }
                        float* dst = ss + lrow * LDS + (warp * SN + t) * 8 + quad * 2;
                        if (mine0) *reinterpret_cast<float2*>(dst) = make_float2(c[0], c[1]);
                        if (mine1) *reinterpret_cast<float2*>(dst + 8 * LDS) = make_float2(c[2], c[3]);
                    }
                }
            }
        }
        __syncthreads();
        // ---- weights: a warp's two heads, two neighbouring keys a lane and 64 keys
        {
            constexpr int KL = KT / 32;                  // keys a lane
            bool seen[KL];
#pragma unroll
            for (int i = 0; i < KL; i += 2) {
                const int2 where = *reinterpret_cast<const int2*>(s_at + (step & 1) * KT + i * 32 + lane * 2);
                seen[i] = where.x >= 0;
                seen[i + 1] = where.y >= 0;
            }
            float s[NH][KL], most = 0.f;
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const bool real = head0 + warp * NH + h < H;                 // (rows past the last head: weights 0)
#pragma unroll
                for (int i = 0; i < KL; i += 2) {
                    const float2 raw = *reinterpret_cast<const float2*>(ss + (warp * NH + h) * LDS + i * 32 + lane * 2);
                    s[h][i] = real && seen[i] ? raw.x * scale : -INFINITY;
                    s[h][i + 1] = real && seen[i + 1] ? raw.y * scale : -INFINITY;
                }
            }
            if (cap > 0.f) {
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int i = 0; i < KL; ++i) {
                        const float y = s[h][i] * inv_cap;                  // (a key is masked by `seen`: the score of one that is may be -infinity too)
                        most = seen[i] && !(fabsf(y) < 0.6f) ? 1.f : most;
                    }
                const bool small = !__any_sync(0xffffffffu, most > 0.f);
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int i = 0; i < KL; ++i) {
                        const float y = s[h][i] * inv_cap;
                        if (seen[i]) s[h][i] = cap * (small ? tdm_tanh_small(y) : tanhf(y));
                    }
            }
            float top[NH], sum[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                top[h] = m_run[h];
#pragma unroll
                for (int i = 0; i < KL; ++i) top[h] = fmaxf(top[h], s[h][i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < NH; ++h) top[h] = fmaxf(top[h], __shfl_xor_sync(0xffffffffu, top[h], o));
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const bool real = head0 + warp * NH + h < H;
                sum[h] = 0.f;
#pragma unroll
                for (int i = 0; i < KL; i += 2) {
                    // (a key that cannot be read weighs nothing, also where every score so far is -infinity)
                    const float p0 = real && seen[i] ? expf(s[h][i] - top[h]) : 0.f, p1 = real && seen[i + 1] ? expf(s[h][i + 1] - top[h]) : 0.f;
                    sum[h] += p0 + p1;
                    uint32_t term[3];
                    gb_split_bf16(p0, p1, term);
#pragma unroll
                    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(sp + (e * HEADS + warp * NH + h) * LDP + i * 32 + lane * 2) = term[e];
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < NH; ++h) sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], o);
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const float corr = top[h] == -INFINITY ? 1.f : expf(m_run[h] - top[h]);
                l_run[h] = l_run[h] * corr + sum[h];
                m_run[h] = top[h];
                if (lane == 0) s_corr[warp * NH + h] = corr;
            }
        }
        __syncthreads();
        // ---- O = O * corr + P V
        {
            const float c0 = s_corr[lrow], c1 = s_corr[lrow + 8];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                acc[j][0] *= c0;
                acc[j][1] *= c0;
                acc[j][2] *= c1;
                acc[j][3] *= c1;
            }
        }
#pragma unroll 1
        for (int part = 0; part < KT / 32; ++part) {     // 32 keys: as many as sums may take before they are added in float32
            constexpr int HALF = KT / 64, NQ = NT < 4 ? NT : 4;              // parts in a group of copies; n tiles under way together
            if (part % HALF == 0) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncwarp();
            }
#pragma unroll
            for (int j0 = 0; j0 < NT; j0 += NQ) {
                float c[NQ][4];
#pragma unroll
                for (int j = 0; j < NQ; ++j) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
                uint32_t av[2][3][4], bv[2][NQ / 2][4];  // (operands of both products first: loads and products issue in order)
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) {
                    const int k0 = part * 32 + kk * 16, key = k0 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
                    for (int j2 = 0; j2 < NQ / 2; ++j2)
                        tdm_ldmatrix<true>(bv[kk][j2], sv + key * (WIDE * 2) + (((warp * NT + j0 + 2 * j2 + (lane >> 4)) ^ (key & 7)) << 4));
#pragma unroll
                    for (int e = 2; e >= 0; --e) tdm_ldmatrix<false>(av[kk][e], sp + (e * HEADS + (lane & 15)) * LDP + k0 + (lane >> 4) * 8);
                }
#pragma unroll
                for (int e = 2; e >= 0; --e)
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                        for (int j = 0; j < NQ; ++j) tdm_mma(c[j], av[kk][e], bv[kk][j / 2][(j & 1) * 2], bv[kk][j / 2][(j & 1) * 2 + 1]);
                float odd = 0.f;                         // (0 times a number that is not finite is NaN)
#pragma unroll
                for (int j = 0; j < NQ; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) odd = fmaf(0.f, c[j][e], odd);
                if (!(odd == 0.f)) {
#pragma unroll
                    for (int j = 0; j < NQ; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (fabsf(c[j][e]) <= FLT_MAX) continue;
                            float sum = 0.f;
                            const int hl = lrow + (e >> 1) * 8, ch = (j0 + j) * 8 + quad * 2 + (e & 1);
#pragma unroll 1
                            for (int k = part * 32; k < part * 32 + 32; ++k) {
                                if (s_at[(step & 1) * KT + k] < 0) continue;
                                float p = 0.f;
#pragma unroll
                                for (int t = 2; t >= 0; --t) p += __bfloat162float(sp[(t * HEADS + hl) * LDP + k]);
                                const unsigned char* v = sv + k * (WIDE * 2) + (((warp * NT + ch / 8) ^ (k & 7)) << 4) + ch % 8 * 2;
                                sum = fmaf(p, __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(v)), sum);
                            }
                            c[j][e] = sum;
                        }
                }
#pragma unroll
                for (int j = 0; j < NQ; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[j0 + j][e] += c[j][e];
            }
            if (part % HALF == HALF - 1) {
                __syncwarp();
                bring_values(step + 1, part / HALF);
            }
        }
        if (step + 2 < steps) {
            __syncthreads();                             // (everyone has brought and seen what these places were looked up for)
            look_up(step + 2);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int h = 0; h < NH; ++h)
        if (lane == 0) {
            s_m[warp * NH + h] = m_run[h];
            s_l[warp * NH + h] = l_run[h];
        }
    __syncthreads();
    const bool final_ = shares == 1;
#pragma unroll
        for (int up = 0; up < 2; ++up) {
            const int hl = lrow + up * 8;
            if (head0 + hl >= H) continue;
            float f = 1.f;
            const float m = s_m[hl], l = s_l[hl];
            if (final_) {
                const float top = unit > 0.f ? fmaxf(0.f, m) : m;
                const float fm = m == -INFINITY ? 0.f : expf(m - top);
                const float den = (unit > 0.f ? unit * expf(-top) : 0.f) + l * fm;
                f = den > 0.f ? fm / den : 0.f;
            }
            const bool none = final_ ? !(f > 0.f) : m == -INFINITY;          // nothing to say: zeros, whatever the sums hold
            const size_t at = ((size_t)share * n + row) * H + head0 + hl;
            float* dst = out + at * WIDE + warp * 8 * NT + quad * 2;
#pragma unroll
            for (int j = 0; j < NT; ++j)
                *reinterpret_cast<float2*>(dst + j * 8) = none ? make_float2(0.f, 0.f) : make_float2(acc[j][up * 2] * f, acc[j][up * 2 + 1] * f);
            if (!final_ && warp == 0 && quad == 0) {
                ml[at * 2] = m;
                ml[at * 2 + 1] = none ? 0.f : l;
            }
        }
}

// heads a block where the kernel is built: wide value rows of 128, 256 or 512 channels whose eights lie in one value head, keys of 64 or
// 128; else 0
GB_EXPORT int gb_talking_decode_mma_heads(int H, int G, int D, int V, int VG) {
    const int wide = VG * V;
    return VG == G && (D == 64 || D == 128) && V % 8 == 0 && (wide == 128 || wide == 256 || wide == 512) ? 16 : 0;
}

template <int NT, int DP>
static int tdm_launch(const void* q, float* out, float* ml, const void* kcache, const void* vcache, const int* block_tables, int max_pages,
                      const int* row_seq, const int* positions, int n, int H, int G, int V, int page_size, long long num_pages, float scale,
                      float cap, float unit, int window, int shares, int* status, cudaStream_t stream) {
    constexpr int bytes = TdmShape<NT>::BYTES;
    cudaFuncSetAttribute(talking_decode_mma_kernel<NT, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    gb_launch(GB_PDL_ATTENTION, talking_decode_mma_kernel<NT, DP>, dim3(n, gb_ceil_div(H, 16), shares), dim3(TDM_THREADS), bytes, stream,
              (const __nv_bfloat16*)q, out, ml, (const __nv_bfloat16*)kcache, (const __nv_bfloat16*)vcache, block_tables, max_pages, row_seq,
              positions, n, H, G, V, page_size, num_pages, scale, cap, unit, window, shares, status);
    return gb_check_launch("gb_talking_attention_decode");
}

// Called by gb_talking_attention_decode where gb_talking_decode_mma_heads says a size is built and the pointers are aligned.
int gb_talking_decode_mma(const void* q, float* out, float* ml, const void* kcache, const void* vcache, const int* block_tables,
                          int max_pages, const int* row_seq, const int* positions, int n, int H, int G, int D, int V, int page_size,
                          long long num_pages, float scale, float cap, float unit, int window, int shares, int* status, cudaStream_t stream) {
    const int nt = G * V / 64, dp = D / 64;
#define TDM_CASE(N, P)                                                                                                                \
    if (nt == N && dp == P)                                                                                                           \
        return tdm_launch<N, P>(q, out, ml, kcache, vcache, block_tables, max_pages, row_seq, positions, n, H, G, V, page_size,       \
                                num_pages, scale, cap, unit, window, shares, status, stream);
    TDM_CASE(2, 1) TDM_CASE(4, 1) TDM_CASE(8, 1) TDM_CASE(2, 2) TDM_CASE(4, 2) TDM_CASE(8, 2)
#undef TDM_CASE
    GB_REQUIRE(false, "gb_talking_attention_decode: head sizes %d / %d are not built", D, V);
}
