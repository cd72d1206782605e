// Causal grouped-query flash attention for prompt portions in the true 32-bit path at head sizes 96 and 128, over the paged cache: float32
// operands, FMA only, online softmax in float32. (Smaller heads: attention_prefill_f32_mma.cu.)
//
// Bound by the FMA pipe: 4 * head_dim operations per visible (query, key) pair against 8 * head_dim bytes per key that 64
// rows share. A block is 64 consecutive query rows of one request for one query head, four warps; a thread holds an 8 x 4
// piece of the 64 x 64 scores and an 8 x (head_dim / 16) piece of the output. Scores pair neighbouring channels in one packed
// FMA (query and key rows lie as they come, so a 16-byte load is two operands); the product with the values pairs two
// query rows (the weights are kept with the rows of a key side by side). Keys arrive a tile ahead through cp.async, the values
// of a tile while its scores are formed; the weights take the place of the tile's keys. One warp per (row, head), which this replaces for prompt portions, walked its keys alone
// and read every key and value row once per query row.
// Measured, one prompt of 1,000 rows, 8/2 heads of 128: 172 us.
//
// Key tiles start at multiples of 64 and a row's masked keys add nothing, so the order of a row's sums depends on its
// position and window alone, not on the batch, on how its prompt was cut, or on which pages hold the keys.
#include "common.cuh"
#include "attention_prefill_f32.h"

#include <float.h>

constexpr int PS_BM = 64, PS_BN = 64, PS_THREADS = 128;

typedef unsigned long long ps_pair;      // two floats in one 64-bit register

__device__ __forceinline__ ps_pair ps_pack(float lo, float hi) {
    ps_pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void ps_unpack(ps_pair v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void ps_fma(ps_pair& c, ps_pair a, ps_pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ ps_pair ps_mul(ps_pair a, ps_pair b) {
    ps_pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void ps_cp16(void* smem, const void* gmem, bool valid) {      // 16 bytes, or zeros
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void ps_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void ps_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }
// the largest / the sum over the 16 threads that hold one row's scores
__device__ __forceinline__ float ps_max16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float ps_sum16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// channels of a thread in the product with the values: pieces of PIECE neighbouring channels, 16 * PIECE apart
template <int HD> struct PsCols {
    static constexpr int N = HD / 16, PIECE = N % 4 == 0 ? 4 : N % 2 == 0 ? 2 : 1, PIECES = N / PIECE;
};

template <int HD> constexpr int ps_smem() { return (PS_BM * (HD + 4) + 2 * PS_BN * (HD + 4 > PS_BM + 4 ? HD + 4 : PS_BM + 4) + PS_BN * HD) * 4; }

template <int HD>
__global__ void __launch_bounds__(PS_THREADS, 1) attention_prefill_f32_kernel(
    const float* __restrict__ q, long long q_stride, float* __restrict__ out, long long out_stride, const float* __restrict__ kcache,
    const float* __restrict__ vcache, const int* __restrict__ block_tables, int max_pages, const int* __restrict__ seq_first_row,
    const int* __restrict__ seq_start_pos, int nh, int nkv, int page_size, long long num_pages, float scale, int window,
    int* __restrict__ status) {
    constexpr int QP = HD + 4;                              // floats from one query (or key) row to the next
    constexpr int PP = PS_BM + 4;                           // ... from one key's weights to the next's
    constexpr int KBUF = PS_BN * (QP > PP ? QP : PP);       // a key buffer also holds the tile's weights
    constexpr int PIECE = PsCols<HD>::PIECE, PIECES = PsCols<HD>::PIECES, CPR = HD / 4;
    extern __shared__ __align__(16) float ps_mem[];
    float* Qs = ps_mem;                                     // [64][QP]
    float* Ks = Qs + PS_BM * QP;                            // two of [64][QP]; in turn the weights [64 keys][PP]
    float* Vs = Ks + 2 * KBUF;                              // [64][HD]
    __shared__ long long off_s[4][PS_BN];                   // where a tile's keys lie in the pool (elements), -1: nowhere

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int qt = gridDim.x - 1 - blockIdx.x;              // later rows see more keys: the longest blocks start first
    const int head = blockIdx.y, seq = blockIdx.z;
    const int row0 = seq_first_row[seq];
    const int nrows = seq_first_row[seq + 1] - row0;
    const int q_lo = qt * PS_BM;
    if (q_lo >= nrows) return;
    const int rows_here = min(PS_BM, nrows - q_lo);
    const int start_pos = seq_start_pos[seq];
    const int reach = max_pages * page_size;                // positions that the block table covers
    // rows of a padding sequence, and rows beyond the table (reported), see nothing and read as zeros
    int pos_hi = start_pos < 0 ? -1 : start_pos + q_lo + rows_here - 1;
    if (pos_hi >= reach) {
        if (tid == 0) atomicOr(status, GB_STATUS_BAD_POSITION);
        pos_hi = reach - 1;
    }
    const int pos_lo = start_pos + q_lo;
    if (start_pos < 0 || pos_lo > pos_hi) {
        for (int i = tid; i < rows_here * CPR; i += PS_THREADS)
            *reinterpret_cast<float4*>(out + (size_t)(row0 + q_lo + i / CPR) * out_stride + (size_t)head * HD + (i % CPR) * 4) =
                make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const int kvh = head / (nh / nkv);
    const int key_lo = (window > 0 && pos_lo + 1 > window) ? pos_lo + 1 - window : 0;
    const int kt_begin = key_lo / PS_BN, kt_end = pos_hi / PS_BN;      // inclusive
    const int* table = block_tables + (size_t)seq * max_pages;

    auto look_up = [&](int kt) {                            // threads 0 .. 63: the tile's key rows
        if (tid < PS_BN && kt <= kt_end) {
            const int key = kt * PS_BN + tid;
            long long off = -1;
            if (key >= key_lo && key <= pos_hi) {
                const long long page = table[key / page_size];
                if (page < 0 || page >= num_pages) atomicOr(status, GB_STATUS_BAD_SLOT);
                else off = ((page * nkv + kvh) * page_size + key % page_size) * HD;
            }
            off_s[kt & 3][tid] = off;
        }
    };
    auto load_keys = [&](int kt, float* dst) {
        for (int c = tid; c < PS_BN * CPR; c += PS_THREADS) {
            const int r = c / CPR, ch = c % CPR;
            const long long off = off_s[kt & 3][r];
            ps_cp16(dst + r * QP + ch * 4, kcache + (off < 0 ? 0 : off) + ch * 4, off >= 0);
        }
    };

    look_up(kt_begin);
    look_up(kt_begin + 1);
    for (int c = tid; c < PS_BM * CPR; c += PS_THREADS) {
        const int r = c / CPR, ch = c % CPR;
        ps_cp16(Qs + r * QP + ch * 4, q + (size_t)(row0 + q_lo + min(r, rows_here - 1)) * q_stride + (size_t)head * HD + ch * 4, r < rows_here);
    }
    __syncthreads();                                        // (off_s)
    load_keys(kt_begin, Ks + (kt_begin & 1) * KBUF);
    ps_commit();

    ps_pair o[PIECES][PIECE][4];                            // [piece][channel][pair of rows]
#pragma unroll
    for (int p = 0; p < PIECES; ++p)
#pragma unroll
        for (int j = 0; j < PIECE; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) o[p][j][i] = 0ull;
    float m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = -FLT_MAX;
        l[i] = 0.f;
    }
    const int valid = pos_hi - pos_lo + 1;                  // rows that see anything
    auto last_of = [&](int i) { return ty * 8 + i < valid ? pos_lo + ty * 8 + i : -1; };      // the keys that a row sees
    auto first_of = [&](int i) { return window > 0 ? max(pos_lo + ty * 8 + i + 1 - window, 0) : 0; };

    for (int kt = kt_begin; kt <= kt_end; ++kt) {
        float* K = Ks + (kt & 1) * KBUF;
        ps_wait<0>();
        __syncthreads();                                    // this tile's keys are there; V and the other buffer are free
        for (int c = tid; c < PS_BN * CPR; c += PS_THREADS) {
            const int r = c / CPR, ch = c % CPR;
            const long long off = off_s[kt & 3][r];
            ps_cp16(Vs + r * HD + ch * 4, vcache + (off < 0 ? 0 : off) + ch * 4, off >= 0);
        }
        ps_commit();
        if (kt < kt_end) load_keys(kt + 1, Ks + ((kt + 1) & 1) * KBUF);
        ps_commit();
        look_up(kt + 2);

        // scores: rows ty * 8 + i, keys tx + 16 j; even and odd channels are summed apart
        ps_pair s2[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            ulonglong2 kv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const ulonglong2*>(K + (tx + 16 * j) * QP + d);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(Qs + (ty * 8 + i) * QP + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    ps_fma(s2[i][j], qv.x, kv[j].x);
                    ps_fma(s2[i][j], qv.y, kv[j].y);
                }
            }
        }
        const int key0 = kt * PS_BN;
        bool there[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) there[j] = off_s[kt & 3][tx + 16 * j] >= 0;
        float p[4][8];
#pragma unroll
        for (int i2 = 0; i2 < 4; ++i2) {
            float corr[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * i2 + h, last = last_of(i), first = first_of(i);
                float top = -FLT_MAX, s[4];
                bool seen[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float lo, hi;
                    ps_unpack(s2[i][j], lo, hi);
                    const int key = key0 + tx + 16 * j;
                    seen[j] = there[j] && key <= last && key >= first;
                    s[j] = seen[j] ? (lo + hi) * scale : -FLT_MAX;
                    top = fmaxf(top, s[j]);
                }
                const float m_new = fmaxf(m[i], ps_max16(top));
                corr[h] = expf(m[i] - m_new);
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    p[j][i] = seen[j] ? expf(s[j] - m_new) : 0.f;
                    sum += p[j][i];
                }
                l[i] = l[i] * corr[h] + ps_sum16(sum);
                m[i] = m_new;
            }
            const ps_pair c2 = ps_pack(corr[0], corr[1]);
#pragma unroll
            for (int pc = 0; pc < PIECES; ++pc)
#pragma unroll
                for (int j = 0; j < PIECE; ++j) o[pc][j][i2] = ps_mul(o[pc][j][i2], c2);
        }
        __syncthreads();                                    // everyone has read this tile's keys: the weights take their place
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* dst = K + (tx + 16 * j) * PP + ty * 8;
            *reinterpret_cast<float4*>(dst) = make_float4(p[j][0], p[j][1], p[j][2], p[j][3]);
            *reinterpret_cast<float4*>(dst + 4) = make_float4(p[j][4], p[j][5], p[j][6], p[j][7]);
        }
        ps_wait<1>();
        __syncthreads();                                    // the weights and the values are there
        // a tile in which some row does not see every key: what a row does not see must not reach it, not even as 0 * inf
        const bool edge = key0 + PS_BN - 1 > pos_lo || valid < rows_here || (window > 0 && pos_lo + valid - window > key0);
        if (!edge) {
#pragma unroll 2
            for (int kk = 0; kk < PS_BN; ++kk) {
                const ulonglong2 pa = *reinterpret_cast<const ulonglong2*>(K + kk * PP + ty * 8);
                const ulonglong2 pb = *reinterpret_cast<const ulonglong2*>(K + kk * PP + ty * 8 + 4);
#pragma unroll
                for (int pc = 0; pc < PIECES; ++pc) {
                    const float* vp = Vs + kk * HD + pc * 16 * PIECE + tx * PIECE;
                    float v[PIECE];
                    if constexpr (PIECE == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(vp);
                    else if constexpr (PIECE == 2) *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(vp);
                    else v[0] = vp[0];
#pragma unroll
                    for (int j = 0; j < PIECE; ++j) {
                        const ps_pair vv = ps_pack(v[j], v[j]);
                        ps_fma(o[pc][j][0], pa.x, vv);
                        ps_fma(o[pc][j][1], pa.y, vv);
                        ps_fma(o[pc][j][2], pb.x, vv);
                        ps_fma(o[pc][j][3], pb.y, vv);
                    }
                }
            }
        } else {
            const int kk_begin = max(key_lo - key0, 0), kk_end = min(pos_hi - key0 + 1, PS_BN);      // (no row sees the others)
            for (int kk = kk_begin; kk < kk_end; ++kk) {
                const float4 pa = *reinterpret_cast<const float4*>(K + kk * PP + ty * 8);
                const float4 pb = *reinterpret_cast<const float4*>(K + kk * PP + ty * 8 + 4);
                const float w[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
                const int key = key0 + kk;
#pragma unroll
                for (int pc = 0; pc < PIECES; ++pc)
#pragma unroll
                    for (int j = 0; j < PIECE; ++j) {
                        const float v = Vs[kk * HD + pc * 16 * PIECE + tx * PIECE + j];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float lo, hi;
                            ps_unpack(o[pc][j][i], lo, hi);
                            if (key <= last_of(2 * i) && key >= first_of(2 * i)) lo = fmaf(w[2 * i], v, lo);
                            if (key <= last_of(2 * i + 1) && key >= first_of(2 * i + 1)) hi = fmaf(w[2 * i + 1], v, hi);
                            o[pc][j][i] = ps_pack(lo, hi);
                        }
                    }
            }
        }
    }

#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = ty * 8 + i;
        if (r >= rows_here) continue;
        const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
        float* dst = out + (size_t)(row0 + q_lo + r) * out_stride + (size_t)head * HD;
#pragma unroll
        for (int pc = 0; pc < PIECES; ++pc)
#pragma unroll
            for (int j = 0; j < PIECE; ++j) {
                float lo, hi;
                ps_unpack(o[pc][j][i / 2], lo, hi);
                dst[pc * 16 * PIECE + tx * PIECE + j] = (i & 1 ? hi : lo) * inv;
            }
    }
}

template <int HD>
static int launch_prefill_f32(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                              const int* block_tables, int max_pages, const int* seq_first_row, const int* seq_start_pos, int num_seqs,
                              int max_rows_per_seq, int nh, int nkv, int page_size, long long num_pages, float scale, int window,
                              int* status, cudaStream_t stream) {
    constexpr int smem = ps_smem<HD>();
    auto kernel = attention_prefill_f32_kernel<HD>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        GB_REQUIRE(e == cudaSuccess, "gb_attention_prefill_f32: %d bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
    }
    dim3 grid(gb_ceil_div(max_rows_per_seq, PS_BM), nh, num_seqs);
    kernel<<<grid, PS_THREADS, smem, stream>>>(q, q_stride, out, out_stride, kcache, vcache, block_tables, max_pages, seq_first_row,
                                               seq_start_pos, nh, nkv, page_size, num_pages, scale, window, status);
    return gb_check_launch("gb_attention_prefill_f32");
}

GB_EXPORT int gb_attention_prefill_f32_supported(int nh, int nkv, int hd) {
    return nkv > 0 && nh % nkv == 0 && (hd == 16 || hd == 32 || hd == 64 || hd == 96 || hd == 128);
}

// Rows of each request are consecutive: request s owns rows seq_first_row[s] .. seq_first_row[s+1]-1, at positions
// seq_start_pos[s] + local index. q, out, caches: float32, rows aligned to 16 bytes.
GB_EXPORT int gb_attention_prefill_f32(const void* q, long long q_stride, void* out, long long out_stride, const void* kcache,
                                       const void* vcache, const int* block_tables, int max_pages, const int* seq_first_row,
                                       const int* seq_start_pos, int rows, int num_seqs, int max_rows_per_seq, int nh, int nkv, int hd, int page_size,
                                       long long num_pages, float scale, int window, int* status, cudaStream_t stream) {
    GB_REQUIRE(gb_attention_prefill_f32_supported(nh, nkv, hd), "gb_attention_prefill_f32: %d/%d heads of %d are not built", nh, nkv, hd);
    GB_REQUIRE(q_stride % 4 == 0 && out_stride % 4 == 0 && ((uintptr_t)q | (uintptr_t)out | (uintptr_t)kcache | (uintptr_t)vcache) % 16 == 0,
               "gb_attention_prefill_f32: rows must be 16-byte aligned");
    GB_REQUIRE(num_seqs >= 0 && num_seqs <= 65535 && nh <= 65535 && max_pages > 0 && page_size > 0 &&
               (long long)max_pages * page_size <= 0x7fffffff, "gb_attention_prefill_f32: bad batch shape");
    if (num_seqs == 0 || max_rows_per_seq <= 0) return 0;
#define GB_CASE(HD_)                                                                                                               \
    if (hd == HD_)                                                                                                                 \
        return launch_prefill_f32<HD_>((const float*)q, q_stride, (float*)out, out_stride, (const float*)kcache, (const float*)vcache, \
                                       block_tables, max_pages, seq_first_row, seq_start_pos, num_seqs, max_rows_per_seq, nh, nkv, page_size, \
                                       num_pages, scale, window, status, stream);
    GB_CASE(96) GB_CASE(128)
#undef GB_CASE
#define GB_CASE(HD_)                                                                                                               \
    if (hd == HD_)                                                                                                                 \
        return gb_launch_prefill_f32_mma<HD_>((const float*)q, q_stride, (float*)out, out_stride, (const float*)kcache, (const float*)vcache, \
                                              block_tables, max_pages, seq_first_row, seq_start_pos, rows, num_seqs, max_rows_per_seq, nh, nkv, \
                                              page_size, num_pages, scale, window, status, stream);
    GB_CASE(16) GB_CASE(32) GB_CASE(64)
#undef GB_CASE
    return 1;
}
