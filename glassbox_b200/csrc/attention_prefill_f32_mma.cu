// Causal grouped-query flash attention for prompt portions in the true 32-bit path at head sizes up to 64, over the paged cache: both
// products on the tensor cores (mma.sync) with the exactness of float32 sums, online softmax in float32.
//
// Every float32 operand (queries, keys, weights, values) is the exact sum of three bfloat16 numbers, each what is left rounded to the
// nearest (Henry, Tang and Heinecke 2019), of whose nine products six stay: what is left out lies below 2^-24 of a product and has either
// sign. The largest product of 16 channels or keys gets an accumulator of its own and is added in float32, since the tensor core cuts what
// it adds to; the five small ones share one per 32 keys.
// Measured against 64 bits (2-norm of the error over that of the result), this / sums by FMA: normal operands, prompts of 2 tokens 3.6e-8 /
// 4.3e-8, of 8 5.9e-8 / 8.3e-8, of 64 8.9e-8 / 1.4e-7, with queries eight times as long 2.1e-7 / 3.5e-7, 500 tokens of these 3.4e-7 / 5.5e-7.
//
// A block is 64 consecutive query rows of one request for one query head: four groups of four warps, each with every fourth tile of 32
// keys (a way), which merge at the end; a warp has 16 rows. A group's tile arrives a turn ahead through cp.async as float32, each piece
// for the thread that splits it and stores the terms as bfloat16 rows (16-byte pieces turned by the row), from which ldmatrix reads the
// fragments; the queries lie so in shared memory for all groups. The longest tiles of all heads and requests start first. The first tiles
// of many requests take blocks of one group that walks the four ways one after the other: three such blocks share a multiprocessor.
// Bound by instructions and their latency (a third of the issue slots with two groups of 64-key tiles, 8 warps an SM) and by shared
// memory's bandwidth (a third of the time). Measured, us, FMA from shared memory / this: 9/3 heads of 64, three prompts of 2,047 rows
// 173 / 60, one of 2,047 rows 294 / 120, with a window of 256 62 / 44; 15/5 heads, 1,200 rows behind 500 267 / 131; 32 prompts of 20 tokens
// 12 / 9.6, of 16 tokens at 32 heads 32 / 24; heads of 32, 1,500 rows 154 / 53, of 16 134 / 38. Two groups of 64-key tiles: 66 and 135 for
// the first two, prompts of 16 tokens at 32 heads 60.
//
// Key tiles start at multiples of 32, a way's are every fourth from a multiple on, and a row's masked keys add nothing, so the order of a
// row's sums depends on its position and window alone, not on the batch, on how its prompt was cut, or on which pages hold the keys. What a row does
// not see does not reach it, not even times zero: values that are no finite numbers are left out of the products and added for the
// rows that see them, scores that come out so are formed again by FMA.
#include "common.cuh"
#include "attention_prefill_f32.h"

constexpr int PM_BM = 64, PM_BN = 32, PM_GROUP = 128, PM_WAYS = 4;
constexpr int PM_PRODUCTS = 6;         // (left term, right term), the smallest first
__device__ constexpr int PM_LEFT[PM_PRODUCTS] = {2, 0, 1, 1, 0, 0}, PM_RIGHT[PM_PRODUCTS] = {0, 2, 1, 0, 1, 0};

__device__ __forceinline__ void pm_mma(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
template <bool TRANS> __device__ __forceinline__ uint4 pm_ldmatrix(const void* smem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    uint4 r;
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(s));
    else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(s));
    return r;
}
__device__ __forceinline__ void pm_cp16(void* smem, const void* gmem, bool valid) {      // 16 bytes, or zeros
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ bool pm_finite(float v) { return fabsf(v) <= FLT_MAX; }
__device__ __forceinline__ bool pm_splits(float v) { return fabsf(v) < __uint_as_float(0x7f7f8000u); }    // (gb_split_bf16: all terms are numbers)

// c (tiles of 8 columns) = left (16 rows, K16 groups of 16) x right: the sums over the groups. left(group, term), right(group, pair of
// tiles, term): fragments.
template <int K16, int N16, typename Left, typename Right>
__device__ __forceinline__ void pm_product(float (&c)[2 * N16][4], Left left, Right right) {
    float lo[2 * N16][4] = {};
#pragma unroll
    for (int n = 0; n < 2 * N16; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[n][e] = 0.f;
#pragma unroll
    for (int k = 0; k < K16; ++k) {
        uint4 a[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) a[e] = left(k, e);
#pragma unroll
        for (int n = 0; n < N16; ++n) {
            uint4 b[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) b[e] = right(k, n, e);
            float hi[2][4] = {};
#pragma unroll
            for (int p = 0; p < PM_PRODUCTS; ++p) {
                const uint4& r = b[PM_RIGHT[p]];
                pm_mma(p == PM_PRODUCTS - 1 ? hi[0] : lo[2 * n], a[PM_LEFT[p]], r.x, r.y);
                pm_mma(p == PM_PRODUCTS - 1 ? hi[1] : lo[2 * n + 1], a[PM_LEFT[p]], r.z, r.w);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[2 * n + i][e] += hi[i][e];
        }
    }
#pragma unroll
    for (int n = 0; n < 2 * N16; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[n][e] += lo[n][e];
}

// What the rows of a lane have come to: sums of weighted values, the largest score, the sum of the weights.
template <int HD> struct PmRows {
    float o[HD / 8][4], m[2], l[2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int n = 0; n < HD / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
        m[0] = m[1] = -FLT_MAX;
        l[0] = l[1] = 0.f;
    }
    __device__ __forceinline__ void sum_lanes() {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int x = 1; x < 4; x <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], x);
    }
    template <typename Other> __device__ __forceinline__ void add(const float (&m1)[2], const float (&l1)[2], Other other) {
        float f0[2], f1[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float top = fmaxf(m[h], m1[h]);
            f0[h] = expf(m[h] - top);
            f1[h] = expf(m1[h] - top);
            m[h] = top;
            l[h] = fmaf(l[h], f0[h], l1[h] * f1[h]);
        }
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) {
            const float4 v = other(n);
            o[n][0] = fmaf(o[n][0], f0[0], v.x * f1[0]);
            o[n][1] = fmaf(o[n][1], f0[0], v.y * f1[0]);
            o[n][2] = fmaf(o[n][2], f0[1], v.z * f1[1]);
            o[n][3] = fmaf(o[n][3], f0[1], v.w * f1[1]);
        }
    }
};

// Two launches may share a call's row tiles: the second then does not wait for the first.
enum { PM_ALONE = 0, PM_FIRST = 1, PM_SECOND = 2 };

// The requests' row tiles behind their first ones, a higher one, whose rows see more keys, before all lower ones: which request has the i-th,
// and which of its tiles is it? Every warp looks for the tile number that i falls on, by how many tiles have a number or a higher one
// (-1: no tile is left). A call of its own, so that its registers are not the kernel's.
__device__ __noinline__ int2 pm_later_tile(int i, const int* __restrict__ first_row, int num_seqs) {
    const int lane = threadIdx.x & 31;
    auto tiles_of = [&](int s) { return s < num_seqs ? (first_row[s + 1] - first_row[s] + PM_BM - 1) / PM_BM : 0; };
    const int own = tiles_of(lane);                         // (of the first 32 requests)
    auto from = [&](int t) {
        int sum = max(own - t, 0);
        for (int s = 32 + lane; s < num_seqs; s += 32) sum += max(tiles_of(s) - t, 0);
        return __reduce_add_sync(0xffffffffu, sum);
    };
    if (from(1) <= i) return make_int2(-1, 0);
    int most = own;
    for (int s = 32 + lane; s < num_seqs; s += 32) most = max(most, tiles_of(s));
    int qt = 1, hi = __reduce_max_sync(0xffffffffu, most);  // from(qt) > i >= from(hi)
    while (hi - qt > 1) {
        const int t = (qt + hi) / 2;
        if (from(t) > i) qt = t;
        else hi = t;
    }
    int nth = i - from(qt + 1);                             // among the requests that have a tile of this number
    for (int s0 = 0; s0 < num_seqs; s0 += 32) {
        const unsigned have = __ballot_sync(0xffffffffu, (s0 ? tiles_of(s0 + lane) : own) > qt);
        if (nth < __popc(have)) {
            const unsigned it = __ballot_sync(0xffffffffu, (have >> lane & 1) && __popc(have & ((1u << lane) - 1)) == nth);
            return make_int2(s0 + __ffs(it) - 1, qt);
        }
        nth -= __popc(have);
    }
    return make_int2(-1, 0);
}

// SEARCH: blocks y are the requests' later tiles (`later` of them at most), then their first ones; else y is the request and z its tile.
template <int HD, int GROUPS, bool SEARCH>
__global__ void __launch_bounds__(PM_GROUP * GROUPS, GROUPS == 1 ? 3 : 1) attention_prefill_f32_mma_kernel(
    const float* __restrict__ q, long long q_stride, float* __restrict__ out, long long out_stride, const float* __restrict__ kcache,
    const float* __restrict__ vcache, const int* __restrict__ block_tables, int max_pages, const int* __restrict__ seq_first_row,
    const int* __restrict__ seq_start_pos, int num_seqs, int nh, int nkv, int page_size, long long num_pages, float scale, int window,
    int* __restrict__ status, int later, int part) {
    constexpr int CPR = HD / 8, K16 = HD / 16;              // 16-byte pieces of a row of one term; groups of 16 channels
    constexpr int TERM = PM_BN * HD * 2, TILE = 3 * TERM;   // bytes of a tile's term; of its terms
    constexpr int LOADS = PM_BN * HD / 4 / PM_GROUP;        // 16-byte loads of a thread and tile
    extern __shared__ __align__(128) unsigned char pm_mem[];
    __shared__ long long off_s[GROUPS][4][PM_BN];           // where a tile's keys lie in the pool (elements), -1: nowhere
    __shared__ unsigned there_s[GROUPS][4];                 // ... which are there, as bits
    __shared__ int odd_s[GROUPS][4];                        // ... and whether the split does not take a value of theirs

    const int tid = threadIdx.x % PM_GROUP, group = threadIdx.x / PM_GROUP, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int head = blockIdx.x;
    // The second of two launches may start when all blocks of the first have passed their wait for what came before both; it waits for
    // the first at its end, so that whoever waits for the second has waited for both.
    if (part != PM_FIRST) gb_pdl_launch_dependents();
    if (part != PM_SECOND) gb_pdl_wait();
    if (part == PM_FIRST) gb_pdl_launch_dependents();
    struct AtEnd {
        bool wait;
        __device__ ~AtEnd() {
            if (wait) gb_pdl_wait();
        }
    } at_end{part == PM_SECOND};
    int seq = blockIdx.y, qt = gridDim.z - 1 - blockIdx.z;  // later rows see more keys: the longest blocks start first
    if (SEARCH) {
        seq -= later;
        if (seq < 0) {
            const int2 at = pm_later_tile(blockIdx.y, seq_first_row, num_seqs);
            if (at.x < 0) return;
            seq = at.x;
            qt = at.y;
        }
    }
    const int row0 = seq_first_row[seq];
    const int nrows = seq_first_row[seq + 1] - row0;
    const int q_lo = qt * PM_BM;
    if (q_lo >= nrows) return;
    const int rows_here = min(PM_BM, nrows - q_lo);
    const int start_pos = seq_start_pos[seq];
    const int reach = max_pages * page_size;                // positions that the block table covers
    // rows of a padding sequence, and rows beyond the table (reported), see nothing and read as zeros
    int pos_hi = start_pos < 0 ? -1 : start_pos + q_lo + rows_here - 1;
    if (pos_hi >= reach) {
        if (threadIdx.x == 0) atomicOr(status, GB_STATUS_BAD_POSITION);
        pos_hi = reach - 1;
    }
    const int pos_lo = start_pos + q_lo;
    if (start_pos < 0 || pos_lo > pos_hi) {
        for (int i = threadIdx.x; i < rows_here * (HD / 4); i += PM_GROUP * GROUPS)
            *reinterpret_cast<float4*>(out + (size_t)(row0 + q_lo + i / (HD / 4)) * out_stride + (size_t)head * HD + (i % (HD / 4)) * 4) =
                make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const int kvh = head / (nh / nkv);
    const int key_lo = (window > 0 && pos_lo + 1 > window) ? pos_lo + 1 - window : 0;
    const int kt_end = pos_hi / PM_BN;                      // inclusive
    const int kt_begin = key_lo / PM_BN;
    // the first tile of a way, and the tile behind one: the next of its way, else (a lone group walks all ways) the first of the next
    auto first_of_way = [&](int way) { return kt_begin + ((way - kt_begin) & (PM_WAYS - 1)); };
    auto next_of = [&](int kt) {
        if (kt < 0 || kt + PM_WAYS <= kt_end) return kt < 0 ? -1 : kt + PM_WAYS;
        if (GROUPS == 1)
            for (int way = (kt & (PM_WAYS - 1)) + 1; way < PM_WAYS; ++way)
                if (first_of_way(way) <= kt_end) return first_of_way(way);
        return -1;
    };
    int kt = first_of_way(group);
    if (kt > kt_end) kt = GROUPS == 1 ? kt_begin : -1;
    if (GROUPS == 1)                                        // (ways in their order, whichever tile is the first)
        for (int way = PM_WAYS - 1; way >= 0; --way)
            if (first_of_way(way) <= kt_end) kt = first_of_way(way);
    const int* table = block_tables + (size_t)seq * max_pages;
    constexpr int Q_TERM = PM_BM * HD * 2, RAW = PM_BN * HD * 4;
    unsigned char* Qs = pm_mem;                             // [3 terms][64 rows][HD] bfloat16
    unsigned char* Ks = pm_mem + 3 * Q_TERM + group * (2 * TILE + 2 * RAW);       // [3 terms][32 keys][HD] bfloat16, then the values'
    unsigned char* Vs = Ks + TILE;
    float* raw_k = reinterpret_cast<float*>(Vs + TILE);     // the next tile as it lies in the cache
    float* raw_v = raw_k + PM_BN * HD;
    auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(PM_GROUP) : "memory"); };

    auto look_up = [&](int kt, int slot) {                  // a warp: the tile's key rows
        if (warp == 0 && kt >= 0) {
            const int key = kt * PM_BN + lane;
            long long off = -1;
            if (key >= key_lo && key <= pos_hi) {
                const long long page = table[key / page_size];
                if (page < 0 || page >= num_pages) atomicOr(status, GB_STATUS_BAD_SLOT);
                else off = ((page * nkv + kvh) * page_size + key % page_size) * HD;
            }
            off_s[group][slot][lane] = off;
            const unsigned there = __ballot_sync(0xffffffffu, off >= 0);
            if (lane == 0) {
                there_s[group][slot] = there;
                odd_s[group][slot] = 0;
            }
        }
    };
    // a thread's pieces of four channels of a tile: piece tid % (HD / 4) of every (PM_GROUP / (HD / 4))th key
    constexpr int KSTEP = PM_GROUP / (HD / 4);
    const int lkey = tid / (HD / 4), lch = tid % (HD / 4) * 4;
    auto raw_of = [&](int i) { return tid * 4 + i * (PM_GROUP * 4); };
    auto fetch = [&](int slot) {                            // ... as float32, which only the thread itself reads
#pragma unroll
        for (int i = 0; i < LOADS; ++i) {
            const long long off = off_s[group][slot][lkey + i * KSTEP];
            pm_cp16(raw_k + raw_of(i), kcache + (off < 0 ? 0 : off + lch), off >= 0);
            pm_cp16(raw_v + raw_of(i), vcache + (off < 0 ? 0 : off + lch), off >= 0);
        }
    };
    auto place = [&](int row, int piece) { return row * (HD * 2) + ((piece ^ ((row / (8 / CPR)) & (CPR - 1))) << 4); };
    auto store = [&](unsigned char* tile, int term, int row, const float4& v) {
        uint32_t lo[3], hi[3];
        gb_split_bf16(v.x, v.y, lo);
        gb_split_bf16(v.z, v.w, hi);
        unsigned char* to = tile + place(row, lch >> 3) + (lch & 4) * 2;
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(to + e * term) = make_uint2(lo[e], hi[e]);
    };

    int ahead = next_of(kt), it = 0;                        // the tile behind this one; turns so far (a tile's slot is its turn)
    look_up(kt, 0);
    look_up(ahead, 1);
    meet();
    if (kt >= 0) fetch(0);
    asm volatile("cp.async.commit_group;");
    for (int r = threadIdx.x / (HD / 4); r < PM_BM; r += PM_GROUP * GROUPS / (HD / 4))
        store(Qs, Q_TERM, r, *reinterpret_cast<const float4*>(q + (size_t)(row0 + q_lo + min(r, rows_here - 1)) * q_stride + (size_t)head * HD + lch));
    __syncthreads();
    const int r_lo = warp * 16 + g;                         // this lane's rows: r_lo and r_lo + 8
    const int valid = pos_hi - pos_lo + 1;                  // rows that see anything
    int last[2], first[2];                                  // the keys that a row sees
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = r_lo + 8 * h;
        last[h] = r < valid ? pos_lo + r : -1;
        first[h] = window > 0 ? max(pos_lo + r + 1 - window, 0) : 0;
    }
    const float* qrow[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) qrow[h] = q + (size_t)(row0 + q_lo + min(r_lo + 8 * h, rows_here - 1)) * q_stride + (size_t)head * HD;
    PmRows<HD> rows, total;                                 // total: a lone group's ways so far
    rows.clear();
    if (GROUPS == 1) total.clear();
    auto& o = rows.o;
    auto& m = rows.m;
    auto& l = rows.l;                                       // (this lane's share)

    while (kt >= 0) {
        const int slot = it & 3;
        asm volatile("cp.async.wait_group 0;");
        meet();                                             // everyone is done with the tile before
        bool odd_v = false;
#pragma unroll 2
        for (int i = 0; i < LOADS; ++i) {
            store(Ks, TERM, lkey + i * KSTEP, *reinterpret_cast<const float4*>(raw_k + raw_of(i)));
            // (values without what the split does not take)
            float4 v = *reinterpret_cast<const float4*>(raw_v + raw_of(i));
            const bool fx = pm_splits(v.x), fy = pm_splits(v.y), fz = pm_splits(v.z), fw = pm_splits(v.w);
            odd_v |= !(fx && fy && fz && fw);
            store(Vs, TERM, lkey + i * KSTEP, make_float4(fx ? v.x : 0.f, fy ? v.y : 0.f, fz ? v.z : 0.f, fw ? v.w : 0.f));
        }
        if (odd_v) odd_s[group][slot] = 1;
        meet();                                             // the tile is there
        const int behind = next_of(ahead);
        if (ahead >= 0) fetch((it + 1) & 3);
        asm volatile("cp.async.commit_group;");
        look_up(behind, (it + 2) & 3);
        const unsigned there = there_s[group][slot];
        const int key0 = kt * PM_BN;
        // a tile in which some row does not see every key
        const bool edge = key0 + PM_BN - 1 > pos_lo || valid < rows_here || (window > 0 && pos_lo + valid - window > key0) || there != 0xffffffffu;
        {
            // scores of keys key0 + 8 j + 2 t4 (+ 1)
            float s[PM_BN / 8][4];
            pm_product<K16, PM_BN / 16>(
                s, [&](int k, int e) { return pm_ldmatrix<false>(Qs + e * Q_TERM + place(16 * warp + (lane & 15), 2 * k + (lane >> 4))); },
                [&](int k, int n, int e) {
                    return pm_ldmatrix<false>(Ks + e * TERM + place(16 * n + (lane & 7) + ((lane >> 4) & 1) * 8, 2 * k + ((lane >> 3) & 1)));
                });
            auto seen = [&](int j, int e) {                 // whether score s[j][e] counts
                const int kk = 8 * j + 2 * t4 + (e & 1), h = e >> 1;
                return key0 + kk <= last[h] && key0 + kk >= first[h] && ((there >> kk) & 1u);
            };
            float top[2] = {-FLT_MAX, -FLT_MAX};
            bool odd = false;
#pragma unroll
            for (int j = 0; j < PM_BN / 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s[j][e] *= scale;
                    const bool in = !edge || seen(j, e);
                    odd |= in && !pm_finite(s[j][e]);
                    if (!in) s[j][e] = -INFINITY;           // (its weight is 0)
                    else top[e >> 1] = fmaxf(top[e >> 1], s[j][e]);
                }
            if (__any_sync(0xffffffffu, odd)) {
                top[0] = top[1] = -FLT_MAX;
#pragma unroll
                for (int j = 0; j < PM_BN / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (edge && !seen(j, e)) continue;
                        if (!pm_finite(s[j][e])) {
                            const float* krow = kcache + off_s[group][slot][8 * j + 2 * t4 + (e & 1)];
                            float v = 0.f;
#pragma unroll 1
                            for (int d = 0; d < HD; ++d) v = fmaf(qrow[e >> 1][d], krow[d], v);
                            s[j][e] = v * scale;
                        }
                        top[e >> 1] = fmaxf(top[e >> 1], s[j][e]);
                    }
                __syncwarp();
            }
            uint4 P[PM_BN / 16][3];                        // the weights as the left operand
            float corr[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int x = 1; x < 4; x <<= 1) top[h] = fmaxf(top[h], __shfl_xor_sync(0xffffffffu, top[h], x));
                const float m_new = fmaxf(m[h], top[h]);
                corr[h] = expf(m[h] - m_new);
                m[h] = m_new;
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < PM_BN / 8; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        s[j][2 * h + e] = expf(s[j][2 * h + e] - m_new);
                        sum += s[j][2 * h + e];
                    }
                l[h] = l[h] * corr[h] + sum;
            }
#pragma unroll
            for (int k = 0; k < PM_BN / 16; ++k) {
                uint32_t w[4][3];
#pragma unroll
                for (int r = 0; r < 4; ++r) gb_split_bf16(s[2 * k + (r >> 1)][2 * (r & 1)], s[2 * k + (r >> 1)][2 * (r & 1) + 1], w[r]);
#pragma unroll
                for (int e = 0; e < 3; ++e) P[k][e] = make_uint4(w[0][e], w[1][e], w[2][e], w[3][e]);
            }
#pragma unroll
            for (int n16 = 0; n16 < HD / 16; ++n16) {
                float c[2][4];
                pm_product<PM_BN / 16, 1>(
                    c, [&](int k, int e) { return P[k][e]; },
                    [&](int k, int, int e) { return pm_ldmatrix<true>(Vs + e * TERM + place(16 * k + (lane & 15), 2 * n16 + (lane >> 4))); });
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[2 * n16 + n][e] = fmaf(o[2 * n16 + n][e], corr[e >> 1], c[n][e]);
            }
            if (odd_s[group][slot]) {                       // (uniform for the group)
#pragma unroll
                for (int j = 0; j < PM_BN / 8; ++j)
#pragma unroll 1
                    for (int x = 0; x < 8; ++x) {
                        const int kk = 8 * j + x, src = (lane & 28) | (x >> 1);
                        float w[2];                         // the weights, as the sums of their terms
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            w[h] = 0.f;
#pragma unroll
                            for (int e = 0; e < 3; ++e) {
                                const uint4& a = P[j >> 1][e];
                                const uint32_t both = __shfl_sync(0xffffffffu, j & 1 ? (h ? a.w : a.z) : (h ? a.y : a.x), src);
                                w[h] += __uint_as_float(x & 1 ? both & 0xffff0000u : both << 16);
                            }
                        }
                        if (!((there >> kk) & 1u)) continue;
                        const float* vrow = vcache + off_s[group][slot][kk];
#pragma unroll
                        for (int n = 0; n < HD / 8; ++n)
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float v = vrow[8 * n + 2 * t4 + (e & 1)];
                                if (!pm_splits(v) && key0 + kk <= last[e >> 1] && key0 + kk >= first[e >> 1]) o[n][e] = fmaf(w[e >> 1], v, o[n][e]);
                            }
                    }
                __syncwarp();
            }
        }
        if (GROUPS == 1 && (ahead < 0 || ((ahead ^ kt) & (PM_WAYS - 1)))) {      // the way ends here
            rows.sum_lanes();
            total.add(m, l, [&](int n) { return make_float4(o[n][0], o[n][1], o[n][2], o[n][3]); });
            rows.clear();
        }
        kt = ahead;
        ahead = behind;
        ++it;
    }

    if (GROUPS > 1) {
        // merge: the other groups leave their rows in shared memory, the first adds them to its own in turn
        constexpr int LANE = HD / 2 + 4, SHARE = 4 * 32 * LANE;
        float* place_of = reinterpret_cast<float*>(pm_mem) + (warp * 32 + lane) * LANE;
        rows.sum_lanes();
        asm volatile("cp.async.wait_group 0;");
        __syncthreads();
        if (group > 0) {
            float* mine = place_of + (group - 1) * SHARE;
#pragma unroll
            for (int n = 0; n < HD / 8; ++n) *reinterpret_cast<float4*>(mine + 4 * n) = make_float4(o[n][0], o[n][1], o[n][2], o[n][3]);
            *reinterpret_cast<float4*>(mine + HD / 2) = make_float4(m[0], m[1], l[0], l[1]);
        }
        __syncthreads();
        if (group > 0) return;
#pragma unroll 1
        for (int i = 0; i < GROUPS - 1; ++i) {
            const float* theirs = place_of + i * SHARE;
            const float4 ml = *reinterpret_cast<const float4*>(theirs + HD / 2);
            const float m1[2] = {ml.x, ml.y}, l1[2] = {ml.z, ml.w};
            rows.add(m1, l1, [&](int n) { return *reinterpret_cast<const float4*>(theirs + 4 * n); });
        }
    }
    const PmRows<HD>& sum = GROUPS == 1 ? total : rows;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = r_lo + 8 * h;
        const float inv = sum.l[h] > 0.f ? 1.0f / sum.l[h] : 0.f;
        if (r >= rows_here) continue;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n)
            *reinterpret_cast<float2*>(out + (size_t)(row0 + q_lo + r) * out_stride + (size_t)head * HD + 8 * n + 2 * t4) =
                make_float2(sum.o[n][2 * h] * inv, sum.o[n][2 * h + 1] * inv);
    }
}

template <int HD, int GROUPS, bool SEARCH>
static int pm_launch(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                     const int* block_tables, int max_pages, const int* seq_first_row, const int* seq_start_pos, int num_seqs, int nh, int nkv, int page_size, long long num_pages, float scale, int window, int* status,
                     cudaStream_t stream, long long y, long long z, int later, int part) {
    constexpr int tiles_bytes = 3 * PM_BM * HD * 2 + GROUPS * 2 * PM_BN * HD * (3 * 2 + 4), merge_bytes = (GROUPS - 1) * 4 * 32 * (HD / 2 + 4) * 4;
    constexpr int smem = tiles_bytes > merge_bytes ? tiles_bytes : merge_bytes;
    auto kernel = attention_prefill_f32_mma_kernel<HD, GROUPS, SEARCH>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    GB_REQUIRE(e == cudaSuccess, "gb_attention_prefill_f32: %d bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
    GB_REQUIRE(y <= 65535 && z <= 65535, "gb_attention_prefill_f32: too many row tiles (%lld x %lld)", y, z);
    gb_launch(GB_PDL_ATTENTION, kernel, dim3(nh, (unsigned)y, (unsigned)z), dim3(PM_GROUP * GROUPS), smem, stream, q, q_stride, out, out_stride, kcache,
              vcache, block_tables, max_pages, seq_first_row, seq_start_pos, num_seqs, nh, nkv, page_size, num_pages, scale, window, status, later, part);
    return gb_check_launch("gb_attention_prefill_f32");
}

template <int HD>
int gb_launch_prefill_f32_mma(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                              const int* block_tables, int max_pages, const int* seq_first_row, const int* seq_start_pos, int rows, int num_seqs,
                              int max_rows_per_seq, int nh, int nkv, int page_size, long long num_pages, float scale, int window,
                              int* status, cudaStream_t stream) {
#define PM_LAUNCH(GROUPS_, SEARCH_, Y_, Z_, LATER_, PART_)                                                                                 \
    pm_launch<HD, GROUPS_, SEARCH_>(q, q_stride, out, out_stride, kcache, vcache, block_tables, max_pages, seq_first_row, seq_start_pos, num_seqs, \
                                    nh, nkv, page_size, num_pages, scale, window, status, stream, Y_, Z_, LATER_, PART_)
    // A recorded step gives its shape's longest possible portion, of which a grid of requests by tiles is mostly empty: where that has twice
    // as many tiles as the requests can have between them (a whole one for every 64 rows, one for each request), these are looked for.
    // The first tiles of many requests (more blocks than multiprocessors) then take one group a block, where a block's start and end
    // count, and the others four, side by side; where a first tile may see many keys, from 512 blocks on (fewer leave a walk of one
    // group alone at the end). All forms give the same bits. Measured, us, recorded shapes, grid of requests by tiles with four groups /
    // by this rule: 32 prompts of 16 tokens at 9, 15, 32 and 64 heads 18 / 11, 33 / 16, 60 / 26 and 118 / 45 (FMA 16, 23, 38 and
    // 67); a prompt of 1,000 beside 31 of 16 tokens 64 / 60, 101 / 79, 209 / 145 and 411 / 282; 16 x 64 tokens behind 500 at 15 heads 79 / 73
    // (first tiles by one group 97); eight of 100 tokens at 9 heads 12.9 / 11.9. Longest portion known: 8 x 100 11.1 without a search
    // (12.0 with), 32 x 16 tokens at 32 heads 23.1 with one group (49 with four).
    const long long tiles = gb_ceil_div(max_rows_per_seq, PM_BM), most = num_seqs * (tiles - 1);
    const long long later = rows / PM_BM < most ? rows / PM_BM : most, blocks = (long long)nh * num_seqs;
    const bool known = num_seqs * tiles <= 2 * (later + num_seqs);
    const bool one = blocks > 148 && (later == 0 || (!known && (blocks >= 512 || (long long)max_pages * page_size <= 256)));
    if (one && later == 0) return PM_LAUNCH(1, false, num_seqs, 1, 0, PM_ALONE);
    if (known) return PM_LAUNCH(PM_WAYS, false, num_seqs, tiles, 0, PM_ALONE);
    if (!one) return PM_LAUNCH(PM_WAYS, true, later + num_seqs, 1, (int)later, PM_ALONE);
    const int rc = PM_LAUNCH(PM_WAYS, true, later, 1, (int)later, PM_FIRST);
    return rc ? rc : PM_LAUNCH(1, false, num_seqs, 1, 0, PM_SECOND);
#undef PM_LAUNCH
}
#define PM_BUILD(HD_)                                                                                                                      \
    template int gb_launch_prefill_f32_mma<HD_>(const float*, long long, float*, long long, const float*, const float*, const int*, int, \
                                                const int*, const int*, int, int, int, int, int, int, long long, float, int, int*, cudaStream_t);
PM_BUILD(16) PM_BUILD(32) PM_BUILD(64)
