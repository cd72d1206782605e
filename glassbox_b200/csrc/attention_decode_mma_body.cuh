// The body of the tensor-core decode attention (see attention_decode_mma.cu for the method) as a device function of
// a *virtual* block (split, kv head, row), so that the same code serves the stand-alone kernel, whose blocks are the
// virtual blocks, and the persistent decode-program kernel (decode_program.cu), whose resident blocks walk over them.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

struct DecodeAttnArgs {
    const __nv_bfloat16* q;
    long long q_stride;
    __nv_bfloat16* out;
    long long out_stride;
    const __nv_bfloat16* kcache;
    const __nv_bfloat16* vcache;
    const int* block_tables;
    int max_pages;
    const int* row_seq;
    const int* positions;
    int nh, nkv, page_size, page_shift;
    long long num_pages;
    float scale;
    int window, splits;     // (window: as gb_first_key's mask)
    float* part_acc;
    float* part_ml;
    int* counters;
    int* status;
    int n;           // rows (used by the persistent kernel to count its virtual blocks)
    int hd, block_keys;
    int late_release;   // let the next kernel in the stream go only after this one's own wait (else at its start)
    // Read only by the SINK instantiations (each may be nullptr): the score, capped as cap * tanh(score / cap) where cap > 0,
    // of a key `dist` tokens back loses
    // r1[head] * ln(1 + r2[head] * dist); the softmax's denominator also holds exp(sink[head]), which has no key and
    // no value; the head's output is multiplied by sigmoid(gate[row * ld_gate + head]) (float32 logits), or, with
    // gate_channels, channel c of it by sigmoid(gate[row * ld_gate + head * HD + c]).
    const float* r1;
    const float* r2;
    const float* sink;
    const float* gate;
    long long ld_gate;
    int gate_channels;
    float cap;
};

constexpr float MMA_NEG_BIG = -1.0e30f;
constexpr int MMA_MAX_PARTS = 2048;   // partial results of a head (splits x warps) at most
constexpr int MMA_MAX_PAGES = 1024;   // page ids of one block's key range kept in shared memory
constexpr int MMA_SCRATCH = 3072;     // floats in which a block's warps add up their results

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// Keys and values are read once: they leave no line behind in L1 (which keeps the small things that are read again:
// page ids, the products' activations). An ordinary load, not a read-only one: in a persistent kernel another block
// of the same launch has written this step's keys and values.
__device__ __forceinline__ uint4 kv_load16(const void* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

template <int WORDS> struct RowLoad;  // WORDS 32-bit words of a value row, widest loads possible
template <> struct RowLoad<1> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, uint32_t (&w)[1]) {
        w[0] = *reinterpret_cast<const uint32_t*>(p);
    }
};
template <> struct RowLoad<2> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, uint32_t (&w)[2]) {
        uint2 v = *reinterpret_cast<const uint2*>(p);
        w[0] = v.x; w[1] = v.y;
    }
};
template <> struct RowLoad<4> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, uint32_t (&w)[4]) {
        uint4 v = kv_load16(p);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
};
template <> struct RowLoad<6> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, uint32_t (&w)[6]) {
        const uint2* q = reinterpret_cast<const uint2*>(p);      // (a share of 24 bytes starts 8-byte aligned)
        const uint2 a = q[0], b = q[1], c = q[2];
        w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y; w[4] = c.x; w[5] = c.y;
    }
};
template <> struct RowLoad<8> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, uint32_t (&w)[8]) {
        uint4 a = *reinterpret_cast<const uint4*>(p), b = *reinterpret_cast<const uint4*>(p + 8);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    }
};

// `sync` says how to wait for the work before (GbPdlSync in the stand-alone kernel, a barrier's wait in a persistent
// one). Queries, which another block of the same launch may have written, are read past L1.
// Shared memory of the body, provided by the caller.
struct __align__(16) DecodeAttnSmem {   // (a multiple of 16 bytes, so that arrays of it keep what follows aligned)
    union {
        int pages[MMA_MAX_PAGES];
        float scratch[MMA_SCRATCH];   // once no page id is needed any more
    };
    int is_last;
};

// NW warps (NW * 32 threads) work on one virtual block: 4, or 8 where few blocks would otherwise leave the chip's
// memory system idle (a small batch): each warp then has half as many blocks of keys to walk through.
// Floats of shared memory that the merge inside a thread-block cluster needs in every block: one (output row, maximum, sum) per head of
// the group and per warp of its own, then (in the first block) per split.
template <int HD>
__host__ __device__ constexpr int decode_attn_cluster_floats(int group, int splits, int warps) { return group * (splits + warps) * (HD + 2); }

// CLUSTER: the blocks of one (row, kv head), one per split, are one thread-block cluster (the caller launches them so; one block may
// stand alone). A block adds up its warps' partial results in its own shared memory (`cluster_part`, decode_attn_cluster_floats<HD>()
// floats, the same offset in every block) and puts one result into the first block's; they meet at the cluster's barrier, and the
// first block merges the splits: no trip through global memory, no counter, no second pass over what other blocks wrote. Otherwise
// the blocks' results go through `part_acc` / `part_ml` and the block that arrives last at `counters` merges them.
template <int HD, int BK, class Sync, int NW = 4, bool CLUSTER = false, bool SINK = false>
__device__ __forceinline__ void attention_decode_mma_body(const DecodeAttnArgs& a, const int split, const int kvh, const int row,
                                                          DecodeAttnSmem& sm, Sync& sync, float* cluster_part = nullptr) {
    constexpr int NTHREADS = NW * 32;
    const __nv_bfloat16* __restrict__ q = a.q;
    const long long q_stride = a.q_stride, out_stride = a.out_stride;
    __nv_bfloat16* __restrict__ out = a.out;
    const __nv_bfloat16* __restrict__ kcache = a.kcache;
    const __nv_bfloat16* __restrict__ vcache = a.vcache;
    const int* __restrict__ block_tables = a.block_tables;
    const int max_pages = a.max_pages;
    const int* __restrict__ row_seq = a.row_seq;
    const int* __restrict__ positions = a.positions;
    const int nh = a.nh, nkv = a.nkv, page_size = a.page_size, page_shift = a.page_shift;
    const long long num_pages = a.num_pages;
    const float scale = a.scale;
    const int window = a.window, splits = a.splits;
    float* __restrict__ part_acc = a.part_acc;
    float* __restrict__ part_ml = a.part_ml;
    int* __restrict__ counters = a.counters;
    int* __restrict__ status = a.status;
    constexpr int KS = HD / 16;   // k16 steps over the channels (scores)
    constexpr int NT = HD / 8;    // n8 tiles over the channels (output)
    constexpr int KT = BK / 8;    // n8 tiles over the keys of a block (scores)
    constexpr int KB = BK / 16;   // k16 steps over the keys of a block (output)
    constexpr int VW = NT / 2;    // 32-bit words of a value row per thread
    const int tid = sync.thread(), lane = tid & 31, warp = tid >> 5;   // NW * 32 threads work on one virtual block
    const int g = lane >> 2, t = lane & 3;
    const int G = nh / nkv;
    const int head0 = kvh * G;
    int& is_last = sm.is_last;
    // SINK: the distance bias of this thread's two heads (rows g and g + 8 of the score tile), and what a merged head's
    // denominator and output still need: the sink's logit joins the maximum and the sum, the gate scales the result
    float sk_b1[2] = {0.f, 0.f}, sk_b2[2] = {0.f, 0.f};
    if constexpr (SINK) {
        if (a.r1 != nullptr) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (g + 8 * h < G) {
                    sk_b1[h] = a.r1[head0 + g + 8 * h];
                    sk_b2[h] = a.r2[head0 + g + 8 * h];
                }
        }
    }
    const float cap = SINK ? a.cap : 0.f, inv_cap2 = cap > 0.f ? 2.0f / cap : 0.f;
    auto sink_logit = [&](int head) { return (SINK && a.sink != nullptr) ? a.sink[head] : MMA_NEG_BIG; };
    auto channel_gate = [&](int head, int c) {
        return (SINK && a.gate != nullptr && a.gate_channels) ? 1.0f / (1.0f + __expf(-a.gate[(size_t)row * a.ld_gate + head * HD + c])) : 1.0f;
    };
    auto gate_factor = [&](int head) {
        return (SINK && a.gate != nullptr && !a.gate_channels) ? 1.0f / (1.0f + __expf(-a.gate[(size_t)row * a.ld_gate + head])) : 1.0f;
    };

    // This kernel's own prologue (positions, block table: step metadata that no kernel writes) runs before it waits
    // for its predecessor, which wrote the queries and this step's keys and values. The next kernel in the stream is
    // let go only after that wait: released earlier, kernels pile up on the SMs, resident and waiting, in the way of
    // the one that works.
    if (!a.late_release) sync.start();
    int pos = positions[row];
    if (pos >= 0 && (pos >> page_shift) >= max_pages) {   // a position the block table does not reach: reported, and the
        if (tid == 0) atomicOr(status, GB_STATUS_BAD_POSITION);   // row is treated as padding (nothing is read)
        pos = -1;
    }
    __nv_bfloat16* orow = out + (size_t)row * out_stride;
    if (pos < 0) {  // padding row
        sync.wait();
        if (a.late_release) sync.start();
        if (sync.gave_up()) return;
        if (split == 0)
            for (int i = tid; i < G * HD; i += NTHREADS) orow[head0 * HD + i] = __float2bfloat16_rn(0.f);
        return;
    }
    if constexpr (CLUSTER)   // every block of the cluster says that it runs (its shared memory exists); waited for before the first store into another block's
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int* table = block_tables + (size_t)row_seq[row] * max_pages;
    const int first = gb_first_key(pos, window);
    const int first_aligned = first / BK * BK;   // blocks of keys start at multiples of BK; keys before `first` are masked
    const int total = pos + 1 - first_aligned;
    const int chunk = ((total + splits - 1) / splits + BK - 1) / BK * BK;
    const int k_begin = first_aligned + split * chunk;
    const int k_end = min(pos + 1, k_begin + chunk);
    const int nblocks = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;

    float m_run[2] = {MMA_NEG_BIG, MMA_NEG_BIG}, l_run[2] = {0.f, 0.f};
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

    // Page ids of this block's key range are staged in shared memory once (bad ids are reported and
    // replaced by page 0, whose rows are then masked like any key outside the range), and blocks of
    // keys start at multiples of BK, so a half-block of 16 keys lies in one page (pages hold a power
    // of two >= 16 keys) and its addresses are a few integer operations. Loads never branch. They
    // run one block of keys ahead of the arithmetic (two register sets), so that a warp always has
    // loads in flight.
    int* pages_s = sm.pages;
    const int page_mask = page_size - 1;
    const int page_lo = k_begin >> page_shift;
    const int n_pages = nblocks > 0 ? ((k_end - 1) >> page_shift) - page_lo + 1 : 0;
    const bool staged = n_pages <= MMA_MAX_PAGES;
    int bad = 0;
    if (staged) {
        for (int i = tid; i < n_pages; i += NTHREADS) {
            int page = table[page_lo + i];
            if (page < 0 || page >= num_pages) {
                // a page wholly before the first visible key may have been given back (window): its
                // keys are masked; any other missing page is an error
                if (((page_lo + i + 1) << page_shift) > first) bad = 1;
                page = 0;
            }
            pages_s[i] = page;
        }
        sync.group_barrier();
    }
    sync.wait();   // the writes of the work before (q, this step's K/V) are visible from here
    if (a.late_release) sync.start();
    if (sync.gave_up()) return;
    // Q as the A operand: rows g and g+8 are query heads head0+g and head0+g+8 (zero beyond G).
    uint32_t qf[KS][4];
    {
        const __nv_bfloat16* q0 = q + (size_t)row * q_stride + (size_t)(head0 + g) * HD;
        const __nv_bfloat16* q1 = q0 + 8 * HD;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            uint2 a = make_uint2(0, 0), b = make_uint2(0, 0);   // (shadow the argument block inside this scope)
            // the four channels that stand for this thread's k indices of step s: any assignment works as long as the
            // keys use the same one; with an even number of steps a thread's channels of two steps are 8 in a row, so
            // that a key's share is one 16-byte load
            const int ch = KS % 2 == 0 ? 32 * (s >> 1) + 8 * t + 4 * (s & 1) : 16 * s + 4 * t;
            if (g < G) a = __ldcg(reinterpret_cast<const uint2*>(q0 + ch));
            if (g + 8 < G) b = __ldcg(reinterpret_cast<const uint2*>(q1 + ch));
            qf[s][0] = a.x; qf[s][1] = b.x; qf[s][2] = a.y; qf[s][3] = b.y;
        }
    }

    // row index (in units of cache rows) of the first key of the 16-key half-block starting at `key`
    auto half_block_row = [&](int key) -> int {
        const int pi = min(key >> page_shift, page_lo + n_pages - 1);
        int page;
        if (staged) {
            page = pages_s[pi - page_lo];
        } else {
            page = table[pi];
            if (page < 0 || page >= num_pages) {
                if (((pi + 1) << page_shift) > first) bad = 1;
                page = 0;
            }
        }
        return (page * nkv + kvh) * page_size + (key & page_mask);
    };

    struct Block {
        uint2 kf[KT][KS];
        uint32_t vf[KB][4][VW];
    };
    auto load_block = [&](int blk, Block& B) {
        const int base = k_begin + blk * BK;
        int hb[KB];
#pragma unroll
        for (int b = 0; b < KB; ++b) hb[b] = half_block_row(base + 16 * b);
#pragma unroll
        for (int j = 0; j < KT; ++j) {
            if constexpr (KS % 2 == 0) {
                const __nv_bfloat16* kp = kcache + (long long)(hb[j >> 1] + 8 * (j & 1) + g) * HD + 8 * t;
#pragma unroll
                for (int s2 = 0; s2 < KS / 2; ++s2) {
                    const uint4 v = kv_load16(kp + 32 * s2);
                    B.kf[j][2 * s2] = make_uint2(v.x, v.y);
                    B.kf[j][2 * s2 + 1] = make_uint2(v.z, v.w);
                }
            } else {
                const __nv_bfloat16* kp = kcache + (long long)(hb[j >> 1] + 8 * (j & 1) + g) * HD + 4 * t;
#pragma unroll
                for (int s = 0; s < KS; ++s) B.kf[j][s] = *reinterpret_cast<const uint2*>(kp + 16 * s);
            }
        }
#pragma unroll
        for (int b = 0; b < KB; ++b)
#pragma unroll
            for (int r = 0; r < 4; ++r)
                RowLoad<VW>::load(vcache + (long long)(hb[b] + 2 * t + (r & 1) + (r >> 1) * 8) * HD + NT * g, B.vf[b][r]);
    };
    auto compute_block = [&](int blk, Block& B) {
        const int base = k_begin + blk * BK;
        // ---- scores
        float s[KT][4];
#pragma unroll
        for (int j = 0; j < KT; ++j) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
                mma16816(s[j], qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3], B.kf[j][ks].x, B.kf[j][ks].y);
        }
        float mx[2] = {MMA_NEG_BIG, MMA_NEG_BIG};
#pragma unroll
        for (int j = 0; j < KT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = base + 8 * j + 2 * t + (e & 1);
                float v = s[j][e] * scale;
                if constexpr (SINK) {
                    if (cap > 0.f) v = gb_cap_fast(v, cap, inv_cap2);
                    if (a.r1 != nullptr) v -= sk_b1[e >> 1] * logf(fmaf(sk_b2[e >> 1], (float)max(pos - key, 0), 1.0f));
                }
                s[j][e] = (key < k_end && key >= first) ? v : MMA_NEG_BIG;
                mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
            }
        float corr[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
            const float m_new = fmaxf(m_run[h], mx[h]);
            corr[h] = __expf(m_run[h] - m_new);
            m_run[h] = m_new;
            l_run[h] *= corr[h];
        }
#pragma unroll
        for (int j = 0; j < KT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = base + 8 * j + 2 * t + (e & 1);
                const float p = (key < k_end && key >= first) ? __expf(s[j][e] - m_run[e >> 1]) : 0.f;
                s[j][e] = p;
                l_run[e >> 1] += p;   // this thread's share; summed over the lane group at the end
            }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            acc[j][0] *= corr[0]; acc[j][1] *= corr[0];
            acc[j][2] *= corr[1]; acc[j][3] *= corr[1];
        }
        // ---- output: P (registers) times V
#pragma unroll
        for (int b = 0; b < KB; ++b) {
            const uint32_t a0 = pack_bf16(s[2 * b][0], s[2 * b][1]), a1 = pack_bf16(s[2 * b][2], s[2 * b][3]);
            const uint32_t a2 = pack_bf16(s[2 * b + 1][0], s[2 * b + 1][1]), a3 = pack_bf16(s[2 * b + 1][2], s[2 * b + 1][3]);
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;   // high or low halves of the two rows' words
                const uint32_t b0 = __byte_perm(B.vf[b][0][j >> 1], B.vf[b][1][j >> 1], sel);
                const uint32_t b1 = __byte_perm(B.vf[b][2][j >> 1], B.vf[b][3][j >> 1], sel);
                mma16816(acc[j], a0, a1, a2, a3, b0, b1);
            }
        }
    };

    Block A, B;
    if (warp < nblocks) load_block(warp, A);
    for (int blk = warp; blk < nblocks; blk += 2 * NW) {
        if (blk + NW < nblocks) load_block(blk + NW, B);
        compute_block(blk, A);
        if (blk + 2 * NW < nblocks) load_block(blk + 2 * NW, A);
        if (blk + NW < nblocks) compute_block(blk + NW, B);
    }

    if (bad) atomicOr(status, GB_STATUS_BAD_SLOT);
    // ---- this warp's partial result
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
    }
    // What a block's warps found comes together in shared memory first, then what the splits found: the same sums in the same order in both
    // ways of merging, so that both give the same bits.
    constexpr int PITCH = HD + 2;                 // a result: HD channels, maximum, sum
    auto put = [&](float* to, int h) {            // this warp's result of its head g + 8 h
        if (t == 0) {
            to[HD] = m_run[h];
            to[HD + 1] = l_run[h];
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            to[NT * (2 * t) + j] = acc[j][2 * h];
            to[NT * (2 * t + 1) + j] = acc[j][2 * h + 1];
        }
    };
    // a head's channel over `parts` results `step` floats apart: its sum, their maximum and their sum (the weights formed by every thread)
    auto merge = [&](const float* pa, int parts, int step, int d, float top, float& m, float& l) {
        m = top;
        for (int i = 0; i < parts; ++i) m = fmaxf(m, pa[i * step + HD]);
        float v = 0.f;
        l = 0.f;
#pragma unroll 8
        for (int i = 0; i < parts; ++i) {
            const float w = __expf(pa[i * step + HD] - m);
            l = fmaf(pa[i * step + HD + 1], w, l);
            v = fmaf(pa[i * step + d], w, v);
        }
        return v;
    };
    // the head's result from its channel's sum v, the maximum m (the sink's logit sk among what it is of) and the sum l
    auto finish = [&](int hi, int d, float sk, float m, float l, float v) {
        if constexpr (SINK) l += __expf(sk - m);
        v *= (l > 0.f ? 1.0f / l : 0.f) * gate_factor(head0 + hi);
        orow[(head0 + hi) * HD + d] = __float2bfloat16_rn(SINK ? v * channel_gate(head0 + hi, d) : v);
    };
    if constexpr (CLUSTER) {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        float* first = cluster.map_shared_rank(cluster_part, 0) + (size_t)NW * G * PITCH;       // [split][head][HD channels, maximum, sum]
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (g + 8 * h < G) put(cluster_part + ((size_t)warp * G + g + 8 * h) * PITCH, h);
        auto last = [&](const float* pa, int parts, int i) {
            const int hi = i / HD, d = i % HD;
            const float sk = sink_logit(head0 + hi);
            float m, l;
            const float v = merge(pa + (size_t)hi * PITCH, parts, G * PITCH, d, sk, m, l);
            finish(hi, d, sk, m, l, v);
        };
        sync.group_barrier();
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        if (splits == 1) {
            for (int i = tid; i < G * HD; i += NTHREADS) last(cluster_part, NW, i);
            return;
        }
        for (int i = tid; i < G * HD; i += NTHREADS) {
            const int hi = i / HD, d = i % HD;
            float m, l;
            const float v = merge(cluster_part + (size_t)hi * PITCH, NW, G * PITCH, d, MMA_NEG_BIG, m, l);
            float* to = first + ((size_t)split * G + hi) * PITCH;
            to[d] = v;
            if (d == 0) {
                to[HD] = m;
                to[HD + 1] = l;
            }
        }
        cluster.sync();                       // (release / acquire: the first block sees what the others stored)
        if (cluster.block_rank() != 0) return;
        for (int i = tid; i < G * HD; i += NTHREADS) last(cluster_part + (size_t)NW * G * PITCH, splits, i);
        return;
    }
    // Through global memory: the block's results, as many heads at a time as the scratch holds, one for every split; the block that arrives
    // last merges them. With every warp's result stored, 48 of them for the last block to merge, 8 rows of 9/3 heads behind 4,000 keys took
    // 10.7 us with a lane a warp for the weights (sums in another order) and 11.1 with a lane a split, 10.4 so; a 135M step of them 751, 763
    // and 734, of 16 such rows 919, 927 and 902.
    constexpr int HEADS = MMA_SCRATCH / (NW * PITCH) < 16 ? MMA_SCRATCH / (NW * PITCH) : 16;
    static_assert(HEADS >= 1, "a head's results of all warps must fit the scratch");
    float* own = sm.scratch;                      // [warp][head of the pass][HD channels, maximum, sum], where the page ids were
    for (int h0 = 0; h0 < G; h0 += HEADS) {
        const int count = min(HEADS, G - h0);
        sync.group_barrier();                     // (the page ids, or the pass before, have been read)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int hi = g + 8 * h - h0;
            if (hi >= 0 && hi < count) put(own + (warp * count + hi) * PITCH, h);
        }
        sync.group_barrier();
        for (int i = tid; i < count * HD; i += NTHREADS) {
            const int hi = i / HD, d = i % HD;
            const float sk = splits == 1 ? sink_logit(head0 + h0 + hi) : MMA_NEG_BIG;
            float m, l;
            const float v = merge(own + hi * PITCH, NW, count * PITCH, d, sk, m, l);
            if (splits == 1) {
                finish(h0 + hi, d, sk, m, l, v);
                continue;
            }
            const size_t slot = ((size_t)row * nh + head0 + h0 + hi) * splits + split;
            part_acc[slot * HD + d] = v;
            if (d == 0) *reinterpret_cast<float2*>(part_ml + slot * 2) = make_float2(m, l);
        }
    }
    if (splits == 1) return;
    __threadfence();
    sync.group_barrier();
    if (tid == 0) {
        int* counter = counters + (size_t)row * nkv + kvh;
        const int prev = atomicAdd(counter, 1);
        is_last = (prev == splits - 1);
        if (is_last) *counter = 0;
    }
    sync.group_barrier();
    if (!is_last) return;
    __threadfence();
    for (int i = tid; i < G * HD; i += NTHREADS) {
        const int hi = i / HD, d = i % HD;
        const float* pa = part_acc + ((size_t)row * nh + head0 + hi) * splits * HD + d;
        const float2* ml = reinterpret_cast<const float2*>(part_ml) + ((size_t)row * nh + head0 + hi) * splits;
        const float sk = sink_logit(head0 + hi);
        float m = sk, l = 0.f, v = 0.f;
        if (splits <= 8) {                        // all asked for before the first is used: one trip to L2
            float2 p[8];
            float pv[8];
#pragma unroll
            for (int sp = 0; sp < 8; ++sp) {
                p[sp] = sp < splits ? __ldcg(ml + sp) : make_float2(MMA_NEG_BIG, 0.f);
                pv[sp] = sp < splits ? __ldcg(pa + (size_t)sp * HD) : 0.f;
            }
#pragma unroll
            for (int sp = 0; sp < 8; ++sp) m = fmaxf(m, p[sp].x);
#pragma unroll
            for (int sp = 0; sp < 8; ++sp)
                if (sp < splits) {
                    const float w = __expf(p[sp].x - m);
                    l = fmaf(p[sp].y, w, l);
                    v = fmaf(pv[sp], w, v);
                }
        } else {
#pragma unroll 8
            for (int sp = 0; sp < splits; ++sp) m = fmaxf(m, __ldcg(ml + sp).x);
#pragma unroll 8
            for (int sp = 0; sp < splits; ++sp) {
                const float2 p = __ldcg(ml + sp);
                const float w = __expf(p.x - m);
                l = fmaf(p.y, w, l);
                v = fmaf(__ldcg(pa + (size_t)sp * HD), w, v);
            }
        }
        finish(hi, d, sk, m, l, v);
    }
}
