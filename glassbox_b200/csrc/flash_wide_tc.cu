// Flash attention for prompt portions whose values are wider than a head (sm_100a, tcgen05): the talking-heads attention, whose
// every query head is applied to the values of all key/value heads (up to 256 channels a block), and attention over a latent
// cache, whose keys are a latent and a rotated part (up to 192 numbers) and whose values are the latents themselves.
//
// One block = 128 consecutive rows of one request for one query head, over tiles of 128 keys. Tensor memory holds two score
// buffers of 128 columns and one accumulator of DV columns; the weights P_j take the place of the scores S_j they come from
// (bfloat16, 64 columns), so nothing else has to fit.
//   warp 0     producer of the query tile and of the keys: page by page through the request's block table, in 64-channel
//              column blocks of 128 rows x 128 bytes (128-byte swizzle; channels past the row are zero-filled)
//   warp 1     issues S_0, S_1, then in turn O += P_j V_j (as soon as P_j is written) and, when that is done, S_(j+2) into the
//              buffer that P_j leaves; meanwhile the softmax warps work on S_(j+1)
//   warps 2-9  softmax, two threads per row: a thread reads 64 of its row's 128 scores, caps and masks them, exchanges its
//              maximum with its partner, and writes its half of P_j. The running maximum is raised (and O rescaled) only when
//              exceeded by more than 2^8 in the exponent, as in attention_prefill_tc.cu.
//   warp 10    producer of the values (not for the latent cache, whose key tile serves both products); puts zeros in the place of
//              keys that no row of the block sees
// Bound by the chain of a tile (scores, the halves' maxima, weights, product, the next scores in the weights' place) in the one block
// that a multiprocessor holds, and by the longest row tiles: over a prompt of 2,048 tokens no unit is above a quarter of its peak
// (tensor pipe 19 %, special functions 16 %, FMA 22 %, issue 28 %; over a latent cache 35, 29, 11, 32). The mma.sync kernels that this replaced formed the scores once per 128 value
// channels and fed both products through ldmatrix. Measured: see gb_talking_attention_flash, gb_latent_flash.
//
// Every wait is bounded: on a timeout the block records GB_STATUS_WAIT_TIMEOUT, waits (bounded) for its copies, frees its tensor
// memory and returns. No multicast.
#include "tcgen05.cuh"

constexpr int FW_BM = 128, FW_BN = 128, FW_WARPS = 11;
constexpr float FW_NEG_BIG = -1.0e30f, FW_LOG2E = 1.4426950408889634f;
constexpr int FW_BLOCK = FW_BM * 128;        // bytes of a column block: 128 rows of 64 bfloat16

struct FwArgs {
    void* out;                 // LATENT: bfloat16 [n, H, DV]; else float32 [n, H, wide]
    const int* block_tables;
    int max_pages;
    const int* seq_first_row;
    const int* seq_start_pos;
    const float* sink;         // LATENT: a logit per head in the denominator, or nullptr
    int H, kv_heads, page_size, page_shift;
    long long num_pages;
    float scale, cap;          // cap > 0: cap * tanh(score / cap)
    int unit;                  // a key of score 0 without a value in the denominator
    int window, wide, vdim;    // channels of a row's output in all; of a value head
    int key_steps;             // 16-channel steps of a key row
    int col_blocks;            // blocks of DV channels that a row's output is cut into
    int merged;                // a page's values of all the block's heads come as one copy (see fw_values_merged)
    int* status;
};

struct __align__(8) FwShared {
    uint64_t q_full, k_full[3], k_empty[3], v_full[2], v_empty[2], s_full[2], p_ready[2], pv_done, o_done, x_bar[4], scored[2], cleared[2];
    float stat[2][2][FW_BM];   // [parity of the tile][half][row]: a half's maximum, at the end its sum
    uint32_t tmem_base;
    int abort_flag, issued[2], consumed[2], q_issued, q_consumed;
};

// KB: column blocks of a key row; DV: value channels of the block
template <int KB, int DV, bool LATENT> struct FwGeometry {
    static constexpr int K_STAGES = 3, V_STAGES = 2, K_BYTES = KB * FW_BLOCK, V_BYTES = LATENT ? 0 : (DV / 64) * FW_BLOCK;
    static constexpr int K_OFF = KB * FW_BLOCK, V_OFF = K_OFF + K_STAGES * K_BYTES, SH_OFF = V_OFF + V_STAGES * V_BYTES;
    static constexpr int SMEM = SH_OFF + (int)sizeof(FwShared) + 1024, O_COL = 2 * FW_BN;
    static_assert(O_COL + DV <= 512 && SMEM <= 227 * 1024, "the block does not fit");
};

__device__ __forceinline__ float fw_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// s <- tanh(s * in) for a warp's scores, as exactly as a call of tanhf (at most 1.1 units in the last place below 1, two beyond; NaN
// stays NaN). The tanh of y is y + y t c(t), t = y^2, with c the interpolation of (tanh(sqrt t) / sqrt t - 1) / t at Chebyshev nodes: of
// [0, 0.0625] for a warp whose scores all lie within a quarter of the cap (most do), of [0, 0.36] and [0, 1] otherwise, fused multiply-adds of two
// scores at a time and no special function. Where a score lies beyond the cap, 1 - 2 / (1 + e^(2|y|)).
__device__ __forceinline__ void fw_tanh(uint32_t (&s)[64], float in) {
    float tops[4] = {0.f, 0.f, 0.f, 0.f};
    const float2 in2 = make_float2(in, in);
#pragma unroll
    for (int k = 0; k < 64; k += 2) {
        const float2 y = __fmul2_rn(make_float2(__uint_as_float(s[k]), __uint_as_float(s[k + 1])), in2);
        s[k] = __float_as_uint(y.x);
        s[k + 1] = __float_as_uint(y.y);
        tops[(k >> 1) & 3] = fmaxf(fmaxf(tops[(k >> 1) & 3], fabsf(y.x)), fabsf(y.y));
    }
    const float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3]));
    auto both = [](float c) { return make_float2(c, c); };
    if (!__any_sync(0xffffffffu, top >= 0.25f)) {
#pragma unroll
        for (int k = 0; k < 64; k += 2) {
            const float2 y = make_float2(__uint_as_float(s[k]), __uint_as_float(s[k + 1])), t = __fmul2_rn(y, y);
            float2 w = __ffma2_rn(both(-0.051974945f), t, both(0.13328698f));
            w = __ffma2_rn(w, t, both(-0.33333316f));
            w = __ffma2_rn(y, __fmul2_rn(w, t), y);
            s[k] = __float_as_uint(w.x);
            s[k + 1] = __float_as_uint(w.y);
        }
        return;
    }
    if (!__any_sync(0xffffffffu, top >= 0.6f)) {
#pragma unroll
        for (int k = 0; k < 64; k += 2) {
            const float2 y = make_float2(__uint_as_float(s[k]), __uint_as_float(s[k + 1])), t = __fmul2_rn(y, y);
            float2 w = __ffma2_rn(both(-0.0062691197f), t, both(0.021110959f));
            w = __ffma2_rn(w, t, both(-0.05387395f));
            w = __ffma2_rn(w, t, both(0.13332915f));
            w = __ffma2_rn(w, t, both(-0.3333333135f));
            w = __ffma2_rn(y, __fmul2_rn(w, t), y);
            s[k] = __float_as_uint(w.x);
            s[k + 1] = __float_as_uint(w.y);
        }
        return;
    }
    const bool beyond = __any_sync(0xffffffffu, top >= 1.0f);
#pragma unroll
    for (int k = 0; k < 64; k += 2) {
        const float2 y = make_float2(__uint_as_float(s[k]), __uint_as_float(s[k + 1])), t = __fmul2_rn(y, y);
        float2 w = __ffma2_rn(both(-0.00042069549f), t, both(0.0025104594f));
        w = __ffma2_rn(w, t, both(-0.0082189217f));
        w = __ffma2_rn(w, t, both(0.021660116f));
        w = __ffma2_rn(w, t, both(-0.05393479f));
        w = __ffma2_rn(w, t, both(0.13333128f));
        w = __ffma2_rn(w, t, both(-0.3333333135f));
        w = __ffma2_rn(y, __fmul2_rn(w, t), y);
        if (beyond) {
            auto far = [](float v) { return copysignf(1.0f - __fdividef(2.0f, 1.0f + fw_exp2(fabsf(v) * (2.0f * FW_LOG2E))), v); };
            if (!(fabsf(y.x) < 1.0f)) w.x = far(y.x);
            if (!(fabsf(y.y) < 1.0f)) w.y = far(y.y);
        }
        s[k] = __float_as_uint(w.x);
        s[k + 1] = __float_as_uint(w.y);
    }
}
// MN-major B operand (rows are keys, 64-channel column blocks `block` bytes apart), 128-byte-swizzled rows
__device__ __forceinline__ uint64_t fw_desc_mn(uint32_t smem_addr, int block) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | (uint64_t)(block >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}
__device__ __forceinline__ void fw_tma_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

template <int KB, int DV, bool LATENT>
__global__ void __launch_bounds__(FW_WARPS * 32) flash_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                   const __grid_constant__ CUtensorMap map_v, const FwArgs a) {
    using G = FwGeometry<KB, DV, LATENT>;
    extern __shared__ __align__(16) unsigned char fw_dyn[];
    unsigned char* smem = fw_dyn + ((1024u - (smem_u32(fw_dyn) & 1023u)) & 1023u);        // swizzled tiles: 1024-byte aligned
    unsigned char* Qs = smem, *Ks = smem + G::K_OFF, *Vs = LATENT ? Ks : smem + G::V_OFF;
    FwShared& sh = *reinterpret_cast<FwShared*>(smem + G::SH_OFF);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // later tiles see more keys: the longest blocks start first (the row tile is the slowest dimension of the grid)
    const int qt = gridDim.z - 1 - blockIdx.z, head = blockIdx.x, seq = blockIdx.y / a.col_blocks, col0 = (blockIdx.y % a.col_blocks) * DV;
    const int row0 = a.seq_first_row[seq], nrows = a.seq_first_row[seq + 1] - row0, q_lo = qt * FW_BM;
    const int start_pos = a.seq_start_pos[seq];
    if (q_lo >= nrows) return;                                  // (uniform for the block, before anything is allocated)
    const int pos_lo = start_pos + q_lo, pos_hi = start_pos + min(nrows, q_lo + FW_BM) - 1;
    // the last position that decides whether the table reaches far enough: of the request (latent), of the tile
    const bool beyond = start_pos >= 0 && ((LATENT ? start_pos + nrows - 1 : pos_hi) >> a.page_shift) >= a.max_pages;
    if (beyond && tid == 0) atomicOr(a.status, GB_STATUS_BAD_POSITION);
    if (start_pos < 0 || beyond) {
        if (LATENT) {                                           // a padding sequence: its rows read as zeros downstream
            gb_pdl_launch_dependents();
            gb_pdl_wait();
            uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + ((size_t)(row0 + q_lo) * a.H + head) * DV);
            for (int i = tid; i < min(FW_BM, nrows - q_lo) * (DV / 8); i += FW_WARPS * 32)
                dst[(size_t)(i / (DV / 8)) * a.H * (DV / 8) + i % (DV / 8)] = make_uint4(0, 0, 0, 0);
        }
        return;
    }
    const int kvh = head / (a.H / a.kv_heads);
    const int key_lo = gb_first_key(pos_lo, a.window);
    const int kt_begin = key_lo / FW_BN, ntiles = pos_hi / FW_BN - kt_begin + 1;
    const int* table = a.block_tables + (size_t)seq * a.max_pages;
    // Where a key's values lie in a tile: column blocks of all 128 keys one behind the other, or (merged) a page's column blocks together
    const bool merged = !LATENT && a.merged;
    const int v_block = merged ? a.page_size * 128 : FW_BLOCK;
    auto value_at = [&](int block, int key) {
        return merged ? (key >> a.page_shift) * (DV / 64) * v_block + block * v_block + (key & (a.page_size - 1)) * 128 : block * FW_BLOCK + key * 128;
    };

    if (tid == 0) {
        mbar_init(&sh.q_full, 1);
        for (int i = 0; i < 3; ++i) { mbar_init(&sh.k_full[i], 1); mbar_init(&sh.k_empty[i], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.v_full[i], 1);
            mbar_init(&sh.v_empty[i], 1);
            mbar_init(&sh.s_full[i], 1);
            mbar_init(&sh.p_ready[i], 8);                       // one arrival per softmax warp
        }
        mbar_init(&sh.pv_done, 1);
        mbar_init(&sh.o_done, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&sh.scored[i], 1); mbar_init(&sh.cleared[i], 1); }
        for (int i = 0; i < 4; ++i) mbar_init(&sh.x_bar[i], 2);   // the two warps of a quarter of the rows
        sh.abort_flag = sh.issued[0] = sh.issued[1] = sh.consumed[0] = sh.consumed[1] = sh.q_issued = sh.q_consumed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
        if (!LATENT) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    volatile int* abort_flag = &sh.abort_flag;
    gb_pdl_launch_dependents();
    gb_pdl_wait();

    // Keys that no row of the block sees have a weight of 0, but what lies in their place in the pages (an earlier request's values,
    // or nothing yet) may be no finite number: zeros take its place before the product. Only the first and the last tile can hold
    // such keys. (The barriers of this exchange have one phase each.)
    const bool edge_first = key_lo % FW_BN != 0 || (ntiles == 1 && pos_hi % FW_BN != FW_BN - 1), edge_last = ntiles > 1 && pos_hi % FW_BN != FW_BN - 1;
    auto clear = [&](unsigned char* values, int j) {            // a warp's work: tile j, whose values have landed
        const int front = max(key_lo - (kt_begin + j) * FW_BN, 0), hi = pos_hi - (kt_begin + j) * FW_BN;
        const int keys = front + max(FW_BN - 1 - hi, 0);
        for (int i = lane; i < keys * (DV / 8); i += 32) {      // 16-byte pieces of a key's values, eight a column block
            const int k = i / (DV / 8), piece = i % (DV / 8), key = k < front ? k : hi + 1 + k - front;
            *reinterpret_cast<uint4*>(values + value_at(piece >> 3, key) + (piece & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.cleared[j == 0 ? 0 : 1]);
    };

    if (warp == 0 || (!LATENT && warp == FW_WARPS - 1)) {
        // ------------------------------------------------------------------------- producers
        const int what = warp == 0 ? 0 : 1;                     // keys, values
        if (what == 0 && lane == 0) {
            mbar_expect_tx(&sh.q_full, KB * FW_BLOCK);
            for (int c = 0; c < KB; ++c) fw_tma_3d(Qs + c * FW_BLOCK, &map_q, &sh.q_full, c * 64, head, row0 + q_lo);
            sh.q_issued = 1;
        }
        const int ppt = FW_BN >> a.page_shift;                  // pages per key tile (1 .. 16): a lane each
        const int boxes = what == 0 ? KB : DV / 64, stages = what == 0 ? G::K_STAGES : G::V_STAGES;
        const int bytes = boxes * FW_BLOCK;
        uint64_t* full = what == 0 ? sh.k_full : sh.v_full;
        uint64_t* empty = what == 0 ? sh.k_empty : sh.v_empty;
        unsigned char* ring = what == 0 ? Ks : Vs;
        int bad = 0;
        const int nowhere = (int)(a.num_pages * a.kv_heads * a.page_size);      // a row past the pool: the load fills in zeros
        constexpr int UNSEEN = (int)0x80000000;
        auto entry_of = [&](int kt) {                           // the table's entry of this lane's page of key tile kt
            int entry = UNSEEN;                                 // (no key of it is seen by any row)
            if (lane < ppt) {
                const int pi = ((kt * FW_BN) >> a.page_shift) + lane, first = pi << a.page_shift;
                if (first <= pos_hi && first + a.page_size > key_lo) entry = pi < a.max_pages ? table[pi] : -1;
            }
            return entry;
        };
        int entry = entry_of(kt_begin);
        int s = 0, round = 0;
        for (int j = 0; j < ntiles; ++j) {
            const int next_entry = j + 1 < ntiles ? entry_of(kt_begin + j + 1) : UNSEEN;   // in flight until the next tile
            int ok = 1;
            if (lane == 0 && round > 0) ok = mbar_wait(&empty[s], (round - 1) & 1, abort_flag, a.status) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&full[s], bytes);
            __syncwarp();
            if (lane < ppt) {
                const bool there = entry >= 0 && entry < a.num_pages;
                if (!there && entry != UNSEEN) bad = 1;
                unsigned char* dst = ring + s * bytes + lane * a.page_size * 128 * (what == 1 && merged ? boxes : 1);
                if (what == 1 && merged)
                    tma_load_2d(dst, &map_v, &full[s], 0, there ? (entry * a.kv_heads + col0 / 64) * a.page_size : nowhere);
                else for (int b = 0; b < boxes; ++b) {
                    if (what == 0) {
                        tma_load_2d(dst + b * FW_BLOCK, &map_k, &full[s], b * 64, there ? (entry * a.kv_heads + kvh) * a.page_size : nowhere);
                    } else {
                        const int col = col0 + b * 64;          // of the wide value row
                        tma_load_2d(dst + b * FW_BLOCK, &map_v, &full[s], col % a.vdim,
                                    there ? (entry * a.kv_heads + col / a.vdim) * a.page_size : nowhere);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) sh.issued[what] = j + 1;
            if (!LATENT && what == 1 && ((j == 0 && edge_first) || (j + 1 == ntiles && edge_last))) {
                if (!mbar_wait_warp(&full[s], round & 1, abort_flag, a.status)) break;
                clear(ring + s * bytes, j);
            }
            entry = next_entry;
            if (++s == stages) { s = 0; ++round; }
        }
        if (bad && what == 0) atomicOr(a.status, GB_STATUS_BAD_SLOT);
    } else if (warp == 1) {
        // ------------------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            const uint32_t idesc_qk = umma_idesc(FW_BM, FW_BN), idesc_pv = umma_idesc(FW_BM, DV) | (1u << 16);     // (B is MN-major)
            const uint64_t q_desc = umma_desc(smem_u32(Qs)), k_desc = umma_desc(smem_u32(Ks)), v_desc = fw_desc_mn(smem_u32(Vs), v_block);
            uint32_t v_step[FW_BN / 16];                        // where 16 keys' values start, in the descriptor's units
#pragma unroll
            for (int kk = 0; kk < FW_BN / 16; ++kk) v_step[kk] = (uint32_t)value_at(0, kk * 16) >> 4;
            bool ok = mbar_wait(&sh.q_full, 0, abort_flag, a.status);
            if (ok) sh.q_consumed = 1;
            auto scores = [&](int j) {
                const int s = j % G::K_STAGES;
                if (!mbar_wait(&sh.k_full[s], (j / G::K_STAGES) & 1, abort_flag, a.status)) return false;
                sh.consumed[0] = j + 1;
                tc_fence_after();
                const uint64_t kd = k_desc + (uint64_t)((s * G::K_BYTES) >> 4);
                for (int k = 0; k < a.key_steps; ++k) {
                    const uint64_t at = (uint64_t)(((k >> 2) * FW_BLOCK + (k & 3) * 32) >> 4);
                    umma_bf16(tmem + (uint32_t)((j & 1) * FW_BN), q_desc + at, kd + at, idesc_qk, k ? 1u : 0u);
                }
                umma_commit(&sh.s_full[j & 1]);
                if (!LATENT) umma_commit(&sh.k_empty[s]);
                if (LATENT && j == 0 && edge_first) umma_commit(&sh.scored[0]);
                if (LATENT && j + 1 == ntiles && edge_last) umma_commit(&sh.scored[1]);
                return true;
            };
            for (int j = 0; j < 2 && j < ntiles && ok; ++j) ok = scores(j);
            for (int j = 0; j < ntiles && ok; ++j) {
                const int s = LATENT ? j % G::K_STAGES : j % G::V_STAGES;
                if (!LATENT && !(ok = mbar_wait(&sh.v_full[s], (j / G::V_STAGES) & 1, abort_flag, a.status))) break;
                if (!LATENT) sh.consumed[1] = j + 1;
                if (j == 0 && edge_first && !(ok = mbar_wait(&sh.cleared[0], 0, abort_flag, a.status))) break;
                if (j + 1 == ntiles && edge_last && !(ok = mbar_wait(&sh.cleared[1], 0, abort_flag, a.status))) break;
                if (!(ok = mbar_wait(&sh.p_ready[j & 1], (j >> 1) & 1, abort_flag, a.status))) break;
                tc_fence_after();
                const uint64_t vd = v_desc + (uint64_t)((s * (LATENT ? G::K_BYTES : G::V_BYTES)) >> 4);
#pragma unroll
                for (int kk = 0; kk < FW_BN / 16; ++kk)         // 16 keys an instruction: 8 columns of P, 16 rows of the values
                    umma_bf16_ts(tmem + (uint32_t)G::O_COL, tmem + (uint32_t)((j & 1) * FW_BN + (kk >> 2) * 64 + (kk & 3) * 8), vd + v_step[kk], idesc_pv,
                                 (j | kk) ? 1u : 0u);
                umma_commit(&sh.pv_done);
                umma_commit(LATENT ? &sh.k_empty[s] : &sh.v_empty[s]);
                if (j + 1 == ntiles) umma_commit(&sh.o_done);   // (a commit covers everything this thread issued before it)
                // S_(j+2) goes where P_j is: only once the product that reads it is done
                if (j + 2 < ntiles) ok = mbar_wait(&sh.pv_done, j & 1, abort_flag, a.status) && scores(j + 2);
            }
        }
    } else if (warp < FW_WARPS - 1) {
        // ------------------------------------------------------------------------- softmax
        const int q = warp & 3, h = (warp - 2) >> 2;            // the quarter of the rows this warp may read; its half of the keys
        const int r = q * 32 + lane, pos = pos_lo + r;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        const float sl2 = a.scale * FW_LOG2E;                   // scores are brought into the base-2 domain
        const float cap2 = a.cap > 0.f ? a.cap * FW_LOG2E : 0.f, cap_in = a.cap > 0.f ? a.scale / a.cap : 0.f;
        const float slx = cap2 > 0.f ? cap2 : sl2;              // what is left to scale
        const int first = gb_first_key(pos, a.window), first_last = gb_first_key(pos_lo + FW_BM - 1, a.window);
        const bool bounded = a.cap > 0.f && a.cap <= 32.f && first_last == 0;      // (and every row sees a key of the first tile)
        float m_run = FW_NEG_BIG, l_run = 0.f;
        float down = 1.0f;          // weights and their sums are held at `down` times themselves
        bool ok = true;
        for (int j = 0; j < ntiles; ++j) {
            const int b = j & 1, key0 = (kt_begin + j) * FW_BN + h * 64;
            if (!mbar_wait_warp(&sh.s_full[b], (j >> 1) & 1, abort_flag, a.status)) { ok = false; break; }
            tc_fence_after();
            uint32_t sv[64];
            tmem_load64(lane_base + (uint32_t)(b * FW_BN + h * 64), sv);
            tc_fence_before();
            if (cap2 > 0.f) fw_tanh(sv, cap_in);                // (the cap itself is left to the scale)
            if (key0 + 63 > pos_lo || key0 < first_last) {      // the tile crosses the diagonal, the window's edge or the last key
#pragma unroll
                for (int k = 0; k < 64; ++k)
                    if (!(key0 + k <= pos && key0 + k >= first)) sv[k] = __float_as_uint(FW_NEG_BIG);
            }
            // Scores that a cap bounds: the first tile's maximum stays, or -16, and the two halves of a row go their own ways, one's caps
            // beside the other's exponentials. A weight may then grow to e^48: the row's weights are held at a power of two times
            // themselves, which changes no bit of them and lets none exceed 2^8, as none does where the maximum is followed. (Where the
            // first tile lies below -4 under a cap of 32, less: the sums have to hold the first tile's weights as well as the last one's.
            // Values from 1e-18 to 1e27 keep their precision whatever the scores do.)
            if (j == 0 || !bounded) {
                float mx4[4] = {FW_NEG_BIG, FW_NEG_BIG, FW_NEG_BIG, FW_NEG_BIG};
#pragma unroll
                for (int k = 0; k < 64; k += 8)
#pragma unroll
                    for (int u = 0; u < 4; ++u) asm("max.f32 %0, %0, %1, %2;" : "+f"(mx4[u]) : "f"(__uint_as_float(sv[k + 2 * u])), "f"(__uint_as_float(sv[k + 2 * u + 1])));
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                // the partner's maximum
                sh.stat[b][h][r] = mx;
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.x_bar[q]);
                if (!mbar_wait_warp(&sh.x_bar[q], j & 1, abort_flag, a.status)) { ok = false; break; }
                mx = fmaxf(mx, sh.stat[b][h ^ 1][r]);
                const bool raise = (mx - m_run) * slx > 8.0f;
                if (j == 0) {
                    if (raise) m_run = bounded ? fmaxf(mx, -16.0f / a.cap) : mx;      // nothing is accumulated yet (scores are in units of the cap)
                    if (!LATENT && bounded) down = __int_as_float((127 - (int)ceilf(fminf(fmaxf(cap2 - m_run * slx - 8.0f, 0.f), 44.f))) << 23);
                } else if (__any_sync(0xffffffffu, raise)) {
                    // (S_j was issued after O += P_(j-2) V_(j-2) was done: the phase of P_(j-1) V_(j-1) is the one to wait for)
                    if (!mbar_wait_warp(&sh.pv_done, (j - 1) & 1, abort_flag, a.status)) { ok = false; break; }
                    tc_fence_after();
                    const float corr = raise ? fw_exp2((m_run - mx) * slx) : 1.0f;
                    if (raise) m_run = mx;
                    l_run *= corr;
#pragma unroll 1
                    for (int c = 0; c < DV / 2; c += 32) {
                        uint32_t ov[32];
                        const uint32_t at = lane_base + (uint32_t)(G::O_COL + h * (DV / 2) + c);
                        tmem_load32(at, ov);
#pragma unroll
                        for (int k = 0; k < 32; ++k) ov[k] = __float_as_uint(__uint_as_float(ov[k]) * corr);
                        tmem_store32(at, ov);
                    }
                }
            }
            // a masked key holds -1e30 and comes out as exactly 0; a row that has seen no key yet must not cancel that
            const float msl = m_run <= FW_NEG_BIG ? 0.f : m_run * slx;
            const float2 scale2 = make_float2(slx, slx), off2 = make_float2(-msl, -msl);
            float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            uint32_t pw[32];
#pragma unroll
            for (int c = 0; c < 64; c += 2) {
                const float2 y = __ffma2_rn(make_float2(__uint_as_float(sv[c]), __uint_as_float(sv[c + 1])), scale2, off2);
                float2 pp = make_float2(fw_exp2(y.x), fw_exp2(y.y));
                if (!LATENT) pp = __fmul2_rn(pp, make_float2(down, down));
                // the denominator sums what the product uses: the weights as rounded to bfloat16
                const uint32_t both = pw[c >> 1] = pack2(__float_as_uint(pp.x), __float_as_uint(pp.y));
                l2[(c >> 1) & 1] = __fadd2_rn(l2[(c >> 1) & 1], make_float2(__uint_as_float(both << 16), __uint_as_float(both & 0xffff0000u)));
            }
            l_run += (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
            tmem_store32(lane_base + (uint32_t)(b * FW_BN + h * 64), pw);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.p_ready[b]);
        }
        if (ok) {                                               // the halves' sums
            const int turn = bounded ? 1 : ntiles;              // exchanges of the halves so far
            sh.stat[turn & 1][h][r] = l_run;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.x_bar[q]);
            ok = mbar_wait_warp(&sh.x_bar[q], turn & 1, abort_flag, a.status);
            // A barrier of its own, with one phase, says that all products are done: nothing orders this look against the last two
            // phases of pv_done, and a parity tells an open phase from its neighbours only (with both complete, the wait for the
            // last but one would take the next, open phase for it and never pass).
            ok = ok && mbar_wait_warp(&sh.o_done, 0, abort_flag, a.status);
        }
        if (ok) {
            tc_fence_after();
            const float up = 1.0f / down;                       // (a power of two)
            float l = (l_run + sh.stat[(bounded ? 1 : ntiles) & 1][h ^ 1][r]) * up, m2 = m_run <= FW_NEG_BIG ? FW_NEG_BIG : m_run * slx;
            float sink2 = FW_NEG_BIG;
            if (LATENT && a.sink != nullptr) sink2 = a.sink[head] * FW_LOG2E;
            if (a.unit) sink2 = 0.f;
            const float top = fmaxf(m2, sink2), corr = fw_exp2(m2 - top);
            l = l * corr + fw_exp2(sink2 - top);
            const float inv = l > 0.f ? corr / l * up : 0.f;
            // Rows turn over where the keys were (all products are done, nothing is on its way there): a store writes 128 bytes of four rows,
            // of bfloat16 64 of eight, and not 16 bytes in each of 32 (float32, 256 channels: 10,800 cycles a block, 2,600 so).
            uint4* stage = reinterpret_cast<uint4*>(Ks) + (warp - 2) * (32 * 8);
            const int live = min(32, nrows - q_lo - q * 32);
            const size_t row0w = (size_t)(row0 + q_lo + q * 32);
#pragma unroll 1
            for (int c = h * (DV / 2); c < (h + 1) * (DV / 2); c += 32) {
                uint32_t ov[32];
                tmem_load32(lane_base + (uint32_t)(G::O_COL + c), ov);
#pragma unroll
                for (int k = 0; k < 32; ++k) ov[k] = __float_as_uint(__uint_as_float(ov[k]) * inv);
                if (LATENT) {
                    tc_turn_put_bf16(stage, lane, ov);
                    __syncwarp();
                    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + (row0w * a.H + head) * a.wide + col0 + c + 8 * (lane & 3);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int rr = 8 * i + (lane >> 2);
                        if (rr < live) *reinterpret_cast<uint4*>(dst + (size_t)rr * a.H * a.wide) = tc_turn_get_bf16(stage, lane, i);
                    }
                } else {
                    tc_turn_put_f32(stage, lane, ov);
                    __syncwarp();
                    float* dst = reinterpret_cast<float*>(a.out) + (row0w * a.H + head) * a.wide + col0 + c + 4 * (lane & 7);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rr = 4 * i + (lane >> 3);
                        if (rr < live) *reinterpret_cast<float4*>(dst + (size_t)rr * a.H * a.wide) = tc_turn_get_f32(stage, lane, i);
                    }
                }
                __syncwarp();      // (the tile is read before it is written again; the next load is the whole warp's)
            }
        }
    } else if (LATENT) {
        // ------------------------------------------------------------------------- clears the ends of the walk
        // (the keys are the values: a tile is cleared once its scores have been formed)
        if (edge_first && mbar_wait_warp(&sh.scored[0], 0, abort_flag, a.status)) clear(Ks, 0);
        if (edge_last && mbar_wait_warp(&sh.scored[1], 0, abort_flag, a.status)) clear(Ks + (ntiles - 1) % G::K_STAGES * G::K_BYTES, ntiles - 1);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (lane == 0 && sh.abort_flag) {                       // copies that nobody consumed may still be in flight
            auto drain = [&](uint64_t* bar, uint32_t parity) {
                const long long t0 = clock64();
                while (!mbar_try_wait(bar, parity) && clock64() - t0 < TC_WAIT_CYCLES) {}
            };
            if (sh.q_issued && !sh.q_consumed) drain(&sh.q_full, 0);
            for (int it = sh.consumed[0]; it < sh.issued[0]; ++it) drain(&sh.k_full[it % G::K_STAGES], (it / G::K_STAGES) & 1);
            for (int it = sh.consumed[1]; it < sh.issued[1]; ++it) drain(&sh.v_full[it % G::V_STAGES], (it / G::V_STAGES) & 1);
        }
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ------------------------------------------------------------------------------------------- host
static int fw_map_q(CUtensorMap* map, const void* q, long long n, int H, int dim, const char* who) {
    TcEncodeTiledFn fn = tc_encode_fn();
    GB_REQUIRE(fn != nullptr, "%s: the driver does not offer cuTensorMapEncodeTiled", who);
    cuuint64_t dims[3] = {(cuuint64_t)dim, (cuuint64_t)H, (cuuint64_t)n};
    cuuint64_t strides[2] = {(cuuint64_t)dim * 2, (cuuint64_t)dim * H * 2};
    cuuint32_t box[3] = {64, 1, FW_BM}, one[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    GB_REQUIRE(r == CUDA_SUCCESS, "%s: cuTensorMapEncodeTiled failed with code %d", who, (int)r);
    return 0;
}

// Value heads of 64 lie one behind the other in a page: a block's heads come in one copy of up to 256 rows, where 16 keys of a product lie in
// one page. A copy a page and head (32 of 2 KB a tile of 256 channels and pages of 16) cost more than the tile's products: 2,048 tokens,
// 16/4 heads, pages of 16 / 32 / 64 / 128 tokens 56.9 / 50.8 / 47.9 / 47.8 us; with this and whole rows stored 41.2 at all of them.
static int fw_values_merged(int vdim, int dv, int page_size) { return vdim == 64 && page_size >= 16 && page_size * (dv / 64) <= 256; }

template <int KB, int DV, bool LATENT>
static int fw_launch(const void* q, const void* kcache, const void* vcache, int n, int dim, int num_seqs, int max_rows, const FwArgs& a,
                     cudaStream_t stream, const char* who) {
    using G = FwGeometry<KB, DV, LATENT>;
    CUtensorMap mq, mk, mv;
    if (fw_map_q(&mq, q, n, a.H, dim, who)) return 1;
    if (tc_make_map_2d(&mk, kcache, a.num_pages * a.kv_heads * a.page_size, dim, dim, a.page_size, 64, who)) return 1;
    if (LATENT) mv = mk;
    else if (tc_make_map_2d(&mv, vcache, a.num_pages * a.kv_heads * a.page_size, a.vdim, a.vdim, a.merged ? a.page_size * (DV / 64) : a.page_size, 64,
                            who)) return 1;
    auto kernel = flash_wide_kernel<KB, DV, LATENT>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
    GB_REQUIRE(e == cudaSuccess, "%s: %d bytes of shared memory refused: %s", who, G::SMEM, cudaGetErrorString(e));
    const int tiles = gb_ceil_div(max_rows, FW_BM);
    GB_REQUIRE(tiles <= 65535 && (long long)num_seqs * a.col_blocks <= 65535, "%s: bad batch shape", who);
    e = gb_launch(GB_PDL_ATTENTION, kernel, dim3(a.H, num_seqs * a.col_blocks, tiles), dim3(FW_WARPS * 32), G::SMEM, stream, mq, mk, mv, a);
    GB_REQUIRE(e == cudaSuccess, "%s: launch failed: %s", who, cudaGetErrorString(e));
    return gb_check_launch(who);
}

static int fw_page_shift(int page_size) {
    int shift = 0;
    while ((1 << shift) < page_size) ++shift;
    return shift;
}
static bool fw_pages_ok(int page_size) { return page_size >= 8 && page_size <= FW_BN && (page_size & (page_size - 1)) == 0; }

// Talking-heads attention of prompt portions: keys of 64 channels, value heads of 64 or 128, the values of all heads a whole
// number of 128-channel blocks.
GB_EXPORT int gb_talking_attention_flash_supported(int D, int V, int VG, int page_size) {
    return D == 64 && (V == 64 || V == 128) && VG > 0 && (VG * V) % 128 == 0 && fw_pages_ok(page_size);
}

// As gb_talking_attention_tiles (talking_attention.cu), VG == G. q bfloat16 [n, H, 64], out float32 [n, H, G * V].
// Measured, 2,048 tokens, 16/4 heads of 64, capped: 395 us in tiles of mma.sync, 37 us here.
GB_EXPORT int gb_talking_attention_flash(const void* q, float* out, const void* kcache, const void* vcache, const int* block_tables, int max_pages,
                                         const int* seq_first_row, const int* seq_start_pos, int n, int num_seqs, int max_rows_per_seq, int H, int G,
                                         int V, int page_size, long long num_pages, float scale, float cap, int unit, int window, int* status,
                                         cudaStream_t stream) {
    GB_REQUIRE(gb_talking_attention_flash_supported(64, V, G, page_size) && H > 0 && H % G == 0,
               "gb_talking_attention_flash: %d/%d heads, values of %d, pages of %d are not built", H, G, V, page_size);
    GB_REQUIRE((((uintptr_t)q | (uintptr_t)out | (uintptr_t)kcache | (uintptr_t)vcache) & 15) == 0, "gb_talking_attention_flash: operands must be 16-byte aligned");
    GB_REQUIRE(n >= 0 && num_seqs >= 0 && max_pages > 0 && num_pages * G * page_size < (1ll << 31), "gb_talking_attention_flash: bad batch shape");
    if (n == 0 || num_seqs == 0 || max_rows_per_seq <= 0) return 0;
    const int wide = G * V;
    FwArgs a = {out, block_tables, max_pages, seq_first_row, seq_start_pos, nullptr, H, G, page_size, fw_page_shift(page_size), num_pages, scale, cap,
                unit, window, wide, V, 4, 1, 0, status};
    if (wide % 256 == 0) {
        a.col_blocks = wide / 256;
        a.merged = fw_values_merged(V, 256, page_size);
        return fw_launch<1, 256, false>(q, kcache, vcache, n, 64, num_seqs, max_rows_per_seq, a, stream, "gb_talking_attention_flash");
    }
    a.col_blocks = wide / 128;
    a.merged = fw_values_merged(V, 128, page_size);
    return fw_launch<1, 128, false>(q, kcache, vcache, n, 64, num_seqs, max_rows_per_seq, a, stream, "gb_talking_attention_flash");
}

GB_EXPORT int gb_latent_flash_supported(int c, int r, int page_size) {
    return c == 128 && (r == 16 || r == 32 || r == 64) && fw_pages_ok(page_size);
}

// Attention of prompt portions over a latent cache [pages, page_size, 128 + r]: q bfloat16 [n, H, 128 + r], out bfloat16
// [n, H, 128]; arguments as gb_latent_attention_mma. Measured, two portions of 1,500 tokens in all
// behind up to 900, 32 heads, 128 + 64: 197 us in tiles of mma.sync, 60 us here.
GB_EXPORT int gb_latent_flash(const void* q, void* out, const void* cache, const int* block_tables, int max_pages, const int* seq_first_row,
                              const int* seq_start_pos, const float* sink, int n, int num_seqs, int max_rows_per_seq, int H, int c, int r,
                              int page_size, long long num_pages, float scale, int window, int* status, cudaStream_t stream) {
    GB_REQUIRE(gb_latent_flash_supported(c, r, page_size) && H > 0, "gb_latent_flash: latent %d, rotated part %d, pages of %d are not built", c, r, page_size);
    GB_REQUIRE((((uintptr_t)q | (uintptr_t)out | (uintptr_t)cache) & 15) == 0, "gb_latent_flash: operands must be 16-byte aligned");
    GB_REQUIRE(n >= 0 && num_seqs >= 0 && max_pages > 0 && num_pages * page_size < (1ll << 31), "gb_latent_flash: bad batch shape");
    if (n == 0 || num_seqs == 0 || max_rows_per_seq <= 0) return 0;
    FwArgs a = {out, block_tables, max_pages, seq_first_row, seq_start_pos, sink, H, 1, page_size, fw_page_shift(page_size), num_pages, scale, 0.f,
                0, window, 128, 128, (c + r) / 16, 1, 0, status};
    return fw_launch<3, 128, true>(q, cache, cache, n, c + r, num_seqs, max_rows_per_seq, a, stream, "gb_latent_flash");
}
