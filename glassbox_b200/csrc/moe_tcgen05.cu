// The experts' products of many rows on the 5th-generation tensor cores: the (row, choice) pairs sorted by expert (moe_sort in
// moe.cu), one persistent grouped product per half.
//
// A tile is 128 of an expert's pairs x BN of its outputs; a block (one per SM) walks the tiles of all experts in turn, an
// expert's tiles next to each other and its rows innermost, so that a piece of its matrix is read from memory once and from L2
// by the expert's other row tiles. Ten warps, as in the dense product (gemm_tcgen05.cu):
//   warp 0     producer: per 64-wide k-block a TMA box of the expert's matrix and the 128 input rows. DOWN, and UP where the rows
//              were gathered before (moe_gather_rows_kernel): the rows are the slots themselves, one box. UP otherwise: the rows of h
//              lie anywhere (sorted[slot] / top); every lane fetches four of them by TMA gather, straight into the swizzled tile.
//   warp 1     issues tcgen05.mma (M 128, N BN, K 16) into one of two accumulators in tensor memory
//   warps 2-9  epilogue, as in the dense product: UP stores bfloat16 relu(c)^2, or one gated unit of every two neighbouring
//              outputs; DOWN scatters float32 rows to pair[pair, :].
// Rows past an expert's last pair are loaded (another row's numbers) and never stored. A k-block takes 1.4 us with 32 gathers, 0.3 with
// a box of rows (the products 0.26), so a pass that brings the rows into slot order (16.8 MB: 4 us) pays from 64 pairs per expert
// on; with fewer a tile needs only a gather or two and the pass would cost its launch. Measured, 2,048 rows, 16 experts, four per
// token (1024 -> 2 x 1024 -> 1024): up half 101 us with gathers, 47 + 4 with the pass, 35 + 4 since the epilogue's units are told apart once
// (me_units); down half 38 -> 23 with the epilogue of eight warps and 16-byte stores. The up half's four rounds of tiles take 700 cycles a
// k-block of 48 KB where the products take 540, behind 7,000 of start. With few pairs per expert it is bound by reading every expert's matrices once.
//
// Every wait is bounded, as in the dense product: on a timeout the block records GB_STATUS_WAIT_TIMEOUT, waits (bounded) for its
// copies, frees its tensor memory and returns. No multicast.
#include "tcgen05.cuh"

constexpr int ME_BM = 128, ME_BK = 64, ME_EPI_WARPS = 8, ME_THREADS = 64 + 32 * ME_EPI_WARPS, ME_MAX_EXPERTS = 512, ME_MAX_STAGES = 8;

struct __align__(8) MeShared {
    uint64_t full[ME_MAX_STAGES], empty[ME_MAX_STAGES], tfull[2], tempty[2];
    uint32_t tmem_base;
    int abort_flag, issued, consumed;
    int row_tiles[ME_MAX_EXPERTS + 1];        // row tiles of the experts before each one
    int offset[ME_MAX_EXPERTS + 1];           // where each expert's slots start
};

template <int BN> struct MeGeometry {
    static constexpr int A_BYTES = ME_BM * ME_BK * 2, W_BYTES = BN * ME_BK * 2, STAGE_BYTES = A_BYTES + W_BYTES;
    static constexpr int STAGES = (192 * 1024 / STAGE_BYTES) < ME_MAX_STAGES ? (192 * 1024 / STAGE_BYTES) : ME_MAX_STAGES;
    static constexpr int SMEM = STAGES * STAGE_BYTES + ME_EPI_WARPS * 32 * 64 + 1024;      // (32 rows x 64 bytes per epilogue warp)
};

// four rows of the tensor map's matrix (box: one row of 64), 128 bytes each, one behind the other
__device__ __forceinline__ void me_gather4(void* dst, const CUtensorMap* map, uint64_t* bar, int col, int r0, int r1, int r2, int r3) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(col), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}

// Gated units with the numbers of gb_gated_unit: v holds 16 pairs of a gate sum and an up sum. Which unit it is is asked once for all of them:
// asked for every pair, in code unrolled over the pairs, the three kinds made an epilogue of 77 KB of instructions that came from
// memory for every tile (16,600 cycles a tile of 128 x 256 sums, whose products take 10,000).
__device__ __forceinline__ void me_units(const uint32_t (&v)[32], uint32_t* u, float limit, float slope) {
    if (slope > 0.f) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float g = fminf(__uint_as_float(v[2 * j]), limit), up = fminf(fmaxf(__uint_as_float(v[2 * j + 1]), -limit), limit);
            u[j] = __float_as_uint(gb_quotient(g, 1.0f + expf(-slope * g)) * (up + 1.0f));
        }
    } else if (slope < 0.f) {
#pragma unroll
        for (int j = 0; j < 16; ++j) u[j] = __float_as_uint(gb_gelu_tanh(__uint_as_float(v[2 * j])) * __uint_as_float(v[2 * j + 1]));
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float g = __uint_as_float(v[2 * j]);
            u[j] = __float_as_uint(gb_quotient(g, 1.0f + expf(-g)) * __uint_as_float(v[2 * j + 1]));
        }
    }
}

template <int BN, bool UP>
__global__ void __launch_bounds__(ME_THREADS) moe_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                                                                 const int* __restrict__ sorted, const int* __restrict__ offsets, int E,
                                                                 int top, int N, int K, void* __restrict__ C, long long ldc, int unit, int gather,
                                                                 float limit, float slope, int* __restrict__ status) {
    using G = MeGeometry<BN>;
    constexpr int STAGES = G::STAGES;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* tiles = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);      // swizzled tiles: 1024-byte aligned
    uint4* epi = reinterpret_cast<uint4*>(tiles + STAGES * G::STAGE_BYTES);
    __shared__ MeShared sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kblocks = (K + ME_BK - 1) / ME_BK;
    const int tiles_n = (N + BN - 1) / BN;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&sh.full[s], 1);
            mbar_init(&sh.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh.tfull[b], 1);
            mbar_init(&sh.tempty[b], ME_EPI_WARPS);
        }
        sh.abort_flag = sh.issued = sh.consumed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(2 * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    // every block adds up the experts' row tiles for itself (one warp, 32 experts a round)
    if (warp == 1) {
        int before = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            const int from = offsets[e < E ? e : E], to = offsets[e < E ? e + 1 : E];
            const int own = (to - from + ME_BM - 1) / ME_BM;
            int sum = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += v;
            }
            if (e < E) {
                sh.row_tiles[e] = before + sum - own;
                sh.offset[e] = from;
            }
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) {
            sh.row_tiles[E] = before;
            sh.offset[E] = offsets[E];
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    volatile int* abort_flag = &sh.abort_flag;
    const int ntiles = sh.row_tiles[E] * tiles_n;

    // a tile: its expert, its first slot, the end of the expert's slots, its first output
    struct Place { int e, m0, m_end, n0; };
    auto place = [&](int tile) {
        int lo = 0, hi = E;                                       // the expert: the last e whose tiles start at or before this one
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (sh.row_tiles[mid] * tiles_n <= tile) lo = mid; else hi = mid;
        }
        // (an expert without pairs shares its start with the next one; the last of equals is the one that has them)
        const int rows = sh.row_tiles[lo + 1] - sh.row_tiles[lo], t = tile - sh.row_tiles[lo] * tiles_n;
        return Place{lo, sh.offset[lo] + (t % rows) * ME_BM, sh.offset[lo + 1], (t / rows) * BN};
    };

    if (warp == 0) {
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
            const Place p = place(tile);
            // Groups of four rows that hold a pair; the rest of the tile keeps what was there, and its sums are not stored. A gather
            // costs as much as a box of 128 rows' share of the load unit: with all 32 for every tile, 24 rows of four of 16 experts
            // 2048 x 2048 took 150 us the feed-forward (mma.sync tiles before: 128), with the live ones 107.
            const int gathers = (min(ME_BM, p.m_end - p.m0) + 3) >> 2;
            int r[4];
            if (UP && gather) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int slot = p.m0 + 4 * lane + i;
                    r[i] = sorted[slot < p.m_end ? slot : p.m0] / top;        // (past the expert's pairs: any row that exists)
                }
            }
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int s = it % STAGES;
                if (it >= STAGES && !mbar_wait_warp(&sh.empty[s], ((it / STAGES) - 1) & 1, abort_flag, status)) { ok = false; break; }
                unsigned char* a_dst = tiles + s * G::STAGE_BYTES;
                if (lane == 0) {
                    mbar_expect_tx(&sh.full[s], UP && gather ? G::W_BYTES + gathers * 512 : G::STAGE_BYTES);
                    tma_load_2d(a_dst + G::A_BYTES, &map_w, &sh.full[s], kb * ME_BK, p.e * N + p.n0);
                    if (!UP || !gather) tma_load_2d(a_dst, &map_a, &sh.full[s], kb * ME_BK, p.m0);
                    sh.issued = it + 1;
                }
                __syncwarp();
                if (UP && gather && lane < gathers) me_gather4(a_dst + lane * 512, &map_a, &sh.full[s], kb * ME_BK, r[0], r[1], r[2], r[3]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(ME_BM, BN);
            const uint64_t a_desc = umma_desc(smem_u32(tiles)), w_desc = umma_desc(smem_u32(tiles) + G::A_BYTES);
            int s = 0, phase = 0, tcount = 0, consumed = 0;
            bool ok = true, ready = false;
            for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++tcount) {
                const int acc = tcount & 1;
                if (tcount >= 2 && !mbar_wait(&sh.tempty[acc], ((tcount >> 1) - 1) & 1, abort_flag, status)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem + (uint32_t)(acc * BN);
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!ready && !mbar_wait(&sh.full[s], phase, abort_flag, status)) { ok = false; break; }
                    ++consumed;
                    tc_fence_after();
                    const uint64_t step = (uint64_t)((s * G::STAGE_BYTES) >> 4);
                    uint64_t* done = &sh.empty[s];
                    if (++s == STAGES) { s = 0; phase ^= 1; }
#pragma unroll
                    for (int k = 0; k < ME_BK / 16; ++k)
                        umma_bf16(d_tmem, a_desc + step + k * 2, w_desc + step + k * 2, idesc, (kb | k) ? 1u : 0u);
                    umma_commit(done);
                    ready = mbar_test(&sh.full[s], phase);
                }
                if (ok) umma_commit(&sh.tfull[acc]);
            }
            sh.consumed = consumed;
        }
    } else {
        const int q = warp & 3;                                   // the quarter of the tensor-memory lanes this warp may read
        const int part = (warp - 2) >> 2;                         // ... and its half of the tile's columns
        uint4* stage = epi + (warp - 2) * (32 * 4);
        const bool vec_f32 = ((uintptr_t)C & 15) == 0 && (ldc & 3) == 0, vec_bf16 = ((uintptr_t)C & 15) == 0 && (ldc & 7) == 0;
        int tcount = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++tcount) {
            const Place p = place(tile);
            const int acc = tcount & 1, slot0 = p.m0 + q * 32;
            const int out_row = UP || slot0 + lane >= p.m_end ? -1 : sorted[slot0 + lane];
            const int rows = min(32, p.m_end - slot0);                        // (may be negative: no row of this warp is live)
            if (!mbar_wait_warp(&sh.tfull[acc], (tcount >> 1) & 1, abort_flag, status)) { ok = false; break; }
            tc_fence_after();
            const uint32_t t_base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN);
            // 32 outputs a turn: of a gated unit, 64 sums
            const int step = UP && unit ? 64 : 32;
#pragma unroll 1
            for (int c0 = part * (BN / 2); c0 < (part + 1) * (BN / 2); c0 += step) {
                if (p.n0 + c0 >= N || rows <= 0) break;                       // (uniform for the warp)
                uint32_t v[32];
                tmem_load32(t_base + (uint32_t)c0, v);
                if (UP) {
                    int col0 = p.n0 + c0, cols = N;
                    if (unit) {
                        // neighbouring outputs are the gate sum and the up sum of one unit
                        col0 >>= 1;
                        cols >>= 1;
                        // (32 units of a row are 64 bytes: two pieces of each half of the turned tile, as tc_turn_put_bf16 lays them)
#pragma unroll 1
                        for (int h = 0; h < 2; ++h) {
                            uint32_t u[16];
                            if (h) tmem_load32(t_base + (uint32_t)(c0 + 32), v);
                            me_units(v, u, limit, slope);
#pragma unroll
                            for (int c = 0; c < 2; ++c)
                                stage[lane * 4 + ((2 * h + c) ^ ((lane >> 1) & 3))] =
                                    make_uint4(pack2(u[8 * c], u[8 * c + 1]), pack2(u[8 * c + 2], u[8 * c + 3]), pack2(u[8 * c + 4], u[8 * c + 5]),
                                               pack2(u[8 * c + 6], u[8 * c + 7]));
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float g = fmaxf(__uint_as_float(v[j]), 0.f);
                            v[j] = __float_as_uint(g * g);
                        }
                        tc_turn_put_bf16(stage, lane, v);
                    }
                    __syncwarp();
                    const int col = col0 + 8 * (lane & 3);
                    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(C) + (size_t)slot0 * ldc + col;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int rr = 8 * i + (lane >> 2);
                        if (rr < rows) tc_store8_bf16(dst + (size_t)rr * ldc, tc_turn_get_bf16(stage, lane, i), col, cols, vec_bf16);
                    }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {                             // 16 columns, 64 bytes a row, at a time
                        if (h) __syncwarp();
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const int j = 16 * h + 4 * c;
                            stage[lane * 4 + (c ^ ((lane >> 1) & 3))] = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                        }
                        __syncwarp();
                        const int col = p.n0 + c0 + 16 * h + 4 * (lane & 3);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int rr = 8 * i + (lane >> 2), row = __shfl_sync(0xffffffffu, out_row, rr);
                            const uint4 w = tc_turn_get_bf16(stage, lane, i);
                            if (rr < rows)
                                tc_store4_f32(reinterpret_cast<float*>(C) + (size_t)row * ldc + col,
                                              make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)),
                                              col, N, vec_f32);
                        }
                    }
                }
                __syncwarp();      // the next load is the whole warp's; lanes of rows past the expert's last pair have taken another way here
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.tempty[acc]);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (lane == 0 && sh.abort_flag) {
            for (int it = sh.consumed; it < sh.issued; ++it) {                // copies that nobody consumed may still be in flight
                const long long t0 = clock64();
                while (!mbar_try_wait(&sh.full[it % STAGES], (it / STAGES) & 1) && clock64() - t0 < TC_WAIT_CYCLES) {}
            }
        }
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
    }
}

template <int BN, bool UP>
static int me_launch(const CUtensorMap& ma, const CUtensorMap& mw, const int* sorted, const int* offsets, int E, int top, int N, int K, void* c,
                     long long ldc, int unit, int gather, float limit, float slope, int* status, long long most_tiles, cudaStream_t stream) {
    auto kernel = moe_tcgen05_kernel<BN, UP>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MeGeometry<BN>::SMEM);
    GB_REQUIRE(e == cudaSuccess, "gb_moe_grouped_gemm: %d bytes of shared memory refused: %s", MeGeometry<BN>::SMEM, cudaGetErrorString(e));
    const int grid = most_tiles < 148 ? (int)most_tiles : 148;                // one block per SM walks the tiles
    e = gb_launch(GB_PDL_GEMM, kernel, dim3(grid), dim3(ME_THREADS), MeGeometry<BN>::SMEM, stream, ma, mw, sorted, offsets, E, top, N, K, c, ldc,
                  unit, gather, limit, slope, status);
    GB_REQUIRE(e == cudaSuccess, "gb_moe_grouped_gemm: launch failed: %s", cudaGetErrorString(e));
    return gb_check_launch("gb_moe_grouped_gemm");
}

// 1 if the grouped tensor-core products take these sizes (rows of 16-byte pieces)
GB_EXPORT int gb_moe_grouped_supported(int d, int ff) { return d % 8 == 0 && ff % 8 == 0 ? 1 : 0; }

// up: a = h [rows, K] (row stride lda), c bfloat16 [pairs, ldc] in slot order; otherwise a = the up half's output [pairs, K] and c
// float32 [pairs, ldc] in pair order. w: the experts' matrices [E * N, K]. sorted, offsets: as moe_sort leaves them.
// gather (up only): the rows of a slot are found through sorted; otherwise a [pairs, K] holds them in slot order.
GB_EXPORT int gb_moe_grouped_gemm(const void* a, long long lda, int rows, const void* w, int N, int K, const int* sorted, const int* offsets,
                                  int E, int top, int pairs, void* c, long long ldc, int up, int unit, float limit, float slope, int gather,
                                  int* status, cudaStream_t stream) {
    GB_REQUIRE(!unit || (up && N % 2 == 0), "gb_moe_grouped_gemm: the gated unit belongs to the up half and needs pairs of rows");
    GB_REQUIRE(N > 0 && K > 0 && K % 8 == 0 && lda % 8 == 0 && pairs >= 0 && E > 0 && E <= ME_MAX_EXPERTS && status != nullptr,
               "gb_moe_grouped_gemm: rows must be whole 16-byte pieces (K=%d), at most %d experts (%d)", K, ME_MAX_EXPERTS, E);
    GB_REQUIRE(((uintptr_t)a & 15) == 0 && ((uintptr_t)w & 15) == 0, "gb_moe_grouped_gemm: operands must be 16-byte aligned");
    GB_REQUIRE((long long)E * N <= 0x7fffffff, "gb_moe_grouped_gemm: too many rows of weights");
    if (pairs == 0) return 0;
    // The width whose rounds of tiles end soonest, as in the dense product (gemm_tcgen05.cu), with its epilogues' times. How many
    // row tiles there are is known on the device alone: every expert's last one is taken to be half full. Measured, microseconds
    // for widths 128 / 256: four of 16 experts 1024 -> 2 x 1024 -> 1024, 2,048 rows up 53.5 / 47.3, down 25.7 / 23.3; 512 rows up
    // 24.1 / 26.2; two of 16 experts 2048 -> 2 x 2048 -> 2048, 1,024 rows down 36.2 / 40.9, 2,048 rows up 105 / 86.
    const long long used = pairs < E ? pairs : E;
    const long long likely = pairs / ME_BM + used / 2, row_tiles = likely > used ? likely : used;
    const int kblocks = gb_ceil_div(K, ME_BK);
    const bool wide = tc_rounds_us(row_tiles * gb_ceil_div(N, 256), 148, kblocks, 256, up ? 3.2f : 4.2f) <=
                      tc_rounds_us(row_tiles * gb_ceil_div(N, 128), 148, kblocks, 128, up ? 1.6f : 2.4f);
    CUtensorMap ma, mw;
    if (tc_make_map_2d(&ma, a, rows, K, lda, up && gather ? 1 : ME_BM, ME_BK, "gb_moe_grouped_gemm")) return 1;
    if (tc_make_map_2d(&mw, w, (long long)E * N, K, K, wide ? 256 : 128, ME_BK, "gb_moe_grouped_gemm")) return 1;
#define ME_CASE(BN_, UP_) me_launch<BN_, UP_>(ma, mw, sorted, offsets, E, top, N, K, c, ldc, unit, gather, limit, slope, status, \
                                              (pairs / ME_BM + used) * gb_ceil_div(N, BN_), stream)
    if (up) return wide ? ME_CASE(256, true) : ME_CASE(128, true);
    return wide ? ME_CASE(256, false) : ME_CASE(128, false);
#undef ME_CASE
}

// Rows of h in the order of the slots: out[slot, :] = h[sorted[slot] / top, :], a warp per row, four of a lane's 16-byte pieces under way.
__global__ void __launch_bounds__(256) moe_gather_rows_kernel(const uint4* __restrict__ h, int pieces, const int* __restrict__ sorted,
                                                              const int* __restrict__ offsets, int E, int top, uint4* __restrict__ out) {
    gb_pdl_launch_dependents();
    gb_pdl_wait();
    const int slot = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (slot >= offsets[E]) return;
    const uint4* src = h + (size_t)(sorted[slot] / top) * pieces;
    uint4* dst = out + (size_t)slot * pieces;
    for (int i0 = lane; i0 < pieces; i0 += 128) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + 32 * u < pieces) v[u] = src[i0 + 32 * u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + 32 * u < pieces) dst[i0 + 32 * u] = v[u];
    }
}

// h bfloat16 [rows, K] and out bfloat16 [pairs, K], both contiguous and 16-byte aligned; sorted, offsets: as moe_sort leaves them.
GB_EXPORT int gb_moe_gather_rows(const void* h, int K, const int* sorted, const int* offsets, int E, int top, int pairs, void* out,
                                 cudaStream_t stream) {
    GB_REQUIRE(K > 0 && K % 8 == 0 && (((uintptr_t)h | (uintptr_t)out) & 15) == 0 && E > 0 && top > 0 && pairs >= 0,
               "gb_moe_gather_rows: rows must be whole 16-byte pieces (K=%d)", K);
    if (pairs == 0) return 0;
    gb_launch(GB_PDL_ELEMENTWISE, moe_gather_rows_kernel, dim3(gb_ceil_div(pairs, 8)), dim3(256), 0, stream, (const uint4*)h, K / 8, sorted,
              offsets, E, top, (uint4*)out);
    return gb_check_launch("gb_moe_gather_rows");
}
