// C[M, N] (+)= X[M, K] * W[N, K]^T for 9 to 64 rows against large matrices (decode batches), on the 5th-generation tensor cores
// with the operands the other way round: a tile is 128 rows of W (the M side of tcgen05.mma, always full) by all rows of X
// (the N side, 16 to 64), so that nothing is spent on padding, and K is split over the blocks of a cluster until the matrix's
// tiles fill the chip. Every weight is read once, by TMA, with up to 192 KB a multiprocessor in flight.
//
//   warp 0     producer: per 128 k two 64-column boxes of W (two of 64 rows, gate and up, when GATED) and two of X into a ring
//              of four stages. The first four stages' weights are asked for before the wait for the kernel before.
//   warp 1     tcgen05.mma (M 128, N 16..64, K 16) into 64 columns of tensor memory
//   warps 2-5  read the accumulator and leave it in shared memory by rows of X: [row][128 outputs], where the stages were
//   all warps  then, after a cluster barrier, block r of the cluster adds up rows r, r + split, ... over the blocks' partial
//              sums through distributed shared memory (in rank order: a fixed order) and runs the epilogue on whole rows: store,
//              add to the residual, squared ReLU, GELU, silu(gate) * up, or rotation and cache write of a stacked QKV product.
//
// Bound by the memory's latency at these sizes (3.5 to 5 TB/s; 67 MB gated, 40 rows, by ncu from a cold start: DRAM 36 % of its peak, tensor
// pipe 9 %, issue 10 %). Measured alone, weights from memory, us at 16 / 40 / 64 rows, this
// and in brackets the better of the weight-streaming and the tile kernel: 6144 x 2048 8.8 / 9.7 / 10.6 (8.8 / 13 / 13);
// 2048 x 2048 5.3 / 6.3 / 6.6 (5.7 / 9.0 / 14); 2 x 8192 x 2048 gated 17 / 21 / 25 (24 / 26 / 26); 2048 x 8192 10 / 12 / 12
// (16 / 33 / 35); 960 x 2560 5.0 / 5.5 / 6.2 (5.2 / 7.5 / 7.8). Below about 5 MB of weights it is no better: what is left is the
// cluster's start and its two barriers.
//
// Every wait on an mbarrier is bounded: on a timeout the block records GB_STATUS_WAIT_TIMEOUT and goes on to the cluster's
// barriers (which every thread of every block reaches), waits for its copies, frees its tensor memory and returns. No multicast.
#include "tcgen05.cuh"

constexpr int GF_BM = 128, GF_BK = 128, GF_ROWS = 64, GF_STAGES = 4, GF_THREADS = 192;
constexpr int GF_W_BYTES = GF_BM * GF_BK * 2, GF_X_BYTES = GF_ROWS * GF_BK * 2, GF_STAGE = GF_W_BYTES + GF_X_BYTES;
constexpr int GF_PITCH = GF_BM + 4;                      // floats from row to row of the partial sums
// k-blocks of a block's slice that are asked for into L2 before the wait: a slice of up to GF_WHOLE whole, of a longer one two past the ring
constexpr int GF_WHOLE = 12, GF_AHEAD = GF_STAGES + 2;
constexpr int GF_SMEM = GF_STAGES * GF_STAGE + 1024;
static_assert(GF_ROWS * GF_PITCH * 4 <= GF_STAGES * GF_STAGE, "the partial sums fit where the stages were");

enum { GF_STORE_BF16 = 0, GF_STORE_F32 = 1, GF_ADD_F32 = 2, GF_GLU_BF16 = 3, GF_ROPE_QKV = 4, GF_RELU2_BF16 = 5, GF_GELU_BF16 = 7 };

struct GfArgs {
    const __nv_bfloat16* w;       // the matrix that map_w describes, its rows ldw numbers apart (read only to ask for it early)
    long long w_rows, ldw;
    void* C;
    long long ldc;
    int mode, M, N, K, split, slice;      // slice: 128-wide k-blocks of a block
    int gate_rows, x_rows;                // x_rows: rows of a box of X, M rounded up to 16
    // rotation and cache write
    const float2* rope;
    const int* positions;
    const int* slots;
    __nv_bfloat16* kcache;
    __nv_bfloat16* vcache;
    int nh, nkv, hd, page_size, max_pos, write_kv;
    long long num_slots;
    int* status;
};

struct __align__(8) GfShared {
    uint64_t full[GF_STAGES], empty[GF_STAGES], tfull;
    uint32_t tmem_base;
    int abort_flag, issued, consumed;
};

__device__ __forceinline__ void gf_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 gf_peer_load(uint32_t addr, uint32_t rank) {      // 16 bytes of block `rank` of the cluster
    uint32_t peer;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer) : "memory");
    return v;
}

// (One block a multiprocessor, by its shared memory, and said so: without it the compiler keeps to 63 registers, and the merge of the
// splits loses its loads under way: 64 rows, N 1024, K 1024 4.6 -> 4.8 us.)
__global__ void __launch_bounds__(GF_THREADS, 1) gemm_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                              const GfArgs a) {
    extern __shared__ __align__(16) unsigned char gf_dyn[];
    unsigned char* stages = gf_dyn + ((1024u - (smem_u32(gf_dyn) & 1023u)) & 1023u);      // swizzled tiles: 1024-byte aligned
    float* part = reinterpret_cast<float*>(stages);                                       // [M][GF_PITCH], once the products are done
    __shared__ GfShared sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x / a.split, rank = blockIdx.x % a.split;
    const bool gated = a.mode == GF_GLU_BF16;
    const int n0 = tile * (gated ? 64 : GF_BM);
    const int kb_all = (a.K + GF_BK - 1) / GF_BK, kb0 = rank * a.slice, kblocks = min(kb_all - kb0, a.slice);
    const int x_bytes = a.x_rows * GF_BK * 2;

    if (tid == 0) {
        for (int s = 0; s < GF_STAGES; ++s) {
            mbar_init(&sh.full[s], 1);
            mbar_init(&sh.empty[s], 1);
        }
        mbar_init(&sh.tfull, 1);
        sh.abort_flag = sh.issued = sh.consumed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(64) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    volatile int* abort_flag = &sh.abort_flag;
    gb_pdl_launch_dependents();

    if (warp == 0) {
        if (elect_one()) {
            auto weights = [&](int it) {
                unsigned char* dst = stages + (it % GF_STAGES) * GF_STAGE;
                uint64_t* bar = &sh.full[it % GF_STAGES];
                mbar_expect_tx(bar, GF_W_BYTES + x_bytes);
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int k = (kb0 + it) * GF_BK + b * 64;
                    if (gated) {
                        tma_load_2d(dst + b * (GF_W_BYTES / 2), &map_w, bar, k, n0);
                        tma_load_2d(dst + b * (GF_W_BYTES / 2) + GF_W_BYTES / 4, &map_w, bar, k, a.gate_rows + n0);
                    } else {
                        tma_load_2d(dst + b * (GF_W_BYTES / 2), &map_w, bar, k, n0);
                    }
                }
            };
            auto rows = [&](int it) {
                unsigned char* dst = stages + (it % GF_STAGES) * GF_STAGE + GF_W_BYTES;
#pragma unroll
                for (int b = 0; b < 2; ++b)
                    tma_load_2d(dst + b * (GF_X_BYTES / 2), &map_x, &sh.full[it % GF_STAGES], (kb0 + it) * GF_BK + b * 64, 0);
            };
            const int first = min(kblocks, GF_STAGES);
            for (int it = 0; it < first; ++it) weights(it);      // (weights: no kernel of the step writes them)
            gb_pdl_wait();
            for (int it = 0; it < first; ++it) rows(it);
            sh.issued = first;
            for (int it = first; it < kblocks; ++it) {
                if (!mbar_wait(&sh.empty[it % GF_STAGES], ((it / GF_STAGES) - 1) & 1, abort_flag, a.status)) break;
                weights(it);
                rows(it);
                sh.issued = it + 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // (X, which the first barrier also waits for, is not requested before this: the limit of the bounded waits must not count
        // the time that the kernel before takes)
        gb_pdl_wait();
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(GF_BM, a.x_rows);
            const uint64_t w_desc = umma_desc(smem_u32(stages)), x_desc = umma_desc(smem_u32(stages) + GF_W_BYTES);
            int consumed = 0;
            bool ok = true;
            for (int it = 0; it < kblocks && ok; ++it) {
                const int s = it % GF_STAGES;
                if (!(ok = mbar_wait(&sh.full[s], (it / GF_STAGES) & 1, abort_flag, a.status))) break;
                consumed = it + 1;
                tc_fence_after();
                const uint64_t step = (uint64_t)((s * GF_STAGE) >> 4);
#pragma unroll
                for (int k = 0; k < GF_BK / 16; ++k)
                    umma_bf16(tmem, w_desc + step + (((k >> 2) * (GF_W_BYTES / 2) + (k & 3) * 32) >> 4),
                              x_desc + step + (((k >> 2) * (GF_X_BYTES / 2) + (k & 3) * 32) >> 4), idesc, (it | k) ? 1u : 0u);
                umma_commit(&sh.empty[s]);
            }
            if (ok) umma_commit(&sh.tfull);
            sh.consumed = consumed;
        }
    } else {
        // A row of the tile a thread: weights beyond the first stages' are asked for into L2 now, a row's part in one piece (the boxes take
        // 256 bytes of each of 128 rows at a time). Weights from memory, 40 rows, us: 2048 x 8192 (slices of 10) 9.9 -> 9.0, 6144 x 2048 8.9 ->
        // 8.4; a long slice whole runs ahead of the ring's own requests: 2 x 8192 x 2048 gated (16) 16.9 -> 18.2, two past the ring 16.7.
        const int r = (warp - 2) * 32 + lane, begin = (kb0 + GF_STAGES) * GF_BK, end = min(a.K, (kb0 + (kblocks <= GF_WHOLE ? kblocks : GF_AHEAD)) * GF_BK);
        const long long row = gated && r >= 64 ? a.gate_rows + n0 + r - 64 : n0 + r, rows = gated && r < 64 ? a.gate_rows : a.w_rows;
        const int bytes = (end - begin) * 2 / 16 * 16;
        if (row < rows && bytes > 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.w + row * a.ldw + begin), "r"(bytes) : "memory");
        gb_pdl_wait();
        const int q = warp & 3;                                   // the quarter of the tensor-memory lanes (outputs) of this warp
        if (mbar_wait_warp(&sh.tfull, 0, abort_flag, a.status)) {
            tc_fence_after();
            for (int c = 0; c < a.x_rows; c += 32) {              // (64 columns are allocated: reading past x_rows is harmless)
                uint32_t v[32];
                tmem_load32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c, v);
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (c + j < a.M) part[(c + j) * GF_PITCH + q * 32 + lane] = __uint_as_float(v[j]);
            }
        }
        tc_fence_before();
    }
    __syncwarp();
    gb_pdl_wait();
    gf_cluster_barrier();                                         // every block's partial sums are in place

    const int heads_total = a.nh + 2 * a.nkv;
    for (int row = rank + (int)warp * a.split; row < a.M; row += a.split * (GF_THREADS / 32)) {
        const uint32_t at = smem_u32(part + row * GF_PITCH + lane * 4);
        float4 s[8];
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (p < a.split) s[p] = gf_peer_load(at, (uint32_t)p);
        float v[4] = {s[0].x, s[0].y, s[0].z, s[0].w};
#pragma unroll
        for (int p = 1; p < 8; ++p)
            if (p < a.split) { v[0] += s[p].x; v[1] += s[p].y; v[2] += s[p].z; v[3] += s[p].w; }
        const int col = n0 + lane * 4;                            // (N is a multiple of 4: four columns are in or out together)
        if (a.mode == GF_STORE_F32 || a.mode == GF_ADD_F32) {
            if (col < a.N) {
                float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.C) + (size_t)row * a.ldc + col);
                float4 r = make_float4(v[0], v[1], v[2], v[3]);
                if (a.mode == GF_ADD_F32) {
                    const float4 o = *dst;
                    r = make_float4(o.x + r.x, o.y + r.y, o.z + r.z, o.w + r.w);
                }
                *dst = r;
            }
            continue;
        }
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.C) + (size_t)row * a.ldc + col;
        bool live = col < a.N;
        if (gated) {
            // lanes 0-15 hold four gate sums, lanes 16-31 the up sums of the same four outputs
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float up = __shfl_xor_sync(0xffffffffu, v[e], 16);
                v[e] = v[e] / (1.0f + __expf(-v[e])) * up;
            }
            live = lane < 16 && col < a.N;
        } else if (a.mode == GF_RELU2_BF16) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { v[e] = fmaxf(v[e], 0.f); v[e] *= v[e]; }
        } else if (a.mode == GF_GELU_BF16) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = gb_gelu_fast(v[e]);
        } else if (a.mode == GF_ROPE_QKV) {
            const int head = col / a.hd, ch = col % a.hd, half = a.hd / 2;      // a tile holds whole heads
            const int pos = a.positions[row];
            const bool is_q = head < a.nh, is_k = !is_q && head < a.nh + a.nkv;
            const bool bad_pos = a.rope != nullptr && pos >= a.max_pos;
            if (bad_pos && lane == 0) atomicOr(a.status, GB_STATUS_BAD_POSITION);
            float other[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) other[e] = __shfl_xor_sync(0xffffffffu, v[e], a.hd / 8);      // the channel half a head away
            if ((is_q || is_k) && a.rope != nullptr && pos >= 0 && !bad_pos) {
                const float4* cs = reinterpret_cast<const float4*>(a.rope + (size_t)pos * half + ch % half);
                const float4 c01 = cs[0], c23 = cs[1];
                const float co[4] = {c01.x, c01.z, c23.x, c23.z}, si[4] = {c01.y, c01.w, c23.y, c23.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = ch < half ? v[e] * co[e] - other[e] * si[e] : v[e] * co[e] + other[e] * si[e];
            }
            live = false;
            if (pos >= 0 && head < heads_total) {
                if (is_q) {
                    live = true;
                } else if (a.write_kv) {
                    const long long slot = a.slots[row];
                    if (slot < 0 || slot >= a.num_slots) {
                        atomicOr(a.status, GB_STATUS_BAD_SLOT);
                    } else {
                        const int kvh = is_k ? head - a.nh : head - a.nh - a.nkv;
                        dst = (is_k ? a.kcache : a.vcache) + (((slot / a.page_size) * a.nkv + kvh) * a.page_size + slot % a.page_size) * a.hd + ch;
                        live = true;
                    }
                }
            }
        }
        if (live)
            *reinterpret_cast<uint2*>(dst) = make_uint2(pack2(__float_as_uint(v[0]), __float_as_uint(v[1])), pack2(__float_as_uint(v[2]), __float_as_uint(v[3])));
    }

    gf_cluster_barrier();                                         // nobody leaves while a block reads its partial sums
    if (warp == 1) {
        if (lane == 0 && sh.abort_flag) {                         // copies that nobody consumed may still be in flight
            for (int it = sh.consumed; it < sh.issued; ++it) {
                const long long t0 = clock64();
                while (!mbar_try_wait(&sh.full[it % GF_STAGES], (it / GF_STAGES) & 1) && clock64() - t0 < TC_WAIT_CYCLES) {}
            }
        }
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(64) : "memory");
    }
}

// ------------------------------------------------------------------------------------------- host
// how many clusters of `size` blocks the chip holds at a time (a block has a multiprocessor to itself)
static int gf_clusters(int size) {
    static int most[9] = {0};
    if (most[size] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(148 / size * size);
        cfg.blockDim = dim3(GF_THREADS);
        cfg.dynamicSmemBytes = GF_SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_few_kernel, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = 1;
        }
        most[size] = n;
    }
    return most[size];
}

static int gf_launch(GfArgs a, const void* x, long long ldx, const void* w, long long w_rows, long long ldw, int tiles, int pdl, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GF_SMEM);
    GB_REQUIRE(e == cudaSuccess, "gb_gemm_few: %d bytes of shared memory refused: %s", GF_SMEM, cudaGetErrorString(e));
    // as many blocks for a tile's K as leave every tile a place on the chip, at least two k-blocks each
    const int kb = gb_ceil_div(a.K, GF_BK);
    a.split = 1;
    for (int s = 2; s <= 8; ++s)
        if (kb >= 2 * s && tiles <= gf_clusters(s)) a.split = s;
    a.slice = gb_ceil_div(kb, a.split);
    a.split = gb_ceil_div(kb, a.slice);                          // (no block without work)
    a.x_rows = (a.M + 15) / 16 * 16;
    a.w = (const __nv_bfloat16*)w;
    a.w_rows = w_rows;
    a.ldw = ldw;
    CUtensorMap mw, mx;
    if (tc_make_map_2d(&mw, w, w_rows, a.K, ldw, a.mode == GF_GLU_BF16 ? 64 : GF_BM, 64, "gb_gemm_few")) return 1;
    if (tc_make_map_2d(&mx, x, a.M, a.K, ldx, a.x_rows, 64, "gb_gemm_few")) return 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * a.split);
    cfg.blockDim = dim3(GF_THREADS);
    cfg.dynamicSmemBytes = GF_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = a.split;
    attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
    ++na;
    if (pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    e = cudaLaunchKernelEx(&cfg, gemm_few_kernel, mw, mx, a);
    GB_REQUIRE(e == cudaSuccess, "gb_gemm_few: launch failed: %s", cudaGetErrorString(e));
    return gb_check_launch("gb_gemm_few");
}

// 1 if the operands are what TMA and the epilogues need
GB_EXPORT int gb_gemm_few_supported(const void* x, const void* w, const void* c, int M, int N, int K, long long ldx, long long ldw, long long ldc) {
    return M > 0 && M <= GF_ROWS && N > 0 && N % 4 == 0 && K > 0 && K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 && ldx >= K && ldw >= K && ldc % 4 == 0 &&
           (((uintptr_t)x | (uintptr_t)w | (uintptr_t)c) & 15) == 0;
}

// mode: 0 store bfloat16, 1 store float32, 2 add into float32, 3 bfloat16(silu(gate) * up) (w: N gate rows, then N up rows),
// 5 bfloat16(max(c, 0)^2), 7 bfloat16(gelu(c)).
GB_EXPORT int gb_gemm_few(const void* x, long long ldx, const void* w, long long ldw, void* c, long long ldc, int mode, int M, int N, int K,
                          int* status, int pdl, cudaStream_t stream) {
    GB_REQUIRE(gb_gemm_few_supported(x, w, c, M, N, K, ldx, ldw, ldc) && ldc >= N && status != nullptr,
               "gb_gemm_few: %d rows (1..%d), N=%d, K=%d or their alignment are not built", M, GF_ROWS, N, K);
    GB_REQUIRE((mode >= 0 && mode <= 3) || mode == GF_RELU2_BF16 || mode == GF_GELU_BF16, "gb_gemm_few: bad mode %d", mode);
    GfArgs a = {};
    a.C = c; a.ldc = ldc; a.mode = mode; a.M = M; a.N = N; a.K = K; a.gate_rows = N; a.status = status; a.hd = 64;
    return gf_launch(a, x, ldx, w, mode == GF_GLU_BF16 ? 2ll * N : N, ldw, gb_ceil_div(N, mode == GF_GLU_BF16 ? 64 : GF_BM), pdl, stream);
}

// Stacked QKV projection with rotation and cache write (arguments as gb_gemm_tcgen05_qkv), head size 64 or 128.
GB_EXPORT int gb_gemm_few_qkv(const void* x, long long ldx, const void* w, long long ldw, void* q_out, long long ldq, int M, int K, const float* rope,
                              int max_pos, const int* positions, const int* slots, void* kcache, void* vcache, int nh, int nkv, int hd, int page_size,
                              long long num_pages, int write_kv, int* status, int pdl, cudaStream_t stream) {
    const int N = (nh + 2 * nkv) * hd;
    GB_REQUIRE((hd == 64 || hd == 128) && nh > 0 && nkv > 0 && page_size > 0, "gb_gemm_few_qkv: head size %d is not built (64, 128)", hd);
    GB_REQUIRE(gb_gemm_few_supported(x, w, q_out, M, N, K, ldx, ldw, ldq) && ldq >= (long long)nh * hd && positions && slots && status,
               "gb_gemm_few_qkv: %d rows (1..%d), N=%d, K=%d or their alignment are not built", M, GF_ROWS, N, K);
    GB_REQUIRE((((uintptr_t)kcache | (uintptr_t)vcache | (uintptr_t)rope) & 15) == 0, "gb_gemm_few_qkv: the cache and the table must be 16-byte aligned");
    GfArgs a = {};
    a.C = q_out; a.ldc = ldq; a.mode = GF_ROPE_QKV; a.M = M; a.N = N; a.K = K; a.status = status;
    a.rope = (const float2*)rope; a.positions = positions; a.slots = slots; a.kcache = (__nv_bfloat16*)kcache; a.vcache = (__nv_bfloat16*)vcache;
    a.nh = nh; a.nkv = nkv; a.hd = hd; a.page_size = page_size; a.max_pos = max_pos; a.write_kv = write_kv;
    a.num_slots = num_pages * page_size;
    return gf_launch(a, x, ldx, w, N, ldw, gb_ceil_div(N, GF_BM), pdl, stream);
}
