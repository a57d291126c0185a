// Grouped bf16 GEMM of a mixture of experts on CTA pairs (tcgen05 cta_group::2): for every work tile, up to 256 rows of A that
// belong to one expert, C[rows] = A[rows] * W[expert]^T.
//
// Operands are swapped, C^T = W * A^T: 256 weight rows are the pair's MMA rows (128 per CTA) and the tile's rows its 16..256
// columns, rounded up to 16 tile by tile. An expert with 13 rows so moves and multiplies 16 rows beside its weights and not 128,
// and one with 188 takes one pass over its weights with 192 columns and not two with 128 each; the pair halves what each CTA
// reads of A. Bound by the weights' bytes where experts have few rows, else by the reads of tiles from L2 and the MMAs.
//
// Qwen3-30B-A3B's experts (128 of 2048 x 768), 200 tokens, 8 experts each: gate / up 240 us and down 149 us with 128 x 128 tiles
// on single CTAs, 141 and 89 us like this, the launches before included (the weights alone: 123 and 62 us). 188 rows per expert:
// 178 and 113 us.
//
// Roles per CTA: warp 0 TMA producer; warp 1 MMA issuer (leader CTA); warps 2-5 epilogue (thread = one output feature). Every
// mbarrier wait is bounded; the cluster-wide barriers (start, end) are reached by every thread on every path.
#include "gemm_common.cuh"

namespace pie {
using namespace sm100;

constexpr int GG_STAGES = 6;
constexpr uint32_t GG_W_BYTES = GEMM_BM * GEMM_BK * 2;              // this CTA's 128 weight rows
constexpr uint32_t GG_X_BYTES = 128 * GEMM_BK * 2;                  // room for its half of up to 256 rows
constexpr uint32_t GG_STAGE_BYTES = GG_W_BYTES + GG_X_BYTES;
constexpr uint32_t GG_SMEM = GG_STAGES * GG_STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
constexpr uint32_t GG_TMEM_COLS = 512;                              // two accumulators of 256 columns

// Work tiles: tile_list[0] of them, entry 1 + i = (first 128-row tile << 9 | rows). Without a list each used 128-row tile is
// one, with all of its rows. Rows from tile max_mtiles on are left out: the list may be of a call with more, or of more routes than
// max_mtiles tiles hold, and A, C and tile_expert end there.
struct GroupedWork {
    const int *tile_expert, *tile_list;
    int max_mtiles;
};
struct GroupedTile {
    int row0, rows, expert;
};
__device__ __forceinline__ int grouped_count(const GroupedWork& w) { return w.tile_list ? min(w.tile_list[0], w.max_mtiles) : w.max_mtiles; }
__device__ __forceinline__ bool grouped_tile(const GroupedWork& w, int i, GroupedTile& t) {
    const int entry = w.tile_list ? w.tile_list[1 + i] : (i << 9 | GEMM_BM);
    const int tile = entry >> 9;
    t.row0 = tile * GEMM_BM;
    t.rows = min(entry & 511, (w.max_mtiles - tile) * GEMM_BM);
    t.expert = (unsigned)tile < (unsigned)w.max_mtiles ? w.tile_expert[tile] : -1;
    return t.expert >= 0;
}

// Boxes of 128 weight rows, and of 8, 16, 32, 64 and 128 rows of A.
struct GroupedMaps {
    CUtensorMap w, x[5];
};
// `rows` (a multiple of 8, up to 128) as one or two boxes (log2 of their rows / 8, -1 for none). A box of its own for every 8 rows
// cost more than the rows themselves: tiles of 48 tokens took longer than tiles of 64 (166 against 148 us for the
// gate / up products above). Rows past `rows` land in the slot and are not read.
__device__ __forceinline__ void grouped_boxes(int rows, int& first, int& second) {
    first = 31 - __clz(rows >> 3);
    const int rest = (rows >> 3) - (1 << first);
    second = rest == 0 ? -1 : 32 - __clz(rest - 1);
    if (second == first) {
        ++first;
        second = -1;
    }
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_grouped_kernel(const __grid_constant__ GroupedMaps maps, bf16* __restrict__ C, int N, int K, int ldc, int* status,
                    const GroupedWork work, const __grid_constant__ EpiArgs ex) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    uint8_t* ring_ptr = smem_raw + (ring - raw);
    const uint32_t bar0 = ring + GG_STAGES * GG_STAGE_BYTES;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (GG_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * GG_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * GG_STAGES + 2 + a); };   // the leader's is the one in use
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ring_ptr + GG_STAGES * GG_STAGE_BYTES + 8 * (2 * GG_STAGES + 4));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank();
    const bool leader = crank == 0;
    const int pid = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int tiles_n = (N + 2 * GEMM_BM - 1) / (2 * GEMM_BM), num_kb = (K + GEMM_BK - 1) / GEMM_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < GG_STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 8);   // 4 epilogue warps of each CTA
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) {
        tmem_alloc_2cta(smem_addr(const_cast<uint32_t*>(tmem_slot)), GG_TMEM_COLS);
        tmem_relinquish_2cta();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers exist before anyone signals across
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();
    pdl_wait();           // the work list is the producing kernels' too
    const int items = grouped_count(work) * tiles_n;

    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_desc(&maps.w);
            const uint32_t leader_full0 = map_to_cta(full_bar(0), 0);
            uint32_t it = 0;
            bool ok = true;
            for (int item = pid; item < items && ok; item += npairs) {
                GroupedTile t;
                if (!grouped_tile(work, item / tiles_n, t)) continue;
                const int half = (t.rows + 15) / 16 * 8;                     // rows of A in this CTA
                int b0, b1;
                grouped_boxes(half, b0, b1);
                const uint32_t bytes = GG_W_BYTES + (uint32_t)((8 << b0) + (b1 >= 0 ? 8 << b1 : 0)) * (GEMM_BK * 2);
                const int x_row = t.row0 + (int)crank * half, w_row = t.expert * N + item % tiles_n * 2 * GEMM_BM + (int)crank * GEMM_BM;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % GG_STAGES;
                    if (!mbar_wait_cluster(empty_bar(s), ((it / GG_STAGES) & 1u) ^ 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    // both CTAs' loads complete on the leader's barrier, armed for the pair's bytes
                    if (leader) mbar_arrive_expect_tx(full_bar(s), 2 * bytes);
                    const uint32_t lbar = leader_full0 + 8u * s, dst = ring + s * GG_STAGE_BYTES;
                    tma_load_2d_pair(dst, &maps.w, lbar, kb * GEMM_BK, w_row);
                    tma_load_2d_pair(dst + GG_W_BYTES, &maps.x[b0], lbar, kb * GEMM_BK, x_row);
                    if (b1 >= 0)
                        tma_load_2d_pair(dst + GG_W_BYTES + (8 << b0) * (GEMM_BK * 2), &maps.x[b1], lbar, kb * GEMM_BK, x_row + (8 << b0));
                }
            }
            // no copy may be in flight when the pair exits: the leader's barriers cover both CTAs
            if (leader) {
                const uint32_t first = it > (uint32_t)GG_STAGES ? it - GG_STAGES : 0u;
                for (uint32_t j = first; j < it; ++j)
                    mbar_wait_cluster(full_bar(j % GG_STAGES), (j / GG_STAGES) & 1u, status, PIE_ERR_WAIT_TMA, 200000000ll);
            }
        }
    } else if (warp == 1) {
        if (leader && elect_one()) {
            uint32_t it = 0, tcount = 0;
            bool ok = true;
            for (int item = pid; item < items && ok; item += npairs) {
                GroupedTile t;
                if (!grouped_tile(work, item / tiles_n, t)) continue;
                const uint32_t acc = tcount & 1u, aph = (tcount >> 1) & 1u;
                ++tcount;
                if (!mbar_wait_cluster(tempty_bar(acc), aph ^ 1u, status, PIE_ERR_WAIT_EPILOGUE)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + acc * 256, idesc = make_idesc_bf16(2 * GEMM_BM, (t.rows + 15) / 16 * 16);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % GG_STAGES;
                    if (!mbar_wait_cluster(full_bar(s), (it / GG_STAGES) & 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t wd = make_smem_desc_sw128(ring + s * GG_STAGE_BYTES);
                    const uint64_t xd = make_smem_desc_sw128(ring + s * GG_STAGE_BYTES + GG_W_BYTES);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k) umma_bf16_2cta(d, wd + 2u * k, xd + 2u * k, idesc, (kb | k) != 0);
                    umma_commit_2cta(empty_bar(s), 3);   // slot s is free in both CTAs
                }
                if (ok) umma_commit_2cta(tfull_bar(acc), 3);
            }
        }
    } else {
        const int q = warp & 3;
        const XieluCoef act(nullptr);
        const uint32_t leader_tempty0 = map_to_cta(tempty_bar(0), 0), leader_tempty1 = map_to_cta(tempty_bar(1), 0);
        uint32_t tcount = 0;
        for (int item = pid; item < items; item += npairs) {
            GroupedTile t;
            if (!grouped_tile(work, item / tiles_n, t)) continue;
            const uint32_t acc = tcount & 1u, aph = (tcount >> 1) & 1u;
            ++tcount;
            const bool got = mbar_wait_cluster(tfull_bar(acc), aph, status, PIE_ERR_WAIT_MMA);
            if (!__all_sync(0xffffffffu, got)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256;
            const int feat = item % tiles_n * 2 * GEMM_BM + (int)crank * GEMM_BM + q * 32 + lane;
            bf16* out = C + (size_t)t.row0 * ldc;
            for (int g = 0; g * 16 < t.rows; ++g) {
                uint32_t r[16];
                float v[16];
                tmem_ld_32x16(t_row + g * 16, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                skinny_store<EPI>(v, feat, g * 16, N, t.rows, out, ldc, nullptr, 0, ex, act);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (leader) mbar_arrive(tempty_bar(acc));
                else mbar_arrive_cluster(acc ? leader_tempty1 : leader_tempty0);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer may still read this CTA's shared memory / signal its barriers
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_2cta(tmem_base, GG_TMEM_COLS);
    }
}

}  // namespace pie

using namespace pie;

extern "C" int pie_make_tma_2d_bf16(CUtensorMap* map, const void* ptr, long rows, long cols, long ld, int box_rows);

template <int EPI>
static int launch_grouped(const GroupedMaps& maps, void* C, int N, int K, int ldc, int* status, int pairs,
                          const GroupedWork& work, const EpiArgs& ex, cudaStream_t st) {
    auto kern = gemm_grouped_kernel<EPI>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GG_SMEM);
    if (e != cudaSuccess) return (int)e;
    e = launch_pdl(kern, dim3(2 * pairs), dim3(GEMM_THREADS), GG_SMEM, st, maps, (bf16*)C, N, K, ldc, status, work, ex);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// A [max_mtiles*128, K] holds token rows sorted by expert in segments padded to 128-row tiles; W is [E, N, K] contiguous;
// tile_expert [max_mtiles] (device) gives each 128-row tile's expert or -1, tile_list [1 + max_mtiles] (device, may be null) the
// work tiles with their rows, as pie_moe_align writes them. C [max_mtiles*128, N] (or N/2 with a GLU epilogue); rows past a
// work tile's are left alone. Graph-safe: the launch shape depends only on max_mtiles.
static int grouped_gemm(const void* A, const void* W, void* C, const int* tile_expert, const int* tile_list, int max_mtiles,
                        int num_experts, int N, int K, int lda, int ldc, int epilogue, int* status, int num_sms, cudaStream_t st,
                        const EpiArgs& ex) {
    if (max_mtiles <= 0 || N <= 0 || num_experts <= 0) return 0;
    if (K <= 0 || K % 8 || N % 8 || ldc % 8) return (int)cudaErrorInvalidValue;
    if ((epilogue == EPI_SWIGLU || epilogue == EPI_CLAMP_GLU) && N % 32) return (int)cudaErrorInvalidValue;
    const long rows = (long)max_mtiles * GEMM_BM;
    GroupedMaps maps;
    if (pie_make_tma_2d_bf16(&maps.w, W, (long)num_experts * N, K, K, GEMM_BM) != 0) return (int)cudaErrorInvalidValue;
    for (int i = 0; i < 5; ++i)
        if (pie_make_tma_2d_bf16(&maps.x[i], A, rows, K, lda, 8 << i) != 0) return (int)cudaErrorInvalidValue;
    const long items = (long)max_mtiles * ((N + 2 * GEMM_BM - 1) / (2 * GEMM_BM));
    const int pairs = (int)(items < num_sms / 2 ? items : num_sms / 2);
    const GroupedWork work{tile_expert, tile_list, max_mtiles};
    switch (epilogue) {
        case EPI_STORE: return launch_grouped<EPI_STORE>(maps, C, N, K, ldc, status, pairs, work, ex, st);
        case EPI_SWIGLU: return launch_grouped<EPI_SWIGLU>(maps, C, N, K, ldc, status, pairs, work, ex, st);
        case EPI_CLAMP_GLU: return launch_grouped<EPI_CLAMP_GLU>(maps, C, N, K, ldc, status, pairs, work, ex, st);
        default: return (int)cudaErrorInvalidValue;
    }
}

PIE_API int pie_grouped_gemm_bf16(const void* A, const void* W, void* C, const int* tile_expert, const int* tile_list, int max_mtiles,
                                  int num_experts, int N, int K, int lda, int ldc, int epilogue, int* status,
                                  int num_sms, cudaStream_t st) {
    if (epilogue != EPI_STORE && epilogue != EPI_SWIGLU) return (int)cudaErrorInvalidValue;
    return grouped_gemm(A, W, C, tile_expert, tile_list, max_mtiles, num_experts, N, K, lda, ldc, epilogue, status, num_sms, st, EpiArgs());
}

// The clamped GLU of experts without biases in the epilogue: C [max_mtiles*128, N/2], see EPI_CLAMP_GLU.
PIE_API int pie_grouped_gemm_clamp_glu(const void* A, const void* W, void* C, const int* tile_expert, const int* tile_list, int max_mtiles,
                                       int num_experts, int N, int K, int lda, int ldc, float limit, int* status,
                                       int num_sms, cudaStream_t st) {
    EpiArgs ex;
    ex.limit = limit;
    return grouped_gemm(A, W, C, tile_expert, tile_list, max_mtiles, num_experts, N, K, lda, ldc, EPI_CLAMP_GLU, status, num_sms, st, ex);
}
