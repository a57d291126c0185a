// bf16 GEMM on CTA pairs (tcgen05 cta_group::2):  C[M,N] = A[M,K] * W[N,K]^T, 256 x bn per pair.
//
// Two CTAs of a 2-CTA cluster share one output tile. Each CTA TMA-loads its own 128 rows of A
// and its own half of the W tile (bn/2 rows) into its shared memory (plain per-CTA loads, no
// multicast); the leader CTA issues tcgen05.mma.cta_group::2, which reads both CTAs' shared
// memory and accumulates 128 rows in each CTA's TMEM. Compared with the single-CTA kernel this
// halves the shared-memory fill per flop (the measured limit of that kernel) and leaves room
// for a deeper TMA ring.
//
// Roles per CTA: warp 0 TMA producer; warp 1 MMA issuer (leader); warps 2-5 epilogue of the CTA's
// own 128 rows. Both CTAs' loads complete on the leader's barriers; tcgen05.commit signals the
// ring-slot and accumulator barriers of both CTAs. Same epilogues and tensor-parallel hooks as
// gemm_tcgen05.cu; every wait on an mbarrier is bounded. The two cluster-wide barriers (start, end)
// are reached by every thread on every path.
//
// Tiles are whole in K and as wide as makes the rounds of the machine short (plan_pairs), where K used to be split over pairs with the
// parts parked in global memory: no workspace, one order of sums. (Walking the tiles in bands of row blocks, for operands that L2 holds
// together, measured no faster.) Weights cold, before and now (us): 512 x 4096 x 14336 80 and 53, 512 x 4096 x 4096 26.4 (on single CTAs)
// and 18.5, 200 x 2048 x 4096 23.4 and 13.5, 1536 x 4096 x 14336 201 and 137, 3661 x 4096 x 4096 129 and 103; 8300 x 28672 x 4096 1.45 ms
// either way: 1.3 PFLOP/s, what the power limit allows.
#include <algorithm>

#include "gemm_common.cuh"

namespace pie {
using namespace sm100;

constexpr int PAIR_M = 2 * GEMM_BM;
constexpr uint32_t PAIR_A_BYTES = GEMM_BM * GEMM_BK * 2;       // a CTA's 128 rows of a k-block
constexpr uint32_t PAIR_RING = 192 * 1024;
constexpr int PAIR_MAX_STAGES = 8;
constexpr uint32_t PAIR_TMEM_COLS = 512;                       // two accumulators of up to 256 columns
constexpr uint32_t PAIR_SMEM = PAIR_RING + 1024 /*align*/ + 512 /*barriers*/ + 16384 /*epilogue staging*/;

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                  bf16* __restrict__ C, const bf16* __restrict__ R, int M, int N, int K, int ldc, int ldr,
                  int* status, const __grid_constant__ TpArgs tp, int bn, int stages, const __grid_constant__ EpiArgs ex) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    uint8_t* ring_ptr = smem_raw + (ring - raw);
    const uint32_t bar0 = ring + PAIR_RING;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (PAIR_MAX_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * PAIR_MAX_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * PAIR_MAX_STAGES + 2 + a); };  // leader's is the one in use
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ring_ptr + PAIR_RING + 8 * (2 * PAIR_MAX_STAGES + 4));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank();
    const bool leader = crank == 0;
    const int pid = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const uint32_t stage_bytes = PAIR_A_BYTES + (uint32_t)bn * GEMM_BK;        // bn / 2 rows of 128 bytes
    const int tiles_m = (M + PAIR_M - 1) / PAIR_M, tiles_n = (N + bn - 1) / bn, num_tiles = tiles_m * tiles_n;
    const int num_kb = (K + GEMM_BK - 1) / GEMM_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
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
        tmem_alloc_2cta(smem_addr(const_cast<uint32_t*>(tmem_slot)), PAIR_TMEM_COLS);
        tmem_relinquish_2cta();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers exist before anyone signals across
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();

    if (warp == 0) {
        // ------------------------------------------------------ TMA producer (each CTA)
        if (elect_one()) {
            tma_prefetch_desc(&tma_a);
            tma_prefetch_desc(&tma_b);
            bool ok = true;
            uint32_t seen = 0, it = 0, ph = 0;
            int s = 0;
            const uint32_t leader_full0 = map_to_cta(full_bar(0), 0);
            pdl_wait();
            for (int tile = pid; tile < num_tiles && ok; tile += npairs) {
                const int m_blk = tile % tiles_m, n_blk = tile / tiles_m;
                const int a_row = m_blk * PAIR_M + (int)crank * GEMM_BM, b_row = n_blk * bn + (int)crank * (bn / 2);
                if (tp.gated && !ag_gate_wait_rows(tp, status, a_row, GEMM_BM, seen)) break;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    if (!mbar_wait_cluster(empty_bar(s), ph ^ 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    // both CTAs' loads complete on the leader's barrier, armed for the pair's bytes
                    if (leader) mbar_arrive_expect_tx(full_bar(s), 2 * stage_bytes);
                    const uint32_t dst = ring + s * stage_bytes, lbar = leader_full0 + 8u * s;
                    tma_load_2d_pair(dst, &tma_a, lbar, kb * GEMM_BK, a_row);
                    tma_load_2d_pair(dst + PAIR_A_BYTES, &tma_b, lbar, kb * GEMM_BK, b_row);
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
            }
            // no copy into this CTA may be in flight when it exits: the leader's barriers cover the pair, and both CTAs meet at the
            // cluster barrier below
            if (leader) {
                const uint32_t first = it > (uint32_t)stages ? it - stages : 0u;
                for (uint32_t j = first; j < it; ++j)
                    mbar_wait_cluster(full_bar(j % stages), (j / stages) & 1u, status, PIE_ERR_WAIT_TMA, 200000000ll);
            }
        }
    } else if (warp == 1) {
        if (leader && elect_one()) {
            // ---------------------------------------------------- leader: MMA issuer of the pair
            const uint32_t idesc = make_idesc_bf16(PAIR_M, bn);
            uint32_t ph = 0, tcount = 0;
            int s = 0;
            bool ok = true;
            for (int tile = pid; tile < num_tiles && ok; tile += npairs, ++tcount) {
                const uint32_t acc = tcount & 1u, aph = (tcount >> 1) & 1u;
                if (!mbar_wait_cluster(tempty_bar(acc), aph ^ 1u, status, PIE_ERR_WAIT_EPILOGUE)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * 256;
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!mbar_wait_cluster(full_bar(s), ph, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = ring + s * stage_bytes;
                    const uint64_t adesc = make_smem_desc_sw128(a_addr);
                    const uint64_t bdesc = make_smem_desc_sw128(a_addr + PAIR_A_BYTES);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k)
                        umma_bf16_2cta(d_tmem, adesc + 2u * k, bdesc + 2u * k, idesc, (kb | k) != 0);
                    umma_commit_2cta(empty_bar(s), 3);   // slot s is free in both CTAs
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit_2cta(tfull_bar(acc), 3);
            }
        }
    } else {
        // ----------------------------------------------------------- epilogue (own 128 rows)
        const int q = warp & 3, chunks = (bn + 63) / 64;
        uint8_t* stage = ring_ptr + PAIR_RING + 512 + (warp - 2) * 4096;
        pdl_wait();          // outputs and residual may still be in use by the previous kernel
        const XieluCoef act(EPI == EPI_XIELU ? ex.act : nullptr);
        const uint32_t leader_tempty0 = map_to_cta(tempty_bar(0), 0);
        const uint32_t leader_tempty1 = map_to_cta(tempty_bar(1), 0);
        uint32_t tcount = 0;
        for (int tile = pid; tile < num_tiles; tile += npairs, ++tcount) {
            const int m_blk = tile % tiles_m, n_blk = tile / tiles_m;
            const uint32_t acc = tcount & 1u, aph = (tcount >> 1) & 1u;
            const bool got = mbar_wait_cluster(tfull_bar(acc), aph, status, PIE_ERR_WAIT_MMA);
            if (!__all_sync(0xffffffffu, got)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256;
            const int row0 = m_blk * PAIR_M + (int)crank * GEMM_BM + q * 32, col0 = n_blk * bn, n_end = min(N, col0 + bn);
#pragma unroll 1
            for (int c = 0; c < chunks; ++c) {
                uint32_t v0[32], v1[32];
                tmem_ld_32x32(t_row + c * 64, v0);
                tmem_ld_32x32(t_row + c * 64 + 32, v1);
                tmem_ld_wait();
                epilogue_store_64<EPI>(v0, v1, stage, row0, col0 + c * 64, M, N, C, ldc, R, ldr, tp, n_end, ex, &act);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (leader) mbar_arrive(tempty_bar(acc));
                else mbar_arrive_cluster(acc ? leader_tempty1 : leader_tempty0);
            }
            if (EPI == EPI_RS) {
                __threadfence_system();
                __syncwarp();
                if (lane == 0) rs_publish_arrival(tp, num_tiles * 8);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer may still read this CTA's shared memory / signal its barriers
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_2cta(tmem_base, PAIR_TMEM_COLS);
    }
}

}  // namespace pie

using namespace pie;

extern "C" int pie_make_tma_2d_bf16(CUtensorMap* map, const void* ptr, long rows, long cols, long ld, int box_rows);

// Tuning aid: tile width of every following launch of more than 128 rows (0: as planned; -1: pairs with the planned width, also where
// the other kernel would be chosen).
static int g_pair_bn = 0;
extern "C" __attribute__((visibility("default"))) int pie_gemm_set_pair_width(int bn) {
    if (bn < -1 || bn > 256 || (bn > 0 && (bn < 64 || bn % 16))) return (int)cudaErrorInvalidValue;
    g_pair_bn = bn;
    return 0;
}

// Width of the tiles: the one whose rounds of the machine take the least time together. A k-block of a tile takes a time that grows with
// bn + 62 (the 256 rows of A are there whatever the width), a round 500 such units and the last tile's epilogue 10 bn: within 1.5 % of
// the best of eleven widths over 96 shapes of 200 to 3661 rows. False where single CTAs are the faster ones (us, pairs against single
// CTAs, weights cold):
//   few tiles of a long K, which single CTAs split: 200 x 1024 x 4096 12.9 / 11.7, but 320 x 1024 x 4096 (32 tiles) 12.9 / 14.1
//   two to four tiles of a short K: 200 x 128 x 512 4.5 / 4.1
//   257 to 384 rows, whose pairs' tiles are up to half empty: 300 x 12352 x 4096 41.7 / 36.0, 320 x 9216 x 512 8.8 / 7.8, but
//     300 x 4096 x 4096 17.6 / 19.8 and 300 x 5120 x 25600 98 / 134
//   one row of tiles, and more than one round of them: 200 x 28672 x 4096 83 / 67, but 200 x 18432 x 4096 (one round) 33 / 37
static bool plan_pairs(int M, int N, int K, int pairs_max, int& width, int& pairs) {
    if (M <= GEMM_BM || N < 128) return false;
    const long num_kb = (K + GEMM_BK - 1) / GEMM_BK, tiles_m = (M + PAIR_M - 1) / PAIR_M;
    long best = -1, rounds = 0;
    for (int bn = 256; bn >= 64; bn -= 16) {
        if (g_pair_bn > 0 && bn != g_pair_bn) continue;
        const long tiles = tiles_m * ((N + bn - 1) / bn), r = (tiles + pairs_max - 1) / pairs_max;
        const long cost = r * (num_kb * (bn + 62) + 500) + 10 * bn;
        if (best >= 0 && cost >= best) continue;
        best = cost;
        rounds = r;
        width = bn;
        pairs = (int)std::min<long>(pairs_max, tiles);
    }
    if (g_pair_bn) return true;
    const long low = tiles_m * ((N + 63) / 64);            // tiles of the least width
    if ((K >= 4096 && low <= 16) || (K <= 512 && low <= 4)) return false;
    if (M > PAIR_M && M <= 3 * GEMM_BM && N >= 6144 && !(rounds == 1 && K >= 8192)) return false;
    return !(M <= PAIR_M && rounds == 2 && K >= 4096);
}

template <int EPI>
static int launch_gemm2(const CUtensorMap& ta, const CUtensorMap& tb, void* C, const void* R, int M, int N,
                        int K, int ldc, int ldr, int* status, int pairs, int bn, cudaStream_t st, const TpArgs& tp,
                        const EpiArgs& ex) {
    auto kern = gemm2_bf16_kernel<EPI>;
    const int stages = std::min<int>(PAIR_MAX_STAGES, PAIR_RING / (PAIR_A_BYTES + bn * GEMM_BK));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM);
    if (e != cudaSuccess) return (int)e;
    e = launch_pdl(kern, dim3(2 * pairs), dim3(GEMM_THREADS), PAIR_SMEM, st, ta, tb, (bf16*)C, (const bf16*)R, M, N, K, ldc, ldr,
                   status, tp, bn, stages, ex);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// CTA-pair GEMM entry used by the public GEMM functions. Sets *handled = 0 (and launches nothing)
// when the shape is better served by the single-CTA kernel.
int pie_gemm2_dispatch(const void* A, const void* W, void* C, const void* R, int M, int N, int K, int lda,
                       int ldw, int ldc, int ldr, int epilogue, int* status, int num_sms, cudaStream_t st,
                       const TpArgs* tp_in, int* handled, const EpiArgs& ex) {
    *handled = 0;
    if (num_sms < 2) return 0;
    int bn = 0, pairs = 0;
    if (!plan_pairs(M, N, K, num_sms / 2, bn, pairs)) return 0;
    CUtensorMap ta, tb;
    if (pie_make_tma_2d_bf16(&ta, A, M, K, lda, GEMM_BM) != 0) return (int)cudaErrorInvalidValue;
    if (pie_make_tma_2d_bf16(&tb, W, N, K, ldw, bn / 2) != 0) return (int)cudaErrorInvalidValue;
    const TpArgs tp = tp_in ? *tp_in : TpArgs{};
    *handled = 1;
    switch (epilogue) {
        case EPI_STORE: return launch_gemm2<EPI_STORE>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        case EPI_RESIDUAL: return launch_gemm2<EPI_RESIDUAL>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        case EPI_SWIGLU: return launch_gemm2<EPI_SWIGLU>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        case EPI_GEGLU: return launch_gemm2<EPI_GEGLU>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        case EPI_XIELU: return launch_gemm2<EPI_XIELU>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        case EPI_STREAM: return launch_gemm2<EPI_STREAM>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        case EPI_RS: return launch_gemm2<EPI_RS>(ta, tb, C, R, M, N, K, ldc, ldr, status, pairs, bn, st, tp, ex);
        default: *handled = 0; return (int)cudaErrorInvalidValue;
    }
}
