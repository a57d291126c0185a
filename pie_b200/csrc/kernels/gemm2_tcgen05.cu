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
// Tiles whole in K are as wide as makes the rounds of the machine short (plan_pairs). (Walking them in bands of row blocks, for operands
// that L2 holds together, measured no faster.) Back to back, weights cold, in tiles of 256 columns or on single CTAs and now (us):
// 512 x 4096 x 4096 23.7 and 16.3, 200 x 2048 x 4096 26.1 and 15.2, 200 x 49152 x 4096 92 and 86;
// 8300 x 28672 x 4096 1.45 ms either way: 1.3 PFLOP/s, what the power limit allows.
//
// Large products whose last round of 256-column tiles would be short have K split over the pairs instead, the parts parked in global
// memory. Whole tiles of another width are faster there (512 x 4096 x 14336 48 us against 62, 1536 x 4096 x 14336 124 against 174), but
// the tensor cores cut every addition off, and the error of a sum grows with the chain: 1.1e-9 of the result's norm for each of K, of
// 14336 1.6e-5 whole and 3.1e-6 to 6.0e-6 in parts, 4 to 7 times as much at 4 to 6 parts. 32-bit streams keep that difference.
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
                  int* status, const __grid_constant__ TpArgs tp, const StreamKArgs sk, int bn, int stages, const __grid_constant__ EpiArgs ex) {
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
            SegmentWalk walk(sk.enabled != 0, num_tiles, num_kb, pid, npairs);
            Segment seg;
            while (ok && walk.next(seg)) {
                const int m_blk = seg.tile % tiles_m, n_blk = seg.tile / tiles_m;
                const int a_row = m_blk * PAIR_M + (int)crank * GEMM_BM, b_row = n_blk * bn + (int)crank * (bn / 2);
                if (tp.gated && !ag_gate_wait_rows(tp, status, a_row, GEMM_BM, seen)) break;
                for (int kb = seg.kb0; kb < seg.kb1; ++kb, ++it) {
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
            SegmentWalk walk(sk.enabled != 0, num_tiles, num_kb, pid, npairs);
            Segment seg;
            for (; ok && walk.next(seg); ++tcount) {
                const uint32_t acc = tcount & 1u, aph = (tcount >> 1) & 1u;
                if (!mbar_wait_cluster(tempty_bar(acc), aph ^ 1u, status, PIE_ERR_WAIT_EPILOGUE)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * 256;
                for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
                    if (!mbar_wait_cluster(full_bar(s), ph, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = ring + s * stage_bytes;
                    const uint64_t adesc = make_smem_desc_sw128(a_addr);
                    const uint64_t bdesc = make_smem_desc_sw128(a_addr + PAIR_A_BYTES);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k)
                        umma_bf16_2cta(d_tmem, adesc + 2u * k, bdesc + 2u * k, idesc, ((kb - seg.kb0) | k) != 0);
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
        pdl_wait();          // outputs, residual and workspace may still be in use by the previous kernel
        const XieluCoef act(EPI == EPI_XIELU ? ex.act : nullptr);
        const uint32_t leader_tempty0 = map_to_cta(tempty_bar(0), 0);
        const uint32_t leader_tempty1 = map_to_cta(tempty_bar(1), 0);
        const long long total_units = (long long)num_tiles * num_kb;
        SegmentWalk walk(sk.enabled != 0, num_tiles, num_kb, pid, npairs);
        Segment seg;
        uint32_t tcount = 0;
        for (; walk.next(seg); ++tcount) {
            const int m_blk = seg.tile % tiles_m, n_blk = seg.tile / tiles_m;
            const uint32_t acc = tcount & 1u, aph = (tcount >> 1) & 1u;
            const bool got = mbar_wait_cluster(tfull_bar(acc), aph, status, PIE_ERR_WAIT_MMA);
            if (!__all_sync(0xffffffffu, got)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256;
            const int row0 = m_blk * PAIR_M + (int)crank * GEMM_BM + q * 32, col0 = n_blk * bn, n_end = min(N, col0 + bn);
            // Part of a tile: parked in the workspace, and the last pair to arrive for these 32 rows (nobody waits) adds up the tile's
            // parts, its own among them, in the order of the pairs. Layout of a slot and warp: [chunk of 32 columns][float4][lane].
            const bool partial = seg.kb0 != 0 || seg.kb1 != num_kb;
            const size_t slot_floats4 = (size_t)PAIR_M * bn / 4, mine4 = (size_t)((int)crank * 4 + q) * (32 * bn / 4) + lane;
            bool finalise = true;
            int c_first = 0, c_last = -1;
            if (partial) {
                uint4* park = reinterpret_cast<uint4*>(sk.ws) + (pid + seg.tile) * slot_floats4 + mine4;
#pragma unroll 1
                for (int c = 0; c < bn / 32; ++c) {
                    uint32_t v[32];
                    tmem_ld_32x32(t_row + c * 32, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) park[(c * 8 + j) * 32] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
                __threadfence();
                __syncwarp();
                c_first = streamk_cta_of((long long)seg.tile * num_kb, total_units, npairs);
                c_last = streamk_cta_of((long long)(seg.tile + 1) * num_kb - 1, total_units, npairs);
                int last = 0;
                if (lane == 0) {
                    int* ctr = sk.cnt + seg.tile * 8 + (int)crank * 4 + q;
                    last = atomicAdd(ctr, 1) == c_last - c_first;
                    if (last) *ctr = 0;
                }
                finalise = __shfl_sync(0xffffffffu, last, 0) != 0;
                if (finalise) __threadfence();
            }
#pragma unroll 1
            for (int c = 0; finalise && c < chunks; ++c) {
                uint32_t v0[32], v1[32];
                tmem_ld_32x32(t_row + c * 64, v0);
                tmem_ld_32x32(t_row + c * 64 + 32, v1);
                tmem_ld_wait();
                if (partial) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v0[j] = v1[j] = 0u;
                    for (int cc = c_first; cc <= c_last; ++cc) {
                        const float4* part = reinterpret_cast<const float4*>(sk.ws) + (cc + seg.tile) * slot_floats4 + mine4 + (size_t)c * 16 * 32;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 a4 = __ldcg(part + j * 32), b4 = __ldcg(part + (8 + j) * 32);
                            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                v0[4 * j + e] = __float_as_uint(__uint_as_float(v0[4 * j + e]) + a[e]);
                                v1[4 * j + e] = __float_as_uint(__uint_as_float(v1[4 * j + e]) + b[e]);
                            }
                        }
                    }
                }
                epilogue_store_64<EPI>(v0, v1, stage, row0, col0 + c * 64, M, N, C, ldc, R, ldr, tp, n_end, ex, &act);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (leader) mbar_arrive(tempty_bar(acc));
                else mbar_arrive_cluster(acc ? leader_tempty1 : leader_tempty0);
            }
            if (EPI == EPI_RS && finalise) {
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

// Products whose K is split over pairs, if at all: from 2e10 multiplications on, from 1e10 with a long K. Below, single CTAs may split it.
bool pie_gemm2_large(int M, int N, int K) {
    const double macs = (double)M * N * K;
    return M > GEMM_BM && N >= 128 && (macs >= 2.0e10 || (macs >= 1.0e10 && K >= 8192));
}

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
// the best of thirteen widths over 96 shapes of 200 to 3661 rows.
//
// Pairs or single CTAs (in tiles of their plan, `single_bn`): what should take less time, by a fit to 2941 products of 129 to 2305 rows,
// 128 to 128256 features and a K of 128 to 14336. The faster kernel to 0.5 % in the mean over them, to 2 % for 94 of 100; over 399 more of
// any size, odd ones among them, 1.2 % and 88 of 100. Pairs against single CTAs, weights cold, back to back (us):
//   a short K, whose rounds are all start and epilogue: 640 x 65536 x 256 39.8 / 28.4, 1024 x 9216 x 128 11.3 / 8.8, 512 x 9216 x 512 9.0 / 8.3
//   257 to 384 rows, whose pairs' tiles are up to half empty: 300 x 12288 x 4096 37.9 / 34.2, but 300 x 4096 x 4096 15.7 / 17.4
//   a last round of either kind that is nearly empty: 640 x 7168 x 2048 18.8 / 16.6, 129 x 24576 x 4096 46.5 / 61.9
// Where K is split - on pairs here, or on single CTAs (single_splits: their plan does so) - is a matter of the error of sums and of their
// order, and stays as it is whatever is the faster way.
struct PairPlan {
    int width, pairs, streamk;
};
static bool plan_pairs(int M, int N, int K, int num_sms, long ws_floats, int cnt_ints, int single_bn, bool single_splits, PairPlan& p) {
    if (M <= GEMM_BM || N < 128) return false;
    const int pairs_max = num_sms / 2;
    const long num_kb = (K + GEMM_BK - 1) / GEMM_BK, tiles_m = (M + PAIR_M - 1) / PAIR_M;
    if (g_pair_bn == 0) {
        const bool large = pie_gemm2_large(M, N, K);
        if (!large && single_splits) return false;
        const int bn = N >= 256 ? 256 : 128;
        const long tiles = tiles_m * ((N + bn - 1) / bn), rounds = (tiles + pairs_max - 1) / pairs_max;
        const long pairs = std::min<long>(tiles * num_kb / 16, pairs_max);         // 16 k-blocks per pair or more
        if (large && pairs >= 1 && tiles % pairs != 0 && tiles <= 2L * pairs_max && (double)tiles / pairs + 0.12 < 0.92 * rounds &&
            (pairs + tiles) * PAIR_M * bn <= ws_floats && tiles * 8 <= cnt_ints) {
            p = PairPlan{bn, (int)pairs, 1};
            return true;
        }
    }
    long best = -1, rounds = 0;
    for (int bn = 256; bn >= 64; bn -= 16) {
        if (g_pair_bn > 0 && bn != g_pair_bn) continue;
        const long tiles = tiles_m * ((N + bn - 1) / bn), r = (tiles + pairs_max - 1) / pairs_max;
        const long cost = r * (num_kb * (bn + 62) + 500) + 10 * bn;
        if (best >= 0 && cost >= best) continue;
        best = cost;
        rounds = r;
        p = PairPlan{bn, (int)std::min<long>(pairs_max, tiles), 0};
    }
    if (g_pair_bn) return true;
    const long tiles_1 = (long)((M + GEMM_BM - 1) / GEMM_BM) * ((N + single_bn - 1) / single_bn), rounds_1 = (tiles_1 + num_sms - 1) / num_sms;
    const double single_ns = rounds_1 * (num_kb * (single_bn + 180.) + 800. + 1.5 * single_bn) + 6. * single_bn + 1200.;
    return rounds * (num_kb * (p.width + 80.) + 1660.) + 20. * p.width < single_ns;
}

template <int EPI>
static int launch_gemm2(const CUtensorMap& ta, const CUtensorMap& tb, void* C, const void* R, int M, int N,
                        int K, int ldc, int ldr, int* status, const PairPlan& p, float* ws, int* cnt, cudaStream_t st,
                        const TpArgs& tp, const EpiArgs& ex) {
    auto kern = gemm2_bf16_kernel<EPI>;
    const int stages = std::min<int>(PAIR_MAX_STAGES, PAIR_RING / (PAIR_A_BYTES + p.width * GEMM_BK));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PAIR_SMEM);
    if (e != cudaSuccess) return (int)e;
    const StreamKArgs sk{ws, cnt, p.streamk, 0, nullptr};
    e = launch_pdl(kern, dim3(2 * p.pairs), dim3(GEMM_THREADS), PAIR_SMEM, st, ta, tb, (bf16*)C, (const bf16*)R, M, N, K, ldc, ldr,
                   status, tp, sk, p.width, stages, ex);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// The plan of a launch: out = {width of the tiles, pairs, K split}. False where the single-CTA kernel takes the product.
bool pie_gemm2_plan(int M, int N, int K, int num_sms, long ws_floats, int cnt_ints, int single_bn, bool single_splits, int* out) {
    PairPlan p{};
    if (num_sms < 2 || !plan_pairs(M, N, K, num_sms, ws_floats, cnt_ints, single_bn, single_splits, p)) return false;
    out[0] = p.width;
    out[1] = p.pairs;
    out[2] = p.streamk;
    return true;
}

// CTA-pair GEMM entry used by the public GEMM functions. Sets *handled = 0 (and launches nothing)
// when the shape is better served by the single-CTA kernel.
int pie_gemm2_dispatch(const void* A, const void* W, void* C, const void* R, int M, int N, int K, int lda,
                       int ldw, int ldc, int ldr, int epilogue, int* status, int num_sms, cudaStream_t st,
                       const TpArgs* tp_in, float* ws, long ws_floats, int* cnt, int cnt_ints, int single_bn, bool single_splits,
                       int* handled, const EpiArgs& ex) {
    *handled = 0;
    if (num_sms < 2) return 0;
    PairPlan p{};
    if (!plan_pairs(M, N, K, num_sms, ws ? ws_floats : 0, cnt_ints, single_bn, single_splits, p)) return 0;
    CUtensorMap ta, tb;
    if (pie_make_tma_2d_bf16(&ta, A, M, K, lda, GEMM_BM) != 0) return (int)cudaErrorInvalidValue;
    if (pie_make_tma_2d_bf16(&tb, W, N, K, ldw, p.width / 2) != 0) return (int)cudaErrorInvalidValue;
    const TpArgs tp = tp_in ? *tp_in : TpArgs{};
    *handled = 1;
    switch (epilogue) {
        case EPI_STORE: return launch_gemm2<EPI_STORE>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        case EPI_RESIDUAL: return launch_gemm2<EPI_RESIDUAL>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        case EPI_SWIGLU: return launch_gemm2<EPI_SWIGLU>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        case EPI_GEGLU: return launch_gemm2<EPI_GEGLU>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        case EPI_XIELU: return launch_gemm2<EPI_XIELU>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        case EPI_STREAM: return launch_gemm2<EPI_STREAM>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        case EPI_RS: return launch_gemm2<EPI_RS>(ta, tb, C, R, M, N, K, ldc, ldr, status, p, ws, cnt, st, tp, ex);
        default: *handled = 0; return (int)cudaErrorInvalidValue;
    }
}
