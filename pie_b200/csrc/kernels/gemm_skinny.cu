// bf16 GEMM for batches of up to 128 rows:  C[M,N] = A[M,K] * W[N,K]^T with M <= 128.
//
// Such a product reads its weights once and does little else, so the kernel is laid out for streaming them:
//   * operands swapped, C^T = W * A^T: 128 weight rows are the MMA's rows, the batch its 16..128 columns, so a CTA moves
//     (128 + batch) x 128 B per 64 columns of K and no more;
//   * K split over the CTAs of a cluster (1, 2, 4 or 8) where the weight tiles alone are too few to keep the memory busy; the
//     partial tiles meet through distributed shared memory, in CTA order, so the sum does not depend on timing. Parking
//     them in global memory behind counters instead cost 4 to 5 us per launch: more than the 33 MB of an output projection take;
//   * at most half of an SM's shared memory and tensor memory per CTA. Two CTAs of one launch share an SM, so uneven tile
//     counts even out (what bounds the launch is memory, and every resident CTA has the same bytes in flight), and under
//     programmatic dependent launch the next product's weights stream in while this one's last tiles are stored.
// The split depends on N and K only: a request's numbers do not change with the batch it runs in, as long as that batch runs here
// (see pie_gemm_skinny_rows); where K is not split they are the general kernels' too.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 epilogue (thread = one output feature). Every mbarrier wait is
// bounded; on a time-out the kernel records a status word and leaves through its normal teardown.
#include <algorithm>

#include "gemm_common.cuh"

namespace pie {
using namespace sm100;

constexpr uint32_t SKINNY_W_BYTES = GEMM_BM * GEMM_BK * 2;     // a 128 x 64 weight tile
constexpr int SKINNY_MAX_STAGES = 8;
constexpr uint32_t SKINNY_RING = 108 * 1024;                   // two CTAs per SM
constexpr uint32_t SKINNY_SMEM = SKINNY_RING + 1024 /*align*/ + 256 /*barriers*/;

// tma_w walks the weights in boxes of 128 rows, tma_x the batch in boxes of all its rows.
// splits = CTAs of a cluster, each with its share of K; with splits > 1 the grid is one cluster per tile.
template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x, bf16* __restrict__ C,
                   const bf16* __restrict__ R, int M, int N, int K, int ldc, int ldr, int* status, int splits, int stages,
                   const __grid_constant__ EpiArgs ex) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    uint8_t* ring_ptr = smem_raw + (ring - raw);
    const uint32_t bar0 = ring + SKINNY_RING;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (SKINNY_MAX_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * SKINNY_MAX_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * SKINNY_MAX_STAGES + 2 + a); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ring_ptr + SKINNY_RING + 8 * (2 * SKINNY_MAX_STAGES + 4));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int cols = (M + 15) / 16 * 16;                       // columns of the MMA
    const uint32_t slot_bytes = SKINNY_W_BYTES + (uint32_t)cols * (GEMM_BK * 2);
    const uint32_t slot_tx = SKINNY_W_BYTES + (uint32_t)M * (GEMM_BK * 2);
    const uint32_t tmem_cols = cols <= 16 ? 32u : (cols <= 32 ? 64u : (cols <= 64 ? 128u : 256u));
    const int tiles = (N + GEMM_BM - 1) / GEMM_BM;
    const int num_kb = (K + GEMM_BK - 1) / GEMM_BK;
    const int part = splits > 1 ? (int)cluster_ctarank() : 0;
    const int kb0 = (int)((long)num_kb * part / splits), kb1 = (int)((long)num_kb * (part + 1) / splits);
    const int tile0 = blockIdx.x / splits, tile_step = gridDim.x / splits;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 4);
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) {
        tmem_alloc(smem_addr(const_cast<uint32_t*>(tmem_slot)), tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();

    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_desc(&tma_w);
            tma_prefetch_desc(&tma_x);
            // Weights that depend on nothing fill the ring at once; the batch's tiles follow when the producing kernel is
            // done. Weights that an earlier launch wrote (fp8 just expanded) wait like the batch.
            int s = 0, parked = 0, parked_kb = kb0;
            uint32_t ph = 0, issued = 0;
            bool ok = true, ready = false;
            auto resolve = [&]() {
                pdl_wait();
                for (int j = 0; j < parked; ++j) {
                    tma_load_2d(ring + j * slot_bytes + SKINNY_W_BYTES, &tma_x, full_bar(j), parked_kb * GEMM_BK, 0);
                    if (++parked_kb == kb1) parked_kb = kb0;
                }
                ready = true;
            };
            if (ex.fresh_w) resolve();
            for (int tile = tile0; tile < tiles && ok; tile += tile_step) {
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!ready && issued == (uint32_t)stages) resolve();
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    const uint32_t dst = ring + s * slot_bytes;
                    mbar_arrive_expect_tx(full_bar(s), slot_tx);
                    tma_load_2d(dst, &tma_w, full_bar(s), kb * GEMM_BK, tile * GEMM_BM);
                    if (ready) tma_load_2d(dst + SKINNY_W_BYTES, &tma_x, full_bar(s), kb * GEMM_BK, 0);
                    else ++parked;
                    ++issued;
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
            }
            if (!ready) resolve();
            // no copy may be in flight when the ring is reused or the CTA exits
            const uint32_t first = issued > (uint32_t)stages ? issued - stages : 0u;
            for (uint32_t j = first; j < issued; ++j)
                mbar_wait(full_bar(j % stages), (j / stages) & 1u, status, PIE_ERR_WAIT_TMA, 200000000ll);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = make_idesc_bf16(GEMM_BM, cols);
            int s = 0;
            uint32_t ph = 0, count = 0;
            bool ok = true;
            for (int tile = tile0; tile < tiles && ok; tile += tile_step, ++count) {
                const uint32_t acc = count & 1u, aph = (count >> 1) & 1u;
                if (!mbar_wait(tempty_bar(acc), aph ^ 1u, status, PIE_ERR_WAIT_EPILOGUE)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + acc * cols;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(full_bar(s), ph, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t wd = make_smem_desc_sw128(ring + s * slot_bytes);
                    const uint64_t xd = make_smem_desc_sw128(ring + s * slot_bytes + SKINNY_W_BYTES);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k) umma_bf16(d, wd + 2u * k, xd + 2u * k, idesc, ((kb - kb0) | k) != 0);
                    umma_commit(empty_bar(s));
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit(tfull_bar(acc));
            }
        }
    } else if (splits == 1) {
        const int q = warp & 3;
        pdl_wait();          // outputs and residual may still be in use by the previous kernel
        const XieluCoef act(EPI == EPI_XIELU ? ex.act : nullptr);
        uint32_t count = 0;
        for (int tile = tile0; tile < tiles; tile += tile_step, ++count) {
            const uint32_t acc = count & 1u, aph = (count >> 1) & 1u;
            const bool got = mbar_wait(tfull_bar(acc), aph, status, PIE_ERR_WAIT_MMA);
            if (!__all_sync(0xffffffffu, got)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * cols;
            const int feat = tile * GEMM_BM + q * 32 + lane;
            for (int g = 0; g < cols / 16; ++g) {
                uint32_t r[16];
                float v[16];
                tmem_ld_32x16(t_row + g * 16, r);
                tmem_ld_wait();
#pragma unroll
                for (int t = 0; t < 16; ++t) v[t] = __uint_as_float(r[t]);
                skinny_store<EPI>(v, feat, g * 16, N, M, C, ldc, R, ldr, ex, act);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(acc));
        }
    }
    if (splits > 1) {
        // Units of 32 features x 16 tokens, 4 quarters x groups of them; unit u is summed and stored by CTA u % splits, from
        // partials that lie in its ring as [unit / splits][source][4 tokens][32 features].
        const int q = warp & 3, groups = cols / 16;
        bool got = true;
        if (warp >= 2) {
            got = __all_sync(0xffffffffu, mbar_wait(tfull_bar(0), 0, status, PIE_ERR_WAIT_MMA));
            tc_fence_after();
        }
        __syncwarp();
        cluster_sync_all();              // every ring of the cluster is free, and every CTA has started
        if (warp >= 2 && got) {
            for (int g = 0; g < groups; ++g) {
                uint32_t r[16];
                tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + g * 16, r);
                tmem_ld_wait();
                const int u = q * groups + g;
                const uint32_t at = map_to_cta(ring + (uint32_t)((u / splits * splits + part) * 2048 + lane * 16), (uint32_t)(u % splits));
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    st_cluster_v4(at + t * 512, __uint_as_float(r[4 * t]), __uint_as_float(r[4 * t + 1]), __uint_as_float(r[4 * t + 2]),
                                  __uint_as_float(r[4 * t + 3]));
            }
        }
        tc_fence_before();
        __syncwarp();
        cluster_sync_all();
        if (warp >= 2 && got) {
            pdl_wait();
            const XieluCoef act(EPI == EPI_XIELU ? ex.act : nullptr);
            for (int slot = warp - 2; slot * splits + part < 4 * groups; slot += 4) {
                const int u = slot * splits + part;
                float v[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) v[t] = 0.f;
                for (int src = 0; src < splits; ++src) {
                    const float4* p = reinterpret_cast<const float4*>(ring_ptr + (slot * splits + src) * 2048) + lane;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const float4 a = p[t * 32];
                        v[4 * t] += a.x; v[4 * t + 1] += a.y; v[4 * t + 2] += a.z; v[4 * t + 3] += a.w;
                    }
                }
                skinny_store<EPI>(v, tile0 * GEMM_BM + u / groups * 32 + lane, u % groups * 16, N, M, C, ldc, R, ldr, ex, act);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

}  // namespace pie

using namespace pie;

extern "C" int pie_make_tma_2d_bf16(CUtensorMap* map, const void* ptr, long rows, long cols, long ld, int box_rows);

// CTAs that share the K of a weight tile: as many as are resident at once (two per SM), each with 4 or more k-blocks.
// Measured at 1 row: 4096 x 4096 in 12.6 / 10.4 / 9.1 us with 2 / 4 / 8 CTAs, 4096 x 14336 in 35.1 / 23.9 / 21.8 us;
// 6144 x 4096 in 12.1 us with 4 (192 CTAs) against 14.7 us with 8 (384: a second wave). A K below 2048 is not split: such
// products keep one summation order whatever the batch size, 129 rows and more included.
static int skinny_splits(int N, int K, int num_sms) {
    const int tiles = (N + GEMM_BM - 1) / GEMM_BM, num_kb = (K + GEMM_BK - 1) / GEMM_BK;
    int s = 1;
    while (K >= 2048 && s < 8 && tiles * 2 * s <= 2 * num_sms && num_kb >= 8 * s) s *= 2;
    return s;
}

// Most rows of a batch that runs here. Every CTA takes 128 weight rows and the whole batch through one SM, where the general kernel
// takes narrower tiles on more SMs; from 96 rows on three ring slots are left, and the epilogue has eight groups of tokens. So
// few tiles or a short K want few rows. Measured with cold caches, this kernel against the general one (us):
//   K >= 4096:        4096 x 4096 18.5 / 22.5 at 64 rows, 4096 x 14336 41 / 58 at 128; 28672 x 4096 59 / 61 at 64, 61 / 61 at 128
//   K < 4096, tiles for all SMs or more (weights bound both; uneven rounds count from K = 1536 on):
//                     51200 x 1536 43 / 47 at 64, 46 / 48 at 128; 28672 x 2040 41 / 39 at 112; 57344 x 768 29 / 31 at 96
//   K split in 8:     1024 x 2880 14.3 / 20.5 at 112 rows, 4096 x 2048 20.5 / 18.4 at 128 (but 2048 x 2048 16.4 / 18.5)
//   K split in 4:     6144 x 2880 20.7 / 22.6 at 112, 6144 x 2048 20.4 / 19.3 at 128
//   K split in 2:     10240 x 2880 and 14336 x 2048 gain up to 12 % at 32 rows, even out at 80, lose 8 % at 112
//   K not split:      2048 x 1024 14.3 / 14.3 at 48 rows, 16.4 / 14.3 at 96; 4096 x 1536 16.4 / 16.4 at 32, 20.5 / 16.4 at 128
int pie_gemm_skinny_rows(int N, int K, int num_sms) {
    if (K >= 4096) return 128;
    if ((N + GEMM_BM - 1) / GEMM_BM >= num_sms) return K >= 1536 ? 96 : 128;
    if (K < 2048) return K >= 1536 ? 48 : 64;
    const int splits = skinny_splits(N, K, num_sms);
    return splits >= 8 ? 128 : splits == 4 ? 112 : 80;
}

template <int EPI>
static int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, void* C, const void* R, int M, int N, int K, int ldc, int ldr,
                         int* status, int num_sms, cudaStream_t st, const EpiArgs& ex) {
    auto kern = gemm_skinny_kernel<EPI>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SKINNY_SMEM);
    if (e != cudaSuccess) return (int)e;
    const int splits = skinny_splits(N, K, num_sms), tiles = (N + GEMM_BM - 1) / GEMM_BM;
    const uint32_t slot = SKINNY_W_BYTES + (uint32_t)((M + 15) / 16 * 16) * (GEMM_BK * 2);
    const int stages = std::min(SKINNY_MAX_STAGES, (int)(SKINNY_RING / slot));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(splits > 1 ? tiles * splits : std::min(tiles, 2 * num_sms));
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = SKINNY_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = g_pie_pdl ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = splits;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = splits > 1 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kern, tw, tx, (bf16*)C, (const bf16*)R, M, N, K, ldc, ldr, status, splits, stages, ex);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// The product of a batch of at most 128 rows (arguments as of the general GEMM).
int pie_gemm_skinny(const void* A, const void* W, void* C, const void* R, int M, int N, int K, int lda, int ldw, int ldc, int ldr,
                    int epilogue, int* status, int num_sms, cudaStream_t st, const EpiArgs& ex) {
    CUtensorMap tw, tx;
    if (pie_make_tma_2d_bf16(&tw, W, N, K, ldw, GEMM_BM) != 0) return (int)cudaErrorInvalidValue;
    if (pie_make_tma_2d_bf16(&tx, A, M, K, lda, M) != 0) return (int)cudaErrorInvalidValue;
    switch (epilogue) {
        case EPI_STORE: return launch_skinny<EPI_STORE>(tw, tx, C, R, M, N, K, ldc, ldr, status, num_sms, st, ex);
        case EPI_RESIDUAL: return launch_skinny<EPI_RESIDUAL>(tw, tx, C, R, M, N, K, ldc, ldr, status, num_sms, st, ex);
        case EPI_SWIGLU: return launch_skinny<EPI_SWIGLU>(tw, tx, C, R, M, N, K, ldc, ldr, status, num_sms, st, ex);
        case EPI_GEGLU: return launch_skinny<EPI_GEGLU>(tw, tx, C, R, M, N, K, ldc, ldr, status, num_sms, st, ex);
        case EPI_XIELU: return launch_skinny<EPI_XIELU>(tw, tx, C, R, M, N, K, ldc, ldr, status, num_sms, st, ex);
        case EPI_STREAM: return launch_skinny<EPI_STREAM>(tw, tx, C, R, M, N, K, ldc, ldr, status, num_sms, st, ex);
        default: return (int)cudaErrorInvalidValue;
    }
}
