// Block-scaled fp8 GEMM on the 5th-generation tensor cores:
//     C[M,N] = sum over 128-deep K blocks b of  sa[m,b] * sw[n,b] * (A8[m, b] . W8[n, b])
// A8 / W8 are fp8 e4m3; sa holds one fp32 scale per (row, 128 columns) of the activation (1 x 128
// quantisation, produced by pie_quant_act_fp8), sw one per (row, 128 columns) of the weight
// (128 x 128 checkpoint blocks expanded to rows when the weight is loaded).
//
// One CTA per 128 x BN output tile, persistent over tiles:
//   warp 0      TMA producer: per K block one 128 x 128-byte tile of A8 and one bn x 128-byte tile
//               of W8 (128-byte swizzle) into a ring of slots
//   warp 1      four tcgen05.mma.kind::f8f6f4 (K = 32 each) per K block into one of two TMEM
//               buffers, starting from zero each block; tcgen05.commit frees the ring slot and
//               publishes the block's partial product
//   warps 2-5   read the partial product from TMEM, scale it by sa * sw and add it to fp32
//               accumulators in registers (one output row per thread); after the last block the
//               usual epilogue (store / +residual / SwiGLU) writes bf16
// The per-block rescale in registers is what block scaling costs; the MMAs of block b+1 overlap it
// through the second TMEM buffer. Every wait is bounded (status word, drain, TMEM freed).
//
// Replaces the reference's dequantise-to-bf16 kernel followed by a library GEMM for block-scaled
// fp8 weights (driver/cuda/src/ops/gemm.cpp:1166-1211, driver/cuda/src/kernels/dequant_fp8.cu:41).
#include <cuda_fp8.h>

#include <algorithm>

#include "gemm_common.cuh"

namespace pie {
using namespace sm100;

constexpr int F8_BK = 128;   // fp8 elements (= bytes) per K block: one swizzle span

template <int BN>
struct Fp8Cfg {
    static constexpr uint32_t A_BYTES = GEMM_BM * F8_BK;
    static constexpr uint32_t B_BYTES = BN * F8_BK;
    static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = BN == 128 ? 5 : 7;
    static constexpr uint32_t TMEM_COLS = 2 * BN;
    static constexpr uint32_t SCALE_BYTES = 4 * 2 * BN * 4;   // per epilogue warp: weight scales of the block being folded, double-buffered
    static constexpr uint32_t SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + SCALE_BYTES + 16384;
};

// Instruction descriptor, kind::f8f6f4: e4m3 x e4m3 -> fp32, both operands K-major.
//   [4,6) D format (1 = f32)  [7,10) A format (0 = e4m3)  [10,13) B format (0 = e4m3)
//   [17,23) N >> 3  [24,29) M >> 4
__host__ __device__ constexpr uint32_t make_idesc_e4m3(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int BN, int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                const float* __restrict__ sa, const float* __restrict__ sw, bf16* __restrict__ C,
                const bf16* __restrict__ R, int M, int N, int K, int ldc, int ldr, int* status, int bn,
                const __grid_constant__ TpArgs tp) {
    using Cfg = Fp8Cfg<BN>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t tiles = (raw + 1023u) & ~1023u;
    uint8_t* tiles_ptr = smem_raw + (tiles - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles_ptr + STAGES * Cfg::STAGE_BYTES);
    const uint32_t bar0 = tiles + STAGES * Cfg::STAGE_BYTES;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
    auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * STAGES + a); };
    auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * STAGES + 2 + a); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 4);
    float* sw_s = reinterpret_cast<float*>(tiles_ptr + STAGES * Cfg::STAGE_BYTES + 256);          // [4 warps][2][BN]
    uint8_t* stage_base = tiles_ptr + STAGES * Cfg::STAGE_BYTES + 256 + Cfg::SCALE_BYTES;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int tiles_m = (M + GEMM_BM - 1) / GEMM_BM;
    const int tiles_n = (N + bn - 1) / bn;
    const int num_tiles = tiles_m * tiles_n;
    const int num_kb = (K + F8_BK - 1) / F8_BK;
    const uint32_t stage_tx = Cfg::A_BYTES + (uint32_t)bn * F8_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
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
        tmem_alloc(smem_addr(const_cast<uint32_t*>(tmem_slot)), Cfg::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_desc(&tma_a);
            tma_prefetch_desc(&tma_b);
            uint32_t it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                const int m_blk = tile % tiles_m, n_blk = tile / tiles_m;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1u;
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    mbar_arrive_expect_tx(full_bar(s), stage_tx);
                    const uint32_t dst = tiles + s * Cfg::STAGE_BYTES;
                    tma_load_2d(dst, &tma_a, full_bar(s), kb * F8_BK, m_blk * GEMM_BM);
                    tma_load_2d(dst + Cfg::A_BYTES, &tma_b, full_bar(s), kb * F8_BK, n_blk * bn);
                }
            }
            const uint32_t first = it > (uint32_t)STAGES ? it - STAGES : 0u;
            for (uint32_t j = first; j < it; ++j)
                mbar_wait(full_bar(j % STAGES), (j / STAGES) & 1u, status, PIE_ERR_WAIT_TMA, 200000000ll);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = make_idesc_e4m3(GEMM_BM, bn);
            uint32_t it = 0;      // counts K blocks = TMEM buffer uses
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t buf = it & 1u, bph = (it >> 1) & 1u;
                    if (!mbar_wait(tempty_bar(buf), bph ^ 1u, status, PIE_ERR_WAIT_EPILOGUE)) { ok = false; break; }
                    if (!mbar_wait(full_bar(s), (it / STAGES) & 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = tiles + s * Cfg::STAGE_BYTES;
                    const uint64_t adesc = make_smem_desc_sw128(a_addr);
                    const uint64_t bdesc = make_smem_desc_sw128(a_addr + Cfg::A_BYTES);
                    const uint32_t d_tmem = tmem_base + buf * BN;
#pragma unroll
                    for (int k = 0; k < F8_BK / 32; ++k)
                        umma_f8(d_tmem, adesc + 2u * k, bdesc + 2u * k, idesc, k != 0);
                    umma_commit(empty_bar(s));
                    umma_commit(tfull_bar(buf));
                }
            }
        }
    } else {
        // accumulate + epilogue: 128 threads, thread = one output row of the tile
        const int q = warp & 3;
        float* sw_w = sw_s + (warp - 2) * 2 * BN;      // this warp's copy: no barrier across warps is needed
        uint32_t it = 0;
        bool ok = true;
        const int kbs = (K + 127) / 128;       // columns of the scale tables
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
            const int m_blk = tile % tiles_m, n_blk = tile / tiles_m;
            const int row = m_blk * GEMM_BM + q * 32 + lane;
            const int n0 = n_blk * bn;
            float acc[BN];
#pragma unroll
            for (int c = 0; c < BN; ++c) acc[c] = 0.f;
            // scales of the next K block are fetched one block ahead (global latency hidden behind
            // the wait for the MMAs and the fold of the current block); lane l keeps the weight
            // scales of columns l, l+32, ... in registers and hands them to its warp through smem
            constexpr int SPL = BN / 32;
            float sw_n[SPL], sa_n;
            auto fetch = [&](int kb) {
#pragma unroll
                for (int u = 0; u < SPL; ++u) {
                    const int c = u * 32 + lane;
                    sw_n[u] = (c < bn && n0 + c < N) ? __ldg(sw + (size_t)(n0 + c) * kbs + kb) : 0.f;
                }
                sa_n = row < M ? __ldg(sa + (size_t)row * kbs + kb) : 0.f;
            };
            fetch(0);
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const uint32_t buf = it & 1u, bph = (it >> 1) & 1u;
                float* sws = sw_w + buf * BN;
#pragma unroll
                for (int u = 0; u < SPL; ++u) sws[u * 32 + lane] = sw_n[u];
                const float sa_r = sa_n;
                if (kb + 1 < num_kb) fetch(kb + 1);
                __syncwarp();
                const bool got = mbar_wait(tfull_bar(buf), bph, status, PIE_ERR_WAIT_MMA);
                if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
                tc_fence_after();
                const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN;
#pragma unroll
                for (int c = 0; c < BN / 32; ++c) {
                    if (c * 32 < bn) {
                        uint32_t v[32];
                        tmem_ld_32x32(t_row + c * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            acc[c * 32 + j] = fmaf(__uint_as_float(v[j]), sa_r * sws[c * 32 + j], acc[c * 32 + j]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(buf));
            }
            if (!ok) break;
            uint8_t* stage = stage_base + (warp - 2) * 4096;
#pragma unroll
            for (int c = 0; c < BN / 64; ++c) {
                if (c * 64 < bn) {
                    uint32_t v0[32], v1[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        v0[j] = __float_as_uint(acc[c * 64 + j]);
                        v1[j] = __float_as_uint(acc[c * 64 + 32 + j]);
                    }
                    epilogue_store_64<EPI>(v0, v1, stage, m_blk * GEMM_BM + q * 32, n0 + c * 64, M, N, C, ldc, R, ldr,
                                           tp, min(N, n0 + bn));
                }
            }
            if (EPI == EPI_RS) {
                // this warp's rows of the tile are in the owners' receive buffers: count the arrival
                __threadfence_system();
                __syncwarp();
                if (lane == 0) rs_publish_arrival(tp, num_tiles * 4);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------ batches of up to 64 rows
// Laid out for streaming the weights, as the bf16 kernel for such batches (gemm_skinny.cu): operands swapped (weight rows are
// the MMA's rows, the batch its 16..64 columns), the ring filled with weights before the producing kernel is done. K is not
// split: the sum over its blocks keeps the order of the kernel above, because the next layer's quantiser turns a last bit into
// a step of 8-bit numbers. (Split over clusters, results of one layer agree to 3e-5, logits of four layers only to 4 %.) A tile has
// `height` weight rows: the MMA's other rows are whatever shared memory holds, each reaches its own accumulator row alone, and
// these are not read.
//
// What block scaling adds: every 128 of K has a partial product of its own in tensor memory, which the epilogue warps scale and
// add up in registers - warp w the 32 features of quarter w % 4 and every other group of 16 tokens. With a hand-over per block that
// chain was what a launch took (0.3 us a block whatever the tile), so blocks are handed over in groups of four, two groups in
// flight: one barrier, and the loads of two blocks under way at once. That takes all of tensor memory and the registers of one CTA
// per SM, which also halves the CTAs that ask L2 for the same rows of the batch. The scales of features and tokens come through
// shared memory, four K blocks at a time and seven such chunks ahead.
//
// Weights cold, at 8 / 24 / 48 / 64 rows (us), with two CTAs per SM and block by block, or by the kernel above where that ran, and like this:
// 5120 x 25600 (20.6 at the memory's rate) 79 / 87 / 88 / 88 and 47 / 50 / 56 / 64; 10240 x 5120 22 / 29 / 27 / 27 and 13 / 14 / 15 / 16;
// 51200 x 5120 43 / 46 / 54 / 60 and 42 / 43 / 44 / 45 (6.3 to 5.8 TB/s); 24576 x 4096 18.8 / 20.2 / 23.6 / 25.8 and 19.2 / 20.2 / 22.0 / 24.1.
// Up to 16 rows in two rounds of tiles are slower than they were by 2 % (24576 x 5120, one row: 22.1 and 22.7) to 4 % (27648 x 2560: 13.8 and
// 14.3).
constexpr int F8S_THREADS = 64 + 256, F8S_CHUNK = 4;
constexpr uint32_t F8S_MMA_BYTES = GEMM_BM * F8_BK;          // what an MMA reads from a slot's start on
constexpr uint32_t F8S_BUFS = 2;                               // groups of F8S_CHUNK blocks in tensor memory
constexpr uint32_t F8S_BLOCK_COLS = 64, F8S_TMEM_COLS = F8S_BUFS * F8S_CHUNK * F8S_BLOCK_COLS;
constexpr int F8S_DEPTH = 8;                                   // chunks of scales: one in use, the others on their way
constexpr uint32_t F8S_RING = 176 * 1024;
constexpr uint32_t F8S_SCALES = F8S_DEPTH * F8S_CHUNK * (64 + GEMM_BM) * 4;
constexpr uint32_t F8S_SMEM = F8S_RING + F8S_SCALES + 1024 /*align*/ + 512 /*barriers*/;
constexpr int F8S_MAX_STAGES = 20;

// height: weight rows of a tile and of its box, a multiple of 16.
template <int EPI>
__global__ void __launch_bounds__(F8S_THREADS, 1)
gemm_fp8_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                       const float* __restrict__ sa, const float* __restrict__ sw, bf16* __restrict__ C, const bf16* __restrict__ R,
                       int M, int N, int K, int ldc, int ldr, int* status, int stages, int height) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    uint8_t* ring_ptr = smem_raw + (ring - raw);
    float* sx = reinterpret_cast<float*>(ring_ptr + F8S_RING);           // [F8S_DEPTH][F8S_CHUNK][64]
    float* swt = sx + F8S_DEPTH * F8S_CHUNK * 64;                        // [F8S_DEPTH][128 features][F8S_CHUNK]
    const uint32_t bar0 = ring + F8S_RING + F8S_SCALES;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (F8S_MAX_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * F8S_MAX_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * F8S_MAX_STAGES + 4 + a); };
    volatile uint32_t* tmem_slot =
        reinterpret_cast<volatile uint32_t*>(ring_ptr + F8S_RING + F8S_SCALES + 8 * (2 * F8S_MAX_STAGES + 8));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int cols = (M + 15) / 16 * 16, groups = cols / 16;
    const uint32_t w_bytes = (uint32_t)height * F8_BK, slot_bytes = w_bytes + (uint32_t)cols * F8_BK, slot_tx = (uint32_t)(height + M) * F8_BK;
    const int tiles = (N + height - 1) / height, num_kb = (K + F8_BK - 1) / F8_BK;
    const int tile0 = blockIdx.x, tile_step = gridDim.x;
    const int quarters = (height + 31) / 32;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (uint32_t a = 0; a < F8S_BUFS; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 2 * quarters);
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) {
        tmem_alloc(smem_addr(const_cast<uint32_t*>(tmem_slot)), F8S_TMEM_COLS);
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
            // the weights depend on nothing and fill the ring at once; the batch's tiles follow when the producing kernel is done
            int s = 0, parked = 0, parked_kb = 0;
            uint32_t ph = 0, issued = 0;
            bool ok = true, ready = false;
            auto resolve = [&]() {
                pdl_wait();
                for (int j = 0; j < parked; ++j) {
                    tma_load_2d(ring + j * slot_bytes + w_bytes, &tma_x, full_bar(j), parked_kb * F8_BK, 0);
                    if (++parked_kb == num_kb) parked_kb = 0;
                }
                ready = true;
            };
            for (int tile = tile0; tile < tiles && ok; tile += tile_step) {
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!ready && issued == (uint32_t)stages) resolve();
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                    const uint32_t dst = ring + s * slot_bytes;
                    mbar_arrive_expect_tx(full_bar(s), slot_tx);
                    tma_load_2d(dst, &tma_w, full_bar(s), kb * F8_BK, tile * height);
                    if (ready) tma_load_2d(dst + w_bytes, &tma_x, full_bar(s), kb * F8_BK, 0);
                    else ++parked;
                    ++issued;
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
            }
            if (!ready) resolve();
            // no copy may be in flight when the CTA exits
            const uint32_t first = issued > (uint32_t)stages ? issued - stages : 0u;
            for (uint32_t j = first; j < issued; ++j)
                mbar_wait(full_bar(j % stages), (j / stages) & 1u, status, PIE_ERR_WAIT_TMA, 200000000ll);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = make_idesc_e4m3(GEMM_BM, cols);
            int s = 0;
            uint32_t ph = 0, buf = 0, bph = 0;
            bool ok = true;
            for (int tile = tile0; tile < tiles && ok; tile += tile_step) {
                for (int kb = 0; kb < num_kb; kb += F8S_CHUNK) {
                    if (!mbar_wait(tempty_bar(buf), bph ^ 1u, status, PIE_ERR_WAIT_EPILOGUE)) { ok = false; break; }
#pragma unroll
                    for (int j = 0; j < F8S_CHUNK; ++j) {
                        if (kb + j >= num_kb) break;
                        if (!mbar_wait(full_bar(s), ph, status, PIE_ERR_WAIT_TMA)) { ok = false; break; }
                        tc_fence_after();
                        const uint64_t wd = make_smem_desc_sw128(ring + s * slot_bytes);
                        const uint64_t xd = make_smem_desc_sw128(ring + s * slot_bytes + w_bytes);
#pragma unroll
                        for (int k = 0; k < F8_BK / 32; ++k)
                            umma_f8(tmem_base + (buf * F8S_CHUNK + j) * F8S_BLOCK_COLS, wd + 2u * k, xd + 2u * k, idesc, k != 0);
                        umma_commit(empty_bar(s));
                        if (++s == stages) { s = 0; ph ^= 1u; }
                    }
                    if (!ok) break;
                    umma_commit(tfull_bar(buf));
                    if (++buf == F8S_BUFS) { buf = 0; bph ^= 1u; }
                }
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2, et = threadIdx.x - 64;
        const bool vec = num_kb % F8S_CHUNK == 0 && ((uintptr_t)sw & 15) == 0, active = q < quarters;
        const int chunks = (num_kb + F8S_CHUNK - 1) / F8S_CHUNK, total = (tiles - tile0 + tile_step - 1) / tile_step * chunks;
        uint32_t buf = 0, bph = 0;
        bool ok = true;
        float acc[2][16];                                                // group 2 i + half, token
        pdl_wait();          // outputs, residual and the tokens' scales may still be in use by the previous kernel
        auto request = [&](int c) {                                      // one group of copies per chunk, empty past the last one
            if (c < total) {
                const int kb = c % chunks * F8S_CHUNK, feat0 = (tile0 + c / chunks * tile_step) * height, b = c % F8S_DEPTH;
                for (int i = et; i < F8S_CHUNK * cols; i += 256) {
                    const int tok = i / F8S_CHUNK, j = i % F8S_CHUNK;
                    const bool live = tok < M && kb + j < num_kb;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_addr(sx + (b * F8S_CHUNK + j) * 64 + tok)),
                                 "l"(live ? sa + (size_t)tok * num_kb + kb + j : sa), "r"(live ? 4 : 0) : "memory");
                }
                if (vec) {
                    if (et < height)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(swt + (b * GEMM_BM + et) * F8S_CHUNK)),
                                     "l"(sw + (size_t)min(feat0 + et, N - 1) * num_kb + kb) : "memory");
                } else {
                    for (int i = et; i < height * F8S_CHUNK; i += 256) {
                        const int f = i / F8S_CHUNK, j = i % F8S_CHUNK;
                        const bool live = kb + j < num_kb;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_addr(swt + (b * GEMM_BM + f) * F8S_CHUNK + j)),
                                     "l"(live ? sw + (size_t)min(feat0 + f, N - 1) * num_kb + kb + j : sw), "r"(live ? 4 : 0) : "memory");
                    }
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        for (int c = 0; c < F8S_DEPTH - 1; ++c) request(c);
        for (int c = 0; c < total; ++c) {
            const int tile = tile0 + c / chunks * tile_step, kb = c % chunks * F8S_CHUNK, b = c % F8S_DEPTH;
            asm volatile("cp.async.wait_group %0;\n" ::"n"(F8S_DEPTH - 2) : "memory");
            asm volatile("bar.sync 1, 256;\n" ::: "memory");             // a warp whose wait ran out still comes here
            request(c + F8S_DEPTH - 1);
            if (!active) continue;
            if (kb == 0) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int t = 0; t < 16; ++t) acc[i][t] = 0.f;
            }
            const float4 of = *reinterpret_cast<const float4*>(swt + (b * GEMM_BM + q * 32 + lane) * F8S_CHUNK);
            const float mine[F8S_CHUNK] = {of.x, of.y, of.z, of.w};
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(tfull_bar(buf), bph, status, PIE_ERR_WAIT_MMA));
            if (ok) {
                tc_fence_after();
                const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + buf * F8S_CHUNK * F8S_BLOCK_COLS;
#pragma unroll
                for (int j1 = 0; j1 < F8S_CHUNK; j1 += 2) {              // two blocks' products in registers at once
                    uint32_t v[2][2][16];
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            if (2 * i + half < groups) tmem_ld_32x16(t_row + (j1 + j) * F8S_BLOCK_COLS + (2 * i + half) * 16, v[j][i]);
                    tmem_ld_wait();
                    if (j1 + 2 == F8S_CHUNK) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(tempty_bar(buf));
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (kb + j1 + j >= num_kb) break;
                        const float* scales = sx + (b * F8S_CHUNK + j1 + j) * 64;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int g = 2 * i + half;
                            if (g >= groups) break;
#pragma unroll
                            for (int t = 0; t < 16; t += 4) {
                                const float4 f = *reinterpret_cast<const float4*>(scales + g * 16 + t);
                                acc[i][t] = fmaf(__uint_as_float(v[j][i][t]), f.x * mine[j1 + j], acc[i][t]);
                                acc[i][t + 1] = fmaf(__uint_as_float(v[j][i][t + 1]), f.y * mine[j1 + j], acc[i][t + 1]);
                                acc[i][t + 2] = fmaf(__uint_as_float(v[j][i][t + 2]), f.z * mine[j1 + j], acc[i][t + 2]);
                                acc[i][t + 3] = fmaf(__uint_as_float(v[j][i][t + 3]), f.w * mine[j1 + j], acc[i][t + 3]);
                            }
                        }
                    }
                }
            }
            if (++buf == F8S_BUFS) { buf = 0; bph ^= 1u; }
            if (kb + F8S_CHUNK >= num_kb && ok) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int g = 2 * i + half;
                    if (g >= groups) break;
                    skinny_store<EPI>(acc[i], tile * height + q * 32 + lane, g * 16, min(N, (tile + 1) * height), M, C, ldc, R, ldr, EpiArgs(),
                                      XieluCoef(nullptr));
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, F8S_TMEM_COLS);
    }
}

// 1 x 128 activation quantisation: one warp per (row, 128-column block).
__global__ void quant_act_fp8_kernel(const bf16* __restrict__ x, int ldx, uint8_t* __restrict__ x8, float* __restrict__ sx,
                                     int M, int K) {
    const int kbs = (K + 127) / 128;
    const long gw = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    pdl_trigger();
    pdl_wait();
    if (gw >= (long)M * kbs) return;
    const int row = (int)(gw / kbs), kb = (int)(gw - (long)row * kbs);
    const int c = kb * 128 + lane * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (c < K) {
        const uint2 raw = *reinterpret_cast<const uint2*>(x + (size_t)row * ldx + c);
        const bf162* p = reinterpret_cast<const bf162*>(&raw);
        const float2 a = __bfloat1622float2(p[0]), b = __bfloat1622float2(p[1]);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    amax = warp_max(amax);
    const float scale = fmaxf(amax, 1e-12f) / 448.f;
    const float inv = 1.f / scale;
    if (c < K) {
        const __nv_fp8x4_storage_t q4 = __nv_cvt_float2_to_fp8x2(make_float2(v[0] * inv, v[1] * inv), __NV_SATFINITE, __NV_E4M3) |
                                        ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v[2] * inv, v[3] * inv), __NV_SATFINITE, __NV_E4M3) << 16);
        *reinterpret_cast<uint32_t*>(x8 + (size_t)row * K + c) = q4;
    }
    if (lane == 0) sx[(size_t)row * kbs + kb] = scale;
}

}  // namespace pie

using namespace pie;

extern "C" int pie_make_tma_2d_bf16(CUtensorMap* map, const void* ptr, long rows, long cols, long ld, int box_rows);

typedef CUresult (*EncodeTiledFn8)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 2-D uint8 row-major [rows, cols]; box = box_rows x 128 bytes with the 128-byte swizzle.
static int make_tma_2d_u8(CUtensorMap* map, const void* ptr, long rows, long cols, long ld, int box_rows) {
    static EncodeTiledFn8 enc = nullptr;
    if (!enc) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return -1;
        enc = reinterpret_cast<EncodeTiledFn8>(p);
    }
    if (((uintptr_t)ptr & 15) || ld % 16) return -2;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld};
    cuuint32_t box[2] = {(cuuint32_t)F8_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return (int)enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// x [M, K] bf16 -> x8 [M, K] e4m3 (dense, leading dimension K) and sx [M, ceil(K/128)].
PIE_API int pie_quant_act_fp8(const void* x, int ldx, void* x8, float* sx, int M, int K, cudaStream_t st) {
    if (M <= 0) return 0;
    if (K % 16 || ldx % 4) return (int)cudaErrorInvalidValue;
    const long warps = (long)M * ((K + 127) / 128);
    const int blocks = (int)((warps * 32 + 255) / 256);
    const cudaError_t e = launch_pdl(quant_act_fp8_kernel, dim3(blocks), dim3(256), 0, st, (const bf16*)x, ldx, (uint8_t*)x8, sx, M, K);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// C[M,N] (or [M,N/2] with SwiGLU) from fp8 operands and their scales (see the header comment).
static int gemm_fp8_launch(const void* A8, const float* sa, const void* W8, const float* sw, void* C,
                           const void* R, int M, int N, int K, int ldc, int ldr, int epilogue, int* status,
                           int num_sms, cudaStream_t st, const TpArgs& tp);

PIE_API int pie_gemm_fp8_blockscaled(const void* A8, const float* sa, const void* W8, const float* sw, void* C,
                                     const void* R, int M, int N, int K, int ldc, int ldr, int epilogue, int* status,
                                     int num_sms, cudaStream_t st) {
    if (epilogue == EPI_RS) return (int)cudaErrorInvalidValue;
    return gemm_fp8_launch(A8, sa, W8, sw, C, R, M, N, K, ldc, ldr, epilogue, status, num_sms, st, TpArgs{});
}

// Tensor-parallel form: with EPI_RS every output row goes to its owner rank's receive buffer
// (`tp_blob` = the communicator's TpArgs, rows_per_rank rows per owner), as in pie_gemm_bf16_tp.
PIE_API int pie_gemm_fp8_blockscaled_tp(const void* A8, const float* sa, const void* W8, const float* sw, void* C,
                                        int M, int N, int K, int ldc, int epilogue, const void* tp_blob,
                                        int rows_per_rank, int* status, int num_sms, cudaStream_t st) {
    TpArgs tp = *reinterpret_cast<const TpArgs*>(tp_blob);
    tp.rows_per_rank = rows_per_rank;
    tp.gated = 0;
    if (epilogue == EPI_RS && (rows_per_rank % 32 || rows_per_rank <= 0)) return (int)cudaErrorInvalidValue;
    return gemm_fp8_launch(A8, sa, W8, sw, C, nullptr, M, N, K, ldc, 0, epilogue, status, num_sms, st, tp);
}

// Weight rows of a tile: where one round of the machine will do, as many as leave 64 tiles or so - what a round takes hardly depends on
// its tiles' rows, and more CTAs ask L2 for the same rows of the batch - else as few as leave the rounds as few. Whole quarters of 32 (two
// warps each), or parts of them where that would end at 128. Measured at 4 / 48 rows (us): 5120 x 25600 in tiles of 24 rows (two rounds)
// 91 / 110, of 40 49 / 57, of 64 48 / 56; 6144 x 4096 of 48 12.6 / 13.0, of 64 11.4 / 12.3, of 96 10.1 / 11.6; 8192 x 8192 of 64 19.3 / 21.0, of
// 128 17.2 / 20.8; 51200 x 5120 of 88 (four rounds) 42.0 / 50.5, of 128 41.5 / 44.2. At 1 / 64 rows: 28672 x 5120 of 104 24.4 / 29.9, of 112
// 24.7 / 29.9, of 128 25.8 / 30.2; 57344 x 5120 (four rounds) of 104 45.9 / 55.9, of 112 47.8 / 56.1, of 128 49.1 / 57.9; 24576 x 5120 of 88
// 22.6 / 29.4, of 96 22.4 / 28.8. Several rounds of a short K are most of all their tiles' starts and ends, and want few tiles: 27648 x 512 of
// 96 5.2 / 7.3, of 128 4.8 / 6.2, 27648 x 2048 12.0 / 14.5 and 10.9 / 14.0, 57344 x 1536 of 104 15.6 / 21.2, of 128 15.5 / 20.3, but 57344 x 2048
// 20.6 / 26.5 and 21.1 / 25.7.
static int fp8_skinny_height(int N, int K, int num_sms) {
    const int rounds = ((N + GEMM_BM - 1) / GEMM_BM + num_sms - 1) / num_sms;
    if (rounds > 1 && K <= (rounds == 2 ? 2048 : 1536)) return GEMM_BM;
    int least = (N + rounds * num_sms - 1) / (rounds * num_sms);
    if (rounds == 1) least = std::min(GEMM_BM, std::max(least, (N + 63) / 64));
    const int height = (least + 31) / 32 * 32;
    if (height < GEMM_BM) return height;
    const int step = rounds > 1 ? 8 : 16;
    return (least + step - 1) / step * step;
}

// Up to 64 rows run here, with the bits of the kernel above. Measured over 128 to 51200 features and a K of 512 to 25600, quantiser and
// product (us, here / above): 1 x 1024 x 1024 4.5 / 6.7, 64 x 1024 x 1024 5.9 / 6.5, 64 x 5120 x 1024 6.5 / 8.1, 16 x 2048 x 8192
// 19.4 / 21.4, 48 x 2048 x 8192 21.7 / 21.9. With few features a launch takes what one tile's sums over K take, and from 49 rows on these are
// the longer ones here: 56 x 1024 x 4096 13.7 / 13.3, 64 x 1536 x 2048 9.2 / 8.8, 64 x 2048 x 8192 24.4 / 22.5, and 24.8 / 24.4 with 2560
// features. Fewer features or a shorter K are not worth the set-up.
static bool fp8_skinny_takes(int M, int N, int K) {
    return M <= 64 && N >= 128 && K >= 512 && !(M > 48 && N <= 2048 && K >= 2048);
}

template <int EPI>
static int launch_fp8_skinny(const void* A8, const float* sa, const void* W8, const float* sw, void* C, const void* R, int M, int N, int K,
                             int ldc, int ldr, int* status, int num_sms, cudaStream_t st) {
    const int height = fp8_skinny_height(N, K, num_sms);
    CUtensorMap tw, tx;
    if (make_tma_2d_u8(&tw, W8, N, K, K, height) != 0) return (int)cudaErrorInvalidValue;
    if (make_tma_2d_u8(&tx, A8, M, K, K, M) != 0) return (int)cudaErrorInvalidValue;      // the box ends with the batch
    auto kern = gemm_fp8_skinny_kernel<EPI>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F8S_SMEM);
    if (e != cudaSuccess) return (int)e;
    const int tiles = (N + height - 1) / height;
    // an MMA reads 128 rows from the last slot's start, too: they have to lie in the ring
    const uint32_t slot = (uint32_t)(height + (M + 15) / 16 * 16) * F8_BK;
    const int stages = (int)std::min({(uint32_t)F8S_MAX_STAGES, F8S_RING / slot, (F8S_RING - F8S_MMA_BYTES) / slot + 1});
    e = launch_pdl(kern, dim3(std::min(tiles, num_sms)), dim3(F8S_THREADS), F8S_SMEM, st, tw, tx, sa, sw, (bf16*)C, (const bf16*)R, M, N, K,
                   ldc, ldr, status, stages, height);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

static int gemm_fp8_launch(const void* A8, const float* sa, const void* W8, const float* sw, void* C,
                           const void* R, int M, int N, int K, int ldc, int ldr, int epilogue, int* status,
                           int num_sms, cudaStream_t st, const TpArgs& tp) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 16 || N % 16 || (epilogue != EPI_RS && ldc % 8) || (epilogue == EPI_RESIDUAL && ldr % 8))
        return (int)cudaErrorInvalidValue;
    if (epilogue == EPI_SWIGLU && N % 32) return (int)cudaErrorInvalidValue;
    if (fp8_skinny_takes(M, N, K)) {
        if (epilogue == EPI_STORE) return launch_fp8_skinny<EPI_STORE>(A8, sa, W8, sw, C, R, M, N, K, ldc, ldr, status, num_sms, st);
        if (epilogue == EPI_RESIDUAL) return launch_fp8_skinny<EPI_RESIDUAL>(A8, sa, W8, sw, C, R, M, N, K, ldc, ldr, status, num_sms, st);
        if (epilogue == EPI_SWIGLU) return launch_fp8_skinny<EPI_SWIGLU>(A8, sa, W8, sw, C, R, M, N, K, ldc, ldr, status, num_sms, st);
    }
    const int tm = (M + GEMM_BM - 1) / GEMM_BM;
    // tile width: the widest of {128, 112, ..., 16} whose tile count fills its waves best
    int bn = 128;
    double best = 1e30;
    for (int cand = 128; cand >= 16; cand -= 16) {
        const long tiles = (long)tm * ((N + cand - 1) / cand);
        const long waves = (tiles + num_sms - 1) / num_sms;
        const double cost = (double)waves * (cand + 24);
        if (cost < best) { best = cost; bn = cand; }
    }
    const int bt = bn <= 64 ? 64 : 128;
    CUtensorMap ta, tb;
    if (make_tma_2d_u8(&ta, A8, M, K, K, GEMM_BM) != 0) return (int)cudaErrorInvalidValue;
    if (make_tma_2d_u8(&tb, W8, N, K, K, bn) != 0) return (int)cudaErrorInvalidValue;
    const long tiles = (long)tm * ((N + bn - 1) / bn);
    const int grid = (int)(tiles < num_sms ? tiles : num_sms);
#define GO(BN_, EPI_)                                                                                         \
    {                                                                                                         \
        auto kern = gemm_fp8_kernel<BN_, EPI_>;                                                               \
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,               \
                                             (int)Fp8Cfg<BN_>::SMEM_BYTES);                                   \
        if (e != cudaSuccess) return (int)e;                                                                  \
        kern<<<grid, GEMM_THREADS, Fp8Cfg<BN_>::SMEM_BYTES, st>>>(ta, tb, sa, sw, (bf16*)C, (const bf16*)R, M, N, K, \
                                                                  ldc, ldr, status, bn, tp);                  \
        return (int)cudaGetLastError();                                                                       \
    }
#define GOE(BN_)                                                  \
    switch (epilogue) {                                           \
        case EPI_STORE: GO(BN_, EPI_STORE)                        \
        case EPI_RESIDUAL: GO(BN_, EPI_RESIDUAL)                  \
        case EPI_SWIGLU: GO(BN_, EPI_SWIGLU)                      \
        case EPI_RS: GO(BN_, EPI_RS)                              \
        default: return (int)cudaErrorInvalidValue;               \
    }
    if (bt == 128) { GOE(128) } else { GOE(64) }
#undef GOE
#undef GO
    return (int)cudaErrorInvalidValue;
}
