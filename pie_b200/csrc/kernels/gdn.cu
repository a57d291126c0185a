// Recurrent mixers of the hybrid models. Mamba-2 (state-space) is at the end of the file; first the
// Gated DeltaNet (linear attention) mixer: the short causal convolution over the
// q | k | v channels with its per-slot tail state, and the gated delta-rule recurrence with the gated
// RMSNorm on its output. One launch serves a ragged batch (prefill chunks and decode rows alike): the
// state of every request lives in its slot of the recurrent-state cache and is carried from fire to fire.
//
//   conv:       y[t, c] = silu( sum_j w[c, j] * x[t - (K-1) + j, c] ), inputs before the first token of
//               this fire come from the slot's last K-1 inputs (zeros after a reset)
//   recurrence: per value head, S in R^{dk x dv} (fp32):
//               S <- S * exp(g);  delta = (v - k^T S) * beta;  S <- S + k (x) delta;  o = q^T S
//               with q, k L2-normalised (q also scaled by dk^-1/2), beta = sigmoid(b),
//               g = -exp(A_log) * softplus(a + dt_bias)
//   output:     out = RMSNorm(o) * w_norm * silu(z)
//
// Five launches for prompts, three for decode: gdn_prep (convolution, SiLU, unit q and k), the convolution's tail,
// [gdn_groups, gdn_walk, gdn_norm] or gdn_step. All arithmetic on the state is 32-bit and exact for any chunking of a
// sequence up to the order of sums.
//
// Counterpart in the reference (behaviour only): driver/cuda/src/kernels/gated_delta_net.cu
// (l2norm, g / beta, recurrent_step*), driver/cuda/src/recurrent_state_cache.cpp (slot layout, slot copy).
#include <type_traits>

#include "common.cuh"

namespace pie {

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

// x: [N, F] fused projection (first C columns are the convolved channels); state: [S, C, K-1] fp32.
template <int K>
__global__ void gdn_conv_kernel(const bf16* __restrict__ x, int x_stride, const bf16* __restrict__ w,
                                const bf16* __restrict__ bias, const float* __restrict__ state,
                                const int* __restrict__ qo_indptr,
                                const int* __restrict__ tok_req, const int* __restrict__ slots,
                                const int* __restrict__ reset, float* __restrict__ y, int n, int c) {
    const int ch = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (ch >= c || t >= n) return;
    const int r = tok_req[t];
    if (slots[r] < 0) return;          // a padding request of a decode graph's bucket: no state, no output
    const int first = qo_indptr[r];
    const int i = t - first;
    const bool fresh = reset[r] != 0;
    const float* st = state + ((size_t)slots[r] * c + ch) * (K - 1);
    float acc = bias ? __bfloat162float(bias[ch]) : 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int idx = i - (K - 1) + j;
        float v;
        if (idx >= 0) v = __bfloat162float(x[(size_t)(first + idx) * x_stride + ch]);
        else v = fresh ? 0.f : st[(K - 1) + idx];
        acc += __bfloat162float(w[ch * K + j]) * v;
    }
    y[(size_t)t * c + ch] = silu_f(acc);
}

// New tail of every request's slot: its last K-1 inputs (older ones come from the previous tail).
template <int K>
__global__ void gdn_conv_state_kernel(const bf16* __restrict__ x, int x_stride, float* __restrict__ state,
                                      const int* __restrict__ qo_indptr, const int* __restrict__ slots,
                                      const int* __restrict__ reset, int c) {
    const int ch = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    pdl_trigger();
    pdl_wait();
    if (ch >= c) return;
    const int first = qo_indptr[r], len = qo_indptr[r + 1] - first;
    if (len <= 0 || slots[r] < 0) return;
    float* st = state + ((size_t)slots[r] * c + ch) * (K - 1);
    const bool fresh = reset[r] != 0;
    float nv[K - 1];
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
        const int idx = len - (K - 1) + j;                 // position within this fire's rows
        if (idx >= 0) nv[j] = __bfloat162float(x[(size_t)(first + idx) * x_stride + ch]);
        else nv[j] = fresh ? 0.f : st[(K - 1) + idx];
    }
#pragma unroll
    for (int j = 0; j < K - 1; ++j) st[j] = nv[j];
}

constexpr int GDN_COEF = 40;               // numbers of a group of four tokens, see gdn_groups_kernel
constexpr int GDN_STAGE = 16;              // tokens of a stage of gdn_walk
constexpr int GDN_WARPS = 4;               // of gdn_walk
constexpr int GDN_STEP_TOKENS = 4;         // of a request that gdn_step still takes

// y = conv + SiLU over q | k | v; then q * rsqrt(q.q + 1e-6) * dk^-1/2 and k * rsqrt(k.k + 1e-6) per head. 128 channels (whole
// heads) of 16 tokens per block: a channel's inputs are read once and slide through registers, and the heads' norms are taken
// here, once, instead of by every value head's block for every token. Bound by memory: 2 bytes in and 4 out per value.
// 2500 tokens x 8192 channels: 173 us with one thread per value, 70 us like this. TILE: tokens of a block, fewer where there are
// few blocks.
template <int DK, int GDN_TILE>
__global__ void __launch_bounds__(128)
gdn_prep_kernel(const bf16* __restrict__ x, int x_stride, const bf16* __restrict__ w, const float* __restrict__ state,
                const int* __restrict__ qo_indptr, const int* __restrict__ tok_req, const int* __restrict__ slots,
                const int* __restrict__ reset, float* __restrict__ y, int n, int c, int qk) {
    __shared__ int s_first[GDN_TILE], s_slot[GDN_TILE], s_fresh[GDN_TILE];
    __shared__ float squares[4][GDN_TILE];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ch = blockIdx.x * 128 + threadIdx.x, t0 = blockIdx.y * GDN_TILE, len = min(GDN_TILE, n - t0);
    const bool own = ch < c;
    pdl_trigger();
    float wt[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) wt[j] = own ? __bfloat162float(w[ch * 4 + j]) : 0.f;
    pdl_wait();
    if (threadIdx.x < len) {
        const int r = tok_req[t0 + threadIdx.x];
        s_first[threadIdx.x] = qo_indptr[r];
        s_slot[threadIdx.x] = slots[r];
        s_fresh[threadIdx.x] = reset[r];
    }
    float in[GDN_TILE];
#pragma unroll
    for (int s = 0; s < GDN_TILE; ++s) in[s] = own && s < len ? __bfloat162float(x[(size_t)(t0 + s) * x_stride + ch]) : 0.f;
    __syncthreads();
    float v[GDN_TILE], sq[GDN_TILE], past[3] = {0.f, 0.f, 0.f};      // past: the three inputs before, oldest first
#pragma unroll
    for (int s = 0; s < GDN_TILE; ++s) {
        v[s] = 0.f;
        if (own && s < len && s_slot[s] >= 0) {
            const int i = t0 + s - s_first[s];
            if (s == 0 || i == 0) {
                const float* st = state + ((size_t)s_slot[s] * c + ch) * 3;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int at = i - 3 + j;                        // position within this fire's rows
                    past[j] = at >= 0 ? __bfloat162float(x[(size_t)(s_first[s] + at) * x_stride + ch]) : s_fresh[s] ? 0.f : st[3 + at];
                }
            }
            v[s] = silu_f(wt[0] * past[0] + wt[1] * past[1] + wt[2] * past[2] + wt[3] * in[s]);
            past[0] = past[1];
            past[1] = past[2];
            past[2] = in[s];
        }
        sq[s] = v[s] * v[s];
    }
    const float part = halving_sum<GDN_TILE, 32>(sq, lane);          // of token lane / (32 / TILE)
    if (lane % (32 / GDN_TILE) == 0) squares[wid][lane / (32 / GDN_TILE)] = part;
    __syncthreads();
    float scale = 1.f;                                               // of token lane % TILE
    if (ch < qk) {
        float sum = 0.f;
        for (int j = 0; j < DK / 32; ++j) sum += squares[wid / (DK / 32) * (DK / 32) + j][lane % GDN_TILE];
        scale = rsqrtf(sum + 1e-6f) * (ch < qk / 2 ? rsqrtf((float)DK) : 1.f);
    }
#pragma unroll
    for (int s = 0; s < GDN_TILE; ++s) {
        const float f = __shfl_sync(0xffffffffu, scale, s);
        if (own && s < len && s_slot[s] >= 0) y[(size_t)(t0 + s) * c + ch] = v[s] * f;
    }
}

// beta = sigmoid(b) and exp(g) of a token and value head
__device__ __forceinline__ float2 gdn_gates(const bf16* xr, int h, int hv, float decay_rate, float bias) {
    return make_float2(1.f / (1.f + __expf(-__bfloat162float(xr[h]))), __expf(decay_rate * softplus_f(__bfloat162float(xr[hv + h]) + bias)));
}

// Four tokens of a request at a time: with S the state before them, G(i, j) the product of the decays of tokens j + 1 .. i,
//   delta_i = beta_i v_i - beta_i G(i, -1) (S^T k_i) - sum_(j < i) beta_i G(i, j) (k_i . k_j) delta_j
//   o_i     = G(i, -1) (S^T q_i) + sum_(j <= i) G(i, j) (q_i . k_j) delta_j
//   S      <- G(3, -1) S + sum_j G(3, j) k_j delta_j^T
// so that all sums over the state's rows start from one state: their latency, and that of the lanes' exchange behind them, is
// paid once per four tokens. The factors that do not depend on a column are worked out here, one warp per (group, key head):
//   [0, 6) beta_i G(i, j) (k_i . k_j), j < i   [8, 24) G(i, j) (q_i . k_j), 4 i + j, 0 for j > i
//   [24, 28) G(i, -1)   [28, 32) beta_i G(i, -1)   [32, 36) beta_i   [36, 40) G(3, j)
// The group that starts at token t of request r lies at t / 4 + r. Missing tokens of a last group count as k = q = beta = 0.
template <int DK>
__global__ void __launch_bounds__(128)
gdn_groups_kernel(const float* __restrict__ y, const bf16* __restrict__ x, int x_stride, const float* __restrict__ a_log,
                  const float* __restrict__ dt_bias, const int* __restrict__ qo_indptr, const int* __restrict__ tok_req,
                  const int* __restrict__ slots, float* __restrict__ coef, int n, int c, int hk, int hv, int gates_at) {
    constexpr int E = DK / 32;
    __shared__ float dots[4][16];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, kh = blockIdx.y, t = blockIdx.x * 4 + wid;
    pdl_trigger();
    pdl_wait();
    if (t >= n) return;
    const int r = tok_req[t], first = qo_indptr[r], len = min(4, qo_indptr[r + 1] - t);
    if (((t - first) & 3) || slots[r] < 0) return;
    float q[4][E], k[4][E], d[16];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float* row = y + (size_t)(t + i) * c + kh * DK + lane + 32 * e;
            q[i][e] = i < len ? row[0] : 0.f;
            k[i][e] = i < len ? row[hk * DK] : 0.f;
        }
    int at = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j, ++at) {
            d[at] = 0.f;
#pragma unroll
            for (int e = 0; e < E; ++e) d[at] += k[i][e] * k[j][e];
        }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j, ++at) {
            d[at] = 0.f;
#pragma unroll
            for (int e = 0; e < E; ++e) d[at] += q[i][e] * k[j][e];
        }
    const float dot = halving_sum<16, 32>(d, lane);
    if ((lane & 1) == 0) dots[wid][lane >> 1] = dot;
    __syncwarp();
    for (int h = kh * (hv / hk); h < (kh + 1) * (hv / hk); ++h) {
        float2 mine = make_float2(0.f, 1.f);
        if (lane < len) mine = gdn_gates(x + (size_t)(t + lane) * x_stride + gates_at, h, hv, -__expf(a_log[h]), dt_bias[h]);
        float beta[4], g[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            beta[i] = __shfl_sync(0xffffffffu, mine.x, i);
            g[i] = __shfl_sync(0xffffffffu, mine.y, i);
        }
        float* dst = coef + ((size_t)(t / 4 + r) * hv + h) * GDN_COEF;
        for (int s = lane; s < GDN_COEF; s += 32) {
            int i, j;                                                // the factor is G(i, j) * f
            float f = 1.f;
            if (s < 6) { i = s < 1 ? 1 : s < 3 ? 2 : 3; j = s - i * (i - 1) / 2; f = dots[wid][s]; }
            else if (s < 8) { i = j = 0; f = 0.f; }
            else if (s < 24) { i = (s - 8) >> 2; j = (s - 8) & 3; f = j <= i ? dots[wid][6 + i * (i + 1) / 2 + j] : 0.f; }
            else if (s < 32) { i = s & 3; j = -1; }
            else if (s < 36) { i = j = s & 3; }
            else { i = 3; j = s & 3; }
            if (s < 6 || (s >= 28 && s < 36)) f *= i == 0 ? beta[0] : i == 1 ? beta[1] : i == 2 ? beta[2] : beta[3];
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (l > j && l <= i) f *= g[l];
            dst[s] = f;
        }
    }
}

// Sums of NV values over LPC lanes: halves change hands until lane g is left with the PER = NV / LPC sums from PER g on.
template <int NV, int LPC, int PER>
__device__ __forceinline__ void halving_sums(const float (&x)[NV], int g, float (&own)[PER]) {
    if constexpr (NV == PER) {
#pragma unroll
        for (int i = 0; i < PER; ++i) own[i] = x[i];
    } else {
        const bool up = g & (LPC / 2);
        float y[NV / 2];
#pragma unroll
        for (int i = 0; i < NV / 2; ++i) {
            const float keep = up ? x[i + NV / 2] : x[i], give = up ? x[i] : x[i + NV / 2];
            y[i] = keep + __shfl_xor_sync(0xffffffffu, give, LPC / 2);
        }
        halving_sums<NV / 2, LPC / 2, PER>(y, g, own);
    }
}

// The state's walk through a request's tokens, four at a time. A warp holds 8 columns of a head's state in registers: lane group
// lane / 8 two of them, lane g = lane % 8 the rows 4 (g + 8 i) + e. Columns never meet, so a head's columns are spread over
// dv / 32 blocks. o takes v's place in `y`; norm and gate, which span the columns, follow in gdn_norm_kernel.
// Bound by the chain from group to group (dot products, exchange, solution, update: 0.8 us) where few prompts run, else by the
// packed multiply-adds (13 per state element and four tokens) and the shared-memory reads beside them. One token at a time
// with block-wide sums, prompts of 1300 + 700 + 500 tokens x 32 heads of 128 x 128 took 3822 us, this form 415 us.
template <int DK, int COLS>
struct GdnStage {
    float q[GDN_STAGE][DK], k[GDN_STAGE][DK], v[GDN_STAGE][COLS], coef[GDN_STAGE / 4][GDN_COEF];
};

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0));
}

template <int DK, int LPC, int CPT>
__global__ void __launch_bounds__(GDN_WARPS * 32)
gdn_walk_kernel(float* __restrict__ y, const float* __restrict__ coef, float* __restrict__ rec_state,
                const int* __restrict__ qo_indptr, const int* __restrict__ slots, const int* __restrict__ reset, int hk, int hv,
                int dv) {
    constexpr int THREADS = GDN_WARPS * 32, COLS = THREADS / LPC * CPT, R = DK / LPC;
    constexpr int NV = 8 * CPT, PER = NV / LPC;                      // sums of a column group, of a lane
    static_assert(R % 4 == 0 && PER >= 1 && (PER <= CPT && CPT % PER == 0) && CPT % 2 == 0, "");
    using Stage = GdnStage<DK, COLS>;
    extern __shared__ __align__(16) uint8_t raw[];
    Stage* stage = reinterpret_cast<Stage*>(raw);
    const int r = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, g = lane % LPC;
    const int cl = (threadIdx.x / LPC) * CPT, c0 = blockIdx.z * COLS + cl;
    pdl_trigger();
    pdl_wait();
    const int first = qo_indptr[r], len = qo_indptr[r + 1] - first, slot = slots[r];
    if (len <= 0 || slot < 0) return;
    const int kh = h / (hv / hk), c = 2 * hk * DK + hv * dv;
    const float* Q = y + (size_t)first * c + kh * DK;
    float* V = y + (size_t)first * c + 2 * hk * DK + h * dv + blockIdx.z * COLS;
    const float* F = coef + ((size_t)(first / 4 + r) * hv + h) * GDN_COEF;
    auto fetch = [&](int t0, int b) {
        for (int i = threadIdx.x; i < GDN_STAGE * DK / 4; i += THREADS) {
            const int t = i / (DK / 4), at = i % (DK / 4) * 4;
            const bool ok = t0 + t < len;
            const float* src = ok ? Q + (size_t)(t0 + t) * c + at : Q;
            copy16_or_zero(&stage[b].q[t][at], src, ok);
            copy16_or_zero(&stage[b].k[t][at], src + hk * DK, ok);
        }
        for (int i = threadIdx.x; i < GDN_STAGE * COLS / 4; i += THREADS) {
            const int t = i / (COLS / 4), at = i % (COLS / 4) * 4;
            const bool ok = t0 + t < len;
            copy16_or_zero(&stage[b].v[t][at], ok ? V + (size_t)(t0 + t) * c + at : V, ok);
        }
        if (threadIdx.x < GDN_STAGE / 4 * (GDN_COEF / 4)) {
            const int m = threadIdx.x / (GDN_COEF / 4), at = threadIdx.x % (GDN_COEF / 4) * 4;
            const bool ok = t0 + 4 * m < len;
            copy16_or_zero(&stage[b].coef[m][at], ok ? F + (size_t)(t0 / 4 + m) * hv * GDN_COEF + at : F, ok);
        }
        asm volatile("cp.async.commit_group;\n");
    };
    fetch(0, 0);
    float* sp = rec_state + (((size_t)slot * hv + h) * DK) * dv + c0;
    const bool fresh = reset[r] != 0;
    F2 S[CPT][R / 2];                                                // two rows each
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
        const float* row = sp + (size_t)(4 * (g + LPC * (i / 2)) + 2 * (i & 1)) * dv;
#pragma unroll
        for (int cc = 0; cc < CPT; cc += 2) {
            float2 a = make_float2(0.f, 0.f), b = a;
            if (!fresh) {
                a = *reinterpret_cast<const float2*>(row + cc);
                b = *reinterpret_cast<const float2*>(row + dv + cc);
            }
            S[cc][i] = f2(a.x, b.x);
            S[cc + 1][i] = f2(a.y, b.y);
        }
    }
    for (int t0 = 0, b = 0; t0 < len; t0 += GDN_STAGE, b ^= 1) {
        if (t0 + GDN_STAGE < len) {
            fetch(t0 + GDN_STAGE, b ^ 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const Stage& st = stage[b];
#pragma unroll 1
        for (int m = 0; m < GDN_STAGE / 4 && t0 + 4 * m < len; ++m) {
            F2 k[4][R / 2];
            float sums[NV];                                          // S^T k_i, then S^T q_i: CPT i + column
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                F2 ya[CPT], za[CPT];
#pragma unroll
                for (int cc = 0; cc < CPT; ++cc) ya[cc] = za[cc] = f2(0.f);
#pragma unroll
                for (int p = 0; p < R / 4; ++p) {
                    const float4 kv = reinterpret_cast<const float4*>(st.k[4 * m + i])[g + LPC * p];
                    const float4 qv = reinterpret_cast<const float4*>(st.q[4 * m + i])[g + LPC * p];
                    k[i][2 * p] = f2(kv.x, kv.y);
                    k[i][2 * p + 1] = f2(kv.z, kv.w);
                    const F2 q0 = f2(qv.x, qv.y), q1 = f2(qv.z, qv.w);
#pragma unroll
                    for (int cc = 0; cc < CPT; ++cc) {
                        ya[cc] = fma2(k[i][2 * p + 1], S[cc][2 * p + 1], fma2(k[i][2 * p], S[cc][2 * p], ya[cc]));
                        za[cc] = fma2(q1, S[cc][2 * p + 1], fma2(q0, S[cc][2 * p], za[cc]));
                    }
                }
#pragma unroll
                for (int cc = 0; cc < CPT; ++cc) {
                    float lo, hi;
                    unpack2(ya[cc], lo, hi);
                    sums[CPT * i + cc] = lo + hi;
                    unpack2(za[cc], lo, hi);
                    sums[4 * CPT + CPT * i + cc] = lo + hi;
                }
            }
            // halves change hands: lane g ends up with sums PER g and on, the first half of the lanes those of k
            float own[PER];
            halving_sums<NV, LPC, PER>(sums, g, own);
            const float* f = st.coef[m];
            float delta[4][CPT];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int cc = 0; cc < CPT; ++cc) {
                    const float s = __shfl_sync(0xffffffffu, own[(CPT * i + cc) % PER], lane - g + (CPT * i + cc) / PER);
                    float dl = f[32 + i] * st.v[4 * m + i][cl + cc] - f[28 + i] * s;
#pragma unroll
                    for (int j = 0; j < i; ++j) dl -= f[i * (i - 1) / 2 + j] * delta[j][cc];
                    delta[i][cc] = dl;
                }
            }
            const int at = (g - LPC / 2) * PER, i_o = at / CPT, c_o = at % CPT;
            if (g >= LPC / 2 && t0 + 4 * m + i_o < len) {
                const float4 w = *reinterpret_cast<const float4*>(f + 8 + 4 * i_o);
                const float gi = f[24 + i_o];
#pragma unroll
                for (int e = 0; e < PER; ++e) {
                    float d[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        d[j] = delta[j][e];
#pragma unroll
                        for (int cc = PER; cc < CPT; cc += PER)
                            if (c_o == cc) d[j] = delta[j][cc + e];
                    }
                    V[(size_t)(t0 + 4 * m + i_o) * c + cl + c_o + e] = gi * own[e] + w.x * d[0] + w.y * d[1] + w.z * d[2] + w.w * d[3];
                }
            }
            const F2 all = f2(f[27]);
#pragma unroll
            for (int cc = 0; cc < CPT; ++cc) {
                F2 e[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) e[j] = f2(f[36 + j] * delta[j][cc]);
#pragma unroll
                for (int i = 0; i < R / 2; ++i) {
                    F2 s = mul2(all, S[cc][i]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) s = fma2(k[j][i], e[j], s);
                    S[cc][i] = s;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
        float* row = sp + (size_t)(4 * (g + LPC * (i / 2)) + 2 * (i & 1)) * dv;
#pragma unroll
        for (int cc = 0; cc < CPT; cc += 2) {
            float a0, b0, a1, b1;
            unpack2(S[cc][i], a0, b0);
            unpack2(S[cc + 1][i], a1, b1);
            *reinterpret_cast<float2*>(row + cc) = make_float2(a0, a1);
            *reinterpret_cast<float2*>(row + dv + cc) = make_float2(b0, b1);
        }
    }
}

// out = RMSNorm(o) * w_norm * silu(z), one warp per (token, value head)
__global__ void __launch_bounds__(256)
gdn_norm_kernel(const float* __restrict__ y, const bf16* __restrict__ x, int x_stride, const bf16* __restrict__ norm_w,
                const int* __restrict__ tok_req, const int* __restrict__ slots, bf16* __restrict__ out, int n, int c, int qk, int hv,
                int dv, float eps) {
    const int lane = threadIdx.x & 31;
    const long at = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_trigger();
    pdl_wait();
    if (at >= (long)n * hv) return;
    const int t = (int)(at / hv), h = (int)(at % hv);
    if (slots[tok_req[t]] < 0) return;
    const float* o = y + (size_t)t * c + qk + h * dv;
    const bf16* z = x + (size_t)t * x_stride + c + h * dv;
    float v[8], zz[8], ms = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const bool ok = 32 * i < dv;
        v[i] = ok ? o[lane + 32 * i] : 0.f;
        zz[i] = ok ? __bfloat162float(z[lane + 32 * i]) : 0.f;
        ms += v[i] * v[i];
    }
    const float f = rsqrtf(warp_sum(ms) / (float)dv + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (32 * i < dv)
            out[((size_t)t * hv + h) * dv + lane + 32 * i] =
                __float2bfloat16(v[i] * f * __bfloat162float(norm_w[lane + 32 * i]) * silu_f(zz[i]));
}

// Decode: a block per (request, value head) with up to 4 LANES columns, four per lane, an eighth of the rows per group of LANES
// threads: the whole state is requested in 16-byte loads before anything waits for it. Both sums of a token run over the old state,
//   delta = beta (v - exp(g) S^T k),  o = exp(g) S^T q + (q . k) delta,  S <- exp(g) S + k delta^T.
// Bound by memory (the state in and out). 40 requests x 32 heads of 128 x 128: 65.7 us token-serial with block-wide sums over
// 64 rows per lane, 33 us like this (5.1 TB/s). Any number of tokens per request is right here.
template <int DK, int LANES>
__global__ void __launch_bounds__(8 * LANES)
gdn_step_kernel(const float* __restrict__ y, const bf16* __restrict__ x, int x_stride, const float* __restrict__ a_log,
                const float* __restrict__ dt_bias, const bf16* __restrict__ norm_w, float* __restrict__ rec_state,
                const int* __restrict__ qo_indptr, const int* __restrict__ slots, const int* __restrict__ reset,
                bf16* __restrict__ out, int hk, int hv, int dv, float eps) {
    constexpr int GROUPS = 8, ROWS = DK / GROUPS;
    __shared__ __align__(16) float sq[DK], sk[DK], part_y[GROUPS][4 * LANES], part_z[GROUPS][4 * LANES];
    __shared__ float red[32];
    const int r = blockIdx.x, h = blockIdx.y, lane = threadIdx.x % LANES, rg = threadIdx.x / LANES, tid = threadIdx.x;
    const bool own = lane * 4 < dv;        // columns past dv are zeros that nobody stores
    pdl_trigger();
    pdl_wait();
    const int first = qo_indptr[r], len = qo_indptr[r + 1] - first, slot = slots[r];
    if (len <= 0 || slot < 0) return;      // a padding request of a decode graph's bucket: no state, no output
    const int kh = h / (hv / hk), c = 2 * hk * DK + hv * dv;
    float* sp = rec_state + (((size_t)slot * hv + h) * DK + rg * ROWS) * dv + lane * 4;
    float4 S[ROWS];
    if (reset[r] || !own) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) S[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) S[i] = *reinterpret_cast<const float4*>(sp + (size_t)i * dv);
    }
    const float decay_rate = -__expf(a_log[h]), bias = dt_bias[h];
    for (int t = first; t < first + len; ++t) {
        const float* row = y + (size_t)t * c;
        float qk = 0.f;
        for (int i = tid; i < DK; i += 8 * LANES) {
            const float q = row[kh * DK + i], k = row[hk * DK + kh * DK + i];
            sq[i] = q;
            sk[i] = k;
            qk += q * k;
        }
        const float2 gates = gdn_gates(x + (size_t)t * x_stride + c + hv * dv, h, hv, decay_rate, bias);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (own) v = *reinterpret_cast<const float4*>(row + 2 * hk * DK + h * dv + lane * 4);
        qk = block_sum(qk, red);
        float4 ys = make_float4(0.f, 0.f, 0.f, 0.f), zs = ys;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const float k = sk[rg * ROWS + i], q = sq[rg * ROWS + i];
            ys.x += k * S[i].x; ys.y += k * S[i].y; ys.z += k * S[i].z; ys.w += k * S[i].w;
            zs.x += q * S[i].x; zs.y += q * S[i].y; zs.z += q * S[i].z; zs.w += q * S[i].w;
        }
        *reinterpret_cast<float4*>(&part_y[rg][lane * 4]) = ys;
        *reinterpret_cast<float4*>(&part_z[rg][lane * 4]) = zs;
        __syncthreads();
        ys = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < GROUPS; ++j) {
            const float4 p = *reinterpret_cast<const float4*>(&part_y[j][lane * 4]);
            ys.x += p.x; ys.y += p.y; ys.z += p.z; ys.w += p.w;
        }
        const float4 d = make_float4((v.x - gates.y * ys.x) * gates.x, (v.y - gates.y * ys.y) * gates.x,
                                     (v.z - gates.y * ys.z) * gates.x, (v.w - gates.y * ys.w) * gates.x);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const float k = sk[rg * ROWS + i];
            S[i].x = gates.y * S[i].x + k * d.x; S[i].y = gates.y * S[i].y + k * d.y;
            S[i].z = gates.y * S[i].z + k * d.z; S[i].w = gates.y * S[i].w + k * d.w;
        }
        constexpr int OUT = LANES < 32 ? 32 : LANES;       // threads that have all columns: output, its norm and gate
        float o[4], ms = 0.f;
        if (tid < OUT) {
            zs = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < GROUPS; ++j) {
                const float4 p = *reinterpret_cast<const float4*>(&part_z[j][lane * 4]);
                zs.x += p.x; zs.y += p.y; zs.z += p.z; zs.w += p.w;
            }
            o[0] = gates.y * zs.x + qk * d.x; o[1] = gates.y * zs.y + qk * d.y;
            o[2] = gates.y * zs.z + qk * d.z; o[3] = gates.y * zs.w + qk * d.w;
            ms = o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3];
#pragma unroll
            for (int s = (LANES < 32 ? LANES : 32) / 2; s; s >>= 1) ms += __shfl_xor_sync(0xffffffffu, ms, s);
        }
        if constexpr (LANES > 32) {
            __syncthreads();               // `red` has been read
            if (lane % 32 == 0 && tid < OUT) red[tid / 32] = ms;
            __syncthreads();
            ms = red[0] + red[1];
        }
        if (tid < OUT) {
            const float f = rsqrtf(ms / (float)dv + eps);
            const bf16* z = x + (size_t)t * x_stride + c + h * dv + lane * 4;
            bf16* dst = out + ((size_t)t * hv + h) * dv + lane * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (own && tid < LANES) dst[i] = __float2bfloat16(o[i] * f * __bfloat162float(norm_w[lane * 4 + i]) * silu_f(__bfloat162float(z[i])));
        }
        __syncthreads();                   // the partial sums and q, k are rewritten by the next token
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (own) *reinterpret_cast<float4*>(sp + (size_t)i * dv) = S[i];
}

// Mamba-2 state update: grid (requests, heads), block = head_dim threads; thread p holds S[p, :] (NS values)
// in registers. conv: [N, inner + 2 * groups * NS] (x | B | C after the convolution); x: the projection
// [N, z | x B C | dt] for dt; y: [N, inner] fp32 (gate and norm follow outside: they span all heads).
template <int NS>
__global__ void __launch_bounds__(256)
mamba2_ssm_kernel(const float* __restrict__ conv, const bf16* __restrict__ x, int x_stride,
                  const float* __restrict__ a_log, const float* __restrict__ dt_bias, const float* __restrict__ d_skip,
                  float* __restrict__ rec_state, const int* __restrict__ qo_indptr, const int* __restrict__ slots,
                  const int* __restrict__ reset, float* __restrict__ y, int heads, int head_dim, int groups) {
    __shared__ float sb[NS], scv[NS], sc[1];
    const int r = blockIdx.x, h = blockIdx.y, p = threadIdx.x;
    const int first = qo_indptr[r], len = qo_indptr[r + 1] - first;
    if (len <= 0 || slots[r] < 0) return;
    const int inner = heads * head_dim, c = inner + 2 * groups * NS;
    const int g = h / (heads / groups);
    float* sp = rec_state + (((size_t)slots[r] * heads + h) * head_dim + p) * NS;
    float S[NS];
    if (reset[r]) {
#pragma unroll
        for (int i = 0; i < NS; ++i) S[i] = 0.f;
    } else {
#pragma unroll
        for (int i = 0; i < NS; ++i) S[i] = sp[i];
    }
    const float a = -__expf(a_log[h]), bias = dt_bias[h], dsk = d_skip[h];
    for (int t = 0; t < len; ++t) {
        const size_t row = (size_t)(first + t);
        const float* cr = conv + row * c;
        for (int i = p; i < NS; i += blockDim.x) {
            sb[i] = cr[inner + g * NS + i];
            scv[i] = cr[inner + groups * NS + g * NS + i];
        }
        if (p == 0) sc[0] = softplus_f(__bfloat162float(x[row * x_stride + inner + c + h]) + bias);
        __syncthreads();
        const float dt = sc[0], xv = cr[h * head_dim + p];
        const float decay = __expf(dt * a), dx = dt * xv;
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            S[i] = S[i] * decay + dx * sb[i];
            acc += S[i] * scv[i];
        }
        y[row * inner + h * head_dim + p] = acc + dsk * xv;
        __syncthreads();                                   // sb / scv / sc are rewritten by the next token
    }
#pragma unroll
    for (int i = 0; i < NS; ++i) sp[i] = S[i];
}

// dst slot <- src slot in both caches of every linear layer (fork of a context).
__global__ void gdn_copy_slot_kernel(float* __restrict__ buf, size_t layer_stride, size_t slot_elems, int layers,
                                     int src, int dst) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= slot_elems) return;
    for (int l = 0; l < layers; ++l) {
        float* base = buf + (size_t)l * layer_stride;
        base[(size_t)dst * slot_elems + i] = base[(size_t)src * slot_elems + i];
    }
}

}  // namespace pie

// The block-per-head step takes fires of short requests (`longest`: most tokens of one), others are walked through in fours: the
// step's chain grows with every token, the walk's with every four. Measured, step against walk: 64 requests of 32 heads of
// 128 x 128 with 3 tokens 108 / 126 us, 4 tokens 125 / 128, 6 tokens 168 / 159; one request with 4 tokens 16.0 / 15.9, 6 tokens 19.6 / 16.9. Of
// 64 x 64 heads, 64 requests with one token: 14 / 30 us.
static bool gdn_steps(int longest) { return longest <= pie::GDN_STEP_TOKENS; }

// 32-bit numbers of workspace (`coef`) that a fire needs.
PIE_API long pie_gdn_coef_elems(int n, int r, int longest, int hv) {
    return gdn_steps(longest) ? 0 : ((long)n / 4 + r + 1) * hv * pie::GDN_COEF;
}

template <int DK>
static int launch_gdn(const void* x, int x_stride, const void* conv_w, const float* a_log, const float* dt_bias, const void* norm_w,
                      float* conv_state, float* rec_state, const int* qo_indptr, const int* tok_req, const int* slots,
                      const int* reset, float* y, float* coef, void* out, int n, int r, int longest, int hk, int hv, int dv, float eps,
                      cudaStream_t st) {
    using namespace pie;
    const int qk = 2 * hk * DK, c = qk + hv * dv;
    const bf16* xb = static_cast<const bf16*>(x);
    const bf16* nw = static_cast<const bf16*>(norm_w);
    // tokens of a block of gdn_prep: fewer where blocks are few. The mixer over 8192 channels: 40 decode rows 43 us with 4 and 53
    // with 16, a prompt of 61 tokens 28 and 31, of 150 tokens 48 and 49, from 300 on the same
    const int tile = (long)n * ((c + 127) / 128) <= 16L * PIE_SMS * 4 ? 4 : 16;
    cudaError_t e = launch_pdl(tile == 4 ? gdn_prep_kernel<DK, 4> : gdn_prep_kernel<DK, 16>, dim3((c + 127) / 128, (n + tile - 1) / tile),
                               dim3(128), 0, st, xb, x_stride, static_cast<const bf16*>(conv_w), conv_state, qo_indptr, tok_req, slots,
                               reset, y, n, c, qk);
    if (e == cudaSuccess)
        e = launch_pdl(gdn_conv_state_kernel<4>, dim3((c + 127) / 128, r), dim3(128), 0, st, xb, x_stride, conv_state, qo_indptr, slots,
                       reset, c);
    if (e != cudaSuccess) return (int)e;
    if (gdn_steps(longest)) {
        auto kern = dv <= 32 ? gdn_step_kernel<DK, 8> : dv <= 64 ? gdn_step_kernel<DK, 16> : gdn_step_kernel<DK, 32>;
        if constexpr (DK < 128)
            if (dv > 128) kern = gdn_step_kernel<DK, 64>;
        const int threads = dv <= 32 ? 64 : dv <= 64 ? 128 : dv <= 128 ? 256 : 512;
        e = launch_pdl(kern, dim3(r, hv), dim3(threads), 0, st, y, xb, x_stride, a_log, dt_bias, nw, rec_state, qo_indptr, slots, reset,
                       static_cast<bf16*>(out), hk, hv, dv, eps);
        return (int)(e != cudaSuccess ? e : cudaGetLastError());
    }
    if (!coef) return (int)cudaErrorInvalidValue;
    e = launch_pdl(gdn_groups_kernel<DK>, dim3((n + 3) / 4, hk), dim3(128), 0, st, y, xb, x_stride, a_log, dt_bias, qo_indptr, tok_req,
                   slots, coef, n, c, hk, hv, c + hv * dv);
    auto walk = [&](auto lpc, auto cpt) {
        constexpr int LPC = decltype(lpc)::value, CPT = decltype(cpt)::value, COLS = GDN_WARPS * 32 / LPC * CPT;
        const int smem = 2 * (int)sizeof(GdnStage<DK, COLS>);
        auto kern = gdn_walk_kernel<DK, LPC, CPT>;
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess)
            e = launch_pdl(kern, dim3(r, hv, dv / COLS), dim3(GDN_WARPS * 32), smem, st, y, coef, rec_state, qo_indptr, slots, reset, hk, hv, dv);
    };
    // Four columns per lane read shared memory half as often as two, but leave half the warps: they win where there are plenty
    // (26 prompts of 100 tokens: 406 against 482 us for the mixer) and lose where a few long prompts run (1300 + 700 + 500 tokens:
    // 679 against 581 us).
    const bool wide = DK == 128 && dv % 64 == 0 && (long)r * hv * (dv / 64) >= 4 * PIE_SMS;
    if (wide) walk(std::integral_constant<int, 8>{}, std::integral_constant<int, DK == 128 ? 4 : 2>{});
    else walk(std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{});
    if (e == cudaSuccess)
        e = launch_pdl(gdn_norm_kernel, dim3((unsigned)(((long)n * hv + 7) / 8)), dim3(256), 0, st, y, xb, x_stride, nw, tok_req, slots,
                       static_cast<bf16*>(out), n, c, qk, hv, dv, eps);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

PIE_API int pie_gdn_mixer(const void* x, int x_stride, const void* conv_w, const float* a_log, const float* dt_bias,
                          const void* norm_w, float* conv_state, float* rec_state, const int* qo_indptr,
                          const int* tok_req, const int* slots, const int* reset, float* conv_scratch, float* coef,
                          void* out, int n, int r, int longest, int hk, int hv, int dk, int dv, int kernel, float eps, cudaStream_t st) {
    using namespace pie;
    if (n <= 0 || r <= 0) return 0;
    if (kernel != 4) return (int)cudaErrorInvalidValue;
    if (dv % 32 != 0 || dv > 256 || (dk == 128 && dv > 128) || hv % hk != 0) return (int)cudaErrorInvalidValue;
    auto launch = dk == 32 ? launch_gdn<32> : dk == 64 ? launch_gdn<64> : dk == 128 ? launch_gdn<128> : nullptr;
    if (!launch) return (int)cudaErrorInvalidValue;
    return launch(x, x_stride, conv_w, a_log, dt_bias, norm_w, conv_state, rec_state, qo_indptr, tok_req, slots, reset, conv_scratch, coef,
                  out, n, r, longest, hk, hv, dv, eps, st);
}

PIE_API int pie_mamba2_mixer(const void* x, int x_stride, const void* conv_w, const void* conv_b, const float* a_log,
                             const float* dt_bias, const float* d_skip, float* conv_state, float* rec_state,
                             const int* qo_indptr, const int* tok_req, const int* slots, const int* reset,
                             float* conv_scratch, float* y, int n, int r, int heads, int head_dim, int state, int groups,
                             cudaStream_t st) {
    using namespace pie;
    if (n <= 0 || r <= 0) return 0;
    if (head_dim > 256 || heads % groups != 0) return (int)cudaErrorInvalidValue;
    const int inner = heads * head_dim, c = inner + 2 * groups * state;
    const bf16* xb = static_cast<const bf16*>(x) + inner;          // the convolved channels follow the gate
    dim3 cg((c + 127) / 128, n);
    gdn_conv_kernel<4><<<cg, 128, 0, st>>>(xb, x_stride, static_cast<const bf16*>(conv_w), static_cast<const bf16*>(conv_b),
                                           conv_state, qo_indptr, tok_req, slots, reset, conv_scratch, n, c);
    dim3 sg((c + 127) / 128, r);
    gdn_conv_state_kernel<4><<<sg, 128, 0, st>>>(xb, x_stride, conv_state, qo_indptr, slots, reset, c);
    dim3 rg(r, heads);
    const bf16* x0 = static_cast<const bf16*>(x);
#define PIE_MAMBA_LAUNCH(NSV)                                                                                   \
    mamba2_ssm_kernel<NSV><<<rg, head_dim, 0, st>>>(conv_scratch, x0, x_stride, a_log, dt_bias, d_skip, rec_state, \
                                                    qo_indptr, slots, reset, y, heads, head_dim, groups)
    if (state == 16) PIE_MAMBA_LAUNCH(16);
    else if (state == 64) PIE_MAMBA_LAUNCH(64);
    else if (state == 128) PIE_MAMBA_LAUNCH(128);
    else return (int)cudaErrorInvalidValue;
#undef PIE_MAMBA_LAUNCH
    return (int)cudaGetLastError();
}

PIE_API int pie_gdn_copy_slot(float* buf, long layer_stride, long slot_elems, int layers, int src, int dst,
                              cudaStream_t st) {
    if (slot_elems <= 0 || layers <= 0 || src == dst) return 0;
    pie::gdn_copy_slot_kernel<<<(unsigned)((slot_elems + 255) / 256), 256, 0, st>>>(buf, (size_t)layer_stride,
                                                                                    (size_t)slot_elems, layers, src, dst);
    return (int)cudaGetLastError();
}
