// Token sampling and probe kernels over bf16 logits.
//
// pie_sample: per row temperature, top-k, top-p, min-p, a seeded counter-based
// random stream and an optional vocabulary bitmask (constrained decoding), all
// on the device. The kept set is found exactly on the 16-bit order key of the
// bf16 logits with histograms of keys, then one token is drawn from the
// renormalised kept set with the Gumbel-max trick, so no sort, no probability
// row in memory and no host round trip is needed.
// Temperature <= 0 selects the arg-max (lowest index on ties).
//
// Reference behaviour: driver/cuda/src/kernels/sample_temp.cu:30-180 (Gumbel-max
// with hash noise, min-p), driver/cuda/src/kernels/sample_flashinfer.cu:19,86
// (top-k / top-p), driver/cuda/src/executor/executor.cpp:2741-2756 (logit masks
// are applied on the host there; here the sampler consumes them),
// driver/cuda/src/kernels/{logprobs,entropy}.cu (probes from unscaled logits).
#include <algorithm>

#include "tcgen05.cuh"

namespace pie {

constexpr int SAMPLE_THREADS = 512;
constexpr int SAMPLE_WARPS = SAMPLE_THREADS / 32;
constexpr int SAMPLE_CLUSTER = 8;                  // most CTAs of a row
constexpr int SAMPLE_BINS = SAMPLE_THREADS;        // one per thread
constexpr uint32_t NEG_INF2 = 0xFF80FF80u;         // two bf16 of -inf
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ uint32_t bf16_key(uint16_t bits) {
    return (bits & 0x8000u) ? (uint32_t)(uint16_t)~bits : (uint32_t)(bits | 0x8000u);
}
// Two bf16 as signed 16-bit numbers of the same order (order key ^ 0x8000 each).
__device__ __forceinline__ uint32_t sortable2(uint32_t w) { return w ^ (((w >> 15) & 0x00010001u) * 0x7FFFu); }
__device__ __forceinline__ float sortable_value(int s) { return __uint_as_float((uint32_t)(s < 0 ? s ^ 0x7FFF : s) << 16); }
__device__ __forceinline__ uint32_t f32_key(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float f32_of_key(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32));
    const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0u);
    return ((unsigned long long)hi << 32) | lo;
}
__device__ __forceinline__ void st_cluster_u64(uint32_t addr, unsigned long long v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// 2^(32 - n): x >> n is the high half of x times it. Arguments, so that they stay products.
struct SampleShift {
    uint32_t by9, by13, by16;
};

// Masses as whole numbers of 2^-40, NaN as bit 63.
constexpr unsigned long long NAN_UNITS = 1ull << 63;
__device__ __forceinline__ unsigned long long add_units(unsigned long long a, unsigned long long b) {
    return ((a & ~NAN_UNITS) + (b & ~NAN_UNITS)) | ((a | b) & NAN_UNITS);
}
__device__ __forceinline__ unsigned long long warp_add_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = add_units(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

struct SampleShared {
    unsigned long long red[SAMPLE_WARPS];
    unsigned long long slot[2][SAMPLE_CLUSTER];    // one word of each CTA of the row, two exchanges deep
    uint32_t cnt[SAMPLE_BINS], mass[3][SAMPLE_BINS];       // masses: whole numbers in three words
    uint32_t wcnt[SAMPLE_WARPS];
    float wmass[SAMPLE_WARPS];
    uint32_t best[4];                              // best score key of a Gumbel pass so far
    int hit;
    uint32_t base_cnt;
    float base_mass;
};

// One row, or a CTA's share of it: vectors of 8 bf16 at (i * cluster + rank) * SAMPLE_THREADS + thread. RESIDENT: they are
// kept in shared memory from the first pass on, each read by the thread that wrote it; else they are read again (L2) in every
// pass. Entries that the mask or the row's end excludes are -inf here, and `allowed` tells them from an -inf of the row where
// it matters.
template <bool RESIDENT>
struct SampleRow {
    const uint4* vec;
    const uint32_t* mask;
    uint4* kept;
    int nvec, cl, rank, count;

    __device__ __forceinline__ bool allowed(int idx) const {
        return idx < nvec * 8 && (!mask || ((mask[idx >> 5] >> (idx & 31)) & 1u));
    }
    __device__ __forceinline__ int index(int i) const { return (i * cl + rank) * SAMPLE_THREADS + (int)threadIdx.x; }
    __device__ __forceinline__ uint4 load(int v) const {
        uint4 p = make_uint4(NEG_INF2, NEG_INF2, NEG_INF2, NEG_INF2);
        if (v < nvec) {
            p = vec[v];
            if (mask) {
                const uint32_t ok = mask[v >> 2] >> ((v & 3) * 8);
                auto excluded = [&](uint32_t w, int k) {
                    if (!((ok >> k) & 1u)) w = (w & 0xFFFF0000u) | (NEG_INF2 & 0xFFFFu);
                    return ((ok >> (k + 1)) & 1u) ? w : (w & 0xFFFFu) | (NEG_INF2 & 0xFFFF0000u);
                };
                p = make_uint4(excluded(p.x, 0), excluded(p.y, 2), excluded(p.z, 4), excluded(p.w, 6));
            }
        }
        return p;
    }
    // largest entry of a vector, sortable
    static __device__ __forceinline__ int top(const uint4& p) {
        const uint32_t m = __vmaxs2(__vmaxs2(sortable2(p.x), sortable2(p.y)), __vmaxs2(sortable2(p.z), sortable2(p.w)));
        return max((int)(int16_t)(m & 0xFFFFu), (int)m >> 16);
    }
    // first pass: as scan, four loads in flight
    template <typename F>
    __device__ __forceinline__ void fetch(F&& f) {
#pragma unroll 1
        for (int i0 = 0; i0 < count; i0 += 4) {
            uint4 p[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u < count) p[u] = load(index(i0 + u));
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u < count) {
                    if (RESIDENT) kept[(i0 + u) * SAMPLE_THREADS + threadIdx.x] = p[u];
                    f(index(i0 + u) * 8, p[u]);
                }
        }
    }
    // f(first index, vector); every thread of a warp makes the same number of calls
    template <typename F>
    __device__ __forceinline__ void scan(F&& f) const {
#pragma unroll 1
        for (int i = 0; i < count; ++i) f(index(i) * 8, RESIDENT ? kept[i * SAMPLE_THREADS + threadIdx.x] : load(index(i)));
    }
};

__device__ __forceinline__ uint32_t word_at(const uint4& p, int k) { return (k & 2) ? ((k & 1) ? p.w : p.z) : ((k & 1) ? p.y : p.x); }
__device__ __forceinline__ float bf16_at(const uint4& p, int k) {
    const uint32_t w = word_at(p, k >> 1);
    return __uint_as_float((k & 1) ? w & 0xFFFF0000u : w << 16);
}
__device__ __forceinline__ uint16_t bits_at(const uint4& p, int k) {
    const uint32_t w = word_at(p, k >> 1);
    return (uint16_t)((k & 1) ? w >> 16 : w & 0xFFFFu);
}

// A row is drawn by a cluster of up to 8 CTAs that keep it in shared memory and exchange one word per CTA at a time. One CTA per
// row, with the row read again from L2 in every pass, took 69 us for one row of 128256 (top-p) and 220 us for 300 rows (top-p,
// top-k, min-p, temperature and greedy in turn); this takes 14 and 71 us. What bounds it is arithmetic, a hash per entry in the
// Gumbel pass, and for few rows the exchanges between the CTAs.
template <bool RESIDENT>
__global__ void __launch_bounds__(SAMPLE_THREADS, 3)
sample_kernel(const bf16* __restrict__ logits, long row_stride, int vocab,
              const float* __restrict__ temperature, const int* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ min_p,
              const unsigned long long* __restrict__ seeds, const uint32_t* __restrict__ mask_bits,
              const int* __restrict__ mask_row, int mask_words, int* __restrict__ out_tokens, int cl, const SampleShift shift) {
    extern __shared__ __align__(16) uint4 kept[];
    __shared__ SampleShared sh;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int row = blockIdx.x / cl;
    if (cl > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    pdl_wait();
    SampleRow<RESIDENT> rv;
    rv.kept = kept;
    rv.vec = reinterpret_cast<const uint4*>(logits + (size_t)row * row_stride);
    rv.nvec = vocab >> 3;
    rv.cl = cl;
    rv.rank = blockIdx.x - row * cl;
    const int mr = mask_row ? mask_row[row] : -1;
    rv.mask = (mask_bits && mr >= 0) ? mask_bits + (size_t)mr * mask_words : nullptr;
    if (tid < 4) sh.best[tid] = 0;                   // seen by all after the first barrier
    rv.count = (rv.nvec + cl * SAMPLE_THREADS - 1) / (cl * SAMPLE_THREADS);

    // ---- exchanges within the row's CTAs. A slot is written again two exchanges later: by then every CTA has read it.
    int turn = 0;
    bool started = cl == 1;
    const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(&sh.slot[0][0]);
    auto exchange = [&](unsigned long long v) {      // v: this CTA's word, the same in all of its threads
        if (cl == 1) {
            if (tid == 0) sh.slot[turn][0] = v;
            __syncthreads();
        } else {
            if (!started) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");   // every CTA has started
            started = true;
            if (tid < cl) st_cluster_u64(sm100::map_to_cta(slot0 + (turn * SAMPLE_CLUSTER + rv.rank) * 8, tid), v);
            __syncwarp();
            sm100::cluster_sync_all();
        }
    };
    auto row_max = [&](unsigned long long v) {       // the exchange before the last one's end: `red` has been read
        v = warp_max_u64(v);
        if (lane == 0) sh.red[wid] = v;
        __syncthreads();
        exchange(warp_max_u64(lane < SAMPLE_WARPS ? sh.red[lane] : 0ull));
        v = warp_max_u64(lane < cl ? sh.slot[turn][lane] : 0ull);
        turn ^= 1;
        return v;
    };
    auto row_sum2 = [&](float& a, float& b) {
        a = warp_sum(a);
        b = warp_sum(b);
        if (lane == 0) sh.red[wid] = ((unsigned long long)__float_as_uint(b) << 32) | __float_as_uint(a);
        __syncthreads();
        const unsigned long long t = lane < SAMPLE_WARPS ? sh.red[lane] : 0ull;
        const float ta = warp_sum(__uint_as_float((uint32_t)t)), tb = warp_sum(__uint_as_float((uint32_t)(t >> 32)));
        exchange(((unsigned long long)__float_as_uint(tb) << 32) | __float_as_uint(ta));
        a = b = 0.f;
        for (int j = 0; j < cl; ++j) {
            a += __uint_as_float((uint32_t)sh.slot[turn][j]);
            b += __uint_as_float((uint32_t)(sh.slot[turn][j] >> 32));
        }
        turn ^= 1;
    };
    auto row_sum_units = [&](unsigned long long v) {
        v = warp_add_u64(v);
        if (lane == 0) sh.red[wid] = v;
        __syncthreads();
        exchange(warp_add_u64(lane < SAMPLE_WARPS ? sh.red[lane] : 0ull));
        v = warp_add_u64(lane < cl ? sh.slot[turn][lane] : 0ull);
        turn ^= 1;
        return v & NAN_UNITS ? __uint_as_float(0x7fffffffu) : __ull2float_rn(v) * 0x1p-40f;
    };

    // ---- arg-max over the allowed entries, the lowest index of equals
    unsigned long long best = 0ull;
    {
        int m = -0x8000, at = 0;
        uint4 where = make_uint4(NEG_INF2, NEG_INF2, NEG_INF2, NEG_INF2);
        rv.fetch([&](int idx0, const uint4& p) {
            const int t = rv.top(p);
            if (t > m) { m = t; at = idx0; where = p; }
        });
        const int neg_inf = (int16_t)(sortable2(NEG_INF2) & 0xFFFFu);
        if (m > neg_inf) {
#pragma unroll
            for (int k = 7; k >= 0; --k)
                if ((int)(bf16_key(bits_at(where, k)) ^ 0x8000u) == (m & 0xFFFF))
                    best = ((unsigned long long)((uint32_t)(m + 0x8000) + 1u) << 32) | (0xffffffffu - (uint32_t)(at + k));
        } else {                                     // -inf is also what stands for excluded entries
            rv.scan([&](int idx0, const uint4& p) {
#pragma unroll 1
                for (int k = 0; k < 8; ++k) {
                    if (!rv.allowed(idx0 + k)) continue;
                    const unsigned long long cand =
                        ((unsigned long long)(bf16_key(bits_at(p, k)) + 1u) << 32) | (0xffffffffu - (uint32_t)(idx0 + k));
                    best = cand > best ? cand : best;
                }
            });
        }
    }
    best = row_max(best);
    const bool writer = rv.rank == 0 && tid == 0;
    const float T = temperature[row];
    if (best == 0ull) {  // nothing allowed: emit token 0
        if (writer) out_tokens[row] = 0;
        return;
    }
    const int arg = (int)(0xffffffffu - (uint32_t)(best & 0xffffffffu));
    if (T <= 0.f) {
        if (writer) out_tokens[row] = arg;
        return;
    }
    const uint32_t kmax = (uint32_t)(best >> 32) - 1u;
    const float xmax = sortable_value((int)kmax - 0x8000);
    const float inv_t = 1.f / T;
    const int K = top_k[row];
    const float P = top_p[row];
    const float MP = min_p[row];
    const bool need_k = K > 0 && K < vocab;
    const bool need_p = P < 1.f;
    uint32_t thr_key = 0;  // keep entries whose key >= thr_key
    // min-p: keep p_i >= min_p * p_max  <=>  x_i >= xmax + T * ln(min_p)
    const float x_floor = (MP > 0.f) ? xmax + T * __logf(MP) : -INFINITY;
    // per-row stream keys from the 64-bit seed; per-element noise is one 32-bit mix of the index
    const unsigned long long seed = splitmix64(seeds[row]);
    const uint32_t s0 = (uint32_t)seed, s1 = (uint32_t)(seed >> 32);
    const float c1 = inv_t == 0.f ? 0x1p-126f : inv_t * LOG2E;         // at an infinite temperature -inf still weighs nothing
    auto weight = [&](float x) { return ex2((x - xmax) * c1); };       // relative to the largest entry's
    auto mix = [&](uint32_t hsh) {
        hsh ^= s1;
        hsh ^= hsh >> 16; hsh *= 0x85EBCA6Bu; hsh ^= hsh >> 13; hsh *= 0xC2B2AE35u; hsh ^= hsh >> 16;
        return hsh;
    };

    // Gumbel-max over the entries with key >= lo (and the min-p floor, and the mask); `salt` separates the noise streams of
    // different rounds. Returns (score key << 32 | ~index) or 0. With Z, adds up the weights of all entries too.
    //
    // The score of an entry of weight w (exp of its scaled distance from the largest) and uniform u is log w - log(-log u). As
    // -log u >= 1 - u, it cannot reach a score b seen before where 1 - u > w exp(-b): that test costs one exponential that the
    // sum of weights needs anyway, and only what passes it (some tens of entries of a row) pays for two logarithms and the
    // exact comparison. The largest entry, whose score every thread works out first, bounds exp(-b). The slack: 2^-16 for the
    // last mixing step of u, left out here as it changes the low half of 32 bits alone; 1e-6 for the error of a fast logarithm
    // near 1 (2^-22) and the bits of u beyond 23; 1e-4 of B for the weights' relative error.
    // Shifts are products' high halves: shifts, logic and comparisons share one pipe of half rate, and it is what the pass is
    // bound by (62 million instructions for 300 rows of 128256, that pipe 65 % busy, before the test was thinned out).
    auto gumbel_pass = [&](uint32_t lo, uint32_t salt, float* Z) -> unsigned long long {
        if (lo > kmax) return 0ull;
        const uint32_t from = s0 + salt * 0x632BE5ABu;
        unsigned long long pick = 0ull;
        auto consider = [&](int idx, uint16_t bits) {
            if (bf16_key(bits) < lo) return;
            const float x = __bfloat162float(__ushort_as_bfloat16(bits));
            if (x < x_floor) return;
            if (!rv.allowed(idx)) return;
            const float u = ((float)(mix(((uint32_t)idx + from) * 0x9E3779B1u) >> 8) + 0.5f) * (1.0f / 16777216.0f);
            const float score = (x - xmax) * inv_t - __logf(-__logf(u));
            const unsigned long long cand = ((unsigned long long)f32_key(score) << 32) | (0xffffffffu - (uint32_t)idx);
            pick = cand > pick ? cand : pick;
        };
        consider(arg, (uint16_t)((kmax & 0x8000u) ? kmax & 0x7fffu : ~kmax));
        uint32_t seen = (uint32_t)(pick >> 32);      // the largest score this thread knows of
        float B = seen ? ex2(f32_of_key(seen) * -LOG2E) * 1.0001f : INFINITY;
        volatile uint32_t* shared_best = &sh.best[salt & 3];
        const float xlow = fmaxf(sortable_value((int)lo - 0x8000), x_floor);    // necessary for key >= lo, not sufficient
        float z = 0.f;
        const bool all = Z || xlow == -INFINITY;
        rv.scan([&](int idx0, const uint4& p) {
            if (!all && !__any_sync(0xffffffffu, !(sortable_value(rv.top(p)) < xlow))) return;
            const uint32_t others = *shared_best;    // one score found anywhere in the CTA spares the other warps theirs
            if (others > seen) {
                seen = others;
                B = ex2(f32_of_key(seen) * -LOG2E) * 1.0001f;
            }
            const uint32_t hb = ((uint32_t)idx0 + from) * 0x9E3779B1u;
            auto passes = [&](int k, float w) {
                uint32_t hsh = (hb + (uint32_t)k * 0x9E3779B1u) ^ s1;
                hsh ^= __umulhi(hsh, shift.by16);
                hsh *= 0x85EBCA6Bu;
                hsh ^= __umulhi(hsh, shift.by13);
                hsh *= 0xC2B2AE35u;
                return !(fmaf(w, B, __uint_as_float(__umulhi(hsh, shift.by9) + 0x3F800000u)) < 2.f - 1.7e-5f);       // 1 + u
            };
            bool maybe = false;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float w = weight(bf16_at(p, k));
                maybe |= passes(k, w);
                if (Z) z += w;
            }
            if (__any_sync(0xffffffffu, maybe)) {
                if (maybe) {
#pragma unroll 1
                    for (int k = 0; k < 8; ++k)
                        if (passes(k, weight(bf16_at(p, k)))) consider(idx0 + k, bits_at(p, k));
                }
                __syncwarp();
                const uint32_t high = __reduce_max_sync(0xffffffffu, (uint32_t)(pick >> 32));
                if (high > seen) {
                    seen = high;
                    B = ex2(f32_of_key(seen) * -LOG2E) * 1.0001f;
                    if (lane == 0) atomicMax(&sh.best[salt & 3], seen);
                }
            }
        });
        if (Z) *Z = z;
        return row_max(pick);
    };

    // Mass of the entries with key >= lo, to the last bit whatever the order of the entries: in whole numbers of 2^-40 for eight
    // entries at a time.
    auto exact_mass = [&](uint32_t lo) {
        unsigned long long units = 0;
        bool nan = false;
        rv.scan([&](int, const uint4& p) {
            float w = 0.f;
#pragma unroll 1
            for (int k = 0; k < 8; ++k) w += bf16_key(bits_at(p, k)) >= lo ? weight(bf16_at(p, k)) : 0.f;
            units += __float2ull_rn(w * 0x1p40f);
            nan |= w != w;
        });
        return row_sum_units(nan ? NAN_UNITS : units);
    };
    // What the order of the additions can change in a 32-bit sum of a row's weights, twice, relative to the sum. It follows the number of
    // CTAs, and so the rows of a batch: a decision that such sums leave open is made on exact masses.
    const float order_error = (float)(rv.count * 8 + 64) * 0x1p-22f;
    if (need_k || need_p) {
        // Rejection rounds (no histogram, no atomics): draw a candidate from the distribution restricted to keys >= lo, then
        // measure how much probability mass lies strictly above its key. It belongs to the kept set iff that is below
        // top-p * Z (ties at the threshold are kept, as in the search below). A rejected candidate proves that every
        // key <= its key is outside the kept set, so the next round draws above it. With top-p = 0.9 a round accepts with
        // probability >= 0.9; after three rejections, and for top-k or a small top-p (where a round rarely accepts), the exact
        // search takes over.
        uint32_t lo = 0;
        const int rounds = (need_p && !need_k && P >= 0.5f) ? 3 : 0;
        float z_thread = 0.f;
        for (int round = 0; round < rounds; ++round) {
            const unsigned long long pick = gumbel_pass(lo, (uint32_t)round, round == 0 ? &z_thread : nullptr);
            if (pick == 0ull) {                       // nothing left above lo: fall back to the arg-max
                if (writer) out_tokens[row] = arg;
                return;
            }
            const int cand = (int)(0xffffffffu - (uint32_t)(pick & 0xffffffffu));
            const uint32_t ckey = bf16_key(reinterpret_cast<const uint16_t*>(rv.vec)[cand]);
            float z = z_thread, above = 0.f;
            rv.scan([&](int, const uint4& p) {
                if (rv.top(p) <= (int)ckey - 0x8000) return;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t sv = sortable2(word_at(p, k >> 1)) << ((k & 1) ? 0 : 16);
                    if ((int)sv > (((int)ckey - 0x8000) * 0x10000 | 0xFFFF)) above += weight(bf16_at(p, k));
                }
            });
            row_sum2(z, above);
            if (fabsf(above - P * z) <= z * order_error) {
                above = exact_mass(ckey + 1u);
                z = exact_mass(0u);
            }
            if (above < P * z) {
                if (writer) out_tokens[row] = cand;
                return;
            }
            lo = ckey + 1u;
        }
        // ---- exact search: the first key from the top at which the count reaches K or the mass P * Z. Keys just below the
        // largest entry's first (entries that can matter are almost always among them), else 128 at a time over all keys and
        // then one by one. A key's mass is its entries' number times their weight; that of 128 keys is added up in whole numbers: neither
        // depends on the order in which the entries come.
        const float Z = need_p ? exact_mass(0u) : 0.f;
        if (need_p && 0.f >= P * Z) {                 // top-p of nothing: the arg-max, also where others equal it
            if (writer) out_tokens[row] = arg;
            return;
        }
        const uint32_t cnt0 = (uint32_t)__cvta_generic_to_shared(&sh.cnt[0]), mass0 = (uint32_t)__cvta_generic_to_shared(&sh.mass[0][0]);
        // a mass of 1 in units, and bits of a word: as many as the entries of a CTA cannot overflow (14 for up to 2^18 of them)
        const int bits = min(14, __clz(rv.count * SAMPLE_THREADS * 8 - 1));
        const float one = (float)(1ull << (3 * bits - 1));
        uint32_t base_cnt = 0;
        float base_mass = 0.f;
        // first bin of `bins` bins of 2^shift keys, downwards from `ktop`, at which a limit is reached, or -1
        auto search = [&](uint32_t ktop, int shift, int bins) -> int {
            __syncthreads();
            sh.cnt[tid] = 0;
            sh.mass[0][tid] = sh.mass[1][tid] = sh.mass[2][tid] = 0;
            if (tid == 0) sh.hit = SAMPLE_BINS;
            __syncthreads();
            const int low = (int)ktop - (bins << shift) + 1 - 0x8000;
            rv.scan([&](int, const uint4& p) {
                if (rv.top(p) < low) return;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t key = bf16_key(bits_at(p, k));
                    const uint32_t bin = (ktop - key) >> shift;       // huge for keys above ktop
                    if (bin >= (uint32_t)bins) continue;
                    atomicAdd(&sh.cnt[bin], 1u);
                    if (need_p && shift) {
                        const unsigned long long units = __float2ull_rn(weight(bf16_at(p, k)) * one);
                        atomicAdd(&sh.mass[0][bin], (uint32_t)units & ((1u << bits) - 1u));
                        atomicAdd(&sh.mass[1][bin], (uint32_t)(units >> bits) & ((1u << bits) - 1u));
                        atomicAdd(&sh.mass[2][bin], (uint32_t)(units >> (2 * bits)));
                    }
                }
            });
            __syncthreads();
            uint32_t c = 0;
            unsigned long long units = 0;
            auto word = [&](int w, uint32_t v) { units += (unsigned long long)v << (w * bits); };
            if (cl > 1) {
                sm100::cluster_sync_all();
                for (int j = 0; j < cl; ++j) {
                    c += ld_cluster_u32(sm100::map_to_cta(cnt0 + tid * 4, j));
                    if (need_p && shift)
                        for (int w = 0; w < 3; ++w) word(w, ld_cluster_u32(sm100::map_to_cta(mass0 + (w * SAMPLE_BINS + tid) * 4, j)));
                }
                sm100::cluster_sync_all();                            // read by all before it changes or its CTA ends
            } else {
                c = sh.cnt[tid];
                for (int w = 0; w < 3; ++w) word(w, sh.mass[w][tid]);
            }
            float m = __ull2float_rn(units) / one;
            if (need_p && !shift && c) m = (float)c * weight(sortable_value((int)ktop - tid - 0x8000));
            const uint32_t c_own = c;
            const float m_own = m;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t cc = __shfl_up_sync(0xffffffffu, c, o);
                const float mm = __shfl_up_sync(0xffffffffu, m, o);
                if (lane >= o) { c += cc; m += mm; }
            }
            if (lane == 31) { sh.wcnt[wid] = c; sh.wmass[wid] = m; }
            __syncthreads();
            uint32_t pc = base_cnt;
            float pm = base_mass;
            for (int w = 0; w < wid; ++w) { pc += sh.wcnt[w]; pm += sh.wmass[w]; }
            c += pc;
            m += pm;
            if ((need_k && c >= (uint32_t)K) || (need_p && m >= P * Z)) atomicMin(&sh.hit, tid);
            __syncthreads();
            const int hit = sh.hit;
            if (tid == hit) { sh.base_cnt = c - c_own; sh.base_mass = m - m_own; }
            __syncthreads();
            return hit < bins ? hit : -1;
        };
        const int near = search(kmax, 0, SAMPLE_BINS);
        if (near >= 0) {
            thr_key = kmax - (uint32_t)near;
        } else {
            const int coarse = search(0xFFFFu, 7, SAMPLE_BINS);
            if (coarse >= 0) {
                base_cnt = sh.base_cnt;
                base_mass = sh.base_mass;
                const uint32_t ktop = 0xFFFFu - (uint32_t)coarse * 128u;
                const int fine = search(ktop, 0, 128);
                thr_key = ktop - (uint32_t)(fine >= 0 ? fine : 127);
            }
        }
    }
    // ---- Gumbel-max over the kept set
    const unsigned long long pick = gumbel_pass(thr_key, 7u, nullptr);
    if (writer) out_tokens[row] = pick ? (int)(0xffffffffu - (uint32_t)(pick & 0xffffffffu)) : arg;
}

constexpr int STATS_THREADS = 1024;

// Per-row max, log-sum-exp and Shannon entropy of the unscaled distribution.
// stats[row] = {max, lse, entropy}.
__global__ void __launch_bounds__(STATS_THREADS)
row_stats_kernel(const bf16* __restrict__ logits, long row_stride, int vocab,
                 float* __restrict__ stats) {
    __shared__ float red[32];
    const int row = blockIdx.x;
    const uint4* vec = reinterpret_cast<const uint4*>(logits + (size_t)row * row_stride);
    const int nvec = vocab >> 3;
    float mx = -INFINITY;
    for (int v = threadIdx.x; v < nvec; v += STATS_THREADS) {
        const uint4 pk = vec[v];
        float f[8];
        unpack8(*reinterpret_cast<const bf16x8*>(&pk), f);
#pragma unroll
        for (int k = 0; k < 8; ++k) mx = fmaxf(mx, f[k]);
    }
    mx = block_max(mx, red);
    float z = 0.f, a = 0.f;  // z = sum e^(x-m), a = sum (x-m) e^(x-m)
    for (int v = threadIdx.x; v < nvec; v += STATS_THREADS) {
        const uint4 pk = vec[v];
        float f[8];
        unpack8(*reinterpret_cast<const bf16x8*>(&pk), f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float d = f[k] - mx;
            const float e = __expf(d);
            z += e;
            a += d * e;
        }
    }
    z = block_sum(z, red);
    a = block_sum(a, red);
    if (threadIdx.x == 0) {
        const float lz = logf(z);
        stats[row * 3 + 0] = mx;
        stats[row * 3 + 1] = mx + lz;
        stats[row * 3 + 2] = lz - a / z;  // H = log Z - E[x - m]
    }
}

}  // namespace pie

using namespace pie;

PIE_API int pie_sample(const void* logits, long row_stride, int rows, int vocab,
                       const float* temperature, const int* top_k, const float* top_p,
                       const float* min_p, const unsigned long long* seeds,
                       const uint32_t* mask_bits, const int* mask_row, int mask_words,
                       int* out_tokens, cudaStream_t st) {
    if (rows <= 0) return 0;
    if (vocab % 8 || row_stride % 8) return (int)cudaErrorInvalidValue;
    // CTAs of a row: as few as hold it in 64 KB each (three per SM), for a row's reductions cost every CTA the same, but up to 8
    // while the machine has room, for latency. Two vectors per thread stay in one CTA (128 rows of 8192 entries at a temperature: 6.9 us,
    // in two CTAs 9.1). Rows beyond 8 x 192 KB are read again in every pass.
    const int nvec = vocab / 8, each = SAMPLE_THREADS * 16;
    int cl = std::min(SAMPLE_CLUSTER, (nvec + 4095) / 4096);
    while (nvec > 2 * SAMPLE_THREADS && cl < SAMPLE_CLUSTER && nvec > cl * SAMPLE_THREADS && (long)rows * (cl + 1) <= 2 * PIE_SMS) ++cl;
    const int count = (nvec + cl * SAMPLE_THREADS - 1) / (cl * SAMPLE_THREADS);
    const bool resident = count * each <= 192 * 1024;
    auto kern = resident ? sample_kernel<true> : sample_kernel<false>;
    if (resident) {
        const cudaError_t a = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 192 * 1024);
        if (a != cudaSuccess) return (int)a;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)rows * cl);
    cfg.blockDim = dim3(SAMPLE_THREADS);
    cfg.dynamicSmemBytes = resident ? count * each : 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = g_pie_pdl ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cl;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cl > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (const bf16*)logits, row_stride, vocab, temperature, top_k, top_p, min_p,
                                             seeds, mask_bits, mask_row, mask_words, out_tokens, cl,
                                             SampleShift{1u << 23, 1u << 19, 1u << 16});
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

PIE_API int pie_row_stats(const void* logits, long row_stride, int rows, int vocab, float* stats,
                          cudaStream_t st) {
    if (rows <= 0) return 0;
    if (vocab % 8 || row_stride % 8) return (int)cudaErrorInvalidValue;
    row_stats_kernel<<<rows, STATS_THREADS, 0, st>>>((const bf16*)logits, row_stride, vocab, stats);
    return (int)cudaGetLastError();
}
