// Temperature + nucleus (top-p) sampling on the device, a cluster of eight blocks per sequence.
//
// Reference: sample_top_p_f32 (src/runtime.rs:1092-1152) -- softmax at the given temperature, tokens sorted by
// descending probability, the shortest prefix whose mass reaches top_p, one coin scaled to that mass, the first
// token at which the running mass reaches it -- and its emitted C99 twin (src/runners/tinystories_smollm.c:506-529),
// which walks the unsorted cumulative distribution instead (`mode` 1).  Both fall back to the greedy rule when
// temperature <= 1e-5 or top_p <= 0.
//
// No sort: the two prefix decisions are thresholds on the probability value, found by an eight-way search over the float
// bit pattern (three bits a round), and ties at a threshold are resolved in index order, the order the CPU checker uses
// for equal probabilities (the reference's unstable sort leaves it open).  Sums are reductions in a fixed order:
// deterministic, but not the reference's sequential order, so a decision that sits within rounding of a threshold can go to
// the neighbouring token.
//
// What bounds it: the number of rounds, each a pass over the row and an exchange.  One block needed 5 us for a pass over
// 128256 probabilities and one bit a round took 62 of them (0.45 ms a step).  Eight blocks hold an eighth of the row each (in
// L1 after the first pass), a round looks at seven thresholds at once and skips the groups of 32 values that are all
// outside the range that is left, and the partial sums travel through distributed
// shared memory: 323 -> 137 us for 128256 nearly equal logits, 326 -> 82 for a peaked row, about 3 us a round.
#include <cooperative_groups.h>
#include <math.h>

#include "vb_internal.cuh"
#include "vb_kernels.cuh"

namespace vb {

namespace {

constexpr int SP_THREADS = 1024, SP_RANKS = 8, SP_WARPS = SP_THREADS / 32;

struct SpShared {
    float red[SP_WARPS][8];
    uint32_t scan[SP_WARPS];
    float tab[2][SP_RANKS][8];  // what every rank's exchange left here; two of them, so that one cluster barrier a round is enough
};
enum SpOp { SP_SUM, SP_MAX, SP_MIN_U32 };
__device__ __forceinline__ float sp_combine(SpOp op, float a, float b) {
    return op == SP_SUM ? a + b : op == SP_MAX ? fmaxf(a, b) : __uint_as_float(min(__float_as_uint(a), __float_as_uint(b)));
}

// The cluster that works on one row: rank r holds the indices [lo, hi).
struct SpRow {
    SpShared* sh;
    float* p;
    uint32_t lo, hi, rank, round, lane, warp;

    // One value per thread of the cluster, combined; the returned table holds every rank's part.
    __device__ __forceinline__ float all(SpOp op, float v, const float (**table)[8] = nullptr) {
        namespace cg = cooperative_groups;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = sp_combine(op, v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
        if (lane == 0) sh->red[warp][0] = v;
        __syncthreads();
        const uint32_t buf = round++ & 1u;
        if (threadIdx.x < SP_RANKS) {
            float t = sh->red[0][0];
            for (int w = 1; w < SP_WARPS; ++w) t = sp_combine(op, t, sh->red[w][0]);
            *cg::this_cluster().map_shared_rank(&sh->tab[buf][rank][0], threadIdx.x) = t;
        }
        cg::this_cluster().sync();
        float t = sh->tab[buf][0][0];
        for (int r = 1; r < SP_RANKS; ++r) t = sp_combine(op, t, sh->tab[buf][r][0]);
        if (table) *table = sh->tab[buf];
        return t;
    }
    // the same for seven sums at once
    __device__ __forceinline__ void all7(float (&v)[8]) {
        namespace cg = cooperative_groups;
        v[7] = 0.0f;
        int o = 16;
#pragma unroll
        for (int n = 8; n > 1; n >>= 1, o >>= 1) {  // lane l is left with the warp's sum of value l >> 2
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < n / 2; ++i) {
                const float send = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
            }
        }
        float r = v[0];
        r += __shfl_xor_sync(0xFFFFFFFFu, r, 2);
        r += __shfl_xor_sync(0xFFFFFFFFu, r, 1);
        if ((lane & 3) == 0) sh->red[warp][lane >> 2] = r;
        __syncthreads();
        const uint32_t buf = round++ & 1u;
        if (threadIdx.x < 8 * SP_RANKS) {
            const uint32_t k = threadIdx.x & 7;
            float t = 0.0f;
#pragma unroll 8
            for (int w = 0; w < SP_WARPS; ++w) t += sh->red[w][k];
            *cg::this_cluster().map_shared_rank(&sh->tab[buf][rank][k], threadIdx.x >> 3) = t;
        }
        cg::this_cluster().sync();
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            float t = 0.0f;
#pragma unroll
            for (int q = 0; q < SP_RANKS; ++q) t += sh->tab[buf][q][k];
            v[k] = t;
        }
    }
    // Largest bit pattern t in [lo_t, hi_t) whose mass (of the probabilities with a pattern >= t; all are positive floats, the
    // pattern orders them) is at least `want`, given that lo_t qualifies and hi_t does not; *above: the mass above it.
    __device__ uint32_t search(uint32_t lo_t, uint32_t hi_t, float want, float* above) {
        float base = 0.0f;  // mass at hi_t and above
        while (hi_t - lo_t > 1) {
            const uint32_t step = (hi_t - lo_t + 7) / 8;
            float s[8] = {};
            for (uint32_t i0 = lo + warp * 32; i0 < hi; i0 += SP_THREADS) {
                const uint32_t i = i0 + lane;
                const float v = i < hi ? p[i] : 0.0f;
                const uint32_t b = __float_as_uint(v);
                const bool in = i < hi && b >= lo_t && b < hi_t;
                if (__any_sync(0xFFFFFFFFu, in)) {
#pragma unroll
                    for (uint32_t k = 0; k < 7; ++k) s[k] += (in && b - lo_t >= (k + 1) * step) ? v : 0.0f;
                }
            }
            all7(s);
            uint32_t k = 0;  // thresholds lo_t + k * step, k = 0..8 (the last one hi_t at most)
#pragma unroll
            for (uint32_t q = 1; q <= 7; ++q)
                if (lo_t + q * step < hi_t && base + s[q - 1] >= want) k = q;
            const uint32_t next = lo_t + (k + 1) * step;
            if (k < 7 && next < hi_t) { hi_t = next; base += s[k]; }
            lo_t += k * step;
        }
        *above = base;
        return lo_t;
    }
    // how many probabilities have the pattern t (counts stay below 2^24 a rank: exact); *table: by rank
    __device__ __forceinline__ uint32_t count(uint32_t t, const float (**table)[8]) {
        uint32_t c = 0;
        for (uint32_t i = lo + threadIdx.x; i < hi; i += SP_THREADS) c += __float_as_uint(p[i]) == t ? 1u : 0u;
        return (uint32_t)all(SP_SUM, (float)c, table);
    }
    // exclusive prefix of one value per thread over the block (thread order = order of the threads' index chunks)
    template <typename T>
    __device__ __forceinline__ T before(T v) {
        T inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const T u = __shfl_up_sync(0xFFFFFFFFu, inc, o); if (lane >= (uint32_t)o) inc += u; }
        __syncthreads();
        if (lane == 31) reinterpret_cast<T*>(sh->scan)[warp] = inc;
        __syncthreads();
        T base = 0;
        for (uint32_t w = 0; w < warp; ++w) base += reinterpret_cast<T*>(sh->scan)[w];
        return base + inc - v;
    }
    __device__ __forceinline__ void chunk(uint32_t* i0, uint32_t* i1) const {
        const uint32_t len = (hi - lo + SP_THREADS - 1) / SP_THREADS;
        *i0 = min(hi, lo + threadIdx.x * len);
        *i1 = min(hi, *i0 + len);
    }
};

struct SampleArgs {
    const float* logits;   // [batch][n]
    float* probs;          // [batch][n] scratch
    uint32_t n;
    float temperature, top_p;
    int mode;              // 0: src/runtime.rs rule, 1: the emitted C99 rule
    const float* coins;    // != null: one coin per sequence (device memory)
    float coin;            // coins == null and use_seed == 0: this coin for every sequence
    int use_seed;          // coins == null: 1 = coin drawn from (seed, sequence, position)
    uint64_t seed;
    SeqState* state;       // != null: inactive sequences are skipped, the winner is fed back and the position advances
    uint32_t* ring;
    uint32_t ring_slots;
    uint32_t* out_token;   // != null: winners [batch]
};

__device__ __forceinline__ float device_coin(uint64_t seed, uint32_t slot, uint32_t pos) {
    const uint64_t h = mix64(stream_key(seed, 0x5A4D504CULL + (uint64_t)slot) + ((uint64_t)pos + 1ULL) * 0x9E3779B97F4A7C15ULL);
    return (float)(uint32_t)(h >> 40) * (1.0f / 16777216.0f);
}

__global__ void __cluster_dims__(SP_RANKS, 1, 1) __launch_bounds__(SP_THREADS) k_sample_top_p(SampleArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ SpShared sh;
    const uint32_t b = blockIdx.y, n = a.n, rank = blockIdx.x;  // (the cluster is the grid's x dimension)
    if (a.state && !a.state[b].active) return;                  // the whole cluster leaves together
    cooperative_groups::this_cluster().sync();                  // every block runs before anyone writes into its shared memory
    const float* lg = a.logits + (size_t)b * n;
    const uint32_t len = ((n + SP_RANKS - 1) / SP_RANKS + 31) / 32 * 32;
    SpRow row;
    row.sh = &sh; row.p = a.probs + (size_t)b * n;
    row.lo = min(n, rank * len); row.hi = min(n, row.lo + len);
    row.rank = rank; row.round = 0; row.lane = threadIdx.x & 31; row.warp = threadIdx.x >> 5;
    float* p = row.p;
    uint32_t tok = 0;
    if (a.temperature <= 1e-5f || a.top_p <= 0.0f) {
        // greedy rule (src/runtime.rs:1078-1088): first index of the maximum, NaN never wins, nothing above -inf -> 0
        float bv = -INFINITY;
        uint32_t bi = 0xFFFFFFFFu;
        for (uint32_t i = row.lo + threadIdx.x; i < row.hi; i += SP_THREADS) {
            const float v = lg[i];
            if (v > bv) { bv = v; bi = i; }
        }
        const float mx = row.all(SP_MAX, bv);
        const uint32_t best = __float_as_uint(row.all(SP_MIN_U32, __uint_as_float((bi != 0xFFFFFFFFu && bv == mx) ? bi : 0xFFFFFFFFu)));
        tok = best == 0xFFFFFFFFu ? 0u : best;
    } else {
        const float coin_raw = a.coins ? a.coins[b] : (a.use_seed ? device_coin(a.seed, b, a.state ? a.state[b].pos : 0u) : a.coin);
        const float inv_temp = 1.0f / a.temperature;
        float m = -INFINITY;
#pragma unroll 8
        for (uint32_t i = row.lo + threadIdx.x; i < row.hi; i += SP_THREADS) m = fmaxf(m, lg[i] * inv_temp);
        const float max_l = row.all(SP_MAX, m);
        float s = 0.0f;
#pragma unroll 4
        for (uint32_t i = row.lo + threadIdx.x; i < row.hi; i += SP_THREADS) {
            const float e = expf(__fsub_rn(__fmul_rn(lg[i], inv_temp), max_l));  // product rounded first, as the reference
            p[i] = e;
            s += e;
        }
        const float sum_exp = row.all(SP_SUM, s);
        if (a.mode == 1) {
            // unsorted walk: first index whose running sum of exp reaches coin * top_p * sum_exp
            const float target = coin_raw * a.top_p * sum_exp;
            uint32_t i0, i1;
            row.chunk(&i0, &i1);
            float part = 0.0f;
            for (uint32_t i = i0; i < i1; ++i) part += p[i];
            const float (*table)[8];
            row.all(SP_SUM, part, &table);
            float base = 0.0f;
            for (uint32_t r = 0; r < rank; ++r) base += table[r][0];
            const float begin = base + row.before(part), end = begin + part;
            // every chunk whose end reaches the target offers its first qualifying index; the lowest one wins
            uint32_t first = 0xFFFFFFFFu;
            if (i1 > i0 && end >= target) {
                float run = begin;
                for (uint32_t i = i0; i < i1; ++i) {
                    run += p[i];
                    if (run >= target) { first = i; break; }
                }
            }
            first = __float_as_uint(row.all(SP_MIN_U32, __uint_as_float(first)));
            tok = first == 0xFFFFFFFFu ? 0u : first;
        } else {
            const float inv_sum = 1.0f / sum_exp;
            float pm = 0.0f, mass = 0.0f;
#pragma unroll 4
            for (uint32_t i = row.lo + threadIdx.x; i < row.hi; i += SP_THREADS) {
                const float v = p[i] * inv_sum;
                p[i] = v;
                pm = fmaxf(pm, v);
                mass += v;
            }
            const uint32_t top_bits = __float_as_uint(row.all(SP_MAX, pm));
            const float total = row.all(SP_SUM, mass);
            const float (*table)[8];
            // nucleus: every probability above the threshold t*, plus the first `m_ties` (index order) equal to it
            uint32_t t_star = 0;
            float above = total;
            if (total >= a.top_p) t_star = row.search(0u, top_bits + 1u, a.top_p, &above);
            const float tau = __uint_as_float(t_star);
            const uint32_t n_ties = row.count(t_star, &table);
            uint32_t m_ties = n_ties;
            if (total >= a.top_p && tau > 0.0f) {
                const float need = ceilf((a.top_p - above) / tau);
                m_ties = need < 1.0f ? 1u : (need > (float)n_ties ? n_ties : (uint32_t)need);
            }
            const float cum = above + (float)m_ties * tau;
            const float coin = fminf(fmaxf(coin_raw, 0.0f), 0.9999f);
            const float target = coin * cum;
            // the token at which the running mass (descending probability, ties by index) reaches the target
            float above2;
            const uint32_t t2 = row.search(t_star, top_bits + 1u, target, &above2);
            const float tau2 = __uint_as_float(t2);
            uint32_t n2 = row.count(t2, &table);
            if (t2 == t_star) n2 = m_ties < n2 ? m_ties : n2;
            uint32_t j = 1;
            if (tau2 > 0.0f && target > above2) {
                const float need = ceilf((target - above2) / tau2);
                j = need < 1.0f ? 1u : (need > (float)n2 ? n2 : (uint32_t)need);
            }
            if (j < 1u) j = 1u;
            // the j-th (1-based, index order) element with the pattern t2
            uint32_t ties = 0;
            for (uint32_t r = 0; r < rank; ++r) ties += (uint32_t)table[r][0];
            uint32_t i0, i1, cnt = 0;
            row.chunk(&i0, &i1);
            for (uint32_t i = i0; i < i1; ++i) cnt += __float_as_uint(p[i]) == t2 ? 1u : 0u;
            ties += row.before(cnt);
            uint32_t pick = 0xFFFFFFFFu;
            if (cnt > 0 && ties < j && j <= ties + cnt) {
                for (uint32_t i = i0; i < i1; ++i)
                    if (__float_as_uint(p[i]) == t2 && ++ties == j) { pick = i; break; }
            }
            pick = __float_as_uint(row.all(SP_MIN_U32, __uint_as_float(pick)));
            tok = pick == 0xFFFFFFFFu ? 0u : pick;
        }
    }
    cooperative_groups::this_cluster().sync();  // no block leaves while another may still write into it (and b's position is read)
    if (rank != 0) return;
    if (threadIdx.x == 0) {
        if (a.out_token) a.out_token[b] = tok;
        if (a.state) {
            const uint32_t pos = a.state[b].pos;
            if (a.ring) a.ring[(size_t)b * a.ring_slots + (pos % a.ring_slots)] = tok;
            seq_advance(a.state + b, tok);
        }
    }
}

}  // namespace

cudaError_t sample_top_p(const LaunchCfg& lc, uint32_t* out_token, const float* logits, float* probs, uint32_t n, uint32_t batch,
                         float temperature, float top_p, int mode, const float* coins, float coin, int use_seed, uint64_t seed,
                         SeqState* state, uint32_t* ring, uint32_t ring_slots) {
    SampleArgs a;
    a.logits = logits; a.probs = probs; a.n = n; a.temperature = temperature; a.top_p = top_p; a.mode = mode; a.coins = coins;
    a.coin = coin; a.use_seed = use_seed; a.seed = seed; a.state = state; a.ring = ring; a.ring_slots = ring_slots; a.out_token = out_token;
    return launch(lc, k_sample_top_p, dim3(SP_RANKS, batch), dim3(SP_THREADS), 0, a);
}

}  // namespace vb

using namespace vb;

extern "C" int32_t vb_op_sample_top_p(uint32_t* out_token, const float* logits, uint32_t n, float temperature, float top_p,
                                      float random_coin, int32_t mode, void* scratch, uint64_t scratch_bytes, void* stream) {
    VB_REQUIRE(out_token && logits && n > 0, "vb_op_sample_top_p: null argument or empty row");
    VB_REQUIRE(mode == 0 || mode == 1, "vb_op_sample_top_p: mode %d (0: runtime rule, 1: emitted C99 rule)", mode);
    VB_REQUIRE(scratch && scratch_bytes >= (uint64_t)n * 4, "vb_op_sample_top_p: scratch of %llu bytes, need %llu",
               (unsigned long long)scratch_bytes, (unsigned long long)n * 4);
    LaunchCfg lc;
    lc.stream = (cudaStream_t)stream;
    VB_CUDA(sample_top_p(lc, out_token, logits, (float*)scratch, n, 1, temperature, top_p, mode, nullptr, random_coin, 0, 0, nullptr,
                         nullptr, 0));
    return VB_OK;
}
