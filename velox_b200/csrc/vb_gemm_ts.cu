// Products of many rows of x on the 5th-generation tensor cores with the WEIGHTS DEQUANTISED INTO TENSOR MEMORY: prompts of
// int4 group-32 and int8 per-channel models, where the weights are what takes time (17 to 128 or 256 rows) or where there is
// no canonical copy to convert (lean contexts, any number of rows).
//     dst[t][o] = sum_k x[t][k] * W[o][k]
//
// Why tensor memory.  A tcgen05.mma (M 128, K 16) takes N / 2 clocks when A comes from tensor memory; with both operands in
// shared memory it also reads 4 KB of A and 32 N bytes of B at 128 bytes a clock, 64 clocks at N = 128 where the arithmetic
// takes 64, and the copies that fill shared memory (64 KB of weight parts, 64 KB of x per 128 of K) compete with it: 0.6 of
// the instruction rate.  Here the weights never pass through shared memory: thread = weight row = tensor-memory lane reads its
// packed weights from global memory (prefetched in registers), makes the fp16 parts in registers and writes them with
// tcgen05.st as the A operand.  Shared memory carries only x, from HBM come only the packed bytes (no fp16 copies of the
// weights are kept), and int4 weights in their tile-major copy are all a lean context has.
//
// Numerics.  x = x_hi + x_lo in fp16 after scaling each row by a power of two to a maximum in [2^13, 2^14) (22 bits of every
// element that matters, no overflow); weights as fp16 hi (+ lo where fp16 does not hold them: int4 group-32 (n - 8) * s is exact
// in hi + lo, others to 22 bits); three (two) products into the same fp32 accumulators, W_lo . x_lo (2^-22) is dropped.  int8
// weights are exact integers, the row scale is applied at the end.
//
// Block: 6 warps, two blocks per SM.  Warp 0 copies x (tiled TMA, [NT rows][64] boxes of hi and lo, 128-byte swizzle), warp 1
// issues, warps 2-5 dequantise 64 of K at a time into a ring of A stages and at the end read the accumulator (lane = weight
// row).  NT = 16..128 rows of x.  Gate and up share a tile: lanes 0-7 of every 16 hold gate rows, lanes 8-15 the same up rows
// (the interleaved int4 copy is laid out that way).  Matrices with few tiles split K over a cluster of up to 8 blocks: the
// partial tiles meet in distributed shared memory and are added in rank order (the same bits every run).
//
// Measured, 8B int4 shape, a product with its k_rows_split, us, for 16 / 64 / 128 rows: QKV 20.6 / 31 / 44, O 14 / 20 / 29, gate/up
// 92 / 127 / 167, down 34 / 51 / 63.  With four rows at a time on vb_gemv_mma.cu a 119-row prompt of the 72B shape took 30 passes
// over 36 GB of weights (0.36 s), now it takes 45 ms.  128 rows and more are bound by the issue: a stage of 12 products (64 of K,
// 128 columns) takes ~1400 clocks where the products alone take 770, which two resident blocks overlap only in part.  There
// the kernel of vb_gemm_tc.cu, whose operands are both in shared memory, is faster (gate/up of 512 rows 342 us, here 570).
// Every wait is bounded; one that runs out sets a block-wide abort flag and the library's error word.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>

#include "vb_kernels.cuh"
#include "vb_tma.cuh"

namespace cg = cooperative_groups;

namespace vb {
namespace {

constexpr int TS_THREADS = 192, TS_Q4_BLK = 1152;
constexpr uint32_t TS_TMEM = 256;  // columns of a block

template <int FMT> struct Ts {
    static constexpr bool q4 = FMT == VB_FMT_Q4G32;
    static constexpr int parts = q4 ? 2 : 1;   // of the weights
    static constexpr int unit = q4 ? 128 : 64; // K of one prefetch
    static constexpr int regs = q4 ? 5 : 4;    // 16-byte registers of one
    static constexpr int depth = 3;            // prefetches in flight
};
template <int FMT, int NT> struct TsShape {
    static constexpr int a_cols = Ts<FMT>::parts * 32;                                     // of one A stage (64 of K)
    static constexpr int d_cols = NT < 32 ? 32 : NT;
    static constexpr int a_stages = (int)TS_TMEM - d_cols >= 4 * a_cols ? 4 : ((int)TS_TMEM - d_cols) / a_cols;
    static constexpr int x_stage = 2 * NT * 128;                                           // hi, lo
    static constexpr int x_stages = NT >= 128 ? 3 : NT >= 64 ? 6 : 8;
    static constexpr int ring = x_stages * x_stage < 96 * 1024 ? (x_stages * x_stage > NT * 512 ? x_stages * x_stage : NT * 512) : x_stages * x_stage;
    // two blocks per SM, not more: tensor memory has room for two
    static constexpr int smem = (ring + 1024 + 512 > 80 * 1024 ? ring + 1024 + 512 : 80 * 1024);
};

struct TsParams {
    const unsigned char *w, *w2;  // int4: tile-major blocks (gate and up interleaved); else the matrix (w2: up)
    const __half *scale, *scale2; // int8: row scales
    const float* unscale;         // [rows of x]
    float* dst;
    const SeqState* state;
    uint32_t rows, K, n_rows, dst_stride, x_lo_row, splits;  // rows of dst; x_lo_row: first row of the lo parts in the x map
    int epilogue;
    uint32_t *err, *stop;
    unsigned long long* trace;
};

__device__ __forceinline__ uint64_t ts_desc(uint32_t addr) {  // K-major, 128-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void ts_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void ts_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ts_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ts_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ts_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                   "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
                   "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void ts_ld16(uint32_t taddr, float (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]), "=f"(r[10]),
                   "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]) : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ bool ts_warp_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, const uint32_t* stop) {
    return __all_sync(0xFFFFFFFFu, wait_or_abort(bar, parity, abort_flag, stop));
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
__device__ __forceinline__ uint32_t word4(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// two fp32 values as fp16 hi and lo pairs
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = h2_bits(h);
    lo = h2_bits(__floats2half2_rn(a - f.x, b - f.y));
}

// 64 of K of one weight row -> the 32 columns of fp16 pairs of the A operand (hi, and lo where parts == 2).
// int4: `half` of a unit of 128.  K order: the order x is stored in; for int4 the middle two of every four are swapped (the
// nibbles of a tile-major word pair up that way without a shuffle), k_rows_split does the same to x.
template <int FMT>
__device__ __forceinline__ void ts_expand(const uint4 (&raw)[Ts<FMT>::regs], int half, bool odd_row, uint32_t (&hi)[32], uint32_t (&lo)[32]) {
    if constexpr (FMT == VB_FMT_Q4G32) {
        // raw[t]: words of the row's four groups, elements 4t..4t+3 (low nibbles) and 16+4t.. (high); raw[4]: half2 per group of
        // the scales of rows g and g + 8
        const __half2 off = __float2half2_rn(-1032.0f), inv16 = __float2half2_rn(0.0625f), off16 = __float2half2_rn(-72.0f);
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
            const uint32_t sp = word4(raw[4], 2 * half + jj);
            const __half2 s = odd_row ? __high2half2(bits_h2(sp)) : __low2half2(bits_h2(sp));
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t u = word4(raw[t], 2 * half + jj), u8 = u >> 8;
                const __half2 v[4] = {__hadd2(bits_h2(lop3_and_or(u, 0x000F000Fu, 0x64006400u)), off), __hadd2(bits_h2(lop3_and_or(u8, 0x000F000Fu, 0x64006400u)), off),
                                      __hfma2(bits_h2(lop3_and_or(u, 0x00F000F0u, 0x64006400u)), inv16, off16),
                                      __hfma2(bits_h2(lop3_and_or(u8, 0x00F000F0u, 0x64006400u)), inv16, off16)};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = jj * 16 + (i >> 1) * 8 + 2 * t + (i & 1);
                    const __half2 h = __hmul2(v[i], s);
                    hi[c] = h2_bits(h);
                    lo[c] = h2_bits(__hfma2(v[i], s, __hneg2(h)));  // exact: 15 bits of (n - 8) * s, 11 of them in h
                }
            }
        }
    } else {
        const __half2 off = __float2half2_rn(-1152.0f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t u = word4(raw[i >> 2], i & 3) ^ 0x80808080u;  // b + 128 in the low byte of 1024 as fp16
            hi[2 * i] = h2_bits(__hadd2(bits_h2(__byte_perm(u, 0x64646464u, 0x4140)), off));
            hi[2 * i + 1] = h2_bits(__hadd2(bits_h2(__byte_perm(u, 0x64646464u, 0x4342)), off));
        }
    }
}

// grid (tiles of NT rows of x, tiles of 128 weight rows, splits), clusters of `splits` along z
template <int FMT, int NT>
__global__ void __launch_bounds__(TS_THREADS, 2) k_gemm_ts(const __grid_constant__ CUtensorMap map_x, const TsParams p) {
    typedef Ts<FMT> F;
    typedef TsShape<FMT, NT> P;
    constexpr int AS = P::a_stages, XS = P::x_stages;
    constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | (8u << 24);  // fp32 accumulate, fp16 operands, M 128
    constexpr int B_XFULL = 0, B_XEMPTY = XS, B_AFULL = 2 * XS, B_AEMPTY = B_AFULL + AS, B_ACC = B_AEMPTY + AS, B_COUNT = B_ACC + 1;
    static_assert(B_COUNT * 8 + 8 <= 512 && AS >= 2, "barriers, A stages");
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = base + P::ring;
    unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + P::ring + B_COUNT * 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.y, split = blockIdx.z, S = p.splits;
    const bool swiglu = p.epilogue == EPI_SWIGLU;
    trace_mark(p.trace, 0);
    if (threadIdx.x == 0) {
        for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_AFULL && i < B_AEMPTY ? 4 : 1);
        *abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TS_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // this block's part of K, in units
    const uint32_t n_units_all = p.K / F::unit, u0 = (uint32_t)((uint64_t)n_units_all * split / S), n_units = (uint32_t)((uint64_t)n_units_all * (split + 1) / S) - u0;
    constexpr int SPU = F::unit / 64;  // A stages per unit
    const uint32_t n_st = n_units * SPU;

    // ---- dequantising warps: where this thread's weight row lies; the first units are requested before the dependency wait ----
    const uint32_t lg = warp & 3, row = lg * 32 + lane;  // tensor-memory lanes 32 * (warp % 4) .. + 31
    const bool deq = warp >= 2;
    const unsigned char* src = nullptr;
    uint4 raw[F::depth][F::regs];
    auto request = [&](uint4 (&r)[F::regs]) {
        if constexpr (F::q4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = ldg_stream(reinterpret_cast<const uint4*>(src) + i);
            const uint32_t back = 64 * (row & 7) + ((row & 8) ? 512 : 0);  // the unit's start is there
            r[4] = __ldg(reinterpret_cast<const uint4*>(src - back + 1024 + 16 * (row & 7)));
            src += TS_Q4_BLK;
        } else {
            constexpr int BYTES = F::regs * 16;
#pragma unroll
            for (int i = 0; i < F::regs; ++i) r[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
            src += BYTES;
        }
    };
    if (deq) {
        if constexpr (F::q4) {
            const uint32_t n_tiles16 = (swiglu ? 2 : 1) * p.rows / 16, t16 = min(tile * 8 + row / 16, n_tiles16 - 1);
            src = p.w + ((size_t)t16 * n_units_all + u0) * TS_Q4_BLK + 64 * (row & 7) + ((row & 8) ? 512 : 0);
        } else {
            const uint32_t r = min(swiglu ? tile * 64 + (row >> 4) * 8 + (row & 7) : tile * 128 + row, p.rows - 1);
            src = ((swiglu && (row & 8)) ? p.w2 : p.w) + ((size_t)r * p.K + (size_t)u0 * F::unit) * (F::regs * 16 / F::unit);
        }
#pragma unroll
        for (int d = 0; d < F::depth; ++d)
            if ((uint32_t)d < n_units) request(raw[d]);
    }
    ts_fence_before();
    __syncthreads();
    ts_fence_after();
    const uint32_t tmem = *tmem_slot, tm_a = tmem + P::d_cols;
    pdl_wait();
    pdl_launch_dependents();
    trace_mark(p.trace, 1);

    if (warp == 0) {
        // ---- x: the hi and the lo box of a stage ----
        if (elect_one()) {
            for (uint32_t i = 0; i < n_st; ++i) {
                const uint32_t s = i % XS;
                if (i >= XS && !wait_or_abort(bar(B_XEMPTY + s), (i / XS + 1) & 1, abort_flag, p.stop)) break;
                mbar_expect_tx(bar(B_XFULL + s), P::x_stage);
                const int kx = (int)(u0 * F::unit + i * 64), y = (int)(blockIdx.x * NT);
                const uint32_t st = base + s * P::x_stage;
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                             ::"r"(st), "l"(&map_x), "r"(kx), "r"(y), "r"(bar(B_XFULL + s)) : "memory");
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                             ::"r"(st + NT * 128), "l"(&map_x), "r"(kx), "r"(y + (int)p.x_lo_row), "r"(bar(B_XFULL + s)) : "memory");
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- tensor-core issue ----
        const bool stopped = stop_set(p.stop);  // an earlier kernel of this context gave up (looked at behind the first copies)
        for (uint32_t i = 0; i < n_st; ++i) {
            const uint32_t xs = i % XS, as = i % AS;
            if (!ts_warp_wait(bar(B_XFULL + xs), (i / XS) & 1, abort_flag, p.stop) || !ts_warp_wait(bar(B_AFULL + as), (i / AS) & 1, abort_flag, p.stop)) break;
            if (i == 0 && __any_sync(0xFFFFFFFFu, stopped)) { *abort_flag = ABORT_STOPPED; break; }
            ts_fence_after();
            if (elect_one()) {
                const uint64_t bh = ts_desc(base + xs * P::x_stage), bl = ts_desc(base + xs * P::x_stage + NT * 128);
                const uint32_t ah = tm_a + as * P::a_cols;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    ts_mma(tmem, ah + 8 * k, bh + 2u * k, IDESC, (i | (uint32_t)k) != 0 ? 1u : 0u);
                    ts_mma(tmem, ah + 8 * k, bl + 2u * k, IDESC, 1u);
                    if (F::parts == 2) ts_mma(tmem, ah + 32 + 8 * k, bh + 2u * k, IDESC, 1u);
                }
                ts_commit(bar(B_AEMPTY + as));
                ts_commit(bar(B_XEMPTY + xs));
                if (i + 1 == n_st) ts_commit(bar(B_ACC));
            }
            __syncwarp();
        }
    } else {
        // ---- weights -> tensor memory ----
        const uint32_t lane_addr = (lg * 32u) << 16;
        uint32_t i = 0;
        bool ok = true;
        for (uint32_t ub = 0; ub < n_units && ok; ub += F::depth) {
#pragma unroll
            for (int d = 0; d < F::depth; ++d) {
                if (ub + d < n_units && ok) {
                    uint32_t hi[SPU][32], lo[32];
#pragma unroll
                    for (int half = 0; half < SPU; ++half) {
                        const uint32_t as = i % AS;
                        if (i >= AS) ok = ts_warp_wait(bar(B_AEMPTY + as), (i / AS + 1) & 1, abort_flag, p.stop);
                        if (!ok) break;
                        ts_fence_after();
                        ts_expand<FMT>(raw[d], half, (row & 8) != 0, hi[half], lo);
                        ts_st32(tm_a + lane_addr + as * P::a_cols, hi[half]);
                        if (F::parts == 2) ts_st32(tm_a + lane_addr + as * P::a_cols + 32, lo);
                        if (half == SPU - 1 && ub + d + F::depth < n_units) request(raw[d]);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        ts_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(B_AFULL + as));
                        ++i;
                    }
                }
            }
        }
    }

    // ---- epilogue: lane = weight row ----
    const bool ok = n_st == 0 || wait_or_abort(bar(B_ACC), 0u, abort_flag, p.stop);
    ts_fence_after();
    const bool good = __syncthreads_and(ok && !*abort_flag);
    const uint32_t o = swiglu ? tile * 64 + (row >> 4) * 8 + (row & 7) : tile * 128 + row;
    const bool o_ok = deq && o < p.rows;
    float sc = 1.0f;
    if (FMT == VB_FMT_I8PC && o_ok) sc = __half2float((swiglu && (row & 8)) ? p.scale2[o] : p.scale[o]);
    const uint32_t t0 = blockIdx.x * NT;
    // 16 values of this lane's row (tokens t, t + 1, ...) -> dst
    auto finish = [&](float (&v)[16], uint32_t t, uint32_t count) {
        const uint32_t tl = t + (lane & 15);
        const bool live = (lane & 15) < count && tl < p.n_rows && (!p.state || p.state[tl].active);
        const uint32_t live_mask = __ballot_sync(0xFFFFFFFFu, live) & 0xFFFFu;
        const float un = live ? p.unscale[tl] : 0.0f;
        float* d = p.dst + (size_t)t * p.dst_stride + o;
        float res[16];
        if (p.epilogue == EPI_RESIDUAL) {
#pragma unroll
            for (int j = 0; j < 16; ++j) res[j] = (o_ok && ((live_mask >> j) & 1u)) ? __ldcg(d + (size_t)j * p.dst_stride) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float a = v[j] * __shfl_sync(0xFFFFFFFFu, un, j) * sc;
            bool store = o_ok && ((live_mask >> j) & 1u);
            if (swiglu) {
                const float up = __shfl_xor_sync(0xFFFFFFFFu, a, 8);
                a = (a / (1.0f + expf(-a))) * up;
                store = store && !(row & 8);
            } else if (p.epilogue == EPI_RESIDUAL) {
                a += res[j];
            }
            if (store) d[(size_t)j * p.dst_stride] = a;
        }
    };
    if (S > 1) {
        // every block of the cluster is past its last product (the ring of x is free): partial rows to the block that owns their
        // tokens, [source rank][token of the owner][128 weight rows]
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        const uint32_t per = NT / S;
        float* recv = reinterpret_cast<float*>(gen);
        if (deq && good) {
#pragma unroll 1
            for (uint32_t c = 0; c < NT; c += 16) {
                float v[16];
                ts_ld16(tmem + ((lg * 32u) << 16) + c, v);
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                    const uint32_t owner = (c + j) / per, slot = (c + j) % per;
                    cluster.map_shared_rank(recv, owner)[(split * per + slot) * 128 + row] = v[j];
                }
            }
        }
        cluster.sync();
        if (deq && good) {
#pragma unroll 1
            for (uint32_t c = 0; c < per; c += 16) {
                const uint32_t count = min(16u, per - c);
                float v[16];
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                    v[j] = 0.0f;
                    if (j < count)
                        for (uint32_t z = 0; z < S; ++z) v[j] += recv[(z * per + c + j) * 128 + row];
                }
                finish(v, t0 + split * per + c, count);
            }
        }
    } else if (deq && good) {
#pragma unroll 1
        for (uint32_t c = 0; c < NT; c += 16) {
            if (t0 + c >= p.n_rows) break;  // uniform
            float v[16];
            ts_ld16(tmem + ((lg * 32u) << 16) + c, v);
            finish(v, t0 + c, 16);
        }
    }
    if (!good) {
        if (threadIdx.x == 0) report_wait(p.err, p.stop, 0x100u);
        // let copies and products that are still in flight land before the memory they use is given back
        abort_drain(abort_flag);
    }
    ts_fence_before();
    __syncthreads();
    if (warp == 1) {
        ts_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TS_TMEM) : "memory");
    }
    trace_exit(p.trace);
}

// ---- x -> hi and lo rows ------------------------------------------------------------------------------------------------
// One block per row: RMSNorm (runtime.rs:588-601), a power of two that brings the row's maximum to [2^13, 2^14), fp16 hi and
// lo.  swap: the middle two of every four elements change places (the K order of int4 weights).  Inactive rows are left alone:
// their columns of the product are not stored.
template <int XR>
__global__ void __launch_bounds__(512) k_rows_split(__half* __restrict__ hi, __half* __restrict__ lo, float* __restrict__ unscale, const float* __restrict__ x,
                                                    const void* __restrict__ norm_w, int norm_fmt, float eps, const SeqState* __restrict__ state, uint32_t K, int swap) {
    __shared__ float red[2][16];
    const uint32_t r = blockIdx.x, K4 = K / 4;
    pdl_launch_dependents();
    float4 w[XR];
    if (norm_w) {  // parameters: on their way before the wait
#pragma unroll
        for (int i = 0; i < XR; ++i) {
            const uint32_t k = threadIdx.x + i * 512;
            w[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < K4) {
                if (norm_fmt == VB_FMT_F32) {
                    w[i] = __ldg(reinterpret_cast<const float4*>(norm_w) + k);
                } else {
                    const uint2 q = __ldg(reinterpret_cast<const uint2*>(norm_w) + k);
                    if (norm_fmt == VB_FMT_F16) {
                        const float2 a = __half22float2(bits_h2(q.x)), b = __half22float2(bits_h2(q.y));
                        w[i] = make_float4(a.x, a.y, b.x, b.y);
                    } else {
                        w[i] = make_float4(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xFFFF0000u), __uint_as_float(q.y << 16), __uint_as_float(q.y & 0xFFFF0000u));
                    }
                }
            }
        }
    }
    pdl_wait();
    if (state && !state[r].active) return;
    const float4* in = reinterpret_cast<const float4*>(x + (size_t)r * K);
    float4 v[XR];
    float ss = 0.0f, mx = 0.0f;
#pragma unroll
    for (int i = 0; i < XR; ++i) {
        const uint32_t k = threadIdx.x + i * 512;
        v[i] = k < K4 ? in[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < XR; ++i) {
        ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
        if (norm_w) { v[i].x *= w[i].x; v[i].y *= w[i].y; v[i].z *= w[i].z; v[i].w *= w[i].w; }
        mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
    }
    ss = warp_sum(ss); mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = ss; red[1][threadIdx.x >> 5] = mx; }
    __syncthreads();
    ss = 0.0f; mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) { ss += red[0][i]; mx = fmaxf(mx, red[1][i]); }
    // norm and scale in one factor: up is a power of two, so (x * w) * (inv * up) rounds like (x * w * inv) does
    const float inv = norm_w ? 1.0f / sqrtf(ss / (float)K + eps) : 1.0f;
    mx *= inv;
    float up = 1.0f;
    if (mx > 0.0f && mx < 3.0e38f) {
        const int e = min(max((int)((__float_as_uint(mx) >> 23) & 255u) - 127, -100), 113);
        up = __uint_as_float((uint32_t)(127 + 13 - e) << 23);
    }
    if (threadIdx.x == 0) unscale[r] = 1.0f / up;
    const float f = inv * up;
    uint2* oh = reinterpret_cast<uint2*>(hi + (size_t)r * K);
    uint2* ol = reinterpret_cast<uint2*>(lo + (size_t)r * K);
#pragma unroll
    for (int i = 0; i < XR; ++i) {
        const uint32_t k = threadIdx.x + i * 512;
        if (k < K4) {
            const float a = v[i].x * f, b = (swap ? v[i].z : v[i].y) * f, c = (swap ? v[i].y : v[i].z) * f, d = v[i].w * f;
            uint2 h, l;
            split2(a, b, h.x, l.x);
            split2(c, d, h.y, l.y);
            oh[k] = h;
            ol[k] = l;
        }
    }
}


template <int FMT, int NT>
cudaError_t ts_launch(const LaunchCfg& lc, const CUtensorMap& map, TsParams p, uint32_t token_tiles, uint32_t row_tiles) {
    typedef TsShape<FMT, NT> P;
    static std::atomic<uint64_t> opted{0};
    const cudaError_t oe = once_per_device(opted, [&]() { return cudaFuncSetAttribute(k_gemm_ts<FMT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::smem); });
    if (oe != cudaSuccess) return oe;
    // Split K over a cluster while that shortens the busiest SM's share (the last wave of whole tiles is mostly empty) and every
    // block keeps eight stages.
    const uint32_t tiles = token_tiles * row_tiles, units = p.K / Ts<FMT>::unit;
    uint32_t best = 1;
    double best_cost = 1e30;
    for (uint32_t s = 1; s <= 8 && s <= (uint32_t)NT; s *= 2) {
        if (s > 1 && units * (Ts<FMT>::unit / 64) < 8 * s) break;
        const double waves = (double)((tiles * s + 147) / 148), cost = waves / s * (1.0 + 0.04 * (s > 1)) + 0.02 * s;
        if (cost < best_cost - 1e-9) { best_cost = cost; best = s; }
    }
    p.splits = best;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(token_tiles, row_tiles, best);
    cfg.blockDim = dim3(TS_THREADS);
    cfg.dynamicSmemBytes = P::smem;
    cfg.stream = lc.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = best;
    cfg.numAttrs = 1;
    if (lc.pdl) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    cfg.attrs = attr;
    if (lc.counter) ++*lc.counter;
    return cudaLaunchKernelEx(&cfg, k_gemm_ts<FMT, NT>, map, p);
}
template <int FMT>
cudaError_t ts_launch_nt(const LaunchCfg& lc, const CUtensorMap& map, const TsParams& p, uint32_t nt, uint32_t row_tiles) {
    const uint32_t tt = (p.n_rows + nt - 1) / nt;
    if (nt == 16) return ts_launch<FMT, 16>(lc, map, p, tt, row_tiles);
    if (nt == 32) return ts_launch<FMT, 32>(lc, map, p, tt, row_tiles);
    if (nt == 64) return ts_launch<FMT, 64>(lc, map, p, tt, row_tiles);
    return ts_launch<FMT, 128>(lc, map, p, tt, row_tiles);
}

}  // namespace

bool gemm_ts_supported(const GemvArgs& a) {
    const bool dual = a.epilogue == EPI_SWIGLU;
    if (a.push.links || a.w.rows == 0 || a.w.cols == 0 || a.w.cols > 32768) return false;
    if (dual && (a.w2.fmt != a.w.fmt || a.w2.rows != a.w.rows || a.w2.cols != a.w.cols)) return false;
    if (a.w.fmt == VB_FMT_Q4G32) return (dual ? a.w.v3_swiglu : a.w.v3) && a.w.cols % 128 == 0 && a.w.rows % (dual ? 8 : 16) == 0;
    return a.w.fmt == VB_FMT_I8PC && a.w.data && a.w.scales && (!dual || (a.w2.data && a.w2.scales)) && a.w.cols % 64 == 0 &&
           (((uintptr_t)a.w.data | (uintptr_t)a.w2.data) & 15) == 0;
}
// rows of x a tile takes: the smallest of 16, 32, 64, 128 that holds them all, else 128
static uint32_t ts_tile_rows(uint32_t n_rows) { return n_rows <= 16 ? 16 : n_rows <= 32 ? 32 : n_rows <= 64 ? 64 : 128; }
uint64_t gemm_ts_workspace_bytes(uint32_t in_dim, uint32_t n_rows) {
    const uint64_t nt = ts_tile_rows(n_rows), pad = (n_rows + nt - 1) / nt * nt;
    return pad * in_dim * 4 + pad * 4 + 1024;
}

cudaError_t gemm_ts(const LaunchCfg& lc, const GemvArgs& a, void* workspace, uint64_t workspace_bytes) {
    if (!gemm_ts_supported(a) || !encode_tiled_fn()) return cudaErrorInvalidValue;
    const uint32_t K = a.w.cols, n_rows = a.batch;
    if (n_rows == 0) return cudaSuccess;
    if (gemm_ts_workspace_bytes(K, n_rows) > workspace_bytes || ((uintptr_t)workspace & 15) != 0) return cudaErrorInvalidValue;
    const bool dual = a.epilogue == EPI_SWIGLU, q4 = a.w.fmt == VB_FMT_Q4G32;
    const uint32_t nt = ts_tile_rows(n_rows), pad = (n_rows + nt - 1) / nt * nt;
    __half* hi = reinterpret_cast<__half*>(workspace);
    __half* lo = hi + (size_t)pad * K;
    float* unscale = reinterpret_cast<float*>(lo + (size_t)pad * K);
    cudaError_t e;
    if (K <= 4096) e = launch(lc, k_rows_split<2>, dim3(n_rows), dim3(512), 0, hi, lo, unscale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, q4 ? 1 : 0);
    else if (K <= 8192) e = launch(lc, k_rows_split<4>, dim3(n_rows), dim3(512), 0, hi, lo, unscale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, q4 ? 1 : 0);
    else if (K <= 20480) e = launch(lc, k_rows_split<10>, dim3(n_rows), dim3(512), 0, hi, lo, unscale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, q4 ? 1 : 0);
    else e = launch(lc, k_rows_split<16>, dim3(n_rows), dim3(512), 0, hi, lo, unscale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, q4 ? 1 : 0);
    if (e != cudaSuccess) return e;
    CUtensorMap map;
    const cuuint64_t dims[2] = {K, 2ull * pad};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, nt}, estr[2] = {1, 1};
    if (encode_tiled_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, hi, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorNotSupported;
    TsParams p = {};
    p.w = (const unsigned char*)(q4 ? (dual ? a.w.v3_swiglu : a.w.v3) : a.w.data);
    p.w2 = (const unsigned char*)a.w2.data;
    p.scale = (const __half*)a.w.scales; p.scale2 = (const __half*)a.w2.scales;
    p.unscale = unscale;
    p.dst = a.dst + a.dst_offset;
    p.state = a.state;
    p.rows = a.w.rows; p.K = K; p.n_rows = n_rows; p.dst_stride = a.dst_stride ? a.dst_stride : a.w.rows; p.x_lo_row = pad;
    p.epilogue = a.epilogue;
    p.trace = a.trace;
    error_words(lc, &p.err, &p.stop);
    const uint32_t row_tiles = (a.w.rows * (dual ? 2 : 1) + 127) / 128;
    return q4 ? ts_launch_nt<VB_FMT_Q4G32>(lc, map, p, nt, row_tiles) : ts_launch_nt<VB_FMT_I8PC>(lc, map, p, nt, row_tiles);
}

}  // namespace vb
