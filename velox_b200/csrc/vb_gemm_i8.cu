// Decode batches over int8 per-channel weights on the integer tensor cores (tcgen05.mma kind::i8): the weights cross
// HBM as the bytes they are stored as -- no fp16 copy, one byte per weight -- and the arithmetic is exact.
//
// What it replaces: the reference's multi-token register-tiled kernels (velox_cuda_runner_k2.cu:480-1085) for the
// projections of a batched decode step, dst[t][o] = sum_k x[t][k] * q[o][k] * scale[o] for up to 32 rows t.
//
//   * x rows (with the reference's RMSNorm folded in, runtime.rs:588-601) become fixed point per row, X = rint(x * p), stored as signed
//     byte planes, the highest first: up to 16 rows as three planes (24 bits, p = 8.3e6 / the row's largest magnitude: X = 65536 * H +
//     256 * M + L, operand rows 0..15 / 16..31 / 32..47), 17 to 32 rows as two (16 bits, p = 32000 / that: X = 256 * H + L, rows 0..31 /
//     32..63) -- k_rows_to_i8;
//   * the weights are read where they lie, canonical int8 [out][K], by tiled TMA ([128 rows][128 bytes] boxes,
//     128-byte swizzle), or from copies in that order; one tcgen05.mma kind::i8 (M 128, N 48 or 64, K 32) per 32 bytes of K accumulates
//     int32 in tensor memory, one column per plane and row, exact;
//   * the epilogue adds the planes' sums in int64, forms their product with scale[o] / p in fp32 and stores / adds the residual / applies
//     SiLU(gate) * up; products with few row tiles split K over several blocks, the last one to arrive sums the fp32
//     partial tiles in split order (the same bits whoever is last).
// Every wait is bounded; a wait that runs out sets a block-wide abort flag and the library's error word.
#include <cuda.h>

#include <algorithm>

#include "vb_kernels.cuh"
#include "vb_tma.cuh"

namespace vb {
namespace {

constexpr int I8_BM = 128;               // weight rows per tile (UMMA M)
constexpr int I8_BK = 128;               // bytes of K per stage: one 128-byte swizzle row
constexpr int I8_W_BYTES = I8_BM * I8_BK;  // 16 KB
// rows of x of a pass, their byte planes, operand rows (UMMA N)
template <int ROWS> struct I8Shape {
    static constexpr int planes = ROWS == 16 ? 3 : 2, n = planes * ROWS, x_bytes = n * I8_BK;
    // instruction descriptor of tcgen05.mma kind::i8: int32 accumulate (bits 4-5 = 2), A and B signed 8-bit (formats 1 at
    // bits 7-9 and 10-12), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    static constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(I8_BM >> 4) << 24);
    static __host__ __device__ constexpr int stage(bool dual) { return (dual ? 2 : 1) * I8_W_BYTES + x_bytes; }
};
constexpr int I8_TMEM = 64;              // columns of a product's accumulators
constexpr int I8_SMEM = 192 * 1024 + 1024 + 256;

__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}"
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void commit_to(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32i(uint32_t taddr, int r[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
                   "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
                   "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
struct I8Params {
    float* dst;                 // [n_rows][dst_stride], column offset applied
    const __half* row_scale;    // [out_dim] weight row scales
    const __half* row_scale2;   // gate/up: the up matrix's
    const float* x_inv_scale;   // [32] 1 / p of every row of x
    const SeqState* state;
    uint32_t out_dim, n_rows, K, dst_stride;
    int epilogue;
    uint32_t *err, *stop;
    float* part;                // [split][tile][32 cols][128 lanes] fp32 partial tiles
    uint32_t* counters;         // [tile], zero between launches
    uint32_t stages;
    unsigned long long* trace;  // time stamps of this launch (vb_trace_read), or null
    // tile-major copies of the weights in shared-memory order (null: tiled TMA from the canonical matrices): a tile is one
    // contiguous 16 KB bulk copy -- sequential DRAM pages instead of 128 rows of 128 bytes a whole matrix row apart
    const unsigned char* w_tiles;
    const unsigned char* w2_tiles;
};

template <bool DUAL, int ROWS>
__global__ void __launch_bounds__(128, 1)
k_gemm_i8(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x,
          const I8Params p) {
    constexpr int W_TILES = DUAL ? 2 : 1;
    typedef I8Shape<ROWS> S;
    constexpr int STAGE_BYTES = S::stage(DUAL);
    constexpr uint32_t TMEM_COLS = W_TILES * I8_TMEM;
    const int STAGES = (int)p.stages;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = base + STAGES * STAGE_BYTES;  // full[STAGES], empty[STAGES], accum, then two words
    const uint32_t bar_accum = bars + 2 * STAGES * 8;
    unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + STAGES * STAGE_BYTES + (2 * STAGES + 1) * 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int row0 = blockIdx.y * I8_BM;
    const int nk_all = (int)((p.K + I8_BK - 1) / I8_BK);
    const int kb_first = (int)(((long long)nk_all * blockIdx.z) / gridDim.z), kb_last = (int)(((long long)nk_all * (blockIdx.z + 1)) / gridDim.z);
    const int nk = kb_last - kb_first;
    trace_mark(p.trace, 0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(bars + s * 8, 1); mbar_init(bars + (STAGES + s) * 8, 1); }
        mbar_init(bar_accum, 1);
        *abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
      if (elect_one()) {
        // weights do not depend on the kernel before this one: the whole ring of weight tiles is requested before the
        // dependency wait, the planes of x (written by the conversion kernel in front) after it
        const int pre = nk < STAGES ? nk : STAGES;
        for (int kb = 0; kb < pre; ++kb) {
            const uint32_t full = bars + kb * 8, st = base + kb * STAGE_BYTES;
            mbar_expect_tx(full, STAGE_BYTES);
            const int kx = (kb_first + kb) * I8_BK;
            if (p.w_tiles) {
                const size_t toff = ((size_t)blockIdx.y * nk_all + kb_first + kb) * I8_W_BYTES;
                tma_load_1d(st, p.w_tiles + toff, I8_W_BYTES, full);
                if (DUAL) tma_load_1d(st + I8_W_BYTES, p.w2_tiles + toff, I8_W_BYTES, full);
            } else {
                tma_2d(st, &map_w, kx, row0, full);
                if (DUAL) tma_2d(st + I8_W_BYTES, &map_w2, kx, row0, full);
            }
        }
        pdl_wait();
        trace_mark(p.trace, 1);
        for (int kb = 0; kb < pre; ++kb) tma_2d(base + kb * STAGE_BYTES + W_TILES * I8_W_BYTES, &map_x, (kb_first + kb) * I8_BK, 0, bars + kb * 8);
        for (int kb = pre; kb < nk; ++kb) {
            const int s = kb % STAGES;
            const uint32_t ph = (uint32_t)(kb / STAGES) & 1u;
            if (!wait_or_abort(bars + (STAGES + s) * 8, ph ^ 1u, abort_flag, p.stop)) break;
            const uint32_t full = bars + s * 8, st = base + s * STAGE_BYTES;
            mbar_expect_tx(full, STAGE_BYTES);
            const int kx = (kb_first + kb) * I8_BK;
            if (p.w_tiles) {
                const size_t toff = ((size_t)blockIdx.y * nk_all + kb_first + kb) * I8_W_BYTES;
                tma_load_1d(st, p.w_tiles + toff, I8_W_BYTES, full);
                if (DUAL) tma_load_1d(st + I8_W_BYTES, p.w2_tiles + toff, I8_W_BYTES, full);
            } else {
                tma_2d(st, &map_w, kx, row0, full);
                if (DUAL) tma_2d(st + I8_W_BYTES, &map_w2, kx, row0, full);
            }
            tma_2d(st + W_TILES * I8_W_BYTES, &map_x, kx, 0, full);
        }
      }
    } else if (warp == 1) {
        const bool stopped = stop_set(p.stop);  // an earlier kernel of this context gave up (looked at behind the first copies)
        // the warp waits together, an elected lane issues (vb_tma.cuh)
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % STAGES;
            const uint32_t ph = (uint32_t)(kb / STAGES) & 1u;
            if (!__all_sync(0xFFFFFFFFu, wait_or_abort(bars + s * 8, ph, abort_flag, p.stop))) break;
            if (kb == 0 && __any_sync(0xFFFFFFFFu, stopped)) { *abort_flag = ABORT_STOPPED; break; }
            fence_after();
            const uint32_t st = base + s * STAGE_BYTES;
            if (elect_one()) {
            const uint64_t da = smem_desc_sw128(st), da2 = smem_desc_sw128(st + I8_W_BYTES), db = smem_desc_sw128(st + W_TILES * I8_W_BYTES);
#pragma unroll
            for (int k = 0; k < I8_BK / 32; ++k) {  // 32 bytes further along the swizzled row: +2 in the address field
                const uint32_t acc = (kb | k) != 0 ? 1u : 0u;
                mma_i8(tmem, da + 2u * k, db + 2u * k, S::idesc, acc);
                if (DUAL) mma_i8(tmem + I8_TMEM, da2 + 2u * k, db + 2u * k, S::idesc, acc);
            }
            commit_to(bars + (STAGES + s) * 8);
            if (kb == nk - 1) commit_to(bar_accum);
            }
            __syncwarp();
        }
    }
    __syncwarp();
    pdl_wait();               // every thread: the epilogue reads the residual stream and x scales of earlier kernels
    pdl_launch_dependents();

    // the scales of x and which of its rows are live, once per block (warp 0), for every lane's 32 columns
    __shared__ float s_inv[32];
    __shared__ uint32_t s_live_mask;
    if (warp == 0) {
        s_inv[lane] = lane < ROWS ? p.x_inv_scale[lane] : 0.0f;
        const bool live = lane < p.n_rows && (!p.state || p.state[lane].active);
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, live);
        if (lane == 0) s_live_mask = m;
    }
    const bool ok = wait_or_abort(bar_accum, 0u, abort_flag, p.stop);
    fence_after();
    const bool good = __syncthreads_and(ok && !*abort_flag);
    if (good) {
        const uint32_t o = (uint32_t)row0 + warp * 32 + lane;
        const bool o_ok = o < p.out_dim;
        const float sc = o_ok ? __half2float(p.row_scale[o]) : 0.0f;
        const float sc2 = (DUAL && o_ok) ? __half2float(p.row_scale2[o]) : 0.0f;
        const uint32_t lane_addr = tmem + ((warp * 32u) << 16);
        const uint32_t n_split = gridDim.z, tile = blockIdx.y, n_tiles = gridDim.y;
        // row j of x: its planes' sums by their powers of 256, exact in int64, to fp32 once
        float v[ROWS], u[ROWS];
        auto sums = [&](float (&y)[ROWS], uint32_t at) {
            int h[32], l[32];
            tmem_ld32i(at, h);
            tmem_ld32i(at + 32, l);  // (three planes: 48 columns, the rest is not looked at)
#pragma unroll
            for (int j = 0; j < ROWS; ++j)
                y[j] = S::planes == 3 ? (float)(((long long)h[j] * 256 + (long long)h[(ROWS + j) & 31]) * 256 + (long long)l[j]) : (float)((long long)h[j] * 256 + (long long)l[j]);
        };
        sums(v, lane_addr);
        if (DUAL) sums(u, lane_addr + I8_TMEM);
        bool reduce = false;
        if (!DUAL && n_split > 1) {
            __shared__ uint32_t s_last;
            float* pt = p.part + (((size_t)blockIdx.z * n_tiles + tile) * ROWS) * 128 + threadIdx.x;
#pragma unroll
            for (int j = 0; j < ROWS; ++j) __stcg(pt + j * 128, v[j]);
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                const uint32_t old = atomicAdd(p.counters + tile, 1u);
                s_last = old == n_split - 1 ? 1u : 0u;
                if (s_last) { p.counters[tile] = 0u; __threadfence(); }
            }
            __syncthreads();
            reduce = s_last != 0u;
            if (reduce) {
#pragma unroll
                for (int j = 0; j < ROWS; ++j) v[j] = 0.0f;
                for (uint32_t z = 0; z < n_split; ++z) {
                    const float* ps = p.part + (((size_t)z * n_tiles + tile) * ROWS) * 128 + threadIdx.x;
#pragma unroll
                    for (int j = 0; j < ROWS; ++j) v[j] += __ldcg(ps + j * 128);
                }
            }
        }
        if ((DUAL || n_split == 1 || reduce) && o_ok) {
            const uint32_t live_mask = s_live_mask;
            float* d0 = p.dst + o;
            float res[ROWS];
            if (!DUAL && p.epilogue == EPI_RESIDUAL) {
#pragma unroll
                for (int j = 0; j < ROWS; ++j) res[j] = ((live_mask >> j) & 1u) ? __ldcg(d0 + (size_t)j * p.dst_stride) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                const float inv = s_inv[j];
                if (!((live_mask >> j) & 1u)) continue;
                const float a = (v[j] * inv) * sc;
                if (DUAL) {
                    const float up = (u[j] * inv) * sc2;
                    d0[(size_t)j * p.dst_stride] = (a / (1.0f + expf(-a))) * up;
                } else if (p.epilogue == EPI_RESIDUAL) {
                    d0[(size_t)j * p.dst_stride] = res[j] + a;
                } else {
                    d0[(size_t)j * p.dst_stride] = a;
                }
            }
        }
    } else {
        if (threadIdx.x == 0) report_wait(p.err, p.stop, 0x80u);
        abort_drain(abort_flag);
    }
    fence_before();
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    trace_exit(p.trace);
}

// What brings a row's largest magnitude (m, below) to the top of its planes; 1 for an all-zero or non-finite row.
template <int ROWS>
__device__ __forceinline__ float row_scale_i8(float m) {
    if (!(m > 0.0f && m <= 3.4028235e38f)) return 1.0f;
    if constexpr (I8Shape<ROWS>::planes == 2) {
        const float pw = m < 8.0e37f ? __fdividef(32000.0f, m) : 32000.0f / m;  // (the fast quotient is 0 from 2^126 on)
        return pw < 3.0e38f ? pw : 1.0f;
    } else {
        return fminf(8300000.0f / m, 5.0e37f);
    }
}
// What takes it back.  A row with a value that is not finite must not give numbers, however many rows share the step.
__device__ __forceinline__ float inv_scale_i8(float m, float pw) { return m <= 3.4028235e38f ? 1.0f / pw : __int_as_float(0x7FC00000); }
// the largest |x| in the order of the bits, NaN on top
__device__ __forceinline__ float row_max_i8(float m, const float4& v) {
    const uint32_t s = 0x7FFFFFFFu;
    return __uint_as_float(max(__float_as_uint(m), max(max(__float_as_uint(v.x) & s, __float_as_uint(v.y) & s), max(__float_as_uint(v.z) & s, __float_as_uint(v.w) & s))));
}
__device__ __forceinline__ float warp_max_i8(float m) { return __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m))); }
// four values as bytes of the planes, `K` apart
template <int ROWS>
__device__ __forceinline__ void store_planes(int8_t* row, size_t plane, uint32_t k, const float4& v, float pw) {
    const float e[4] = {v.x, v.y, v.z, v.w};
    constexpr int P = I8Shape<ROWS>::planes;
    uint32_t w[P] = {};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int X = __float2int_rn(e[j] * pw);
        constexpr int most = P == 2 ? 32639 : 8355711;
        X = max(-most, min(most, X));
#pragma unroll
        for (int i = P - 1; i > 0; --i) {
            const int H = (X + 128) >> 8;
            w[i] |= (uint32_t)((X - (H << 8)) & 0xFF) << (8 * j);
            X = H;
        }
        w[0] |= (uint32_t)(X & 0xFF) << (8 * j);
    }
#pragma unroll
    for (int i = 0; i < P; ++i) reinterpret_cast<uint32_t*>(row + i * plane)[k] = w[i];
}

// One block per row of x (ROWS blocks): planes[i * ROWS + r][k] = plane i (the highest first) of X = rint(norm(x) * p); inv_scale[r] = 1 / p.
// Rows of inactive slots and rows past n_rows are zeros.
template <int ROWS>
__global__ void __launch_bounds__(256)
k_rows_to_i8(int8_t* __restrict__ planes, float* __restrict__ inv_scale, const float* __restrict__ x, const void* __restrict__ norm_w, int norm_fmt,
             float eps, const SeqState* __restrict__ state, uint32_t K, uint32_t n_rows) {
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t r = blockIdx.x;
    int8_t* row = planes + (size_t)r * K;
    const size_t plane = (size_t)ROWS * K;
    const bool live = r < n_rows && (!state || state[r].active);
    const uint32_t K4 = K / 4;
    if (!live) {
        for (uint32_t k = threadIdx.x; k < K4; k += blockDim.x) store_planes<ROWS>(row, plane, k, make_float4(0.f, 0.f, 0.f, 0.f), 0.0f);
        if (threadIdx.x == 0) inv_scale[r] = 0.0f;
        return;
    }
    __shared__ float part[8], part_mx[8];
    const float4* in4 = reinterpret_cast<const float4*>(x + (size_t)r * K);
    float inv = 1.0f;
    if (norm_w) {
        float ss = 0.0f;
        for (uint32_t k = threadIdx.x; k < K4; k += blockDim.x) {
            const float4 v = in4[k];
            ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
        }
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
        __syncthreads();
        float tot = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) tot += part[i];
        inv = 1.0f / sqrtf(tot / (float)K + eps);
    }
    auto normed = [&](uint32_t k) {
        float4 v = in4[k];
        if (norm_w) {
            float4 w;
            if (norm_fmt == VB_FMT_F16) {
                const uint2 raw = reinterpret_cast<const uint2*>(norm_w)[k];
                const float2 w01 = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), w23 = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
                w = make_float4(w01.x, w01.y, w23.x, w23.y);
            } else {
                w = reinterpret_cast<const float4*>(norm_w)[k];
            }
            v.x = (v.x * inv) * w.x; v.y = (v.y * inv) * w.y; v.z = (v.z * inv) * w.z; v.w = (v.w * inv) * w.w;
        }
        return v;
    };
    float mx = 0.0f;
    for (uint32_t k = threadIdx.x; k < K4; k += blockDim.x) {
        mx = row_max_i8(mx, normed(k));
    }
    mx = warp_max_i8(mx);
    if ((threadIdx.x & 31) == 0) part_mx[threadIdx.x >> 5] = mx;
    __syncthreads();
    float gmax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) gmax = row_max_i8(gmax, make_float4(part_mx[i], 0.f, 0.f, 0.f));
    const float pw = row_scale_i8<ROWS>(gmax);
    if (threadIdx.x == 0) inv_scale[r] = inv_scale_i8(gmax, pw);
    for (uint32_t k = threadIdx.x; k < K4; k += blockDim.x) store_planes<ROWS>(row, plane, k, normed(k), pw);
}

// The same conversion for rows of up to 4096 * XR elements in one trip through memory: 1024 threads hold the row in
// registers (XR float4 each), so the sum of squares, the largest magnitude and the two byte planes all come from one
// load; the three passes of the kernel above cost three dependent round trips per row (5-9 us, four times a layer).
template <int XR, int ROWS>
__global__ void __launch_bounds__(1024)
k_rows_to_i8_regs(int8_t* __restrict__ planes, float* __restrict__ inv_scale, const float* __restrict__ x, const void* __restrict__ norm_w,
                  int norm_fmt, float eps, const SeqState* __restrict__ state, uint32_t K, uint32_t n_rows) {
    pdl_launch_dependents();  // the product's set-up (tensor maps, tensor memory, its first weight tiles) runs beside this
    const uint32_t r = blockIdx.x, K4 = K / 4, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int8_t* row = planes + (size_t)r * K;
    const size_t plane = (size_t)ROWS * K;
    __shared__ float red[32];
    __shared__ float bc[2];
    // norm weights are weights: on their way before the producer of x is done
    float4 w[XR];
    if (norm_w) {
#pragma unroll
        for (int i = 0; i < XR; ++i) {
            const uint32_t k = threadIdx.x + i * 1024;
            w[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < K4) {
                if (norm_fmt == VB_FMT_F16) {
                    const uint2 raw = reinterpret_cast<const uint2*>(norm_w)[k];
                    const float2 w01 = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), w23 = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
                    w[i] = make_float4(w01.x, w01.y, w23.x, w23.y);
                } else {
                    w[i] = reinterpret_cast<const float4*>(norm_w)[k];
                }
            }
        }
    }
    pdl_wait();
    const bool live = r < n_rows && (!state || state[r].active);
    if (!live) {
        for (uint32_t k = threadIdx.x; k < K4; k += blockDim.x) store_planes<ROWS>(row, plane, k, make_float4(0.f, 0.f, 0.f, 0.f), 0.0f);
        if (threadIdx.x == 0) inv_scale[r] = 0.0f;
        return;
    }
    const float4* in4 = reinterpret_cast<const float4*>(x + (size_t)r * K);
    float4 v[XR];
#pragma unroll
    for (int i = 0; i < XR; ++i) {
        const uint32_t k = threadIdx.x + i * 1024;
        v[i] = k < K4 ? in4[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (norm_w) {
        // the same order of squares within a thread as the three-pass kernel would not be reproducible anyway (other
        // thread count); the checker's bound is on the product, not on these bits
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < XR; ++i) { ss = fmaf(v[i].x, v[i].x, ss); ss = fmaf(v[i].y, v[i].y, ss); ss = fmaf(v[i].z, v[i].z, ss); ss = fmaf(v[i].w, v[i].w, ss); }
        ss = warp_sum(ss);
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        if (warp == 0) {
            float t = warp_sum(red[lane]);
            if (lane == 0) bc[0] = 1.0f / sqrtf(t / (float)K + eps);
        }
        __syncthreads();
        const float inv = bc[0];
#pragma unroll
        for (int i = 0; i < XR; ++i) {
            v[i].x = (v[i].x * inv) * w[i].x; v[i].y = (v[i].y * inv) * w[i].y; v[i].z = (v[i].z * inv) * w[i].z; v[i].w = (v[i].w * inv) * w[i].w;
        }
    }
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < XR; ++i) mx = row_max_i8(mx, v[i]);
    mx = warp_max_i8(mx);
    __syncthreads();  // red[] is read no more
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    if (warp == 0) {
        const float g = warp_max_i8(red[lane]);
        if (lane == 0) bc[1] = g;
    }
    __syncthreads();
    const float gmax = bc[1], pw = row_scale_i8<ROWS>(gmax);
    if (threadIdx.x == 0) inv_scale[r] = inv_scale_i8(gmax, pw);
#pragma unroll
    for (int i = 0; i < XR; ++i) {
        const uint32_t k = threadIdx.x + i * 1024;
        if (k < K4) store_planes<ROWS>(row, plane, k, v[i], pw);
    }
}

// dst tile (row tile rt, k block kb) at ((rt * n_kb) + kb) * 16 KB: byte b of the 16-byte piece c of row r at
// r * 128 + ((c ^ (r & 7)) << 4) + b -- what a tiled TMA copy with the 128-byte swizzle would have written; rows past the
// matrix are zeros.  One thread per 16-byte piece.
__global__ void __launch_bounds__(256)
k_tile_i8_umma(uint4* __restrict__ dst, const int8_t* __restrict__ src, uint32_t rows, uint32_t K, uint32_t n_kb, uint64_t n_pieces) {
    const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n_pieces) return;
    const uint32_t c = (uint32_t)(i & 7), r = (uint32_t)((i >> 3) & 127);
    const uint64_t tile = i >> 10;
    const uint32_t kb = (uint32_t)(tile % n_kb), rt = (uint32_t)(tile / n_kb);
    const uint32_t row = rt * 128 + r;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (row < rows) v = *reinterpret_cast<const uint4*>(src + (size_t)row * K + (size_t)kb * 128 + c * 16);
    dst[tile * 1024 + r * 8 + (c ^ (r & 7))] = v;
}

// int8 [rows][K] row-major, boxes of [box_rows][128 bytes], 128-byte swizzle, zeros outside the matrix
bool make_map_i8(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t K, uint32_t box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {K, rows};
    const cuuint64_t strides[1] = {K};
    const cuuint32_t box[2] = {I8_BK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr uint64_t I8_COUNTER_BYTES = 64 * 1024, I8_PART_BYTES = 4 * 1024 * 1024;

}  // namespace

bool gemm_i8_half_ring = true;  // vb_set_option("i8_half_ring", 0): every block of k_gemm_i8 takes a whole SM's shared memory
bool gemm_i8_tiles = true;  // vb_set_option("i8_tiles", 0): weight tiles by tiled TMA from the canonical matrices instead of the tile-major copies
bool gemm_i8_enabled = true;  // vb_set_option("decode_gemm_i8", 0): decode batches over int8 weights go through the fp16 copies again

// a kernel's shared memory is set once per device, as much as its deepest ring takes
template <bool DUAL, int ROWS>
static cudaError_t launch_i8(const LaunchCfg& lc, dim3 grid, const CUtensorMap& mw, const CUtensorMap& mw2, const CUtensorMap& mx, const I8Params& p) {
    static std::atomic<uint64_t> opted{0};
    const cudaError_t e = once_per_device(opted, []() { return cudaFuncSetAttribute(k_gemm_i8<DUAL, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, I8_SMEM); });
    if (e != cudaSuccess) return e;
    return launch(lc, k_gemm_i8<DUAL, ROWS>, grid, dim3(128), (size_t)p.stages * I8Shape<ROWS>::stage(DUAL) + 1024 + 256, mw, mw2, mx, p);
}
template <int ROWS>
static cudaError_t launch_rows(const LaunchCfg& lc, const GemvArgs& a, int8_t* planes, float* inv_scale) {
    const uint32_t K = a.w.cols;
    if (K <= 4096) return launch(lc, k_rows_to_i8_regs<1, ROWS>, dim3(ROWS), dim3(1024), 0, planes, inv_scale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, a.batch);
    if (K <= 8192) return launch(lc, k_rows_to_i8_regs<2, ROWS>, dim3(ROWS), dim3(1024), 0, planes, inv_scale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, a.batch);
    if (K <= 20480) return launch(lc, k_rows_to_i8_regs<5, ROWS>, dim3(ROWS), dim3(1024), 0, planes, inv_scale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, a.batch);
    return launch(lc, k_rows_to_i8<ROWS>, dim3(ROWS), dim3(256), 0, planes, inv_scale, a.x, a.norm_w, a.norm_fmt, a.eps, a.state, K, a.batch);
}

bool gemm_i8_supported(const GemvArgs& a) {
    if (!gemm_i8_enabled || a.w.fmt != VB_FMT_I8PC || a.batch == 0 || a.batch > 32 || !a.w.data || !a.w.scales) return false;
    if (a.w.cols % 16 != 0 || a.w.rows == 0 || ((uintptr_t)a.w.data & 15) != 0) return false;
    if (a.epilogue == EPI_SWIGLU && (a.w2.fmt != VB_FMT_I8PC || a.w2.rows != a.w.rows || a.w2.cols != a.w.cols || !a.w2.data || !a.w2.scales ||
                                     ((uintptr_t)a.w2.data & 15) != 0))
        return false;
    return a.push.links == nullptr;
}

uint64_t gemm_i8_tiles_bytes(uint32_t rows, uint32_t K) {
    return K % I8_BK ? 0 : (uint64_t)((rows + I8_BM - 1) / I8_BM) * (K / I8_BK) * I8_W_BYTES;
}
cudaError_t gemm_i8_make_tiles(const LaunchCfg& lc, void* dst, const void* src_i8, uint32_t rows, uint32_t K) {
    if (K % I8_BK != 0 || ((uintptr_t)dst & 15) != 0 || ((uintptr_t)src_i8 & 15) != 0) return cudaErrorInvalidValue;
    const uint32_t n_kb = K / I8_BK;
    const uint64_t n_pieces = gemm_i8_tiles_bytes(rows, K) / 16;
    return launch(lc, k_tile_i8_umma, dim3((unsigned)((n_pieces + 255) / 256)), dim3(256), 0, reinterpret_cast<uint4*>(dst),
                  reinterpret_cast<const int8_t*>(src_i8), rows, K, n_kb, n_pieces);
}

// workspace head: tile counters (zero before the first call) and partial tiles, then the planes of x and their scales
uint64_t gemm_i8_workspace_bytes(uint32_t in_dim) {
    return I8_COUNTER_BYTES + I8_PART_BYTES + (((uint64_t)64 * in_dim + 1023) / 1024 * 1024) + 1024;
}

template <int ROWS>
static cudaError_t gemm_i8_rows(const LaunchCfg& lc, const GemvArgs& a, void* workspace, uint64_t workspace_bytes, bool counters_zeroed) {
    const bool dual = a.epilogue == EPI_SWIGLU;
    const uint32_t K = a.w.cols, out_dim = a.w.rows, n_rows = a.batch;
    if (gemm_i8_workspace_bytes(K) > workspace_bytes || ((uintptr_t)workspace & 1023) != 0) return cudaErrorInvalidValue;
    unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
    int8_t* planes = reinterpret_cast<int8_t*>(ws + I8_COUNTER_BYTES + I8_PART_BYTES);
    float* inv_scale = reinterpret_cast<float*>(ws + I8_COUNTER_BYTES + I8_PART_BYTES + (((uint64_t)64 * K + 1023) / 1024 * 1024));
    const cudaError_t e = launch_rows<ROWS>(lc, a, planes, inv_scale);
    if (e != cudaSuccess) return e;
    CUtensorMap mw, mw2, mx;
    if (!make_map_i8(&mw, a.w.data, out_dim, K, I8_BM) || !make_map_i8(&mx, planes, I8Shape<ROWS>::n, K, I8Shape<ROWS>::n)) return cudaErrorNotSupported;
    if (dual) { if (!make_map_i8(&mw2, a.w2.data, out_dim, K, I8_BM)) return cudaErrorNotSupported; } else mw2 = mw;
    I8Params p;
    p.dst = a.dst + a.dst_offset;
    p.row_scale = (const __half*)a.w.scales;
    p.row_scale2 = dual ? (const __half*)a.w2.scales : nullptr;
    p.x_inv_scale = inv_scale;
    p.state = a.state;
    p.out_dim = out_dim; p.n_rows = n_rows; p.K = K;
    p.dst_stride = a.dst_stride ? a.dst_stride : out_dim;
    p.epilogue = a.epilogue;
    error_words(lc, &p.err, &p.stop);
    p.counters = reinterpret_cast<uint32_t*>(ws);
    p.part = reinterpret_cast<float*>(ws + I8_COUNTER_BYTES);
    const uint32_t tiles = (out_dim + I8_BM - 1) / I8_BM, nk = (K + I8_BK - 1) / I8_BK;
    uint32_t splits = 1;
    if (!dual && counters_zeroed && gemm_tc_split_k && tiles * 2 <= 148) {
        splits = std::min(std::min(148u / tiles, 8u), std::max(nk / 8u, 1u));
        if ((uint64_t)splits * tiles * 128 * ROWS * 4 > I8_PART_BYTES || tiles * 4 > I8_COUNTER_BYTES) splits = 1;
    }
    // single products with more tiles than SMs (the lm_head: 1188): half the shared memory of an SM per block (4 stages),
    // two blocks per SM, so that one block's weights are on the way while the other is in its epilogue: 123 -> 94 us.
    // One-wave products measured ~1 us slower that way and keep the whole ring, as does gate/up (two weight tiles per stage).
    p.stages = (uint32_t)(192 * 1024 / I8Shape<ROWS>::stage(dual));
    if (!dual && gemm_i8_half_ring && tiles * splits > 148) p.stages = 4;
    p.trace = a.trace;
    const bool use_tiles = gemm_i8_tiles && a.w.i8_tiles && (!dual || a.w2.i8_tiles) && K % I8_BK == 0;
    p.w_tiles = use_tiles ? reinterpret_cast<const unsigned char*>(a.w.i8_tiles) : nullptr;
    p.w2_tiles = (use_tiles && dual) ? reinterpret_cast<const unsigned char*>(a.w2.i8_tiles) : p.w_tiles;
    const dim3 grid(1, tiles, splits);
    return dual ? launch_i8<true, ROWS>(lc, grid, mw, mw2, mx, p) : launch_i8<false, ROWS>(lc, grid, mw, mw2, mx, p);
}

cudaError_t gemm_i8(const LaunchCfg& lc, const GemvArgs& a, void* workspace, uint64_t workspace_bytes, bool counters_zeroed) {
    if (!gemm_i8_supported(a)) return cudaErrorInvalidValue;
    return a.batch <= 16 ? gemm_i8_rows<16>(lc, a, workspace, workspace_bytes, counters_zeroed) : gemm_i8_rows<32>(lc, a, workspace, workspace_bytes, counters_zeroed);
}

}  // namespace vb
