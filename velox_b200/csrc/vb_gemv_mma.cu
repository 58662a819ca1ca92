// Products of a few rows of x with int4, fp16 or bf16 weights on mma.sync: decode batches, speculative verify passes,
// short prompts, and batch 1 of the q4 group-64 format.
//
// Why mma.sync.  m16n8k16 issues every 8 clocks on each of an SM's four schedulers (measured; m16n8k32.s8 the same):
// 128 weights a clock and SM for eight columns, where HBM delivers 41 int4 weights (11 of 16 bits).  So up to three
// groups of eight columns cost no more time than the stream itself, without the detour through shared or tensor memory
// that tcgen05 operands take (dequantised hi + lo halves of int4 weights would be 164 bytes a clock of shared-memory
// writes, more than an SM has).  What has to be kept down is instructions: 16 x 128 weights (1152 bytes) arrive every 50
// clocks, 200 issue slots.
//
// Weights.  A = 16 weight rows x 16 of K.  int4 group-32: a masked nibble IS an fp16 operand, the subnormal n * 2^-24 (bits 0-3)
// or n * 2^-20 (bits 4-7, its x is stored divided by 16), exact: one AND per two weights and no conversion.  Groups keep their
// own accumulator: symmetric group-32 (n - 8) * s: the accumulator starts at -8 * sum(x), then acc += s * d; group-64
// n * s + m = (n - 8) * s + (m + 8 s): acc += s * d + (m + 8 s) * sum(x).  The tensor core aligns a subnormal operand's products
// by its exponent, not by its leading bit, and drops bits below: 1e-6 of a product's result, which the integer kernel's x (1.7e-5)
// does not notice, but group-64 weights, whose other kernels compute in fp32 (1.1e-7), do: their nibbles become n - 8 by one
// addition (1.1..1.9e-7; 5 % of a decode step of the 8B shape).  Block layout: the "v3" tiles of vb_gemv_imma.cu (a lane's 16 bytes are its words of
// four groups, so that one mma pair stays inside a group).  fp16 / bf16: rows g and g + 8 of the canonical matrix, 16 bytes
// a lane: the lane's 8 elements of K are its share of two mma (the order of K inside them is free as long as x follows it).
//
// Activations.  x becomes fp16 (bf16 for bf16 weights) parts whose sum carries x: two parts = 22 bits for group-32 weights,
// three = all 24 bits of fp32 for the others; each part a column of B (2 or 4 columns per row of x).  fp16 rows are scaled
// by a power of two to a maximum in [2^13, 2^14), so neither range nor subnormals cost accuracy.  One small kernel
// (k_x_frag, RMSNorm included) writes them in fragment order, 512 contiguous bytes per (32 of K, 8 columns), each weight
// block's share (with its sums) contiguous.  The products stream it through a ring of bulk copies in shared memory: read
// through L1 instead, every block of K waited a trip to L2 (gate/up of the 8B shape, 4 rows: 23 us).
//
// Sums.  The tensor core truncates what it accumulates: 16-bit products left in one accumulator along K were off by 3e-6 (K 4096) to
// 9e-6 (14336), all to the same side.  Every 64 of K start from zero and are added with a rounding: 1.3..1.8e-7 (fp32 kernel 1.0..1.4e-7),
// for 4 % of a step of 5 rows and more.
//
// Split.  A block is 4 warps on 4 row tiles (8 on 16 for 32 columns) over the same range of K, so that they share the
// fragments.  Matrices with few tiles split K over a cluster of up to 8 blocks; the partials meet in distributed shared memory
// and are added in rank order (the same bits every run).  A warp streams its tiles through a ring of its own, filled before the
// grid-dependency wait.
//
// Measured, 8B shape, a product with its k_x_frag in a graph: gate/up with 4 rows 22.9 us, with 8 rows 30.7, with 16 46.5
// (vb_gemv_imma.cu: 19.3 us for every 4 rows); down 15.8 / 21.4 / 42 (21.6 for every 4); fp16 gate/up with 4 rows 46.6 (235 MB:
// 5.0 TB/s; fp32 kernel 72).  A step of one group-64 row 2.09 ms (fp32 kernel: 3.9).  The steady state is bound by issue
// and latency (IPC 1.6 of 4, ~115 instructions a block and 8 columns): 5.0 TB/s of int4, 6.0 of fp16.
#include <cooperative_groups.h>

#include <algorithm>

#include "vb_internal.cuh"
#include "vb_kernels.cuh"
#include "vb_tma.cuh"

namespace cg = cooperative_groups;

namespace vb {
namespace {

constexpr int MM_Q4_BLK = 1152;  // 16 rows x 128 columns of nibbles + 128 bytes of scales

template <int FMT> struct Mm {
    static constexpr bool q4 = FMT == VB_FMT_Q4G32 || FMT == VB_FMT_Q4G64REF;
    static constexpr int parts = FMT == VB_FMT_Q4G32 ? 2 : 3, cols = FMT == VB_FMT_Q4G32 ? 2 : 4;  // columns a row of x takes
    static constexpr int rows = 8 / cols;          // rows of x per 8 columns
    static constexpr int kb = q4 ? 128 : 64;       // K of one weight block
    static constexpr int sx_k = FMT == VB_FMT_Q4G32 ? 32 : 64;  // K one sum covers
    static constexpr int frags = kb / 32;          // fragments of 512 bytes per weight block and 8 columns ...
    static constexpr int sums = q4 ? kb / sx_k : 0;  // ... then so many sums per column
    static constexpr int sum_bytes = FMT == VB_FMT_Q4G32 ? 64 : 32;  // of one sum over 8 columns (group-32: each pair twice, an accumulator)
    static constexpr int x_bytes = frags * 512 + sums * sum_bytes;  // of one weight block and 8 columns
};
constexpr int MM_SLOT_BLKS = 2;  // weight blocks per slot of the x ring
// T groups of 8 columns: row tiles per warp, warps of a block, blocks of an SM, slots of the x ring, blocks of a warp's weight ring
template <int FMT, int T> struct MmShape {
    static constexpr int mt = T == 4 ? 2 : 1, warps = T == 4 ? 8 : 4, per_sm = T == 4 ? 2 : T == 2 ? 4 : 5,
                         slots = T == 4 ? 2 : T == 2 ? 3 : 4, depth = T == 4 ? 3 : T == 2 ? 4 : 5;
    static constexpr int slot = MM_SLOT_BLKS * T * Mm<FMT>::x_bytes;
    static constexpr int w_blk = Mm<FMT>::q4 ? MM_Q4_BLK : 2048;
    static constexpr int smem = slots * slot + warps * depth * mt * w_blk + 128;
};

struct MmArgs {
    const unsigned char *w, *w2;  // q4: v3 blocks (gate and up interleaved for SwiGLU); else the matrix (w2: up)
    uint32_t rows, K;             // rows of dst
    uint32_t n_tiles;
    const unsigned char* xf;      // [weight blocks of K] x { [frags][T][32 lanes] uint4, q4: [sums][T][8] floats }
    uint32_t* err;
    const float* unscale;         // [rows of x]
    float* dst;
    const SeqState* state;
    uint32_t batch, dst_stride, dst_offset, splits;
    int epilogue;
    unsigned long long* trace;
};

template <int FMT>
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (FMT == VB_FMT_BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// d = a . b + c into registers of its own
__device__ __forceinline__ void mma16816_from(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const float4& c) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
}
__device__ __forceinline__ uint32_t word_of(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// the words of rows g and g + 8 as the A operands of two mma, subnormal (see the head of the file)
__device__ __forceinline__ void nibbles(uint32_t (&A)[8], uint32_t u, uint32_t v) {
    A[0] = u & 0x000F000Fu; A[1] = v & 0x000F000Fu; A[2] = u & 0x00F000F0u; A[3] = v & 0x00F000F0u;
    u >>= 8; v >>= 8;
    A[4] = u & 0x000F000Fu; A[5] = v & 0x000F000Fu; A[6] = u & 0x00F000F0u; A[7] = v & 0x00F000F0u;
}

__device__ __forceinline__ uint32_t hadd2_bits(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// the same as normal numbers: n - 8 (bits 0-3) and 16 * (n - 8) (bits 4-7)
__device__ __forceinline__ void nibbles_normal(uint32_t (&A)[8], uint32_t u, uint32_t v) {
    constexpr uint32_t LOW = 0xE408E408u, HIGH = 0xE480E480u;  // -1032, -1152
    A[0] = hadd2_bits(lop3_and_or(u, 0x000F000Fu, 0x64006400u), LOW); A[1] = hadd2_bits(lop3_and_or(v, 0x000F000Fu, 0x64006400u), LOW);
    A[2] = hadd2_bits(lop3_and_or(u, 0x00F000F0u, 0x64006400u), HIGH); A[3] = hadd2_bits(lop3_and_or(v, 0x00F000F0u, 0x64006400u), HIGH);
    u >>= 8; v >>= 8;
    A[4] = hadd2_bits(lop3_and_or(u, 0x000F000Fu, 0x64006400u), LOW); A[5] = hadd2_bits(lop3_and_or(v, 0x000F000Fu, 0x64006400u), LOW);
    A[6] = hadd2_bits(lop3_and_or(u, 0x00F000F0u, 0x64006400u), HIGH); A[7] = hadd2_bits(lop3_and_or(v, 0x00F000F0u, 0x64006400u), HIGH);
}

// Bounded wait (vb_tma.cuh); one that runs out is reported and the block carries on with what is there.
__device__ __forceinline__ void mm_wait(uint32_t bar, uint32_t parity, uint32_t* err) {
    if (mbar_try_wait(bar, parity)) return;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > 2000000000LL) { atomicOr(err, 0x80u); return; }
}

__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}

// grid: (tile groups * splits) blocks, clusters of `splits`; T groups of 8 columns, MT row tiles per warp
template <int FMT, int T>
__global__ void __launch_bounds__(MmShape<FMT, T>::warps * 32, MmShape<FMT, T>::per_sm) k_gemv_mma(const MmArgs a) {
    typedef Mm<FMT> F;
    typedef MmShape<FMT, T> P;
    constexpr int MT = P::mt, D = P::depth, MM_WARPS = P::warps, MM_SLOTS = P::slots, SLOT = P::slot, BLK_X = T * F::x_bytes, WB = P::w_blk;
    constexpr int NV = MT * T * (F::cols == 2 ? 2 : 1);      // sums a lane ends up with
    extern __shared__ __align__(128) unsigned char smem[];   // the ring of x, every warp's ring of weights, barriers
    __shared__ float recv[8 * NV * 32];
    const uint32_t ring = smem_u32(smem), full = ring + P::smem - 128, empty = full + 8 * MM_SLOTS;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < MM_SLOTS; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, MM_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t S = a.splits, rank = blockIdx.x % S, group = blockIdx.x / S;
    trace_mark(a.trace, 0);
    pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    if (S > 1) cluster.barrier_arrive();  // every block of the cluster runs before anyone writes into its shared memory

    const uint32_t KT = a.K / F::kb, kb0 = KT * rank / S, n_kb = KT * (rank + 1) / S - kb0;
    const uint32_t tile0 = (group * MM_WARPS + warp) * MT;
    const bool any = tile0 < a.n_tiles;
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    // weights of this lane: int4: the tile's blocks; else rows g and g + 8 of each tile (SwiGLU: the same row of gate and up)
    const unsigned char *pa[MT], *pb[F::q4 ? 1 : MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const uint32_t tile = min(tile0 + m, a.n_tiles - 1);
        if constexpr (F::q4) {
            pa[m] = a.w + ((size_t)tile * KT + kb0) * MM_Q4_BLK + 16 * lane;
        } else {
            const uint32_t r0 = min(swiglu ? tile * 8 + g : tile * 16 + g, a.rows - 1), r1 = min(swiglu ? r0 : tile * 16 + 8 + g, a.rows - 1);
            pa[m] = a.w + ((size_t)r0 * a.K + kb0 * F::kb + 8 * t) * 2;
            pb[m] = (swiglu ? a.w2 : a.w) + ((size_t)r1 * a.K + kb0 * F::kb + 8 * t) * 2;
        }
    }
    // This warp's ring: D blocks of every tile.  16-byte asynchronous copies: with the blocks held in registers instead, the
    // loads in flight waited for each other (four deep no faster than two, 4.4 TB/s of fp16 weights).
    const unsigned char* wring = smem + MM_SLOTS * SLOT + warp * (D * MT * WB);
    const uint32_t wring_s = smem_u32(wring);
    uint32_t w_in = 0;  // byte offset of the slot the next block goes to
    auto request = [&](bool there) {
        if (there) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const uint32_t dst = wring_s + w_in + m * WB + 16 * lane;
                if constexpr (F::q4) {
                    cp_async16(dst, pa[m]);
                    cp_async16(dst + 512, pa[m] + 512);
                    if (lane < 8) cp_async16(dst + 1024, pa[m] + 1024);
                    pa[m] += MM_Q4_BLK;
                } else {
                    cp_async16(dst, pa[m]); cp_async16(dst + 512, pb[m]);
                    cp_async16(dst + 1024, pa[m] + 64); cp_async16(dst + 1536, pb[m] + 64);
                    pa[m] += 128; pb[m] += 128;
                }
            }
            w_in = w_in == (D - 1) * MT * WB ? 0 : w_in + MT * WB;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int d = 0; d < D - 1; ++d) request(any && (uint32_t)d < n_kb);

    pdl_wait();
    trace_mark(a.trace, 1);
    float acc[MT][T][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < T; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.0f;
    // x: thread 0 keeps the ring full; every warp waits for a slot once per MM_SLOT_BLKS blocks and gives it back
    const unsigned char* xsrc = a.xf + (size_t)kb0 * BLK_X;
    const uint32_t n_slots = (n_kb + MM_SLOT_BLKS - 1) / MM_SLOT_BLKS;
    auto fill = [&](uint32_t i) {
        const uint32_t bytes = min((uint32_t)MM_SLOT_BLKS, n_kb - i * MM_SLOT_BLKS) * BLK_X, bar = full + 8 * (i % MM_SLOTS);
        mbar_expect_tx(bar, bytes);
        tma_load_1d(ring + (i % MM_SLOTS) * SLOT, xsrc + (size_t)i * SLOT, bytes, bar);
    };
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < min((uint32_t)MM_SLOTS, n_slots); ++i) fill(i);
    uint32_t at = 0, phase = 0;  // slot of the ring of x, how often it came round
    uint32_t w_out = 0;          // slot of the weight ring
#pragma unroll 1
    for (uint32_t blk = 0; blk < n_kb; blk += MM_SLOT_BLKS) {
        // thread 0 refills the slot before this one once every warp has left it
        const uint32_t gone = phase * MM_SLOTS + at;  // slots finished so far
        if (threadIdx.x == 0 && gone > 0 && gone - 1 + MM_SLOTS < n_slots) {
            mm_wait(empty + 8 * ((gone - 1) % MM_SLOTS), ((gone - 1) / MM_SLOTS) & 1u, a.err);
            fill(gone - 1 + MM_SLOTS);
        }
        __syncwarp();
        mm_wait(full + 8 * at, phase & 1u, a.err);
#pragma unroll
        for (int q = 0; q < MM_SLOT_BLKS; ++q) {
            if (blk + q < n_kb) {
                request(any && blk + q + D - 1 < n_kb);
                asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
                __syncwarp();
                const unsigned char* xb = smem + at * SLOT + q * BLK_X;
                const uint4* xp = reinterpret_cast<const uint4*>(xb) + lane;
                const unsigned char* sp = xb + F::frags * T * 512 + (FMT == VB_FMT_Q4G32 ? 16 : 8) * t;
                const uint4* wp = reinterpret_cast<const uint4*>(wring + w_out);
                w_out = w_out == (D - 1) * MT * WB ? 0 : w_out + MT * WB;
                uint4 w0[MT], w1[MT], w2[F::q4 ? MT : 1], w[F::q4 ? 1 : MT][4];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    if constexpr (F::q4) {
                        w0[m] = wp[m * (WB / 16) + lane]; w1[m] = wp[m * (WB / 16) + 32 + lane]; w2[m] = wp[m * (WB / 16) + 64 + g];
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) w[m][i] = wp[m * (WB / 16) + i * 32 + lane];
                    }
                }
                if constexpr (FMT == VB_FMT_Q4G32) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t A[MT][8];
                        float2 s[MT];
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            nibbles(A[m], word_of(w0[m], j), word_of(w1[m], j));
                            const uint32_t sc = word_of(w2[m], j);
                            s[m] = __half22float2(*reinterpret_cast<const __half2*>(&sc));
                        }
#pragma unroll
                        for (int n = 0; n < T; ++n) {
                            const uint4 bx = xp[(j * T + n) * 32];
                            const float4 c = *reinterpret_cast<const float4*>(sp + (j * T + n) * 64);
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                float e[4];
                                mma16816_from(e, A[m][0], A[m][1], A[m][2], A[m][3], bx.x, bx.y, c);
                                mma16816<FMT>(e, A[m][4], A[m][5], A[m][6], A[m][7], bx.z, bx.w);
                                acc[m][n][0] = fmaf(e[0], s[m].x, acc[m][n][0]); acc[m][n][1] = fmaf(e[1], s[m].x, acc[m][n][1]);
                                acc[m][n][2] = fmaf(e[2], s[m].y, acc[m][n][2]); acc[m][n][3] = fmaf(e[3], s[m].y, acc[m][n][3]);
                            }
                        }
                    }
                } else if constexpr (FMT == VB_FMT_Q4G64REF) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t A[MT][2][8];
                        float2 s0[MT], s1[MT];  // (scale, minimum) of rows g and g + 8
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) nibbles_normal(A[m][i], word_of(w0[m], 2 * h + i), word_of(w1[m], 2 * h + i));
                            const uint32_t z0 = word_of(w2[m], h), z1 = word_of(w2[m], 2 + h);
                            s0[m] = __half22float2(*reinterpret_cast<const __half2*>(&z0));
                            s1[m] = __half22float2(*reinterpret_cast<const __half2*>(&z1));
                            s0[m].y = fmaf(8.0f, s0[m].x, s0[m].y); s1[m].y = fmaf(8.0f, s1[m].x, s1[m].y);  // n * s + m = (n - 8) * s + (m + 8 * s)
                        }
#pragma unroll
                        for (int n = 0; n < T; ++n) {
                            const uint4 b0 = xp[(2 * h * T + n) * 32], b1 = xp[((2 * h + 1) * T + n) * 32];
                            const float2 c = *reinterpret_cast<const float2*>(sp + (h * T + n) * 32);
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                float e[4];
                                mma16816_from(e, A[m][0][0], A[m][0][1], A[m][0][2], A[m][0][3], b0.x, b0.y, make_float4(0.f, 0.f, 0.f, 0.f));
                                mma16816<FMT>(e, A[m][0][4], A[m][0][5], A[m][0][6], A[m][0][7], b0.z, b0.w);
                                mma16816<FMT>(e, A[m][1][0], A[m][1][1], A[m][1][2], A[m][1][3], b1.x, b1.y);
                                mma16816<FMT>(e, A[m][1][4], A[m][1][5], A[m][1][6], A[m][1][7], b1.z, b1.w);
                                acc[m][n][0] = fmaf(e[0], s0[m].x, fmaf(c.x, s0[m].y, acc[m][n][0])); acc[m][n][1] = fmaf(e[1], s0[m].x, fmaf(c.y, s0[m].y, acc[m][n][1]));
                                acc[m][n][2] = fmaf(e[2], s1[m].x, fmaf(c.x, s1[m].y, acc[m][n][2])); acc[m][n][3] = fmaf(e[3], s1[m].x, fmaf(c.y, s1[m].y, acc[m][n][3]));
                            }
                        }
                    }
                } else {
#pragma unroll
                    for (int n = 0; n < T; ++n) {
                        const uint4 b0 = xp[n * 32], b1 = xp[(T + n) * 32];
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            const uint4 &u0 = w[m][0], &v0 = w[m][1], &u1 = w[m][2], &v1 = w[m][3];
                            float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                            mma16816<FMT>(e, u0.x, v0.x, u0.y, v0.y, b0.x, b0.y);
                            mma16816<FMT>(e, u0.z, v0.z, u0.w, v0.w, b0.z, b0.w);
                            mma16816<FMT>(e, u1.x, v1.x, u1.y, v1.y, b1.x, b1.y);
                            mma16816<FMT>(e, u1.z, v1.z, u1.w, v1.w, b1.z, b1.w);
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[m][n][i] += e[i];
                        }
                    }
                }
                __syncwarp();  // before the next block's request overwrites what other lanes may still read
            }
        }
        if (lane == 0) mbar_arrive(empty + 8 * at);
        if (++at == MM_SLOTS) { at = 0; ++phase; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    // parts of a row of x -> one sum.  Two columns: lane (g,t) has row 4n + t of x for weight rows g and g + 8.  Four: its
    // even lane gets row 2n + t/2 for weight row g, the odd one for g + 8 (the fourth column is never written: left out)
    float y[NV];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < T; ++n) {
            const float* e = acc[m][n];
            if constexpr (F::cols == 2) {
                y[(m * T + n) * 2] = e[0] + e[1];
                y[(m * T + n) * 2 + 1] = e[2] + e[3];
            } else {
                const bool odd = t & 1;
                const float own0 = odd ? e[0] : e[0] + e[1], own1 = odd ? e[2] : e[2] + e[3];
                const float got = __shfl_xor_sync(0xFFFFFFFFu, odd ? own0 : own1, 1);
                y[m * T + n] = (odd ? own1 : own0) + got;
            }
        }
    bool final_here = true;
    if (S > 1) {
        // warp w's tiles are finished by block w % S of the cluster
        const uint32_t slot = warp / S, owner = warp % S, per = (MM_WARPS + S - 1) / S;
        cluster.barrier_wait();
        float* dst = cluster.map_shared_rank(recv, owner) + (size_t)((rank * per + slot) * NV) * 32 + lane;
#pragma unroll
        for (int i = 0; i < NV; ++i) dst[i * 32] = y[i];
        cluster.sync();
        final_here = owner == rank;
        if (final_here) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                float s = 0.0f;
                for (uint32_t r = 0; r < S; ++r) s += recv[((r * per + slot) * NV + i) * 32 + lane];
                y[i] = s;
            }
        }
    }
    if (final_here) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const uint32_t tile = tile0 + m;
#pragma unroll
            for (int n = 0; n < T; ++n) {
                const uint32_t b = F::cols == 2 ? n * 4 + t : n * 2 + (t >> 1);  // row of x
                const bool live = tile < a.n_tiles && b < a.batch && (!a.state || a.state[b].active);
                const float un = live ? a.unscale[b] : 0.0f;
                float* d = a.dst + (size_t)b * a.dst_stride + a.dst_offset;
                float v0, v1;  // weight rows g and g + 8
                bool has0 = live, has1 = live;
                if constexpr (F::cols == 2) {
                    v0 = y[(m * T + n) * 2]; v1 = y[(m * T + n) * 2 + 1];
                } else {
                    v0 = v1 = y[m * T + n];
                    if (swiglu) {
                        const float other = __shfl_xor_sync(0xFFFFFFFFu, v0, 1);
                        if (t & 1) v0 = other; else v1 = other;
                        has0 = live && !(t & 1);
                    } else {
                        has0 = live && !(t & 1); has1 = live && (t & 1);
                    }
                }
                v0 *= un; v1 *= un;
                if (swiglu) {
                    const uint32_t o = tile * 8 + g;
                    if (has0 && o < a.rows) d[o] = (v0 / (1.0f + expf(-v0))) * v1;
                } else {
                    const uint32_t o = tile * 16 + g;
                    if (has0 && o < a.rows) d[o] = a.epilogue == EPI_RESIDUAL ? d[o] + v0 : v0;
                    if (has1 && o + 8 < a.rows) d[o + 8] = a.epilogue == EPI_RESIDUAL ? d[o + 8] + v1 : v1;
                }
            }
        }
    }
    trace_exit(a.trace);
}

// ---- x -> parts in fragment order ---------------------------------------------------------------------------------
struct XfArgs {
    const float* x;
    unsigned char* xf; float* unscale;
    const void* norm_w; int norm_fmt; float eps;
    const SeqState* state;
    uint32_t K, T;
};
__device__ __forceinline__ float4 norm4(const void* w, int fmt, uint32_t i4) {
    if (fmt == VB_FMT_F32) return __ldg(reinterpret_cast<const float4*>(w) + i4);
    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(w) + i4);
    if (fmt == VB_FMT_F16) {
        const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), q = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        return make_float4(p.x, p.y, q.x, q.y);
    }
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xFFFF0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xFFFF0000u));
}

constexpr int XF_THREADS = 512;
// grid (K / 4096 rounded up, rows of x): every block reads the whole row for its norm and scale (from L2) and converts its
// own 4096 elements, one lane's share of 32 of K per thread.  Latency is all there is to it: the norm weights are fetched
// before the dependency wait, the row's loads are issued together.
template <int FMT>
__global__ void __launch_bounds__(XF_THREADS) k_x_frag(const XfArgs a) {
    typedef Mm<FMT> F;
    constexpr bool SCALED = FMT != VB_FMT_BF16;
    constexpr int U = 4;  // float4s a thread loads at once: rows of up to 8192 in one trip
    __shared__ float red_s[XF_THREADS / 32], red_m[XF_THREADS / 32];
    const uint32_t b = blockIdx.y, K = a.K, K4 = K / 4;
    const float* x = a.x + (size_t)b * K;
    pdl_launch_dependents();
    // q4: elements 4t, 4t+2 | 16+4t, 18+4t | 4t+1, 4t+3 | 17+4t, 19+4t (the nibbles' places in a v3 word), else 8t .. 8t+7
    const uint32_t unit = blockIdx.x * XF_THREADS + threadIdx.x, k32 = unit >> 2, t = unit & 3;  // lane t's share of K [32 k32, +32)
    const bool in = k32 * 32 < K;
    const uint32_t e0 = k32 * 32 + (F::q4 ? 4 * t : 8 * t), e1 = e0 + (F::q4 ? 16 : 4);
    float4 wr[U], wp, wq;
    if (a.norm_w) {
#pragma unroll
        for (int i = 0; i < U; ++i)
            if (threadIdx.x + i * XF_THREADS < K4) wr[i] = norm4(a.norm_w, a.norm_fmt, threadIdx.x + i * XF_THREADS);
        if (in) { wp = norm4(a.norm_w, a.norm_fmt, e0 / 4); wq = norm4(a.norm_w, a.norm_fmt, e1 / 4); }
    }
    pdl_wait();
    const bool active = !a.state || a.state[b].active;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
    if (in) { p = *reinterpret_cast<const float4*>(x + e0); q = *reinterpret_cast<const float4*>(x + e1); }
    float inv = 1.0f, up = 1.0f;
    if (a.norm_w || SCALED) {
        float ss = 0.0f, mx = 0.0f;
        for (uint32_t i0 = threadIdx.x; i0 < K4; i0 += U * XF_THREADS) {
            float4 v[U];
#pragma unroll
            for (int i = 0; i < U; ++i) v[i] = i0 + i * XF_THREADS < K4 ? reinterpret_cast<const float4*>(x)[i0 + i * XF_THREADS] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < U; ++i) {
                if (a.norm_w && i0 + i * XF_THREADS < K4) {
                    ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
                    const float4 w = i0 == threadIdx.x ? wr[i] : norm4(a.norm_w, a.norm_fmt, i0 + i * XF_THREADS);
                    v[i] = make_float4(v[i].x * w.x, v[i].y * w.y, v[i].z * w.z, v[i].w * w.w);
                }
                mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
            }
        }
        ss = warp_sum(ss); mx = warp_max(mx);
        if ((threadIdx.x & 31) == 0) { red_s[threadIdx.x >> 5] = ss; red_m[threadIdx.x >> 5] = mx; }
        __syncthreads();
        ss = 0.0f; mx = 0.0f;
#pragma unroll
        for (int i = 0; i < XF_THREADS / 32; ++i) { ss += red_s[i]; mx = fmaxf(mx, red_m[i]); }
        if (a.norm_w) { inv = 1.0f / sqrtf(ss / (float)K + a.eps); mx *= inv; }
        if (SCALED && mx > 0.0f && mx < 3.0e38f) {
            // 2^(13 - floor(log2 max)), kept inside the exponents of a float
            const int e = min(max((int)((__float_as_uint(mx) >> 23) & 255u) - 127, -100), 127);
            up = __uint_as_float((uint32_t)(127 + 13 - e) << 23);
        }
    }
    if (!active) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.unscale[b] = (FMT == VB_FMT_Q4G32 ? 16777216.0f : 1.0f) / up;
    if (a.norm_w && in) {
        p.x = (p.x * inv) * wp.x; p.y = (p.y * inv) * wp.y; p.z = (p.z * inv) * wp.z; p.w = (p.w * inv) * wp.w;
        q.x = (q.x * inv) * wq.x; q.y = (q.y * inv) * wq.y; q.z = (q.z * inv) * wq.z; q.w = (q.w * inv) * wq.w;
    }
    float v[8];
    if constexpr (F::q4) { v[0] = p.x; v[1] = p.z; v[2] = q.x; v[3] = q.z; v[4] = p.y; v[5] = p.w; v[6] = q.y; v[7] = q.w; }
    else { v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w; }
    const uint32_t n = b / F::rows, col0 = (b % F::rows) * F::cols;
    unsigned char* blk = a.xf + (size_t)(k32 / F::frags) * a.T * F::x_bytes;  // the weight block's share
    uint4* frag = reinterpret_cast<uint4*>(blk) + ((k32 % F::frags) * a.T + n) * 32;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= up;
#pragma unroll
    for (int part = 0; part < F::parts; ++part) {
        uint32_t h[4];
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f0 = v[2 * i], f1 = v[2 * i + 1];
            float r0, r1;
            if constexpr (FMT == VB_FMT_BF16) {
                const __nv_bfloat162 c = __floats2bfloat162_rn(f0, f1);
                r0 = __low2float(c); r1 = __high2float(c);
                h[i] = *reinterpret_cast<const uint32_t*>(&c);
            } else {
                __half2 c = __floats2half2_rn(f0, f1);
                r0 = __low2float(c); r1 = __high2float(c);
                if (F::q4 && (i & 1)) c = __hmul2(c, __float2half2_rn(0.0625f));  // meets n * 2^-20
                h[i] = *reinterpret_cast<const uint32_t*>(&c);
            }
            v[2 * i] = f0 - r0; v[2 * i + 1] = f1 - r1;  // what is left for the next part, exact
            sum += r0 + r1;
        }
        if (in) frag[(col0 + part) * 4 + t] = make_uint4(h[0], h[1], h[2], h[3]);
        if constexpr (F::q4) {
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
            if (F::sx_k == 64) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 4);
            if (in && unit % (F::sx_k / 8) == 0) {
                unsigned char* sums = blk + F::frags * a.T * 512 + ((k32 % F::frags) / (F::sx_k / 32) * a.T + n) * F::sum_bytes;
                const uint32_t c = col0 + part;
                if constexpr (FMT == VB_FMT_Q4G32) {  // lane t's accumulator start: columns 2t, 2t+1 for its two weight rows
                    float* f = reinterpret_cast<float*>(sums) + (c >> 1) * 4 + (c & 1);
                    f[0] = f[2] = sum * (-8.0f / 16777216.0f);
                } else {
                    reinterpret_cast<float*>(sums)[c] = sum;
                }
            }
        }
    }
}

template <int FMT, int T>
cudaError_t launch_mma(const LaunchCfg& lc, MmArgs a) {
    typedef MmShape<FMT, T> P;
    const uint32_t groups = (a.n_tiles + P::warps * P::mt - 1) / (P::warps * P::mt), KT = a.K / Mm<FMT>::kb;
    // Few tiles: split K over a cluster while all its blocks find a place at once and every warp keeps four weight blocks (a
    // cluster that has to wait starts a wave of its own: QKV of the 8B shape in 8 parts 11.5 us, in 4 parts 10.6).  Pairs may
    // go a quarter beyond: they slip in as soon as two blocks leave (its gate/up: 26.3 us whole, 22.9 in pairs).
    const uint32_t places = 148 * P::per_sm;
    a.splits = 1;
    while (a.splits < 8 && KT >= 8 * a.splits && groups * a.splits * 2 <= (a.splits == 1 ? places * 5 / 4 : places)) a.splits *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups * a.splits);
    cfg.blockDim = dim3(P::warps * 32);
    cfg.dynamicSmemBytes = P::smem;
    cfg.stream = lc.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    if (lc.pdl) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    cfg.attrs = attr;
    static std::atomic<uint64_t> opted{0};
    const cudaError_t oe = once_per_device(opted, [&]() { return cudaFuncSetAttribute(k_gemv_mma<FMT, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::smem); });
    if (oe != cudaSuccess) return oe;
    if (lc.counter) ++*lc.counter;
    return cudaLaunchKernelEx(&cfg, k_gemv_mma<FMT, T>, a);
}

// one pass: the rows of x that fit T groups of 8 columns
template <int FMT>
cudaError_t pass_mma(const LaunchCfg& lc, MmArgs a, XfArgs f, unsigned char* ws) {
    const uint32_t tiles = (a.batch + Mm<FMT>::rows - 1) / Mm<FMT>::rows, T = tiles <= 2 ? tiles : 4;
    f.T = T;
    f.xf = ws;
    f.unscale = reinterpret_cast<float*>(ws + (size_t)(f.K / Mm<FMT>::kb) * T * Mm<FMT>::x_bytes);
    a.xf = f.xf; a.unscale = f.unscale;
    cudaError_t e = launch(lc, k_x_frag<FMT>, dim3((f.K + 4095) / 4096, a.batch), dim3(XF_THREADS), 0, f);
    if (e != cudaSuccess) return e;
    if (T == 1) return launch_mma<FMT, 1>(lc, a);
    if (T == 2) return launch_mma<FMT, 2>(lc, a);
    return launch_mma<FMT, 4>(lc, a);
}

}  // namespace

// fragments of 4 groups of 8 columns and their sums (18 bytes per element of K and group), the rows' scales
uint64_t gemv_mma_workspace_bytes(uint32_t max_in_dim) { return (uint64_t)max_in_dim * 4 * (16 + 2) + 4096; }

cudaError_t gemv_mma(const LaunchCfg& lc, const GemvArgs& g, bool* handled) {
    *handled = false;
    const bool swiglu = g.epilogue == EPI_SWIGLU, q4 = g.w.fmt == VB_FMT_Q4G32 || g.w.fmt == VB_FMT_Q4G64REF;
    const uint32_t K = g.w.cols;
    if (!g.frag_ws || gemv_mma_workspace_bytes(K) > g.frag_ws_bytes || g.push.links) return cudaSuccess;
    const uint64_t weights = (uint64_t)g.w.rows * K * (swiglu ? 2 : 1);
    if (g.w.fmt == VB_FMT_Q4G32) {
        // One row: the integer kernel stages x itself and needs one launch.  2..4 rows are one pass of its multi-row flavour too,
        // faster (8B shape: O 6.2 against 8.2 us, gate/up 17.5 / 22.9, head 55 / 64) unless four rows of x are long to stage
        // (down: 19.7 / 15.8) or the tiles of a large matrix fill the last of several rounds of SMs badly (QKV: 384 tiles on 296
        // places, 14.7 / 10.4).  Below 8M weights, or in a single round, its one launch is ahead however the tiles fall (models of
        // 1024 / 1536 / 2048 columns, a step of 2 rows: 387 / 391 / 297 us, by the fill alone 509 / 426 / 334).
        if (g.batch < 2) return cudaSuccess;
        const uint32_t tiles = (swiglu ? 2 : 1) * g.w.rows / 16, places = 2 * 148, rounds = (tiles + places - 1) / places;
        if (g.batch <= 4 && K <= 8192 && (rounds == 1 || weights < 8000000ull || tiles * 4 >= rounds * places * 3)) return cudaSuccess;
    } else {
        // The fp32 kernel needs one launch and no conversion, and takes small matrices in one wave: ahead there, and with one or two
        // rows of 16-bit weights (it streams those at 5..6 TB/s).  Where the line lies (decode steps of models of 768 to 2048
        // columns, products from the named size on taken here, us; 16-bit / group-64):
        //   3 rows: 1024 columns from 1M weights 521 / 589, 4M 415 / 420, 10M 457 / 451; 2048 columns 4M 553 / 529, 10M 592 / 560
        //   8 rows, one pass of 16-bit: 1024 columns 839 / 1142, 592 / 692, 664 / 680; 2048 columns 884 / 1007, 923 / 960
        //   32 rows: 1024 columns 3062 / 4353, 1760 / 2092, 1814 / 1946; 1536 columns 2165 / 2650 from 4M, 1957 / 2411 from 10M
        if (!q4 && g.batch < 3) return cudaSuccess;
        const uint32_t one_pass = q4 ? 4 : 8;
        if (weights < (g.batch > 1 && g.batch <= one_pass ? 4000000ull : 8000000ull)) return cudaSuccess;
    }
    MmArgs a;
    if (q4) {
        a.w = (const unsigned char*)(swiglu ? g.w.v3_swiglu : g.w.v3);
        if (!a.w || K % 128 != 0) return cudaSuccess;
        a.n_tiles = swiglu ? g.w.rows / 8 : g.w.rows / 16;
    } else if (g.w.fmt == VB_FMT_F16 || g.w.fmt == VB_FMT_BF16) {
        a.w = (const unsigned char*)g.w.data; a.w2 = (const unsigned char*)g.w2.data;
        if (!a.w || K % 64 != 0) return cudaSuccess;
        a.n_tiles = swiglu ? (g.w.rows + 7) / 8 : (g.w.rows + 15) / 16;
    } else {
        return cudaSuccess;
    }
    a.err = nullptr;
    fast_error_word(&a.err);
    a.rows = g.w.rows; a.K = K; a.epilogue = g.epilogue; a.trace = g.trace;
    a.dst_stride = g.dst_stride ? g.dst_stride : g.w.rows; a.dst_offset = g.dst_offset;
    XfArgs f;
    f.norm_w = g.norm_w; f.norm_fmt = g.norm_fmt; f.eps = g.eps; f.K = K;
    *handled = true;
    const uint32_t per = 4 * (g.w.fmt == VB_FMT_Q4G32 ? 4 : 2);
    for (uint32_t b0 = 0; b0 < g.batch; b0 += per) {
        a.batch = std::min(per, g.batch - b0);
        a.dst = g.dst + (size_t)b0 * a.dst_stride;
        a.state = f.state = g.state ? g.state + b0 : nullptr;
        f.x = g.x + (size_t)b0 * K;
        unsigned char* ws = (unsigned char*)g.frag_ws;
        const cudaError_t e = g.w.fmt == VB_FMT_Q4G32 ? pass_mma<VB_FMT_Q4G32>(lc, a, f, ws)
                            : g.w.fmt == VB_FMT_Q4G64REF ? pass_mma<VB_FMT_Q4G64REF>(lc, a, f, ws)
                            : g.w.fmt == VB_FMT_F16 ? pass_mma<VB_FMT_F16>(lc, a, f, ws) : pass_mma<VB_FMT_BF16>(lc, a, f, ws);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace vb
