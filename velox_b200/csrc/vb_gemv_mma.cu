// Products of a few rows of x with int4, fp16 or bf16 weights on mma.sync: decode batches, speculative verify passes,
// short prompts, and batch 1 of the q4 group-64 format.
//
// Why mma.sync.  m16n8k16 issues every 8 clocks on each of an SM's four schedulers (measured; m16n8k32.s8 the same):
// 128 weights a clock and SM for eight columns, where HBM delivers 41 int4 weights (11 of 16 bits).  So the
// products of up to three groups of eight columns take no longer than the stream, without the detour through shared or tensor memory
// that tcgen05 operands take (dequantised hi + lo halves of int4 weights would be 164 bytes a clock of shared-memory
// writes, more than an SM has).  What they cost is instructions and fragment reads (a step of 4 rows, one group: 1.82 ms, of 5, two
// groups: 2.45): 16 x 128 weights (1152 bytes) arrive every 50 clocks, 200 issue slots.
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
// block's share (with its sums) contiguous; bulk copies bring it to shared memory: read through L1 instead, every block of K waited
// a trip to L2 (gate/up of the 8B shape, 4 rows: 23 us).
//
// Sums.  The tensor core truncates what it accumulates: 16-bit products left in one accumulator along K were off by 3e-6 (K 4096) to
// 9e-6 (14336), all to the same side.  Every 64 of K start from zero and are added with a rounding: 1.3..1.8e-7 (fp32 kernel 1.0..1.4e-7),
// for 4 % of a step of 5 rows and more.
//
// Split, 16-bit weights.  A block is 4 warps on 4 row tiles (8 on 16 for 32 columns) over the same range of K, so that they share the
// fragments, which go round a ring.  Matrices with few tiles split K over a cluster of up to 8 blocks; the partials meet in distributed
// shared memory and are added in rank order (the same bits every run).  A warp streams its tiles through a ring of its own, filled before
// the grid-dependency wait.
//
// Split, int4 weights.  There the fragments are as many bytes as the weights (8 columns: 1152 of 1152 a block), so every ring of them
// doubled what the blocks moved, and its barriers what they waited.  One block per SM keeps x for good and takes tile after tile; the
// warps split K, not the tiles, so that all of a matrix's tiles come out even to a sixteenth of a tile's time.  Two weight blocks a
// step: one wait, one set of addresses, one loop for both.
//
// Measured, a step of the 8B shape, ms (as above with int4 weights too, 2..4 int4 rows on vb_gemv_imma.cu -> now): int4, 2 / 3 / 4 / 5 / 8 rows
// 2.16 / 2.24 / 2.06 / 2.74 / 2.79 -> 1.73 / 1.80 / 1.82 / 2.45 / 2.46; group-64, 1 / 2 / 4 / 8 rows 2.09 / 2.26 / 2.52 / 4.55 -> 1.64 / 1.73 / 2.24 /
// 4.24 (0.1..0.2 of it at 2 and 3 rows is the attention's).  fp16 gate/up with 4 rows 46.6 us (235 MB: 5.0 TB/s; fp32 kernel 72).
// What bounds the int4 products is issue and latency: ~115 instructions a weight block and 8 columns, IPC 1.9 of 4 in gate/up.
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
// 16-bit weights, T groups of 8 columns: row tiles per warp, warps of a block, blocks of an SM, slots of the x ring, blocks of a warp's
// weight ring
template <int FMT, int T> struct MmShape {
    static constexpr int mt = T == 4 ? 2 : 1, warps = T == 4 ? 8 : 4, per_sm = T == 4 ? 2 : T == 2 ? 4 : 5,
                         slots = T == 4 ? 2 : T == 2 ? 3 : 4, depth = T == 4 ? 3 : T == 2 ? 4 : 5;
    static constexpr int slot = MM_SLOT_BLKS * T * Mm<FMT>::x_bytes;
    static constexpr int w_blk = 2048;
    static constexpr int smem = slots * slot + warps * depth * mt * w_blk + 128;
};

struct MmArgs {
    const unsigned char *w, *w2;  // q4: v3 blocks (gate and up interleaved for SwiGLU); else the matrix (w2: up)
    uint32_t rows, K;             // rows of dst
    uint32_t n_tiles;
    const float* x;               // rows of x and the norm's weights, where a product converts them itself
    const void* norm_w; int norm_fmt; float eps;
    const unsigned char* xf;      // [weight blocks of K] x { [frags][T][32 lanes] uint4, q4: [sums][T][8] floats }
    uint32_t *err, *stop;
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
__device__ __forceinline__ void mm_wait(uint32_t bar, uint32_t parity, uint32_t* err, uint32_t* stop) {
    if (!wait_or_stop(bar, parity, stop)) report_wait(err, stop, 0x200u);
}

__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}

// One block of 128 of K of a tile: acc[n] += its products with T groups of 8 columns (w0, w1: the words of rows g and g + 8; w2: scales)
template <int FMT, int T>
__device__ __forceinline__ void q4_block(float (&acc)[T][4], const uint4& w0, const uint4& w1, const uint4& w2, const uint4* xp, const unsigned char* sp) {
    if constexpr (FMT == VB_FMT_Q4G32) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t A[8];
            nibbles(A, word_of(w0, j), word_of(w1, j));
            const uint32_t sc = word_of(w2, j);
            const float2 s = __half22float2(*reinterpret_cast<const __half2*>(&sc));
#pragma unroll
            for (int n = 0; n < T; ++n) {
                const uint4 bx = xp[(j * T + n) * 32];
                const float4 c = *reinterpret_cast<const float4*>(sp + (j * T + n) * 64);
                float e[4];
                mma16816_from(e, A[0], A[1], A[2], A[3], bx.x, bx.y, c);
                mma16816<FMT>(e, A[4], A[5], A[6], A[7], bx.z, bx.w);
                acc[n][0] = fmaf(e[0], s.x, acc[n][0]); acc[n][1] = fmaf(e[1], s.x, acc[n][1]);
                acc[n][2] = fmaf(e[2], s.y, acc[n][2]); acc[n][3] = fmaf(e[3], s.y, acc[n][3]);
            }
        }
    } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t A[2][8];
#pragma unroll
            for (int i = 0; i < 2; ++i) nibbles_normal(A[i], word_of(w0, 2 * h + i), word_of(w1, 2 * h + i));
            const uint32_t z0 = word_of(w2, h), z1 = word_of(w2, 2 + h);  // (scale, minimum) of rows g and g + 8
            float2 s0 = __half22float2(*reinterpret_cast<const __half2*>(&z0)), s1 = __half22float2(*reinterpret_cast<const __half2*>(&z1));
            s0.y = fmaf(8.0f, s0.x, s0.y); s1.y = fmaf(8.0f, s1.x, s1.y);  // n * s + m = (n - 8) * s + (m + 8 * s)
#pragma unroll
            for (int n = 0; n < T; ++n) {
                const uint4 b0 = xp[(2 * h * T + n) * 32], b1 = xp[((2 * h + 1) * T + n) * 32];
                const float2 c = *reinterpret_cast<const float2*>(sp + (h * T + n) * 32);
                float e[4];
                mma16816_from(e, A[0][0], A[0][1], A[0][2], A[0][3], b0.x, b0.y, make_float4(0.f, 0.f, 0.f, 0.f));
                mma16816<FMT>(e, A[0][4], A[0][5], A[0][6], A[0][7], b0.z, b0.w);
                mma16816<FMT>(e, A[1][0], A[1][1], A[1][2], A[1][3], b1.x, b1.y);
                mma16816<FMT>(e, A[1][4], A[1][5], A[1][6], A[1][7], b1.z, b1.w);
                acc[n][0] = fmaf(e[0], s0.x, fmaf(c.x, s0.y, acc[n][0])); acc[n][1] = fmaf(e[1], s0.x, fmaf(c.y, s0.y, acc[n][1]));
                acc[n][2] = fmaf(e[2], s1.x, fmaf(c.x, s1.y, acc[n][2])); acc[n][3] = fmaf(e[3], s1.x, fmaf(c.y, s1.y, acc[n][3]));
            }
        }
    }
}
// Parts of a row of x -> one sum.  Two columns: lane (g,t) has row 4n + t of x for weight rows g and g + 8.  Four: its
// even lane gets row 2n + t/2 for weight row g, the odd one for g + 8 (the fourth column is never written: left out)
template <int FMT, int T>
__device__ __forceinline__ void lane_sums(float* y, const float (&acc)[T][4], uint32_t t) {
#pragma unroll
    for (int n = 0; n < T; ++n) {
        const float* e = acc[n];
        if constexpr (Mm<FMT>::cols == 2) {
            y[n * 2] = e[0] + e[1];
            y[n * 2 + 1] = e[2] + e[3];
        } else {
            const bool odd = t & 1;
            const float own0 = odd ? e[0] : e[0] + e[1], own1 = odd ? e[2] : e[2] + e[3];
            const float got = __shfl_xor_sync(0xFFFFFFFFu, odd ? own0 : own1, 1);
            y[n] = (odd ? own1 : own0) + got;
        }
    }
}

// fp16 and bf16 weights.  Grid: (tile groups * splits) blocks, clusters of `splits`; T groups of 8 columns, MT row tiles per warp
template <int FMT, int T>
__global__ void __launch_bounds__(MmShape<FMT, T>::warps * 32, MmShape<FMT, T>::per_sm) k_gemv_mma(const MmArgs a) {
    typedef Mm<FMT> F;
    typedef MmShape<FMT, T> P;
    constexpr int MT = P::mt, D = P::depth, MM_WARPS = P::warps, MM_SLOTS = P::slots, SLOT = P::slot, BLK_X = T * F::x_bytes, WB = P::w_blk;
    static_assert(!F::q4 && F::cols == 4, "16-bit weights");
    constexpr int NV = MT * T;                               // sums a lane ends up with
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
    // weights of this lane: rows g and g + 8 of each tile (SwiGLU: the same row of gate and up)
    const unsigned char *pa[MT], *pb[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const uint32_t tile = min(tile0 + m, a.n_tiles - 1);
        const uint32_t r0 = min(swiglu ? tile * 8 + g : tile * 16 + g, a.rows - 1), r1 = min(swiglu ? r0 : tile * 16 + 8 + g, a.rows - 1);
        pa[m] = a.w + ((size_t)r0 * a.K + kb0 * F::kb + 8 * t) * 2;
        pb[m] = (swiglu ? a.w2 : a.w) + ((size_t)r1 * a.K + kb0 * F::kb + 8 * t) * 2;
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
                cp_async16(dst, pa[m]); cp_async16(dst + 512, pb[m]);
                cp_async16(dst + 1024, pa[m] + 64); cp_async16(dst + 1536, pb[m] + 64);
                pa[m] += 128; pb[m] += 128;
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
            mm_wait(empty + 8 * ((gone - 1) % MM_SLOTS), ((gone - 1) / MM_SLOTS) & 1u, a.err, a.stop);
            fill(gone - 1 + MM_SLOTS);
        }
        __syncwarp();
        mm_wait(full + 8 * at, phase & 1u, a.err, a.stop);
#pragma unroll
        for (int q = 0; q < MM_SLOT_BLKS; ++q) {
            if (blk + q < n_kb) {
                request(any && blk + q + D - 1 < n_kb);
                asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
                __syncwarp();
                const unsigned char* xb = smem + at * SLOT + q * BLK_X;
                const uint4* xp = reinterpret_cast<const uint4*>(xb) + lane;
                const uint4* wp = reinterpret_cast<const uint4*>(wring + w_out);
                w_out = w_out == (D - 1) * MT * WB ? 0 : w_out + MT * WB;
                uint4 w[MT][4];
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[m][i] = wp[m * (WB / 16) + i * 32 + lane];
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
                __syncwarp();  // before the next block's request overwrites what other lanes may still read
            }
        }
        if (lane == 0) mbar_arrive(empty + 8 * at);
        if (++at == MM_SLOTS) { at = 0; ++phase; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    float y[NV];
#pragma unroll
    for (int m = 0; m < MT; ++m) lane_sums<FMT, T>(y + m * T, acc[m], t);
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
                const uint32_t b = n * 2 + (t >> 1);  // row of x
                const bool live = tile < a.n_tiles && b < a.batch && (!a.state || a.state[b].active);
                const float un = live ? a.unscale[b] : 0.0f;
                float* d = a.dst + (size_t)b * a.dst_stride + a.dst_offset;
                float v0 = y[m * T + n], v1 = v0;  // weight rows g and g + 8
                bool has0 = live && !(t & 1), has1 = live && (t & 1);
                if (swiglu) {
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, v0, 1);
                    if (t & 1) v0 = other; else v1 = other;
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

__device__ __forceinline__ float4 norm4(const void* w, int fmt, uint32_t i4) {
    if (fmt == VB_FMT_F32) return __ldg(reinterpret_cast<const float4*>(w) + i4);
    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(w) + i4);
    if (fmt == VB_FMT_F16) {
        const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), q = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        return make_float4(p.x, p.y, q.x, q.y);
    }
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xFFFF0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xFFFF0000u));
}

// 2^(13 - floor(log2 max)), kept inside the exponents of a float: what brings a row's maximum into [2^13, 2^14)
__device__ __forceinline__ float x_scale(float mx) {
    if (!(mx > 0.0f && mx < 3.0e38f)) return 1.0f;
    const int e = min(max((int)((__float_as_uint(mx) >> 23) & 255u) - 127, -100), 127);
    return __uint_as_float((uint32_t)(127 + 13 - e) << 23);
}
// Lane t's share of K [32 k32, +32) of row b of x (p, q: its two runs of four elements; `in`: it exists), times `up`, as parts into the
// fragments at xf (T groups of 8 columns); the `first` lane of a sum's K stores the sums.  Four (group-64: eight) lanes call together.
template <int FMT>
__device__ __forceinline__ void x_unit(unsigned char* xf, uint32_t T, uint32_t k32, uint32_t t, uint32_t b, const float4& p, const float4& q, float up, bool in, bool first) {
    typedef Mm<FMT> F;
    float v[8];
    if constexpr (F::q4) { v[0] = p.x; v[1] = p.z; v[2] = q.x; v[3] = q.z; v[4] = p.y; v[5] = p.w; v[6] = q.y; v[7] = q.w; }
    else { v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w; }
    const uint32_t n = b / F::rows, col0 = (b % F::rows) * F::cols;
    unsigned char* blk = xf + (size_t)(k32 / F::frags) * T * F::x_bytes;  // the weight block's share
    uint4* frag = reinterpret_cast<uint4*>(blk) + ((k32 % F::frags) * T + n) * 32;
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
            if (in && first) {
                unsigned char* sums = blk + F::frags * T * 512 + ((k32 % F::frags) / (F::sx_k / 32) * T + n) * F::sum_bytes;
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

// ---- int4 weights: x resident in shared memory --------------------------------------------------------------------------
// One persistent block of 16 warps per SM: two groups of 8 warps, each group on its own row tile, whose K its warps split by pairs of
// weight blocks; x comes in chunks of a pair for each warp, two of them: a row of up to 4096 stays for all tiles of the block, a
// longer one goes round.
template <int FMT, int T> struct MrShape {
    static constexpr int warps = 8, groups = 2, threads = groups * warps * 32;
    static constexpr int chunk = 2 * warps;                     // weight blocks of a chunk of x
    static constexpr int slots = 2, places = T == 1 ? 2 : 1;    // chunks in shared memory; of the warps' sums
    static constexpr int depth = T == 1 ? 3 : 2, pair = 2 * MM_Q4_BLK;  // pairs of a warp's weight ring
    static constexpr int blk_x = T * Mm<FMT>::x_bytes, slot = chunk * blk_x;
    static constexpr int nv = T * (Mm<FMT>::cols == 2 ? 2 : 1); // sums a lane ends up with
    static constexpr int ring = slots * slot, red = ring + groups * warps * depth * pair, bars = red + groups * places * warps * nv * 128, smem = bars + 16 * slots;
    static_assert(smem <= 232448 - 1024, "shared memory");
};

// where x comes from: fragments that k_x_frag wrote, resident or in a ring of chunks, or the rows themselves (K up to 4096)
enum { MR_RING, MR_RES, MR_SELF };
template <int FMT, int T, int X>
__global__ void __launch_bounds__(MrShape<FMT, T>::threads, 1) k_gemv_mma_res(const MmArgs a) {
    constexpr bool RES = X != MR_RING;
    typedef Mm<FMT> F;
    typedef MrShape<FMT, T> P;
    static_assert(F::q4, "v3 tiles");
    constexpr int D = P::depth, NV = P::nv;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float un_s[T * F::rows];
    const uint32_t xs = smem_u32(smem), full = xs + P::bars, empty = full + 8 * P::slots;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5, group = wid / P::warps, warp = wid % P::warps, g = lane >> 2, t = lane & 3;
    const uint32_t gt = threadIdx.x % (P::warps * 32);  // thread of the group
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < P::slots; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, P::groups * P::warps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    trace_mark(a.trace, 0);
    pdl_launch_dependents();
    const uint32_t KT = a.K / F::kb, n_ch = (KT + P::chunk - 1) / P::chunk, vstride = P::groups * gridDim.x, tile0 = blockIdx.x + group * gridDim.x;
    const uint32_t rounds = (a.n_tiles - blockIdx.x + vstride - 1) / vstride;  // of the block's first group: the other one has no more
    const bool swiglu = a.epilogue == EPI_SWIGLU;

    // weights: this warp's pairs warp, warp + 8, ... of tile after tile, through a ring of its own
    const uint32_t my_ch = 2 * warp < KT ? (KT - 2 * warp + P::chunk - 1) / P::chunk : 0;  // pairs of a tile
    const uint32_t my_tiles = tile0 < a.n_tiles ? (a.n_tiles - tile0 + vstride - 1) / vstride : 0;
    uint32_t r_left = my_ch * my_tiles, r_ch = my_ch;  // pairs to request, of this tile
    const unsigned char* src = a.w + ((size_t)tile0 * KT + 2 * warp) * MM_Q4_BLK + 16 * lane;
    const size_t jump = ((size_t)vstride * KT - (size_t)my_ch * P::chunk) * MM_Q4_BLK;  // from behind a tile's last pair to the next tile's first
    const bool odd_end = my_ch && 2 * warp + (my_ch - 1) * P::chunk + 1 >= KT;         // the last pair is one block
    const unsigned char* const wring = smem + P::ring + wid * (D * P::pair);
    const uint32_t wring_s = smem_u32(wring) + 16 * lane;
    uint32_t w_in = 0, w_out = 0;
    auto request = [&]() {
        if (r_left) {
            const uint32_t dst = wring_s + w_in;
            cp_async16(dst, src);
            cp_async16(dst + 512, src + 512);
            if (r_ch == 1 && odd_end) {
                if (lane < 8) cp_async16(dst + 1024, src + 1024);
            } else {
                cp_async16(dst + 1024, src + 1024);
                cp_async16(dst + 1536, src + 1536);
                if (lane < 16) cp_async16(dst + 2048, src + 2048);
            }
            w_in = w_in == (D - 1) * P::pair ? 0 : w_in + P::pair;
            src += P::chunk * MM_Q4_BLK;
            --r_left;
            if (--r_ch == 0) { r_ch = my_ch; src += jump; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int d = 0; d < D - 1; ++d) request();

    [[maybe_unused]] float4 wp4 = make_float4(1.f, 1.f, 1.f, 1.f), wq4 = wp4;
    const uint32_t k32 = threadIdx.x >> 2, e0 = k32 * 32 + 4 * t, e1 = e0 + 16;  // MR_SELF: this thread's share of a row
    const bool in_row = k32 * 32 < a.K;
    if constexpr (X == MR_SELF)
        if (a.norm_w && in_row) { wp4 = norm4(a.norm_w, a.norm_fmt, e0 / 4); wq4 = norm4(a.norm_w, a.norm_fmt, e1 / 4); }
    pdl_wait();
    trace_mark(a.trace, 1);
    if constexpr (X == MR_SELF) {
        // every block converts all rows: less than a kernel before this one and its hand-over (3.3 us, of which 2.7 are its own)
        constexpr int ROWS = T * F::rows;
        __shared__ float red_s[ROWS][P::threads / 32], red_m[ROWS][P::threads / 32];
        float4 p[ROWS], q[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            p[r] = q[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in_row && (uint32_t)r < a.batch) {
                p[r] = *reinterpret_cast<const float4*>(a.x + (size_t)r * a.K + e0);
                q[r] = *reinterpret_cast<const float4*>(a.x + (size_t)r * a.K + e1);
            }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            float ss = 0.0f;
            if (a.norm_w) {
                ss = fmaf(p[r].x, p[r].x, fmaf(p[r].y, p[r].y, fmaf(p[r].z, p[r].z, p[r].w * p[r].w)));
                ss = fmaf(q[r].x, q[r].x, fmaf(q[r].y, q[r].y, fmaf(q[r].z, q[r].z, fmaf(q[r].w, q[r].w, ss))));
                p[r].x *= wp4.x; p[r].y *= wp4.y; p[r].z *= wp4.z; p[r].w *= wp4.w;
                q[r].x *= wq4.x; q[r].y *= wq4.y; q[r].z *= wq4.z; q[r].w *= wq4.w;
                ss = warp_sum(ss);
            }
            const float mx = warp_max(fmaxf(fmaxf(fmaxf(fabsf(p[r].x), fabsf(p[r].y)), fmaxf(fabsf(p[r].z), fabsf(p[r].w))),
                                            fmaxf(fmaxf(fabsf(q[r].x), fabsf(q[r].y)), fmaxf(fabsf(q[r].z), fabsf(q[r].w)))));
            if (lane == 0) { red_s[r][wid] = ss; red_m[r][wid] = mx; }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if ((uint32_t)r < a.batch) {  // (an inactive row's products are not written)
                float ss = 0.0f, mx = 0.0f, inv = 1.0f;
#pragma unroll
                for (int w = 0; w < P::threads / 32; ++w) { ss += red_s[r][w]; mx = fmaxf(mx, red_m[r][w]); }
                if (a.norm_w) { inv = 1.0f / sqrtf(ss / (float)a.K + a.eps); mx *= inv; }
                const float up = x_scale(mx);
                if (threadIdx.x == 0) un_s[r] = (FMT == VB_FMT_Q4G32 ? 16777216.0f : 1.0f) / up;
                const float f = inv;
                p[r].x *= f; p[r].y *= f; p[r].z *= f; p[r].w *= f;
                q[r].x *= f; q[r].y *= f; q[r].z *= f; q[r].w *= f;
                x_unit<FMT>(smem, T, k32, t, (uint32_t)r, p[r], q[r], up, in_row, threadIdx.x % (F::sx_k / 8) == 0);
            }
        }
        __syncthreads();
    }
    const uint32_t n_fill = RES ? n_ch : n_ch * rounds;
    auto fill = [&](uint32_t q) {  // one thread: chunk q % n_ch of x
        const uint32_t ch = RES ? q : q % n_ch, slot = RES ? q : q % P::slots, bytes = min((uint32_t)P::chunk, KT - ch * P::chunk) * P::blk_x;
        mbar_expect_tx(full + 8 * slot, bytes);
        tma_load_1d(xs + slot * P::slot, a.xf + (size_t)ch * P::slot, bytes, full + 8 * slot);
    };
    // (a bulk copy holds its thread for ~400 clocks: every warp issues one in its turn)
    if (X != MR_SELF && lane == 0 && wid < min((uint32_t)P::slots, n_fill)) fill(wid);

    // the thread that writes: sums (n, lane) of a tile; its row of x
    const uint32_t b = F::cols == 2 ? (gt >> 5) * 4 + t : (gt >> 5) * 2 + (t >> 1);
    const bool writer = gt < T * 32, live = writer && b < a.batch && (!a.state || a.state[b].active);
    const float un = !live ? 0.0f : X == MR_SELF ? un_s[b] : a.unscale[b];
    float* const dst = a.dst + (size_t)(live ? b : 0) * a.dst_stride + a.dst_offset;
    const unsigned char* const x0 = smem + 2 * warp * P::blk_x;
    uint32_t q = 0;
#pragma unroll 1
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t tile = tile0 + r * vstride;
        const bool has = tile < a.n_tiles;
        // what the sums are added to, fetched early
        const bool has0 = live && has && (F::cols == 2 || !(t & 1)), has1 = live && has && !swiglu && (F::cols == 2 || (t & 1));
        float res0 = 0.0f, res1 = 0.0f;
        if (a.epilogue == EPI_RESIDUAL) {
            if (has0) res0 = dst[tile * 16 + g];
            if (has1) res1 = dst[tile * 16 + g + 8];
        }
        float acc[T][4];
#pragma unroll
        for (int n = 0; n < T; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = 0.0f;
        uint32_t left = has ? my_ch : 0, x_at = 0;
#pragma unroll 1
        for (uint32_t ch = 0; ch < (RES ? left : n_ch); ++ch) {
            if constexpr (RES) {
                if (X == MR_RES && r == 0) mm_wait(full + 8 * ch, 0, a.err, a.stop);
            } else {
                const uint32_t slot = q % P::slots;
                if (q > 0 && q - 1 + P::slots < n_fill && wid == q % (P::groups * P::warps) && lane == 0) {
                    mm_wait(empty + 8 * ((q - 1) % P::slots), ((q - 1) / P::slots) & 1u, a.err, a.stop);
                    fill(q - 1 + P::slots);
                }
                __syncwarp();
                mm_wait(full + 8 * slot, (q / P::slots) & 1u, a.err, a.stop);
                x_at = slot * P::slot;
            }
            if (RES || ch < left) {
                request();
                asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
                __syncwarp();
                const unsigned char* xb = x0 + x_at;
                const uint4* wp = reinterpret_cast<const uint4*>(wring + w_out);
                w_out = w_out == (D - 1) * P::pair ? 0 : w_out + P::pair;
                q4_block<FMT, T>(acc, wp[lane], wp[32 + lane], wp[64 + g], reinterpret_cast<const uint4*>(xb) + lane,
                                 xb + F::frags * T * 512 + (FMT == VB_FMT_Q4G32 ? 16 : 8) * t);
                if (ch + 1 < left || !odd_end)
                    q4_block<FMT, T>(acc, wp[72 + lane], wp[104 + lane], wp[136 + g], reinterpret_cast<const uint4*>(xb + P::blk_x) + lane,
                                     xb + P::blk_x + F::frags * T * 512 + (FMT == VB_FMT_Q4G32 ? 16 : 8) * t);
                __syncwarp();  // before the next request overwrites what other lanes may still read
            }
            if constexpr (RES) x_at += P::slot;
            else {
                if (lane == 0) mbar_arrive(empty + 8 * (q % P::slots));
                ++q;
            }
        }
        if (has) {
            float y[NV];
            lane_sums<FMT, T>(y, acc, t);
            // the 8 warps' sums through shared memory; with two places in turn one barrier of the group per tile is enough
            float* red = reinterpret_cast<float*>(smem + P::red) + (group * P::places + (P::places == 2 ? r & 1 : 0)) * (P::warps * NV * 32);
#pragma unroll
            for (int i = 0; i < NV; ++i) red[(warp * NV + i) * 32 + lane] = y[i];
            asm volatile("bar.sync %0, %1;" ::"r"(1u + group), "n"(P::warps * 32) : "memory");
            if (writer) {
                const uint32_t n = gt >> 5;
                float v0 = 0.0f, v1 = 0.0f;
#pragma unroll
                for (int w = 0; w < P::warps; ++w) {
                    if constexpr (F::cols == 2) { v0 += red[(w * NV + 2 * n) * 32 + lane]; v1 += red[(w * NV + 2 * n + 1) * 32 + lane]; }
                    else v0 += red[(w * NV + n) * 32 + lane];
                }
                if constexpr (F::cols != 2) {
                    v1 = v0;
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, v0, 1);
                    if (swiglu) v1 = other;  // (the even lane writes)
                }
                v0 *= un; v1 *= un;
                if (swiglu) {
                    if (has0) dst[tile * 8 + g] = (v0 / (1.0f + expf(-v0))) * v1;
                } else {
                    if (has0) dst[tile * 16 + g] = res0 + v0;
                    if (has1) dst[tile * 16 + g + 8] = res1 + v1;
                }
            }
            if constexpr (P::places == 1) asm volatile("bar.sync %0, %1;" ::"r"(1u + group), "n"(P::warps * 32) : "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
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
        if (SCALED) up = x_scale(mx);
    }
    if (!active) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.unscale[b] = (FMT == VB_FMT_Q4G32 ? 16777216.0f : 1.0f) / up;
    if (a.norm_w && in) {
        p.x = (p.x * inv) * wp.x; p.y = (p.y * inv) * wp.y; p.z = (p.z * inv) * wp.z; p.w = (p.w * inv) * wp.w;
        q.x = (q.x * inv) * wq.x; q.y = (q.y * inv) * wq.y; q.z = (q.z * inv) * wq.z; q.w = (q.w * inv) * wq.w;
    }
    x_unit<FMT>(a.xf, a.T, k32, t, b, p, q, up, in, unit % (F::sx_k / 8) == 0);
}

template <int FMT, int T>
cudaError_t launch_mma(const LaunchCfg& lc, MmArgs a) {
    typedef MmShape<FMT, T> P;
    const uint32_t groups = (a.n_tiles + P::warps * P::mt - 1) / (P::warps * P::mt), KT = a.K / Mm<FMT>::kb;
    // Few tiles: split K over a cluster while all its blocks find a place at once and every warp keeps four weight blocks (a
    // cluster that has to wait starts a wave of its own).  Pairs may go a quarter beyond: they slip in as soon as two blocks leave.
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

template <int FMT, int T, int X>
cudaError_t launch_mma_res(const LaunchCfg& lc, const MmArgs& a) {
    typedef MrShape<FMT, T> P;
    static std::atomic<uint64_t> opted{0};
    const cudaError_t oe = once_per_device(opted, [&]() { return cudaFuncSetAttribute(k_gemv_mma_res<FMT, T, X>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::smem); });
    if (oe != cudaSuccess) return oe;
    return launch(lc, k_gemv_mma_res<FMT, T, X>, dim3(std::min(148u, a.n_tiles)), dim3(P::threads), P::smem, a);
}

// one pass: the rows of x that fit T groups of 8 columns
template <int FMT>
cudaError_t pass_mma(const LaunchCfg& lc, MmArgs a, XfArgs f, unsigned char* ws) {
    const uint32_t tiles = (a.batch + Mm<FMT>::rows - 1) / Mm<FMT>::rows, T = tiles <= 2 ? tiles : 4;
    f.T = T;
    f.xf = ws;
    f.unscale = reinterpret_cast<float*>(ws + (size_t)(f.K / Mm<FMT>::kb) * T * Mm<FMT>::x_bytes);
    a.xf = f.xf; a.unscale = f.unscale;
    if constexpr (Mm<FMT>::q4) {
        // Up to three rows that a block's threads hold, 8 elements each: converted by the product itself (8B shape, a step, ms: one row of
        // group-64 1.78 -> 1.61, two 1.83 -> 1.72; int4, two rows 1.80 -> 1.73, three 1.81 -> 1.78, four 1.82 -> 1.85).
        if (T == 1 && a.batch <= 3 && f.K <= MrShape<FMT, 1>::threads * 8) {
            a.x = f.x; a.norm_w = f.norm_w; a.norm_fmt = f.norm_fmt; a.eps = f.eps;
            return launch_mma_res<FMT, 1, MR_SELF>(lc, a);
        }
    }
    cudaError_t e = launch(lc, k_x_frag<FMT>, dim3((f.K + 4095) / 4096, a.batch), dim3(XF_THREADS), 0, f);
    if (e != cudaSuccess) return e;
    if constexpr (Mm<FMT>::q4) {
        const bool fits = f.K <= (uint32_t)(MrShape<FMT, 1>::slots * MrShape<FMT, 1>::chunk * Mm<FMT>::kb);
        if (T == 1) return fits ? launch_mma_res<FMT, 1, MR_RES>(lc, a) : launch_mma_res<FMT, 1, MR_RING>(lc, a);
        return fits ? launch_mma_res<FMT, 2, MR_RES>(lc, a) : launch_mma_res<FMT, 2, MR_RING>(lc, a);
    } else {
        if (T == 1) return launch_mma<FMT, 1>(lc, a);
        return T == 2 ? launch_mma<FMT, 2>(lc, a) : launch_mma<FMT, 4>(lc, a);
    }
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
        // One row: the integer kernel streams fastest.  2..4 rows: its multi-row flavour is one launch and ahead for small matrices
        // (models of 1024 / 1536 / 2048 columns, a step of 2 rows: 387 / 391 / 297 us, here 509 / 426 / 334); at the 8B shape all products of
        // a step here are (2 / 3 / 4 rows 1.80 / 1.80 / 1.82 ms, all there 1.88 / 1.93 / 2.00, each the faster way for itself 1.90 .. 2.1:
        // the two kernels in turn cost more than either).
        if (g.batch < 2 || (g.batch <= 4 && weights < 8000000ull)) return cudaSuccess;
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
    error_words(lc, &a.err, &a.stop);
    a.rows = g.w.rows; a.K = K; a.epilogue = g.epilogue; a.trace = g.trace;
    a.dst_stride = g.dst_stride ? g.dst_stride : g.w.rows; a.dst_offset = g.dst_offset;
    XfArgs f;
    f.norm_w = g.norm_w; f.norm_fmt = g.norm_fmt; f.eps = g.eps; f.K = K;
    *handled = true;
    // rows of a pass: 16 columns of int4 weights (32 of them in one pass, on a kernel that kept two row tiles a warp: 9 rows 4.57 ms a step
    // of the 8B shape, now 3.99, 16 rows 4.76 / 4.71; group-64, 5 rows 4.42 / 3.81), 32 of the others
    const uint32_t per = g.w.fmt == VB_FMT_Q4G32 ? 8 : q4 ? 4 : 8;
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
