// Multi-head latent attention decode on the 5th-generation tensor cores: both products of the absorbed form run as
// tcgen05.mma with their accumulators in tensor memory.
//
// Same contract as k_mla_decode (vb_mla_decode.cu; model shape examples/deepseek_v3_mla.vlx:18-45, decode scope
// :117-150): per sequence, all heads share every latent row [c_kv 512 | k_rope 64] (bf16),
//     S[heads x tokens] = Q[heads x 576] . L^T,   P = softmax rows,   O[heads x 512] = P . L[:, :512].
//
// One block = 128 heads (the tensor-memory lanes) x one half of the 512 output dimensions (O needs 128 lanes x 512 fp32
// columns = all of tensor memory, so two blocks split the columns; each computes S for itself), 256 threads, one block per SM.
// The batch's 64-token tiles are dealt to 74 such pairs in equal contiguous runs that may begin and end inside a sequence
// (a run's part of a sequence = a piece), so no SM waits for a longer context than its share.  Per tile:
//   * warp 0 (one lane): tiled TMA brings the tile in as nine [64 rows][64 columns] boxes with the 128-byte swizzle, two tiles'
//     room: the five boxes that only S reads are free when S is done, the four of this block's output columns when P . L is.
//     Q (bf16, converted once by a small kernel): four boxes in shared memory, the last 320 of its 576 columns in tensor memory;
//   * warp 1: S = Q . L^T, 36 tcgen05.mma kind::f16 (bf16 operands, M 128, N 64, K 16), 16 with A from shared memory, 20 from
//     tensor memory;
//   * warp 2: O += P . L[:, half], four instructions (N 256, K 16) with P read FROM TENSOR MEMORY (bf16 pairs written by the
//     softmax warps with tcgen05.st) and the SAME staged boxes as the B operand, read MN-major (tokens are K);
//   * warps 4-7 (128 threads, one head row = one tensor-memory lane each): read their S row, free it for the next tile's product
//     at once, running maximum and sum without any shuffle, probabilities to bf16 into tensor memory.  The maximum is lazy: O is
//     rescaled (tcgen05.ld / st of 256 columns) only when a tile's maximum exceeds the one in use by more than 8 (in e), so that
//     probabilities stay below e^8 and almost every tile skips the rescale.
// Every hand-over is an mbarrier with a bounded wait and a block-wide abort flag (a wait that runs out sets a status word at
// the head of the scratch area: the merge kernel then fills the output with NaN).  Rows of the last tile past the end of the
// context are zeroed in shared memory before P . L (their probabilities are 0, but 0 x garbage must not be NaN).
//
// What a tensor instruction costs (M 128, K 16, measured back to back): N / 2 clocks of arithmetic; with A from shared memory at
// least 4 KB + the B tile at 128 bytes a clock: 45 clocks at N 16, 53 at N 64, 67 at N 128; with A from tensor memory N / 2 at
// every N.  Hence 64 tokens a tile (16: three times the clocks per token) and as much of Q as fits in tensor memory: 16 x 53 +
// 20 x 33 + 4 x 129 = 2.0 k clocks a tile.  These rates need the issuing lane chosen by elect.sync (vb_tma.cuh) and descriptors known at
// compile time up to a base: issued by `lane == 0` from a loop with run-time column blocks the same instructions came 183 clocks
// apart and the kernel took 270 us instead of 177.
// Measured, 64 sequences of 1024..8192 tokens (mean 4609): 132 us with conversion (6) and merge (14), 3.2 k clocks a tile, tensor
// pipe and shared memory (operands 170 KB + copies 72 KB a tile at 128 bytes a clock: 1.9 k) both about 60 % busy; 16-token tiles
// in 1024-row slices: 350 us.  On the way: nine barriers a tile instead of two 177; two buffers of P and five boxes of Q 158.
#include <cuda.h>
#include <cuda_bf16.h>

#include "vb_internal.cuh"
#include "vb_kernels.cuh"
#include "vb_tma.cuh"

namespace vb {
namespace {

constexpr int MT_LAT = 576, MT_V = 512;
constexpr int MT_M = 128;                 // heads per block = tensor-memory lanes
constexpr int MT_T = 64;                  // tokens per tile
constexpr int MT_KB = MT_LAT / 64;        // nine column blocks of 64 elements (128 bytes)
constexpr int MT_QS = 4, MT_QT = MT_KB - MT_QS;  // column blocks of Q in shared memory, in tensor memory
constexpr int MT_DH = 256;                // output dimensions per block
constexpr int MT_YB = MT_DH / 64, MT_XB = MT_KB - MT_YB;  // column blocks that S and P . L read, that only S reads
constexpr int MT_BOX = MT_T * 128, MT_QBOX = MT_M * 128, MT_TILE = MT_KB * MT_BOX;  // bytes
constexpr int MT_L_OFF = MT_QS * MT_QBOX, MT_BAR_OFF = MT_L_OFF + 2 * MT_TILE;      // two tiles
constexpr int MT_SMEM = MT_BAR_OFF + 128 + 1024;
static_assert(MT_SMEM <= 232448 - 64, "shared memory of one block");
constexpr int MT_THREADS = 256;
constexpr uint32_t MT_TMEM_COLS = 512;
constexpr uint32_t MT_TM_S = 0, MT_TM_P = 64, MT_TM_Q = 96, MT_TM_O = 256;  // scores; probabilities as bf16 pairs (32 columns); the last
                                                                             // column blocks of Q; the output
static_assert(MT_TM_Q + MT_QT * 32 <= MT_TM_O, "tensor memory columns");
constexpr int MT_ROW = MT_V + 8;          // floats of a partial row: output, maximum, sum, padding to whole 32 bytes
constexpr uint32_t MT_PAIRS = 74;         // pairs of blocks: one block per SM
constexpr float MT_LAZY = 8.0f * 1.4426950408889634f;

// instruction descriptors, kind::f16: fp32 accumulate (bit 4), A and B bf16 (1 at bits 7 and 10), N >> 3 at bit 17,
// M >> 4 at bit 24; bit 16 = B is MN-major
constexpr uint32_t MT_IDESC_S = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MT_T >> 3) << 17) | ((uint32_t)(MT_M >> 4) << 24);
constexpr uint32_t MT_IDESC_O = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(MT_DH >> 3) << 17) | ((uint32_t)(MT_M >> 4) << 24);

// K-major operand, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t desc_k_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// MN-major operand, 128-byte swizzle: 64 elements of MN contiguous (one 128-byte row per K index), the next 64 elements
// of MN `lbo` bytes further, groups of 8 K indices 1024 bytes apart
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void mma_bf16_ss(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// A from tensor memory (lane = row, two bf16 of K per 32-bit column), B from shared memory
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void commit_to(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// tcgen05.ld of 32 columns; the values are there only after tmem_ld_wait on them
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, float* u) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=f"(u[0]), "=f"(u[1]), "=f"(u[2]), "=f"(u[3]), "=f"(u[4]), "=f"(u[5]), "=f"(u[6]), "=f"(u[7]), "=f"(u[8]), "=f"(u[9]), "=f"(u[10]), "=f"(u[11]), "=f"(u[12]), "=f"(u[13]), "=f"(u[14]), "=f"(u[15]), "=f"(u[16]), "=f"(u[17]), "=f"(u[18]), "=f"(u[19]), "=f"(u[20]), "=f"(u[21]), "=f"(u[22]), "=f"(u[23]), "=f"(u[24]), "=f"(u[25]), "=f"(u[26]), "=f"(u[27]), "=f"(u[28]), "=f"(u[29]), "=f"(u[30]), "=f"(u[31])
                 : "r"(taddr) : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld_wait(float (&r)[N]) {  // (the registers go through it: nothing reads them before)
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+f"(r[i]));
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&r)[32]) {
    tmem_ld32_nowait(taddr, r);
    tmem_ld_wait(r);
}
__device__ __forceinline__ float exp2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float r[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])), "r"(__float_as_uint(r[3])),
                   "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])), "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7])),
                   "r"(__float_as_uint(r[8])), "r"(__float_as_uint(r[9])), "r"(__float_as_uint(r[10])), "r"(__float_as_uint(r[11])),
                   "r"(__float_as_uint(r[12])), "r"(__float_as_uint(r[13])), "r"(__float_as_uint(r[14])), "r"(__float_as_uint(r[15])),
                   "r"(__float_as_uint(r[16])), "r"(__float_as_uint(r[17])), "r"(__float_as_uint(r[18])), "r"(__float_as_uint(r[19])),
                   "r"(__float_as_uint(r[20])), "r"(__float_as_uint(r[21])), "r"(__float_as_uint(r[22])), "r"(__float_as_uint(r[23])),
                   "r"(__float_as_uint(r[24])), "r"(__float_as_uint(r[25])), "r"(__float_as_uint(r[26])), "r"(__float_as_uint(r[27])),
                   "r"(__float_as_uint(r[28])), "r"(__float_as_uint(r[29])), "r"(__float_as_uint(r[30])), "r"(__float_as_uint(r[31]))
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ bool wait_abort(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 128; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > 2000000000LL) { *abort_flag = 1u; return false; }
    }
}

// the same answer in every lane of a warp (the tensor-memory loads and __syncwarp that follow need the whole warp)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    return __all_sync(0xFFFFFFFFu, wait_abort(bar, parity, abort_flag));
}

struct MlaTcParams {
    const uint32_t* ctx_len;   // [B]
    float* out;                // [B][n_heads][512]
    float* partial;            // [pieces][min(n_heads, 128)][MT_ROW]
    const __nv_bfloat16* q16;  // [B][q_rows_per_seq][576]
    uint32_t* status;          // one word: nonzero when a wait ran out
    uint2* spans;              // [entries] first and last run of an entry
    uint32_t n_seq, n_heads, hbs, q_rows_per_seq;  // hbs: blocks of 128 heads, q_rows_per_seq = hbs * 128
    uint32_t min_tiles;        // of a run
    uint32_t max_rows;         // rows a sequence counts with at most: the launch and the scratch area are sized for them
    uint32_t direct;           // out takes 32-byte stores: sequences of one piece go straight there
    uint64_t cache_stride;     // rows between sequences
    float scale;
};

// The deal: entry e = (sequence e / hbs, head block e % hbs) has ceil(ctx / 64) tiles; all tiles in a row, runs of `run` each.
// Piece of run p in entry e: number p + e (each next piece raises one of the two by one).
// A device-side ctx_len beyond max_rows (a captured step whose context has outgrown its max_ctx) ends at max_rows.
__device__ __forceinline__ uint32_t mla_ctx(const MlaTcParams& p, uint32_t b) { return min(p.ctx_len[b], p.max_rows); }
__device__ __forceinline__ uint32_t mla_tiles(const MlaTcParams& p, uint32_t e) { return (mla_ctx(p, e / p.hbs) + MT_T - 1) / MT_T; }
__device__ __forceinline__ uint32_t mla_run(uint32_t total, uint32_t min_tiles) { return max((total + MT_PAIRS - 1) / MT_PAIRS, min_tiles); }
// sum over the block of one value per thread (every thread gets it); red: one word per warp
__device__ __forceinline__ uint32_t block_total(uint32_t v, uint32_t* red) {
    v = __reduce_add_sync(0xFFFFFFFFu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t s = 0;
    for (uint32_t i = 0; i < blockDim.x / 32; ++i) s += red[i];
    return s;
}

// the j-th column block of Q and L that S takes: the other half's, the rope block, then this block's own output columns
__device__ __forceinline__ uint32_t mla_block(uint32_t j, uint32_t dh) { return j < 4 ? (1 - dh) * 4 + j : (j == 4 ? 8 : dh * 4 + j - 5); }

__global__ void __launch_bounds__(MT_THREADS, 1)
k_mla_decode_tc(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_l, const MlaTcParams p) {
    const uint32_t pair = blockIdx.x >> 1, dh = blockIdx.x & 1, warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint32_t red[MT_THREADS / 32], s_entry, s_off;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t q_s = base, l_s = base + MT_L_OFF, bars = base + MT_BAR_OFF;
    // barriers (8 bytes each); q_t, s_free and p_full: the four softmax warps, the others one arrival
    constexpr int B_QFULL = 0, B_XFULL = 1, B_YFULL = 3, B_PVDONE = 5, B_SFULL = 7, B_QT = 9, B_SFREE = 10, B_PFULL = 11, B_COUNT = 12;
    auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + MT_BAR_OFF + B_COUNT * 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    if (threadIdx.x == 0) {
        for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_QT ? 4 : 1);
        *abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(MT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_launch_dependents();
    // ---- this pair's run of tiles (the kernel before this one, q's conversion, was launched behind everything that may have
    // written ctx_len: only q16 has to be waited for) ---------------------------------------------------------------------------------------
    const uint32_t n_entries = p.n_seq * p.hbs;
    uint32_t mine = 0;
    for (uint32_t e = threadIdx.x; e < n_entries; e += MT_THREADS) mine += mla_tiles(p, e);
    const uint32_t total = block_total(mine, red), run = mla_run(total, p.min_tiles), lo = pair * run;
    for (uint32_t e0 = 0, before = 0; e0 < n_entries && before <= lo; e0 += MT_THREADS) {
        // where the run begins: exclusive scan of 256 entries at a time
        const uint32_t e = e0 + threadIdx.x, v = e < n_entries ? mla_tiles(p, e) : 0;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t n = __shfl_up_sync(0xFFFFFFFFu, incl, o); if (lane >= (uint32_t)o) incl += n; }
        __syncthreads();
        if (lane == 31) red[warp] = incl;
        __syncthreads();
        uint32_t excl = before + incl - v;
        for (uint32_t w = 0; w < MT_THREADS / 32; ++w) { if (w < warp) excl += red[w]; before += red[w]; }
        if (v > 0 && excl <= lo && lo < excl + v) { s_entry = e; s_off = lo - excl; }
    }
    pdl_wait();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_o = tmem + MT_TM_O;

    // Tile m (counted over the whole run) lies in slot m & 1 (its five S-only boxes free when S is there, the other four when
    // P . L is done).  A barrier's n-th completion has parity (n - 1) & 1, and a wait is safe only while the barrier can be at most one completion past it: every barrier that
    // two roles may see apart by a tile exists once per slot.
    uint32_t n = 0, e = s_entry, off = s_off, left = lo < total ? min(run, total - lo) : 0;
    uint32_t pieces = 0;
    for (; left > 0; ++e, off = 0) {
        const uint32_t b = e / p.hbs, hb = e % p.hbs, ctx = mla_ctx(p, b), tiles_e = (ctx + MT_T - 1) / MT_T;
        const uint32_t nt = min(left, tiles_e - off);
        if (nt == 0) continue;
        left -= nt;
        const uint32_t qph = pieces & 1;
        if (threadIdx.x == 0 && dh == 0) {
            if (off == 0) p.spans[e].x = pair;
            if (off + nt == tiles_e) p.spans[e].y = pair;
        }
        if (warp == 0) {
            if (lane == 0) {
                // ---- producer: Q (nothing of the piece before is in flight any more), then the tiles -------------------------
                mbar_expect_tx(bar(B_QFULL), MT_QS * MT_QBOX);
                const int q_row = (int)(b * p.q_rows_per_seq + hb * MT_M);
                for (uint32_t j = 0; j < MT_QS; ++j) tma_2d(q_s + j * MT_QBOX, &map_q, (int)mla_block(j, dh) * 64, q_row, bar(B_QFULL));
                const long long row0 = (long long)b * (long long)p.cache_stride + (long long)off * MT_T;
                for (uint32_t i = 0; i < nt; ++i) {
                    const uint32_t m = n + i, slot = m & 1, dst = l_s + slot * MT_TILE;
                    const int y = (int)(row0 + (long long)i * MT_T);
                    if (m >= 2 && !wait_abort(bar(B_SFULL + slot), ((m >> 1) + 1) & 1, abort_flag)) break;  // S of tile m - 2 is there
                    mbar_expect_tx(bar(B_XFULL + slot), MT_XB * MT_BOX);
                    for (uint32_t j = 0; j < MT_XB; ++j) tma_2d(dst + j * MT_BOX, &map_l, (int)mla_block(j, dh) * 64, y, bar(B_XFULL + slot));
                    if (m >= 2 && !wait_abort(bar(B_PVDONE + slot), ((m >> 1) + 1) & 1, abort_flag)) break;
                    mbar_expect_tx(bar(B_YFULL + slot), MT_YB * MT_BOX);
                    for (uint32_t j = MT_XB; j < MT_KB; ++j) tma_2d(dst + j * MT_BOX, &map_l, (int)mla_block(j, dh) * 64, y, bar(B_YFULL + slot));
                }
            }
        } else if (warp == 1) {
            // ---- S = Q . L^T (the warp waits together, an elected lane issues: see the head of the file) -----------------------
            bool ok = warp_wait(bar(B_QFULL), qph, abort_flag) && warp_wait(bar(B_QT), qph, abort_flag);
            for (uint32_t i = 0; i < nt && ok; ++i) {
                const uint32_t m = n + i, slot = m & 1, lt = l_s + slot * MT_TILE;
                auto blocks = [&](int j0, int j1) {  // the four K steps of each column block
#pragma unroll
                    for (int j = j0; j < j1; ++j) {
                        const uint64_t db = desc_k_sw128(lt + j * MT_BOX), da = desc_k_sw128(q_s + j * MT_QBOX);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (j < MT_QS) mma_bf16_ss(tmem + MT_TM_S, da + 2u * k, db + 2u * k, MT_IDESC_S, (j | k) != 0 ? 1u : 0u);
                            else mma_bf16_ts(tmem + MT_TM_S, tmem + MT_TM_Q + (j - MT_QS) * 32 + k * 8, db + 2u * k, MT_IDESC_S, (j | k) != 0 ? 1u : 0u);
                        }
                    }
                };
                ok = warp_wait(bar(B_XFULL + slot), (m >> 1) & 1, abort_flag) && (m == 0 || warp_wait(bar(B_SFREE), (m + 1) & 1, abort_flag));
                if (!ok) break;
                fence_after();
                if (elect_one()) blocks(0, MT_XB);
                __syncwarp();
                ok = warp_wait(bar(B_YFULL + slot), (m >> 1) & 1, abort_flag);
                if (!ok) break;
                fence_after();
                if (elect_one()) { blocks(MT_XB, MT_KB); commit_to(bar(B_SFULL + slot)); }
                __syncwarp();
            }
        } else if (warp == 2) {
            // ---- O += P . L -----------------------------------------------------------------------------------------------------
            for (uint32_t i = 0; i < nt; ++i) {
                const uint32_t m = n + i, slot = m & 1;
                if (!warp_wait(bar(B_PFULL), m & 1, abort_flag)) break;
                fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < MT_T / 16; ++k)
                        mma_bf16_ts(tmem_o, tmem + MT_TM_P + k * 8, desc_mn_sw128(l_s + slot * MT_TILE + MT_XB * MT_BOX + k * 2048, MT_BOX), MT_IDESC_O,
                                    (i | (uint32_t)k) != 0 ? 1u : 0u);
                    commit_to(bar(B_PVDONE + slot));
                }
                __syncwarp();
            }
        } else if (warp >= 4) {
            // ---- softmax: thread = head row = tensor-memory lane ------------------------------------------------------------
            const uint32_t lg = warp & 3, row = lg * 32 + lane;  // the lanes this warp may touch: 32 * (warp % 4)
            const uint32_t lane_addr = (lg * 32u) << 16;
            {
                // the last column blocks of this head's Q (the products that read the ones before are done)
                const __nv_bfloat16* q_head = p.q16 + ((size_t)b * p.q_rows_per_seq + hb * MT_M + row) * MT_LAT;
#pragma unroll
                for (int c = 0; c < MT_QT; ++c) {
                    const uint4* q = reinterpret_cast<const uint4*>(q_head + mla_block(MT_QS + c, dh) * 64);
                    float r[32];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint4 v = q[i];
                        r[4 * i] = __uint_as_float(v.x); r[4 * i + 1] = __uint_as_float(v.y); r[4 * i + 2] = __uint_as_float(v.z); r[4 * i + 3] = __uint_as_float(v.w);
                    }
                    tmem_st32(tmem + lane_addr + MT_TM_Q + c * 32, r);
                }
                tmem_st_wait();
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_QT));
            }
            const float sl2 = p.scale * 1.4426950408889634f;
            float m_use = -INFINITY, l_run = 0.0f;
            bool ok = true;
            // has P . L of tile t completed?
            auto pv_done = [&](uint32_t t) { return warp_wait(bar(B_PVDONE + (t & 1)), (t >> 1) & 1, abort_flag); };
            for (uint32_t i = 0; i < nt && ok; ++i) {
                const uint32_t m = n + i;
                ok = warp_wait(bar(B_SFULL + (m & 1)), (m >> 1) & 1, abort_flag);
                if (!ok) break;
                fence_after();
                float s[MT_T];
                tmem_ld32_nowait(tmem + lane_addr + MT_TM_S, s);
                tmem_ld32_nowait(tmem + lane_addr + MT_TM_S + 32, s + 32);
                tmem_ld_wait(s);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_SFREE));
                const uint32_t valid = min((uint32_t)MT_T, ctx - (off + i) * MT_T);
                float mx = -INFINITY;
                if (valid < (uint32_t)MT_T) {
#pragma unroll
                    for (int j = 0; j < MT_T; ++j) s[j] = (uint32_t)j < valid ? s[j] : -INFINITY;
                }
#pragma unroll
                for (int j = 0; j < MT_T; ++j) mx = fmaxf(mx, s[j]);
                mx *= sl2;  // scores in units of log2
                // lazy maximum: move only when the tile's exceeds the one in use by more than MT_LAZY (always on the first tile)
                const bool move = mx > m_use + MT_LAZY || i == 0;
                const float m_new = move ? mx : m_use;
                const float alpha = move ? (i == 0 ? 0.0f : exp2f(m_use - m_new)) : 1.0f;
                float packed[MT_T / 2];
                float sum = 0.0f;
#pragma unroll
                for (int j = 0; j < MT_T / 2; ++j) {
                    const __nv_bfloat162 pr = __floats2bfloat162_rn(exp2_fast(fmaf(s[2 * j], sl2, -m_new)), exp2_fast(fmaf(s[2 * j + 1], sl2, -m_new)));
                    sum += __bfloat162float(pr.x) + __bfloat162float(pr.y);  // the rounded values: numerator and denominator agree
                    packed[j] = __uint_as_float(*reinterpret_cast<const uint32_t*>(&pr));
                }
                l_run = l_run * alpha + sum;
                m_use = m_new;
                if (i >= 1 && __any_sync(0xFFFFFFFFu, move)) {
                    // rescale this warp's 32 rows of O (256 columns) once every product issued so far is done; lanes that did
                    // not move multiply by 1
                    ok = pv_done(m - 1);
                    if (!ok) break;
                    fence_after();
#pragma unroll 1
                    for (int c = 0; c < MT_DH / 32; ++c) {
                        float o[32];
                        tmem_ld32(tmem_o + lane_addr + c * 32, o);
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] *= alpha;
                        tmem_st32(tmem_o + lane_addr + c * 32, o);
                    }
                    tmem_st_wait();
                } else if (i >= 1) {
                    ok = pv_done(m - 1);  // the product of the tile before has read its probabilities (long since: S came after it)
                    if (!ok) break;
                }
                if (valid < (uint32_t)MT_T) {
                    // the last tile: rows past the context's end hold whatever followed in the cache; zero them for P . L (the
                    // tile has landed, and S of this tile is done with it)
                    const uint32_t yt = MT_L_OFF + (m & 1) * MT_TILE + MT_XB * MT_BOX, n_zero = (MT_T - valid) * MT_YB * 8;  // (row, column block, 16-byte piece)
                    for (uint32_t z = row; z < n_zero; z += 128) {
                        const uint32_t piece = z & 7, cb = (z >> 3) % MT_YB, r = valid + (z >> 3) / MT_YB;
                        *reinterpret_cast<uint4*>(gen + yt + cb * MT_BOX + r * 128 + piece * 16) = make_uint4(0, 0, 0, 0);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic stores, read by the tensor core
                }
                tmem_st32(tmem + lane_addr + MT_TM_P, packed);  // the A operand of P . L
                tmem_st_wait();
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_PFULL));
            }
            // ---- the piece's output: final when it is the whole sequence, else unnormalised with maximum and sum -------------
            if (ok) ok = pv_done(n + nt - 1);
            if (ok) {
                fence_after();
                const uint32_t h = hb * MT_M + row, h_slot = min(p.n_heads, (uint32_t)MT_M);
                const bool whole = p.direct && nt == tiles_e;
                float* dst = whole ? p.out + ((size_t)b * p.n_heads + h) * MT_V : p.partial + ((size_t)(pair + e) * h_slot + row) * MT_ROW;
                const float f = whole ? 1.0f / l_run : 1.0f;
#pragma unroll 1
                for (int c = 0; c < MT_DH / 32; ++c) {
                    float o[32];
                    tmem_ld32(tmem_o + lane_addr + c * 32, o);  // every lane of the warp takes part, rows past n_heads just do not store
                    if (h < p.n_heads) {
#pragma unroll
                        for (int j = 0; j < 32; j += 8) {  // a lane's row is far from its neighbour's: whole 32-byte sectors per store
                            asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + dh * MT_DH + c * 32 + j), "f"(o[j] * f), "f"(o[j + 1] * f),
                                         "f"(o[j + 2] * f), "f"(o[j + 3] * f), "f"(o[j + 4] * f), "f"(o[j + 5] * f), "f"(o[j + 6] * f), "f"(o[j + 7] * f) : "memory");
                        }
                    }
                }
                if (!whole && dh == 0 && h < p.n_heads) { dst[MT_V] = m_use; dst[MT_V + 1] = l_run; }
            }
            fence_before();
        }
        n += nt;
        ++pieces;
        __syncthreads();  // the next piece overwrites Q, O and the tensor-memory part of Q
        fence_after();
        if (*abort_flag) break;
    }
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicOr(p.status, 1u);
        // let copies in flight land before the block (and its shared memory) goes away
        const long long t0 = clock64();
        while (clock64() - t0 < 20000000LL) {}
        __syncthreads();
    }
    if (warp == 3) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MT_TMEM_COLS) : "memory");
    }
}

// out[b][h][:] = sum over the pieces of the sequence of partial * 2^(m - M) / L; sequences of one piece are final already.
// grid (2 heads, B), 256 threads, four dimensions each.  Bound by latency: one trip for the entry's runs, which the main kernel
// left in `spans`, one for every four pieces (working the deal out here, a head a block: 20 us for 64 sequences of two pieces, 37 MB; now 13.7, cold).
__global__ void __launch_bounds__(256) k_mla_merge_tc(const MlaTcParams p) {
    const uint32_t h = blockIdx.x * 2 + (threadIdx.x >> 7), b = blockIdx.y, d4 = threadIdx.x & 127;
    pdl_wait();
    if (h >= p.n_heads) return;
    const uint32_t e = b * p.hbs + h / MT_M, status = *p.status, ctx = p.ctx_len[b];
    const uint2 span = p.spans[e];  // first and last run (written by them; stale for an empty sequence)
    float* o = p.out + ((size_t)b * p.n_heads + h) * MT_V + d4 * 4;
    if (status || ctx == 0) {
        // status: a wait in the tensor-core kernel ran out: the partials are not to be trusted, and the caller must see it
        o[0] = o[1] = o[2] = o[3] = status ? __int_as_float(0x7FC00000) : 0.0f;
        return;
    }
    if (p.direct && span.x == span.y) return;
    const size_t stride = (size_t)min(p.n_heads, (uint32_t)MT_M) * MT_ROW;
    const float* base = p.partial + (size_t)(span.x + e) * stride + (size_t)(h % MT_M) * MT_ROW;
    const uint32_t live = span.y - span.x + 1;
    float M = -INFINITY, L = 0.0f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t s0 = 0; s0 < live; s0 += 4) {
        float2 ml[4];
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ml[i] = make_float2(-INFINITY, 0.0f);
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s0 + i < live) {
                ml[i] = *reinterpret_cast<const float2*>(base + (s0 + i) * stride + MT_V);
                v[i] = *reinterpret_cast<const float4*>(base + (s0 + i) * stride + d4 * 4);
            }
        }
        const float Mn = fmaxf(M, fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x))), f = exp2f(M - Mn);
        M = Mn;
        L *= f; acc.x *= f; acc.y *= f; acc.z *= f; acc.w *= f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float w = exp2f(ml[i].x - Mn);
            L = fmaf(ml[i].y, w, L);
            acc.x = fmaf(v[i].x, w, acc.x); acc.y = fmaf(v[i].y, w, acc.y); acc.z = fmaf(v[i].z, w, acc.z); acc.w = fmaf(v[i].w, w, acc.w);
        }
    }
    const float inv = 1.0f / L;
    o[0] = acc.x * inv; o[1] = acc.y * inv; o[2] = acc.z * inv; o[3] = acc.w * inv;
}

// q fp32 [B][n_heads][576] -> bf16 [B][rows_per_seq][576] (times sign), rows past n_heads zero; eight elements a thread
__global__ void __launch_bounds__(256)
k_mla_q_bf16(uint4* __restrict__ dst, const float* __restrict__ q, uint32_t n_heads, uint32_t rows_per_seq, uint32_t n8, float sign, uint32_t* status) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i == 0) *status = 0u;
    if (i >= n8) return;
    const uint32_t row = i / (MT_LAT / 8), c = i % (MT_LAT / 8), b = row / rows_per_seq, r = row % rows_per_seq;
    uint32_t v[4] = {0u, 0u, 0u, 0u};
    if (r < n_heads) {
        const float2* src = reinterpret_cast<const float2*>(q + ((size_t)b * n_heads + r) * MT_LAT + c * 8);  // (q is 8-byte aligned)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = src[k];
            const __nv_bfloat162 h = __floats2bfloat162_rn(f.x * sign, f.y * sign);
            v[k] = *reinterpret_cast<const uint32_t*>(&h);
        }
    }
    dst[i] = make_uint4(v[0], v[1], v[2], v[3]);
}

// bf16 [rows][576] row-major, boxes of [box_rows][64 columns], 128-byte swizzle, zeros outside the matrix
bool make_map_bf16(CUtensorMap* m, const void* ptr, uint64_t rows, uint32_t box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {MT_LAT, rows};
    const cuuint64_t strides[1] = {MT_LAT * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

static uint32_t mla_min_tiles(uint32_t split_tokens) { return split_tokens ? (split_tokens + MT_T - 1) / MT_T : 4; }
// Contexts end where the mma.sync kernel's last slice does: max_ctx in whole slices of split_tokens (0: 1024).
static uint64_t mla_max_rows(uint32_t max_ctx, uint32_t split_tokens) {
    const uint64_t slice = split_tokens ? split_tokens : 1024;
    return (max_ctx + slice - 1) / slice * slice;
}
static uint64_t mla_total_tiles(uint32_t batch, uint32_t hbs, uint32_t max_ctx, uint32_t split_tokens) {
    return (uint64_t)batch * hbs * ((mla_max_rows(max_ctx, split_tokens) + MT_T - 1) / MT_T);
}

uint64_t mla_tc_extra_scratch_bytes(uint32_t batch, uint32_t n_heads) {
    const uint64_t rows = (uint64_t)((n_heads + MT_M - 1) / MT_M) * MT_M;
    return 1024 + (uint64_t)batch * rows * MT_LAT * 2 + (uint64_t)batch * (rows / MT_M) * sizeof(uint2);
}

// pieces: one per run of tiles and per (sequence, block of heads) at most
uint64_t mla_tc_partial_bytes(uint32_t batch, uint32_t n_heads, uint32_t max_ctx, uint32_t split_tokens) {
    const uint32_t hbs = (n_heads + MT_M - 1) / MT_M;
    const uint64_t entries = (uint64_t)batch * hbs, m = mla_min_tiles(split_tokens), runs = (mla_total_tiles(batch, hbs, max_ctx, split_tokens) + m - 1) / m, slots = (runs < MT_PAIRS ? runs : MT_PAIRS) + entries;
    return slots * (n_heads < (uint32_t)MT_M ? n_heads : (uint32_t)MT_M) * MT_ROW * 4 + 32;
}

// extra: the area of mla_tc_extra_scratch_bytes (16-byte aligned): a status word, then Q in bf16, then the entries' spans
cudaError_t mla_decode_tc(const LaunchCfg& lc, float* out, const float* q, const void* cache, const uint32_t* ctx_len, float* partial, void* extra,
                          uint32_t batch, uint32_t n_heads, uint32_t max_ctx, uint32_t split_tokens, uint64_t cache_stride, float scale) {
    static std::atomic<uint64_t> opted{0};
    cudaError_t e = once_per_device(opted, []() { return cudaFuncSetAttribute(k_mla_decode_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM); });
    if (e != cudaSuccess) return e;
    const uint32_t hbs = (n_heads + MT_M - 1) / MT_M, rows_per_seq = hbs * MT_M;
    uint32_t* status = reinterpret_cast<uint32_t*>(extra);
    __nv_bfloat16* q16 = reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<unsigned char*>(extra) + 1024);
    CUtensorMap mq, ml;
    if (!make_map_bf16(&mq, q16, (uint64_t)batch * rows_per_seq, MT_M) || !make_map_bf16(&ml, cache, (uint64_t)batch * cache_stride, MT_T))
        return cudaErrorNotSupported;
    MlaTcParams p = {};
    p.ctx_len = ctx_len; p.out = out; p.q16 = q16; p.status = status;
    p.partial = reinterpret_cast<float*>(((uintptr_t)partial + 31) & ~(uintptr_t)31);  // (the scratch is 16-byte aligned)
    p.spans = reinterpret_cast<uint2*>(q16 + (size_t)batch * rows_per_seq * MT_LAT);
    p.n_seq = batch; p.n_heads = n_heads; p.hbs = hbs; p.q_rows_per_seq = rows_per_seq;
    p.min_tiles = mla_min_tiles(split_tokens);
    p.direct = ((uintptr_t)out & 31) == 0 ? 1u : 0u;
    p.cache_stride = cache_stride; p.scale = scale == 0.0f ? 1e-30f : fabsf(scale);  // the sign goes into q; 0 would turn masked scores into NaN
    const uint64_t max_rows = mla_max_rows(max_ctx, split_tokens), runs = (mla_total_tiles(batch, hbs, max_ctx, split_tokens) + p.min_tiles - 1) / p.min_tiles;
    p.max_rows = max_rows < 0xFFFFFFC0ull ? (uint32_t)max_rows : 0xFFFFFFC0u;
    const uint32_t n8 = batch * rows_per_seq * (MT_LAT / 8);
    LaunchCfg chained = lc;  // each of the three starts its prologue while the one before it runs
    chained.pdl = true;
    if ((e = launch(lc, k_mla_q_bf16, dim3((n8 + 255) / 256), dim3(256), 0, reinterpret_cast<uint4*>(q16), q, n_heads, rows_per_seq, n8, scale < 0.0f ? -1.0f : 1.0f, status)) != cudaSuccess) return e;
    if ((e = launch(chained, k_mla_decode_tc, dim3(2 * (unsigned)(runs < MT_PAIRS ? runs : MT_PAIRS)), dim3(MT_THREADS), MT_SMEM, mq, ml, p)) != cudaSuccess) return e;
    return launch(chained, k_mla_merge_tc, dim3((n_heads + 1) / 2, batch), dim3(256), 0, p);
}

}  // namespace vb
